"""The gather of the face fluxes on both sides of the size from which the cells
off the sides have a kernel of their own, with every source that it takes, bit
for bit against the oracle."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import oracle
from asam_gb300 import TransportBlock
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu

# 38912 padded cells are what 152 SMs hold at once: exactly those, a plane more,
# and boxes above it with none, one or few cells off the sides along an axis
SIZES = [(30, 30, 36), (30, 30, 37), (2, 100, 100), (100, 2, 100), (100, 100, 2), (3, 80, 100), (80, 3, 100),
         (100, 80, 3), (100, 4, 70)]


@pytest.mark.parametrize("diffusion", [False, True])
@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_advection(built_lib, nx, ny, nz, periodic, diffusion):
    rng = np.random.default_rng(nx + ny + nz)
    grid = G.Grid(nx, ny, nz, 100.0, 130.0, G.stretched_levels(nz, 50.0, 90.0), periodic, periodic, False)
    geo = G.cut_cell_geometry(grid, rng.uniform(0.0, 60.0, (ny, nx)))
    vel = G.closed_face_velocity(geo, 3.0, seed=1)
    o = oracle.Oracle(geo)
    c = o.exchange_cell(rng.uniform(0.5, 1.5, (3,) + grid.pshape))
    with TransportBlock(geo, 3) as blk:
        blk.set_velocity(*vel)
        if diffusion:
            coefs = G.diffusion_coefficients(geo, c[0])
            blk.set_diffusion(*coefs)
            o.set_diffusion(*coefs)
        got = blk.Fcn(c)
    np.testing.assert_array_equal(got, o.fcn(c, vel))


@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_momentum_sources(built_lib, nx, ny, nz):
    geo, vel, st, pos, (dx, dy, dz), bound = G.hill_dyn_case(nx, ny, nz, seed=3)
    o = oracle.Oracle(geo)
    _, pre = o.thermo(st.c, 0, pos["th"], rv_pos=pos.get("qv", -1))
    with TransportBlock(geo, st.c.shape[0]) as blk:
        blk.set_velocity(*vel)
        blk.proj_setup(dx, dy, dz)
        blk.dyn_setup(pos["th"], pos["mom"], rv_pos=pos.get("qv", -1), bound_cells=bound)
        got = blk.FcnMet(st.c, pre)
    np.testing.assert_array_equal(got, o.fcn_dyn(st.c, vel, pre, pos["mom"], dx, dy, dz))


@pytest.mark.parametrize("nx,ny,nz,launches", [(24, 24, 16, 1), (30, 30, 36, 1), (30, 30, 37, 2)])
def test_small_blocks_take_one_launch(built_lib, nx, ny, nz, launches):
    """The gather's launches beside phi and the three face fluxes, on a GPU of 152 SMs."""
    geo, vel, st = G.hill_case(nx, ny, nz, seed=2)
    with TransportBlock(geo, st.c.shape[0]) as blk:
        blk.set_velocity(*vel)
        count = lambda: ctypes.c_longlong(blk.lib.asam_launch_count()).value  # noqa: E731
        blk.Fcn(st.c)
        n0 = count()
        blk.Fcn(st.c)
        assert count() - n0 == 4 + launches
