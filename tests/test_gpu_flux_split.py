"""The flux right-hand side bit for bit against the oracle where its kernels
split and shortcut: blocks with no, one or few cells off the sides, and fields
whose differences are zero, next to Eps, subnormal or huge."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from asam_gb300 import TransportBlock
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _fields(rng, shape):
    """Component values over a density of 1: smooth, constant, steps of the
    size of Eps, the 2^-45 below which Eps counts, subnormal and huge values."""
    out = [np.ones(shape), rng.standard_normal(shape), np.full(shape, 0.25), 1e-30 * rng.integers(-3, 4, shape),
           2.0 ** -45 * rng.integers(-2, 3, shape) * (1 + 2.0 ** -52 * rng.integers(-2, 3, shape)),
           5e-324 * rng.integers(0, 9, shape), 1e200 * rng.standard_normal(shape),
           rng.standard_normal(shape) * 10.0 ** rng.integers(-200, 1, shape)]
    return np.ascontiguousarray(np.stack(out))


@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 1), (2, 2, 2), (3, 3, 3), (3, 2, 5), (4, 1, 3), (5, 3, 4), (33, 4, 3)])
def test_flux_bitwise(built_lib, nx, ny, nz, periodic):
    rng = np.random.default_rng(10 * nx + ny + periodic)
    grid = G.Grid(nx, ny, nz, 100.0, 130.0, G.stretched_levels(nz, 50.0, 90.0), periodic, periodic, False)
    h = rng.uniform(0.0, 60.0, (ny, nx))
    geo = G.cut_cell_geometry(grid, h)
    vel = G.closed_face_velocity(geo, 3.0, seed=nx + nz)
    c = _fields(rng, grid.pshape)
    o = oracle.Oracle(geo)
    c = o.exchange_cell(c)
    with TransportBlock(geo, c.shape[0]) as blk:
        blk.set_velocity(*vel)
        np.testing.assert_array_equal(blk.Fcn(c), o.fcn(c, vel))
