"""NaN, infinities, signed zeros and the ends of the range in the operands that
the flux and matrix kernels compare or shortcut: velocities, volumes, areas and
densities."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from asam_gb300 import TransportBlock, ros_coeffs
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _case(periodic):
    nx, ny, nz = 7, 6, 5
    rng = np.random.default_rng(5 + periodic)
    grid = G.Grid(nx, ny, nz, 100.0, 130.0, G.stretched_levels(nz, 50.0, 90.0), periodic, periodic, False)
    geo = G.cut_cell_geometry(grid, rng.uniform(0.0, 60.0, (ny, nx)))
    vel = [np.array(v) for v in G.closed_face_velocity(geo, 3.0, seed=1)]
    c = oracle.Oracle(geo).exchange_cell(rng.uniform(0.5, 1.5, (3,) + grid.pshape))
    return rng, geo, vel, c


def _fcn(geo, vel, c, precision):
    with TransportBlock(geo, c.shape[0], precision=precision) as blk:
        blk.set_velocity(*vel)
        return blk.Fcn(c)


@pytest.mark.parametrize("precision", ["fp64", "fp32_refined"])
@pytest.mark.parametrize("nan", [np.nan, -np.nan])
@pytest.mark.parametrize("periodic", [True, False])
def test_face_with_a_nan_velocity_has_no_flux(built_lib, periodic, nan, precision):
    """NaN flows in neither direction, so the faces give what resting ones give."""
    rng, geo, vel, c = _case(periodic)
    rest = [v.copy() for v in vel]
    for v, r in zip(vel, rest):
        inner = v[1:-1, 1:-1, 1:-1]  # off the walls, whose inflow is not a comparison
        hit = rng.random(inner.shape) < 0.2
        inner[hit] = nan
        r[1:-1, 1:-1, 1:-1][hit] = 0.0
    np.testing.assert_array_equal(_fcn(geo, vel, c, precision), _fcn(geo, rest, c, precision))


@pytest.mark.parametrize("value", [np.nan, -np.nan, -0.0, 0.0])
@pytest.mark.parametrize("periodic", [True, False])
def test_volumes_that_compare_false(built_lib, periodic, value):
    """Neither a NaN volume nor a negative zero next to zero is the smaller one."""
    rng, geo, vel, c = _case(periodic)
    inner = geo.volc[1:-1, 1:-1, 1:-1]
    inner[rng.random(inner.shape) < 0.2] = 0.0
    inner[rng.random(inner.shape) < 0.2] = value
    np.testing.assert_array_equal(_fcn(geo, vel, c, "fp64"), oracle.Oracle(geo).fcn(c, vel))


@pytest.mark.parametrize("where", ["velocity", "density", "area", "volume"])
@pytest.mark.parametrize("periodic", [True, False])
def test_matrix_of_special_operands(built_lib, periodic, where):
    """The terms that the direction of the flow makes 0 are so only for
    ordinary areas, volumes and densities: 0*inf, 0/0 and NaN elsewhere."""
    rng, geo, vel, c = _case(periodic)
    values = [np.nan, np.inf, -np.inf, 0.0, -0.0, 1.5e308, -1.5e308, 5e-324, -1e-30, -1.0]
    for a in {"velocity": vel, "density": [c[0]], "area": [geo.fu, geo.fv, geo.fw], "volume": [geo.volc]}[where]:
        hit = rng.random(a.shape) < 0.2
        a[hit] = rng.choice(values, hit.sum())
    for v in vel if where != "velocity" else []:  # both signs and rest
        v[...] = rng.choice([0.0, 1.0, -1.0], v.shape) * rng.uniform(0.5, 2.0, v.shape)
    with TransportBlock(geo, c.shape[0]) as blk:
        blk.set_velocity(*vel)
        blk.Jac(c, 2.0)
        got = blk.jac_matrix()
    want = oracle.Oracle(geo).jac(c[0], vel, ros_coeffs("RosRK3")[1], 2.0)
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 0.0, 2.0 ** -46, 2.0 ** -45, -1.0, 1e-30, 5e-324])
def test_momentum_sources_of_special_areas(built_lib, value):
    """F/(F+Eps) is 1 for finite areas from 2^-45 on only."""
    geo, vel, st, pos, (dx, dy, dz), bound = G.hill_dyn_case(7, 6, 5, seed=3)
    rng = np.random.default_rng(3)
    vel = [np.zeros_like(v) for v in vel]  # the sources alone
    for a in (geo.fu, geo.fv, geo.fw):
        a[...] = rng.uniform(0.5, 2.0, a.shape)
        a[rng.random(a.shape) < 0.2] = value
    pre = rng.uniform(8e4, 1e5, geo.grid.pshape)
    with TransportBlock(geo, st.c.shape[0]) as blk:
        blk.set_velocity(*vel)
        blk.proj_setup(dx, dy, dz)
        blk.dyn_setup(pos["th"], pos["mom"], rv_pos=pos.get("qv", -1), bound_cells=bound)
        got = blk.FcnMet(st.c, pre)
    if np.isfinite(value):
        want = oracle.Oracle(geo).fcn_dyn(st.c, vel, pre, pos["mom"], dx, dy, dz)
        for q in pos["mom"]:
            np.testing.assert_array_equal(got[q], want[q])
        return
    # (the oracle's flux over such a face is 0*inf as well; a resting face inside the block has none here, while
    # the inflow through the outer walls is |u| - u times the area)
    nx, ny, nz = 7, 6, 5
    grid = geo.grid
    wall = np.zeros((nz, ny, nx), dtype=bool)
    for axis, F, periodic in ((2, geo.fu, grid.periodic_x), (1, geo.fv, grid.periodic_y), (0, geo.fw, grid.periodic_z)):
        if periodic:
            continue
        w, F = np.moveaxis(wall, axis, -1), np.moveaxis(F, axis, -1)
        w[..., 0] |= ~np.isfinite(F[..., 1])
        w[..., -1] |= ~np.isfinite(F[..., w.shape[-1] + 1])
    for comp, F in ((1, geo.fu[:, :, 2:nx + 1]), (3, geo.fv[:, 2:ny + 1]), (5, geo.fw[2:nz + 1])):
        box = tuple(slice(0, m) for m in F.shape)
        g = got[pos["mom"][comp]][1:-1, 1:-1, 1:-1][box]
        with np.errstate(invalid="ignore"):
            np.testing.assert_array_equal(np.isnan(g), np.isnan(F / (F + 1e-30)) | wall[box])
