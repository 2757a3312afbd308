"""The plane solves of the multigrid with their coarse plane levels resident in
shared memory: sizes for which all, some or few of the levels fit, odd rows
and lines, more planes than SMs, closed and periodic sides, against the
oracle's zebra order bit for bit (FP64) and against the FP64 result (FP32)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from asam_gb300 import TransportBlock
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu

# (nx, ny, nz): lines x planes x rows of the finest plane level
SIZES = [(33, 4, 33),    # whole plane resident, odd rows and lines, two warps of lines
         (64, 3, 32),    # whole plane resident, just below the limit
         (100, 6, 48),   # the finest plane level streams, the others resident
         (101, 5, 49),   # the same with odd sizes
         (301, 4, 99),   # two streaming levels, more lines than threads take at once in the ring's first warps
         (12, 310, 10),  # more planes of one parity than SMs: two CTAs per SM
         (3, 2, 150)]    # long columns, two lines


def _geometry(nx, ny, nz, periodic):
    if not periodic:
        return G.closed_hill_case(nx, ny, nz, seed=nx + nz)
    grid = G.Grid(nx, ny, nz, 200.0, 200.0, G.stretched_levels(nz, 50.0, 400.0))
    return G.close_dead_faces(G.cut_cell_geometry(grid, G.gaussian_hill_terrain(grid, 600.0, 800.0, 50.0, 600.0,
                                                                                 seed=nx + nz)))


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_vcycle_bitwise(built_lib, nx, ny, nz, periodic):
    geo = _geometry(nx, ny, nz, periodic)
    W, dx, dy, dz, _ = G.projection_inputs(geo, seed=3)
    o = oracle.OracleProj(geo, dx, dy, dz, W, zebra=1)
    o.lapl_compute(0.435866521508459, 2.0)
    rng = np.random.default_rng(nx * ny)
    b = rng.standard_normal((nz, ny, nx))
    with TransportBlock(geo, 3) as blk:
        blk.proj_setup(dx, dy, dz)
        blk.proj_weights(*W)
        blk.JacAccGrav(0.435866521508459, 2.0)
        np.testing.assert_array_equal(blk.VCycleCG(b), o.vcycle(b))
        if periodic:
            x = rng.standard_normal(o.nvec)
            np.testing.assert_array_equal(blk.PSolve1(x), o.psolve1(x))


@pytest.mark.parametrize("kind", ["closed", "psolve1", "periodic"])
@pytest.mark.parametrize("nx,ny,nz", SIZES[:5])
def test_fp32_vcycle_close_to_fp64(built_lib, nx, ny, nz, kind):
    """The FP32 cycle runs some 2^7 dependent relaxations, each contracting:
    2^7 roundings of 2^-24 with a factor 16 for the unevenly scaled rows."""
    geo = _geometry(nx, ny, nz, kind != "closed")
    W, dx, dy, dz, _ = G.projection_inputs(geo, seed=3)
    live = geo.volc[1:-1, 1:-1, 1:-1].reshape(-1) > 0
    out = []
    for prec in ("fp64", "fp32"):
        with TransportBlock(geo, 3) as blk:
            blk.proj_setup(dx, dy, dz)
            if kind != "closed":
                blk.proj_set_preconditioner(kind)
            blk.proj_set_precision(prec)
            blk.proj_weights(*W)
            blk.JacAccGrav(0.435866521508459, 2.0)
            x = np.zeros(blk.proj_nvec)
            # cells without volume have a zero right-hand side in the projection
            x[:live.size] = np.random.default_rng(7).standard_normal(live.size) * live
            out.append(np.asarray(blk.PSolve1(x)).reshape(-1)[:live.size][live])
    err = np.abs(out[1] - out[0]).max() / np.abs(out[0]).max()
    assert err <= 2.0 ** 7 * 2.0 ** -24 * 16
