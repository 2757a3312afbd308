"""The two FP32 x-line kernels give the same bits: a box whose rows fit shared
memory against one with the same rows, cut off from the rest of rows that do
not fit."""
from __future__ import annotations

import numpy as np
import pytest

from asam_gb300 import TransportBlock
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _solve(nx, val, b):
    """val (7, nz+2, ny+2, nx+2), b (ncomp, ...): the preconditioned b."""
    ny, nz = b.shape[2] - 2, b.shape[1] - 2
    grid = G.Grid(nx, ny, nz, 100.0, 100.0, G.uniform_levels(nz, 100.0), False, False, False)
    with TransportBlock(G.cut_cell_geometry(grid, None), b.shape[0], precision="fp32_refined",
                        inner_precond="xline") as blk:
        blk.set_jac_matrix(val.reshape(7, -1))
        return blk.inner_psolve(b)


@pytest.mark.parametrize("nx", [1, 5, 6, 7, 30, 255])
def test_rows_in_shared_memory_against_chunks(built_lib, nx, ny=2, nz=2, ncomp=10, far=4700):
    rng = np.random.default_rng(nx)
    val = np.zeros((7, nz + 2, ny + 2, far + 2))
    val[3] = rng.uniform(1.0, 4.0, val[3].shape)
    for d in (2, 4):  # columns i of rows i+1 and i-1
        val[d, ..., :nx + 2] = rng.uniform(-0.3, 0.3, val[d, ..., :nx + 2].shape)
    val[2, ..., nx + 1] = val[4, ..., 0] = 0.0  # nothing leaves the first nx+2 cells
    b = rng.standard_normal((ncomp, nz + 2, ny + 2, far + 2))
    long = _solve(far, val, b)
    short = _solve(nx, np.ascontiguousarray(val[..., :nx + 2]), np.ascontiguousarray(b[..., :nx + 2]))
    assert np.any(short[..., 1:nx + 1])
    np.testing.assert_array_equal(short[..., 1:nx + 1], long[..., 1:nx + 1])
