"""The FP64 Gauss-Seidel tiles against the oracle's lexicographic sweeps, bit
for bit: boxes that end inside, at and just beyond a tile, component counts on
both sides of every grouping, zero couplings and zero right-hand sides."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from asam_gb300 import TransportBlock
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu


# padded widths nx+2: 16 (one tile), 15, 17, 33; 4 x 4 lines likewise in y and z
@pytest.mark.parametrize("nx,ny,nz,ncomp", [(14, 2, 2, 1), (13, 3, 5, 2), (15, 1, 6, 3), (31, 6, 3, 8), (32, 9, 10, 9),
                                            (1, 1, 1, 5), (47, 14, 13, 16)])
def test_psolve_bitwise(built_lib, nx, ny, nz, ncomp):
    grid = G.Grid(nx, ny, nz, 100.0, 100.0, G.uniform_levels(nz, 100.0))
    geo = G.cut_cell_geometry(grid, None)
    rng = np.random.default_rng(nx * 100 + ncomp)
    val = rng.uniform(-0.3, 0.3, (7, grid.npad))
    val[3] = rng.uniform(1.0, 4.0, grid.npad)
    val[:3][rng.random((3, grid.npad)) < 0.2] = 0.0
    val[4:][rng.random((3, grid.npad)) < 0.2] = 0.0
    # no coupling leaves the box (slot m of a column acts on the row m away: the
    # flat storage would wrap it into the next line)
    v = val.reshape((7,) + grid.pshape)
    v[2, :, :, -1] = v[4, :, :, 0] = v[1, :, -1] = v[5, :, 0] = v[0, -1] = v[6, 0] = 0.0
    b = rng.standard_normal((ncomp,) + grid.pshape)
    b[:, : (nz + 2) // 2] *= rng.random((ncomp, (nz + 2) // 2, ny + 2, nx + 2)) < 0.5
    with TransportBlock(geo, ncomp) as blk:
        blk.set_jac_matrix(val)
        np.testing.assert_array_equal(blk.PSolve(b), oracle.Oracle(geo).psolve(val, b))
