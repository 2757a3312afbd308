"""FP64 BiCGStab against the oracle at row widths on both sides of those that the
update-and-norm pass takes in one piece less with more cells a lane."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from asam_gb300 import TransportBlock
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu


# padded widths 128 | 129 .. 160 | 161 and 256 | 257 .. 320 | 321
@pytest.mark.parametrize("nx", [126, 127, 150, 158, 159, 254, 255, 318, 319])
def test_row_widths(built_lib, nx, ny=3, nz=2, ncomp=3):
    grid = G.Grid(nx, ny, nz, 100.0, 100.0, G.uniform_levels(nz, 100.0))
    geo = G.cut_cell_geometry(grid, None)
    o = oracle.Oracle(geo)
    rng = np.random.default_rng(nx)
    val = rng.uniform(-0.15, 0.15, (7, grid.npad))
    val[3] = rng.uniform(1.0, 2.0, grid.npad)
    v = val.reshape((7,) + grid.pshape)  # no coupling leaves the box
    v[2, :, :, -1] = v[4, :, :, 0] = v[1, :, -1] = v[5, :, 0] = v[0, -1] = v[6, 0] = 0.0
    b = o.exchange_cell(rng.standard_normal((ncomp,) + grid.pshape))
    want, got = np.zeros_like(b), np.zeros_like(b)
    o.bicgstab_halfsteps(val, want, b, 4)
    with TransportBlock(geo, ncomp) as blk:
        blk.set_jac_matrix(val)
        iters, resid = blk.BiCGStabMetSp(got, b, 2, 1e-300)
        assert iters == 4  # the limit, after both halves of two iterations
    # the sums of the dot products in another order: some 1e-15, amplified a hundredfold at most in four half-steps
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
