"""The FP32 x-line solve against a tridiagonal solve in FP64: rows shorter and
longer than the register batches, last CTAs with fewer rows, component counts
on both sides of a warp, and rows too long for shared memory."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import tests.pyref as pyref
from asam_gb300 import TransportBlock
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu

# Off-diagonal entries of at most 0.3 each against a diagonal of at least 1:
# every rounding (2^-24, three a row each way) is damped by 0.3/(1 - 0.3) a row
# and the solution is at most 2.5 times the right-hand side, so 2.5 * 6 * 2^-24
# / (1 - 0.43)^2 < 3e-6 of the largest value.
TOL = 1e-5


def _matrix(rng, grid):
    val = rng.uniform(-0.3, 0.3, (7, grid.npad))
    val[3] = rng.uniform(1.0, 4.0, grid.npad)
    v = val.reshape((7,) + grid.pshape)  # no coupling leaves the box
    v[2, :, :, -1] = v[4, :, :, 0] = v[1, :, -1] = v[5, :, 0] = v[0, -1] = v[6, 0] = 0.0
    return val


@pytest.mark.parametrize("nx,ny,nz,ncomp", [(1, 1, 1, 1), (5, 3, 4, 16), (6, 30, 20, 10), (7, 40, 36, 3), (8, 2, 2, 7),
                                            (32, 5, 41, 1), (255, 50, 30, 10), (1100, 3, 2, 16), (4700, 1, 2, 10)])
def test_x_lines(built_lib, nx, ny, nz, ncomp):
    grid = G.Grid(nx, ny, nz, 100.0, 100.0, G.uniform_levels(nz, 100.0))
    geo = G.cut_cell_geometry(grid, None)
    rng = np.random.default_rng(nx * 100 + ncomp)
    val = _matrix(rng, grid)
    b = rng.standard_normal((ncomp,) + grid.pshape)
    o = oracle.Oracle(geo)
    x = pyref.line_solve(val, grid, o.exchange_cell(b), 0).reshape(b.shape)
    x[:, [0, -1]] = x[:, :, [0, -1]] = x[..., [0, -1]] = 0.0
    x = o.exchange_cell(x)
    with TransportBlock(geo, ncomp, precision="fp32_refined", inner_precond="xline") as blk:
        blk.set_jac_matrix(val)
        got = blk.inner_psolve(b)
    assert np.abs(got - x).max() <= TOL * np.abs(x).max()


# padded widths 4, 17, 18, 259: products of two cells and of one cell a thread
@pytest.mark.parametrize("nx,ny,nz", [(2, 3, 4), (15, 6, 5), (16, 6, 5), (257, 4, 3)])
def test_refined_step(built_lib, nx, ny, nz):
    """Both precisions solve the stage systems to 1e-12 of the right-hand side;
    the stage matrices of a short step are I + O(1), so the states agree to a
    few hundred times that."""
    geo, vel, st = G.hill_case(nx, ny, nz, seed=nx)
    out = []
    for precision, kw in (("fp64", {}), ("fp32_refined", {"inner_precond": "xline"})):
        c = st.c.copy()
        with TransportBlock(geo, c.shape[0], bicgstab_tol=1e-12, precision=precision, **kw) as blk:
            blk.set_velocity(*vel)
            blk.Ros3MetC(c, 1.0)
        out.append(c)
    for a, b in zip(out[1], out[0]):
        assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max()
