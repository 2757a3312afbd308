"""The FP32 product and its dot products, seen through the first pass of the
refinement: its BiCGStab runs on them alone, and the FP64 residual of the
correction is the returned one when it already meets the tolerance."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
import tests.pyref as pyref
from asam_gb300 import TransportBlock
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _bicgstab(o, grid, val, b, tol):
    """One run from 0 in FP64, with the x-line preconditioner: (iterations, the
    norm of the residual of its x, that of b, the smallest distance of a norm to
    the limit)."""
    inner = (slice(None), slice(1, -1), slice(1, -1), slice(1, -1))
    dot = lambda x, y: float((x[inner] * y[inner]).sum())  # noqa: E731

    def precond(r):
        x = pyref.line_solve(val, grid, r, 0).reshape(b.shape)
        x[:, [0, -1]] = x[:, :, [0, -1]] = x[..., [0, -1]] = 0.0
        return x

    matvec = lambda x: o.matvec(val, x).reshape(b.shape)  # noqa: E731
    r, rt, p, x = b.copy(), b.copy(), b.copy(), np.zeros_like(b)
    n0, gap = dot(b, b) ** 0.5, np.inf
    rho = dot(rt, r)
    for it in range(1, 30):
        if it > 1:
            old, rho = rho, dot(rt, r)
            p = r + rho / old * alpha / omega * (p - omega * v)
        ph = precond(p)
        v = matvec(ph)
        alpha = rho / dot(rt, v)
        r = r - alpha * v
        x = x + alpha * ph
        for half in (0, 1):
            if half:
                rh = precond(r)
                t = matvec(rh)
                omega = dot(t, r) / dot(t, t)
                r = r - omega * t
                x = x + omega * rh
            rel = dot(r, r) ** 0.5 / n0
            gap = min(gap, abs(rel / tol - 1.0))
            if rel <= tol:
                res = b - matvec(x)
                return it, dot(res, res) ** 0.5, n0, gap
    raise AssertionError("no convergence")


# Couplings of one sign and row sums of 0.75, so that the step lengths are far
# from 1.  Rounding: some ten roundings of 2^-24 an entry, product and update, a
# dozen passes: below 1e-5 of |b|.  A coupling missed in one cell alone moves the
# residual by 5e-5 of |b| or more at these sizes, a wrong step length by far more.
# Padded widths 4, 17, 18, 34, 259: products of two cells and of one cell a thread.
@pytest.mark.parametrize("nx,ny,nz,ncomp", [(2, 3, 4, 1), (2, 4, 1, 2), (15, 6, 5, 10), (16, 6, 5, 10), (16, 1, 7, 3),
                                            (32, 9, 2, 3), (257, 4, 3, 10)])
def test_first_refinement_pass(built_lib, nx, ny, nz, ncomp):
    grid = G.Grid(nx, ny, nz, 100.0, 100.0, G.uniform_levels(nz, 100.0), False, False, False)
    geo = G.cut_cell_geometry(grid, None)
    o = oracle.Oracle(geo)
    tol = 1e-2
    for seed in range(100):  # a system whose norms stay off the limit, and whose residual is not tiny
        rng = np.random.default_rng(seed)
        val = rng.uniform(0.05, 0.2, (7, grid.npad))
        val[3] = rng.uniform(1.0, 1.5, grid.npad)
        v = val.reshape((7,) + grid.pshape)
        for d, axis, side in ((0, 1, -1), (6, 1, 0), (1, 2, -1), (5, 2, 0), (2, 3, -1), (4, 3, 0)):
            w = np.moveaxis(v, axis, -1)  # the halo cells couple to nothing: column d of the last interior cell too
            w[d, ..., side] = w[d, ..., side - 1 if side else 1] = w[d, ..., 0 if side else -1] = 0.0
        b = np.zeros((ncomp,) + grid.pshape)
        b[:, 1:-1, 1:-1, 1:-1] = rng.standard_normal((ncomp, nz, ny, nx))
        it, want, n0, gap = _bicgstab(o, grid, val, b, 0.5 * tol)  # the limit of the first inner solve
        if gap > 0.05 and want > 1e-3 * n0:
            break
    else:
        raise AssertionError("no such system")
    with TransportBlock(geo, ncomp, precision="fp32_refined", inner_precond="xline") as blk:
        blk.set_jac_matrix(val)
        x = np.zeros_like(b)
        iters, resid = blk.BiCGStabMetSp(x, b, 30, tol)
    assert iters == it
    assert abs(resid - want) <= 2e-5 * n0
