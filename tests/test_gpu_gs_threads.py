"""The FP32 Gauss-Seidel kernels from several host threads whose contexts take
different shared-memory sizes (components per CTA): the size that a kernel may
take is a setting of the kernel, not of the thread."""
from __future__ import annotations

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from asam_gb300 import Batch, TransportBlock
from asam_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def _case(ncomp):
    geo, vel, st = G.hill_case(20, 14, 10, seed=3)
    c = np.ascontiguousarray(np.concatenate([st.c] * 2)[:ncomp])
    return geo, vel, c


@pytest.mark.parametrize("sched", ["persistent", "levels"])
def test_threads_with_other_group_sizes(built_lib, sched):
    geo, vel, c = _case(16)
    with TransportBlock(geo, 16, precision="fp32_refined", gs_schedule=sched, gs_group=16) as wide, \
            TransportBlock(geo, 16, precision="fp32_refined", gs_schedule=sched, gs_group=8) as narrow, \
            ThreadPoolExecutor(1) as one, ThreadPoolExecutor(1) as two:
        for blk in (wide, narrow):
            blk.set_velocity(*vel)
            blk.Jac(c, 2.0)
        want = one.submit(wide.inner_psolve, c).result()
        for _ in range(2):
            assert np.array_equal(two.submit(narrow.inner_psolve, c).result(), want)
            assert np.array_equal(one.submit(wide.inner_psolve, c).result(), want)


@pytest.mark.parametrize("sched", ["persistent", "levels"])
def test_batch_with_other_group_sizes(built_lib, sched):
    geo, vel, c0 = _case(16)
    groups = (16, 8, 16, 5)
    blocks = [TransportBlock(geo, 16, bicgstab_tol=1e-8, precision="fp32_refined", gs_schedule=sched, gs_group=g)
              for g in groups]
    for blk in blocks:
        blk.set_velocity(*vel)
        blk.set_graphs(0)  # every launch from its worker
    states = [c0.copy() for _ in groups]
    with Batch(blocks, nthreads=2) as batch:
        _, status = batch.ros_step(states, 2.0, nsteps=3)
    assert not any(status)
    for s in states[1:]:
        assert np.array_equal(s, states[0])
    for blk in blocks:
        blk.close()
