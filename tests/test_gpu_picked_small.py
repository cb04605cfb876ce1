"""Groups of few requests of nvshmemx_batch_execute_picked take the route of
nvshmemx_batch_execute, by which the variants are timed: one launch, whose error
reaches the call's status."""
import numpy as np
import pytest
import torch

from nvshmem_b200 import DT_INT, ERR_NOMEM, REQ_PUT
from nvshmem_b200 import picker as P
from test_gpu_picker_runtime import _picker
from _util import heap_images, requests

pytestmark = pytest.mark.gpu

NPES, HEAP = 2, 8 << 20
VARIANT = 8  # 3 x 8 KiB rings, 8 warps to a CTA


class Handle:
    """One-class table where only VARIANT was measured: every group runs it."""

    def __init__(self):
        tt = np.full((1, 12), np.nan, np.float32)
        tt[0, VARIANT] = 1.0
        self.net = P.MLP(seed=1)
        self.h, self.keep = _picker(self.net, np.full((1, 6), 100.0, np.float32), tt)


def rows(n, nbytes):
    return requests([dict(src_off=16 * k, dst_off=HEAP // 2 + k * nbytes, bytes=nbytes, src_pe=k % 2, dst_pe=1, op=REQ_PUT,
                          dtype=DT_INT) for k in range(n)])


def kernels(call):
    """Names of the batch kernels that copy, of those that a call launches."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return sorted({e.key for e in prof.key_averages() if "batch_exec" in e.key or "batch_small" in e.key})


@pytest.mark.parametrize("n", [300, 4000])
def test_runs_the_kernels_that_are_timed(shmem_factory, n):
    sh, p = shmem_factory(NPES, HEAP), Handle()
    reqs = rows(n, 512)
    with sh.batch(len(reqs), int(reqs["bytes"].sum()), 256) as b:
        b.upload(reqs)
        b.execute(1)
        assert b.execute_picked(p, reqs)[0] == 0
        timed = kernels(lambda: b.execute(1))
        picked = kernels(lambda: b.execute_picked(p, reqs))
    assert len(timed) == 1 and picked == timed
    assert sh.status() == 0


def test_an_error_reaches_the_status(shmem_factory):
    sh, p = shmem_factory(NPES, HEAP), Handle()
    reqs = rows(40, 65536)
    before = heap_images(sh, NPES, HEAP)
    with sh.batch(len(reqs), 0, 256) as b:  # a work table of 41 items for 160 chunks
        for _ in range(2):
            assert b.execute_picked(p, reqs)[0] == ERR_NOMEM
            assert np.array_equal(heap_images(sh, NPES, HEAP), before)
        assert b.execute_picked(p, rows(30, 4096))[0] == 0  # the next call starts without it
