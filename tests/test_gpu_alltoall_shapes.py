"""All-to-all rounds at the numbers of PEs where the thread form changes its CTA
(a warp, 128 threads, more), and in the CTA form at messages around its rounds
of tiles."""
import numpy as np
import pytest

from nvshmem_b200 import DT_INT, MODE_BLOCK, MODE_BULK, MODE_THREAD, REQ_GET, REQ_PUT
from oracle.model import Model
from _util import heap_images

pytestmark = pytest.mark.gpu


def check(shmem_factory, npes, heap, nbytes, mode, op, ctas=0):
    sh, om = shmem_factory(npes, heap), Model(npes, heap)
    for pe in range(npes):
        sh.fill_random(pe, 0, heap, 12)
        om.fill_random(pe, 0, heap, 12)
    sh.alltoall(op, DT_INT, 0, heap // 2, nbytes, rounds=2, mode=mode, ctas_per_pe=ctas)
    assert sh.status() == 0
    om.alltoall(1 if op == REQ_GET else 0, 0, heap // 2, nbytes, rounds=2)
    assert np.array_equal(heap_images(sh, npes, heap), om.heap)


@pytest.mark.parametrize("npes", [33, 34, 65, 129, 130, 148])
@pytest.mark.parametrize("nbytes", [260, 4096, 4100])
def test_thread_form(shmem_factory, npes, nbytes):
    check(shmem_factory, npes, 2 << 20, nbytes, MODE_THREAD, REQ_GET if nbytes == 4096 else REQ_PUT)


@pytest.mark.parametrize("nbytes", [508, 4100, 16384, 16388, 49_152, 49_156, 65_540, 100_000])
@pytest.mark.parametrize("mode", [MODE_BLOCK, MODE_BULK])
def test_cta_form(shmem_factory, nbytes, mode):
    check(shmem_factory, 3, 1 << 20, nbytes, mode, REQ_PUT, ctas=2)
