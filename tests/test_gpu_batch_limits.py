"""Batches on both sides of the size up to which one launch plans and executes
them, for both CTA sizes, submitted and executed again."""
import pytest

from oracle.model import Model
from _util import first_diff, heap_images, random_requests

pytestmark = pytest.mark.gpu

NPES, HEAP = 4, 32 << 20


@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("base", [512, 1024])
@pytest.mark.parametrize("extra", [-1, 0])
def test_one_launch_and_two(shmem_factory, threads, base, extra):
    n = base + 12 * threads + extra
    sh, om = shmem_factory(NPES, HEAP), Model(NPES, HEAP)
    for pe in range(NPES):
        sh.fill_random(pe, 0, HEAP, 22)
        om.fill_random(pe, 0, HEAP, 22)
    reqs = random_requests(n, n, NPES, HEAP, max_bytes=16000)
    assert len(reqs) == n
    with sh.batch(n, int(reqs["bytes"].sum()), 1024) as b:
        b.set_config(dict(tma_stages=2, tma_stage_bytes=4096, threads=threads, chunk_bytes=4096))
        assert b.submit(reqs)[0] == 0
        b.execute(1)
    assert sh.status() == 0
    om.apply_requests(reqs)
    assert first_diff(heap_images(sh, NPES, HEAP), om.heap) is None
