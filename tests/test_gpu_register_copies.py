"""Register-copy batches: every number of accesses in flight, with sources 4, 8
and 12 bytes and single bytes off their destinations, at the lengths where a
copy's head, rounds of vectors and tail meet."""
import pytest

from nvshmem_b200 import DT_INT, REQ_GET, REQ_PUT
from oracle.model import Model
from _util import first_diff, heap_images, requests

pytestmark = pytest.mark.gpu

HEAP = 16 << 20
SIZES = [4, 12, 16, 28, 508, 512, 1024, 1536, 1540, 2044, 2048, 4100, 16400]


@pytest.mark.parametrize("unroll", [1, 2, 4, 8])
@pytest.mark.parametrize("skews", [(0, 4, 8, 12), (0, 1, 6)])
def test_bit_exact(shmem_factory, unroll, skews):
    sh, om = shmem_factory(2, HEAP), Model(2, HEAP)
    for pe in range(2):
        sh.fill_random(pe, 0, HEAP, 31)
        om.fill_random(pe, 0, HEAP, 31)
    rows, at = [], HEAP // 2
    for ds in skews:
        for ss in skews:
            for k, nb in enumerate(SIZES):
                rows.append(dict(src_off=20_000 * (len(rows) % 50) + ss, dst_off=at + ds, bytes=nb, src_pe=k % 2,
                                 dst_pe=(k // 2) % 2, op=REQ_PUT if k % 3 else REQ_GET, dtype=DT_INT))
                at += (nb + 32) // 16 * 16
    assert at <= HEAP
    reqs = requests(rows)
    with sh.batch(len(reqs), int(reqs["bytes"].sum()), 1024) as b:
        for threads, chunk in ((128, 1024), (1024, 16384)):
            b.set_config(dict(unroll=unroll, threads=threads, chunk_bytes=chunk))
            assert b.submit(reqs)[0] == 0
    om.apply_requests(reqs)
    assert first_diff(heap_images(sh, 2, HEAP), om.heap) is None
