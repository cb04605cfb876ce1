"""The thread form's long copies, shared by a cluster of four CTAs of 128
threads: sizes around the smallest shared copy and its pieces, lists of fewer
and of more requests than a cluster, and a CTA whose threads all list one."""
import pytest

from nvshmem_b200 import DT_INT, MODE_THREAD, REQ_G, REQ_GET, REQ_P, REQ_PUT, REQ_SIGNAL
from oracle.model import Model
from _util import first_diff, heap_images, requests

pytestmark = pytest.mark.gpu

HEAP = 64 << 20
SIZES = [65532, 65536, 65540, 98304, 98308, 131068, 300_004]


def run(shmem_factory, rows):
    sh, om = shmem_factory(2, HEAP), Model(2, HEAP)
    for pe in range(2):
        sh.fill_random(pe, 0, HEAP, 11)
        om.fill_random(pe, 0, HEAP, 11)
    reqs = requests(rows)
    sh.exec_requests(reqs, MODE_THREAD)
    assert sh.status() == 0
    om.apply_requests(reqs)
    assert first_diff(heap_images(sh, 2, HEAP), om.heap) is None


@pytest.mark.parametrize("n", [1, 7, 127, 129, 511, 513, 1100])
@pytest.mark.parametrize("skew", [0, 1, 4])
def test_long_copies_between_short_requests(shmem_factory, n, skew):
    rows, at = [], HEAP // 2
    for k in range(n):
        nb = SIZES[(k // 9) % len(SIZES)] if k % 9 == 0 else 4 * (k % 700)
        kind = k % 13
        if kind == 5:
            rows.append(dict(dst_off=at, dst_pe=k % 2, op=REQ_SIGNAL, value=k))
        elif kind == 7:
            rows.append(dict(src_off=k, dst_off=at, dst_pe=k % 2, op=REQ_P, dtype=DT_INT))
        elif kind == 11:
            rows.append(dict(src_off=4 * k, dst_off=at, src_pe=k % 2, dst_pe=(k // 2) % 2, op=REQ_G, dtype=DT_INT))
        else:
            rows.append(dict(src_off=(k * 4096) % (HEAP // 4) + skew, dst_off=at, bytes=nb, src_pe=k % 2,
                             dst_pe=(k // 2) % 2, op=REQ_PUT if k % 2 else REQ_GET, dtype=DT_INT))
        at += (nb + 47) // 16 * 16
    assert at <= HEAP
    run(shmem_factory, rows)


def test_every_thread_of_a_cta_lists_a_copy(shmem_factory):
    rows = [dict(src_off=(k * 65536) % (HEAP // 4), dst_off=HEAP // 2 + k * 66000, bytes=65540, src_pe=k % 2,
                 dst_pe=1, op=REQ_PUT, dtype=DT_INT) for k in range(130)]
    run(shmem_factory, rows)
