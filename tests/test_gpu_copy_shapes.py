"""The register copies at the sizes where their parts meet: edge words, lane
copies, rows, tiles and long rounds, for every distance of source and
destination modulo 16 (whole words and single bytes), in every caller form."""
import numpy as np
import pytest

from nvshmem_b200 import (DT_INT, MODE_BLOCK, MODE_BULK, MODE_THREAD, MODE_WARP, REQ_GET, REQ_PUT, REQ_SIGNAL)
from oracle.model import Model
from _util import first_diff, heap_images, requests

pytestmark = pytest.mark.gpu

HEAP = 32 << 20
# around: one word, a vector, four vectors (a lane's own copy), a row of 512
# bytes, a 4 KiB tile, the 16 KiB long copies and their 6 and 8 KiB rounds
SIZES = [0, 4, 12, 16, 60, 64, 68, 80, 508, 516, 2044, 4096, 4100, 8188, 16380, 16384, 16400, 24592, 65556]


def shaped(skews, sizes, npes=2):
    rows, cursor, k = [], HEAP // 2, 0
    for ds in skews:
        for ss in skews:
            for nb in sizes:
                rows.append(dict(src_off=4096 * (k % 64) + ss, dst_off=cursor + ds, bytes=nb, src_pe=k % npes,
                                 dst_pe=(k // 2) % npes, op=REQ_PUT if k % 3 else REQ_GET, dtype=DT_INT))
                cursor += (nb + 32) // 16 * 16
                k += 1
                if k % 11 == 0:  # lanes without a copy in between
                    rows.append(dict(dst_off=cursor, dst_pe=k % npes, op=REQ_SIGNAL, value=k))
                    cursor += 16
    assert cursor <= HEAP
    return requests(rows)


@pytest.mark.parametrize("skews", [(0, 4, 8, 12), (0, 1, 6)])
@pytest.mark.parametrize("mode", [MODE_THREAD, MODE_WARP, MODE_BLOCK, MODE_BULK])
def test_copy_shapes_bit_exact(shmem_factory, mode, skews):
    sh, om = shmem_factory(2, HEAP), Model(2, HEAP)
    for pe in range(2):
        sh.fill_random(pe, 0, HEAP, 5)
        om.fill_random(pe, 0, HEAP, 5)
    reqs = shaped(skews, SIZES)
    sh.exec_requests(reqs, mode)
    assert sh.status() == 0
    om.apply_requests(reqs)
    assert first_diff(heap_images(sh, 2, HEAP), om.heap) is None


@pytest.mark.parametrize("lanes", [1, 15, 16, 31, 33])
def test_thread_form_with_few_lanes(shmem_factory, lanes):
    """A warp that is not full: copies alone, and together with fewer lanes."""
    sh, om = shmem_factory(2, HEAP), Model(2, HEAP)
    for pe in range(2):
        sh.fill_random(pe, 0, HEAP, 6)
        om.fill_random(pe, 0, HEAP, 6)
    reqs = shaped((4, 8), [20, 4100, 20004])[:lanes]
    sh.exec_requests(reqs, MODE_THREAD)
    assert sh.status() == 0
    om.apply_requests(reqs)
    assert first_diff(heap_images(sh, 2, HEAP), om.heap) is None


def test_thread_form_in_an_all_to_all_of_odd_messages(shmem_factory):
    npes, nbytes = 5, 16384 + 20
    sh, om = shmem_factory(npes, 1 << 20), Model(npes, 1 << 20)
    for pe in range(npes):
        sh.fill_random(pe, 0, 1 << 20, 7)
        om.fill_random(pe, 0, 1 << 20, 7)
    for mode in (MODE_THREAD, MODE_WARP, MODE_BLOCK):
        sh.alltoall(REQ_GET, DT_INT, 0, 1 << 19, nbytes, rounds=2, mode=mode, ctas_per_pe=2)
    om.alltoall(1, 0, 1 << 19, nbytes, rounds=1)
    assert np.array_equal(heap_images(sh, npes, 1 << 20), om.heap)


@pytest.mark.parametrize("op", [REQ_PUT, REQ_GET])
@pytest.mark.parametrize("nbytes,ctas", [(16, 3), (64, 1), (10 * 1024, 2), (64 * 1024 + 16, 1), (100_000, 5)])
@pytest.mark.parametrize("apart", [True, False])
def test_ring_across_rounds(shmem_factory, op, nbytes, ctas, apart):
    """Rounds of the CTA-wide TMA mode over rotating buffer sets: shares below a
    chunk, of several messages and of more chunks than the ring has stages;
    with receive buffers that a later round sends from again (`apart` false),
    where no load may pass a barrier."""
    npes, nsets, rounds = 5, 3, 7
    one = (npes * nbytes + 15) // 16 * 16
    heap = 8 << 20
    recv = 4 << 20 if apart else one  # set s is received where set s + 1 is sent from
    sh, om = shmem_factory(npes, heap), Model(npes, heap)
    for pe in range(npes):
        sh.fill_random(pe, 0, heap, 8)
        om.fill_random(pe, 0, heap, 8)
    sh.alltoall(op, DT_INT, 0, recv, nbytes, rounds=rounds, nsets=nsets, set_stride=one, mode=MODE_BULK,
                ctas_per_pe=ctas)
    assert sh.status() == 0
    om.alltoall(1 if op == REQ_GET else 0, 0, recv, nbytes, rounds=rounds, nsets=nsets, set_stride=one)
    assert np.array_equal(heap_images(sh, npes, heap), om.heap)


def test_all_to_all_by_threads_of_several_warps(shmem_factory):
    npes, nbytes, heap = 40, 1028, 256 << 10
    sh, om = shmem_factory(npes, heap), Model(npes, heap)
    for pe in range(npes):
        sh.fill_random(pe, 0, heap, 9)
        om.fill_random(pe, 0, heap, 9)
    sh.alltoall(REQ_PUT, DT_INT, 0, 128 << 10, nbytes, rounds=2, mode=MODE_THREAD)
    om.alltoall(0, 0, 128 << 10, nbytes, rounds=2)
    assert np.array_equal(heap_images(sh, npes, heap), om.heap)


@pytest.mark.parametrize("mode,n", [(MODE_BLOCK, 6145), (MODE_BULK, 12289)])
def test_cta_forms_with_many_requests(shmem_factory, mode, n):
    """From here on the CTA forms run with 128 threads to a CTA."""
    sh, om = shmem_factory(2, HEAP), Model(2, HEAP)
    for pe in range(2):
        sh.fill_random(pe, 0, HEAP, 10)
        om.fill_random(pe, 0, HEAP, 10)
    sizes = [4, 100, 1000, 2052] * (n // 4) + [70_004]
    rows, at = [], HEAP // 2
    for k, nb in enumerate(sizes):
        rows.append(dict(src_off=(k * 64) % 4_000_000 + 4 * (k % 4), dst_off=at, bytes=nb, src_pe=k % 2,
                         dst_pe=(k // 2) % 2, op=REQ_PUT if k % 2 else REQ_GET, dtype=DT_INT))
        at += (nb + 15) // 16 * 16
    assert len(rows) == n and at <= HEAP
    reqs = requests(rows)
    sh.exec_requests(reqs, mode)
    assert sh.status() == 0
    om.apply_requests(reqs)
    assert first_diff(heap_images(sh, 2, HEAP), om.heap) is None
