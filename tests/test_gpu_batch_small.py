"""Batches that run as one launch: around the sizes at which the requests stop
fitting the kernel's parameters (120 full, 240 compact), a CTA's threads (256)
and the launch itself (4096), in every entry point, with the errors that must
leave the heap untouched."""
import numpy as np
import pytest

from nvshmem_b200 import (DT_INT, ERR_BOUNDS, ERR_INVALID, ERR_NOMEM, REQ_P, REQ_PUT, ShmemError, to_compact)
from oracle.model import Model
from _util import first_diff, heap_images, random_requests, requests

pytestmark = pytest.mark.gpu

NPES, HEAP = 4, 16 << 20


def start(shmem_factory):
    sh, om = shmem_factory(NPES, HEAP), Model(NPES, HEAP)
    for pe in range(NPES):
        sh.fill_random(pe, 0, HEAP, 21)
        om.fill_random(pe, 0, HEAP, 21)
    return sh, om


@pytest.mark.parametrize("entry", ["submit", "compact", "resident"])
@pytest.mark.parametrize("n", [1, 31, 120, 121, 240, 241, 256, 257, 2049, 4095, 4096])
def test_sizes_bit_exact(shmem_factory, n, entry):
    sh, om = start(shmem_factory)
    reqs = random_requests(n, n, NPES, HEAP, max_bytes=12000)
    if entry == "compact":  # no compact form for the bits of a double
        reqs = reqs[~((reqs["op"] == REQ_P) & (reqs["dtype"] == 2))]
    assert len(reqs) > n * 0.8
    with sh.batch(len(reqs), int(reqs["bytes"].sum()), 256) as b:
        if entry == "submit":
            st, _ = b.submit(reqs)
        elif entry == "compact":
            st, _ = b.submit_compact(to_compact(reqs))
        else:
            b.upload(reqs)
            b.execute(2)
            st = 0
        assert st == 0 and sh.status() == 0
        om.apply_requests(reqs)
        assert first_diff(heap_images(sh, NPES, HEAP), om.heap) is None
        # the requests stay resident
        for pe in range(NPES):
            sh.fill_random(pe, 0, HEAP, 21)
        b.execute(1)
        assert first_diff(heap_images(sh, NPES, HEAP), om.heap) is None


@pytest.mark.parametrize("shape", [dict(tma_stages=2, tma_stage_bytes=1024, threads=128, chunk_bytes=256),
                                   dict(tma_stages=4, tma_stage_bytes=4096, threads=256, chunk_bytes=768),
                                   dict(tma_stages=3, tma_stage_bytes=8192, threads=256, chunk_bytes=1 << 20)])
def test_one_long_request_among_short_ones(shmem_factory, shape):
    """Pieces are counted per request: one of 6 MB beside empty and tiny ones."""
    sh, om = start(shmem_factory)
    rows, at = [], HEAP // 2
    for k, nb in enumerate([0, 4, 6_000_004, 0, 16, 20, 0, 1028, 0]):
        rows.append(dict(src_off=64 + 4 * (k % 4), dst_off=at, bytes=nb, src_pe=k % NPES, dst_pe=1, op=REQ_PUT,
                         dtype=DT_INT))
        at += (nb + 31) // 16 * 16
    reqs = requests(rows)
    with sh.batch(len(reqs), int(reqs["bytes"].sum()), 256) as b:
        b.set_config(shape)
        assert b.submit(reqs)[0] == 0
        assert b.stats()[0] == sum(-(-int(x) // shape["chunk_bytes"]) for x in reqs["bytes"])
    om.apply_requests(reqs)
    assert first_diff(heap_images(sh, NPES, HEAP), om.heap) is None


@pytest.mark.parametrize("n", [5, 300])
@pytest.mark.parametrize("what", ["op", "bounds", "table"])
def test_errors_run_nothing(shmem_factory, n, what):
    sh, _ = start(shmem_factory)
    reqs = random_requests(3, n, NPES, HEAP, ops=(REQ_PUT,), max_bytes=9000)
    reqs["bytes"] = 8192
    before = heap_images(sh, NPES, HEAP)
    bad = len(reqs) - 1
    if what == "op":
        reqs["op"][bad] = 9
        code = ERR_INVALID
    elif what == "bounds":
        reqs["dst_off"][bad] = HEAP - 8
        code = ERR_BOUNDS
    else:
        code, bad = ERR_NOMEM, -1
    payload = 0 if what == "table" else int(reqs["bytes"].sum())
    with sh.batch(len(reqs), payload, 1024) as b:
        b.set_config(dict(tma_stages=3, tma_stage_bytes=8192, threads=256, chunk_bytes=1024))
        assert b.submit(reqs)[0] == code
        with pytest.raises(ShmemError) as e:
            b.execute(1)
        assert e.value.code == code and f"request {bad} " in str(e.value)
    assert np.array_equal(heap_images(sh, NPES, HEAP), before)
