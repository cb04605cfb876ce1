"""Resident requests reach the per-call kernel unchecked: one with a dtype that no
type has is a copy of whole words in the TMA form, of 8 bytes for every 4 in the
others."""
import numpy as np
import pytest

from nvshmem_b200 import MODE_BLOCK, MODE_BULK, MODE_THREAD, MODE_WARP, REQ_PUT
from _util import requests

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,times", [(MODE_THREAD, 2), (MODE_WARP, 2), (MODE_BLOCK, 2), (MODE_BULK, 1)])
@pytest.mark.parametrize("nbytes", [4, 1028, 8192])
def test_unknown_dtype(shmem_factory, mode, times, nbytes):
    heap = 1 << 20
    sh = shmem_factory(2, heap)
    for pe in range(2):
        sh.fill_random(pe, 0, heap, 50 + pe)
    want = sh.read(1, 0, heap)
    want[heap // 2:heap // 2 + times * nbytes] = sh.read(0, 64, times * nbytes)
    with sh.batch(1, nbytes, 256) as b:
        b.upload(requests([dict(src_off=64, dst_off=heap // 2, bytes=nbytes, src_pe=0, dst_pe=1, op=REQ_PUT, dtype=3)]))
        b.percall(mode, 1)
    assert sh.status() == 0
    assert np.array_equal(sh.read(1, 0, heap), want)
