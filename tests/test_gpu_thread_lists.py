"""Thread-form lists long enough that a warp takes several requests (as many as
keep the warps of two CTAs of 128 threads to an SM busy, 32 at most): long
copies that fill a CTA's share of the list, beside short ones of every length
and distance from their destinations."""
import numpy as np
import pytest

from nvshmem_b200 import DT_DOUBLE, DT_FLOAT, DT_INT, MODE_THREAD, REQ_GET, REQ_PUT, REQ_SIGNAL, REQUEST_DTYPE
from oracle.model import Model
from _util import first_diff, heap_images

pytestmark = pytest.mark.gpu

HEAP, SMS = 128 << 20, 148


def lists(n, lanes):
    """n requests in warps of `lanes`; the first CTA's are all long copies, as is every 997th."""
    k = np.arange(n)
    r = np.zeros(n, dtype=REQUEST_DTYPE)
    short = np.array([4, 8, 60, 64, 68, 76, 252, 516, 1028, 2048, 0, 4100])
    r["bytes"] = short[(k * 7 + k // 12) % len(short)]
    first = 4 * lanes  # a CTA's requests
    long = (k < first) | (k % 997 == 0)
    r["bytes"][long] = np.array([65536, 65540, 98_308, 131_068])[k[long] % 4]
    r["bytes"][k % 503 == 5] = 20_004
    r["dtype"] = np.array([DT_INT, DT_FLOAT, DT_INT, DT_DOUBLE])[k % 4]
    r["bytes"] = np.where(r["dtype"] == DT_DOUBLE, r["bytes"] // 8 * 8, r["bytes"])
    r["op"] = np.where(k % 3 == 0, REQ_GET, REQ_PUT)
    sig = k % 101 == 7
    r["op"][sig], r["bytes"][sig], r["dtype"][sig], r["value"] = REQ_SIGNAL, 0, DT_INT, k
    skew = np.where(r["dtype"] == DT_DOUBLE, 8, 4)
    r["src_off"] = (k * 4096) % (HEAP // 4) + k // 5 % 4 * skew % 16
    size = (np.maximum(r["bytes"], 4).astype(np.int64) + 16 + 15) // 16 * 16
    r["dst_off"] = HEAP // 2 + np.cumsum(size) - size + np.where(sig, 0, k // 7 % 4 * skew % 16)
    r["src_pe"], r["dst_pe"] = k % 2, k // 2 % 2
    assert r["dst_off"][-1] + size[-1] <= HEAP
    return r


@pytest.mark.parametrize("n", [1185, SMS * 8 * 16 + 1, SMS * 8 * 31 + 5])
def test_several_requests_to_a_warp(shmem_factory, n):
    lanes = min(32, -(-n // (SMS * 8)))
    assert lanes in (2, 17, 32)
    sh, om = shmem_factory(2, HEAP), Model(2, HEAP)
    for pe in range(2):
        sh.fill_random(pe, 0, HEAP, 13)
        om.fill_random(pe, 0, HEAP, 13)
    reqs = lists(n, lanes)
    sh.exec_requests(reqs, MODE_THREAD)
    assert sh.status() == 0
    om.apply_requests(reqs)
    assert first_diff(heap_images(sh, 2, HEAP), om.heap) is None
