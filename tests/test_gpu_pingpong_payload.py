"""The payload of a ping-pong: after the exchanges PE 1 holds what PE 0 sent,
with whole vectors (copied straight) and with words outside them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [256, 260, 264])
@pytest.mark.parametrize("words", [0, 1, 3, 4, 5, 12, 16, 63, 64, 67, 1024, 4099, 8192])
def test_payload(shmem_factory, at, words):
    heap = 64 << 10
    sh = shmem_factory(2, heap)
    for pe in range(2):
        sh.fill_random(pe, 0, heap, 40 + pe)
    before = [sh.read(pe, 0, heap) for pe in range(2)]
    ns, total = sh.pingpong(0, at, words, 7, 3)
    assert len(ns) == 7 and total > 0
    want = before[1].copy()
    want[at:at + 4 * words] = before[0][at:at + 4 * words]
    assert np.array_equal(sh.read(0, 4, heap - 4), before[0][4:])
    assert np.array_equal(sh.read(1, 4, heap - 4), want[4:])
    assert all(sh.read(pe, 0, 4).view(np.int32)[0] == 10 for pe in range(2))
