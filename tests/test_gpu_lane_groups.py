"""Thread-form calls of one length by groups of lanes: from a few warps each lane
copies for itself, from many the group copies together, on both sides of the
lengths at which that changes."""
import pytest

from nvshmem_b200 import REQ_GET, REQ_PUT
from test_gpu_device_calls import ALL, HEAP, HEAP_OPERAND, Rows, check, exe  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [0x55555555, 0x5555D555, ALL])
@pytest.mark.parametrize("op", [REQ_PUT, REQ_GET])
def test_few_warps(exe, tmp_path, lanes, op):  # noqa: F811
    m = Rows()
    n = 2 * bin(lanes).count("1") + 3
    check(exe, tmp_path, [(0, lanes, HEAP_OPERAND, m.make([nb], n, op=op, skew=skew))
                          for nb in (124, 132, 144, 148, 260, 516, 528, 4100, 16_380, 16_384) for skew in (4, 16)])


@pytest.mark.parametrize("nbytes,warps", [(260, 200), (260, 700), (388, 700), (1028, 310)])
def test_many_warps(exe, tmp_path, nbytes, warps):  # noqa: F811
    m = Rows()
    rows = m.make([nbytes], 32 * warps, op=REQ_PUT)
    assert m.at <= HEAP
    check(exe, tmp_path, [(0, ALL, HEAP_OPERAND, rows)])
