"""The public device calls as an application's kernels make them
(tests/native/device_calls.cu, linked against libnvshmem.a the plain way and
with device LTO), against the CPU oracle: puts and gets by groups of lanes of
every kind, of lengths around the parts of the shared copy, with the local
operand in the heap, in shared memory and in a thread's own array, and the
warp, CTA and TMA forms of every type."""
import os
import subprocess

import numpy as np
import pytest

from nvshmem_b200 import DT_DOUBLE, DT_FLOAT, DT_INT, REQ_GET, REQ_PUT
from oracle.model import Model
from _util import requests

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.environ.get("DEVICE_CALLS_LIB", os.path.join(REPO, "df-nvshmem-prototype_b200", "lib"))
NPES, HEAP = 2, 32 << 20
HEAP_OPERAND, OWN, SHARED, SHARED_ONE = range(4)
ALL = 0xFFFFFFFF
# 1, 15, 16 (a half, and every other lane), 17, 31 and 32 lanes
LANES = [0x100, 0x7FFF, 0xFFFF0000, 0x55555555, 0x5555D555, 0x7FFFFFFF, ALL]


@pytest.fixture(scope="module", params=["plain", "lto"])
def exe(request, tmp_path_factory):
    d = tmp_path_factory.mktemp(request.param)
    src, out = os.path.join(REPO, "tests", "native", "device_calls.cu"), str(d / "device_calls")
    inc, libs = ["-I", os.path.join(REPO, "include")], ["-L", LIB, "-lnvshmem", "-L/usr/local/cuda/lib64/stubs", "-lcuda"]
    final = ["-gencode", "arch=compute_100a,code=sm_100a", "-rdc=true"]
    if request.param == "plain":
        cmds = [["nvcc", *final, *inc, src, "-o", out, *libs]]
    else:
        cmds = [["nvcc", "-gencode", "arch=compute_100a,code=lto_100a", "-rdc=true", *inc, "-c", src, "-o", out + ".o"],
                ["nvcc", *final, "-dlto", out + ".o", "-o", out, *libs]]
    for c in cmds:
        r = subprocess.run(c, capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-3000:]
    return out


def check(exe, tmp_path, lists):
    """lists: (form, lanes, operand, rows)."""
    om = Model(NPES, HEAP)
    for pe in range(NPES):
        om.fill_random(pe, 0, HEAP, 3)
    with open(tmp_path / "in", "wb") as f:
        f.write(np.array([NPES, len(lists)], np.int32).tobytes() + np.array([HEAP], np.uint64).tobytes())
        f.write(om.heap.tobytes())
        for form, lanes, operand, rows in lists:
            f.write(np.array([form, lanes, len(rows), operand], np.uint32).tobytes() + requests(rows).tobytes())
    r = subprocess.run([exe, str(tmp_path / "in"), str(tmp_path / "out")], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
    got = np.fromfile(tmp_path / "out", dtype=np.uint8).reshape(NPES, HEAP)
    for form, lanes, operand, rows in lists:
        om.apply_requests(requests(rows))
        for k, q in enumerate(rows):
            at = slice(q["dst_off"], q["dst_off"] + q["bytes"])
            assert np.array_equal(got[q["dst_pe"], at], om.heap[q["dst_pe"], at]), (form, hex(lanes), operand, k, q)
    assert np.array_equal(got, om.heap)


class Rows:
    """Requests with destinations of their own in the upper half of the heap."""

    def __init__(self):
        self.at = HEAP // 2

    def make(self, sizes, n, dtype=DT_INT, op=None, skew=4, same_source=False):
        w, rows = (8 if dtype == DT_DOUBLE else 4), []
        for k in range(n):
            nb = sizes[(k * 5 + k // len(sizes)) % len(sizes)] // w * w
            ds, ss = (k % 4) * skew, (k // 3 % 4) * skew
            if w == 8:
                ds, ss = ds // 8 * 8, ss // 8 * 8
            src = 0 if same_source else 4096 * (k % 97) * 8 + ss
            rows.append(dict(src_off=src, dst_off=self.at + ds, bytes=nb, src_pe=0 if same_source else k % NPES,
                             dst_pe=(k // 2) % NPES, op=op if op is not None else (REQ_PUT if k // 32 % 2 else REQ_GET),
                             dtype=dtype))
            self.at += (nb + 48) // 16 * 16
        assert self.at <= HEAP
        return rows


@pytest.mark.parametrize("operand", [OWN, SHARED])
def test_local_operand_of_the_thread(exe, tmp_path, operand):
    """Lengths on both sides of four vectors, the first that lanes share."""
    m = Rows()
    lists = []
    for lanes in LANES:
        n = 3 * bin(lanes).count("1") + 2
        for op in (REQ_PUT, REQ_GET):
            lists.append((0, lanes, operand, m.make([0, 4, 60, 64, 68, 76, 80, 128, 252, 256], n, op=op)))
            lists.append((0, lanes, operand, m.make([64, 72, 80, 88, 248, 256], n, dtype=DT_DOUBLE, op=op)))
    check(exe, tmp_path, lists)


def test_long_copies_from_shared_memory(exe, tmp_path):
    """From 16 KiB on a copy prefetches its source, and the TMA form loads it
    into its ring: both only from global memory."""
    m = Rows()
    lists = [(0, lanes, SHARED_ONE, m.make([nb], bin(lanes).count("1"), op=REQ_PUT, same_source=True))
             for lanes in (0x100, 0x7FFF, ALL) for nb in (16384, 20484, 24576)]
    lists += [(form, ALL, SHARED_ONE, m.make([nb], 5, op=REQ_PUT, same_source=True))
              for form in (1, 2, 3) for nb in (4100, 24576)]
    check(exe, tmp_path, lists)


@pytest.mark.parametrize("dtype", [DT_INT, DT_FLOAT, DT_DOUBLE])
@pytest.mark.parametrize("skew", [4, 1])
def test_groups_of_lanes(exe, tmp_path, dtype, skew):
    """Mixed lengths and offsets within a group, and puts beside gets."""
    m = Rows()
    sizes = [0, 4, 60, 68, 520, 4100, 16384, 70_000]
    lists = []
    for lanes in LANES:
        n = 2 * bin(lanes).count("1") + 1
        lists.append((0, lanes, HEAP_OPERAND, m.make(sizes if n < 40 else sizes[:-1], n, dtype=dtype, skew=skew)))
        for op in (REQ_PUT, REQ_GET):
            lists.append((0, lanes, HEAP_OPERAND, m.make(sizes[:-2], n, dtype=dtype, op=op, skew=skew)))
    mixed = m.make(sizes, 40, dtype=dtype, skew=skew)
    for k, q in enumerate(mixed):
        q["op"] = REQ_PUT if k % 3 else REQ_GET
    check(exe, tmp_path, lists + [(0, ALL, HEAP_OPERAND, mixed)])


@pytest.mark.parametrize("form", [1, 2, 3])
def test_cooperative_forms(exe, tmp_path, form):
    m = Rows()
    sizes = [0, 4, 12, 60, 516, 2044, 4096, 4100, 16384, 20_004, 65_556]
    lists = []
    for dtype in (DT_INT, DT_FLOAT, DT_DOUBLE):
        for skew in (4, 1) if dtype != DT_DOUBLE else (8, 4):
            for op in (REQ_PUT, REQ_GET):
                lists.append((form, ALL, HEAP_OPERAND, m.make(sizes, 45, dtype=dtype, op=op, skew=skew)))
    check(exe, tmp_path, lists)
