"""Registers that the device calls cost an application's kernel: linked with device
LTO, a kernel that puts or gets by its warps or by its block runs with 1024
threads, one whose threads put and get with 512; the plain link leaves room for
384."""
import os
import re
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(REPO, "df-nvshmem-prototype_b200", "lib")

SOURCE = """
#include "nvshmem.h"
#include "nvshmem_device.h"
#include "nvshmemx.h"
__global__ void by_warp(float *d, float *s, size_t stride, int n, int get) {
  const size_t k = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 32;
  if (get) nvshmemx_float_get_warp(d + k * stride, s + k * stride, n, 1);
  else nvshmemx_float_put_warp(d + k * stride, s + k * stride, n, 1);
}
__global__ void by_block(float *d, float *s, size_t stride, int n, int get) {
  if (get) nvshmemx_float_get_block(d + blockIdx.x * stride, s + blockIdx.x * stride, n, 1);
  else nvshmemx_float_put_block(d + blockIdx.x * stride, s + blockIdx.x * stride, n, 1);
}
__global__ void by_thread(float *d, float *s, size_t stride, int n, int get) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (get) nvshmem_float_get(d + k * stride, s + k * stride, n, 1);
  else nvshmem_float_put(d + k * stride, s + k * stride, n, 1);
}
int main() {
  by_warp<<<1, 32>>>(0, 0, 0, 0, 0);
  by_block<<<1, 32>>>(0, 0, 0, 0, 0);
  by_thread<<<1, 32>>>(0, 0, 0, 0, 0);
}
"""


def registers(text):
    """Kernel name -> registers, from ptxas (LTO) or nvlink (plain)."""
    got, name = {}, None
    for line in text.splitlines():
        if "entry function" in line or ("Function properties" in line and "nvlink" in line):
            m = re.search(r"_Z\d+(by_[a-z]+?)Pf", line)
            name = m.group(1) if m else None
        m = re.search(r"[uU]sed (\d+) registers", line)
        if m and name:
            got[name], name = int(m.group(1)), None
    return got


@pytest.mark.parametrize("link,most", [("lto", {"by_warp": 64, "by_block": 64, "by_thread": 104}),
                                       ("plain", {"by_warp": 168, "by_block": 168, "by_thread": 168})])
def test_registers_of_a_calling_kernel(tmp_path, link, most):
    if not os.path.exists(os.path.join(LIB, "libnvshmem.a")):
        pytest.skip("the library is not built")
    src, out = tmp_path / "app.cu", str(tmp_path / "app")
    src.write_text(SOURCE)
    inc = ["-I", os.path.join(REPO, "include")]
    libs = ["-L", LIB, "-lnvshmem", "-L/usr/local/cuda/lib64/stubs", "-lcuda"]
    final = ["-gencode", "arch=compute_100a,code=sm_100a", "-rdc=true"]
    if link == "plain":
        cmds = [["nvcc", *final, *inc, str(src), "-o", out, *libs, "-Xnvlink", "-v"]]
    else:
        cmds = [["nvcc", "-gencode", "arch=compute_100a,code=lto_100a", "-rdc=true", *inc, "-c", str(src), "-o", out + ".o"],
                ["nvcc", *final, "-dlto", out + ".o", "-o", out, *libs, "-Xptxas", "-v"]]
    for c in cmds:
        r = subprocess.run(c, capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
    got = registers(r.stdout + r.stderr)
    print(link, got)
    assert set(got) == set(most)
    assert all(got[k] <= most[k] for k in most), got
