"""The kernels that are held to few registers a thread keep their state in them:
the linker's report of the shared library's kernels names no spills."""
import glob
import os
import re
import subprocess

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "df-nvshmem-prototype_b200")


@pytest.fixture(scope="module")
def spills(tmp_path_factory):
    """Bytes of spill stores of each kernel (mangled name), as the library's link reports them."""
    objs = sorted(glob.glob(os.path.join(PKG, "_build", "lto", "*.o")))
    if not objs:
        pytest.skip("the library's objects are not built")
    out = str(tmp_path_factory.mktemp("link") / "lib.so")
    r = subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-dlto", "-shared", "-rdc=true", "-cudart",
                        "static", "-Xptxas", "-v", *objs, "-o", out, "-lpthread", "-ldl", "-lrt"],
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-2000:]
    got, name = {}, None
    for line in (r.stdout + r.stderr).splitlines():
        m = re.search(r"Compiling entry function '(\w+)'", line)
        name = m.group(1) if m else name
        m = re.search(r"(\d+) bytes spill stores", line)
        if m and name:
            got[name], name = int(m.group(1)), None
    return got


def test_register_copy_kernels_do_not_spill(spills):
    named = {k: v for k, v in spills.items() if "batch_exec_kernel" in k}
    assert len(named) == 12
    assert not any(named.values()), named
