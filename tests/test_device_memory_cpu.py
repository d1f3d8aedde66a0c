"""The rules of the library's device memory -- what stays with the library when
buffers are freed, what a failing allocation gets back -- on the CPU, over a
stand-in for the CUDA runtime's allocator (tests/native/device_memory.cpp)."""
import os
import pathlib
import shutil
import subprocess

import pytest

from conftest import PKG_DIR, ROOT


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc")
    if not shutil.which("g++") or not nvcc:
        pytest.skip("no compiler")
    cuda = pathlib.Path(os.path.realpath(nvcc)).parent.parent
    out = tmp_path_factory.mktemp("mem") / "device_memory"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(cuda / "include"), "-I", str(ROOT / "include"),
                    "-I", str(PKG_DIR / "csrc"), "-x", "c++", str(PKG_DIR / "csrc" / "qcp_mem.cu"),
                    str(ROOT / "tests" / "native" / "device_memory.cpp"), "-o", str(out)], check=True, timeout=300)
    return out


@pytest.mark.parametrize("what", ["idle_after_frees", "give_back", "large_gets_the_rest", "lasting_and_small",
                                  "other_device", "refused_free", "shared_buffers"])
def test_rule(exe, what):
    r = subprocess.run([str(exe), what], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
