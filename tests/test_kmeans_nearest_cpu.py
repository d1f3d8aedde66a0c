"""The k-means assignment's search for the centre at a known distance: the
lowest of equal ones, and a centre of the group whatever the distance (no sums
or counts are written out of range should two evaluations ever differ)."""
import os
import pathlib
import shutil
import subprocess

import pytest

from conftest import PKG_DIR, ROOT


def test_first_at_distance(tmp_path):
    nvcc = shutil.which("nvcc")
    if not shutil.which("g++") or not nvcc:
        pytest.skip("no compiler")
    cuda = pathlib.Path(os.path.realpath(nvcc)).parent.parent
    exe = tmp_path / "nearest"
    subprocess.run(["g++", "-std=c++17", "-ffp-contract=off", "-I", str(cuda / "include"), "-I", str(PKG_DIR / "csrc"),
                    str(ROOT / "tests" / "native" / "kmeans_nearest.cpp"), "-o", str(exe)], check=True, timeout=300)
    ask = [(0, 8, 0.0, 0), (0, 8, 9.0, 3), (4, 8, 9.0, 5), (16, 20, 361.0, 19),
           (0, 8, 9.5, 0), (8, 16, 9.0, 8), (16, 20, float("inf"), 16), (16, 20, float("nan"), 16)]
    out = subprocess.run([str(exe)], input="\n".join(f"{a} {b} {d}" for a, b, d, _ in ask), check=True,
                         capture_output=True, text=True, timeout=60).stdout.split()
    assert [int(v) for v in out] == [w for *_, w in ask]
