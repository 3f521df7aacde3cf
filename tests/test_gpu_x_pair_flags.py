"""The words through which pairs of SMs hand over the parts of a cut tile, looked at from a C++ program that holds them
(`pair_flags_check.cu`): all zero after every launch, and the same bits from launches that follow one another or run beside
those of another stream, also where a tile of many holders is left to the one that began it."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_words_are_handed_back(tmp_path):
    import aotx_b200.library as library
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    lib_dir = os.path.dirname(library.LIB_PATH)
    assert os.path.exists(library.LIB_PATH)
    exe = str(tmp_path / "pair_flags_check")
    build = subprocess.run(
        [nvcc, "-O2", "-std=c++17", "-diag-suppress", "20011", "-gencode", "arch=compute_100a,code=sm_100a",
         "-I", os.path.join(ROOT, "aotx_b200", "csrc"), "-o", exe, os.path.join(ROOT, "tests", "pair_flags_check.cu"),
         "-L", lib_dir, "-laotx_q8_b200", "-Xlinker", "-rpath", "-Xlinker", lib_dir],
        capture_output=True, text=True, timeout=900)
    assert build.returncode == 0, build.stderr[-2000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, (run.stdout[-3000:], run.stderr[-2000:])
    assert run.stdout.strip().endswith("pass")
