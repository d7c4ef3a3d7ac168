"""Index arithmetic and tables behind the unchecked kernels, evaluated on the host by a program that is compiled
against the library's own headers and linked with it (tests/cpp/index_tables.cu): no GPU is used."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_index_tables(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    libdir = os.path.join(ROOT, "hyteg_b200")
    if not os.path.exists(nvcc):
        pytest.skip("no CUDA compiler")
    if not os.path.exists(os.path.join(libdir, "libhyteg_b200.so")):
        pytest.skip("library not built")
    exe = str(tmp_path / "index_tables")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(libdir, "csrc"),
                    "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "index_tables.cu"), "-L", libdir,
                    "-lhyteg_b200", "-Xlinker", f"-rpath={libdir}", "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout
