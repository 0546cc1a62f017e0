"""A re-ingestion that fails: before the handle's arrays are written it leaves the
matrix that was there, after that none, never half of each.  The failing steps are
those of a stand-in for the CUDA runtime, so no GPU takes part."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "spmspv-adaptive_b200", "csrc")


def test_failed_input_coo(tmp_path):
    nvcc = shutil.which("nvcc")
    if not nvcc:
        pytest.skip("needs nvcc to compile ingest.cu")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    obj, exe = str(tmp_path / "ingest.o"), str(tmp_path / "ingest_failure")
    subprocess.run(["make", "-s", "-C", CSRC, "OBJDIR=" + str(tmp_path), obj], check=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", cuda, "-I", CSRC,
                    "-I", os.path.join(CSRC, "..", "..", "include"),
                    os.path.join(HERE, "ingest_fake_cuda.cpp"), obj, "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
