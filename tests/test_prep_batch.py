"""Host layout of a batch whose problems are prepared side by side: the same
as each problem's own, and the first failing problem's error."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "slamplay_gb300", "csrc")
CUDA_INC = "/usr/local/cuda/include"


@pytest.mark.parametrize("threads", ["1", "8"])
def test_batch_equals_its_problems(tmp_path, threads):
    if shutil.which("g++") is None or not os.path.isdir(CUDA_INC):
        pytest.skip("g++ or the CUDA headers are missing")
    out = str(tmp_path / "prep_batch")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    "-I", CUDA_INC, os.path.join(ROOT, "tests", "cpu", "prep_batch.cpp"),
                    os.path.join(CSRC, "prep.cpp"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=300, env=dict(os.environ, GBA_HOST_THREADS=threads))
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
