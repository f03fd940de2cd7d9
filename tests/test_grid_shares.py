"""The grid PCG's split of a problem over its CTAs (tests/cpu/grid_shares.cpp)
and, on a GPU, problems whose split leaves CTAs without a share."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from slamplay_gb300 import BALProblem, Solver

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "slamplay_gb300", "csrc")
CUDA_INC = "/usr/local/cuda/include"


def test_shares_cover_the_problem(tmp_path):
    if shutil.which("g++") is None or not os.path.isdir(CUDA_INC):
        pytest.skip("g++ or the CUDA headers are missing")
    out = str(tmp_path / "grid_shares")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "cpu", "grid_shares.cpp"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


def _solve(b, **kw):
    g = b.copy()
    with Solver(max_num_iterations=4, function_tolerance=0.0, gradient_tolerance=0.0, parameter_tolerance=0.0,
                pcg_tolerance=1e-8, max_linear_solver_iterations=120, schur="explicit", **kw) as s:
        return g, s.solve(g)


# 20 of 150 CTAs own nothing on the walk of 30 cameras, 10 of 152 on that of
# 33, 3 on the ring of 33.  (Any CTA count set for a test selects the grid
# form; 500 is more than a launch has.)  Tolerance: none, the two-kernel PCG's
# additions in the same order.
@pytest.mark.gpu
@pytest.mark.parametrize("layout,cams,points", [(1, 30, 1500), (1, 33, 1500), (0, 33, 900), (3, 3, 100)])
def test_ctas_without_a_share(monkeypatch, layout, cams, points):
    b = BALProblem.synthetic(layout, seed=cams, num_cameras=cams, num_points=points)
    ref, sr = _solve(b, persistent_pcg=0)
    monkeypatch.setenv("GBA_TEST_GRID_CTAS", "500")
    got, sg = _solve(b, persistent_pcg=1)
    np.testing.assert_array_equal(sg.trace_cost, sr.trace_cost)
    np.testing.assert_array_equal(sg.trace_linear_iterations, sr.trace_linear_iterations)
    assert np.array_equal(got.parameters(), ref.parameters())
