"""The key by which a handle replays a captured solve (tests/cpu/graph_key.cpp)
and, on a GPU, the two batches of equal totals one after the other on a
handle."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from slamplay_gb300 import BALProblem, Solver

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "slamplay_gb300", "csrc")
CUDA_INC = "/usr/local/cuda/include"


def test_key_holds_every_launch_parameter(tmp_path):
    if shutil.which("g++") is None or not os.path.isdir(CUDA_INC):
        pytest.skip("g++ or the CUDA headers are missing")
    out = str(tmp_path / "graph_key")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "include"), "-I", CSRC,
                    "-I", CUDA_INC, os.path.join(ROOT, "tests", "cpu", "graph_key.cpp"),
                    os.path.join(CSRC, "prep.cpp"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr


def _ring(ci, pi, nc, seed):
    """Cameras around a cloud of points, pixels with noise, a start off the truth."""
    r = np.random.default_rng(seed)
    npt = int(pi.max()) + 1
    a, X = 2 * np.pi * r.random(nc), 4 * r.random((npt, 3)) - 2
    # (a rotation about y by a, the cloud ten units in front)
    R = np.zeros((nc, 3, 3))
    R[:, 0, 0] = R[:, 2, 2] = np.cos(a)
    R[:, 0, 2], R[:, 2, 0], R[:, 1, 1] = np.sin(a), -np.sin(a), 1.0
    P = np.einsum("nij,nj->ni", R[ci], X[pi]) + np.array([0.0, 0.0, -10.0])
    uv = -500.0 * P[:, :2] / P[:, 2:] + 0.5 * r.standard_normal((len(ci), 2))
    cams = np.zeros((nc, 9))
    cams[:, 1] = np.where(a > np.pi, a - 2 * np.pi, a)
    cams[:, 5], cams[:, 6] = -10.0, 500.0
    cams[:, :3] += 0.01 * r.standard_normal((nc, 3))
    X = X + 0.05 * r.standard_normal(X.shape)
    return BALProblem.from_arrays(nc, npt, ci, pi, uv, np.concatenate([cams.ravel(), X.ravel()]))


def _groups(n, seed):
    """n groups of 8 cameras, each with 32 points that all of its cameras see."""
    j = np.arange(32 * n)
    return _ring((j[:, None] // 32 * 8 + np.arange(8)).ravel(), np.repeat(j, 8), 8 * n, seed)


def _pairs(n, seed):
    """n cameras, a point for each two of them."""
    a, b = np.triu_indices(n, 1)
    return _ring(np.stack([a, b], 1).ravel(), np.repeat(np.arange(len(a)), 2), n, seed)


# Tolerance: none, a replay of the right graph gives the bits of a fresh handle.
@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_equal_totals_other_split_on_one_handle(precision):
    opts = dict(max_num_iterations=4, function_tolerance=0.0, gradient_tolerance=0.0, parameter_tolerance=0.0,
                pcg_tolerance=1e-8, max_linear_solver_iterations=60, schur="explicit", precision=precision)
    batches = [[_pairs(40, 1), _groups(6, 2), _groups(6, 3)], [_pairs(40, 1), _groups(10, 2), _groups(2, 3)]]
    with Solver(**opts) as s:
        for probs in batches + batches[:1]:
            got, ref = [p.copy() for p in probs], [p.copy() for p in probs]
            sums = s.batch_solve(got)
            with Solver(**opts) as f:
                want = f.batch_solve(ref)
            for g, r, x, y in zip(got, ref, sums, want):
                np.testing.assert_array_equal(x.trace_cost, y.trace_cost)
                assert np.array_equal(g.parameters(), r.parameters())
