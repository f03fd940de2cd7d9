"""FP64 formation of the explicit Schur complement at its edges: rounds of 64
pairs staged 32 at a time and shared by three runs, two CTAs a block.

Four cameras that all see every point: each of the six blocks has one pair
per point.  At radius 1 the Jacobi-scaled reduced system's condition number
is below 13 (column blocks of J of norms at most 3 and sqrt(3), damping 1),
so with the PCG at 1e-13 the step agrees with the CPU oracle's to about
13 * 1e-13 plus rounding; 1e-10 in the relative norm is asked for.  A pair
left out or counted twice moves these steps by 1e-3 and more.
"""
import numpy as np
import pytest

from oracle import oracle_py as O
from slamplay_gb300 import BALProblem, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npt", [1, 2, 3, 31, 32, 33, 34, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191])
def test_formation_pair_counts(npt):
    nc = 4
    b = BALProblem.synthetic(0, seed=npt, num_cameras=nc, num_points=npt)
    ci, pi = np.repeat(np.arange(nc), npt), np.tile(np.arange(npt), nc)
    blank = BALProblem.from_arrays(nc, npt, ci, pi, np.zeros(2 * nc * npt), b.parameters())
    with Solver() as s:
        seen, _, _ = s.evaluate(blank)
    obs = seen + np.random.default_rng(npt).normal(scale=2.0, size=seen.shape)
    d = BALProblem.from_arrays(nc, npt, ci, pi, obs, b.parameters())
    opts = dict(pcg_tolerance=1e-13, max_linear_solver_iterations=500)
    with Solver(schur="explicit", **opts) as s:
        step, _, _ = s.compute_step(d, 1.0)
        _, J, _ = s.evaluate(d)
    want, _, _, ok = O.compute_step(O.Problem.from_bal(d), 1.0, linear_solver="pcg_schur", **opts)
    assert ok
    sq = (J * J).sum(axis=1)
    cam, pt = np.zeros((nc, 9)), np.zeros((npt, 3))
    np.add.at(cam, ci, sq[:, :9])
    np.add.at(pt, pi, sq[:, 9:])
    scale = 1.0 + np.sqrt(np.concatenate([cam.ravel(), pt.ravel()]))
    assert np.linalg.norm(scale * (step - want)) <= 1e-10 * np.linalg.norm(scale * want)
