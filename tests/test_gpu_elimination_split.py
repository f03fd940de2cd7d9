"""FP64 point elimination with one and with two CTAs a chunk.

A problem alone, of at most half as many chunks as the GPU has SMs, takes two
CTAs a chunk; in a batch of more chunks one.  The sums are the same, so each
problem gets the same bits either way (the camera side and the formation read
what the elimination wrote)."""
import numpy as np
import pytest

from slamplay_gb300 import BALProblem, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,npt", [(1, 3), (2, 40), (5, 300), (9, 1500), (40, 700)])
def test_alone_equals_batch(nc, npt):
    probs = [BALProblem.synthetic(3, index=0, seed=nc, num_cameras=nc, num_points=npt)]
    probs += [BALProblem.synthetic(3, index=i, seed=5, num_cameras=30, num_points=3000) for i in range(1, 4)]
    opts = dict(max_num_iterations=4, schur="explicit", pcg_tolerance=1e-10, max_linear_solver_iterations=200,
                function_tolerance=0.0, gradient_tolerance=0.0, parameter_tolerance=0.0)
    with Solver(**opts) as s:
        a = probs[0].copy()
        sa = s.solve(a)
        qs = [p.copy() for p in probs]
        sb = s.batch_solve(qs)
    assert np.array_equal(a.parameters(), qs[0].parameters())
    assert sa.final_cost == sb[0].final_cost
