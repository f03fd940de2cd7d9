"""The grid PCG (FP64, one problem over the whole GPU) where its CTAs hold
more rows than their shared memory was planned for, as beside other kernels
that hold SMs: fewer CTAs launched (GBA_TEST_GRID_CTAS at handle creation).

Tolerance: none.  Every CTA count runs the two-kernel PCG's additions in the
same order, so parameters, traces and iteration counts agree bitwise."""
import numpy as np
import pytest

from slamplay_gb300 import BALProblem, Solver

pytestmark = pytest.mark.gpu

OPTS = dict(max_num_iterations=3, function_tolerance=0.0, gradient_tolerance=0.0, parameter_tolerance=0.0,
            pcg_tolerance=1e-8, max_linear_solver_iterations=40, schur="explicit")


def _solve(b, **kw):
    g = b.copy()
    with Solver(**{**OPTS, **kw}) as s:
        sm = s.solve(g)
        s.set_profiling(True)
        s.solve(b.copy())
        grid = {e["name"]: e["launches"] for e in s.profile()}.get("pcg_grid", 0) > 0
    return g, sm, grid


# 1: every exchange within one CTA; 2, 7: several passes over the rows, more
# camera blocks than one round of the update; 38: a quarter of the SMs; 0: all.
# 300 cameras: ten chunks of p.q sums, 38 camera blocks; a ring of 70: rows
# of more than 64 blocks.
@pytest.mark.parametrize("layout,cams,points", [(1, 300, 6000), (0, 70, 1500)])
@pytest.mark.parametrize("ctas", [0, 1, 2, 7, 38])
def test_grid_pcg_any_cta_count(monkeypatch, layout, cams, points, ctas):
    b = BALProblem.synthetic(layout, seed=5, num_cameras=cams, num_points=points)
    ref, sr, two = _solve(b, persistent_pcg=0)
    monkeypatch.setenv("GBA_TEST_GRID_CTAS", str(ctas))
    got, sg, one = _solve(b, persistent_pcg=1)
    assert one and not two
    np.testing.assert_array_equal(sg.trace_cost, sr.trace_cost)
    np.testing.assert_array_equal(sg.trace_linear_iterations, sr.trace_linear_iterations)
    assert np.array_equal(got.parameters(), ref.parameters())


def test_grid_pcg_quadratic_criterion():
    b = BALProblem.synthetic(1, seed=6, num_cameras=90, num_points=3000)
    kw = dict(pcg_criterion="quadratic_model", eta=1e-4)
    ref, sr, _ = _solve(b, persistent_pcg=0, **kw)
    got, sg, one = _solve(b, persistent_pcg=1, **kw)
    assert one
    np.testing.assert_array_equal(sg.trace_linear_iterations, sr.trace_linear_iterations)
    assert np.array_equal(got.parameters(), ref.parameters())
