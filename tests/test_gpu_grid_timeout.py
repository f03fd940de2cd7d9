"""The grid PCG's waits that run out, where a CTA's shares take another path
through the kernel: one CTA (every exchange with itself, rows in several
passes, camera blocks in several rounds), a few, and the quadratic-model
test.  GBA_TEST_GRID_WAIT lets every wait look for a tag that nothing writes:
a bounded wait, an error code, and a context that stays usable."""
import numpy as np
import pytest

from slamplay_gb300 import BALProblem, GBAError, Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas,opts", [(1, {}), (7, {}), (38, {}), (500, dict(pcg_criterion="quadratic_model", eta=1e-4))])
def test_wait_runs_out(monkeypatch, ctas, opts):
    b = BALProblem.synthetic(1, seed=5, num_cameras=90, num_points=2500)
    opts = dict(max_num_iterations=2, pcg_tolerance=1e-6, max_linear_solver_iterations=40, schur="explicit", **opts)
    monkeypatch.setenv("GBA_TEST_GRID_CTAS", str(ctas))
    ref = b.copy()
    with Solver(**opts) as s:
        s.solve(ref)
    monkeypatch.setenv("GBA_TEST_GRID_WAIT", "1")
    with Solver(**opts) as s:
        with pytest.raises(GBAError) as e:
            s.solve(b.copy())
        assert e.value.status == 5  # GBA_ERR_TIMEOUT
    monkeypatch.delenv("GBA_TEST_GRID_WAIT")
    got = b.copy()
    with Solver(**opts) as s:
        s.solve(got)
    assert np.array_equal(got.parameters(), ref.parameters())
