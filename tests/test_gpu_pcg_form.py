"""Which form of the FP64 PCG a solve runs, as the profile tells it: a cluster
per problem for small problems and batches, the whole GPU for a larger single
problem, two kernels per iteration otherwise."""
import pytest

from slamplay_gb300 import BALProblem, Solver

pytestmark = pytest.mark.gpu


def _form(probs, **opts):
    with Solver(max_num_iterations=2, pcg_tolerance=1e-6, max_linear_solver_iterations=20, schur="explicit", **opts) as s:
        s.set_profiling(True)
        s.batch_solve([p.copy() for p in probs])
        prof = {e["name"]: e for e in s.profile()}
    one, cluster = prof["pcg_grid"]["launches"], prof["pcg_cluster64"]["launches"]
    assert prof["pcg_cluster64"]["total_ms"] == 0.0
    if one == 0:
        assert cluster == 0 and prof["pcg_camera"]["launches"] > 0
        return "two kernels"
    assert cluster in (0, one) and prof["pcg_grid"]["total_ms"] > 0.0
    return "cluster" if cluster else "grid"


def _walk(cams, points, index=0):
    return BALProblem.synthetic(3, index=index, seed=7, num_cameras=cams, num_points=points)


@pytest.mark.parametrize("cams,points,form", [(8, 400, "cluster"), (23, 900, "cluster"), (160, 3000, "grid")])
def test_single_problem(cams, points, form):
    assert _form([_walk(cams, points)]) == form


@pytest.mark.parametrize("cams,form", [(40, "cluster"), (128, "cluster"), (129, "two kernels")])
def test_batch(cams, form):
    assert _form([_walk(cams, 1500), _walk(6, 250, 1)]) == form


def test_switches(monkeypatch):
    assert _form([_walk(23, 900)], persistent_pcg=0) == "two kernels"
    monkeypatch.setenv("GBA_TEST_GRID_CTAS", "500")
    assert _form([_walk(23, 900)]) == "grid"
