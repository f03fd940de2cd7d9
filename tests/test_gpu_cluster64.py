"""The FP64 cluster PCG (one thread-block cluster per problem) against the
two-kernel FP64 PCG, through the C ABI.

Tolerance: none.  Both forms run the same additions in the same order, so
parameters, costs, cost traces and PCG iteration counts agree bitwise, alone
and in a batch."""
import numpy as np
import pytest

from slamplay_gb300 import BALProblem, Solver

pytestmark = pytest.mark.gpu

OPTS = dict(max_num_iterations=5, function_tolerance=0.0, gradient_tolerance=0.0, parameter_tolerance=0.0,
            pcg_tolerance=1e-8, max_linear_solver_iterations=120, schur="explicit")


def _batch(probs, **opts):
    gs = [p.copy() for p in probs]
    with Solver(**{**OPTS, **opts}) as s:
        sums = s.batch_solve(gs) if len(gs) > 1 else [s.solve(gs[0])]
        s.set_profiling(True)
        s.batch_solve([p.copy() for p in probs])
        one_launch = {e["name"]: e["launches"] for e in s.profile()}.get("pcg_grid", 0) > 0
    return gs, sums, one_launch


def _same(probs, **opts):
    ga, sa, one = _batch(probs, persistent_pcg=1, **opts)
    gb, sb, two = _batch(probs, persistent_pcg=0, **opts)
    assert one and not two
    for a, b, x, y in zip(ga, gb, sa, sb):
        np.testing.assert_array_equal(x.trace_cost, y.trace_cost)
        np.testing.assert_array_equal(x.trace_linear_iterations, y.trace_linear_iterations)
        assert np.array_equal(a.parameters(), b.parameters())
    return ga


# cameras: one and two camera blocks and their edges (8, 9, 16, 17), one and
# two chunks of the p.q sums (32, 33), rows of more than 32 blocks (dense
# rings of 33 and 60), the most blocks a cluster updates (128)
@pytest.mark.parametrize("layout,cams,points", [(0, 2, 60), (0, 3, 80), (3, 5, 200), (0, 8, 300), (3, 9, 400),
                                                (0, 16, 700), (3, 17, 700), (3, 32, 900), (0, 33, 900),
                                                (0, 60, 1200), (3, 128, 1500)])
def test_cluster64_equals_two_kernel_bitwise(layout, cams, points):
    kw = dict(min_views=2, max_views=2) if cams < 4 else {}
    b = BALProblem.synthetic(layout, seed=cams, num_cameras=cams, num_points=points, **kw)
    _same([b, BALProblem.synthetic(3, index=1, seed=3, num_cameras=6, num_points=250)])


@pytest.mark.parametrize("crit", ["residual", "quadratic_model"])
def test_cluster64_single_and_criteria(crit):
    b = BALProblem.synthetic(3, seed=4, num_cameras=21, num_points=900)
    _same([b], pcg_criterion=crit, eta=1e-4)


def test_cluster64_uneven_batch_equals_alone():
    """Problems of 5 to 40 cameras, one with a camera that sees points twice
    (a block with itself) and one without observations: the batch gives each
    problem the bits of its own solve."""
    probs = [BALProblem.synthetic(3, index=i, seed=7, num_cameras=c, num_points=p)
             for i, (c, p) in enumerate([(5, 250), (40, 1500), (23, 333), (12, 800)])]
    d = probs[2]
    dup = np.nonzero(d.camera_index() == 1)[0][:10]
    probs[2] = BALProblem.from_arrays(d.num_cameras(), d.num_points(),
                                      np.concatenate([d.camera_index(), d.camera_index()[dup]]),
                                      np.concatenate([d.point_index(), d.point_index()[dup]]),
                                      np.concatenate([d.observations().reshape(-1, 2),
                                                      d.observations().reshape(-1, 2)[dup] + 0.3]), d.parameters())
    e = probs[0]
    probs.append(BALProblem.from_arrays(e.num_cameras(), e.num_points(), [], [], [], e.parameters()))
    got = _same(probs)
    for p, g in zip(probs[:4], got):
        q = p.copy()
        with Solver(**OPTS) as s:
            s.solve(q)
        assert np.array_equal(q.parameters(), g.parameters())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_late_shape_equals_alone(precision):
    """Thirty problems that end at different LM iterations: once few of them
    run, a launch of another shape takes over; each problem keeps the bits of
    its own solve, with the graph and with the host-driven loop."""
    probs = [BALProblem.synthetic(3, index=i, seed=11, num_cameras=5 + i, num_points=200 + 40 * i) for i in range(30)]
    opts = dict(max_num_iterations=30, schur="explicit", pcg_tolerance=1e-6, max_linear_solver_iterations=60,
                precision=precision)
    runs = []
    for graphs in (1, 0):
        gs = [p.copy() for p in probs]
        with Solver(use_graphs=graphs, **opts) as s:
            sums = s.batch_solve(gs)
        runs.append(gs)
    its = sorted(x.num_iterations for x in sums)
    assert its[0] < its[-1]
    for p, a, b in zip(probs, *runs):
        q = p.copy()
        with Solver(**opts) as s:
            s.solve(q)
        assert np.array_equal(q.parameters(), a.parameters()) and np.array_equal(q.parameters(), b.parameters())
