"""The FP64 cluster PCG where one camera shares points with every other (a
hub) and the others with few: the mean row of S is short, so the product runs
by warps over several rows a pass, and the hub's nine rows are longer than a
warp.

Tolerance: none.  The cluster form runs the two-kernel PCG's additions in the
same order, so parameters, costs, cost traces and PCG iteration counts agree
bitwise."""
import numpy as np
import pytest

from slamplay_gb300 import BALProblem, Solver

pytestmark = pytest.mark.gpu

OPTS = dict(max_num_iterations=5, function_tolerance=0.0, gradient_tolerance=0.0, parameter_tolerance=0.0,
            pcg_tolerance=1e-8, max_linear_solver_iterations=120, schur="explicit")


def _project(cam, X):
    w, th = cam[:3], np.linalg.norm(cam[:3])
    k, c, s = w / th, np.cos(th), np.sin(th)
    P = X * c + np.cross(k, X) * s + np.outer(X @ k, k) * (1 - c) + cam[3:6]
    xy = -P[:, :2] / P[:, 2:3]
    r2 = (xy * xy).sum(1)
    return cam[6] * (1 + r2 * (cam[7] + cam[8] * r2))[:, None] * xy, P[:, 2] < -0.5  # (in front of the camera)


def _hub(cams, points, hub, seed):
    """A walk's window whose camera `hub` sees a point of every other camera."""
    b = BALProblem.synthetic(3, seed=seed, num_cameras=cams, num_points=points)
    ci, pi = b.camera_index(), b.point_index()
    uv, front = _project(b.parameters()[9 * hub:9 * hub + 9], b.parameters()[9 * cams:].reshape(-1, 3))
    seen, add = set(pi[ci == hub].tolist()), []
    for c in range(cams):
        own = pi[ci == c]
        if c == hub or seen.intersection(own.tolist()):
            continue
        add.append(own[front[own]][0])
        seen.add(int(add[-1]))
    add = np.array(add, dtype=np.int32)
    ci, pi = np.concatenate([ci, np.full(len(add), hub, np.int32)]), np.concatenate([pi, add])
    covisible = [set() for _ in range(cams)]
    for p in range(points):
        see = ci[pi == p].tolist()
        for c in see:
            covisible[c].update(see)
    rows = [len(s) for s in covisible]  # blocks of the camera's rows of S, the diagonal one among them
    assert rows[hub] == cams and sum(rows) < 17 * cams
    return BALProblem.from_arrays(cams, points, ci, pi,
                                  np.concatenate([b.observations().reshape(-1, 2), uv[add]]), b.parameters())


def _solve(probs, **opts):
    gs = [p.copy() for p in probs]
    with Solver(**{**OPTS, **opts}) as s:
        sums = s.batch_solve(gs) if len(gs) > 1 else [s.solve(gs[0])]
        s.set_profiling(True)
        s.batch_solve([p.copy() for p in probs])
        prof = {e["name"]: e["launches"] for e in s.profile()}
    return gs, sums, prof


# one problem: rows of 32 and 33 blocks (the edge of a pass) to 50 (two runs
# of 32); in a batch also 65 and 96 (three), 97 and 128 (four).  Hubs: the
# first camera (its rows are the warps' first passes), one further in, the last.
@pytest.mark.parametrize("cams,points,batch,hub", [(c, p, False, h) for c, p in ((32, 500), (33, 500), (36, 600), (40, 600),
                                                                                 (44, 700), (50, 800))
                                                   for h in (0, c // 2, c - 1)] +
                         [(c, p, True, h) for c, p in ((40, 600), (65, 900), (96, 1000), (97, 1000), (128, 1200))
                          for h in (0, c // 3)])
def test_hub_camera_equals_two_kernel_bitwise(cams, points, batch, hub):
    probs = [_hub(cams, points, hub, cams)]
    if batch:
        probs.append(BALProblem.synthetic(3, index=1, seed=3, num_cameras=6, num_points=250))
    ga, sa, pa = _solve(probs, persistent_pcg=1)
    gb, sb, pb = _solve(probs, persistent_pcg=0)
    assert pa["pcg_cluster64"] > 0 and pb["pcg_grid"] == 0
    for a, b, x, y in zip(ga, gb, sa, sb):
        np.testing.assert_array_equal(x.trace_cost, y.trace_cost)
        np.testing.assert_array_equal(x.trace_linear_iterations, y.trace_linear_iterations)
        assert np.array_equal(a.parameters(), b.parameters())
