"""gba_evaluate_noalloc at the sizes where its kernel's form changes.

From 2,432 runs of 256 observations a warp takes a whole run, below that a
warp takes 32 observations.  Either form evaluates an observation by the same
instructions, so the residuals of a large problem equal, bit for bit, those of
its slices below the line.  The cost is a sum of non-negative terms over at
most 5 + 8 + 10 + 13 additions in a chain: relative error below 36 * 2^-53,
about 4e-15, plus 3 roundings a term; 1e-14 is asked for.
"""
import ctypes
import math

import numpy as np
import pytest

from slamplay_gb300 import _native as N

pytestmark = pytest.mark.gpu
LINE = 2432 * 256


def _call(torch, cams, pts, obs, ci, pi):
    n = ci.numel()
    dp = N.DeviceProblem(cams.shape[0], pts.shape[0], n, ci.data_ptr(), pi.data_ptr(), obs.data_ptr(),
                         cams.data_ptr(), pts.data_ptr())
    res = torch.full((2 * n,), 7.0, dtype=torch.float64, device="cuda")
    cost = torch.full((1,), -1.0, dtype=torch.float64, device="cuda")
    st = N.lib().gba_evaluate_noalloc(ctypes.byref(dp), 0, 1.0, ctypes.c_void_p(res.data_ptr()),
                                      ctypes.c_void_p(cost.data_ptr()),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    N.check(st, None, "gba_evaluate_noalloc")
    torch.cuda.synchronize()
    return res.cpu().numpy().reshape(-1, 2), float(cost.item())


@pytest.mark.parametrize("n", [LINE - 256, LINE - 255, LINE, LINE + 1, LINE + 7 * 256 + 33, LINE + 8 * 256])
def test_both_forms_agree(n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    nc, npt = 37, 1001
    cams = np.concatenate([rng.normal(0, 0.3, (nc, 3)), rng.normal(0, 0.5, (nc, 3)),
                           np.tile([500.0, -0.1, 0.05], (nc, 1))], axis=1)
    pts = rng.normal(0, 1, (npt, 3)) + [0, 0, -8]
    dev = lambda a, t: torch.tensor(a, dtype=t, device="cuda")
    cams, pts = dev(cams, torch.float64), dev(pts, torch.float64)
    ci = dev(rng.integers(0, nc, n), torch.int32)
    pi = dev(rng.integers(0, npt, n), torch.int32)
    obs = dev(rng.normal(0, 100, (n, 2)), torch.float64)
    res, cost = _call(torch, cams, pts, obs, ci, pi)
    half = n // 2
    for sl in (slice(0, half), slice(half, n)):
        part, _ = _call(torch, cams, pts, obs[sl].contiguous(), ci[sl].contiguous(), pi[sl].contiguous())
        assert np.array_equal(res[sl], part)
    want = math.fsum(0.5 * (res * res).sum(axis=1))
    assert abs(cost - want) <= 1e-14 * want
    ci[n - 1] = nc  # outside: NaN there and in the cost, nothing else changes
    bad, cost = _call(torch, cams, pts, obs, ci, pi)
    assert np.isnan(bad[n - 1]).all() and np.isnan(cost)
    assert np.array_equal(bad[: n - 1], res[: n - 1])
