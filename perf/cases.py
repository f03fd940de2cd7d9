"""Workloads of the bundle-adjustment library as its users run them, for timing and for comparing results.

A case is a plain dict. `listed()` names the fixed ones, `draw(rng)` gives another one of the same ranges,
`prepare` makes the problems and the solver handle a program holds, `run` is one pass through the public entry
points, `work` what a pass cannot do without, and `exact` the same result from plain torch in 64 bits.

Kinds of case:
  window     one or several local bundle-adjustment windows in the BAL camera model (5-40 cameras on a short walk)
  ring       the small all-around problem: cameras on a ring, every point in 4-10 of them
  request    one reconstruction of a map that grew over a walk, as a serving queue or an offline job hands it in
  loops      a large map: closed loops with more cameras than one cluster takes, the sparse two-kernel solver
  local_ba   stereo windows of a SLAM backend (poses on SE3, outlier test), one by one or as a batch
  step       one damped linear solve, for a program that drives its own trust region
  residuals  residuals and cost of a problem that is already in device memory (a tracking thread, a merge check)
"""
import ctypes
import math
import random

import numpy as np
import torch

from slamplay_gb300 import BALProblem, LocalBAWindow, Solver
from slamplay_gb300 import _native as native
from slamplay_gb300.solver import G2O_VARIANT, LOCAL_BA

# mean observations per point of each generator layout
_VIEWS = {"window": 4.9, "ring": 7.0, "request": 4.9, "step": 4.9, "loops": 5.8, "residuals": 5.0}
_SYNTH = {"window": 3, "ring": 0, "request": 1, "step": 1, "loops": 2}

# the benchmark's rule for capped solves: a fixed number of LM iterations, PCG to 1e-6 or 100 iterations
_CAPPED = dict(function_tolerance=0.0, gradient_tolerance=0.0, parameter_tolerance=0.0, pcg_tolerance=1e-6,
               max_linear_solver_iterations=100)
# what the mixed form is run with to convergence
_MIXED = dict(pcg_tolerance=1e-6, max_linear_solver_iterations=100)


def listed():
    return [
        # a SLAM backend's call after each keyframe: 7 stereo keyframes, the smallest call there is
        {"name": "local_ba_window", "kind": "local_ba", "batch": 1, "cameras": 7, "points": 600,
         "precision": "fp64"},
        # the same windows of many sessions, gathered by a server
        {"name": "local_ba_batch_mixed", "kind": "local_ba", "batch": 64, "cameras": 7, "points": 600,
         "precision": "mixed"},
        # the smallest benchmark problem, Ceres' default tolerances
        {"name": "ring16", "kind": "ring", "cameras": 16, "points": 2000, "precision": "fp64", "rule": "default",
         "loss": "trivial"},
        # one local window through the drop-in call (Huber loss, Ceres' defaults)
        {"name": "window", "kind": "window", "batch": 1, "cameras": 23, "points": 2600, "precision": "fp64",
         "rule": "default", "loss": "huber"},
        # uneven windows solved together: the drop-in precision, and the mixed one that is meant for batches
        {"name": "window_batch", "kind": "window", "batch": 48, "sizes": 5, "precision": "fp64", "rule": "default",
         "loss": "trivial"},
        {"name": "window_batch_mixed", "kind": "window", "batch": 192, "sizes": 6, "precision": "mixed",
         "rule": "default", "loss": "trivial"},
        # a reconstruction of ordinary size, g2o's policy (the other back end a user may come from)
        {"name": "request_g2o", "kind": "request", "cameras": 75, "points": 9001, "precision": "fp64", "rule": "g2o",
         "loss": "huber"},
        # the benchmark's medium problem, both precisions, 50 LM iterations with the PCG capped
        {"name": "walk250", "kind": "request", "cameras": 250, "points": 60000, "precision": "fp64",
         "rule": "capped", "iterations": 50, "loss": "trivial"},
        {"name": "walk250_mixed", "kind": "request", "cameras": 250, "points": 60000, "precision": "mixed",
         "rule": "capped", "iterations": 50, "loss": "trivial"},
        # a map with closed loops, the first iterations after a loop closure
        {"name": "loops_mixed", "kind": "loops", "cameras": 1800, "points": 200000, "precision": "mixed",
         "rule": "capped", "iterations": 10, "loss": "trivial"},
        # one damped linear solve at the reference's start radius
        {"name": "step250", "kind": "step", "cameras": 250, "points": 40000, "precision": "fp64", "radius": 1e3},
        # the cost of a whole map in device memory
        {"name": "residuals_map", "kind": "residuals", "cameras": 1800, "observations": 5000001, "loss": "trivial"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the listed ranges."""
    kind = rng.choice(["window", "window", "window", "ring", "request", "request", "loops", "local_ba", "local_ba",
                       "step", "residuals"])
    precision = rng.choice(["fp64", "mixed"])
    loss = rng.choice(["trivial", "huber", "cauchy"])
    if kind == "window":
        if rng.random() < 0.5:
            return {"kind": kind, "batch": 1, "cameras": rng.randint(5, 40), "points": _log_int(rng, 200, 5000),
                    "precision": precision, "rule": rng.choice(["default", "capped"]), "iterations": 10,
                    "loss": loss}
        return {"kind": kind, "batch": _log_int(rng, 2, 48 if precision == "fp64" else 192),
                "sizes": rng.randint(100, 10 ** 6), "precision": precision, "rule": "default", "loss": loss}
    if kind == "ring":
        return {"kind": kind, "cameras": rng.randint(10, 64), "points": _log_int(rng, 300, 6000),
                "precision": precision, "rule": "default", "loss": loss}
    if kind == "request":
        rule = rng.choice(["default", "capped", "g2o"])
        return {"kind": kind, "cameras": _log_int(rng, 10, 250), "points": _log_int(rng, 1000, 40000),
                "precision": precision, "rule": rule, "iterations": rng.randint(5, 30),
                "loss": "huber" if rule == "g2o" else loss}
    if kind == "loops":
        return {"kind": kind, "cameras": rng.randint(1030, 1800), "points": _log_int(rng, 20000, 200000),
                "precision": "mixed", "rule": "capped", "iterations": rng.randint(3, 10), "loss": loss}
    if kind == "local_ba":
        return {"kind": kind, "batch": rng.choice([1, _log_int(rng, 2, 64)]), "cameras": rng.randint(3, 16),
                "points": _log_int(rng, 100, 1500), "precision": precision}
    if kind == "step":
        return {"kind": kind, "cameras": _log_int(rng, 10, 250), "points": _log_int(rng, 1000, 40000),
                "precision": "fp64", "radius": 10.0 ** rng.randint(1, 3)}
    return {"kind": kind, "cameras": _log_int(rng, 1, 1800), "observations": _log_int(rng, 500, 5000000),
            "loss": loss}


# ---- inputs -----------------------------------------------------------------


def _options(case):
    """The solver options of a case."""
    o = dict(precision=case["precision"])
    if case["kind"] == "local_ba":
        return {**LOCAL_BA, **o}
    if case["kind"] == "step":
        return dict(o, pcg_tolerance=1e-12, max_linear_solver_iterations=2000)
    o.update(loss=case["loss"], loss_scale=1.0)
    if case["rule"] == "capped":
        return dict(o, **_CAPPED, max_num_iterations=case["iterations"])
    if case["rule"] == "g2o":
        o = {**G2O_VARIANT, **o, "max_num_iterations": 15}
    if case["precision"] == "mixed":
        o.update(_MIXED)
    return o


def _window_sizes(case):
    if case.get("batch", 1) == 1:
        return [(case["cameras"], case["points"])]
    r = random.Random(case["sizes"])
    return [(r.randint(5, 40), r.randint(200, 5000)) for _ in range(case["batch"])]


def _problems(case, seed):
    k = _SYNTH[case["kind"]]
    if case["kind"] == "window":
        return [BALProblem.synthetic(k, index=i, seed=seed, num_cameras=nc, num_points=npt)
                for i, (nc, npt) in enumerate(_window_sizes(case))]
    return [BALProblem.synthetic(k, seed=seed, num_cameras=case["cameras"], num_points=case["points"])]


def _features(case):
    """Features of one stereo window: a landmark is tracked in most of its window's images, not in all."""
    return int(0.8 * case["cameras"] * case["points"])


def _window(case, seed):
    """A stereo window of just these sizes: the generator drops landmarks that leave the images, so it starts with
    more of them; some of the features are lost, as a tracker loses them."""
    nk, npt, no = case["cameras"], case["points"], _features(case)
    w = LocalBAWindow.synthetic(seed=seed, num_keyframes=nk, num_landmarks=npt + npt // 4 + 20)
    seen = np.nonzero(w.landmark_index < npt)[0]
    keep = np.sort(np.random.default_rng(seed).permutation(seen)[:no])
    return LocalBAWindow(w.keyframe_index[keep], w.landmark_index[keep], w.rig_camera[keep],
                         w.observations.reshape(-1, 2)[keep], w.poses, w.landmarks[:3 * npt], w.fx, w.fy, w.cx, w.cy,
                         w.extrinsics)


def _windows(case, seed):
    return [_window(case, seed * 1000 + i) for i in range(case["batch"])]


def _resident(case, seed, device):
    """A ring of cameras around a cloud of points in BAL order (by point), in device memory."""
    g = torch.Generator(device=device).manual_seed(seed)
    f = dict(device=device, dtype=torch.float64, generator=g)
    nc, no = case["cameras"], case["observations"]
    npt = max(1, no // 5)
    cams = torch.zeros(nc, 9, device=device, dtype=torch.float64)
    cams[:, 1] = 2 * math.pi * torch.rand(nc, **f) - math.pi
    cams[:, 0:3] += 0.05 * torch.randn(nc, 3, **f)
    cams[:, 5] = -10.0
    cams[:, 3:6] += 0.1 * torch.randn(nc, 3, **f)
    cams[:, 6] = 500.0 * (1 + 0.01 * torch.randn(nc, **f))
    cams[:, 7] = 0.1 * torch.rand(nc, **f) - 0.05
    cams[:, 8] = 0.01 * torch.rand(nc, **f) - 0.005
    pts = 4 * torch.rand(npt, 3, **f) - 2
    ci = torch.randint(0, nc, (no,), device=device, dtype=torch.int32, generator=g)
    pi = (torch.arange(no, device=device) * npt // no).to(torch.int32)
    uv = _snavely(cams, pts, ci.long(), pi.long())[0] + 0.5 * torch.randn(no, 2, **f)
    cams[:, 0:3] += 0.01 * torch.randn(nc, 3, **f)
    pts += 0.1 * torch.randn(npt, 3, **f)
    return cams, pts, ci, pi, uv.contiguous()


def prepare(case, seed):
    if case["kind"] == "residuals":
        cams, pts, ci, pi, uv = _resident(case, seed, "cuda")
        p = native.DeviceProblem(cams.shape[0], pts.shape[0], ci.shape[0], ci.data_ptr(), pi.data_ptr(),
                                 uv.data_ptr(), cams.data_ptr(), pts.data_ptr())
        out = torch.empty(ci.shape[0], 2, device="cuda", dtype=torch.float64)
        cost = torch.empty(1, device="cuda", dtype=torch.float64)
        return {"case": case, "problem": p, "keep": (cams, pts, ci, pi, uv), "residuals": out, "cost": cost,
                "loss": native.LOSS[case["loss"]]}
    s = {"case": case, "solver": Solver(**_options(case))}
    if case["kind"] == "local_ba":
        s["windows"] = _windows(case, seed)
        s["start"] = [(w.poses.copy(), w.landmarks.copy()) for w in s["windows"]]
    else:
        s["problems"] = _problems(case, seed)
        s["start"] = [b.parameters().copy() for b in s["problems"]]
    return s


# ---- one pass -----------------------------------------------------------------


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "residuals":
        stream = torch.cuda.current_stream().cuda_stream
        native.check(native.lib().gba_evaluate_noalloc(ctypes.byref(state["problem"]), state["loss"], 1.0,
                                                       state["residuals"].data_ptr(), state["cost"].data_ptr(), stream),
                     None, "gba_evaluate_noalloc")
        return {"residuals": state["residuals"], "cost": state["cost"]}
    if kind == "step":
        delta, model, _ = state["solver"].compute_step(state["problems"][0], case["radius"])
        return {"delta": delta, "model_cost_change": model}
    if kind == "local_ba":
        ws = state["windows"]
        for w, (poses, landmarks) in zip(ws, state["start"]):
            w.poses[:] = poses
            w.landmarks[:] = landmarks
        got = state["solver"].local_ba(ws)
        return {"poses": np.concatenate([w.poses for w in ws]), "landmarks": np.concatenate([w.landmarks for w in ws]),
                "cost": np.array([s.final_cost for s, _ in got]),
                "outlier": np.concatenate([r["outlier"] for _, r in got])}
    ps = state["problems"]
    for b, x in zip(ps, state["start"]):
        b.parameters()[:] = x
    if len(ps) == 1:
        sums = [state["solver"].solve(ps[0])]
    else:
        sums = state["solver"].batch_solve(ps)
    return {"parameters": np.concatenate([b.parameters() for b in ps]),
            "cost": np.array([s.final_cost for s in sums])}


# ---- what a pass cannot do without ----------------------------------------------


def work(case):
    """Bytes: indices, observations and parameters in, results out, once. Flops: per LM iteration and observation
    one projection with its Jacobian (about 250), the point's and the camera's 3x3, 3x9 and 9x9 products (about
    350) and the back-substitution (about 60); iterations as capped, else ten."""
    kind = case["kind"]
    if kind == "residuals":
        no, npt = case["observations"], max(1, case["observations"] // 5)
        return {"bytes": no * (8 + 16 + 16) + npt * 24 + case["cameras"] * 72, "flops": no * 45}
    if kind == "local_ba":
        no = case["batch"] * _features(case)
        npar = case["batch"] * (6 * case["cameras"] + 3 * case["points"])
        return {"bytes": no * (8 + 1 + 16 + 1) + 16 * npar, "flops": 10 * no * 660}
    sizes = _window_sizes(case) if kind == "window" else [(case["cameras"], case["points"])]
    no = int(sum(p for _, p in sizes) * _VIEWS[kind])
    npar = sum(9 * c + 3 * p for c, p in sizes)
    its = 1 if kind == "step" else case.get("iterations", 10) if case["rule"] == "capped" else 10
    return {"bytes": no * 24 + 16 * npar, "flops": its * no * 660}


# ---- the same results in plain torch, 64 bits -------------------------------------


def _skew(v):
    z = torch.zeros_like(v[..., 0])
    return torch.stack([z, -v[..., 2], v[..., 1], v[..., 2], z, -v[..., 0], -v[..., 1], v[..., 0], z],
                       -1).reshape(*v.shape[:-1], 3, 3)


def _rotation(w):
    """Rotation matrices of angle-axis vectors, (n, 3, 3)."""
    th2 = (w * w).sum(-1)
    th = th2.sqrt()
    K = _skew(w)
    small = th2 <= 2.220446049250313e-16
    s = torch.where(small, torch.ones_like(th), torch.sin(th) / torch.where(small, torch.ones_like(th), th))
    c = torch.where(small, torch.zeros_like(th), (1 - torch.cos(th)) / torch.where(small, torch.ones_like(th), th2))
    eye = torch.eye(3, dtype=w.dtype, device=w.device)
    return eye + s[:, None, None] * K + c[:, None, None] * (K @ K)


def _rotation_derivative(w, R):
    """dR/dw_k, (n, 3, 3, 3) with k first: ([w]_x w_k + [w x (I - R) e_k]_x) R / |w|^2 (Gallego and Yezzi 2015)."""
    th2 = (w * w).sum(-1)
    small = th2 <= 2.220446049250313e-16
    eye = torch.eye(3, dtype=w.dtype, device=w.device)
    out = []
    for k in range(3):
        ek = eye[k].expand_as(w)
        v = torch.linalg.cross(w, ek - R[:, :, k])
        D = (w[:, k, None, None] * _skew(w) + _skew(v)) @ R / torch.where(small, torch.ones_like(th2), th2)[:, None, None]
        out.append(torch.where(small[:, None, None], _skew(ek), D))
    return torch.stack(out, 1)


def _snavely(cams, pts, ci, pi, jacobian=False):
    """Predicted pixels (no, 2), and with `jacobian` the derivatives by camera (no, 2, 9) and point (no, 2, 3)."""
    R = _rotation(cams[:, :3])
    X = pts[pi]
    P = (R[ci] @ X[:, :, None])[:, :, 0] + cams[ci, 3:6]
    xy = -P[:, :2] / P[:, 2:3]
    f, k1, k2 = cams[ci, 6], cams[ci, 7], cams[ci, 8]
    r2 = (xy * xy).sum(1)
    d = 1 + r2 * (k1 + k2 * r2)
    uv = (f * d)[:, None] * xy
    if not jacobian:
        return uv, None, None
    M = d[:, None, None] * torch.eye(2, dtype=P.dtype) + 2 * (k1 + 2 * k2 * r2)[:, None, None] * xy[:, :, None] * xy[:, None, :]
    Z = -torch.cat([torch.eye(2, dtype=P.dtype).expand(len(ci), 2, 2), xy[:, :, None]], 2) / P[:, 2, None, None]
    A = f[:, None, None] * (M @ Z)
    dR = _rotation_derivative(cams[:, :3], R)
    dP = torch.stack([(dR[:, k][ci] @ X[:, :, None])[:, :, 0] for k in range(3)], 2)
    Jc = torch.cat([A @ dP, A, (d[:, None] * xy)[:, :, None], ((f * r2)[:, None] * xy)[:, :, None],
                    ((f * r2 * r2)[:, None] * xy)[:, :, None]], 2)
    return uv, Jc, A @ R[ci]


def _rho(loss, a, s):
    """rho(s), rho'(s) and rho''(s) of the robust losses."""
    one, zero = torch.ones_like(s), torch.zeros_like(s)
    if loss == "huber":
        out = s > a * a
        r = torch.where(out, s, one).sqrt()
        return torch.where(out, 2 * a * r - a * a, s), torch.where(out, a / r, one), \
            torch.where(out, -a / r / (2 * torch.where(out, s, one)), zero)
    if loss == "cauchy":
        t = 1 + s / (a * a)
        return a * a * t.log(), 1 / t, -1 / (a * a * t * t)
    return s, one, zero


def _correct(loss, a, r, Jc, Jp):
    """The robust loss folded into residuals and Jacobians (Triggs' correction, as Ceres applies it)."""
    if loss == "trivial":
        return r, Jc, Jp
    s = (r * r).sum(1)
    _, r1, r2 = _rho(loss, a, s)
    q = r1.sqrt()
    use = (s > 0) & (r2 > 0)
    alpha = torch.where(use, 1 - (1 + 2 * s * r2 / r1).clamp_min(0).sqrt(), torch.zeros_like(s))
    rs = q / (1 - alpha)
    an = torch.where(use, alpha / torch.where(use, s, torch.ones_like(s)), torch.zeros_like(s))

    def fix(J):
        rJ = (r[:, :, None] * J).sum(1, keepdim=True)
        return q[:, None, None] * (J - an[:, None, None] * r[:, :, None] * rJ)

    return rs[:, None] * r, fix(Jc), fix(Jp)


class _Snavely:
    """A BAL problem for `_minimise`."""

    def __init__(self, b, so3):
        self.nc, self.np = b.num_cameras(), b.num_points()
        self.ci = torch.from_numpy(b.camera_index().astype(np.int64))
        self.pi = torch.from_numpy(b.point_index().astype(np.int64))
        self.uv = torch.from_numpy(b.observations().reshape(-1, 2).copy())
        self.x = torch.from_numpy(b.parameters().copy())
        self.so3 = so3

    def split(self, x):
        return x[:9 * self.nc].reshape(-1, 9), x[9 * self.nc:].reshape(-1, 3)

    def residuals(self, x, jacobian):
        c, p = self.split(x)
        uv, Jc, Jp = _snavely(c, p, self.ci, self.pi, jacobian)
        if jacobian and self.so3:  # rotation columns by dw of R <- exp(dw) R: dP/dw = -[R X]_x
            RX = (_rotation(c[:, :3])[self.ci] @ p[self.pi][:, :, None])[:, :, 0]
            Jc[:, :, :3] = -Jc[:, :, 3:6] @ _skew(RX)
        return uv - self.uv, Jc, Jp

    def plus(self, x, dc, dp):
        c, p = self.split(x)
        c2 = c + dc
        if self.so3:
            c2[:, :3] = _log(_rotation(dc[:, :3]) @ _rotation(c[:, :3]))
        return torch.cat([c2.reshape(-1), (p + dp).reshape(-1)])


class _Rig:
    """A stereo window for `_minimise`: the reference's pose Jacobian, taken at the rig camera."""

    def __init__(self, w):
        self.nc, self.np = w.num_keyframes, w.num_landmarks
        self.ci = torch.from_numpy(w.keyframe_index.astype(np.int64))
        self.pi = torch.from_numpy(w.landmark_index.astype(np.int64))
        self.side = torch.from_numpy(w.rig_camera.astype(np.int64))
        self.uv = torch.from_numpy(w.observations.reshape(-1, 2).copy())
        self.x = torch.from_numpy(np.concatenate([w.poses, w.landmarks]))
        self.f = torch.tensor([w.fx, w.fy], dtype=torch.float64)
        self.c = torch.tensor([w.cx, w.cy], dtype=torch.float64)
        self.E = torch.from_numpy(w.extrinsics.copy())

    def split(self, x):
        return x[:6 * self.nc].reshape(-1, 6), x[6 * self.nc:].reshape(-1, 3)

    def residuals(self, x, jacobian):
        T, p = self.split(x)
        R, ER = _rotation(T[:, :3]), _rotation(self.E[:, :3])
        P = (R[self.ci] @ p[self.pi][:, :, None])[:, :, 0] + T[self.ci, 3:]
        Q = (ER[self.side] @ P[:, :, None])[:, :, 0] + self.E[self.side, 3:]
        r = self.uv - (self.f * Q[:, :2] / Q[:, 2:3] + self.c)
        if not jacobian:
            return r, None, None
        D = torch.zeros(len(Q), 2, 3, dtype=Q.dtype)
        D[:, 0, 0], D[:, 1, 1] = -self.f[0] / Q[:, 2], -self.f[1] / Q[:, 2]
        D[:, :, 2] = self.f * Q[:, :2] / (Q[:, 2:3] ** 2)
        Jc = torch.zeros(len(Q), 2, 9, dtype=Q.dtype)
        Jc[:, :, :3], Jc[:, :, 3:6] = -D @ _skew(Q), D
        return r, Jc, D @ ER[self.side] @ R[self.ci]

    def plus(self, x, dc, dp):
        T, p = self.split(x)
        w, u = dc[:, :3], dc[:, 3:6]
        th2 = (w * w).sum(1)
        th = th2.sqrt()
        tiny = th < 1e-4
        ok = torch.where(tiny, torch.ones_like(th), th)
        a = torch.where(tiny, 0.5 - th2 / 24, (1 - torch.cos(ok)) / ok ** 2)
        b = torch.where(tiny, 1 / 6 - th2 / 120, (ok - torch.sin(ok)) / ok ** 3)
        K, dR = _skew(w), _rotation(w)
        V = torch.eye(3, dtype=w.dtype) + a[:, None, None] * K + b[:, None, None] * (K @ K)
        t = (dR @ T[:, 3:, None] + V @ u[:, :, None])[:, :, 0]
        return torch.cat([torch.cat([_log(dR @ _rotation(T[:, :3])), t], 1).reshape(-1), (p + dp).reshape(-1)])


def _log(R):
    """Angle-axis of rotation matrices, through the largest component of the quaternion."""
    m = R.reshape(-1, 9)
    d = torch.stack([1 + m[:, 0] + m[:, 4] + m[:, 8], 1 + m[:, 0] - m[:, 4] - m[:, 8],
                     1 - m[:, 0] + m[:, 4] - m[:, 8], 1 - m[:, 0] - m[:, 4] + m[:, 8]], 1)
    s = [m[:, 7] - m[:, 5], m[:, 2] - m[:, 6], m[:, 3] - m[:, 1]]
    t = [m[:, 1] + m[:, 3], m[:, 2] + m[:, 6], m[:, 5] + m[:, 7]]
    q = torch.stack([torch.stack([d[:, 0], s[0], s[1], s[2]], 1), torch.stack([s[0], d[:, 1], t[0], t[1]], 1),
                     torch.stack([s[1], t[0], d[:, 2], t[2]], 1), torch.stack([s[2], t[1], t[2], d[:, 3]], 1)], 1)
    q = q[torch.arange(len(m)), d.argmax(1)]
    q = q / q.norm(dim=1, keepdim=True)
    q = torch.where(q[:, :1] < 0, -q, q)
    n = q[:, 1:].norm(dim=1)
    return q[:, 1:] * torch.where(n > 0, 2 * torch.atan2(n, q[:, 0]) / torch.where(n > 0, n, torch.ones_like(n)),
                                  2 * torch.ones_like(n))[:, None]


def _damped_solve(m, r, Jc, Jp, dc2, dp2):
    """y of (J^T J + D^2) y = J^T r with the points eliminated and a dense factorisation of the cameras."""
    nc, npt = m.nc, m.np
    C = torch.zeros(npt, 3, 3, dtype=r.dtype).index_add_(0, m.pi, Jp.mT @ Jp) + torch.diag_embed(dp2)
    gp = torch.zeros(npt, 3, dtype=r.dtype).index_add_(0, m.pi, (Jp.mT @ r[:, :, None])[:, :, 0])
    gc = torch.zeros(nc, 9, dtype=r.dtype).index_add_(0, m.ci, (Jc.mT @ r[:, :, None])[:, :, 0])
    Ci = torch.linalg.inv(C)
    Y = Jc.mT @ Jp
    Z = Y @ Ci[m.pi]
    S = torch.zeros(nc * nc, 9, 9, dtype=r.dtype)
    S.index_add_(0, m.ci * nc + m.ci, Jc.mT @ Jc)
    order = torch.argsort(m.pi, stable=True)
    k = 0
    while True:  # the pairs of observations of one point, k places apart
        a, b = order[:len(order) - k], order[k:]
        same = m.pi[a] == m.pi[b]
        if not bool(same.any()):
            break
        a, b = a[same], b[same]
        blk = Z[a] @ Y[b].mT
        S.index_add_(0, m.ci[a] * nc + m.ci[b], -blk)
        if k:
            S.index_add_(0, m.ci[b] * nc + m.ci[a], -blk.mT)
        k += 1
    S = S.reshape(nc, nc, 9, 9).permute(0, 2, 1, 3).reshape(9 * nc, 9 * nc) + torch.diag(dc2.reshape(-1))
    v = gc.index_add(0, m.ci, -(Z @ gp[m.pi][:, :, None])[:, :, 0])
    yc = torch.cholesky_solve(v.reshape(-1, 1), torch.linalg.cholesky(S)).reshape(nc, 9)
    w = torch.zeros(npt, 3, dtype=r.dtype).index_add_(0, m.pi, (Y.mT @ yc[m.ci][:, :, None])[:, :, 0])
    return yc, (Ci @ (gp - w)[:, :, None])[:, :, 0]


def _norms(m, Jc, Jp):
    return (torch.zeros(m.nc, 9, dtype=Jc.dtype).index_add_(0, m.ci, (Jc * Jc).sum(1)),
            torch.zeros(m.np, 3, dtype=Jc.dtype).index_add_(0, m.pi, (Jp * Jp).sum(1)))


def _scaled_step(m, r, Jc, Jp, sc, sp, radius, damping=None):
    """The step and its predicted decrease, in the scaled parameters' own units."""
    Jc, Jp = Jc * sc[m.ci][:, None, :], Jp * sp[m.pi][:, None, :]
    if damping is None:
        dc2, dp2 = (n.clamp(1e-6, 1e32) / radius for n in _norms(m, Jc, Jp))
    else:
        dc2, dp2 = torch.full_like(sc, damping), torch.full_like(sp, damping)
    yc, yp = _damped_solve(m, r, Jc, Jp, dc2, dp2)
    u = -((Jc @ yc[m.ci][:, :, None]) + (Jp @ yp[m.pi][:, :, None]))[:, :, 0]
    return -yc * sc, -yp * sp, float(-(u * (r + u / 2)).sum())


def _minimise(m, o):
    """Ceres' trust-region Levenberg-Marquardt, or g2o's, with exact linear solves: (parameters, cost)."""
    loss, a, g2o = o.get("loss", "trivial"), o.get("loss_scale", 1.0), o.get("lm_policy") == "g2o"
    cap, ftol = o.get("max_num_iterations", 50), o.get("function_tolerance", 1e-6)
    gtol, ptol = o.get("gradient_tolerance", 1e-10), o.get("parameter_tolerance", 1e-8)

    def cost_of(x):
        r = m.residuals(x, False)[0]
        return float(0.5 * _rho(loss, a, (r * r).sum(1))[0].sum())

    x, cost = m.x, cost_of(m.x)
    r, Jc, Jp = _correct(loss, a, *m.residuals(x, True))
    nc2, np2 = _norms(m, Jc, Jp)
    sc, sp = (torch.ones_like(nc2), torch.ones_like(np2)) if g2o else (1 / (1 + nc2.sqrt()), 1 / (1 + np2.sqrt()))
    radius, shrink = (1 / (1e-5 * float(max(nc2.max(), np2.max()))) if g2o else 1e4), 2.0
    it = trials = 0
    while it < cap:
        dc, dp, model = _scaled_step(m, r, Jc, Jp, sc, sp, radius, 1 / radius if g2o else None)
        new = m.plus(x, dc, dp)
        c = cost_of(new)
        c = c if math.isfinite(c) else math.inf
        trials += 1
        it += 0 if g2o else 1
        gain = 2 * (cost - c) / (2 * model + 1e-3) if g2o else (cost - c) / model
        if not g2o and (float((new - x).norm()) <= ptol * (float(x.norm()) + ptol) or abs(cost - c) <= ftol * cost):
            break
        if gain > (0.0 if g2o else 1e-3):
            x, cost = new, c
            t = 1 - (2 * gain - 1) ** 3
            radius /= max(1 / 3, min(2 / 3, t) if g2o else t)
            radius, shrink = (radius if g2o else min(1e16, radius)), 2.0
            it, trials = it + (1 if g2o else 0), 0
            r, Jc, Jp = _correct(loss, a, *m.residuals(x, True))
            g = max(float(torch.zeros(m.nc, 9, dtype=r.dtype).index_add_(0, m.ci, (Jc.mT @ r[:, :, None])[:, :, 0]).abs().max()),
                    float(torch.zeros(m.np, 3, dtype=r.dtype).index_add_(0, m.pi, (Jp.mT @ r[:, :, None])[:, :, 0]).abs().max()))
            if not g2o and g <= gtol:
                break
        else:
            radius /= shrink
            shrink *= 2
            if g2o and (trials >= 10 or gain == 0.0):
                break
    return x, cost


def exact(case, seed):
    """What `run` returns, in plain torch; None where a dense solve of the cameras would take too long or where the
    PCG's cap, not the solution, decides the steps."""
    kind = case["kind"]
    if kind == "residuals":
        cams, pts, ci, pi, uv = _resident(case, seed, "cuda")
        r = _snavely(cams, pts, ci.long(), pi.long())[0] - uv
        return {"residuals": r, "cost": (0.5 * _rho(case["loss"], 1.0, (r * r).sum(1))[0].sum()).reshape(1)}
    if kind == "step":
        m = _Snavely(_problems(case, seed)[0], False)
        r, Jc, Jp = m.residuals(m.x, True)
        nc2, np2 = _norms(m, Jc, Jp)
        dc, dp, model = _scaled_step(m, r, Jc, Jp, 1 / (1 + nc2.sqrt()), 1 / (1 + np2.sqrt()), case["radius"])
        return {"delta": torch.cat([dc.reshape(-1), dp.reshape(-1)]), "model_cost_change": model}
    if case.get("batch", 1) > 4 or kind == "loops" or case.get("rule") == "capped":
        return None
    if case["cameras"] * case["points"] > 10 ** 6 if "cameras" in case else False:
        return None
    o = _options(case)
    if kind == "local_ba":
        got = [_minimise(_Rig(w), o) for w in _windows(case, seed)]
        n = 6 * case["cameras"]
        return {"poses": torch.cat([x[:n] for x, _ in got]), "landmarks": torch.cat([x[n:] for x, _ in got]),
                "cost": np.array([c for _, c in got]), "outlier": None}
    got = [_minimise(_Snavely(b, o.get("camera_update") == "so3_left"), o) for b in _problems(case, seed)]
    # (points seen at almost no parallax slide along their rays: a walk's parameters, and the mixed form's, are one of
    # many minimisers, and only the cost has a value of its own)
    free = kind == "request" or case["precision"] == "mixed"
    return {"parameters": None if free else torch.cat([x for x, _ in got]), "cost": np.array([c for _, c in got])}
