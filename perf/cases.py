"""Workloads this framework is timed on, through its public entry points.

Each case is a dict of plain values; ``kind`` names the entry point:

residual   ReprojectionResidual forward and backward (FP32), or residual_f64 (FP64 forward): the
           differentiable reprojection residual a learned pipeline calls per optimisation step.
product    Plan.schur_product: y = S_lambda x of the reduced camera system of a resident survey, the
           operator a program's own Krylov loop applies.
refresh    refresh_reprojection: the landmarks' residuals after a solve, from host arrays to host arrays.
two_view   CudaBundleAdjuster.solve of an initial pair (two poses, fixed baseline).
window     CudaBundleAdjuster.solve of one local window: a ring of calibrated, self-calibrating or
           spherical (angular residual) cameras, direct or PCG steps.
batch      CudaBundleAdjuster.solve_batched of independent local windows.
survey     Plan.solve of a resident survey with per-camera intrinsics: the global adjustment, FP64 or
           mixed precision, PCG or direct steps, a bounded number of LM iterations and the certificate.

Iterative solves ask for accurate camera steps (a PCG tolerance of 1e-10 or below), so that a result
does not depend on the PCG iteration at which a loose tolerance happens to be met.

Everything is made from the seed alone, on the GPU where that is quicker, with the noise model of
``synthetic`` (0.5 px pixel noise, 5 % outliers, perturbed poses and points).
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "openmvg-rs_b200"))

from openmvg_ba_cuda import BundleProblem, CameraIntrinsics, Gauge, RobustLoss, SolveConfig, abi, autograd, synthetic  # noqa: E402
from openmvg_ba_cuda.adjuster import CudaBundleAdjuster  # noqa: E402
from openmvg_ba_cuda.sfm import LandmarkTracks, refresh_reprojection  # noqa: E402

WIDTH, HEIGHT = synthetic.WIDTH, synthetic.HEIGHT


def listed():
    return [
        # one local window's residuals: a few launches, latency bound
        {"name": "residual_window", "kind": "residual", "dtype": "f32", "observations": 8009, "cameras": 20, "points": 2000},
        # a city-scale reconstruction's residuals: the largest differentiable call
        {"name": "residual_10m", "kind": "residual", "dtype": "f32", "observations": 10_000_000, "cameras": 3000, "points": 2_000_000},
        # the FP64 forward, for finite-difference checks and FP64 evaluation
        {"name": "residual_f64", "kind": "residual", "dtype": "f64", "observations": 1_200_001, "cameras": 500, "points": 200_000},
        # the reduced-system product of the 500-camera survey
        {"name": "product_plane500", "kind": "product", "cameras": 500, "points": 200_000, "extent": 100.0},
        # every landmark of the 3,000-camera survey measured again after its solve
        {"name": "refresh_2m", "kind": "refresh", "views": 3000, "landmarks": 2_000_000, "mixed_models": False},
        # the initial pair of an incremental reconstruction
        {"name": "two_view_pair", "kind": "two_view", "points": 700, "loss": "huber"},
        # one calibrated local window, direct steps: what incremental SfM runs after every added view
        {"name": "window_direct", "kind": "window", "model": "calibrated", "cameras": 20, "points": 2000, "solver": "direct", "loss": "huber", "iterations": 12},
        # the same window with a shared free focal and distortion
        {"name": "window_selfcal", "kind": "window", "model": "self_calibrating", "cameras": 20, "points": 2000, "solver": "direct", "loss": "huber", "iterations": 12},
        # a 360-degree rig's window: angular residuals, Cauchy continuation, PCG steps
        {"name": "window_spherical_pcg", "kind": "window", "model": "spherical", "cameras": 32, "points": 6001, "solver": "iterative", "loss": "cauchy", "iterations": 12},
        # a batch of uneven local windows in one call
        {"name": "batch_32", "kind": "batch", "windows": 32, "max_cameras": 40, "max_points": 5290, "iterations": 8},
        # the 500-camera survey, FP64, direct steps on the banded reduced system
        {"name": "survey500_direct", "kind": "survey", "cameras": 500, "points": 200_000, "extent": 100.0, "precision": "fp64", "solver": "direct", "iterations": 4},
        # the 3,000-camera, 12M-observation survey, mixed precision, PCG steps
        {"name": "survey3000_mixed", "kind": "survey", "cameras": 3000, "points": 2_000_000, "extent": 245.0, "precision": "mixed", "solver": "iterative", "iterations": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["residual", "residual", "product", "refresh", "two_view", "window", "batch", "survey"])
    if kind == "residual":
        n = _log_int(rng, 1000, 10_000_000)
        return {"kind": kind, "dtype": rng.choice(["f32", "f32", "f32", "f64"]), "observations": n,
                "cameras": max(2, min(3000, _log_int(rng, 5, 3000), n // 50)), "points": max(100, min(2_000_000, n // rng.randint(3, 9)))}
    if kind == "refresh":
        n = _log_int(rng, 1000, 2_000_000)
        return {"kind": kind, "views": max(10, n // rng.randint(300, 900)), "landmarks": n, "mixed_models": rng.random() < 0.5}
    if kind == "two_view":
        return {"kind": kind, "points": _log_int(rng, 30, 5000), "loss": rng.choice(["huber", "squared", "cauchy"])}
    if kind == "window":
        cams = rng.randint(6, 40)
        return {"kind": kind, "model": rng.choice(["calibrated", "self_calibrating", "spherical"]), "cameras": cams,
                "points": _log_int(rng, 500, 8000), "solver": rng.choice(["direct", "iterative"]), "loss": rng.choice(["huber", "cauchy"]),
                "iterations": rng.randint(5, 12)}
    if kind == "batch":
        return {"kind": kind, "windows": rng.randint(2, 32), "max_cameras": rng.randint(12, 40), "max_points": _log_int(rng, 700, 5290),
                "iterations": rng.randint(5, 9)}
    cams = _log_int(rng, 60, 1000)  # the survey grids' camera density: 500 cameras over 100 x 100
    c = {"kind": kind, "cameras": cams, "points": cams * rng.randint(150, 450), "extent": round(100.0 * math.sqrt(cams / 500.0), 3)}
    if kind == "product":
        return c
    solver = rng.choice(["direct", "iterative"])
    # few iterations: beyond them the survey's weakest points amplify rounding to the eighth digit
    return {**c, "precision": "mixed" if solver == "iterative" and rng.random() < 0.5 else "fp64", "solver": solver,
            "iterations": rng.randint(2, 4)}


# ---- inputs -----------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, device="cuda", dtype=torch.float64, generator=g) * (hi - lo) + lo


def _normal(g, sigma, *shape):
    return torch.randn(*shape, device="cuda", dtype=torch.float64, generator=g) * sigma


def _integers(g, lo, hi, *shape):
    return torch.randint(lo, hi, shape, device="cuda", generator=g)


def _exp_so3(w):
    th = torch.linalg.vector_norm(w, dim=1)
    z = torch.zeros_like(th)
    k = torch.stack([z, -w[:, 2], w[:, 1], w[:, 2], z, -w[:, 0], -w[:, 1], w[:, 0], z], dim=1).reshape(-1, 3, 3)
    safe = torch.where(th > 1e-12, th, torch.ones_like(th))
    a = torch.where(th > 1e-12, torch.sin(th) / safe, torch.ones_like(th))
    b = torch.where(th > 1e-12, (1 - torch.cos(th)) / safe**2, torch.full_like(th, 0.5))
    return torch.eye(3, device=w.device, dtype=w.dtype) + a[:, None, None] * k + b[:, None, None] * (k @ k)


def _np(t, dtype=None):
    a = t.cpu().numpy()
    return a if dtype is None else a.astype(dtype)


def _residual_inputs(case, seed):
    """synthetic.residual_inputs on the GPU: points in front of an owning camera, observed in no order by
    those of the 16 cameras with the closest viewing directions that see them; pixels with noise and
    outliers, as a reconstruction's are."""
    g = _generator(seed)
    n, cameras, points = case["observations"], case["cameras"], case["points"]
    rotvec = _normal(g, 1.0, cameras, 3)
    rotvec = rotvec * (_uniform(g, 0.0, math.pi, cameras) / torch.linalg.vector_norm(rotvec, dim=1))[:, None]
    trans = _uniform(g, 0.0, 1.0, cameras, 3)
    intr = torch.stack([_uniform(g, 400, 600, cameras), _uniform(g, -0.1, 0.0, cameras), _uniform(g, 0.0, 0.01, cameras)], dim=1)
    owner = _integers(g, 0, cameras, points)
    depth = _uniform(g, 2.0, 50.0, points)
    pc = torch.cat([_uniform(g, -0.4, 0.4, points, 2) * depth[:, None], depth[:, None]], dim=1)
    R = _exp_so3(rotvec)
    X = torch.einsum("nji,nj->ni", R[owner], pc - trans[owner])
    axis = R[:, 2, :]
    order = torch.argsort(axis @ axis.T, dim=1, descending=True, stable=True)
    near, away = order[:, :16], order[:, -1]
    pt = _integers(g, 0, points, n)
    own = owner[pt]

    def camera_point(c):
        return torch.einsum("nij,nj->ni", R[c], X[pt]) + trans[c]

    cam = near[own, _integers(g, 0, near.shape[1], n)]
    q = camera_point(cam)
    cam = torch.where((q[:, 2] > 1.0) & (q[:, 0] ** 2 + q[:, 1] ** 2 < 0.5 * q[:, 2] ** 2), cam, own)  # the owner sees its points
    behind = (torch.rand(n, device="cuda", generator=g) < 0.002) & (camera_point(away[own])[:, 2] < -0.5)
    cam = torch.where(behind, away[own], cam)  # a few observations behind their camera
    q = camera_point(cam)
    xy = q[:, :2] / q[:, 2:]
    r2 = (xy * xy).sum(1)
    pixel = (intr[cam, 0] * (1 + intr[cam, 1] * r2 + intr[cam, 2] * r2 * r2))[:, None] * xy + _normal(g, 0.5, n, 2)
    outlier = (torch.rand(n, device="cuda", generator=g) < 0.05) | behind
    pixel = torch.where(outlier[:, None], _uniform(g, -300, 300, n, 2), pixel)
    dtype = torch.float32 if case["dtype"] == "f32" else torch.float64
    state = {"cam": cam.to(torch.int32), "pt": pt.to(torch.int32), "pixel": pixel.to(dtype),
             "leaves": [a.to(dtype).contiguous() for a in (rotvec, trans, intr, X)]}
    if case["dtype"] == "f32":
        state["grad"] = _normal(g, 1.0, n, 2).to(dtype)
        for leaf in state["leaves"]:
            leaf.requires_grad_()
    return state


def _survey(seed, cameras, points, extent, free_intrinsics, mean_track=6.5, altitude=16.0, chunk=250_000):
    """synthetic.plane_problem on the GPU: serpentine rows of cameras over a ground plane, tracks of
    3 + a geometric number of the cameras that see each point (all of them where fewer do)."""
    g = _generator(seed)
    rows = int(round(math.sqrt(cameras * 0.8)))
    cols = int(math.ceil(cameras / rows))
    idx = torch.arange(cameras, device="cuda")
    r, c = idx // cols, idx % cols
    c = torch.where(r % 2 == 0, c, cols - 1 - c)
    cell_w, cell_h = extent / cols, extent / rows
    C = torch.stack([(c + 0.5) * cell_w, (r + 0.5) * cell_h, torch.full((cameras,), altitude, device="cuda")], dim=1).double()
    C = C + _normal(g, 1.0, cameras, 3) * torch.tensor([0.1, 0.1, 0.3], device="cuda", dtype=torch.float64)
    zero = torch.zeros(cameras, device="cuda", dtype=torch.float64)
    yaw = _exp_so3(torch.stack([zero, zero, torch.where(r % 2 == 0, zero, zero + math.pi)], dim=1))
    down = torch.diag(torch.tensor([1.0, -1.0, -1.0], device="cuda", dtype=torch.float64))
    R = _exp_so3(_normal(g, 0.03, cameras, 3)) @ down @ yaw.transpose(1, 2)
    f0, ppx, ppy = 500.0, WIDTH / 2, HEIGHT / 2
    if free_intrinsics:
        k1s, k2s, fs = _uniform(g, -0.12, -0.06, cameras), _uniform(g, 0.0, 0.02, cameras), f0 * _uniform(g, 0.97, 1.03, cameras)
    else:
        k1s, k2s, fs = zero - 0.09, zero + 0.01, zero + f0
    X = torch.stack([_uniform(g, 0, extent, points), _uniform(g, 0, extent, points), _uniform(g, 0, 2.0, points)], dim=1)
    rad = altitude * (WIDTH / 2) / f0 * 1.3
    kx, ky = int(math.ceil(rad / cell_w)) + 1, int(math.ceil(rad / cell_h)) + 1
    off_c, off_r = (a.reshape(-1) for a in torch.meshgrid(torch.arange(-kx, kx + 1, device="cuda"),
                                                          torch.arange(-ky, ky + 1, device="cuda"), indexing="ij"))
    cam_at = torch.full((rows, cols), -1, device="cuda", dtype=torch.int64)
    cam_at[r, c] = idx
    want = 3 + torch.empty(points, device="cuda", dtype=torch.float64).geometric_(1.0 / (mean_track - 2.0), generator=g).long() - 1
    parts = []
    for start in range(0, points, chunk):
        Xc = X[start:start + chunk]
        cc = torch.clamp((Xc[:, 0] / cell_w).long(), 0, cols - 1)[:, None] + off_c
        rr = torch.clamp((Xc[:, 1] / cell_h).long(), 0, rows - 1)[:, None] + off_r
        inside = (cc >= 0) & (cc < cols) & (rr >= 0) & (rr < rows)
        cand = torch.where(inside, cam_at[rr.clamp(0, rows - 1), cc.clamp(0, cols - 1)], -1)
        ci = cand.clamp(min=0)
        d = Xc[:, None, :] - C[ci]
        xc = torch.einsum("nmij,nmj->nmi", R[ci], d)
        xn, yn = xc[..., 0] / xc[..., 2], xc[..., 1] / xc[..., 2]
        r2 = xn * xn + yn * yn
        s = fs[ci] * (1.0 + k1s[ci] * r2 + k2s[ci] * r2 * r2)
        u, v = s * xn + ppx, s * yn + ppy
        vis = (cand >= 0) & (xc[..., 2] > 0.5) & (r2 < 0.81) & (u > 8) & (u < WIDTH - 8) & (v > 8) & (v < HEIGHT - 8)
        key = torch.where(vis, torch.rand(cand.shape, device="cuda", generator=g), 2.0)
        order = torch.argsort(key, dim=1)
        take = torch.minimum(want[start:start + chunk], vis.sum(dim=1))
        sel_p, rank = torch.nonzero(torch.arange(cand.shape[1], device="cuda")[None] < take[:, None], as_tuple=True)
        sel = order[sel_p, rank]
        parts.append((sel_p + start, cand[sel_p, sel], u[sel_p, sel], v[sel_p, sel]))
        del d, xc, xn, yn, r2, s, u, v, vis, key, order, cand, ci, cc, rr, inside
    obs_point, obs_pose, u, v = (torch.cat(a) for a in zip(*parts))
    n = len(u)
    pix = torch.stack([u, v], dim=1) + _normal(g, 0.5, n, 2)
    outlier = torch.rand(n, device="cuda", generator=g) < 0.05
    pix = torch.where(outlier[:, None], torch.stack([_uniform(g, 0, WIDTH, n), _uniform(g, 0, HEIGHT, n)], dim=1), pix)
    pose_np = _np(obs_pose, np.uint32)
    if free_intrinsics:
        f_init, k1_init = fs * (1.0 + _normal(g, 0.005, cameras)), k1s + _normal(g, 0.005, cameras)
        intr = [CameraIntrinsics(model=abi.CAMERA_BROWN_CONRADY, fx=f, fy=f, cx=ppx, cy=ppy, radial_kind=abi.RADIAL_K1K2, k1=a, k2=b,
                                 variables=abi.INTRINSIC_FOCAL | abi.INTRINSIC_RADIAL)
                for f, a, b in zip(f_init.tolist(), k1_init.tolist(), k2s.tolist())]
        obs_intr = pose_np.copy()
    else:
        intr = [CameraIntrinsics(model=abi.CAMERA_BROWN_CONRADY, fx=f0, fy=f0, cx=ppx, cy=ppy, radial_kind=abi.RADIAL_K1K2, k1=-0.09, k2=0.01)]
        obs_intr = np.zeros_like(pose_np)
    return BundleProblem(
        rotations=_np(_exp_so3(_normal(g, 0.01, cameras, 3)) @ R), centers=_np(C + _normal(g, 0.05, cameras, 3)),
        pose_variables=np.full(cameras, abi.POSE_FREE, dtype=np.uint32), intrinsics=intr, points=_np(X + _normal(g, 0.02, points, 3)),
        point_fixed=np.zeros(points, dtype=np.uint8), observation_pose=pose_np, observation_intrinsic=obs_intr,
        observation_point=_np(obs_point, np.uint32), observation_pixel=_np(pix), robust_loss=RobustLoss.huber(1.0), gauge=Gauge())


def _look_at(C):
    z = -C / torch.linalg.vector_norm(C, dim=1, keepdim=True)
    x = torch.linalg.cross(torch.tensor([0.0, 0.0, 1.0], device="cuda", dtype=torch.float64).expand_as(z), z)
    x = x / torch.linalg.vector_norm(x, dim=1, keepdim=True)
    return torch.stack([x, torch.linalg.cross(z, x), z], dim=1)


def _ring(case, seed):
    """synthetic.ring_problem on the GPU: cameras on a ring looking inwards, 3-8 observations a point;
    spherical cameras' residuals are angles."""
    g = _generator(seed)
    cameras, points, model = case["cameras"], case["points"], case["model"]
    radius = {"calibrated": 10.0, "self_calibrating": 3.0, "spherical": 3.0}[model]
    ang = torch.arange(cameras, device="cuda", dtype=torch.float64) * (2 * math.pi / cameras)
    C = torch.stack([radius * torch.cos(ang), radius * torch.sin(ang), 0.05 * radius * torch.sin(3 * ang)], dim=1)
    R = _look_at(C)
    X = _uniform(g, -1.0, 1.0, points, 3)
    longest = min(8, cameras)
    counts = _integers(g, 3, longest + 1, points)
    order = torch.argsort(torch.rand(points, cameras, device="cuda", generator=g), dim=1)[:, :longest]
    obs_point, rank = torch.nonzero(torch.arange(longest, device="cuda")[None] < counts[:, None], as_tuple=True)
    pose = order[obs_point, rank]
    n = len(pose)
    q = torch.einsum("nij,nj->ni", R[pose], X[obs_point] - C[pose])
    extra = {}
    scale = {"huber": RobustLoss.huber, "cauchy": RobustLoss.cauchy}[case["loss"]]
    if model == "spherical":
        width = 2048
        lon, lat = torch.atan2(q[:, 0], q[:, 2]), torch.atan2(q[:, 1], torch.hypot(q[:, 0], q[:, 2]))
        pix = torch.stack([(lon + math.pi) * width / (2 * math.pi) - 0.5, (lat + math.pi / 2) * (width // 2) / math.pi - 0.5], dim=1)
        pix = pix + _normal(g, 0.3, n, 2)
        intr = CameraIntrinsics(model=abi.CAMERA_SPHERICAL, width=width, height=width // 2)
        loss = RobustLoss(abi.LOSS_HUBER if case["loss"] == "huber" else abi.LOSS_CAUCHY, 1e-3, abi.RESIDUAL_ANGULAR)
        extra["residual_space"] = abi.RESIDUAL_ANGULAR
        rot, centre, move = 0.005, 0.02, 0.01
    else:
        f, cx, cy, k1, k2, k3 = 500.0, 320.0, 240.0, -0.1, 0.01, (-0.001 if model == "calibrated" else 0.0)
        xn, yn = q[:, 0] / q[:, 2], q[:, 1] / q[:, 2]
        r2 = xn * xn + yn * yn
        s = f * (1.0 + k1 * r2 + k2 * r2 * r2 + k3 * r2**3)
        pix = torch.stack([s * xn + cx, s * yn + cy], dim=1) + _normal(g, 0.5, n, 2)
        outlier = torch.rand(n, device="cuda", generator=g) < 0.05
        pix = torch.where(outlier[:, None], torch.stack([_uniform(g, 0, WIDTH, n), _uniform(g, 0, HEIGHT, n)], dim=1), pix)
        if model == "calibrated":
            intr = CameraIntrinsics(model=abi.CAMERA_BROWN_CONRADY, fx=f, fy=f, cx=cx, cy=cy, radial_kind=abi.RADIAL_K1K2K3, k1=k1, k2=k2, k3=k3)
        else:
            intr = CameraIntrinsics(model=abi.CAMERA_BROWN_CONRADY, fx=505.0, fy=505.0, cx=cx, cy=cy, radial_kind=abi.RADIAL_K1K2,
                                    k1=-0.09, k2=0.0, variables=abi.INTRINSIC_FOCAL | abi.INTRINSIC_RADIAL)
        loss = scale(1.0 if case["loss"] == "huber" else 2.0)
        rot, centre, move = 0.01, 0.05, 0.02
    return BundleProblem(
        rotations=_np(_exp_so3(_normal(g, rot, cameras, 3)) @ R), centers=_np(C + _normal(g, centre, cameras, 3)),
        pose_variables=np.full(cameras, abi.POSE_FREE, dtype=np.uint32), intrinsics=[intr], points=_np(X + _normal(g, move, points, 3)),
        point_fixed=np.zeros(points, dtype=np.uint8), observation_pose=_np(pose, np.uint32),
        observation_intrinsic=np.zeros(n, dtype=np.uint32), observation_point=_np(obs_point, np.uint32), observation_pixel=_np(pix),
        robust_loss=loss, gauge=Gauge(), **extra)


def _pair(case, seed):
    """An initial pair: points 2-6 units in front of two cameras a short baseline apart, 0.5 px noise."""
    g = _generator(seed)
    points = case["points"]
    X = torch.cat([_uniform(g, -0.8, 0.8, points, 2), _uniform(g, 0.0, 1.0, points, 1)], dim=1)
    X[:, 2] = 2.0 + 4.0 * X[:, 2]
    t = torch.tensor([0.8, 0.1, 0.15], device="cuda", dtype=torch.float64)
    R = _exp_so3(torch.tensor([[0.04, -0.08, 0.025]], device="cuda", dtype=torch.float64))[0]
    cams = [dict(fx=500.0, fy=510.0, cx=320.0, cy=240.0), dict(fx=520.0, fy=515.0, cx=315.0, cy=238.0)]

    def pixels(cam, q):
        p = torch.stack([cam["fx"] * q[:, 0] / q[:, 2] + cam["cx"], cam["fy"] * q[:, 1] / q[:, 2] + cam["cy"]], dim=1)
        return p + _normal(g, 0.5, points, 2)

    pix = torch.cat([pixels(cams[0], X), pixels(cams[1], X @ R.T + t)])
    t0 = t + _normal(g, 0.02, 3)
    baseline = torch.linalg.vector_norm(t)
    t0 = t0 * baseline / torch.linalg.vector_norm(t0)
    R0 = _exp_so3(_normal(g, 0.01, 1, 3))[0] @ R
    z = np.zeros(points, dtype=np.uint32)
    loss = {"huber": RobustLoss.huber(1.0), "squared": RobustLoss.squared(), "cauchy": RobustLoss.cauchy(2.0)}[case["loss"]]
    centre = -_np(R0).T @ _np(t0)
    return BundleProblem(
        rotations=np.stack([np.eye(3), _np(R0)]), centers=np.stack([np.zeros(3), centre]),
        pose_variables=np.array([0, abi.POSE_FREE], dtype=np.uint32),
        intrinsics=[CameraIntrinsics(model=abi.CAMERA_PINHOLE, **c) for c in cams], points=_np(X + _normal(g, 0.02, points, 3)),
        point_fixed=np.zeros(points, dtype=np.uint8), observation_pose=np.concatenate([z, z + 1]),
        observation_intrinsic=np.concatenate([z, z + 1]), observation_point=np.tile(np.arange(points, dtype=np.uint32), 2),
        observation_pixel=_np(pix), robust_loss=loss, gauge=Gauge.fixed_baseline(0, 1, float(np.linalg.norm(centre))))


_REFRESH_CAMERAS = [
    CameraIntrinsics(model=abi.CAMERA_BROWN_CONRADY, fx=650.0, fy=640.0, cx=330.0, cy=245.0, radial_kind=abi.RADIAL_K1K2K3, k1=-0.08,
                     k2=0.01, k3=0.001, tangential_kind=abi.TANGENTIAL_P1P2, p1=1e-3, p2=-5e-4),
    CameraIntrinsics(model=abi.CAMERA_PINHOLE, fx=700.0, fy=690.0, cx=320.0, cy=240.0),
    CameraIntrinsics(model=abi.CAMERA_FISHEYE, fx=300.0, fy=300.0, cx=320.0, cy=240.0),
    CameraIntrinsics(model=abi.CAMERA_SPHERICAL, width=2048, height=1024),
]


def _refresh_project(model, q):
    """Pixels of camera points q under row `model` of _REFRESH_CAMERAS, plain FP64."""
    c = _REFRESH_CAMERAS[model]
    if model < 2:
        x, y = q[:, 0] / q[:, 2], q[:, 1] / q[:, 2]
        if model == 0:
            r2 = x * x + y * y
            s = 1.0 + c.k1 * r2 + c.k2 * r2**2 + c.k3 * r2**3
            x, y = (x * s + 2 * c.p1 * x * y + c.p2 * (r2 + 2 * x * x), y * s + c.p1 * (r2 + 2 * y * y) + 2 * c.p2 * x * y)
        return torch.stack([c.fx * x + c.cx, c.fy * y + c.cy], dim=1)
    if model == 2:
        radial = torch.hypot(q[:, 0], q[:, 1])
        s = torch.atan2(radial, q[:, 2]) / radial
        return torch.stack([c.fx * q[:, 0] * s + c.cx, c.fy * q[:, 1] * s + c.cy], dim=1)
    lon, lat = torch.atan2(q[:, 0], q[:, 2]), torch.atan2(q[:, 1], torch.hypot(q[:, 0], q[:, 2]))
    return torch.stack([(lon + math.pi) * c.width / (2 * math.pi) - 0.5, (lat + math.pi / 2) * c.height / math.pi - 0.5], dim=1)


def _refresh_inputs(case, seed):
    """A ring of views around the landmarks, tracks of 2-10 views (mean 6), a few views without a pose,
    some observations outside the support, inactive landmarks, 3 % gross outliers."""
    g = _generator(seed)
    L, V = case["landmarks"], case["views"]
    ang = torch.arange(V, device="cuda", dtype=torch.float64) * (2 * math.pi / V)
    C = torch.stack([4.0 * torch.cos(ang), 4.0 * torch.sin(ang), 0.3 * torch.sin(2 * ang)], dim=1)
    R = _look_at(C)
    view_model = torch.arange(V, device="cuda") % 4 if case["mixed_models"] else torch.arange(V, device="cuda") % 2
    posed = torch.rand(V, device="cuda", generator=g) > 0.03
    X = _uniform(g, -1.0, 1.0, L, 3)
    counts = _integers(_generator(L), 2, 11, L)  # the track lengths belong to the case, not to the seed
    offset = torch.zeros(L + 1, device="cuda", dtype=torch.int64)
    offset[1:] = torch.cumsum(counts, 0)
    n = int(offset[-1])
    owner = torch.repeat_interleave(torch.arange(L, device="cuda"), counts)
    first = _integers(g, 0, V, L)  # consecutive views of a trajectory, as a track has them
    view = (first[owner] + (torch.arange(n, device="cuda") - offset[owner])) % V
    q = torch.einsum("nij,nj->ni", R[view], X[owner] - C[view])
    pix = torch.empty(n, 2, device="cuda", dtype=torch.float64)
    model = view_model[view]
    for m in range(4):
        at = torch.nonzero(model == m)[:, 0]
        pix[at] = _refresh_project(m, q[at])
    pix = pix + _normal(g, 0.7, n, 2)
    outlier = torch.rand(n, device="cuda", generator=g) < 0.03
    pix = torch.where(outlier[:, None], pix + _uniform(g, -100, 100, n, 2), pix)
    support = torch.rand(n, device="cuda", generator=g) > 0.08
    active = torch.rand(L, device="cuda", generator=g) > 0.02
    pose = torch.where(posed[view], view, abi.NO_POSE)
    tracks = LandmarkTracks(points=_np(X), active=_np(active, np.uint8), track_offset=_np(offset, np.uint64),
                            track_pose=_np(pose, np.uint32), track_intrinsic=_np(model, np.uint32), track_pixel=_np(pix),
                            track_support=_np(support, np.uint8))
    return _np(R), _np(C), tracks


def _config(case):
    """Solve options of the window and survey cases."""
    if case["kind"] == "window":
        direct = case["solver"] == "direct"
        return SolveConfig(linear_solver=abi.SOLVER_DIRECT if direct else abi.SOLVER_ITERATIVE, max_iterations=case["iterations"],
                           pcg_relative_tolerance=0.0 if direct else 1e-10)
    direct = case.get("solver") == "direct"
    return SolveConfig(linear_solver=abi.SOLVER_DIRECT if direct else abi.SOLVER_ITERATIVE, max_iterations=case.get("iterations", 1),
                       precision=abi.PRECISION_MIXED if case.get("precision") == "mixed" else abi.PRECISION_FP64,
                       pcg_relative_tolerance=0.0 if direct else 1e-11)


_adjusters = []


def _adjuster():
    """The one solver context a program opens at start-up."""
    if not _adjusters:
        _adjusters.append(CudaBundleAdjuster(torch.cuda.current_device()))
    return _adjusters[0]


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "residual":
        return {**state, **_residual_inputs(case, seed)}
    state["adjuster"] = _adjuster()
    if kind == "refresh":
        R, C, tracks = _refresh_inputs(case, seed)
        return {**state, "rotations": R, "centers": C, "tracks": tracks}
    if kind == "two_view":
        return {**state, "problem": _pair(case, seed), "config": SolveConfig()}
    if kind == "window":
        return {**state, "problem": _ring(case, seed), "config": _config(case)}
    if kind == "batch":
        rng = np.random.Generator(np.random.PCG64(case["windows"]))  # the windows' sizes belong to the case
        cams = rng.integers(5, case["max_cameras"] + 1, size=case["windows"])
        pts = np.exp(rng.uniform(math.log(500), math.log(case["max_points"]), size=case["windows"])).astype(int)
        problems = [_ring({"model": "calibrated", "loss": "huber", "cameras": int(c), "points": int(p)}, 1000 * seed + w)
                    for w, (c, p) in enumerate(zip(cams, pts))]
        return {**state, "problems": problems, "config": SolveConfig(max_iterations=case["iterations"])}
    problem = _survey(seed, case["cameras"], case["points"], case["extent"], True)
    state["plan"] = state["adjuster"].plan(problem, _config(case))
    if kind == "product":
        dim = state["plan"].info()["reduced_dimension"]
        state["x"] = _normal(_generator(seed + 1), 1.0, dim)
        state["y"] = torch.empty_like(state["x"])
        torch.cuda.synchronize()
        state["plan"].schur_product(state["x"].data_ptr(), state["y"].data_ptr(), 0.1)  # linearizes once
    return state


def _solution(s):
    held = np.zeros(len(s.points), dtype=np.uint8)
    held[s.quarantined_points.astype(np.int64)] = 1
    return {"rotations": s.rotations, "centers": s.centers, "points": s.points,
            "intrinsics": np.array([[c.fx, c.k1, c.k2] for c in s.intrinsics]), "quarantined": held,
            "cost": s.report["final_objective"],
            "counts": np.array([s.report[k] for k in ("iteration_count", "accepted_step_count", "status", "observability")])}


def run(state):
    kind = state["case"]["kind"]
    if kind == "residual":
        if state["case"]["dtype"] == "f64":
            return autograd.residual_f64(state["cam"], state["pt"], state["pixel"], *state["leaves"])
        residual = autograd.reprojection_residual(state["cam"], state["pt"], state["pixel"], *state["leaves"])
        return [residual.detach(), *torch.autograd.grad(residual, state["leaves"], state["grad"])]
    if kind == "product":
        state["plan"].schur_product(state["x"].data_ptr(), state["y"].data_ptr(), 0.1)
        return state["y"]
    if kind == "refresh":
        r = refresh_reprojection(state["adjuster"], state["rotations"], state["centers"], _REFRESH_CAMERAS, state["tracks"])
        return {"update": r.landmark_update, "error": r.reprojection_error, "support": r.track_support,
                "counts": np.array([r.rejected_landmarks, r.removed_observations])}
    if kind == "batch":
        out = [_solution(s) for s in state["adjuster"].solve_batched(state["problems"], state["config"])]
        return {k: np.concatenate([np.atleast_1d(o[k]).reshape(-1) for o in out]) for k in out[0]}
    if kind == "survey":
        return _solution(state["plan"].solve())
    return _solution(state["adjuster"].solve(state["problem"], state["config"]))


def work(case):
    """Bytes: every input read once and every output written once. Flops: the projections, their
    Jacobians and, for solves, the point elimination of every observation and LM iteration."""
    kind = case["kind"]
    if kind == "residual":
        n, s = case["observations"], 4 if case["dtype"] == "f32" else 8
        tables = (9 * case["cameras"] + 3 * case["points"]) * s
        fwd = n * (8 + 4 * s) + tables
        return {"bytes": fwd, "flops": 60 * n} if s == 8 else {"bytes": fwd + n * 8 + 4 * s * n // 2 + 2 * tables, "flops": 260 * n}
    if kind == "product":
        n = 6 * case["points"]
        return {"bytes": n * (24 * 8 + 4) + 48 * case["points"], "flops": 150 * n}
    if kind == "refresh":
        n = 6 * case["landmarks"]
        return {"bytes": n * 26 + case["landmarks"] * 50, "flops": 80 * n}
    if kind == "two_view":
        return {"bytes": case["points"] * (2 * 28 + 2 * 24), "flops": case["points"] * 2000.0}
    if kind == "window":
        n = 5 * case["points"]
        return {"bytes": n * 28 + case["points"] * 48, "flops": case["iterations"] * 600 * n}
    if kind == "batch":
        mean = (case["max_points"] - 500) / math.log(case["max_points"] / 500)
        n = 5.5 * mean * case["windows"]
        return {"bytes": n * 28 + n * 8, "flops": case["iterations"] * 600 * n}
    n = 6 * case["points"]
    return {"bytes": n * 28 + case["points"] * 48, "flops": (case["iterations"] + 1) * 600.0 * n}


# ---- the same in plain FP64 ----------------------------------------------------------------------
def _exact_residual(case, seed):
    state = _residual_inputs(case, seed)
    cam, pt, pixel = state["cam"].long(), state["pt"].long(), state["pixel"].double()
    leaves = [a.detach().double().requires_grad_() for a in state["leaves"]]
    rotvec, trans, intr, X = leaves
    w2 = (rotvec * rotvec).sum(1)
    th = torch.sqrt(w2)
    z = torch.zeros_like(th)
    K = torch.stack([z, -rotvec[:, 2], rotvec[:, 1], rotvec[:, 2], z, -rotvec[:, 0], -rotvec[:, 1], rotvec[:, 0], z], dim=1).reshape(-1, 3, 3)
    R = torch.eye(3, device="cuda", dtype=torch.float64) + (torch.sin(th) / th)[:, None, None] * K + ((1 - torch.cos(th)) / w2)[:, None, None] * (K @ K)
    with torch.no_grad():  # the admissible observations: in front, inside the first radial turn, positive distortion determinant
        q = torch.einsum("nij,nj->ni", R[cam], X[pt]) + trans[cam]
        ok = q[:, 2] > 64 * 2.220446049250313e-16 * q.abs().amax(dim=1)
        k1, k2 = intr[cam, 1], intr[cam, 2]
        r2 = torch.where(ok, (q[:, 0] ** 2 + q[:, 1] ** 2) / q[:, 2] ** 2, 0.0)
        # smallest positive root of 1 + 3 k1 s + 5 k2 s^2
        disc = 9 * k1 * k1 - 20 * k2
        root = torch.where(disc >= 0, -2.0 / (3 * k1 - torch.sqrt(disc.clamp(min=0))), math.inf)
        dist = 1 + k1 * r2 + k2 * r2 * r2
        det = dist * (dist + 2 * r2 * (k1 + 2 * k2 * r2))
        ok &= ~((disc >= 0) & (root > 0) & (r2 >= root)) & (det > 1e-12)
    at = torch.nonzero(ok)[:, 0]
    cam, pt = cam[at], pt[at]
    q = torch.einsum("nij,nj->ni", R[cam], X[pt]) + trans[cam]
    n = q[:, :2] / q[:, 2:]
    r2 = (n * n).sum(1)
    part = (intr[cam, 0] * (1 + intr[cam, 1] * r2 + intr[cam, 2] * r2 * r2))[:, None] * n - pixel[at]
    residual = torch.full_like(pixel, math.nan)
    residual[at] = part.detach()
    if case["dtype"] == "f64":
        return residual
    return [residual, *torch.autograd.grad(part, leaves, state["grad"].double()[at])]


def _exact_refresh(case, seed):
    R, C, tracks = _refresh_inputs(case, seed)
    dev = lambda a, t=torch.float64: torch.from_numpy(a.astype(np.int64) if t is torch.int64 else a).cuda().to(t)  # noqa: E731
    R, C, X, pix = dev(R), dev(C), dev(tracks.points), dev(tracks.track_pixel)
    pose, model, offset = dev(tracks.track_pose, torch.int64), dev(tracks.track_intrinsic, torch.int64), dev(tracks.track_offset, torch.int64)
    L = len(X)
    owner = torch.repeat_interleave(torch.arange(L, device="cuda"), offset[1:] - offset[:-1])
    supporting = dev(tracks.track_support) > 0
    posed = pose != abi.NO_POSE
    at = pose.clamp(max=len(R) - 1)
    q = torch.einsum("nij,nj->ni", R[at], X[owner] - C[at])
    r = torch.zeros(len(pix), device="cuda", dtype=torch.float64)
    valid = torch.ones(len(pix), device="cuda", dtype=torch.bool)
    for m in range(4):
        i = torch.nonzero(model == m)[:, 0]
        c, o = _REFRESH_CAMERAS[m], pix[i]
        if m < 2:
            r[i] = torch.linalg.vector_norm(_refresh_project(m, q[i]) - o, dim=1)
            continue
        if m == 2:
            d = (o - torch.tensor([c.cx, c.cy], device="cuda")) / c.fx
            td = torch.linalg.vector_norm(d, dim=1)
            b = torch.cat([d * (torch.sin(td) / td)[:, None], torch.cos(td)[:, None]], dim=1)
            scale = c.fx
        else:
            lon, lat = (o[:, 0] + 0.5) * (2 * math.pi) / c.width - math.pi, (o[:, 1] + 0.5) * math.pi / c.height - math.pi / 2
            b = torch.stack([torch.cos(lat) * torch.sin(lon), torch.sin(lat), torch.cos(lat) * torch.cos(lon)], dim=1)
            valid[i] = (o[:, 1] >= -0.5) & (o[:, 1] <= c.height - 0.5)
            scale = c.width / (2 * math.pi)
        e = q[i] / torch.linalg.vector_norm(q[i], dim=1, keepdim=True) - b
        r[i] = 2 * torch.asin(0.5 * torch.linalg.vector_norm(e, dim=1)) * scale
    keep = supporting & posed & valid
    zero = torch.zeros(L, device="cuda", dtype=torch.float64)
    kept = zero.index_add(0, owner, keep.double())
    total = zero.index_add(0, owner, torch.where(keep, r, 0.0))
    done = (dev(tracks.active) > 0) & (kept >= 2)
    return {"update": None, "error": torch.where(done, total / kept.clamp(min=1), 0.0), "support": None, "counts": None}


def exact(case, seed):
    """Solves and reduced-system products have no closed form outside this framework: None."""
    if case["kind"] == "residual":
        return _exact_residual(case, seed)
    if case["kind"] == "refresh":
        return _exact_refresh(case, seed)
    return None
