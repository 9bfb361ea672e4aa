"""The residual forward's shared-memory camera table (csrc/residual.cu: at least 2^18 observations, 32 per
camera, the table within 200 KB, aligned pixels) at the edges of its rule, against the kernel that
recomputes the camera per observation (reached by calls of fewer observations) and the FP64 forward; and
the adjoint on few cameras and points, where every warp's contributions meet in the same accumulators,
against torch's FP64 autograd of the same formula.

Tolerances: FP32 predictions of pixels up to ~1e3 carry a few units of 6e-8 relative, 2e-3 px covers them
(the tolerance of the FP32 forward's parity test); the adjoint's relative norm 2e-4 likewise."""
import numpy as np
import pytest

from openmvg_ba_cuda import synthetic

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EDGE = 1 << 18


def _dev(d, dtype):
    return (torch.as_tensor(d["camera_index"].astype(np.int32), device="cuda"),
            torch.as_tensor(d["point_index"].astype(np.int32), device="cuda"),
            *(torch.as_tensor(d[k], dtype=dtype, device="cuda")
              for k in ("pixel", "rotvec", "translation", "intrinsics", "points")))


@pytest.mark.parametrize("observations,cameras", [(EDGE, 1), (EDGE + 7, 40), (EDGE + 255, 1600), (EDGE, 3200),
                                                  (EDGE + 1, 3201)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_table_forward_equals_the_per_observation_forward(observations, cameras, dtype):
    from openmvg_ba_cuda.autograd import reprojection_residual, residual_f64
    d = synthetic.residual_inputs(seed=cameras, observations=observations, cameras=cameras, points=20_000,
                                  dtype=np.float64)
    cam, pt, px, rv, tr, it, X = _dev(d, dtype)
    cam[3], pt[5] = cameras, -1  # out of range: NaN in both kernels
    f = reprojection_residual if dtype == torch.float32 else residual_f64
    whole = f(cam, pt, px, rv, tr, it, X)
    half = observations // 2
    parts = torch.cat([f(cam[s].contiguous(), pt[s].contiguous(), px[s].contiguous(), rv, tr, it, X)
                       for s in (slice(0, half), slice(half, observations))])
    assert torch.equal(torch.isnan(whole), torch.isnan(parts))
    assert bool(torch.isnan(whole[3]).all()) and bool(torch.isnan(whole[5]).all())
    near = torch.nan_to_num(parts).abs() < 1e4  # a point next to a camera's plane projects far outside
    tol = 2e-3 if dtype == torch.float32 else 1e-9
    assert float((torch.nan_to_num(whole) - torch.nan_to_num(parts))[near].abs().max()) < tol


def test_unaligned_pixels_take_the_per_observation_forward():
    from openmvg_ba_cuda.autograd import reprojection_residual
    d = synthetic.residual_inputs(seed=2, observations=EDGE, cameras=50, points=20_000, dtype=np.float64)
    cam, pt, px, rv, tr, it, X = _dev(d, torch.float32)
    flat = torch.empty(2 * EDGE + 1, device="cuda")
    view = flat[1:].view(EDGE, 2)  # contiguous, 4-byte aligned
    view.copy_(px)
    a, b = reprojection_residual(cam, pt, view, rv, tr, it, X), reprojection_residual(cam, pt, px, rv, tr, it, X)
    assert torch.equal(torch.isnan(a), torch.isnan(b))
    near = torch.nan_to_num(b).abs() < 1e4
    assert float((torch.nan_to_num(a) - torch.nan_to_num(b))[near].abs().max()) < 2e-3


@pytest.mark.parametrize("observations,cameras,points", [(1, 1, 1), (31, 1, 2), (33, 2, 1), (5000, 3, 7), (70_001, 5, 300)])
def test_adjoint_of_crowded_accumulators(observations, cameras, points):
    from openmvg_ba_cuda.autograd import vjp
    rng = np.random.default_rng(observations)
    rv = 0.1 * rng.normal(size=(cameras, 3)) + 0.01
    tr = rng.uniform(0.0, 0.5, size=(cameras, 3))
    it = np.stack([rng.uniform(400, 600, cameras), rng.uniform(-0.1, 0, cameras), rng.uniform(0, 0.01, cameras)], axis=1)
    X = np.concatenate([rng.uniform(-1, 1, size=(points, 2)), rng.uniform(4, 8, size=(points, 1))], axis=1)
    cam, pt = rng.integers(0, cameras, observations), rng.integers(0, points, observations)
    px, g = rng.uniform(-200, 200, size=(observations, 2)), rng.normal(size=(observations, 2))
    f32 = lambda a: torch.as_tensor(a, dtype=torch.float32, device="cuda")  # noqa: E731
    i32 = lambda a: torch.as_tensor(a.astype(np.int32), device="cuda")  # noqa: E731
    got = vjp(i32(cam), i32(pt), f32(px), f32(rv), f32(tr), f32(it), f32(X), f32(g))
    leaves = [f32(a).double().requires_grad_() for a in (rv, tr, it, X)]
    w, t, f, P = leaves
    th = torch.linalg.vector_norm(w, dim=1)[:, None, None]
    z = torch.zeros_like(w[:, 0])
    K = torch.stack([z, -w[:, 2], w[:, 1], w[:, 2], z, -w[:, 0], -w[:, 1], w[:, 0], z], dim=1).reshape(-1, 3, 3)
    R = torch.eye(3, device="cuda", dtype=torch.float64) + torch.sin(th) / th * K + (1 - torch.cos(th)) / th**2 * (K @ K)
    ci, pi = torch.as_tensor(cam, device="cuda"), torch.as_tensor(pt, device="cuda")
    q = torch.einsum("nij,nj->ni", R[ci], P[pi]) + t[ci]
    n = q[:, :2] / q[:, 2:]
    r2 = (n * n).sum(1)
    res = (f[ci, 0] * (1 + f[ci, 1] * r2 + f[ci, 2] * r2 * r2))[:, None] * n - f32(px).double()
    want = torch.autograd.grad(res, leaves, f32(g).double())
    for a, b in zip(got, want):
        assert float(torch.linalg.vector_norm(a.double() - b)) <= 2e-4 * float(torch.linalg.vector_norm(b)) + 1e-12


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 1e30])
def test_adjoint_of_a_camera_without_a_finite_rotation(bad):
    """Its observations are inadmissible, so it contributes nothing anywhere: its gradients are zero, and the
    other cameras' are those of the call without its observations."""
    from openmvg_ba_cuda.autograd import vjp
    d = synthetic.residual_inputs(seed=3, observations=5000, cameras=7, points=500, dtype=np.float64)
    cam, pt, px, rv, tr, it, X = _dev(d, torch.float32)
    rv[2, 1] = bad
    g = torch.ones_like(px)
    got = vjp(cam, pt, px, rv, tr, it, X, g)
    g[cam == 2] = 0.0
    want = vjp(cam, pt, px, torch.nan_to_num(rv, nan=0.0, posinf=0.0).clamp(max=10.0), tr, it, X, g)
    for a, b in zip(got[:3], want[:3]):
        assert float(a[2].abs().max()) == 0.0
        assert torch.equal(a, b)
    assert torch.equal(got[3], want[3])


@pytest.mark.parametrize("count", [1 << 32, 1 << 58, 1 << 59, (1 << 64) - 1])
def test_a_camera_count_whose_products_wrap_takes_the_per_observation_forward(count):
    """The count only bounds the indices: the arrays hold the cameras that the observations name. The same
    bits as that kernel's, which calls of fewer observations take."""
    import ctypes as C
    from openmvg_ba_cuda import abi
    from openmvg_ba_cuda._lib import lib
    from openmvg_ba_cuda.autograd import residual_f64
    d = synthetic.residual_inputs(seed=4, observations=EDGE, cameras=40, points=20_000, dtype=np.float64)
    cam, pt, px, rv, tr, it, X = _dev(d, torch.float64)
    half = EDGE // 2
    want = torch.cat([residual_f64(cam[s].contiguous(), pt[s].contiguous(), px[s].contiguous(), rv, tr, it, X)
                      for s in (slice(0, half), slice(half, EDGE))])
    got, err = torch.empty_like(want), abi.Error()
    assert lib().omvgba_residual_forward_f64(torch.cuda.current_stream().cuda_stream, EDGE, cam.data_ptr(),
                                             pt.data_ptr(), px.data_ptr(), count, rv.data_ptr(), tr.data_ptr(),
                                             it.data_ptr(), X.shape[0], X.data_ptr(), got.data_ptr(),
                                             C.byref(err)) == 0
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(want))
