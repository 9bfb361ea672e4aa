"""PCG of a small system in one cluster kernel (k_pcg_loop) against the graph of per-iteration kernels over
the matrix-free product: one block, one task per row, the last size whose tasks fit (64 blocks in rows of
64), the first that does not, a shared intrinsic group, masks, angular residuals, and runs that end at the
iteration limit or at a loose tolerance.

The two take the same recurrences over products that agree to rounding: the same iteration and acceptance
counts, the final cost to 1e-9, parameters to 1e-7 (the parity tests' tolerances)."""
import numpy as np
import pytest

from openmvg_ba_cuda import SolveConfig, abi, synthetic

pytestmark = pytest.mark.gpu


def _ring(cameras, **kw):
    return synthetic.ring_problem(seed=10, cameras=cameras, points=900, radius=3.0, **kw)


def _one_camera():
    masks = np.zeros(8, dtype=np.uint32)
    masks[3] = abi.POSE_FREE
    return _ring(8, pose_variables=masks)


def _masks():
    return _ring(20, pose_variables=np.array([0, 0] + [1, 2, 3] * 6, dtype=np.uint32))


CASES = {"one_camera": _one_camera, "masks": _masks, "ring_8": lambda: _ring(8), "ring_33": lambda: _ring(33),
         "ring_65": lambda: _ring(65), "ring_66": lambda: _ring(66),
         "shared_group": lambda: _ring(20, self_calibrating=True)}


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("tolerance,limit", [(1e-10, 0), (1e-10, 3), (1e-1, 0)])
def test_cluster_pcg_equals_the_graph_pcg(adjuster, case, tolerance, limit):
    p = CASES[case]()
    cfg = SolveConfig(linear_solver=abi.SOLVER_ITERATIVE, max_iterations=6, pcg_relative_tolerance=tolerance,
                      pcg_max_iterations=limit)
    a = adjuster.solve(p, cfg)
    b = adjuster.solve(p, cfg.with_(matvec=abi.MATVEC_IMPLICIT))
    for k in ("iteration_count", "accepted_step_count", "rejected_step_count", "rejected_step_solve", "status",
              "pcg_iteration_count", "observability", "unconstrained_intrinsic_count"):
        assert a.report[k] == b.report[k], (k, a.report[k], b.report[k])
    assert abs(a.report["final_objective"] - b.report["final_objective"]) <= 1e-9 * b.report["final_objective"]
    assert np.max(np.abs(a.rotations - b.rotations)) < 1e-7 and np.max(np.abs(a.centers - b.centers)) < 1e-7
    assert np.max(np.abs(a.points - b.points)) < 1e-7
    again = adjuster.solve(p, cfg)
    assert np.array_equal(a.points, again.points) and np.array_equal(a.centers, again.centers)


def test_plan_product_of_an_explicit_operator(adjuster):
    """A plan whose PCG uses the explicit rows builds them for its product too."""
    torch = pytest.importorskip("torch")
    p = _ring(20)
    cfg = SolveConfig(linear_solver=abi.SOLVER_ITERATIVE, max_iterations=2)
    out = []
    for matvec in (abi.MATVEC_AUTO, abi.MATVEC_EXPLICIT, abi.MATVEC_IMPLICIT):
        with adjuster.plan(p, cfg.with_(matvec=matvec)) as plan:
            d = plan.info()["reduced_dimension"]
            x = torch.linspace(-1.0, 1.0, d, dtype=torch.float64, device="cuda")
            y = torch.empty_like(x)
            torch.cuda.synchronize()
            plan.schur_product(x.data_ptr(), y.data_ptr(), 0.1)
            torch.cuda.synchronize()
            out.append(y)
    for y in out[:2]:
        assert float((y - out[2]).abs().max()) <= 1e-9 * float(out[2].abs().max())


def _unobserved_pose():
    p = _ring(20)
    return _without(p, p.observation_pose == 5)


def _unobserved_group():
    p = _ring(20, self_calibrating=True)
    p.intrinsics = p.intrinsics + [p.intrinsics[0]]  # free, and no observation names it
    return p


def _without(p, drop):
    for k in ("observation_pose", "observation_intrinsic", "observation_point", "observation_pixel"):
        setattr(p, k, getattr(p, k)[~drop])
    return p


@pytest.mark.parametrize("case", [_unobserved_pose, _unobserved_group])
@pytest.mark.parametrize("limit", [0, 3])
def test_a_free_block_without_observations(adjuster, case, limit):
    """Its row of S is zero: the product there is lambda diag x and its step is zero, in the cluster kernel
    as in the matrix-free product; the rank test sees a zero row whichever operator took the steps."""
    p = case()
    cfg = SolveConfig(linear_solver=abi.SOLVER_ITERATIVE, max_iterations=6, pcg_relative_tolerance=1e-10,
                      pcg_max_iterations=limit)
    a = adjuster.solve(p, cfg)
    b = adjuster.solve(p, cfg.with_(matvec=abi.MATVEC_IMPLICIT))
    for k in ("iteration_count", "accepted_step_count", "rejected_step_count", "rejected_step_solve", "status",
              "pcg_iteration_count", "observability", "unconstrained_intrinsic_count"):
        assert a.report[k] == b.report[k], (k, a.report[k], b.report[k])
    assert abs(a.report["final_objective"] - b.report["final_objective"]) <= 1e-9 * b.report["final_objective"]
    assert np.max(np.abs(a.rotations - b.rotations)) < 1e-7 and np.max(np.abs(a.centers - b.centers)) < 1e-7
    assert np.max(np.abs(a.points - b.points)) < 1e-7
    again = adjuster.solve(p, cfg)
    assert np.array_equal(a.points, again.points) and np.array_equal(a.centers, again.centers)
