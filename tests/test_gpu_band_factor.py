"""The banded tiled factor, its solve and the camera step they give, at the sizes where the tiles can go
wrong: systems of less than a panel, of exactly one tile and one more, ragged last tiles, bands of one tile
and bands wider than the solve's cluster. One direct step is one LM iteration: its state is compared with
the oracle's dense-band Cholesky at the parity tests' tolerances (cost 1e-9 relative, parameters 1e-7)."""
import numpy as np
import pytest

import oracle as O
from openmvg_ba_cuda import SolveConfig, abi, synthetic

pytestmark = pytest.mark.gpu


def _ring(cameras, dims):
    masks = np.full(cameras, abi.POSE_FREE, dtype=np.uint32)
    masks[0] = 0
    left = dims
    for c in range(1, cameras):  # free coordinates: 6 a camera, 3 or none for the last ones
        masks[c] = abi.POSE_FREE if left >= 6 else (abi.POSE_ROTATION if left >= 3 else 0)
        left -= 6 if left >= 6 else (3 if left >= 3 else 0)
    return synthetic.ring_problem(seed=8, cameras=cameras, points=400, pose_variables=masks)


@pytest.mark.parametrize("cameras,dims", [(8, 6), (8, 9), (13, 63), (13, 66), (23, 129), (36, 192), (60, 351), (122, 723)])
def test_direct_step_matches_oracle(adjuster, cameras, dims):
    p = _ring(cameras, dims)
    cfg = SolveConfig(linear_solver=abi.SOLVER_DIRECT, max_iterations=2)
    g, o = adjuster.solve(p, cfg), O.solve(p, cfg)
    assert g.report["reduced_dimension"] == dims
    for k in ("iteration_count", "accepted_step_count", "rejected_step_count", "status", "observability"):
        assert g.report[k] == o.report[k], k
    assert abs(g.report["final_objective"] - o.report["final_objective"]) <= 1e-9 * o.report["final_objective"]
    assert np.max(np.abs(g.rotations - o.rotations)) < 1e-7
    assert np.max(np.abs(g.centers - o.centers)) < 1e-7


def test_wide_band_step_matches_oracle(adjuster):
    """90 cameras with their own intrinsics over a grid, D about 800: a band of several tiles over a
    cluster of more than one CTA, and the selected inverse of the certificate."""
    p = synthetic.plane_problem(seed=15, cameras=90, points=9000, mean_track=8.0, extent=42.0)
    # points seen three times or more: a point with little parallax leaves the certificate to rounding
    keep = (np.bincount(p.observation_point, minlength=len(p.points)) >= 3)[p.observation_point]
    points, index = np.unique(p.observation_point[keep], return_inverse=True)
    p.points, p.point_fixed, p.observation_point = p.points[points], p.point_fixed[points], index.astype(np.uint32)
    p.observation_pose, p.observation_intrinsic = p.observation_pose[keep], p.observation_intrinsic[keep]
    p.observation_pixel = p.observation_pixel[keep]
    cfg = SolveConfig(linear_solver=abi.SOLVER_DIRECT, max_iterations=2)
    g, o = adjuster.solve(p, cfg), O.solve(p, cfg)
    for k in ("iteration_count", "accepted_step_count", "status", "observability"):
        assert g.report[k] == o.report[k], k
    assert np.array_equal(g.unconstrained_intrinsics, o.unconstrained_intrinsics)
    assert abs(g.report["final_objective"] - o.report["final_objective"]) <= 1e-9 * o.report["final_objective"]


@pytest.mark.parametrize("cameras,unobserved", [(13, 3), (13, 12), (60, 20)])
@pytest.mark.parametrize("solver", [abi.SOLVER_DIRECT, abi.SOLVER_AUTO])
def test_a_free_camera_without_observations_takes_a_zero_step(adjuster, cameras, unobserved, solver):
    """S is zero there and the damping its only diagonal: the factor succeeds, the camera stays, and the rank
    test of the undamped system finds the zero row, as in the oracle."""
    p = synthetic.ring_problem(seed=8, cameras=cameras, points=400)
    keep = p.observation_pose != unobserved
    for k in ("observation_pose", "observation_intrinsic", "observation_point", "observation_pixel"):
        setattr(p, k, getattr(p, k)[keep])
    cfg = SolveConfig(linear_solver=solver, max_iterations=2)
    g, o = adjuster.solve(p, cfg), O.solve(p, cfg)
    for k in ("iteration_count", "accepted_step_count", "rejected_step_count", "status", "observability"):
        assert g.report[k] == o.report[k], k
    assert g.report["accepted_step_count"] > 0
    assert abs(g.report["final_objective"] - o.report["final_objective"]) <= 1e-9 * o.report["final_objective"]
    assert np.max(np.abs(g.rotations - o.rotations)) < 1e-7
    assert np.max(np.abs(g.centers - o.centers)) < 1e-7
