"""The explicit reduced camera system built from camera pairs (csrc/pair_rows.cuh) against the
matrix-free product of the same linearization, where its pair lists, items and blocks can go wrong:
cameras that see a point twice, pose masks and the S^2 chart (pose dimensions 2 to 6), fixed poses with
free intrinsics, one shared intrinsic group (a block that collects every pair), a group per camera (the
9-parameter products), fixed points, angular residuals, and few cameras with long lists.

Both products sum the same terms in FP64 in different orders, so they agree to rounding of the largest
entries: 1e-9 of the product's largest value, the tolerance of the operator parity tests."""
import numpy as np
import pytest

from openmvg_ba_cuda import CameraIntrinsics, Gauge, RobustLoss, SolveConfig, abi, synthetic

pytestmark = pytest.mark.gpu


def _ring(**kw):
    return synthetic.ring_problem(seed=6, **kw)


def _seen_twice():
    p = _ring(points=300)
    keep = np.arange(0, p.observation_count, 3)  # a third of the observations once more, moved by a pixel
    p.observation_pose = np.concatenate([p.observation_pose, p.observation_pose[keep]])
    p.observation_intrinsic = np.concatenate([p.observation_intrinsic, p.observation_intrinsic[keep]])
    p.observation_point = np.concatenate([p.observation_point, p.observation_point[keep]])
    p.observation_pixel = np.vstack([p.observation_pixel, p.observation_pixel[keep] + 1.0])
    return p


def _masks():
    return _ring(points=400, pose_variables=np.array([0, 0] + [1, 2, 3] * 6, dtype=np.uint32))


def _baseline():
    p = _ring(points=400)
    p.pose_variables[0] = 0
    p.gauge = Gauge.fixed_baseline(0, 3, float(np.linalg.norm(p.centers[3] - p.centers[0])))
    return p


def _shared_group():
    return _ring(self_calibrating=True, radius=3.0)


def _two_groups_fixed_pose():
    p = _ring(points=500, self_calibrating=True, radius=3.0)
    second = CameraIntrinsics(model=abi.CAMERA_BROWN_CONRADY, fx=498.0, fy=498.0, cx=320.0, cy=240.0,
                              radial_kind=abi.RADIAL_K1K2, k1=-0.1, k2=0.0, variables=abi.INTRINSIC_FOCAL)
    p.intrinsics = p.intrinsics + [second]
    p.observation_intrinsic = (p.observation_pose % 2).astype(np.uint32)
    p.pose_variables[[0, 5]] = 0
    return p


def _group_per_camera():
    p = synthetic.plane_problem(seed=12, cameras=37, points=3001, mean_track=6.5, extent=27.0)
    # without damping a point needs parallax: keep those with three views
    keep = (np.bincount(p.observation_point, minlength=len(p.points)) >= 3)[p.observation_point]
    points, index = np.unique(p.observation_point[keep], return_inverse=True)
    p.points, p.point_fixed, p.observation_point = p.points[points], p.point_fixed[points], index.astype(np.uint32)
    p.observation_pose, p.observation_intrinsic = p.observation_pose[keep], p.observation_intrinsic[keep]
    p.observation_pixel = p.observation_pixel[keep]
    return p


def _fixed_points():
    p = _ring(points=400)
    p.point_fixed[::4] = 1
    return p


def _few_cameras():
    return _ring(cameras=8, points=6001)


CASES = {f.__name__[1:]: f for f in (_seen_twice, _masks, _baseline, _shared_group, _two_groups_fixed_pose,
                                     _group_per_camera, _fixed_points, _few_cameras)}


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("damping", [0.0, 1e-2])
def test_pair_rows_equal_the_matrix_free_product(adjuster, case, damping):
    p = CASES[case]()
    p.robust_loss = RobustLoss.huber(1.0)
    d = adjuster.debug_schur_product(p, None)
    rng = np.random.default_rng(1)
    for _ in range(2):
        x = rng.standard_normal(d)
        free, explicit = adjuster.debug_schur_product(p, x, damping)
        assert np.max(np.abs(free - explicit)) <= 1e-9 * np.max(np.abs(explicit))


def test_a_budget_without_room_for_the_pairs_builds_by_block_rows(adjuster):
    """The two builds of S take the same steps: a budget that leaves no room for the pair lists uses
    k_block_rows, and the solves agree to rounding."""
    p = _ring(points=600)
    cfg = SolveConfig(linear_solver=abi.SOLVER_DIRECT, max_iterations=6)
    free = adjuster.solve(p, cfg)
    budget = 1 << 20  # grow until the solve is accepted: the first accepted budget has no slack for the pairs
    while True:
        try:
            tight = adjuster.solve(p, cfg.with_(workspace_budget_bytes=budget))
            break
        except Exception as e:
            assert "budget" in str(e)
            budget += 1 << 16
    assert tight.report["iteration_count"] == free.report["iteration_count"]
    rel = abs(tight.report["final_objective"] - free.report["final_objective"]) / free.report["final_objective"]
    assert rel <= 1e-9
    assert np.max(np.abs(tight.points - free.points)) <= 1e-7
    assert np.max(np.abs(tight.centers - free.centers)) <= 1e-7


@pytest.mark.parametrize("cameras", [393_152, 393_153, 393_216, 393_217])
def test_camera_counts_at_the_limit_of_the_neighbour_bitmap(adjuster, cameras):
    """A neighbour bitmap, a bit per camera, has the 48 KB of a CTA's shared memory less the kernel's own
    variables (two words, and what the compiler aligns); S is built by block rows above that. Fixed cameras
    that see nothing change no result."""
    p = _ring(points=200)
    cfg = SolveConfig(linear_solver=abi.SOLVER_DIRECT, max_iterations=3)
    few = adjuster.solve(p, cfg)
    more = cameras - len(p.centers)
    p.rotations = np.concatenate([p.rotations, np.broadcast_to(np.eye(3), (more, 3, 3))])
    p.centers = np.concatenate([p.centers, np.zeros((more, 3))])
    p.pose_variables = np.concatenate([p.pose_variables, np.zeros(more, dtype=np.uint32)])
    many = adjuster.solve(p, cfg)
    assert many.report["iteration_count"] == few.report["iteration_count"]
    assert abs(many.report["final_objective"] - few.report["final_objective"]) <= 1e-9 * few.report["final_objective"]
    assert np.max(np.abs(many.points - few.points)) <= 1e-7
    assert np.max(np.abs(many.centers[:len(few.centers)] - few.centers)) <= 1e-7


def _three_views(p):
    keep = (np.bincount(p.observation_point, minlength=len(p.points)) >= 3)[p.observation_point]
    points, index = np.unique(p.observation_point[keep], return_inverse=True)
    p.points, p.point_fixed, p.observation_point = p.points[points], p.point_fixed[points], index.astype(np.uint32)
    p.observation_pose, p.observation_intrinsic = p.observation_pose[keep], p.observation_intrinsic[keep]
    p.observation_pixel = p.observation_pixel[keep]
    return p


def test_device_memory_that_others_hold_leaves_the_solve_with_block_rows(adjuster):
    """Whatever of the pair tables the device has no room for, the solve goes on: by block rows, and with the
    tables given back where the factor or the selected inverse needs their memory. The rest of a solve with
    its tables was measured, the memory left to it runs from what block rows need to all of it."""
    torch = pytest.importorskip("torch")
    from openmvg_ba_cuda.adjuster import CudaBundleAdjuster
    p = _three_views(synthetic.plane_problem(seed=13, cameras=250, points=60_000, mean_track=7.0, extent=70.0))
    cfg = SolveConfig(linear_solver=abi.SOLVER_DIRECT, max_iterations=2)

    def solve(room):
        """A plan's solve with `room` bytes of device memory free at its start (None: all of it), and what it took."""
        with CudaBundleAdjuster(0) as own, own.plan(p, cfg) as plan:
            torch.cuda.empty_cache()
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            filler = torch.empty(before - room, dtype=torch.uint8, device="cuda") if room else None
            try:
                s = plan.solve()
                return s, before - torch.cuda.mem_get_info()[0]
            finally:
                del filler
                torch.cuda.empty_cache()

    want, grown = solve(None)
    launches = set()
    n = p.observation_count
    assert grown > 2 * 27 * 8 * n  # the operands alone
    for share in (0.35, 0.5, 0.6, 0.7, 0.8, 0.9, 0.95, 1.0):
        got, _ = solve(int(share * grown) + (16 << 20))
        launches.add(got.report["kernel_launches"])
        for k in ("iteration_count", "accepted_step_count", "status", "observability"):
            assert got.report[k] == want.report[k], (share, k)
        assert abs(got.report["final_objective"] - want.report["final_objective"]) <= 1e-9 * want.report["final_objective"]
        assert np.max(np.abs(got.points - want.points)) <= 1e-7
    # the tightest took block rows from the start: one kernel a build and no tables
    assert min(launches) < want.report["kernel_launches"] and len(launches) > 1


def _long_tracks_of_one_group():
    """1,000 cameras that share one free intrinsic group and meet in most pairs: the group's blocks collect
    every pair again."""
    cameras, points, track = 1000, 400, 60
    p = synthetic.ring_problem(seed=14, cameras=cameras, points=points, self_calibrating=True, radius=3.0)
    rng = np.random.default_rng(14)
    p.observation_pose = np.concatenate([rng.choice(cameras, track, replace=False) for _ in range(points)]).astype(np.uint32)
    p.observation_point = np.repeat(np.arange(points), track).astype(np.uint32)
    p.observation_intrinsic = np.zeros(points * track, dtype=np.uint32)
    px, _ = synthetic._project(p.rotations[p.observation_pose], p.centers[p.observation_pose],
                               p.points[p.observation_point], 500.0, 320.0, 240.0, -0.1, 0.01, 0.0)
    p.observation_pixel = px + rng.normal(size=px.shape)
    return p


def _pair_table_bytes(p):
    """The tables of the pair build that a solver keeps, for cameras of 9 parameters in one group: operands,
    list entries, at least one partial product per pair, the neighbours, and the contributions of a pair
    to the blocks of its poses, its poses with the group (twice) and the group itself."""
    cameras = len(p.centers)
    seen = np.zeros((cameras, len(p.points)), dtype=np.int64)
    np.add.at(seen, (p.observation_pose, p.observation_point), 1)
    meet = seen @ seen.T
    neighbours, entries = np.count_nonzero(meet), int(np.triu(meet).sum())
    pairs = (neighbours + cameras) // 2
    return 2 * 27 * 8 * p.observation_count + 8 * entries + 8 * 81 * pairs + 4 * neighbours + 8 * 4 * neighbours


@pytest.mark.parametrize("case", [_long_tracks_of_one_group, lambda: _ring(points=600)])
def test_a_budget_holds_the_pair_tables_or_the_solve_takes_block_rows(adjuster, case):
    """The build that a budget leaves is read from the number of launches: the smallest budget that the
    solve is accepted with takes block rows, a large one the pairs, and the smallest one that takes the
    pairs has room for their tables."""
    p = case()
    cfg = SolveConfig(linear_solver=abi.SOLVER_DIRECT, max_iterations=1)

    def launches(budget):
        try:
            return adjuster.solve(p, cfg.with_(workspace_budget_bytes=budget)).report["kernel_launches"]
        except Exception as e:
            assert "budget" in str(e)
            return 0

    def smallest(low, high, good):  # to a quarter megabyte
        while high - low > 1 << 18:
            mid = (low + high) // 2
            low, high = (low, mid) if good(launches(mid)) else (mid, high)
        return high

    pairs = adjuster.solve(p, cfg).report["kernel_launches"]
    assert launches(1 << 36) == pairs
    accepted = smallest(0, 1 << 36, lambda n: n > 0)
    assert 0 < launches(accepted) < pairs
    with_pairs = smallest(accepted, 1 << 36, lambda n: n == pairs)
    if len(p.centers) == 1000:
        assert with_pairs - (accepted - (1 << 18)) >= _pair_table_bytes(p)
