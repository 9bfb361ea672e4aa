"""Calls from several threads: plans of one context on streams of their own, and batches on one context. Every
solve gives the bits that it gives alone."""
import threading

import numpy as np
import pytest

from openmvg_ba_cuda import SolveConfig, abi, synthetic

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _in_threads(calls):
    """The results of the calls, all started together, each on its own thread."""
    out, start = [None] * len(calls), threading.Barrier(len(calls))

    def run(k):
        start.wait()
        try:
            out[k] = calls[k]()
        except Exception as e:  # noqa: BLE001
            out[k] = e

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for o in out:
        if isinstance(o, Exception):
            raise o
    return out


def _same(a, b):
    assert a.report["iteration_count"] == b.report["iteration_count"]
    assert a.report["final_objective"] == b.report["final_objective"]
    assert np.array_equal(a.points, b.points) and np.array_equal(a.centers, b.centers)


@pytest.mark.parametrize("solver", [abi.SOLVER_DIRECT, abi.SOLVER_ITERATIVE])
def test_plans_of_one_context_on_their_own_streams(adjuster, solver):
    problems = [synthetic.ring_problem(seed=20 + k, cameras=20 + 4 * k, points=900, radius=3.0) for k in range(3)]
    streams = [torch.cuda.Stream() for _ in problems]
    plans = []
    try:
        for p, s in zip(problems, streams):
            cfg = SolveConfig(linear_solver=solver, max_iterations=8, pcg_relative_tolerance=1e-10, stream=s.cuda_stream)
            plans.append(adjuster.plan(p, cfg))
        alone = [plan.solve() for plan in plans]
        alone = [plan.solve() for plan in plans]  # the tables and graphs of a first solve are in place
        together = _in_threads([lambda plan=plan: [plan.solve() for _ in range(6)] for plan in plans])
        for a, repeats in zip(alone, together):
            for b in repeats:
                _same(a, b)
    finally:
        for plan in plans:
            plan.close()


def test_batches_on_one_context(adjuster):
    """More batches at a time than one, of different sizes, twice over: each has workers of its own."""
    windows = synthetic.window_problems(seed=32, windows=10, total_observations=30_000, min_points=200, max_points=2000,
                                        max_cameras=16)
    cfg = SolveConfig(max_iterations=10)
    alone = [adjuster.solve(w, cfg) for w in windows]
    for _ in range(2):
        together = _in_threads([lambda n=n: adjuster.solve_batched(windows[:n], cfg) for n in (10, 3, 7)])
        for batch in together:
            for a, b in zip(alone, batch):
                _same(a, b)
