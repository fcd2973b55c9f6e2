"""The lines between the two ways a step takes its sources: fewer sources never cost a step more than many.

Up to a number of sources one CTA takes their CFL bounds, past it a grid-wide pass does; in the persistent kernel
the tiles' CTAs add up to 1024 of them. The sums are the same, so results are exact on both sides of each line
(tolerance zero). A step's time below a line is at most 15 % above that with 1500 sources, which is past every line: the
lines are set where both sides take about the same time, and repeated best-of-5 timings differ by a few per cent.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle.resident_oracle import ResidentOracle

from ._valley import MANNING, dam, valley_grid

pytestmark = pytest.mark.gpu

# (kernel, the last count on the near side of a line)
LINES = [("persistent", 64), ("persistent", 1024), ("staged", 64), ("tiled", 128)]


@pytest.fixture(scope="module")
def grid():
    return valley_grid()


def rates(grid, count: int) -> np.ndarray:
    """``count`` seeded sources, a quarter of them under the dam or near it."""
    rng = np.random.default_rng(count)
    near = np.flatnonzero(grid.centroid[:, 0] < 160.0)
    at = rng.choice(near, count // 4, replace=False)
    at = np.concatenate([at, rng.choice(np.setdiff1d(np.arange(grid.N), at), count - at.size, replace=False)])
    out = np.zeros(grid.N, np.float32)
    out[at] = rng.uniform(1e-5, 0.02, count)
    return out


@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize(("kernel", "line"), LINES)
def test_both_sides_of_a_line_match_the_oracle(kernel: str, line: int, side: int, grid) -> None:
    from inundation_b200.backend import SWESolverB200Resident

    h0, z, n = dam(grid), np.zeros(grid.N, np.float32), np.full(grid.N, MANNING, np.float32)
    solver, oracle = SWESolverB200Resident(grid, None, h0, z, z, n), ResidentOracle(grid, h0, z, z, n)
    solver.stage_kernel = kernel
    src = rates(grid, line + side)
    kw = dict(t_end=3.0, output_interval_s=1.5, dt_max=1.0, dt_init=0.01, cfl_interval=1, progress=False, source_rate=src)
    a, _ = solver.run(**kw)
    b, _ = oracle.run(**kw)
    assert solver.steps_total == oracle.steps_total
    assert all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b, strict=True))
    for name in ("hu", "hv", "h_residual"):
        x, y = getattr(solver, f"download_{name}")(), getattr(oracle, f"download_{name}")()
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))


def us_per_step(grid, kernel: str, count: int, steps: int = 100) -> float:
    from inundation_b200.batch import BatchedSolver, BatchMember

    h0, z, n = dam(grid), np.zeros(grid.N, np.float32), np.full(grid.N, MANNING, np.float32)
    solver = BatchedSolver([BatchMember(grid, h0, z, z, n, source_rate=rates(grid, count))])
    solver.stage_kernel = kernel
    times = []
    for _ in range(5):
        solver.reset()
        solver.start(1.0, 0.01)
        submit = solver._graph(steps)
        first, last = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with torch.cuda.stream(solver._stream):
            submit.replay()
            first.record()
            submit.replay()
            last.record()
        last.synchronize()
        times.append(first.elapsed_time(last) * 1000.0 / steps)
    return min(times)


@pytest.mark.parametrize("kernel", ["persistent", "staged", "tiled"])
def test_fewer_sources_do_not_cost_more(kernel: str, grid) -> None:
    many = us_per_step(grid, kernel, 1500)
    slow = {c: us_per_step(grid, kernel, c) for c in (64, 128, 256, 384, 512, 1024)}
    slow = {c: t for c, t in slow.items() if t > 1.15 * many}
    assert not slow, (many, slow)
