"""Sources and early-ended submits of the whole-step kernels, bit for bit against the FP32 oracle.

Up to 1024 sources are added by the CTAs of their tiles, with one more barrier in
steps that have a source outside the active blocks; more run as grid-wide passes.
A submit ends as soon as no instance has time left, so short windows leave most of
a submit's steps out. All results are exact: the tolerance is zero.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle.resident_oracle import ResidentOracle

from ._valley import DX, MANNING, NX, NY, cell_near, dam, valley_grid

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grid():
    return valley_grid()


def rates(grid, count: int) -> np.ndarray:
    """``count`` sources: one under the dam, one sink there, the rest seeded, most of them on dry ground."""
    rng = np.random.default_rng(count)
    out = np.zeros(grid.N, np.float32)
    at = rng.choice(grid.N, count, replace=False)
    out[at] = rng.uniform(1e-5, 0.02, count)
    first = cell_near(grid, NX * DX * 0.1, NY * DX / 2)
    if out[first] == 0.0:
        out[at[0]] = 0.0
    out[first] = 0.5
    if count > 2:
        out[at[1]] = -0.01 if at[1] != first else out[at[1]]
    assert np.count_nonzero(out) == count
    return out


@pytest.mark.parametrize("kernel", ["persistent", "staged"])
@pytest.mark.parametrize("ctas", [None, 3])
@pytest.mark.parametrize("active_set", [True, False])
@pytest.mark.parametrize("compensated", [True, False])
@pytest.mark.parametrize("count", [1, 40, 1024, 1025, 5000])
def test_sources_match_the_oracle(count: int, compensated: bool, active_set: bool, ctas: int | None, kernel: str, grid) -> None:
    from inundation_b200.backend import SWESolverB200Resident

    h0, z, n = dam(grid), np.zeros(grid.N, np.float32), np.full(grid.N, MANNING, np.float32)
    solver = SWESolverB200Resident(grid, None, h0, z, z, n)
    solver.stage_kernel, solver.max_grid = kernel, ctas
    oracle = ResidentOracle(grid, h0, z, z, n)
    for s in (solver, oracle):
        s.compensated, s.active_set, s.steps_per_graph = compensated, active_set, 30
    kw = dict(output_interval_s=1.5, dt_max=1.0, dt_init=0.01, cfl_interval=1, progress=False)
    for t0, t1, src in ((0.0, 3.0, rates(grid, count)), (3.0, 4.5, rates(grid, max(1, count // 2)))):
        a, _ = solver.run(t_end=t1, t_start=t0, resume=t0 > 0.0, source_rate=src, **kw)
        b, _ = oracle.run(t_end=t1, t_start=t0, resume=t0 > 0.0, source_rate=src, **kw)
        assert len(a) == len(b) and all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))
    for name in ("h", "hu", "hv", "h_residual"):
        x, y = getattr(solver, f"download_{name}")(), getattr(oracle, f"download_{name}")()
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))
    assert solver.steps_total == oracle.steps_total


@pytest.mark.parametrize("kernel", ["persistent", "staged", "mixed"])
@pytest.mark.parametrize("per_submit", [1, 2, 7, 200])
def test_submits_that_end_early_change_nothing(per_submit: int, kernel: str, grid) -> None:
    """Windows of a few steps: the clock, the state and the flags of whole submits, whatever their length."""
    from inundation_b200.backend import SWESolverB200Resident

    h0, z, n = dam(grid), np.zeros(grid.N, np.float32), np.full(grid.N, MANNING, np.float32)
    solver = SWESolverB200Resident(grid, None, h0, z, z, n)
    oracle = ResidentOracle(grid, h0, z, z, n)
    solver.steps_per_graph = per_submit
    if kernel == "mixed":  # the kernels take turns, each from the lists and flags the other left
        names = iter(["persistent", "staged", "tiled", "staged", "plain", "persistent"] * 1000)
        replay = solver._graph

        def turn(*a):
            solver.stage_kernel = next(names)
            return replay(*a)

        solver._graph = turn
    else:
        solver.stage_kernel = kernel
    kw = dict(t_end=2.0, output_interval_s=0.25, dt_max=0.5, dt_init=0.01, cfl_interval=1, progress=False)
    a, ta = solver.run(**kw)
    b, tb = oracle.run(**kw)
    assert ta == tb and solver.steps_total == oracle.steps_total
    assert all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b, strict=True))
    np.testing.assert_array_equal(solver.download_block_flags()[:, 0], oracle.download_block_flags()[:, 0])


def test_batch_instances_that_end_apart_match_their_own_runs() -> None:
    """A batch on the staged whole-step kernel: instances of other sizes, clocks and sources, some done long before
    the last, on a grid of a few CTAs; each equals its own oracle run."""
    from inundation_b200.batch import BatchedSolver, BatchMember

    members, oracles = [], []
    for k, (nx, ny) in enumerate([(64, 32), (40, 30), (16, 16), (128, 64)]):
        g = valley_grid(nx=nx, ny=ny)
        h0, z, n = dam(g, nx=nx, ny=ny), np.zeros(g.N, np.float32), np.full(g.N, MANNING, np.float32)
        rate = None
        if k % 2:
            rate = np.zeros(g.N, np.float32)
            rate[[g.N // 2, g.N - 1]] = (0.05, 0.001)
        members.append(BatchMember(g, h0, z, z, n, source_rate=rate))
        oracles.append((ResidentOracle(g, h0, z, z, n), rate))
    ends = [2.0, 0.25, 1.0, 0.5]
    solver = BatchedSolver(members)
    solver.stage_kernel, solver.max_grid = "staged", 5
    solver.run(ends, 0.5, 0.01, 0.5)
    for i, (oracle, rate) in enumerate(oracles):
        oracle.run(t_end=ends[i], output_interval_s=0.5, dt_max=0.5, dt_init=0.01, source_rate=rate)
        for name in ("h", "hu", "hv", "h_residual"):
            x, y = getattr(solver, f"download_{name}")(i), getattr(oracle, f"download_{name}")()
            np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32), err_msg=f"{name} of {i}")


def test_rain_on_every_cell_matches_the_oracle(grid) -> None:
    """A source in every cell (the pruned bounds), the ground dry at first but for the dam: cells wet one after
    another, beside dry neighbours, and the sources' bounds set dt."""
    from inundation_b200.backend import SWESolverB200Resident

    h0, z, n = dam(grid), np.zeros(grid.N, np.float32), np.full(grid.N, MANNING, np.float32)
    rain = np.random.default_rng(5).uniform(1e-5, 2e-3, grid.N).astype(np.float32)
    rain[grid.N // 3] = 5.0
    solver = SWESolverB200Resident(grid, None, h0, z, z, n)
    solver.stage_kernel = "staged"
    oracle = ResidentOracle(grid, h0, z, z, n)
    kw = dict(t_end=3.0, output_interval_s=1.0, dt_max=0.5, dt_init=0.01, cfl_interval=1, progress=False, source_rate=rain)
    a, _ = solver.run(**kw)
    b, _ = oracle.run(**kw)
    assert solver.steps_total == oracle.steps_total
    assert all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b, strict=True))
    for name in ("hu", "hv", "h_residual"):
        x, y = getattr(solver, f"download_{name}")(), getattr(oracle, f"download_{name}")()
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32))
