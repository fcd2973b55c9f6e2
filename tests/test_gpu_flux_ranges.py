"""States outside the flux's branch-free range: every kernel still equals the FP32 oracle bit for bit.

Water at rest (numerators exactly zero), films and momenta down to denormals, depths and speeds far above
anything physical, and a gravity or dry tolerance for which the whole run takes the IEEE operations.
"""

from __future__ import annotations

import numpy as np
import pytest

from oracle.resident_oracle import ResidentOracle

from ._valley import MANNING, dam, valley_grid

pytestmark = pytest.mark.gpu


def states(grid):
    rng = np.random.default_rng(11)
    n = grid.N
    calm = np.full(n, 2.0, np.float32)
    z = np.zeros(n, np.float32)
    tiny = (10.0 ** rng.uniform(-44, -3, n)).astype(np.float32)
    h = np.where(rng.random(n) < 0.5, dam(grid) + np.float32(2e-3), tiny).astype(np.float32)
    slow = (10.0 ** rng.uniform(-45, -20, n) * np.where(rng.random(n) < 0.5, -1, 1)).astype(np.float32)
    huge = (10.0 ** rng.uniform(4, 6.5, n)).astype(np.float32)
    fast = (huge * 10.0 ** rng.uniform(-2, 2, n)).astype(np.float32)
    flat = grid.zb.max() - grid.zb
    return {"calm": ((flat + calm).astype(np.float32), z, z), "tiny": (h, slow, slow[::-1].copy()),
            "huge": (huge, fast, -fast[::-1].copy())}


@pytest.mark.parametrize("kernel", ["persistent", "staged", "tiled"])
@pytest.mark.parametrize("case", ["calm", "tiny", "huge", "gravity", "film"])
def test_states_outside_the_plain_range(case: str, kernel: str) -> None:
    from inundation_b200.backend import SWESolverB200Resident

    grid = valley_grid(nx=64, ny=48)
    h, hu, hv = states(grid)["tiny" if case in ("gravity", "film") else case]
    kw = {"gravity": {"g": 0.01}, "film": {"dry_tol": 1e-10}}.get(case, {})
    n = np.full(grid.N, MANNING, np.float32)
    solver = SWESolverB200Resident(grid, None, h, hu, hv, n, **kw)
    solver.stage_kernel = kernel
    oracle = ResidentOracle(grid, h, hu, hv, n, **kw)
    t = 2.0**-12
    run = dict(t_end=t, output_interval_s=t, dt_max=2.0**-16, dt_init=2.0**-16, cfl_interval=1, progress=False)
    for s in (solver, oracle):
        s.steps_per_graph = 20
        s.run(**run)
    assert solver.steps_total == oracle.steps_total >= 16
    for name in ("h", "hu", "hv", "h_residual"):
        x, y = getattr(solver, f"download_{name}")(), getattr(oracle, f"download_{name}")()
        same = (x.view(np.uint32) == y.view(np.uint32)) | (np.isnan(x) & np.isnan(y))
        assert same.all(), (name, int((~same).sum()), x[~same][:3], y[~same][:3])


@pytest.mark.parametrize("kernel", ["persistent", "staged", "tiled"])
def test_films_under_the_smallest_gravity_of_the_plain_range(kernel: str) -> None:
    """Depths from 2^-100 to 2^-60 and a gravity just above 1/16: celerity arguments down to 2^-85 and below."""
    from inundation_b200.backend import SWESolverB200Resident

    grid = valley_grid(nx=64, ny=48)
    rng = np.random.default_rng(12)
    h = np.where(rng.random(grid.N) < 0.2, 0.01, 2.0 ** rng.uniform(-100, -60, grid.N)).astype(np.float32)
    z, n, kw = np.zeros(grid.N, np.float32), np.full(grid.N, MANNING, np.float32), {"g": 0.07, "dry_tol": 1e-9}
    solver, oracle = SWESolverB200Resident(grid, None, h, z, z, n, **kw), ResidentOracle(grid, h, z, z, n, **kw)
    solver.stage_kernel = kernel
    t = 2.0**-6
    for s in (solver, oracle):
        s.steps_per_graph = 20
        s.run(t_end=t, output_interval_s=t, dt_max=t / 16, dt_init=t / 16, cfl_interval=1, progress=False)
    assert solver.steps_total == oracle.steps_total >= 16
    for name in ("h", "hu", "hv", "h_residual"):
        x, y = getattr(solver, f"download_{name}")(), getattr(oracle, f"download_{name}")()
        np.testing.assert_array_equal(x.view(np.uint32), y.view(np.uint32), err_msg=name)
