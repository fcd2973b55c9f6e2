"""The block kernel's stages, one launch each, and the edges of the whole-step block kernel's range.

Without packed records, and where its CTAs cannot hold every block, "staged" runs stage by stage. All results are
exact against the FP32 oracle: the tolerance is zero.
"""

from __future__ import annotations

import numpy as np
import pytest

from inundation_b200.engine import DENSE_TAKEN_BLOCKS, _DenseSubmit
from inundation_b200.scenarios import open_channel
from inundation_b200.tuning import OPEN_INFLOW, OPEN_NORMAL

from ._valley import MANNING, dam, point_source, valley_grid
from .test_gpu_packed_blocks import oracle_of, same_run, solver_of

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grid():
    return valley_grid()


@pytest.mark.parametrize("max_grid", [None, 5])
@pytest.mark.parametrize("sources", [0, 1])
@pytest.mark.parametrize("compensated", [True, False])
def test_staged_stages_match_the_oracle(compensated: bool, sources: int, max_grid: int | None, grid) -> None:
    solver, oracle = solver_of(grid, dam(grid)), oracle_of(grid, dam(grid))
    solver.stage_kernel, solver.packed_blocks, solver.max_grid = "staged", False, max_grid
    solver.compensated = oracle.compensated = compensated
    solver.steps_per_graph = 40
    assert not isinstance(solver._graph(), _DenseSubmit)
    same_run(solver, oracle, source_rate=point_source(grid, 0.5, 60.0, 128.0) if sources else None)


@pytest.mark.parametrize("blocks", [DENSE_TAKEN_BLOCKS, DENSE_TAKEN_BLOCKS + 2])
def test_one_cta_takes_as_many_blocks_as_its_list_holds(blocks: int) -> None:
    """All blocks of the mesh on one CTA: the list's length runs whole steps, a row of blocks more the stages."""
    geom = valley_grid(nx=512, ny=blocks // 2)
    h0 = np.where(geom.centroid[:, 0] < 700.0, 0.5, 0.0).astype(np.float32)
    solver, oracle = solver_of(geom, h0), oracle_of(geom, h0)
    assert solver.n_blocks == blocks
    solver.stage_kernel, solver.max_grid, solver.steps_per_graph = "staged", 1, 8
    assert isinstance(solver._graph(), _DenseSubmit) == (blocks == DENSE_TAKEN_BLOCKS)
    run = dict(t_end=2.0**-4, output_interval_s=2.0**-4, dt_max=2.0**-7, dt_init=2.0**-7, cfl_interval=1, progress=False)
    for s in (solver, oracle):
        s.active_set = False  # every block is on the list
        s.run(**run)
    assert solver.steps_total == oracle.steps_total >= 8
    for name in ("h", "hu", "hv", "h_residual"):
        p, q = getattr(solver, f"download_{name}")(), getattr(oracle, f"download_{name}")()
        np.testing.assert_array_equal(p.view(np.uint32), q.view(np.uint32), err_msg=name)


# -- the clamp tally in the block kernels: a CFL number at which the update does draw cells below zero ----------------
CFL = 4.0


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("compensated", [True, False])
def test_the_clamp_tally_of_the_block_kernels(compensated: bool, packed: bool, grid) -> None:
    rng = np.random.default_rng(7)
    h0 = np.where(rng.random(grid.N) < 0.5, dam(grid) + np.float32(1.2e-3), 0.0).astype(np.float32)
    solver, oracle = solver_of(grid, h0, cfl=CFL), oracle_of(grid, h0, cfl=CFL)
    solver.stage_kernel, solver.packed_blocks = "staged", packed
    for s in (solver, oracle):
        s.compensated, s.track_clamp = compensated, True
    same_run(solver, oracle, dt_max=2.0)
    clamped = oracle.download_clamp_mass()
    assert (clamped > 0.0).any()
    np.testing.assert_array_equal(solver.download_clamp_mass().view(np.uint32), clamped.view(np.uint32))
    assert isinstance(solver._graph(), _DenseSubmit) == packed


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("compensated", [True, False])
def test_the_clamp_tally_of_an_open_mesh(compensated: bool, packed: bool) -> None:
    sc = open_channel(cells=200, across=20, depth=0.4)
    h0 = (sc.h0 * (np.random.default_rng(1).random(sc.geom.N) < 0.5)).astype(np.float32)
    solver = solver_of(sc.geom, h0, cfl=CFL, open_edges=sc.meta["open_edges"])
    oracle = oracle_of(sc.geom, h0, cfl=CFL, open_edges=sc.meta["open_edges"])
    solver.stage_kernel, solver.packed_blocks = "staged", packed
    up, down = (e.size for e in sc.meta["open_edges"])
    for s in (solver, oracle):
        s.compensated, s.track_clamp = compensated, True
        s.set_open_conditions(np.repeat([OPEN_INFLOW, OPEN_NORMAL], [up, down]).astype(np.uint32),
                              np.repeat([0.6, 0.9], [up, down]).astype(np.float32))
    same_run(solver, oracle, t_end=12.0, output_interval_s=4.0, dt_max=8.0, dt_init=0.5)
    clamped = oracle.download_clamp_mass()
    assert (clamped > 0.0).any()
    np.testing.assert_array_equal(solver.download_clamp_mass().view(np.uint32), clamped.view(np.uint32))
    np.testing.assert_array_equal(solver.download_open_volumes(), oracle.download_open_volumes())
    assert isinstance(solver._graph(), _DenseSubmit) == packed
