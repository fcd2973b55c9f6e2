"""Where the packed records are made, where they are refused, and the stage-by-stage blocks that run then.

The whole-step block kernel needs its records packed and a CTA for every block; the block kernel's stages, one launch
each, are the fallback. All results are exact against the FP32 oracle: the tolerance is zero.
"""

from __future__ import annotations

import numpy as np
import pytest

from inundation_b200.engine import KERNELS, _DenseSubmit
from inundation_b200.mesh.geometry import with_bed
from oracle.resident_oracle import ResidentOracle

from ._valley import MANNING, dam, point_source, valley_grid

pytestmark = pytest.mark.gpu


def solver_of(geom, h0, **kw):
    from inundation_b200.backend import SWESolverB200Resident

    z, n = np.zeros(geom.N, np.float32), np.full(geom.N, MANNING, np.float32)
    return SWESolverB200Resident(geom, None, h0, z, z, n, **kw)


def oracle_of(geom, h0, **kw):
    z, n = np.zeros(geom.N, np.float32), np.full(geom.N, MANNING, np.float32)
    return ResidentOracle(geom, h0, z, z, n, **kw)


def same_run(a, b, **kw) -> None:
    run = {**dict(t_end=2.0, output_interval_s=0.5, dt_max=0.5, dt_init=0.01, cfl_interval=1, progress=False), **kw}
    x, _ = a.run(**run)
    y, _ = b.run(**run)
    assert a.steps_total == b.steps_total
    assert all(np.array_equal(p.view(np.uint32), q.view(np.uint32)) for p, q in zip(x, y, strict=True))
    for name in ("h", "hu", "hv", "h_residual"):
        p, q = getattr(a, f"download_{name}")(), getattr(b, f"download_{name}")()
        np.testing.assert_array_equal(p.view(np.uint32), q.view(np.uint32), err_msg=name)


def test_a_mesh_that_is_always_seated_is_packed_when_asked_for() -> None:
    """512 tiles have a CTA each: "auto" never leaves the persistent kernel, so nothing is packed until "staged" is
    chosen; the sources set before that come along."""
    grid = valley_grid()
    solver, oracle = solver_of(grid, dam(grid)), oracle_of(grid, dam(grid))
    assert 4 * solver.n_blocks <= solver.grid(KERNELS["persistent"])
    assert solver._blocks is None and not solver._blocks_t
    src = point_source(grid, 0.5, 60.0, 128.0)
    same_run(solver, oracle, source_rate=src)
    assert solver._blocks is None
    solver.stage_kernel = "staged"
    assert isinstance(solver._graph(), _DenseSubmit) and solver._blocks is not None
    solver.steps_total = oracle.steps_total = 0
    same_run(solver, oracle, source_rate=src)


def test_a_larger_mesh_is_packed_at_once() -> None:
    geom = valley_grid(nx=256, ny=256)
    solver = solver_of(geom, dam(geom, ny=256))
    assert 4 * solver.n_blocks > solver.grid(KERNELS["persistent"])
    assert solver._blocks is not None


def test_bed_steps_out_of_range_leave_no_records_behind() -> None:
    """A step of 10^6 m is past what the range check of the branch-free flux relies on."""
    geom = valley_grid(nx=256, ny=256)
    zb = geom.zb.copy()
    zb[geom.N - 1] = 1e6
    geom = with_bed(geom, zb)
    solver, oracle = solver_of(geom, dam(geom, ny=256)), oracle_of(geom, dam(geom, ny=256))
    assert solver._blocks is None and not solver._blocks_t
    solver.stage_kernel = "staged"
    assert not isinstance(solver._graph(), _DenseSubmit)
    same_run(solver, oracle)


def test_perimeters_bound_the_sum_of_a_cells_edges() -> None:
    geom = valley_grid(nx=256, ny=256)
    around = solver_of(geom, dam(geom, ny=256))._blocks_t["perim"].cpu().numpy().astype(np.float64)
    want = np.zeros(geom.N)
    for side in (geom.edge_cellL, geom.edge_cellR):
        np.add.at(want, side[side >= 0], geom.edge_len[side >= 0].astype(np.float64))
    assert (around[: geom.N] >= want * (1.0 + 1e-5)).all() and (around[: geom.N] <= want * (1.0 + 1e-3)).all()
    assert (around[geom.N :] == 0.0).all()
