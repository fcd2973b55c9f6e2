"""Which kernel a calibration's forward segment takes, on a stub (no device).

The persistent kernel where "auto" would take it and its tiles' CTAs add the sources themselves; graphs of the
per-step kernels otherwise, among them for a mesh that the gauged kernel's grid cannot hold (the library refuses it).
"""

from __future__ import annotations

import ctypes

import pytest

from inundation_b200 import native
from inundation_b200.adjoint import GaugeCalibration
from inundation_b200.engine import KERNELS, PERSISTENT_FUSED_SOURCES

SWE_OK, SWE_ERR_CUDA, SWE_ERR_TOO_LARGE = 0, 2, 3


class Graph:
    def __init__(self, log: list) -> None:
        self.log = log

    def replay(self) -> None:
        self.log.append("graph")


class Stub(GaugeCalibration):
    _cuda_stream = ctypes.c_void_p(0)


class Lib:
    def __init__(self, log: list, status: int) -> None:
        self.log, self.status = log, status

    def swe_steps_gauged(self, *args) -> int:
        if self.status == SWE_OK:
            self.log.append("persistent")
        return self.status


def segment(active: int, sources: int = 0, n_blocks: int = 1000, status: int = SWE_OK, **attributes) -> list:
    p = Stub.__new__(Stub)
    log: list = []
    p.n_blocks, p._active_blocks, p._src_count = n_blocks, active, sources
    p._sms, p._per_sm, p.ctas_per_sm, p.max_grid = 148, {k: 4 for k in KERNELS.values()}, None, None
    p._mesh, p._state, p._gauges = native.SweMesh(), native.SweState(), native.SweGauges()
    p._params, p._sources = native.SweParams, native.SweSources
    p._stream, p._lib = None, Lib(log, status)
    p._segment_graph = lambda n_steps, record: Graph(log)
    for name, value in attributes.items():
        setattr(p, name, value)
    p._forward_steps(4, 1)
    return log


@pytest.mark.parametrize(
    ("active", "n_blocks", "want"),
    [(250, 1000, "persistent"), (251, 1000, "graph"), (148, 148, "persistent"), (149, 149, "graph")],
)
def test_the_active_blocks_decide_as_for_auto(active: int, n_blocks: int, want: str) -> None:
    assert segment(active, n_blocks=n_blocks) == [want]


@pytest.mark.parametrize(("sources", "want"), [(0, "persistent"), (PERSISTENT_FUSED_SOURCES, "persistent"),
                                               (PERSISTENT_FUSED_SOURCES + 1, "graph"), (250_000, "graph")])
def test_many_sources_take_the_graph(sources: int, want: str) -> None:
    """Rain on every cell took six times as long in the persistent kernel (250k cells: 98 ms against 17)."""
    assert segment(50, sources=sources) == [want]


def test_a_mesh_that_the_gauged_grid_cannot_hold_takes_the_graph() -> None:
    assert segment(50, status=SWE_ERR_TOO_LARGE) == ["graph"]
    with pytest.raises(RuntimeError, match="swe_steps_gauged"):
        segment(50, status=SWE_ERR_CUDA)


@pytest.mark.parametrize("attributes", [{"persistent_forward": False}, {"stage_kernel": "plain"}, {"track_clamp": True}])
def test_the_other_kernels_and_the_clamp_tally_take_the_graph(attributes: dict) -> None:
    assert segment(50, **attributes) == ["graph"]
