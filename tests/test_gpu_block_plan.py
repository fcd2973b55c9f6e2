"""Blocks that fit the dynamic shared memory but not beside the dense kernel's own: configured as 0 CTAs, not an error."""

from __future__ import annotations

import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(("bytes_left", "fits"), [(0, False), (2048, False), (16384, True)])
def test_static_shared_memory_counts(bytes_left: int, fits: bool) -> None:
    """Only the occupancy query runs: the addresses are placeholders that nothing dereferences."""
    from inundation_b200 import native

    lib = native.load()
    mesh = native.SweMesh(n_cells=256, n_blocks=1, max_tile_edges=64, n_inst=1, max_sub_edges=64, max_sub_slots=64)
    for name, kind in native.SweMesh._fields_:
        if kind is native._P and name != "open_cond":
            setattr(mesh, name, 0x10000)
    # 227 KB hold 128 B of barrier words, 64 records of 24 B, 256 + halo cells of 16 B and 1040 B of pointers
    halo = (227 * 1024 - bytes_left - 128 - 24 * 64 - 1040) // 16 - 256
    blocks = native.SweBlocks(max_halo=halo, **{n: 0x30000 for n, kind in native.SweBlocks._fields_ if kind is native._P})
    per_sm = ctypes.c_int(7)
    assert lib.swe_configure_blocks(ctypes.byref(mesh), ctypes.byref(blocks), ctypes.byref(per_sm)) == 0
    assert (per_sm.value == 1) if fits else (per_sm.value == 0)
