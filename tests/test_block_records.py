"""Halo lists and local record indices of the 256-cell tiles (host side): they name the records' own cells."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from inundation_b200.layout import NO_CELL, build_batch_layout, build_tile_layout, halo_records
from inundation_b200.scenarios import open_channel, voronoi_geometry


@pytest.mark.parametrize("cells", [60, 256, 257, 3000, 20_000])
def test_local_indices_name_the_records_cells(cells: int) -> None:
    if cells == 60:
        layout = build_tile_layout(open_channel(cells=12, across=5).geom)
    elif cells == 3000:
        layout = build_batch_layout([voronoi_geometry(n, 10.0 * n**0.5, n) for n in (700, 1500, 800)])
    else:
        layout = build_tile_layout(voronoi_geometry(cells, 10.0 * cells**0.5, cells))
    T = layout.blocks
    H = halo_records(T, torch.from_numpy(T.cl), torch.from_numpy(T.cr), layout.n_padded_cells)
    halo, halo_ptr = H.halo.numpy(), H.halo_ptr.numpy().astype(np.int64)
    local = H.local.numpy().view(np.uint32)
    tile = np.repeat(np.arange(T.n_tiles), np.diff(T.ptr.astype(np.int64)))
    real = T.edge >= 0

    def cell(index: np.ndarray) -> np.ndarray:
        place = halo_ptr[tile] + np.maximum(index.astype(np.int64) - 256, 0)
        return np.where(index < 256, 256 * tile + index, halo[np.minimum(place, halo.size - 1)])

    left, right = local & 0xFFFF, local >> 16
    np.testing.assert_array_equal(cell(left)[real], T.cl[real])
    inner = real & (T.cr >= 0)
    np.testing.assert_array_equal(cell(right)[inner], T.cr[inner])
    assert (right[real & (T.cr < 0)] == NO_CELL).all() and (left[real & (T.cr < 0)] < 256).all()
    for t in range(T.n_tiles):  # each cell outside once
        own = halo[halo_ptr[t] : halo_ptr[t + 1]]
        assert np.unique(own).size == own.size and not ((own // 256) == t).any()
    assert H.max_halo == int(np.diff(halo_ptr).max(initial=0))
