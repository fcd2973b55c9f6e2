"""The forward of a calibration in the persistent kernel: the per-step kernels' losses, records and gradients, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

from inundation_b200.scenarios import calibration

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gauges", [1, 40, 300])
@pytest.mark.parametrize(("steps", "every"), [(1, 1), (23, 8), (40, 50)])
def test_persistent_forward_matches_the_per_step_kernels(steps: int, every: int, gauges: int) -> None:
    from inundation_b200.adjoint import GaugeCalibration

    sc = calibration(9000, seed=3, knots=6, gauges=gauges, spacing=10.0)
    z, q = sc.geom.zb.astype(np.float32), sc.hydrographs[0].knot_q.astype(np.float32)
    out = []
    for persistent in (True, False):
        p = GaugeCalibration(sc.geom, sc.h0, sc.hu0, sc.hv0, gauges=sc.meta["gauges"], steps=steps,
                             hydrographs=sc.hydrographs, checkpoint_every=every, dt_max=1.0, dt_init=0.05)
        p.persistent_forward, p.cut_depth = persistent, 4e-4
        seen = p.observe(sc.meta["n_true"], z, q)
        losses = [p.loss(sc.manning, z, q), p.loss(sc.manning, z, q)]
        out.append((seen, np.array(losses), *p.gradient(), p.download_state("h"), p.download_block_flags()[:, 0]))
    assert out[0][1][0] == out[0][1][1]
    for a, b in zip(*out, strict=True):
        np.testing.assert_array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))
