"""GPU: the two forms of the counter-based stream (inlined and by a call) are one stream.

The wavefront engine's source stage draws through the called form, the persistent kernel through the inlined one:
for the same photons the counts that only the source decides (launched, accepted at the collimator, rejected) are
the same whole numbers, for photon counts below, at and above a warp and with an offset into the stream.
"""
from __future__ import annotations

import numpy as np
import pytest

from tardiis_and_claritas_gb300 import abi, scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,offset", [(1, 0), (31, 5), (33, 1000), (50_000, 123_456)])
def test_called_and_inlined_streams_agree(n, offset):
    from tardiis_and_claritas_gb300 import lib as L
    from tardiis_and_claritas_gb300.build_ext import build
    build()
    cfg = S.small_cell_config(particle_surface_rms_slope_deg=0.0, wave_surface_rms_height_m=0.0)
    parts = S.quartz_particles(100.0, n_bins=8)
    ctx = L.Context(0)
    ctx.set_scene(cfg.to_scene_params())
    ctx.build_particles(parts.spec(cfg), cfg.sediment_spec())
    t = []
    for flags in (0, abi.RUN_PERSISTENT_KERNEL):
        r, _ = ctx.trace(S.run_params(n, seed=9, ray_offset=offset, rng_mode=abi.RNG_PHILOX, flags=flags))
        t.append(r)
    ctx.close()
    assert t[0]["status_counts"].sum() == t[1]["status_counts"].sum() == n
    assert t[0]["status_counts"][3] == t[1]["status_counts"][3]
    k = abi.RF_NAMES.index("source_accepted")
    np.testing.assert_array_equal(t[0]["ray_flags"][k], t[1]["ray_flags"][k])
