"""GPU: drawing photons into free slots, at the sizes where lanes and scenarios change over.

Warps draw photon numbers 32 at a time across scenario boundaries and hand out free slots from chunks of 32. Every
photon's result is a function of its number alone, so integer tallies of tiny scenarios traced together equal those
of each traced alone, and those of one trace equal the sum over any split of it (runs of a few photons, and more
photons than the pool has slots).
"""
from __future__ import annotations

import numpy as np
import pytest

import parity_scenes as PS
from tardiis_and_claritas_gb300 import abi, scene as S

pytestmark = pytest.mark.gpu

COUNTS = [1, 31, 32, 33, 2, 1, 1, 65, 7, 4097, 3, 128]


@pytest.fixture(scope="module")
def ctx():
    from tardiis_and_claritas_gb300 import lib as L
    from tardiis_and_claritas_gb300.build_ext import build
    build()
    c = L.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("rng", [abi.RNG_REFERENCE_XORSHIFT, abi.RNG_PHILOX])
def test_tiny_scenarios_together_equal_each_alone(ctx, rng):
    scs = S.sweep_workload(len(COUNTS), sampler_seed=8, n_bins=8)
    scenes, parts, seds = S.sweep_specs(scs)
    runs = [S.run_params(n, seed=5 + i, ray_offset=10 * i, rng_mode=rng, scenario_id=i) for i, n in enumerate(COUNTS)]
    ctx.sweep_build(scenes, parts, seds)
    got = ctx.sweep_trace(runs)
    for i, n in enumerate(COUNTS):
        ctx.set_scene(scenes[i])
        ctx.build_particles(parts[i], seds[i])
        want, _ = ctx.trace(runs[i])
        for k in PS.TALLY_KEYS:
            np.testing.assert_array_equal(got[i][k], want[k], err_msg=f"scenario {i}: {k}")
        assert int(np.sum(want["status_counts"])) == n


@pytest.mark.parametrize("n,split", [(1, 1), (33, 32), (1000, 31), (3_000_001, 1_234_567)])
def test_trace_equals_the_sum_of_its_parts(ctx, n, split):
    cfg = S.small_cell_config()
    ctx.set_scene(cfg.to_scene_params())
    ctx.build_particles(S.quartz_particles(n_bins=8, concentration_mg_l=200.0).spec(cfg), cfg.sediment_spec())

    def trace(count, offset):
        return ctx.trace(S.run_params(count, seed=3, ray_offset=offset, rng_mode=abi.RNG_REFERENCE_XORSHIFT))[0]

    whole = trace(n, 0)
    parts = [trace(split, 0)] + ([trace(n - split, split)] if n > split else [])
    for k in PS.TALLY_KEYS:
        np.testing.assert_array_equal(whole[k], sum(np.asarray(p[k]) for p in parts), err_msg=k)
