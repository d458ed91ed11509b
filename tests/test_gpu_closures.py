"""GPU: closures (the conditional sampler) wherever the counter-based stream runs them.

A closure's trials run in a lane (tail kernel, GEOM's first ones), across a warp from the first (COND stage) or in
a lane and then across the warp (COND stage with diagnostics on). Trial t of a closure has its own substream, so a
photon's history is the same in all of them up to the rounding of separately compiled kernels: a few photons per
million take another path (0.1 % of the rays is far above that), and the trial counters differ by those photons'
trials. Weakly absorbing particles make closures of an absorbed target hundreds of trials long; a small trial limit
makes them end in the middle of a warp's batch.
"""
from __future__ import annotations

import numpy as np
import pytest

from tardiis_and_claritas_gb300 import abi, scene as S

pytestmark = pytest.mark.gpu

COND = abi.STAGE_NAMES.index("COND")
ALL_TAIL = {"tail_photons": 1 << 20, "pass_batch": 1}
NO_TAIL = {"tail_photons": 1}


@pytest.fixture(scope="module")
def ctx():
    from tardiis_and_claritas_gb300 import lib as L
    from tardiis_and_claritas_gb300.build_ext import build
    build()
    c = L.Context(0)
    yield c
    c.set_engine_config(None)
    c.close()


POPULATIONS = {
    # every event is a closure, and the few absorbed targets take hundreds of trials
    "absorbing": dict(concentration_mg_l=2000.0, n_bins=24, k=2e-4),
    # transparent: a closure follows only an event whose sphere does not fit beside a wall (it starts in GEOM); with
    # nearly the water's index no trial is a wave event, and beside a wall none may ever fit
    "coarse": dict(concentration_mg_l=100_000.0, n_bins=8, d_min_um=200.0, d_max_um=400.0, median_um=300.0),
}


def _scene(ctx, population, retries):
    cfg = S.small_cell_config(particle_event_model="hybrid_mie_exact_rate")
    cfg.validate()
    parts = S.quartz_particles(**POPULATIONS[population], **(dict(n=cfg.n_water * 1.0002) if population == "coarse" else {}))
    sp = cfg.to_scene_params()
    sp.conditional_retries = retries
    ctx.set_scene(sp)
    ctx.build_particles(parts.spec(cfg), cfg.sediment_spec())


def _closures(t):
    c = np.asarray(t["conditional_stats"], dtype=np.int64)
    return int(c[6] + c[7] + c[8] + c[9])  # absorbed, scattered, failed, exhausted: each closure ends in one


def _trace(ctx, engine, n, seed=3, **run):
    ctx.set_engine_config(engine)
    try:
        return ctx.trace(S.run_params(n, seed=seed, rng_mode=abi.RNG_PHILOX, **run), records=True)
    finally:
        ctx.set_engine_config(None)


@pytest.mark.parametrize("provenance", [False, True])
@pytest.mark.parametrize("retries", [45, 512])
def test_a_closure_of_at_most_512_trials_is_one_visit_of_the_tail(ctx, provenance, retries):
    _scene(ctx, "absorbing", retries)
    ctx.set_provenance(provenance)
    try:
        t, _ = _trace(ctx, ALL_TAIL, 20_000)
        assert ctx.engine_stats()["tail_photons"] > 0
    finally:
        ctx.set_provenance(False)
    closures, trials = _closures(t), int(t["conditional_stats"][0])
    assert closures > 1000 and trials > closures + 1000  # long closures among them
    assert 0 < int(t["sched_stats"][COND]) <= closures


@pytest.mark.parametrize("population,retries", [("absorbing", 13), ("absorbing", 20), ("absorbing", 45),
                                                ("absorbing", 16384), ("coarse", 20), ("coarse", 16384)])
def test_diagnostic_closures_equal_those_of_the_tail_and_of_the_plain_stage(ctx, population, retries):
    n = 300_000 if population == "coarse" else 60_000
    _scene(ctx, population, retries)
    got = {}
    for name, engine, provenance in (("stage", NO_TAIL, True), ("tail", ALL_TAIL, True), ("plain", NO_TAIL, False)):
        ctx.set_provenance(provenance)
        try:
            t, rec = _trace(ctx, engine, n)
            prov = ctx.read_provenance_records(n)[0] if provenance else None
        finally:
            ctx.set_provenance(False)
        got[name] = (t, np.stack([rec[k] for k in abi.RECORD_INT_FIELDS], axis=1), prov)
    t, ints, prov = got["stage"]
    assert t["sched_stats"][COND] > 0 and t["device_error"] == 0
    if population == "absorbing" and retries < 512:
        assert t["conditional_stats"][9] > 0  # some closures run out of trials
    for other in ("tail", "plain"):
        t2, ints2, prov2 = got[other]
        same = np.all(ints == ints2, axis=1)
        assert same.mean() >= 0.999, (other, same.mean())
        np.testing.assert_allclose(np.asarray(t["conditional_stats"], dtype=np.float64),
                                   np.asarray(t2["conditional_stats"], dtype=np.float64), rtol=5e-3, atol=40, err_msg=other)
        assert abs(_closures(t) - _closures(t2)) <= 2e-3 * _closures(t)
        if prov2 is not None:
            assert (prov[same] != prov2[same]).any(axis=1).mean() <= 1e-3, other
