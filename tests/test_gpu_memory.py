"""GPU: what a context keeps of its largest scene is given back when it turns to much smaller ones (two in a row).

A scene's tables lie in one arena that the next build reuses. A scene of 9001 angles and 1500 orders has 217 MB of
angular functions alone; a build of 257 angles and small particles needs under 2 MB.
"""
from __future__ import annotations

import pytest

from tardiis_and_claritas_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    from tardiis_and_claritas_gb300 import lib as L
    from tardiis_and_claritas_gb300.build_ext import build
    build()
    torch.cuda.init()
    c = L.Context(0)
    yield c
    c.close()


def _build(ctx, n_theta, d_max_um):
    import torch
    cfg = S.small_cell_config(mie_phase_grid_size=n_theta)
    cfg.validate()
    ctx.set_scene(cfg.to_scene_params())
    ctx.build_particles(S.quartz_particles(n_bins=4, d_min_um=1.0, d_max_um=d_max_um).spec(cfg), cfg.sediment_spec())
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0], ctx.physics()


def test_a_small_scene_gives_the_memory_of_a_large_one_back(ctx):
    free_small, want = _build(ctx, 257, 5.0)
    free_large, _ = _build(ctx, 9001, 300.0)
    assert free_small - free_large > 200 << 20
    _build(ctx, 257, 5.0)
    free_again, got = _build(ctx, 257, 5.0)
    assert free_again - free_large > 200 << 20
    assert all((got[k] == want[k]).all() for k in ("qext", "phase_cdf"))


@pytest.mark.parametrize("others", [[(6001, 300.0), (6001, 300.0)], [(257, 5.0), (9001, 300.0), (257, 5.0)]])
def test_scenes_of_similar_size_or_in_turn_keep_it(ctx, others):
    _build(ctx, 9001, 300.0)
    free_large, _ = _build(ctx, 9001, 300.0)
    for n_theta, d_max_um in others:
        free, _ = _build(ctx, n_theta, d_max_um)
        assert abs(free - free_large) < 32 << 20
