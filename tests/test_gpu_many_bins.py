"""GPU: the phase tables of a sweep equal a single scene's at every number of bins.

The phase pdf takes one bin to a warp or, without the table of the angular functions (above 256 MB of it), four from
160 bins on, in both arithmetics. Every bin has the same operations in the same order in all of them, so the tables of
a scenario are those of its single build bit for bit: hundreds of bins with the table, totals below, at and above the
line without it, a last group of four with missing bins, and angles that fill neither a warp nor a block.
"""
from __future__ import annotations

import numpy as np
import pytest

from tardiis_and_claritas_gb300 import abi, scene as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from tardiis_and_claritas_gb300 import lib as L
    from tardiis_and_claritas_gb300.build_ext import build
    build()
    c = L.Context(0)
    yield c
    c.close()


def _check(ctx, sizes, n_theta, d_max_um, arithmetic, compare):
    cfg = S.small_cell_config(mie_phase_grid_size=n_theta)
    cfg.validate()
    parts = [S.quartz_particles(n_bins=k, d_min_um=1.0 + 0.1 * i, d_max_um=d_max_um) for i, k in enumerate(sizes)]
    specs = [p.spec(cfg, table_arithmetic=arithmetic) for p in parts]
    ctx.sweep_build([cfg.to_scene_params()] * len(sizes), specs, [cfg.sediment_spec()] * len(sizes))
    swept = {i: ctx.sweep_physics(i, sizes[i], n_theta) for i in compare}
    ctx.set_scene(cfg.to_scene_params())
    for i in compare:
        ctx.build_particles(specs[i], cfg.sediment_spec())
        one = ctx.physics()
        for key in ("qext", "qsca", "asym_g", "theta", "phase_cdf"):
            assert np.array_equal(swept[i][key], one[key]), (i, key)
        assert np.all(one["phase_cdf"].reshape(sizes[i], n_theta)[:, -1] == 1.0)


@pytest.mark.parametrize("arithmetic", [abi.TABLES_REFERENCE, abi.TABLES_FAST])
@pytest.mark.parametrize("last", [43, 44, 47])  # 607, 608 and 611 bins: a multiple of four and not
def test_sweep_tables_equal_single_builds(ctx, arithmetic, last):
    _check(ctx, [47] * 12 + [last], 1801, 60.0, arithmetic, range(13))


@pytest.mark.parametrize("n_theta,arithmetic", [(12289, abi.TABLES_REFERENCE), (24001, abi.TABLES_FAST)])
@pytest.mark.parametrize("sizes", [[47, 47, 47, 18], [47, 47, 47, 19], [47] * 13])  # 159, 160 and 611 bins
def test_without_the_angular_table(ctx, n_theta, arithmetic, sizes):
    _check(ctx, sizes, n_theta, 300.0, arithmetic, (0, len(sizes) - 1))
