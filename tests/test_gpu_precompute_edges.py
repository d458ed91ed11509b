"""GPU: the scene-table kernels at the edges of their work splits, against the CPU oracle.

The meridional solver shares a bin's rows out over a cluster of CTAs, whose size follows from the number of bins
and the grid (rows that do not divide evenly, odd row lengths, one bin, all of the chip's bins); the phase CDF of a
bin is kept in shared memory up to a limit on the angles; the angular functions come from a table up to a limit on
its size (256 MB, passed by the last two cases), else from the pdf kernel's own recurrence. The solver's arithmetic is the oracle's, operation by
operation, so its field may differ by what the two machines' libm functions differ in the coefficients (an ulp or
two, 1e-15, carried through a contraction of at most a few thousand sweeps: 1e-9 is far above it), and its
iteration count is the oracle's. cos(theta) of the two machines may differ by two ulps (2^-53 each), which at the
first angles of the grid (pi / (n_theta - 1)) moves theta by 2^-53 n_theta / pi and a pdf whose forward lobe is 1/x
wide by x times that: four times x 2^-53 n_theta / pi, and 1e-13 for the sums.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle_harness as H
import parity_scenes as PS
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


@pytest.mark.parametrize("nr,nz,n_bins", [(16, 32, 1), (17, 33, 5), (31, 97, 64), (45, 64, 20), (100, 100, 30)])
def test_meridional_field_equals_oracle(ctx, nr, nz, n_bins):
    over, pk, _ = PS.SCENES["meridional_solver"]
    cfg = S.small_cell_config(**dict(over, meridional_grid_nr=nr, meridional_grid_nz=nz, meridional_solver_tolerance=1e-3))
    cfg.validate()
    parts = S.quartz_particles(**dict(pk, n_bins=n_bins))
    ctx.set_scene(cfg.to_scene_params())
    ctx.build_particles(parts.spec(cfg), cfg.sediment_spec())
    got = ctx.sediment_field()
    orc = H.OracleRun("port", cfg, parts)
    want = orc.sediment_field()
    orc.close()
    assert got["iterations"] == want["iterations"]
    np.testing.assert_allclose(got["grid"], want["grid"], rtol=1e-9, atol=0)


@pytest.mark.parametrize("n_theta,d_max_um,arithmetic", [
    (257, 5.0, "reference"), (258, 5.0, "fast"), (1801, 300.0, "reference"), (12288, 5.0, "reference"),
    (12289, 5.0, "reference"), (12289, 300.0, "reference"), (24001, 300.0, "fast")])
def test_phase_cdf_equals_oracle(ctx, n_theta, d_max_um, arithmetic):
    cfg = S.small_cell_config(mie_phase_grid_size=n_theta)
    parts = S.quartz_particles(n_bins=3, d_min_um=0.5, d_max_um=d_max_um)
    ctx.set_scene(cfg.to_scene_params())
    arith = abi.TABLES_FAST if arithmetic == "fast" else abi.TABLES_REFERENCE
    ctx.build_particles(parts.spec(cfg, table_arithmetic=arith), cfg.sediment_spec())
    got = ctx.physics()
    orc = H.OracleRun("port", cfg, parts)
    want = orc.physics()
    orc.close()
    x = float(want["size_parameter"].max())
    np.testing.assert_allclose(got["phase_cdf"], want["phase_cdf"], rtol=0, atol=1e-13 + 4 * x * 2.0**-53 * n_theta / np.pi)
