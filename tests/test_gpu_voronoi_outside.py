"""Voronoi cells of particles whose coordinate along the sightline is outside the box
(by a tenth of it, by a whole box length) or not finite, against the C oracle: the
distance to an image is the same number there, and a cell without a finite distance
owns no point."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [1, 2, 3])
@pytest.mark.parametrize("kind", ["tenth", "box", "nan", "inf", "mixed"])
@pytest.mark.parametrize("box,n", [(100.0, 3), (102.4, 40), (700.0, 600)])
def test_cells_outside_the_box(fsg, port, axis, kind, box, n):
    from fake_spectra_gb300._spectra_priv import _Particle_Interpolate
    rng = np.random.default_rng(73 * axis + n)
    x = rng.uniform(0, box, n)
    if n == 3:
        x[:] = (0.95 * box, 0.97 * box, 0.3 * box)
    pos = rng.uniform(0.45 * box, 0.55 * box, (n, 3))
    pos[:, axis - 1] = x
    some = np.arange(n) % 3 == 0                       # with three cells, the one at 0.95
    far = pos[:, axis - 1]
    if kind in ("tenth", "mixed"):
        far[some & (x > 0.9 * box)] -= box
        far[some & (x < 0.1 * box)] += box
    if kind in ("box", "mixed"):
        far[some] += np.where(x[some] < 0.5 * box, box, -box)
    if kind in ("nan", "mixed"):
        far[n // 2] = np.nan
    if kind in ("inf", "mixed"):
        far[n - 1] = np.inf
    cofm = np.full((2, 3), 0.5 * box)
    cofm[1] += 0.01 * box
    t = synth.LYA
    for ct in (0, 1):
        args = (ct, 300, 2, box, synth.cosmology()[2], 0.25, t.lambda_cm, t.gamma, t.fosc,
                t.amumass, 1e-7, pos.astype(np.float32),
                (40 * rng.standard_normal((n, 3))).astype(np.float32),
                (rng.lognormal(0, 1, n) * 1e11).astype(np.float32),
                (1e4 * rng.lognormal(0, 0.3, n)).astype(np.float32),
                np.full(n, 0.3 * box, np.float32), np.full(2, axis, np.int32), cofm)
        want = port.particle_interpolate(*args)
        got = _Particle_Interpolate(*args)
        assert np.isfinite(want).all() and (want != 0).any()
        # as tests/test_gpu_voronoi.py
        np.testing.assert_allclose(got, want, rtol=1e-11, atol=1e-14 * np.abs(want).max())
