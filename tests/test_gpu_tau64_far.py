"""FP64 optical depths of cold absorbers far from the line centre (more than 1000
thermal widths, beyond the range of the integer node sums) where the first far-field
tile starts as close to the multipole radius as it can, against the C oracle, each
particle on a sightline of its own and tautail = 0 so that every pixel counts."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins,kernel", [(3000, 1), (3000, 2), (2999, 3), (8000, 1), (12500, 0)])
def test_tiles_next_to_the_multipole_radius(fsg, port, nbins, kernel):
    from fake_spectra_gb300._spectra_priv import _Particle_Interpolate
    rng = np.random.default_rng(nbins)
    velfac, line = synth.cosmology()[2], synth.CIV
    box = 2e4 * nbins / 3000
    px = box * velfac / nbins
    bfac = np.sqrt(2 * 1.3806504e-16 / (line.amumass * 1.67262178e-24)) / 1e5
    pos, hh, temp = [], [], []
    while len(pos) < 96:
        t, h = 10 ** rng.uniform(2.2, 3.2), box * 10 ** rng.uniform(-2.3, -1.2)
        b = bfac * np.sqrt(t)
        umax = 0.75 * (np.float32(h) * velfac) / b     # the outermost node
        x = max(4.5 * umax, umax + 12) * b / px
        k = int(x + 2)                                 # pixels to the first tile
        if not 1.02 < k - x < 1.3 or x > 0.4 * nbins:
            continue
        tile = 64 * rng.integers(0, nbins // 64)
        pos.append(((tile - k) % nbins + 0.98) * px / velfac)
        hh.append(h)
        temp.append(t)
    n = len(pos)
    pos = np.stack([pos, np.tile(np.arange(12), n // 12) * box / 12,
                    np.repeat(np.arange(n // 12), 12) * box / (n // 12)], axis=1)
    pos = pos.astype(np.float32)
    args = (1, nbins, kernel, box, velfac, 0.25, line.lambda_cm, line.gamma, line.fosc,
            line.amumass, 0.0, pos, np.zeros_like(pos),
            (10 ** rng.uniform(12, 14, n)).astype(np.float32), np.float32(temp), np.float32(hh),
            np.ones(n, np.int32), pos.astype(np.float64))
    got, want = _Particle_Interpolate(*args), port.particle_interpolate(*args)
    assert (want > 0).mean() > 0.99
    # 1e-11, the FP64 form's tolerance, and the 128-bit sums' unit (2^-124 of a bound at
    # most 2^13 of the row's largest value, times the pairs of a row, 2^3 at most)
    bad = np.abs(got - want) > 1e-11 * want + 2.0 ** -108 * want.max(axis=1, keepdims=True)
    assert not bad.any(), (len(np.unique(np.argwhere(bad)[:, 0])), np.argwhere(bad)[:4],
                           got[bad][:4], want[bad][:4])
