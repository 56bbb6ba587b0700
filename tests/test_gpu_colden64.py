"""FP64 column densities (integer interior pixels, double edge pixels) against
the C oracle: pixels from far narrower to far wider than the smoothing
lengths, pairs that graze the kernel's support, every kernel, row lengths at
the shared-memory limits, one to many sightlines."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


def _case(seed, n, nlos, hmax, box=1e4):
    rng = np.random.default_rng(seed)
    g = dict(pos=rng.uniform(0, box, (n, 3)).astype(np.float32),
             dens=(10 ** rng.uniform(9, 14, n)).astype(np.float32),
             hh=(hmax * 10 ** rng.uniform(-2, 0, n)).astype(np.float32),
             axis=rng.integers(1, 4, nlos).astype(np.int32),
             cofm=rng.uniform(0, box, (nlos, 3)), box=box)
    # sightlines through particles and at the edge of their support
    for l in range(0, nlos, 2):
        p = rng.integers(n)
        off = g["hh"][p] * rng.choice([0.0, 0.5, 0.99, 0.9999])
        g["cofm"][l] = g["pos"][p].astype(np.float64)
        g["cofm"][l, g["axis"][l] % 3] += off
    return g


def _check(g, nbins, kernel, port):
    from fake_spectra_gb300._spectra_priv import _Particle_Interpolate
    vel = np.zeros_like(g["pos"])
    temp = np.full_like(g["hh"], 1e4)
    t = synth.LYA
    args = (0, nbins, kernel, g["box"], synth.cosmology()[2], 0.25, t.lambda_cm, t.gamma, t.fosc,
            t.amumass, 1e-7, g["pos"], vel, g["dens"], temp, g["hh"], g["axis"], g["cofm"])
    got = _Particle_Interpolate(*args)
    want = port.particle_interpolate(*args)
    assert (want > 0).any()
    # the sums are integers in units of 2^-124 of the sightline's bound (the sum
    # over its pairs of dens x largest kernel value x pixel x windows), half a
    # unit per contribution: far below a pixel's value except in rows that hold
    # both the strongest cores and single kernel tails 27 orders fainter
    n = len(g["hh"])
    pix = g["box"] / nbins
    wraps = np.ceil(2 * g["hh"].max() / pix / nbins) + 1
    unit = 2.0 ** -124 * 2 * n * g["dens"].max() * 8 * pix * wraps
    np.testing.assert_allclose(got, want, rtol=1e-11, atol=0.5 * n * wraps * unit)


@pytest.mark.parametrize("kernel", [0, 1, 3])
@pytest.mark.parametrize("nbins", [1, 31, 33, 900, 11152, 14100, 20000])
def test_pixel_widths(fsg, port, kernel, nbins):
    _check(_case(nbins + kernel, 300, 7, 1500.0), nbins, kernel, port)


@pytest.mark.parametrize("nlos", [1, 40, 400])
def test_sightline_counts(fsg, port, nlos):
    _check(_case(nlos, 500, nlos, 900.0), 257, 1, port)
