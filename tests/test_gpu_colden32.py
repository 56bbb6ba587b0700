"""FP32 column densities: the end pixels (integer arithmetic away from grazing
pairs, double at them) and the interior against the C oracle; every kernel,
pixels from far narrower to far wider than the smoothing lengths, particles at
the edge of their support.  1e-5 is the FP32 form's stated accuracy."""
import numpy as np
import pytest

from test_gpu_colden64 import _case
from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1, 3])
@pytest.mark.parametrize("nbins", [1, 33, 900, 14100])
def test_end_pixels(fsg, port, kernel, nbins):
    from fake_spectra_gb300._spectra_priv import _Particle_Interpolate
    g = _case(nbins + kernel, 300, 7, 1500.0)
    vel, temp, t = np.zeros_like(g["pos"]), np.full_like(g["hh"], 1e4), synth.LYA
    args = (0, nbins, kernel, g["box"], synth.cosmology()[2], 0.25, t.lambda_cm, t.gamma, t.fosc,
            t.amumass, 1e-7, g["pos"], vel, g["dens"], temp, g["hh"], g["axis"], g["cofm"])
    got = _Particle_Interpolate(*args, precision="fp32")
    want = port.particle_interpolate(*args)
    assert (want > 0).any()
    # a pixel of a row is a sum of positive terms, each within 1e-5 of its own
    # value, in units of about 2^-60 of the row's bound
    np.testing.assert_allclose(got, want, rtol=1e-5, atol=1e-12 * want.max())
