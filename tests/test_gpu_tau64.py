"""FP64 optical depths through the staged kernel (multipole wing, far-field
tiles, shared sightlines) against the C oracle: row lengths around the tile
widths and the shared-memory limits, line constants from negligible to strong
damping, cold and hot gas, strong absorbers whose wings wrap round the row."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu

# the repository's FP64 tolerance: relative 1e-11, and the contributions below
# tautail that the stop rule may move by one pixel
RTOL, ATOL = 1e-11, 5e-7


def _case(seed, n=400, nlos=5, box=1e4):
    rng = np.random.default_rng(seed)
    dens = 10 ** rng.uniform(9, 14, n)
    dens[:3] = 1e20                                    # wings that cover the whole row
    temp = 10 ** rng.uniform(3.6, 5.0, n)
    temp[3:6] = (30.0, 3e6, 300.0)                     # strong damping / hot / cold
    return dict(pos=rng.uniform(0, box, (n, 3)).astype(np.float32),
                vel=(60 * rng.standard_normal((n, 3))).astype(np.float32),
                dens=dens.astype(np.float32), temp=temp.astype(np.float32),
                hh=(box / 6 * rng.uniform(0.1, 1.0, n)).astype(np.float32),
                axis=rng.integers(1, 4, nlos).astype(np.int32),
                cofm=rng.uniform(0, box, (nlos, 3)), box=box)


def _args(g, nbins, kernel, line, gamma=None):
    velfac = synth.cosmology()[2]
    return (1, nbins, kernel, g["box"], velfac, 0.25, line.lambda_cm,
            line.gamma if gamma is None else gamma, line.fosc, line.amumass, 1e-7, g["pos"],
            g["vel"], g["dens"], g["temp"], g["hh"], g["axis"], g["cofm"])


def _check(args, port):
    from fake_spectra_gb300._spectra_priv import _Particle_Interpolate
    got = _Particle_Interpolate(*args)
    want = port.particle_interpolate(*args)
    assert (want > 0).any()
    bad = np.abs(got - want) > RTOL * np.abs(want) + ATOL
    assert not bad.any(), (np.argwhere(bad)[:4], got[bad][:4], want[bad][:4])


@pytest.mark.parametrize("nbins", [2, 63, 64, 65, 257, 1115, 3001, 8700, 11152, 13900, 17000])
def test_row_lengths(fsg, port, nbins):
    _check(_args(_case(nbins), nbins, 1, synth.LYA), port)


@pytest.mark.parametrize("kernel", [0, 1, 3])
@pytest.mark.parametrize("gamma", [0.0, 1e3, 6.265e8, 3e11, 3e13])
def test_damping_and_kernels(fsg, port, kernel, gamma):
    _check(_args(_case(7), 900, kernel, synth.LYA, gamma), port)


@pytest.mark.parametrize("nlos", [1, 39, 160])
def test_sightline_counts(fsg, port, nlos):
    """One sightline per cluster of blocks, several waves, and one block per sightline."""
    _check(_args(_case(nlos, n=300, nlos=nlos), 300, 1, synth.CIV), port)
