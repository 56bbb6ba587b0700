"""The flux power at the edges of the transforms' ranges, against numpy's FFT:
lengths in shared memory (direct and chirp-z) and the first ones beyond, one or
many pairs per block, an odd last row, rows of very different size, constant
rows, a NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _want(tau, mean):
    f = np.exp(-tau) / mean - 1.0
    n = tau.shape[1]
    return (np.abs(np.fft.rfft(f, axis=1)) ** 2).sum(0) / n ** 2 / tau.shape[0]


def _got(tau, mean):
    import ctypes
    import torch
    from fake_spectra_gb300 import _lib
    from fake_spectra_gb300 import fluxstatistics as st
    ctx = st._context()
    st._bind(ctx)
    d = torch.as_tensor(tau, device="cuda")
    out = np.empty(tau.shape[1] // 2 + 1)
    eb = _lib.errbuf()
    rc = _lib.load().fsg_flux_power_device(
        ctx.handle, ctypes.c_void_p(d.data_ptr()), tau.shape[0], tau.shape[1],
        ctypes.c_double(1.0), ctypes.c_double(mean), ctypes.c_double(1.0),
        ctypes.c_void_p(out.ctypes.data), eb, 512)
    _lib.raise_for(rc, eb.value.decode(errors="replace"))
    return out


# 13888 points fit: direct lengths to 13824, chirp-z lengths to 13824 (pixels to 6912)
@pytest.mark.parametrize("npix,nspec", [
    (1, 3), (2, 5), (3, 1), (11, 700), (13, 2), (128, 1000), (210, 9), (301, 20001), (1024, 305),
    (2401, 4), (4099, 3), (6561, 2), (6911, 5), (6917, 3), (6949, 3), (13824, 3), (14000, 3),
    (13889, 2)])
def test_lengths(fsg, npix, nspec):
    rng = np.random.default_rng(npix)
    tau = np.exp(rng.normal(0, 1.5, (nspec, 1)) + rng.normal(0, 1, (nspec, npix)))
    got, want = _got(tau, 0.7), _want(tau, 0.7)
    # both transforms are within about 1e-15 sqrt(log n) of the row's norm per
    # frequency: relative to a frequency's power that is 2 sqrt(mean power / power)
    tol = 1e-13 * np.sqrt(want * want.mean()) + 1e-13 * want + 1e-27 * want.sum()
    assert (np.abs(got - want) <= tol).all(), (np.abs(got - want) / tol).max()


@pytest.mark.parametrize("npix", [512, 6911])
def test_unequal_rows(fsg, npix):
    rng = np.random.default_rng(1)
    big = np.abs(rng.normal(0, 1, (2, npix)))
    small = 0.3566749439387324 + 1e-6 * rng.normal(0, 1, (2, npix))    # exp(-tau) / 0.7 - 1 ~ 1e-6
    const = np.full((3, npix), 0.3566749439387324)
    for rows in (small, np.vstack([big, small, const]), const):
        got, want = _got(rows, 0.7), _want(rows, 0.7)
        # a row's d is known to 2^-53 of 1 (exp and the mean flux)
        assert np.abs(got - want).max() <= 1e-13 * want.max() + 1e-15 * np.sqrt(want.max()) + 1e-31


def test_nan_row(fsg):
    tau = np.ones((4, 300))
    tau[2, 17] = np.nan
    assert np.isnan(_got(tau, 0.7)).all()
