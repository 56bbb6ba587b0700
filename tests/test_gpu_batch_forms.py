"""Batched deposits whose forms need different buffers: a column density before an
optical depth (the shared-sightline state of the second is larger, and near the
shared-memory limit only one of the two keeps its accumulators on chip), in a
context that has made no call yet."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nbins", [300, 13900, 14300])
def test_column_density_first(fsg, nbins, precision):
    import torch
    from fake_spectra_gb300 import _lib, interp as I
    w = synth.config4(nside=16, nlos=20)
    w.nbins = nbins
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    pos, vel, temp, hh, d = T(w.pos), T(w.vel), T(w.temp), T(w.hh), T(w.dens["HI"])
    t = synth.LYA
    lines = [(t, d, False, True), (t, d, True, False), (t, d, True, True)]
    fresh = _lib.Context(0)
    for rep in range(2):
        outs = I.spectra_batch_device(fresh, nbins, w.kernel, w.box, w.velfac, w.atime, w.tautail,
                                      pos, vel, temp, hh, w.axis, w.cofm, lines,
                                      precision=precision, tune=-1)
    other = _lib.Context(0)
    for (_, _, want_tau, want_col), (tau, col) in zip(lines, outs):
        for ct, got in ((1, tau), (0, col)):
            if got is not None:
                ref = I.particle_interpolate_device(other, *w.call_args(t, ct)[:11], pos, vel, d,
                                                    temp, hh, w.axis, w.cofm,
                                                    precision=precision, tune=-1)
                assert torch.equal(got, ref), ct
