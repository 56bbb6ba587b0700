"""FP32 optical depths of few sightlines, shared between blocks: the bits of the
launch with a block per sightline (threads given), for one to many sightlines,
rows with and without far-field tiles, sightlines without pairs, very unequal
ones and one with a NaN."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlos", [1, 5, 120, 400])
@pytest.mark.parametrize("nbins", [50, 1115, 9000])
def test_same_bits(ctx, nlos, nbins):
    import torch
    from fake_spectra_gb300 import interp as I
    w = synth.config4(nside=24, nlos=nlos)
    w.nbins = nbins
    rng = np.random.default_rng(nlos)
    w.cofm[nlos // 2:] = w.cofm[:1]                    # the same busy place, other axes
    if nlos > 3:
        w.cofm[1] = -5 * w.box                         # no particle near
    for bad in (False, True):
        if bad:
            w.dens["HI"] = w.dens["HI"].copy()
            w.dens["HI"][rng.integers(w.npart, size=3)] = np.nan
        a = list(w.call_args(synth.LYA, 1))
        for k in range(11, 16):
            a[k] = torch.from_numpy(np.ascontiguousarray(a[k])).cuda()
        got = I.particle_interpolate_device(ctx, *a, precision="fp32", tune=-1)
        want = I.particle_interpolate_device(ctx, *a, precision="fp32", threads=512)
        # (a sightline with a NaN is summed by FP64 atomics, in no fixed order)
        clean = ~want.isnan().any(dim=1)
        assert torch.equal(got.view(torch.int64)[clean], want.view(torch.int64)[clean])
        assert torch.equal(got.isnan(), want.isnan())
        assert torch.allclose(got, want, rtol=1e-12, atol=0, equal_nan=True)
        # again (the shared words are cleared)
        again = I.particle_interpolate_device(ctx, *a, precision="fp32", tune=-1)
        assert torch.equal(again.view(torch.int64)[clean], want.view(torch.int64)[clean])
