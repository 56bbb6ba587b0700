"""FP32 column densities of sightlines that pass through particles exactly, with
smoothing lengths whose square is exact in float: the kernel's support then ends at
q = 1 exactly.  Single and multi-channel entries against the C oracle; 1e-5 is the
FP32 form's stated accuracy."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu

H = np.array([1, 2, 2.5, 37, 64, 100, 12.25, 200], np.float32)


@pytest.mark.parametrize("kernel", [1, 3])
@pytest.mark.parametrize("nbins", [1, 33, 900, 14100])
def test_particle_on_its_sightline(ctx, port, kernel, nbins):
    import torch
    from fake_spectra_gb300 import interp as I
    rng = np.random.default_rng(nbins + kernel)
    box, velfac, t, n = 1500.0, synth.cosmology()[2], synth.LYA, 3 * H.size
    pos = rng.uniform(0, box, (n, 3)).astype(np.float32)
    pos[:4, 0] = (0.0, 0.5, box, box - 0.5)            # windows that wrap round the row
    hh = np.tile(H, 3)
    dens = (10 ** rng.uniform(9, 14, (3, n))).astype(np.float32)
    axis = np.repeat([1, 2, 3], H.size).astype(np.int32)
    cofm = pos.astype(np.float64)
    vel, temp = np.zeros_like(pos), np.full_like(hh, 1e4)
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    chan = I.colden_channels_device(ctx, nbins, kernel, box, velfac, T(pos), T(hh), axis, cofm,
                                    [T(d) for d in dens], precision="fp32")
    for c in range(3):
        args = (0, nbins, kernel, box, velfac, 0.25, t.lambda_cm, t.gamma, t.fosc, t.amumass,
                1e-7, pos, vel, dens[c], temp, hh, axis, cofm)
        want = port.particle_interpolate(*args)
        assert (want.max(axis=1) > 0).all()
        dev = list(args)
        for k in range(11, 16):
            dev[k] = T(dev[k])
        got = I.particle_interpolate_device(ctx, *dev, precision="fp32", tune=-1).cpu().numpy()
        for g in (got, chan[c].cpu().numpy()):
            # sums of positive terms, each within 1e-5 of its own value, in units of
            # about 2^-60 of the row's bound
            np.testing.assert_allclose(g, want, rtol=1e-5, atol=1e-12 * want.max())
