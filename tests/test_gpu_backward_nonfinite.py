"""Gradients for a dL/dtau with an infinity: a particle whose window holds that pixel
gets an infinity of the sign of its own derivative there, also where the window reaches
the pixel through far-field tiles, and every other particle a finite gradient."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins,boost", [(202, 1e5), (1116, 1e6), (3000, 1e5)])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
def test_one_infinite_pixel(ctx, port, nbins, boost, value):
    import torch
    from fake_spectra_gb300.autograd import particle_tau
    w = synth.config4(nside=16, nlos=2)
    t = synth.LYA
    off, part, _ = port.near_particles(w.pos, w.hh, w.axis, w.cofm, w.box)
    rng = np.random.default_rng(nbins)
    near = np.unique(part)
    keep = np.sort(rng.choice(near, size=min(300, near.size), replace=False))
    dens = (w.dens["HI"][keep] * np.where(rng.random(keep.size) < 0.5, boost, 1.0))
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
    leaves = [T(w.vel[keep]), T(dens), T(np.maximum(w.temp[keep], 3e3))]
    for a in leaves:
        a.requires_grad_(True)
    tau = particle_tau(ctx, nbins, w.kernel, w.box, w.velfac, w.atime, t.lambda_cm, t.gamma,
                       t.fosc, t.amumass, w.tautail, T(w.pos[keep]), *leaves, T(w.hh[keep]),
                       w.axis, w.cofm)

    def grads(g):
        return torch.autograd.grad(tau, leaves, torch.as_tensor(g).cuda().to(tau.dtype),
                                   retain_graph=True)

    seen = 0
    for pixel in rng.integers(0, nbins, size=4):
        G = np.zeros((w.nlos, nbins))
        G[0, pixel] = 1.0
        unit = grads(G)                                # each particle's derivative there
        G = rng.normal(size=G.shape)
        G[0, pixel] = value
        for name, one, got in zip(("vel", "dens", "temp"), unit, grads(G)):
            assert not got.isnan().any(), (name, pixel, int(got.isnan().sum()))
            # (the last pixel of a window may go either way)
            sure = one.abs() > 1e-4 * one.abs().max()
            want = torch.sign(one[sure]) * value
            assert torch.equal(got[sure], want), (name, pixel)
            assert got[one == 0].isfinite().float().mean() > 0.99
            seen += int(sure.sum())
    assert seen > 100
