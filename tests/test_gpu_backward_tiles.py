"""The backward kernel on long damping wings (pixels reached through the nodes
of far-field tiles) against the dense FP64 PyTorch form: rows shorter than a
tile, with a ragged last tile, longer than shared memory holds, absorbers whose
window covers the whole row, sub-sampled pixels.  Tolerances are those of the
other gradient tests (the window's last pixels may differ)."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbins,boost,npart", [
    (50, 1.0, 400), (64, 1e4, 400), (202, 1e5, 400), (1116, 1e3, 400), (1116, 1e6, 200),
    (3000, 1e5, 100), (37002, 1e5, 12)])
def test_gradients_through_tiles(ctx, port, nbins, boost, npart):
    import torch
    from dense_ref import dense_tau
    from fake_spectra_gb300.autograd import particle_tau
    w = synth.config4(nside=16, nlos=2)
    t = synth.LYA
    off, part, dr2 = port.near_particles(w.pos, w.hh, w.axis, w.cofm, w.box)
    rng = np.random.default_rng(nbins)
    near = np.unique(part)
    keep = np.sort(rng.choice(near, size=min(npart, near.size), replace=False))
    pos, vel, hh = w.pos[keep], w.vel[keep], w.hh[keep]
    dens = (w.dens["HI"][keep] * np.where(rng.random(keep.size) < 0.5, boost, 1.0))
    dens = dens.astype(np.float32)
    temp = np.maximum(w.temp[keep], np.float32(3e3))
    off, part, dr2 = port.near_particles(pos, hh, w.axis, w.cofm, w.box)
    line = np.repeat(np.arange(w.nlos), np.diff(off))
    G = torch.as_tensor(rng.normal(size=(w.nlos, nbins)))

    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    leaves = [T(a).requires_grad_(True) for a in (vel, dens, temp)]
    tau = particle_tau(ctx, nbins, w.kernel, w.box, w.velfac, w.atime, t.lambda_cm, t.gamma,
                       t.fosc, t.amumass, w.tautail, T(pos), *leaves, T(hh), w.axis, w.cofm)
    tau.backward(G.cuda().to(tau.dtype))

    f64 = lambda a: torch.tensor(np.asarray(a, dtype=np.float64))
    ax = w.axis[line] - 1
    v, d, k = f64(vel).requires_grad_(True), f64(dens).requires_grad_(True), \
        f64(temp).requires_grad_(True)
    pi = torch.from_numpy(part.astype(np.int64))
    axt = torch.from_numpy(ax.astype(np.int64))
    want = dense_tau((t.lambda_cm, t.gamma, t.fosc, t.amumass), nbins, w.box, w.velfac, w.tautail,
                     w.nlos, torch.from_numpy(line), f64(dr2), f64(pos[part, ax]), v[pi, axt],
                     d[pi], k[pi], f64(hh[part]))
    (want * G).sum().backward()
    for name, got, ref in zip(("vel", "dens", "temp"), leaves, (v, d, k)):
        got, ref = got.grad.double().cpu(), ref.grad
        err = (got - ref).abs()
        # dens spans many decades: its gradients are per unit density
        assert (err <= 2e-3 * ref.abs() + 2e-4 * ref.abs().max()).all(), (name, err.max())
