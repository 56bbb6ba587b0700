"""Optical depths and density gradients with tautail = 0: every window covers the row,
so no pixel is left to the stop rule and the values are compared by themselves, without
the absolute slack that the rule needs elsewhere."""
import numpy as np
import pytest

from test_gpu_tau64 import _args, _case
from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


def _no_tail(args):
    args = list(args)
    args[10] = 0.0
    return args


@pytest.mark.parametrize("nbins,kernel,gamma", [
    (64, 1, 6.265e8), (65, 3, 3e11), (257, 0, 6.265e8), (900, 1, 1e3), (1115, 3, 6.265e8),
    (1115, 1, 3e11), (1115, 1, 3e13), (3001, 1, 6.265e8), (8700, 1, 6.265e8), (17000, 3, 1e3)])
@pytest.mark.parametrize("line", [synth.LYA, synth.CIV])
def test_fp64_values(fsg, port, nbins, kernel, gamma, line):
    from fake_spectra_gb300._spectra_priv import _Particle_Interpolate
    args = _no_tail(_args(_case(nbins, n=150, nlos=3), nbins, kernel, line, gamma))
    got = _Particle_Interpolate(*args)
    want = port.particle_interpolate(*args)
    # 1e-11, the FP64 form's tolerance, of every pixel; and the 128-bit sums' unit, 2^-124
    # of a bound at most 2^13 of the row's largest value, times 150 terms
    tol = 1e-11 * want + 2.0 ** -103 * want.max(axis=1, keepdims=True)
    bad = np.abs(got - want) > tol
    assert (want > 0).all() and not bad.any(), (np.argwhere(bad)[:4], got[bad][:4], want[bad][:4])


@pytest.mark.parametrize("nbins,boost", [(50, 1.0), (202, 1e5), (1116, 1.0), (1116, 1e6),
                                         (3000, 1e3)])
def test_density_gradient_of_every_particle(ctx, port, nbins, boost):
    import torch
    from dense_ref import dense_tau
    from fake_spectra_gb300.autograd import particle_tau
    w = synth.config4(nside=16, nlos=2)
    t = synth.LYA
    off, part, _ = port.near_particles(w.pos, w.hh, w.axis, w.cofm, w.box)
    rng = np.random.default_rng(nbins)
    near = np.unique(part)
    keep = np.sort(rng.choice(near, size=min(150, near.size), replace=False))
    pos, vel, hh = w.pos[keep], w.vel[keep], w.hh[keep]
    dens = (w.dens["HI"][keep] * np.where(rng.random(keep.size) < 0.5, boost, 1.0))
    dens = dens.astype(np.float32)
    temp = np.maximum(w.temp[keep], np.float32(3e3))
    off, part, dr2 = port.near_particles(pos, hh, w.axis, w.cofm, w.box)
    line = np.repeat(np.arange(w.nlos), np.diff(off))
    G = torch.as_tensor(rng.uniform(0.5, 1.5, size=(w.nlos, nbins)))
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d = T(dens).requires_grad_(True)
    tau = particle_tau(ctx, nbins, w.kernel, w.box, w.velfac, w.atime, t.lambda_cm, t.gamma,
                       t.fosc, t.amumass, 0.0, T(pos), T(vel), d, T(temp), T(hh), w.axis, w.cofm)
    tau.backward(G.cuda().to(tau.dtype))
    f64 = lambda a: torch.tensor(np.asarray(a, dtype=np.float64))
    ax = w.axis[line] - 1
    pi, axt = torch.from_numpy(part.astype(np.int64)), torch.from_numpy(ax.astype(np.int64))
    ref = f64(dens).requires_grad_(True)
    want = dense_tau((t.lambda_cm, t.gamma, t.fosc, t.amumass), nbins, w.box, w.velfac, 0.0,
                     w.nlos, torch.from_numpy(line), f64(dr2), f64(pos[part, ax]),
                     f64(vel)[pi, axt], ref[pi], f64(temp)[pi], f64(hh[part]))
    (want * G).sum().backward()
    got, ref = d.grad.double().cpu(), ref.grad
    # all terms are positive: the profile's and the tiles' errors (a few 1e-6) and float sums
    assert (ref[pi] > 0).all()
    err = (got - ref).abs() / ref.clamp(min=1e-300)
    assert err[pi].max() <= 1e-4, err[pi].max()
