"""The warp-wide sightline search against the oracle's pairs: sightlines per cell
from few to many, smoothing lengths from tiny to half the box, particles in
clusters and spread thin (a warp's box wraps around the periodic edge or spans
the domain), outside the box, with lengths that are zero, negative or not
finite.  The pair lists are compared through the particles near any sightline
and through column densities of known pairs (a count per sightline)."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nlos,hmax,spread", [
    (31, 1, 0.3, 1.0), (33, 40, 0.01, 1.0), (5000, 3, 0.02, 0.01), (5000, 300, 0.05, 0.02),
    (20000, 2000, 0.01, 1.0), (3000, 2000, 0.6, 1.0), (64, 5000, 0.02, 1.0)])
@pytest.mark.parametrize("axes", [(1, 2, 3), (2,)])
def test_pairs(fsg, ctx, port, n, nlos, hmax, spread, axes):
    import torch
    from fake_spectra_gb300 import interp
    from fake_spectra_gb300._spectra_priv import _Particle_Interpolate
    rng = np.random.default_rng(n + nlos)
    box = 1000.0
    centre = rng.choice([0.0, 0.5, 0.999], size=(n, 3))
    pos = np.mod(centre + spread * (rng.random((n, 3)) - 0.5), 1.0) * box
    pos = pos.astype(np.float32)
    hh = (hmax * box * 10 ** rng.uniform(-2, 0, n)).astype(np.float32)
    odd = rng.random(n) < 0.02
    pos[odd] += np.float32(box) * rng.choice([-1, 1], size=(int(odd.sum()), 1)).astype(np.float32)
    hh[::97] = 0.0
    hh[13::97] = -1.0
    axis = rng.choice(axes, size=nlos).astype(np.int32)
    cofm = rng.uniform(0, box, size=(nlos, 3))
    near = rng.integers(n, size=(nlos + 1) // 2)         # sightlines at the edge of supports
    cofm[::2] = pos[near]
    cofm[::2, 2] += np.maximum(hh[near], 0) * (1 + rng.choice([-1e-6, 0, 1e-6], near.size))
    off, part, _ = port.near_particles(pos, hh, axis, cofm, box)
    got = interp.near_lines_device(ctx, box, torch.from_numpy(pos).cuda(),
                                   torch.from_numpy(hh).cuda(), axis, cofm)
    np.testing.assert_array_equal(got.cpu().numpy(),
                                  np.unique(np.asarray(part[:off[-1]])).astype(np.int32))
    # every pair: the sightlines' column densities with one wide pixel
    t = synth.LYA
    args = (0, 1, 0, box, 0.1, 0.25, t.lambda_cm, t.gamma, t.fosc, t.amumass, 1e-7, pos,
            np.zeros_like(pos), rng.random(n).astype(np.float32) + 1, np.full(n, 1e4, np.float32),
            hh, axis, cofm)
    want = port.particle_interpolate(*args)
    assert ctx is not None
    np.testing.assert_allclose(_Particle_Interpolate(*args), want, rtol=1e-11,
                               atol=1e-13 * max(want.max(), 1e-300))
