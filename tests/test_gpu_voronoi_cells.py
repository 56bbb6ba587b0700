"""Voronoi cells against the C oracle where the block's candidate list matters:
more near-equidistant cells than it holds, particles at the same place (ties go
to the smaller index), a single cell, point counts around a block of points."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


def _case(kind, rng, box):
    if kind == "crowded":
        # a thin shell around the sightlines: every cell is nearly as far as any other
        n = 1500
        phi = rng.uniform(0, 2 * np.pi, n)
        r = 0.2 * box * (1 + 1e-4 * rng.random(n))
        pos = np.stack([rng.uniform(0, box, n), 0.5 * box + r * np.cos(phi),
                        0.5 * box + r * np.sin(phi)], axis=1)
        hh = np.full(n, 0.3 * box)
    elif kind == "ties":
        pos = np.repeat(rng.uniform(0, box, (40, 3)), 3, axis=0)[rng.permutation(120)]
        hh = np.full(120, 0.35 * box)
    else:
        pos = np.full((1, 3), 0.5 * box)
        hh = np.full(1, 0.3 * box)
    n = len(pos)
    return dict(pos=pos.astype(np.float32), hh=hh.astype(np.float32),
                vel=(40 * rng.standard_normal((n, 3))).astype(np.float32),
                dens=(rng.lognormal(0, 1, n) * 1e11).astype(np.float32),
                temp=(1e4 * rng.lognormal(0, 0.3, n)).astype(np.float32),
                axis=np.array([1, 1], np.int32),
                cofm=np.array([[0, 0.5 * box, 0.5 * box], [0, 0.48 * box, 0.51 * box]]))


# 0.1 kpc/h points: 1023, 1024, 1025 and many blocks of them
@pytest.mark.parametrize("kind,box", [("crowded", 102.35), ("crowded", 700.0), ("ties", 102.45),
                                      ("ties", 1500.0), ("single", 102.55)])
def test_cells(fsg, port, kind, box):
    from fake_spectra_gb300._spectra_priv import _Particle_Interpolate
    g = _case(kind, np.random.default_rng(11), box)
    t = synth.LYA
    for ct in (0, 1):
        args = (ct, 300, 2, box, synth.cosmology()[2], 0.25, t.lambda_cm, t.gamma, t.fosc,
                t.amumass, 1e-7, g["pos"], g["vel"], g["dens"], g["temp"], g["hh"], g["axis"],
                g["cofm"])
        want = port.particle_interpolate(*args)
        got = _Particle_Interpolate(*args)
        assert (want != 0).any()
        # as tests/test_gpu_voronoi.py
        np.testing.assert_allclose(got, want, rtol=1e-11, atol=1e-14 * np.abs(want).max())
