"""CPU check of the integer kernel integral at the edge of the support
(fsg_spline_fix.cuh, the form of the FP32 column density's end pixels) against
numpy's extended precision: pixels clipped at the support on one side or both,
particles on their sightline and off it, smoothing lengths that are exact in a few
bits (the clipped edge is then at q = 1 exactly) and others."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "fake_spectra_gb300", "csrc")
LD = np.longdouble


def _kernel(cubic, q):
    """The kernel and the magnitude of its derivative, as sums of the terms' magnitudes."""
    t = 1 - q
    if t <= 0:
        return LD(0), LD(0)
    if cubic:
        return (1 - 6 * q * q * t, 12 * q + 18 * q * q) if q < 0.5 else (2 * t ** 3, 6 * t * t)
    third = LD(1) / 3
    r, d = t ** 5, 5 * t ** 4
    for c, b in ((-6, third), (15, 2 * third)):
        if t > b:
            r += c * (t - b) ** 5
            d += 5 * abs(c) * (t - b) ** 4
    return r, d


@pytest.mark.parametrize("cubic", [1, 0])
@pytest.mark.parametrize("h", [1.0, 2.0, 2.5, 37.0, 64.0, 100.0, 12.25, float(np.float32(37.123))])
def test_clipped_pixels(tmp_path, cubic, h):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    if np.finfo(LD).eps > 1e-18:
        pytest.skip("no extended precision")
    exe = str(tmp_path / "spline_edges")
    subprocess.run([cc, "-O2", "-std=c++17", "-x", "c++", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "spline_edges.cpp")], check=True)
    rng = np.random.default_rng(3)
    cases = []
    for dr2 in (0.0, 1e-300, 1e-20 * h * h, 1e-9 * h * h, 0.01 * h * h, 0.5 * h * h, 0.99 * h * h):
        zr = float(np.sqrt(np.float64(np.float32(h) * np.float32(h)) - dr2))
        if zr > h:
            continue
        cases += [(dr2, zr, -zr, zr), (dr2, zr, -zr, -zr), (dr2, zr, zr, zr)]
        for w in (1e-12, 1e-7, 1e-3, 0.1, 0.3, 0.9, 1.0, 1.5, 1.99):
            for f in (1.0, rng.random()):
                d = min(w * f * zr, 2 * zr)
                cases += [(dr2, zr, -zr, -zr + d), (dr2, zr, zr - d, zr)]
    text = "\n".join(" ".join([str(cubic), h.hex()] + [v.hex() for v in c]) for c in cases)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
    got = [float.fromhex(s) for s in out.split()]
    assert len(got) == len(cases)
    for (dr2, _, a, b), g in zip(cases, got):
        want = tol = LD(0)
        for j in range(9):
            z = (LD(a) + (LD(b) - LD(a)) * j / 8) / LD(h)
            q = np.sqrt(LD(dr2) / LD(h) / LD(h) + z * z)
            k, dk = _kernel(cubic, q)
            # z / h and dr2 / h^2 in double are good to 2^-51 of q, and to 2^-49 where the
            # scale is 8 units lower (the derivative where q is that much smaller); the
            # squares to 2^-63, the root to 2^-61 and every product to a unit of 2^-59
            dq = LD(2) ** (-50 if dr2 > 1e-14 * h * h else -48)
            dk = max(dk, _kernel(cubic, max(q - dq, LD(0)))[1])
            c = LD(1) / 2 if j in (0, 8) else LD(1)
            want += c * k
            tol += c * (dk * dq + LD(2) ** -55)
        assert abs(g - want) <= tol, (dr2, a, b, g, float(want), float(tol))
