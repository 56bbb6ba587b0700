"""CPU check of the integer kernel integral (fsg_spline_fix.cuh) against
numpy's extended precision: pixels from a millionth of the smoothing length to
the whole support, through the centre, at the breaks of the splines and up to
the last pixel the integer form takes (1 - q^2 = 2^-8)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "fake_spectra_gb300", "csrc")
LD = np.longdouble


def _kernel(cubic, q):
    t = 1 - q
    if cubic:
        return 1 - 6 * q * q * t if q < 0.5 else 2 * t ** 3
    third = LD(1) / 3
    r = t ** 5
    r -= 6 * (t - third) ** 5 if t > third else 0
    r += 15 * (t - 2 * third) ** 5 if t > 2 * third else 0
    return r


def test_pixel_integrals(tmp_path):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    if np.finfo(LD).eps > 1e-18:
        pytest.skip("no extended precision")
    exe = str(tmp_path / "spline_fix")
    subprocess.run([cc, "-O2", "-std=c++17", "-x", "c++", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "spline_fix.cpp")], check=True)
    rng = np.random.default_rng(5)
    grid = lambda v: float(np.floor(v * 2.0 ** 50)) / 2.0 ** 50
    # through the particle itself, a node at z = 0 exactly
    cases = [(c, -w, w, B) for c in (0, 1) for w in (2.0 ** -40, 2.0 ** -10, 0.25, 0.9)
             for B in (0.0, 2.0 ** -50)]
    for k in range(6000):
        B = rng.random() ** rng.choice([0.05, 1.0, 4.0, 40.0]) * 0.996
        lim = 1 - 2.0 ** -8 - B
        if lim <= 0:
            continue
        zl = np.sqrt(lim)
        wd = rng.choice([1e-6, 1e-3, 0.02, 0.3, 2.0]) * rng.random()
        a = rng.choice([rng.uniform(-zl, zl), -zl, zl - wd, -wd / 2, np.sqrt(max(0, .25 - B))])
        if abs(a) <= zl and abs(a + wd) <= zl:
            cases.append((k % 2, grid(a), grid(a + wd), grid(B)))
    assert len(cases) > 3000
    text = "\n".join("%d %s %s %s" % (c, a.hex(), b.hex(), B.hex()) for c, a, b, B in cases)
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout
    got = [float.fromhex(s) for s in out.split()]
    worst = []
    for (c, a, b, B), g in zip(cases, got):
        want = LD(0)
        for j in range(9):
            z = LD(a) + (LD(b) - LD(a)) * j / 8
            want += _kernel(c, np.sqrt(LD(B) + z * z)) / (2 if j in (0, 8) else 1)
        worst.append(float(abs(g - want) / want))
    # 2^-59 per node against sums of at least 2^-12 (quintic tails), and the
    # extended reference's own cancellation
    assert max(worst) < 4e-14 and np.median(worst) < 3e-16
