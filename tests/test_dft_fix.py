"""CPU check of the fixed-point transforms (fsg_dft_fix.cuh): every radix alone
and combined, both directions, against an extended-precision DFT: noise, a
single spike and a single frequency at the largest norm the scaling allows."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "fake_spectra_gb300", "csrc")


@pytest.mark.parametrize("radices", [[2], [3], [4], [5], [7], [8], [16], [16, 8], [8, 16], [2, 3],
                                     [16, 16, 3], [7, 7, 5], [16, 4, 3, 5], [3, 3, 3, 3]])
def test_fixed_point_transform(tmp_path, radices):
    LD = np.longdouble
    if np.finfo(LD).eps > 1e-18:
        pytest.skip("no extended precision")
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "dft_fix")
    subprocess.run([cc, "-O2", "-std=c++17", "-x", "c++", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "dft_fix.cpp")], check=True)
    n = int(np.prod(radices))
    two_pi = 2 * LD("3.14159265358979323846264338327950288")
    ang = two_pi * np.arange(n).astype(LD) / n
    c, s = np.cos(ang), -np.sin(ang)
    k = (np.arange(n)[:, None] * np.arange(n)[None, :]) % n
    rng = np.random.default_rng(n)
    spike = np.zeros(n, complex)
    spike[n // 2] = 0.6 + 0.8j
    freq = np.exp(2j * np.pi * (np.arange(n) * (n // 3) % n) / n)
    for z in (rng.normal(size=n) + 1j * rng.normal(size=n), spike, freq):
        z = z / np.linalg.norm(z) * 2 ** 0.79          # the scaling's bound is 2^60.8
        text = "\n".join("%s %s" % (float(v.real).hex(), float(v.imag).hex()) for v in z)
        text += "\n" + "\n".join("%s %s" % (float(a).hex(), float(b).hex()) for a, b in zip(c, s))
        x, y = z.real.astype(LD), z.imag.astype(LD)
        wr, wi = c[k] @ x - s[k] @ y, c[k] @ y + s[k] @ x
        for way in ("dif", "dit"):
            out = subprocess.run([exe, way, *map(str, radices)], input=text, capture_output=True,
                                 text=True, check=True)
            got = np.array([[float.fromhex(v) for v in line.split()]
                            for line in out.stdout.splitlines()])
            err = np.hypot(got[:, 0] - wr, got[:, 1] - wi)
            # per pass: the table's 2^-54 of the value, and about a unit per
            # rounding (2^-60 of the norm, times the 2 sqrt(n) of the scale)
            norm = np.sqrt(n) * 2 ** 0.8
            tol = len(radices) * (2.0 ** -53 * np.hypot(wr, wi) + 2.0 ** -51 * norm / np.sqrt(n)
                                  + 2.0 ** -57 * norm)
            assert (err <= tol).all(), (way, (err / tol).max())
