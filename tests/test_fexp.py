"""CPU check of the flux passes' exponential (fsg_fexp.cuh) with a scale other
than one: exp(s t) of the exact product s t against extended precision, both
signs, results across the normal range, table edges, subnormal and tiny scales."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "fake_spectra_gb300", "csrc")


@pytest.mark.parametrize("seed,lo,hi", [(0, -60, 0), (1, -8, 6.5), (2, 5.0, 6.55)])
def test_scaled_exponential(tmp_path, seed, lo, hi):
    LD = np.longdouble
    if np.finfo(LD).eps > 1e-18:
        pytest.skip("no extended precision")
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "fexp")
    subprocess.run([cc, "-O2", "-std=c++17", "-x", "c++", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "fexp.cpp")], check=True)
    rng = np.random.default_rng(seed)
    y = np.exp(rng.uniform(lo, hi, 20000)) * rng.choice([-1.0, 1.0], 20000)
    s = np.exp(rng.uniform(-5, 5, y.size)) * rng.choice([-1.0, 1.0], y.size)
    s[:40] = 10.0 ** -np.arange(0, 320, 8)
    # results at the edges of the table's intervals
    k = np.arange(2000)
    y[100:2100] = -k * np.log(2.0) / 1024 * (1 + 2.0 ** -52 * rng.integers(-2, 3, k.size))
    t = y / s
    t[:40] = rng.uniform(0, 1, 40)
    text = "\n".join("%s %s" % (float(a).hex(), float(b).hex()) for a, b in zip(s, t))
    out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True)
    got = np.array([float.fromhex(v) for v in out.stdout.split()])
    p = LD(s) * LD(t)
    want = np.exp(p)
    # half an ulp of rounding (2^-53 relative), 2^-53 for f held to 2^-54 and the
    # polynomial, and the extended product's own rounding
    tol = (2.0 + np.abs(p) * 2.0 ** -10) * LD(2.0) ** -53
    assert (np.abs(LD(got) - want) <= tol * want).all()
