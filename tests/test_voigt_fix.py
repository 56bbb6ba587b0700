"""CPU check of the integer Voigt node sums (fsg_voigt_fix.cuh) against the
oracle's Voigt function, over the damping range they serve and around the
edges of their tables: x = 2, 4, 8 (row scales), octaves above, the last row,
and nodes close to and far from the line centre."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "fake_spectra_gb300", "csrc")


def _weights(rng, kind):
    p2 = rng.random()
    q = np.sqrt(p2 + (1 - p2) * (np.arange(-3, 4) / 4.0) ** 2)
    if kind == 0:
        w = np.ones(7)
    else:
        w = np.where(q < 0.5, 1 - 6 * q * q + 6 * q ** 3, 2 * (1 - q) ** 3)
    return w / w.max()


def test_node_sums(tmp_path, port):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "voigt_fix")
    subprocess.run([cc, "-O2", "-std=c++17", "-x", "c++", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "voigt_fix.cpp")], check=True)
    rng = np.random.default_rng(3)
    grid = lambda v: float(np.floor(v * 2.0 ** 40)) / 2.0 ** 40   # exact in the fixed units
    cases = []
    for x in (0.0, 1e-9, 1 / 32, 0.999999, 2.0, 4.0, 8.0, 16.0, 511.9, 997.0):
        for eps in (-1e-7, 0.0, 1e-7):
            for a in (1e-8, 4.7e-4, 2.0 ** -8):
                cases.append((a, 0.0, grid(abs(x + eps)), np.eye(7)[3]))
    for k in range(6000):
        a = 2.0 ** rng.uniform(-26, -8)
        u1 = grid(rng.choice([0.0, rng.uniform(0, 1), rng.uniform(0, 12)]))
        cases.append((a, u1, grid(rng.uniform(0, 4.5 * 3 * u1 + 13)), _weights(rng, k % 2)))
    text = "\n".join(" ".join(float(v).hex() for v in (a, u, v, *w)) for a, u, v, w in cases)
    r = subprocess.run([exe], input=text, capture_output=True, text=True, check=True)
    got = np.array([float.fromhex(s) for s in r.stdout.split()])
    want = np.array([sum(w[i] * port.voigt(abs((i - 3) * u - v), a) for i in range(7))
                     for a, u, v, w in cases])
    assert got.shape == want.shape
    # the oracle's own profile is good to 5e-15
    assert np.max(np.abs(got - want) / want) < 2e-14
    assert np.median(np.abs(got - want) / want) < 2e-15
