"""CPU check of the integer Voigt arithmetic (fsg_voigt_fix.cuh): the node sums
against the oracle's Voigt function, over the damping range they serve and
around the edges of their tables: x = 2, 4, 8 (row scales), octaves above, the
last row, and nodes close to and far from the line centre; the far wing's
polynomial and the velocity in units of b against extended precision."""
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


def _build(tmp_path):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "voigt_fix")
    subprocess.run([cc, "-O2", "-std=c++17", "-x", "c++", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "voigt_fix.cpp")], check=True)
    return exe


def test_far_wing(tmp_path):
    LD = np.longdouble
    if np.finfo(LD).eps > 1e-18:
        pytest.skip("no extended precision")
    exe = _build(tmp_path)
    rng = np.random.default_rng(8)
    cases = []
    for _ in range(4000):
        b, vmp = 10 ** rng.uniform(-0.5, 2.5), rng.uniform(12, 300)
        V = vmp * (1 + 10 ** rng.uniform(-5, 2.5))
        r = [(2 * k + 1) / 20.25 ** k * rng.random() for k in range(1, 16)]
        cases.append((b, vmp, 10 ** rng.uniform(-30, 30), 2 * V * b * rng.choice([-1, 1]),
                      float(rng.choice([2, 4, 6, 7, 11, 16])), *r))
    text = "\n".join(" ".join(float(v).hex() for v in c) for c in cases)
    out = subprocess.run([exe, "far"], input=text, capture_output=True, text=True, check=True)
    for c, line in zip(cases, out.stdout.splitlines()):
        got, v = (float.fromhex(s) for s in line.split())
        V = abs(LD(c[3])) / 2 * LD(1.0 / c[0])
        y = LD(c[1] * c[1]) / (V * V)
        want = LD(c[2]) * (y + sum(LD(c[4 + k]) * y ** (k + 1) for k in range(1, int(c[4]))))
        assert abs(got - want) < 3e-16 * want, c
        if V < 1000:
            assert abs(v - V) < 2.5e-16 * V


def test_node_sums(tmp_path, port):
    exe = _build(tmp_path)
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
