"""The buffer of shared sightlines is optional: where the device has no room for it a
call runs with a block per sightline and gives the same bits, alone and batched, the
calls after it are shared again, and the buffer makes room for one that is needed.
The failures come from a preloaded cudaMalloc, in a process of its own."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def _child(precision, nlos, nbins):
    import ctypes
    import torch
    from fake_spectra_gb300 import _lib, interp as I
    fake = ctypes.CDLL(None)
    fake.fake_malloc_limit.argtypes = [ctypes.c_size_t]

    def case(nside):
        w = synth.config4(nside=nside, nlos=nlos)
        w.nbins = nbins
        a = list(w.call_args(synth.LYA, 1))
        for k in range(11, 16):
            a[k] = torch.from_numpy(np.ascontiguousarray(a[k])).cuda()
        want = I.particle_interpolate_device(ctx, *a, precision=precision, persistent=0)
        return w, a, want

    def check(w, a, want):
        got = I.particle_interpolate_device(ctx, *a, precision=precision, tune=-1)
        assert torch.equal(got, want)
        (tau, _), = I.spectra_batch_device(ctx, nbins, w.kernel, w.box, w.velfac, w.atime,
                                           w.tautail, a[11], a[12], a[14], a[15], w.axis, w.cofm,
                                           [(synth.LYA, a[13], True, False)],
                                           precision=precision, tune=-1)
        assert torch.equal(tau, want)

    ctx = _lib.Context(0)
    small = case(12)               # a launch that does not share allocates everything else
    other = _lib.Context(0)
    ctx, keep = other, ctx
    large = case(20)
    ctx = keep
    # 16 bytes a pixel for the shared buffer, 8 for a row of the output
    fake.fake_malloc_limit(12 * nlos * nbins)
    check(*small)
    assert fake.fake_malloc_failed() >= 2
    fake.fake_malloc_limit(ctypes.c_size_t(-1).value)
    before = fake.fake_malloc_failed()
    check(*small)                  # shared
    assert fake.fake_malloc_failed() == before
    fake.fake_malloc_fail_next(1)  # the pair lists of the larger call
    check(*large)
    assert fake.fake_malloc_failed() == before + 1
    check(*small)
    print("child ok")


@pytest.mark.parametrize("precision,nlos,nbins", [("fp64", 1100, 2000), ("fp32", 400, 9000)])
def test_call_without_room_to_share(fsg, tmp_path, precision, nlos, nbins):
    cc = shutil.which("gcc")
    if cc is None:
        pytest.skip("no C compiler")
    so = str(tmp_path / "fake_malloc.so")
    subprocess.run([cc, "-O1", "-shared", "-fPIC", "-o", so,
                    os.path.join(HERE, "fake_malloc.c"), "-ldl"], check=True)
    r = subprocess.run([sys.executable, os.path.abspath(__file__), precision, str(nlos),
                        str(nbins)], env=dict(os.environ, LD_PRELOAD=so,
                                              PYTHONPATH=os.path.dirname(HERE)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "child ok" in r.stdout, r.stderr[-4000:]


if __name__ == "__main__":
    _child(sys.argv[1], int(sys.argv[2]), int(sys.argv[3]))
