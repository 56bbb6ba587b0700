"""The autotuner where an FP32 optical depth's sightlines are shared between blocks: it
times the launches that such a call can run (pairs staged per warp), the statistics
name the launch that ran, and a call with a block per sightline keeps its own choice."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlos", [20, 400])
def test_times_what_runs(ctx, nlos):
    import torch
    from fake_spectra_gb300 import _lib, interp as I
    _lib.tune_cache_clear()
    w = synth.config4(nside=24, nlos=nlos)
    a = list(w.call_args(synth.LYA, 1))
    for k in range(11, 16):
        a[k] = torch.from_numpy(np.ascontiguousarray(a[k])).cuda()

    def call(**kw):
        before = ctx.stats()["gpu_launches"]
        out = I.particle_interpolate_device(ctx, *a, precision="fp32", **kw)
        st = ctx.stats()
        return out, st["launch"], st["tune"], st["gpu_launches"] - before

    want, launch, tune, plain = call(tune=-1)
    assert not launch["tuned"] and launch["threads"] == 1024 and launch["records"] == 0
    got, chosen, tune, n = call()
    assert tune["ran"] and tune["candidates"] <= 3 and n <= plain + 2 * 3
    assert chosen["tuned"] and chosen["threads"] == 1024 and chosen["chunk"] in (2, 4, 8)
    assert 0 < tune["ms_best"] <= tune["ms_default"] and torch.equal(got, want)
    got, again, tune, n = call()
    assert not tune["ran"] and again == chosen and n == plain and torch.equal(got, want)
    # asked for, a block per sightline
    got, launch, tune, n = call(threads=512)
    assert launch["threads"] == 512 and not launch["tuned"] and torch.equal(got, want)
