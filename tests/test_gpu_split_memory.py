"""The buffer of shared sightlines is optional: with too little device memory for it a
call runs with a block per sightline and gives the same bits, alone and batched, and
the calls after it are shared again."""
import numpy as np
import pytest

from fake_spectra_gb300 import synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _fill(torch, leave):
    """Device memory held until about `leave` bytes are free."""
    held, size = [], 64 << 30
    while size >= 2 * MB:
        free = torch.cuda.mem_get_info()[0]
        if free - size < leave:
            size //= 2
            continue
        held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
    return held


@pytest.mark.parametrize("precision,nlos,nbins", [("fp64", 1100, 6000), ("fp32", 400, 9000)])
def test_call_without_room_to_share(fsg, precision, nlos, nbins):
    import torch
    from fake_spectra_gb300 import _lib, interp as I
    w = synth.config4(nside=12, nlos=nlos)
    w.nbins = nbins
    ctx = _lib.Context(0)
    held = []
    try:
        a = list(w.call_args(synth.LYA, 1))
        for k in range(11, 16):
            a[k] = torch.from_numpy(np.ascontiguousarray(a[k])).cuda()
        want = torch.empty((nlos, nbins), dtype=torch.float64, device="cuda")
        got = torch.empty_like(want)
        batch = [(synth.LYA, a[13], True, False)]

        def both():
            kw = dict(precision=precision, tune=-1)
            I.particle_interpolate_device(ctx, *a, out=got, **kw)
            assert np.array_equal(got.cpu().numpy(), want_h)
            (tau, _), = I.spectra_batch_device(ctx, nbins, w.kernel, w.box, w.velfac, w.atime,
                                               w.tautail, a[11], a[12], a[14], a[15], w.axis,
                                               w.cofm, batch, **kw)
            assert np.array_equal(tau.cpu().numpy(), want_h)

        # a launch that does not share allocates and loads everything else
        I.particle_interpolate_device(ctx, *a, out=want, precision=precision, persistent=0)
        want_h = want.cpu().numpy()                    # compared on the host
        spare = torch.empty_like(want)                 # room for the batched call's output
        shared = 16 * nlos * nbins                     # the buffer, without its tile nodes
        held = _fill(torch, leave=shared // 3)
        del spare
        assert torch.cuda.mem_get_info()[0] < shared // 2
        both()
        del held[:]
        torch.cuda.empty_cache()
        both()
    finally:
        del held[:]
        ctx.close()
        torch.cuda.empty_cache()
