"""Performance cases of the sightline-interpolation path.

Each case is one call (or one step) that a program makes through the package's
public entry points, on synthetic snapshots of the recipes in
``fake_spectra_gb300.synth`` (box sizes, clumping, temperatures, smoothing
lengths), with the sizes of this repository's workloads or smaller and ragged
ones.  ``kind`` names the entry point:

  dropin    _spectra_priv._Particle_Interpolate on host arrays (the call a user
            of the reference makes; FP64 by default, FP32 on request)
  device    interp.particle_interpolate_device on device-resident arrays
  noalloc   interp.particle_interpolate_noalloc (caller owns the GPU memory)
  batch     interp.spectra_batch_device: Ly-a, Ly-b, CIV tau and two column
            densities after one search
  train     autograd.particle_tau: flux, loss and gradients of one fitting step
  channels  interp.colden_channels_device: weighted column densities
  near      interp.near_lines_device: which particles are near any skewer
  flux      fluxstatistics: PDF and 1-D power at a fixed mean flux
"""
import math

import numpy as np
import torch

from fake_spectra_gb300 import _lib, autograd, fluxstatistics, interp, synth
from fake_spectra_gb300 import _spectra_priv as priv

LINES = {"lya": synth.LYA, "lyb": synth.LYB, "civ": synth.CIV}
# synth recipe -> (box in kpc/h); 1: L = 60 Mpc/h, clumps of 100 kpc/h; 3: L = 100 Mpc/h,
# lognormal clumps; 4: L = 20 Mpc/h
BOX = {1: 6e4, 3: 1e5, 4: 2e4}
CUBIC, TOP_HAT, VORONOI, QUINTIC = 1, 0, 2, 3
MEAN_FLUX = 0.68                       # <F> at z = 3
TAUTAIL = 1e-7


def _case(name=None, **kw):
    base = dict(kind="device", recipe=1, nside=64, nlos=100, axis=3, nbins=1000, tau=True,
                line="lya", kernel=CUBIC, precision="fp64", channels=0)
    base.update(kw)
    if name:
        base["name"] = name
    return base


def listed():
    return [
        # a short reference-style call: one small box, 64 skewers, coarse pixels
        _case("dropin tau fp64 32^3", kind="dropin", recipe=4, nside=32, nlos=64, axis=1,
              nbins=223),
        # the same call on a mid-sized box: metal line, quintic kernel, all three axes
        _case("dropin civ fp64 128^3", kind="dropin", recipe=4, nside=128, nlos=400, axis=0,
              nbins=1115, line="civ", kernel=QUINTIC),
        # default precision on a device-resident 256^3 snapshot at 1 km/s
        _case("device tau fp64 256^3", recipe=1, nside=256, nlos=72, axis=3, nbins=6691),
        # Voronoi cells (moving-mesh snapshots)
        _case("dropin voronoi fp64 64^3", kind="dropin", recipe=4, nside=64, nlos=100, axis=2,
              nbins=557, kernel=VORONOI),
        # column densities of a 60 x 60 survey of skewers, host arrays in and out
        _case("dropin colden fp64 256^3", kind="dropin", recipe=1, nside=256, nlos=3600, axis=3,
              nbins=6691, tau=False),
        # the largest survey: 512^3 particles, 32768 skewers over three axes
        _case("device tau fp32 512^3", recipe=3, nside=512, nlos=32768, axis=0, nbins=11152,
              precision="fp32"),
        # the smallest call, where launches and synchronisations count
        _case("noalloc tau fp32 48^3", kind="noalloc", recipe=4, nside=48, nlos=33, axis=2,
              nbins=1115, line="lyb", precision="fp32"),
        # several transitions of one snapshot
        _case("batch fp32 256^3", kind="batch", recipe=1, nside=256, nlos=3600, axis=3,
              nbins=6691, precision="fp32"),
        # one step of a gradient-based fit (forward and backward)
        _case("train fp32 128^3", kind="train", recipe=4, nside=128, nlos=1024, axis=1,
              nbins=1115, precision="fp32"),
        # velocity-, temperature- and density-weighted column densities
        _case("channels fp32 256^3", kind="channels", recipe=1, nside=256, nlos=1800, axis=3,
              nbins=6691, tau=False, precision="fp32", channels=5),
        # which particles are near any skewer (the reference's read filter)
        _case("near lines 256^3", kind="near", recipe=1, nside=256, nlos=3600, axis=0, nbins=0,
              tau=False),
        # flux statistics of a set of spectra (an odd, prime number of pixels)
        _case("flux 3600 x 6691", kind="flux", nside=0, nlos=3600, nbins=6691),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "dropin", "device", "device", "device", "noalloc", "batch",
                       "train", "channels", "near", "flux"])
    recipe = rng.choice([1, 3, 4])
    line = rng.choice(["lya", "lyb", "civ"])
    kernel = rng.choice([CUBIC, CUBIC, QUINTIC, TOP_HAT])
    axis = rng.choice([0, 1, 2, 3])
    if kind == "flux":
        npix = _log_int(rng, 300, 12000)
        return _case(kind="flux", nside=0, nbins=npix,
                     nlos=_log_int(rng, 16, max(17, 24000000 // npix)))
    if kind == "near":
        return _case(kind="near", recipe=recipe, nside=_log_int(rng, 32, 256), axis=axis,
                     nlos=_log_int(rng, 16, 3600), nbins=0, tau=False)
    if kind == "noalloc":
        tau = rng.random() < 0.7
        return _case(kind=kind, recipe=4, nside=_log_int(rng, 24, 64), axis=axis, tau=tau,
                     nlos=_log_int(rng, 16, 128), nbins=_log_int(rng, 300, 2300), line=line,
                     kernel=kernel, precision="fp32" if tau else rng.choice(["fp32", "fp64"]))
    if kind == "train":
        return _case(kind=kind, recipe=4, nside=_log_int(rng, 32, 128), axis=axis, line=line,
                     nlos=_log_int(rng, 32, 1024), nbins=_log_int(rng, 300, 2300),
                     kernel=kernel, precision="fp32")
    if kind == "batch":
        return _case(kind=kind, recipe=recipe, nside=_log_int(rng, 48, 256), axis=axis,
                     nlos=_log_int(rng, 64, 2000), nbins=_log_int(rng, 700, 11152),
                     precision="fp32")
    if kind == "channels":
        return _case(kind=kind, recipe=recipe, nside=_log_int(rng, 48, 256), axis=axis,
                     nlos=_log_int(rng, 64, 1200), nbins=_log_int(rng, 700, 6691), tau=False,
                     kernel=kernel, precision=rng.choice(["fp32", "fp64"]),
                     channels=rng.choice([2, 3, 5, 8]))
    tau = rng.random() < 0.75
    precision = rng.choice(["fp64", "fp64", "fp32"])
    nside = _log_int(rng, 32, 256)
    nbins = _log_int(rng, 200, 11152)
    if tau and precision == "fp64":
        # FP64 optical depths: no more pair-pixels than the listed 256^3 case
        per_px = 1 + 2 * 0.1115 * BOX[recipe] / nbins / 6.0      # sub-samples of wide pixels
        top = min(1024, int(1.2e8 / (nside * nbins * per_px)))
        nlos = _log_int(rng, 8, max(16, top)) if top > 8 else 8
    else:
        nlos = _log_int(rng, 32, 3600)
    return _case(kind=kind, recipe=recipe, nside=nside, nlos=nlos, axis=axis, nbins=nbins,
                 tau=tau, line=line, kernel=kernel, precision=precision)


# ------------------------------------------------------------------ inputs
_CTX = None


def _context():
    # one context for the program, as an application keeps it
    global _CTX
    if _CTX is None:
        _CTX = _lib.Context(torch.cuda.current_device())
    return _CTX


def _snapshot(case, seed):
    """The synth recipe with this case's particle count, skewers and species density."""
    w = synth.generate_torch(case["recipe"], seed=seed, device="cuda", nside=case["nside"],
                             nlos=case["nlos"])
    if case["recipe"] != 3 or case["axis"] != 0:
        rng = np.random.default_rng(seed + 1)
        n = case["nlos"]
        axis = rng.integers(1, 4, size=n) if case["axis"] == 0 else np.full(n, case["axis"])
        w.axis = axis.astype(np.int32)
        w.cofm = rng.uniform(0.0, w.box, size=(n, 3))
    if "CIV" not in w.dens:
        # n_CIV = 10^-4.5 n_HI (delta+1)^0.3, delta+1 from the smoothing length
        mean = 2.0 * w.box / case["nside"]
        w.dens["CIV"] = (w.dens["HI"].double() * 10 ** -4.5 *
                         (mean / w.hh.double()) ** 0.9).float()
    return w


def _tau_field(case, seed):
    """Correlated lognormal optical depths with a few saturated stretches."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n, npix = case["nlos"], case["nbins"]
    x = torch.randn(n, 1, npix + 128, generator=g, device="cuda")
    k = torch.exp(-0.5 * (torch.linspace(-2.5, 2.5, 129, device="cuda")) ** 2)
    x = torch.nn.functional.conv1d(x, (k / k.square().sum().sqrt()).reshape(1, 1, -1))[:, 0]
    return torch.exp(1.8 * x.double() - 1.5)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "flux":
        return {"case": case, "tau": _tau_field(case, seed), "vmax": 1.0 * case["nbins"]}
    w = _snapshot(case, seed)
    st = {"case": case, "w": w, "line": LINES[case["line"]]}
    dens = w.dens[st["line"].species]
    if kind == "dropin":
        st["host"] = [t.cpu().numpy() for t in (w.pos, w.vel, dens, w.temp, w.hh)]
        w.pos = w.vel = w.temp = w.hh = None
        w.dens = {}
    else:
        st["dev"] = (w.pos, w.vel, dens, w.temp, w.hh)
        st["ctx"] = _context()
    if kind == "channels":
        # weights of velocity, temperature and density, as the weighted column densities use them
        base = dens
        weights = [base, base * w.vel[:, 0], base * w.vel[:, 1], base * w.vel[:, 2],
                   base * (w.temp * 1e-4), base * w.vel[:, 0].abs(), base * w.hh * 1e-2,
                   base * 0.5]
        st["dens"] = [t.contiguous() for t in weights[:case["channels"]]]
    if kind == "train":
        g = torch.Generator(device="cuda")
        g.manual_seed(seed + 2)
        st["target"] = torch.rand(case["nlos"], case["nbins"], generator=g, device="cuda")
        pos, vel, dn, temp, hh = st["dev"]
        st["params"] = [t.clone().requires_grad_(True) for t in (vel, dn, temp)]
    return st


def _args(case, w, line):
    return (int(case["tau"]), case["nbins"], case["kernel"], w.box, w.velfac, w.atime,
            line.lambda_cm, line.gamma, line.fosc, line.amumass, TAUTAIL)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "flux":
        bins, pdf = fluxstatistics.flux_pdf(state["tau"], nbins=20, mean_flux_desired=MEAN_FLUX)
        k, power = fluxstatistics.flux_power(state["tau"], state["vmax"],
                                             mean_flux_desired=MEAN_FLUX)
        return {"pdf": pdf, "power": power}
    w, line = state["w"], state["line"]
    if kind == "dropin":
        pos, vel, dens, temp, hh = state["host"]
        return priv._Particle_Interpolate(*_args(case, w, line), pos, vel, dens, temp, hh, w.axis,
                                          w.cofm, precision=case["precision"])
    ctx = state["ctx"]
    pos, vel, dens, temp, hh = state["dev"]
    if kind == "near":
        # the reader's filter: a mask over the particles
        idx = interp.near_lines_device(ctx, w.box, pos, hh, w.axis, w.cofm)
        keep = torch.zeros(pos.shape[0], dtype=torch.bool, device=pos.device)
        keep[idx.long()] = True
        return keep
    if kind == "device":
        return interp.particle_interpolate_device(ctx, *_args(case, w, line), pos, vel, dens,
                                                  temp, hh, w.axis, w.cofm,
                                                  precision=case["precision"])
    if kind == "noalloc":
        return interp.particle_interpolate_noalloc(*_args(case, w, line), pos, vel, dens, temp,
                                                   hh, w.axis, w.cofm,
                                                   precision=case["precision"])
    if kind == "batch":
        hi, civ = w.dens["HI"], w.dens["CIV"]
        out = interp.spectra_batch_device(
            ctx, case["nbins"], case["kernel"], w.box, w.velfac, w.atime, TAUTAIL, pos, vel,
            temp, hh, w.axis, w.cofm,
            [(synth.LYA, hi, True, True), (synth.LYB, hi, True, False),
             (synth.CIV, civ, True, True)], precision=case["precision"])
        return [t for pair in out for t in pair if t is not None]
    if kind == "channels":
        return interp.colden_channels_device(ctx, case["nbins"], case["kernel"], w.box, w.velfac,
                                             pos, hh, w.axis, w.cofm, state["dens"],
                                             precision=case["precision"])
    # train: single-precision flux against its target, gradients of the particle fields
    vel, dens, temp = state["params"]
    tau = autograd.particle_tau(ctx, *_args(case, w, line)[1:], pos, vel, dens, temp, hh, w.axis,
                                w.cofm)
    flux = torch.exp(-tau).float()
    loss = (flux - state["target"]).square().sum()
    gv, gd, gt = torch.autograd.grad(loss, (vel, dens, temp))
    return {"flux": flux.detach(), "vel": gv, "dens": gd, "temp": gt}


# ------------------------------------------------------------------ work
def _pairs_per_line(case):
    # 4 pi nside x the mean of (delta+1)^(-2/3) seen by a skewer, about 0.87 in these recipes
    return 10.9 * case["nside"]


def work(case):
    """Bytes: inputs read once, outputs written once.  Flops: 7 profile values of 32 flops (or
    one kernel integral of 9 nodes of 12 flops) for the pixels within four thermal widths (the
    kernel support) of each pair; the damping wings need far fewer values than pixels."""
    if case["kind"] == "flux":
        n = case["nlos"] * case["nbins"]
        return {"bytes": 8.0 * n, "flops": n * (20.0 + 2.5 * math.log2(case["nbins"]))}
    n, nlos, nbins = case["nside"] ** 3, case["nlos"], case["nbins"]
    if case["kind"] == "near":
        return {"bytes": 16.0 * n, "flops": 10.0 * n}
    pairs = _pairs_per_line(case) * nlos
    outs = {"batch": 5, "channels": case["channels"]}.get(case["kind"], 1)
    kms = 1.115e-1 * BOX[case["recipe"]] / nbins           # pixel width, velfac = 0.1115
    core = min(nbins, 8 * 13.0 / kms + 1)                  # b = 13 km/s: Ly-a at 10^4 K
    support = min(nbins, 2.0 * 1.3 * BOX[case["recipe"]] / case["nside"] * 0.1115 / kms + 1)
    flops = 0.0
    if case["tau"]:
        lines = 3 if case["kind"] == "batch" else 1
        flops += pairs * core * 7 * 32.0 * lines * (3 if case["kind"] == "train" else 1)
    if not case["tau"] or case["kind"] == "batch":
        flops += pairs * support * 9 * 12.0
    fields = 16.0 * n + 4.0 * 3 * pairs + 4.0 * max(1, case["channels"]) * pairs
    grads = 20.0 * n if case["kind"] == "train" else 0.0
    return {"bytes": fields + grads + 8.0 * outs * nlos * nbins, "flops": flops}


# ------------------------------------------------------------------ 64-bit values
PI = math.pi
_SIGMA_T, _KB, _MP, _C_KMS = 6.652458558e-25, 1.3806504e-16, 1.67262178e-24, 299792.458
_TRAP_H = math.sqrt(PI / 14.0)


def _faddeeva(x, a, want_l=False):
    """H = Re w and (want_l) L = Im w of w(x + i a), 0 < a: the trapezoidal rule for
    (i/pi) int exp(-t^2)/(z - t) dt with its pole correction, at t = k h or (k + 1/2) h,
    whichever keeps the nodes away from x."""
    h = _TRAP_H
    frac = torch.remainder(x / h, 1.0)
    half = (frac < 0.25) | (frac > 0.75)                   # the shifted nodes are farther
    x2, a2 = x * x, a * a
    f = 4.0 * a2 * x2
    hsum = torch.where(half, torch.zeros_like(x), 0.5 * a / (x2 + a2))
    lsum = torch.where(half, torch.zeros_like(x), 0.5 * x / (x2 + a2)) if want_l else None
    for k in range(14):
        t2 = torch.where(half, (k + 0.5) ** 2, (k + 1.0) ** 2).to(x) * (h * h)
        d = x2 - a2 - t2
        g = torch.exp(-t2) / (d * d + f)
        hsum = hsum + g * a * (x2 + a2 + t2)
        if want_l:
            lsum = lsum + g * x * (x2 + a2 - t2)
    # 2 exp(-z^2) / (1 -+ exp(-2 pi i z / h)), + for the shifted nodes
    s = torch.where(half, 1.0, -1.0).to(x)
    e = torch.exp(2.0 * PI * a / h)
    th = 2.0 * PI * x / h
    dr, di = 1.0 + s * e * torch.cos(th), -s * e * torch.sin(th)
    m = 2.0 * torch.exp(a2 - x2) / (dr * dr + di * di)
    c, sn = torch.cos(2.0 * x * a), -torch.sin(2.0 * x * a)
    H = 2.0 * h / PI * hsum + m * (c * dr + sn * di)
    if not want_l:
        return H, None
    return H, 2.0 * h / PI * lsum + m * (sn * dr - c * di)


def _spline(kernel, q):
    if kernel == TOP_HAT:
        return torch.full_like(q, 3.0 / 4.0 / PI)
    t = 1.0 - q
    zero = torch.zeros_like(q)
    if kernel == CUBIC:
        v = torch.where(q < 0.5, 1 - 6 * q * q + 6 * q ** 3, 2 * t ** 3) * (8.0 / PI)
    else:
        n = 9.0 / 40 / PI
        v = torch.where(q < 1. / 3, 6 * n * (11 - 90 * q ** 2 + 405 * q ** 4 - 405 * q ** 5),
                        torch.where(q < 2. / 3, n * ((3 * t) ** 5 - 6 * (2 - 3 * q) ** 5),
                                    243 * n * t ** 5))
    return torch.where(q >= 1, zero, v)


def _pairs(pos, hh, axis, cofm, box):
    """(line, particle, dr2) of every particle within its smoothing length of a line."""
    lines, parts, dists = [], [], []
    h2 = (hh * hh).double()
    for i, (ax, c) in enumerate(zip(axis.tolist(), cofm.tolist())):
        p, q = {1: (1, 2), 2: (0, 2), 3: (0, 1)}[ax]
        d1 = (pos[:, p].double() - c[p]).abs()
        d1 = torch.where(d1 > 0.5 * box, box - d1, d1)
        d2 = (pos[:, q].double() - c[q]).abs()
        d2 = torch.where(d2 > 0.5 * box, box - d2, d2)
        dr2 = d1 * d1 + d2 * d2
        k = (dr2 < h2).nonzero()[:, 0]
        lines.append(torch.full_like(k, i))
        parts.append(k)
        dists.append(dr2[k])
    return torch.cat(lines), torch.cat(parts), torch.cat(dists)


def _chunks(n, size):
    return (slice(s, min(n, s + size)) for s in range(0, n, size))


def _exact_tau(case, w, line, fields, gtau=None):
    """tau, or with gtau = dL/dtau the gradients (vel, dens, temp), in 64 bits."""
    pos, vel, dens, temp, hh = fields
    nbins, kernel = case["nbins"], case["kernel"]
    pl, pp, pd = _pairs(pos, hh, w.axis, w.cofm, w.box)
    sigma = math.sqrt(3.0 * PI * _SIGMA_T / 8.0) * line.lambda_cm * line.fosc
    bfac = math.sqrt(2.0 * _KB / (line.amumass * _MP)) / 1e5
    vfac = line.gamma * line.lambda_cm / (4.0 * PI) / 1e5
    width = w.box * w.velfac / nbins
    ax = torch.from_numpy(w.axis.astype(np.int64)).to(pos.device)[pl] - 1
    b = bfac * temp[pp].double().sqrt()
    v0 = w.velfac * pos[pp, ax].double() + vel[pp, ax].double()
    vdr2 = w.velfac * pd * w.velfac
    vs = w.velfac * hh[pp].double()
    vh = (vs * vs - vdr2).clamp(min=0).sqrt()
    dv = 2.0 * vh / 8
    nodes = dv[:, None] * torch.arange(1, 8, device=pos.device) - vh[:, None]
    wt = _spline(kernel, (vdr2[:, None] + nodes * nodes).sqrt() / vs[:, None])
    unit = sigma / math.sqrt(PI) * _C_KMS / b * dv / w.velfac       # times dens times sum w H
    dn = dens[pp].double()
    zmax = torch.floor(v0 / width)
    npts = torch.where(b / 2 > width, torch.ones_like(b), 2 * torch.ceil(width / b) + 1)
    out = torch.zeros(case["nlos"] * nbins, dtype=torch.float64, device=pos.device)
    grads = None
    if gtau is not None:
        grads = [torch.zeros(vel.numel(), dtype=torch.float64, device=pos.device),
                 torch.zeros_like(dens, dtype=torch.float64),
                 torch.zeros_like(temp, dtype=torch.float64)]
        gtau = gtau.reshape(-1)
    half, block = nbins // 2, 128
    for npt in npts.unique().tolist():
        npt = int(npt)
        group = (npts == npt).nonzero()[:, 0]
        for sl in _chunks(len(group), 1 << 14):
            for sign in (1, -1):
                live = group[sl]
                for k0 in range(0, half, block):
                    if not len(live):
                        break
                    k = torch.arange(k0, min(half, k0 + block), device=pos.device)
                    z = zmax[live, None] + (k if sign > 0 else -1 - k)
                    low = z * width - v0[live, None]
                    sums = [0.0, 0.0, 0.0]
                    for s in range(npt):
                        at = low + (0.5 * width if npt == 1 else s * width / (npt - 1))
                        wq = 1.0 if npt == 1 else (0.5 if s in (0, npt - 1) else 1.0) / (npt - 1)
                        for i in range(7):
                            u = (nodes[live, i, None] - at) / b[live, None]
                            a = (vfac / b[live])[:, None]
                            H, L = _faddeeva(u, a, gtau is not None)
                            c = wq * wt[live, i, None]
                            sums[0] = sums[0] + c * H
                            if gtau is not None:
                                hu = -2.0 * (u * H - a * L)
                                ha = 2.0 * (u * L + a * H) - 2.0 / math.sqrt(PI)
                                sums[1] = sums[1] + c * hu
                                sums[2] = sums[2] + c * (H + u * hu + a * ha)
                    tl = (unit * dn)[live, None] * sums[0]
                    below = tl < TAUTAIL
                    keep = below.long().cumsum(1) - below.long() == 0
                    j = pl[live, None] * nbins + torch.remainder(z, nbins).long()
                    if gtau is None:
                        out.index_add_(0, j[keep], tl[keep])
                    else:
                        g = torch.where(keep, gtau[j], torch.zeros_like(tl))
                        p = pp[live]
                        grads[0].index_add_(0, 3 * p + ax[live],
                                            (unit * dn / b)[live] * (g * sums[1]).sum(1))
                        grads[1].index_add_(0, p, unit[live] * (g * sums[0]).sum(1))
                        grads[2].index_add_(0, p, -(unit * dn)[live] / (2 * temp[p].double())
                                            * (g * sums[2]).sum(1))
                    live = live[~below.any(1)]
    if gtau is not None:
        return grads[0].reshape(vel.shape), grads[1], grads[2]
    return out.reshape(case["nlos"], nbins)


def _exact_colden(case, w, pos, hh, densities):
    nbins, kernel = case["nbins"], case["kernel"]
    pl, pp, pd = _pairs(pos, hh, w.axis, w.cofm, w.box)
    ax = torch.from_numpy(w.axis.astype(np.int64)).to(pos.device)[pl] - 1
    p1 = pos[pp, ax].double()
    h = hh[pp].double()
    h2 = (hh * hh).double()[pp]                             # float product, as the inputs' type
    zr = (h2 - pd).sqrt()
    pix = w.box / nbins
    lo = torch.floor((p1 - zr) / pix)
    n = (torch.ceil((p1 + zr) / pix) - lo + 1).long()
    outs = [torch.zeros(case["nlos"] * nbins, dtype=torch.float64, device=pos.device)
            for _ in densities]
    order = torch.argsort(n)
    for sl in _chunks(len(order), 1 << 14):
        e = order[sl]
        for k0 in range(0, int(n[e].max()), 256):
            k = torch.arange(k0, min(int(n[e].max()), k0 + 256), device=pos.device)
            z = lo[e, None] + k
            a = torch.maximum(pix * z - p1[e, None], -zr[e, None])
            b = torch.minimum(pix * z - p1[e, None] + pix, zr[e, None])
            d = b - a
            if kernel == TOP_HAT:
                f = 3.0 / 4.0 / PI * d.clamp(min=0)
            else:
                f = 0.0
                for i in range(9):
                    x = b if i == 8 else a + i * (d / 8)
                    q = (pd[e, None] + x * x).sqrt() / h[e, None]
                    f = f + _spline(kernel, q) * (0.5 if i in (0, 8) else 1.0)
                f = torch.where(d < 0, torch.zeros_like(d), f * d / 8)
            use = k[None, :] < n[e, None]
            j = (pl[e, None] * nbins + torch.remainder(z, nbins).long())[use]
            for out, dens in zip(outs, densities):
                out.index_add_(0, j, (dens[pp[e]].double()[:, None] * f)[use])
    return [o.reshape(case["nlos"], nbins) for o in outs]


def _exact_flux(tau):
    scale, old = 1.0, 0.0
    while abs(scale - old) > 1e-5 * scale:
        old = scale
        f = torch.exp(-scale * tau)
        mean, slope = f.mean().item(), (tau * f).mean().item()
        scale = old + (mean - MEAN_FLUX) / slope
        if scale <= 0:
            scale = 1e-10
    f = torch.exp(-scale * tau)
    edges = torch.arange(21, dtype=torch.float64, device=tau.device) / 20.0
    j = torch.bucketize(f, edges, right=True) - 1
    j = torch.where(f == 1.0, torch.full_like(j, 19), j)
    n = torch.bincount(j.reshape(-1), minlength=20).double()
    power = 0.0
    npix = tau.shape[1]
    for sl in _chunks(tau.shape[0], 1 << 10):
        m = torch.fft.rfft(f[sl] / MEAN_FLUX - 1.0)
        power = power + (m.real.square() + m.imag.square()).sum(0)
    vmax = 1.0 * npix
    return {"pdf": (n / (edges[1:] - edges[:-1]) / n.sum()).cpu().numpy(),
            "power": (vmax * power / npix ** 2 / tau.shape[0]).cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "flux":
        return _exact_flux(_tau_field(case, seed))
    if kind in ("near", "batch") or case["kernel"] == VORONOI:
        return None                     # whole numbers; too long; a search over cells
    cost = _pairs_per_line(case) * case["nlos"] * case["nbins"] * 7.0
    if case["tau"]:
        # 1 km/s pixels against b/2 of cold gas: up to a few sub-samples where pixels are wide
        kms = 1.115e-1 * BOX[case["recipe"]] / case["nbins"]
        cost *= 1 + 2 * kms / 6.0
        if cost > (7e9 if kind == "train" else 1.8e10):
            return None
    elif case["nlos"] * case["nside"] ** 3 > 7e10:
        return None
    st = prepare(case, seed)
    w, line = st["w"], st["line"]
    if "host" in st:
        fields = [torch.from_numpy(a).cuda() for a in st["host"]]
    else:
        fields = st["dev"]
    if kind == "train":
        tau = _exact_tau(case, w, line, fields)
        flux = torch.exp(-tau)
        gtau = -flux * 2.0 * (flux - st["target"].double())
        gv, gd, gt = _exact_tau(case, w, line, fields, gtau)
        return {"flux": flux, "vel": gv, "dens": gd, "temp": gt}
    if case["tau"]:
        tau = _exact_tau(case, w, line, fields)
        return tau if kind != "dropin" else tau.cpu().numpy()
    if kind == "channels":
        return _exact_colden(case, w, fields[0], fields[4], st["dens"])
    out = _exact_colden(case, w, fields[0], fields[4], [fields[2]])[0]
    return out if kind != "dropin" else out.cpu().numpy()
