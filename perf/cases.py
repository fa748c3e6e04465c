"""Measured workloads of the correlators, through the public entry points.

Each case is one call that an XPCS analysis makes: correlate a stack of dense
frames (uint8 or uint16, on the device or in pinned host memory, with or
without the deviation or a two-time matrix), correlate per-pixel event lists,
correlate a per-frame CSR stack, or compress frames to event lists.

Counts are synthetic speckle: a complex Gaussian field that moves smoothly
through independent key fields ``key`` frames apart, intensity mu * |E|^2,
Poisson counts; the q-bins are equal-width annuli around the frame's centre.
"""
import math

import numpy as np
import torch

from dynamix_gb300.correlator import (DenseCorrelator, EventCorrelator, FramesCompressor, MatMulCorrelator,
                                      SparseCorrelator)

DEV = "cuda"


def listed():
    return [
        # a quick look during alignment: a small region of interest, 1,000 frames, 8 narrow rings
        dict(name="dense_small", kind="dense", H=128, W=128, T=1000, bins=8, r0=0, r1=64, dtype="uint8", mu=0.05,
             key=64, where="device"),
        # the usual measurement: a 0.5 Mpx photon-counting detector, 10,000 sparse frames, 16 rings
        dict(name="dense_detector", kind="dense", H=514, W=1030, T=10000, bins=16, r0=20, r1=400, dtype="uint8",
             mu=0.1, key=64, where="device"),
        # a short ragged series: odd frame sides, no round frame count, few rings
        dict(name="dense_ragged", kind="dense", H=487, W=619, T=1777, bins=7, r0=11, r1=290, dtype="uint8", mu=0.2,
             key=32, where="device"),
        # a bright sample on the same kind of detector: counts above 16
        dict(name="dense_bright", kind="dense", H=512, W=512, T=3001, bins=24, r0=10, r1=250, dtype="uint8", mu=1.0,
             key=64, where="device"),
        # frames that a reader has just left in pinned host memory
        dict(name="dense_host", kind="dense", H=514, W=1030, T=3000, bins=16, r0=20, r1=400, dtype="uint8", mu=0.1,
             key=64, where="host"),
        # an integrating detector: uint16 frames, mean 50 counts
        dict(name="dense_u16", kind="dense", H=256, W=256, T=5000, bins=12, r0=8, r1=128, dtype="uint16", mu=50.0,
             key=128, where="device"),
        # the same, strongly exposed: counts above 2048, odd sides
        dict(name="dense_u16_wide", kind="dense", H=195, W=487, T=1500, bins=6, r0=8, r1=190, dtype="uint16",
             mu=400.0, key=64, where="device"),
        # g2 with its deviation, as for error bars in a fit
        dict(name="dense_std", kind="std", H=256, W=256, T=2000, bins=8, r0=8, r1=128, dtype="uint8", mu=0.5, key=64,
             where="device"),
        # g2 and then the two-time matrix of one ring, for an ageing sample
        dict(name="two_time", kind="two_time", H=256, W=256, T=2000, bins=8, r0=8, r1=128, dtype="uint8", mu=0.5,
             key=64, where="device", q=4),
        # event lists of a 1 Mpx detector at very low flux
        dict(name="events", kind="events", H=1062, W=1028, T=20000, bins=32, r0=20, r1=500, mu=0.005, key=200,
             where="device"),
        # a 4.5 Mpx detector's frames as CSR, 20,000 frames
        dict(name="csr", kind="csr", H=2162, W=2068, T=20000, bins=32, r0=20, r1=1000, mu=0.005, key=200,
             where="device"),
        # dense frames to event lists, for storage or the event correlator
        dict(name="compress", kind="compress", H=514, W=1030, T=4000, dtype="uint8", mu=0.1, key=64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: sizes, counts and rings over the ranges that the listed ones stand for."""
    kind = rng.choice(["dense", "dense", "dense", "dense16", "std", "two_time", "events", "csr", "compress"])
    H, W = int(_log(rng, 100, 1100)), int(_log(rng, 100, 1100))
    r1 = round(min(H, W) * rng.uniform(0.3, 0.6))
    c = dict(kind=kind, H=H, W=W, bins=int(_log(rng, 4, 48)), r0=round(r1 * rng.uniform(0.0, 0.3)), r1=r1,
             key=rng.choice([16, 32, 64, 128]))
    if kind == "dense":
        T = min(int(_log(rng, 300, 12000)), int(4e9 / (H * W)))
        c.update(T=T, dtype="uint8", mu=round(_log(rng, 0.01, 1.0), 3), where=rng.choice(["device", "device", "host"]),
                 cls=rng.choice(["matmul", "dense"]))
    elif kind == "dense16":
        T = min(int(_log(rng, 300, 6000)), int(6e8 / (H * W)))
        c.update(kind="dense", T=T, dtype="uint16", mu=round(_log(rng, 0.5, 600.0), 2),
                 where=rng.choice(["device", "device", "host"]), cls=rng.choice(["matmul", "dense"]))
    elif kind in ("std", "two_time"):
        H, W = min(H, 400), min(W, 400)
        r1 = round(min(H, W) * rng.uniform(0.3, 0.6))
        c.update(H=H, W=W, r0=r1 // 5, r1=r1, T=int(_log(rng, 200, 3000)), bins=rng.randint(2, 16), dtype="uint8",
                 mu=round(_log(rng, 0.2, 2.0), 3), where="device")
        if kind == "two_time":
            c["q"] = rng.randint(1, c["bins"])
    elif kind in ("events", "csr"):
        mu = _log(rng, 0.001, 0.02)
        T = min(int(_log(rng, 1000, 20000)), int(1e8 / (H * W * mu)))
        c.update(T=T, mu=round(mu, 5), key=rng.choice([50, 100, 200]), where=rng.choice(["device", "device", "host"]))
    else:
        c = dict(kind=kind, H=H, W=W, T=min(int(_log(rng, 300, 6000)), int(2e9 / (H * W))),
                 dtype=rng.choice(["uint8", "uint8", "uint16"]), mu=round(_log(rng, 0.01, 0.5), 3), key=c["key"])
    return c


def _rings(case):
    """Labels 1..bins of the annuli between r0 and r1, 0 elsewhere (int32)."""
    H, W = case["H"], case["W"]
    y, x = np.mgrid[0:H, 0:W]
    r = np.sqrt((y - H / 2.0) ** 2 + (x - W / 2.0) ** 2)
    q = np.floor((r - case["r0"]) / ((case["r1"] - case["r0"]) / float(case["bins"]))).astype(np.int64) + 1
    q[(r < case["r0"]) | (r >= case["r1"]) | (q > case["bins"])] = 0
    return q.astype(np.int32)


def _field(shape, g):
    return torch.randn((2,) + shape, generator=g, device=DEV) * math.sqrt(0.5)


def _frames(case, seed):
    """The (T, H, W) stack on the device."""
    H, W, T, L = case["H"], case["W"], case["T"], case["key"]
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    wide = case["dtype"] == "uint16"
    out = torch.empty((T, H, W), dtype=torch.uint16 if wide else torch.uint8, device=DEV)
    a = _field((H, W), g)
    for t0 in range(0, T, L):
        b = _field((H, W), g)
        n = min(L, T - t0)
        phase = torch.arange(n, device=DEV, dtype=torch.float32) * (math.pi / (2 * L))
        co, si = torch.cos(phase).view(n, 1, 1), torch.sin(phase).view(n, 1, 1)
        lam = (co * a[0] + si * b[0]).square_().add_((co * a[1] + si * b[1]).square_()).mul_(case["mu"])
        counts = torch.poisson(lam, generator=g)
        if wide:
            out[t0:t0 + n] = counts.clamp_(max=4095).to(torch.int32).to(torch.uint16)
        else:
            out[t0:t0 + n] = counts.clamp_(max=255).to(torch.uint8)
        a = b
    return out


def _filled(mu):
    """Share of non-zero counts of a stack with exponential intensities of mean mu."""
    return 1.0 - 1.0 / (1.0 + mu)


def _thinned(case, frames):
    """The stack with 97 % of the expected non-zero counts, whatever the seed: some of
    them, evenly spread, are set to zero (event lists of one case have one length)."""
    flat = frames.view(-1)
    filled = torch.nonzero(flat.view(torch.int16) if flat.dtype == torch.uint16 else flat).view(-1)
    extra = filled.numel() - int(0.97 * _filled(case["mu"]) * flat.numel())
    if extra > 0:
        flat[filled[torch.arange(extra, device=DEV) * (filled.numel() // extra)]] = 0
    return frames


def _photons(case, seed, by_pixel):
    """(pixel, frame, count) of every non-zero element of a very sparse stack, in
    pixel-major (frame inside a pixel) or frame-major (pixel inside a frame) order."""
    npix, T, L = case["H"] * case["W"], case["T"], case["key"]
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    keys = []
    for t0 in range(0, T, L):
        n = min(L, T - t0)
        lam = _field((npix,), g).square_().sum(0).mul_(case["mu"] * n)
        per = torch.poisson(lam, generator=g).to(torch.int64)
        pix = torch.repeat_interleave(torch.arange(npix, device=DEV), per)
        t = t0 + torch.randint(0, n, pix.shape, generator=g, device=DEV)
        keys.append(pix * T + t if by_pixel else t * npix + pix)
    key, count = torch.unique_consecutive(torch.sort(torch.cat(keys))[0], return_counts=True)
    minor = T if by_pixel else npix
    major = torch.div(key, minor, rounding_mode="floor")
    return major, key - major * minor, count.clamp_(max=255).to(torch.uint8)


def _offsets(index, n):
    """Exclusive running counts of index values 0..n-1 (int64, n + 1)."""
    out = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    out[1:] = torch.cumsum(torch.bincount(index, minlength=n), 0)
    return out


def _events(case, seed):
    """(times int32, data uint8, offsets int64) in the event correlator's layout."""
    pix, t, v = _photons(case, seed, True)
    return t.to(torch.int32), v, _offsets(pix, case["H"] * case["W"])


def _csr(case, seed):
    """(data uint8, indices int32, indptr int32, offsets int64): per-frame CSR."""
    H, W, T = case["H"], case["W"], case["T"]
    t, pix, v = _photons(case, seed, False)
    row = torch.div(pix, W, rounding_mode="floor")
    indptr = torch.zeros((T, H + 1), dtype=torch.int64, device=DEV)
    indptr[:, 1:] = torch.cumsum(torch.bincount(t * H + row, minlength=T * H).view(T, H), 1)
    return v, (pix - row * W).to(torch.int32), indptr.to(torch.int32).view(-1), _offsets(t, T)


def _placed(case, tensors):
    """The tensors as they are, or in pinned host memory."""
    if case.get("where") != "host":
        return tensors
    return tuple(torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t) for t in tensors)


def prepare(case, seed):
    shape, kind = (case["H"], case["W"]), case["kind"]
    if kind == "compress":
        return dict(case=case, args=(_thinned(case, _frames(case, seed)),))
    q = _rings(case)
    if kind == "events":
        times, data, offsets = _events(case, seed)
        corr = EventCorrelator(shape, case["T"], case["T"], total_events_count=len(data), qmask=q)
        return dict(case=case, corr=corr, args=_placed(case, (times, data, offsets)))
    if kind == "csr":
        args = _csr(case, seed)
        if case["where"] == "host":       # the readers write one index type
            args = (args[0], args[1], args[2], args[3].to(torch.int32))
        return dict(case=case, corr=SparseCorrelator(shape, case["T"], qmask=q), args=_placed(case, args))
    cls = DenseCorrelator if case.get("cls") == "dense" else MatMulCorrelator
    return dict(case=case, corr=cls(shape, case["T"], qmask=q), args=_placed(case, (_frames(case, seed),)))


def run(state):
    kind = state["case"]["kind"]
    if kind == "compress":
        data, times, offsets = FramesCompressor.compress_all_stack(*state["args"])
        return {"data": data, "times": times, "offsets": offsets}
    if kind == "std":
        res = state["corr"].correlate(*state["args"], calc_std=True)
        return {"g2": res.res, "dev": res.dev}
    g2 = state["corr"].correlate(*state["args"])
    if kind == "two_time":
        return {"g2": g2, "ttcf": state["corr"].two_time(state["case"]["q"])}
    return {"g2": g2}


def work(case):
    H, W, T, kind = case["H"], case["W"], case["T"], case["kind"]
    npix = float(H * W)
    eb = 2 if case.get("dtype") == "uint16" else 1
    if kind == "compress":
        return {"bytes": npix * T * (eb + _filled(case["mu"]) * (4 + eb)) + 8 * npix, "flops": 0.0}
    P = float(np.count_nonzero(_rings(case)))
    out = 4.0 * case["bins"] * T
    if kind in ("events", "csr"):
        n = T * case["mu"]                                    # events per pixel; pairs of one: n^2 / 2
        pairs = P * n * n / 2 * (1 + case["key"] / T)
        if kind == "events":
            return {"bytes": P * (5 * n + 8) + out, "flops": 2 * pairs}
        return {"bytes": npix * n * 5 + 4.0 * (H + 1) * T + 8 * T + out, "flops": 2 * pairs}
    flops = 2 * P * T * (T + 1) / 2
    if kind == "std":
        return {"bytes": P * T * eb + 2 * out, "flops": flops}
    if kind == "two_time":
        return {"bytes": P * T * eb + out + 4.0 * T * T, "flops": flops}
    return {"bytes": P * T * eb + out, "flops": flops}


def _autocorr(x):
    """Sum over columns of sum_t x(t) x(t + tau) of integer-valued columns (T, n): float64 (T,)."""
    n = 1 << (2 * x.shape[0] - 1).bit_length()
    f = torch.fft.rfft(x.T.to(torch.float64).contiguous(), n=n, dim=1)
    power = torch.view_as_real(f).square_().sum((0, 2))
    return torch.round(torch.fft.irfft(power.to(torch.complex128), n=n))[:x.shape[0]]


def _g2(numer, sums, npix):
    T = sums.shape[1]
    den = torch.stack([_autocorr(s.view(T, 1)) for s in sums])
    return (npix[:, None] * numer / den).cpu().numpy()


def _exact_dense(case, frames, q):
    T, kind = case["T"], case["kind"]
    flat = frames.view(T, -1)
    numer, sums, npix = [], [], []
    extra = {}
    devs = []
    for b in range(1, case["bins"] + 1):
        idx = torch.from_numpy(np.flatnonzero(q.ravel() == b)).to(DEV)
        part = max(1, int(3e8 / (4 * T)))
        N = torch.zeros(T, dtype=torch.float64, device=DEV)
        S = torch.zeros(T, dtype=torch.float64, device=DEV)
        G = torch.zeros((T, T), dtype=torch.float64, device=DEV) if kind in ("std", "two_time") else None
        for k in range(0, idx.numel(), part):
            sel = idx[k:k + part]
            if flat.dtype == torch.uint16:
                x = flat.view(torch.int16)[:, sel].to(torch.float64)
            else:
                x = flat[:, sel].to(torch.float64)
            N += _autocorr(x)
            S += x.sum(1)
            if G is not None:
                G.addmm_(x, x.T)
        numer.append(N)
        sums.append(S)
        P = float(idx.numel())
        npix.append(P)
        if kind == "std":
            ratio = (G / P) / torch.outer(S / P, S / P)
            dev = torch.empty(T, dtype=torch.float64, device=DEV)
            for tau in range(T):
                d = torch.diagonal(ratio, tau)
                dev[tau] = torch.std(d, unbiased=False) / math.sqrt(T - tau)
            devs.append(dev)
        elif kind == "two_time" and b == case["q"]:
            trc = torch.triu(G, 1) * P / T / (torch.outer(S, S) / T)
            if float(torch.diagonal(trc, -5).sum()) < 1:
                trc = trc + trc.T
            first = torch.diagonal(trc, 1)
            mean = first[first > 0].mean()
            torch.diagonal(trc)[:T - 1] = mean
            extra["ttcf"] = trc.cpu().numpy()
    if kind == "std":
        extra["dev"] = torch.stack(devs).cpu().numpy()
    out = {"g2": _g2(torch.stack(numer), torch.stack(sums), torch.tensor(npix, dtype=torch.float64, device=DEV))}
    out.update(extra)
    return out


def _exact_pairs(case, seed, q):
    """Pair sums over the photons of every binned pixel."""
    T, nb = case["T"], case["bins"]
    label = torch.from_numpy(q.ravel().astype(np.int64)).to(DEV)
    pix, t, v = _photons(case, seed, True)
    keep = label[pix] > 0
    pix, t, v = pix[keep], t[keep], v[keep].to(torch.float64)
    base = (label[pix] - 1) * T
    sums = torch.bincount(base + t, weights=v, minlength=nb * T).view(nb, T)
    numer = torch.zeros(nb * T, dtype=torch.float64, device=DEV)
    left = torch.arange(pix.numel(), device=DEV)              # events with a partner k places on
    for k in range(int(torch.bincount(pix).max()) if pix.numel() else 0):
        left = left[left + k < pix.numel()]
        left = left[pix[left] == pix[left + k]]
        numer += torch.bincount(base[left] + t[left + k] - t[left], weights=v[left] * v[left + k], minlength=nb * T)
    npix = torch.bincount(label, minlength=nb + 1)[1:].to(torch.float64)
    return {"g2": _g2(numer.view(nb, T), sums, npix)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "compress":
        return None                                           # whole numbers only
    q = _rings(case)
    if kind in ("events", "csr"):
        if case["H"] * case["W"] * case["T"] * case["mu"] > 2e8:
            return None                                       # more than 20 s
        return _exact_pairs(case, seed, q)
    return _exact_dense(case, _frames(case, seed), q)
