"""Performance cases of the X-engine library: what programs ask of it, through
the Python binding of its C ABI (dsax).

A program keeps one context per block geometry (with its beam weights or its
trained net loaded once) and hands it block after block, so `prepare` keeps
the context of the geometry it was last asked for and every state of that
geometry uses it; a training run and a captured batch keep a context of their
own, as they own the net or the graph inside it.  `run` enqueues on the
context's stream and does not wait, except where the call itself returns host
results (host buffers, a training step's loss).

The FP64 values (`exact`) restate the definitions in include/dsax.h with plain
torch and do not use the library.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dsa110-xengine_b200"))

import dsax  # noqa: E402

NBL = 2080
NST = 64
FORMATS = {"captured": dsax.FMT_CAPTURED, "reordered": dsax.FMT_REORDERED}
LF_LAYERS = [(8, 32), (32, 64), (64, 64), (64, 1)]


# ---------------------------------------------------------------------- cases
def listed():
    return [
        # The shortest call a correlator user makes: a quick-look subband of a
        # few channels over an eighth of a block, where launches and latency count.
        _corr("corr_quicklook", npkt=256, nant=63, nchan=16, fmt="captured", data="gauss"),
        # The instrument's block: 2048 packets x 63 antennas x 384 channels, one
        # call per block.
        _corr("corr_block", npkt=2048, nant=63, nchan=384, fmt="captured", data="gauss"),
        # The same block from a host program that already did the corner turn
        # (the REORDER key), as behind the reference's dsaX_reorder_raw.
        _corr("corr_reordered", npkt=2048, nant=64, nchan=384, fmt="reordered", data="gauss"),
        # Several consecutive blocks handed over together.
        _case("corr_stream", "corr_many", npkt=2048, nant=63, nchan=384, nblk=4),
        # The drop-in use: a pinned ring-buffer block in, visibilities out to
        # the host, one subband width down from the full block.
        _case("corr_host", "corr_host", npkt=2048, nant=63, nchan=192),
        # 256 Stokes-I beams of the full block, BF16 operands.
        _beam("beam_block", npkt=2048, nant=63, nchan=384, nbeam=256, ppo=16, fp8=False),
        # FP8 operands on an uneven subband: 25 channel groups, half the beams
        # and four times the time resolution.
        _beam("beam_fp8_uneven", npkt=1936, nant=64, nchan=200, nbeam=128, ppo=4, fp8=True),
        # RFI masks and statistics of one block of beams (FP32 Stokes-I).
        _flag("flag_masks", nbeam=256, ntime=4096, nchan=48),
        # The search node: 16 subbands' beams placed into its 1024-channel uint8
        # filterbank, then normalised, flagged and cleaned in place.
        _case("search_node", "search", nbeam=64, ntime=16384, nsrc=16, nc=48, guard=128),
        # The learned flagger on one block of beams.
        _case("learned_logits", "learned", nbeam=256, ntime=4096, nchan=48, tds=32),
        # One training step of its net on a batch of beams.
        _case("learned_train", "train", nbeam=16, ntime=4096, nchan=48, tds=32),
        # Consecutive blocks of mixed subband widths: correlate, beamform and
        # flag each, as one captured graph.
        _case("batch_mixed", "batch", npkt=2048, nant=63, widths="768,192,384,768,192,384",
              nbeam=256, ppo=16),
    ]


def _case(name, kind, **kw):
    return {"name": name, "kind": kind, **kw} if name else {"kind": kind, **kw}


def _corr(name, **kw):
    return _case(name, "corr", accumulate=kw.pop("accumulate", False), **kw)


def _beam(name, **kw):
    return _case(name, "beam", **kw)


def _flag(name, **kw):
    return _case(name, "flag", **kw)


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["corr", "corr", "corr_many", "corr_host", "beam", "beam", "flag", "flag",
                       "search", "learned", "train", "batch"])
    nant = rng.choice([63, 63, 64, rng.randint(8, 64)])
    if kind == "corr":
        return _corr(None, npkt=_logint(rng, 64, 2048), nant=nant, nchan=_logint(rng, 8, 512),
                     fmt=rng.choice(["captured", "captured", "reordered"]),
                     data=rng.choice(["gauss", "uniform"]), accumulate=rng.random() < 0.25)
    if kind == "corr_many":
        return _case(None, kind, npkt=_logint(rng, 256, 2048), nant=nant,
                     nchan=_logint(rng, 16, 384), nblk=rng.randint(2, 6))
    if kind == "corr_host":
        return _case(None, kind, npkt=_logint(rng, 256, 2048), nant=nant, nchan=_logint(rng, 16, 192))
    if kind == "beam":
        ppo = rng.choice([4, 8, 16, 16, 32])
        step = max(16, ppo)
        return _beam(None, npkt=step * max(1, _logint(rng, 64, 2048) // step), nant=nant,
                     nchan=8 * _logint(rng, 2, 48), nbeam=64 * rng.choice([1, 2, 2, 3, 4, 4, 6]),
                     ppo=ppo, fp8=rng.random() < 0.5)
    if kind == "flag":
        nchan = 4 * _logint(rng, 8, 256)
        ntime = _logint(rng, 512, 16384)
        top = max(1, min(256, (1 << 26) // (nchan * ntime)))
        return _flag(None, nbeam=_logint(rng, 1, top), ntime=ntime, nchan=nchan)
    if kind == "search":
        nsrc, nc = rng.choice([(16, 48), (8, 48), (4, 96), (16, 24), (2, 48)])
        guard = 16 * rng.randint(1, 8)
        return _case(None, kind, nbeam=_logint(rng, 4, 64), ntime=128 * _logint(rng, 8, 128),
                     nsrc=nsrc, nc=nc, guard=guard)
    if kind in ("learned", "train"):
        nchan = 4 * rng.randint(8, 16)
        return _case(None, kind, nbeam=_logint(rng, 1, 256 if kind == "learned" else 16),
                     ntime=128 * _logint(rng, 4, 32), nchan=nchan, tds=rng.choice([16, 32, 32, 64]))
    widths = [32 * _logint(rng, 2, 24) for _ in range(rng.randint(2, 5))]
    return _case(None, kind, npkt=32 * _logint(rng, 8, 64), nant=nant,
                 widths=",".join(str(w) for w in widths), nbeam=128 * rng.randint(1, 2), ppo=16)


# ------------------------------------------------------------------- contexts
_kept = {}


def _context(**cfg):
    """The context of one configuration; the last one asked for is kept."""
    key = tuple(sorted(cfg.items()))
    if key not in _kept:
        _kept.clear()
        _kept[key] = dsax.Context(dsax.default_config(**cfg))
    return _kept[key]


def _bf_scale(ppo):
    """uint8 level 128 / 4 at the mean power of sigma 2.5 samples and unit weights."""
    return 32.0 / (2 * 8 * 2 * ppo * NST * 2 * 6.25)


def _unit_weights(ngrp, nbeam):
    """Unit-magnitude weights with seeded phases [ngrp][2 pol][nbeam][64], FP64."""
    r = np.random.default_rng(ngrp * 1000 + nbeam)
    ph = r.uniform(0.0, 2.0 * np.pi, size=(ngrp, 2, nbeam, NST))
    return np.cos(ph), np.sin(ph)


def _net():
    """He-normal parameters of the learned flagger's net, biases near zero."""
    r = np.random.default_rng(11)
    out = []
    for ci, co in LF_LAYERS:
        out += [r.standard_normal(co * 9 * ci) * math.sqrt(2.0 / (9 * ci)),
                0.02 * r.standard_normal(co)]
    return np.concatenate(out).astype(np.float32)


def _beam_context(nchan, case, fp8):
    ctx = _context(npkt=case["npkt"], nant_in=case["nant"], nchan=nchan, nbeam=case["nbeam"],
                   bf_pkt_per_out=case["ppo"], bf_scale=_bf_scale(case["ppo"]), bf_fp8=int(fp8))
    if not getattr(ctx, "weighted", False):
        ctx.set_weights(*_unit_weights(nchan // 8, case["nbeam"]))
        ctx.weighted = True
    return ctx


# --------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _samples(n, gen, data="gauss"):
    """n packed 4+4-bit samples: Gaussian sigma 2.5 rounded and clipped to
    [-8, 7], or uniform on [-8, 7]."""
    if data == "uniform":
        return torch.randint(0, 256, (n,), generator=gen, device="cuda", dtype=torch.uint8)
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    step = 1 << 26
    for s in range(0, n, step):
        m = min(step, n - s)
        q = [(2.5 * torch.randn(m, generator=gen, device="cuda")).round_().clamp_(-8, 7).to(torch.int8)
             for _ in range(2)]
        out[s:s + m] = ((q[0] & 15) | ((q[1] & 15) << 4)).view(torch.uint8)
    return out


def _captured(case, nchan, gen, data="gauss"):
    return _samples(case["npkt"] * case["nant"] * nchan * 4, gen, data)


def _filterbank(nbeam, ntime, nchan, gen, seed):
    """Stokes-I: exponential noise (mean 2) with persistent tones, bursts and
    drifting tones; and the channels and samples that carry a tone or a burst."""
    x = torch.rand((nbeam, ntime, nchan), generator=gen, device="cuda")
    x.clamp_(min=1e-7).log_().mul_(-2.0)
    cm = torch.zeros((nbeam, nchan), dtype=torch.uint8, device="cuda")
    tm = torch.zeros((nbeam, ntime), dtype=torch.uint8, device="cuda")
    r = np.random.default_rng(seed)
    t = torch.arange(ntime, device="cuda")
    for _ in range(max(1, nbeam // 4)):
        b, c, w = int(r.integers(nbeam)), int(r.integers(nchan - 3)), int(r.integers(1, 4))
        x[b, :, c:c + w] += float(r.uniform(10, 40))
        cm[b, c:c + w] = 1
        b, t0, w = int(r.integers(nbeam)), int(r.integers(ntime - 8)), int(r.integers(1, 9))
        x[b, t0:t0 + w] += float(r.uniform(6, 20))
        tm[b, t0:t0 + w] = 1
    for _ in range(nbeam // 8):
        b, c, d = int(r.integers(nbeam)), float(r.uniform(0, nchan - 1)), float(r.uniform(-8, 8))
        x[b, t, (c + d * t / ntime).round().clamp(0, nchan - 1).long()] += float(r.uniform(10, 30))
    return x, cm, tm


def _search_data(case, seed):
    """Two consecutive blocks of uint8 beams as received from every subband
    [nsrc][nbeam][ntime][nc]: a bandpass around 48 with sigma 6, and the same
    persistent tones and some bursts in each."""
    gen = _gen(seed)
    nsrc, B, T, nc = case["nsrc"], case["nbeam"], case["ntime"], case["nc"]
    r = np.random.default_rng(seed)
    band = torch.from_numpy(r.uniform(42, 54, size=(nsrc, 1, 1, nc)).astype(np.float32)).cuda()
    tones = [(int(r.integers(nsrc)), int(r.integers(B)), int(r.integers(nc)), float(r.uniform(10, 60)))
             for _ in range(max(1, B // 4))]
    blocks = []
    for _ in range(2):
        blk = torch.empty((nsrc, B, T, nc), dtype=torch.uint8, device="cuda")
        for s in range(nsrc):
            z = torch.randn((B, T, nc), generator=gen, device="cuda").mul_(6.0).add_(band[s])
            for ts, b, c, amp in tones:
                if ts == s:
                    z[b, :, c] += amp
            blk[s] = z.round_().clamp_(0, 255).to(torch.uint8)
        for _ in range(max(1, B // 8)):
            b, t0, w = int(r.integers(B)), int(r.integers(T - 8)), int(r.integers(1, 9))
            blk[:, b, t0:t0 + w] += 40
        blocks.append(blk)
    return blocks


def _flag_params(case):
    return dsax.flag_params(case["nbeam"], case["ntime"], case["nchan"])


# -------------------------------------------------------------------- prepare
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_corr(c, seed):
    ctx = _context(npkt=c["npkt"], nant_in=c["nant"], nchan=c["nchan"])
    if c["fmt"] == "captured":
        blk = _captured(c, c["nchan"], _gen(seed), c["data"])
    else:   # [pkt][2 nchan][64][2 pol], absent antennas zero
        blk = _samples(c["npkt"] * 2 * c["nchan"] * NST * 2, _gen(seed), c["data"])
        blk.view(-1, NST, 2)[:, c["nant"]:] = 0
    return {"kind": "corr", "ctx": ctx, "blk": blk, "fmt": FORMATS[c["fmt"]],
            "accumulate": c["accumulate"],
            "vis": torch.zeros((2 * c["nchan"], NBL, 4, 2), device="cuda")}


def _prepare_corr_many(c, seed):
    ctx = _context(npkt=c["npkt"], nant_in=c["nant"], nchan=c["nchan"])
    gen = _gen(seed)
    return {"kind": "corr_many", "ctx": ctx,
            "blks": [_captured(c, c["nchan"], gen) for _ in range(c["nblk"])],
            "vis": [torch.zeros((2 * c["nchan"], NBL, 4, 2), device="cuda") for _ in range(c["nblk"])]}


def _prepare_corr_host(c, seed):
    ctx = _context(npkt=c["npkt"], nant_in=c["nant"], nchan=c["nchan"])
    return {"kind": "corr_host", "ctx": ctx,
            "blk": _captured(c, c["nchan"], _gen(seed)).cpu().pin_memory(),
            "vis": torch.zeros((2 * c["nchan"], NBL, 4, 2)).pin_memory()}


def _prepare_beam(c, seed):
    shape = (c["npkt"] // c["ppo"], c["nbeam"], c["nchan"] // 8)
    return {"kind": "beam", "ctx": _beam_context(c["nchan"], c, c["fp8"]),
            "blk": _captured(c, c["nchan"], _gen(seed)),
            "u8": torch.zeros(shape, dtype=torch.uint8, device="cuda"),
            "power": torch.zeros(shape, device="cuda")}


def _prepare_flag(c, seed):
    B, T, C = c["nbeam"], c["ntime"], c["nchan"]
    x, _, _ = _filterbank(B, T, C, _gen(seed), seed)
    stats = torch.zeros(4 * B * C + B * T, device="cuda")
    return {"kind": "flag", "ctx": _context(npkt=16, nchan=8), "p": _flag_params(c), "x": x,
            "cm": torch.zeros((B, C), dtype=torch.uint8, device="cuda"),
            "tm": torch.zeros((B, T), dtype=torch.uint8, device="cuda"), "stats": stats,
            "moments": stats[:4 * B * C].view(4, B, C), "series": stats[4 * B * C:].view(B, T)}


def _prepare_search(c, seed):
    B, T, C = c["nbeam"], c["ntime"], c["nsrc"] * c["nc"] + 2 * c["guard"]
    ctx = _context(npkt=16, nchan=8)
    p = dsax.flag_params(B, T, C, guard=c["guard"], ts_base=T // 16)
    s = {"kind": "search", "ctx": ctx, "blks": _search_data(c, seed), "turn": 0,
         "fs": ctx.flag_state(p, dsax.flag_clean_params(naver=1), dsax.DTYPE_U8),
         "shape": (c["nsrc"], B, T, c["nc"], T, C, c["guard"]),
         "fil": torch.zeros((B, T, C), dtype=torch.uint8, device="cuda"),
         "cm": torch.zeros((B, C), dtype=torch.uint8, device="cuda"),
         "tm": torch.zeros((B, T), dtype=torch.uint8, device="cuda")}
    torch.cuda.synchronize()
    _run_search(s)   # the first block gives the baseline and starts the flagging
    ctx.sync()
    return s


def _prepare_learned(c, seed):
    B, T, C = c["nbeam"], c["ntime"], c["nchan"]
    x, _, _ = _filterbank(B, T, C, _gen(seed), seed)
    ctx = _context(npkt=16, nchan=8)
    if not getattr(ctx, "trained", False):
        ctx.lf_set_params(_net())
        ctx.trained = True
    shape = (B, T // c["tds"], C)
    return {"kind": "learned", "ctx": ctx, "p": _flag_params(c), "x": x, "tds": c["tds"],
            "mask": torch.zeros(shape, dtype=torch.uint8, device="cuda"),
            "logits": torch.zeros(shape, device="cuda")}


def _prepare_train(c, seed):
    x, cm, tm = _filterbank(c["nbeam"], c["ntime"], c["nchan"], _gen(seed), seed)
    ctx = dsax.Context(dsax.default_config(npkt=16, nchan=8))
    ctx.lf_set_params(_net())
    return {"kind": "train", "ctx": ctx, "p": _flag_params(c), "x": x, "cm": cm, "tm": tm,
            "tds": c["tds"]}


def _widths(c):
    return [int(w) for w in c["widths"].split(",")]


def _prepare_batch(c, seed):
    gen, widths, nout = _gen(seed), _widths(c), c["npkt"] // c["ppo"]
    ctx = dsax.Context(dsax.default_config(npkt=c["npkt"], nant_in=c["nant"], nchan=max(widths),
                                           nbeam=c["nbeam"], bf_pkt_per_out=c["ppo"],
                                           bf_scale=_bf_scale(c["ppo"])))
    ctx.set_weights(*_unit_weights(max(widths) // 8, c["nbeam"]))
    u8 = dict(dtype=torch.uint8, device="cuda")
    return {"kind": "batch", "ctx": ctx, "descs": [
        {"blk": _captured(c, w, gen), "nchan": w,
         "vis": torch.zeros((2 * w, NBL, 4, 2), device="cuda"),
         "beams": torch.zeros((nout, c["nbeam"], w // 8), **u8),
         "chanmask": torch.zeros((c["nbeam"], w // 8), **u8),
         "tsmask": torch.zeros((c["nbeam"], nout), **u8)} for w in widths]}


# ------------------------------------------------------------------------ run
def run(s):
    return globals()["_run_" + s["kind"]](s)


def _run_corr(s):
    s["ctx"].correlate(s["blk"], s["vis"], fmt=s["fmt"], accumulate=s["accumulate"])
    return s["vis"]


def _run_corr_many(s):
    s["ctx"].correlate_many(s["blks"], s["vis"])
    return s["vis"]


def _run_corr_host(s):
    s["ctx"].correlate(s["blk"], s["vis"], dsax.MEM_HOST)
    return s["vis"]


def _run_beam(s):
    s["ctx"].beamform(s["blk"], s["u8"], s["power"])
    return {"u8": s["u8"], "power": s["power"]}


def _run_flag(s):
    s["ctx"].flag(s["p"], s["x"], s["cm"], s["tm"], stats=s["stats"])
    return {"cm": s["cm"], "tm": s["tm"], "moments": s["moments"], "series": s["series"]}


def _run_search(s):
    nsrc, B, T, nc, fil_nt, fil_nc, ch0 = s["shape"]
    s["ctx"].ct_unpack(s["blks"][s["turn"]], nsrc, B, T, nc, s["fil"], fil_nt, fil_nc, 0, ch0)
    s["turn"] ^= 1
    s["fs"].clean(s["fil"], s["cm"], s["tm"])
    return {"fil": s["fil"], "cm": s["cm"], "tm": s["tm"]}


def _run_learned(s):
    # the mask is the sign of the logits inside the guard band
    s["ctx"].flag_learned(s["p"], s["x"], s["mask"], s["logits"], tds=s["tds"])
    return s["logits"]


def _run_train(s):
    loss, grads = s["ctx"].lf_train_step(s["p"], s["x"], s["cm"], s["tm"], tds=s["tds"], lr=1e-3,
                                         pos_weight=3.0, want_grads=True)
    return {"loss": loss, "grads": grads}


def _run_batch(s):
    s["ctx"].run_batch(s["descs"])
    return [[d["vis"], d["beams"], d["chanmask"], d["tsmask"]] for d in s["descs"]]


# ----------------------------------------------------------------------- work
def _vis_bytes(nchan):
    return 2 * nchan * NBL * 4 * 8


def _corr_work(npkt, nant, nchan, extra=0.0):
    """The block read and the visibilities written once; the products of every
    baseline (8 operations per complex multiply-add)."""
    return {"bytes": npkt * nant * nchan * 4 + _vis_bytes(nchan) * (1.0 + extra),
            "flops": 8.0 * NBL * 4 * 2 * nchan * npkt}


def _beam_flops(npkt, nchan, nbeam):
    return 8.0 * nbeam * NST * 2 * nchan * 2 * npkt


def _net_flops():
    return sum(2.0 * 9 * ci * co for ci, co in LF_LAYERS)


def work(c):
    k = c["kind"]
    if k == "corr":
        return _corr_work(c["npkt"], NST if c["fmt"] == "reordered" else c["nant"], c["nchan"],
                          1.0 if c["accumulate"] else 0.0)
    if k == "corr_host":
        return _corr_work(c["npkt"], c["nant"], c["nchan"])
    if k == "corr_many":
        return {m: v * c["nblk"] for m, v in _corr_work(c["npkt"], c["nant"], c["nchan"]).items()}
    if k == "beam":
        out = c["npkt"] // c["ppo"] * c["nbeam"] * (c["nchan"] // 8)
        return {"bytes": c["npkt"] * c["nant"] * c["nchan"] * 4 + 5.0 * out,
                "flops": _beam_flops(c["npkt"], c["nchan"], c["nbeam"])}
    if k == "flag":
        B, T, C = c["nbeam"], c["ntime"], c["nchan"]
        return {"bytes": 4.0 * B * T * C + 17.0 * B * C + 5.0 * B * T, "flops": 0.0}
    if k == "search":
        B, T, C = c["nbeam"], c["ntime"], c["nsrc"] * c["nc"] + 2 * c["guard"]
        return {"bytes": float(B * T * (c["nsrc"] * c["nc"] + C) + B * (C + T)), "flops": 0.0}
    if k in ("learned", "train"):
        B, T, C = c["nbeam"], c["ntime"], c["nchan"]
        px = B * (T // c["tds"]) * C
        if k == "learned":
            return {"bytes": 4.0 * B * T * C + 5.0 * px, "flops": _net_flops() * px}
        n = sum(9 * ci * co + co for ci, co in LF_LAYERS)
        return {"bytes": 4.0 * B * T * C + B * (T + C) + 4.0 * n * 7,
                "flops": (3.0 * _net_flops() - 2.0 * 9 * 8 * 32) * px}
    out = {"bytes": 0.0, "flops": 0.0}
    for w in _widths(c):
        v = _corr_work(c["npkt"], c["nant"], w)
        nout = c["npkt"] // c["ppo"]
        out["bytes"] += v["bytes"] + nout * c["nbeam"] * (w // 8) + c["nbeam"] * (w // 8 + nout)
        out["flops"] += v["flops"] + _beam_flops(c["npkt"], w, c["nbeam"])
    return out


# ---------------------------------------------------------------------- exact
def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return f(case, seed) if f else None


def _nibbles(b):
    """(re, im) FP64 of packed samples."""
    v = b.to(torch.int16)
    return ((((v & 15) ^ 8) - 8).double(), ((((v >> 4) & 15) ^ 8) - 8).double())


def _correlate64(x, nchan):
    """x [pkt][ant][nchan][2 t][2 pol] packed -> visibilities [2 nchan][2080][4][2]."""
    npkt, nant = x.shape[:2]
    vis = torch.empty((2 * nchan, NBL, 4, 2), dtype=torch.float64, device="cuda")
    i, j = torch.tril_indices(NST, NST, device="cuda")
    for ch in range(nchan):
        for t in range(2):
            re = torch.zeros((2, NST, 2, npkt), dtype=torch.float64, device="cuda")
            a, b = _nibbles(x[:, :, ch, t])
            re[0, :nant], re[1, :nant] = a.permute(1, 2, 0), b.permute(1, 2, 0)
            r, m = re[0].reshape(2 * NST, npkt), re[1].reshape(2 * NST, npkt)
            c = m @ r.T
            for part, v in ((0, r @ r.T + m @ m.T), (1, c - c.T)):
                v = v.view(NST, 2, NST, 2)[i, :, j]          # [bl][pol_i][pol_j]
                vis[2 * ch + t, :, :, part] = v.reshape(NBL, 4)
    return vis


def _exact_corr(c, seed):
    if c["fmt"] == "captured":
        x = _captured(c, c["nchan"], _gen(seed), c["data"]).view(c["npkt"], c["nant"], c["nchan"], 2, 2)
    else:
        x = _samples(c["npkt"] * 2 * c["nchan"] * NST * 2, _gen(seed), c["data"])
        x.view(-1, NST, 2)[:, c["nant"]:] = 0
        x = x.view(c["npkt"], c["nchan"], 2, NST, 2).permute(0, 3, 1, 2, 4)
    return _correlate64(x, c["nchan"])


def _exact_corr_many(c, seed):
    gen, shape = _gen(seed), (c["npkt"], c["nant"], c["nchan"], 2, 2)
    blks = [_captured(c, c["nchan"], gen).view(shape) for _ in range(c["nblk"])]
    return [_correlate64(b, c["nchan"]) for b in blks]


def _exact_corr_host(c, seed):
    x = _captured(c, c["nchan"], _gen(seed)).view(c["npkt"], c["nant"], c["nchan"], 2, 2)
    return _correlate64(x, c["nchan"])


def _beams64(x, nchan, nbeam, ppo):
    """Stokes-I power [npkt/ppo][nbeam][nchan/8] of packed x [pkt][ant][nchan][2][2]."""
    npkt, nant = x.shape[:2]
    wre, wim = _unit_weights(nchan // 8, nbeam)
    out = torch.zeros((npkt // ppo, nbeam, nchan // 8), dtype=torch.float64, device="cuda")
    for g in range(nchan // 8):
        for pol in range(2):
            w = torch.complex(torch.from_numpy(wre[g, pol, :, :nant]).cuda(),
                              torch.from_numpy(wim[g, pol, :, :nant]).cuda())
            re, im = _nibbles(x[:, :, 8 * g:8 * g + 8, :, pol])
            v = torch.complex(re, im).permute(1, 0, 2, 3).reshape(nant, -1)
            y = w @ v
            p = (y.real ** 2 + y.imag ** 2).view(nbeam, npkt // ppo, -1).sum(2)
            out[:, :, g] += p.T
    return out


def _exact_beam(c, seed):
    x = _captured(c, c["nchan"], _gen(seed)).view(c["npkt"], c["nant"], c["nchan"], 2, 2)
    return {"u8": None, "power": _beams64(x, c["nchan"], c["nbeam"], c["ppo"])}


def _exact_batch(c, seed):
    gen, out = _gen(seed), []
    for w in _widths(c):
        x = _captured(c, w, gen).view(c["npkt"], c["nant"], w, 2, 2)
        out.append([_correlate64(x, w), None, None, None])
    return out


def _lower_median(v):
    return v.sort(dim=-1).values[..., (v.shape[-1] + 1) // 2 - 1].unsqueeze(-1)


def _moments64(x, p):
    """Per (beam, channel) mean, variance, maximum and peak-to-peak of the
    tbin-sample means."""
    B, T, C = x.shape
    xd = x.double()
    mean = xd.mean(1)
    var = ((xd * xd).mean(1) - mean * mean).clamp(min=0.0)
    nb = T // p.tbin
    bins = xd[:, :nb * p.tbin].view(B, nb, p.tbin, C).mean(2) if nb else None
    pp = bins.amax(1) - bins.amin(1) if nb else torch.zeros_like(mean)
    return mean, var, xd.amax(1), pp


def _detrended(s, p):
    """Channels [guard, C - guard) less the lower median of the filt channels
    from each on (the last windows end at the guard band), and the MAD."""
    C, G, F = s.shape[1], p.guard, p.filt
    j = torch.arange(G, C - G, device="cuda")
    w0 = torch.where(C - G - j >= F, j, torch.full_like(j, C - G - F))
    win = s[:, w0[:, None] + torch.arange(F, device="cuda")]
    d = s[:, G:C - G] - _lower_median(win).squeeze(-1)
    return d, _lower_median((d - _lower_median(d)).abs())


def _boxcar(pp, p):
    """FBIN-channel mean of pp less its median, and the MAD."""
    C, G = pp.shape[1], p.guard
    inner = pp[:, G:C - G]
    med = _lower_median(inner)
    v = pp.unfold(1, p.fbin, 1).mean(-1)[:, G:C - G - p.fbin] - med
    return v, _lower_median((inner - med).abs())


def _exact_flag(c, seed):
    p, C = _flag_params(c), c["nchan"]
    x, _, _ = _filterbank(c["nbeam"], c["ntime"], C, _gen(seed), seed)
    moments = _moments64(x, p)
    mask = torch.zeros((c["nbeam"], C), dtype=torch.bool, device="cuda")
    for s, thr in zip(moments, (p.thresh, p.thresh + p.var_add, p.thresh)):
        d, mad = _detrended(s, p)
        mask[:, p.guard:C - p.guard] |= d.abs() > thr * mad
    v, mad = _boxcar(moments[3], p)
    mask[:, p.guard:C - p.guard - p.fbin] |= v > p.thresh / math.sqrt(p.fbin) * mad
    series = torch.where(mask[:, None, :], torch.full((), 48.0, dtype=torch.float64, device="cuda"),
                         x.double()).mean(2)
    return {"cm": None, "tm": None, "moments": torch.stack(moments), "series": series}


def _slog(v):
    return v.sign() * v.abs().log1p()


def _features64(x, p, tds):
    """The net's eight features per pixel [B][8][T/tds][C] (see dsax_lf_features)."""
    B, T, C = x.shape
    G, H = p.guard, T // tds
    mean, var, mx, pp = _moments64(x, p)
    f = torch.zeros((B, 8, H, C), dtype=torch.float64, device="cuda")
    mu = mean.mean(1)[:, None, None]
    sd = ((var + mean * mean).mean(1)[:, None, None] - mu * mu).sqrt()
    px = x.view(B, H, tds, C).double()
    f[:, 0] = _slog((px.mean(2) - mu) / sd * math.sqrt(tds))
    f[:, 1] = _slog((px.amax(2) - mu) / sd)
    ts = x.double().mean(2)
    med = _lower_median(ts[:, :p.ts_base])
    zt = ((ts - med) / (p.ts_thresh * _lower_median((ts[:, :p.ts_base] - med).abs()))).view(B, H, tds)
    f[:, 2] = _slog(10.0 * (zt.amax(2) - 1.0))[:, :, None]
    for k, (s, thr) in enumerate(zip((mean, var, mx), (p.thresh, p.thresh + p.var_add, p.thresh))):
        z = torch.zeros((B, C), dtype=torch.float64, device="cuda")
        d, mad = _detrended(s, p)
        z[:, G:C - G] = d / (thr * mad)
        f[:, 3 + k] = _slog(10.0 * (z.abs() - 1.0))[:, None, :]
    z = torch.zeros((B, C), dtype=torch.float64, device="cuda")
    v, mad = _boxcar(pp, p)
    z[:, G:C - G - p.fbin] = v / (p.thresh / math.sqrt(p.fbin) * mad)
    f[:, 6] = _slog(10.0 * (z - 1.0))[:, None, :]
    f[:, 7] = _slog(zt.mean(2))[:, :, None]
    return f


def _layers64():
    flat, o, out = torch.from_numpy(_net()).double().cuda(), 0, []
    for ci, co in LF_LAYERS:
        w, b = flat[o:o + co * 9 * ci].view(co, 3, 3, ci), flat[o + co * 9 * ci:o + co * 9 * ci + co]
        out.append((w.clone().requires_grad_(), b.clone().requires_grad_()))
        o += co * 9 * ci + co
    return out


def _forward64(layers, f):
    for k, (w, b) in enumerate(layers):
        f = torch.nn.functional.conv2d(f, w.permute(0, 3, 1, 2), b, padding=1)
        if k < len(layers) - 1:
            f = f.relu()
    return f[:, 0]


def _exact_learned(c, seed):
    x, _, _ = _filterbank(c["nbeam"], c["ntime"], c["nchan"], _gen(seed), seed)
    f, layers = _features64(x, _flag_params(c), c["tds"]), _layers64()
    with torch.no_grad():
        return torch.cat([_forward64(layers, f[b:b + 16]) for b in range(0, c["nbeam"], 16)])


def _exact_train(c, seed):
    x, cm, tm = _filterbank(c["nbeam"], c["ntime"], c["nchan"], _gen(seed), seed)
    p, B, C, H = _flag_params(c), c["nbeam"], c["nchan"], c["ntime"] // c["tds"]
    inside = torch.zeros(C, dtype=torch.bool, device="cuda")
    inside[p.guard:C - p.guard] = True
    row = tm.view(B, H, c["tds"]).amax(2).bool()[:, :, None] & inside
    y = (cm.bool()[:, None, :] | row).double()
    layers = _layers64()
    z = _forward64(layers, _features64(x, p, c["tds"]))
    wgt = torch.where(y > 0, 3.0, 1.0) * inside
    loss = (wgt * (torch.nn.functional.softplus(z) - y * z)).sum() / (B * H * int(inside.sum()))
    grads = torch.autograd.grad(loss, [t for wb in layers for t in wb])
    return {"loss": loss.detach(), "grads": torch.cat([g.reshape(-1) for g in grads])}
