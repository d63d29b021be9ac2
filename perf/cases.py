"""The work a receiver or a training program has this package do, as cases to time.

Every case is one pass through a public entry point on data of a seeded
transmission: payload bits -> BCH, LDPC, bit interleave, constellation ->
channel -> the package.  Es/N0 is given relative to the MODCOD's measured
threshold (``margin``, dB).  The kinds, and the ranges ``draw`` covers:

  pipeline  FecPipeline.decode: cells -> payload bytes; 1..75 FEC Blocks of
            16200 or 64800 bits, every rate and constellation, AWGN with one
            sigma2 or Rayleigh with one per cell
  stream    FecPipeline.decode_stream: the same from a time-interleaved PLP
            cell stream (hybrid or convolutional de-interleaver)
  demap     demap.demap: soft bits alone; sigma2 scalar, per Block, per cell
            or estimated; codeword or transmission order
  demap64   demap.demap_f64: the double-precision soft bits of one long row
  minsum    GpuMinSum.decode: host LLRs in, host decisions out, in the
            decoder's four types
  cpe       cpe.cpe_correct_device: common phase error of an OFDM cell pool
  sp        ldpc.sp_decode: exact sum-product of the Blocks min-sum left open
  train     one training step of the unrolled weighted min-sum: forward,
            loss, backward to the weights
  uneven    batch.UnevenBatch.run: Blocks of many MODCODs in one graph
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from atsc3_b200 import batch, codes, cpe, demap, ldpc, learned, synth, thresholds, timeint
from atsc3_b200.pipeline import FecPipeline

DEV = "cuda"
MODS = ("QPSK", "16QAM", "64QAM", "256QAM", "1024QAM", "4096QAM")
CELLS_PER_FRAME = 1_216_939


def listed():
    return [
        # a low-rate service that hands over each short Block as it arrives:
        # one call, one codeword, latency is all
        {"name": "block_16200", "kind": "pipeline", "n": 16200, "mod": "16QAM", "rate": "11/15",
         "nblk": 1, "chan": "awgn", "margin": 1.0},
        # a mid-rate PLP, one TI block at a time: few long Blocks, fewer than the chip holds
        {"name": "few_64800_256qam", "kind": "pipeline", "n": 64800, "mod": "256QAM",
         "rate": "10/15", "nblk": 7, "chan": "awgn", "margin": 1.5},
        # the headline: one frame of 75 long Blocks under Rayleigh fading near
        # and below the code's threshold, sigma2 per cell
        {"name": "frame_64800_16qam", "kind": "pipeline", "n": 64800, "mod": "16QAM",
         "rate": "6/15", "nblk": 75, "chan": "rayleigh", "margin": 0.0},
        # a PLP straight from the hybrid time interleaver, good reception
        {"name": "stream_64800_64qam", "kind": "stream", "n": 64800, "mod": "64QAM",
         "rate": "8/15", "nblk": 45, "ncols": 15, "ti": "hybrid", "margin": 1.0},
        # soft bits of the densest constellation, a frame at a time
        {"name": "demap_4096qam", "kind": "demap", "n": 64800, "mod": "4096QAM", "rate": "10/15",
         "nblk": 75, "sigma": "cell", "deint": True},
        # soft bits with the noise estimated from the cells, transmission order
        {"name": "demap_estimate", "kind": "demap", "n": 64800, "mod": "1024QAM", "rate": "9/15",
         "nblk": 5, "sigma": "none", "deint": False},
        # the receiver's default double-precision soft bits: one row, noise estimated
        {"name": "demap_f64_row", "kind": "demap64", "mod": "256QAM", "rate": "9/15",
         "ncell": 113_401},
        # the receiver's min-sum call: host LLRs of short Blocks in double precision
        {"name": "minsum_f64", "kind": "minsum", "n": 16200, "rate": "8/15", "mod": "64QAM",
         "nblk": 37, "dtype": "float64", "margin": 1.0},
        # phase correction of a whole frame's cell pool, two PLPs' constellations
        {"name": "cpe_frame", "kind": "cpe", "nsym": 61, "per_sym": 19_949, "mod0": "256QAM",
         "mod1": "16QAM", "rate": "9/15"},
        # the rescue of the Blocks a frame's min-sum left open (at most eight)
        {"name": "sp_rescue", "kind": "sp", "n": 64800, "mod": "16QAM", "rate": "6/15",
         "nblk": 8, "iters": 100, "margin": -0.75},
        # one step of weight training at the trainer's default batch and depth
        {"name": "train_step", "kind": "train", "n": 64800, "mod": "64QAM", "rate": "8/15",
         "nblk": 64, "iters": 12, "buckets": "degree", "margin": 0.0},
        # several PLPs of a multiplex decoded together
        {"name": "uneven_12_modcods", "kind": "uneven", "nmod": 12, "nblk": 96, "mix": 5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("pipeline", "pipeline", "stream", "demap", "demap", "demap64", "minsum",
                       "cpe", "sp", "train", "uneven"))
    n, mod, rate = rng.choice(thresholds.modcods())
    margin = rng.choice((0.5, 1.0, 1.5, 2.0))
    if kind == "pipeline":
        return {"kind": kind, "n": n, "mod": mod, "rate": rate, "nblk": _log(rng, 1, 75),
                "chan": rng.choice(("awgn", "rayleigh")), "margin": margin}
    if kind == "stream":
        ncols = rng.randint(3, 25)
        return {"kind": kind, "n": n, "mod": mod, "rate": rate, "ncols": ncols,
                "nblk": ncols * rng.randint(1, 3), "margin": margin,
                "ti": rng.choice(("hybrid", "convolutional"))}
    if kind == "demap":
        return {"kind": kind, "n": n, "mod": mod, "rate": rate, "nblk": _log(rng, 1, 75),
                "sigma": rng.choice(("none", "scalar", "row", "cell")),
                "deint": rng.random() < 0.7}
    if kind == "demap64":
        mod = rng.choice(MODS)
        cap = 200_000 if codes.MOD_BITS[mod] <= 8 else 20_000
        return {"kind": kind, "mod": mod, "rate": rate, "ncell": _log(rng, 1350, cap)}
    if kind == "minsum":
        dtype = rng.choice(("float64", "float32", "bfloat16", "float16"))
        return {"kind": kind, "n": 16200, "rate": rate, "mod": rng.choice(("QPSK", "64QAM")),
                "nblk": _log(rng, 1, 60), "dtype": dtype, "margin": margin + 0.5}
    if kind == "cpe":
        return {"kind": kind, "nsym": _log(rng, 1, 70), "per_sym": _log(rng, 500, 20_000),
                "mod0": rng.choice(MODS[:4]), "mod1": rng.choice(MODS[:4]), "rate": rate}
    if kind == "sp":
        return {"kind": kind, "n": n, "mod": rng.choice(("QPSK", "16QAM", "64QAM")), "rate": rate,
                "nblk": rng.randint(1, 8), "iters": rng.choice((50, 100)),
                "margin": rng.choice((-0.75, -0.25))}
    if kind == "train":
        rate = rng.choice(("6/15", "8/15", "10/15"))
        return {"kind": kind, "n": 64800, "mod": {"6/15": "16QAM", "8/15": "64QAM"}.get(rate, "256QAM"),
                "rate": rate, "nblk": _log(rng, 4, 60), "iters": rng.randint(3, 12),
                "buckets": rng.choice(("degree", "row")), "margin": margin}
    return {"kind": "uneven", "nmod": rng.randint(2, 12), "nblk": _log(rng, 8, 96),
            "mix": rng.randint(0, 10_000)}


# ---- inputs -----------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _tx(n, mod, rate):
    return synth.Transmitter(n, mod, rate, device=DEV)


@functools.lru_cache(maxsize=None)
def _points(mod, rate):
    return torch.from_numpy(np.asarray(codes.alphabet(mod, rate), np.complex128)).to(DEV)


@functools.lru_cache(maxsize=None)
def _order(n, mod, rate):
    """codeword position of every transmitted bit"""
    return torch.from_numpy(np.asarray(codes.bicm_map(n, mod, rate), np.int64)).to(DEV)


def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _blocks(n, mod, rate, nblk, chan, margin, g):
    """received cells (nblk, ncell), their sigma2, the codewords"""
    tx = _tx(n, mod, rate)
    pay = torch.randint(0, 2, (nblk, tx.kp), generator=g, device=DEV, dtype=torch.uint8)
    x, cw = tx.encode(pay)
    y, s2 = synth.channel(x, thresholds.lookup(n, mod, rate) + margin, chan, g)
    return y, s2, cw


def _edges(rate, n):
    return len(codes.csr(rate, n)[1])


@functools.lru_cache(maxsize=None)
def _minsum(rate, n, dtype):
    cptr, cidx, _, _ = codes.csr(rate, n)
    checks = [cidx[a:b].tolist() for a, b in zip(cptr[:-1], cptr[1:])]
    return ldpc.GpuMinSum(checks, n, dtype=dtype)


@functools.lru_cache(maxsize=None)
def _wms(rate, n, buckets):
    return learned.WmsCode(rate, n, DEV, buckets)


def _mix(case):
    """the uneven case's Blocks: ``nmod`` MODCODs, ``nblk`` Blocks in a mixed order"""
    r = np.random.default_rng(case["mix"])
    mcs = thresholds.modcods()
    some = [mcs[i] for i in r.choice(len(mcs), case["nmod"], replace=False)]
    return [some[i] for i in r.integers(0, len(some), case["nblk"])]


def _llr(case, g):
    y, s2, cw = _blocks(case["n"], case["mod"], case["rate"], case["nblk"], "awgn",
                        case["margin"], g)
    return demap.demap(y, case["mod"], case["rate"], sigma2=s2, n=case["n"]), cw


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "pipeline":
        n, mod, rate = case["n"], case["mod"], case["rate"]
        y, s2, _ = _blocks(n, mod, rate, case["nblk"], case["chan"], case["margin"], g)
        pipe = FecPipeline(n, mod, rate)
        hard = torch.zeros((case["nblk"], (n + 31) // 32 * 4), dtype=torch.uint8, device=DEV)
        return {"case": case, "pipe": pipe, "y": y, "s2": s2, "out": {"hard": hard}}
    if kind == "stream":
        n, mod, rate = case["n"], case["mod"], case["rate"]
        y, s2, _ = _blocks(n, mod, rate, case["nblk"], "awgn", case["margin"], g)
        ncell = y.shape[1]
        if case["ti"] == "hybrid":
            ti = timeint.HybridTI(ncell, case["ncols"], nti=case["nblk"] // case["ncols"])
            cells = ti.interleave(y)
        else:
            ti = timeint.ConvolutionalTI(256, 31, C=17, nblk=case["nblk"], ncell=ncell)
            pre = torch.cat([torch.zeros(17, dtype=y.dtype, device=DEV), y.reshape(-1)])
            cells = ti.interleave(pre, pre.numel() + 256 * 256)
        pipe = FecPipeline(n, mod, rate)
        hard = torch.zeros((case["nblk"], (n + 31) // 32 * 4), dtype=torch.uint8, device=DEV)
        return {"case": case, "pipe": pipe, "cells": cells, "ti": ti, "s2": s2,
                "out": {"hard": hard}}
    if kind == "demap":
        y, s2, _ = _blocks(case["n"], case["mod"], case["rate"], case["nblk"],
                           "rayleigh" if case["sigma"] == "cell" else "awgn", 1.0, g)
        s2 = {"none": lambda: None, "scalar": lambda: s2, "cell": lambda: s2,
              "row": lambda: torch.full((case["nblk"],), s2, device=DEV)}[case["sigma"]]()
        return {"case": case, "y": y, "s2": s2}
    if kind == "demap64":
        pts = _points(case["mod"], case["rate"])
        k = torch.randint(0, pts.numel(), (case["ncell"],), generator=g, device=DEV)
        n0 = 10.0 ** (-(3.0 * codes.MOD_BITS[case["mod"]] - 3.0) / 10.0)
        nz = torch.randn((case["ncell"], 2), generator=g, device=DEV, dtype=torch.float64)
        y = pts[k] + torch.view_as_complex(nz) * math.sqrt(n0 / 2)
        return {"case": case, "y": y[None]}
    if kind == "minsum":
        lam, _ = _llr(case, g)
        return {"case": case, "dec": _minsum(case["rate"], case["n"], case["dtype"]),
                "lam": lam.double().cpu().numpy()}
    if kind == "cpe":
        nsym, per = case["nsym"], case["per_sym"]
        n = nsym * per
        al = [_points(case["mod0"], case["rate"]), _points(case["mod1"], case["rate"])]
        u = torch.rand(n, generator=g, device=DEV)
        region = ((u > 0.6).to(torch.uint8) + (u > 0.85).to(torch.uint8))
        dummy = (1.0 - 2.0 * torch.randint(0, 2, (n,), generator=g, device=DEV)).to(torch.complex128)
        x = torch.where(region == 2, dummy,
                        torch.where(region == 1,
                                    al[1][torch.randint(0, al[1].numel(), (n,), generator=g, device=DEV)],
                                    al[0][torch.randint(0, al[0].numel(), (n,), generator=g, device=DEV)]))
        mag = 1.0 + 0.1 * torch.randn(nsym, generator=g, device=DEV, dtype=torch.float64)
        ang = 0.04 * (2.0 * torch.rand(nsym, generator=g, device=DEV, dtype=torch.float64) - 1.0)
        gain = torch.polar(mag, ang).repeat_interleave(per)
        nz = torch.view_as_complex(torch.randn((n, 2), generator=g, device=DEV, dtype=torch.float64))
        ptr = torch.arange(0, n + 1, per, device=DEV, dtype=torch.int32)
        return {"case": case, "pool": 1.7 * x * gain + nz * math.sqrt(0.5 * 10 ** -2.4), "ptr": ptr,
                "region": region, "al": al, "dummy": dummy}
    if kind == "sp":
        lam, _ = _llr(case, g)
        return {"case": case, "lam": lam.double(),
                "tab": ldpc.sp_tables(codes.csr(case["rate"], case["n"]), case["n"])}
    if kind == "train":
        lam, cw = _llr(case, g)
        code = _wms(case["rate"], case["n"], case["buckets"])
        a, b = code.init_params(case["iters"], 0.8, 0.05)
        a += 0.05 * torch.rand(a.shape, generator=g, device=DEV)
        return {"case": case, "lam": lam, "cw": cw, "code": code, "a": a.requires_grad_(True),
                "b": b.requires_grad_(True)}
    specs = _mix(case)
    cells, s2 = [None] * len(specs), [0.0] * len(specs)
    for mc in sorted(set(specs)):
        at = [i for i, s in enumerate(specs) if s == mc]
        y, v, _ = _blocks(*mc, len(at), "awgn", 1.0, g)
        for j, i in enumerate(at):
            cells[i], s2[i] = y[j], v
    ub = batch.UnevenBatch(specs)
    ub.hard.zero_()
    ub.load(cells, s2)
    ub.capture()
    return {"case": case, "batch": ub}


# ---- one pass ---------------------------------------------------------------

_KEYS = ("lam", "hard", "conv", "its", "bad", "syn", "ok", "payload")


def run(state):
    kind = state["case"]["kind"]
    if kind == "pipeline":
        ws = state["pipe"].decode(state["y"], state["s2"], out=state["out"])
        return {k: ws[k] for k in _KEYS}
    if kind == "stream":
        ws = state["pipe"].decode_stream(state["cells"], state["ti"], state["s2"],
                                         out=state["out"])
        return {k: ws[k] for k in _KEYS}
    if kind == "demap":
        c = state["case"]
        return demap.demap(state["y"], c["mod"], c["rate"], sigma2=state["s2"],
                           n=c["n"], deinterleave=c["deint"])
    if kind == "demap64":
        return demap.demap_f64(state["y"], state["case"]["mod"], state["case"]["rate"])
    if kind == "minsum":
        return state["dec"].decode(state["lam"])
    if kind == "cpe":
        return cpe.cpe_correct_device(state["pool"], state["ptr"], state["region"], state["al"],
                                      state["dummy"])
    if kind == "sp":
        o = ldpc.sp_decode(state["tab"], state["lam"], iters=state["case"]["iters"])
        return {k: o[k] for k in ("bits", "conv", "its", "bad")}
    if kind == "train":
        out = learned.WeightedMinSum.apply(state["lam"], state["a"], state["b"], state["code"],
                                           False)
        loss = learned.bce_loss(out, state["cw"])
        ga, gb = torch.autograd.grad(loss, (state["a"], state["b"]))
        return {"out": out, "loss": loss, "ga": ga, "gb": gb}
    ub = state["batch"]
    ub.run()
    return {"llr": ub.llr, "hard": ub.hard, "payload": ub.payload, "conv": ub.conv,
            "its": ub.its, "bad": ub.bad, "syn": ub.syn, "ok": ub.ok}


# ---- what a pass cannot do without --------------------------------------------

def _demap_work(n, mod, cell_s2):
    """one Block: cells (and sigma2) in, float32 LLRs out; per cell and point
    five operations of the metric and two minima"""
    nb = codes.MOD_BITS[mod]
    ncell = n // nb
    return 8 * ncell + (4 * ncell if cell_s2 else 0) + 4 * n, ncell * 7.0 * (1 << nb)


def _decode_work(n, rate, its):
    """one codeword: decisions and flags out; per edge and iteration about
    eight operations (subtract, two minima, sign, scale, select, add, subtract)"""
    return n // 8 + codes.kpayload(rate, n) // 8 + 34, 8.0 * its * _edges(rate, n)


def _its(margin):
    return 50 if margin <= 0 else 20 if margin < 1.0 else 12


def work(case):
    kind = case["kind"]
    nblk = case.get("nblk", 1)
    if kind in ("pipeline", "stream"):
        db, df = _demap_work(case["n"], case["mod"], case.get("chan") == "rayleigh")
        lb, lf = _decode_work(case["n"], case["rate"], _its(case["margin"]))
        return {"bytes": nblk * (db + lb), "flops": nblk * (df + lf)}
    if kind == "demap":
        db, df = _demap_work(case["n"], case["mod"], case["sigma"] == "cell")
        return {"bytes": nblk * db, "flops": nblk * df}
    if kind == "demap64":
        nb = codes.MOD_BITS[case["mod"]]
        return {"bytes": case["ncell"] * (16 + 8 * nb), "flops": case["ncell"] * 7.0 * (1 << nb)}
    if kind == "minsum":
        size = {"float64": 8, "float32": 4}.get(case["dtype"], 2)
        lb, lf = _decode_work(case["n"], case["rate"], _its(case["margin"]))
        return {"bytes": nblk * (size * case["n"] + case["n"] + 9), "flops": nblk * lf}
    if kind == "cpe":
        n = case["nsym"] * case["per_sym"]
        m = 0.6 * (1 << codes.MOD_BITS[case["mod0"]]) + 0.25 * (1 << codes.MOD_BITS[case["mod1"]])
        return {"bytes": n * 49 + 16 * case["nsym"], "flops": 3.0 * n * (6 * m + 20)}
    if kind == "sp":
        # tanh, log, exp and atanh of every edge and iteration, some twenty operations each
        return {"bytes": nblk * (9 * case["n"] + 9),
                "flops": 80.0 * nblk * min(case["iters"], 30) * _edges(case["rate"], case["n"])}
    if kind == "train":
        n, t = case["n"], case["iters"]
        return {"bytes": nblk * n * 9, "flops": 30.0 * nblk * t * _edges(case["rate"], n)}
    b = f = 0.0
    for n, mod, rate in _mix(case):
        db, df = _demap_work(n, mod, False)
        lb, lf = _decode_work(n, rate, 12)
        b, f = b + db + lb, f + df + lf
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits ------------------------------------------------------

def _llr64(z, pts, nb):
    """(cells, nb) undivided max-log LLRs and (cells,) nearest squared distances"""
    z = z.reshape(-1).to(torch.complex128)
    out = torch.empty((z.numel(), nb), dtype=torch.float64, device=z.device)
    near = torch.empty(z.numel(), dtype=torch.float64, device=z.device)
    step = max(1, (1 << 26) // pts.numel())
    p2 = pts.real ** 2 + pts.imag ** 2
    for lo in range(0, z.numel(), step):
        w = z[lo:lo + step, None]
        q = p2 - 2.0 * (w.real * pts.real + w.imag * pts.imag)
        for i in range(nb):
            m = q.view(-1, 1 << i, 2, 1 << (nb - 1 - i)).amin(dim=(1, 3))
            out[lo:lo + step, i] = m[:, 1] - m[:, 0]
        near[lo:lo + step] = q.amin(1) + w[:, 0].real ** 2 + w[:, 0].imag ** 2
    return out, near


def _soft64(y, s2, n, mod, rate, deint=True):
    """(nblk, n) LLRs of received cells (nblk, ncell); s2: None, a number, per row or per cell"""
    nb = codes.MOD_BITS[mod]
    nblk, ncell = y.shape
    q, near = _llr64(y, _points(mod, rate), nb)
    q = q.view(nblk, ncell, nb)
    if s2 is None:
        s2 = near.view(nblk, ncell).mean(1).clamp_min(1e-9)
    if isinstance(s2, torch.Tensor):
        s2 = s2.double().view(nblk, -1, 1)
    elif y.dtype == torch.complex64:
        s2 = float(np.float32(s2))
    q = (q / s2).reshape(nblk, ncell * nb)
    if not deint:
        return q
    lam = torch.empty_like(q)
    lam[:, _order(n, mod, rate)] = q
    return lam


def _cpe64(s):
    pool, nsym, per = s["pool"], s["case"]["nsym"], s["case"]["per_sym"]
    z = pool / pool.abs().square().mean().sqrt()
    total = torch.ones(nsym, dtype=torch.complex128, device=DEV)
    for _ in range(3):
        h = s["dummy"].clone()
        for r in (0, 1):
            at = (s["region"] == r).nonzero()[:, 0]
            for part in at.split(1 << 16):
                d = (z[part][:, None] - s["al"][r][None, :]).abs()
                h[part] = s["al"][r][d.argmin(1)]
        num = (h.conj() * z).view(nsym, per).sum(1)
        den = h.abs().square().view(nsym, per).sum(1).clamp_min(1e-12)
        c = num / den
        z = (z.view(nsym, per) / c[:, None]).reshape(-1)
        total = total * c
    return z, total


def _train64(s):
    """The unrolled weighted min-sum and its gradient, a few Blocks at a time."""
    c = s["case"]
    cptr, cidx, _, _ = codes.csr(c["rate"], c["n"])
    deg = np.diff(cptr)
    nc, dmax = len(deg), int(deg.max())
    col = np.arange(dmax)
    on = col[None, :] < deg[:, None]
    idx = np.full((nc, dmax), c["n"], np.int64)
    idx[on] = cidx
    idx, on = torch.from_numpy(idx).to(DEV), torch.from_numpy(on).to(DEV)
    bucket = s["code"].t["cbucket"].long()
    a = s["a"].detach().double().requires_grad_(True)
    b = s["b"].detach().double().requires_grad_(True)
    outs, loss = [], 0.0
    ga, gb = torch.zeros_like(a), torch.zeros_like(b)
    ar = torch.arange(dmax, device=DEV)
    for lo in range(0, c["nblk"], 8):
        llr = s["lam"][lo:lo + 8].double()
        nb = llr.shape[0]
        tot, m = llr, torch.zeros((nb, nc, dmax), dtype=torch.float64, device=DEV)
        zero = torch.zeros((nb, 1), dtype=torch.float64, device=DEV)
        for t in range(c["iters"]):
            x = torch.cat([tot, zero], 1)[:, idx] - m
            neg = (x < 0) & on
            mag = torch.where(on, x.abs(), torch.inf)
            two = torch.topk(mag, 2, dim=-1, largest=False, sorted=True)
            mu = torch.where(ar == two.indices[..., :1], two.values[..., 1:], two.values[..., :1])
            v = torch.relu(a[t][bucket][None, :, None] * mu - b[t][bucket][None, :, None])
            par = (neg.sum(-1, keepdim=True) % 2).bool()
            m = torch.where(on, torch.where(par ^ neg, -v, v), 0.0)
            sums = torch.zeros((nb, c["n"] + 1), dtype=torch.float64, device=DEV)
            tot = llr + sums.index_add(1, idx.reshape(-1), m.reshape(nb, -1))[:, :c["n"]]
        part = torch.nn.functional.binary_cross_entropy_with_logits(
            -tot, s["cw"][lo:lo + 8].double(), reduction="sum") / (c["nblk"] * c["n"])
        da, db = torch.autograd.grad(part, (a, b))
        ga, gb, loss = ga + da, gb + db, loss + part.detach()
        outs.append(tot.detach())
    return {"out": torch.cat(outs), "loss": loss, "ga": ga, "gb": gb}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("minsum", "sp"):
        return None                  # decisions and counts only
    s = prepare(case, seed)
    if kind == "pipeline":
        lam = _soft64(s["y"], s["s2"], case["n"], case["mod"], case["rate"])
        return {k: lam if k == "lam" else None for k in _KEYS}
    if kind == "stream":
        nblk, ncell = s["ti"].nblk, s["ti"].ncell
        b = torch.arange(nblk, device=DEV)[:, None]
        r = torch.arange(ncell, device=DEV)[None, :]
        if case["ti"] == "hybrid":
            nc = case["ncols"]
            at = (b // nc) * (nc * ncell) + ncell * ((b % nc - r % nc) % nc) + r
        else:
            i = 17 + b * ncell + r
            at = i + 256 * ((31 + i) % 256)
        lam = _soft64(s["cells"][at], s["s2"], case["n"], case["mod"], case["rate"])
        return {k: lam if k == "lam" else None for k in _KEYS}
    if kind == "demap":
        return _soft64(s["y"], s["s2"], case["n"], case["mod"], case["rate"], case["deint"])
    if kind == "demap64":
        return _soft64(s["y"], None, 0, case["mod"], case["rate"], False)
    if kind == "cpe":
        return _cpe64(s)
    if kind == "train":
        return _train64(s)
    ub = s["batch"]
    llr = torch.empty(ub.llr.numel(), dtype=torch.float64, device=DEV)
    s2 = ub.sigma2.tolist()
    for i, (n, mod, rate) in enumerate(ub.specs):
        o, ncell = int(ub.cell_off[i]), ub.ncell[i]
        lo = int(ub.llr_off[i])
        llr[lo:lo + n] = _soft64(ub.cells[o:o + ncell][None], s2[i], n, mod, rate)[0]
    none = dict.fromkeys(("hard", "payload", "conv", "its", "bad", "syn", "ok"))
    return {"llr": llr, **none}
