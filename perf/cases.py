"""Performance cases: what a user of the selector has it do, through its public
entry points (the C ABI as the Python package binds it).

    listed()            the fixed cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs in GPU memory and the handle a program keeps
    run(state)          one call, as a program makes it
    work(case)          bytes a call cannot do without (input read once, answers written once)
    exact(case, seed)   the same answers by a 64-bit sort in torch

A case names its entry point ("entry"):
    bucket / smos   ggms_bucket_multiselect_* / ggms_iterative_smos_*: ks and answers on the host
    ex              ggms_multiselect_*_ex: ks and answers in device memory, stream-ordered
    topk            ggms_topk_*: the K largest values, answers on the host
    batch           ggms_multiselect_segmented_*: many vectors of uneven length at once
    noalloc         ggms_multiselect_noalloc_f32: host ks, device answers, no allocation
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ggms-distributed_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ggms_b200 as G  # noqa: E402

NP = {"f32": np.float32, "f64": np.float64, "u32": np.uint32, "i32": np.int32}
TORCH = {"f32": torch.float32, "f64": torch.float64, "u32": torch.int32, "i32": torch.int32}  # u32: its bits
SIZE = {"f32": 4, "f64": 8, "u32": 4, "i32": 4}
CHUNK = 1 << 26  # values generated at a time


def listed():
    return [
        # five-number summary of a short vector: the smallest call, latency and launches only
        {"name": "summary_f32", "entry": "bucket", "dtype": "f32", "n": 1000, "values": "normal", "ks": "percentiles",
         "nk": 5},
        # all percentiles of a million values, as the reference's callers ask for them
        {"name": "percentiles_f32", "entry": "bucket", "dtype": "f32", "n": 1 << 20, "values": "uniform",
         "ks": "percentiles", "nk": 101},
        # some ranks of a few million integers at a ragged length, inside a device-side program
        {"name": "ranks_i32", "entry": "ex", "dtype": "i32", "n": 3_000_017, "values": "uniform", "ks": "random",
         "nk": 33},
        # the iterativeSMOS benchmark: 2^26 unsigned integers, 1001 random ranks
        {"name": "random_u32", "entry": "smos", "dtype": "u32", "n": 1 << 26, "values": "uniform", "ks": "random",
         "nk": 1001},
        # the same in double precision, ks and answers on the device
        {"name": "random_f64", "entry": "ex", "dtype": "f64", "n": 1 << 26, "values": "normal", "ks": "random",
         "nk": 1001},
        # the headline: ranks clustered in the top 1% of 2^28 half-normal values, plus both extremes
        {"name": "tail_f32", "entry": "ex", "dtype": "f32", "n": 1 << 28, "values": "half_normal", "ks": "top1pct",
         "nk": 1026},
        # the same vector, ranks spread over all of it
        {"name": "spread_f32", "entry": "ex", "dtype": "f32", "n": 1 << 28, "values": "half_normal", "ks": "random",
         "nk": 1024},
        # many ranks of uneven data: a mixture of 8 Gaussians, 2^14 random ranks
        {"name": "mixture_f32", "entry": "ex", "dtype": "f32", "n": 1 << 28, "values": "mixture8", "ks": "random",
         "nk": 1 << 14},
        # top-k of a long score vector, answers on the host
        {"name": "topk_f32", "entry": "topk", "dtype": "f32", "n": 20_000_003, "values": "normal", "ks": "topk",
         "nk": 1000},
        # the batched benchmark: 4096 vectors, lengths log-uniform over 14 octaves, 2^30 values in all, 1-512 ranks each
        {"name": "batch_f32", "entry": "batch", "dtype": "f32", "nseg": 4096, "n": 1 << 30, "octaves": 14.0,
         "values": "uniform_normal", "ks": "random", "kmax": 512, "shape_seed": 41},
        # many short rows (per-row quantiles of a table), a few ranks each
        {"name": "rows_u32", "entry": "batch", "dtype": "u32", "nseg": 20_000, "n": 12_000_000, "octaves": 4.0,
         "values": "uniform", "ks": "random", "kmax": 8, "shape_seed": 7},
        # a latency-critical loop that must not allocate
        {"name": "noalloc_f32", "entry": "noalloc", "dtype": "f32", "n": (1 << 22) + 3, "values": "mixture8",
         "ks": "random", "nk": 300},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["bucket", "smos", "ex", "ex", "ex", "topk", "batch", "batch", "noalloc"])
    if entry == "batch":
        n = _log(rng, 1 << 16, 1 << 29)
        nseg = min(_log(rng, 16, 30_000), n // 64)
        # no more ranks than about one in 16 values
        kmax = min(_log(rng, 1, 512), max(1, n // (8 * nseg)))
        dtype = rng.choice(["f32", "u32"])
        return {"entry": "batch", "dtype": dtype, "nseg": nseg, "n": n, "octaves": round(rng.uniform(0.0, 14.0), 2),
                "values": "uniform_normal" if dtype == "f32" else "uniform", "ks": "random", "kmax": kmax,
                "shape_seed": rng.randrange(1 << 20)}
    dtype = "f32" if entry == "noalloc" else rng.choice(["f32", "f32", "f64", "u32", "i32"])
    n = _log(rng, 256, 1 << 27) if dtype == "f64" or entry == "noalloc" else _log(rng, 256, 1 << 28)
    n = max(256, n - rng.randrange(0, 16))
    most = 1024 if entry == "noalloc" else 1 << 14
    nk = min(_log(rng, 1, most), n // 16)
    values = rng.choice(["uniform", "normal", "half_normal", "cauchy", "lognormal", "mixture8", "distinct256"]) \
        if dtype in ("f32", "f64") else rng.choice(["uniform", "sorted", "distinct256"])
    ks = "topk" if entry == "topk" else rng.choice(["random", "random", "percentiles", "top1pct"])
    if ks == "top1pct":
        nk = max(2, min(nk, n // 100))
    return {"entry": entry, "dtype": dtype, "n": n, "values": values, "ks": ks, "nk": max(1, nk)}


# ------------------------------------------------------------------ inputs
def _fill(dtype, kind, out, g, seed):
    """Values of one distribution into the flat tensor `out`, a chunk at a time."""
    n, dev = out.numel(), out.device
    wide = torch.float64 if dtype == "f64" else torch.float32
    r = np.random.default_rng(seed)
    if kind == "mixture8":  # means U[-100, 100], std log-uniform [0.01, 10], weights Dirichlet(1)
        mean = torch.tensor(r.uniform(-100.0, 100.0, 8), dtype=wide, device=dev)
        std = torch.tensor(np.exp(r.uniform(np.log(0.01), np.log(10.0), 8)), dtype=wide, device=dev)
        edge = torch.tensor(np.cumsum(r.dirichlet(np.ones(8)))[:7], dtype=torch.float32, device=dev)
    elif kind == "distinct256":
        if dtype in ("u32", "i32"):
            table = torch.tensor(r.integers(-(1 << 31), 1 << 31, 256), dtype=torch.int32, device=dev)
        else:
            table = torch.tensor(100.0 * r.standard_normal(256), dtype=wide, device=dev)
    for a in range(0, n, CHUNK):
        b = min(n, a + CHUNK)
        m = b - a
        if kind == "distinct256":
            v = table[torch.randint(0, 256, (m,), generator=g, device=dev)]
        elif dtype in ("u32", "i32"):
            if kind == "sorted":  # one value of each of n equal strata, descending
                i = torch.arange(n - 1 - a, n - 1 - b, -1, device=dev, dtype=torch.float64)
                u = (i + torch.rand(m, generator=g, device=dev, dtype=torch.float64)) * (2.0 ** 32 / n)
                v = u.to(torch.int64).clamp_(0, (1 << 32) - 1)
                v = (v if dtype == "u32" else v - (1 << 31)).to(torch.int32)
            else:
                v = torch.randint(-(1 << 31), 1 << 31, (m,), generator=g, device=dev, dtype=torch.int32)
        elif kind == "uniform":
            v = torch.rand(m, generator=g, device=dev, dtype=wide)
        elif kind == "cauchy":
            v = torch.tan(math.pi * (torch.rand(m, generator=g, device=dev, dtype=torch.float64) - 0.5))
        else:
            v = torch.randn(m, generator=g, device=dev, dtype=wide)
            if kind == "half_normal":
                v = v.abs_()
            elif kind == "lognormal":
                v = torch.exp_(v.mul_(2.0))
            elif kind == "mixture8":
                c = torch.bucketize(torch.rand(m, generator=g, device=dev), edge)
                v = mean[c] + std[c] * v
        out[a:b] = v


def _ks(case, seed):
    """1-based k-th-largest ranks."""
    n, nk, r = case["n"], case["nk"], np.random.default_rng(seed + 1)
    if case["ks"] == "percentiles":
        p = np.arange(nk, dtype=np.float64) / max(nk - 1, 1)
        return (np.round(p * (n - 1)) + 1).astype(np.uint32)
    if case["ks"] == "topk":
        return np.arange(1, nk + 1, dtype=np.uint32)
    if case["ks"] == "top1pct":
        ks = r.integers(1, max(2, n // 100) + 1, nk)
        ks[0], ks[-1] = 1, n
        return ks.astype(np.uint32)
    return r.integers(1, n + 1, nk).astype(np.uint32)


def _lengths(case):
    """Segment lengths (log-uniform over the case's octaves, scaled to its total) and ks per segment."""
    r = np.random.default_rng(case["shape_seed"])
    w = np.exp2(r.uniform(0.0, case["octaves"], case["nseg"]))
    lens = np.maximum(1, (w * (case["n"] / w.sum())).astype(np.int64))
    nks = np.minimum(r.integers(1, case["kmax"] + 1, case["nseg"]), lens)
    return lens, nks


def _inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if case["entry"] != "batch":
        v = torch.empty(case["n"], dtype=TORCH[case["dtype"]], device="cuda")
        _fill(case["dtype"], case["values"], v, g, seed)
        return {"v": v, "ks": _ks(case, seed)}
    lens, nks = _lengths(case)
    off = np.concatenate([[0], np.cumsum(lens)])
    k_off = np.concatenate([[0], np.cumsum(nks)])
    v = torch.empty(int(off[-1]), dtype=TORCH[case["dtype"]], device="cuda")
    if case["values"] == "uniform_normal":  # every other segment uniform, the others normal
        _fill(case["dtype"], "uniform", v, g, seed)
        for s in range(1, case["nseg"], 2) if case["nseg"] <= 4096 else range(1, 4096, 2):
            v[off[s]:off[s + 1]].normal_(generator=g)
    else:
        _fill(case["dtype"], case["values"], v, g, seed)
    r = np.random.default_rng(seed + 1)
    ks = (r.random(int(k_off[-1])) * np.repeat(lens, nks)).astype(np.int64) + 1
    return {"v": v, "off": off, "k_off": k_off, "ks": np.minimum(ks, np.repeat(lens, nks)).astype(np.uint32)}


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case, np=NP[case["dtype"]])
    entry = case["entry"]
    if entry in ("ex", "topk", "batch"):
        s["ctx"] = G.Context(0)
    if entry in ("ex", "batch"):
        s["d_ks"] = torch.from_numpy(s["ks"].astype(np.int32)).cuda()
    if entry == "ex":
        s["opts"] = G.default_opts(ks_on_device=1, out_on_device=1)
    if entry == "batch":
        s["d_off"] = torch.from_numpy(s["off"]).cuda()
        s["d_k_off"] = torch.from_numpy(s["k_off"]).cuda()
    if entry in ("ex", "batch", "noalloc"):
        s["out"] = torch.empty(len(s["ks"]), dtype=s["v"].dtype, device="cuda")
    return s


# ------------------------------------------------------------------ one call
def _ok(rc, what):
    if rc:
        raise G.GGMSError(rc, what)


def run(s):
    case, v = s["case"], s["v"]
    entry = case["entry"]
    if entry in ("bucket", "smos"):
        name = "bucket_multiselect" if entry == "bucket" else "iterative_smos"
        return G.dropin(name, v.data_ptr(), v.numel(), s["ks"], s["np"])
    if entry == "topk":
        return G.topk(s["ctx"], v.data_ptr(), v.numel(), case["nk"], s["np"])
    stream = torch.cuda.current_stream().cuda_stream
    if entry == "ex":
        _ok(G.multiselect_ex(s["ctx"], v.data_ptr(), v.numel(), s["d_ks"].data_ptr(), len(s["ks"]),
                             s["out"].data_ptr(), s["np"], s["opts"], stream), "multiselect_ex")
    elif entry == "batch":
        _ok(G.segmented(s["ctx"], v.data_ptr(), s["d_off"].data_ptr(), case["nseg"], s["d_ks"].data_ptr(),
                        s["d_k_off"].data_ptr(), s["out"].data_ptr(), s["np"], None, stream), "segmented")
    else:
        _ok(G.multiselect_noalloc_f32(v.data_ptr(), v.numel(), s["ks"], s["out"].data_ptr(), stream), "noalloc")
    return s["out"]


def work(case):
    size = SIZE[case["dtype"]]
    if case["entry"] == "batch":
        lens, nks = _lengths(case)
        return {"bytes": int(lens.sum()) * size + int(nks.sum()) * (4 + size) + 16 * (case["nseg"] + 1), "flops": 0}
    return {"bytes": case["n"] * size + case["nk"] * (4 + size), "flops": 0}


# ------------------------------------------------------------------ the same answers in 64 bits
def _wide(case, v):
    if case["dtype"] == "u32":
        return v.to(torch.int64) & 0xFFFFFFFF
    return v.to(torch.int64) if case["dtype"] == "i32" else v.to(torch.float64)


def exact(case, seed):
    s = _inputs(case, seed)
    v = s["v"]
    ks = torch.from_numpy(s["ks"].astype(np.int64)).cuda()
    if case["entry"] != "batch":
        return torch.sort(_wide(case, v)).values[v.numel() - ks]
    off, k_off = s["off"], s["k_off"]
    out = torch.empty(len(s["ks"]), dtype=_wide(case, v[:1]).dtype, device="cuda")
    a = 0
    while a < case["nseg"]:  # groups of segments of up to 2^26 values: by value, then stably by segment
        b = max(a + 1, int(np.searchsorted(off, off[a] + (1 << 26), side="right")) - 1)
        w, order = torch.sort(_wide(case, v[off[a]:off[b]]))
        lens = torch.from_numpy(np.diff(off[a:b + 1])).cuda()
        seg = torch.repeat_interleave(torch.arange(b - a, device="cuda", dtype=torch.int32), lens)[order]
        w = w[torch.sort(seg, stable=True).indices]
        nks = torch.from_numpy(np.diff(k_off[a:b + 1])).cuda()
        end = torch.repeat_interleave(torch.from_numpy(off[a + 1:b + 1] - off[a]).cuda(), nks)
        out[k_off[a]:k_off[b]] = w[end - ks[k_off[a]:k_off[b]]]
        a = b
    return out if case["dtype"] == "f32" else out.to(torch.int32)
