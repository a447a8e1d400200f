"""The workloads this library is timed on: what a user of the jagged hot path has it do.

Every case is one pass through the public entry points on arrays that already
live on the GPU.  A jagged array is (offsets int64 [lists + 1], content), as
awkward's ListOffsetArray stores it; list lengths are Poisson with some forced
empty lists (events with a few particles, sentences with a few words), or
heavy-tailed (a few lists of tens of thousands of elements among many short
ones).  `listed()` names the cases, `draw()` samples the ranges they stand for:
10^3 to 10^7 lists and up to 80 million elements.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import awkward_gb300
from awkward_gb300 import autograd, jagged
from awkward_gb300.batch import Batch

DEV = "cuda"
TORCH = {"float64": torch.float64, "float32": torch.float32, "int64": torch.int64}
NP = {"float64": np.float64, "float32": np.float32, "int64": np.int64}


def listed():
    return [
        # ak.sum / ak.max / ak.argmax(axis=-1) of one small chunk of events: launches and latency
        {"name": "reduce_small", "kind": "reduce", "lists": 1_003, "mean": 8.0, "tail": False,
         "dtype": "float64", "values": "normal"},
        # the same on a whole data set (the benchmark's own shape)
        {"name": "reduce_large", "kind": "reduce", "lists": 10_000_000, "mean": 8.0, "tail": False,
         "dtype": "float64", "values": "normal"},
        # the same on heavy-tailed lists of float32 (documents, graphs by degree)
        {"name": "reduce_tail", "kind": "reduce", "lists": 200_003, "mean": 60.0, "tail": True,
         "dtype": "float32", "values": "positive"},
        # array[array > cut]: a jagged boolean mask that keeps 40 %
        {"name": "select_mask", "kind": "mask", "lists": 4_000_000, "mean": 8.0,
         "dtype": "float64", "keep": 0.4},
        # array[ak.argsort(...)[:, :2]]: a jagged integer index of up to two entries a list
        {"name": "select_index", "kind": "index", "lists": 1_000_000, "mean": 8.0,
         "dtype": "float32", "picks": 2},
        # array[..., 1:] on the inner lists of a two-level array
        {"name": "select_range", "kind": "range", "lists": 1_000_000, "mean": 4.0, "inner": 6.0,
         "dtype": "float64", "start": 1, "stop": None, "step": None},
        # ak.combinations(array, 2): all pairs inside each list
        {"name": "pairs", "kind": "combinations", "lists": 1_000_000, "mean": 6.0, "n": 2,
         "replacement": False},
        # ak.argsort(axis=-1) of many short lists
        {"name": "argsort_short", "kind": "sort", "lists": 2_000_000, "mean": 8.0, "tail": False,
         "dtype": "float64", "arg": True, "ascending": False},
        # ak.sort(axis=-1) of a few long lists
        {"name": "sort_long", "kind": "sort", "lists": 301, "mean": 30_000.0, "tail": False,
         "dtype": "float32", "arg": False, "ascending": True},
        # ak.sum(axis=0): the regrouping above the innermost axis, the carry and the sum
        {"name": "sum_axis0", "kind": "outer", "lists": 2_000_000, "mean": 8.0, "bins": 1,
         "dtype": "float64"},
        # attention pooling of ragged sets, forward and backward: softmax, weighted sum, max
        {"name": "pool_train", "kind": "pool", "lists": 1_000_000, "mean": 16.0, "dtype": "float32"},
        # many arrays at once, replayed from one CUDA graph: sum, max, argmax, count, array[mask]
        {"name": "batch", "kind": "batch", "arrays": 10, "min_lists": 10_000, "max_lists": 300_000,
         "mean": 30.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["reduce", "reduce", "mask", "index", "range", "combinations", "sort", "sort",
                       "outer", "pool", "batch"])
    floating = rng.choice(["float64", "float64", "float32"])
    if kind == "reduce":
        mean = round(math.exp(rng.uniform(math.log(2), math.log(300))), 2)
        return {"kind": kind, "lists": _log_int(rng, 1_000, min(10_000_000, 80_000_000 / mean)),
                "mean": mean, "tail": rng.random() < 0.3,
                "dtype": rng.choice(["float64", "float64", "float32", "int64"]),
                "values": rng.choice(["normal", "normal", "positive", "sparse"])}
    if kind == "mask":
        mean = round(rng.uniform(2, 40), 2)
        return {"kind": kind, "lists": _log_int(rng, 1_000, min(4_000_000, 32_000_000 / mean)),
                "mean": mean, "dtype": floating, "keep": round(rng.uniform(0.05, 0.95), 3)}
    if kind == "index":
        return {"kind": kind, "lists": _log_int(rng, 1_000, 4_000_000),
                "mean": round(rng.uniform(2, 12), 2), "dtype": floating, "picks": rng.randint(1, 5)}
    if kind == "range":
        start, stop, step = rng.choice([(1, None, None), (None, 2, None), (None, -1, None),
                                        (-2, None, None), (None, None, 2), (None, None, -1)])
        return {"kind": kind, "lists": _log_int(rng, 1_000, 1_000_000),
                "mean": round(rng.uniform(2, 4), 2), "inner": round(rng.uniform(2, 8), 2),
                "dtype": floating, "start": start, "stop": stop, "step": step}
    if kind == "combinations":
        n = rng.choice([2, 2, 3])
        return {"kind": kind, "lists": _log_int(rng, 1_000, 1_000_000 if n == 2 else 500_000),
                "mean": round(rng.uniform(2, 8 if n == 2 else 5), 2), "n": n,
                "replacement": rng.random() < 0.25}
    if kind == "sort":
        mean = round(math.exp(rng.uniform(math.log(3), math.log(40_000))), 2)
        return {"kind": kind, "lists": max(3, _log_int(rng, max(3, 20_000 / mean), 16_000_000 / mean)),
                "mean": mean, "tail": mean < 200 and rng.random() < 0.3,
                "dtype": rng.choice(["float64", "float32", "int64"]), "arg": rng.random() < 0.6,
                "ascending": rng.random() < 0.5}
    if kind == "outer":
        rows = _log_int(rng, 1_000, 2_000_000)
        return {"kind": kind, "lists": rows, "mean": round(rng.uniform(2, 10), 2),
                "bins": rng.choice([1, 1, max(1, rows // 100), max(1, rows // 8)]), "dtype": floating}
    if kind == "pool":
        return {"kind": kind, "lists": _log_int(rng, 1_000, 1_000_000),
                "mean": round(rng.uniform(4, 24), 2), "dtype": rng.choice(["float32", "float32", "float64"])}
    lo = _log_int(rng, 200, 10_000)
    return {"kind": kind, "arrays": rng.randint(4, 10), "min_lists": lo, "max_lists": 30 * lo,
            "mean": round(rng.uniform(4, 30), 2)}


# ---------------------------------------------------------------- inputs
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed((seed * 1_000_003 + salt) & 0x7FFFFFFF)


def _lengths(order, n, mean, tail=False, empty=0.01):
    """List lengths: one sample of the distribution, in an order drawn from
    `order` (so that arrays of two seeds differ but hold as many elements)."""
    g = _gen(n, 1)
    if tail:
        # log-normal lengths (sigma 1.5): the longest of 200,000 lists is a thousand times the median
        z = torch.randn(n, generator=g, device=DEV, dtype=torch.float64)
        L = (torch.exp(1.5 * z) * (mean / math.exp(1.125))).floor().to(torch.int64)
        L.clamp_(max=200_000)
    else:
        L = torch.poisson(torch.full((n,), float(mean), device=DEV), generator=g).to(torch.int64)
    L[torch.rand(n, generator=g, device=DEV) < empty] = 0
    return L[torch.randperm(n, generator=order, device=DEV)]


def _mask(g, n, keep):
    m = torch.zeros(n, dtype=torch.bool, device=DEV)
    m[torch.randperm(n, generator=g, device=DEV)[:int(round(keep * n))]] = True
    return m


def _offsets(L):
    off = torch.zeros(L.numel() + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(L, 0, out=off[1:])
    return off


def _content(g, n, dtype, values="normal"):
    if dtype == "int64":
        return torch.randint(-1_000_000, 1_000_000, (n,), generator=g, device=DEV)
    x = torch.randn(n, generator=g, device=DEV, dtype=TORCH[dtype])
    if values == "positive":  # momenta, weights: positive over a few decades
        x = torch.exp(1.2 * x)
    elif values == "sparse":  # thresholded signals: a fifth are exact zeros
        x[torch.rand(n, generator=g, device=DEV) < 0.2] = 0
    return x


def _list_ids(off):
    L = off[1:] - off[:-1]
    return torch.repeat_interleave(torch.arange(L.numel(), device=DEV), L)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "batch":
        arrays = []
        lo, hi = math.log(case["min_lists"]), math.log(case["max_lists"])
        for n in np.exp(np.linspace(lo, hi, case["arrays"])).astype(np.int64):
            off = _offsets(_lengths(g, int(n), case["mean"]))
            x = _content(g, int(off[-1]), "float64")
            arrays.append((off, x, _mask(g, x.numel(), 0.4)))
        st["batch"] = b = Batch(arrays)
        st["plan"] = b.plan()
        st["graph"] = b.graph(st["plan"])
        torch.cuda.synchronize()
        kept = [int(m.sum()) for _o, _x, m in arrays]
        st["out"] = [(b.out_sum[i], b.out_max[i], b.out_argmax[i], b.out_count[i],
                      b.sel_offsets[i], b.sel_content[i][:k]) for i, k in enumerate(kept)]
        return st
    n = case["lists"]
    if kind == "outer":
        bins = case["bins"]
        # rows of each outer list: an even split with jitter (one bin takes all of them)
        cuts = torch.sort(torch.randint(0, n + 1, (bins - 1,), generator=g, device=DEV))[0]
        st["outer"] = torch.cat([cuts.new_zeros(1), cuts, cuts.new_full((1,), n)])
    L = _lengths(g, n, case["mean"], case.get("tail", False))
    off = _offsets(L)
    if kind == "range":
        st["outer"] = off
        off = _offsets(_lengths(g, int(off[-1]), case["inner"]))
        st.update(start=case["start"], stop=case["stop"], step=case["step"])
    st["off"], E = off, int(off[-1])
    if kind == "combinations":
        st.update(n=case["n"], replacement=case["replacement"])
        return st
    st["x"] = x = _content(g, E, case["dtype"], case.get("values", "normal"))
    st["dtype"] = case["dtype"]
    if kind == "reduce":
        dt = x.dtype
        st["out"] = {"sum": torch.empty(n, dtype=dt, device=DEV),
                     "max": torch.empty(n, dtype=dt, device=DEV),
                     "argmax": torch.empty(n, dtype=torch.int64, device=DEV)}
    elif kind == "mask":
        st["mask"] = _mask(g, E, case["keep"])
    elif kind == "index":
        K = torch.clamp(L, max=case["picks"])
        st["ioff"] = _offsets(K)
        ids = _list_ids(st["ioff"])
        # any position of the list, a third of them counted from its end
        u = torch.rand(ids.numel(), generator=g, device=DEV, dtype=torch.float64)
        pos = torch.minimum((u * L[ids]).to(torch.int64), L[ids] - 1)
        back = torch.rand(ids.numel(), generator=g, device=DEV) < 1 / 3
        st["idx"] = torch.where(back, pos - L[ids], pos)
    elif kind == "sort":
        st.update(arg=case["arg"], ascending=case["ascending"])
        st["out"] = torch.empty(E, dtype=torch.int64 if case["arg"] else x.dtype, device=DEV)
    elif kind == "pool":
        st["score"] = _content(g, E, case["dtype"]).requires_grad_()
        st["x"] = x.requires_grad_()
        st["grads"] = (_content(g, n, case["dtype"]), _content(g, n, case["dtype"]))
        st["filled"] = L > 0
    return st


# ---------------------------------------------------------------- one pass
def run(st):
    return _RUN[st["kind"]](st)


def _run_reduce(st):
    be = awkward_gb300.backend()
    off, x, out = st["off"], st["x"], st["out"]
    n, dt = off.numel() - 1, NP[st["dtype"]]
    lowest = -np.inf if st["dtype"] != "int64" else np.iinfo(np.int64).min
    be["awkward_reduce_sum", dt, dt, np.int64](out["sum"], x, off, n)
    be["awkward_reduce_max", dt, dt, np.int64](out["max"], x, off, n, lowest)
    be["awkward_reduce_argmax", np.int64, dt, np.int64, np.int64](out["argmax"], x, off, off[:-1], n)
    return out


def _run_mask(st):
    return jagged.mask_select(st["off"], st["x"], st["mask"])


def _run_index(st):
    return jagged.index_select(st["off"], st["x"], st["ioff"], st["idx"])


def _run_range(st):
    return jagged.getitem_inner_range(st["outer"], st["off"], st["x"], st["start"], st["stop"],
                                      st["step"])


def _run_combinations(st):
    be = awkward_gb300.backend()
    off, n, rep = st["off"], st["n"], st["replacement"]
    N, i8 = off.numel() - 1, np.int64
    total = torch.empty(1, dtype=torch.int64, device=DEV)
    offsets = torch.empty(N + 1, dtype=torch.int64, device=DEV)
    starts, stops = off[:-1], off[1:]
    be["awkward_ListArray_combinations_length", i8, i8, i8, i8](total, offsets, n, rep, starts, stops, N)
    be.synchronize()
    tuples = int(total.item())
    rows = [torch.empty(tuples, dtype=torch.int64, device=DEV) for _ in range(n)]
    toindex = torch.empty(n, dtype=torch.int64, device=DEV)
    fromindex = torch.zeros(n, dtype=torch.int64, device=DEV)
    be["awkward_ListArray_combinations", i8, i8, i8, i8, i8](rows, toindex, fromindex, n, rep, starts,
                                                           stops, N)
    be.synchronize()
    return {"offsets": offsets, "rows": rows, "toindex": toindex}


def _run_sort(st):
    be = awkward_gb300.backend()
    off, x, dt = st["off"], st["x"], NP[st["dtype"]]
    if st["arg"]:
        be["awkward_argsort", np.int64, dt, np.int64](st["out"], x, x.numel(), off, off.numel(),
                                                      st["ascending"], True)
    else:
        be["awkward_sort", dt, dt, np.int64](st["out"], x, x.numel(), off, off.numel(),
                                             st["ascending"], True)
    return st["out"]


def _run_outer(st):
    be = awkward_gb300.backend()
    off, outer, x, dt = st["off"], st["outer"], st["x"], NP[st["dtype"]]
    rows, bins, E = off.numel() - 1, outer.numel() - 1, x.numel()

    def ints(k):
        return torch.empty(k, dtype=torch.int64, device=DEV)

    maxcount, copy = ints(1), ints(rows + 1)
    be.by_name("awkward_ListOffsetArray_reduce_nonlocal_maxcount_offsetscopy_64")(maxcount, copy, off, rows)
    be.synchronize()
    M = int(maxcount.item())
    nb = bins * M
    carry, nextoffsets, last, distincts = ints(E), ints(nb + 1), ints(1), ints(nb)
    be.by_name("awkward_ListOffsetArray_reduce_nonlocal_preparenext_64")(
        carry, nextoffsets, E, last, distincts, nb, copy, off, rows, outer, bins, M)
    be.synchronize()
    out = torch.empty(nb, dtype=x.dtype, device=DEV)
    be["awkward_reduce_sum", dt, dt, np.int64](out, jagged.take(x, carry), nextoffsets, nb)
    starts, stops = ints(bins), ints(bins)
    be.by_name("awkward_ListOffsetArray_reduce_nonlocal_outstartsstops_64")(starts, stops, distincts, nb, bins)
    be.synchronize()
    return {"sum": out, "carry": carry, "offsets": nextoffsets, "last": last, "distincts": distincts,
            "starts": starts, "stops": stops}


def _run_pool(st):
    off, score, x = st["off"], st["score"], st["x"]
    w = autograd.jagged_softmax(score, off)
    mean = autograd.segment_sum(w * x, off)
    peak = autograd.segment_max(x, off)
    gs, gx = torch.autograd.grad((mean, peak), (score, x), st["grads"])
    return {"weights": w.detach(), "mean": mean.detach(), "peak": peak.detach(), "grad_score": gs,
            "grad_x": gx}


def _run_batch(st):
    st["graph"].replay()
    return st["out"]


_RUN = {"reduce": _run_reduce, "mask": _run_mask, "index": _run_index, "range": _run_range,
        "combinations": _run_combinations, "sort": _run_sort, "outer": _run_outer, "pool": _run_pool,
        "batch": _run_batch}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "batch":
        lo, hi = math.log(case["min_lists"]), math.log(case["max_lists"])
        n = case["arrays"] * (case["max_lists"] - case["min_lists"]) / (hi - lo)
        e = n * case["mean"]
        # offsets, content and mask in; four results a list, new offsets and 40 % of the content out
        return {"bytes": int(8 * n + 9 * e + 40 * n + 3.2 * e), "flops": int(3 * e)}
    n, e = case["lists"], case["lists"] * case["mean"]
    s = 4 if case.get("dtype") == "float32" else 8
    if kind == "reduce":  # content and offsets in, three results a list out
        return {"bytes": int(s * e + 8 * n + (2 * s + 8) * n), "flops": int(3 * e)}
    if kind == "mask":
        return {"bytes": int((s + 1) * e + 16 * n + case["keep"] * s * e), "flops": 0}
    if kind == "index":  # the gathered elements, both offsets and the index in; offsets and elements out
        k = n * min(case["picks"], case["mean"])
        return {"bytes": int(24 * n + 8 * k + 2 * s * k), "flops": 0}
    if kind == "range":
        inner = e
        elements = inner * case["inner"]
        if case["step"] is not None:
            kept = elements / abs(case["step"])
        elif case["start"] == 1 or case["stop"] == -1:
            kept = elements - inner
        else:
            kept = min(2.0, case["inner"]) * inner
        return {"bytes": int(16 * inner + 2 * s * kept), "flops": 0}
    if kind == "combinations":  # for Poisson lengths E[L(L-1)...] = mean^n
        k, m = case["n"], case["mean"]
        per = m**k / math.factorial(k)
        if case["replacement"]:
            per = m + m * m / 2 if k == 2 else m + m * m + m**3 / 6
        return {"bytes": int(8 * n + 8 * n + 8 * k * per * n), "flops": 0}
    if kind == "sort":
        return {"bytes": int(s * e + 8 * n + (8 if case["arg"] else s) * e), "flops": 0}
    if kind == "outer":  # content and offsets in; offsets copy and carry out (sums are few)
        return {"bytes": int(s * e + 16 * n + 8 * e + 24 * case["bins"] * 2 * case["mean"]), "flops": int(e)}
    # pool: scores, values and offsets in, weights and both gradients out, 4 values a list
    return {"bytes": int(5 * s * e + 8 * n + 4 * s * n), "flops": int(20 * e)}


# ---------------------------------------------------------------- the values in 64 bits
def _segment_sums(x, off):
    """Sums by list, exact to 2^-60 per element: each value split into two
    integers whose (wrapping) running sums are differenced."""
    if not x.is_floating_point():
        c = torch.cat([x.new_zeros(1), torch.cumsum(x, 0)])
        return c[off[1:]] - c[off[:-1]]
    x = x.to(torch.float64)
    out = None
    for bits in (20, 60):
        k = torch.round(x * 2.0**bits)
        x = x - k * 2.0**-bits
        c = torch.cat([off.new_zeros(1), torch.cumsum(k.to(torch.int64), 0)])
        part = (c[off[1:]] - c[off[:-1]]).to(torch.float64) * 2.0**-bits
        out = part if out is None else out + part
    return out


def _segment_max(x, off):
    out = torch.full((off.numel() - 1,), -math.inf, dtype=torch.float64, device=DEV)
    return out.scatter_reduce_(0, _list_ids(off), x.to(torch.float64), "amax")


def exact(case, seed):
    st = prepare(case, seed)
    kind = case["kind"]
    if kind == "combinations":
        return None
    if kind == "batch":
        return [(_segment_sums(x, o), _segment_max(x, o), None, None, None, x[m])
                for o, x, m in st["batch"].arrays]
    off, x = st["off"], st["x"]
    if kind == "reduce":
        if case["dtype"] == "int64":
            return None
        return {"sum": _segment_sums(x, off), "max": _segment_max(x, off), "argmax": None}
    if kind == "mask":
        return None, x[st["mask"]].to(torch.float64)
    if kind == "index":
        ids = _list_ids(st["ioff"])
        at = off[ids] + torch.where(st["idx"] < 0, st["idx"] + (off[ids + 1] - off[ids]), st["idx"])
        return None, x[at].to(torch.float64)
    if kind == "range":
        ids = _list_ids(off)
        pos = torch.arange(x.numel(), device=DEV) - off[ids]
        L = (off[1:] - off[:-1])[ids]
        start, stop, step = case["start"], case["stop"], case["step"]
        if step == -1:
            return None, None, x[off[ids + 1] - 1 - pos].to(torch.float64)
        a = 0 if start is None else (L + start).clamp(min=0) if start < 0 else start
        b = L if stop is None else L + stop if stop < 0 else stop
        keep = (pos >= a) & (pos < b) & (pos % (1 if step is None else step) == 0)
        return None, None, x[keep].to(torch.float64)
    if kind == "sort":
        if case["arg"] or case["dtype"] == "int64":
            return None
        ids = _list_ids(off)
        v, order = torch.sort(x.to(torch.float64), descending=not case["ascending"], stable=True)
        return v[torch.sort(ids[order], stable=True)[1]]
    if kind == "outer":
        got = {"sum": None, "carry": None, "offsets": None, "last": None, "distincts": None,
               "starts": None, "stops": None}
        ids = _list_ids(off)
        row_bin = torch.searchsorted(st["outer"], torch.arange(off.numel() - 1, device=DEV), right=True) - 1
        M = int((off[1:] - off[:-1]).max())
        key = row_bin[ids] * M + torch.arange(x.numel(), device=DEV) - off[ids]
        skey, order = torch.sort(key, stable=True)
        noff = torch.searchsorted(skey, torch.arange(case["bins"] * M + 1, device=DEV))
        got["sum"] = _segment_sums(x[order], noff)
        return got
    # pool
    score, v = st["score"].detach().to(torch.float64), x.detach().to(torch.float64)
    gm, gp = (t.to(torch.float64) for t in st["grads"])
    ids, n = _list_ids(off), off.numel() - 1

    def total(t):
        return torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, ids, t)

    e = torch.exp(score - _segment_max(score, off)[ids])
    w = e / total(e)[ids]
    mean, peak = total(w * v), _segment_max(v, off)
    at = torch.arange(v.numel(), device=DEV)
    first = torch.full((n,), v.numel(), device=DEV).scatter_reduce_(
        0, ids, torch.where(v == peak[ids], at, v.numel()), "amin")
    grad_x = w * gm[ids]
    grad_x[first[st["filled"]]] += gp[st["filled"]]
    return {"weights": w, "mean": mean, "peak": peak, "grad_score": w * (v - mean[ids]) * gm[ids],
            "grad_x": grad_x}
