"""The searches that users of this framework run, as cases to be timed.

Twelve cases over the public entry points, in four families:

* the exact linear index (`LinearIndex.search`, mode "exact") -- one query at a time, a small ragged
  inner-product batch, and a large batch;
* its tensor-core form (`LinearIndex.search_tc`) -- the 1M x 384 batch, a serving-size inner-product
  batch at dim 768, and the scaled-FP8 form at 4M x 256;
* the IVF index (`IVFIndex.search`) -- the BF16 tensor-core form at the benchmark's batch and one query
  at a time, the SQ8-code tensor-core form from host buffers, and the exact SQ8 selection;
* what surrounds a search: the IVF build (`IVFIndex.fit`) and the competition plugin's one query per call
  (`Algorithm.query`).

Data: L2-normalised Gaussian mixtures (list sizes by a clipped Zipf law for the IVF cases), or normalised
Gaussian rows, drawn on the device from the seed; queries from the same distribution.
"""
from __future__ import annotations

import math

import numpy as np
import torch

DEV = "cuda:0"


# ---- cases -------------------------------------------------------------------------------------------

def listed():
    return [
        # one query against a resident 1M x 384 base: the interactive lookup, bound by reading the base
        {"name": "flat_exact_1q", "kind": "flat", "data": "mixture", "metric": "l2", "n": 1_000_000, "dim": 384,
         "c": 2048, "sigma": 0.3, "nq": 1, "k": 100},
        # a small ragged inner-product batch: odd row count, a dim that is no multiple of 32, k = 10
        {"name": "flat_exact_ragged_ip", "kind": "flat", "data": "normal", "metric": "ip", "n": 50_021, "dim": 100,
         "c": 1, "sigma": 1.0, "nq": 9, "k": 10},
        # the exact ground truth of a query set: 1,000 queries over 1M x 384
        {"name": "flat_exact_batch", "kind": "flat", "data": "mixture", "metric": "l2", "n": 1_000_000, "dim": 384,
         "c": 2048, "sigma": 0.3, "nq": 1000, "k": 100},
        # tensor-core exact search, the benchmark's 10k batch (R = 400)
        {"name": "flat_tc_batch", "kind": "flat_tc", "data": "mixture", "metric": "l2", "precision": "bf16",
         "n": 1_000_000, "dim": 384, "c": 2048, "sigma": 0.3, "nq": 10_000, "k": 100, "refine": 400},
        # the server's exact inner-product route: one gathered batch of requests over 1M x 768
        {"name": "flat_tc_ip_serving", "kind": "flat_tc", "data": "mixture", "metric": "ip", "precision": "bf16",
         "n": 1_000_000, "dim": 768, "c": 1024, "sigma": 0.35, "nq": 77, "k": 100, "refine": 400},
        # the scaled-FP8 form at 4M x 256 with norms spread over 0.5-2 (R = 500)
        {"name": "flat_fp8_batch", "kind": "flat_tc", "data": "scaled", "metric": "l2", "precision": "e4m3",
         "n": 4_000_000, "dim": 256, "c": 4096, "sigma": 0.4, "nq": 5000, "k": 100, "refine": 500},
        # the benchmark's headline: IVF on the tensor cores, BF16 keys, 10k queries at the tuned point
        {"name": "ivf_tc_batch", "kind": "ivf", "mode": "tc", "host": False, "n": 1_000_000, "dim": 384, "c": 2048,
         "sigma": 0.3, "nq": 10_000, "k": 100, "nprobe": 2, "refine": 100, "sample_div": 16},
        # the same index, one query per call: serving latency
        {"name": "ivf_tc_1q", "kind": "ivf", "mode": "tc", "host": False, "n": 1_000_000, "dim": 384, "c": 2048,
         "sigma": 0.3, "nq": 1, "k": 100, "nprobe": 4, "refine": 150, "sample_div": 8},
        # SQ8 codes on the tensor cores, a ragged batch from host buffers to host arrays (end to end)
        {"name": "ivf_sq8_tc_host", "kind": "ivf", "mode": "tc_sq8", "host": True, "n": 1_000_000, "dim": 384,
         "c": 2048, "sigma": 0.3, "nq": 3001, "k": 100, "nprobe": 2, "refine": 150, "sample_div": 8},
        # exact SQ8 selection, the plugin backend gpu_ivf_sq8's search at its default probe count and 4k re-rank
        {"name": "ivf_exact_batch", "kind": "ivf", "mode": "exact", "host": False, "n": 1_000_000, "dim": 384,
         "c": 2048, "sigma": 0.3, "nq": 2000, "k": 100, "nprobe": 8, "refine": -1, "sample_div": 8},
        # building an IVF index: 15 k-means rounds, the lists and the SQ8 codes, then its state read out
        {"name": "ivf_fit", "kind": "fit", "n": 50_000, "dim": 384, "c": 256, "sigma": 0.3, "iters": 15},
        # the competition harness's pattern: one host query per call through the plugin's default backend
        {"name": "plugin_linear_1q", "kind": "plugin", "data": "normal", "n": 100_000, "dim": 384, "k": 100},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed families, sizes spread over their ranges."""
    kind = rng.choice(["flat", "flat", "flat", "flat_tc", "flat_tc", "flat_fp8", "ivf", "ivf", "ivf", "ivf", "fit",
                       "plugin"])
    if kind == "flat":
        n, dim, nq = _log_int(rng, 20_000, 1_000_000), _log_int(rng, 64, 768), _log_int(rng, 1, 1000)
        if n * dim * nq > 3.8e11:
            nq = max(1, int(3.8e11 // (n * dim)))
        data = rng.choice(["mixture", "normal"])
        return {"kind": "flat", "data": data, "metric": rng.choice(["l2", "l2", "ip"]), "n": n, "dim": dim,
                "c": min(2048, max(1, n // 400)), "sigma": 0.3, "nq": nq, "k": rng.choice([1, 10, 50, 100, 100])}
    if kind == "flat_tc":
        n, dim, nq = _log_int(rng, 50_000, 1_000_000), _log_int(rng, 64, 768), _log_int(rng, 1, 10_000)
        if n * dim * nq > 3.8e12:
            nq = max(1, int(3.8e12 // (n * dim)))
        k = rng.choice([10, 100])
        return {"kind": "flat_tc", "data": "mixture", "metric": rng.choice(["l2", "ip"]), "precision": "bf16", "n": n,
                "dim": dim, "c": min(2048, max(1, n // 400)), "sigma": rng.choice([0.3, 0.35]), "nq": nq, "k": k,
                "refine": 4 * k}
    if kind == "flat_fp8":
        n, nq = _log_int(rng, 500_000, 4_000_000), _log_int(rng, 64, 5000)
        return {"kind": "flat_tc", "data": "scaled", "metric": "l2", "precision": "e4m3", "n": n,
                "dim": rng.choice([128, 200, 256]), "c": min(4096, n // 400), "sigma": 0.4, "nq": nq, "k": 100,
                "refine": 500}
    if kind == "ivf":
        n, dim = _log_int(rng, 100_000, 1_000_000), _log_int(rng, 96, 400)
        mode = rng.choice(["tc", "tc", "tc_sq8", "exact"])
        nq = _log_int(rng, 1, 10_000 if mode != "exact" else 2000)
        return {"kind": "ivf", "mode": mode, "host": rng.random() < 0.3, "n": n, "dim": dim,
                "c": min(2048, max(64, n // 500)), "sigma": 0.3, "nq": nq, "k": rng.choice([10, 100]),
                "nprobe": rng.choice([2, 3, 4, 8]), "refine": rng.choice([100, 150, 200]),
                "sample_div": rng.choice([4, 8, 16])}
    if kind == "fit":
        return {"kind": "fit", "n": _log_int(rng, 10_000, 50_000), "dim": _log_int(rng, 64, 384),
                "c": _log_int(rng, 16, 256), "sigma": 0.3, "iters": 15}
    return {"kind": "plugin", "data": "normal", "n": _log_int(rng, 10_000, 100_000), "dim": _log_int(rng, 64, 384),
            "k": rng.choice([10, 100])}


# ---- data ----------------------------------------------------------------------------------------------

def _zipf_sizes(n, c, s=1.1, lo=20):
    """List sizes clip(round(C0 r^-s), lo, n / 25), C0 chosen so that they sum to n."""
    hi = max(lo, n // 25)
    r = np.arange(1, c + 1, dtype=np.float64) ** -s
    a, b = 0.0, 4.0 * n
    for _ in range(100):
        m = 0.5 * (a + b)
        a, b = (m, b) if np.clip(np.round(m * r), lo, hi).sum() < n else (a, m)
    sizes = np.clip(np.round(b * r), lo, hi).astype(np.int64)
    i, diff = c - 1, n - int(sizes.sum())
    while diff and i >= 0:
        step = int(max(lo - sizes[i], min(hi - sizes[i], diff)))
        sizes[i] += step
        diff -= step
        i -= 1
    sizes[0] += diff
    return sizes


def _data(kind, n, dim, nq, c, sigma, seed):
    """(base, queries, centres, list of each row) on the device; kind: normal, mixture, scaled or zipf."""
    g = torch.Generator(device=DEV).manual_seed(1_000_003 * (seed + 1))
    norm = torch.nn.functional.normalize
    if kind == "normal":
        base = norm(torch.randn(n, dim, generator=g, device=DEV), dim=1)
        return base, norm(torch.randn(nq, dim, generator=g, device=DEV), dim=1), None, None
    centres = torch.randn(c, dim, generator=g, device=DEV)
    if kind == "zipf":
        sizes = torch.from_numpy(_zipf_sizes(n, c)).to(DEV)
        assign = torch.repeat_interleave(torch.arange(c, device=DEV), sizes)
        assign = assign[torch.randperm(n, generator=g, device=DEV)]
        qc = torch.multinomial(sizes.double() / n, nq, replacement=True, generator=g)
    else:
        assign = torch.randint(0, c, (n,), generator=g, device=DEV)
        qc = torch.randint(0, c, (nq,), generator=g, device=DEV)
    base = torch.empty(n, dim, device=DEV)
    for s in range(0, n, 1 << 19):
        e = min(n, s + (1 << 19))
        base[s:e] = norm(centres[assign[s:e]] + sigma * torch.randn(e - s, dim, generator=g, device=DEV), dim=1)
    queries = norm(centres[qc] + sigma * torch.randn(nq, dim, generator=g, device=DEV), dim=1)
    if kind == "scaled":
        base.mul_(torch.rand(n, 1, generator=g, device=DEV) * 1.5 + 0.5)
        queries.mul_(torch.rand(nq, 1, generator=g, device=DEV) * 1.5 + 0.5)
    return base, queries, norm(centres, dim=1), assign


def _inputs(case, seed):
    kind = case["kind"]
    if kind in ("ivf", "fit"):
        return _data("zipf", case["n"], case["dim"], case.get("nq", 1), case["c"], case["sigma"], seed)
    return _data(case["data"], case["n"], case["dim"], case.get("nq", 1), case.get("c", 1), case.get("sigma", 1.0),
                 seed)


# ---- prepare and run -------------------------------------------------------------------------------------

def prepare(case, seed):
    base, queries, centres, assign = _inputs(case, seed)
    kind = case["kind"]
    st = {"case": case, "queries": queries}
    if kind in ("flat", "flat_tc"):
        from annvedi_b200.linear import LinearIndex
        ix = LinearIndex(device=0, metric=case["metric"], mode="exact")
        ix.fit(base)
        if kind == "flat_tc":
            ix.set_tc_precision(case["precision"])
            ix.search_tc(queries[:1], case["k"], refine_r=case["refine"])  # lays out the operand copy once
        st["index"] = ix
    elif kind == "ivf":
        from annvedi_b200.ivf import IVFIndex
        ix = IVFIndex(device=0, mode="exact", num_threads=16)
        ix.fit(base, 1, 0, case["c"], centroids=centres, assign=assign.int())
        ix.set_option("sample_div", case["sample_div"])
        if case["mode"] != "exact":
            ix.search(queries[:1], case["k"], 0, case["nprobe"], case["refine"], mode=case["mode"])
        st["index"] = ix
        if case["host"]:
            st["queries"] = queries.cpu().pin_memory()
            st["ids"] = torch.empty(case["nq"], case["k"], dtype=torch.int64, pin_memory=True)
            st["dists"] = torch.empty(case["nq"], case["k"], dtype=torch.float32, pin_memory=True)
    elif kind == "fit":
        st["base"] = base
    else:
        from annvedi_b200.algorithm import Algorithm
        algo = Algorithm()
        algo.fit(base, backend="linear")
        st["index"] = algo
        st["queries"] = queries.cpu().numpy()
    torch.cuda.synchronize()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "flat":
        return st["index"].search(st["queries"], case["k"], mode="exact")
    if kind == "flat_tc":
        return st["index"].search_tc(st["queries"], case["k"], refine_r=case["refine"])
    if kind == "ivf":
        out = {"out_ids": st["ids"], "out_dists": st["dists"]} if case["host"] else {}
        return st["index"].search(st["queries"], case["k"], 0, case["nprobe"], case["refine"], mode=case["mode"], **out)
    if kind == "fit":
        from annvedi_b200.ivf import IVFIndex
        ix = IVFIndex(device=0, mode="exact", num_threads=16)
        ix.fit(st["base"], 1, 0, case["c"], kmeans_iters=case["iters"])
        s = ix.export_state()
        return [s[key] for key in ("centroids", "original_data", "quantized_data", "scale", "offset",
                                   "reordered_to_original", "table_offsets")]
    return st["index"].query(st["queries"][0], case["k"])


# ---- what a pass cannot do without ------------------------------------------------------------------------

def work(case):
    n, dim, kind = case["n"], case["dim"], case["kind"]
    if kind == "fit":  # rows read, codes and reordered rows written; every round's assignment
        return {"bytes": n * dim * 9 + 4 * n, "flops": 2 * n * dim * case["c"] * (case["iters"] + 1)}
    if kind == "plugin":
        return {"bytes": 4 * n * dim + 4 * dim + 8 * case["k"], "flops": 2 * n * dim}
    nq = case["nq"]
    io = nq * (4 * dim + 12 * case["k"])
    if kind in ("flat", "flat_tc"):
        size = 4 if kind == "flat" else (2 if case["precision"] == "bf16" else 1)
        return {"bytes": size * n * dim + io, "flops": 2 * n * dim * nq}
    # IVF: each query's first list is met in proportion to its size, the other probes are any lists; the rows of
    # the lists that the batch probes are read once, at a code or a BF16 value an element
    sizes = _zipf_sizes(n, case["c"]).astype(np.float64)
    p = sizes / n
    cands = nq * (float((sizes * p).sum()) + (case["nprobe"] - 1) * n / case["c"])
    miss = np.exp(nq * np.log1p(-np.minimum(p, 0.999)) + nq * (case["nprobe"] - 1) * math.log1p(-1.0 / case["c"]))
    rows = float((sizes * (1.0 - miss)).sum())
    size = 2 if case["mode"] == "tc" else 1
    return {"bytes": int(size * rows * dim + 4 * case["c"] * dim + io),
            "flops": int(2 * dim * (cands + nq * case["c"]))}


# ---- the values in 64 bits ----------------------------------------------------------------------------------

def _exact_flat(case, seed):
    base, q, _, _ = _inputs(case, seed)
    k, ip = case["k"], case["metric"] == "ip"
    best = None
    step = max(1, int(6e8 // case["nq"]))
    for s in range(0, case["n"], step):
        x = base[s:s + step].double()
        dots = q.double() @ x.T
        key = -dots if ip else (x * x).sum(1)[None, :] - 2.0 * dots
        top = torch.topk(key, min(k, key.shape[1]), largest=False, sorted=False)
        cur = (top.values, top.indices + s)
        if best is not None:
            v = torch.cat([best[0], cur[0]], 1)
            i = torch.cat([best[1], cur[1]], 1)
            t = torch.topk(v, min(k, v.shape[1]), largest=False, sorted=False)
            cur = (t.values, torch.gather(i, 1, t.indices))
        best = cur
    out = torch.empty(case["nq"], best[1].shape[1], dtype=torch.float64, device=DEV)
    for s in range(0, case["nq"], 1000):  # the distances of the best rows, by differences
        x, y = base[best[1][s:s + 1000]].double(), q[s:s + 1000].double()[:, None, :]
        out[s:s + 1000] = (x * y).sum(-1) if ip else ((x - y) ** 2).sum(-1)
    return None, torch.sort(out, 1, descending=ip).values


def _exact_ivf(case, seed):
    """The search's definition in 64 bits: lists by centroid distance, the best R rows by the mode's key over
    the probed lists (every row for a query whose lists hold fewer than k), re-ranked by their squared
    distances."""
    base, q, cen, assign = _inputs(case, seed)
    nq, k, C = case["nq"], case["k"], case["c"]
    R = max(k, case["refine"] if case["refine"] > 0 else 4 * k)
    npc = min(case["nprobe"], C)
    order = torch.argsort(assign, stable=True)
    off = torch.cat([torch.zeros(1, dtype=torch.int64, device=DEV), torch.cumsum(torch.bincount(assign, minlength=C), 0)])
    cd = (cen.double() ** 2).sum(1)[None, :] - 2.0 * q.double() @ cen.double().T
    probes = torch.topk(cd, npc, largest=False).indices
    lo, hi = base.min(0).values, base.max(0).values  # per-dimension SQ8
    scale = (hi - lo) * torch.tensor(1.0 / 255.0, dtype=torch.float32, device=DEV)

    def decoded(x):
        return torch.round((x - lo) / scale).clamp_(0, 255).double() * scale.double()
    sizes = (off[1:] - off[:-1]).cpu().numpy()
    offh, ph = off.cpu().numpy(), probes.cpu().numpy()
    keys = torch.full((nq, npc * R), math.inf, dtype=torch.float64, device=DEV)
    rows = torch.zeros((nq, npc * R), dtype=torch.int64, device=DEV)
    flat = np.argsort(ph.reshape(-1), kind="stable")
    lists, starts = np.unique(ph.reshape(-1)[flat], return_index=True)
    ends = np.append(starts[1:], len(flat))
    for l, s, e in zip(lists, starts, ends):
        if sizes[l] == 0:
            continue
        pairs = torch.from_numpy(flat[s:e]).to(DEV)
        qi, slot = pairs // npc, pairs % npc
        r = order[int(offh[l]):int(offh[l + 1])]
        if case["mode"] == "tc":
            x = base[r]
            key = (x.double() ** 2).sum(1)[None, :] - 2.0 * q[qi].bfloat16().double() @ x.bfloat16().double().T
        else:
            code = decoded(base[r])
            w = q[qi].double() - lo.double()
            if case["mode"] == "tc_sq8":
                w = -2.0 * scale.double() * w
                a = 127.0 / w.abs().amax(1, keepdim=True)
                key = (code ** 2).sum(1)[None, :] + (torch.round(w * a) / a) @ (code / scale.double()).T
            else:
                key = (code ** 2).sum(1)[None, :] - 2.0 * w @ code.T
            if case["mode"] == "exact":
                key = key + (w ** 2).sum(1, keepdim=True)
        m = min(R, r.shape[0])
        t = torch.topk(key, m, largest=False, sorted=False)
        at = (slot * R)[:, None] + torch.arange(m, device=DEV)[None, :]
        keys[qi[:, None], at] = t.values
        rows[qi[:, None], at] = r[t.indices]
    top = torch.topk(keys, min(R, keys.shape[1]), largest=False)
    cand = torch.gather(rows, 1, top.indices)
    for i in torch.nonzero(torch.isinf(top.values[:, k - 1])).flatten().tolist():  # short of k: every row, by SQ8
        w = q[i].double() - lo.double()
        key = torch.cat([((decoded(base[s:s + 200_000]) - w) ** 2).sum(1) for s in range(0, case["n"], 200_000)])
        t = torch.topk(key, cand.shape[1], largest=False)
        top.values[i], cand[i] = t.values, t.indices
    out = torch.empty(nq, k, dtype=torch.float64, device=DEV)
    for s in range(0, nq, 500):
        d = ((base[cand[s:s + 500]].double() - q[s:s + 500].double()[:, None, :]) ** 2).sum(-1)
        d = torch.where(torch.isfinite(top.values[s:s + 500]), d, torch.full_like(d, math.inf))
        out[s:s + 500] = torch.sort(d, 1).values[:, :k]
    return None, out.cpu() if case["host"] else out


def exact(case, seed):
    if case["kind"] in ("flat", "flat_tc"):
        return _exact_flat(case, seed)
    if case["kind"] == "ivf":
        return _exact_ivf(case, seed)
    return None  # ids alone, or a k-means state whose later rounds follow its own roundings
