"""The calls that programs built on this framework make, at the sizes they make them.

Each case is one call (or, for the serving loop, one batch of requests) through
the public entry points on inputs that are resident on the GPU.  Sizes come
from the benchmark's configurations and the tests; ``draw`` spreads the same
calls over the whole range between the smallest and the largest.

Outputs are exact for integer scans, compaction, sorting and selection.  Sums
of floating values are FP32 results of FP32 (or better) accumulation.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pytorch-tcuscan_b200"))

import tcuscan_ops  # noqa: E402
from tcuscan_b200 import batch, serve, workloads  # noqa: E402

DTYPES = {"int8": torch.int8, "int16": torch.int16, "float16": torch.float16, "float32": torch.float32,
          "int32": torch.int32}
BYTES = {"int8": 1, "int16": 2, "float16": 2, "float32": 4, "int32": 4}


def listed():
    return [
        # a prefix sum of a short vector (offsets of a batch, a histogram): latency is all there is
        {"name": "scan_f16_short", "kind": "scan", "dtype": "float16", "n": 1021, "S": 64},
        # the ordinary single call: 2^20 fp16 values
        {"name": "scan_f16_1m", "kind": "scan", "dtype": "float16", "n": 1 << 20, "S": 64},
        # the headline scan: 2^28 int8 values to int32
        {"name": "scan_i8_2e28", "kind": "scan", "dtype": "int8", "n": 1 << 28, "S": 0},
        # thousands of uneven fp32 rows scanned in one launch
        {"name": "rows_f32_4096", "kind": "rows", "dtype": "float32", "rows": 4096, "lo": 256, "hi": 1 << 20},
        # a segmented scan by start flags at a ragged length
        {"name": "seg_scan_f16_flags", "kind": "seg_scan", "dtype": "float16", "n": (1 << 26) + 4321, "p": 0.01},
        # per-segment sums over row pointers, segments of 64 elements on average
        {"name": "seg_sum_f16_mean64", "kind": "seg_sum", "dtype": "float16", "n": 1 << 28, "mean": 64,
         "wide": True},
        # y = A x for a square CSR matrix with Zipf row lengths
        {"name": "spmv_f32_zipf", "kind": "spmv", "dtype": "float32", "rows": 1 << 20, "nnz": 1 << 24},
        # stream compaction of 2^28 fp16 values, 30 % kept
        {"name": "compress_f16_2e28", "kind": "compact", "op": "compress", "dtype": "float16", "n": 1 << 28, "p": 0.3},
        # values and positions of the kept elements, an ordinary ragged length
        {"name": "compress_ind_f32_10m", "kind": "compact", "op": "positions", "dtype": "float32", "n": 10_000_019,
         "p": 0.3},
        # the largest sort of the reference's tests: values and positions
        {"name": "sort_f16_25m", "kind": "sort", "dtype": "float16", "n": 25165824},
        # the largest top-k of the reference's tests: k = sqrt(n)
        {"name": "topk_f16_20m", "kind": "topk", "dtype": "float16", "n": 20 * 1024 * 1024 - 10, "k": 4579},
        # the serving loop: a burst of mixed requests (scan / seg_sum / compress), all waiting at once
        {"name": "served_48", "kind": "served", "count": 48, "hi": 1 << 24},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "rows", "seg_scan", "seg_sum", "spmv", "compact", "compact", "sort", "topk",
                       "served"])
    if kind == "scan":
        return {"kind": kind, "dtype": rng.choice(["int8", "float16", "float32"]), "n": _log_int(rng, 1 << 10, 1 << 28),
                "S": rng.choice([0, 64, 128])}
    if kind == "rows":
        lo = _log_int(rng, 64, 1024)
        return {"kind": kind, "dtype": rng.choice(["float16", "float32", "int8"]), "rows": _log_int(rng, 64, 4096),
                "lo": lo, "hi": _log_int(rng, 4 * lo, 1 << 18)}
    if kind == "seg_scan":
        return {"kind": kind, "dtype": rng.choice(["float16", "float16", "int8"]), "n": _log_int(rng, 1 << 12, 1 << 28),
                "p": rng.choice([0.001, 0.01, 0.05, 0.5])}
    if kind == "seg_sum":
        return {"kind": kind, "dtype": rng.choice(["float16", "int8", "float32"]), "n": _log_int(rng, 1 << 12, 1 << 28),
                "mean": rng.choice([4, 16, 64, 1024]), "wide": rng.random() < 0.5}
    if kind == "spmv":
        rows = _log_int(rng, 1 << 10, 1 << 20)
        return {"kind": kind, "dtype": rng.choice(["float16", "float32"]), "rows": rows,
                "nnz": rows * rng.choice([4, 16])}
    if kind == "compact":
        return {"kind": kind, "op": rng.choice(["compress", "positions", "gather", "split"]),
                "dtype": rng.choice(["int16", "float16", "float32"]), "n": _log_int(rng, 1 << 12, 1 << 28),
                "p": rng.choice([0.01, 0.3, 0.9])}
    if kind == "sort":
        return {"kind": kind, "dtype": rng.choice(["float16", "int16", "float32"]), "n": _log_int(rng, 1 << 12, 1 << 25)}
    if kind == "topk":
        n = _log_int(rng, 1 << 12, 40 * 1024 * 1024)
        return {"kind": kind, "dtype": rng.choice(["float16", "int16"]), "n": n,
                "k": rng.choice([1, 5, 64, int(n ** 0.5), n // 8])}
    return {"kind": "served", "count": rng.randint(8, 48), "hi": _log_int(rng, 1 << 18, 1 << 24)}


# ---------------------------------------------------------------------------
# inputs

LAYOUT = 11  # seed of what fixes the outputs' shapes: row lengths, segment lengths, numbers of ones


def _gen(dev, seed):
    return torch.Generator(device=dev).manual_seed(seed)


def _values(n, dtype, dev, seed):
    """int8 in [-8, 8], fp16 uniform [-1, 1), fp32 N(0, 1)."""
    if dtype == "float32":
        return torch.randn(n, device=dev, generator=_gen(dev, seed))
    return workloads.scan_input(n, DTYPES[dtype], dev, seed)


def _bounds(n, mean, wide, dev, seed):
    """CSR row pointers of n elements with geometric segment lengths: one set of lengths, in an order of the seed's."""
    steps = torch.empty(int(n / mean * 1.02) + 1024, device=dev).geometric_(1.0 / mean, generator=_gen(dev, LAYOUT))
    pts = torch.cumsum(steps.to(torch.int64), 0)
    pts = torch.cat([pts[pts < n], torch.full((1,), n, dtype=torch.int64, device=dev)])
    lens = torch.diff(pts, prepend=torch.zeros_like(pts[:1]))
    lens = lens[torch.randperm(lens.numel(), device=dev, generator=_gen(dev, seed))]
    b = torch.cat([torch.zeros_like(pts[:1]), torch.cumsum(lens, 0)])
    return b if wide else b.to(torch.int32)


def _mask(n, p, dev, seed):
    """Bernoulli(p) mask whose number of ones is the same for every seed (the outputs' shapes are the case's)."""
    shift = int(np.random.default_rng(seed).integers(0, n))
    return torch.roll(workloads.bernoulli_mask(n, p, dev, LAYOUT), shift)


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    kind = case["kind"]
    st = {"case": case}
    if kind == "scan":
        st["x"] = _values(case["n"], case["dtype"], dev, seed)
    elif kind == "rows":
        lens = np.diff(workloads.uneven_rows(case["rows"], case["lo"], case["hi"], LAYOUT))
        offs = np.concatenate([[0], np.cumsum(np.random.default_rng(seed).permutation(lens))])
        st["x"] = _values(int(offs[-1]), case["dtype"], dev, seed)
        st["offsets"] = torch.from_numpy(offs).to(dev)
    elif kind == "seg_scan":
        st["x"] = _values(case["n"], case["dtype"], dev, seed)
        st["flags"] = workloads.bernoulli_mask(case["n"], case["p"], dev, seed + 1)
    elif kind == "seg_sum":
        st["x"] = _values(case["n"], case["dtype"], dev, seed)
        st["indptr"] = _bounds(case["n"], case["mean"], case["wide"], dev, seed + 1)
    elif kind == "spmv":
        st["vals"], st["indptr"], st["cols"], st["x"] = workloads.zipf_csr(
            rows=case["rows"], cols=case["rows"], target_nnz=case["nnz"], dtype=DTYPES[case["dtype"]], device=dev,
            seed=seed)
    elif kind == "compact":
        n = case["n"]
        v = torch.randint(-1000, 1000, (n,), dtype=torch.int16, device=dev, generator=_gen(dev, seed))
        st["x"] = v.to(DTYPES[case["dtype"]])
        st["mask"] = _mask(n, case["p"], dev, seed + 1)
        if case["op"] == "gather":
            st["idx"] = torch.arange(n, dtype=torch.int32, device=dev)
    elif kind in ("sort", "topk"):
        n, dt = case["n"], DTYPES[case["dtype"]]
        if dt == torch.int16:
            st["x"] = torch.randint(-32768, 32768, (n,), dtype=dt, device=dev, generator=_gen(dev, seed))
        else:
            st["x"] = torch.rand(n, device=dev, generator=_gen(dev, seed)).to(dt)
    else:
        st["stream"] = workloads.ServedStream(case["count"], dev, LAYOUT, lo=1 << 10, hi=case["hi"])
        for i, pool in enumerate(st["stream"].pools):
            pool.copy_(workloads.scan_input(pool.numel(), pool.dtype, dev, seed + 1 + i))
        st["server"] = serve.Server(dev, budget_bytes=8 << 30, keep_results=True)
    return st


# ---------------------------------------------------------------------------
# one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "scan":
        return tcuscan_ops.run_scan_multi_core(state["x"], case["S"] or None)
    if kind == "rows":
        return batch.scan_rows(state["x"], state["offsets"])
    if kind == "seg_scan":
        return tcuscan_ops.run_seg_scan(state["x"], state["flags"], 64)
    if kind == "seg_sum":
        return tcuscan_ops.run_seg_sum_multi_core(state["x"], state["indptr"], 64)
    if kind == "spmv":
        return tcuscan_ops.run_spmv_v2(state["vals"], state["indptr"], state["cols"], state["x"], 64)
    if kind == "compact":
        op, x, mask = case["op"], state["x"], state["mask"]
        if op == "compress":
            return tcuscan_ops.run_compress(x, mask, 64)
        if op == "positions":
            return tcuscan_ops.run_compress_ind_no_arange(x, mask, 64)
        if op == "gather":
            return tcuscan_ops.run_compress_ind(x, state["idx"], mask, 64)
        return tcuscan_ops.run_split(x, mask, 64)
    if kind == "sort":
        return tcuscan_ops.run_radix_sort(state["x"], 128)
    if kind == "topk":
        lo, hi = (-32768, 32767) if case["dtype"] == "int16" else (0.0, 1.0)
        f = tcuscan_ops.run_topk_int16 if case["dtype"] == "int16" else tcuscan_ops.run_topk_fp16
        return f(state["x"], case["k"], lo, hi, 128)
    server, stream = state["server"], state["stream"]
    server.release()  # the results of the burst before this one
    ids = server.submit_many(*stream.arrays(), np.full(case["count"], server.now()))
    server.run()
    return [server.result(i) for i in ids]


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    """Each input read once, each output written once; one addition per element (two operations per nonzero)."""
    kind = case["kind"]
    eb = BYTES.get(case.get("dtype"), 0)
    if kind == "scan":
        return {"bytes": case["n"] * (eb + 4), "flops": case["n"]}
    if kind == "rows":
        lo, hi = case["lo"], case["hi"]
        n = int(case["rows"] * (hi - lo) / math.log(hi / lo))
        return {"bytes": n * (eb + 4) + 8 * (case["rows"] + 1), "flops": n}
    if kind == "seg_scan":
        return {"bytes": case["n"] * (eb + 1 + 4), "flops": case["n"]}
    if kind == "seg_sum":
        segs = case["n"] / case["mean"] + 1
        return {"bytes": int(case["n"] * eb + segs * ((8 if case["wide"] else 4) + 4)), "flops": case["n"]}
    if kind == "spmv":
        return {"bytes": case["nnz"] * (eb + 4) + case["rows"] * (4 + 4 + eb), "flops": 2 * case["nnz"]}
    if kind == "compact":
        n, k = case["n"], int(case["n"] * case["p"])
        out = {"compress": k * eb, "positions": k * (eb + 4), "gather": 4 * n + k * (eb + 4), "split": n * eb}
        return {"bytes": n * (eb + 1) + out[case["op"]], "flops": n}
    if kind == "sort":
        return {"bytes": case["n"] * (2 * eb + 4), "flops": case["n"]}
    if kind == "topk":
        return {"bytes": case["n"] * eb + case["k"] * (eb + 4), "flops": case["n"]}
    n = case["count"] * (case["hi"] - 1024) / math.log(case["hi"] / 1024)  # log-uniform sizes
    eb = 0.4 * 1 + 0.4 * 2 + 0.2 * 4
    return {"bytes": int(n * (0.5 * (eb + 4) + 0.3 * (eb + 8 / 64) + 0.2 * (eb + 1 + 0.3 * eb))), "flops": int(n)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("compact", "sort", "topk") or case.get("dtype") == "int8":
        return "exact"
    # FP32 results of sums accumulated in FP32 or better: 1e-8 to 1.2e-7 from the 64-bit results, and up to 2.4e-7
    # of a value between two runs that add their carries in another order; about four times that
    return {"rel": 5e-7, "max": 2e-6}


# ---------------------------------------------------------------------------
# the same results in 64 bits

def _scan64(x, starts=None):
    """Inclusive sums of x, restarted at each of the sorted positions `starts`."""
    x = x.to(torch.int64) if x.dtype == torch.int8 else x.double()
    cs = torch.cumsum(x, 0)
    if starts is None or starts.numel() == 0:
        return cs
    head = torch.zeros_like(cs)
    base = torch.where(starts > 0, cs[(starts - 1).clamp_min(0)], torch.zeros_like(cs[:1]))
    head[starts] = torch.diff(base, prepend=torch.zeros_like(base[:1]))
    return cs.sub_(torch.cumsum(head, 0))


def _sums64(x, indptr):
    x = x.to(torch.int64) if x.dtype == torch.int8 else x.double()
    cs = torch.cat([torch.zeros_like(x[:1]), torch.cumsum(x, 0)])
    ends = cs[indptr.long()]
    return ends[1:] - ends[:-1]


def exact(case, seed):
    st = prepare(dict(case), seed)
    kind, x = case["kind"], st.get("x")
    whole = torch.int32 if case.get("dtype") == "int8" else torch.float64
    if kind == "scan":
        return _scan64(x).to(whole)
    if kind == "rows":
        return _scan64(x, st["offsets"][:-1]).to(whole)
    if kind == "seg_scan":
        return _scan64(x, torch.nonzero(st["flags"]).flatten()).to(whole)
    if kind == "seg_sum":
        return _sums64(x, st["indptr"]).to(whole)
    if kind == "spmv":
        return _sums64(st["vals"].double() * x.double()[st["cols"].long()], st["indptr"])
    if kind == "compact":
        m = st["mask"].bool()
        if case["op"] == "compress":
            return x[m]
        if case["op"] == "split":
            return torch.cat([x[m], x[~m]])
        return x[m], torch.nonzero(m).flatten().to(torch.int32)
    if kind == "sort":
        v, i = torch.sort(x, stable=True)
        return v, i.to(torch.int32)
    if kind == "topk":
        thr = torch.sort(x).values[x.numel() - case["k"]]
        tie = x == thr
        keep = (x > thr) | (tie & (torch.cumsum(tie, 0) <= case["k"] - (x > thr).sum()))
        return x[keep], torch.nonzero(keep).flatten().to(torch.int32)
    out = []
    for i in range(case["count"]):
        op, xi, aux = st["stream"].request(i)
        i8 = xi.dtype == torch.int8
        if op == serve.SCAN:
            out.append(_scan64(xi).to(torch.int32 if i8 else torch.float64))
        elif op == serve.SEG_SUM:
            out.append(_sums64(xi, aux).to(torch.int32 if i8 else torch.float64))
        else:
            out.append(xi[aux.bool()])
    return out
