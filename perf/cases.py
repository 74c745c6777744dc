"""Workloads of the index, each one call (or one short sequence of calls) of
the public entry points on prepared inputs:

* ``query``       FalconnPP.query on host arrays (the reference's Python call);
* ``batched``     the batched form on device buffers, uniform or per-query k
                  and qProbes, FP32 / BF16 / FP8 rerank;
* ``build``       index construction followed by one batch of queries on the
                  new index (the tables themselves stay on the device);
* ``bruteforce``  the low-precision block rerank over every point;
* ``truth``       the exact FP64 top-k that recall is measured against.

The data are Gaussian mixtures with log-normal norms (the shapes of
``falconnpp_b200.synth``), drawn on the GPU from the seed; queries are held
out from the same mixture.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import falconnpp_b200
from falconnpp_b200 import capi

CENTRES = 256
SIGMA = 0.3
NORM_SIGMA = 0.4
PRECISION = {"fp32": 0, "bf16": 1, "fp8": 2}
ROW_BYTES = {"fp32": 4, "bf16": 2, "fp8": 1}


def _index(n, d, tables, proj, min_size, iprobes):
    return {"n": n, "d": d, "tables": tables, "proj": proj, "min_size": min_size, "scale": 0.01, "iprobes": iprobes}


# the two benchmark indexes of the repository, and the 128-dimensional shape
# of its precision workload at a size that builds in well under a second
SMALL = _index(100_000, 200, 50, 256, 500, 1)
LARGE = _index(1_000_000, 200, 100, 256, 1000, 3)
NARROW = _index(2_000_000, 128, 64, 128, 50, 3)


def listed():
    return [
        # one interactive lookup through the Python class: latency and launches
        {"name": "lookup-1", "kind": "query", **LARGE, "queries": 1, "k": 20, "qprobes": 10,
         "form": "plain", "precision": "fp32", "shortlist": 4},
        # the reference's CPU-sized configuration: 1,000 queries in one call
        {"name": "query-100Kx200", "kind": "query", **SMALL, "queries": 1000, "k": 20, "qprobes": 10,
         "form": "plain", "precision": "fp32", "shortlist": 4},
        # the whole query set in one call of the default form, as the
        # reference's integration script does
        {"name": "query-1Mx200", "kind": "query", **LARGE, "queries": 10_000, "k": 20, "qprobes": 10,
         "form": "plain", "precision": "fp32", "shortlist": 4},
        # the benchmark's operating point: resident data, FP8 first pass
        {"name": "batched-fp8", "kind": "batched", **LARGE, "queries": 10_000, "k": 20, "qprobes": 2,
         "mixed": False, "precision": "fp8", "shortlist": 2, "graph": True},
        # an uneven mixed batch: per-query k and qProbes, ragged size
        {"name": "batched-bf16-mixed", "kind": "batched", **LARGE, "queries": 2047, "k": 20, "qprobes": 80,
         "mixed": True, "precision": "bf16", "shortlist": 2, "graph": True},
        # the bit-exact batched form at a high recall setting (two probes per table)
        {"name": "batched-fp32-qp80", "kind": "batched", **LARGE, "queries": 3000, "k": 20, "qprobes": 80,
         "mixed": False, "precision": "fp32", "shortlist": 4, "graph": False},
        # 128 dimensions, 128 projections: another rotation size, small buckets
        {"name": "batched-fp8-128d", "kind": "batched", **NARROW, "queries": 10_000, "k": 10, "qprobes": 40,
         "mixed": False, "precision": "fp8", "shortlist": 4, "graph": False},
        # the reference's own setting: L = 50 and qProbes in the thousands
        {"name": "batched-qp1000", "kind": "batched", **SMALL, "queries": 1000, "k": 20, "qprobes": 1000,
         "mixed": False, "precision": "fp32", "shortlist": 4, "graph": False},
        # index construction from a host array (the Python class)
        {"name": "build-100Kx200", "kind": "build", **SMALL, "queries": 256, "k": 20, "qprobes": 10, "host": True},
        # index construction from resident data at the benchmark's size
        {"name": "build-1Mx200", "kind": "build", **LARGE, "queries": 256, "k": 20, "qprobes": 10, "host": False},
        # the block rerank: every point against a batch of queries
        {"name": "bruteforce-bf16", "kind": "bruteforce", **SMALL, "n": 1_000_000, "tables": 4, "queries": 10_000,
         "k": 20, "precision": "bf16", "shortlist": 4},
        # the recall ground truth of a benchmark run (500-query sample)
        {"name": "truth-f64", "kind": "truth", "n": 1_000_000, "d": 200, "queries": 500, "k": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: 20 thousand to a million points, 48
    to 256 dimensions (odd ones too), 1 to 10,000 queries."""
    kind = rng.choice(["query", "query", "batched", "batched", "batched", "build", "bruteforce", "truth"])
    n = _log_int(rng, 20_000, 1_000_000)
    d = rng.choice([64, 100, 128, 200, 256, rng.randint(48, 256), rng.randint(48, 256)])
    k = rng.choice([1, 5, 10, 20, 50, 100])
    if kind == "truth":
        return {"kind": kind, "n": n, "d": d, "queries": _log_int(rng, 10, 500), "k": k}
    proj = rng.choice([64, 128, 256, 256])
    tables = rng.randint(8, 100)
    case = {"kind": kind, **_index(n, d, tables, proj, rng.choice([50, 200, 500, 1000]), rng.choice([1, 2, 3])),
            "queries": _log_int(rng, 1, 10_000), "k": k, "qprobes": _log_int(rng, 1, 80)}
    if kind == "query":
        form = rng.choice(["plain", "plain", "batched"])
        precision = "fp32" if form == "plain" else rng.choice(["fp32", "bf16", "fp8"])
        return {**case, "form": form, "precision": precision, "shortlist": rng.choice([2, 4])}
    if kind == "batched":
        return {**case, "mixed": rng.random() < 0.3, "precision": rng.choice(["fp32", "bf16", "fp8"]),
                "shortlist": rng.choice([2, 4]), "graph": rng.random() < 0.5}
    if kind == "build":
        return {**case, "queries": min(case["queries"], 256), "host": rng.random() < 0.5}
    return {**case, "tables": 4, "precision": rng.choice(["bf16", "fp8"]), "shortlist": 2}


def _mixture(gen, centres, n):
    d = centres.shape[1]
    x = torch.empty((n, d), dtype=torch.float32, device="cuda")
    for s in range(0, n, 1 << 18):
        m = min(1 << 18, n - s)
        label = torch.randint(0, centres.shape[0], (m,), generator=gen, device="cuda")
        p = centres[label] + SIGMA * torch.randn((m, d), generator=gen, device="cuda")
        norm = torch.exp(NORM_SIGMA * torch.randn((m, 1), generator=gen, device="cuda"))
        x[s:s + m] = p / p.norm(dim=1, keepdim=True) * norm
    return x


def _data(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    centres = torch.randn((CENTRES, case["d"]), generator=gen, device="cuda")
    return _mixture(gen, centres, case["n"]), _mixture(gen, centres, case["queries"])


def _mixed_arrays(case, seed):
    """Per-query k and qProbes of a mixed batch, bounded by the case's own."""
    rng = np.random.default_rng(seed)
    ks = np.array([v for v in (1, 5, 10, 20, 50, 100) if v <= case["k"]], np.int32)
    qps = np.array([v for v in (1, 5, 10, 20, 80) if v <= case["qprobes"]], np.int32)
    return rng.choice(ks, case["queries"]).astype(np.int32), rng.choice(qps, case["queries"]).astype(np.int32)


def _set_param(index, case):
    args = (case["tables"], case["proj"], case["min_size"], case["scale"], case["iprobes"], 8, 42)
    (index.set_index_param if isinstance(index, capi.Index) else index.setIndexParam)(*args)


def prepare(case, seed):
    x, q = _data(case, seed)
    torch.cuda.synchronize()  # the index runs on streams of its own
    kind, k, nq = case["kind"], case["k"], case["queries"]
    state = {"case": case, "stream": torch.cuda.Stream()}
    if kind == "truth":
        out = torch.zeros((nq, k), dtype=torch.int32, device="cuda")
        return {**state, "x": x, "q": q, "ids": out, "scores": torch.zeros((nq, k), dtype=torch.float64, device="cuda")}
    host = kind == "query" and case["form"] == "plain" or kind == "build" and case["host"]
    if host:
        index = falconnpp_b200.FalconnPP.FalconnPP(case["n"], case["d"])
    else:
        index = capi.Index(case["n"], case["d"])
    _set_param(index, case)
    state["index"] = index
    if kind == "build":
        index.set_qProbes(case["qprobes"]) if host else index.set_qprobes(case["qprobes"])
        if host:
            return {**state, "x": x.cpu().numpy(), "q": q.cpu().numpy()}
        state.update(x=x, q=q)
    elif host:
        index.build(x.cpu().numpy().T)
        index.set_qProbes(case["qprobes"])
        return {**state, "q": q.cpu().numpy()}
    else:
        index.build_device(x.data_ptr())
        if kind != "bruteforce":
            index.set_qprobes(case["qprobes"])
        if kind == "query":
            index.set_query_form(1, PRECISION[case["precision"]], case["shortlist"])
            return {**state, "q": q.cpu().pin_memory().numpy()}
        state["q"] = q
    if kind == "batched":
        index.set_query_form(1, PRECISION[case["precision"]], case["shortlist"])
        index.set_option("use_graph", int(case["graph"]))
        if case["mixed"]:
            ks, qps = _mixed_arrays(case, seed)
            state["ks"], state["qps"] = torch.from_numpy(ks).cuda(), torch.from_numpy(qps).cuda()
    state["ids"] = torch.zeros((nq, k), dtype=torch.int32, device="cuda")
    state["scores"] = torch.zeros((nq, k), dtype=torch.float32, device="cuda")
    if kind == "build":
        state["counts"] = torch.zeros((nq, 2), dtype=torch.int32, device="cuda")
    return state


def run(state):
    case = state["case"]
    kind, nq, k = case["kind"], case["queries"], case["k"]
    stream = state["stream"].cuda_stream
    if kind == "truth":
        capi.bruteforce_topk_f64(state["x"].data_ptr(), case["n"], case["d"], state["q"].data_ptr(), nq, k,
                                 state["ids"].data_ptr(), state["scores"].data_ptr(), stream)
        return {"ids": state["ids"], "scores": state["scores"]}
    index = state["index"]
    if kind == "query":
        if case["form"] == "plain":
            return {"ids": index.query(state["q"].T, k)}
        return {"ids": index.query(state["q"], k)}
    if kind == "build":
        if case["host"]:
            index.build(state["x"].T)
            return {"ids": index.query(state["q"].T, k)}
        index.build_device(state["x"].data_ptr(), stream)
        index.query_batched_dump(state["q"].data_ptr(), nq, k, state["ids"].data_ptr(), state["scores"].data_ptr(),
                                 None, state["counts"].data_ptr(), stream)
        info = index.info()
        return {"ids": state["ids"], "scores": state["scores"], "counts": state["counts"],
                "stored": info["n_ids"], "largest": info["max_kept"]}
    if kind == "bruteforce":
        index.bruteforce_lowp(state["q"].data_ptr(), nq, k, PRECISION[case["precision"]], case["shortlist"],
                              state["ids"].data_ptr(), state["scores"].data_ptr(), stream)
        return {"ids": state["ids"], "scores": state["scores"]}
    ks, qps = state.get("ks"), state.get("qps")
    index.query_batched(state["q"].data_ptr(), nq, ks.data_ptr() if ks is not None else None,
                        qps.data_ptr() if qps is not None else None, k, case["qprobes"], state["ids"].data_ptr(), k,
                        state["scores"].data_ptr(), stream)
    return {"ids": state["ids"], "scores": state["scores"]}


def _per_query(case):
    """Candidates and unique candidates per query: a probed bucket of this
    data holds about min(min_size, n * iprobes / 1000) ids, and what a query
    gathers lies mostly in its own cluster of n / CENTRES points."""
    qp = case["qprobes"] if not case.get("mixed") else max(1, case["qprobes"] // 3)
    cand = qp * max(1.0, min(case["min_size"], case["n"] * case["iprobes"] / 1000))
    cluster = case["n"] / CENTRES
    return cand, cand * cluster / (cand + cluster)


def work(case):
    kind, n, d, nq, k = case["kind"], case["n"], case["d"], case["queries"], case["k"]
    call = nq * (4 * d + 8 * k)  # queries in, ids and scores out
    if kind in ("truth", "bruteforce"):
        return {"bytes": n * d * ROW_BYTES[case.get("precision", "fp32")] + call, "flops": 2.0 * n * nq * d}
    fht = 1 << (max(d, case["proj"]) - 1).bit_length()
    hashing = 6.0 * case["tables"] * fht * math.log2(fht)
    cand, unique = _per_query(case)
    query = {"bytes": call + nq * (4 * cand + 8 * case["qprobes"])
             + min(n, nq * unique) * d * ROW_BYTES[case.get("precision", "fp32")],
             "flops": nq * (hashing + 2 * unique * d)}
    if kind != "build":
        return query
    tables = 4.0 * case["tables"] * (n * case["iprobes"] + 4 * case["proj"] ** 2)
    return {"bytes": 8.0 * n * d + tables + query["bytes"], "flops": n * hashing + query["flops"]}


def exact(case, seed):
    """The scores of the exact top-k in 64 bits, computed by torch.  The ids
    have no such value (an approximate search may return others)."""
    kind, k, nq = case["kind"], case["k"], case["queries"]
    if kind == "query" or kind == "build" and case["host"]:
        return None
    if kind == "batched" and _per_query({**case, "qprobes": 1} if case["mixed"] else case)[0] < 25 * k:
        return None  # so few candidates that the search misses many neighbours
    x, q = _data(case, seed)
    x, q = x.double(), q.double()
    if kind != "truth":
        x = x - x.mean(dim=0, keepdim=True)
    scores = torch.empty((nq, k), dtype=torch.float64, device="cuda")
    for s in range(0, nq, 256):
        scores[s:s + 256] = torch.topk(q[s:s + 256] @ x.T, k, dim=1).values
    if case.get("mixed"):
        ks = torch.from_numpy(_mixed_arrays(case, seed)[0]).cuda()
        scores[torch.arange(k, device="cuda")[None, :] >= ks[:, None]] = 0.0
    got = {"ids": None, "scores": scores}
    if kind == "build":
        got.update(counts=None, stored=None, largest=None)
    return got
