"""The work that performance is measured on: calls of the selector as a serving process makes them.

A case is one pass of such a process: the selections of one decode step (`layers` calls, one per
indexer layer, eager or as the replayed CUDA graph a decode loop keeps), one prefill chunk, one step
of the fused indexer, or one batch whose logits are in host memory. `op` names the entry point:

  select   fast_topk_v3 / fast_topk      fp32 logits, k = 2048
  warm     fast_topk_v3_warm             the same, with the thresholds of the step before
  general  fast_topk_general             any k, fp32 / fp16 / bf16 logits
  paged    fast_topk_transform_fused     prefill chunk, indices mapped through the page table
  indexer  FusedIndexerTopk              logits from q and the key cache, selected as they are produced
  host     fast_topk_v3_host             logits, lengths and result in host memory

The ops hand out a row's indices in no particular order, so a pass ends the way a masked attention
uses them: they are marked in a byte mask over the keys (two small torch kernels per pass, whatever
the number of layers). Rows shorter than k are padded with -1, which is folded onto index 0 - a key
that such a row has selected anyway.
"""
from __future__ import annotations

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "flash-float-jit-kernels_b200"))

from jit_kernel import _native  # noqa: E402
from jit_kernel.indexer import FusedIndexerTopk  # noqa: E402
from jit_kernel.topk_indexer import (  # noqa: E402
    fast_topk, fast_topk_general, fast_topk_transform_fused, fast_topk_v3, fast_topk_v3_host, fast_topk_v3_warm)

K = 2048
HEADS, DIM = 64, 128
MARGIN = 1 << 18  # key units, about 3 % of a logit: what covers a query that drifts from step to step
DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16, "fp8": torch.float8_e4m3fn}


def _case(op, batch, length, layers=1, values="normal", ragged=False, k=K, dtype="fp32", graph=False, overlap=False,
          cold=False):
    return {"op": op, "batch": batch, "length": length, "layers": layers, "values": values, "ragged": ragged, "k": k,
            "dtype": dtype, "graph": graph, "overlap": overlap, "cold": cold}


def listed():
    return [
        # one short request, called eagerly: host time and launch latency are most of it
        dict(name="decode_b1_16k", **_case("select", 1, 16384)),
        # a decode step of a model with eight indexer layers, replayed as a CUDA graph: one request of
        # a medium context (odd length: rows grow by one token per step) ...
        dict(name="decode_b1_96k_graph", **_case("select", 1, 98305, layers=8, values="heads", graph=True)),
        # ... and of the longest context
        dict(name="decode_b1_1m_graph", **_case("select", 1, 1048576, layers=8, values="heads", graph=True)),
        # the same loop carrying every row's threshold from step to step, a few requests
        dict(name="warm_b4_200k_graph", **_case("warm", 4, 200001, layers=4, values="heads", graph=True)),
        # a full decode batch of requests of all lengths, one eager call
        dict(name="ragged_b64_128k", **_case("select", 64, 131072, ragged=True)),
        # the same batch as a stream of independent calls that may overlap
        dict(name="ragged_b64_128k_stream", **_case("select", 64, 131072, layers=8, ragged=True, graph=True, overlap=True)),
        # a prefill chunk of two requests of 2048 queries each, page tables applied: the largest
        dict(name="prefill_b4096_32k_paged", **_case("paged", 4096, 32768, values="heads")),
        # half-width logits and a smaller k
        dict(name="bf16_k1024_b24_70k", **_case("general", 24, 70001, ragged=True, k=1024, dtype="bf16")),
        # logits in pinned host memory
        dict(name="host_b16_64k", **_case("host", 16, 65536, ragged=True)),
        # the fused indexer in a decode loop: one request with an fp8 key cache, as a graph ...
        dict(name="indexer_fp8_b1_128k_graph", **_case("indexer", 1, 131072, layers=4, dtype="fp8", graph=True)),
        # ... a full ragged batch with a bf16 key cache ...
        dict(name="indexer_bf16_b64_128k", **_case("indexer", 64, 131072, ragged=True, dtype="bf16")),
        # ... and the first step of new requests, which has no thresholds to start from
        dict(name="indexer_fp8_b8_64k_cold", **_case("indexer", 8, 65537, ragged=True, dtype="fp8", cold=True)),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["select", "select", "select", "warm", "general", "paged", "indexer", "indexer", "host"])
    values = rng.choice(["normal", "normal", "heads", "heads", "ties", "tail"])
    if op == "paged":
        length = spread(4096, 65536)
        batch = max(2, min(spread(128, 4096), (7 << 24) // length)) & ~1
        return _case(op, batch, length, values=values)
    if op == "indexer":
        length = spread(4096, 1 << 20)
        batch = max(1, min(spread(1, 64), (1 << 23) // length))
        graph = rng.random() < 0.5
        return _case(op, batch, length, layers=rng.choice([1, 2, 4]) if graph and batch * length <= 1 << 20 else 1,
                     ragged=batch > 1, dtype=rng.choice(["bf16", "fp8"]), graph=graph, cold=rng.random() < 0.25)
    if op == "host":
        length = spread(4096, 1 << 18)
        batch = max(1, min(spread(1, 64), (1 << 22) // length))
        return _case(op, batch, length, values=values, ragged=batch > 1)
    length = spread(4096, 1 << 20)
    batch = max(1, min(spread(1, 256), (1 << 24) // length))
    graph = rng.random() < 0.5
    layers = max(1, min(rng.choice([1, 2, 4, 8]), (1 << 24) // (batch * length))) if graph else 1
    ragged = batch > 1 and rng.random() < 0.6
    if op == "general":
        return _case(op, batch, length, layers=layers, values=values, ragged=ragged, k=rng.choice([512, 1024, 1025, 3000, 4096]),
                     dtype=rng.choice(["fp32", "fp16", "bf16"]), graph=graph)
    return _case(op, batch, length, layers=layers, values=values, ragged=ragged, graph=graph,
                 overlap=op == "select" and graph and batch >= 16 and rng.random() < 0.5)


# ---- inputs --------------------------------------------------------------------------------------
def _fill_logits(values, gen, out):
    """Indexer logits: N(0,1); the sum over 64 heads of w_h * relu(N(0,1)); 70 % exact zeros, a
    log-normal rest and 5 % copies of one value at the threshold; N(0,1) with a tail of 0.1 %."""
    if values == "heads":
        w = torch.rand(HEADS, generator=gen, device=out.device).tolist()
        x = torch.empty_like(out)
        out.zero_()
        for h in range(HEADS):
            out.add_(x.normal_(generator=gen).relu_(), alpha=w[h])
        return
    out.normal_(generator=gen)
    if values == "tail":
        out.add_(6.0 * (torch.rand(out.shape, generator=gen, device=out.device) < 0.001))
    elif values == "ties":
        u = torch.rand(out.shape, generator=gen, device=out.device)
        out.exp_().masked_fill_(u < 0.70, 0.0)
        top = torch.topk(out.masked_fill(u >= 0.95, -1.0), min(K, out.size(1)), dim=1).values[:, -1:]
        out.copy_(torch.where(u >= 0.95, top, out))


def _lengths(case, gen, batch, length, device):
    if not case["ragged"]:
        return torch.full((batch,), length, dtype=torch.int32, device=device)
    return torch.randint(min(1024, length), length + 1, (batch,), generator=gen, device=device, dtype=torch.int32)


def _mean_length(case):
    B, L = case["batch"], case["length"]
    if case["op"] == "paged":
        return sum(n for _, n in _chunk(case)) / B
    return (min(1024, L) + L) / 2 if case["ragged"] else L


def _chunk(case):
    """(request, valid keys) of every query row of a prefill chunk of two requests: one at the end of
    a prompt as long as the logits are wide, one a quarter of the way through (causal: a row sees the
    keys up to its own position)."""
    B, L = case["batch"], case["length"]
    n = B // 2
    ends = (L, max(n, L // 4))
    return [(r, max(1, ends[r] - n + 1 + i)) for r in range(2) for i in range(n)]


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    B, L, n, op = case["batch"], case["length"], case["layers"], case["op"]
    dtype = DTYPES[case["dtype"]]
    s = {"case": case, "graph": None}
    s["mask"] = torch.zeros(n * B, L, dtype=torch.uint8, device="cpu" if op == "host" else dev)
    if op == "indexer":
        _prepare_indexer(s, gen, dev, dtype)
    else:
        s["lengths"] = _lengths(case, gen, B, L, dev)
        s["score"] = []
        for _ in range(n):
            x = torch.empty(B, L, device=dev)
            _fill_logits(case["values"], gen, x)
            s["score"].append(x if dtype == torch.float32 else x.to(dtype))
        s["idx"] = torch.empty(n * B, case["k"], dtype=torch.int32, device=dev)
        if op == "warm":
            # the step before this one: every row one logit shorter
            s["thr"] = torch.zeros(n, B, dtype=torch.int32, device=dev)
            for i in range(n):
                fast_topk_v3_warm(s["score"][i], s["lengths"] - 1, K, s["thr"][i])
        elif op == "paged":
            rows = _chunk(case)
            s["lengths"] = torch.tensor([c for _, c in rows], dtype=torch.int32, device=dev)
            s["cu"] = torch.tensor([0, B // 2, B], dtype=torch.int32, device=dev)
            s["pages"] = torch.stack([torch.randperm(L, generator=gen, device=dev) for _ in range(2)]).to(torch.int32)
        elif op == "host":
            s["score"] = [s["score"][0].cpu().pin_memory()]
            s["lengths"] = s["lengths"].cpu().pin_memory()
            s["idx"] = torch.empty(B, K, dtype=torch.int32).pin_memory()
    if case["graph"]:
        _capture(s)
    return s


def _prepare_indexer(s, gen, dev, dtype):
    case = s["case"]
    B, L, n = case["batch"], case["length"], case["layers"]
    s["lengths"] = _lengths(case, gen, B, L, dev)
    s["idx"] = torch.empty(n * B, K, dtype=torch.int32, device=dev)
    s["layer"] = []
    for i in range(n):
        q = torch.randn(B, HEADS, DIM, generator=gen, device=dev) * 0.5
        before = q + 0.025 * torch.randn(B, HEADS, DIM, generator=gen, device=dev)
        keys = torch.empty(B, L, DIM, dtype=dtype, device=dev)
        for b in range(B):
            keys[b] = (torch.randn(L, DIM, generator=gen, device=dev) * 0.5).to(dtype)
        w = torch.rand(B, HEADS, generator=gen, device=dev)
        scale = torch.rand(B, L, generator=gen, device=dev) + 0.5 if case["dtype"] == "fp8" else None
        f = FusedIndexerTopk(B, L, dev)
        f.logits.zero_()  # (columns beyond a row's length are never written)
        if not case["cold"]:  # the step before this one, with the query it had
            f(before.to(dtype), keys, w, s["lengths"], k_scale=scale)
        s["layer"].append((f, q.to(dtype), keys, w, scale))


def _capture(s):
    """The decode step as a CUDA graph, the way a decode loop keeps it."""
    overlap = s["case"]["overlap"]
    kept = [t.clone() for t in _thresholds(s)]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        _step(s)  # (first calls set kernel attributes, which a capture may not)
        for t, was in zip(_thresholds(s), kept):
            t.copy_(was)
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    if overlap:
        _native.set_overlap(True)
    try:
        with torch.cuda.graph(graph):
            s["out"] = _step(s)
    finally:
        if overlap:
            _native.set_overlap(False)
    s["graph"] = graph


def _thresholds(s):
    return [s["thr"]] if "thr" in s else [layer[0].thresholds for layer in s.get("layer", [])]


# ---- one pass -------------------------------------------------------------------------------------
def run(s):
    if s["graph"] is not None:
        s["graph"].replay()
        return s["out"]
    return _step(s)


def _step(s):
    case = s["case"]
    op, B, n = case["op"], case["batch"], case["layers"]
    idx, lengths = s.get("idx"), s["lengths"]
    out = {}
    if op == "select" and n == 1:
        idx = fast_topk_v3(s["score"][0], lengths, K)
    elif op == "select":
        for i in range(n):
            fast_topk(s["score"][i], idx[i * B:(i + 1) * B], lengths)
    elif op == "warm":
        for i in range(n):
            fast_topk_v3_warm(s["score"][i], lengths, K, s["thr"][i], margin=MARGIN, out=idx[i * B:(i + 1) * B])
        out["thresholds"] = s["thr"]
    elif op == "general":
        picked = [fast_topk_general(s["score"][i], lengths, case["k"]) for i in range(n)]
        idx = picked[0] if n == 1 else torch.cat(picked)
    elif op == "paged":
        idx = fast_topk_transform_fused(s["score"][0], lengths, s["pages"], s["cu"], K)
    elif op == "host":
        fast_topk_v3_host(s["score"][0], lengths, K, out=idx)
        torch.cuda.current_stream().synchronize()  # (the caller reads the result on the host)
    else:
        for i, (f, q, keys, w, scale) in enumerate(s["layer"]):
            if case["cold"]:
                f.thresholds.zero_()
            f(q, keys, w, lengths, margin=MARGIN, out=idx[i * B:(i + 1) * B], k_scale=scale)
        out["logits"] = [layer[0].logits for layer in s["layer"]]
        # (a positive logit's key is its bit pattern with the sign bit set: its negative as a float)
        out["thresholds"] = [layer[0].thresholds.view(torch.float32) for layer in s["layer"]]
    if case["ragged"] or op == "paged":
        idx = idx.clamp_(min=0)
    out["mask"] = s["mask"].zero_().scatter_(1, idx, 1)
    return out


# ---- what a pass cannot do without -----------------------------------------------------------------
def work(case):
    B, n = case["batch"], case["layers"]
    keys = n * B * _mean_length(case)
    picks = 4 * n * B * case["k"]
    if case["op"] == "indexer":
        per_key = 256 if case["dtype"] == "bf16" else 132
        return {"bytes": keys * (per_key + 4) + n * B * (HEADS * DIM * (per_key // 128) + HEADS * 4) + picks,
                "flops": keys * 2 * HEADS * DIM}
    width = 4 if case["dtype"] == "fp32" else 2
    table = 4 * 2 * case["length"] if case["op"] == "paged" else 0
    return {"bytes": keys * width + 4 * n * B + picks + table, "flops": 0}


def tolerance(case):
    if case["op"] == "indexer":
        # fp32 sums over 128 products and 64 heads, against the same sums in 64 bits: 1.1e-7 in norm and
        # 3.5e-7 at most (torch in fp32: 0.5e-7 and 2.2e-7); four times that, and the few picks whose
        # logits lie closer to the threshold (none seen in two rows of 65,537 keys)
        return {"rel": 5e-7, "max": 1.5e-6, "differ": 1e-4}
    return "exact"
