"""The work a user of annc_b200 has it do, as cases that can be timed and compared.

A case is a dict of plain values; `kind` names the path and the rest its sizes:

  dlrm             DlrmPipeline.forward: one inference pass of the DLRM-style model
  bags             device.BagPlan.run: grouped embedding bags over device-resident id buffers
  segment_reduce   the KPFusedSparseSegmentReduce operator, one table per call
  gather_unique    the KPFusedGather operator: unique keys, inverse map, their rows
  matmul_add_relu  the `__matmul_add_relu` custom call
  layout_matmul    the `__layout_matmul` custom call (kn4-packed weight, on the host as a graph
                   compiler holds a constant, or on the device)
  bmm_softmax      the `__batch_matmul` custom call followed by the row softmax
  bmm_sigmoid      the KPFusedBatchMatMulAddSigmoid operator (fp32)
  mlp_bf16         device.gemm chain of the wide BF16 MLP: bias + ReLU layers, sigmoid at the end

Sizes and distributions are those of the benchmark configurations and the tests.  Inputs are
drawn on the GPU from the seed alone.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from annc_b200 import device as dev
from annc_b200 import ops, synth
from annc_b200._lib import (ACT_RELU, ACT_SIGMOID, IO_A_BF16, IO_B_BF16, IO_C_BF16, MATH_BF16, MATH_FP32)
from annc_b200.dlrm import DlrmPipeline

_LUT = 1 << 22  # distinct popularity ranks of a table's ids


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # one serving request batch: latency and launches are what a user waits for
        dict(name="dlrm_b200", kind="dlrm", batch=200, max_rows=100_000, max_bag=20),
        # a throughput batch of the benchmark model
        dict(name="dlrm_b65536", kind="dlrm", batch=65536, max_rows=1_000_000, max_bag=20),
        # hash-bucket ids, 6.6 GB of tables, sum pooling (the embedding benchmark configuration)
        dict(name="bags_hash_sum", kind="bags", tables=26, rows=1_000_000, dim=64, batch=16384, min_bag=1,
             max_bag=20, ids="hash", mean=False, zipf=1.05),
        # plain row numbers, empty bags among them, mean pooling, wide rows (the recsys shape)
        dict(name="bags_rows_mean", kind="bags", tables=64, rows=50_000, dim=128, batch=1999, min_bag=0,
             max_bag=50, ids="i64", mean=True, zipf=1.2),
        # one table of a rewritten TF graph at a serving batch: the operator call with its allocation callback
        dict(name="segment_reduce_b256", kind="segment_reduce", rows=100_000, dim=64, batch=256, max_bag=20,
             ids="i64", mean=False, zipf=1.05),
        # unique keys of a large id column and their rows
        dict(name="gather_unique_300k", kind="gather_unique", rows=1_000_000, dim=64, nnz=300_001, zipf=1.05),
        # one MLP layer of a compiled graph, addend as the full broadcast matrix
        dict(name="matmul_add_relu_512", kind="matmul_add_relu", m=512, k=1024, n=1024),
        # constant-folded prepacked weight: a large batch, device-resident ...
        dict(name="layout_matmul_8192", kind="layout_matmul", m=8192, k=2048, n=4096, weight="device"),
        # ... and a serving batch with the weight a host constant of the executable
        dict(name="layout_matmul_200", kind="layout_matmul", m=200, k=2048, n=4096, weight="host"),
        # attention scores and their row softmax
        dict(name="bmm_softmax_64x256", kind="bmm_softmax", b=64, m=256, k=64, n=256),
        # target-attention scoring layer in fp32, bias per output column
        dict(name="bmm_sigmoid_256x50", kind="bmm_sigmoid", b=256, m=50, k=128, n=256, rhs_batched=False),
        # concat of 64 pooled vectors through the BF16 MLP
        dict(name="mlp_bf16_16384", kind="mlp_bf16", batch=16384, k=8192, h1=1024, h2=512),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["dlrm", "dlrm", "bags", "bags", "segment_reduce", "gather_unique", "matmul_add_relu",
                       "layout_matmul", "layout_matmul", "bmm_softmax", "bmm_sigmoid", "mlp_bf16"])
    if kind == "dlrm":
        batch = _log(rng, 64, 65536)
        return dict(kind=kind, batch=batch, max_rows=_log(rng, 20_000, 1_000_000), max_bag=rng.randint(1, 20))
    if kind == "bags":
        dim = rng.choice([16, 32, 64, 64, 128, 128, 256, 8, 48, 100])
        tables = _log(rng, 1, 100)
        # lookups * dim stays below that of the listed cases
        most = min(65536, max(64, 200_000_000 // (tables * dim * 20)))
        return dict(kind=kind, tables=tables, rows=_log(rng, 1000, min(1_000_000, 400_000_000 // (tables * dim))),
                    dim=dim, batch=_log(rng, 32, most), min_bag=rng.randint(0, 1), max_bag=rng.randint(1, 40),
                    ids=rng.choice(["hash", "i64", "i32"]), mean=rng.random() < 0.5,
                    zipf=rng.choice([1.05, 1.2]))
    if kind == "segment_reduce":
        return dict(kind=kind, rows=_log(rng, 1000, 1_000_000), dim=rng.choice([16, 32, 64, 128, 20]),
                    batch=_log(rng, 16, 16384), max_bag=rng.randint(1, 40), ids=rng.choice(["i64", "i32"]),
                    mean=rng.random() < 0.5, zipf=rng.choice([1.05, 1.2]))
    if kind == "gather_unique":
        return dict(kind=kind, rows=_log(rng, 1000, 1_000_000), dim=rng.choice([8, 16, 32, 64, 128, 12]),
                    nnz=_log(rng, 200, 1_000_000), zipf=rng.choice([1.05, 1.2]))
    if kind == "matmul_add_relu":
        m = _log(rng, 1, 8192)
        k, n = _log(rng, 16, 2048), _log(rng, 16, 2048)
        if rng.random() < 0.75:  # layer widths of real models are multiples of four, batches are not
            k, n = (k + 3) // 4 * 4, (n + 3) // 4 * 4
        else:
            k, n, m = min(k, 512), min(n, 512), min(m, 2048)
        return dict(kind=kind, m=m, k=k, n=n)
    if kind == "layout_matmul":
        m = _log(rng, 1, 8192)
        return dict(kind=kind, m=m, k=_log(rng, 8, 512) * 4, n=_log(rng, 8, 1024) * 4,
                    weight=rng.choice(["device", "host"]))
    if kind == "bmm_softmax":
        return dict(kind=kind, b=_log(rng, 1, 128), m=_log(rng, 1, 512), k=_log(rng, 4, 32) * 4,
                    n=rng.choice([_log(rng, 4, 128) * 4, _log(rng, 16, 512)]))
    if kind == "bmm_sigmoid":
        return dict(kind=kind, b=_log(rng, 1, 512), m=_log(rng, 1, 100), k=_log(rng, 4, 256), n=_log(rng, 1, 256),
                    rhs_batched=rng.random() < 0.5)
    return dict(kind=kind, batch=_log(rng, 256, 16384), k=rng.choice([16, 32, 64]) * 128,
                h1=rng.choice([512, 1024]), h2=rng.choice([256, 512]))


# ---------------------------------------------------------------- inputs

def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)


def _normal(g, *shape, scale=1.0):
    return torch.randn(shape, device="cuda", generator=g) * scale


def _ranks(g, n: int, a: float):
    """Zipf-like popularity ranks in [1, 2^22]: floor of a Pareto variable of tail index a - 1, what
    lies beyond the map spread evenly over it."""
    x = torch.rand(n, device="cuda", generator=g, dtype=torch.float64).clamp_(min=1e-18) ** (-1.0 / (a - 1.0))
    far = torch.randint(1, _LUT, (n,), device="cuda", generator=g)
    return torch.where(x < _LUT, x.clamp(max=float(_LUT)).to(torch.int64), far)


def _ids62(g, n: int, a: float, table: int):
    """Raw 62-bit ids: every rank has one fixed id, scattered over the whole range."""
    h = (_ranks(g, n, a) + table * 0x51ED2701) * 0x1E3779B97F4A7C15
    h = h ^ ((h >> 29) & 0x7FFFFFFFF)
    return (h * 0x3F58476D1CE4E5B9) & ((1 << 62) - 1)


def _bags(g, batch: int, lo: int, hi: int):
    """Index matrix [nnz, 2] (sample, position) of bags of U{lo..hi} lookups, sorted by sample."""
    lens = torch.randint(lo, hi + 1, (batch,), device="cuda", generator=g)
    if int(lens.sum()) == 0:
        lens[0] = 1
    seg = torch.repeat_interleave(torch.arange(batch, device="cuda"), lens)
    pos = torch.arange(seg.shape[0], device="cuda") - (torch.cumsum(lens, 0) - lens)[seg]
    return torch.stack([seg, pos], 1).contiguous()


def _dlrm_inputs(case, seed):
    """Tensors of the DLRM-style model: 26 tables of log-uniform size, 13 dense features."""
    g = _gen(seed)
    dim, tables, top_in = 64, 26, 64 + 27 * 26 // 2
    r = np.random.default_rng(seed)
    rows = [int(round(10 ** u)) for u in r.uniform(3.0, math.log10(case["max_rows"]), tables)]
    layer = lambda k, n: (_normal(g, k, n, scale=k ** -0.5), _normal(g, n, scale=0.01))
    d = dict(bottom=[layer(13, 512), layer(512, 256), layer(256, dim)],
             top=[layer(top_in, 512), layer(512, 256), layer(256, 1)],
             dense=_normal(g, case["batch"], 13),
             tables=[torch.rand((n, dim), device="cuda", generator=g) * 0.1 - 0.05 for n in rows], bags=[])
    for t in range(tables):
        seg = _bags(g, case["batch"], 1, case["max_bag"])
        d["bags"].append((_ids62(g, seg.shape[0], 1.05, t), seg))
    return d


def _bag_inputs(case, seed):
    g = _gen(seed)
    tabs = [torch.rand((case["rows"], case["dim"]), device="cuda", generator=g) * 0.1 - 0.05
            for _ in range(case["tables"])]
    ids, segs = [], []
    for t in range(case["tables"]):
        seg = _bags(g, case["batch"], case["min_bag"], case["max_bag"])
        raw = _ids62(g, seg.shape[0], case["zipf"], t)
        if case["ids"] != "hash":
            raw = (raw % case["rows"]).to(torch.int64 if case["ids"] == "i64" else torch.int32)
        ids.append(raw)
        segs.append(seg)
    return tabs, ids, segs


def _reduce_inputs(case, seed):
    g = _gen(seed)
    tab = torch.rand((case["rows"], case["dim"]), device="cuda", generator=g) * 0.1 - 0.05
    seg = _bags(g, case["batch"], 1, case["max_bag"])
    rows = _ids62(g, seg.shape[0], case["zipf"], 0) % case["rows"]
    return tab, (rows if case["ids"] == "i64" else rows.to(torch.int32)), seg


def _matmul_inputs(case, seed):
    g = _gen(seed)
    m, k, n = case["m"], case["k"], case["n"]
    if case["kind"] == "layout_matmul":
        return _normal(g, m, k), _normal(g, k, n, scale=1 / 64)
    x = torch.rand((m, k), device="cuda", generator=g) * 2 - 1
    w = _normal(g, k, n, scale=1 / 32)
    addend = _normal(g, n, scale=0.1).expand(m, n).contiguous()
    return x, w, addend


def _bmm_inputs(case, seed):
    g = _gen(seed)
    b, m, k, n = case["b"], case["m"], case["k"], case["n"]
    if case["kind"] == "bmm_softmax":
        return _normal(g, b, m, k, scale=1 / 8), _normal(g, b, k, n, scale=1 / 8)
    rhs = _normal(g, b, k, n, scale=k ** -0.5) if case["rhs_batched"] else _normal(g, k, n, scale=k ** -0.5)
    return _normal(g, b, m, k), rhs, _normal(g, n, scale=0.1)


def _mlp_inputs(case, seed):
    """Activations and weights as fp32 values that bf16 holds exactly (the bf16 copies are the inputs)."""
    g = _gen(seed)
    sizes = (case["k"], case["h1"], case["h2"], 1)
    x = (_normal(g, case["batch"], case["k"], scale=0.05)).to(torch.bfloat16)
    layers = [(_normal(g, a, b, scale=a ** -0.5), _normal(g, b, scale=0.01)) for a, b in zip(sizes, sizes[1:])]
    return x, layers


# ---------------------------------------------------------------- what a user's program has in hand

def prepare(case, seed):
    kind = case["kind"]
    if kind == "dlrm":
        d = _dlrm_inputs(case, seed)
        host = lambda t: t.cpu().numpy()
        bags = [synth.BagInputs(host(i), host(s)) for i, s in d["bags"]]
        emb = synth.EmbeddingWorkload([host(t) for t in d["tables"]], bags, case["batch"], 64)
        layers = lambda ls: [(host(w), host(b)) for w, b in ls]
        model = synth.DlrmModel(layers(d["bottom"]), layers(d["top"]), emb, host(d["dense"]),
                                [t.shape[0] for t in d["tables"]])
        del d
        return kind, DlrmPipeline(model, torch.device("cuda", torch.cuda.current_device()))
    if kind == "bags":
        tabs, ids, segs = _bag_inputs(case, seed)
        out = torch.empty((case["batch"], case["tables"], case["dim"]), device="cuda")
        plan = dev.BagPlan(tabs, ids, segs, out, 0, case["batch"], id_kind={"i32": 0, "i64": 1, "hash": 2}[case["ids"]],
                           col=0, combiner=int(case["mean"]))
        return kind, plan
    if kind == "segment_reduce":
        tab, rows, seg = _reduce_inputs(case, seed)
        return kind, (tab, rows, seg, np.zeros(2, np.int32), np.zeros(1, np.int32), int(case["mean"]))
    if kind == "gather_unique":
        g = _gen(seed)
        tab = torch.rand((case["rows"], case["dim"]), device="cuda", generator=g) * 0.1 - 0.05
        # as many different keys as such a column has on average, each at least once, the rest by popularity
        n, u = case["nnz"], _unique_keys(case)
        pool = torch.randperm(case["rows"], device="cuda", generator=g)[:u]
        keys = torch.cat([pool, pool[_ranks(g, n - u, case["zipf"]) % u]])[torch.randperm(n, device="cuda", generator=g)]
        keys = torch.stack([torch.arange(case["nnz"], device="cuda"), keys], 1).contiguous()
        return kind, (tab, keys, np.array([0, 1], np.int32))
    if kind == "matmul_add_relu":
        x, w, addend = _matmul_inputs(case, seed)
        return kind, (torch.zeros_like(addend), addend, x, w)
    if kind == "layout_matmul":
        x, w = _matmul_inputs(case, seed)
        packed = dev.kn4_pack(w)
        return kind, (x, packed.cpu().numpy() if case["weight"] == "host" else packed)
    if kind in ("bmm_softmax", "bmm_sigmoid"):
        return kind, _bmm_inputs(case, seed)
    if kind == "mlp_bf16":
        x, layers = _mlp_inputs(case, seed)
        weights = [dev.bf16_weight(w) for w, _ in layers[:-1]] + [layers[-1][0]]
        bf, f32 = dict(dtype=torch.bfloat16, device="cuda"), dict(dtype=torch.float32, device="cuda")
        acts = [torch.empty((case["batch"], case["h1"]), **bf), torch.empty((case["batch"], case["h2"]), **f32),
                torch.empty((case["batch"], 1), **f32)]
        return kind, (x, list(zip(weights, [b for _, b in layers], [w.shape for w, _ in layers])), acts)
    raise ValueError(kind)


def run(state):
    kind, s = state
    if kind == "dlrm":
        return s.forward()
    if kind == "bags":
        s.run()
        return s.out
    if kind == "segment_reduce":
        return ops.kp_fused_sparse_segment_reduce(*s)
    if kind == "gather_unique":
        return ops.kp_fused_gather(*s)
    if kind == "matmul_add_relu":
        return ops.xla_matmul_add_relu(*s)
    if kind == "layout_matmul":
        return ops.xla_layout_matmul(*s)
    if kind == "bmm_softmax":
        return ops.xla_softmax(ops.xla_batch_matmul(*s))
    if kind == "bmm_sigmoid":
        return ops.kp_fused_batch_matmul_add_sigmoid(*s)
    x, layers, acts = s
    b = x.shape[0]
    for i, ((w, bias, (k, n)), y) in enumerate(zip(layers, acts)):
        if i == len(layers) - 1:
            dev.gemm(x, w, y, m=b, n=n, k=k, bias=bias, activation=ACT_SIGMOID, math=MATH_FP32)
        else:
            flags = IO_A_BF16 | IO_B_BF16 | (IO_C_BF16 if y.dtype == torch.bfloat16 else 0)
            dev.gemm(x, w, y, m=b, n=n, k=k, trans_b=True, bias=bias, activation=ACT_RELU, math=MATH_BF16,
                     io_flags=flags)
        x = y
    return acts


# ---------------------------------------------------------------- what a pass cannot do without

def _distinct(n: float, rows: float, a: float) -> float:
    """Expected number of different table rows that n lookups of Zipf-like ids read."""
    edges = np.unique(np.floor(np.logspace(0, math.log10(_LUT), 400)))
    lo, hi = edges[:-1], edges[1:]
    t = a - 1.0
    tail = _LUT ** -t / _LUT
    p = (lo ** -t - hi ** -t) / (hi - lo) + tail
    ids = float(((hi - lo) * -np.expm1(-n * p)).sum())
    return rows * -math.expm1(-ids / rows)


def _unique_keys(case):
    return max(1, min(case["nnz"], int(_distinct(case["nnz"], case["rows"], case["zipf"]))))


def _bag_bytes(tables, rows, dim, batch, mean_bag, id_bytes, a):
    n = batch * mean_bag
    return tables * (n * (id_bytes + 8) + _distinct(n, rows, a) * 4 * dim + batch * 4 * dim)


def work(case):
    kind = case["kind"]
    if kind == "dlrm":
        b, mean_bag = case["batch"], (1 + case["max_bag"]) / 2
        us = np.linspace(3.0, math.log10(case["max_rows"]), 26)
        n = b * mean_bag
        emb = sum(n * 16 + _distinct(n, 10 ** u, 1.05) * 256 for u in us)
        weights = 13 * 512 + 512 * 256 + 256 * 64 + 415 * 512 + 512 * 256 + 256
        return {"bytes": emb + b * (13 + 1) * 4 + weights * 4, "flops": b * (2.0 * weights + 27 * 26 * 64 + 26 * mean_bag * 64)}
    if kind == "bags":
        mean_bag = (case["min_bag"] + case["max_bag"]) / 2
        n = case["tables"] * case["batch"] * mean_bag
        return {"bytes": _bag_bytes(case["tables"], case["rows"], case["dim"], case["batch"], mean_bag,
                                    4 if case["ids"] == "i32" else 8, case["zipf"]), "flops": n * case["dim"]}
    if kind == "segment_reduce":
        mean_bag = (1 + case["max_bag"]) / 2
        return {"bytes": _bag_bytes(1, case["rows"], case["dim"], case["batch"], mean_bag,
                                    4 if case["ids"] == "i32" else 8, case["zipf"]),
                "flops": case["batch"] * mean_bag * case["dim"]}
    if kind == "gather_unique":
        u = _unique_keys(case)
        return {"bytes": case["nnz"] * (8 + 4) + u * (8 + 8 * case["dim"]), "flops": 0}
    if kind in ("matmul_add_relu", "layout_matmul"):
        m, k, n = case["m"], case["k"], case["n"]
        c = 2 if kind == "matmul_add_relu" else 1
        return {"bytes": 4 * (m * k + k * n + c * m * n), "flops": 2.0 * m * n * k}
    if kind == "bmm_softmax":
        b, m, k, n = case["b"], case["m"], case["k"], case["n"]
        return {"bytes": 4 * b * (m * k + k * n + m * n), "flops": 2.0 * b * m * n * k}
    if kind == "bmm_sigmoid":
        b, m, k, n = case["b"], case["m"], case["k"], case["n"]
        return {"bytes": 4 * (b * m * k + (b if case["rhs_batched"] else 1) * k * n + n + b * m * n),
                "flops": 2.0 * b * m * n * k}
    b, k, h1, h2 = case["batch"], case["k"], case["h1"], case["h2"]
    return {"bytes": 2 * (b * k + k * h1 + h1 * h2 + b * h1) + 4 * (b * h2 + h2 + b),
            "flops": 2.0 * b * (k * h1 + h1 * h2 + h2)}


# ---------------------------------------------------------------- results

def tolerance(case):
    """About four times the distance to exact() measured over the ranges."""
    kind = case["kind"]
    if kind == "gather_unique":
        return "exact"  # whole numbers and copied rows
    if kind in ("bags", "segment_reduce"):
        return {"rel": 4e-7, "max": 1e-5}  # fp32 sums of up to 50 rows (8e-8 measured)
    if kind == "bmm_sigmoid":
        return {"rel": 1e-6, "max": 1e-5}  # fp32 sums, the sigmoid in fp32 (3e-7)
    if kind == "dlrm":
        return {"rel": 4e-4, "max": 5e-3}  # TF32 layers and the TF32 interaction under a sigmoid (9e-5)
    if kind == "bmm_softmax":
        return {"rel": 4e-4, "max": 5e-3}  # TF32 products under a softmax (1e-4)
    if kind == "mlp_bf16":
        return {"rel": 7e-3, "max": 5e-2}  # bf16 activations between the layers (1.7e-3)
    return {"rel": 3e-3, "max": 1.5e-2}    # TF32 products, fp32 sums (8e-4)


def _exact_bags(tab, rows, seg, batch, mean):
    out = torch.zeros((batch, tab.shape[1]), dtype=torch.float64, device="cuda")
    out.index_add_(0, seg[:, 0], tab[rows.long()].double())
    if mean:
        lens = torch.bincount(seg[:, 0], minlength=batch).clamp(min=1)
        out /= lens[:, None]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "dlrm":
        d = _dlrm_inputs(case, seed)
        x = d["dense"].double()
        for w, b in d["bottom"]:
            x = torch.relu(x @ w.double() + b.double())
        z = [x]
        for tab, (ids, seg) in zip(d["tables"], d["bags"]):
            z.append(_exact_bags(tab, ids % tab.shape[0], seg, case["batch"], False))
        z = torch.stack(z, 1)
        i, j = torch.tril_indices(27, 27, offset=-1, device="cuda")
        outs = []
        for part in z.split(8192):
            y = torch.cat([part[:, 0], torch.bmm(part, part.transpose(1, 2))[:, i, j]], 1)
            for k, (w, b) in enumerate(d["top"]):
                y = y @ w.double() + b.double()
                y = torch.sigmoid(y) if k == 2 else torch.relu(y)
            outs.append(y)
        return torch.cat(outs)
    if kind == "bags":
        tabs, ids, segs = _bag_inputs(case, seed)
        out = torch.empty((case["batch"], case["tables"], case["dim"]), dtype=torch.float64, device="cuda")
        for t in range(case["tables"]):
            out[:, t] = _exact_bags(tabs[t], ids[t] % case["rows"], segs[t], case["batch"], case["mean"])
        return out
    if kind == "segment_reduce":
        tab, rows, seg = _reduce_inputs(case, seed)
        return _exact_bags(tab, rows, seg, case["batch"], case["mean"]), None
    if kind == "gather_unique":
        return None
    if kind == "matmul_add_relu":
        x, w, addend = _matmul_inputs(case, seed)
        return torch.relu(x.double() @ w.double() + addend.double())
    if kind == "layout_matmul":
        x, w = _matmul_inputs(case, seed)
        return x.double() @ w.double()
    if kind == "bmm_softmax":
        q, kt = _bmm_inputs(case, seed)
        return torch.softmax(torch.bmm(q.double(), kt.double()), -1)
    if kind == "bmm_sigmoid":
        lhs, rhs, bias = _bmm_inputs(case, seed)
        return torch.sigmoid(torch.matmul(lhs.double(), rhs.double()) + bias.double())
    x, layers = _mlp_inputs(case, seed)
    y, outs = x.double(), []
    for i, (w, b) in enumerate(layers):
        w = w.to(torch.bfloat16).double() if i < 2 else w.double()
        y = y @ w + b.double()
        y = torch.sigmoid(y) if i == 2 else torch.relu(y)
        outs.append(y)
    return outs
