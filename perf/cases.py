"""The framework's work as a list of cases, each one pass through a public
entry point: the relational folds and pipelines of ``einfold_b200.kernels``
over host and device tables, the tensor-level attention and products of
``einfold_b200.autograd``, and the ranking entry of the C ABI.

``listed()`` holds the cases, ``draw(rng)`` gives another one of the same
ranges, ``prepare(case, seed)`` the inputs, ``run(state)`` one pass and its
outputs, ``work(case)`` the bytes and operations a pass cannot do without,
and ``exact(case, seed)`` the outputs as plain torch or numpy computes them
in 64 bits.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import pyarrow as pa
import torch

from einfold_b200 import _lib, ir
from einfold_b200 import autograd as A
from einfold_b200 import cases as C
from einfold_b200 import kernels as K
from einfold_b200 import synthetic as S


def listed():
    return [
        # A small GROUP BY product between two tables in host memory, rows
        # shuffled and in four batches each: what a query engine hands over
        # for an ordinary query. Latency, copies and launches count.
        {"name": "fold_host_512", "kind": "fold_host", "m": 512, "k": 512, "n": 256, "nulls": False},
        # The same fold at the size of the headline benchmark, tables and
        # result in HBM.
        {"name": "fold_device_8192", "kind": "fold_device", "m": 8192, "k": 8192, "n": 8192},
        # A sparse contraction on keys that are no positions (strings and
        # hashes with Zipf frequencies): ranking, sorting, grouped sums.
        {"name": "fold_sorted_50000", "kind": "fold_sorted", "rows": 50000},
        # Dense ranking of 64-bit keys with repeats, the step under every
        # join and group of the sorting path.
        {"name": "rank_64m", "kind": "rank", "rows": 1 << 26},
        # A training step's attention at a short odd length: launches and
        # host round trips count.
        {"name": "attention_train_short", "kind": "attention", "batch": 2, "heads": 3, "tq": 100, "tk": 100, "d": 32,
         "mask": "causal", "precision": "split", "backward": True},
        # The headline benchmark's causal attention, forward and backward.
        {"name": "attention_train_4096", "kind": "attention", "batch": 4, "heads": 16, "tq": 4096, "tk": 4096, "d": 64,
         "mask": "causal", "precision": "split", "backward": True},
        # One query a group against a long table of keys, as in decoding or a
        # lookup.
        {"name": "attention_one_query", "kind": "attention", "batch": 2, "heads": 8, "tq": 1, "tk": 8191, "d": 64,
         "mask": "none", "precision": "split", "backward": False},
        # Groups of very different lengths in a window, padded to the longest.
        {"name": "attention_ragged", "kind": "ragged", "groups": 64, "d": 128, "window": 512},
        # The FP64 form of the attention, asked for by precision=FP64.
        {"name": "attention_train_fp64", "kind": "attention", "batch": 2, "heads": 16, "tq": 2048, "tk": 2048, "d": 64,
         "mask": "causal", "precision": "fp64", "backward": True},
        # A layer's batched products with their gradients, odd sizes.
        {"name": "matmul_train_batched", "kind": "matmul", "batch": 6, "m": 333, "k": 450, "n": 201,
         "precision": "split", "backward": True},
        # Attention as a relational pipeline over tables in HBM (placement,
        # kernels, result assembly).
        {"name": "pipeline_attention", "kind": "pipeline", "batch": 2, "heads": 4, "t": 1000, "d": 64},
        # The Gaussian smoother: row-expression scores, unshifted weights.
        {"name": "smoother_64x1m", "kind": "smoother", "groups": 64, "x": 1 << 20, "y": 256},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["fold_host", "fold_device", "fold_sorted", "rank", "attention", "attention", "attention",
                       "ragged", "matmul", "pipeline", "smoother"])
    if kind == "fold_host":
        return {"kind": kind, "m": _log(rng, 8, 512), "k": _log(rng, 8, 512), "n": _log(rng, 8, 512),
                "nulls": rng.random() < 0.5}
    if kind == "fold_device":
        return {"kind": kind, "m": _log(rng, 64, 8192), "k": _log(rng, 64, 8192), "n": _log(rng, 64, 8192)}
    if kind == "fold_sorted":
        return {"kind": kind, "rows": _log(rng, 500, 50000)}
    if kind == "rank":
        return {"kind": kind, "rows": _log(rng, 1 << 12, 1 << 27)}
    if kind == "attention":
        precision = rng.choice(["split", "split", "fp64"])
        backward = rng.random() < 0.6
        d = rng.choice([16, 32, 40, 64])
        if not backward and rng.random() < 0.5:  # few queries, many keys
            return {"kind": kind, "batch": rng.randint(1, 4), "heads": rng.choice([1, 4, 8]), "tq": rng.randint(1, 16),
                    "tk": _log(rng, 500, 16384), "d": rng.choice([64, 128]), "mask": "none", "precision": "split",
                    "backward": False}
        t = _log(rng, 32, 3000)
        return {"kind": kind, "batch": rng.randint(1, 4), "heads": rng.choice([1, 3, 8]), "tq": t, "tk": t, "d": d,
                "mask": rng.choice(["causal", "causal", "window", "none"]), "precision": precision,
                "backward": backward}
    if kind == "ragged":
        return {"kind": kind, "groups": _log(rng, 4, 48), "d": rng.choice([64, 128]), "window": _log(rng, 64, 1024)}
    if kind == "matmul":
        precision = rng.choice(["split", "split", "split", "fp64"])
        top = 1024 if precision == "split" else 512
        return {"kind": kind, "batch": _log(rng, 1, 12), "m": _log(rng, 16, top), "k": _log(rng, 16, top),
                "n": _log(rng, 16, top), "precision": precision, "backward": rng.random() < 0.7}
    if kind == "pipeline":
        return {"kind": kind, "batch": rng.randint(1, 3), "heads": rng.choice([1, 2, 4]), "t": _log(rng, 50, 1500),
                "d": rng.choice([16, 32, 64])}
    return {"kind": kind, "groups": _log(rng, 1, 48), "x": _log(rng, 1000, 1 << 20), "y": _log(rng, 16, 256)}


# ---- the descriptions -------------------------------------------------------


def _product_fold():
    """SUM(a.v * b.v) GROUP BY i, k of a(i, j, v) and b(j, k, v)."""
    e = ir.EQ
    return ir.Fold([e, e, e], [ir.Operand([(0, 0), (1, 1)], 2), ir.Operand([(1, 0), (2, 1)], 2)],
                   [ir.Output(0), ir.Output(2)])


def _attention_pipeline():
    """Causal softmax attention over q(b, h, t, d, x), k(b, h, t, d, x) and
    v(b, h, t, c, x). Dimensions: 0 b, 1 h, 2 tq, 3 d, 4 tk, 5 c."""
    e = ir.EQ
    producer = ir.Fold([e] * 5, [ir.Operand([(0, 0), (1, 1), (2, 2), (3, 3)], 4),
                                 ir.Operand([(0, 0), (1, 1), (4, 2), (3, 3)], 4)],
                       [ir.Output(0), ir.Output(1), ir.Output(2), ir.Output(4)])
    producer = producer.with_conditions([ir.Condition(2, ir.Comparison.GREATER_OR_EQUAL, 4, 0)])
    return ir.Pipeline(producer, ir.Weight.exp(), [e], ir.Operand([(0, 0), (1, 1), (4, 2), (5, 3)], 4), [0, 1, 2, 5],
                       ir.Normalizer.KEPT_GROUPS)


def _conditions(case):
    if case["mask"] == "causal":
        return A.causal()
    if case["mask"] == "window":
        return A.window(max(1, case["tq"] // 8))
    return []


def _precision(case):
    return K.Precision.FP64 if case["precision"] == "fp64" else K.Precision.SPLIT


# ---- inputs -----------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(shape, g, sd=1.0):
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g) * sd


def _host_values(case, seed):
    """The host fold's values: a [m][k], b [k][n] uniform[-1, 1], and which
    of b's are NULL (1%, or none)."""
    rng = np.random.RandomState(seed)
    a = rng.uniform(-1, 1, (case["m"], case["k"]))
    b = rng.uniform(-1, 1, (case["k"], case["n"]))
    nulls = rng.uniform(size=b.shape) < 0.01 if case["nulls"] else np.zeros(b.shape, dtype=bool)
    return a, b, nulls, rng


def _host_relation(names, values, nulls, rng):
    """Every key pair with its value, rows shuffled, in four batches."""
    keys = np.indices(values.shape).reshape(2, -1)
    order = rng.permutation(values.size)
    cuts = [0, *sorted(rng.randint(0, values.size + 1, 3).tolist()), values.size]
    schema = pa.schema([(names[0], pa.int64()), (names[1], pa.int64()), ("v", pa.float64())])
    flat, mask = values.reshape(-1), None if nulls is None else nulls.reshape(-1)
    batches = []
    for lo, hi in zip(cuts[:-1], cuts[1:]):
        rows = order[lo:hi]
        v = pa.array(flat[rows], mask=None if mask is None else mask[rows])
        batches.append(pa.record_batch([pa.array(keys[0][rows]), pa.array(keys[1][rows]), v], schema=schema))
    return K.Relation(schema, batches)


def _grid_relation(names, extents, values):
    keys = S.grid_keys(extents)
    schema = pa.schema([(c, pa.int64()) for c in names] + [("x", pa.float64())])
    return K.DeviceRelation(schema, list(keys) + [values.reshape(-1)])


def _attention_inputs(case, seed):
    g = _generator(seed)
    lead = (case["batch"], case["heads"])
    q = _randn((*lead, case["tq"], case["d"]), g)
    k = _randn((*lead, case["tk"], case["d"]), g)
    v = _randn((*lead, case["tk"], case["d"]), g)
    d_out = _randn(q.shape, g) if case["backward"] else None
    return q, k, v, d_out


def _zipf(rng, n, pool, s=1.1):
    """n indices into a pool, index r drawn with frequency proportional to (r + 1)^-s."""
    cdf = np.cumsum(np.arange(1, pool + 1, dtype=np.float64) ** -s)
    return np.searchsorted(cdf / cdf[-1], rng.uniform(size=n), side="right").clip(0, pool - 1)


def _sorted_tables(case, seed):
    """a(i, j, v) and b(j, k, v): i and k 16-hex-digit strings, j 63-bit
    hashes with Zipf(1.1) frequencies, v normal(0, 1). Which rows share a key
    is the same for every seed (so results have the same size); the keys, the
    rows' order and the values are the seed's."""
    rows = case["rows"]
    law, rng = np.random.RandomState(0), np.random.RandomState(seed)
    words = [rng.randint(0, 1 << 62, n, dtype=np.int64).astype(np.uint64) for n in (rows, rows, 4 * rows)]
    hashes = words[2].astype(np.int64)
    picks = [(law.randint(0, rows, rows), _zipf(law, rows, 4 * rows)) for _ in range(2)]
    (ia, ja), (kb, jb) = ((p[order], z[order]) for p, z in picks for order in [rng.permutation(rows)])
    va, vb = rng.normal(size=rows), rng.normal(size=rows)
    a = pa.record_batch([S.hex_strings(words[0][ia]), pa.array(hashes[ja]), pa.array(va)], names=["i", "j", "v"])
    b = pa.record_batch([pa.array(hashes[jb]), S.hex_strings(words[1][kb]), pa.array(vb)], names=["j", "k", "v"])
    return a, b


def _ragged_inputs(case, seed):
    """q, k, v [groups][longest][d], zero past each group's length: the
    lengths of C.ragged_lengths (log-uniform in [128, 8192]) in an order of
    the seed's."""
    g = _generator(seed)
    lengths = C.ragged_lengths(case["groups"])
    lengths = lengths[torch.from_numpy(np.random.RandomState(seed).permutation(case["groups"]))]
    shape = (case["groups"], int(lengths.max()), case["d"])
    pad = torch.arange(shape[1], device="cuda")[None, :, None] >= lengths.cuda()[:, None, None]
    q, k, v = (_randn(shape, g).masked_fill_(pad, 0.0) for _ in range(3))
    return q, k, v, lengths


def _matmul_inputs(case, seed):
    g = _generator(seed)
    a = _randn((case["batch"], case["m"], case["k"]), g)
    b = _randn((case["batch"], case["k"], case["n"]), g, case["k"] ** -0.5)
    d_c = _randn((case["batch"], case["m"], case["n"]), g) if case["backward"] else None
    return a, b, d_c


def _pipeline_inputs(case, seed):
    g = _generator(seed)
    shape = (case["batch"], case["heads"], case["t"], case["d"])
    return [_randn(shape, g, sd) for sd in (1 / 8, 1.0, 1.0)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fold_host":
        a, b, nulls, rng = _host_values(case, seed)
        return {"kind": "fold", "fold": _product_fold(), "a": _host_relation(["i", "j"], a, None, rng),
                "b": _host_relation(["j", "k"], b, nulls if case["nulls"] else None, rng), "options": K.Options()}
    if kind == "fold_device":
        g = _generator(seed)
        u = [torch.rand(shape, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
             for shape in ((case["m"], case["k"]), (case["k"], case["n"]))]
        return {"kind": "fold", "fold": _product_fold(),
                "a": _grid_relation(["i", "j"], list(u[0].shape), u[0]),
                "b": _grid_relation(["j", "k"], list(u[1].shape), u[1]), "options": K.Options(result_on_device=True)}
    if kind == "fold_sorted":
        a, b = _sorted_tables(case, seed)
        return {"kind": "fold", "fold": _product_fold(), "a": K.Relation(a.schema, [a]),
                "b": K.Relation(b.schema, [b]), "options": K.Options(result_on_device=True)}
    if kind == "rank":
        n = case["rows"]
        # Keys drawn from a pool of n/2: which rows share one is the same for
        # every seed, the keys and the rows' order are the seed's.
        pool = S.u64(seed, 7, n // 2)
        pick = (S.u64(0, 8, n) % (n // 2))[torch.randperm(n, device="cuda", generator=_generator(seed))]
        return {"kind": kind, "words": pool[pick].contiguous(),
                "rank": torch.empty(n, dtype=torch.int32, device="cuda"),
                "first": torch.empty(n, dtype=torch.int32, device="cuda")}
    if kind == "attention":
        q, k, v, d_out = _attention_inputs(case, seed)
        for t in (q, k, v):
            t.requires_grad_(case["backward"])
        return {"kind": kind, "q": q, "k": k, "v": v, "d_out": d_out, "conditions": _conditions(case),
                "scale": case["d"] ** -0.5, "precision": _precision(case)}
    if kind == "ragged":
        q, k, v, lengths = _ragged_inputs(case, seed)
        return {"kind": kind, "q": q, "k": k, "v": v, "lengths": lengths, "conditions": A.window(case["window"]),
                "scale": case["d"] ** -0.5}
    if kind == "matmul":
        a, b, d_c = _matmul_inputs(case, seed)
        for t in (a, b):
            t.requires_grad_(case["backward"])
        return {"kind": kind, "a": a, "b": b, "d_c": d_c, "precision": _precision(case)}
    if kind == "pipeline":
        q, k, v = _pipeline_inputs(case, seed)
        rels = [_grid_relation(["b", "h", "t", d], list(x.shape), x) for x, d in ((q, "d"), (k, "d"), (v, "c"))]
        return {"kind": "pipeline", "pipeline": _attention_pipeline(), "operands": rels}
    q, k, v, _, _, _ = C.smoother_tables(case["groups"], case["x"], case["y"], seed)
    return {"kind": "pipeline", "pipeline": C.smoother_pipeline(0.01), "operands": [q, k, v]}


# ---- one pass ---------------------------------------------------------------


def _column(array):
    """A host result column's values (and validity, where some are NULL), or
    a string column's offsets and bytes, without a copy of the buffers."""
    values = np.asarray(array.fill_null(0)) if array.null_count else array.to_numpy(zero_copy_only=True)
    return [values, np.asarray(array.is_valid())] if array.null_count else values


def _device_batch(batch):
    return [list(batch.strings(i)) if batch.formats[i] in (b"u", b"z") else batch.column(i)
            for i in range(len(batch.formats))]


def run(state):
    kind = state["kind"]
    if kind == "fold":
        got = K.fold(state["fold"], state["a"], state["b"], options=state["options"])
        if state["options"].result_on_device:
            return [_device_batch(b) for b in got.batches]
        return [[_column(c) for c in b.columns] for b in got.batches]
    if kind == "rank":
        words, distinct = state["words"], ctypes.c_int64(0)
        stream = torch.cuda.current_stream().cuda_stream or 1
        status = _lib.load().einfold_rank_words(_lib.context(0), words.data_ptr(), words.numel(),
                                                state["rank"].data_ptr(), state["first"].data_ptr(),
                                                ctypes.byref(distinct), ctypes.c_void_p(stream))
        if status != _lib.OK:
            raise RuntimeError(_lib.load().einfold_last_error().decode())
        return [state["rank"], state["first"][:distinct.value], distinct.value]
    if kind == "attention":
        q, k, v = state["q"], state["k"], state["v"]
        if state["d_out"] is None:
            return list(A.attention_forward(q, k, v, state["conditions"], state["scale"], state["precision"]))
        out = A.attention(q, k, v, state["conditions"], state["scale"], state["precision"])
        return [out, *torch.autograd.grad(out, (q, k, v), state["d_out"])]
    if kind == "ragged":
        return list(A.attention_forward(state["q"], state["k"], state["v"], state["conditions"], state["scale"],
                                        q_lengths=state["lengths"], k_lengths=state["lengths"]))
    if kind == "matmul":
        c = A.matmul(state["a"], state["b"], state["precision"])
        if state["d_c"] is None:
            return c
        return [c, *torch.autograd.grad(c, (state["a"], state["b"]), state["d_c"])]
    got = K.pipeline(state["pipeline"], state["operands"], options=K.Options(result_on_device=True))
    return [_device_batch(b) for b in got.batches]


# ---- what a pass cannot do without ------------------------------------------


def _pairs(tq, tk, mask):
    if mask == "causal":
        return sum(min(x + 1, tk) for x in range(tq))
    if mask == "window":
        r = max(1, tq // 8)
        return sum(max(0, min(x + r, tk - 1) - max(x - r, 0) + 1) for x in range(tq))
    return tq * tk


def work(case):
    kind = case["kind"]
    if kind in ("fold_host", "fold_device"):
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 24 * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    if kind == "fold_sorted":
        a, b = _sorted_tables(case, 0)
        pairs = S.joined_pairs(a.column(1).to_numpy(), b.column(0).to_numpy())
        # Nearly every pair is a group of its own: two 16-byte strings, their
        # offsets and a value each.
        return {"bytes": 2 * 36 * case["rows"] + 48 * pairs, "flops": 2 * pairs}
    if kind == "rank":
        return {"bytes": 14 * case["rows"], "flops": 0}
    if kind == "attention":
        groups, tq, tk, d = case["batch"] * case["heads"], case["tq"], case["tk"], case["d"]
        pairs = groups * _pairs(tq, tk, case["mask"])
        once = 8 * d * groups * (2 * tq + 2 * tk)
        if not case["backward"]:
            return {"bytes": once + 8 * groups * tq, "flops": 4 * d * pairs}
        return {"bytes": once + 8 * d * groups * (2 * tq + 2 * tk), "flops": 14 * d * pairs}
    if kind == "ragged":
        lengths = C.ragged_lengths(case["groups"])
        rows, pairs = int(lengths.sum()), C.allowed_pairs(lengths, case["window"])
        return {"bytes": 8 * rows * (4 * case["d"] + 1), "flops": 4 * case["d"] * pairs}
    if kind == "matmul":
        b, m, k, n = case["batch"], case["m"], case["k"], case["n"]
        once, times = m * k + k * n + m * n, 3 if case["backward"] else 1
        return {"bytes": 8 * b * once * (2 if case["backward"] else 1), "flops": 2 * times * b * m * k * n}
    if kind == "pipeline":
        groups, t, d = case["batch"] * case["heads"], case["t"], case["d"]
        return {"bytes": 4 * 40 * groups * t * d, "flops": 4 * d * groups * _pairs(t, t, "causal")}
    rows, keys = case["groups"] * case["x"], case["groups"] * case["y"]
    # A subtraction, a square, a division, an exponential and two sums a pair.
    return {"bytes": (32 + 24) * rows + 56 * keys, "flops": 7 * rows * case["y"]}


# ---- the same in 64 bits by plain torch and numpy ----------------------------


def _softmax_average(q, k, v, scale, allowed):
    s = scale * (q @ k.transpose(-1, -2))
    if allowed is not None:
        s = s.masked_fill(~allowed, float("-inf"))
    lse = torch.logsumexp(s, dim=-1)
    return torch.exp(s - lse[..., None]) @ v, lse


def _allowed(tq, tk, mask):
    if mask == "none":
        return None
    x = torch.arange(tq, device="cuda")[:, None]
    j = torch.arange(tk, device="cuda")[None, :]
    return x >= j if mask == "causal" else (x - j).abs() <= max(1, tq // 8)


def _exact_attention(case, seed):
    q, k, v, d_out = _attention_inputs(case, seed)
    allowed = _allowed(case["tq"], case["tk"], case["mask"])
    scale = case["d"] ** -0.5
    flat = [None if t is None else t.flatten(0, 1) for t in (q, k, v, d_out)]
    parts = []
    for g in range(flat[0].shape[0]):
        qg, kg, vg = (t[g].clone().requires_grad_(case["backward"]) for t in flat[:3])
        out, lse = _softmax_average(qg, kg, vg, scale, allowed)
        if case["backward"]:
            parts.append([out.detach(), *torch.autograd.grad(out, (qg, kg, vg), flat[3][g])])
        else:
            parts.append([out, lse])
    return [torch.stack(p).unflatten(0, q.shape[:2]) for p in zip(*parts)]


def _exact_sorted(case, seed):
    a, b = _sorted_tables(case, seed)
    _, ri = np.unique(np.array(a.column(0).to_pylist(), dtype="S16"), return_inverse=True)
    names, rk = np.unique(np.array(b.column(1).to_pylist(), dtype="S16"), return_inverse=True)
    jb = b.column(0).to_numpy()
    order = np.argsort(jb, kind="stable")
    lo = np.searchsorted(jb[order], a.column(1).to_numpy(), side="left")
    count = np.searchsorted(jb[order], a.column(1).to_numpy(), side="right") - lo
    gpu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    lo, count, ri, rk = gpu(lo), gpu(count), gpu(ri), gpu(rk[order])
    left = torch.repeat_interleave(torch.arange(len(count), device="cuda"), count)
    begin = torch.cumsum(count, 0) - count
    right = lo[left] + torch.arange(left.numel(), device="cuda") - begin[left]
    groups, inverse = torch.unique(ri[left] * len(names) + rk[right], return_inverse=True)
    products = gpu(a.column(2).to_numpy())[left] * gpu(b.column(2).to_numpy()[order])[right]
    return torch.zeros(groups.numel(), dtype=torch.float64, device="cuda").index_add_(0, inverse, products)


def exact(case, seed):
    kind = case["kind"]
    if kind == "fold_host":
        a, b, nulls, _ = _host_values(case, seed)
        return [[None, None, (a @ np.where(nulls, 0.0, b)).reshape(-1)]]
    if kind == "fold_device":
        g = _generator(seed)
        a, b = [torch.rand(shape, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
                for shape in ((case["m"], case["k"]), (case["k"], case["n"]))]
        return [[None, None, (a @ b).reshape(-1)]]
    if kind == "fold_sorted":
        return [[None, None, _exact_sorted(case, seed)]]
    if kind == "rank":
        return None
    if kind == "attention":
        return _exact_attention(case, seed)
    if kind == "ragged":
        q, k, v, lengths = _ragged_inputs(case, seed)
        out = torch.full_like(q, float("nan"))
        lse = torch.full(q.shape[:-1], float("nan"), dtype=torch.float64, device="cuda")
        for g, t in enumerate(lengths.tolist()):
            x = torch.arange(t, device="cuda")
            near = (x[:, None] - x[None, :]).abs() <= case["window"]
            out[g, :t], lse[g, :t] = _softmax_average(q[g, :t], k[g, :t], v[g, :t], case["d"] ** -0.5, near)
        return [out, lse]
    if kind == "matmul":
        a, b, d_c = _matmul_inputs(case, seed)
        if d_c is None:
            return a @ b
        return [a @ b, d_c @ b.transpose(-1, -2), a.transpose(-1, -2) @ d_c]
    if kind == "pipeline":
        q, k, v = _pipeline_inputs(case, seed)
        out, _ = _softmax_average(q, k, v, 1.0, _allowed(case["t"], case["t"], "causal"))
        return [[None] * 4 + [out.reshape(-1)]]
    _, _, _, xs, ys, vs = C.smoother_tables(case["groups"], case["x"], case["y"], seed)
    groups, y = case["groups"], case["y"]
    out = torch.empty_like(xs).view(groups, -1)
    step = max(1, (1 << 27) // y)
    for g in range(groups):
        x, yg, vg = xs.view(groups, -1)[g], ys.view(groups, y)[g], vs.view(groups, y)[g]
        for at in range(0, x.numel(), step):
            w = torch.exp(-((x[at:at + step, None] - yg) ** 2) / 0.01)
            out[g, at:at + step] = (w @ vg) / w.sum(1)
    return [[None, None, out.reshape(-1)]]
