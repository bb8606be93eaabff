"""The workloads this library is measured on: the searches, the permutation and extension
filters, the canonical form, the extend step and the ordering model's training step, each
through the public entry point a program calls.

``listed()`` names the fixed cases, ``draw(rng)`` gives further ones of the same ranges.
``prepare(case, seed)`` makes what a program holds before the call (inputs, slot, model),
``run(state)`` makes one pass and returns its outputs, ``work(case)`` counts the bytes and
operations no implementation can do without and ``exact(case, seed)`` computes the floating
outputs in 64 bits with torch, numpy or plain Python.

A search returns verdicts (and, for staged calls, the depth that decided them), not the
sequences: warps race, so which of the valid sequences comes back differs between two runs
of one build.
"""
from __future__ import annotations

import ctypes
import math
import struct
import zlib

import numpy as np
import torch

from tdp1375_b200 import api, extensions, frontier, native, order_model
from tdp1375_b200.cases import MIN_RATE, config_cases, three_permutation

RATE = float(MIN_RATE)
QUEUE_BYTES = 3000 << 20
TABLE_2M = 1 << 21   # the drop-in's table
TABLE_2P26 = 1 << 26  # the proof driver's table
TABLE_2P28 = 1 << 28  # the learned evaluation's table
TABLE_2P30 = 1 << 30  # the batched evaluation's table
MAX_ROWS = 1 << 20   # rows the reference's filter returns at most
vp = ctypes.c_void_p


def listed():
    return [
        # the proof generator's smallest nodes: two bad small components, depths 4 and 5, one
        # native call per depth (latency of a call)
        {"name": "calls_small", "kind": "calls", "components": 2, "big": 0, "count": 8, "table": TABLE_2M},
        # the combination step's configurations (3-norm above 8, n up to about 40, both sides of the
        # 32-symbol layout), staged to depth 11
        {"name": "calls_comb", "kind": "calls", "components": 0, "big": 1, "count": 8, "table": TABLE_2M},
        # 3-permutations of 4..6 cycles, full sorting: the parity workload of the CPU path
        {"name": "batch_full_m4_6", "kind": "batch", "m_lo": 4, "m_hi": 6, "count": 1000, "depth": 11, "full": 1,
         "levels": 0, "table": TABLE_2M},
        # the drop-in range up to 8 cycles, two of the largest: a few exhaustive searches fill the chip
        {"name": "batch_full_m4_8", "kind": "batch", "m_lo": 4, "m_hi": 7, "top": 8, "tops": 2, "count": 40,
         "depth": 11, "full": 1, "levels": 0, "table": TABLE_2P30},
        # many uneven instances (geometric m in 3..10, 10% random permutations), partial mode
        {"name": "batch_uneven", "kind": "uneven", "count": 8192, "depth": 11, "table": TABLE_2P28},
        # 3..10 cycles under the learned order: features, tensor-core MLP, sort, search
        {"name": "batch_learned", "kind": "batch", "m_lo": 3, "m_hi": 10, "count": 2000, "depth": 11, "full": 0,
         "levels": 1, "table": TABLE_2P28},
        # the permutation filter at an interactive size and at the size of the benchmark
        {"name": "pi_filter_n9", "kind": "pi_filter", "n": 9, "cycle": 5, "skip": 0},
        {"name": "pi_filter_n12", "kind": "pi_filter", "n": 12, "cycle": 7, "skip": 0},
        # every one-3-cycle extension of 1,000 bases of six 3-cycles
        {"name": "extension_filter", "kind": "extension_filter", "m": 6, "count": 1000, "unoriented": 0},
        # canonical form of a large frontier
        {"name": "canonical", "kind": "canonical", "m_lo": 3, "m_hi": 10, "count": 250_000},
        # the extend step over a level's bad cases
        {"name": "insertions", "kind": "insertions", "m_lo": 3, "m_hi": 8, "count": 500},
        # one optimiser step of the ordering model at the training batch
        {"name": "train_step", "kind": "train", "rows": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["calls", "calls", "batch", "batch", "uneven", "learned", "pi_filter", "pi_filter",
                       "extension_filter", "extension_filter", "canonical", "canonical", "insertions", "train"])
    if kind == "calls":
        if rng.random() < 0.5:
            return {"kind": "calls", "components": rng.randint(2, 3), "big": 0, "count": rng.randint(4, 12),
                    "table": TABLE_2M}
        return {"kind": "calls", "components": 0, "big": 1, "count": rng.randint(4, 9),
                "table": rng.choice([TABLE_2M, TABLE_2P26])}
    if kind == "batch":
        lo = rng.randint(3, 5)
        return {"kind": "batch", "m_lo": lo, "m_hi": rng.randint(lo, 6), "count": _log_int(rng, 100, 1000),
                "depth": rng.randint(9, 11), "full": rng.randint(0, 1), "levels": 0,
                "table": rng.choice([TABLE_2M, TABLE_2P26])}
    if kind == "uneven":
        return {"kind": "uneven", "count": _log_int(rng, 700, 8192), "depth": 11, "table": TABLE_2P28}
    if kind == "learned":
        return {"kind": "batch", "m_lo": 3, "m_hi": rng.randint(8, 10), "count": _log_int(rng, 300, 2000), "depth": 11,
                "full": 0, "levels": rng.randint(1, 2), "table": TABLE_2P28}
    if kind == "pi_filter":
        n = rng.randint(8, 12)
        return {"kind": "pi_filter", "n": n, "cycle": rng.randint(5, min(n, 9)), "skip": int(rng.random() < 0.25)}
    if kind == "extension_filter":
        if rng.random() < 0.5:  # random bases: nearly every extension is rejected
            return {"kind": "extension_filter", "m": rng.randint(3, 6), "count": _log_int(rng, 100, 1000),
                    "unoriented": 0}
        # bases without a 2-move inside a cycle, as the proof's bad cases
        return {"kind": "extension_filter", "m": rng.randint(3, 9), "count": _log_int(rng, 30, 1000),
                "unoriented": 1}
    if kind == "canonical":
        lo = rng.randint(2, 6)
        return {"kind": "canonical", "m_lo": lo, "m_hi": rng.randint(lo, 20), "count": _log_int(rng, 150, 100_000)}
    if kind == "insertions":
        lo = rng.randint(2, 5)
        return {"kind": "insertions", "m_lo": lo, "m_hi": rng.randint(lo, 9), "count": _log_int(rng, 20, 500)}
    return {"kind": "train", "rows": 8 * _log_int(rng, 64, 512)}


# ---------------------------------------------------------------- inputs
def _rng(case, seed):
    text = repr(sorted((k, v) for k, v in case.items() if k != "name"))
    return np.random.Generator(np.random.PCG64([seed, zlib.crc32(text.encode())]))


def _three_cycles(rng, count, m_lo, m_hi, unoriented=False):
    """`count` products of m disjoint 3-cycles (m uniform in m_lo..m_hi, pi the identity):
    rows of 64 successors, sizes, and the cycles' symbols in cycle order."""
    m = rng.integers(m_lo, m_hi + 1, size=count)
    width = 3 * m_hi
    keys = rng.random((count, width))
    keys[np.arange(width)[None, :] >= 3 * m[:, None]] = 2.0
    q = np.argsort(keys, axis=1).reshape(count, m_hi, 3)
    if unoriented:  # x > y > z along the cycle: no 2-move on its own symbols
        q = -np.sort(-q, axis=2)
    spi = np.zeros((count, 64), np.uint8)
    live = (np.arange(m_hi)[None, :] < m[:, None])
    for t in range(3):
        r, c = np.nonzero(live)
        spi[r, q[r, c, t]] = q[r, c, (t + 1) % 3]
    return spi, (3 * m).astype(np.uint8), q, live


def _component_chain(rng, components, big):
    """A configuration of the combination step: bad small components inserted into one another
    at random positions; `big`: until the 3-norm passes 8."""
    parts = [extensions._successor_of(t) for t in extensions.BAD_SMALL_COMPONENTS]
    spi, norm, used = [], 0, 0
    while (norm <= 8) if big else (used < components):
        comp = parts[int(rng.integers(0, len(parts) if big else 2))]
        at, k = int(rng.integers(0, len(spi) + 1)), len(comp)
        move = [x if x < at else x + k for x in range(len(spi))]
        out = [0] * (len(spi) + k)
        for x, y in enumerate(spi):
            out[move[x]] = move[y]
        for x, y in enumerate(comp):
            out[at + x] = at + y
        spi, used = out, used + 1
        norm = (len(spi) - frontier.odd_cycles(spi)) // 2
    return spi


# ---------------------------------------------------------------- what a program keeps
_kept = {"table": 0, "levels": None, "model": None}


def _slot(table):
    """One slot with the asked table, as a program creates once."""
    if _kept["table"] != table:
        _kept["table"] = 0
        api.GPUSortingSearch.destroySlots()
        api.GPUSortingSearch.initSlots(1, 1, QUEUE_BYTES, table)
        _kept.update(table=table, levels=0)


def _targets(q, live):
    """A training target per row: the positions of the first cycle that admits a 2-move on its
    own symbols (pi is the identity), else of the first cycle."""
    x, y, z = q[:, :, 0], q[:, :, 1], q[:, :, 2]
    cyclic = ((x > y).astype(int) + (y > z) + (z > x)) <= 1
    pick = np.argmax(cyclic & live, axis=1)
    s = np.sort(q[np.arange(len(q)), pick], axis=1)
    return order_model.LEX32[s[:, 0], s[:, 1], s[:, 2]].astype(np.int32)


def _order_model():
    if _kept["model"] is None:
        rng = np.random.Generator(np.random.PCG64(1375))
        spi, n, q, live = _three_cycles(rng, 16384, 8, 10)
        pi = np.where(np.arange(64)[None, :] < n[:, None], np.arange(64), 0).astype(np.uint8)
        model = order_model.OrderModel()
        order_model.train(model, spi, pi, n, _targets(q, live), epochs=8, batch=1024)
        _kept["model"] = model
    return _kept["model"]


def _set_levels(levels):
    if _kept["levels"] == levels:
        return
    if levels:
        _order_model().install(0, enable=True, levels=levels)
    elif native.load().tdp_enable_order_model(0, 0) != 0:
        raise RuntimeError(native.last_error())
    _kept["levels"] = levels


def prepare(case, seed):
    rng, kind = _rng(case, seed), case["kind"]
    if kind in ("calls", "batch", "uneven"):
        _slot(case["table"])
        _set_levels(case.get("levels", 0))
    if kind == "calls":
        calls = []
        for _ in range(case["count"]):
            spi = _component_chain(rng, case["components"], case["big"])
            ub = frontier.upper_bound(spi, MIN_RATE)
            depths = [4] + ([min(ub, 8)] if ub > 4 else []) + ([min(ub, 11)] if ub > 8 else [])
            calls.append((list(range(len(spi))), spi, frontier.odd_cycles(spi), depths))
        return {"run": _run_calls, "calls": calls}
    if kind == "batch":
        span = case["m_hi"] - case["m_lo"] + 1
        ms = [case["m_lo"] + i % span for i in range(case["count"])] + [case.get("top", 0)] * case.get("tops", 0)
        cases = [three_permutation(m, rng) for m in ms]
        return {"run": _run_batch, "count": len(cases),
                "instances": api.make_instances(cases, case["depth"], bool(case["full"]))}
    if kind == "uneven":
        cases = [c[:3] for c in config_cases(4, case["count"], start=int(rng.integers(1 << 40)))]
        return {"run": _run_batch, "count": len(cases), "instances": api.make_instances(cases, case["depth"], False)}
    if kind == "pi_filter":
        n = case["n"]
        cycle = [int(v) for v in rng.permutation(n)[:case["cycle"]]]
        triple = [int(v) for v in rng.permutation(n)[:3]]
        return {"run": _run_pi_filter, "n": n, "skip": case["skip"], "cycle": (ctypes.c_uint8 * len(cycle))(*cycle),
                "triple": (ctypes.c_uint8 * 3)(*triple), "rows": (ctypes.c_uint8 * (MAX_ROWS * n))()}
    if kind == "extension_filter":
        spi, n, _, _ = _three_cycles(rng, case["count"], case["m"], case["m"], bool(case["unoriented"]))
        pi = np.where(np.arange(64) < 3 * case["m"], np.arange(64), 0).astype(np.uint8)
        per = native.load().tdp_extension_count(3 * case["m"])
        return {"run": _run_extension_filter, "n": 3 * case["m"], "count": case["count"],
                "spi": torch.from_numpy(spi).cuda(), "pi": torch.from_numpy(np.tile(pi, (case["count"], 1))).cuda(),
                "keep": torch.zeros(case["count"] * per, dtype=torch.uint8, device="cuda")}
    if kind == "canonical":
        spi, n, _, _ = _three_cycles(rng, case["count"], case["m_lo"], case["m_hi"])
        return {"run": _run_canonical, "count": case["count"], "spi": torch.from_numpy(spi).cuda(),
                "n": torch.from_numpy(n).cuda(),
                "signature": torch.zeros((case["count"], 64), device="cuda"),
                "hash": torch.zeros(case["count"], dtype=torch.int32, device="cuda"),
                "variant": torch.zeros(case["count"], dtype=torch.int32, device="cuda")}
    if kind == "insertions":
        # half the configurations without a 2-move inside a cycle, as the bad cases are
        half = case["count"] // 2
        a = _three_cycles(rng, half, case["m_lo"], case["m_hi"], True)
        b = _three_cycles(rng, case["count"] - half, case["m_lo"], case["m_hi"])
        spi, n = np.concatenate([a[0], b[0]]), np.concatenate([a[1], b[1]])
        max_n = int(n.max())
        slots = case["count"] * int(native.load().tdp_insertion_extension_slots(max_n))
        return {"run": _run_insertions, "count": case["count"], "max_n": max_n, "spi": torch.from_numpy(spi).cuda(),
                "n": torch.from_numpy(n).cuda(),
                "gates": torch.zeros(case["count"], dtype=torch.int64, device="cuda"),
                "flags": torch.zeros(slots, dtype=torch.uint8, device="cuda"),
                "out": torch.zeros((slots, 64), dtype=torch.uint8, device="cuda")}
    x, n, target, model = _train_inputs(case, seed)
    return {"run": _run_train, "x": x, "n": n, "target": target, "model": model}


def _train_inputs(case, seed):
    """A batch of states with their targets, and a model in the middle of its training (biases
    and Adam moments away from zero)."""
    rng = _rng(case, seed)
    spi, n, q, live = _three_cycles(rng, case["rows"], 4, 10)
    pi = np.where(np.arange(64)[None, :] < n[:, None], np.arange(64), 0).astype(np.uint8)
    d_n = torch.from_numpy(n).cuda()
    x = order_model.features(torch.from_numpy(spi).cuda(), torch.from_numpy(pi).cuda(), d_n)
    model = order_model.OrderModel(seed=int(rng.integers(1 << 30)))
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 30)))
    for k in range(8):
        like = model.m[k]
        model.m[k] = torch.randn(like.shape, generator=g, device="cuda") * 1e-4
        model.v[k] = torch.rand(like.shape, generator=g, device="cuda") * 1e-7 + 1e-8
    for layer in range(4):
        model.bias[layer] = torch.randn(model.bias[layer].shape, generator=g, device="cuda") * 0.05
    model.step = 100
    return x, d_n, torch.from_numpy(_targets(q, live)).cuda(), model


# ---------------------------------------------------------------- one pass
def run(state):
    return state["run"](state)


def _check(rc):
    if rc < 0:
        raise RuntimeError(native.last_error())
    return rc


def _stream():
    return vp(torch.cuda.current_stream().cuda_stream)


def _run_calls(s):
    decided = []
    for pi, spi, even, depths in s["calls"]:
        at = 0
        for depth in depths:
            if api.GPUSortingSearch.searchForSortingSeq(pi, spi, even, RATE, depth, False, 0):
                at = depth
                break
        decided.append(at)
    return {"decided": np.array(decided, np.int32)}


def _run_batch(s):
    results = api.search_batch(0, s["instances"], s["count"], RATE)
    raw = np.frombuffer(results, np.int32).reshape(len(results), -1)
    return {"status": raw[:, 0]}


def _run_pi_filter(s):
    hits = _check(native.load().tdp_pi_filter(s["cycle"], len(s["cycle"]), s["triple"], 3, s["n"], s["skip"],
                                              s["rows"], MAX_ROWS))
    return {"hits": hits, "rows": np.frombuffer(s["rows"], np.uint8)}  # the first `hits` rows of n bytes


def _run_extension_filter(s):
    _check(native.load().tdp_extension_filter_device(vp(s["spi"].data_ptr()), vp(s["pi"].data_ptr()), s["n"],
                                                     s["count"], vp(s["keep"].data_ptr()), _stream()))
    return {"keep": s["keep"]}


def _run_canonical(s):
    _check(native.load().tdp_canonical_device(vp(s["spi"].data_ptr()), vp(s["n"].data_ptr()), s["count"],
                                              vp(s["signature"].data_ptr()), vp(s["hash"].data_ptr()),
                                              vp(s["variant"].data_ptr()), _stream()))
    return {"signature": s["signature"], "hash": s["hash"], "variant": s["variant"]}


def _run_insertions(s):
    _check(native.load().tdp_insertion_extensions_device(
        vp(s["spi"].data_ptr()), vp(s["n"].data_ptr()), s["count"], s["max_n"], vp(s["gates"].data_ptr()),
        vp(s["flags"].data_ptr()), vp(s["out"].data_ptr()), _stream()))
    return {"gates": s["gates"], "flags": s["flags"], "out": s["out"]}


def _run_train(s):
    model = s["model"]
    loss, top1 = model.train_step(s["x"], s["n"], s["target"])
    return {"loss": loss, "top1": top1, "master": model.master, "weight": model.weight, "bias": model.bias,
            "m": model.m, "v": model.v}


# ---------------------------------------------------------------- what a pass cannot do without
def _mean_insertions(case):
    """Slots and written rows per configuration: one row per multiset of three positions."""
    ns = [3 * m for m in range(case["m_lo"], case["m_hi"] + 1)]
    rows = sum((n + 2) * (n + 1) * n / 6 - n for n in ns) / len(ns)
    n = ns[-1]
    return (n + 2) * (n + 1) * n / 6, rows


def work(case):
    kind = case["kind"]
    if kind in ("calls", "batch", "uneven"):
        # instance in, result out; every root child judged once (three cycle words each).  How
        # many nodes lie below a root depends on the instance and is not counted.
        n = 3 * case["m_hi"] if kind == "batch" else 30 if kind == "uneven" or case["big"] else 6 * case["components"]
        return {"bytes": case["count"] * (136 + 208), "flops": case["count"] * 3.0 * (n * (n - 1) * (n - 2) // 6)}
    if kind == "pi_filter":
        # every hit written once is data-dependent; what is certain is the visit of the first
        # symbols' arrangements, counted as one operation per cycle arrangement
        return {"bytes": 64 + 8, "flops": float(math.perm(case["n"] - 1, min(case["n"] - 1, case["cycle"])))}
    if kind == "extension_filter":
        n = 3 * case["m"]
        per = 2 * math.comb(n, 3) + 2 * math.comb(n + 3, 3)
        return {"bytes": case["count"] * (128 + per), "flops": 0.0}
    if kind == "canonical":
        n = 3 * (case["m_lo"] + case["m_hi"]) / 2
        # 2n signatures of n values, each at least one checksum step per byte
        return {"bytes": case["count"] * (65 + 256 + 8), "flops": case["count"] * 2 * n * n * 4}
    if kind == "insertions":
        slots, rows = _mean_insertions(case)
        return {"bytes": case["count"] * (65 + 8 + slots + 64 * rows), "flops": 0.0}
    rows, layers = case["rows"], order_model.LAYERS
    weights = sum(a * b for a, b in layers)
    biases = sum(a for a, _ in layers)
    # forward, weight gradients, and input gradients of all layers but the first; the batch
    # read once, weights, masters and both moments read and written
    flops = 2.0 * rows * (3 * weights - layers[0][0] * layers[0][1])
    return {"bytes": rows * (order_model.FEATURES * 2 + 5) + weights * (3 * 8 + 2 * 2) + biases * 3 * 8,
            "flops": flops}


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "canonical" and case["count"] * case["m_hi"] ** 2 <= 100_000:
        return _exact_canonical(case, seed)
    return None  # verdicts, bytes and whole numbers


def _exact_train(case, seed):
    x, n, target, model = _train_inputs(case, seed)
    rows = x.shape[0]
    w = [t.double() for t in model.weight]
    b = [t.double() for t in model.bias]
    acts = [x.double()]
    for layer in range(3):
        acts.append(torch.relu(acts[-1] @ w[layer].T + b[layer]))
    logits = acts[-1] @ w[3].T + b[3]
    # column c = (i < j < k) is valid when k < n
    last = np.full(order_model.TRIPLES_PADDED, 255)
    i, j, k = np.nonzero(order_model.LEX32 >= 0)
    last[order_model.LEX32[i, j, k]] = k
    valid = torch.from_numpy(last).cuda()[None, :] < n[:, None].long()
    logits = logits.masked_fill(~valid, float("-inf"))
    logp = torch.log_softmax(logits, dim=1)
    at = target.long()[:, None]
    loss = -logp.gather(1, at)
    grad = logp.exp()
    grad.scatter_add_(1, at, torch.full_like(loss, -1.0))
    grad /= rows
    del logits, logp, valid
    gw, gb = [None] * 4, [None] * 4
    for layer in (3, 2, 1, 0):
        gw[layer] = grad.T @ acts[layer]
        gb[layer] = grad.sum(0)
        if layer:
            grad = (grad @ w[layer]) * (acts[layer] > 0)
    step = model.step + 1
    c1, c2 = 1 - 0.9 ** step, 1 - 0.999 ** step
    value, m, v = [], [], []
    for old, g, m0, v0 in zip(model.master + model.bias, gw + gb, model.m, model.v):
        m.append(0.9 * m0.double() + 0.1 * g)
        v.append(0.999 * v0.double() + 0.001 * g * g)
        value.append(old.double() - 1e-3 * (m[-1] / c1) / ((v[-1] / c2).sqrt() + 1e-8))
    value[3][order_model.TRIPLES:] = 0.0
    return {"loss": float(loss.mean()), "top1": None, "master": value[:4], "weight": value[:4], "bias": value[4:],
            "m": m, "v": v}


def _exact_canonical(case, seed):
    """The canonical signature by its definition: of the 2n signatures of a configuration (pi
    started at each symbol, and the mirror of each), the one whose CRC32 is least, then the
    lexicographically least."""
    spi, sizes, _, _ = _three_cycles(_rng(case, seed), case["count"], case["m_lo"], case["m_hi"])
    out = np.zeros((case["count"], 64))
    for row in range(case["count"]):
        n = int(sizes[row])
        succ = [int(v) for v in spi[row, :n]]
        inv = [0] * n
        for x, y in enumerate(succ):
            inv[y] = x
        best = None
        for variant in range(2 * n):
            r = variant >> 1
            if variant & 1:  # symbols at pi positions i and n-1-i swapped, the cycles run backwards
                nxt = [n - 1 - (inv[(r + n - 1 - p) % n] - r) % n for p in range(n)]
            else:
                nxt = [(succ[(r + p) % n] - r) % n for p in range(n)]
            value, label = [0.0] * n, 0
            for p in range(n):
                if value[p]:
                    continue
                label += 1
                cycle = [p]
                while nxt[cycle[-1]] != p:
                    cycle.append(nxt[cycle[-1]])
                oriented = sum(a < b for a, b in zip(cycle, cycle[1:] + cycle[:1])) > 1
                for t, q in enumerate(cycle):
                    value[q] = label + (t + 1) / 100 if oriented else float(label)
            code = zlib.crc32(struct.pack(">%df" % n, *value))
            code = (code - (1 << 32) if code >> 31 else code, value)
            if best is None or code < best:
                best = code
        out[row, :n] = best[1]
    return {"signature": torch.from_numpy(out), "hash": None, "variant": None}
