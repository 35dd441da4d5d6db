"""The work a user of libatc has it do, as cases that can be timed and compared.

A case is a dict of plain values.  Its "kind" names the call:

  count      atc.tc on a resident oriented CSR (the counting programs' hot loop)
  kcl        atc.kcl on a resident oriented CSR (the k-clique program)
  pretc      atc.pretc_device: raw pairs on the device -> oriented CSR
  program    atc.pretc_host_ptr + atc.tc: pinned host pairs -> CSR -> count, a whole
             counting program's run
  adirection atc.adirection: host pairs -> oriented host pairs (the A-direction program)
  batch      Batch.run: many graphs of uneven sizes in one replay
  select     atc.graph_features + MLP.select on device pairs (the learned selector's use)
  gradients  MLP.gradients: forward and backward of the selector's network (its training)

Graphs are the benchmark's and the tests' generators: R-MAT (Graph500 parameters), Chung-Lu
and random geometric graphs.  `pairs` cuts an R-MAT sample list at any length, so sizes need
not be powers of two.  Where the outputs are edge lists (pretc, adirection) the input holds
exactly `edges` distinct edges among `pairs` raw pairs, the rest repeats (as symmetrised edge
files have them), so that every seed gives outputs of one size.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "accelerating-tc_gb300")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

import atc  # noqa: E402


def listed():
    return [
        # the smallest call: a graph of a thousand vertices, where launches and waits are all
        # there is (the smoke test's graph)
        {"name": "count-rmat10", "kind": "count", "graph": "rmat", "scale": 10, "pairs": 16 << 10,
         "dir": "ADIRECTION", "order": "NONE", "kernel": "AUTO"},
        # an ordinary social-network-like graph of odd size, default kernel
        {"name": "count-chunglu700k", "kind": "count", "graph": "chunglu", "n": 700001, "gamma": 2.3, "degree": 37.0,
         "dir": "ADIRECTION", "order": "NONE", "kernel": "AUTO"},
        # a kernel family asked for by name, as tric_gpu does, on a degree orientation
        {"name": "count-rmat20-tricore", "kind": "count", "graph": "rmat", "scale": 20, "pairs": 16 << 20,
         "dir": "DEGREE_LOWID", "order": "NONE", "kernel": "TRICORE"},
        # the headline: R-MAT scale 24, A-direction + A-order
        {"name": "count-rmat24", "kind": "count", "graph": "rmat", "scale": 24, "pairs": 16 << 24,
         "dir": "ADIRECTION", "order": "AORDER", "kernel": "AUTO"},
        # k-cliques of a spatial graph (every candidate set small)
        {"name": "kcl-rgg20-k5", "kind": "kcl", "graph": "rgg", "n": 1 << 20, "degree": 32.0, "dir": "ADIRECTION",
         "order": "NONE", "k": 5},
        # k-cliques of a skewed graph (large candidate sets)
        {"name": "kcl-rmat18-k4", "kind": "kcl", "graph": "rmat", "scale": 18, "pairs": 16 << 18,
         "dir": "ADIRECTION", "order": "NONE", "k": 4},
        # a small input built for counting, degree orientation, an odd number of pairs
        {"name": "pretc-rmat14", "kind": "pretc", "graph": "rmat", "scale": 14, "pairs": 200003, "edges": 150001,
         "dir": "DEGREE", "order": "NONE"},
        # a large input built for counting, A-direction
        {"name": "pretc-rmat22", "kind": "pretc", "graph": "rmat", "scale": 22, "pairs": 16 << 22, "edges": 61000000,
         "dir": "ADIRECTION", "order": "NONE"},
        # a whole run on host data: A-direction + A-order, then the count
        {"name": "program-rmat20", "kind": "program", "graph": "rmat", "scale": 20, "pairs": 16 << 20,
         "dir": "ADIRECTION", "order": "AORDER", "kernel": "AUTO"},
        # the A-direction program's work on pageable host pairs
        {"name": "adirection-rmat17", "kind": "adirection", "graph": "rmat", "scale": 17, "pairs": 1500001,
         "edges": 750003},
        # many graphs of uneven sizes
        {"name": "batch-chunglu48", "kind": "batch", "graphs": 48, "n_lo": 1000, "n_hi": 200000},
        # a training step's gradients for the selector's network (the timing fixture's shape)
        {"name": "gradients-480x24", "kind": "gradients", "rows": 480, "hidden": 64, "outputs": 24},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, lo, hi):
    """A graph of about lo..hi edges."""
    m = _log_uniform(rng, lo, hi)
    g = rng.choice(("rmat", "rmat", "chunglu", "rgg"))
    if g == "rmat":
        ef = rng.uniform(8.0, 24.0)
        scale = max(8, min(24, int(math.log2(m / ef))))
        return {"graph": "rmat", "scale": scale, "pairs": m}
    degree = round(rng.uniform(8.0, 64.0), 2)
    n = max(300, int(2 * m / degree))
    if g == "chunglu":
        return {"graph": "chunglu", "n": n, "gamma": round(rng.uniform(2.05, 2.95), 3), "degree": degree}
    return {"graph": "rgg", "n": n, "degree": degree}


def _with_edges(rng, case):
    """Fixes the distinct edges of a drawn graph: some of the raw pairs repeat one."""
    most = case["pairs"] if case["graph"] == "rmat" else int(case["n"] * case["degree"] / 2)
    case["edges"] = int(most * rng.uniform(0.5, 0.8))
    case["pairs"] = int(case["edges"] * rng.uniform(1.0, 2.0))
    return case


DIRS = ("ADIRECTION", "ADIRECTION", "DEGREE", "DEGREE_LOWID", "KCORE")


def draw(rng):
    kind = rng.choice(("count", "count", "count", "count", "kcl", "kcl", "pretc", "pretc", "program", "adirection",
                       "batch", "select", "gradients"))
    c = {"kind": kind}
    if kind in ("count", "pretc", "program"):
        c.update(_draw_graph(rng, 1 << 13, 1 << 25))
        if kind == "pretc":
            _with_edges(rng, c)
        c["dir"] = rng.choice(DIRS)
        c["order"] = rng.choice(("NONE", "NONE", "DEGREE_DESC"))
        if c["graph"] == "rmat" and c["pairs"] > 1 << 18:  # A-order needs a skewed graph of some size
            c["order"] = rng.choice(("NONE", "AORDER", "DEGREE_DESC"))
        if kind != "pretc":
            c["kernel"] = rng.choice(("AUTO", "AUTO", "AUTO", "BISSON", "HU", "FOX", "TRICORE"))
    elif kind == "kcl":
        c.update(_draw_graph(rng, 1 << 13, 1 << 21))
        c["dir"] = rng.choice(DIRS)
        c["order"] = "NONE"
        c["k"] = rng.choice((4, 4, 5, 5, 6)) if c["graph"] != "rmat" or c["pairs"] < 1 << 19 else 4
    elif kind == "adirection":
        c.update(_with_edges(rng, _draw_graph(rng, 1 << 13, 1 << 22)))
    elif kind == "batch":
        c.update({"graphs": rng.randrange(5, 64), "n_lo": 1000, "n_hi": _log_uniform(rng, 4000, 200000)})
    elif kind == "select":
        c.update(_draw_graph(rng, 1 << 13, 1 << 24))
        c.update({"hidden": 64, "outputs": rng.choice((24, 60))})
    else:
        c.update({"rows": _log_uniform(rng, 16, 4096), "hidden": rng.choice((32, 64, 100)),
                  "outputs": rng.choice((24, 60))})
    return c


# ---- inputs ---------------------------------------------------------------------------
def _stream():
    return torch.cuda.current_stream().cuda_stream


def _raise(status):
    if status != 0:
        raise atc.ATCError(status, atc.lib().atc_last_error().decode(errors="replace"))


def _device_pairs(case, seed):
    """The case's raw pairs, an int32 (m, 2) tensor on the device."""
    if "edges" not in case:
        return _samples(case, seed)
    # distinct edges without loops, (0, n - 1) among them, in random order and direction
    n = 1 << case["scale"] if case["graph"] == "rmat" else case["n"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    more = 1.3
    while True:
        p = _samples(_grown(case, more), seed).to(torch.int64)
        keys = torch.unique(p.amin(1) * n + p.amax(1))
        lo, hi = torch.div(keys, n, rounding_mode="floor"), keys % n
        keys = keys[(lo != hi) & (keys != n - 1)]
        if keys.numel() >= case["edges"] - 1:
            break
        more *= 1.3
    keys = keys[torch.randperm(keys.numel(), generator=g, device="cuda")[: case["edges"] - 1]]
    keys = torch.cat([keys, keys.new_tensor([n - 1])])
    e = torch.stack([torch.div(keys, n, rounding_mode="floor"), keys % n], 1).to(torch.int32)
    flip = torch.rand(e.shape[0], generator=g, device="cuda") < 0.5
    e = torch.where(flip[:, None], e.flip(1), e)
    return torch.cat([e, e[: case["pairs"] - e.shape[0]].flip(1)]).contiguous()


def _grown(case, more):
    """The case's graph with `more` times the samples."""
    if case["graph"] == "rmat":
        return {**case, "pairs": int(case["edges"] * more)}
    return {**case, "degree": 2 * case["edges"] / case["n"] * more}


def _samples(case, seed):
    s = _stream()
    if case["graph"] == "rmat":
        pairs, scale = case["pairs"], case["scale"]
        ef = -(-pairs // (1 << scale))
        out = torch.empty((ef << scale, 2), dtype=torch.int32, device="cuda")
        _raise(atc.lib().atc_gen_rmat_device(scale, ef, *atc.GRAPH500, seed, out.data_ptr(), s))
        return out[:pairs]
    if case["graph"] == "chunglu":
        return atc.gen_chunglu_device(case["n"], case["gamma"], case["degree"], seed, stream=s)
    import ctypes
    cap = int(case["n"] * case["degree"] * 0.6) + 4096  # the mean is n * degree / 2
    out = torch.empty((cap, 2), dtype=torch.int32, device="cuda")
    cnt = ctypes.c_uint64(0)
    _raise(atc.lib().atc_gen_rgg_device(case["n"], case["degree"], seed, out.data_ptr(), cap, ctypes.byref(cnt), s))
    return out[: cnt.value]


def _csr(case, seed):
    p = _device_pairs(case, seed)
    return atc.pretc_device(p.data_ptr(), p.shape[0], atc.Dir[case["dir"]], atc.Order[case["order"]], stream=_stream())


def _batch_graphs(case, seed):
    rng = np.random.default_rng(seed)
    for g in range(case["graphs"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        yield {"graph": "chunglu", "n": n, "gamma": float(rng.uniform(2.05, 3.0)), "degree": float(rng.uniform(4, 64)),
               "dir": "ADIRECTION", "order": "NONE"}, seed * 1000 + g


def _mlp_values(case, seed):
    """Weights, standardisation and (for gradients) rows of the selector's network."""
    rng = np.random.default_rng(seed)
    i, h, o = 6, case["hidden"], case["outputs"]
    w = [rng.uniform(-1, 1, (a, b)) * math.sqrt(6.0 / a) for a, b in ((i, h), (h, h), (h, o))]
    b = [rng.uniform(-0.1, 0.1, k) for k in (h, h, o)]
    params = np.concatenate([np.concatenate([x.ravel(), y]) for x, y in zip(w, b)]).astype(np.float32)
    mean = np.array([13.0, 15.0, 3.0, 6.0, 8.0, 14.0], dtype=np.float32)
    std = np.array([2.0, 2.0, 0.7, 2.0, 1.5, 3.0], dtype=np.float32)
    rows = case.get("rows", 0)
    x = (mean + std * rng.normal(size=(rows, i))).astype(np.float32)
    t = rng.normal(1.0, 1.5, (rows, o)).astype(np.float32)  # log-times
    mask = (rng.uniform(size=(rows, o)) < 0.9).astype(np.float32)  # triples that could not be timed
    return params, mean, std, x, t, mask


def prepare(case, seed):
    atc.init(torch.cuda.current_device())
    kind = case["kind"]
    if kind == "count":
        return kind, _csr(case, seed), atc.Kernel[case["kernel"]]
    if kind == "kcl":
        return kind, _csr(case, seed), case["k"]
    if kind == "pretc":
        return kind, _device_pairs(case, seed), atc.Dir[case["dir"]], atc.Order[case["order"]]
    if kind == "program":
        host = _device_pairs(case, seed).cpu().pin_memory()
        return kind, host, atc.Dir[case["dir"]], atc.Order[case["order"]], atc.Kernel[case["kernel"]]
    if kind == "adirection":
        return kind, _device_pairs(case, seed).cpu().numpy()
    if kind == "batch":
        b = atc.Batch()
        for g, s in _batch_graphs(case, seed):
            c = _csr(g, s)
            b.add(c, stream=_stream())
            c.free()
        return kind, b, {"group_by_source": 2}
    params, mean, std, x, t, mask = _mlp_values(case, seed)
    net = atc.MLP(6, case["hidden"], case["outputs"])
    net.params(params)
    net.scaling(mean, std)
    if kind == "select":
        return kind, net, _device_pairs(case, seed)
    return kind, net, x, t, mask


class _Array:
    """A device array of a CSR, which it keeps alive."""

    def __init__(self, csr, ptr, count, typestr):
        self.csr = csr
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _csr_outputs(csr):
    st = csr.struct
    out = {"n": csr.n, "m": csr.m, "wedges": csr.wedges, "wedges_min": csr.wedges_min, "max_outdeg": csr.max_outdeg}
    out["offsets"] = torch.as_tensor(_Array(csr, st.offsets, csr.n + 1, "<i8"), device="cuda")
    if csr.m:
        out["cols"] = torch.as_tensor(_Array(csr, st.cols, csr.m, "<i4"), device="cuda")
    return out


def run(state):
    kind = state[0]
    if kind == "count":
        return atc.tc(state[1], state[2], stream=_stream())[0]
    if kind == "kcl":
        return atc.kcl(state[1], state[2], stream=_stream())[0]
    if kind == "pretc":
        _, p, d, o = state
        return _csr_outputs(atc.pretc_device(p.data_ptr(), p.shape[0], d, o, stream=_stream()))
    if kind == "program":
        _, p, d, o, k = state
        csr = atc.pretc_host_ptr(p.data_ptr(), p.shape[0], d, o, stream=_stream())
        count = atc.tc(csr, k, stream=_stream())[0]
        csr.free()
        return count
    if kind == "adirection":
        return atc.adirection(state[1], want_prio=True, stream=_stream())
    if kind == "batch":
        return state[1].run(state[2], stream=_stream())[0]
    if kind == "select":
        f = atc.graph_features(state[2].data_ptr(), state[2].shape[0], stream=_stream())
        choice, predicted = state[1].select(f)
        return {"features": f, "choice": choice, "predicted": predicted}
    loss, grads = state[1].gradients(*state[2:])
    return {"loss": loss, "grads": grads}


# ---- what a pass cannot do without ------------------------------------------------------
def _size(case):
    """(vertices, raw pairs, edges) of the case's graph, near enough: R-MAT samples repeat."""
    if "edges" in case:
        return 1 << case["scale"] if case["graph"] == "rmat" else case["n"], case["pairs"], case["edges"]
    if case["graph"] == "rmat":
        return 1 << case["scale"], case["pairs"], int(case["pairs"] * 0.93)
    m = int(case["n"] * case["degree"] / 2)
    return case["n"], m, m


def work(case):
    """Inputs read once and outputs written once: a CSR is 8 bytes a vertex and 4 an edge, a raw
    pair 8.  Counting has no multiplications; the network's layers have."""
    kind = case["kind"]
    if kind == "batch":
        mean_n = (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])
        return {"bytes": case["graphs"] * (8.0 * mean_n + 4.0 * mean_n * 17 + 8), "flops": 0.0}
    if kind == "gradients":
        i, h, o, r = 6, case["hidden"], case["outputs"], case["rows"]
        params = i * h + h + h * h + h + h * o + o
        return {"bytes": 4.0 * (2 * params + r * (i + 2 * o)), "flops": 2.0 * r * (2 * i * h + 3 * h * h + 3 * h * o)}
    n, pairs, m = _size(case)
    csr = 8.0 * (n + 1) + 4.0 * m
    if kind in ("count", "kcl"):
        return {"bytes": csr + 8, "flops": 0.0}
    if kind == "pretc":
        return {"bytes": 8.0 * pairs + csr, "flops": 0.0}
    if kind == "program":
        return {"bytes": 8.0 * pairs + 8, "flops": 0.0}
    if kind == "adirection":
        return {"bytes": 8.0 * pairs + 8.0 * m + 4.0 * n, "flops": 0.0}
    return {"bytes": 8.0 * pairs, "flops": 2.0 * (6 * case["hidden"] + case["hidden"] ** 2 + case["hidden"] * case["outputs"])}


# ---- the floating outputs in 64 bits ----------------------------------------------------
def _network64(params, i, h, o, z):
    at, layers = 0, []
    for a, b in ((i, h), (h, h), (h, o)):
        w = params[at: at + a * b].reshape(a, b)
        at += a * b
        layers.append((w, params[at: at + b]))
        at += b
    (w1, b1), (w2, b2), (w3, b3) = layers
    a1 = np.maximum(z @ w1 + b1, 0.0)
    a2 = np.maximum(a1 @ w2 + b2, 0.0)
    return a1, a2, a2 @ w3 + b3, w2, w3


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("select", "gradients"):
        return None  # whole numbers
    params, mean, std, x, t, mask = (v.astype(np.float64) for v in _mlp_values(case, seed))
    h, o = case["hidden"], case["outputs"]
    if kind == "select":
        raw = _device_pairs(case, seed).to(torch.int64)
        n = int(raw.max()) + 1
        p = raw[raw[:, 0] != raw[:, 1]]
        m = p.shape[0]
        deg = torch.bincount(p.reshape(-1), minlength=n)
        a, b = p[:, 0], p[:, 1]
        a_src = (deg[a] < deg[b]) | ((deg[a] == deg[b]) & (a > b))
        out = torch.bincount(torch.where(a_src, a, b), minlength=n)
        d = deg.double()
        mu = float(d.sum()) / n
        var = float((d * d).sum()) / n - mu * mu
        tail_v = out[out * n > 2 * m]
        tail = float(tail_v.sum()) - tail_v.numel() * (m / n)
        f = np.log1p(np.array([n, m, mu, max(var, 0.0), float(deg.max()), max(tail, 0.0)], dtype=np.float64))
        y = _network64(params, 6, h, o, ((f - mean) / std)[None, :])[2]
        return {"features": f, "choice": None, "predicted": y[0]}
    z = (x - mean) / std
    a1, a2, y, w2, w3 = _network64(params, 6, h, o, z)
    cnt = max(mask.sum(), 1.0)
    loss = 0.5 * (mask * (y - t) ** 2).sum() / cnt
    dy = mask * (y - t) / cnt
    d2 = (dy @ w3.T) * (a2 > 0)
    d1 = (d2 @ w2.T) * (a1 > 0)
    grads = np.concatenate([np.concatenate([(u.T @ v).ravel(), v.sum(0)]) for u, v in ((z, d1), (a1, d2), (a2, dy))])
    return {"loss": float(loss), "grads": grads}
