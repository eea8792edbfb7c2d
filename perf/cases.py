"""Timed workloads of the matcher, one pass each through the public entry points.

A case is a dict of plain values: ``kind`` names the call, the other keys its
sizes and options. Descriptors follow the recipe of
``matching_sift_b200.datagen`` (128 Exp(1) values, 38 zeroed, norm 512,
rounded to uint8; half of the queries are noisy copies of base rows), drawn on
the GPU from the seed so that a million rows take milliseconds to make.

Kinds:
  match      match() of two CUDA tensors: uint8, float16 (SIFT components / 512)
             or general float32 rows (unit-normalised uniform values)
  drop_in    cublas_2nn_sift(FLOAT_DEVICE) on float32 SIFT components / 512
  host       cublas_2nn_sift(U8_HOST) on pinned host buffers
  plan       BatchPlan.run(): many uneven image pairs, one graph replay
  batch      match_batch() of uneven image pairs given for the first time
  mutual     match_mutual_batch(): both directions of every pair, cross-checked
  lsh_index  HashIndex.lsh().search(): a base hashed once, searched many times
  lsh        lsh_match(): base and queries hashed, bucketed and searched in one call
  learned    MlpHash.match(): the learned hash in one call, exact fallback included
  grad       mlp_loss_grad(): forward and backward of one training step
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import matching_sift_b200 as ms

DIM = 128
DEV = "cuda:0"
THRESHOLD = 0.8


def listed():
    return [
        # One image pair with few keypoints: the smallest call, all latency.
        {"name": "pair_517x733", "kind": "match", "dtype": "u8", "q": 517, "r": 733},
        # The reference's small benchmark configuration on uint8 rows.
        {"name": "u8_1000x10000", "kind": "match", "dtype": "u8", "q": 1000, "r": 10000},
        # The same sizes as a caller of the reference issues them: float rows
        # of SIFT components / 512 through cublas_2nn_sift.
        {"name": "drop_in_f32_1000x10000", "kind": "drop_in", "q": 1000, "r": 10000},
        # The headline: ANN_SIFT1M's sizes, exact.
        {"name": "u8_10000x1000000", "kind": "match", "dtype": "u8", "q": 10000, "r": 1000000},
        # The headline from host buffers, copies included.
        {"name": "host_u8_10000x1000000", "kind": "host", "q": 10000, "r": 1000000},
        # Half rows (the reference's HALF_DEVICE type) at ragged sizes.
        {"name": "f16_2561x500003", "kind": "match", "dtype": "f16", "q": 2561, "r": 500003},
        # General float rows: the reference benchmark's default data.
        {"name": "f32_2053x131077", "kind": "match", "dtype": "f32", "q": 2053, "r": 131077},
        # A photo collection's image pairs, sizes of both sides log-uniform in [500, 8000], planned once.
        {"name": "plan_512_pairs", "kind": "plan", "pairs": 512, "lo": 500, "hi": 8000, "sizes": 0},
        # What a geometric verifier starts from: both directions of every pair, cross-checked.
        {"name": "mutual_128_pairs", "kind": "mutual", "pairs": 128, "lo": 500, "hi": 8000, "sizes": 1},
        # A served LSH index: 8 tables of 16 bits, 16 buckets per table.
        {"name": "lsh_index_4096x1000000", "kind": "lsh_index", "q": 4096, "r": 1000000, "L": 8, "k": 16,
         "probes": 16},
        # The learned hash on a new base: base hash, buckets, probes, scan and fallback.
        {"name": "learned_4096x1000000", "kind": "learned", "q": 4096, "r": 1000000, "k": 16, "probes": 8,
         "min_candidates": 16},
        # One training step of the learned hash at its default batch.
        {"name": "grad_2048_k16", "kind": "grad", "batch": 2048, "k": 16},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(("match", "match", "match", "drop_in", "host", "plan", "batch", "mutual", "lsh_index", "lsh",
                       "learned", "grad"))
    if kind == "match":
        dtype = rng.choice(("u8", "u8", "f16", "f32"))
        if dtype == "u8":
            return {"kind": kind, "dtype": dtype, "q": _log_int(rng, 200, 10000), "r": _log_int(rng, 300, 1000000)}
        if dtype == "f16":
            return {"kind": kind, "dtype": dtype, "q": _log_int(rng, 300, 4000), "r": _log_int(rng, 1000, 500000)}
        return {"kind": kind, "dtype": dtype, "q": _log_int(rng, 300, 4000), "r": _log_int(rng, 1000, 200000)}
    if kind == "drop_in":
        return {"kind": kind, "q": _log_int(rng, 300, 4000), "r": _log_int(rng, 500, 200000)}
    if kind == "host":
        return {"kind": kind, "q": _log_int(rng, 500, 10000), "r": _log_int(rng, 5000, 1000000)}
    if kind in ("plan", "batch", "mutual"):
        most = {"plan": 512, "batch": 256, "mutual": 128}[kind]
        lo = _log_int(rng, 100, 1000)
        return {"kind": kind, "pairs": _log_int(rng, 2, most), "lo": lo, "hi": _log_int(rng, 2 * lo, 8000),
                "sizes": rng.randrange(1 << 30)}
    if kind in ("lsh_index", "lsh"):
        L = rng.choice((1, 2, 4, 8))
        return {"kind": kind, "q": _log_int(rng, 300, 4096), "r": _log_int(rng, 20000, 1000000), "L": L,
                "k": rng.choice((14, 16, 20)), "probes": rng.choice((1, 4, 8, 16))}
    if kind == "learned":
        return {"kind": kind, "q": _log_int(rng, 300, 4096), "r": _log_int(rng, 20000, 1000000),
                "k": rng.choice((14, 16, 20)), "probes": rng.choice((1, 4, 8, 16)),
                "min_candidates": rng.choice((0, 8, 16))}
    return {"kind": "grad", "batch": _log_int(rng, 100, 4096), "k": rng.choice((8, 16, 20, 24, 32))}


# --------------------------------------------------------------------- inputs

def _gen(seed: int, stream: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed((seed * 16 + stream) % (1 << 62))


def _fresh(n: int, g: torch.Generator) -> torch.Tensor:
    """n SIFT-like uint8 rows."""
    out = torch.empty((n, DIM), dtype=torch.uint8, device=DEV)
    for s in range(0, n, 1 << 18):
        m = min(1 << 18, n - s)
        x = torch.empty((m, DIM), device=DEV).exponential_(generator=g)
        drop = torch.rand((m, DIM), device=DEV, generator=g).topk(38, dim=1).indices
        x.scatter_(1, drop, 0.0)
        x *= 512.0 / x.norm(dim=1, keepdim=True).clamp_min(1e-20)
        out[s:s + m] = x.round_().clamp_(0, 255).to(torch.uint8)
    return out


def _noisy(src: torch.Tensor, g: torch.Generator) -> torch.Tensor:
    x = src.float() + 8.0 * torch.randn(src.shape, device=DEV, generator=g)
    return x.round_().clamp_(0, 255).to(torch.uint8)


def _queries(n: int, base: torch.Tensor, g: torch.Generator) -> torch.Tensor:
    """Half noisy copies of base rows, half fresh rows, in random order."""
    q = _fresh(n, g)
    half = torch.randperm(n, device=DEV, generator=g)[:n // 2]
    src = torch.randint(0, base.shape[0], (n // 2,), device=DEV, generator=g)
    q[half] = _noisy(base[src], g)
    return q


def _workload(case, seed):
    r = _fresh(case["r"], _gen(seed, 0))
    return _queries(case["q"], r, _gen(seed, 1)), r


def _floats(case, seed):
    """Unit-normalised uniform float32 rows."""
    g = _gen(seed, 2)
    out = []
    for n in (case["q"], case["r"]):
        x = torch.rand((n, DIM), device=DEV, generator=g)
        out.append(x / x.norm(dim=1, keepdim=True))
    return out


def _pair_sizes(case) -> np.ndarray:
    """(pairs, 2) keypoint counts, a part of the case and not of the seed."""
    rng = np.random.default_rng(case["sizes"])
    return np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), (case["pairs"], 2))).astype(np.int64)


def _pairs(case, seed):
    """All first sets, all second sets (40% noisy copies of first-set rows), pair table."""
    sizes = _pair_sizes(case)
    a = _fresh(int(sizes[:, 0].sum()), _gen(seed, 3))
    g = _gen(seed, 4)
    b = _fresh(int(sizes[:, 1].sum()), g)
    a_off = np.concatenate([[0], np.cumsum(sizes[:, 0])])
    b_off = np.concatenate([[0], np.cumsum(sizes[:, 1])])
    pair_of = torch.from_numpy(np.repeat(np.arange(len(sizes)), sizes[:, 1])).to(DEV)
    first = torch.from_numpy(a_off[:-1]).to(DEV)[pair_of]
    count = torch.from_numpy(sizes[:, 0]).to(DEV)[pair_of]
    u = torch.rand(b.shape[0], device=DEV, generator=g)
    src = first + (u * count).long().clamp_max(count - 1)
    copied = torch.rand(b.shape[0], device=DEV, generator=g) < 0.4
    b[copied] = _noisy(a[src[copied]], g)
    table = np.stack([sizes[:, 0], sizes[:, 1], b_off[:-1]], axis=1).astype(np.uint32)
    return a, b, table


def _planes(case, seed):
    x = 32.0 * torch.randn((case["L"], case["k"], DIM), device=DEV, generator=_gen(seed, 5))
    return x.round_().clamp_(-127, 127).to(torch.int8)


def _mlp_params(k: int, seed: int) -> torch.Tensor:
    """Flat parameters (W1, b1, W2 padded to 32 rows, b2 padded to 32) at the scale training starts from."""
    g = _gen(seed, 6)
    w2 = torch.zeros((32, 256), device=DEV)
    w2[:k] = 0.0884 * torch.randn((k, 256), device=DEV, generator=g)
    b2 = torch.zeros(32, device=DEV)
    b2[:k] = 0.1 * torch.randn(k, device=DEV, generator=g)
    return torch.cat([0.125 * torch.randn(256 * DIM, device=DEV, generator=g),
                      0.3 * torch.randn(256, device=DEV, generator=g), w2.reshape(-1), b2])


def _step_rows(case, seed):
    """Rows of one training step: queries, neighbours (noisy copies), random rows."""
    n = case["batch"]
    g = _gen(seed, 7)
    near = _fresh(n, g)
    return torch.cat([_noisy(near, g), near, _fresh(n, g)])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "match":
        if case["dtype"] == "f32":
            q, r = _floats(case, seed)
        else:
            q, r = _workload(case, seed)
            if case["dtype"] == "f16":
                q, r = (q.half() / 512), (r.half() / 512)
        return {"kind": kind, "q": q, "r": r}
    if kind == "drop_in":
        q, r = _workload(case, seed)
        return {"kind": kind, "q": q.float() / 512, "r": r.float() / 512,
                "matches": torch.empty(case["q"], dtype=torch.int32, device=DEV)}
    if kind == "host":
        q, r = _workload(case, seed)
        return {"kind": kind, "q": q.cpu().pin_memory(), "r": r.cpu().pin_memory(),
                "matches": torch.empty(case["q"], dtype=torch.int32).pin_memory()}
    if kind in ("plan", "batch", "mutual"):
        a, b, table = _pairs(case, seed)
        state = {"kind": kind, "a": a, "b": b, "pairs": table}
        if kind == "plan":
            state["plan"] = ms.BatchPlan(a, b, table, threshold=THRESHOLD)
        return state
    if kind in ("lsh_index", "lsh"):
        q, r = _workload(case, seed)
        planes = _planes(case, seed)
        state = {"kind": kind, "q": q, "r": r, "planes": planes, "probes": case["probes"]}
        if kind == "lsh_index":
            state["index"] = ms.HashIndex.lsh(r, planes)
        return state
    if kind == "learned":
        q, r = _workload(case, seed)
        return {"kind": kind, "q": q, "r": r, "model": ms.MlpHash.from_params(_mlp_params(case["k"], seed), case["k"]),
                "probes": case["probes"], "min_candidates": case["min_candidates"]}
    return {"kind": kind, "x": _step_rows(case, seed), "batch": case["batch"], "k": case["k"],
            "params": _mlp_params(case["k"], seed)}


# ---------------------------------------------------------------- one pass

def run(state):
    kind = state["kind"]
    if kind == "match":
        return ms.match(state["q"], state["r"], THRESHOLD)
    if kind in ("drop_in", "host"):
        q, r = state["q"], state["r"]
        rc = ms.cublas_2nn_sift(q, r, ms.FLOAT_DEVICE if kind == "drop_in" else ms.U8_HOST, q.shape[0], r.shape[0],
                                state["matches"], THRESHOLD)
        return {"status": rc, "matches": state["matches"]}
    if kind == "plan":
        return state["plan"].run()
    if kind == "batch":
        return ms.match_batch(state["a"], state["b"], state["pairs"], THRESHOLD)
    if kind == "mutual":
        return ms.match_mutual_batch(state["a"], state["b"], state["pairs"], THRESHOLD)
    if kind == "lsh_index":
        return state["index"].search(state["q"], probes=state["probes"])
    if kind == "lsh":
        return ms.lsh_match(state["q"], state["r"], state["planes"], probes=state["probes"], candidates=True)
    if kind == "learned":
        return state["model"].match(state["q"], state["r"], n_probes=state["probes"],
                                    min_candidates=state["min_candidates"])
    loss, grads = ms.mlp_loss_grad(state["x"], state["batch"], state["k"], state["params"])
    return {"loss": loss, "grads": grads}


# ------------------------------------------------------------ necessary work

def work(case):
    kind = case["kind"]
    if kind in ("match", "drop_in", "host"):
        q, r = case["q"], case["r"]
        size = {"u8": 1, "f16": 2, "f32": 4}[case.get("dtype", "f32" if kind == "drop_in" else "u8")]
        out = 20 if kind == "match" else 4  # matches, two indices, two distances per query
        return {"bytes": (q + r) * DIM * size + q * out, "flops": 2 * q * r * DIM}
    if kind in ("plan", "batch", "mutual"):
        sizes = _pair_sizes(case)
        a, b = int(sizes[:, 0].sum()), int(sizes[:, 1].sum())
        # A mutual search needs the products of each pair once: the reverse direction has the same ones.
        return {"bytes": (a + b) * DIM + a * 20, "flops": 2 * DIM * int((sizes[:, 0] * sizes[:, 1]).sum())}
    if kind in ("lsh_index", "lsh", "learned"):
        q, r, k, probes = case["q"], case["r"], case["k"], case["probes"]
        tables = case.get("L", 1)
        # Members of the probed buckets if codes were spread evenly, at 3 operations an element.
        members = q * min(r, r * tables * probes / 2.0 ** k)
        hashed = q + (0 if kind == "lsh_index" else r)
        per_row = 2 * (DIM * 256 + 256 * k) if kind == "learned" else 2 * DIM * tables * k
        return {"bytes": int((q + r) * DIM + q * 24 + min(members * 4, tables * r * 4)),
                "flops": int(hashed * per_row + members * 3 * DIM)}
    rows, k = 3 * case["batch"], case["k"]
    params = 256 * DIM + 256 + 32 * 256 + 32
    return {"bytes": rows * DIM + 2 * params * 4,
            "flops": 2 * rows * (256 * DIM + 256 * k) + 2 * rows * (2 * 256 * k + 256 * DIM)}


# ------------------------------------------------------- the same in 64 bits

def _top2(q: torch.Tensor, r: torch.Tensor, member=None):
    """Two smallest squared distances of every row of q to the rows of r (FLT_MAX where absent), float64."""
    absent = float(np.finfo(np.float32).max)
    qd = q.double()
    qn = (qd * qd).sum(1, keepdim=True)
    best = torch.full((q.shape[0], 2), absent, dtype=torch.float64, device=q.device)
    step = max(2, min(r.shape[0], (1 << 29) // max(1, q.shape[0])))
    for s in range(0, r.shape[0], step):
        rd = r[s:s + step].double()
        d = qn + (rd * rd).sum(1) - 2.0 * (qd @ rd.T)
        if member is not None:
            d.masked_fill_(~member(s, s + rd.shape[0]), absent)
        for _ in range(2):
            m, at = d.min(dim=1)
            best = torch.cat([best, m[:, None]], 1).sort(1).values[:, :2]
            d.scatter_(1, at[:, None], absent)
    return best.clamp_min(0.0)


def _lsh_top2(q, r, planes, probes):
    """_top2 over the members of the probed buckets of every table."""
    L, k = planes.shape[0], planes.shape[1]
    bits = 2 ** torch.arange(k, device=DEV)
    flip = min(6, k)
    masks = torch.arange(1 << flip, device=DEV)
    use = ((masks[:, None] >> torch.arange(flip, device=DEV)) & 1).double()
    code_r, probe_q = [], []
    for t in range(L):
        p = planes[t].double().T
        code_r.append(torch.cat([((c.double() @ p < 0) * bits).sum(1) for c in r.split(1 << 18)]))
        z = q.double() @ p
        code = ((z < 0) * bits).sum(1)
        mag, bit = z.abs().sort(dim=1, stable=True)
        weight = mag[:, :flip] @ use.T
        pick = weight.sort(dim=1, stable=True).indices[:, :probes]
        flips = (use.long()[pick] * bits[bit[:, :flip]][:, None, :]).sum(2)
        probe_q.append(code[:, None] ^ flips)
    out = []
    rows = max(1, (1 << 30) >> k)
    for s in range(0, q.shape[0], rows):
        n = min(rows, q.shape[0] - s)
        wanted = [torch.zeros((n, 1 << k), dtype=torch.bool, device=DEV).scatter_(1, pq[s:s + n], True)
                  for pq in probe_q]

        def member(lo, hi):
            m = wanted[0][:, code_r[0][lo:hi]]
            for t in range(1, L):
                m |= wanted[t][:, code_r[t][lo:hi]]
            return m

        out.append(_top2(q[s:s + n], r, member))
    return torch.cat(out)


def _grad64(x, batch, k, params):
    """Loss and gradients in float64. The model itself rounds its weights and hidden values to
    BF16; gradients pass straight through the roundings."""
    bf = lambda v: v.float().to(torch.bfloat16).double()
    p = params.double()
    n1 = 256 * DIM
    w1, b1 = bf(p[:n1]).view(256, DIM), p[n1:n1 + 256]
    w2, b2 = bf(p[n1 + 256:n1 + 256 + 32 * 256]).view(32, 256)[:k], p[n1 + 256 + 32 * 256:][:k]
    xs = x.double() / 64
    h = bf((xs @ w1.T + b1).clamp_min(0))
    t = torch.tanh(h @ w2.T + b2)
    rows = 3 * batch
    tq, tp, tn = t[:batch], t[batch:2 * batch], t[2 * batch:]
    sp, sn = (tq * tp).sum(1) / k, (tq * tn).sum(1) / k
    mean = t.mean(0)
    pos, neg, bal = (1 - sp).mean(), (sn * sn).mean(), (mean * mean).sum()
    dt = (2 * mean / rows).repeat(rows, 1)
    cn = (2 * sn / (k * batch))[:, None]
    dt[:batch] += -tp / (k * batch) + cn * tn
    dt[batch:2 * batch] += -tq / (k * batch)
    dt[2 * batch:] += cn * tq
    dz = dt * (1 - t * t)
    dh = (dz @ w2) * (h > 0)
    g2 = torch.zeros((32, 256), dtype=torch.float64, device=x.device)
    g2[:k] = dz.T @ h
    gb2 = torch.zeros(32, dtype=torch.float64, device=x.device)
    gb2[:k] = dz.sum(0)
    grads = torch.cat([(dh.T @ xs).reshape(-1), dh.sum(0), g2.reshape(-1), gb2])
    return np.array([float(pos + neg + bal), float(pos), float(neg), float(bal)]), grads


def exact(case, seed):
    kind = case["kind"]
    if kind in ("drop_in", "host", "learned"):
        # Whole numbers only, or buckets chosen by the sign of a rounded sum.
        return None
    if kind == "match":
        if case["dtype"] == "f32":
            q, r = _floats(case, seed)
        else:
            q, r = _workload(case, seed)
        d = _top2(q, r)
        if case["dtype"] == "f16":
            d = torch.where(d < 1e30, d / 512.0 ** 2, d)
        return {"matches": None, "nn_idx": None, "nn_dist": d}
    if kind in ("plan", "batch", "mutual"):
        a, b, table = _pairs(case, seed)
        dist, off = [], 0
        for n_a, n_b, b_off in table.astype(np.int64):
            dist.append(_top2(a[off:off + n_a], b[b_off:b_off + n_b]))
            off += n_a
        return {"matches": None, "nn_idx": None, "nn_dist": torch.cat(dist)}
    if kind in ("lsh_index", "lsh"):
        q, r = _workload(case, seed)
        d = _lsh_top2(q, r, _planes(case, seed), case["probes"])
        out = {"matches": None, "nn_idx": None, "nn_dist": d, "candidates": None}
        if kind == "lsh_index":
            out["fallback"] = None
        return out
    loss, grads = _grad64(_step_rows(case, seed), case["batch"], case["k"], _mlp_params(case["k"], seed))
    return {"loss": loss, "grads": grads}
