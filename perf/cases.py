"""Performance cases of the engine: the work a program gives it, each case one
pass through a public entry point.

A case is a dict with a "kind":

* knn        the neighbour table of a point set (stages.knn): the plain FP32
             search and the BF16 search with its exact rerank;
* fit        NCVis.fit_transform up to the start of the optimizer
             (n_epochs = 0: preprocessing, neighbours, symmetrization, initial
             embedding), numpy in and out or CUDA tensors;
* batched    NCVis.fit_transform_batched of several data sets, likewise;
* symmetrize neighbour table to graph (stages.symmetrize);
* init       graph to initial embedding (stages.init_embedding);
* optimize   the last epochs of the optimizer on an embedding that has
             settled (stages.optimize);
* nce        the differentiable loss, forward and backward (nce.nce_loss).

The optimizer's chains race on the embedding as the reference's threads do.
Over the epochs of a whole fit a difference in the last bit grows to another
embedding altogether, so the fits here stop before the optimizer and the
optimizer is run over its last epochs, where the steps are short and two runs
stay near one another.
"""
import math

import numpy as np
import torch

import ncvis_gb300 as ncvis
from ncvis_gb300 import nce, stages

A, B = 0.76687364, 1.22256382  # the curve of the default min_dist 0.4, spread 1
SEED = 42                      # the engine's default seed
EPOCHS = 50
DISTANCES = {"euclidean": 0, "inner_product": 1, "cosine": 2, "correlation": 3}
DEV = "cuda"


def listed():
    return [
        # A small table in one call, the size of the classic toy sets:
        # launches and waits are most of it.
        {"name": "knn_fp32_1000x32", "kind": "knn", "n": 1000, "dim": 32, "k": 15,
         "distance": "euclidean", "precision": "fp32", "data": "mixture"},
        # The reference's default configuration, 10,000 x 64, as its users call
        # it: numpy in, numpy out, FP32 search.
        {"name": "fit_fp32_10000x64_numpy", "kind": "fit", "n": 10_000, "dim": 64, "k": 15,
         "d": 2, "distance": "euclidean", "precision": "fp32", "data": "mixture", "host": True},
        # The plain FP32 search where the pairs dominate, odd size,
        # preprocessing that centres and scales the rows.
        {"name": "knn_fp32_60013x100", "kind": "knn", "n": 60_013, "dim": 100, "k": 15,
         "distance": "correlation", "precision": "fp32", "data": "sphere"},
        # Word-vector-like rows (131,072 x 100, cosine), BF16 search with rerank.
        {"name": "knn_bf16_131072x100", "kind": "knn", "n": 131_072, "dim": 100, "k": 15,
         "distance": "cosine", "precision": "bf16", "data": "sphere"},
        # A million word-vector-like rows already on the GPU: every stage before
        # the optimizer at the largest size.
        {"name": "fit_bf16_1024000x100", "kind": "fit", "n": 1_024_000, "dim": 100, "k": 15,
         "d": 2, "distance": "cosine", "precision": "bf16", "data": "sphere", "host": False},
        # Many small independent data sets of uneven sizes in one run.
        {"name": "batched_bf16_48x64", "kind": "batched", "problems": 48, "low": 500,
         "high": 20_000, "dim": 64, "k": 15, "d": 2, "precision": "bf16"},
        # Graph construction from a large table (hubs included).
        {"name": "symmetrize_800000x15", "kind": "symmetrize", "n": 800_000, "k": 15},
        # The initial embedding of a large graph, odd size, three dimensions.
        {"name": "init_500001_d3", "kind": "init", "n": 500_001, "k": 15, "d": 3},
        # The optimizer's last epochs at a large size (noise staged in windows).
        {"name": "optimize_1000000_d2", "kind": "optimize", "n": 1_000_000, "k": 15, "d": 2,
         "staged": True, "epochs": 5},
        # The same at the default configuration's size (unstaged noise).
        {"name": "optimize_10000_d2", "kind": "optimize", "n": 10_000, "k": 15, "d": 2,
         "staged": False, "epochs": 5},
        # One batch of 2^20 edges for a torch optimizer, plane embedding.
        {"name": "nce_200000_d2", "kind": "nce", "n": 200_000, "edges": 1 << 20, "d": 2,
         "noise": 5, "spread": 3.0},
        # The same in 16 dimensions from the start of a training, ragged batch.
        {"name": "nce_200000_d16", "kind": "nce", "n": 200_000, "edges": 700_001, "d": 16,
         "noise": 5, "spread": 0.01},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["knn", "knn", "knn", "fit", "batched", "symmetrize", "init", "optimize",
                       "optimize", "nce", "nce"])
    if kind == "knn":
        precision = rng.choice(["fp32", "bf16"])
        data = rng.choice(["mixture", "sphere"])
        distance = (rng.choice(["cosine", "correlation", "inner_product"]) if data == "sphere"
                    else "euclidean")
        return {"kind": kind, "n": _log_int(rng, 500, 70_000 if precision == "fp32" else 250_000),
                "dim": rng.randint(8, 126), "k": rng.randint(5, 30), "distance": distance,
                "precision": precision, "data": data}
    if kind == "fit":
        host = rng.random() < 0.5
        precision = rng.choice(["fp32", "bf16"])
        return {"kind": kind, "n": _log_int(rng, 2000, 40_000 if precision == "fp32" else 300_000),
                "dim": rng.randint(16, 126), "k": rng.randint(8, 20), "d": rng.randint(1, 4),
                "distance": "cosine", "precision": precision, "data": "sphere", "host": host}
    if kind == "batched":
        return {"kind": kind, "problems": rng.randint(4, 60), "low": rng.randint(200, 500),
                "high": rng.randint(2000, 15_000), "dim": rng.randint(16, 100),
                "k": rng.randint(8, 20), "d": rng.randint(1, 4),
                "precision": rng.choice(["fp32", "bf16"])}
    if kind == "symmetrize":
        return {"kind": kind, "n": _log_int(rng, 2000, 800_000), "k": rng.randint(5, 30)}
    if kind == "init":
        return {"kind": kind, "n": _log_int(rng, 2000, 800_000), "k": rng.randint(5, 25),
                "d": rng.choice([1, 2, 2, 3, 4, 8])}
    if kind == "optimize":
        staged = rng.random() < 0.5
        n = _log_int(rng, 70_000, 900_000) if staged else _log_int(rng, 3000, 60_000)
        return {"kind": kind, "n": n, "k": rng.randint(8, 20), "d": rng.choice([1, 2, 2, 3, 4]),
                "staged": staged, "epochs": rng.randint(2, 5)}
    return {"kind": kind, "n": _log_int(rng, 5000, 400_000), "edges": _log_int(rng, 10_000, 1 << 20),
            "d": rng.choice([1, 2, 2, 3, 4, 8, 16, 24]), "noise": rng.randint(1, 12),
            "spread": rng.choice([0.01, 1.0, 3.0])}


# ---- inputs ---------------------------------------------------------------------


def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFF)
    return g


def _mixture(n, dim, g, comps=10):
    """Gaussian mixture: centres of standard deviation 5, unit clusters."""
    centres = 5.0 * torch.randn((comps, dim), generator=g, device=DEV)
    label = torch.randint(0, comps, (n,), generator=g, device=DEV)
    return centres[label] + torch.randn((n, dim), generator=g, device=DEV)


def _sphere(n, dim, g, comps=128):
    """Unit vectors around `comps` mean directions, at about the spread of a von
    Mises-Fisher mixture of concentration 50 in 100 dimensions."""
    mu = torch.nn.functional.normalize(torch.randn((comps, dim), generator=g, device=DEV), dim=1)
    label = torch.randint(0, comps, (n,), generator=g, device=DEV)
    x = torch.randn((n, dim), generator=g, device=DEV)
    m = mu[label]
    x -= (x * m).sum(1, keepdim=True) * m
    x = torch.nn.functional.normalize(x, dim=1)
    w = (0.42 + 0.07 * torch.randn((n, 1), generator=g, device=DEV)).clamp_(-0.9, 0.9)
    return w * m + (1 - w * w).sqrt() * x


def _points(case, seed):
    make = _sphere if case["data"] == "sphere" else _mixture
    return make(case["n"], case["dim"], _gen(seed, 1))


def _groups(n, seed):
    """The points of every group of a table of n rows, as (first group, ids
    [groups, points]) blocks: about 512 points a group, a group's points far
    apart in the numbering.  The seed says which group has which numbers; the
    order within a group stays, and with it the size of the table's graph."""
    m = max(64, min(512, n // 8))
    count = n // m
    m, more = n // count, n % count  # `more` groups have one point more
    place = torch.randperm(count, generator=_gen(seed, 2), device=DEV)
    ids = torch.arange(m, device=DEV)[None, :] * count + place[:, None]
    extra = m * count + torch.randperm(more, generator=_gen(seed, 3), device=DEV)
    blocks = [(0, torch.cat([ids[:more], extra[:, None]], 1))] if more else []
    return blocks + [(more, ids[more:])], count


def _table(n, k, seed):
    """A neighbour table in the engine's row order (descending distance) with
    hubs: exact neighbours of 24-dimensional Gaussian points within their groups."""
    g = _gen(n, k)
    inds = torch.empty((n, k), dtype=torch.int32, device=DEV)
    dists = torch.empty((n, k), dtype=torch.float32, device=DEV)
    for _, every in _groups(n, seed)[0]:
        for ids in every.split(256):
            count, m = ids.shape
            x = torch.randn((count, m, 24), generator=g, device=DEV)
            d2 = torch.cdist(x, x, compute_mode="donot_use_mm_for_euclid_dist").square()
            d2.diagonal(dim1=1, dim2=2).fill_(float("inf"))
            near, where = torch.topk(d2, k, dim=2, largest=False, sorted=True)
            to = torch.gather(ids.unsqueeze(1).expand(count, m, m), 2, where).flip(2)
            inds[ids.reshape(-1)] = to.reshape(-1, k).to(torch.int32)
            dists[ids.reshape(-1)] = near.flip(2).reshape(-1, k)
    return inds, dists * 2.0 ** (seed % 5)  # data of another unit


def _layout(n, d, seed):
    """An embedding as it looks late in a fit: the points of a group close by,
    the groups spread over the plane (space)."""
    g = _gen(seed, 4)
    blocks, count = _groups(n, seed)
    centres = 8.0 * torch.randn((count, d), generator=g, device=DEV)
    y = 0.7 * torch.randn((n, d), generator=g, device=DEV)
    for first, ids in blocks:
        y[ids.reshape(-1)] += centres[first:first + ids.shape[0]].repeat_interleave(ids.shape[1], 0)
    return y


def _sizes(case):
    """Points per problem, log-uniform; the case alone says them."""
    rng = np.random.default_rng([case["problems"], case["low"], case["high"]])
    u = rng.uniform(math.log(case["low"]), math.log(case["high"]), case["problems"])
    return [int(v) for v in np.exp(u)]


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "knn":
        state["X"] = _points(case, seed)
    elif kind == "fit":
        X = _points(case, seed)
        state["X"] = X.cpu().numpy() if case["host"] else X
        state["vis"] = ncvis.NCVis(d=case["d"], n_neighbors=case["k"], n_epochs=0,
                                   random_seed=SEED, a=A, b=B, distance=case["distance"],
                                   knn_precision=case["precision"])
    elif kind == "batched":
        g = _gen(seed, 3)
        state["Xs"] = [_mixture(n, case["dim"], g, 4 + i % 17)
                       for i, n in enumerate(_sizes(case))]
        state["vis"] = ncvis.NCVis(d=case["d"], n_neighbors=case["k"], n_epochs=0,
                                   random_seed=SEED, a=A, b=B,
                                   knn_precision=case["precision"])
    elif kind == "symmetrize":
        state["inds"], state["dists"] = _table(case["n"], case["k"], seed)
    elif kind == "init":
        inds, dists = _table(case["n"], case["k"], seed)
        state["row_ptr"], state["cols"], _, _ = stages.symmetrize(inds, dists)
    elif kind == "optimize":
        inds, dists = _table(case["n"], case["k"], seed)
        _, state["dst"], _, state["src"] = stages.symmetrize(inds, dists)
        state["Y"] = _layout(case["n"], case["d"], seed)
        state["Q"] = torch.full((1,), -2.0, device=DEV)
        state["plan"] = ncvis.default_noise_plan(EPOCHS)
    else:
        # A batch of the edges of a symmetrized graph, from an offset on.
        n, k = case["n"], 15
        inds, dists = _table(n, k, seed)
        _, dst, _, src = stages.symmetrize(inds, dists)
        e = min(case["edges"], src.shape[0])
        state["offset"] = int(np.random.default_rng(seed).integers(0, src.shape[0] - e + 1))
        at = slice(state["offset"], state["offset"] + e)
        state["src"], state["dst"] = src[at].clone(), dst[at].clone()
        g = _gen(seed, 5)
        state["Y"] = (case["spread"] * torch.randn((n, case["d"]), generator=g,
                                                   device=DEV)).requires_grad_()
        state["Q"] = torch.ones((), device=DEV, requires_grad=True)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "knn":
        return stages.knn(state["X"], case["k"], DISTANCES[case["distance"]],
                          precision=1 if case["precision"] == "bf16" else 0)
    if kind == "fit":
        return state["vis"].fit_transform(state["X"])
    if kind == "batched":
        return state["vis"].fit_transform_batched(state["Xs"])
    if kind == "symmetrize":
        return stages.symmetrize(state["inds"], state["dists"])
    if kind == "init":
        return stages.init_embedding(state["row_ptr"], state["cols"], case["d"], SEED, 20,
                                     1.0 / case["k"])
    if kind == "optimize":
        Y, Q = state["Y"].clone(), state["Q"].clone()
        return stages.optimize(Y, Q, state["src"], state["dst"], SEED, state["plan"], A, B,
                               epoch_begin=EPOCHS - case["epochs"], staged=case["staged"])
    loss = nce.nce_loss(state["Y"], state["Q"], state["src"], state["dst"], case["noise"], A, B,
                        SEED, 7, state["offset"])
    return (loss, *torch.autograd.grad(loss, [state["Y"], state["Q"]]))


def work(case):
    kind = case["kind"]
    k = case.get("k", 15)
    if kind == "batched":
        sizes = _sizes(case)
        return {"bytes": 4.0 * sum(sizes) * (case["dim"] + case["d"]),
                "flops": sum(2.0 * n * n * case["dim"] + 20 * 1.6 * n * k * 2 * case["d"]
                             for n in sizes)}
    n = case["n"]
    edges = 1.6 * n * k  # of the symmetrized graph, about
    if kind == "knn":
        return {"bytes": 4 * n * case["dim"] + 8 * n * k, "flops": 2.0 * n * n * case["dim"]}
    if kind == "fit":
        return {"bytes": 4 * n * (case["dim"] + case["d"]),
                "flops": 2.0 * n * n * case["dim"] + 20 * edges * 2 * case["d"]}
    if kind == "symmetrize":
        return {"bytes": 8 * n * k + 8 * n + 12 * edges, "flops": edges * math.log2(2 * k)}
    if kind == "init":
        return {"bytes": 8 * n + 4 * edges + 4 * n * case["d"],
                "flops": 20 * (2 * edges + 6 * n) * case["d"]}
    if kind == "optimize":
        noise = int(ncvis.default_noise_plan(EPOCHS)[EPOCHS - case["epochs"]:].sum())
        return {"bytes": 8 * edges + 8 * n * case["d"],
                "flops": edges * (case["epochs"] + noise) * (20 + 7 * case["d"])}
    e = case["edges"]
    return {"bytes": 2 * 8 * e + 3 * 4 * n * case["d"],
            "flops": 2 * e * (1 + case["noise"]) * (30 + 6 * case["d"])}


# ---- the same in 64 bits ----------------------------------------------------------


def _exact_knn(case, seed):
    x = _points(case, seed).double()
    n, k = case["n"], case["k"]
    if case["distance"] == "correlation":
        x = x - x.mean(1, keepdim=True)
    if case["distance"] in ("correlation", "cosine"):
        x = x / x.norm(dim=1, keepdim=True)
    euclid = case["distance"] == "euclidean"
    near = torch.empty((n, k), dtype=torch.float64, device=DEV)
    # Candidates by a 32-bit product, far more than are kept; their distances in 64.
    y = x.float()
    half = y.square().sum(1) / 2
    keep = min(n, 4 * k + 16)
    step = max(1, min(n, (1 << 28) // n))
    for s in range(0, n, step):
        score = y[s:s + step] @ y.T
        if euclid:
            score -= half
        cand = torch.topk(score, keep, dim=1, sorted=False).indices
        q = x[s:s + step]
        d = torch.empty(cand.shape, dtype=torch.float64, device=DEV)
        for b in range(0, q.shape[0], 2048):
            c = x[cand[b:b + 2048]]
            p = q[b:b + 2048, None, :]
            d[b:b + 2048] = ((p - c) ** 2).sum(2) if euclid else 1 - (p * c).sum(2)
        d = torch.sort(d, dim=1).values[:, 1:k + 1]
        near[s:s + step] = d.flip(1)
    return None, near


def _uniform(count):
    """The start of the initial embedding: U[0, 1) in 32 bits, the stream of
    pcg64(SEED), whose first state is one step from SEED plus the increment."""
    mult = 2549297995355413924 << 64 | 4865540595714422341
    inc = 6364136223846793005 << 64 | 1442695040888963407
    gen = np.random.PCG64()
    first = ((SEED + inc) * mult + inc) % (1 << 128)
    gen.state = {"bit_generator": "PCG64", "state": {"state": first, "inc": inc},
                 "has_uint32": 0, "uinteger": 0}
    u = gen.random_raw(count).astype(np.float32) * np.float32(2.0 ** -64)
    return np.minimum(u, np.float32(0.99999994))


def _exact_init(case, seed):
    n, d = case["n"], case["d"]
    inds, dists = _table(n, case["k"], seed)
    row_ptr, cols, _, src = stages.symmetrize(inds, dists)  # the input, as prepare() has it
    cols, src = cols.long(), src.long()
    y = torch.from_numpy(_uniform(n * d)).to(DEV).double().view(n, d)
    alpha = float(np.float32(1.0 / case["k"]))
    for _ in range(20):
        z = torch.zeros_like(y)
        for c in range(d):
            z[:, c].index_add_(0, src, alpha * y[:, c][cols])
        z = z - z.mean(0)
        y = z / z.square().mean(0).sqrt()
    return y


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11) on uint64 arrays."""
    low = np.uint64(0xFFFFFFFF)
    m0, m1 = np.uint64(0xD2511F53), np.uint64(0xCD9E8D57)
    for r in range(10):
        p0, p1 = m0 * c0, m1 * c2
        q0 = (k0 + np.uint64(r * 0x9E3779B9 & 0xFFFFFFFF)) & low
        q1 = (k1 + np.uint64(r * 0xBB67AE85 & 0xFFFFFFFF)) & low
        c0, c1, c2, c3 = ((p1 >> np.uint64(32)) ^ c1 ^ q0, p1 & low,
                          (p0 >> np.uint64(32)) ^ c3 ^ q1, p0 & low)
    return c0, c1, c2, c3


def _bounded(lo, hi, n):
    n = np.uint64(n)
    return (hi * n + (lo * n >> np.uint64(32))) >> np.uint64(32)


def _noise(src, n, noise, tag, offset):
    """The loss's documented noise: counter (edge, tag, sample pair), key from the seed."""
    e = np.arange(offset, offset + len(src), dtype=np.uint64)
    zero = np.zeros_like(e)
    k0, k1 = np.uint64(SEED), np.uint64(0x5EED1)
    out = np.empty((len(src), noise), np.int64)
    i = src.astype(np.uint64)
    for s in range(noise):
        r = _philox(e, zero, zero + np.uint64(tag), zero + np.uint64(s >> 1), k0, k1)
        o = _bounded(r[2 * (s & 1)], r[2 * (s & 1) + 1], n)
        for retry in range(1, 65):
            at = np.nonzero(o == i)[0]
            if not len(at):
                break
            z = zero[at]
            r = _philox(e[at], z + np.uint64(retry << 16), z + np.uint64(tag),
                        z + np.uint64((s >> 1) | 0x80000000), k0 ^ np.uint64(retry), k1)
            o[at] = _bounded(r[0], r[1], n)
        out[:, s] = o
    return out


def _exact_nce(case, seed):
    state = prepare(case, seed)
    n, nu = case["n"], case["noise"]
    src, dst = state["src"].long(), state["dst"].long()
    other = torch.from_numpy(_noise(state["src"].cpu().numpy(), n, nu, 7, state["offset"])).to(DEV)
    y = state["Y"].detach().double().requires_grad_()
    q = state["Q"].detach().double().requires_grad_()
    a, b = float(np.float32(A)), float(np.float32(B))
    log_nu = math.log(nu)
    loss = 0.0
    for s in range(nu + 1):
        d2 = (y[src] - y[dst if s == 0 else other[:, s - 1]]).square().sum(1)
        # d2 == 0 (a point with itself) is held off zero: its gradient is zero.
        log_ph = -torch.log1p(a * d2.clamp_min(1e-300) ** b)
        u = (log_nu + q - log_ph) if s == 0 else (log_ph - q - log_nu)
        loss = loss + torch.nn.functional.softplus(u, threshold=60).sum()
    gy, gq = torch.autograd.grad(loss, [y, q])
    return loss.detach(), gy, gq


def exact(case, seed):
    kind = case["kind"]
    if kind == "knn" and case["n"] <= 150_000:
        return _exact_knn(case, seed)
    if kind == "init":
        return _exact_init(case, seed)
    if kind == "nce":
        return _exact_nce(case, seed)
    # fit, batched: the graph below the embedding has no closed 64-bit form
    # (the rows' order and the removal of doubles go by 32-bit ties); the
    # graph's values are copies of the table's; the optimizer's chains race.
    return None
