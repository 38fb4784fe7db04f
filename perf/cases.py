"""The searches and builds that a user of pynear_gb300 runs, as timed cases.

``listed()`` gives the named cases, ``draw(rng)`` further ones of the same
ranges, ``prepare`` the index and the queries that a program holds before the
call, ``run`` one call through the public classes, ``work`` the bytes and
operations that no implementation can avoid, and ``exact`` the same results
in 64 bits.

Host arrays go in and come out wherever the public call takes host arrays (the
flat, tensor-core flat, k-means and binary IVF classes); the IVF batch and the
Voronoi raster use the calls on CUDA tensors.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import pynear_gb300 as pn
from pynear_gb300 import workloads

FLAT = {"l2": pn.FlatL2Index, "l1": pn.FlatL1Index, "linf": pn.FlatChebyshevIndex}


def listed():
    return [
        # one query against a small table: an interactive lookup, all latency
        {"name": "flat_l2_one", "op": "flat", "metric": "l2", "n": 20_000, "d": 64, "nq": 1, "k": 10},
        # a few queries against a table larger than L2: a service answering requests as they come
        {"name": "flat_l2_few_1m", "op": "flat", "metric": "l2", "n": 1_000_000, "d": 128, "nq": 8, "k": 10},
        # the exact L2 benchmark configuration: one batch of 1,000 against 100k short rows
        {"name": "flat_l2_batch", "op": "flat", "metric": "l2", "n": 100_000, "d": 32, "nq": 1000, "k": 5},
        # ragged everything and a long result list: L1 over rows of 97 floats, 100 neighbours each
        {"name": "flat_l1_odd", "op": "flat", "metric": "l1", "n": 30_011, "d": 97, "nq": 513, "k": 100},
        # the Hamming benchmark configuration: 10,000 queries over a million 512-bit codes
        {"name": "hamming_batch", "op": "hamming", "n": 1_000_000, "nbytes": 64, "nq": 10_000, "k": 10},
        # binary IVF as image matching uses it: build over 256-bit descriptors, then one frame's 1,000 queries
        {"name": "ivfbin_build", "op": "ivfbin", "n": 200_000, "nbytes": 32, "nlist": 256, "nprobe": 8, "nq": 1000,
         "k": 10, "max_iter": 20},
        # bulk exact L2 through the tensor-core shortlist (its benchmark configuration)
        {"name": "tcflat_batch", "op": "tcflat", "n": 1_000_000, "d": 128, "nq": 10_000, "k": 10, "shortlist": 40},
        # the largest IVF batch of the benchmark's 1..4,096 range, queries already on the device
        {"name": "ivf_tc_batch", "op": "ivf", "engine": "tc", "device": True, "n": 400_000, "d": 512, "nlist": 1024,
         "n_probe": 28, "nq": 4096, "k": 10},
        # a small IVF batch from host memory: the other end of that range
        {"name": "ivf_tc_small", "op": "ivf", "engine": "tc", "device": False, "n": 200_000, "d": 256, "nlist": 512,
         "n_probe": 16, "nq": 16, "k": 10},
        # IVFFlatL2Index as its constructor makes it (FP32 engine, the reference's distances)
        {"name": "ivf_fp32_batch", "op": "ivf", "engine": "fp32", "device": False, "n": 200_000, "d": 128,
         "nlist": 512, "n_probe": 10, "nq": 1000, "k": 10},
        # building a coarse quantiser
        {"name": "kmeans_build", "op": "kmeans", "n": 100_000, "d": 64, "k": 256, "max_iter": 20},
        # the Voronoi demo at 4K with its colours
        {"name": "voronoi_4k", "op": "voronoi", "width": 3840, "height": 2160, "seeds": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["flat", "flat", "flat", "hamming", "hamming", "ivfbin", "tcflat", "ivf_tc", "ivf_tc", "ivf_fp32",
                     "kmeans", "voronoi"])
    if op == "flat":
        n, d, k = _log(rng, 1000, 1_000_000), _log(rng, 2, 512), _log(rng, 1, 256)
        n = min(n, 128_000_000 // d)
        nq = min(_log(rng, 1, 1024), max(1, 3_200_000_000 // (n * d)))
        return {"op": "flat", "metric": rng.choice(["l2", "l2", "l1", "linf"]), "n": n, "d": d, "nq": nq, "k": k}
    if op == "hamming":
        n, nb = _log(rng, 1000, 1_000_000), rng.choice([8, 16, 20, 32, 33, 61, 64, 64, 96, 128])
        n = min(n, 64_000_000 // nb)
        nq = min(_log(rng, 1, 10_000), max(1, 640_000_000_000 // (n * nb)))
        return {"op": "hamming", "n": n, "nbytes": nb, "nq": nq, "k": _log(rng, 1, 100)}
    if op == "ivfbin":
        return {"op": "ivfbin", "n": _log(rng, 10_000, 200_000), "nbytes": rng.choice([8, 16, 20, 32, 32]),
                "nlist": _log(rng, 32, 256), "nprobe": _log(rng, 1, 16), "nq": _log(rng, 1, 1000),
                "k": _log(rng, 1, 50), "max_iter": 20}
    if op == "tcflat":
        n, d = _log(rng, 10_000, 1_000_000), rng.randint(16, 256)
        n = min(n, 128_000_000 // d)
        nq = min(_log(rng, 16, 10_000), 1_280_000_000_000 // (n * d))
        return {"op": "tcflat", "n": n, "d": d, "nq": nq, "k": rng.randint(1, 32), "shortlist": rng.choice([32, 40])}
    if op == "ivf_tc":
        n, d, nlist = _log(rng, 50_000, 400_000), rng.randint(64, 512), _log(rng, 128, 1024)
        return {"op": "ivf", "engine": "tc", "device": rng.random() < 0.5, "n": n, "d": d, "nlist": nlist,
                "n_probe": rng.randint(4, 28), "nq": _log(rng, 1, 4096), "k": rng.randint(1, 20)}
    if op == "ivf_fp32":
        n, d, nlist = _log(rng, 10_000, 200_000), rng.randint(16, 128), _log(rng, 64, 512)
        return {"op": "ivf", "engine": "fp32", "device": rng.random() < 0.5, "n": n, "d": d, "nlist": nlist,
                "n_probe": rng.randint(1, 10), "nq": _log(rng, 1, 1000), "k": _log(rng, 1, 100)}
    if op == "kmeans":
        return {"op": "kmeans", "n": _log(rng, 4000, 100_000), "d": rng.randint(8, 64), "k": _log(rng, 16, 256),
                "max_iter": rng.randint(5, 20)}
    return {"op": "voronoi", "width": _log(rng, 200, 3840), "height": _log(rng, 150, 2160),
            "seeds": _log(rng, 4, 4096)}


# ── inputs ─────────────────────────────────────────────────────────────────
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _mixture(g, n, d, nq, centres, sigma, zipf):
    """Rows, queries and the row's component of a Gaussian mixture: centres N(0, I), noise sigma,
    Zipf(1.1) or equal component sizes (the benchmark's generator, drawn on the device)."""
    c = torch.randn(centres, d, generator=g, device="cuda")
    if zipf:
        sizes = torch.from_numpy(workloads.zipf_sizes(n, centres, 1.1)).cuda()
        comp = torch.repeat_interleave(torch.arange(centres, device="cuda"), sizes)
        comp = comp[torch.randperm(n, generator=g, device="cuda")]
    else:
        comp = torch.randint(0, centres, (n,), generator=g, device="cuda")
    x = torch.randn(n, d, generator=g, device="cuda").mul_(sigma).add_(c[comp])
    qc = comp[torch.randint(0, n, (nq,), generator=g, device="cuda")]
    q = torch.randn(nq, d, generator=g, device="cuda").mul_(sigma).add_(c[qc])
    return x, q, comp, c


def _flat_inputs(case, seed):
    g = _gen(seed)
    n, d, nq = case["n"], case["d"], case["nq"]
    return torch.rand(n, d, generator=g, device="cuda"), torch.rand(nq, d, generator=g, device="cuda")


def _binary_inputs(case, seed, flips):
    """Uniform codes; each query is a row with about `flips` of every 512 bits flipped."""
    g = _gen(seed)
    n, nb, nq = case["n"], case["nbytes"], case["nq"]
    db = torch.randint(0, 256, (n, nb), generator=g, device="cuda", dtype=torch.uint8)
    src = torch.randint(0, n, (nq,), generator=g, device="cuda")
    bits = torch.rand(nq, nb, 8, generator=g, device="cuda") < flips / 512.0
    mask = (bits.to(torch.uint8) << torch.arange(8, device="cuda", dtype=torch.uint8)).sum(-1).to(torch.uint8)
    return db, db[src] ^ mask


def _descriptor_inputs(case, seed):
    """Descriptors as image features give them: 512 prototype codes, each row a prototype with about 8 % of its
    bits flipped; queries drawn the same way."""
    g = _gen(seed)
    n, nb, nq = case["n"], case["nbytes"], case["nq"]
    proto = torch.randint(0, 256, (512, nb), generator=g, device="cuda", dtype=torch.uint8)
    which = torch.randint(0, 512, (n + nq,), generator=g, device="cuda")
    bits = torch.rand(n + nq, nb, 8, generator=g, device="cuda") < 0.08
    mask = (bits.to(torch.uint8) << torch.arange(8, device="cuda", dtype=torch.uint8)).sum(-1).to(torch.uint8)
    rows = proto[which] ^ mask
    return rows[:n].contiguous(), rows[n:].contiguous()


def _tc_inputs(case, seed):
    x, q, _, _ = _mixture(_gen(seed), case["n"], case["d"], case["nq"], 1024, 0.3, False)
    return x, q


def _ivf_inputs(case, seed):
    """Mixture with twice as many components as lists; every component belongs to the nearest of nlist chosen
    centres, and a list's centroid is its rows' mean (what k-means over such data ends in)."""
    g = _gen(seed)
    nlist = case["nlist"]
    x, q, comp, c = _mixture(g, case["n"], case["d"], case["nq"], 2 * nlist, 0.3, True)
    pick = torch.randperm(2 * nlist, generator=g, device="cuda")[:nlist]
    labels = torch.cdist(c, c[pick]).argmin(1)[comp]
    cent = torch.zeros(nlist, case["d"], dtype=torch.float64, device="cuda")
    # one list at a time in a fixed order of the rows, so that the same seed gives the same centroids
    order = torch.argsort(labels, stable=True)
    counts = torch.bincount(labels, minlength=nlist)
    ends = torch.cumsum(counts, 0).tolist()
    begin = 0
    for i, end in enumerate(ends):
        if end > begin:
            cent[i] = x[order[begin:end]].to(torch.float64).mean(0)
        begin = end
    return x, q, cent.to(torch.float32), labels.to(torch.int32)


def _kmeans_inputs(case, seed):
    x, _, _, _ = _mixture(_gen(seed), case["n"], case["d"], 1, 2 * case["k"], 0.6, True)
    return x


def prepare(case, seed):
    op = case["op"]
    state = {"op": op, "case": case}
    if op == "flat":
        x, q = _flat_inputs(case, seed)
        ix = FLAT[case["metric"]]()
        ix.set(x.cpu().numpy())
        state.update(index=ix, q=q.cpu().numpy())
    elif op == "hamming":
        x, q = _binary_inputs(case, seed, 24)
        ix = pn.FlatHammingIndex()
        ix.set(x.cpu().numpy())
        state.update(index=ix, q=q.cpu().numpy())
    elif op == "ivfbin":
        x, q = _descriptor_inputs(case, seed)
        ix = pn.IVFFlatBinaryIndex(nlist=case["nlist"], nprobe=case["nprobe"], max_iter=case["max_iter"])
        state.update(index=ix, data=x.cpu().numpy(), q=q.cpu().numpy())
    elif op == "tcflat":
        x, q = _tc_inputs(case, seed)
        ix = pn.FlatL2TCIndex(shortlist=case["shortlist"])
        ix.set(x.cpu().numpy())
        state.update(index=ix, q=q.cpu().numpy())
    elif op == "ivf":
        x, q, cent, labels = _ivf_inputs(case, seed)
        ix = pn.IVFFlatL2Index(n_clusters=case["nlist"], n_probe=case["n_probe"], engine=case["engine"])
        ix.set_assigned(x.cpu().numpy(), cent.cpu().numpy(), labels.cpu().numpy())
        state.update(index=ix)
        if case["device"]:
            nq, k = case["nq"], case["k"]
            state.update(q=q.contiguous(), out=(torch.empty((nq, k), dtype=torch.int64, device="cuda"),
                                                torch.empty((nq, k), dtype=torch.float32, device="cuda"),
                                                torch.empty((nq,), dtype=torch.int64, device="cuda")))
        else:
            state.update(q=q.cpu().numpy())
    elif op == "kmeans":
        state.update(data=_kmeans_inputs(case, seed).cpu().numpy())
    else:
        g = _gen(seed)
        xs = torch.linspace(0, 1, case["width"], device="cuda", dtype=torch.float32)
        ys = torch.linspace(0, 1, case["height"], device="cuda", dtype=torch.float32)
        state.update(seeds=torch.rand(case["seeds"], 2, generator=g, device="cuda"), xs=xs, ys=ys,
                     palette=torch.randint(0, 256, (case["seeds"], 4), generator=g, device="cuda",
                                           dtype=torch.uint8))
    torch.cuda.synchronize()
    return state


# ── one call ───────────────────────────────────────────────────────────────
def run(state):
    op, case = state["op"], state["case"]
    if op in ("flat", "hamming", "tcflat"):
        idx, dist = state["index"].search_knn_arrays(state["q"], case["k"])
        return {"idx": idx, "dist": dist}
    if op == "ivfbin":
        ix = state["index"]
        ix.set(state["data"])
        idx, dist, cnt = ix.search_knn_arrays(state["q"], case["k"])
        cent, labels = ix.export()
        # entries past a query's count carry no result
        keep = np.arange(idx.shape[1])[None, :] < cnt[:, None]
        return {"centroids": cent, "labels": labels, "idx": np.where(keep, idx, -1), "dist": np.where(keep, dist, 0),
                "count": cnt}
    if op == "ivf":
        if case["device"]:
            idx, dist, cnt = state["out"]
            state["index"].search_knn_device(state["q"], case["k"], idx, dist, cnt)
        else:
            idx, dist, cnt = state["index"].search_knn_arrays(state["q"], case["k"])
        return {"idx": idx, "dist": dist, "count": cnt}
    if op == "kmeans":
        labels, cent = pn.kmeans_l2(state["data"], case["k"], max_iter=case["max_iter"])
        return {"labels": labels, "centroids": cent}
    r = pn.voronoi_raster_device(state["seeds"], state["xs"], state["ys"], palette=state["palette"])
    return {"ids": r.ids, "rgba": r.rgba}


# ── what a pass cannot do without ──────────────────────────────────────────
def work(case):
    op = case["op"]
    if op == "flat":
        n, d, nq, k = case["n"], case["d"], case["nq"], case["k"]
        return {"bytes": 4 * d * (n + nq) + 12 * nq * k, "flops": 3 * n * nq * d}
    if op == "hamming":  # per pair and 32-bit word: exclusive or, bit count, add
        n, nb, nq, k = case["n"], case["nbytes"], case["nq"], case["k"]
        return {"bytes": nb * (n + nq) + 16 * nq * k, "flops": 3 * n * nq * math.ceil(nb / 4)}
    if op == "ivfbin":  # seeding and one assignment score every row against every list; the search its probed lists
        n, nb, nq = case["n"], case["nbytes"], case["nq"]
        pairs = 2 * n * case["nlist"] + nq * (case["nlist"] + n * case["nprobe"] // case["nlist"])
        return {"bytes": 2 * nb * n + nb * nq + 4 * n, "flops": 3 * pairs * math.ceil(nb / 4)}
    if op == "tcflat":  # 16-bit scores of every pair, then k exact rows per query
        n, d, nq, k = case["n"], case["d"], case["nq"], case["k"]
        return {"bytes": 2 * d * n + 4 * d * nq + nq * k * (4 * d + 12), "flops": 2 * n * nq * d}
    if op == "ivf":
        n, d, nq, k, nlist = case["n"], case["d"], case["nq"], case["k"], case["nlist"]
        rows = nq * case["n_probe"] * (n // nlist)
        size = 2 if case["engine"] == "tc" else 4
        return {"bytes": size * d * min(n, rows) + 4 * d * (nq + nlist) + 20 * nq * k,
                "flops": 2 * d * (rows + nq * nlist)}
    if op == "kmeans":  # seeding distances, then one inner product per row, centroid and iteration
        n, d, k = case["n"], case["d"], case["k"]
        return {"bytes": 4 * n * d + 4 * k * d + 4 * n, "flops": (3 + 2 * case["max_iter"]) * n * d * k}
    px = case["width"] * case["height"]  # one distance per pixel at least; ids and colours out
    return {"bytes": 8 * px + 12 * case["seeds"], "flops": 6 * px}


# ── the same results in 64 bits ────────────────────────────────────────────
def _nearest(x, q, k, allowed=None):
    """The k smallest squared distances per query in 64 bits: candidates by the expanded form, then the
    difference form. allowed(a, b): for queries a..b, the (b - a, n) mask of rows that count."""
    x = x.to(torch.float64)
    q = q.to(torch.float64)
    xn = (x * x).sum(1)
    out = torch.full((q.shape[0], k), math.inf, dtype=torch.float64, device=x.device)
    step = max(1, min(q.shape[0], 400_000_000 // x.shape[0]))
    m = min(x.shape[0], k + 8)
    for a in range(0, q.shape[0], step):
        s = torch.addmm(xn, q[a:a + step], x.T, alpha=-2.0)
        if allowed is not None:
            s.masked_fill_(~allowed(a, min(q.shape[0], a + step)), math.inf)
        v, i = torch.topk(s, m, dim=1, largest=False)
        del s
        e = ((x[i] - q[a:a + step, None, :]) ** 2).sum(2).masked_fill_(torch.isinf(v), math.inf)
        e = torch.sort(e, dim=1).values[:, :k]
        out[a:a + step, :e.shape[1]] = e
    return out


def exact(case, seed):
    op = case["op"]
    if op == "flat":
        x, q = _flat_inputs(case, seed)
        k = min(case["k"], case["n"])
        if case["metric"] == "l2":
            dist = _nearest(x, q, k).sqrt()
        else:
            p = 1.0 if case["metric"] == "l1" else math.inf
            x, q = x.to(torch.float64), q.to(torch.float64)
            step = max(1, 200_000_000 // x.shape[0])
            dist = torch.cat([torch.sort(torch.topk(torch.cdist(q[a:a + step], x, p=p), k, dim=1,
                                                    largest=False).values, dim=1).values
                              for a in range(0, q.shape[0], step)])
        return {"idx": None, "dist": dist}
    if op == "tcflat":
        x, q = _tc_inputs(case, seed)
        return {"idx": None, "dist": _nearest(x, q, case["k"]).sqrt()}
    if op == "ivf":
        x, q, cent, labels = _ivf_inputs(case, seed)
        c = cent.to(torch.float64)
        q64, lab = q.to(torch.float64), labels.long()
        full = torch.bincount(lab, minlength=case["nlist"]) > 0  # empty lists are dropped
        probed = torch.zeros(q.shape[0], case["nlist"], dtype=torch.bool, device="cuda")
        near = ((c * c).sum(1) - 2.0 * (q64 @ c.T)).masked_fill(~full, math.inf)
        probed.scatter_(1, torch.topk(near, min(case["n_probe"], int(full.sum())), dim=1, largest=False).indices,
                        True)
        dist = _nearest(x, q, case["k"], lambda a, b: probed[a:b][:, lab])
        # a query whose probed lists hold fewer than k rows has no value past its count
        return {"idx": None, "dist": dist if bool(torch.isfinite(dist).all()) else None, "count": None}
    # Hamming, binary IVF and the raster give whole numbers only; Lloyd's iterations from the library's own
    # seeds have no 64-bit counterpart (one label that flips changes every later step)
    return None
