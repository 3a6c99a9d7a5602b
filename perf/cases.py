"""Workloads of the IVF-PQ engine, through its public Python entry points.

What a program that uses this engine has it do: answer query batches (one query at a time in a request
path, thousands at a time in an offline job), re-rank the candidates exactly, encode vectors with a
trained model, and reload an index with fresh vectors.  Every case names the shape of the data set and of
the index, the options of the call and the size of the batch; `prepare` makes the data from a seed and
lays out what such a program keeps (the index with its trained model, parameter objects, output arrays of
the throughput cases), `run` is one call -- or the two or three calls that belong together.

Data are seeded Gaussian mixtures with the value distributions of the benchmark's generators: unit-norm
anisotropic float vectors, 8-bit integer vectors, unit-norm half-precision embeddings.  The model of an
index is trained here on the GPU with integer-valued sums, so that one seed always gives the same model
bit for bit: list centres from a sample of the rows and one Lloyd step, codebooks from sampled residuals
and a few Lloyd steps.
"""
import math

import numpy as np
import torch

from cuvs_b200 import ivf_pq, refine
from cuvs_b200 import helpers

_NP = {"float32": np.float32, "float16": np.float16, "uint8": np.uint8, "int8": np.int8}
_BYTES = {"float": 4, "deep": 4, "half": 2, "sift": 1, "int8": 1}


def _search(name, data, n_rows, dim, n_lists, pq_dim, n_queries, n_probes, k, *, pq_bits=8, metric="sqeuclidean",
            lut="float32", internal="float32", coarse="float32", batch=4096, refine_to=0, kept=1.0, wait=True):
    """`refine_to` > 0: the k candidates are re-ranked exactly to so many; `kept` < 1: a bitset filter lets
    that fraction of the rows through; `wait`: the call returns when the result is there (the default of the
    entry point), else results of several batches are in flight as in an offline job."""
    return {"name": name, "op": "search", "data": data, "n_rows": n_rows, "dim": dim, "n_lists": n_lists,
            "pq_dim": pq_dim, "pq_bits": pq_bits, "metric": metric, "n_queries": n_queries, "n_probes": n_probes,
            "k": k, "lut": lut, "internal": internal, "coarse": coarse, "batch": batch, "refine_to": refine_to,
            "kept": kept, "wait": wait}


def listed():
    return [
        # one request against a small index with the default table type: the latency of a call
        _search("one query, 100k rows", "float", 100_000, 128, 1024, 64, 1, 32, 10),
        # a micro-batch of requests against a mid-sized index (thousands of lists)
        _search("100 queries, 2M rows", "deep", 2_000_000, 96, 10_000, 48, 100, 20, 10, lut="float16"),
        # the benchmark's headline workload: an offline batch with exact re-ranking of twice the wanted rows
        _search("10k queries, 10M rows, re-ranked", "deep", 10_000_000, 96, 50_000, 48, 10_000, 20, 20,
                lut="float16", batch=10_000, refine_to=10, wait=False),
        # 8-bit image descriptors, long lists, many neighbours: candidate generation
        _search("10k queries, u8, k 100", "sift", 4_000_000, 128, 4000, 64, 10_000, 64, 100, lut="uint8",
                batch=10_000, wait=False),
        # signed 8-bit vectors, many probes of lists of about 490 rows
        _search("4k queries, i8, 128 probes", "int8", 6_000_000, 128, 12_288, 64, 4000, 128, 10, lut="uint8",
                batch=4000, wait=False),
        # half-precision text embeddings, inner product, 4-bit codes
        _search("2k queries, 768-d f16, 4-bit", "half", 1_000_000, 768, 4096, 384, 2000, 100, 10, pq_bits=4,
                metric="inner_product", lut="float16", batch=2000, wait=False),
        # everything left at its default, cosine distance, a dimension that is no multiple of anything
        _search("5k queries, 100-d cosine, defaults", "float", 500_000, 100, 1024, 0, 5003, 20, 10, metric="cosine"),
        # a thousand candidates per query for a later ranking stage
        _search("500 queries, k 1000", "deep", 1_000_000, 96, 2000, 48, 500, 30, 1000, lut="float16"),
        # only a fifth of the rows may be returned; 6-bit codes, half-precision tables and sums
        _search("777 queries, filtered, 6-bit", "float", 1_000_000, 64, 3000, 32, 777, 40, 10, pq_bits=6,
                lut="float16", internal="float16", coarse="float16", kept=0.2),
        # exact re-ranking alone: 200 candidates per query out of half-precision embeddings
        {"name": "re-rank 4k x 200, 768-d f16", "op": "refine", "data": "half", "n_rows": 1_000_000, "dim": 768,
         "n_queries": 4000, "n_candidates": 200, "k": 100, "metric": "inner_product"},
        # encoding: a million new vectors to list labels and codes with a trained model
        {"name": "encode 1M rows", "op": "transform", "data": "deep", "n_rows": 1_000_003, "dim": 96,
         "n_lists": 16_384, "pq_dim": 48, "pq_bits": 8, "metric": "sqeuclidean"},
        # an index reloaded with fresh vectors under the same model, then the first batch of queries
        {"name": "reload 300k u8 rows, search", "op": "reload", "data": "sift", "n_rows": 300_000, "dim": 128,
         "n_lists": 1024, "pq_dim": 64, "pq_bits": 8, "metric": "sqeuclidean", "n_queries": 500, "n_probes": 20,
         "k": 10, "lut": "float32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _index_shape(rng, data):
    dim = rng.choice((128, 128, 96, 64, 100, 160)) if data in ("sift", "int8") else \
        rng.choice((256, 384, 768)) if data == "half" else rng.choice((64, 96, 96, 100, 128, 200, rng.randint(33, 160)))
    bits = rng.choice((8, 8, 8, 8, 6, 5)) if data != "half" else rng.choice((8, 4, 4))
    pq_dim = max(8, (dim // rng.choice((2, 2, 4))) // 8 * 8)
    if data == "float" and rng.random() < 0.3:
        pq_dim, bits = 0, 8    # left to the engine
    return dim, pq_dim, bits


def draw(rng):
    op = rng.choice(("search",) * 7 + ("refine", "transform", "reload"))
    data = rng.choice(("deep", "deep", "float", "sift", "int8", "half"))
    if op == "refine":
        dim = rng.choice((768, 384)) if data == "half" else rng.choice((96, 128, rng.randint(33, 160)))
        cand = _log(rng, 16, 250)
        return {"op": op, "data": data, "n_rows": _log(rng, 20_000, 1_000_000), "dim": dim,
                "n_queries": _log(rng, 1, 4000), "n_candidates": cand, "k": max(1, min(100, cand // rng.choice((1, 2, 4)))),
                "metric": rng.choice(("sqeuclidean", "inner_product", "cosine"))}
    dim, pq_dim, bits = _index_shape(rng, data)
    metric = rng.choice(("sqeuclidean", "sqeuclidean", "euclidean", "inner_product")) if data != "float" else \
        rng.choice(("sqeuclidean", "inner_product", "cosine"))
    if op == "transform":
        return {"op": op, "data": data, "n_rows": _log(rng, 1000, min(1_000_000, 150_000_000 // dim)), "dim": dim,
                "n_lists": _log(rng, 256, 16_384), "pq_dim": pq_dim, "pq_bits": bits, "metric": metric}
    if op == "reload":
        return {"op": op, "data": data, "n_rows": _log(rng, 20_000, min(300_000, 60_000_000 // dim)), "dim": dim,
                "n_lists": _log(rng, 64, 2048), "pq_dim": pq_dim, "pq_bits": bits, "metric": metric,
                "n_queries": _log(rng, 1, 500), "n_probes": _log(rng, 4, 32), "k": _log(rng, 1, 50),
                "lut": rng.choice(("float32", "float16"))}
    while True:
        n_rows = _log(rng, 50_000, min(4_000_000, 400_000_000 // dim))
        n_lists = max(64, n_rows // _log(rng, 100, 1000))
        n_queries, n_probes = _log(rng, 1, 10_000), min(_log(rng, 8, 128), n_lists // 4)
        k = rng.choice((1, 10, 10, 10, 20, 32, 50, 100, 100, 200, 500))
        if n_queries * n_probes * (n_rows / n_lists) * (pq_dim or dim) <= (1e10 if k <= 128 else 1e9):
            break
    lut = rng.choice(("float32", "float16", "float16", "uint8"))
    throughput = n_queries >= 1000
    return _search("", data, n_rows, dim, n_lists, pq_dim, n_queries, n_probes, k, pq_bits=bits, metric=metric, lut=lut,
                   internal=rng.choice(("float32", "float32", "float32", "float16")) if lut != "float32" else "float32",
                   coarse=rng.choice(("float32", "float32", "float32", "float16")),
                   batch=rng.choice((4096, 10_000)), kept=rng.choice((1.0, 1.0, 1.0, 0.2, 0.6)),
                   wait=not throughput) | {"name": "drawn"}


# ---- data ----------------------------------------------------------------------------------------
def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed((seed * 1_000_003 + salt) % (1 << 62))


def _mixture(case, seed):
    """Centres and scales of the mixture: one component for about 2,000 rows."""
    g, dim, data = _generator(seed, 1), case["dim"], case["data"]
    n = max(32, case["n_rows"] // 2000)
    if data == "sift":
        c = torch.rand(n, dim, generator=g, device="cuda") * 60.0
        return c + torch.empty(n, dim, device="cuda").exponential_(1.0 / 20.0, generator=g), 12.0
    if data == "int8":
        return torch.rand(n, dim, generator=g, device="cuda") * 200.0 - 100.0, 12.0
    if data == "float":
        return torch.rand(n, dim, generator=g, device="cuda") * 2.0 - 1.0, 0.15
    c = torch.randn(n, dim, generator=g, device="cuda")
    if data == "half":
        return torch.nn.functional.normalize(c, dim=1), 0.75 / math.sqrt(dim)
    s = torch.exp(torch.rand(n, dim, generator=g, device="cuda") * math.log(10.0) + math.log(0.05))
    return c, s * (c.norm(dim=1, keepdim=True) / math.sqrt(dim))


def _rows(case, mixture, n, g):
    centers, scales = mixture
    data, out = case["data"], []
    for start in range(0, n, 2_000_000):
        m = min(2_000_000, n - start)
        comp = torch.randint(0, centers.shape[0], (m,), generator=g, device="cuda")
        x = torch.randn(m, case["dim"], generator=g, device="cuda")
        x.mul_(scales[comp] if isinstance(scales, torch.Tensor) else scales).add_(centers[comp])
        if data == "sift":
            x = x.round_().clamp_(0, 255).to(torch.uint8)
        elif data == "int8":
            x = x.round_().clamp_(-128, 127).to(torch.int8)
        elif data != "float":
            x = torch.nn.functional.normalize(x, dim=1)
            x = x.half() if data == "half" else x
        out.append(x)
    return out[0] if len(out) == 1 else torch.cat(out)


# ---- the trained model ---------------------------------------------------------------------------
def _as_float(case, x):
    """Rows in the units the model works in (integers scaled, cosine rows normalised)."""
    f = x.float() / {torch.uint8: 256.0, torch.int8: 128.0}.get(x.dtype, 1.0)
    return torch.nn.functional.normalize(f, dim=1) if case["metric"] == "cosine" else f


def _means(points, labels, old):
    """Mean of the points of every label, summed as integers (the same bits in any order)."""
    n, fix = old.shape[0], 2.0 ** 24
    sums = torch.zeros(old.shape, dtype=torch.int64, device="cuda")
    sums.index_add_(0, labels, (points * fix).to(torch.int64))
    count = torch.bincount(labels, minlength=n).unsqueeze(1)
    return torch.where(count > 0, (sums.double() / (count.clamp(min=1) * fix)).float(), old)


def _model(case, rows, seed):
    """An index with a trained model and no rows."""
    g, dim, n_lists, bits = _generator(seed, 3), case["dim"], case["n_lists"], case["pq_bits"]
    params = ivf_pq.IndexParams(n_lists=n_lists, metric=case["metric"], pq_bits=bits, pq_dim=case["pq_dim"])
    pq_dim = case["pq_dim"] or max(1, (dim // 2 if dim >= 128 else dim) // 32 * 32)
    length, book = -(-dim // pq_dim), 1 << bits
    rot_dim = pq_dim * length
    if rot_dim == dim:
        rotation = torch.eye(dim, device="cuda")
    else:
        a = torch.randn(rot_dim, rot_dim, generator=torch.Generator().manual_seed(7), dtype=torch.float64)
        rotation = torch.linalg.qr(a)[0][:, :dim].float().contiguous().cuda()

    def index_of(centers, codebooks):
        return ivf_pq.build_precomputed(params, dim, codebooks, centers, (centers @ rotation.T).contiguous(), rotation)

    pick = torch.randperm(rows.shape[0], generator=g, device="cuda")
    train = rows[pick[: min(rows.shape[0], max(20 * n_lists, 40_000))]].contiguous()
    train_f = _as_float(case, train)
    centers = train_f[torch.arange(n_lists, device="cuda") % train.shape[0]].contiguous()
    if train.shape[0] < n_lists:    # more lists than rows to sample: spread the repeated ones
        centers = centers * (1 + 0.02 * torch.randn(centers.shape, generator=g, device="cuda"))
    no_books = torch.zeros(pq_dim, length, book, device="cuda")
    labels = ivf_pq.transform(index_of(centers, no_books), train)[0].to(torch.int64)
    centers = _means(train_f, labels, centers)
    if case["metric"] == "cosine":
        centers = torch.nn.functional.normalize(centers, dim=1)
    sample, sample_f = train[:16_384], train_f[:16_384]
    labels = ivf_pq.transform(index_of(centers, no_books), sample)[0].to(torch.int64)
    r = ((sample_f - centers[labels]) @ rotation.T).view(-1, pq_dim, length).transpose(0, 1).contiguous()
    first = torch.randint(0, r.shape[1], (book,), generator=g, device="cuda")
    books = r[:, first].contiguous()                                      # [pq_dim, book, length]
    offset = torch.arange(pq_dim, device="cuda").unsqueeze(1) * book
    for _ in range(3):
        near = torch.empty(r.shape[:2], dtype=torch.int64, device="cuda")
        for j in range(0, pq_dim, 32):
            d2 = books[j:j + 32].square().sum(2).unsqueeze(1) - 2.0 * torch.bmm(r[j:j + 32], books[j:j + 32].transpose(1, 2))
            near[j:j + 32] = d2.argmin(2)
        books = _means(r.reshape(-1, length), (near + offset).reshape(-1), books.reshape(-1, length)).view(pq_dim, book, length)
    return index_of(centers, books.transpose(1, 2).contiguous())


def _search_params(case):
    return ivf_pq.SearchParams(n_probes=case["n_probes"], lut_dtype=_NP[case["lut"]],
                               internal_distance_dtype=_NP[case.get("internal", "float32")],
                               coarse_search_dtype=_NP[case.get("coarse", "float32")],
                               max_internal_batch_size=case.get("batch", 4096))


# ---- the interface -------------------------------------------------------------------------------
def prepare(case, seed):
    mixture = _mixture(case, seed)
    rows = _rows(case, mixture, case["n_rows"], _generator(seed, 2))
    s = {"case": case, "rows": rows}
    if case["op"] == "transform":
        s["index"] = _model(case, rows, seed)
        return s
    s["queries"] = _rows(case, mixture, case["n_queries"], _generator(seed, 4))
    if case["op"] == "refine":
        s["candidates"] = torch.randint(0, case["n_rows"], (case["n_queries"], case["n_candidates"]),
                                        generator=_generator(seed, 5), device="cuda")
        return s
    s["index"], s["ids"] = _model(case, rows, seed), torch.arange(case["n_rows"], device="cuda")
    s["params"] = _search_params(case)
    if case["op"] == "reload":
        return s
    ivf_pq.extend(s["index"], rows, s["ids"])
    s["filter"] = None
    if case["kept"] < 1.0:
        keep = torch.rand(-(-case["n_rows"] // 32) * 32, generator=_generator(seed, 6), device="cuda") < case["kept"]
        bit = torch.ones((), dtype=torch.int64, device="cuda") << torch.arange(32, device="cuda")
        s["filter"] = (keep.view(-1, 32) * bit).sum(1).to(torch.uint32)
    if not case["wait"]:
        n, k = case["n_queries"], case["k"]
        s["out"] = (torch.empty((n, k), dtype=torch.int64, device="cuda"), torch.empty((n, k), device="cuda"))
    if case["refine_to"] == 0:
        s["rows"] = None
    return s


def run(state):
    case = state["case"]
    if case["op"] == "transform":
        return ivf_pq.transform(state["index"], state["rows"])
    if case["op"] == "refine":
        return refine(state["rows"], state["queries"], state["candidates"], k=case["k"], metric=case["metric"])
    if case["op"] == "reload":
        helpers.reset_index(state["index"])
        ivf_pq.extend(state["index"], state["rows"], state["ids"])
        return ivf_pq.search(state["params"], state["index"], state["queries"], case["k"])
    neighbors, distances = state.get("out", (None, None))
    found = ivf_pq.search(state["params"], state["index"], state["queries"], case["k"], neighbors, distances,
                          sync=case["wait"], filter=state["filter"])
    if case["refine_to"] == 0:
        return found
    return refine(state["rows"], state["queries"], found[1], k=case["refine_to"], metric=case["metric"], sync=case["wait"])


def work(case):
    """Bytes: inputs and outputs once, and of the index the centres and the codes of the lists that the
    batch probes (expected number of distinct lists).  Operations: the products with the centres and one
    addition per code of every row in a probed list (search); the products with the candidate rows
    (re-ranking); the products with centres and codebooks (encoding)."""
    dim, n, width = case["dim"], case["n_rows"], _BYTES[case["data"]]
    if case["op"] == "refine":
        pairs = case["n_queries"] * case["n_candidates"]
        distinct = n * -math.expm1(-pairs / n)
        return {"bytes": distinct * dim * width + case["n_queries"] * (dim * width + 12 * case["k"]) + 8 * pairs,
                "flops": 2 * pairs * dim}
    n_lists, book = case["n_lists"], 1 << case["pq_bits"]
    pq_dim = case["pq_dim"] or max(1, (dim // 2 if dim >= 128 else dim) // 32 * 32)
    code = pq_dim * case["pq_bits"] / 8
    encode = {"bytes": n * (dim * width + 4 + code) + 4 * n_lists * dim, "flops": 2.0 * n * dim * (n_lists + book)}
    if case["op"] == "transform":
        return encode
    q, p = case["n_queries"], min(case["n_probes"], n_lists)
    k_out = case.get("refine_to") or case["k"]
    probed = n * -math.expm1(q * math.log1p(-p / n_lists)) if p < n_lists else n
    found = {"bytes": q * (dim * width + 12 * k_out) + 4 * n_lists * dim + 4 * book * dim + probed * code,
             "flops": 2.0 * q * n_lists * dim + q * p * (n / n_lists) * pq_dim}
    if case["op"] == "reload":
        return {"bytes": encode["bytes"] + 16 * n + found["bytes"], "flops": encode["flops"] + found["flops"]}
    if case.get("refine_to"):
        found["bytes"] += q * case["k"] * dim * width
        found["flops"] += 2.0 * q * case["k"] * dim
    if case["kept"] < 1.0:
        found["bytes"] += n / 8 + 8 * probed
    return found


def tolerance(case):
    """Labels and codes are whole numbers and the same in every correct implementation.  Distances are sums
    of at most a few hundred 32-bit terms (16-bit ones where the caller asks for half-precision sums); ids
    may trade places where distances tie to within that."""
    if case["op"] == "transform":
        return "exact"
    if case.get("internal") == "float16":
        return {"rel": 1e-3, "differ": 1e-2}
    return {"rel": 1e-5, "max": 1e-4, "differ": 1e-3}
