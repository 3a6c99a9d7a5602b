#!/usr/bin/env python
"""Benchmark of the IVF-PQ search path.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference] [--config 1..5]

Workload (default, --config 2): the deep-embedding-shaped configuration -- 10,000,000 x 96 fp32
L2-normalised draws from a 4,096-component anisotropic Gaussian mixture (seed 1), 10,000 queries,
n_lists 50,000, pq_dim 48, pq_bits 8, k = 10, fp16 look-up table, fp32 internal distances, n_probes
swept over {20, 50, 100, 200}, one batch of 10,000 queries per step.  --config 1, 3, 4, 5 run the other
four benchmark configurations (3 and 4 at the size one GPU holds: 100 M rows and the 125 M-row prefix).
The public datasets these imitate are not available offline; the seeded synthetic generators below
stand in for them.

A step = one search of the whole query batch.  `value` is queries/s with queries resident in HBM;
`e2e` is the same through the C interface with pinned host buffers and the copies inside the timed
region.  Times come from CUDA events on the stream the library launches on (torch's current
stream); the kernels of the fine search are timed by the library's own events around their launches.  `parity`
compares, id for id, what the GPU search returned for the CPU leg's sample of queries with what the
CPU oracle returned for them; with several GPUs `mg_parity` compares the merged result with the
single-GPU result of the same index.

`cpu_baseline` is the CPU oracle (the port of the reference search arithmetic, all host threads) on a
bounded sample of the same queries against the same index.  --impl reference reports that the
reference itself cannot be built offline.
"""
from __future__ import annotations

import argparse
import hashlib
import json
import os
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

# The five benchmark configurations.  `gen` names the generator; `batches` are the small batches whose
# latency is reported beside the throughput batch; `refine_ratio` > 1 re-ranks refine_ratio * k
# candidates exactly (the reference benchmark's own route to high recall with PQ).
CONFIGS = {
    1: dict(name="config 1: small L2, 100k x 128 f32", gen="uniform_centers", n_rows=100_000, dim=128,
            n_components=1024, seed=0, n_queries=1000, n_lists=1024, pq_dim=64, pq_bits=8, k=10,
            probes=(32,), lut="float32", internal="float32", kmeans_n_iters=20,
            kmeans_trainset_fraction=0.5, refine_ratio=1, metric="sqeuclidean", batches=(1, 100)),
    2: dict(name="deep-embedding-shaped L2, 10M x 96 f32", gen="deep", n_rows=10_000_000, dim=96,
            n_components=4096, seed=1, n_queries=10_000, n_lists=50_000, pq_dim=48, pq_bits=8,
            k=10, probes=(20, 50, 100, 200), lut="float16", internal="float32",
            kmeans_n_iters=10, kmeans_trainset_fraction=0.1, refine_ratio=2, metric="sqeuclidean",
            batches=(1, 100)),
    3: dict(name="SIFT-shaped L2, 100M x 128 u8", gen="sift", n_rows=100_000_000, dim=128,
            n_components=16384, seed=2, n_queries=10_000, n_lists=100_000, pq_dim=64, pq_bits=8, k=100,
            probes=(64,), lut="uint8", internal="float32", kmeans_n_iters=8,
            kmeans_trainset_fraction=0.02, refine_ratio=1, metric="sqeuclidean", batches=(1, 100)),
    4: dict(name="int8 L2, 125M-row prefix of 1B x 128 i8", gen="int8", n_rows=125_000_000, dim=128,
            n_components=65536, seed=3, n_queries=10_000, n_lists=262_144, pq_dim=64, pq_bits=8, k=10,
            probes=(128,), lut="uint8", internal="float32", kmeans_n_iters=6,
            kmeans_trainset_fraction=0.02, refine_ratio=1, metric="sqeuclidean", batches=(1, 100)),
    5: dict(name="text-embedding-shaped inner product, 10M x 768 f16, 4-bit codes", gen="vmf",
            n_rows=10_000_000, dim=768, n_components=2048, seed=4, n_queries=10_000, n_lists=32_768,
            pq_dim=384, pq_bits=4, k=10, probes=(100,), lut="float16", internal="float32",
            kmeans_n_iters=8, kmeans_trainset_fraction=0.1, refine_ratio=1, metric="inner_product",
            batches=(1, 10)),
}
# A slice of configuration 3 run beside the headline workload (its own scan roofline: long lists, 8-bit
# look-up table, k = 100 -- the regime where the code scan rather than the table build dominates).
LONG_LISTS = dict(CONFIGS[3], name="config 3 slice: SIFT-shaped L2, 4M x 128 u8", n_rows=4_000_000,
                  n_lists=4000, n_components=2048, n_queries=10_000, kmeans_trainset_fraction=0.1)
METRIC = "IVF-PQ search QPS @ recall@10>=0.95"
FALLBACK_HBM_GBS = 6650.0


def log(*a):
    if int(os.environ.get("RANK", "0")) == 0:
        print(*a, file=sys.stderr, flush=True)


# --------------------------------------------------------------------------------------------
# synthetic data (seeded per chunk, so any prefix or shard can be regenerated independently)
# --------------------------------------------------------------------------------------------
def mixture_model(wl, device):
    import torch
    g = torch.Generator(device="cpu").manual_seed(wl["seed"] * 7919 + 17)
    nc, dim = wl["n_components"], wl["dim"]
    kind = wl["gen"]
    if kind == "sift":
        # centres in [0, 60] plus a per-dimension exponential offset (mean 20): mass skewed to 0-40
        centers = torch.rand(nc, dim, generator=g) * 60.0
        centers = centers + torch.empty(nc, dim).exponential_(1.0 / 20.0, generator=g)
        return centers.to(device), torch.tensor(12.0, device=device)
    if kind == "int8":
        centers = torch.rand(nc, dim, generator=g) * 200.0 - 100.0
        return centers.to(device), torch.tensor(12.0, device=device)
    if kind == "uniform_centers":
        centers = torch.rand(nc, dim, generator=g) * 2.0 - 1.0
        return centers.to(device), torch.tensor(0.15, device=device)
    if kind == "vmf":
        # unit centres; isotropic noise whose norm makes the mean cosine to the centre about 0.8
        centers = torch.nn.functional.normalize(torch.randn(nc, dim, generator=g), dim=1)
        return centers.to(device), torch.tensor(0.75 / np.sqrt(dim), device=device)
    centers = torch.randn(nc, dim, generator=g)
    lo, hi = np.log(0.05), np.log(0.5)
    scales = torch.exp(torch.rand(nc, dim, generator=g) * (hi - lo) + lo)
    # per-component scale is relative to the centre norm, so clusters keep their identity after
    # the rows are L2-normalised
    scales = scales * (centers.norm(dim=1, keepdim=True) / np.sqrt(dim))
    return centers.to(device), scales.to(device)


def data_dtype(wl):
    import torch
    return {"sift": torch.uint8, "int8": torch.int8, "vmf": torch.float16}.get(wl["gen"], torch.float32)


def gen_rows(wl, model, start, count, device, stream_id=0):
    import torch
    centers, scales = model
    g = torch.Generator(device=device).manual_seed(wl["seed"] * 1_000_003 + start + stream_id * 977)
    comp = torch.randint(0, wl["n_components"], (count,), generator=g, device=device)
    noise = torch.randn(count, wl["dim"], generator=g, device=device)
    x = centers[comp] + (scales[comp] if scales.dim() == 2 else scales) * noise
    kind = wl["gen"]
    if kind == "sift":
        return x.round_().clamp_(0, 255).to(torch.uint8)
    if kind == "int8":
        return x.round_().clamp_(-128, 127).to(torch.int8)
    if kind == "uniform_centers":
        return x
    x = torch.nn.functional.normalize(x, dim=1)
    return x.to(torch.float16) if kind == "vmf" else x


def gen_dataset(wl, device):
    import torch
    model = mixture_model(wl, device)
    x = torch.empty((wl["n_rows"], wl["dim"]), device=device, dtype=data_dtype(wl))
    step = 1_000_000
    for s in range(0, wl["n_rows"], step):
        c = min(step, wl["n_rows"] - s)
        x[s:s + c] = gen_rows(wl, model, s, c, device)
    q = gen_rows(wl, model, 0, wl["n_queries"], device, stream_id=1)
    return x, q


def ground_truth(x, q, k, metric="sqeuclidean"):
    """Exact top-k in fp32, in row chunks: smallest squared L2 distance, or largest inner product."""
    import torch
    q = q.float()
    ip = metric == "inner_product"
    qn = (q * q).sum(1, keepdim=True)
    best_d = torch.full((q.shape[0], k), float("inf"), device=q.device)
    best_i = torch.zeros((q.shape[0], k), dtype=torch.int64, device=q.device)
    step = 200_000
    for s in range(0, x.shape[0], step):
        xb = x[s:s + step].float()
        dots = q @ xb.T
        d = -dots if ip else qn + (xb * xb).sum(1)[None, :] - 2.0 * dots
        dd, ii = torch.topk(d, min(k, d.shape[1]), dim=1, largest=False)
        cat_d = torch.cat([best_d, dd], 1)
        cat_i = torch.cat([best_i, ii + s], 1)
        best_d, sel = torch.topk(cat_d, k, dim=1, largest=False)
        best_i = torch.gather(cat_i, 1, sel)
    return best_i


def recall_at_k(found, truth):
    import torch
    hits = (found.unsqueeze(2) == truth.unsqueeze(1)).any(2).sum().item()
    return hits / truth.numel()


# --------------------------------------------------------------------------------------------
# clocks
# --------------------------------------------------------------------------------------------
class ClockSampler:
    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.samples, self.proc, self.gpu = [], None, gpu_index

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.samples.append(line.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=2)
        except Exception:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for s in self.samples:
            p = [t.strip() for t in s.split(",")]
            try:
                sm.append(float(p[0]))
                mx.append(float(p[1]))
                for n, v in zip(names, p[3:7]):
                    if v.lower().startswith("active"):
                        reasons.add(n)
            except Exception:
                pass
        return {"sm_mhz": float(np.median(sm)) if sm else None,
                "sm_max_mhz": float(max(mx)) if mx else None, "reasons": sorted(reasons),
                "samples": len(sm)}


# --------------------------------------------------------------------------------------------
# fixture: dataset, index file, ground truth -- cached in a temp dir for back-to-back runs
# --------------------------------------------------------------------------------------------
def builder_version():
    """Hash of the sources that decide what an index built here contains (a cached fixture of another
    builder is not reused)."""
    h = hashlib.sha1()
    here = os.path.dirname(os.path.abspath(__file__))
    for name in ("build.cu", "index.cu"):
        with open(os.path.join(here, "cuvs_b200", "csrc", name), "rb") as f:
            h.update(f.read())
    return h.hexdigest()[:8]


def cache_dir(wl):
    key = hashlib.sha1((json.dumps(wl, sort_keys=True, default=str) + builder_version()).encode()).hexdigest()[:12]
    base = "/dev/shm" if os.path.isdir("/dev/shm") else tempfile.gettempdir()
    d = os.path.join(base, f"cuvs_b200_bench_{key}")
    os.makedirs(d, exist_ok=True)
    return d


def lut_np(wl):
    return {"float32": np.float32, "float16": np.float16, "uint8": np.uint8}[wl["lut"]]


def k0_of(wl):
    return int(wl["refine_ratio"] * wl["k"]) if wl["refine_ratio"] > 1 else wl["k"]


def single_result_path(d, p, k0):
    return os.path.join(d, f"single_p{p}_k{k0}.npz")


def prepare_fixture(wl, device, need_dataset=False, single_results=False):
    """Returns dict(index_path, queries (device), truth (device), build_s).  Builds what is missing.
    `single_results`: also keep, beside the index, what the single-GPU search returns for every
    n_probes of the workload (k0 candidates, before refinement) -- the multi-GPU parity check reads it."""
    import torch

    from cuvs_b200 import ivf_pq
    d = cache_dir(wl)
    ipath, qpath, tpath = (os.path.join(d, n) for n in ("index.ivfpq", "queries.npy", "truth.npy"))
    done = os.path.join(d, "done")
    out = {"index_path": ipath, "build_s": None, "dir": d}
    if not os.path.exists(done):
        t0 = time.time()
        x, q = gen_dataset(wl, device)
        torch.cuda.synchronize()
        log(f"[bench] generated {tuple(x.shape)} {x.dtype} in {time.time() - t0:.1f}s")
        t0 = time.time()
        params = ivf_pq.IndexParams(n_lists=wl["n_lists"], pq_dim=wl["pq_dim"], pq_bits=wl["pq_bits"],
                                    metric=wl["metric"], kmeans_n_iters=wl["kmeans_n_iters"],
                                    kmeans_trainset_fraction=wl["kmeans_trainset_fraction"])
        index = ivf_pq.build(params, x)
        torch.cuda.synchronize()
        out["build_s"] = time.time() - t0
        log(f"[bench] built index in {out['build_s']:.1f}s")
        t0 = time.time()
        truth = ground_truth(x, q, wl["k"], wl["metric"])
        torch.cuda.synchronize()
        log(f"[bench] exact ground truth in {time.time() - t0:.1f}s")
        ivf_pq.save(ipath, index)
        np.save(qpath, q.cpu().numpy())
        np.save(tpath, truth.cpu().numpy())
        del x, index
        torch.cuda.empty_cache()
        open(done, "w").write("ok")
    out["queries"] = torch.from_numpy(np.load(qpath)).to(device)
    out["truth"] = torch.from_numpy(np.load(tpath)).to(device)
    k0 = k0_of(wl)
    if single_results and not all(os.path.exists(single_result_path(d, p, k0)) for p in wl["probes"]):
        index = ivf_pq.load(ipath)
        nq = out["queries"].shape[0]
        for p in wl["probes"]:
            sp = ivf_pq.SearchParams(n_probes=p, lut_dtype=lut_np(wl),
                                     internal_distance_dtype={"float32": np.float32, "float16": np.float16}[wl["internal"]],
                                     max_internal_batch_size=nq)
            dd, ii = ivf_pq.search(sp, index, out["queries"], k0)
            np.savez(single_result_path(d, p, k0), d=dd.cpu().numpy(), i=ii.cpu().numpy())
        del index
        torch.cuda.empty_cache()
    if need_dataset:      # regenerated from the seeds (refinement reads the original vectors)
        out["dataset"] = gen_dataset(wl, device)[0]
    return out


# --------------------------------------------------------------------------------------------
# parity: GPU result against another result of the same queries, id for id
# --------------------------------------------------------------------------------------------
def parity_record(d_gpu, i_gpu, d_ref, i_ref, tol):
    """Rows must hold the same ids in the same places with bit-equal distances; a row may differ only
    where distances tie within `tol` (relative): every id the GPU returned that the other side did not
    must lie within tol of the other side's distance at that place or of its k-th distance."""
    d_gpu, i_gpu, d_ref, i_ref = (np.asarray(a) for a in (d_gpu, i_gpu, d_ref, i_ref))
    same = (i_gpu == i_ref).all(axis=1)
    bits = (d_gpu.view(np.uint32) == d_ref.view(np.uint32)) | ~np.isfinite(d_ref)
    identical = int((same & bits.all(axis=1)).sum())
    tie_rows, failed = 0, 0
    for r in np.nonzero(~(same & bits.all(axis=1)))[0]:
        ref = dict(zip(i_ref[r].tolist(), d_ref[r].tolist()))
        kth = float(d_ref[r][-1])
        ok = True
        for idv, dv in zip(i_gpu[r].tolist(), d_gpu[r].tolist()):
            want = ref.get(idv, kth)
            if not (abs(dv - want) <= tol * max(abs(want), 1e-30) + 1e-30):
                ok = False
                break
        tie_rows += int(ok)
        failed += int(not ok)
    return {"rows": int(same.shape[0]), "identical": identical, "tie_rows": tie_rows, "failed_rows": failed,
            "tol": tol, "passed": failed == 0 and tie_rows <= max(1, same.shape[0] // 50)}


# --------------------------------------------------------------------------------------------
# CPU baseline (oracle port), bounded sample
# --------------------------------------------------------------------------------------------
def cpu_baseline(index_path, queries_np, wl, n_probes, budget_s=12.0, steps=1, warmup=0,
                 dataset_np=None):
    """The CPU port on all host threads: IVF-PQ search for k0 candidates and, when the workload
    refines, exact re-ranking of those candidates with numpy.  Also returns what the search itself
    (before re-ranking) found for the sample, for the parity check against the GPU."""
    from oracle import oracle as O
    t0 = time.time()
    # all host cores, whatever OMP_NUM_THREADS the launcher put into the environment
    O.lib().orc_set_num_threads(os.cpu_count() or 1)
    ix = O.OracleIndex.load(index_path)
    ix.flat()
    log(f"[bench] oracle loaded the index in {time.time() - t0:.1f}s")
    cores = O.lib().orc_num_threads()
    lut = {"float32": O.CUDA_R_32F, "float16": O.CUDA_R_16F, "uint8": O.CUDA_R_8U}[wl["lut"]]
    internal = {"float32": O.CUDA_R_32F, "float16": O.CUDA_R_16F}[wl["internal"]]
    k = wl["k"]
    k0 = k0_of(wl) if dataset_np is not None else k
    ip = wl["metric"] == "inner_product"
    found = {}

    def run(q):
        d, i = O.search(ix, q, k0, n_probes=n_probes, lut_dtype=lut, internal_dtype=internal)
        found["d"], found["i"] = d, i
        if k0 > k:
            safe = np.where(i == O.OUT_OF_BOUNDS, 0, i)
            v = dataset_np[safe].astype(np.float32)                # [n, k0, dim]
            qf = q.astype(np.float32)
            dd = -(v * qf[:, None, :]).sum(2) if ip else ((v - qf[:, None, :]) ** 2).sum(2)
            dd = np.where(i == O.OUT_OF_BOUNDS, np.inf, dd)
            o = np.argsort(dd, axis=1)[:, :k]
            i = np.take_along_axis(i, o, 1)
        return i

    # size the sample from a probe run
    n0 = min(len(queries_np), max(cores, 32))
    t0 = time.time()
    run(queries_np[:n0])
    per_q = (time.time() - t0) / n0
    n = int(min(len(queries_np), max(n0, budget_s / max(per_q, 1e-9))))
    times = []
    for it in range(warmup + steps):
        t0 = time.time()
        run(queries_np[:n])
        if it >= warmup:
            times.append(time.time() - t0)
    dt = float(np.mean(times))
    what = f"first {n} of {len(queries_np)} queries, n_probes={n_probes}, k={k}"
    if k0 > k:
        what += f", {k0} candidates re-ranked exactly"
    return {"value": n / dt, "unit": "queries/s", "cores": int(cores), "kind": "port",
            "sample": what + "; same index file; C port of the reference arithmetic, OpenMP over queries"}, dt, n, found


# --------------------------------------------------------------------------------------------
def hbm_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        try:
            return float(json.load(open(p))["hbm_gbs"]), "measured"
        except Exception:
            pass
    return FALLBACK_HBM_GBS, "fallback"


# DRAM bytes (read + write) of the bounding kernel per DISTINCT 32-row group of a launch, from an ncu
# capture on a 2 M-row case of this workload (129.8 MB over 67,421 distinct groups of 3 x 512 B).  Traffic
# grows with the distinct groups of a launch, so the full-size figure is this constant times the
# launch's distinct groups.
DRAM_BYTES_PER_UNIQUE_GROUP = 1926.0


def fine_search_record(stats, wl, two_steps, peak):
    """Roofline figures of the kernel that goes over the probed lists, from the library's counters.

    Two steps (large batches): `filter_kernel` decodes every probed list once for up to 128 queries, so its bytes
    are the codes of the distinct lists, one operand row per (query, list) pair and four bounds per pair and
    32-row group; `rescore_kernel` then scores exactly what the bounds leave.  Tables: `scan_kernel` goes over the
    codes of every pair.  `pair_scan`: the codes of every pair's list (what scanning each pair on its own would
    read) over the time of the whole fine search, to compare the two and several GPUs; a list that many queries
    share makes it exceed the peak."""
    nb = max(1, stats.batches)
    scan_ms, merge_ms = stats.scan_ms / nb, stats.merge_ms / nb
    group = -(-wl["pq_dim"] // (128 // wl["pq_bits"])) * 512
    pair_bytes, unique_bytes = stats.scan_groups / nb * group, stats.unique_groups / nb * group
    algo, kernel = pair_bytes, "scan_kernel (LUT build + code scan + top-k)"
    if two_steps:
        length = wl["dim"] // wl["pq_dim"]          # 2 in every workload: no padding in the operand
        chunks = -(-(wl["pq_dim"] * length // 8 + 1) // 2) * 2
        algo = unique_bytes + stats.pairs / nb * chunks * 16 + stats.scan_groups / nb * 16
        kernel = "filter_kernel (tensor-core bounds of every row of the probed lists)"
    ms = scan_ms + (merge_ms if two_steps else 0.0)
    rate = lambda b, t: round(b / (t * 1e-3) / 1e9, 1) if t > 0 else None  # noqa: E731
    ach = rate(algo, scan_ms)
    return {"bound": "hbm", "kernel": kernel, "achieved": ach, "peak": peak, "unit": "GB/s",
            "frac": round(ach / peak, 4) if ach else None, "kernel_ms": round(scan_ms, 4),
            "algorithmic_bytes_per_launch": int(algo), "unique_bytes_per_launch": int(unique_bytes),
            "pair_scan": {"bytes": int(pair_bytes), "ms": round(ms, 4), "rate": rate(pair_bytes, ms), "unit": "GB/s",
                          "kernels": "filter_kernel + rescore_kernel" if two_steps else "scan_kernel"}}


def workload_from_args(args):
    if args.workload == "sift" and args.config == 2:      # older spelling of a configuration-3 slice
        wl = dict(CONFIGS[3], name="SIFT-shaped L2, 20M x 128 u8", n_rows=20_000_000, n_lists=20_000,
                  kmeans_trainset_fraction=0.1, kmeans_n_iters=10)
    else:
        wl = dict(CONFIGS[args.config])
    if args.rows:
        per_list = max(1, wl["n_rows"] // wl["n_lists"])
        wl.update(n_rows=args.rows, n_lists=max(64, args.rows // per_list),
                  n_queries=min(wl["n_queries"], max(100, args.rows // 100)))
        wl["name"] += f" (shrunk to {args.rows} rows)"
    if args.lists:
        wl["n_lists"] = args.lists
        wl["name"] += f" ({args.lists} lists)"
    if args.refine_ratio is not None:
        wl["refine_ratio"] = args.refine_ratio
    return wl


def long_list_record(res, device, peak, steps):
    """The fine search on long lists: a 4 M-row slice of configuration 3 (lists of about 1,000 rows,
    8-bit look-up table, k = 100, n_probes 64), its own roofline figures."""
    import ctypes as C

    import torch

    from cuvs_b200 import _lib as L
    from cuvs_b200 import ivf_pq
    wl = dict(LONG_LISTS)
    fx = prepare_fixture(wl, device)
    index = ivf_pq.load(fx["index_path"])
    q = fx["queries"]
    nq, k, p = q.shape[0], wl["k"], wl["probes"][0]
    sp = ivf_pq.SearchParams(n_probes=p, lut_dtype=np.uint8, max_internal_batch_size=nq)
    lib = L.load()
    d, i = ivf_pq.search(sp, index, q, k, resources=res)
    rec = recall_at_k(i, fx["truth"])
    stats = L.SearchStats()
    L.check(lib.cuvsB200StatsEnable(res.handle, True))
    L.check(lib.cuvsB200StatsGet(res.handle, C.byref(stats), True))
    for _ in range(max(3, steps)):
        ivf_pq.search(sp, index, q, k, resources=res, sync=False)
    L.check(lib.cuvsB200StatsGet(res.handle, C.byref(stats), True))
    L.check(lib.cuvsB200StatsEnable(res.handle, False))
    b = max(1, stats.batches)
    del index
    torch.cuda.empty_cache()
    return {"workload": wl["name"], "n_lists": wl["n_lists"], "n_probes": p, "k": k, "lut_dtype": "uint8",
            "recall_at_k": round(rec, 4), "ms_per_batch": round(sum(getattr(stats, f) for f in
                                                                    ("prep_ms", "coarse_ms", "sort_ms", "scan_ms", "merge_ms")) / b, 4),
            "roofline": fine_search_record(stats, wl, True, peak)}


def run_ours(args):
    import ctypes as C

    import torch
    import torch.distributed as dist

    from cuvs_b200 import _lib as L
    from cuvs_b200 import ivf_pq, mg, refine
    from cuvs_b200.common import Resources, default_resources

    wl = workload_from_args(args)
    probes = tuple(int(p) for p in args.probes.split(",")) if args.probes else wl["probes"]
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local_rank)
    device = torch.device("cuda", local_rank)
    if world > 1:
        # keep stdout to the one JSON line (NCCL prints its version banner there at VERSION level)
        if os.environ.get("NCCL_DEBUG", "").upper() in ("", "VERSION"):
            os.environ["NCCL_DEBUG"] = "WARN"
        dist.init_process_group("nccl", device_id=device)
    res = default_resources()
    lib = L.load()
    k = wl["k"]
    k0 = k0_of(wl)
    refining = k0 > k
    metric = wl["metric"]

    # ---- fixture: rank 0 builds (or finds) it, everyone loads its shard ----
    if rank == 0:
        fx = prepare_fixture(wl, device, need_dataset=refining, single_results=world > 1)
    if world > 1:
        dist.barrier()
    if rank != 0:
        fx = prepare_fixture(wl, device, need_dataset=refining)
    index = mg.load_shard(fx["index_path"], rank, world, res) if world > 1 else ivf_pq.load(fx["index_path"])
    queries, truth = fx["queries"], fx["truth"]
    dataset = fx.get("dataset")
    nq = queries.shape[0]
    lut_dt = lut_np(wl)
    int_dt = {"float32": np.float32, "float16": np.float16}[wl["internal"]]
    comm = mg.RankComm(None, res) if world > 1 else None

    def make_sp(p):
        return ivf_pq.SearchParams(n_probes=p, lut_dtype=lut_dt, internal_distance_dtype=int_dt,
                                   max_internal_batch_size=max(nq, 1))

    cand_i = torch.empty((nq, k0), dtype=torch.int64, device=device)
    cand_d = torch.empty((nq, k0), dtype=torch.float32, device=device)
    out_i0 = torch.empty((nq, k), dtype=torch.int64, device=device)
    out_d0 = torch.empty((nq, k), dtype=torch.float32, device=device)

    def ann_search(sp, q, r, cm, ci, cd):
        """IVF-PQ search for k0 candidates: one call into the C++ host side either way (with several
        GPUs the call enqueues probe slice, all-gathers, scan and merge)."""
        if world > 1:
            return mg.search(sp, index, q, k0, resources=r, sync=False, comm=cm, out=(cd, ci))
        return ivf_pq.search(sp, index, q, k0, ci, cd, r, sync=False)

    def one_search(sp, q=None, outs=None):
        """The whole step: the search above and, with a refine ratio above 1, exact re-ranking to k."""
        q = queries if q is None else q
        out_i, out_d = outs if outs is not None else (out_i0, out_d0)
        d, i = ann_search(sp, q, res, comm, cand_i, cand_d)
        if refining:
            d, i = refine(dataset, q, i, k=k, metric=metric, indices=out_i, distances=out_d,
                          resources=res, sync=False)
        elif outs is not None:
            out_i.copy_(i)
            out_d.copy_(d)
            d, i = out_d, out_i
        return d, i

    def timed(fn, steps, warmup, tail=None):
        for _ in range(warmup):
            fn()
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        t_host = time.perf_counter()
        for _ in range(steps):
            fn()
        t_host = time.perf_counter() - t_host
        if tail is not None:
            tail()          # e.g. make the timing stream wait for copies still in flight
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        if rank == 0:
            log(f"[bench] timed {steps} steps: device {ms / steps:.3f} ms/step, "
                f"host issue {t_host / steps * 1e3:.3f} ms/step")
        if world > 1:
            t = torch.tensor([ms], device=device)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = t.item()
        return ms / steps, t_host / steps * 1e3

    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()

    # ---- recall / QPS sweep over n_probes (the configuration's list, plus smaller values that show
    # where recall starts to fall: on this generator it saturates early) ----
    def sweep_entry(p):
        sp = make_sp(p)
        d, i = one_search(sp)
        torch.cuda.synchronize()
        rec = recall_at_k(i, truth)
        rec_ann = recall_at_k(cand_i[:, :k], truth) if refining else rec
        ms, _ = timed(lambda: one_search(sp), max(2, min(args.steps, 5)), 2)
        log(f"[bench] n_probes={p}: recall@{k}={rec:.4f} (without refinement {rec_ann:.4f})  {nq / ms * 1e3:,.0f} q/s")
        return {"n_probes": p, f"recall_at_{k}": round(rec, 4), "recall_without_refinement": round(rec_ann, 4),
                "qps": round(nq / ms * 1e3, 1), "ms_per_batch": round(ms, 3)}

    sweep = [sweep_entry(p) for p in probes]
    below = [] if (args.probes or args.no_e2e) else [sweep_entry(p) for p in (1, 2, 5, 10) if p < min(probes)]
    rkey = f"recall_at_{k}"
    ok = [s for s in sweep if s[rkey] >= 0.95]
    if ok:
        chosen, target_met = ok[0], True
    else:
        best = max(s[rkey] for s in sweep)
        chosen = [s for s in sweep if s[rkey] >= best - 0.005][0]
        target_met = False
    p_star = chosen["n_probes"]
    sp = make_sp(p_star)

    # ---- multi-GPU parity: the merged result against the single-GPU search of the same index ----
    mg_parity = None
    if world > 1 and rank == 0:
        ref = np.load(single_result_path(fx["dir"], p_star, k0)) if os.path.exists(
            single_result_path(fx["dir"], p_star, k0)) else None
    if world > 1:
        d, i = ann_search(sp, queries, res, comm, cand_i, cand_d)
        torch.cuda.synchronize()
        if rank == 0 and ref is not None:
            # equal distances may come out in another order across parts: tolerance 0 on the values
            mg_parity = parity_record(d.cpu().numpy(), i.cpu().numpy(), ref["d"], ref["i"], 0.0)
            mg_parity["against"] = "single-GPU search of the same index file, same queries, same n_probes"
            log(f"[bench] multi-GPU parity: {mg_parity}")

    # ---- the timed region: K steps, device-resident queries ----
    L.check(lib.cuvsB200StatsEnable(res.handle, True))
    stats = L.SearchStats()
    one_search(sp)
    L.check(lib.cuvsB200StatsGet(res.handle, C.byref(stats), True))
    if comm is not None:
        comm.stats(reset=True)
    launches_before = stats.launches
    ms_step, host_ms = timed(lambda: one_search(sp), args.steps, args.warmup)
    ms_single = ms_step
    L.check(lib.cuvsB200StatsGet(res.handle, C.byref(stats), True))
    n_calls = args.steps + args.warmup
    gpu_launches = int(round((stats.launches - launches_before) * args.steps / n_calls))
    nb = max(1, stats.batches)
    scan_ms = stats.scan_ms / nb
    n_pieces = -(-wl["pq_dim"] // (128 // wl["pq_bits"]))
    unique_groups = stats.unique_groups / nb
    # which kernels a batch takes (every workload here has straight-line codes): see the library's dispatch
    two_steps = comm is None and nq * p_star > 16384 and k0 <= 128
    peak, peak_kind = hbm_peak()
    roofline = fine_search_record(stats, wl, two_steps, peak)
    if comm is None:
        names = {"scan_ms": "bounds_ms", "merge_ms": "exact_scores_ms"} if two_steps else {}
        stage = {names.get(k2, k2): round(getattr(stats, k2) / nb, 4)
                 for k2 in ("prep_ms", "coarse_ms", "sort_ms", "scan_ms", "merge_ms")}
    else:
        # the one-call step of a rank: its own five stages; the scan stage contains the fine search
        # whose kernel time is reported beside it
        cs = comm.stats(reset=True)
        stage = {"select_probes_slice_ms": round(cs["select_ms"], 4),
                 "allgather_probes_ms": round(cs["gather_probes_ms"], 4),
                 "scan_owned_lists_ms": round(cs["scan_ms"], 4), "scan_kernel_ms": round(scan_ms, 4),
                 "allgather_results_ms": round(cs["gather_results_ms"], 4),
                 "merge_parts_ms": round(cs["merge_ms"], 4)}
    stage["host_issue_ms"] = round(host_ms, 4)
    L.check(lib.cuvsB200StatsEnable(res.handle, False))
    ms_ann_only = None
    if refining:
        t, _ = timed(lambda: refine(dataset, queries, cand_i, k=k, metric=metric, indices=out_i0,
                                    distances=out_d0, resources=res, sync=False), args.steps, 1)
        stage["refine_ms"] = round(t, 4)
        ms_ann_only, _ = timed(lambda: ann_search(sp, queries, res, comm, cand_i, cand_d), args.steps, 2)

    # Throughput mode: three batches in flight per GPU (--in-flight), each on its own stream, resources handle and (with
    # several GPUs) communicator -- the serving pattern of the reference's benchmark in throughput
    # mode: several host threads, one stream each -- so that the small kernels and the exchanges of one
    # batch fill the tails of the other's large kernels.  The per-kernel figures above (stage times,
    # roofline, launches) come from the single-stream pass.
    n_streams = max(1, args.in_flight)
    lanes = []
    for _ in range(n_streams):
        r = Resources()
        lanes.append(dict(stream=torch.cuda.Stream(device), res=r,
                          comm=mg.RankComm(None, r) if world > 1 else None,
                          ci=torch.empty_like(cand_i), cd=torch.empty_like(cand_d),
                          oi=torch.empty_like(out_i0), od=torch.empty_like(out_d0)))
    lane_state = {"i": 0}

    def lane_search(q, outs=None, stream_wait=None):
        """One step on the next lane; returns the lane (its stream carries the step)."""
        lane = lanes[lane_state["i"] % n_streams]
        lane_state["i"] += 1
        with torch.cuda.stream(lane["stream"]):
            if stream_wait is not None:
                for ev in stream_wait:
                    lane["stream"].wait_event(ev)
            lane["res"].use_current_stream()
            d, i = ann_search(sp, q, lane["res"], lane["comm"], lane["ci"], lane["cd"])
            oi, od = outs if outs is not None else (lane["oi"], lane["od"])
            if refining:
                refine(dataset, q, i, k=k, metric=metric, indices=oi, distances=od,
                       resources=lane["res"], sync=False)
            elif outs is not None:
                oi.copy_(i)
                od.copy_(d)
        return lane

    def lanes_join():
        main = torch.cuda.current_stream()
        for lane in lanes:
            main.wait_stream(lane["stream"])

    for lane in lanes:
        lane["stream"].wait_stream(torch.cuda.current_stream())
    ms_step, _ = timed(lambda: lane_search(queries), args.steps, args.warmup + n_streams, tail=lanes_join)
    log(f"[bench] {n_streams} batches in flight: {ms_step:.4f} ms/step (one at a time: {ms_single:.4f})")

    # ---- the configuration's small batches: latency per call, synchronised ----
    small = []
    if not args.no_e2e:
        for b in wl["batches"]:
            if b >= nq:
                continue
            qb = queries[:b].contiguous()
            cb_i = torch.empty((b, k0), dtype=torch.int64, device=device)
            cb_d = torch.empty((b, k0), dtype=torch.float32, device=device)
            ob_i = torch.empty((b, k), dtype=torch.int64, device=device)
            ob_d = torch.empty((b, k), dtype=torch.float32, device=device)

            def small_step():
                d, i = ann_search(sp, qb, res, comm, cb_i, cb_d)
                if refining:
                    refine(dataset, qb, i, k=k, metric=metric, indices=ob_i, distances=ob_d,
                           resources=res, sync=False)
                torch.cuda.synchronize()      # latency mode: the caller waits for every batch

            for _ in range(5):
                small_step()
            t0 = time.perf_counter()
            n_rep = 50
            for _ in range(n_rep):
                small_step()
            dt = (time.perf_counter() - t0) / n_rep
            small.append({"batch": b, "latency_ms": round(dt * 1e3, 4), "qps": round(b / dt, 1)})
            log(f"[bench] batch {b}: {dt * 1e3:.3f} ms per call, {b / dt:,.0f} q/s")

    # ---- end to end: pinned host buffers, copies inside the timed region ----
    # Every step copies its queries host -> device and its results device -> host.  The copies run on
    # their own streams with four sets of buffers (two batches are in flight, so two sets would make
    # an input copy wait for the search two steps back to finish): step s+1's and s+2's input copies
    # and step s-1's result copy overlap step s's search (a serving loop's usual multi-buffering); the
    # timed region ends only when the last result has reached the host.
    n_slots = 4
    q_host = queries.cpu().pin_memory()
    q_dev = [torch.empty_like(queries) for _ in range(n_slots)]
    o_dev = [(torch.empty((nq, k), dtype=torch.int64, device=device),
              torch.empty((nq, k), dtype=torch.float32, device=device)) for _ in range(n_slots)]
    i_host = [torch.empty((nq, k), dtype=torch.int64).pin_memory() for _ in range(n_slots)]
    d_host = [torch.empty((nq, k), dtype=torch.float32).pin_memory() for _ in range(n_slots)]
    s_in, s_out = torch.cuda.Stream(device), torch.cuda.Stream(device)
    ev_in = [torch.cuda.Event() for _ in range(n_slots)]
    ev_done = [torch.cuda.Event() for _ in range(n_slots)]
    ev_out = [torch.cuda.Event() for _ in range(n_slots)]
    e2e_state = {"step": 0}

    def e2e_step():
        s = e2e_state["step"]
        slot = s % n_slots
        with torch.cuda.stream(s_in):
            if s >= n_slots:
                s_in.wait_event(ev_done[slot])       # the search n_slots steps back has read this buffer
            q_dev[slot].copy_(q_host, non_blocking=True)
            ev_in[slot].record(s_in)
        # the search runs on its lane's stream, behind this step's input copy and the result copy that
        # last used the output buffer
        lane = lane_search(q_dev[slot], o_dev[slot], [ev_in[slot]] + ([ev_out[slot]] if s >= n_slots else []))
        ev_done[slot].record(lane["stream"])
        with torch.cuda.stream(s_out):
            s_out.wait_event(ev_done[slot])
            i_host[slot].copy_(o_dev[slot][0], non_blocking=True)
            d_host[slot].copy_(o_dev[slot][1], non_blocking=True)
            ev_out[slot].record(s_out)
        e2e_state["step"] = s + 1

    def e2e_tail():
        main = torch.cuda.current_stream()
        for ev in ev_out:
            main.wait_event(ev)
        lanes_join()

    if args.no_e2e:
        ms_e2e, e2e_rec = float("nan"), float("nan")
    else:
        ms_e2e, _ = timed(e2e_step, args.steps, args.warmup, tail=e2e_tail)
        last = (e2e_state["step"] - 1) % n_slots
        e2e_rec = recall_at_k(i_host[last].to(device), truth)
    clocks = sampler.stop() if rank == 0 else None

    if rank != 0:
        if world > 1:
            dist.barrier()
            dist.destroy_process_group()
        return

    traffic = int(DRAM_BYTES_PER_UNIQUE_GROUP * unique_groups) if wl["gen"] == "deep" and two_steps else None
    config = {"workload": wl["name"], "n_rows": wl["n_rows"], "dim": wl["dim"],
              "n_lists": wl["n_lists"], "pq_dim": wl["pq_dim"], "pq_bits": wl["pq_bits"], "metric": metric,
              "k": k, "recall_k": k, "batch": nq, "n_probes": p_star, "lut_dtype": wl["lut"],
              "internal_distance_dtype": wl["internal"], "refine_ratio": wl["refine_ratio"],
              rkey: chosen[rkey], "recall_without_refinement": chosen["recall_without_refinement"],
              "recall_target_met": target_met, "sweep": sweep, "sweep_below_the_configured_probes": below,
              "recall_note": "on this generator recall is flat over the configured n_probes (queries fall next to "
                             "their component's lists) and falls only below about 10 probes (see "
                             "sweep_below_the_configured_probes): the operating point is the first configured "
                             "n_probes; what lifts recall over 0.95 is the exact re-ranking" if refining else None,
              "small_batches": small,
              "parallelism": f"list-sharded x{world}, one process per GPU, one C++ call per batch" if world > 1
              else "single GPU",
              "batches_in_flight": n_streams, "ms_per_step_one_batch_in_flight": round(ms_single, 4),
              "ms_per_step_without_refinement": round(ms_ann_only, 4) if ms_ann_only else round(ms_single, 4),
              "l2": f"inputs larger than L2: {wl['n_rows'] * n_pieces * 16 // 1_000_000} MB of codes per pass",
              "stage_ms": stage, "build_s": fx.get("build_s")}
    line = {
        "metric": METRIC, "value": round(nq / ms_step * 1e3, 1), "unit": "queries/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": round(ms_step, 4), "higher_is_better": True,
        # the index and the query batch are the same at every number of GPUs
        "scaling": "strong", "vs_baseline": None,
        "dtype": "f32" if wl["lut"] != "uint8" else "f32 (8-bit float look-up table)",
        "data": "synthetic",
        "config": config,
        "e2e": {"value": round(nq / ms_e2e * 1e3, 1), "unit": "queries/s",
                "h2d_bytes_per_step": int(q_host.numel() * q_host.element_size()),
                "d2h_bytes_per_step": int(nq * k * 12), "ms_per_step": round(ms_e2e, 4),
                "copies": "every step, on side streams with four sets of buffers (overlap the neighbouring steps)",
                rkey: round(e2e_rec, 4)},
        "gpu_launches": gpu_launches,
        "clocks": clocks,
        "roofline": dict(roofline, peak_kind=f"of {peak_kind}", traffic=traffic),
    }
    if mg_parity is not None:
        line["mg_parity"] = mg_parity
    failed = mg_parity is not None and not mg_parity["passed"]
    if world == 1 and not args.no_cpu:
        index_gb = os.path.getsize(fx["index_path"]) / 1e9
        if index_gb > 3.0:
            line["cpu_baseline"] = {"value": None, "unit": "queries/s", "cores": os.cpu_count(), "kind": "port",
                                    "sample": f"skipped: the oracle would have to load a {index_gb:.1f} GB index "
                                              "through Python; the CPU leg runs on --config 1 and 2"}
        else:
            q_np = queries.cpu().numpy()
            cb, _, n_cpu, found = cpu_baseline(fx["index_path"], q_np, wl, p_star,
                                               dataset_np=dataset.cpu().numpy() if refining else None)
            cb["value"] = round(cb["value"], 1)
            line["cpu_baseline"] = cb
            # id-level parity of the timed configuration: the GPU's candidates (before re-ranking)
            # for the CPU leg's sample against the oracle's
            d, i = ivf_pq.search(sp, index, queries[:n_cpu].contiguous(), k0, resources=res)
            tol = 1e-5 if wl["lut"] == "float32" else 1e-2
            par = parity_record(d.cpu().numpy(), i.cpu().numpy(), found["d"][:n_cpu], found["i"][:n_cpu], tol)
            par["against"] = "CPU oracle, same index file, same queries, before re-ranking"
            line["parity"] = par
            log(f"[bench] parity: {par}")
            failed = failed or not par["passed"]
    if world == 1 and args.config == 2 and not args.rows and not args.no_e2e and args.workload == "deep":
        del index
        torch.cuda.empty_cache()
        line["config"]["long_lists"] = long_list_record(res, device, peak, args.steps)
    emit(line)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    if failed:
        log("[bench] PARITY FAILED")
        sys.exit(3)


def run_reference(args):
    """The reference arm would time the reference's own build.  There is none: see the line it prints."""
    if int(os.environ.get("RANK", "0")) == 0:
        emit({"impl": "reference",
              "unavailable": "the reference needs RAFT, RMM and other RAPIDS sources that are not available offline: it "
                             "cannot be built or installed here (its arithmetic restated for the host cores is timed as "
                             "cpu_baseline of the other arm)"})


def emit(line: dict):
    """Write the one JSON line to the process's original stdout."""
    data = (json.dumps(line) + "\n").encode()
    os.write(_REAL_STDOUT, data)


_REAL_STDOUT = 1


def main():
    # Libraries (NCCL's version banner, for one) print to stdout; the contract is ONE JSON line
    # there.  Keep the original stdout for that line and point fd 1 at stderr for everything else.
    global _REAL_STDOUT
    sys.stdout.flush()
    _REAL_STDOUT = os.dup(1)
    os.dup2(2, 1)
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--in-flight", type=int, default=3, dest="in_flight",
                    help="batches in flight per GPU in the throughput passes (streams / resources handles)")
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--rows", type=int, default=0, help="shrink the dataset (testing only)")
    ap.add_argument("--lists", type=int, default=0, help="override n_lists (profiling the coarse stage on a small dataset)")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline leg")
    ap.add_argument("--config", type=int, default=2, choices=[1, 2, 3, 4, 5],
                    help="which of the five benchmark configurations to run (default: 2, the headline)")
    ap.add_argument("--workload", default="deep", choices=["deep", "sift"],
                    help="sift = a 20 M-row slice of configuration 3 (older spelling; see --config)")
    ap.add_argument("--probes", default="", help="comma-separated n_probes to sweep (default: the workload's)")
    ap.add_argument("--no-e2e", action="store_true", help="skip the end-to-end leg (profiling runs)")
    ap.add_argument("--refine-ratio", type=float, default=None,
                    help="candidates fetched per result before exact re-ranking (1 = no refinement)")
    args = ap.parse_args()
    args.warmup = max(3, args.warmup)
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
