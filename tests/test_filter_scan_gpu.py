"""The two-step fine search (tensor-core bounds, then exact scores of what they leave), forced on at every size,
against the CPU oracle: ids and distance bits."""
import numpy as np
import pytest

from conftest import make_mixture
from test_search_gpu import LUT, assert_parity, build_case, gpu_search

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(autouse=True)
def two_step():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cuvs_b200 import _lib as L
    L.check(L.load().cuvsB200SetScanCodebookHome(4))
    yield
    L.check(L.load().cuvsB200SetScanCodebookHome(0))


@pytest.fixture(scope="module")
def ivf():
    from cuvs_b200 import ivf_pq
    return ivf_pq


def check(ivf, O, ix, path, q, k, p, lut, internal, tol=1e-5):
    d, i = gpu_search(ivf, ivf.load(path), q, k, p, lut, internal)
    do, io = O.search(ix, q, k, n_probes=p, lut_dtype=LUT[lut][1], internal_dtype=LUT[internal][1])
    assert_parity(d, i, do, io, tol)


# code widths x components per subspace (padded to 1, 2, 4 or a multiple of 8 in the operand)
@pytest.mark.parametrize("bits,dim,pq_dim", [(8, 16, 16), (8, 96, 48), (8, 57, 19), (8, 32, 8), (8, 40, 8), (8, 64, 8),
                                             (8, 96, 8), (4, 16, 16), (4, 64, 32), (4, 32, 8), (4, 48, 6), (4, 90, 10),
                                             (5, 32, 16), (6, 48, 12), (7, 80, 16), (6, 100, 8)])
@pytest.mark.parametrize("metric", [0, 6])
def test_code_widths_and_lengths(ivf, oracle_mod, tmp_path, bits, dim, pq_dim, metric):
    x, q, ix, path = build_case(oracle_mod, tmp_path, "w", n=1500, dim=dim, n_lists=12, pq_dim=pq_dim, pq_bits=bits,
                                metric=metric, nq=40)
    for lut in ("f32", "f16"):
        check(ivf, oracle_mod, ix, path, q, 10, 5, lut, "f32", 1e-5 if lut == "f32" else 1e-2)


@pytest.mark.parametrize("metric,lut,internal", [(0, "f32", "f32"), (1, "f16", "f32"), (0, "fp8", "f32"), (0, "f16", "f16"),
                                                 (0, "fp8", "f16"), (2, "f32", "f32"), (2, "f16", "f32"), (6, "f16", "f32")])
# (k > 128 takes the look-up tables, forced or not)
@pytest.mark.parametrize("k", [1, 16, 17, 64, 65, 100, 128, 300])
def test_k_and_types(ivf, oracle_mod, tmp_path, metric, lut, internal, k):
    x, q, ix, path = build_case(oracle_mod, tmp_path, "k", n=4000, dim=48, n_lists=16, pq_dim=24, metric=metric, nq=24)
    check(ivf, oracle_mod, ix, path, q, k, 6, lut, internal, 1e-5 if lut == "f32" else 1e-2)


@pytest.mark.parametrize("n_queries", [1, 16, 17, 128, 129, 400])
def test_list_sizes_and_queries_per_list(ivf, oracle_mod, tmp_path, n_queries):
    """Lists around the edges of groups (32 rows) and tiles (256 rows), empty ones among them, each probed by every
    query: one tile of pairs, its edges, and several."""
    O = oracle_mod
    x, q, ix, path = build_case(O, tmp_path, "r", n=2000, n_lists=12, nq=n_queries)
    sizes = [0, 1, 31, 32, 33, 0, 255, 256, 257, 64, 700, 5]
    rng = np.random.default_rng(0)
    codes, ids, nxt = [], [], 0
    for s in sizes:
        c = rng.integers(0, 256, size=(s, ix.pq_dim), dtype=np.uint8)
        codes.append(O.pack_list(c, 8) if s else np.zeros(0, np.uint8))
        ids.append(np.arange(nxt, nxt + s, dtype=np.int64) * 3 + 7)
        nxt += s
    ix.list_sizes = np.array(sizes, dtype=np.uint32)
    ix.list_codes, ix.list_ids, ix._flat = codes, ids, None
    ix.save(path)
    for p in (1, 5, 12):
        check(ivf, O, ix, path, q, 20, p, "f32", "f32")


def test_filter_and_few_candidates(ivf, oracle_mod, tmp_path):
    """A bitset that lets a handful of rows through: fewer than k results, padded."""
    x, q, ix, path = build_case(oracle_mod, tmp_path, "f", n=3000, n_lists=16, nq=200)
    g = ivf.load(path)
    for keep in (3, 200, 2500):
        allowed = np.zeros(3008, bool)
        allowed[np.random.default_rng(keep).choice(3000, keep, replace=False)] = True
        words = np.packbits(allowed, bitorder="little").view(np.uint32)
        sp = ivf.SearchParams(n_probes=8)
        d, i = ivf.search(sp, g, torch.from_numpy(q).cuda(), 10, filter=torch.from_numpy(words).cuda())
        d, i = d.cpu().numpy(), i.cpu().numpy()
        do, io = oracle_mod.search(ix, q, 10, n_probes=8, bitset=words)
        assert_parity(d, i, do, io, 1e-5)


@pytest.mark.parametrize("scale", [1e-6, 1.0, 300.0, 1e6])
def test_data_scale(ivf, oracle_mod, tmp_path, scale):
    """Operands are scaled into half precision: tiny and huge data, tables whose entries overflow their type, and queries
    far outside the data (differences that half precision cannot hold)."""
    O = oracle_mod
    from conftest import make_mixture
    x = (make_mixture(2000, 32, 30, 0.15, 0) * scale).astype(np.float32)
    q = (make_mixture(48, 32, 30, 0.15, 1) * scale).astype(np.float32)
    q[5] *= 3000.0
    q[6] *= 1e-4
    ix = O.build_index(x, 16, pq_dim=16, pq_bits=8, kmeans_iters=3)
    path = str(tmp_path / "s.ivfpq")
    ix.save(path)
    for lut in ("f32", "fp8") + (("f16",) if scale < 1e3 else ()):
        check(ivf, O, ix, path, q, 10, 6, lut, "f32", 1e-5 if lut == "f32" else 1e-2)


@pytest.mark.parametrize("dim,pq_dim,bits,n_lists,rows,n_queries,metric,lut,batches", [
    # bounds of 501 KB per query, but the look-up tables score these: one batch
    (16, 8, 8, 64, 1_000_000, 5000, "inner_product", np.uint8, 1),
    # the same size with bounds, and a query operand of 803 KB: 2 GiB at a time
    (16, 8, 8, 64, 1_000_000, 5000, "inner_product", np.float16, 2),
    (768, 384, 4, 512, 20_000, 3000, "inner_product", np.float16, 2)])
def test_size_of_an_internal_batch(ivf, dim, pq_dim, bits, n_lists, rows, n_queries, metric, lut, batches):
    import ctypes as C
    from cuvs_b200 import _lib as L
    from cuvs_b200.common import Resources
    g = torch.Generator(device="cuda").manual_seed(4)
    normal = lambda *shape: torch.randn(*shape, generator=g, device="cuda")  # noqa: E731
    centers = normal(n_lists, dim)
    index = ivf.build_precomputed(ivf.IndexParams(n_lists=n_lists, pq_dim=pq_dim, pq_bits=bits, metric=metric), dim,
                                  normal(pq_dim, dim // pq_dim, 1 << bits) * 0.3, centers, centers,
                                  torch.eye(dim, device="cuda"))
    x = centers[torch.arange(rows, device="cuda") % n_lists] + 0.3 * normal(rows, dim)
    ivf.extend(index, x, torch.arange(rows, device="cuda"))
    q = x[:n_queries] + 0.1 * normal(n_queries, dim)
    res, lib, stats = Resources(), L.load(), L.SearchStats()
    L.check(lib.cuvsB200StatsEnable(res.handle, True))
    p = dict(n_probes=n_lists, lut_dtype=lut)
    d, i = ivf.search(ivf.SearchParams(max_internal_batch_size=n_queries, **p), index, q, 10, resources=res)
    L.check(lib.cuvsB200StatsGet(res.handle, C.byref(stats), True))
    assert stats.batches == batches
    d2, i2 = ivf.search(ivf.SearchParams(max_internal_batch_size=1000, **p), index, q, 10, resources=res)
    assert bool((i == i2).all()) and bool((d == d2).all())


@pytest.mark.parametrize("lut,internal,bits,k", [("f32", "f32", 8, 10), ("fp8", "f32", 8, 100), ("f16", "f16", 6, 17)])
def test_a_wait_that_runs_out_scores_every_row(ivf, oracle_mod, tmp_path, lut, internal, bits, k):
    """One block of every CTA's first tile never comes and the limit is about a millisecond: the bounding kernel gives up,
    the exact pass scores every row of the probed lists, the handle counts the batch, and the next search is a healthy
    one.  (Sixteen lists: the coarse search does not run on the tensor cores.)"""
    import ctypes as C
    from cuvs_b200 import _lib as L
    from cuvs_b200.common import Resources
    x, q, ix, path = build_case(oracle_mod, tmp_path, "t", n=3000, dim=48, n_lists=16, pq_dim=24, pq_bits=bits, nq=40)
    do, io = oracle_mod.search(ix, q, k, n_probes=9, lut_dtype=LUT[lut][1], internal_dtype=LUT[internal][1])
    g, lib, res = ivf.load(path), L.load(), Resources()
    sp = ivf.SearchParams(n_probes=9, lut_dtype=LUT[lut][0], internal_distance_dtype=LUT[internal][0])

    def search():
        d, i = ivf.search(sp, g, torch.from_numpy(q).cuda(), k, resources=res)
        n = C.c_uint64(0)
        L.check(lib.cuvsStreamSync(res.handle))
        L.check(lib.cuvsB200CoarseTimeouts(res.handle, C.byref(n)))
        assert_parity(d.cpu().numpy(), i.cpu().numpy(), do, io, 1e-5 if lut == "f32" else 1e-2)
        return n.value

    try:
        L.check(lib.cuvsB200SetCoarseWaitTest(1000, 1))
        assert search() == 1
    finally:
        L.check(lib.cuvsB200SetCoarseWaitTest(0, 0))
    assert search() == 1


def odd_queries(q):
    """NaN, infinities, zeros, and values at the ends of the ranges of fp32, half precision and the 8-bit float."""
    q = q.copy()
    q[0, 3], q[1], q[2, 5], q[3], q[4] = np.nan, np.nan, np.inf, -np.inf, 0.0
    q[5], q[6, 0], q[8], q[9, 1], q[10], q[11], q[12] = 1e30, -1e30, 1e4, 3e4, 1e19, 3e18, 300.0
    q[7] *= 1e-7
    q[13] *= 1e12
    return q


@pytest.mark.parametrize("metric,bits,dim,pq_dim", [(0, 8, 64, 32), (1, 8, 64, 64), (0, 6, 48, 24), (2, 8, 40, 24), (6, 8, 64, 32),
                                                    (6, 4, 64, 32)])
@pytest.mark.parametrize("lut,internal", [("f32", "f32"), ("f16", "f32"), ("fp8", "f32"), ("f16", "f16"), ("fp8", "f16")])
def test_odd_queries_answer_as_with_tables(ivf, oracle_mod, tmp_path, metric, bits, dim, pq_dim, lut, internal):
    from cuvs_b200 import _lib as L
    x, q, _, path = build_case(oracle_mod, tmp_path, "o", n=2500, dim=dim, n_lists=16, pq_dim=pq_dim, pq_bits=bits, metric=metric,
                               nq=80)
    g, q = ivf.load(path), odd_queries(q)
    for k in (1, 10, 100):
        d2, i2 = gpu_search(ivf, g, q, k, 7, lut, internal)
        L.check(L.load().cuvsB200SetScanCodebookHome(2))
        d0, i0 = gpu_search(ivf, g, q, k, 7, lut, internal)
        L.check(L.load().cuvsB200SetScanCodebookHome(4))
        assert (i0 == i2).all(), np.nonzero((i0 != i2).any(1))[0]
        assert (d0.view(np.uint32) == d2.view(np.uint32)).all(), np.nonzero((d0.view(np.uint32) != d2.view(np.uint32)).any(1))[0]


# (squares and products that underflow fp32 partly or wholly, and large ones)
@pytest.mark.parametrize("data_scale,query_scale", [(1.0, 1e-14), (1.0, 1e-17), (1.0, 1e-20), (1.0, 1e-38), (1.0, 1e18), (1e-13, 1e-13),
                                                    (1e-17, 1e-17), (1e-19, 1e-19), (1e-20, 1.0), (1e16, 1e16)])
@pytest.mark.parametrize("metric", [0, 6])
def test_scales_at_the_ends_of_fp32_answer_as_with_tables(ivf, oracle_mod, tmp_path, metric, data_scale, query_scale):
    from cuvs_b200 import _lib as L
    x, q, ix, path = build_case(oracle_mod, tmp_path, "e", n=2500, dim=48, n_lists=16, pq_dim=24, metric=metric, nq=80)
    for a in (ix.pq_centers, ix.centers, ix.centers_rot):
        a *= np.float32(data_scale)
    ix.centers[:, 48] *= np.float32(data_scale)
    ix.save(path)
    g, q = ivf.load(path), (q * np.float32(query_scale)).astype(np.float32)
    for lut in ("f32", "f16"):
        d2, i2 = gpu_search(ivf, g, q, 10, 7, lut)
        L.check(L.load().cuvsB200SetScanCodebookHome(2))
        d0, i0 = gpu_search(ivf, g, q, 10, 7, lut)
        L.check(L.load().cuvsB200SetScanCodebookHome(4))
        assert (i0 == i2).all(), np.nonzero((i0 != i2).any(1))[0]
        assert (d0.view(np.uint32) == d2.view(np.uint32)).all()


def test_workspace_of_a_skewed_index(ivf):
    """One list of 400,000 rows, 4,000 of 25, each query probes 512 of them: bounds 2.1 GB, operand 0.33 GB, and tiles for what
    10,000 queries can probe (25 MB; a bound by the longest list alone asks for 9 GB)."""
    from cuvs_b200.common import Resources
    g = torch.Generator(device="cuda").manual_seed(4)
    n_lists, dim, long_list = 4001, 16, 400_000
    centers = torch.randn(n_lists, dim, generator=g, device="cuda") * 4
    index = ivf.build_precomputed(ivf.IndexParams(n_lists=n_lists, pq_dim=8), dim,
                                  torch.randn(8, 2, 256, generator=g, device="cuda") * 0.3, centers, centers,
                                  torch.eye(dim, device="cuda"))
    which = torch.cat([torch.zeros(long_list, dtype=torch.int64, device="cuda"),
                       torch.arange(100_000, device="cuda") % (n_lists - 1) + 1])
    x = centers[which] + 0.2 * torch.randn(which.numel(), dim, generator=g, device="cuda")
    ivf.extend(index, x, torch.arange(which.numel(), device="cuda"))
    assert int(index.list_sizes.to(torch.int64).max()) > 300_000
    q = x[torch.randint(0, x.shape[0], (10_000,), generator=g, device="cuda")].contiguous()
    sp = lambda b: ivf.SearchParams(n_probes=512, lut_dtype=np.float16, max_internal_batch_size=b)  # noqa: E731
    torch.cuda.empty_cache()
    free, res = torch.cuda.mem_get_info()[0], Resources()
    d, i = ivf.search(sp(10_000), index, q, 10, resources=res)
    used = free - torch.cuda.mem_get_info()[0]
    assert used < 4 << 30, used
    d2, i2 = ivf.search(sp(500), index, q, 10)
    assert bool((i == i2).all()) and bool((d == d2).all())


# rows left by their distance above the unit's value: tight bounds (steps saturate), wide bounds with many neighbours, signed scores,
# lists that end inside a unit; against the tables bit for bit
@pytest.mark.parametrize("metric,lut,k", [("sqeuclidean", "f16", 20), ("sqeuclidean", "f32", 128), ("sqeuclidean", "fp8", 100),
                                          ("inner_product", "f16", 10), ("cosine", "f32", 65)])
@pytest.mark.parametrize("dim,pq_dim,bits", [(96, 48, 8), (64, 32, 4), (50, 24, 6)])
def test_row_codes_leave_what_the_tables_find(ivf, metric, lut, k, dim, pq_dim, bits):
    from cuvs_b200 import _lib as L
    x = make_mixture(60_001, dim, 60, 0.3, seed=dim)
    q = make_mixture(900, dim, 60, 0.3, seed=dim + 1)
    g = ivf.build(ivf.IndexParams(n_lists=150, pq_dim=pq_dim, pq_bits=bits, metric=metric, kmeans_n_iters=3), torch.from_numpy(x).cuda())
    L.check(L.load().cuvsB200SetScanCodebookHome(4))
    try:
        d2, i2 = gpu_search(ivf, g, q, k, 20, lut, "f32")
        L.check(L.load().cuvsB200SetScanCodebookHome(2))
        d0, i0 = gpu_search(ivf, g, q, k, 20, lut, "f32")
    finally:
        L.check(L.load().cuvsB200SetScanCodebookHome(0))
    assert (i0 == i2).all() and (d0.view(np.uint32) == d2.view(np.uint32)).all()


# few neighbours (no row codes) and more (with them), narrow and wide bounds, every straight-line shape, the general loop, and a codebook that
# exceeds shared memory; against the tables bit for bit
@pytest.mark.parametrize("metric,lut,internal", [("sqeuclidean", "f32", "f32"), ("sqeuclidean", "f16", "f32"), ("sqeuclidean", "f16", "f16"),
                                                 ("sqeuclidean", "fp8", "f32"), ("inner_product", "f16", "f32"), ("cosine", "f32", "f32")])
@pytest.mark.parametrize("dim,pq_dim,bits", [(96, 48, 8), (64, 16, 8), (64, 32, 4), (81, 27, 8), (56, 40, 5), (200, 100, 8)])
def test_with_and_without_row_codes(ivf, metric, lut, internal, dim, pq_dim, bits):
    from cuvs_b200 import _lib as L
    x = make_mixture(60_001, dim, 60, 0.3, seed=dim)
    q = make_mixture(900, dim, 60, 0.3, seed=dim + 1)
    g = ivf.build(ivf.IndexParams(n_lists=150, pq_dim=pq_dim, pq_bits=bits, metric=metric, kmeans_n_iters=3), torch.from_numpy(x).cuda())
    for k in (1, 9, 40):
        L.check(L.load().cuvsB200SetScanCodebookHome(4))
        d2, i2 = gpu_search(ivf, g, q, k, 20, lut, internal)
        L.check(L.load().cuvsB200SetScanCodebookHome(2))
        d0, i0 = gpu_search(ivf, g, q, k, 20, lut, internal)
        assert (i0 == i2).all() and (d0.view(np.uint32) == d2.view(np.uint32)).all()


# rows and queries whose distances are many orders below the longest codeword, which sets the scale of the half-precision operands:
# |r|^2 of the near rows underflows there.  Against the tables bit for bit
@pytest.mark.parametrize("lut,internal", [("f32", "f32"), ("f16", "f32"), ("fp8", "f32"), ("f16", "f16")])
@pytest.mark.parametrize("pq_dim,length,bits", [(16, 1, 8), (16, 2, 8), (24, 4, 8), (32, 2, 4), (16, 8, 8)])
@pytest.mark.parametrize("longest,near", [(3.0, 1.0), (300.0, 0.05), (30_000.0, 0.05), (300.0, 1e-3)])
def test_distances_far_below_the_longest_codeword(ivf, lut, internal, pq_dim, length, bits, longest, near):
    from cuvs_b200 import _lib as L
    rng = np.random.default_rng(pq_dim + length)
    dim, n_lists, n, book = pq_dim * length, 20, 6000, 1 << bits
    books = near * rng.standard_normal((pq_dim, length, book))
    books[:, :, book - 2:] *= longest / near
    centers = rng.standard_normal((n_lists, dim))
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    g = ivf.build_precomputed(ivf.IndexParams(n_lists=n_lists, pq_dim=pq_dim, pq_bits=bits), dim, to(books), to(centers), to(centers),
                              to(np.eye(dim)))
    rows = centers[rng.integers(0, n_lists, n)] + near * rng.standard_normal((n, dim))
    rows[::50] += longest * rng.standard_normal((len(rows[::50]), dim))
    ivf.extend(g, to(rows), torch.arange(n, device="cuda"))
    q = (rows[rng.integers(0, n, 300)] + 0.01 * near * rng.standard_normal((300, dim))).astype(np.float32)
    for k in (1, 10, 40):
        L.check(L.load().cuvsB200SetScanCodebookHome(4))
        d2, i2 = gpu_search(ivf, g, q, k, 4, lut, internal)
        L.check(L.load().cuvsB200SetScanCodebookHome(2))
        d0, i0 = gpu_search(ivf, g, q, k, 4, lut, internal)
        assert (i0 == i2).all() and (d0.view(np.uint32) == d2.view(np.uint32)).all()
