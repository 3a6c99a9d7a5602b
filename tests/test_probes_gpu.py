"""Probe selection of large batches (two passes over the lists' values, no score matrix) against the exact product with
row selection: the same probes in the same order, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from conftest import make_mixture

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def mods():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cuvs_b200 import _lib, ivf_pq, mg
    return ivf_pq, mg, _lib


def index_of(ivf, centers, metric):
    n_lists, dim = centers.shape
    rng = np.random.default_rng(1)
    books = rng.standard_normal((2, dim // 2, 16)).astype(np.float32)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    return ivf.build_precomputed(ivf.IndexParams(n_lists=n_lists, pq_dim=2, pq_bits=4, metric=metric), dim, to(books), to(centers),
                                 to(centers), to(np.eye(dim)))


def redone(mods, res):
    """Queries whose probes were worked out over all lists, since the handle was made."""
    counts = (C.c_uint64 * 3)()
    mods[2].check(mods[2].load().cuvsB200RedoCounts(res.handle, counts))
    return counts[0]


def both(mods, index, q, n_probes, mode=0):
    """(probes as search selects them, probes of the exact product, queries that the former left to all lists)"""
    from cuvs_b200.common import Resources
    ivf, mg, L = mods
    lib, got, res = L.load(), [], Resources()
    for mode in (mode, 1):
        try:
            lib.cuvsB200SetCoarseMode(mode)
            got.append(mg.select_probes(index, q, n_probes, resources=res).to(torch.int64))
        finally:
            lib.cuvsB200SetCoarseMode(0)
    return *got, redone(mods, res)


# edges of the 256-query and 256-list tiles; 8, 32, 64 and 128 lists per maximum; one, two, three and more K blocks
@pytest.mark.parametrize("metric", ["sqeuclidean", "inner_product", "cosine"])
@pytest.mark.parametrize("n_lists,n_q,dim,n_probes", [(257, 8200, 14, 1), (513, 4300, 62, 32), (1024, 2305, 130, 20), (4001, 700, 96, 128),
                                                      (4096, 513, 256, 256), (9000, 257, 128, 20), (20000, 255, 66, 200),
                                                      (40000, 100, 32, 50)])
def test_probes(mods, n_lists, n_q, dim, n_probes, metric):
    centers = make_mixture(n_lists, dim, 60, 0.4, 2)
    q = make_mixture(n_q, dim, 60, 0.4, 3)
    if metric == "cosine":
        centers /= np.linalg.norm(centers, axis=1, keepdims=True)
    index = index_of(mods[0], centers, metric)
    fast, exact, n = both(mods, index, torch.from_numpy(q).cuda(), n_probes)
    assert bool((fast == exact).all())
    assert n <= n_q // 256                                         # ordinary data: the two passes settle it


# the fewest queries that go through the two passes (by probes and lists, by pairs, beyond 16,384 lists by queries), and one less
@pytest.mark.parametrize("metric", ["sqeuclidean", "inner_product"])
@pytest.mark.parametrize("n_lists,n_q,dim,n_probes", [(513, 9728, 30, 32), (1000, 9000, 40, 60), (4001, 2559, 96, 128), (4096, 9766, 24, 256),
                                                      (9000, 1235, 130, 200), (16384, 257, 66, 160), (20000, 129, 32, 30), (40000, 257, 32, 63), (32768, 64, 62, 64),
                                                      (40000, 64, 98, 200), (1000, 2098, 20, 5)])
def test_where_the_two_passes_begin(mods, n_lists, n_q, dim, n_probes, metric):
    index = index_of(mods[0], make_mixture(n_lists, dim, 60, 0.4, 2), metric)
    q = torch.from_numpy(make_mixture(n_q, dim, 60, 0.4, 3)).cuda()
    fast, exact, n = both(mods, index, q, n_probes)
    assert bool((fast == exact).all()) and n <= n_q // 256
    below, exact, _ = both(mods, index, q[:n_q - 1], n_probes)     # (the other path's guard is wider: it redoes more)
    assert bool((below == exact).all()) and bool((below == fast[:n_q - 1]).all())


# lists in the order of their components, or of the branches of a tree: neighbours are alike
@pytest.mark.parametrize("metric", ["sqeuclidean", "inner_product"])
@pytest.mark.parametrize("n_lists,n_q,dim,n_probes", [(2048, 2000, 96, 20), (4000, 2000, 128, 64), (12288, 1000, 64, 128),
                                                      (20000, 1000, 64, 20), (65536, 300, 32, 50)])
@pytest.mark.parametrize("tree", [False, True])
def test_the_order_of_the_lists_does_not_matter(mods, n_lists, n_q, dim, n_probes, metric, tree):
    rng = np.random.default_rng(n_lists)
    if tree:
        centers, level = np.zeros((1, dim)), 1.0
        while len(centers) < n_lists:
            level *= 0.7
            centers = np.repeat(centers, 8, 0)
            centers = centers + level * rng.standard_normal(centers.shape)
        centers = centers[:n_lists]
    else:
        component = np.sort(rng.integers(0, n_lists // 16, n_lists))
        centers = rng.standard_normal((n_lists // 16, dim))[component] + 0.3 * rng.standard_normal((n_lists, dim))
    q = centers[rng.integers(0, n_lists, n_q)] + 0.3 * np.abs(centers).mean() * rng.standard_normal((n_q, dim))
    index = index_of(mods[0], centers.astype(np.float32), metric)
    fast, exact, n = both(mods, index, torch.from_numpy(q.astype(np.float32)).cuda(), n_probes)
    assert bool((fast == exact).all())
    assert n <= n_q // 256


# small integers: most lists have the score of several others; two, or many of them, across the last probe
@pytest.mark.parametrize("n_lists,n_q,dim,n_probes,top", [(2048, 1100, 16, 40, 16), (4096, 600, 30, 200, 9), (20000, 150, 12, 33, 8)])
@pytest.mark.parametrize("metric", ["sqeuclidean", "inner_product"])
def test_equal_scores(mods, n_lists, n_q, dim, n_probes, top, metric):
    rng = np.random.default_rng(top)
    centers, q = rng.integers(0, top, (n_lists, dim)), rng.integers(0, top, (n_q, dim))
    index = index_of(mods[0], centers.astype(np.float32), metric)
    fast, exact, n = both(mods, index, torch.from_numpy(q.astype(np.float32)).cuda(), n_probes)
    assert bool((fast == exact).all())
    assert n < n_q // 2                                            # (what is tested is the order of those ranked at once)


def test_a_last_batch_with_larger_chunks(mods):
    """The exact product of 12,000 queries takes one chunk, that of the 16,384 before them two smaller ones, in one workspace."""
    ivf, mg, _ = mods
    index = index_of(ivf, make_mixture(1100, 16, 60, 0.4, 2), "sqeuclidean")
    q = torch.from_numpy(make_mixture(16_384 + 12_000, 16, 60, 0.4, 3)).cuda()
    got = mg.select_probes(index, q, 300)                          # (more probes than the two product passes take)
    assert bool((got[:16_384].to(torch.int64) == mg.select_probes(index, q[:16_384], 300).to(torch.int64)).all())
    assert bool((got[16_384:].to(torch.int64) == mg.select_probes(index, q[16_384:], 300).to(torch.int64)).all())


def test_odd_queries_and_equal_lists(mods):
    """Queries without a bound (NaN, infinities, values at the ends of fp32, zeros) and lists that are equal or nearly so in numbers
    beyond what a query has room for."""
    rng = np.random.default_rng(5)
    centers = make_mixture(4096, 48, 60, 0.4, 2)
    centers[100:130] = centers[7]                                  # ties: lowest list first
    centers[1000:1600] = centers[8] + 1e-6 * rng.standard_normal((600, 48))
    q = make_mixture(1500, 48, 60, 0.4, 3)
    q[0], q[1, 3], q[2, 4], q[3] = 0.0, np.nan, np.inf, 1e30
    q[4] *= 1e-30
    q[5] *= 1e18
    q[10:40] = centers[7]
    q[40:80] = centers[8]
    for metric in ("sqeuclidean", "inner_product"):
        index = index_of(mods[0], centers, metric)
        fast, exact, n = both(mods, index, torch.from_numpy(q.astype(np.float32)).cuda(), 40)
        assert 41 <= n <= 120                                      # those at centers[8], without a bound, and few others
        fine = torch.ones(len(q), dtype=torch.bool, device="cuda")
        fine[1] = fine[2] = False                                  # (NaN scores have no order)
        assert bool((fast == exact).all(1)[fine].all())


# queries that many equal lists are nearest to, beyond what there is room for: as many as the whole grid scores, one more, and
# many; the scores in rows of 16 and of fewer queries per block; both paths that leave queries to the redo
@pytest.mark.parametrize("n_lists,n_q,dim,n_probes", [(1024, 9000, 40, 20), (4001, 3000, 102, 64), (100_000, 700, 30, 10)])
@pytest.mark.parametrize("m", [1, 64, 65, 500, 0])
def test_queries_redone(mods, n_lists, n_q, dim, n_probes, m):
    rng = np.random.default_rng(m)
    centers = make_mixture(n_lists, dim, 60, 0.4, 2)
    centers[rng.permutation(n_lists)[:600]] = centers[8] + 1e-6 * rng.standard_normal((600, dim))
    q = make_mixture(n_q, dim, 60, 0.4, 3)
    m = m or n_q
    q[rng.permutation(n_q)[:m]] = centers[8] + 1e-3 * rng.standard_normal((m, dim))
    index = index_of(mods[0], centers.astype(np.float32), "sqeuclidean")
    for mode in (0, 2) if n_lists > 50_000 else (0,):              # (2: shapes that path covers)
        fast, exact, n = both(mods, index, torch.from_numpy(q.astype(np.float32)).cuda(), n_probes, mode)
        assert bool((fast == exact).all())
        assert m <= n <= m + n_q // 16, (mode, n)


def test_redoing_a_whole_batch_costs_a_few_exact_products(mods):
    """One centre at thirty times the others' length widens every query's bound: the whole batch is redone.  Measured: 49 times
    the exact product with a thread per list and its centre row read by itself, 2 to 3 times through shared memory."""
    from cuvs_b200.common import Resources
    ivf, mg, L = mods
    centers = make_mixture(4000, 128, 60, 0.4, 2)
    ordinary = index_of(ivf, centers, "sqeuclidean")
    centers[5] *= 30.0 * np.linalg.norm(centers, axis=1).mean() / np.linalg.norm(centers[5])
    index = index_of(ivf, centers, "sqeuclidean")
    q = torch.from_numpy(make_mixture(10_000, 128, 60, 0.4, 3)).cuda()

    def timed(index, res):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        mg.select_probes(index, q, 64, resources=res)
        b.record()
        torch.cuda.synchronize()
        return a.elapsed_time(b)

    redo, exact = [], []
    for _ in range(3):
        res = Resources()
        timed(ordinary, res)                                       # (buffers)
        redo.append(timed(index, res))
        assert redone(mods, res) >= 9000
        try:
            L.load().cuvsB200SetCoarseMode(1)
            timed(index, res)
            exact.append(timed(index, res))
        finally:
            L.load().cuvsB200SetCoarseMode(0)
    assert min(redo) < 8.0 * min(exact)


# one product pass times out; every query is redone exactly and the handle counts the batch
@pytest.mark.parametrize("dim", [40, 300])
def test_a_wait_that_runs_out_redoes_every_query(mods, dim):
    ivf, mg, L = mods
    from cuvs_b200.common import Resources
    centers = make_mixture(2100, dim, 60, 0.4, 2)
    q = torch.from_numpy(make_mixture(1100, dim, 60, 0.4, 3)).cuda()
    index = index_of(ivf, centers, "sqeuclidean")
    lib, res = L.load(), Resources()

    def run():
        out = mg.select_probes(index, q, 20, resources=res).to(torch.int64)
        m = C.c_uint64(0)
        L.check(lib.cuvsStreamSync(res.handle))
        L.check(lib.cuvsB200CoarseTimeouts(res.handle, C.byref(m)))
        return out, m.value

    healthy, m0 = run()
    try:
        L.check(lib.cuvsB200SetCoarseWaitTest(1000, 1))
        timed_out, m1 = run()
    finally:
        L.check(lib.cuvsB200SetCoarseWaitTest(0, 0))
    again, m2 = run()
    assert m0 == 0 and m1 == 1 and m2 == m1
    assert bool((healthy == timed_out).all()) and bool((healthy == again).all())


@pytest.mark.parametrize("per_cluster", [False, True])
def test_a_model_is_complete_on_return(mods, per_cluster):
    """Nothing of the derived state is still being made when the C call that lays out a model returns: a handle on another
    stream may search at once."""
    from cuvs_b200.common import DLTensorRef, Resources
    ivf, _, L = mods
    n_lists, dim = 30_000, 128
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    centers = to(make_mixture(n_lists, dim, 60, 0.4, 2))
    books = torch.rand((n_lists if per_cluster else 2, dim // 2, 16), device="cuda")
    params = ivf.IndexParams(n_lists=n_lists, pq_dim=2, pq_bits=4, codebook_kind="cluster" if per_cluster else "subspace")
    stream = torch.cuda.Stream()
    res, index = Resources(stream.cuda_stream), ivf.Index()
    refs = [DLTensorRef(t) for t in (books, centers, centers, to(np.eye(dim)))]
    torch.cuda.synchronize()
    L.check(L.load().cuvsIvfPqBuildPrecomputed(res.handle, params._p, C.c_uint32(dim), *[r.ref() for r in refs], index._h))
    assert stream.query()


def test_a_handle_leaves_the_passes_where_they_do_not_pay(mods):
    """A batch that left more than a sixteenth of its queries to the redo sends the next calls of that shape to the exact product;
    other shapes stay, and after a while the passes are tried again."""
    from cuvs_b200.common import Resources
    ivf, mg, _ = mods
    centers = make_mixture(2048, 64, 60, 0.4, 2)
    ordinary = index_of(ivf, centers, "sqeuclidean")
    far = centers.copy()
    far[5] *= 30.0 * np.linalg.norm(centers, axis=1).mean() / np.linalg.norm(far[5])
    index = index_of(ivf, far, "sqeuclidean")
    q = torch.from_numpy(make_mixture(2000, 64, 60, 0.4, 3)).cuda()
    res = Resources()

    def run(index, n_probes=20):
        before = redone(mods, res)                                 # (synchronises: the last batch's counters have arrived)
        out = mg.select_probes(index, q, n_probes, resources=res).to(torch.int64)
        return out, redone(mods, res) - before

    first, n = run(index)
    assert n > len(q) // 4
    for _ in range(16):
        out, n = run(index)
        assert n == 0 and bool((out == first).all())
    assert run(ordinary, 30)[1] <= len(q) // 256                   # (another shape takes the passes)
    assert run(index)[1] > len(q) // 4                             # the next try
    for _ in range(32):
        assert run(index)[1] == 0
    assert run(ordinary)[1] <= len(q) // 256                       # a try that succeeds
    assert run(index)[1] > len(q) // 4
    for _ in range(16):
        assert run(index)[1] == 0
    assert run(index)[1] > len(q) // 4
