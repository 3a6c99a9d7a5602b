"""Labels and codes of `transform` against a float64 statement: the labelling on the tensor cores (and the exact pass below
its size), and the encoder for every number of components per subspace."""
import ctypes as C

import numpy as np
import pytest

from conftest import make_mixture

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ivf():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cuvs_b200 import ivf_pq
    return ivf_pq


def model(ivf, dim, n_lists, pq_dim, bits, metric="sqeuclidean", scale=1.0, seed=0):
    rng = np.random.default_rng(seed)
    length = -(-dim // pq_dim)
    rot_dim = pq_dim * length
    centers = (make_mixture(n_lists, dim, 40, 0.3, seed) * scale).astype(np.float32)
    books = (rng.standard_normal((pq_dim, length, 1 << bits)) * 0.2 * scale).astype(np.float32)
    rot = np.eye(dim) if rot_dim == dim else np.linalg.qr(rng.standard_normal((rot_dim, rot_dim)))[0][:, :dim]
    rot = rot.astype(np.float32)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    index = ivf.build_precomputed(ivf.IndexParams(n_lists=n_lists, pq_dim=pq_dim, pq_bits=bits, metric=metric), dim,
                                  to(books), to(centers), to(centers @ rot.T), to(rot))
    return index, centers, books, rot


def check_labels(labels, x, centers):
    x64, c64 = torch.from_numpy(x).cuda().double(), torch.from_numpy(centers).cuda().double()
    d = torch.cdist(x64, c64)
    best = d.min(1).values
    got = d.gather(1, labels.to(torch.int64).unsqueeze(1)).squeeze(1)
    # the label's squared distance is the smallest up to the rounding of an fp32 chain over |x||c|
    tol = 1e-5 * (x64.norm(dim=1) + c64.norm(dim=1).max()) ** 2
    assert bool((got ** 2 <= best ** 2 + tol).all())
    assert float((got == best).double().mean()) > 0.99


# edges of the 128-row and 256-list tiles, one and several K blocks, row tile resident (dim <= 382) and not, few rows (lists
# shared between SMs), and sizes below the tensor-core path
@pytest.mark.parametrize("n,dim,n_lists", [(65536, 14, 256), (70001, 61, 257), (20000, 62, 1000), (16387, 126, 2049),
                                           (9000, 127, 5000), (20001, 384, 1023), (17000, 768, 1100), (100, 32, 300)])
@pytest.mark.parametrize("scale", [1.0, 3e4])
def test_labels(ivf, n, dim, n_lists, scale):
    pq_dim = 8 if dim >= 8 else 1
    index, centers, _, _ = model(ivf, dim, n_lists, pq_dim, 8, scale=scale)
    x = (make_mixture(n, dim, 40, 0.3, 5) * scale).astype(np.float32)
    x[3] = centers[7]            # exactly a centre
    x[4] *= 1e-3                 # far from the scale of the others
    x[5] *= 1e5
    labels, _ = ivf.transform(index, torch.from_numpy(x).cuda())
    check_labels(labels, x, centers)


def test_equal_centres_take_the_lowest_list(ivf):
    index, centers, books, rot = model(ivf, 32, 512, 16, 8)
    centers[100:356] = centers[44]          # ties inside and across tiles: all rows near them are redone exactly
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    index = ivf.build_precomputed(ivf.IndexParams(n_lists=512, pq_dim=16), 32, to(books), to(centers),
                                  to(centers @ rot.T), to(rot))
    x = make_mixture(40000, 32, 40, 0.3, 3)
    x[:300] = centers[44] + 1e-3
    labels = ivf.transform(index, to(x))[0].to(torch.int64)
    assert bool((labels[:300] == 44).all()) and not bool(((labels >= 100) & (labels < 356)).any())


@pytest.mark.parametrize("bits,pq_dim,length", [(8, 16, 1), (8, 24, 2), (8, 6, 2), (8, 10, 3), (8, 5, 4), (4, 8, 5), (8, 4, 8),
                                                (5, 8, 2), (6, 12, 4), (7, 8, 16), (8, 2, 130), (4, 64, 2)])
@pytest.mark.parametrize("n", [1, 1025])
def test_codes(ivf, bits, pq_dim, length, n):
    dim = pq_dim * length
    index, centers, books, _ = model(ivf, dim, 20, pq_dim, bits)
    x = make_mixture(n, dim, 40, 0.3, 9)
    labels, packed = ivf.transform(index, torch.from_numpy(x).cuda())
    labels, packed = labels.cpu().numpy().astype(np.int64), packed.cpu().numpy()
    stream = np.unpackbits(packed, axis=1, bitorder="little")[:, :pq_dim * bits].reshape(n, pq_dim, bits)
    codes = (stream * (1 << np.arange(bits))).sum(2)
    r = (x - centers[labels]).astype(np.float32).reshape(n, pq_dim, length)
    d = ((r[:, :, :, None].astype(np.float64) - books[None]) ** 2).sum(2)
    got = np.take_along_axis(d, codes[:, :, None], 2)[:, :, 0]
    assert (got <= d.min(2) * (1 + 1e-5) + 1e-9).all() and (codes == d.argmin(2)).mean() > 0.999


# through tables of cells (at most four components, 7 and 8 bits, so many rows or more), against the comparison of all distances
# (fewer rows at a time), bit for bit: normal and heavy-tailed residuals, equal codewords, a subspace whose codewords are
# all equal or far from zero for their spread, components that do not count, rows far outside, infinities and NaN
@pytest.mark.parametrize("length,n", [(1, 24576), (2, 24577), (3, 131073), (4, 393217)])
@pytest.mark.parametrize("bits", [7, 8])
@pytest.mark.parametrize("rotated", [False, True])
def test_codes_by_cells(ivf, length, n, bits, rotated):
    pq_dim, n_lists = 8 if bits < 8 else 7, 20
    dim = pq_dim * length - (1 if rotated else 0)
    rot_dim, book = pq_dim * length, 1 << bits
    rng = np.random.default_rng(10 * length + bits)
    books = rng.standard_normal((pq_dim, length, book)).astype(np.float32)
    books[1] *= np.exp(rng.uniform(-4, 1, book)).astype(np.float32)          # heavy tails
    books[2, :, book // 2:] = books[2, :, :book - book // 2]                 # every codeword twice
    books[3] = 0.25                                                          # all equal
    books[4] = 100.0 + 1e-4 * books[4]                                       # far from zero for their spread
    books[5, 0] = -0.5                                                       # a component that is always the same
    centers = rng.standard_normal((n_lists, dim)).astype(np.float32)
    rot = np.eye(dim) if not rotated else np.linalg.qr(rng.standard_normal((rot_dim, rot_dim)))[0][:, :dim]
    rot = rot.astype(np.float32)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    index = ivf.build_precomputed(ivf.IndexParams(n_lists=n_lists, pq_dim=pq_dim, pq_bits=bits), dim, to(books), to(centers),
                                  to(centers @ rot.T), to(rot))
    x = (centers[rng.integers(0, n_lists, n)] + rng.standard_normal((n, dim)) * np.exp(rng.uniform(-5, 1, (n, 1)))).astype(np.float32)
    x[::7] = x[::7] * 30.0
    x[5], x[6, 0], x[7, 0] = 1e30, np.inf, np.nan
    if not rotated:
        near = centers[3].reshape(pq_dim, length)                            # midway between codewords, and on them
        x[100:100 + book] = (near + books.transpose(2, 0, 1)).reshape(book, dim)
        x[1000:1000 + book] = (near + 0.5 * (books + np.roll(books, 1, 2)).transpose(2, 0, 1)).reshape(book, dim)
    labels, codes = ivf.transform(index, to(x))
    for r0 in range(0, n, 20000):
        few_labels, few = ivf.transform(index, to(x[r0:r0 + 20000]))
        assert bool((few_labels == labels[r0:r0 + 20000]).all())
        assert bool((few == codes[r0:r0 + 20000]).all())


# at the number of rows from which the tables are used, which depends on the number of subspaces, and one row below it: against fewer
# rows at a time, bit for bit (subspaces that do not fill the last block of either encoder)
@pytest.mark.parametrize("length,bits,pq_dim,n", [(1, 8, 37, 17_405), (1, 7, 64, 40_625), (2, 8, 65, 17_846), (2, 7, 24, 55_333),
                                                  (3, 8, 33, 99_393), (3, 7, 40, 137_500), (4, 8, 41, 238_414), (4, 7, 72, 201_944),
                                                  (2, 8, 1, 264_000), (2, 8, 8, 24_576), (4, 8, 3, 1_041_666)])
def test_where_tables_of_cells_begin(ivf, length, bits, pq_dim, n):
    rng = np.random.default_rng(n)
    dim, n_lists, book = pq_dim * length, 20, 1 << bits
    books = (rng.standard_normal((pq_dim, length, book)) * np.exp(rng.uniform(-2, 1, (pq_dim, 1, 1)))).astype(np.float32)
    centers = rng.standard_normal((n_lists, dim)).astype(np.float32)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()  # noqa: E731
    index = ivf.build_precomputed(ivf.IndexParams(n_lists=n_lists, pq_dim=pq_dim, pq_bits=bits), dim, to(books), to(centers),
                                  to(centers), to(np.eye(dim)))
    x = to(centers)[torch.from_numpy(rng.integers(0, n_lists, n)).cuda()]
    x = x + torch.randn(n, dim, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda")
    from cuvs_b200 import _lib as L
    from cuvs_b200.common import Resources
    res, launches, stats = Resources(), [0], L.SearchStats()

    def transform(rows):
        out = ivf.transform(index, rows, resources=res)
        L.check(L.load().cuvsB200StatsGet(res.handle, C.byref(stats), False))
        launches.append(stats.launches)
        return out

    labels_below, codes_below = transform(x[:n - 1])
    labels, codes = transform(x)
    # (the tables are made by one kernel more)
    assert launches[2] - launches[1] == launches[1] + 1
    assert bool((labels_below == labels[:n - 1]).all()) and bool((codes_below == codes[:n - 1]).all())
    for r0 in range(0, n, 12_000):
        few_labels, few = ivf.transform(index, x[r0:r0 + 12_000])
        assert bool((few_labels == labels[r0:r0 + 12_000]).all())
        assert bool((few == codes[r0:r0 + 12_000]).all())


# one and several K blocks: row tile resident, and streamed beside the lists
@pytest.mark.parametrize("n,dim,n_lists", [(20000, 62, 1000), (17000, 300, 1100), (17000, 768, 1100)])
def test_a_wait_that_runs_out_redoes_every_label(ivf, n, dim, n_lists):
    """One list block of every CTA's first tile never comes and the limit is about a millisecond: the labelling kernel gives
    up, every row is labelled by the exact product, and the handle counts the call."""
    import ctypes as C
    from cuvs_b200 import _lib as L
    from cuvs_b200.common import Resources
    index, _, _, _ = model(ivf, dim, n_lists, 4, 8)
    x = torch.from_numpy(make_mixture(n, dim, 40, 0.3, 5)).cuda()
    lib, res = L.load(), Resources()

    def labels():
        out = ivf.transform(index, x, resources=res)[0]
        m = C.c_uint64(0)
        L.check(lib.cuvsStreamSync(res.handle))
        L.check(lib.cuvsB200CoarseTimeouts(res.handle, C.byref(m)))
        return out.to(torch.int64), m.value

    healthy, m0 = labels()
    try:
        L.check(lib.cuvsB200SetCoarseWaitTest(1000, 1))
        timed_out, m1 = labels()
    finally:
        L.check(lib.cuvsB200SetCoarseWaitTest(0, 0))
    again, m2 = labels()
    assert m0 == 0 and m1 >= 1 and m2 == m1
    assert bool((healthy == timed_out).all()) and bool((healthy == again).all())


# more lists within reach of a row than the first pass keeps (four units of eight per column quarter), than a block of the
# finish kernel has room for, and than the second pass keeps; one, two, three and more K blocks.  second, full: rows go through
# a second pass (there is none for so few rows that the first has as many shares), and to the exact product over all lists.
@pytest.mark.parametrize("n,dim,n_lists,alike,second,full",
                         [(4097, 40, 4096, 64, False, True), (9000, 96, 4100, 12, False, True), (8200, 128, 2050, 10, False, True),
                          (8200, 130, 2050, 10, False, True), (17000, 200, 1030, 6, False, True), (20000, 64, 1024, 512, False, True),
                          (41000, 96, 4096, 12, True, True), (40001, 130, 2050, 64, True, True), (150000, 32, 2048, 8, True, False)])
def test_many_lists_within_reach(ivf, n, dim, n_lists, alike, second, full):
    """Centres in groups that differ by some 1e-5 of their length: the labels equal those of the exact product (the labelling
    kernel's waits made to run out)."""
    from cuvs_b200 import _lib as L
    from cuvs_b200.common import Resources
    rng = np.random.default_rng(dim)
    groups = make_mixture(-(-n_lists // alike), dim, 40, 0.3, 1)
    centers = groups[rng.permutation(n_lists) % len(groups)] + 1e-5 * rng.standard_normal((n_lists, dim))
    centers = centers.astype(np.float32)
    books = rng.standard_normal((4, dim // 2, 16)).astype(np.float32) if dim % 4 else \
        rng.standard_normal((4, dim // 4, 16)).astype(np.float32)
    if dim % 4:
        books = books[:2]
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    eye = np.eye(dim, dtype=np.float32)
    index = ivf.build_precomputed(ivf.IndexParams(n_lists=n_lists, pq_dim=len(books), pq_bits=4), dim, to(books), to(centers),
                                  to(centers), to(eye))
    x = to((groups[rng.integers(0, len(groups), n)] + 0.05 * rng.standard_normal((n, dim))).astype(np.float32))
    lib, res, counts = L.load(), Resources(), (C.c_uint64 * 3)()
    labels = ivf.transform(index, x, resources=res)[0].to(torch.int64)
    L.check(lib.cuvsB200RedoCounts(res.handle, counts))
    assert (counts[1] > 0) == second and (counts[2] > 0) == full
    try:
        L.check(lib.cuvsB200SetCoarseWaitTest(1000, 1))
        exact = ivf.transform(index, x)[0].to(torch.int64)
    finally:
        L.check(lib.cuvsB200SetCoarseWaitTest(0, 0))
    assert bool((labels == exact).all())
