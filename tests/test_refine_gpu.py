"""GPU tests of cuvsRefine (exact re-ranking of candidates) against a float64 numpy statement,
in the spirit of the reference's cpp/tests/neighbors/refine.cu (candidates from brute force with
extra noise, refined result must equal the exact top-k)."""
import numpy as np
import pytest

from conftest import make_mixture

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def exact_refine(x, q, cand, k, metric):
    x64, q64 = x.astype(np.float64), q.astype(np.float64)
    out_i = np.zeros((q.shape[0], k), np.int64)
    out_d = np.zeros((q.shape[0], k), np.float64)
    for r in range(q.shape[0]):
        c = cand[r]
        v = x64[c]
        if metric == "inner_product":
            s = -(v @ q64[r])
        elif metric == "cosine":
            s = 1.0 - (v @ q64[r]) / (np.linalg.norm(v, axis=1) * np.linalg.norm(q64[r]))
        else:
            s = ((v - q64[r]) ** 2).sum(1)
        o = np.argsort(s, kind="stable")[:k]
        out_i[r] = c[o]
        out_d[r] = s[o]
    if metric == "inner_product":
        out_d = -out_d
    if metric == "euclidean":
        out_d = np.sqrt(out_d)
    return out_d, out_i


@pytest.mark.parametrize("metric", ["sqeuclidean", "euclidean", "inner_product", "cosine"])
@pytest.mark.parametrize("dtype", [np.float32, np.uint8])
def test_refine_matches_exact_reranking(metric, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cuvs_b200 import refine
    if dtype == np.uint8:
        x = make_mixture(5000, 48, 20, 15.0, 1, np.uint8, 20, 200)
        q = make_mixture(200, 48, 20, 15.0, 2, np.uint8, 20, 200)
    else:
        x = make_mixture(5000, 48, 20, 0.3, 1)
        q = make_mixture(200, 48, 20, 0.3, 2)
    rng = np.random.default_rng(3)
    cand = np.stack([rng.choice(5000, size=64, replace=False) for _ in range(200)]).astype(np.int64)
    k = 10
    d, i = refine(torch.from_numpy(x).cuda(), torch.from_numpy(q).cuda(), torch.from_numpy(cand).cuda(),
                  k=k, metric=metric)
    d, i = d.cpu().numpy(), i.cpu().numpy()
    ed, ei = exact_refine(x, q, cand, k, metric)
    same = (i == ei).all(axis=1)
    assert same.mean() > 0.99            # rows may differ only at fp32-level ties
    assert np.allclose(d[same], ed[same], rtol=2e-5, atol=1e-5)


def test_refine_ignores_missing_candidates_and_checks_arguments():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cuvs_b200 import refine
    from cuvs_b200._lib import CuvsError
    x = make_mixture(1000, 16, 8, 0.3, 4)
    q = make_mixture(8, 16, 8, 0.3, 5)
    cand = np.tile(np.arange(12, dtype=np.int64), (8, 1))
    cand[:, 5:] = np.iinfo(np.int64).max            # only 5 real candidates per query
    d, i = refine(torch.from_numpy(x).cuda(), torch.from_numpy(q).cuda(), torch.from_numpy(cand).cuda(), k=8)
    i, d = i.cpu().numpy(), d.cpu().numpy()
    assert (np.sort(i[:, :5], axis=1) == np.arange(5)).all()
    assert (i[:, 5:] == np.iinfo(np.int64).max).all() and np.isinf(d[:, 5:]).all()
    with pytest.raises(CuvsError, match="cannot be smaller than k"):
        refine(torch.from_numpy(x).cuda(), torch.from_numpy(q).cuda(), torch.from_numpy(cand[:, :4].copy()).cuda(), k=8)


@pytest.mark.parametrize("dtype", [np.float32, np.float16, np.int8, np.uint8])
@pytest.mark.parametrize("dim,n_q,n_cand,k", [(1, 3, 5, 5), (33, 1, 250, 100), (130, 70, 33, 33), (137, 2, 100, 64),
                                              (768, 5, 200, 10), (64, 5000, 20, 10)])
def test_refine_row_lengths_and_splits(dtype, dim, n_q, n_cand, k):
    """Every way a row can be read (16-byte, 4-byte and shifted words, tails), one and several warps per query."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from cuvs_b200 import refine
    rng = np.random.default_rng(dim * 7 + n_q)
    if dtype in (np.int8, np.uint8):
        x, q = (rng.integers(0, 100, size=(n, dim)).astype(dtype) for n in (1001, n_q))
    else:
        x, q = (rng.standard_normal((n, dim)).astype(dtype) for n in (1001, n_q))
    cand = np.stack([rng.choice(1001, size=n_cand, replace=False) for _ in range(n_q)]).astype(np.int64)
    cand[:, n_cand // 2] = np.iinfo(np.int64).max if k < n_cand else cand[:, n_cand // 2]
    for metric in ("sqeuclidean", "inner_product", "cosine"):
        d, i = refine(torch.from_numpy(x).cuda(), torch.from_numpy(q).cuda(), torch.from_numpy(cand).cuda(), k=k,
                      metric=metric)
        d, i = d.cpu().numpy().astype(np.float64), i.cpu().numpy()
        valid = np.where(cand < 1001, cand, 0)
        v, qq = x.astype(np.float64)[valid], q.astype(np.float64)[:, None, :]
        dots = (v * qq).sum(2)
        s = {"sqeuclidean": ((v - qq) ** 2).sum(2), "inner_product": -dots,
             "cosine": 1.0 - dots / (np.linalg.norm(v, axis=2) * np.linalg.norm(qq, axis=2) + 1e-30)}[metric]
        s = np.where(cand < 1001, s, np.inf)
        want = np.sort(s, axis=1)[:, :k] * (-1.0 if metric == "inner_product" else 1.0)
        scale = np.abs(want).max() + 1.0
        assert np.allclose(d, want, rtol=3e-5, atol=3e-5 * scale), (metric, np.abs(d - want).max())
        got = np.take_along_axis(s, (cand[:, :, None] == i[:, None, :]).argmax(1), 1)   # the returned ids' own scores
        assert np.allclose(got * (-1.0 if metric == "inner_product" else 1.0), want, rtol=3e-5, atol=3e-5 * scale)
