"""The projection kernels at the edges of their forms, against the oracle:
tensor cores with features whose energy sits in the leading or the trailing
dimensions (the code bound weighs a dimension by the roundings it takes part
in), whose magnitudes are far from 1, or whose sampled rows say nothing of the
others (inexact in fp16, or past the sample's scale, only where the sample does
not look); column blocks past 256 columns; and the SIMT tiling of more than 64
columns with ragged edges in points, columns and dimensions."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def check(culsh, X, A, b, W):
    L, M, D = A.shape
    ht = culsh.HashTables()
    ht.reset(X.shape[0], D, L, M, W, A=A, b=b)
    ht.index(X)
    ref = oracle.build_index(X, A, b, W)
    np.testing.assert_array_equal(ht.getBuckets(), ref.buckets)
    for l in range(L):
        np.testing.assert_array_equal(ht.getBuckets_codes(l), ref.codes(l), err_msg=f"table {l}")
        np.testing.assert_array_equal(ht.getBuckets_totalIndices(l), ref.ids(l), err_msg=f"table {l}")
    return ht.profile()


def features(kind, N, D, rng):
    X = rng.normal(0, 1, (N, D))
    if kind == "front":
        X *= np.exp(-6.0 * np.arange(D) / D)
    elif kind == "back":
        X *= np.exp(-6.0 * np.arange(D)[::-1] / D)
    elif kind == "tiny":
        X *= 1e-6
    elif kind == "huge":
        X *= 1e6
    elif kind in ("late_inexact", "late_large"):
        # every second row is sampled (N / 4096 = 2): integers there
        X = np.rint(20 * X)
        if kind == "late_inexact":
            X[1::2] += 0.1 * rng.normal(0, 1, X[1::2].shape)
        else:
            X[1::2] *= 4096
    return np.ascontiguousarray(X, np.float32)


def projection(L, M, D, W, rng):
    return rng.normal(0, 1, (L, M, D)).astype(np.float32), rng.uniform(0, W, (L, M)).astype(np.float32)


@pytest.mark.parametrize("kind", ["plain", "front", "back", "tiny", "huge", "late_inexact", "late_large"])
@pytest.mark.parametrize("D,L,M", [(128, 4, 12), (67, 3, 7), (96, 20, 14), (320, 2, 9)])
def test_tensor_core_codes(culsh, kind, D, L, M, monkeypatch):
    monkeypatch.setenv("CULSH_PROJECT_TC", "1")
    rng = np.random.default_rng(D + L)
    N = 8501
    X = features(kind, N, D, rng)
    W = float(0.25 * np.sqrt(np.mean(np.sum(X.astype(np.float64) ** 2, axis=1))))
    A, b = projection(L, M, D, W, rng)
    assert check(culsh, X, A, b, W)["tensor_cores"] == 1


@pytest.mark.parametrize("D,L,M", [(216, 14, 7), (256, 5, 13), (250, 10, 11), (200, 3, 37)])
def test_narrow_last_column_block(culsh, D, L, M):
    """Two column blocks of which the last holds at least sixteen columns
    fewer: only columns that exist are recomputed (each other column of a block
    would add a code per point)."""
    rng = np.random.default_rng(D + L)
    N = 6001
    X = features("plain", N, D, rng)
    W = float(2 * np.sqrt(D))
    A, b = projection(L, M, D, W, rng)
    p = check(culsh, X, A, b, W)
    assert p["tensor_cores"] == 1 and p["recomputed"] < 0.02 * N * L * M


@pytest.mark.parametrize("N,D,L,M", [(1027, 33, 4, 16), (1027, 33, 5, 13), (130, 128, 8, 16), (2049, 130, 3, 43),
                                     (127, 7, 16, 16), (5, 64, 6, 12)])
def test_simt_codes(culsh, N, D, L, M, monkeypatch):
    monkeypatch.setenv("CULSH_PROJECT_SIMT", "1")
    rng = np.random.default_rng(N + D + M)
    X = features("plain", N, D, rng)
    A, b = projection(L, M, D, 3.0, rng)
    assert check(culsh, X, A, b, 3.0)["tensor_cores"] == 0


@pytest.mark.parametrize("Q", [1, 2, 3, 64, 65, 511])
@pytest.mark.parametrize("D,L,M", [(128, 3, 7), (256, 5, 13), (256, 3, 8), (33, 4, 16), (15, 1, 3), (257, 3, 8)])
def test_few_queries(culsh, Q, D, L, M):
    """The few-queries projection (2 or 8 rows a block of 64 columns, up to 256
    dimensions) and the tiling past it, on host rows and on device rows: probes
    and distances are the oracle's."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(Q + D + L)
    N, K, T, W = 3000, 5, 6, 12.0
    X = rng.normal(0, 2, (N, D)).astype(np.float32)
    q = np.ascontiguousarray(X[rng.integers(0, N, Q)] + 0.1 * rng.normal(0, 1, (Q, D)), np.float32)
    A, b = projection(L, M, D, W, rng)
    ht = culsh.HashTables()
    ht.reset(N, D, L, M, W, A=A, b=b)
    ht.index(X)
    ref = oracle.search(oracle.build_index(X, A, b, W), X, q, K, T)
    st = culsh.SearchTables()
    st.reset(ht, K, T)
    for _ in range(2):
        st.search(q, dataset=X)
        for l in range(L):
            np.testing.assert_array_equal(st.getQueryBuckets(l), ref["qbuckets"][l].reshape(Q, T), err_msg=f"table {l}")
        np.testing.assert_array_equal(st.getKnnIds(), ref["knn_ids"])
        np.testing.assert_array_equal(st.getKnnDistances(), ref["knn_dists"])
    dq = torch.from_numpy(q).cuda()
    ids = torch.empty(Q * K, dtype=torch.int32, device="cuda")
    dists = torch.empty(Q * K, dtype=torch.float32, device="cuda")
    st.search_device(dq.data_ptr(), Q, ids.data_ptr(), dists.data_ptr())
    torch.cuda.synchronize()
    np.testing.assert_array_equal(ids.cpu().numpy(), ref["knn_ids"].astype(np.int32).reshape(-1))
    np.testing.assert_array_equal(dists.cpu().numpy(), ref["knn_dists"].reshape(-1))


@pytest.mark.parametrize("share", [0.001, 0.4, 1.0])
@pytest.mark.parametrize("D", [64, 320])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_that_are_not_numbers(culsh, D, share, bad):
    """Rows with a value that is not finite, few of the sample or all: the build
    reports them."""
    rng = np.random.default_rng(D)
    N, L, M, W = 8192, 2, 8, 64.0
    X = np.round(rng.normal(0, 20, (N, D))).astype(np.float32)
    X[rng.random(N) < share, rng.integers(0, D)] = bad
    X[5, 1] = bad
    A = rng.normal(0, 1, (L, M, D)).astype(np.float32)
    ht = culsh.HashTables()
    ht.reset(N, D, L, M, W, A=A, b=np.zeros((L, M), np.float32))
    with pytest.raises(culsh.CulshError) as ei:
        ht.index(X)
    assert ei.value.code == culsh.ERR_NUMERIC
    X[~np.isfinite(X)] = 1.0
    ht.index(X)   # the object serves the next build
    assert ht.getBuckets(0) > 0
