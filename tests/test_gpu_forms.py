"""Forms of the probe and candidate kernels that a rule on sizes picks, at the
edges of their rules, against the oracle: a warp per query for a handful of
candidates, selection in place of sorted lists (sets of every size, few and
many queries, rows staged through shared memory or read directly, merges of
partitions), and the probe with a warp per (table, query) pair."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _check(st, want, L, Q, T):
    np.testing.assert_array_equal(st.getKnnIds(), want["knn_ids"])
    np.testing.assert_array_equal(st.getKnnDistances(), want["knn_dists"])
    assert st.getTotalCandidates_unique() == int(want["unique"].sum())
    assert st.getTotalCandidates_nonUnique() == int(want["nonunique"].sum())
    for l in range(L):
        np.testing.assert_array_equal(st.getQueryBuckets(l), want["qbuckets"][l].reshape(Q, T))


def _index(culsh, X, A, b, W):
    L, M, D = A.shape
    ht = culsh.HashTables()
    ht.reset(X.shape[0], D, L, M, W, A=A, b=b)
    ht.index(X)
    return ht


@pytest.mark.parametrize("D,K", [(4, 1), (13, 10), (96, 40), (160, 10), (164, 10), (1024, 5), (1028, 5)])
def test_few_candidates(culsh, D, K):
    """Queries of 0 to some 60 candidates (32 is the most a warp takes), with
    duplicates over the tables and exact copies in the data."""
    rng = np.random.default_rng(D)
    N, L, M, T, W = 3000, 5, 3, 4, 1.1 * np.sqrt(D)
    X = rng.normal(0, 1, (N, D)).astype(np.float32)
    X[1::9] = X[::9][: len(X[1::9])]
    Qm = (X[rng.integers(0, N, 500)] + rng.normal(0, 0.05, (500, D))).astype(np.float32)
    Qm[:5] = 50.0
    A = rng.normal(0, 1, (L, M, D)).astype(np.float32)
    A[:, 1:] *= 3.0
    b = (rng.random((L, M)) * W).astype(np.float32)
    want = oracle.search(oracle.build_index(X, A, b, W), X, Qm, K, T)
    st = culsh.SearchTables()
    st.reset(_index(culsh, X, A, b, W), K, T)
    st.search(Qm, dataset=X)
    _check(st, want, L, 500, T)


SIZES = [1, 31, 32, 33, 63, 64, 65, 1023, 1024, 1025, 2047, 2048, 2049, 4000]


@pytest.mark.parametrize("Q", [14, 1400])
@pytest.mark.parametrize("D,K", [(16, 1), (128, 32), (100, 33), (17, 100), (12, 2048), (164, 10)])
def test_set_sizes(culsh, Q, D, K):
    """Buckets of exact sizes around the selection's and the set's limits, one
    table and probe, a third of each bucket's points at equal distances; few
    queries (partitioned) and many (whole sets as one item)."""
    rng = np.random.default_rng(K)
    X = np.concatenate([np.full((n, D), 0.0, np.float32) for n in SIZES])
    X += rng.integers(-8, 9, X.shape).astype(np.float32) / 4
    at = 0
    for i, n in enumerate(SIZES):
        X[at:at + n // 3] = X[at]
        X[at:at + n, 0] = i + 0.5
        at += n
    X = np.ascontiguousarray(X[rng.permutation(len(X))])
    Qm = (rng.integers(-8, 9, (Q, D)) / 4).astype(np.float32)
    Qm[:, 0] = np.arange(Q) % len(SIZES) + 0.5
    A = np.zeros((1, 1, D), np.float32)
    A[0, 0, 0] = 1.0
    b = np.zeros((1, 1), np.float32)
    want = oracle.search(oracle.build_index(X, A, b, 1.0), X, Qm, K, 1)
    assert sorted(set(want["unique"].tolist())) == SIZES
    st = culsh.SearchTables()
    st.reset(_index(culsh, X, A, b, 1.0), K, 1)
    st.set_tuning(dense_min=1 << 30)   # no dense queries: the item kernels take all
    st.search(Qm, dataset=X)
    _check(st, want, 1, Q, 1)


@pytest.mark.parametrize("M,T,Q", [(1, 1, 9), (1, 6, 9), (8, 2, 200), (8, 16, 40), (12, 33, 100), (16, 64, 30),
                                   (16, 64, 20000), (15, 5, 1023), (15, 5, 1025), (17, 16, 40)])
@pytest.mark.parametrize("ties", [False, True])
def test_warp_probe(culsh, M, T, Q, ties):
    """Query buckets, counts and results when the probe takes a warp per (table,
    query) pair, around the pair count up to which it does; with ties, many of
    a query's boundary distances are equal (the reference's heap order)."""
    rng = np.random.default_rng(100 * M + T)
    N, D, L, K = 2000, 10, 5, 4
    if ties:
        X = rng.integers(-3, 4, (N, D)).astype(np.float32)
        Qm = rng.integers(-3, 4, (Q, D)).astype(np.float32)
        A = rng.integers(-1, 2, (L, M, D)).astype(np.float32)
        b = np.zeros((L, M), np.float32)
        W = 4.0
    else:
        X = rng.normal(0, 1, (N, D)).astype(np.float32)
        Qm = rng.normal(0, 1, (Q, D)).astype(np.float32)
        A = rng.normal(0, 1, (L, M, D)).astype(np.float32)
        W = 3.0
        b = (rng.random((L, M)) * W).astype(np.float32)
    want = oracle.search(oracle.build_index(X, A, b, W), X, Qm, K, T)
    ht = _index(culsh, X, A, b, W)
    st = culsh.SearchTables()
    st.reset(ht, K, T)
    st.search(Qm, dataset=X)
    _check(st, want, L, Q, T)


@pytest.mark.parametrize("D", [4, 60, 64, 68, 124, 132])
@pytest.mark.parametrize("wt", [64, 128, 256, 512, 0])
def test_gather_steps(culsh, wt, D):
    """Candidate lists of lengths around the gather's steps of every width (one
    or two ids a thread; wt = 0: the per-query kernel) and rows around the eight
    16-byte loads a lane keeps in flight."""
    sizes = [33, 63, 64, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 3000]
    rng = np.random.default_rng(wt + D)
    G, K, T, L, M, W = len(sizes), 10, 1, 2, 1, 4.0
    X = rng.normal(0, 1, (sum(sizes), D)).astype(np.float32)
    X[:, 0] = np.repeat(np.arange(G), sizes) * 100.0 + rng.random(sum(sizes)) * 3.9   # a bucket each
    Qm = np.zeros((2 * G, D), np.float32)
    Qm[:, 0] = np.tile(np.arange(G) * 100.0 + 2.0, 2)
    A = np.zeros((L, M, D), np.float32)
    A[:, 0, 0] = 1.0
    b = np.zeros((L, M), np.float32)
    want = oracle.search(oracle.build_index(X, A, b, W), X, Qm, K, T)
    st = culsh.SearchTables()
    st.reset(_index(culsh, X, A, b, W), K, T)
    st.set_tuning(dense_min=1 << 30, **({"ws_threads": wt} if wt else {"candidates_mode": 0}))
    st.search(Qm, dataset=X)
    _check(st, want, L, 2 * G, T)
