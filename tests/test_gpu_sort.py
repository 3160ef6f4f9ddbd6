"""The index order of multi-word keys: digit passes over the top key word,
then each run of equal top words ordered by its lower words and id (sort form
1), and the passes over every word it falls back to when a run is too long
(form 2, and forced with CULSH_SORT_ALL_WORDS), against the oracle. The data
put points in clusters that share the leading columns' codes exactly and
differ in the trailing columns, with cluster sizes across every run class:
single points, 2 to 8, 9 to 32, 33 to 2,048, and one of 2,049 where asked."""

import os

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def clustered(sizes, seed):
    """D = 12: dims 0-3 fix the leading six columns (one value per cluster,
    spread so that clusters differ there), dims 4-11 drive the trailing six;
    some points repeat exactly."""
    rng = np.random.default_rng(seed)
    D, L, M, W = 12, 2, 12, 1.0
    A = np.zeros((L, M, D), np.float32)
    A[:, :6, :4] = rng.normal(0, 1, (L, 6, 4))
    A[:, 6:, 4:] = rng.normal(0, 1, (L, 6, 8))
    b = rng.uniform(0, W, (L, M)).astype(np.float32)
    parts = []
    for c, n in enumerate(sizes):
        pts = np.empty((n, D), np.float32)
        pts[:, :4] = rng.normal(0, 30, 4).astype(np.float32)
        pts[:, 4:] = rng.normal(0, 4, (n, 8)).astype(np.float32)
        if n > 3:
            pts[n // 2] = pts[0]          # an exact duplicate inside the run
        parts.append(pts)
    X = np.concatenate(parts)
    X = X[rng.permutation(X.shape[0])]
    return np.ascontiguousarray(X), A, b, W


def check(culsh, X, A, b, W):
    L, M, D = A.shape
    N = X.shape[0]
    ht = culsh.HashTables()
    ht.reset(N, D, L, M, W, A=A, b=b)
    ht.index(X)
    ref = oracle.build_index(X, A, b, W)
    np.testing.assert_array_equal(ht.getBuckets(), ref.buckets)
    for l in range(L):
        np.testing.assert_array_equal(ht.getBuckets_totalIndices(l), ref.ids(l), err_msg=f"table {l}")
        np.testing.assert_array_equal(ht.getBuckets_startingIndices(l), ref.starts(l), err_msg=f"table {l}")
        np.testing.assert_array_equal(ht.getBuckets_sizes(l), ref.sizes(l), err_msg=f"table {l}")
        np.testing.assert_array_equal(ht.getBuckets_codes(l), ref.codes(l), err_msg=f"table {l}")
    return ht.profile()


SIZES = [1] * 800 + [2] * 200 + [3] * 60 + [7] * 40 + [8] * 10 + [9] * 10 + [20] * 6 + [32] * 12 + [33] * 6 + [100] * 6 + [700] * 2 + [2048]


def test_top_word_then_runs(culsh):
    X, A, b, W = clustered(SIZES, 1)
    p = check(culsh, X, A, b, W)
    assert p["key_words"] >= 2
    assert p["sort_form"] == 1


def test_run_too_long_falls_back(culsh):
    X, A, b, W = clustered(SIZES + [2049], 2)
    p = check(culsh, X, A, b, W)
    assert p["key_words"] >= 2
    assert p["sort_form"] == 2


def test_all_words_form_agrees(culsh, monkeypatch):
    X, A, b, W = clustered(SIZES, 3)
    monkeypatch.setenv("CULSH_SORT_ALL_WORDS", "1")
    p = check(culsh, X, A, b, W)
    assert p["sort_form"] == 0


@pytest.mark.parametrize("M,W", [(10, 0.02), (11, 0.02), (16, 0.02), (20, 0.02)])
def test_keys_wider_than_128_bits(culsh, M, W):
    """Bucket keys of 4 to 8 words: buckets, codes and a search whose queries
    are indexed points, against the oracle."""
    rng = np.random.default_rng(M)
    N, D, L, T, K = 5000, 32, 3, 4, 5
    X = rng.normal(0, 1, (N, D)).astype(np.float32)
    X[N // 2:] = X[:N // 2] + rng.normal(0, 1e-5, (N // 2, D)).astype(np.float32)
    A = rng.normal(0, 1, (L, M, D)).astype(np.float32)
    b = (rng.random((L, M)) * W).astype(np.float32)
    p = check(culsh, X, A, b, W)
    assert p["key_words"] >= (5 if M > 11 else 4)
    ht = culsh.HashTables()
    ht.reset(N, D, L, M, W, A=A, b=b)
    ht.index(X)
    st = culsh.SearchTables()
    st.reset(ht, K, T)
    st.search(X[:200], dataset=X)
    want = oracle.search(oracle.build_index(X, A, b, W), X, X[:200], K, T)
    np.testing.assert_array_equal(st.getKnnIds(), want["knn_ids"])
    np.testing.assert_array_equal(st.getKnnDistances(), want["knn_dists"])


@pytest.mark.parametrize("form", ["parts", "in place"])
@pytest.mark.parametrize("N,M,dup", [(1, 8, 1), (3, 8, 1), (4096, 8, 1), (4097, 12, 1), (8191, 12, 3), (20000, 16, 1),
                                     (60000, 12, 1), (60000, 12, 5000)])
def test_hash_tables_find_every_bucket(culsh, form, N, M, dup, monkeypatch):
    """Both forms of the hash tables (by parts of 2,048 groups, one part or
    many, a last tile of any length; and in place): the points themselves as
    queries all find their own buckets, and the first probes' buckets are the
    oracle's."""
    monkeypatch.setenv("CULSH_HASH_PARTS_MIN", "1" if form == "parts" else "1000000000000")
    rng = np.random.default_rng(N + M)
    D, L, W = 16, 3, 2.0
    X = rng.normal(0, 4, (max(N // dup, 1), D)).astype(np.float32)
    X = np.ascontiguousarray(X[rng.integers(0, X.shape[0], N)] if dup > 1 else X)
    A = rng.normal(0, 1, (L, M, D)).astype(np.float32)
    b = rng.uniform(0, W, (L, M)).astype(np.float32)
    ht = culsh.HashTables()
    ht.reset(N, D, L, M, W, A=A, b=b)
    ht.index(X)
    q = X[rng.permutation(N)[:2000]]
    st = culsh.SearchTables()
    st.reset(ht, 1, 4)
    st.search(q, dataset=X)
    ref = oracle.search(oracle.build_index(X, A, b, W), X, q, 1, 4)
    for l in range(L):
        qb = st.getQueryBuckets(l)
        assert (qb[:, 0] >= 0).all()
        np.testing.assert_array_equal(qb, ref["qbuckets"][l].reshape(q.shape[0], 4), err_msg=f"table {l}")
    np.testing.assert_array_equal(ht.getBuckets_sizes(0), oracle.build_index(X, A, b, W).sizes(0))


@pytest.mark.parametrize("N,env,form,spills", [
    (4_090, {}, 1, False),            # one part
    (8_300, {}, 1, None),             # four parts, a last tile of 108 keys
    (60_000, {}, 1, None),            # sixteen
    (240_001, {}, 1, True),           # 64, nearly half full: keys that probe past a part's end
    (60_000, {"CULSH_HASH_PART_CAP": "3600"}, 1, True),    # records past a part's space
    (60_000, {"CULSH_HASH_PART_CAP": "0", "CULSH_HASH_SPILL": "200000"}, 1, True),   # every key placed afterwards
    (60_000, {"CULSH_HASH_PART_CAP": "3600", "CULSH_HASH_SPILL": "64"}, 2, True),   # too many: again in place
    (60_000, {"CULSH_HASH_PART_CAP": "0", "CULSH_HASH_SPILL": "0"}, 2, True),
])
def test_hash_tables_by_parts(culsh, monkeypatch, N, env, form, spills):
    """The form by parts with one part and many, records or probes past a part's
    end, and the rebuild in place when those outgrow their list: every point
    finds its own bucket, the first probes' buckets are the oracle's, and keys
    that no point has are not found."""
    import ctypes
    monkeypatch.setenv("CULSH_HASH_PARTS_MIN", "1")
    monkeypatch.setenv("CULSH_HASH_SPILL", str(N))   # the list of a small build must fit its codes' space
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    rng = np.random.default_rng(N)
    D, L, M, W = 16, 3, 12, 2.0
    X = rng.normal(0, 4, (N, D)).astype(np.float32)
    A = rng.normal(0, 1, (L, M, D)).astype(np.float32)
    b = rng.uniform(0, W, (L, M)).astype(np.float32)
    ht = culsh.HashTables()
    ht.reset(N, D, L, M, W, A=A, b=b)
    for _ in range(2):   # a second build of the same object starts afresh
        ht.index(X)
    spilled = ctypes.c_uint()
    assert culsh.lib().culsh_index_hash_form(ht._h, ctypes.byref(spilled)) == form
    if spills is not None:
        assert (spilled.value > 0) == spills
    if env.get("CULSH_HASH_PART_CAP") == "0":
        assert spilled.value == sum(ht.getBuckets(l) for l in range(L))
    own = min(N, 60_000)
    q = np.concatenate([X[-own:], rng.normal(0, 4, (500, D)).astype(np.float32)])
    ref = oracle.build_index(X, A, b, W)
    want = oracle.search(ref, X, q, 1, 4)
    st = culsh.SearchTables()
    st.reset(ht, 1, 4)
    st.search(q, dataset=X)
    for l in range(L):
        qb = st.getQueryBuckets(l)
        assert (qb[:own, 0] >= 0).all()
        np.testing.assert_array_equal(qb, want["qbuckets"][l].reshape(q.shape[0], 4), err_msg=f"table {l}")
        np.testing.assert_array_equal(ht.getBuckets_sizes(l), ref.sizes(l))


def test_fallback_without_room_gives_scratch_back(culsh, monkeypatch):
    """The passes over every word after a run too long: where their buffers
    do not fit beside the first form's, those are freed first."""
    torch = pytest.importorskip("torch")
    X, A, b, W = clustered([1] * 100 + [30_000] * 20, 5)
    L, M, D = A.shape
    ref = oracle.build_index(X, A, b, W)
    left = {}
    for limit in (None, "1000"):
        if limit:
            monkeypatch.setenv("CULSH_SCRATCH_MAX_BYTES", limit)
        ht = culsh.HashTables()
        ht.reset(X.shape[0], D, L, M, W, A=A, b=b)
        before = torch.cuda.mem_get_info()[0]
        for _ in range(2):   # and the next build's first form, beside theirs
            ht.index(X)
        left[limit] = before - torch.cuda.mem_get_info()[0]
        assert ht.profile()["sort_form"] == 2
        for l in range(L):
            np.testing.assert_array_equal(ht.getBuckets_totalIndices(l), ref.ids(l))
        del ht
    assert left["1000"] + (8 << 20) <= left[None]   # 4 bytes a point and table at least, and the runs' lists
