"""Forms that take over where the usual one does not apply: dense queries
whose tensor-core buffers do not fit the device, or whose data that path does
not take, against the oracle."""

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _case(seed, N, D, L, M, W, Q, scale=1.0):
    rng = np.random.default_rng(seed)
    X = (rng.normal(0, scale, (N, D))).astype(np.float32)
    Qm = (rng.normal(0, scale, (Q, D))).astype(np.float32)
    A = rng.normal(0, 1, (L, M, D)).astype(np.float32)
    b = (rng.random((L, M)) * W).astype(np.float32)
    return X, Qm, A, b


def _search(culsh, X, A, b, W, K, T, **tuning):
    L, M, D = A.shape
    ht = culsh.HashTables()
    ht.reset(X.shape[0], D, L, M, W, A=A, b=b)
    ht.index(X)
    st = culsh.SearchTables()
    st.reset(ht, K, T)
    if tuning:
        st.set_tuning(**tuning)
    return st


def _check(st, want):
    np.testing.assert_array_equal(st.getKnnIds(), want["knn_ids"])
    np.testing.assert_array_equal(st.getKnnDistances(), want["knn_dists"])
    assert st.getTotalCandidates_unique() == int(want["unique"].sum())
    assert st.getTotalCandidates_nonUnique() == int(want["nonunique"].sum())


@pytest.mark.parametrize("N", [30_000, 1_900_000])
def test_dense_without_room(culsh, monkeypatch, N):
    """The tensor-core path's buffers do not fit: the bitmap kernel, or (bits of
    more points than a block holds) the per-query kernel serves the queries
    that were listed as dense, and later searches plan without the path until
    there is room."""
    D, L, M, W, Q, K, T = 4, 2, 2, 4.0, 6, 10, 4
    X, Qm, A, b = _case(N, N, D, L, M, W, Q)
    want = oracle.search(oracle.build_index(X, A, b, W), X, Qm, K, T)
    monkeypatch.setenv("CULSH_SCRATCH_MAX_BYTES", "1000")
    st = _search(culsh, X, A, b, W, K, T)
    for _ in range(2):
        st.search(Qm, dataset=X)
        _check(st, want)
        assert st.profile()["knn_queries"] == 0
    monkeypatch.delenv("CULSH_SCRATCH_MAX_BYTES")
    st.search(Qm, dataset=X)
    _check(st, want)
    assert st.profile()["knn_queries"] > 0


def test_probe_form_without_room(culsh, monkeypatch):
    """Narrow buckets and eight or more probes: the lookups behind the key filter
    want a hash and a mask per probe; without room the fused form runs."""
    N, D, L, M, W, Q, K, T = 20_000, 16, 4, 8, 1.0, 5_000, 5, 8
    X, _, A, b = _case(7, N, D, L, M, W, 1)
    Qm = X[:Q]
    want = oracle.search(oracle.build_index(X, A, b, W), X, Qm, K, T)
    held = {}
    for limit in (None, "1000"):
        if limit:
            monkeypatch.setenv("CULSH_SCRATCH_MAX_BYTES", limit)
        st = _search(culsh, X, A, b, W, K, T)
        st.search(Qm, dataset=X)
        _check(st, want)
        for l in range(L):
            np.testing.assert_array_equal(st.getQueryBuckets(l), want["qbuckets"][l].reshape(Q, T))
        held[limit] = culsh.lib().culsh_search_device_bytes(st._h)
    assert held["1000"] + 12 * L * Q * T <= held[None]


@pytest.mark.parametrize("how", ["set", "set_other", "restore", "autotune"])
def test_probe_form_survives_tuning(culsh, how):
    """The probe form follows the shape until a form is set: a tuning that is
    read and written back, changed elsewhere, or set and restored keeps it.
    (The form behind the key filter shows by its buffers.)"""
    N, D, L, M, W, Q, K, T = 20_000, 16, 4, 8, 1.0, 20_000, 5, 8
    X, _, A, b = _case(8, N, D, L, M, W, 1)
    st = _search(culsh, X, A, b, W, K, T)
    created = st.get_tuning()
    if how == "set":
        st.set_tuning()
    elif how == "set_other":
        st.set_tuning(ws_threads=256)
    elif how == "restore":
        st.set_tuning(probe_split=1, probe_batch=4)
        st.set_tuning(**created)
    else:   # the tuner times that form too: what it returns, set again, is what it timed
        torch = pytest.importorskip("torch")
        q = torch.from_numpy(X).cuda()
        ids = torch.empty((Q, K), dtype=torch.int32, device="cuda")
        d = torch.empty((Q, K), dtype=torch.float32, device="cuda")
        tune = st.autotune(q.data_ptr(), Q, ids.data_ptr(), d.data_ptr())
        own = _search(culsh, X, A, b, W, K, T)
        own.set_tuning(**{k: tune[k] for k in created if k not in ("search_ms", "configs_tried")})
        for s in (st, own):
            culsh.lib().culsh_search_release(s._h)
            s.search(X, dataset=X)
        assert culsh.lib().culsh_search_device_bytes(st._h) == culsh.lib().culsh_search_device_bytes(own._h)
        return
    st.search(X, dataset=X)
    want = _search(culsh, X, A, b, W, K, T)
    want.search(X, dataset=X)
    assert culsh.lib().culsh_search_device_bytes(st._h) == culsh.lib().culsh_search_device_bytes(want._h)
    st.set_tuning(probe_batch=1)   # a form set: no filter buffers
    culsh.lib().culsh_search_release(st._h)
    st.search(X, dataset=X)
    assert (culsh.lib().culsh_search_device_bytes(st._h) + 12 * L * Q * T
            == culsh.lib().culsh_search_device_bytes(want._h))


@pytest.mark.parametrize("margin", [None, "0"])
@pytest.mark.parametrize("Q", [256, 257, 700])
def test_dense_queries_in_turns(culsh, monkeypatch, Q, margin):
    """More dense queries than one turn's membership rows hold (here 256), the
    last turn full or not, with queries that are scanned exactly in every turn:
    values outside the path's range, and (margin 0) survivors past the lists."""
    N, D, L, M, W, K, T = 6_000, 20, 3, 2, 6.0, 10, 4
    X, Qm, A, b = _case(Q, N, D, L, M, W, Q)
    Qm[::90] *= np.float32(1e-13) / np.abs(Qm[::90]).max()
    want = oracle.search(oracle.build_index(X, A, b, W), X, Qm, K, T)
    monkeypatch.setenv("CULSH_KNN_CHUNK_BYTES", "0")
    if margin:
        monkeypatch.setenv("CULSH_KNN_LIST_MARGIN", margin)
    st = _search(culsh, X, A, b, W, K, T, dense_min=1)
    for _ in range(2):
        st.search(Qm, dataset=X)
        _check(st, want)
        p = st.profile()
        assert p["knn_queries"] == int((want["nonunique"] > 0).sum()) > Q - 20
        assert p["knn_fallback"] >= (Q + 89) // 90


def test_dense_values_outside_every_dense_form(culsh):
    """Values whose squares leave the tensor-core path's range, more points than
    the bitmap kernel's block holds: listed as dense, served per query."""
    N, D, L, M, W, Q, K, T = 1_900_000, 4, 2, 2, 4e18, 4, 10, 4
    X, Qm, A, b = _case(3, N, D, L, M, W, Q, scale=1e18)
    want = oracle.search(oracle.build_index(X, A, b, W), X, Qm, K, T)
    assert want["nonunique"].min() > N // 16
    st = _search(culsh, X, A, b, W, K, T)
    for _ in range(2):
        st.search(Qm, dataset=X)
        _check(st, want)
        assert st.profile()["knn_queries"] == 0
