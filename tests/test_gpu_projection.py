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


@pytest.mark.parametrize("N,D,L,M", [(1027, 33, 4, 16), (1027, 33, 5, 13), (130, 128, 8, 16), (2049, 130, 3, 43),
                                     (127, 7, 16, 16), (5, 64, 6, 12)])
def test_simt_codes(culsh, N, D, L, M, monkeypatch):
    monkeypatch.setenv("CULSH_PROJECT_SIMT", "1")
    rng = np.random.default_rng(N + D + M)
    X = features("plain", N, D, rng)
    A, b = projection(L, M, D, 3.0, rng)
    assert check(culsh, X, A, b, 3.0)["tensor_cores"] == 0
