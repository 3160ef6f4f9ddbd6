"""Launches that depend on what ran before in the process: shared memory is
opted into per kernel and only ever grows, so a size that needs it is tried
in a process of its own."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MEMBERSHIP = """
import numpy as np, culsh_gb300 as culsh, oracle
N, L, M, W = {N}, {L}, {M}, {W}
D, Q, K, T = 8, 16, 10, 4
rng = np.random.default_rng(N)
X = rng.normal(0, 1, (N, D)).astype(np.float32)
Qm = rng.normal(0, 1, (Q, D)).astype(np.float32)
A = rng.normal(0, 1, (L, M, D)).astype(np.float32)
b = (rng.random((L, M)) * W).astype(np.float32)
ht = culsh.HashTables()
ht.reset(N, D, L, M, W, A=A, b=b)
ht.index(X)
st = culsh.SearchTables()
st.reset(ht, K, T)
st.set_tuning(dense_min=1)
st.search(Qm, dataset=X)
assert st.profile()["knn_queries"] > 0
largest = max(int(ht.getBuckets_sizes(l).max()) for l in range(L))
assert (largest >= 512) == {bank}, largest
want = oracle.search(oracle.build_index(X, A, b, W), X, Qm, K, T)
np.testing.assert_array_equal(st.getKnnIds(), want["knn_ids"])
np.testing.assert_array_equal(st.getKnnDistances(), want["knn_dists"])
assert st.getTotalCandidates_unique() == int(want["unique"].sum())
"""


@pytest.mark.parametrize("bank", [True, False], ids=["bank_lists", "ids"])
@pytest.mark.parametrize("N", [268_000, 271_000, 280_000, 293_800, 294_900, 296_000])
def test_membership_rows_around_48_kb(N, bank):
    """The membership kernel's bits are 33 to 37 KB at these N, on either side of
    what its static shared memory leaves of the 48 KB that need no opt-in."""
    L, M, W = (3, 2, 6.0) if bank else (8, 6, 1.0)
    r = subprocess.run([sys.executable, "-c", MEMBERSHIP.format(N=N, L=L, M=M, W=W, bank=bank)], cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr

THREADS = """
import threading
import numpy as np, culsh_gb300 as culsh
SHAPES = [(2_000, 16, 1, 4, 4.0), (2_000, 256, 4, 16, 16.0), (2_000, 64, 4, 8, 8.0), (2_000, 300, 8, 16, 16.0)]
errors = []
def work(i):
    try:
        N, D, L, M, W = SHAPES[i % len(SHAPES)]
        rng = np.random.default_rng(i)
        X = np.round(rng.normal(0, 20, (N, D))).astype(np.float32)
        A = rng.normal(0, 0.2, (L, M, D)).astype(np.float32)
        b = (rng.random((L, M)) * W).astype(np.float32)
        ht = culsh.HashTables()
        ht.reset(N, D, L, M, W, A=A, b=b)
        st = culsh.SearchTables()
        first = None
        for _ in range(60):
            ht.index(X)
            st.reset(ht, 5, 2)
            st.set_tuning(dense_min=1)
            st.search(X[:64], dataset=X)
            got = (ht.getBuckets_totalIndices(0), st.getKnnIds())
            first = first or got
            assert all(np.array_equal(a, b) for a, b in zip(first, got))
        assert ht.profile()["tensor_cores"] == 1
    except Exception as e:
        errors.append(f"{i}: {e}")
ts = [threading.Thread(target=work, args=(i,)) for i in range(8)]
for t in ts: t.start()
for t in ts: t.join()
assert not errors, errors
"""


def test_threads_with_indexes_of_different_shapes():
    """Eight threads build and search indexes whose kernels want different
    amounts of shared memory: none takes back what another opted into."""
    r = subprocess.run([sys.executable, "-c", THREADS], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
