"""A database whose tables for new profiles (where each rare group enters each
window of rows, the members in two bytes, the bit columns) do not fit in the
memory that is free: it is made without them, holds its operand, groups (members
in four bytes) and maps alone, and every batch searches the groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 9, 16383, 16384, 16385, 40961, 70001])
@pytest.mark.parametrize("tau", [0, 100000])
def test_queries_without_the_tables(pkg, monkeypatch, n, tau):
    """Row counts around the windows of 16 384 and past two-byte row numbers,
    alleles of single rows, of a few and of most rows, ids the database never
    saw, one profile to more than a tile of them; automatic tau and every allele
    rare: the count on the ids, and the answers of a database with the tables."""
    rng = np.random.default_rng(n + tau)
    L, m = 37, 130
    top = np.maximum(2, (n * rng.random(L) ** 4).astype(np.int64))
    A = rng.integers(0, top[None, :] + 1, size=(n, L)).astype(np.uint64)
    Q = A[rng.integers(0, n, m)].copy()
    fresh = rng.random((m, L)) < 0.2
    Q[fresh] = rng.integers(2**40, 2**41, size=int(fresh.sum()), dtype=np.uint64)
    Q[rng.random((m, L)) < 0.05] = 0
    with pkg.Database(A, tau=tau) as db:
        info = db.info()
        want = db.query(Q)[0]
    for r in range(0, m, 13):
        np.testing.assert_array_equal(want[r], ((A != Q[r]) & (A != 0) & (Q[r] != 0)).sum(1))
    counts = [np.unique(A[:, k][A[:, k] != 0], return_counts=True)[1] for k in range(L)]
    slots = sum(len(c) + 1 for c in counts)
    members = sum(int(c[c < info["tau"]].sum()) for c in counts)
    tables = (4 * (slots * -(-n // 16384) + 1) - 2 * members
              + (info["d_onehot"] + L) * (-(-n // 1024) * 1024 // 8))
    monkeypatch.setenv("TCH_FORCE_GROUP_SEARCH", "1")
    with pkg.Database(A, tau=tau) as db:
        assert info["device_bytes"] - db.info()["device_bytes"] == tables
        for k in (1, 8, 9, m):
            np.testing.assert_array_equal(db.query(Q[:k])[0], want[:k])
