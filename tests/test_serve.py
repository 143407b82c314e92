"""Serving: new profiles against a resident database, through the C ABI
(tch_db_query, tch_server_*), every distance against the oracle's brute-force
count of the joint profile set (check.py:39-44)."""
import importlib
import threading

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
PKG = "cgmlst-hamming-gpu_gb300"


@pytest.fixture(scope="module")
def tch(pkg):
    assert pkg.device_count() > 0, "no CUDA device visible"
    return pkg


def expected(db_calls, q):
    """(q x db, q x q) distances by the oracle on the joint set."""
    n = len(db_calls)
    x = oracle.dense_ranks(np.concatenate([db_calls, q]))[0]
    m = len(q)
    qdb = oracle.hamming_block(x, n, n + m, 0, n)
    qq = oracle.hamming_block(x, n, n + m, n, n + m)
    return qdb, qq


def check(qdb, qq, exp_qdb, exp_qq):
    np.testing.assert_array_equal(qdb, exp_qdb)
    if qq is not None and len(qq) > 1:
        iu = np.triu_indices(len(qq), 1)
        np.testing.assert_array_equal(qq[iu], exp_qq[iu])


def profiles(n, L, seed, alleles=40):
    synth = importlib.import_module(PKG + ".synth")
    return synth.zipf_profiles(n, L, seed, 1.2, lambda rng, L: rng.integers(2, alleles, L),
                               lambda rng, L: rng.uniform(0.0, 0.05, L), hashed_frac=0.05)


@pytest.mark.parametrize("tau", [0, 2, 16, 100000])
def test_query_against_database(tch, tau):
    A = profiles(900, 150, seed=1)
    db_calls, q = A[:700], A[700:]
    q = q.copy()
    q[0, :20] = np.arange(1, 21, dtype=np.uint64) + np.uint64(2**62)  # ids the database has never seen
    q[1] = 0                                                          # all missing
    q[2] = db_calls[5]                                                # a database row again
    exp_qdb, exp_qq = expected(db_calls, q)
    with tch.Database(db_calls, tau=tau) as db:
        for m in (1, 3, 57, 200):
            qdb, qq = db.query(q[:m])
            check(qdb, qq, exp_qdb[:m], exp_qq[:m, :m])
    assert exp_qdb[2, 5] == 0


def test_query_wide_database(tch):
    """More database rows than one pass of the shared-memory counters (65 536)."""
    rng = np.random.default_rng(3)
    n, L = 70001, 10
    A = rng.integers(1, 4000, size=(n + 40, L)).astype(np.uint64)  # mostly rare alleles
    A[:, :2] = rng.integers(1, 5, size=(n + 40, 2))
    with tch.Database(A[:n], tau=64) as db:
        qdb, qq = db.query(A[n:])
    exp_qdb, exp_qq = expected(A[:n], A[n:])
    check(qdb, qq, exp_qdb, exp_qq)


def test_server_results_same_alone_and_in_the_mix(tch):
    A = profiles(1500, 200, seed=4)
    db_calls = A[:1000]
    rng = np.random.default_rng(5)
    batches = []
    for _ in range(14):
        m = int(rng.integers(1, 120))
        idx = rng.integers(1000, 1500, size=m)
        batches.append(A[idx].copy())
    with tch.Database(db_calls) as db:
        alone = [db.query(b) for b in batches]
        with tch.Server(db, slots=4) as sv:
            # submitted from several threads at once: they run concurrently
            ids = [None] * len(batches)

            def put(k):
                ids[k] = sv.submit(batches[k])

            ts = [threading.Thread(target=put, args=(k,)) for k in range(len(batches))]
            for t in ts:
                t.start()
            for t in ts:
                t.join()
            mixed = [sv.wait(i) for i in ids]
    for b, (qa, qqa), (qm, qqm, queued, lat) in zip(batches, alone, mixed):
        np.testing.assert_array_equal(qm, qa)
        if len(b) > 1:
            iu = np.triu_indices(len(b), 1)
            np.testing.assert_array_equal(qqm[iu], qqa[iu])
        assert lat >= queued >= 0
        exp_qdb, exp_qq = expected(db_calls, b)
        check(qm, qqm, exp_qdb, exp_qq)


def test_server_admission_by_memory(tch):
    """A budget below two requests runs them one at a time, still exact."""
    A = profiles(800, 120, seed=6)
    with tch.Database(A[:600]) as db:
        budget = db.query_bytes(100) + db.query_bytes(100) // 2
        with tch.Server(db, slots=3, budget=budget) as sv:
            ids = [sv.submit(A[600 + 50 * k: 700 + 50 * k]) for k in range(3)]
            res = [sv.wait(i) for i in ids]
    for k, (qdb, qq, queued, lat) in enumerate(res):
        exp_qdb, exp_qq = expected(A[:600], A[600 + 50 * k: 700 + 50 * k])
        check(qdb, qq, exp_qdb, exp_qq)


def test_query_errors(tch):
    A = profiles(300, 50, seed=7)
    with tch.Database(A[:200]) as db:
        with pytest.raises(tch.TchError):
            db.query(A[200:, :40])  # wrong locus count


def test_query_against_k_chunked_database(tch):
    """A database whose operand rows are split along K into several
    allocations: the new profiles' rows follow the same split."""
    A = profiles(600, 300, seed=9, alleles=120)
    try:
        tch.set_max_chunk_bytes(1024 * 512)  # rows padded to 512 -> chunks of 1 KB of K
        with tch.Database(A[:500], tau=8) as db:
            assert db.info()["k_chunks"] > 1
            qdb, qq = db.query(A[500:])
    finally:
        tch.set_max_chunk_bytes(0)
    exp_qdb, exp_qq = expected(A[:500], A[500:])
    check(qdb, qq, exp_qdb, exp_qq)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 9, 16383, 16384, 16385, 65537, 70001])
@pytest.mark.parametrize("tau", [0, 100000])
def test_query_window_edges(pkg, n, tau):
    """Database sizes around the windows of the rare counts (16 384 rows) and
    past two-byte row numbers; alleles of single rows, of a few and of most
    rows; ids the database never saw; automatic tau and every allele rare."""
    rng = np.random.default_rng(n)
    L, m = 37, 5
    top = np.maximum(2, (n * rng.random(L) ** 4).astype(np.int64))
    A = rng.integers(0, top[None, :] + 1, size=(n, L)).astype(np.uint64)
    Q = A[rng.integers(0, n, m)].copy()
    fresh = rng.random((m, L)) < 0.2
    Q[fresh] = rng.integers(2**40, 2**41, size=int(fresh.sum()), dtype=np.uint64)
    Q[rng.random((m, L)) < 0.05] = 0
    want = np.stack([((A != q) & (A != 0) & (q != 0)).sum(1) for q in Q])
    with pkg.Database(A, tau=tau) as db:
        got, qq = db.query(Q)
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(db.query(Q[:1], want_qq=False)[0], want[:1])
    both = np.stack([((Q != q) & (Q != 0) & (q != 0)).sum(1) for q in Q])
    np.testing.assert_array_equal(np.triu(qq, 1), np.triu(both, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1025, 2051])
@pytest.mark.parametrize("L", [1, 15, 17, 511, 513, 1100])
def test_few_profiles_by_bit_columns(pkg, n, L):
    """One, eight (the most that go by the bit columns) and nine profiles (the
    tile pass) give the same distances, at row counts around the columns' words
    and CTAs and locus counts around the warps' shares."""
    rng = np.random.default_rng(n * 7 + L)
    A = rng.integers(0, rng.integers(2, 30, size=L)[None, :], size=(n, L)).astype(np.uint64)
    Q = rng.integers(0, 30, size=(9, L)).astype(np.uint64)
    want = np.stack([((A != q) & (A != 0) & (q != 0)).sum(1) for q in Q])
    with pkg.Database(A, tau=max(2, n // 12)) as db:
        for m in (1, 8, 9):
            np.testing.assert_array_equal(db.query(Q[:m])[0], want[:m])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16500, 16504])
@pytest.mark.parametrize("m", [255, 256, 257, 600])
@pytest.mark.parametrize("pinned", [False, True])
def test_results_copied_in_blocks(pkg, n, m, pinned):
    """Results large enough to go back block by block (256 profiles each) beside
    the kernels, rows packed and pitched, into page-locked and pageable buffers,
    twice in a row on the same lane and from two threads."""
    rng = np.random.default_rng(n + m)
    L = 21
    A = rng.integers(0, 12, size=(n, L)).astype(np.uint64)
    Q = rng.integers(0, 13, size=(m, L)).astype(np.uint64)
    want = np.zeros((m, n), np.uint16)
    both = np.zeros((m, m), np.uint16)
    for k in range(L):
        want += (Q[:, k, None] != A[None, :, k]) & (Q[:, k, None] != 0) & (A[None, :, k] != 0)
        both += (Q[:, k, None] != Q[None, :, k]) & (Q[:, k, None] != 0) & (Q[None, :, k] != 0)
    with pkg.Database(A, tau=600) as db:
        def one():
            out = pkg.pinned_empty((m, n)) if pinned else np.empty((m, n), np.uint16)
            for _ in range(2):
                out[:] = 0xFFFF
                qdb, qq = db.query(Q, out=out)
                np.testing.assert_array_equal(qdb, want)
                np.testing.assert_array_equal(np.triu(qq, 1), np.triu(both, 1))
        errors = []

        def guarded():
            try:
                one()
            except BaseException as e:  # noqa: BLE001
                errors.append(e)

        threads = [threading.Thread(target=guarded) for _ in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors[0]


@pytest.mark.gpu
@pytest.mark.parametrize("n,L", [(2048, 2047), (2049, 2048), (2047, 2049), (16385, 40), (40961, 9), (700, 4100), (3, 1)])
@pytest.mark.parametrize("m", [1, 3, 8])
def test_few_profiles_at_the_clusters_edges(pkg, n, L, m):
    """Row counts around a CTA's 2 048 and a cluster's 16 384 rows, locus counts
    around a chunk's 2 048: rare, frequent, new and missing ids in every profile,
    id lists of any length (none, one, thousands)."""
    rng = np.random.default_rng(n * 3 + L + m)
    high = rng.choice([1, 2, 6, 40, 3000], size=L)
    A = rng.integers(0, high[None, :], size=(n, L)).astype(np.uint64) * 3
    Q = rng.integers(0, 3 * high[None, :] + 2, size=(m, L)).astype(np.uint64)
    Q[::2] = np.where(rng.random((len(Q[::2]), L)) < 0.6, A[rng.integers(0, n, size=len(Q[::2]))], Q[::2])
    want = np.zeros((m, n), np.uint16)
    for k in range(L):
        want += (Q[:, k, None] != A[None, :, k]) & (Q[:, k, None] != 0) & (A[None, :, k] != 0)
    with pkg.Database(A, tau=max(2, n // 9)) as db:
        np.testing.assert_array_equal(db.query(Q)[0], want)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [2, 31, 32, 33, 65, 200])
@pytest.mark.parametrize("L", [1, 7, 8, 64, 513, 1030])
def test_batch_pairs_at_tile_edges(pkg, m, L):
    """The batch's own pairs around the tiles of 32 x 32 and the loci's eighths
    and chunks of 64: ids that differ in one half only, missing calls."""
    rng = np.random.default_rng(m * 11 + L)
    low, top = (rng.integers(0, 3, size=(m, L), dtype=np.uint64) for _ in range(2))
    Q = low | top << np.uint64(32)
    A = Q[: max(1, m // 2)]
    want = np.zeros((m, m), np.uint16)
    for k in range(L):
        want += (Q[:, k, None] != Q[None, :, k]) & (Q[:, k, None] != 0) & (Q[None, :, k] != 0)
    with pkg.Database(A) as db:
        got, qq = db.query(Q)
    np.testing.assert_array_equal(np.triu(qq, 1), np.triu(want, 1))
    np.testing.assert_array_equal(got, want[:, : len(A)])
