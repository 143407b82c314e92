"""The device encoder (allele calls -> ranks, operands, rare CSR on the GPU)
against the oracle: every cell of the upper triangle, and the encoder's sizes
(one-hot columns, rare pairs) against the restated reference host encoder."""
import importlib

import numpy as np
import pytest

import oracle
import refgen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["dense", "lists"])
def tch(pkg, request):
    """Every test runs for both holdings of the rare term: per-stripe dense
    counts from the rare groups, and the reference's pair lists."""
    assert pkg.device_count() > 0, "no CUDA device visible"
    pkg.set_rare_term(request.param == "dense")
    yield pkg
    pkg.set_rare_term(True)


def upper_equal(H, ref):
    iu = np.triu_indices(ref.shape[0], 1)
    bad = np.nonzero(H[iu] != ref[iu])[0]
    assert len(bad) == 0, f"{len(bad)} cells differ"


@pytest.mark.parametrize("case_idx", [0, 1, 2])
@pytest.mark.parametrize("tau", [0, 1, 2, 8, 100000])
def test_checkpy_cases_device_encoder(tch, golden, case_idx, tau):
    c = golden["cases"][case_idx]
    A, _ = refgen.checkpy_make(c["n"], c["L"], c["seed"], c["hashed"])
    calls = A.astype(np.uint64)
    with tch.Solver.from_calls(calls, tau=tau) as s:
        info = s.info()
        H, _ = s.run(128)
    assert "%016x" % oracle.rollhash(H) == c["rollhash"]
    if tau > 0:  # same encoding sizes as the reference host (main.rs:366-444)
        x, cnt = oracle.dense_ranks(calls)
        e = oracle.encode(x, cnt, tau)
        assert info["d_onehot"] == e.D and info["n_rare"] == len(e.js) and info["tau"] == tau


def test_run_calls_contract(tch):
    rng = np.random.default_rng(9)
    A = rng.integers(0, 2**64 - 1, size=(333, 77), dtype=np.uint64, endpoint=True) % np.uint64(13)
    A[A == 0] = 0
    A[:, :5] = rng.integers(1, 2**63, size=(333, 5), dtype=np.uint64)  # 64-bit ids, all distinct
    A[::7, 5] = A[0, 5]
    H, secs, tau, sink = tch.run_calls(A, stripe=40)
    assert tau >= 2
    assert [c[0] for c in sink.calls] == list(range(0, 333, 40))
    upper_equal(H, oracle.hamming(oracle.dense_ranks(A)[0]))


@pytest.mark.parametrize("n,L", [(1, 1), (2, 1), (9, 3), (129, 64), (257, 65), (300, 0), (5, 200)])
def test_edge_shapes_device_encoder(tch, n, L):
    rng = np.random.default_rng(n + 7 * L)
    A = rng.integers(0, 5, size=(n, L)).astype(np.uint64)
    with tch.Solver.from_calls(A, tau=3) as s:
        H, _ = s.run(64)
    x = oracle.dense_ranks(A)[0] if L else np.zeros((n, 1), np.uint16)
    upper_equal(H, oracle.hamming(x))


def test_many_alleles_per_locus(tch):
    """A locus near the 65 535-allele limit and one above it."""
    n = 70000
    rng = np.random.default_rng(1)
    A = np.zeros((n, 2), np.uint64)
    A[:, 0] = rng.permutation(n).astype(np.uint64) % np.uint64(65535) + np.uint64(1)
    A[:, 1] = rng.integers(1, 4, n)
    with tch.Solver.from_calls(A, tau=2) as s:
        info = s.info()
    assert info["n"] == n
    A[:, 0] = np.arange(1, n + 1, dtype=np.uint64)  # 70 000 distinct ids
    with pytest.raises(tch.TchError, match="65535"):
        tch.Solver.from_calls(A, tau=2)


def test_longtail_sample_device_vs_host_encoder(tch):
    synth = __import__("importlib").import_module("cgmlst-hamming-gpu_gb300.synth")
    A = synth.longtail(n=3000, L=400, seed=5)
    x, nd = tch.dense_ranks(A)
    for tau in (32, 128):
        enc = tch.encode_host(x, nd, tau)
        with tch.Solver.from_calls(A, tau=tau) as s:
            info = s.info()
            Hd, _ = s.run(512)
        assert info["d_onehot"] == enc.D and info["n_rare"] == enc.n_rare
        Hh, _, _, _ = tch.run(enc, stripe=512)
        iu = np.triu_indices(3000, 1)
        np.testing.assert_array_equal(Hd[iu], Hh[iu])
    upper_equal(Hd, oracle.hamming(x))


def test_rare_term_mode_reported(tch, pkg):
    rng = np.random.default_rng(12)
    A = rng.integers(1, 30, size=(200, 40)).astype(np.uint64)
    with tch.Solver.from_calls(A, tau=8) as s:
        info = s.info()
        H, _ = s.run(64)
    upper_equal(H, oracle.hamming(oracle.dense_ranks(A)[0]))
    x, cnt = oracle.dense_ranks(A)
    assert info["n_rare"] == len(oracle.encode(x, cnt, 8).js)
    assert info["rare_dense"] in (0, 1)


def test_more_loci_than_threads(tch):
    """More loci than one CTA pass of the rare-count kernel covers (1024)."""
    rng = np.random.default_rng(21)
    n, L = 400, 2500
    A = rng.integers(1, 12, size=(n, L)).astype(np.uint64)
    A[rng.random((n, L)) < 0.02] = 0
    x = oracle.dense_ranks(A)[0]
    ref = oracle.hamming(x)
    for tau in (4, 64, 1000):
        with tch.Solver.from_calls(A, tau=tau) as s:
            H, _ = s.run(96)
        upper_equal(H, ref)


def test_wide_stripe_blocks(tch):
    """n above 65 536 columns: the rare counts of a row take several passes
    of the shared-memory counters.  Rows checked against the oracle's block."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(33)
    n, L = 70001, 12
    A = rng.integers(1, 3000, size=(n, L)).astype(np.uint64)  # ~23 rows per allele: rare at tau 64
    A[:, :3] = rng.integers(1, 4, size=(n, 3))  # frequent loci
    x = oracle.dense_ranks(A)[0]
    with tch.Solver.from_calls(A, tau=64) as s:
        assert s.info()["n_rare"] > 0
        for r0, rows in ((0, 200), (4097, 131), (n - 300, 300)):
            ldo = (n - r0 + 7) // 8 * 8
            out = torch.zeros((rows, ldo), dtype=torch.int16, device="cuda")
            s.stripe(r0, rows, out.data_ptr(), ldo, torch.cuda.current_stream().cuda_stream)
            s.check()
            got = out.cpu().numpy().view(np.uint16)
            ref = oracle.hamming_block(x, r0, r0 + rows, r0, n)
            for r in range(rows):
                np.testing.assert_array_equal(got[r, r + 1: n - r0], ref[r, r + 1:])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 7, 8, 9, 33, 255, 257, 600])
@pytest.mark.parametrize("groups", ["pairs", "eights", "whole", "mixed"])
def test_row_runs_piece_edges(pkg, n, groups):
    """Rare groups of two rows, of about eight (one 16-byte piece of members),
    of every row, and of all sizes, so that runs start, end and lie anywhere in
    their pieces; more loci than runs are staged at a time; stripes whose
    counters start at even and odd columns."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    L = 1300
    high = {"pairs": max(2, n // 2), "eights": max(2, n // 8), "whole": 2, "mixed": 0}[groups]
    if high:
        A = rng.integers(1, high, size=(n, L))
    else:
        A = rng.integers(1, rng.integers(2, n + 2, size=L) + 1, size=(n, L))
    A[rng.random((n, L)) < 0.05] = 0
    A = A.astype(np.uint64)
    want = oracle.hamming(pkg.dense_ranks(A)[0])
    with pkg.Solver.from_calls(A, tau=65536) as s:  # every allele rare
        for r0 in (0, 1, n // 2):
            rows, ldo = n - r0, (n - r0 + 7) // 8 * 8
            d = torch.zeros((max(rows, 1), ldo), dtype=torch.int16, device="cuda:0")
            s.stripe(r0, rows, d.data_ptr(), ldo, torch.cuda.current_stream().cuda_stream)
            s.check()
            got = d.cpu().numpy().view(np.uint16)
            for r in range(rows):
                np.testing.assert_array_equal(got[r, r + 1:rows], want[r0 + r, r0 + r + 1:])


@pytest.mark.gpu
@pytest.mark.parametrize("distinct", [(5, 511), (512, 513), (3000, 2049), (8000, 4), (8193, 40), (9100, 9100)])
def test_distinct_counts_around_table_sizes(pkg, distinct):
    """Loci with as many distinct ids as a small hash table holds, with more (the
    tables are built again), and around the rank kernel's one id per thread."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(distinct[0])
    n = 9100
    cols = []
    for d in distinct + (3,):
        ids = rng.choice(2**62, size=d, replace=False).astype(np.uint64) + np.uint64(1)
        cols.append(rng.permutation(np.concatenate([ids, ids[rng.integers(0, d, n - d)]])))
    A = np.stack(cols, axis=1)
    with pkg.Solver.from_calls(A, tau=4) as s:
        ldo = (n + 7) // 8 * 8
        d = torch.zeros((n, ldo), dtype=torch.int16, device="cuda:0")
        s.stripe(0, n, d.data_ptr(), ldo, torch.cuda.current_stream().cuda_stream)
        s.check()
        t = torch.from_numpy(A.view(np.int64)).cuda()
        want = sum((t[:, k, None] != t[None, :, k]).to(torch.int16) for k in range(A.shape[1]))
        assert bool((torch.triu(d[:, :n], 1) == torch.triu(want, 1)).all())


@pytest.mark.gpu
@pytest.mark.parametrize("tau", [1, 2, 32, 128, 129, 130, 1000])
def test_tables_around_group_sizes(pkg, tau):
    """Alleles seen 1, 2, 31-33, 127-129 and 300 times at loci of 1 to 70
    alleles: the encoding's sizes against the host encoder's, the distances
    against the count, with tau on either side of every size."""
    rng = np.random.default_rng(tau)
    n, sizes = 900, [1, 2, 31, 32, 33, 127, 128, 129, 300]
    cols = []
    for k in range(12):
        col, left, a = [], n, 1
        if k >= 8:
            col = [1000 + i for i in range(60)]  # more alleles than lanes
            left -= 60
        for size in rng.permutation(sizes):
            if size <= left:
                col += [a] * int(size)
                left -= int(size)
                a += 1
        cols.append(rng.permutation(np.array(col + [0] * left)))
    A = np.stack(cols, axis=1).astype(np.uint64)
    x, nd = pkg.dense_ranks(A)
    want = oracle.hamming(x)
    counts = [np.bincount(x[:, k])[1:] for k in range(x.shape[1])]
    with pkg.Solver.from_calls(A, tau=tau) as s:
        info = s.info()
        assert info["d_onehot"] == sum(int((c >= tau).sum()) for c in counts)
        assert info["n_rare"] == sum(int((c * (c - 1) // 2)[(c < tau) & (c >= 2)].sum()) for c in counts)
        H, _ = s.run(200)
    iu = np.triu_indices(n, 1)
    np.testing.assert_array_equal(H[iu], want[iu])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [9000, 21000])
def test_rows_of_many_rare_pairs(pkg, n):
    """Sets above and below the pairs per row at which the launch shape changes,
    with rows on both sides of its widths: sampled rows against the count."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    for L in (6, 40):
        A = rng.integers(1, 7, size=(n, L)).astype(np.uint64)  # n / 6 rows per allele, all rare at tau 65536
        with pkg.Solver.from_calls(A, tau=65536) as s:
            assert (s.info()["n_rare"] > 32768 * n) == (n * L / 12 > 32768)
            ldo = (n + 7) // 8 * 8
            d = torch.zeros((n, ldo), dtype=torch.int16, device="cuda:0")
            s.stripe(0, n, d.data_ptr(), ldo, torch.cuda.current_stream().cuda_stream)
            s.check()
            for i in (0, 1, 519, n - 20480 - 1, n - 20480, n - 8193, n - 8192, n - 300, n - 2):
                if 0 <= i < n:
                    want = (A[i + 1:] != A[i]).sum(1)
                    np.testing.assert_array_equal(d[i, i + 1:n].cpu().numpy(), want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [129, 4096, 8193, 131072, 131073, 270000])
def test_rows_sorted_by_bit_maps(pkg, n):
    """Groups of more rows than a warp sorts, over row counts around the words, the
    threads' shares and the windows (131 072 rows) of the bit maps: new profiles'
    distances read every group in its order."""
    rng = np.random.default_rng(n)
    L, m = 6, 9
    top = np.array([1, 2, 3, max(1, n // 300), max(1, n // 129), min(n, 65535)])
    A = rng.integers(1, top[None, :] + 1, size=(n, L)).astype(np.uint64)
    Q = A[rng.integers(0, n, size=m)]
    want = np.zeros((m, n), np.uint16)
    for k in range(L):
        want += Q[:, k, None] != A[None, :, k]
    with pkg.Database(A, tau=n + 1) as db:
        np.testing.assert_array_equal(db.query(Q)[0], want)
        np.testing.assert_array_equal(db.query(Q[:1])[0], want[:1])
    if n <= 8193:
        with pkg.Solver.from_calls(A, tau=n + 1) as s:
            H, _ = s.run(n)
        full = (A[:, None, :] != A[None, : min(n, 600), :]).sum(2).T
        iu = np.triu_indices(min(n, 600), 1, n)
        np.testing.assert_array_equal(H[: min(n, 600)][iu], full[iu])


@pytest.mark.gpu
@pytest.mark.parametrize("tau", [4, 5, 6, 7, 8, 9, 10, 12, 14, 20, 28, 40])
def test_counts_around_quarter_octaves(pkg, tau):
    """The sizes the tau model sums from its bins are those of the encoding: counts
    on either side of the bins' edges, at taus on and off them."""
    rng = np.random.default_rng(tau)
    sizes = [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 19, 20, 23, 24, 27, 28, 31, 32, 39, 40]
    col = np.concatenate([np.full(s, a + 1) for a, s in enumerate(sizes)])
    A = np.stack([rng.permutation(col) for _ in range(9)], axis=1).astype(np.uint64)
    with pkg.Solver.from_calls(A, tau=tau) as s:
        info = s.info()
        assert info["d_onehot"] == 9 * sum(c >= tau for c in sizes)
        assert info["n_rare"] == 9 * sum(c * (c - 1) // 2 for c in sizes if c < tau)


@pytest.mark.gpu
def test_refined_tau_keeps_distances(pkg):
    """A set large enough for a tau between the powers of two: the distances are
    those of another tau."""
    synth = importlib.import_module(pkg.__name__ + ".synth")
    A = synth.longtail(n=9000, L=1343, seed=3)
    with pkg.Solver.from_calls(A) as s:
        H, _ = s.run(4096)
    with pkg.Solver.from_calls(A, tau=64) as s:
        assert s.info()["tau"] == 64
        want, _ = s.run(4096)
    iu = np.triu_indices(9000, 1)
    np.testing.assert_array_equal(H[iu], want[iu])
