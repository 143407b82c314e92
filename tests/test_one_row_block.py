"""Stripes, query batches and sets of at most 128 rows, whose tiles go to CTA pairs
or to CTAs by themselves as their number decides: both against the count on the
ids, around the 128 rows and around the numbers of tiles (240 columns each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def counts(torch, A, rows):
    """Distances of the given rows to every row of A, counted locus by locus."""
    t = torch.from_numpy(A.view(np.int64)).cuda()
    d = torch.zeros((len(rows), len(A)), dtype=torch.int16, device="cuda")
    q = t[torch.as_tensor(rows, device="cuda")]
    for k in range(A.shape[1]):
        a, b = q[:, k, None], t[None, :, k]
        d += ((a != b) & (a != 0) & (b != 0)).to(torch.int16)
    return d


@pytest.mark.parametrize("n", [2000, 18240, 18241, 36480, 36481, 60000])
@pytest.mark.parametrize("split", [False, True])
def test_stripes_of_few_rows(pkg, n, split):
    """77 tiles and more than one wave of pairs, 152 and 153, several tiles per CTA;
    rows at the set's start, at an odd row and at its end; operands whole and split
    along K."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    L = 23
    A = rng.integers(0, 40, size=(n, L)).astype(np.uint64)
    ld = (n + 7) // 8 * 8
    pkg.set_max_chunk_bytes(256 * (-(-n // 256) * 256) if split else 0)  # 256 bytes of a row per piece
    try:
        s = pkg.Solver.from_calls(A, tau=max(2, n // 41))
    finally:
        pkg.set_max_chunk_bytes(0)
    assert s.info()["d_onehot"] > 100 and s.info()["n_rare"] > 0
    assert (s.info()["k_chunks"] > 1) == split
    for rows in (1, 33, 127, 128, 129):
        for r0 in (0, 7, n - rows):
            out = torch.full((rows, ld), -1, dtype=torch.int16, device="cuda")
            s.stripe(r0, rows, out.data_ptr(), ld, torch.cuda.current_stream().cuda_stream)
            s.check()
            want = counts(torch, A, np.arange(r0, r0 + rows))[:, r0:]
            assert bool((torch.triu(out[:, :n - r0], 1) == torch.triu(want, 1)).all())
            assert bool((out[:, n - r0:] == -1).all())
    s.close()


@pytest.mark.parametrize("n", [18241, 36481])
def test_query_batches_of_one_row_block(pkg, n):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    A = rng.integers(0, 60, size=(n + 129, 19)).astype(np.uint64)
    want = counts(torch, A, np.arange(n, n + 129))[:, :n].cpu().numpy()
    with pkg.Database(A[:n], tau=n // 50) as db:
        for m in (9, 64, 127, 128, 129):
            np.testing.assert_array_equal(db.query(A[n:n + m])[0], want[:m])


@pytest.mark.parametrize("shapes", ["small", "edge", "mixed", "few"])
def test_batches_of_small_sets(pkg, shapes):
    """400 sets of 1 to 128 profiles; sets of 127 to 129; small ones beside large
    ones, in two launches; fewer small sets than pairs."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(len(shapes))
    sizes = {"small": rng.integers(1, 129, 400), "edge": rng.integers(127, 130, 300),
             "mixed": np.concatenate([rng.integers(2, 129, 500), [700, 1300, 241]]), "few": rng.integers(2, 129, 40)}
    sets = [rng.integers(0, 30, size=(int(n), int(rng.integers(1, 400)))).astype(np.uint64) for n in sizes[shapes]]
    with pkg.Batch(sets, taus=[3] * len(sets)) as b:
        off, ld = b.layout()
        out = torch.full((int(off[-1]) + 8,), -1, dtype=torch.int16, device="cuda")
        b.set_schedule(0)
        for _ in range(2):
            b.run(out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        b.check()
        got = out.cpu().numpy()
    for A, o, w in zip(sets, off, ld):
        n = len(A)
        H = got[int(o):int(o) + n * int(w)].reshape(n, int(w))[:, :n]
        want = ((A[:, None, :] != A[None]) & (A[:, None, :] != 0) & (A[None] != 0)).sum(2)
        iu = np.triu_indices(n, 1)
        np.testing.assert_array_equal(H[iu], want[iu])
