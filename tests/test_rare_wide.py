"""Rare counts of sets of more than 65 536 profiles, whose group members take four
bytes: stripes of every width class with the row runs, and with groups so large
that the runs are found per locus instead, against the count on the ids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alleles,L", [(2, 40), (9, 40), (2, 300)])
def test_wide_sets_with_crowded_groups(pkg, alleles, L):
    """More and fewer than eight rare pairs per row and column; the last rows,
    narrow ones, the widest that one pass holds, and ones that need two; more loci
    than a narrow row's CTA takes at a time."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(L + alleles)
    n = 70001
    A = rng.integers(0, alleles + 1, size=(n, L)).astype(np.uint64)
    t = torch.from_numpy(A.astype(np.int16)).cuda()
    with pkg.Solver.from_calls(A, tau=65536) as s:
        assert (s.info()["n_rare"] > 8 * n * n) == (L * (alleles / (alleles + 1)) ** 2 / alleles / 2 > 8)
        for width in (1, 3, 255, 8192, 8193, 20000, 65536, n):
            r0, rows = n - width, min(width, 40)
            ld = (width + 7) // 8 * 8
            out = torch.full((rows, ld), -1, dtype=torch.int16, device="cuda")
            s.stripe(r0, rows, out.data_ptr(), ld, torch.cuda.current_stream().cuda_stream)
            s.check()
            for r in range(0, rows, 13):
                q, x = t[r0 + r], t[r0 + r + 1:]
                want = ((x != q) & (x != 0) & (q != 0)).sum(1).to(torch.int16)
                assert bool((out[r, r + 1:width] == want).all())
