"""The sums behind the automatic tau: the counts go into bins of a quarter of an
octave, and a candidate's one-hot columns, rare pairs and rare cells are sums of
whole bins."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def allele_counts(A):
    return np.concatenate([np.unique(c[c != 0], return_counts=True)[1] for c in A.T]).astype(np.float64)


def table(sizes, loci, rng):
    col = np.concatenate([np.full(s, a + 1) for a, s in enumerate(sizes)])
    return np.stack([rng.permutation(col) for _ in range(loci)], axis=1).astype(np.uint64)


@pytest.mark.parametrize("sizes", [range(1, 41), [2**k + d for k in range(2, 10) for d in (-1, 0, 1)],
                                   [5 * 2**k // 4 + d for k in range(3, 9) for d in (-1, 0)], [1] * 300, [4000, 1, 1]])
def test_sums_of_the_candidates(pkg, sizes):
    """Counts on either side of every power of two (and of the quarters between
    them): each candidate's columns, pairs and cells, as the features give them,
    against the counts of the table."""
    A = table(list(sizes), 9, np.random.default_rng(len(list(sizes))))
    c = allele_counts(A)
    f = pkg.tau_features(A)
    assert set(f["taus"].tolist()) == {2**k for k in range(1, 17)}
    for tau, row in zip(f["taus"], f["feats"]):
        rare = c[(c < tau) & (c >= 2)]
        # f32 logarithms of whole numbers: half a unit in the last place each
        want = [np.log(tau), np.log1p((c >= tau).sum()), np.log1p((rare * (rare - 1) / 2).sum()), np.log1p(rare.sum())]
        np.testing.assert_allclose(row[6:10], want, rtol=2.0**-23, atol=0)


def picks(c, n, L, gemm=4.8e15, dense=1.9e12):
    """The power of two with the least estimate, and what the quarters of the
    octaves beside it make of it."""
    def est(tau):
        rare = c[c < tau]
        k = max(256, -(-(L + int((c >= tau).sum())) // 256) * 256)
        return n * (n - 1) / 2 * k / gemm + (rare * (rare - 1) / 2).sum() / dense

    best = min((2**k for k in range(1, 17)), key=est)
    refined, least = best, 0.985 * est(best)
    if best >= 8 and est(best) >= 1e-4:
        lg = best.bit_length() - 1
        for first in range(4 * lg - 3, 4 * lg + 4):
            tau = ((4 + first % 4) << (first // 4)) // 4
            if est(tau) < least:
                refined, least = tau, est(tau)
    return best, refined


@pytest.mark.parametrize("n,L,seed", [(9000, 1343, 3), (10000, 1142, 5), (12000, 600, 1), (2000, 300, 1)])
def test_automatic_tau_is_the_refined_minimum(pkg, n, L, seed):
    """The solver's tau is the one that the sums give: between two powers of two
    for the first two sets, a power of two where that gains too little, and where
    the set is too small to be refined."""
    synth = importlib.import_module(pkg.__name__ + ".synth")
    A = synth.longtail(n=n, L=L, seed=seed)
    best, refined = picks(allele_counts(A), n, L)
    with pkg.Solver.from_calls(A) as s:
        assert s.info()["tau"] == refined
    assert (refined != best) == (n in (9000, 10000))
    assert (refined & (refined - 1) != 0) == (n in (9000, 10000))
