"""The tile pass starts beside the kernel that writes its rare counts
(programmatic dependent launch).  What the earlier kernel writes may not be read
through the read-only path (__ldg, ld.global.nc), which is for data that nobody
writes while a kernel runs, and every solve must see the counts of its own rows
when solves follow one another through the same block of memory."""
import os
import re

import numpy as np
import oracle
import pytest

from conftest import PKG_NAME, ROOT


def test_rare_counts_are_not_read_through_the_read_only_path():
    with open(os.path.join(ROOT, PKG_NAME, "csrc", "k_tc.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    reads = re.findall(r"([^;{}]*)reinterpret_cast<const uint4\*>\(rdense", text)
    assert reads, "the tile pass no longer reads its counts as 16-byte words"
    for before in reads:
        assert "__ldg" not in before and "ldg" not in before and ".nc" not in before, before.strip()
    assert not re.search(r"__restrict__\s+rdense|ld\.global\.nc", text)


def test_bounded_waits_do_not_cover_the_launch_before():
    """The epilogue waits for the counts' launch, without a limit; the roles whose
    limited waits hang on the epilogue (producer and issuer, from their third
    tile on) wait for that launch first, so that a long one is no timeout."""
    with open(os.path.join(ROOT, PKG_NAME, "csrc", "k_tc.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    body = text[text.index("tc_stripe_kernel("):text.index("cuTensorMapEncodeTiled", text.index("tc_stripe_kernel("))]
    loops = body.split("for (int t = t_begin")[1:]
    assert len(loops) == 3  # producer, issuer, epilogue
    for loop in loops[:2]:
        head = loop[:loop.index("mbar_wait")]
        assert re.search(r"if \(nth == 2\) grid_wait\(\);", head)
    assert "grid_wait();" in body[:body.index("for (int t = t_begin; t < t_end")]


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 32, 300])
def test_few_rows_against_long_counts(pkg, rows):
    """Stripes of fewer rows than SMs, whose tile pass starts at once beside the
    counts and takes several tiles per CTA pair while it waits for them."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(rows)
    n, L = 60000, 60
    A = rng.integers(0, 4, size=(n, L)).astype(np.uint64)
    ld = (n + 7) // 8 * 8
    with pkg.Solver.from_calls(A, tau=65536) as s:
        for r0 in (0, 3000):
            out = torch.zeros((rows, ld), dtype=torch.int16, device="cuda:0")
            s.stripe(r0, rows, out.data_ptr(), ld, torch.cuda.current_stream().cuda_stream)
            s.check()
            got = out.cpu().numpy().view(np.uint16)
            for r in range(0, rows, max(1, rows // 5)):
                i = r0 + r
                want = ((A[i + 1:] != A[i]) & (A[i + 1:] != 0) & (A[i] != 0)).sum(1)
                np.testing.assert_array_equal(got[r, r + 1:n - r0], want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [300, 1301])
def test_solves_in_turn_through_one_block(pkg, n):
    """Two sets of one shape and other rare alleles, solved in turn on one stream
    without a wait between them: the pool hands both the same block of counts."""
    torch = pytest.importorskip("torch")
    L, rounds = 90, 12
    sets, want = [], []
    for seed in (1, 2):
        rng = np.random.default_rng(seed * n)
        A = rng.integers(0, max(2, n // (3 * seed)), size=(n, L)).astype(np.uint64)
        sets.append(A)
        want.append(np.triu(oracle.hamming(pkg.dense_ranks(A)[0]), 1))
    ld = (n + 7) // 8 * 8
    with pkg.Solver.from_calls(sets[0], tau=65536) as a, pkg.Solver.from_calls(sets[1], tau=65536) as b:
        out = torch.zeros((2 * rounds, n, ld), dtype=torch.int16, device="cuda:0")
        st = torch.cuda.current_stream().cuda_stream
        for q in range(2 * rounds):
            (a, b)[q % 2].stripe(0, n, out[q].data_ptr(), ld, st)
        a.check()
        b.check()
    for q in range(2 * rounds):
        got = np.triu(out[q, :, :n].cpu().numpy().view(np.uint16), 1)
        np.testing.assert_array_equal(got, want[q % 2])
