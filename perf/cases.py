"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values; ``prepare`` makes what a user's program holds
before the call (inputs from a seed, on the GPU or in host memory as the entry
point takes them, and the solver, database or batch that such a program keeps),
``run`` is one pass through the public entry points.  Kinds:

triangle   a device-resident whole upper triangle, ``Solver.stripe``: the main
           path, from the smallest sets (launches and latency) to the 63 005
           profiles of the long-tail outbreak shape
run_calls  allele calls in host memory to u16 stripes in host memory (device
           encoder, triangle, copy-out, the caller's callback)
run_bits   the reference's own entry point ``tch_run``: bit-packed operands and
           pair lists in host memory, stripes back to the callback
query      new profiles against a database resident on the device, one isolate
           at a time or a batch of them
batch      many uneven sets solved by one replay of a captured schedule
mst        the minimum spanning tree of a full matrix in device memory
neighbors  the k nearest profiles of every profile of such a matrix
table      what the command-line tool does: the TSV table parsed on the GPU,
           encoded, solved, and the matrix formatted as TSV text

Only cells that the entry points define are returned: the triangle entry points
leave the cells at and below the diagonal unspecified, so a caller takes the
rectangles right of its diagonal blocks as they lie and masks the blocks.
"""
import importlib
import math

import numpy as np
import torch

tch = importlib.import_module("cgmlst-hamming-gpu_gb300")

DEV = "cuda:0"
LOCI = (1142, 1343, 2794, 3016)  # schemes of the batched benchmark


# ------------------------------------------------------------------ profiles

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _profiles(n, L, law, seed):
    """n x L allele ids (int64 bit patterns on the GPU, 0 = missing).

    small     distinct alleles per locus lognormal (mean 40, at most 500), Zipf(1.1) calls, 2% missing
    longtail  median 60 with a tail to 3 000, Zipf(1.2), 1-5% missing per locus, 5% hashed 64-bit ids
    founders  50 founder alleles per locus drawn uniformly, 1% mutated to fresh ids, 2% missing
    uneven    the batched sets: Zipf(1.0-1.4), 0-8% missing
    clonal    one ancestor (long-tail law) per 40 profiles, 0-3% of the loci mutated: outbreak clusters"""
    g = _gen(seed)
    if law == "clonal":
        anc = _profiles(max(2, n // 40), L, "longtail", seed + 7919)
        x = anc[torch.randint(0, anc.shape[0], (n,), generator=g, device=DEV)]
        rate = 0.03 * torch.rand((n, 1), generator=g, device=DEV)
        hit = torch.rand((n, L), generator=g, device=DEV) < rate
        donors = torch.randint(0, anc.shape[0], (n,), generator=g, device=DEV)
        x = torch.where(hit, anc[donors], x)
        return x.contiguous()
    if law == "founders":
        k = torch.full((L,), 50, device=DEV)
        s, miss = 0.0, torch.full((L, 1), 0.02, device=DEV)
    else:
        z = torch.randn((L,), generator=g, device=DEV)
        if law == "longtail":
            k, s = torch.exp(math.log(60.0) + 1.26 * z).round().clamp(2, 3000).long(), 1.2
            miss = 0.01 + 0.04 * torch.rand((L, 1), generator=g, device=DEV)
        else:
            k, s = torch.exp(math.log(40.0) - 0.5 + z).round().clamp(2, 500).long(), 1.1
            miss = torch.full((L, 1), 0.02, device=DEV)
            if law == "uneven":
                s = 1.0 + 0.4 * float(torch.rand((1,), generator=g, device=DEV))
                miss = torch.full((L, 1), 0.08 * float(torch.rand((1,), generator=g, device=DEV)), device=DEV)
    kmax = int(k.max())
    rank = torch.arange(1, kmax + 1, device=DEV, dtype=torch.float64)
    cdf = torch.where(rank[None, :] <= k[:, None], rank.pow(-s)[None, :], 0.0).cumsum(1)
    cdf = (cdf / cdf[:, -1:]).float()
    ids = torch.randint(1, 2**32, (L, kmax), generator=g, device=DEV)
    if law == "longtail":
        hashed = torch.rand((L, kmax), generator=g, device=DEV) < 0.05
        ids = torch.where(hashed, torch.randint(2**32, 2**63 - 1, (L, kmax), generator=g, device=DEV), ids)
    u = torch.rand((L, n), generator=g, device=DEV)
    idx = torch.minimum(torch.searchsorted(cdf, u, right=True), k[:, None] - 1)
    x = ids.gather(1, idx)
    del idx
    if law == "founders":
        mut = torch.rand((L, n), generator=g, device=DEV) < 0.01
        x = torch.where(mut, torch.randint(2**32, 2**63 - 1, (L, n), generator=g, device=DEV), x)
    x.masked_fill_(u.uniform_(generator=g) < miss, 0)
    return x.t().contiguous()


def _host(x):
    return x.cpu().numpy().view(np.uint64)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _up8(n):
    return (n + 7) // 8 * 8


# ------------------------------------------------------------- result shapes

def _triangle(H, n):
    """The strict upper triangle of H (n x ld): the rectangle right of each
    diagonal block, a view, and the diagonal blocks with j <= i zeroed."""
    B = max(512, -(-n // 30))
    ld = H.stride(0)
    full = n // B
    out = [H[a:a + B, a + B:n] for a in range(0, n - B, B)]
    if full:
        out.append(torch.triu(H.as_strided((full, B, B), (B * ld + B, ld, 1)), 1))
    if n % B:
        out.append(torch.triu(H[full * B:n, full * B:n], 1))
    return out


class _HostMatrix:
    """A callback that keeps the stripes as one host matrix, with the cells at
    and below the diagonal zero."""

    def __init__(self, n, stripe):
        self.H = np.zeros((n, n), np.uint16)
        self.mask = np.triu(np.ones((min(stripe, n),) * 2, np.uint16), 1)

    def __call__(self, ctx, r0, rows, w, ptr):
        s = np.ctypeslib.as_array(ptr, shape=(rows, w))
        dst = self.H[r0:r0 + rows, r0:]
        dst[:, rows:] = s[:, rows:]
        np.multiply(s[:, :rows], self.mask[:rows, :rows], out=dst[:, :rows])


# --------------------------------------------------------------------- cases

def listed():
    return [
        # one outbreak's isolates: launches and latency are the whole cost
        {"name": "triangle_outbreak", "kind": "triangle", "n": 151, "L": 1142, "law": "small", "tau": 0},
        # a national collection of ordinary size
        {"name": "triangle_small", "kind": "triangle", "n": 2000, "L": 1142, "law": "small", "tau": 0},
        # the founder-allele shape: tens of thousands of frequent one-hot columns or very large rare groups
        {"name": "triangle_founders", "kind": "triangle", "n": 12011, "L": 5000, "law": "founders", "tau": 0},
        # the headline shape, an international database in one pass
        {"name": "triangle_longtail", "kind": "triangle", "n": 63005, "L": 1142, "law": "longtail", "tau": 0},
        # from allele calls in host memory to a matrix in host memory
        {"name": "run_calls", "kind": "run_calls", "n": 10007, "L": 1343, "law": "longtail", "stripe": 512},
        # a Rust host linked against the reference's entry point
        {"name": "run_bits", "kind": "run_bits", "n": 12001, "L": 1142, "law": "longtail", "tau": 256,
         "stripe": 4096},
        # one new isolate against the resident database: latency
        {"name": "query_one", "kind": "query", "n": 200000, "L": 1142, "m": 1, "law": "longtail"},
        # a sequencing run's isolates against it
        {"name": "query_many", "kind": "query", "n": 200000, "L": 1142, "m": 701, "law": "longtail"},
        # many independent collections, 50 to 5 000 profiles each, schedule tuned once
        {"name": "batch_uneven", "kind": "batch", "count": 48, "low": 50, "high": 5000, "shapes": 1},
        # outbreak clusters joined by their minimum spanning tree
        {"name": "mst_clusters", "kind": "mst", "n": 30011, "L": 1142, "law": "clonal"},
        # the ten nearest profiles of every profile
        {"name": "neighbors_10", "kind": "neighbors", "n": 40009, "L": 1142, "law": "longtail", "k": 10},
        # the command-line tool's run: table in, matrix text out
        {"name": "table_to_text", "kind": "table", "n": 4001, "L": 1142, "law": "longtail"},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["triangle", "triangle", "triangle", "run_calls", "run_bits", "query", "query", "batch", "mst",
                       "neighbors", "table"])
    law = rng.choice(["small", "longtail", "longtail", "uneven", "clonal"])
    L = rng.choice(LOCI + (97, 1142))
    if kind == "triangle":
        if rng.random() < 0.25:
            return {"kind": kind, "n": _log_uniform(rng, 500, 12011), "L": rng.choice([1000, 3001, 5000]),
                    "law": "founders", "tau": rng.choice([0, 0, 16])}
        n = _log_uniform(rng, 50, 63005)
        return {"kind": kind, "n": n, "L": L if n < 30000 else min(L, 1142), "law": law,
                "tau": rng.choice([0, 0, 0, 64])}
    if kind == "run_calls":
        return {"kind": kind, "n": _log_uniform(rng, 60, 10007), "L": L, "law": law,
                "stripe": rng.choice([512, 512, 2048])}
    if kind == "run_bits":
        return {"kind": kind, "n": _log_uniform(rng, 60, 12001), "L": min(L, 1343), "law": law,
                "tau": rng.choice([64, 256]), "stripe": rng.choice([512, 4096])}
    if kind == "query":
        n = _log_uniform(rng, 2000, 200000)
        m = _log_uniform(rng, 1, min(1500, 200000 * 701 // n))
        return {"kind": kind, "n": n, "L": min(L, 1142) if n > 60000 else L, "m": m, "law": law}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(8, 48), "low": 50, "high": rng.choice([1000, 3000, 5000]),
                "shapes": rng.randrange(1000)}
    if kind == "mst":
        return {"kind": kind, "n": _log_uniform(rng, 100, 30011), "L": L, "law": law}
    if kind == "neighbors":
        return {"kind": kind, "n": _log_uniform(rng, 100, 40009), "L": L, "law": law, "k": rng.choice([1, 5, 10, 32])}
    return {"kind": "table", "n": _log_uniform(rng, 60, 4001), "L": min(L, 1343), "law": law}


def _batch_sets(case):
    """(n, L) of every set: sizes log-uniform, fixed by the case."""
    rng = np.random.default_rng(case["shapes"])
    lo, hi = math.log(case["low"]), math.log(case["high"])
    return [(int(round(math.exp(rng.uniform(lo, hi)))), int(rng.choice(LOCI))) for _ in range(case["count"])]


def _table_text(x, ids):
    """The profiles as the tool's input table: header, then id and calls per line ("-" for missing)."""
    n, L = x.shape
    v = x.clone()
    v[v < 0] = 1
    width = len(str(int(v.max())))
    cells = torch.zeros((n, L, width + 1), dtype=torch.uint8, device=DEV)
    cells[:, :, 0] = 9  # tab
    rest = v.clone()
    for p in range(width, 0, -1):
        digit = (48 + rest % 10).to(torch.uint8)
        cells[:, :, p] = torch.where((rest > 0) | (p == width), digit, 0)
        rest //= 10
    cells[:, :, width] = torch.where(v == 0, 45, cells[:, :, width])
    rows, lens = cells.reshape(n, -1), (cells != 0).reshape(n, -1).sum(1).cpu().numpy()
    flat = rows[rows != 0].cpu().numpy().tobytes()
    parts, at = ["FILE".encode() + b"".join(b"\tL%d" % k for k in range(L))], 0
    for i in range(n):
        parts.append(ids[i].encode() + flat[at:at + int(lens[i])])
        at += int(lens[i])
    return b"\n".join(parts) + b"\n"


def _full_matrix(case, seed):
    """The full symmetric matrix in device memory, n x up(n, 8)."""
    n = case["n"]
    H = torch.zeros((n, _up8(n)), dtype=torch.int16, device=DEV)
    with tch.Solver.from_calls(_host(_profiles(n, case["L"], case["law"], seed))) as s:
        s.stripe(0, n, H.data_ptr(), H.stride(0), _stream())
        s.check()
    for a in range(0, n, 4096):
        b = min(n, a + 4096)
        H[a:b, a:b].triu_(1)
        H[a:b, a:b] += H[a:b, a:b].t().clone()
        if b < n:
            H[b:n, a:b] = H[a:b, b:n].t()
    return H


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sets = _batch_sets(case)
        batch = tch.Batch([_host(_profiles(n, L, "uneven", seed + 7919 * q)) for q, (n, L) in enumerate(sets)])
        off, ld = batch.layout()
        out = torch.zeros(int(off[-1]), dtype=torch.int16, device=DEV)
        keep = torch.zeros_like(out)  # 1 at the cells i < j < n
        for (n, _), o, w in zip(sets, off, ld):
            keep[int(o):int(o) + n * int(w)].view(n, int(w))[:, :n].copy_(
                torch.ones((n, n), dtype=torch.int16, device=DEV).triu_(1))
        batch.tune(out.data_ptr(), _stream())
        return {"kind": kind, "batch": batch, "out": out, "keep": keep}
    n, L = case["n"], case["L"]
    if kind in ("mst", "neighbors"):
        return {"kind": kind, "H": _full_matrix(case, seed), "n": n, "k": case.get("k")}
    if kind == "query":
        x = _profiles(n + case["m"], L, case["law"], seed)
        m = case["m"]
        return {"kind": kind, "db": tch.Database(_host(x[:n])), "q": _host(x[n:]),
                "out": tch.pinned_empty((m, n)), "qq": tch.pinned_empty((m, m)),
                "keep": np.triu(np.ones((m, m), np.uint16), 1)}
    x = _profiles(n, L, case["law"], seed)
    if kind == "table":
        ids = ["isolate_%06d" % i for i in range(n)]
        room = n * (5 * n + 20) + 20 * (n + 2)  # four digits and a separator per distance, ids, header
        return {"kind": kind, "text": _table_text(x, ids), "ids": ids, "out": np.zeros(room, np.uint8)}
    calls = _host(x)
    if kind == "triangle":
        return {"kind": kind, "solver": tch.Solver.from_calls(calls, tau=case["tau"]), "n": n,
                "H": torch.zeros((n, _up8(n)), dtype=torch.int16, device=DEV)}
    sink = _HostMatrix(n, case["stripe"])
    if kind == "run_calls":
        return {"kind": kind, "calls": calls, "stripe": case["stripe"], "sink": sink}
    ranks, distinct = tch.dense_ranks(calls)
    return {"kind": kind, "enc": tch.encode_host(ranks, distinct, tau=case["tau"]), "stripe": case["stripe"],
            "sink": sink}


def run(state):
    kind = state["kind"]
    if kind == "triangle":
        H = state["H"]
        state["solver"].stripe(0, state["n"], H.data_ptr(), H.stride(0), _stream())
        return _triangle(H, state["n"])
    if kind == "run_calls":
        return tch.run_calls(state["calls"], stripe=state["stripe"], sink=state["sink"])[0].view(np.int16)
    if kind == "run_bits":
        return tch.run(state["enc"], stripe=state["stripe"], sink=state["sink"])[0].view(np.int16)
    if kind == "query":
        qdb, qq = state["db"].query(state["q"], out=state["out"], out_qq=state["qq"], stream=_stream())
        return [qdb.view(np.int16), (qq * state["keep"]).view(np.int16)]
    if kind == "batch":
        state["batch"].run(state["out"].data_ptr(), _stream())
        return state["out"] * state["keep"]
    if kind == "mst":
        H = state["H"]
        return list(tch.mst_device(H.data_ptr(), H.stride(0), state["n"], _stream()))
    if kind == "neighbors":
        H = state["H"]
        return list(tch.neighbors_device(H.data_ptr(), H.stride(0), state["n"], state["k"], _stream()))
    out, at = state["out"], 0

    def keep(chunk):
        nonlocal at
        out[at:at + len(chunk)] = np.frombuffer(chunk, np.uint8)
        at += len(chunk)

    with tch.Tsv(state["text"]) as t:
        with t.solver() as s:
            s.write_tsv(state["ids"], sink=keep)
    return [out, at]


def work(case):
    """Profiles read once as two-byte ranks (eight-byte ids where the call takes
    them), distances written once; one compare and one add per pair and locus."""
    kind = case["kind"]
    if kind == "batch":
        sets = _batch_sets(case)
        return {"bytes": sum(2 * n * L + n * (n - 1) for n, L in sets), "flops": sum(n * (n - 1) * L for n, L in sets)}
    n, L = case["n"], case["L"]
    pairs = n * (n - 1) / 2
    if kind == "triangle":
        return {"bytes": 2 * n * L + 2 * pairs, "flops": 2 * pairs * L}
    if kind in ("run_calls", "run_bits"):
        return {"bytes": (8 if kind == "run_calls" else 2) * n * L + 2 * pairs, "flops": 2 * pairs * L}
    if kind == "query":
        m = case["m"]
        return {"bytes": 2 * n * L + 8 * m * L + 2 * m * n + m * (m - 1), "flops": 2 * (m * n + m * (m - 1) / 2) * L}
    if kind == "mst":
        return {"bytes": 2 * n * n + 10 * n, "flops": n * n}
    if kind == "neighbors":
        return {"bytes": 2 * n * n + 6 * n * case["k"], "flops": n * n}
    return {"bytes": 10 * n * L + 4 * n * n, "flops": 2 * pairs * L}


def _count(x, y):
    """Distances of every row of x to every row of y, counted locus by locus."""
    d = torch.zeros((x.shape[0], y.shape[0]), dtype=torch.int64, device=DEV)
    for k in range(x.shape[1]):
        a, b = x[:, k, None], y[None, :, k]
        d += (a != b) & (a != 0) & (b != 0)
    return d


def exact(case, seed):
    """Distances by direct count; None for the other
    results and for sets that would take too long."""
    kind = case["kind"]
    if kind not in ("triangle", "run_calls", "run_bits", "query"):
        return None
    n, L, m = case["n"], case["L"], case.get("m", case["n"])
    if n * m * L > 6e9:
        return None
    if kind == "query":
        x = _profiles(n + m, L, case["law"], seed)
        return [_count(x[n:], x[:n]), torch.triu(_count(x[n:], x[n:]), 1)]
    x = _profiles(n, L, case["law"], seed)
    H = _count(x, x)
    return _triangle(H, n) if kind == "triangle" else torch.triu(H, 1)
