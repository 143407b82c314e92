// Dense rare counts of a stripe, built on the device from the rare groups.
//
// The rare term R[i, j] = #{loci k : x[i,k] == x[j,k] != 0 and that allele is
// rare} (the reference applies it pair by pair from the host-built lists,
// tensorcore/rs/src/main.rs:416-447 and tensorcore/rs/cuda/tch.cu:31-38).
// Here the encoder keeps every rare allele as a group of rows (ascending)
// plus each row's own place in its groups; row i's partners at locus k are
// the group members after its own entry.  Per stripe this kernel counts them
// into a u16 block laid out like the output, which the tensor-core epilogue
// subtracts with 16-byte loads: no pair list is ever materialised.
//
// A CTA per stripe row (persistent over the rows).  The counters of the row's
// columns sit in shared memory as u16 pairs (65 536 columns per pass), each
// partner adds 1 with a shared atomic, and the finished row is written out with
// coalesced 16-byte stores.  Triangle solves read the rows' partner runs as the
// encoder laid them out (rare_runs_kernel); where there are none (stripes wider
// than one pass) or the groups are too crowded for them (launch_rare_dense), the
// runs of two loci per thread are found at a time, laid end to end by a block-wide
// scan of their lengths and cut into equal parts, one per warp (rare_dense_kernel).
//
// What bounds rare_runs_kernel: the shared atomics.  Random columns put 3.4
// lanes of a warp on one bank, so an atomic takes 3.4 of the L1's data cycles,
// and with the member loads and the run cursor those are 75-79 % busy (ncu,
// 12 011 x 5 000 founders); at the margin it counts 2.0e12 pairs/s, of 6.7 per
// cycle and SM.  63 005 x 1 142 long-tail, tau 1 024 (3.4e9 pairs): 2.69 ms,
// 4.72 before, when each member went through the run cursor by itself and one
// 1 024-thread CTA per SM took every row; 0.6 ms of it is the 4 GB block.

#include <climits>
#include <cstdlib>

#include "rare_walk.cuh"
#include "tch_internal.cuh"

namespace tch {
namespace {

#ifndef TCH_RARE_NARROW_T
#define TCH_RARE_NARROW_T 128
#endif
constexpr int NT = TCH_RARE_NARROW_T;      // threads per CTA of the narrow-row kernels (one row each)
constexpr int RD_WORDS = 32768;          // u32 counter words in shared memory (128 KB): 65 536 columns per pass

// Counter words a launch needs (a narrow stripe takes less shared memory, so
// more CTAs fit on an SM when several solves run side by side).
inline int counter_words(size_t width) { return (int)std::min<size_t>(RD_WORDS, width / 2); }
template <int T>
inline int rd_smem(int cwords) { return cwords * 4 + (2 * T + 1) * 4 + 2 * T * 4 + 64 * 4; }
// Runs of a row staged at a time by the row-run kernels.
template <int T>
constexpr int kCap = T >= 256 ? 2 * T : 512;
constexpr int kMinCap = 512;
template <int T>
constexpr int runs_smem(int cwords, int cap = kCap<T>) { return cwords * 4 + (2 * cap + 2 + 64) * 4; }
constexpr unsigned FULL = 0xFFFFFFFFu;

__device__ __forceinline__ uint64_t lower_bound_m(const uint32_t* __restrict__ m, uint64_t lo, uint64_t hi,
                                                  uint32_t key) {
    while (lo < hi) {
        const uint64_t mid = lo + (hi - lo) / 2;
        if (__ldg(m + mid) < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Partner run of row i at locus k inside columns [jlo, jhi): members[lo, lo +
// len).  a = x[i, k], mp = mpos[i, k], coff = cnt_off[k], loaded by the caller.
__device__ __forceinline__ uint32_t partner_run(const RareGroups& g, int i, uint32_t a, uint32_t mp, uint64_t coff,
                                                uint32_t jlo, uint32_t jhi, uint32_t* lo_out) {
    if (!a || mp == kNoGroup) return 0;  // missing, or in no rare group: no lookup at all
    const uint64_t g1 = __ldg(g.goff + coff + a + 1);
    uint64_t b = (uint64_t)mp + 1, e = g1;  // empty when i is the group's last member
    if (b >= e) return 0;
    // members after i's own entry are > i; clip to the pass's columns (only a
    // pass that starts after i + 1 or ends before n needs it)
    if (jlo > (uint32_t)i + 1 && b < e && __ldg(g.members + b) < jlo) b = lower_bound_m(g.members, b, e, jlo);
    if (jhi < (uint32_t)g.n && b < e && __ldg(g.members + e - 1) >= jhi) e = lower_bound_m(g.members, b, e, jhi);
    *lo_out = (uint32_t)b;
    return (uint32_t)(e - b);
}

// This thread's two loci of a row: ranks and own positions.
struct CellPair {
    uint32_t a0 = 0, a1 = 0, m0 = 0, m1 = 0;
};

__device__ __forceinline__ CellPair load_cells(const RareGroups& g, int i, int k0) {
    CellPair c;
    const size_t base = (size_t)i * g.L + k0;
    if (k0 < g.L) {
        c.a0 = g.x[base];
        c.m0 = g.mpos[base];
    }
    if (k0 + 1 < g.L) {
        c.a1 = g.x[base + 1];
        c.m1 = g.mpos[base + 1];
    }
    return c;
}

// A part whose runs hold this many items on average is walked run by run
// (measured on the long-tail profiles: 256 beats 0, 64, 1024 and never).
constexpr uint32_t kWalkMin = 256;

__device__ __forceinline__ void count_col(uint32_t* cnt, uint32_t c) {
    atomicAdd(cnt + (c >> 1), 1u << ((c & 1u) * 16u));
}

// Items [e_begin, e_end) of runs laid end to end (run q: items pre[q] ..
// pre[q + 1] - 1, members run[q] ..; pre[nr] bounds the last one), counted at
// column j - wb by one warp.  A part of long runs (kWalkMin items or more on
// average) is walked run by run, the lanes on consecutive members; otherwise
// 256 items at a time, lane l on items e + l + 32 u, several short runs in one
// pass, each lane keeping its current run (start, end, first member) in
// registers.
__device__ __forceinline__ void walk_part(uint32_t* cnt, const uint32_t* pre, const uint32_t* run, int nr,
                                          uint32_t e_begin, uint32_t e_end, const uint32_t* __restrict__ members,
                                          int wb, int lane) {
    if (e_begin >= e_end) return;
    int p = 0;  // the run holding e_begin: the last p with pre[p] <= e_begin
    {
        int hi = nr;
        while (hi - p > 1) {
            const int m = (p + hi) >> 1;
            if (pre[m] <= e_begin) p = m; else hi = m;
        }
    }
    // long runs on average: walk run by run, the lanes on consecutive members
    // with no per-item bookkeeping
    int pe = p;  // the run holding e_end - 1
    {
        int hi = nr;
        while (hi - pe > 1) {
            const int m = (pe + hi) >> 1;
            if (pre[m] <= e_end - 1) pe = m; else hi = m;
        }
    }
    if ((e_end - e_begin) >= kWalkMin * (uint32_t)(pe - p + 1)) {
        uint32_t e = e_begin;
        for (int q = p; e < e_end; q++) {
            const uint32_t stop = min(pre[q + 1], e_end);
            const uint32_t* src = members + run[q] + (e - pre[q]);
            const uint32_t c = stop - e;
            uint32_t k = (uint32_t)lane;
            for (; k + 224 < c; k += 256) {  // eight loads in flight per lane
                uint32_t jj[8];
#pragma unroll
                for (int u = 0; u < 8; u++) jj[u] = __ldg(src + k + 32 * u);
#pragma unroll
                for (int u = 0; u < 8; u++) count_col(cnt, jj[u] - (uint32_t)wb);
            }
            if (k + 96 < c) {
                uint32_t jj[4];
#pragma unroll
                for (int u = 0; u < 4; u++) jj[u] = __ldg(src + k + 32 * u);
#pragma unroll
                for (int u = 0; u < 4; u++) count_col(cnt, jj[u] - (uint32_t)wb);
                k += 128;
            }
            for (; k < c; k += 32) count_col(cnt, __ldg(src + k) - (uint32_t)wb);
            e = stop;
        }
        return;
    }
    uint32_t a = pre[p], b = pre[p + 1], r = run[p];  // this lane's current run
    uint32_t e0 = e_begin;
    for (; e0 + 256 <= e_end; e0 += 256) {  // whole batches: no bounds checks
        uint32_t j[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const uint32_t e = e0 + (uint32_t)(u * 32 + lane);
            while (e >= b) {  // next run (pre[nr] = total > e bounds it)
                ++p;
                a = b;
                b = pre[p + 1];
                r = run[p];
            }
            j[u] = __ldg(members + r + (e - a));
        }
#pragma unroll
        for (int u = 0; u < 8; u++) count_col(cnt, j[u] - (uint32_t)wb);
    }
    for (; e0 < e_end; e0 += 256) {  // the last, partial batch
        uint32_t idx[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const uint32_t e = e0 + (uint32_t)(u * 32 + lane);
            idx[u] = 0xFFFFFFFFu;
            if (e < e_end) {
                while (e >= b) {  // next run (pre[nr] = total > e bounds it)
                    ++p;
                    a = b;
                    b = pre[p + 1];
                    r = run[p];
                }
                idx[u] = r + (e - a);
            }
        }
        uint32_t j[8];
#pragma unroll
        for (int u = 0; u < 8; u++) j[u] = idx[u] != 0xFFFFFFFFu ? __ldg(members + idx[u]) : 0u;
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (idx[u] != 0xFFFFFFFFu) count_col(cnt, j[u] - (uint32_t)wb);
    }
}

// Lays this thread's two runs (l0 partners from members[lo0], l1 from
// members[lo1]) end to end with every other thread's non-empty runs (a block
// scan of item and run counts compacts them), cuts the items into one equal
// part per warp, and counts every partner j at column j - wb (walk_part).
// Called by all threads of the CTA (it synchronises them).
template <int T>
__device__ __forceinline__ void count_runs(uint32_t* cnt, uint32_t* pre, uint32_t* run, uint32_t* wsum, uint32_t l0,
                                           uint32_t lo0, uint32_t l1, uint32_t lo1,
                                           const uint32_t* __restrict__ members, int wb) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NWARPS = T / 32;
    __shared__ uint32_t tot[2];  // items, runs
    const uint32_t mi = l0 + l1, mc = (l0 ? 1u : 0u) + (l1 ? 1u : 0u);
    uint32_t ii = mi, ic = mc;  // inclusive warp scans of items and runs
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t ti = __shfl_up_sync(FULL, ii, d), tc = __shfl_up_sync(FULL, ic, d);
        if (lane >= d) ii += ti, ic += tc;
    }
    if (lane == 31) wsum[warp] = ii, wsum[32 + warp] = ic;
    __syncthreads();  // also orders the counter zeroing and the previous chunk's readers
    if (warp == 0) {
        const uint32_t vi = lane < NWARPS ? wsum[lane] : 0u, vc = lane < NWARPS ? wsum[32 + lane] : 0u;
        uint32_t xi = vi, xc = vc;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t ti = __shfl_up_sync(FULL, xi, d), tc = __shfl_up_sync(FULL, xc, d);
            if (lane >= d) xi += ti, xc += tc;
        }
        if (lane < NWARPS) wsum[lane] = xi - vi, wsum[32 + lane] = xc - vc;
        if (lane == 31) tot[0] = xi, tot[1] = xc;
    }
    __syncthreads();
    {
        const uint32_t ei = wsum[warp] + ii - mi;        // items before this thread's runs
        uint32_t q = wsum[32 + warp] + ic - mc;          // their places among the non-empty runs
        if (l0) pre[q] = ei, run[q] = lo0, q++;
        if (l1) pre[q] = ei + l0, run[q] = lo1;
        if (tid == 0) pre[tot[1]] = tot[0];
    }
    __syncthreads();
    const uint32_t total = tot[0];
    const uint32_t part = (total + NWARPS - 1) / NWARPS;
    const uint32_t e_begin = min(total, (uint32_t)warp * part), e_end = min(total, e_begin + part);
    walk_part(cnt, pre, run, (int)tot[1], e_begin, e_end, members, wb, lane);
}

// Copies runs [c0, c0 + cn) of the row whose runs are [q0, q1) into `run`, and
// the piece after the last of them into run[cn].x.
template <int T>
__device__ __forceinline__ void stage_runs(const RareGroups& g, int i, uint64_t q0, uint64_t q1, uint32_t c0,
                                           uint32_t cap, uint2* run) {
    const uint32_t nrun = (uint32_t)(q1 - q0), cn = min(cap, nrun - c0);
    for (uint32_t t = threadIdx.x; t < cn; t += T) {
        run[t] = make_uint2(__ldg(g.rpre + q0 + c0 + t), __ldg(g.rlo + q0 + c0 + t));
    }
    if (threadIdx.x == 0)
        run[cn] = make_uint2(c0 + cn < nrun ? __ldg(g.rpre + q0 + c0 + cn) : __ldg(g.rtot + i), 0u);
}

// Counts every run of row i; the first `cap` of them are staged and visible to
// all threads.  Called by all threads of the CTA.
template <int T, class M>
__device__ __forceinline__ void count_staged_row(const Counters& c, uint2* run, const RareGroups& g, const M* members, int i, uint64_t q0, uint64_t q1, uint32_t cap) {
    constexpr int NWARPS = T / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nrun = (uint32_t)(q1 - q0);
    for (uint32_t c0 = 0; c0 < nrun; c0 += cap) {
        if (c0) {
            __syncthreads();  // the previous runs' readers
            stage_runs<T>(g, i, q0, q1, c0, cap, run);
            __syncthreads();
        }
        const uint32_t cn = min(cap, nrun - c0);
        const uint32_t first = run[0].x >> 3, total = (run[cn].x >> 3) - first;
        const uint32_t part = (total + NWARPS - 1) / NWARPS;
        const uint32_t e_begin = first + min(total, (uint32_t)warp * part);
        const uint32_t e_end = first + min(total, (uint32_t)warp * part + part);
        walk_pieces<M>(c, run, (int)cn, e_begin, e_end, members, lane);
    }
}

// Rows [row_begin, row_end) of a stripe whose rows have precomputed runs, each in
// one pass of the counters: `cwords` of them hold row_begin's width, the widest.
// Persistent over the rows: the finished row is written out and its counters
// cleared in one sweep, which also stages the next row's runs.
template <int T, class M>
__global__ void __launch_bounds__(T, T >= 1024 ? 1 : 1536 / T)
    rare_runs_kernel(const RareGroups g, int r0, int row_begin, int row_end, uint16_t* __restrict__ R, size_t ldr,
                     int cend, int cwords, int cap) {
    extern __shared__ uint4 smem_rd[];
    uint32_t* cnt = reinterpret_cast<uint32_t*>(smem_rd);
    uint2* run = reinterpret_cast<uint2*>(cnt + cwords);  // cap + 1
    grid_release();
    const M* members = sizeof(M) == 2 ? reinterpret_cast<const M*>(g.members16) : reinterpret_cast<const M*>(g.members);
    const int tid = threadIdx.x;
    int r = row_begin + (int)blockIdx.x;
    for (int w = tid; w < cwords / 4; w += T) smem_rd[w] = make_uint4(0, 0, 0, 0);
    uint64_t q0 = g.roff[r0 + r], q1 = g.roff[r0 + r + 1];
    if (q1 > q0) stage_runs<T>(g, r0 + r, q0, q1, 0, cap, run);
    for (;;) {
        const int next = r + (int)gridDim.x;
        uint64_t n0 = 0, n1 = 0;
        if (next < row_end) n0 = g.roff[r0 + next], n1 = g.roff[r0 + next + 1];
        __syncthreads();  // counters zero, runs staged
        const int cbeg = r0 + (r & ~(kRareDenseAlign - 1));  // first column of the row's diagonal tile
        count_staged_row<T, M>(counters_at(cnt, cbeg), run, g, members, r0 + r, q0, q1, (uint32_t)cap);
        __syncthreads();  // row counted
        if (n1 > n0) stage_runs<T>(g, r0 + next, n0, n1, 0, cap, run);
        uint4* dst = reinterpret_cast<uint4*>(R + (size_t)r * ldr + (size_t)(cbeg - r0));
        const int nq = (cend - cbeg) >> 3;
        const bool more = next < row_end;
        for (int w = tid; w < nq; w += T) {
            dst[w] = smem_rd[w];
            if (more) smem_rd[w] = make_uint4(0, 0, 0, 0);
        }
        if (!more) break;
        r = next;
        q0 = n0;
        q1 = n1;
    }
    grid_wait();  // a band does not complete before the one launched ahead of it
}

// Many sets' whole triangles in one launch (batched solves): the rows of
// every job laid end to end (row_job: the job of every row), one CTA per row
// as in rare_runs_kernel, each row counted in one pass (the launcher checks
// that every job's width fits the counters).
struct RareJob {
    RareGroups g;
    uint16_t* R;
    size_t ldr;
    int cend;  // up(n, 256): the job's stripe is its whole triangle (r0 = 0)
    int row0;  // the job's first row in the launch
};

template <int T>
__global__ void __launch_bounds__(T, 1536 / T)
    rare_batch_kernel(const RareJob* __restrict__ jobs, const int* __restrict__ row_job, int total_rows,
                      int cwords) {
    extern __shared__ uint4 smem_rd[];
    uint32_t* cnt = reinterpret_cast<uint32_t*>(smem_rd);
    uint32_t* wsum = cnt + cwords;          // 64: per-warp totals of the scans
    uint2* runs = reinterpret_cast<uint2*>(wsum + 64);   // kCap<T> + 1 staged row runs, or
    uint32_t* run = wsum + 64;              // kCap<T>: first member of each run found per locus
    uint32_t* pre = run + kCap<T>;          // kCap<T> + 1: exclusive prefix of the run lengths
    const int tid = threadIdx.x;
    grid_release();
    for (int gr = blockIdx.x; gr < total_rows; gr += gridDim.x) {
        const RareJob& jb = jobs[__ldg(row_job + gr)];
        const RareGroups g = jb.g;
        const int i = gr - jb.row0;
        const int n = g.n, L = g.L;
        const int cbeg = i & ~(kRareDenseAlign - 1);  // first column of the row's diagonal tile
        const int nq = (jb.cend - cbeg) >> 3;
        for (int w = tid; w < nq; w += T) smem_rd[w] = make_uint4(0, 0, 0, 0);
        const uint32_t jlo = (uint32_t)(i + 1), jhi = (uint32_t)n;
        if (g.members16) {  // the row's precomputed runs
            const uint64_t q0 = g.roff[i], q1 = g.roff[i + 1];
            if (q1 > q0) stage_runs<T>(g, i, q0, q1, 0, kCap<T>, runs);
            __syncthreads();
            count_staged_row<T, uint16_t>(counters_at(cnt, cbeg), runs, g, g.members16, i, q0, q1, kCap<T>);
        } else {
            for (int kc = 0; jlo < jhi && kc < L; kc += (2 * T)) {
                const int k0 = kc + 2 * tid;
                uint32_t lo0 = 0, lo1 = 0, l0 = 0, l1 = 0;
                const CellPair c = load_cells(g, i, k0);
                if (k0 < L) l0 = partner_run(g, i, c.a0, c.m0, g.cnt_off[k0], jlo, jhi, &lo0);
                if (k0 + 1 < L) l1 = partner_run(g, i, c.a1, c.m1, g.cnt_off[k0 + 1], jlo, jhi, &lo1);
                count_runs<T>(cnt, pre, run, wsum, l0, lo0, l1, lo1, g.members, cbeg);
            }
        }
        __syncthreads();
        uint4* dst = reinterpret_cast<uint4*>(jb.R + (size_t)i * jb.ldr + (size_t)cbeg);
        for (int w = tid; w < nq; w += T) dst[w] = smem_rd[w];
        __syncthreads();
    }
}

template <int T>
__global__ void __launch_bounds__(T, 1024 / T)
    rare_dense_kernel(const RareGroups g, int r0, int rows, uint16_t* __restrict__ R, size_t ldr, int cend,
                      int cwords) {
    extern __shared__ uint4 smem_rd[];
    uint32_t* cnt = reinterpret_cast<uint32_t*>(smem_rd);
    uint32_t* pre = cnt + cwords;          // 2T + 1: exclusive prefix of the run lengths
    uint32_t* run = pre + (2 * T) + 1;     // 2T: first member index of each run
    uint32_t* wsum = run + (2 * T);        // 64: per-warp totals of the scans
    const int tid = threadIdx.x;
    const int n = g.n, L = g.L;
    grid_release();
    // with every locus in one scan (L <= 2T) a thread keeps the same two
    // loci for all rows: their count offsets stay in registers and the next
    // row's ranks and positions are fetched while this row is counted
    const bool one_chunk = L <= (2 * T);
    uint64_t co0 = 0, co1 = 0;
    if (one_chunk) {
        if (2 * tid < L) co0 = g.cnt_off[2 * tid];
        if (2 * tid + 1 < L) co1 = g.cnt_off[2 * tid + 1];
    }
    CellPair next;
    if (one_chunk && (int)blockIdx.x < rows) next = load_cells(g, r0 + (int)blockIdx.x, 2 * tid);
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const int i = r0 + r;
        const CellPair cur = next;
        if (one_chunk && r + (int)gridDim.x < rows) next = load_cells(g, i + (int)gridDim.x, 2 * tid);
        const int cbeg = r0 + (r & ~(kRareDenseAlign - 1));  // first column of the row's diagonal tile
        uint4* Rrow = reinterpret_cast<uint4*>(R + (size_t)r * ldr + (size_t)(cbeg - r0));
        for (int wb = cbeg; wb < cend; wb += 2 * cwords) {
            const int we = min(cend, wb + 2 * cwords);
            const int nq = (we - wb) >> 3;  // uint4 of counters (8 columns each); we - wb is a multiple of 256
            for (int w = tid; w < nq; w += T) smem_rd[w] = make_uint4(0, 0, 0, 0);
            const uint32_t jlo = (uint32_t)max(wb, i + 1), jhi = (uint32_t)min(we, n);
            for (int kc = 0; jlo < jhi && kc < L; kc += (2 * T)) {
                // this thread's two loci, then a block-wide exclusive scan of the run lengths
                const int k0 = kc + 2 * tid;
                uint32_t lo0 = 0, lo1 = 0, l0 = 0, l1 = 0;
                if (one_chunk) {
                    l0 = partner_run(g, i, cur.a0, cur.m0, co0, jlo, jhi, &lo0);
                    l1 = partner_run(g, i, cur.a1, cur.m1, co1, jlo, jhi, &lo1);
                } else {
                    const CellPair c = load_cells(g, i, k0);
                    if (k0 < L) l0 = partner_run(g, i, c.a0, c.m0, g.cnt_off[k0], jlo, jhi, &lo0);
                    if (k0 + 1 < L) l1 = partner_run(g, i, c.a1, c.m1, g.cnt_off[k0 + 1], jlo, jhi, &lo1);
                }
                count_runs<T>(cnt, pre, run, wsum, l0, lo0, l1, lo1, g.members, wb);
            }
            __syncthreads();
            uint4* dst = Rrow + ((wb - cbeg) >> 3);
            for (int w = tid; w < nq; w += T) dst[w] = smem_rd[w];
            __syncthreads();
        }
    }
}

// Rare counts of m new profiles against every row of the set:
// R[r * ldr + j] = loci where new profile r and row j share an allele that is
// rare in the set, for j < n (0 up to cend).  One CTA per profile and window of
// kQueryWindow columns.  A new profile's partners at a locus are a whole group,
// and the encoder laid down where each group enters each window, so a run costs
// two neighbouring loads; a warp takes 32 loci, lays their runs end to end and
// walks them by pieces, with no step that waits for another warp but the
// clearing and the write-out.
//
// Bound by the chains of dependent loads (rank, window entry, members), which
// the windows' CTAs overlap: five of them on an SM.  701 profiles against 200 000
// x 1 142 (tau 4 096): 0.35 ms; one CTA per profile with four passes of 65 536
// columns, two binary searches per locus in each, took 0.67.
// Databases without the window entries (they did not fit) keep the members in four
// bytes, and a run's ends are found by binary search (WINDOWS false): 64 profiles
// against 20 000 x 3 016 and 200 000 x 1 142 take 0.304 and 0.500 ms in the call,
// with the entries 0.230 and 0.437.
constexpr int QT = 256;
template <bool WINDOWS>
__global__ void __launch_bounds__(QT, 5)
    rare_query_kernel(const RareGroups g, const uint32_t* __restrict__ xq, uint16_t* __restrict__ R, size_t ldr,
                      int cend) {
    __shared__ uint4 counters[kQueryWindow / 8];
    __shared__ uint2 runs[QT / 32][33];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    grid_release();
    const int w = blockIdx.x, r = blockIdx.y;
    const int wb = w * kQueryWindow, nq = (min(cend, wb + kQueryWindow) - wb) >> 3;
    for (int q = tid; q < nq; q += QT) counters[q] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const Counters c = WINDOWS ? window_counters(counters) : counters_at(counters, wb);
    constexpr uint32_t G = WINDOWS ? kPiece<uint16_t> : kPiece<uint32_t>;
    uint2* run = runs[warp];
    for (int k0 = 32 * warp; k0 < g.L; k0 += QT) {
        const int k = k0 + lane;
        uint32_t lo = 0, hi = 0;
        if (k < g.L) {
            const uint32_t a = __ldg(xq + (size_t)r * g.L + k);
            if (a && a != kNovelRank) {  // empty for an allele that is frequent in the set
                const uint64_t slot = __ldg(g.cnt_off + k) + a;
                if (WINDOWS) {
                    const uint32_t* e = g.wpos + slot * (uint64_t)g.windows + w;
                    lo = __ldg(e);
                    hi = __ldg(e + 1);
                } else {
                    const uint64_t end = __ldg(g.goff + slot + 1);
                    const uint64_t first = lower_bound_m(g.members, __ldg(g.goff + slot), end, (uint32_t)wb);
                    lo = (uint32_t)first;
                    hi = (uint32_t)lower_bound_m(g.members, first, end, (uint32_t)wb + kQueryWindow);
                }
            }
        }
        const uint32_t pieces = hi > lo ? (hi - 1) / G - lo / G + 1 : 0;
        uint32_t inc = pieces;  // inclusive scan
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, inc, d);
            if (lane >= d) inc += t;
        }
        const uint32_t total = __shfl_sync(FULL, inc, 31);
        const unsigned has = __ballot_sync(FULL, pieces > 0);
        __syncwarp();  // the previous runs' readers
        if (pieces) run[__popc(has & ((1u << lane) - 1u))] = make_uint2((inc - pieces) << 3 | ((hi - 1) % G), lo);
        if (lane == 0) run[__popc(has)] = make_uint2(total << 3, 0);
        __syncwarp();
        if (WINDOWS) walk_pieces<uint16_t>(c, run, __popc(has), 0, total, g.members16, lane);
        else walk_pieces<uint32_t>(c, run, __popc(has), 0, total, g.members, lane);
    }
    __syncthreads();
    uint4* dst = reinterpret_cast<uint4*>(R + (size_t)r * ldr + wb);
    for (int q = tid; q < nq; q += QT) dst[q] = counters[q];
}

// The same block from pair lists: one CTA per stripe row (persistent), the
// row's partners read once per counter pass with consecutive threads on
// consecutive entries, each partner in the pass's columns adding 1 with a
// shared atomic.  A partner outside (i, n) is reported and skipped.
__global__ void __launch_bounds__(1024, 1)
    rare_lists_kernel(const uint32_t* __restrict__ start, const uint32_t* __restrict__ js, int n, int r0, int rows,
                      uint16_t* __restrict__ R, size_t ldr, int cend, int cwords, int* err) {
    extern __shared__ uint4 smem_rd[];
    uint32_t* cnt = reinterpret_cast<uint32_t*>(smem_rd);
    const int tid = threadIdx.x;
    grid_release();
    for (int r = blockIdx.x; r < rows; r += gridDim.x) {
        const int i = r0 + r;
        const uint32_t pa = __ldg(start + i), pb = __ldg(start + i + 1);
        const int cbeg = r0 + (r & ~(kRareDenseAlign - 1));  // first column of the row's diagonal tile
        uint4* Rrow = reinterpret_cast<uint4*>(R + (size_t)r * ldr + (size_t)(cbeg - r0));
        for (int wb = cbeg; wb < cend; wb += 2 * cwords) {
            const int we = min(cend, wb + 2 * cwords);
            const int nq = (we - wb) >> 3;
            for (int w = tid; w < nq; w += blockDim.x) smem_rd[w] = make_uint4(0, 0, 0, 0);
            __syncthreads();
            for (uint32_t p = pa + (uint32_t)tid; p < pb; p += blockDim.x) {
                const uint32_t j = __ldg(js + p);
                if (j <= (uint32_t)i || j >= (uint32_t)n) {
                    if (wb == cbeg) atomicOr(err, DEVERR_RARE_PAIR);
                    continue;
                }
                if (j >= (uint32_t)wb && j < (uint32_t)we) count_col(cnt, j - (uint32_t)wb);
            }
            __syncthreads();
            uint4* dst = Rrow + ((wb - cbeg) >> 3);
            for (int w = tid; w < nq; w += blockDim.x) dst[w] = smem_rd[w];
            __syncthreads();
        }
    }
}

}  // namespace

cudaError_t launch_rare_from_lists(const uint32_t* start, const uint32_t* js, int n, int r0, int rows, uint16_t* R,
                                   size_t ldr, int* err, int sms, cudaStream_t st) {
    if (rows <= 0) return cudaSuccess;
    const size_t width = up((size_t)(n - r0), kRareDenseAlign);
    if (ldr < width || (ldr & 7) || ((uintptr_t)R & 15)) return cudaErrorInvalidValue;
    static bool attrs[kMaxDevices] = {};
    bool& attr = attrs[current_device()];
    if (!attr) {
        const cudaError_t e = cudaFuncSetAttribute(rare_lists_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   RD_WORDS * 4);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    const int cwords = counter_words(width);
    rare_lists_kernel<<<std::max(1, std::min(rows, sms)), 1024, cwords * 4, st>>>(start, js, n, r0, rows, R, ldr,
                                                                                 r0 + (int)width, cwords, err);
    return cudaGetLastError();
}

cudaError_t rare_batch_prepare(const std::vector<RareBatchItem>& items, RareBatchPlan* plan) {
    std::vector<RareJob> jobs;
    std::vector<int> row_job;
    int row0 = 0, cwords = 1;
    for (const RareBatchItem& it : items) {
        if (it.g.n < 2) continue;
        const size_t width = up((size_t)it.g.n, kRareDenseAlign);
        if (it.ldr < width || (it.ldr & 7) || ((uintptr_t)it.R & 15)) return cudaErrorInvalidValue;
        if (width > (size_t)2 * RD_WORDS) return cudaErrorInvalidValue;  // one counter pass per row
        RareJob j;
        j.g = it.g;
        j.R = it.R;
        j.ldr = it.ldr;
        j.cend = (int)width;
        j.row0 = row0;
        row0 += it.g.n;
        cwords = std::max(cwords, (int)(width / 2));
        row_job.insert(row_job.end(), (size_t)it.g.n, (int)jobs.size());
        jobs.push_back(j);
    }
    rare_batch_release(plan);
    plan->njobs = (int)jobs.size();
    plan->total_rows = row0;
    plan->cwords = cwords;
    if (jobs.empty()) return cudaSuccess;
    cudaError_t e = device_alloc(&plan->d_jobs, jobs.size() * sizeof(RareJob));
    if (e == cudaSuccess) e = device_alloc(&plan->d_row_job, row_job.size() * sizeof(int));
    if (e == cudaSuccess)
        e = cudaMemcpy(plan->d_jobs, jobs.data(), jobs.size() * sizeof(RareJob), cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(plan->d_row_job, row_job.data(), row_job.size() * sizeof(int), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return e;
    static bool attrs[kMaxDevices] = {};
    bool& attr = attrs[current_device()];
    if (!attr) {
        e = cudaFuncSetAttribute(rare_batch_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 runs_smem<NT>(RD_WORDS));
        if (e != cudaSuccess) return e;
        attr = true;
    }
    return cudaSuccess;
}

cudaError_t launch_rare_batch(const RareBatchPlan& plan, int sms, cudaStream_t st) {
    if (!plan.njobs || !plan.total_rows) return cudaSuccess;
    // one CTA per row, as the per-set launches: rows differ widely in work
    // (the sets' widths and taus), and the block scheduler balances them
    (void)sms;
    const int grid = std::max(1, plan.total_rows);
    rare_batch_kernel<NT><<<grid, NT, runs_smem<NT>(plan.cwords), st>>>(
        static_cast<const RareJob*>(plan.d_jobs), static_cast<const int*>(plan.d_row_job), plan.total_rows,
        plan.cwords);
    return cudaGetLastError();
}

void rare_batch_release(RareBatchPlan* plan) {
    if (plan->d_jobs) cudaFree(plan->d_jobs);
    if (plan->d_row_job) cudaFree(plan->d_row_job);
    plan->d_jobs = plan->d_row_job = nullptr;
    plan->njobs = plan->total_rows = 0;
}

// Shared memory of one CTA when an SM holds `per_sm` of them (1 KB of it is the
// system's).
constexpr int runs_room(int per_sm) { return (227 * 1024) / per_sm - 1024; }

// Narrow rows, in columns: a CTA of NT (128) threads each, so that many rows' chains
// of dependent steps overlap (5 000 profiles, tau 64: 0.039 ms, with 512 threads
// 0.060; from 8 192 columns on the two are alike).
constexpr int kNarrow = 8192;
// TCH_RARE_SMALL_ROWS: only for stripes of fewer rows than this.
static bool narrow_rows(int rows) {
    static const int limit = [] {
        const char* v = getenv("TCH_RARE_SMALL_ROWS");
        return v ? std::max(0, atoi(v)) : INT_MAX;
    }();
    return rows < limit;
}

// One launch of rare_runs_kernel over rows [ra, rb) of the stripe: `per_sm` CTAs
// of T threads on an SM, as many of them as hold the widest row's counters; the
// runs staged at a time take what is left, up to a row's most.
template <int T, class M>
static cudaError_t launch_runs(const RareGroups& g, int r0, int ra, int rb, uint16_t* R, size_t ldr, int cend,
                               int per_sm, bool persistent, int sms, cudaStream_t st) {
    const int cwords = (cend - r0 - (ra & ~(kRareDenseAlign - 1))) / 2;
    while (per_sm > 1 && runs_smem<T>(cwords, kMinCap) > runs_room(per_sm)) per_sm--;
    const int left = (runs_room(per_sm) - runs_smem<T>(cwords, 0)) / 8;
    const int cap = std::max(std::min(left, (int)up((size_t)g.L, 32)), kMinCap);
    const int grid = persistent ? std::min(per_sm * sms, rb - ra) : rb - ra;
    // a band after the first fills the SMs that the one before it leaves
    return launch_after(ra > 0, rare_runs_kernel<T, M>, dim3((unsigned)grid), T, runs_smem<T>(cwords, cap), st, g, r0, ra,
                        rb, R, ldr, cend, cwords, cap);
}

// The stripe's rows in bands of like width, each with as many CTAs per SM as
// its counters leave room for: rows of 63 005 columns take the whole SM, those of
// half the width share it in twos and threes.
template <class M>
static cudaError_t launch_rare_runs(const RareGroups& g, int r0, int rows, uint16_t* R, size_t ldr, int sms,
                                    cudaStream_t st) {
    const int width = (int)up((size_t)(g.n - r0), kRareDenseAlign), cend = r0 + width;
    // widest row that leaves room for two CTAs on an SM
    constexpr int kWide = (runs_room(2) - runs_smem<512>(0, kMinCap)) / 2 / kRareDenseAlign * kRareDenseAlign;
    // sets with more than 32 768 rare pairs per row keep many warps per row busy:
    // 256 threads a row, a CTA each, up to 20 480 columns (10 000 x 1 142, tau 1 024,
    // 91 000 pairs per row: 0.552 ms, with 512 and 128 threads 0.658; 12 011
    // founders: 4.04 and 4.60; wider rows run better on 512: 63 005 profiles 2.69
    // ms, 2.89 when 256 threads take them up to 28 672)
    const bool heavy = g.pairs > (size_t)32768 * g.n;
    constexpr int kHeavyWidth = 20480;
    cudaError_t e = cudaSuccess;
    static bool attrs[kMaxDevices] = {};  // once per device (also keeps it out of graph captures)
    bool& attr = attrs[current_device()];
    if (!attr) {
        const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
        e = cudaFuncSetAttribute(rare_runs_kernel<1024, M>, at, runs_room(1));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(rare_runs_kernel<512, M>, at, runs_room(1));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(rare_runs_kernel<NT, M>, at, runs_room(1));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(rare_runs_kernel<256, M>, at, runs_room(1));
        if (e != cudaSuccess) return e;
        attr = true;
    }
    for (int ra = 0; ra < rows && e == cudaSuccess;) {
        const int w = width - (ra & ~(kRareDenseAlign - 1));
        // the end of the rows from ra on that are wider than `limit` columns
        auto wider = [&](int limit) { return w <= limit ? ra : std::min(rows, width - limit); };
        int rb;
        if ((rb = wider(kWide)) > ra) {
            e = launch_runs<1024, M>(g, r0, ra, rb, R, ldr, cend, 1, true, sms, st);
        } else if ((rb = wider(28672)) > ra) {
            e = launch_runs<512, M>(g, r0, ra, rb, R, ldr, cend, 2, true, sms, st);
        } else if ((rb = wider(heavy ? kHeavyWidth : narrow_rows(rows) ? kNarrow : 0)) > ra) {
            e = launch_runs<512, M>(g, r0, ra, rb, R, ldr, cend, 3, true, sms, st);
        } else {
            rb = rows;
            e = heavy ? launch_runs<256, M>(g, r0, ra, rb, R, ldr, cend, 6, false, sms, st)
                      : launch_runs<NT, M>(g, r0, ra, rb, R, ldr, cend, 8, false, sms, st);
        }
        ra = rb;
    }
    return e;
}

cudaError_t launch_rare_dense(const RareGroups& g, int r0, int rows, uint16_t* R, size_t ldr, int sms,
                              cudaStream_t st) {
    if (rows <= 0) return cudaSuccess;
    const size_t width = up((size_t)(g.n - r0), kRareDenseAlign);
    if (ldr < width || (ldr & 7) || ((uintptr_t)R & 15)) return cudaErrorInvalidValue;
    // Every row's precomputed runs, where the widest row fits one counter pass.  Not
    // with four-byte members in groups so large that a row has more than eight rare
    // pairs per column: lanes on consecutive members of such runs meet fewer banks
    // twice than lanes on pieces of four (70 001 x 200, tau 65 536, 13 pairs per
    // column: the last 8 192 rows 0.48 and 0.59 ms, 20 480 3.35 and 3.48; x 1 142, tau
    // 4 096, 4.7 pairs: 0.36 and 0.29, 1.95 and 1.46).
    const bool crowded = !g.members16 && g.pairs / 8 > (size_t)g.n * g.n;
    if (g.roff && width <= (size_t)2 * RD_WORDS && !crowded)
        return g.members16 ? launch_rare_runs<uint16_t>(g, r0, rows, R, ldr, sms, st)
                           : launch_rare_runs<uint32_t>(g, r0, rows, R, ldr, sms, st);
    static bool attrs[kMaxDevices] = {};  // once per device (also keeps it out of graph captures)
    bool& attr = attrs[current_device()];
    if (!attr) {
        const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
        cudaError_t e = cudaFuncSetAttribute(rare_dense_kernel<1024>, at, rd_smem<1024>(RD_WORDS));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(rare_dense_kernel<NT>, at, rd_smem<NT>(kNarrow / 2));
        if (e != cudaSuccess) return e;
        attr = true;
    }
    const int cwords = counter_words(width);
    if (width <= (size_t)kNarrow && narrow_rows(rows))  // a CTA of 128 threads per row, as in bands of runs
        rare_dense_kernel<NT><<<rows, NT, rd_smem<NT>(cwords), st>>>(g, r0, rows, R, ldr, r0 + (int)width, cwords);
    else
        rare_dense_kernel<1024><<<std::max(1, std::min(rows, sms)), 1024, rd_smem<1024>(cwords), st>>>(
            g, r0, rows, R, ldr, r0 + (int)width, cwords);
    return cudaGetLastError();
}

cudaError_t launch_rare_query(const RareGroups& g, const uint32_t* xq, int m, uint16_t* R, size_t ldr,
                              cudaStream_t st) {
    const size_t width = up((size_t)std::max(g.n, 1), kRareDenseAlign);
    if (ldr < width || (ldr & 7) || ((uintptr_t)R & 15)) return cudaErrorInvalidValue;
    if (g.wpos ? g.windows != query_windows(g.n) || !g.members16 : !g.goff || !g.members) return cudaErrorInvalidValue;
    const auto kernel = g.wpos ? rare_query_kernel<true> : rare_query_kernel<false>;
    for (int r0 = 0; r0 < m; r0 += 65535) {  // the grid's second dimension
        const dim3 grid(query_windows(g.n), std::min(65535, m - r0));
        kernel<<<grid, QT, 0, st>>>(g, xq + (size_t)r0 * g.L, R + (size_t)r0 * ldr, ldr, (int)width);
    }
    return cudaGetLastError();
}

}  // namespace tch
