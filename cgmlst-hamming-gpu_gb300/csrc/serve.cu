// Serving: a profile database resident in HBM and query batches of new
// profiles against it (no reference counterpart; the reference computes one
// matrix per run).
//
// tch_db holds the database encoded on the device (operand rows, rare groups
// including single-row groups, and the maps that encode new profiles like the
// database's own: ids in rank order per locus, frequent column per allele).
// A query batch of m new profiles runs on the caller's stream, allocating only
// from a stream-ordered pool:
//   ranks      each id looked up in its locus's sorted ids (new ids -> novel)
//   operand    packed fp4 rows in the database's column layout (presence +
//              frequent one-hot, the A side of the tile pass; a novel id is
//              present but matches nothing); the database keeps only its
//              B-side copy (one-hot columns negated)
//   rare       u16 counts of rare equal alleles against every database row
//   distances  the tcgen05 tile pass over the m x n rectangle, subtracting them;
//              for a few profiles ranks, rare counts and distances come out of
//              one kernel, from the database's bit columns (query_few_kernel)
//   q x q      the batch's own upper triangle by a direct count on the calls
//              (ids compared as given; 0 = missing)
// Every distance is exact; the database's tau only decides which alleles go
// through the one-hot columns and which through the rare counts.
//
// tch_server runs query batches from many callers: a FIFO of requests, a set
// of worker threads with one stream each (the slots), and admission by device
// memory: a request starts when its estimated bytes fit in the budget next to
// the requests already running, so batches that arrive while others are on the
// GPU overlap with them.

#include <math.h>
#include <string.h>

#include <chrono>
#include <condition_variable>
#include <deque>
#include <map>
#include <mutex>
#include <thread>
#include <type_traits>
#include <vector>

#include <cooperative_groups.h>

#include "rare_walk.cuh"
#include "tch_internal.cuh"

namespace cg = cooperative_groups;

namespace tch {
namespace {

// Distances of one new profile (blockIdx.y) to every row of the database, straight
// from its ids: a row differs at the loci whose bit column (that of the profile's
// allele, DeviceEncoding::bits) has its bit, less those where the two share a rare
// allele.  A cluster of eight CTAs takes one window of kQueryWindow rows:
//   ranks    each CTA looks up an eighth of the ids, four lanes to an id, every
//            step leaving a fifth of the locus's ids, and hands the columns to
//            the other seven;
//   rare     it counts the rare partners that its eighth of the loci has in the
//            window, 16 bytes of members per lane;
//   bits     it adds up all loci's columns for its own 2 048 rows: a warp takes
//            1 024 of them (lane = 32 rows) and a sixteenth of the loci, eight
//            columns at a time through carry-save adders into binary counters
//            held as planes of bits, spread into row counts at the end;
//   out      it adds the eight CTAs' rare counts of its rows and writes.
// Loci go by in chunks of FEW_LOCI.
//
// Bound by chains of dependent loads at one profile (ids, window entries, members,
// columns: each a trip to memory), at several by the columns' read, n / 8 bytes
// per locus.  One profile against 200 000 x 1 142: 28 us with cold caches, the
// whole call 44; three kernels (ranks; rare counts, a CTA per window; columns), one
// after the other with their results in memory, took 60, the call 91.
constexpr int FEW_T = 1024, FEW_CTAS = 8, FEW_ROWS = kQueryWindow / FEW_CTAS, FEW_LOCI = 2048;
constexpr int FEW_PLANES = 13;                       // a warp counts at most 4 096 of 65 535 loci
constexpr int FEW_RUNS = FEW_LOCI / FEW_CTAS / 32;   // loci a warp looks up in a chunk: 8
static_assert(FEW_ROWS == 2 * 1024 && FEW_RUNS * 4 == 32, "two warps' rows and four lanes per locus");
struct FewShared {
    uint4 counters[kQueryWindow / 8];  // rare partners, u16 pairs
    uint32_t count[2][32 * 33];        // row (i & 31) * 33 + (i >> 5) of each half
    uint32_t sel[FEW_LOCI];            // bit column per locus, ~0 for a missing call
    uint2 runs[FEW_T / 32][FEW_RUNS + 1];
};
__device__ __forceinline__ uint32_t carry_add(uint32_t& a, uint32_t b, uint32_t c) {
    const uint32_t carry = (a & b) | (a & c) | (b & c);
    a = a ^ b ^ c;
    return carry;
}
__global__ void __cluster_dims__(FEW_CTAS, 1, 1) __launch_bounds__(FEW_T)
    query_few_kernel(const uint64_t* __restrict__ q, const RareGroups g, const uint64_t* __restrict__ slot_ids,
                     const int32_t* __restrict__ col, const uint32_t* __restrict__ base, uint32_t D,
                     const uint32_t* __restrict__ bits, size_t words, uint16_t* __restrict__ out, size_t ldo) {
    extern __shared__ uint4 few_smem[];
    FewShared& sm = *reinterpret_cast<FewShared*>(few_smem);
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, L = g.L;
    const int rank = (int)cluster.block_rank(), window = blockIdx.x / FEW_CTAS, r = blockIdx.y;
    for (int t = tid; t < kQueryWindow / 8; t += FEW_T) sm.counters[t] = make_uint4(0, 0, 0, 0);
    for (int t = tid; t < 2 * 32 * 33; t += FEW_T) (&sm.count[0][0])[t] = 0;
    const Counters counters = window_counters(sm.counters);
    const int half = warp >> 4, share = warp & 15;
    const size_t word = (size_t)window * (kQueryWindow / 32) + rank * (FEW_ROWS / 32) + half * 32 + lane;
    uint32_t p[FEW_PLANES];
#pragma unroll
    for (int b = 0; b < FEW_PLANES; b++) p[b] = 0;
    for (int c0 = 0; c0 < L; c0 += FEW_LOCI) {
        const int nl = min(FEW_LOCI, L - c0), per = (nl + FEW_CTAS - 1) / FEW_CTAS;
        // the cluster's CTAs run and are done with the last chunk's columns
        cluster.sync();
        {
            const int at = (tid >> 2) + rank * per, k = c0 + at, s = lane & 3;
            const bool mine = (tid >> 2) < per && at < nl;
            const uint64_t v = mine ? __ldg(q + (size_t)r * L + k) : 0;
            uint64_t first = 0, lo = 0, hi = 0;
            if (v) {  // ids of locus k ascend at slots cnt_off[k] + 1 .. cnt_off[k + 1] - 1
                first = __ldg(g.cnt_off + k);
                lo = first + 1;
                hi = __ldg(g.cnt_off + k + 1);
            }
            const uint64_t end = hi;
            while (__any_sync(0xFFFFFFFFu, lo < hi)) {
                const uint64_t len = hi - lo;
                const bool less = lo < hi && __ldg(slot_ids + lo + len * (s + 1) / 5) < v;
                const int below = __popc(__ballot_sync(0xFFFFFFFFu, less) >> (lane & ~3) & 15u);
                if (lo < hi) {
                    if (below < 4) hi = lo + len * (below + 1) / 5;
                    if (below) lo = lo + len * below / 5 + 1;
                }
            }
            const bool known = v && lo < end && __ldg(slot_ids + lo) == v;
            uint32_t e = 0;
            if (known) {  // empty for an allele that is frequent in the set
                if (s < 2) e = __ldg(g.wpos + lo * (uint64_t)g.windows + window + s);
            }
            if (mine) {
                const int32_t c = known ? __ldg(col + lo) : -1;
                const uint32_t m = !v ? ~0u : c >= 0 ? __ldg(base + k) + (uint32_t)c : D + (uint32_t)k;
                cluster.map_shared_rank(sm.sel, 2 * s)[at] = m;
                cluster.map_shared_rank(sm.sel, 2 * s + 1)[at] = m;
            }
            cluster.barrier_arrive();
            // the warp's runs, end to end (lanes 4 q hold run q)
            const uint32_t last = __shfl_sync(0xFFFFFFFFu, e, lane | 1);
            const uint32_t pieces = s == 0 && last > e ? (last - 1) / 8 - e / 8 + 1 : 0;
            uint32_t inc = pieces;
#pragma unroll
            for (int d = 4; d < 32; d <<= 1) {
                const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, d);
                if (lane >= d) inc += t;
            }
            const uint32_t total = __shfl_sync(0xFFFFFFFFu, inc, 28);
            const unsigned has = __ballot_sync(0xFFFFFFFFu, pieces > 0);
            uint2* run = sm.runs[warp];
            if (pieces) run[__popc(has & ((1u << lane) - 1u))] = make_uint2((inc - pieces) << 3 | ((last - 1) & 7u), e);
            if (lane == 0) run[__popc(has)] = make_uint2(total << 3, 0);
            __syncwarp();
            walk_pieces<uint16_t>(counters, run, __popc(has), 0, total, g.members16, lane);
            __syncwarp();
            cluster.barrier_wait();
        }
        if (word < words) {
            const uint32_t* mine = bits + word;
            const int part = ((nl + 15) / 16 + 7) & ~7, k1 = min(nl, (share + 1) * part);
#pragma unroll 2
            for (int k = share * part; k < k1; k += 8) {
                uint32_t x[8];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const uint32_t c = k + e < k1 ? sm.sel[k + e] : ~0u;
                    x[e] = c != ~0u ? __ldg(mine + (size_t)c * words) : 0u;
                }
                const uint32_t a0 = carry_add(p[0], x[0], x[1]), a1 = carry_add(p[0], x[2], x[3]);
                const uint32_t b0 = carry_add(p[1], a0, a1);
                const uint32_t a2 = carry_add(p[0], x[4], x[5]), a3 = carry_add(p[0], x[6], x[7]);
                const uint32_t b1 = carry_add(p[1], a2, a3);
                uint32_t c = carry_add(p[2], b0, b1);
#pragma unroll
                for (int b = 3; b < FEW_PLANES; b++) {
                    const uint32_t t = p[b] & c;
                    p[b] ^= c;
                    c = t;
                }
            }
        }
    }
#pragma unroll 4
    for (int i = 0; i < 32; i++) {
        uint32_t v = 0;
#pragma unroll
        for (int b = 0; b < FEW_PLANES; b++) v |= ((p[b] >> i) & 1u) << b;
        if (v) atomicAdd(&sm.count[half][i * 33 + lane], v);
    }
    cluster.sync();
    {
        uint32_t rare = 0;  // rows 2 tid and 2 tid + 1 of this CTA's; neither half reaches 65 536
#pragma unroll
        for (int c = 0; c < FEW_CTAS; c++)
            rare += reinterpret_cast<const uint32_t*>(cluster.map_shared_rank(sm.counters, c))[rank * (FEW_ROWS / 2) + tid];
        const int i = 2 * tid & 1023, j = window * kQueryWindow + rank * FEW_ROWS + 2 * tid;
        const uint32_t* count = sm.count[tid >> 9] + (i >> 5);
        const uint32_t d0 = count[(i & 31) * 33] - (rare & 0xFFFFu), d1 = count[((i & 31) + 1) * 33] - (rare >> 16);
        if (j < g.n) *reinterpret_cast<uint32_t*>(out + (size_t)r * ldo + j) = (d0 & 0xFFFFu) | d1 << 16;
    }
    cluster.sync();  // no CTA leaves while others read its counters
}

// +1.0 at column col of row `row` (zeroed before); two columns of one byte
// belong to different cells, hence the atomic OR on the word.
__device__ __forceinline__ void set_fp4_one(const KChunks& X, size_t row, size_t col) {
    uint32_t* w = reinterpret_cast<uint32_t*>(X.at(row, (int)((col >> 1) & ~(size_t)3)));
    atomicOr(w, kFp4One << (4 * (col & 7)));
}

// The batch's ranks and operand rows (zeroed before).
__global__ void query_pack_kernel(const uint64_t* __restrict__ q, int m, int L, const uint64_t* __restrict__ cnt_off,
                                  const uint64_t* __restrict__ slot_ids, const int32_t* __restrict__ col,
                                  const uint32_t* __restrict__ base, uint32_t* xq, KChunks X) {
    const size_t total = (size_t)m * L;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t i = t / L;
        const int k = (int)(t % L);
        const uint64_t v = q[t];
        uint32_t r = 0;
        if (v) {
            set_fp4_one(X, i, (size_t)k);
            // ids of locus k ascend at slots cnt_off[k] + 1 .. cnt_off[k + 1] - 1
            const uint64_t first = cnt_off[k], end = cnt_off[k + 1];
            uint64_t lo = first + 1, hi = end;
            while (lo < hi) {
                const uint64_t mid = lo + (hi - lo) / 2;
                if (slot_ids[mid] < v) lo = mid + 1; else hi = mid;
            }
            r = kNovelRank;
            if (lo < end && slot_ids[lo] == v) {
                r = (uint32_t)(lo - first);
                const int32_t c = col[lo];
                if (c >= 0) set_fp4_one(X, i, (size_t)L + base[k] + (size_t)c);
            }
        }
        xq[t] = r;
    }
}

// Direct count of the batch's own pairs (ids compared as given): a cluster of
// eight CTAs per 32 x 32 pairs, each with an eighth of the loci, 64 of them staged
// in shared memory at a time, 2 x 2 pairs per thread.  Two profiles differ at the
// loci where the presence of a call agrees less those where the ids (or the two
// missing calls) are equal: the first by the rows' bit masks, taken as the ids are
// staged, so a pair and locus costs one 64-bit compare.
//
// Bound by the compares for large batches and by the chain of load, barrier and
// count for small ones, which the split of the loci shortens.  40 / 200 / 1 000
// profiles of 1 142 loci: 15 / 23 / 179 us; 16 x 16 pairs per CTA, all loci in one
// CTA and one pair per thread took 60 / 61 / 285.
constexpr int QQ_T = 32, QQ_K = 64, QQ_CTAS = 8;
__global__ void __cluster_dims__(QQ_CTAS, 1, 1) __launch_bounds__(256)
    qq_kernel(const uint64_t* __restrict__ q, int m, int L, uint16_t* out, size_t ldo) {
    const int a0 = blockIdx.y * QQ_T, b0 = blockIdx.x / QQ_CTAS * QQ_T;
    if (b0 < a0) return;  // below the diagonal, the whole cluster
    __shared__ uint64_t ids[2 * QQ_T][QQ_K + 1];  // rows of the two groups
    __shared__ uint32_t present[2 * QQ_T][QQ_K / 32];
    __shared__ uint32_t part[QQ_T * QQ_T];
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & 15, ty = tid >> 4;
    const int rank = (int)cluster.block_rank(), per = (L + QQ_CTAS - 1) / QQ_CTAS;
    const int k1 = min(L, (rank + 1) * per);
    uint32_t d[2][2] = {};
    for (int k0 = rank * per; k0 < k1; k0 += QQ_K) {
#pragma unroll
        for (int e = 0; e < 2 * QQ_T / 8; e++) {
            const int t = warp + 8 * e, row = t < QQ_T ? a0 + t : b0 + t - QQ_T;
#pragma unroll
            for (int w = 0; w < QQ_K / 32; w++) {
                const int k = k0 + 32 * w + lane;
                const uint64_t v = row < m && k < k1 ? __ldg(q + (size_t)row * L + k) : 0;
                ids[t][32 * w + lane] = v;
                const uint32_t mask = __ballot_sync(0xFFFFFFFFu, v != 0);
                if (lane == 0) present[t][w] = mask;
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int v = 0; v < 2; v++)
#pragma unroll
                for (int w = 0; w < QQ_K / 32; w++)
                    d[u][v] += __popc(~(present[ty + 16 * u][w] ^ present[QQ_T + tx + 16 * v][w]));
#pragma unroll 8
        for (int k = 0; k < QQ_K; k++) {
            const uint64_t x0 = ids[ty][k], x1 = ids[ty + 16][k];
            const uint64_t y0 = ids[QQ_T + tx][k], y1 = ids[QQ_T + tx + 16][k];
            d[0][0] -= x0 == y0;
            d[0][1] -= x0 == y1;
            d[1][0] -= x1 == y0;
            d[1][1] -= x1 == y1;
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
        for (int v = 0; v < 2; v++) part[(ty + 16 * u) * QQ_T + tx + 16 * v] = d[u][v];
    cluster.sync();
    constexpr int SHARE = QQ_T * QQ_T / QQ_CTAS;
    if (tid < SHARE) {
        const int t = rank * SHARE + tid, a = a0 + t / QQ_T, b = b0 + t % QQ_T;
        uint32_t sum = 0;
#pragma unroll
        for (int c = 0; c < QQ_CTAS; c++) sum += cluster.map_shared_rank(part, c)[t];
        if (a < m && b < m && b > a) out[(size_t)a * ldo + b] = (uint16_t)sum;
    }
    cluster.sync();  // no CTA leaves while others read its counts
}

double now_s() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

}  // namespace

// A stream for a query's result copies and the events that order it against the
// query's own stream.
constexpr int kCopyBlocks = 16;
struct CopyLane {
    cudaStream_t st = nullptr;
    cudaEvent_t ev[kCopyBlocks + 2] = {};
    void destroy() {
        if (st) cudaStreamDestroy(st);
        for (cudaEvent_t x : ev)
            if (x) cudaEventDestroy(x);
    }
};
}  // namespace tch

using namespace tch;

struct tch_db {
    int device = 0, n = 0, L = 0, sms = 0;
    DeviceEncoding enc;
    cudaMemPool_t pool = nullptr;
    // copy lanes not in use: one per query that runs at the same time, kept for
    // the next and destroyed with the database
    std::mutex lanes_mu;
    std::vector<tch::CopyLane*> lanes;
};

namespace tch {
namespace {

cudaError_t take_lane(tch_db* db, CopyLane** out) {
    {
        std::lock_guard<std::mutex> lk(db->lanes_mu);
        if (!db->lanes.empty()) {
            *out = db->lanes.back();
            db->lanes.pop_back();
            return cudaSuccess;
        }
    }
    CopyLane* l = new CopyLane();
    cudaError_t e = cudaStreamCreateWithFlags(&l->st, cudaStreamNonBlocking);
    for (cudaEvent_t& x : l->ev)
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        l->destroy();
        delete l;
        return e;
    }
    *out = l;
    return cudaSuccess;
}

void give_lane(tch_db* db, CopyLane* l) {
    std::lock_guard<std::mutex> lk(db->lanes_mu);
    db->lanes.push_back(l);
}

// Batches of at most this many profiles go by the bit columns, whose read grows
// with them, larger ones by the tile pass, whose does not up to 256.  1 / 8 / 12 /
// 16 profiles, by columns: 44 / 215 / 322 / 404 us against 200 000 x 1 142, 67 /
// 154 / 207 / 258 against 50 000 x 3 016, 42 / 77 / 77 / 103 against 20 000 x
// 1 142; by tiles: 231 / 264 / 275 / 285, 188 / 203 / 219 / 222, 80 / 93 / 101 /
// 102.
constexpr int kBitProfiles = 8;
bool by_bits(const tch_db* db, int m) { return m <= kBitProfiles && db->enc.bits; }

size_t query_bytes(const tch_db* db, int m) {
    const size_t mr = up((size_t)std::max(m, 1), 256);
    return (size_t)m * db->L * 12 + mr * (size_t)db->enc.kb + (size_t)m * up((size_t)db->n, kRareDenseAlign) * 2 +
           (size_t)m * up((size_t)db->n, 8) * 2 + (size_t)m * up((size_t)m, 8) * 2 + (1u << 20);
}

// Results of at least this many bytes are copied beside the kernels.
constexpr size_t kOverlapBytes = (size_t)8 << 20;

// rows x w u16 to the host from device rows of stride ld.
cudaError_t copy_rows(uint16_t* dst, size_t w, const uint16_t* src, size_t ld, int rows, cudaStream_t st) {
    if (ld == w) return cudaMemcpyAsync(dst, src, (size_t)rows * w * 2, cudaMemcpyDeviceToHost, st);
    return cudaMemcpy2DAsync(dst, w * 2, src, ld * 2, w * 2, rows, cudaMemcpyDeviceToHost, st);
}

int db_query(tch_db* db, int m, const uint64_t* qcalls, uint16_t* h_qdb, uint16_t* h_qq, cudaStream_t st, Err& e) {
    const int n = db->n, L = db->L;
    const DeviceEncoding& enc = db->enc;
    const size_t mr = up((size_t)std::max(m, 1), 256);
    const size_t ldr = up((size_t)n, kRareDenseAlign), ldo = up((size_t)n, 8), ldq = up((size_t)m, 8);
    uint64_t* dq = nullptr;
    uint32_t* xq = nullptr;
    uint16_t *R = nullptr, *out = nullptr, *qq = nullptr;
    int* derr = nullptr;
    Fp4Operands QX;  // the batch's A-side rows: the database's K layout, m rows
    QX.pos = enc.X.neg;
    for (int c = 0; c < kMaxKChunks; c++) QX.pos.p[c] = nullptr;
    QX.n_rows = mr;
    QX.kb = enc.kb;
    KChunks& X = QX.pos;
    const bool bits = by_bits(db, m);
    // a large result goes back block by block on a stream of its own, while the
    // next block and the batch's own triangle are computed: 701 profiles against
    // 200 000, 280 MB, 2.08 ms against 2.66 in one piece after the last kernel.  A
    // block is a row block of the tile pass (256), more when there would be more
    // than kCopyBlocks.
    const int block = (int)up((size_t)std::max((m + kCopyBlocks - 1) / kCopyBlocks, 1), 256);
    CopyLane* lane = nullptr;
    cudaError_t ce = cudaSuccess;
    // TCH_VERBOSE=1: device time of each phase on stderr
    const char* vb = getenv("TCH_VERBOSE");
    const bool verbose = vb && vb[0] == '1';
    cudaEvent_t ev[8] = {};
    int nev = 0;
    auto mark = [&]() {
        if (verbose && nev < 8 && cudaEventCreate(&ev[nev]) == cudaSuccess) cudaEventRecord(ev[nev++], st);
    };
    if (m <= 0) return e.set("empty query batch");
    if (!qcalls) return e.set("null query calls");
    if (cudaSetDevice(db->device) != cudaSuccess) return e.set("cudaSetDevice(%d) failed", db->device);
    // one allocation for all of it: each costs the call about 2 us
    char* work = nullptr;
    size_t bytes = 0, zero_at = 0, zero = 0;
    auto place = [&](auto** p, size_t want) {  // two passes: sizes, then addresses
        if (work) *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(work + bytes);
        bytes += up(want, 256);
    };
    for (int pass = 0; pass < 2; pass++) {
        bytes = 0;
        place(&dq, (size_t)m * L * 8);
        if (h_qdb) place(&out, (size_t)m * ldo * 2);
        if (h_qq && m > 1) place(&qq, (size_t)m * ldq * 2);
        if (h_qdb && !bits) {
            place(&xq, (size_t)m * L * 4);
            place(&R, (size_t)m * ldr * 2);
            zero_at = bytes;  // zeroed: the operand rows and the error word
            for (int c = 0; c < X.n; c++) place(&X.p[c], mr * (size_t)X.width_of(c));
            place(&derr, 4);
            zero = bytes - zero_at;
        }
        if (pass == 0) ce = pool_alloc(&work, bytes, db->pool, st);
        if (ce != cudaSuccess) goto done;
    }
    mark();
    ce = cudaMemcpyAsync(dq, qcalls, (size_t)m * L * 8, cudaMemcpyHostToDevice, st);
    if (ce == cudaSuccess && zero) ce = cudaMemsetAsync(work + zero_at, 0, zero, st);
    if (ce != cudaSuccess) goto done;
    {
        const int grid = (int)std::min<size_t>(((size_t)m * L + 255) / 256, (size_t)db->sms * 16);
        if (h_qdb) {
            mark();
            if (!bits) {
                query_pack_kernel<<<grid, 256, 0, st>>>(dq, m, L, enc.cnt_off, enc.slot_ids, enc.col, enc.base, xq, X);
                ce = cudaGetLastError();
                if (ce != cudaSuccess) goto done;
            }
            RareGroups g;
            g.cnt_off = enc.cnt_off;
            g.goff = enc.goff;
            g.members = enc.members;
            g.members16 = enc.members16;
            g.wpos = enc.wpos;
            g.windows = query_windows(n);
            g.n = n;
            g.L = L;
            mark();
            StripeArgs a;
            a.n = n;
            a.ldo = ldo;
            a.err = derr;
            a.rect = true;
            if ((size_t)m * n * 2 >= kOverlapBytes) ce = take_lane(db, &lane);
            if (ce != cudaSuccess) goto done;
            const int step = lane ? block : m;
            for (int r0 = 0, k = 0; r0 < m; r0 += step, k++) {
                const int rows = std::min(step, m - r0);
                if (bits) {
                    query_few_kernel<<<dim3((unsigned)(g.windows * FEW_CTAS), rows), FEW_T, sizeof(FewShared), st>>>(
                        dq + (size_t)r0 * L, g, enc.slot_ids, enc.col, enc.base, (uint32_t)enc.D, enc.bits,
                        enc.bit_words, out + (size_t)r0 * ldo, ldo);
                    ce = cudaGetLastError();
                } else {
                    uint16_t* Rb = R + (size_t)r0 * ldr;
                    ce = launch_rare_query(g, xq + (size_t)r0 * L, rows, Rb, ldr, st);
                    if (ce != cudaSuccess) goto done;
                    a.r0 = r0;
                    a.rows = rows;
                    a.out = out + (size_t)r0 * ldo;
                    a.after_counts = true;
                    ce = launch_tc_stripe(QX, &enc.X, Rb, ldr, a, db->sms, st);
                }
                if (ce == cudaSuccess && lane) ce = cudaEventRecord(lane->ev[k], st);
                if (ce != cudaSuccess) goto done;
            }
        }
        if (qq) {
            mark();
            const unsigned tiles = (unsigned)((m + QQ_T - 1) / QQ_T);
            qq_kernel<<<dim3(tiles * QQ_CTAS, tiles), 256, 0, st>>>(dq, m, L, qq, ldq);
            ce = cudaGetLastError();
            if (ce == cudaSuccess && lane) ce = cudaEventRecord(lane->ev[kCopyBlocks], st);
            if (ce != cudaSuccess) goto done;
        }
        mark();
        // the copies last, as one into pageable memory holds this thread
        const cudaStream_t cs = lane ? lane->st : st;
        if (h_qdb) {
            const int step = lane ? block : m;
            for (int r0 = 0, k = 0; r0 < m && ce == cudaSuccess; r0 += step, k++) {
                const int rows = std::min(step, m - r0);
                if (lane) ce = cudaStreamWaitEvent(cs, lane->ev[k], 0);
                // one linear copy when the rows are packed (ldo == n), a pitched one otherwise
                if (ce == cudaSuccess)
                    ce = copy_rows(h_qdb + (size_t)r0 * n, (size_t)n, out + (size_t)r0 * ldo, ldo, rows, cs);
            }
            if (ce != cudaSuccess) goto done;
        }
        if (qq) {
            if (lane) ce = cudaStreamWaitEvent(cs, lane->ev[kCopyBlocks], 0);
            if (ce == cudaSuccess) ce = copy_rows(h_qq, (size_t)m, qq, ldq, m, cs);
            if (ce != cudaSuccess) goto done;
        }
    }
done:
    {
        int herr = 0;
        if (lane) {  // what follows on this stream (the buffers' release) comes after the copies
            cudaError_t le = cudaEventRecord(lane->ev[kCopyBlocks + 1], lane->st);
            if (le == cudaSuccess) le = cudaStreamWaitEvent(st, lane->ev[kCopyBlocks + 1], 0);
            if (le != cudaSuccess) cudaStreamSynchronize(lane->st);
            if (ce == cudaSuccess) ce = le;
        }
        if (derr && ce == cudaSuccess) ce = cudaMemcpyAsync(&herr, derr, 4, cudaMemcpyDeviceToHost, st);
        if (work) cudaFreeAsync(work, st);
        mark();
        const cudaError_t se = cudaStreamSynchronize(st);
        if (ce == cudaSuccess) ce = se;
        if (lane) give_lane(db, lane);
        if (nev > 1) {
            static const char* names[] = {"h2d", "rank+pack", "counts + distances", "q x q", "d2h", "", "", ""};
            fprintf(stderr, "tch query m=%d:", m);
            for (int k = 0; k + 1 < nev; k++) {
                float ms = 0;
                cudaEventElapsedTime(&ms, ev[k], ev[k + 1]);
                fprintf(stderr, " %s %.2f ms", names[k], ms);
            }
            fprintf(stderr, "\n");
        }
        for (int k = 0; k < nev; k++) cudaEventDestroy(ev[k]);
        if (ce != cudaSuccess) return e.set("query batch: %s", cudaGetErrorString(ce));
        if (herr) return e.set("query batch: device reported error 0x%x", herr);
    }
    return 0;
}

struct Request {
    int64_t id = 0;
    int m = 0;
    const uint64_t* q = nullptr;
    uint16_t* h_qdb = nullptr;
    uint16_t* h_qq = nullptr;
    size_t bytes = 0;
    double t_submit = 0, t_start = 0, t_done = 0;
    bool done = false;
    int rc = 0;
    char err[256] = {0};
};

}  // namespace
}  // namespace tch

struct tch_server {
    tch_db* db = nullptr;
    size_t budget = 0, in_use = 0;
    int running = 0;
    bool stop = false;
    std::mutex mu;
    std::condition_variable cv;
    std::deque<Request*> queue;
    std::map<int64_t, Request*> reqs;
    int64_t next_id = 1;
    std::vector<std::thread> workers;
};

namespace tch {
namespace {

void worker_loop(tch_server* sv) {
    cudaSetDevice(sv->db->device);
    cudaStream_t st = nullptr;
    cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    for (;;) {
        Request* r = nullptr;
        {
            std::unique_lock<std::mutex> lk(sv->mu);
            // FIFO; the head starts when it fits next to the running requests
            // (or alone, whatever its size)
            sv->cv.wait(lk, [&] {
                return sv->stop ||
                       (!sv->queue.empty() && (sv->running == 0 || sv->in_use + sv->queue.front()->bytes <= sv->budget));
            });
            if (sv->stop && sv->queue.empty()) break;
            r = sv->queue.front();
            sv->queue.pop_front();
            sv->in_use += r->bytes;
            sv->running++;
            r->t_start = now_s();
        }
        Err e{r->err, (int)sizeof(r->err)};
        const int rc = db_query(sv->db, r->m, r->q, r->h_qdb, r->h_qq, st, e);
        {
            std::lock_guard<std::mutex> lk(sv->mu);
            sv->in_use -= r->bytes;
            sv->running--;
            r->rc = rc;
            r->t_done = now_s();
            r->done = true;
        }
        sv->cv.notify_all();
    }
    if (st) cudaStreamDestroy(st);
}

}  // namespace
}  // namespace tch

extern "C" {

int tch_db_create(int device, int n, int L, const uint64_t* calls, int tau, tch_db** out, char* err, int errlen) {
    Err e{err, errlen};
    uint64_t* d_calls = nullptr;
    tch_db* db = nullptr;
    if (!out) return e.set("null output handle");
    *out = nullptr;
    if (n < 1 || L < 1) return e.set("the database needs n >= 1 profiles and L >= 1 loci (got n=%d, L=%d)", n, L);
    if (L > 65535) return e.set("more than 65535 loci (u16 distances)");
    if (!calls) return e.set("null input buffer");
    db = new tch_db();
    db->device = device;
    db->n = n;
    db->L = L;
    {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        uint64_t keep = ~0ull;
        TCH_CK(e, cudaSetDevice(device));
        TCH_CK(e, cudaDeviceGetAttribute(&db->sms, cudaDevAttrMultiProcessorCount, device));
        TCH_CK(e, cudaMemPoolCreate(&db->pool, &props));
        TCH_CK(e, cudaMemPoolSetAttribute(db->pool, cudaMemPoolAttrReleaseThreshold, &keep));
        TCH_CK(e, cudaFuncSetAttribute(query_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(FewShared)));
    }
    TCH_CK(e, device_alloc(&d_calls, (size_t)n * L * 8));
    TCH_CK(e, cudaMemcpy(d_calls, calls, (size_t)n * L * 8, cudaMemcpyHostToDevice));
    {
        TauModel model;
        if (encode_on_device(device, n, L, d_calls, tau, model, false, max_chunk_bytes(), ENC_QUERY, &db->enc, e))
            goto fail;
    }
    cudaFree(d_calls);
    cudaStreamSynchronize(0);  // the working pool lets go of what it does not keep
    // the database's own triangle is not served: drop its ranks and positions,
    // and its A-side operand copy (queries are the A side)
    cudaFree(db->enc.x);
    cudaFree(db->enc.mpos);
    db->enc.bytes -= (size_t)n * L * 6;
    db->enc.x = nullptr;
    db->enc.mpos = nullptr;
    for (int c = 0; c < kMaxKChunks; c++)
        if (db->enc.X.pos.p[c]) {
            cudaFree(db->enc.X.pos.p[c]);
            db->enc.X.pos.p[c] = nullptr;
            db->enc.bytes -= db->enc.x_rows * (size_t)db->enc.X.pos.width_of(c);
        }
    *out = db;
    return 0;
fail:
    if (d_calls) cudaFree(d_calls);
    if (db) {
        if (db->pool) cudaMemPoolDestroy(db->pool);
        delete db;
    }
    return 1;
}

void* tch_host_alloc(size_t bytes) {
    void* p = nullptr;
    return cudaMallocHost(&p, std::max<size_t>(bytes, 16)) == cudaSuccess ? p : nullptr;
}

void tch_host_free(void* p) {
    if (p) cudaFreeHost(p);
}

void tch_db_destroy(tch_db* db) {
    if (!db) return;
    cudaSetDevice(db->device);
    cudaDeviceSynchronize();
    free_device_encoding(&db->enc);
    for (CopyLane* l : db->lanes) {
        l->destroy();
        delete l;
    }
    if (db->pool) cudaMemPoolDestroy(db->pool);
    delete db;
}

int tch_db_info(const tch_db* db, int* n, int* L, int* tau, size_t* d_onehot, size_t* device_bytes, int* k_chunks) {
    if (!db) return 1;
    if (k_chunks) *k_chunks = db->enc.X.neg.n;
    if (n) *n = db->n;
    if (L) *L = db->L;
    if (tau) *tau = db->enc.tau;
    if (d_onehot) *d_onehot = db->enc.D;
    if (device_bytes) *device_bytes = db->enc.bytes;
    return 0;
}

size_t tch_db_query_bytes(const tch_db* db, int m) { return db && m > 0 ? query_bytes(db, m) : 0; }

int tch_db_query(tch_db* db, int m, const uint64_t* qcalls, uint16_t* qdb, uint16_t* qq, void* stream, char* err,
                 int errlen) {
    Err e{err, errlen};
    if (!db) return e.set("null database");
    return db_query(db, m, qcalls, qdb, qq, (cudaStream_t)stream, e);
}

int tch_server_create(tch_db* db, int slots, size_t budget, tch_server** out, char* err, int errlen) {
    Err e{err, errlen};
    if (!db || !out) return e.set("null argument");
    if (slots < 1 || slots > 64) return e.set("slots must be in [1, 64] (got %d)", slots);
    tch_server* sv = new tch_server();
    sv->db = db;
    if (!budget) {
        size_t f = 0;
        cudaSetDevice(db->device);
        free_memory(db->device, &f);
        budget = f / 2;
    }
    sv->budget = budget;
    for (int s = 0; s < slots; s++) sv->workers.emplace_back(worker_loop, sv);
    *out = sv;
    return 0;
}

int64_t tch_server_submit(tch_server* sv, int m, const uint64_t* qcalls, uint16_t* qdb, uint16_t* qq) {
    if (!sv || m <= 0 || !qcalls) return -1;
    Request* r = new Request();
    r->m = m;
    r->q = qcalls;
    r->h_qdb = qdb;
    r->h_qq = qq;
    r->bytes = query_bytes(sv->db, m);
    r->t_submit = now_s();
    {
        std::lock_guard<std::mutex> lk(sv->mu);
        r->id = sv->next_id++;
        sv->reqs[r->id] = r;
        sv->queue.push_back(r);
    }
    sv->cv.notify_all();
    return r->id;
}

int tch_server_wait(tch_server* sv, int64_t id, double* queued_s, double* latency_s, char* err, int errlen) {
    Err e{err, errlen};
    if (!sv) return e.set("null server");
    Request* r = nullptr;
    {
        std::unique_lock<std::mutex> lk(sv->mu);
        auto it = sv->reqs.find(id);
        if (it == sv->reqs.end()) return e.set("unknown request %lld", (long long)id);
        r = it->second;
        // claimed before the wait releases the lock: a second wait on the
        // same id finds it unknown instead of sharing (and deleting) it
        sv->reqs.erase(it);
        sv->cv.wait(lk, [&] { return r->done; });
    }
    if (queued_s) *queued_s = r->t_start - r->t_submit;
    if (latency_s) *latency_s = r->t_done - r->t_submit;
    const int rc = r->rc;
    if (rc) e.set("%s", r->err);
    delete r;
    return rc;
}

void tch_server_destroy(tch_server* sv) {
    if (!sv) return;
    {
        std::lock_guard<std::mutex> lk(sv->mu);
        sv->stop = true;
    }
    sv->cv.notify_all();
    for (auto& t : sv->workers) t.join();
    for (auto& kv : sv->reqs) delete kv.second;
    delete sv;
}

}  // extern "C"
