// Tensor-core tile pass for sm_103a: block-scaled fp4 tcgen05.mma
// (kind::mxf4, every scale factor 1.0) with TMEM accumulators, operands staged
// by TMA, one fused epilogue writing u16 distances.
//
// Operands (Fp4Operands): packed e2m1 rows [presence | one-hot | zeros], two
// elements per byte, 0 or +1.0 in the `pos` copy, which is read as A, and 0
// or +1.0 / -1.0 (one-hot part) in the `neg` copy, which is read as B.  One
// output tile (256 rows i x 240 columns j) is
//
//   D = pos_i . neg_j^T  =  P Pt - O Ot
//
// Every product is 0 or +-1 and every partial sum an integer of magnitude at
// most the number of loci (< 2^24), so the fp32 accumulation is exact; the
// epilogue re-checks the integrality of every value and reports a device
// error if it ever fails.  This replaces the reference's two CUTLASS b1 GEMMs
// (tensorcore/rs/cuda/tch.cu:22-32, 128-129): on GB300 the b1 warp MMA issues
// at ~150 TOPS, kind::i8 does not exist on sm_103a, and the fp4 kinds run at
// twice the fp8 rate from half the operand bytes (tch-peak).  The fp4 kinds
// have no negate bit, hence the second operand copy with the one-hot sign in
// the data.
//
// A CTA pair (cluster of two, tcgen05 cta_group::2) per tile, 10 warps per
// CTA, one CTA per SM, persistent over the stripe's tiles (upper triangle
// only, or every tile of a rectangle):
//   warp 0    TMA producer   ring of 6 or 7 stages (A 128 x 128 B, B 120 x 128 B): each
//                            CTA its 128 rows of A and its half of the columns'
//                            rows, completing on the first CTA's barrier
//   warp 1    MMA issuer     (first CTA) 4 x tcgen05.mma (M 256, N 240, K = 64
//                            elements) per stage into one of two 240-column
//                            accumulators in both CTAs' TMEM
//   warps 2-9 epilogue       two per TMEM lane quarter, one per column half:
//                            tcgen05.ld 32 columns x 16 rows -> u16 pairs -> quad
//                            transpose -> minus the dense rare counts (loaded
//                            while the MMAs run) -> 16-byte stores
// TMEM: accumulators at columns 0 and 240, the scale factors (1.0, written
// once by the epilogue warps before the first MMA) in columns 480-511.
// Tiles are visited in raster groups of row blocks, column-major inside a
// group, so that the pairs running at the same time share A and B tiles in L2.
//
// What bounds it: the shared-memory data path.  A stage's 31 KB per CTA are
// written by TMA and read by the MMAs at 128 bytes a cycle, 496 cycles in all (as
// many as the 64 bytes a cycle that an SM takes in from L2 allow), while its MMAs
// take 480 (16 384 MACs per cycle and SM, the probe's rate); 503 cycles per stage
// measured, and the epilogue's accesses come on top, 1.9 us per tile with seven
// stages.  One CTA per tile (128 x 224) takes 44 KB for 448 cycles of MMAs and
// stops at 0.61 of the probe's rate: 8.46 ms for the triangle of 63 005 long-tail
// profiles at tau 1 024, 5.95 ms in pairs (0.88).
// Three more things were needed to get there, each measured on that triangle
// (8.38 ms as a plain pair):
//   - the next stage's barrier is looked at before a stage's MMAs are issued:
//     a wait between two stages costs the issuing thread about 130 cycles that
//     the tensor pipe then idles (8.38 -> 8.18);
//   - the epilogue touches whole 64-byte row pieces (8.18 -> 7.60, below);
//   - producer and issuer run under elect.sync (7.60 -> 6.27): under
//     `lane == 0` an MMA takes 86 cycles to issue, as its descriptors move
//     through vector registers;
// raster groups of 16 and the smaller shared-memory configuration did the rest.
//
// Stripes and sets of at most 128 rows, where there are enough of their tiles, take
// the same kernel with a CTA by itself per tile (128 x 240, 4 stages of 46 KB).
//
// Every mbarrier wait is bounded (about 2 s of %globaltimer, none of it spent on the
// launch before); on a timeout the CTA records DEVERR_TIMEOUT, stops issuing work,
// drains what it issued, frees its TMEM and returns.

#include <cuda.h>
#include <cudaTypedefs.h>
#include <limits.h>

#include <algorithm>
#include <functional>
#include <numeric>
#include <queue>
#include <utility>
#include <vector>

#include "tc_ptx.cuh"
#include "tch_internal.cuh"

namespace tch {
namespace {

constexpr int BM = 128;             // tile rows of one CTA (TMEM lanes)
constexpr int PM = 2 * BM;          // tile rows of a CTA pair (MMA M)
constexpr int BN = 240;             // tile columns (MMA N)
constexpr int BH = BN / 2;          // column rows staged by each CTA of the pair
constexpr int BK = 128;             // bytes of K per stage: one 128-byte swizzle row, 256 elements
// Stages of the ring: seven fit, but with six the 196 KB configuration of shared
// memory leaves the epilogue's loads 32 KB more of L1.  63 005 profiles, tau 1 024
// (50 stages of K per tile): 6.19 ms with seven, 5.95 with six (6.42 with six in
// the 228 KB configuration); 12 011 founders with 997 stages of K: 4.22 and 4.34;
// alike with 81 stages, and for many sets in one launch.
constexpr int FEW_STAGES = 6, ALL_STAGES = 7;
constexpr int FEW_STAGES_K = 100;  // six up to this many stages of K per tile
constexpr int A_BYTES = BM * BK;    // 16 KB
constexpr int B_BYTES = BH * BK;    // 15 KB: the column rows of one TMA box
// One CTA's stage: a CTA by itself (below) holds the column rows of both boxes.
__host__ __device__ constexpr int stage_bytes(bool pair) { return A_BYTES + (pair ? 1 : 2) * B_BYTES; }
constexpr int ONE_STAGES = 4;       // of 46 KB
// For the schedule of a batch, in K stages of a pair: a tile's epilogue beyond its
// MMAs, and a launch.
constexpr long long kEpilogueStages = 4, kLaunchStages = 16;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int ACC_STRIDE = BN;      // TMEM columns from one accumulator to the next
constexpr int SF_COL = 480;         // 32 TMEM columns of scale factors
constexpr int TMEM_COLS = 512;
constexpr int CHUNK = 32;           // accumulator columns per tcgen05.ld (16 lanes each)
constexpr int CHUNKS = (BN + CHUNK - 1) / CHUNK;
constexpr int WARP_CHUNKS = (CHUNKS + 1) / 2;  // chunks of the first column half (the second has the rest)
// 128-row blocks per raster group (TCH_TC_GROUP overrides): 63 005 profiles, tau
// 1 024: 4 -> 6.82 ms, 8 -> 6.31, 16 -> 6.24, 32 -> 6.40
constexpr int GROUP_M = 16;
constexpr int BAR_BYTES = 256;
constexpr int smem_bytes(bool pair, int stages) { return 1024 + stages * stage_bytes(pair) + BAR_BYTES; }
static_assert(smem_bytes(true, ALL_STAGES) <= 232448 && smem_bytes(false, ONE_STAGES) <= 232448, "shared memory per CTA");
static_assert(BN % 16 == 0 && BN <= 256 && ACC_STRIDE + BN <= SF_COL && SF_COL + 32 <= TMEM_COLS, "TMEM layout");
static_assert(ACC_STRIDE + CHUNKS * CHUNK <= TMEM_COLS, "the last chunk's loads stay inside TMEM");
static_assert(BH % 8 == 0, "whole 8-row swizzle atoms per CTA");
static_assert(A_BYTES % 1024 == 0 && B_BYTES % 1024 == 0, "stages stay 1024-byte aligned (128-byte swizzle)");

using namespace ptx;

// 128-row blocks per raster group: GROUP_M unless TCH_TC_GROUP gives another
// count in [1, 256].  Larger groups read the column side of the operand fewer
// times (once per group) at the cost of a larger row-side working set.
int group_row_blocks() {
    static int g = 0;
    if (!g) {
        const char* v = getenv("TCH_TC_GROUP");
        const int x = v ? atoi(v) : 0;
        g = (x >= 1 && x <= 256) ? x : GROUP_M;
    }
    return g;
}

// Row blocks of a pair (PM rows) per raster group, from the schedule's 128-row blocks.
int pair_group(int group) { return std::max(1, (group > 0 ? std::min(group, 256) : group_row_blocks()) / 2); }

// ---------------------------------------------------------------- tile order
// Row block bi covers rows a_r0 + PM bi .. + PM of the A operand, column block
// bj columns c0 + BN bj .. + BN.  In a triangle (c0 = r0) the row block's
// first column block is the one holding its first diagonal cell.
struct TileSpace {
    int nbi, nbj;  // row blocks of the stripe, column blocks of [c0, n)
    int gs;        // row blocks per raster group
    int rect;      // 1: every tile (rows of one set against columns of another)
};

__host__ __device__ __forceinline__ int first_col(const TileSpace& ts, int bi) {
    return ts.rect ? 0 : (PM * bi) / BN;
}
// The last row block present in column block bj.
__host__ __device__ __forceinline__ int last_row(const TileSpace& ts, int bj) {
    const int r = ((bj + 1) * BN - 1) / PM;
    return ts.rect || r > ts.nbi - 1 ? ts.nbi - 1 : r;
}

__host__ __device__ __forceinline__ long long tiles_in(const TileSpace& ts, int b0, int b1) {
    long long c = 0;
    for (int bi = b0; bi < b1; bi++) c += ts.nbj > first_col(ts, bi) ? ts.nbj - first_col(ts, bi) : 0;
    return c;
}

constexpr int MAX_GROUPS = 1024;  // raster groups with a precomputed first tile

// First tile index of every raster group, so a tile's coordinates cost a
// binary search over groups plus a few steps.
struct GroupTable {
    int ngroups;
    int first[MAX_GROUPS + 1];
};

// t -> (bi, bj).
__device__ bool tile_coords(const TileSpace& ts, const GroupTable& gt, int t, int* bi_out, int* bj_out) {
    int lo = 0, hi = gt.ngroups;  // last group whose first tile is <= t
    while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (gt.first[mid] <= t) lo = mid; else hi = mid;
    }
    t -= gt.first[lo];
    const int g0 = lo * ts.gs, g1 = min(ts.nbi, g0 + ts.gs);
    // columns that hold only part of the group (those that cross the diagonal)
    int bj = first_col(ts, g0);
    for (; bj < ts.nbj; bj++) {
        const int rows = min(g1 - 1, last_row(ts, bj)) - g0 + 1;  // rows g0 .. of the group in column bj
        if (rows == g1 - g0) break;  // from here on every column holds the whole group
        if (t < rows) {
            *bi_out = g0 + t;
            *bj_out = bj;
            return true;
        }
        t -= rows;
    }
    const int full = g1 - g0;
    bj += t / full;
    if (bj >= ts.nbj) return false;
    *bi_out = g0 + t % full;
    *bj_out = bj;
    return true;
}

// Tensor maps of every K chunk: A boxes (128 rows of the pos copy) and B
// boxes (BH rows of the neg copy), and the 128-byte K blocks of each chunk.
struct TcMaps {
    CUtensorMap a[kMaxKChunks];
    CUtensorMap b[kMaxKChunks];
    int kblocks[kMaxKChunks];
    int n;
};

// One triangle of a batch: its geometry, K stages, tensor maps and output.
struct TcJob {
    int n, rows, kblocks;  // rows [0, rows) against columns [0, n) of one set (r0 = c0 = 0)
    int nchunks;           // K chunks: A maps at jmaps[map0 ..), B maps at jmaps[map0 + nchunks ..)
    int kbl[kMaxKChunks];  // K stages of each chunk
    int map0;
    TileSpace ts;          // one raster group
    const uint16_t* rdense;
    size_t ldr;
    uint16_t* out;
    size_t ldo;
    int vec_store;
};

// One stripe (the fields below `err` unused), or a batch of triangles
// (MULTI: `jobs`, their tensor maps `jmaps`, and the CTA pairs' tiles, pair p's
// (job, tile of the job) at tiles[first[p]] .. tiles[first[p + 1] - 1], all in
// device memory, written before the launch).
struct TcParams {
    int n, r0, rows;  // columns end at n; rows [r0, r0 + rows) of the A operand
    int c0;           // first column: r0 (upper triangle) or 0 (rectangle)
    int kblocks;      // K stages per tile
    TileSpace ts;
    GroupTable gt;
    int num_tiles;
    const uint16_t* rdense;  // dense rare counts (row stride ldr, column j at j - c0), or null
    size_t ldr;
    uint16_t* out;
    size_t ldo;
    int vec_store;  // 1: 16-byte stores (ldo a multiple of 8, out 16-byte aligned)
    int* err;
    const TcJob* jobs;
    const CUtensorMap* jmaps;
    const int2* tiles;
    const int* first;
};

// t -> (bi, bj) when the whole triangle is one raster group (a batch job).
__device__ bool tile_coords_one_group(const TileSpace& ts, int t, int* bi_out, int* bj_out) {
    const int g1 = ts.nbi;
    int bj = first_col(ts, 0);
    for (; bj < ts.nbj; bj++) {
        const int rows = min(g1 - 1, last_row(ts, bj)) + 1;
        if (rows == g1) break;
        if (t < rows) {
            *bi_out = t;
            *bj_out = bj;
            return true;
        }
        t -= rows;
    }
    bj += t / g1;
    if (bj >= ts.nbj) return false;
    *bi_out = t % g1;
    *bj_out = bj;
    return true;
}

// Lane quads transpose 4 x 4 words: lane c of a quad gives w[r] to lane r and
// ends with word r from lane r of the quad, its own in place.
__device__ __forceinline__ void quad_transpose(uint32_t (&w)[4], int c) {
    constexpr unsigned ALL = 0xFFFFFFFFu;
    const bool odd = c & 1, upper = c & 2;
    const uint32_t s0 = __shfl_xor_sync(ALL, odd ? w[0] : w[1], 1);
    const uint32_t s1 = __shfl_xor_sync(ALL, odd ? w[2] : w[3], 1);
    if (odd) w[0] = s0, w[2] = s1;
    else w[1] = s0, w[3] = s1;
    const uint32_t t0 = __shfl_xor_sync(ALL, upper ? w[0] : w[2], 2);
    const uint32_t t1 = __shfl_xor_sync(ALL, upper ? w[1] : w[3], 2);
    if (upper) w[0] = t0, w[1] = t1;
    else w[2] = t0, w[3] = t1;
}

// Two exact fp32 integers as u16 halves of a word (modulo 2^16): added to 1.5
// x 2^23, an integer of magnitude below 2^22 stands in the low mantissa bits.
// `bad` is set when one is not an integer.
__device__ __forceinline__ uint32_t pack_u16(uint32_t v0, uint32_t v1, bool* bad) {
    constexpr float kShift = 12582912.0f;
    const float f0 = __uint_as_float(v0), f1 = __uint_as_float(v1);
    const float x0 = __fadd_rn(f0, kShift), x1 = __fadd_rn(f1, kShift);
    *bad |= (__fsub_rn(x0, kShift) != f0) | (__fsub_rn(x1, kShift) != f1);
    return __byte_perm(__float_as_uint(x0), __float_as_uint(x1), 0x5410);
}

// PAIR false: a CTA by itself per tile of 128 x 240, for stripes and sets of at most
// 128 rows, whose pairs would work half for nothing (see one_cta).
template <bool MULTI, bool PAIR, int STAGES>
__global__ void __cluster_dims__(PAIR ? 2 : 1, 1, 1) __launch_bounds__(THREADS, 1)
    tc_stripe_kernel(const __grid_constant__ TcMaps maps, const TcParams p) {
    constexpr int CTAS = PAIR ? 2 : 1;  // of a tile
    constexpr int STAGE_BYTES = stage_bytes(PAIR), CTA_B_BYTES = STAGE_BYTES - A_BYTES;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* stage_a = smem;
    uint8_t* stage_b = smem + STAGES * A_BYTES;
    uint64_t* bars = (uint64_t*)(smem + STAGES * STAGE_BYTES);
    uint64_t* full = bars;                     // STAGES
    uint64_t* empty = bars + STAGES;           // STAGES
    uint64_t* tfull = bars + 2 * STAGES;       // 2
    uint64_t* tempty = bars + 2 * STAGES + 2;  // 2
    uint64_t* drain = bars + 2 * STAGES + 4;   // 1
    uint64_t* scales = bars + 2 * STAGES + 5;  // 1: the scale factors stand in both CTAs' TMEM
    uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 6);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    // this pair's tiles: every (gridDim.x / 2)-th one, or its list of a batch's
    const int pair = blockIdx.x / CTAS;
    const int t_begin = MULTI ? p.first[pair] : pair, t_end = MULTI ? p.first[pair + 1] : p.num_tiles;
    const int t_step = MULTI ? 1 : gridDim.x / CTAS;
    const uint32_t rank = PAIR ? cluster_rank() : 0;  // 0: the CTA that issues the pair's MMAs

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], CTAS * EPI_WARPS);  // both CTAs' epilogues
        }
        mbar_init(drain, 1);
        mbar_init(scales, 4 * CTAS);  // four warps of each CTA
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (!MULTI)
            for (int c = 0; c < maps.n; c++) {
                asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&maps.a[c]) : "memory");
                asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&maps.b[c]) : "memory");
            }
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                         "r"(TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    tc_fence_before();
    __syncwarp();
    cluster_sync();  // barriers initialised and TMEM allocated in both CTAs
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------------------ producer
        if (elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            int issued[STAGES];
            uint32_t issued_ph[STAGES];
            for (int q = 0; q < STAGES; q++) issued[q] = 0, issued_ph[q] = 0;
            int last_job = -1;  // MULTI: the job whose maps this thread has acquired
            for (int t = t_begin, nth = 0; ok && t < t_end; t += t_step, nth++) {
                if (nth == 2) grid_wait();  // as the issuer
                int bi, bj, y_a, y_b, kblocks;
                const CUtensorMap* ma = maps.a;
                const CUtensorMap* mb = maps.b;
                const int* kbls = maps.kblocks;
                if (!MULTI) {
                    if (!tile_coords(p.ts, p.gt, t, &bi, &bj)) break;
                    y_a = p.r0 + bi * PM;
                    y_b = p.c0 + bj * BN;
                    kblocks = p.kblocks;
                } else {
                    const int2 tile = __ldg(p.tiles + t);
                    const int job = tile.x;
                    const TcJob& jb = p.jobs[job];
                    if (!tile_coords_one_group(jb.ts, tile.y, &bi, &bj)) break;
                    y_a = bi * PM;
                    y_b = bj * BN;
                    kblocks = jb.kblocks;
                    ma = p.jmaps + jb.map0;
                    mb = ma + jb.nchunks;
                    kbls = jb.kbl;
                    if (job != last_job) {
                        for (int c = 0; c < 2 * jb.nchunks; c++) tensormap_acquire(ma + c);
                        last_job = job;
                    }
                }
                y_a += (int)rank * BM;  // this CTA's half of the rows and of the columns
                y_b += (int)rank * BH;
                int ch = 0, kbl = 0;  // K chunk and block inside it
                int kbl_end = kbls[0];
                for (int kb = 0; kb < kblocks; kb++) {
                    if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.err)) { ok = false; break; }
                    // both CTAs' loads complete on the issuing CTA's barrier
                    if (rank == 0) mbar_expect_tx(&full[s], CTAS * STAGE_BYTES);
                    uint8_t *sa = stage_a + s * A_BYTES, *sb = stage_b + s * CTA_B_BYTES;
                    if (PAIR) {
                        const uint32_t bar = peer_addr(&full[s], 0);
                        tma_load_2d_pair(ma + ch, bar, sa, kbl * BK, y_a);
                        tma_load_2d_pair(mb + ch, bar, sb, kbl * BK, y_b);
                    } else {
                        const uint32_t bar = smem_u32(&full[s]);
                        tma_load_2d(ma + ch, bar, sa, kbl * BK, y_a);
                        tma_load_2d(mb + ch, bar, sb, kbl * BK, y_b);
                        tma_load_2d(mb + ch, bar, sb + B_BYTES, kbl * BK, y_b + BH);
                    }
                    if (++kbl == kbl_end) {
                        kbl = 0;
                        if (++ch < kMaxKChunks) kbl_end = kbls[ch];
                    }
                    issued[s] = 1;
                    issued_ph[s] = ph;
                    if (++s == STAGES) s = 0, ph ^= 1;
                }
            }
            if (ok) {
                // tail: every stage released by the MMA warp (all commits arrived)
                for (int q = 0; q < STAGES; q++) {
                    if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.err)) break;
                    if (++s == STAGES) s = 0, ph ^= 1;
                }
            } else if (rank == 0) {
                // abort: let the loads already issued land before the pair exits
                for (int q = 0; q < STAGES; q++)
                    if (issued[q]) {
                        const unsigned long long t0 = gtimer();
                        while (!mbar_test(&full[q], issued_ph[q]) && gtimer() - t0 < WAIT_NS) {}
                    }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = make_idesc_mx(kE2M1, 1, CTAS * BM, BN);
            const uint32_t sf = tmem_base + SF_COL;
            int s = 0, acc = 0;
            uint32_t ph = 0, aph = 0;
            bool ready = false;  // stage s is known to hold its operands
            bool ok = mbar_wait(scales, 0, abort_flag, p.err);
            tc_fence_after();
            for (int t = t_begin, nth = 0; ok && t < t_end; t += t_step, nth++) {
                // the first two tiles have an accumulator each; the third waits for
                // the epilogue, and so for the launch before, however long that
                // takes: the bound of the waits begins when it is done
                if (nth == 2) grid_wait();
                const int kblocks = MULTI ? p.jobs[__ldg(&p.tiles[t].x)].kblocks : p.kblocks;
                if (!mbar_wait(&tempty[acc], aph ^ 1, abort_flag, p.err)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(acc * ACC_STRIDE);
                for (int kb = 0; kb < kblocks; kb++) {
                    if (!ready && !mbar_wait(&full[s], ph, abort_flag, p.err)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a0 = smem_u32(stage_a + s * A_BYTES), b0 = smem_u32(stage_b + s * CTA_B_BYTES);
                    // look at the next stage's barrier before this stage's MMAs are
                    // issued: the look's latency then hides behind them instead of
                    // leaving the tensor pipe idle between two stages
                    const int sn = s + 1 == STAGES ? 0 : s + 1;
                    ready = mbar_peek(&full[sn], sn ? ph : ph ^ 1);
#pragma unroll
                    for (int k = 0; k < BK / 32; k++) {
                        const uint64_t da = sw128_desc(a0 + 32 * k), db = sw128_desc(b0 + 32 * k);
                        const uint32_t accumulate = (kb | k) ? 1u : 0u;
                        if (PAIR) tc_mma_mxf4_pair(d_tmem, da, db, idesc, sf, sf, accumulate);
                        else tc_mma_mxf4(d_tmem, da, db, idesc, sf, sf, accumulate);
                    }
                    // stage free in both CTAs once these MMAs have read it
                    if (PAIR) tc_commit_pair(&empty[s]);
                    else tc_commit(&empty[s]);
                    if (++s == STAGES) s = 0, ph ^= 1;
                }
                if (!ok) break;
                if (PAIR) tc_commit_pair(&tfull[acc]);  // accumulator ready for both epilogues
                else tc_commit(&tfull[acc]);
                if (++acc == 2) acc = 0, aph ^= 1;
            }
            // every MMA issued by this thread has completed before TMEM is freed
            if (PAIR) tc_commit_pair_local(drain);
            else tc_commit(drain);
            const unsigned long long t0 = gtimer();
            while (!mbar_test(drain, 0) && gtimer() - t0 < WAIT_NS) {}
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue
        const int q = warp & 3;           // TMEM lanes [32 q, 32 q + 32) belong to this warp
        const int half = (warp - 2) / 4;  // column half of the tile
        if (half == 0) {
            // scale factors 1.0 in every lane of the 32 scale-factor columns, one
            // warp per lane quarter; the first loads are under way meanwhile
            tmem_fill32(tmem_base + ((uint32_t)(q * 32) << 16) + SF_COL, 0x01010101u * kUe8m0One);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(peer_addr(scales, 0));
        }
        // the operands do not depend on the launch before, so its tail overlaps the
        // first tiles' MMAs; the rare counts do, and the output may still be read
        grid_wait();
        int acc = 0;
        uint32_t aph = 0;
        bool bad = false;
        for (int t = t_begin; t < t_end; t += t_step) {
            int bi, bj;
            int n = p.n, r0 = p.r0, c0 = p.c0, iend = p.r0 + p.rows, vec_store = p.vec_store;
            const uint16_t* rdense = p.rdense;
            uint16_t* out = p.out;
            size_t ldo = p.ldo, ldr = p.ldr;
            const bool tri = MULTI || !p.ts.rect;
            if (!MULTI) {
                if (!tile_coords(p.ts, p.gt, t, &bi, &bj)) break;
            } else {
                const int2 tile = __ldg(p.tiles + t);
                const TcJob& jb = p.jobs[tile.x];
                if (!tile_coords_one_group(jb.ts, tile.y, &bi, &bj)) break;
                n = jb.n;
                r0 = 0;
                c0 = 0;
                iend = jb.rows;
                vec_store = jb.vec_store;
                rdense = jb.rdense;
                out = jb.out;
                ldo = jb.ldo;
                ldr = jb.ldr;
            }
            const bool dense = rdense != nullptr;
            // A chunk is 32 columns of the warp's 32 rows, in two passes of 16 rows.
            // After the quad transpose a lane holds 8 consecutive columns (16
            // bytes) of rows l / 4 and l / 4 + 8 of the pass, so one 16-byte access
            // of the warp covers 64 bytes of 8 rows.  (With a row per lane, as
            // 32x32b loads give it, each access touched 32 rows; the L1 then spent
            // 7 700 of a tile's cycles on them, which the MMAs need to fetch
            // operands: 8.18 ms against 7.60 on the 63 005-profile triangle.)
            const int i0 = r0 + bi * PM + (int)rank * BM + q * 32;  // the warp's first row
            const int j0 = c0 + bj * BN;
            const int c_begin = half * WARP_CHUNKS, c_end = half ? CHUNKS : WARP_CHUNKS;
            const int quad = lane & 3, lrow = lane >> 2;
            // a chunk with no cell above the diagonal is skipped
            const int j_min = tri ? i0 + 2 - CHUNK : INT_MIN;
            // columns of this tile and set: [j0, j_end)
            const int j_end = min(n, j0 + BN);
            // the rare counts, fetched while the MMAs of the tile run; a row of the
            // block is at least up(n - c0, 8) wide, so a live 16 bytes is in bounds.
            // Plain loads: the kernel that writes the block may still run when this
            // one starts, and the read-only path (ld.global.nc, __ldg) may only be
            // used on what nobody writes while a kernel runs.
            uint4 r4[WARP_CHUNKS][4];
#pragma unroll
            for (int cc = 0; cc < WARP_CHUNKS; cc++) {
                const int cb = j0 + (c_begin + cc) * CHUNK, j = cb + 8 * quad;
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    const int i = i0 + 8 * g + lrow;
                    r4[cc][g] = make_uint4(0, 0, 0, 0);
                    if (dense && c_begin + cc < c_end && cb >= j_min && i < iend && j < j_end)
                        r4[cc][g] = *reinterpret_cast<const uint4*>(rdense + (size_t)(i - r0) * ldr + (j - c0));
                }
            }
            if (!mbar_wait(&tfull[acc], aph, abort_flag, p.err)) break;
            tc_fence_after();
            const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * ACC_STRIDE);
#pragma unroll
            for (int cc = 0; cc < WARP_CHUNKS; cc++) {
                const int c = c_begin + cc;
                const int cb = j0 + c * CHUNK;  // first column of the chunk
                const bool skip = c >= c_end || cb < j_min || cb >= j_end;  // uniform over the warp
                uint32_t v[2][16];
                if (!skip) {
                    tmem_ld_16x256b_x4(tbase + (uint32_t)(c * CHUNK), v[0]);
                    tmem_ld_16x256b_x4(tbase + (16u << 16) + (uint32_t)(c * CHUNK), v[1]);
                    tmem_wait_ld();
                }
                if (cc == WARP_CHUNKS - 1) {  // this warp's part of the accumulator is read: hand it back
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(peer_addr(&tempty[acc], 0));
                }
                if (skip) continue;
                const int j = cb + 8 * quad;
#pragma unroll
                for (int g = 0; g < 4; g++) {  // rows 8 g + l / 4 of the warp's 32
                    const int i = i0 + 8 * g + lrow;
                    uint32_t w[4];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        bool odd = false;
                        w[r] = pack_u16(v[g / 2][4 * r + 2 * (g & 1)], v[g / 2][4 * r + 2 * (g & 1) + 1], &odd);
                        bad |= odd && cb + 8 * r < j0 + BN;  // columns past BN are not this accumulator's
                    }
                    quad_transpose(w, quad);
                    const uint4 rr = r4[cc][g];
                    w[0] = __vsub2(w[0], rr.x);
                    w[1] = __vsub2(w[1], rr.y);
                    w[2] = __vsub2(w[2], rr.z);
                    w[3] = __vsub2(w[3], rr.w);
                    if (i >= iend || j >= j_end) continue;
                    uint16_t* dst = out + (size_t)(i - r0) * ldo + (j - c0);
                    if (vec_store && j + 8 <= n) {
                        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; e += 2) {
                            if (j + e + 1 < n) *reinterpret_cast<uint32_t*>(dst + e) = w[e / 2];
                            else if (j + e < n) dst[e] = (uint16_t)w[e / 2];
                        }
                    }
                }
            }
            if (++acc == 2) acc = 0, aph ^= 1;
        }
        if (bad) atomicOr(p.err, DEVERR_OVERFLOW);
    }

    // neither CTA leaves (or frees TMEM) while the other may still use its
    // barriers, its operand stages or its accumulators
    tc_fence_before();
    __syncwarp();
    cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        if (PAIR)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS)
                         : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS)
                         : "memory");
    }
}

// ---------------------------------------------------------------- host side
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

// rows x kb bytes, boxes of 128 bytes of K x box_rows rows, 128-byte swizzle.
bool make_map(CUtensorMap* m, const uint8_t* X, size_t rows, int kb, int box_rows) {
    auto fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)kb, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)kb};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)X, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool same_chunking(const KChunks& x, const KChunks& y) { return x.n == y.n && x.width == y.width && x.kb == y.kb; }

// Shared memory of one CTA, and the smallest configuration of it: left to itself
// a launch beside the rare counts' tail stays in theirs (228 KB).
template <bool MULTI, bool PAIR, int STAGES>
cudaError_t set_attributes() {
    constexpr int bytes = smem_bytes(PAIR, STAGES);
    const auto kernel = tc_stripe_kernel<MULTI, PAIR, STAGES>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    constexpr int kPercent = (100 * (bytes + 1024) + 228 * 1024 - 1) / (228 * 1024);
    return cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, kPercent);
}

// Whether `tiles` tiles of one row block of at most 128 rows go to CTAs by
// themselves.  Half of a pair's rows would be padding; a CTA alone takes about half
// as long again per tile (46 KB a stage, at the 64 bytes a cycle that an SM takes in
// from L2), but twice as many run at a time.  Stripes of 64 rows, pairs and single
// CTAs: 6 000 columns, 169 stages 0.063 and 0.085 ms (25 tiles), 20 000, 303 stages
// 0.202 and 0.154 (84), 33 000, 365 stages 0.256 and 0.241 (138), 40 000, 388 stages
// 0.388 and 0.427 (167), 63 005, 440 stages 0.592 and 0.540 (263).
bool one_cta(int tiles, int num_sms) {
    auto waves = [&](int at_a_time) { return (tiles + at_a_time - 1) / std::max(at_a_time, 1); };
    return 3 * waves(num_sms) < 2 * waves(std::max(num_sms / 2, 1));
}

cudaError_t launch_one(const Fp4Operands& A, const Fp4Operands& B, const uint16_t* R, size_t ldr,
                       const StripeArgs& a, int num_sms, cudaStream_t st) {
    static bool attrs[kMaxDevices] = {};
    const int dev = current_device();
    if (!attrs[dev]) {
        cudaError_t e = set_attributes<false, true, FEW_STAGES>();
        if (e == cudaSuccess) e = set_attributes<false, true, ALL_STAGES>();
        if (e == cudaSuccess) e = set_attributes<false, false, ONE_STAGES>();
        if (e != cudaSuccess) return e;
        attrs[dev] = true;
    }
    const KChunks& ka = A.pos;
    const KChunks& kb = B.neg;
    if (A.kb <= 0 || (A.kb % BK) || B.kb != A.kb) return cudaErrorInvalidValue;
    if (ka.n < 1 || ka.kb != A.kb || !same_chunking(ka, kb) || (ka.width % BK)) return cudaErrorInvalidValue;
    if ((a.ldo & 1) || ((uintptr_t)a.out & 3)) return cudaErrorInvalidValue;
    if (R && ((ldr & 7) || ((uintptr_t)R & 15))) return cudaErrorInvalidValue;
    TcMaps maps;
    TcParams p;
    maps.n = ka.n;
    for (int c = 0; c < ka.n; c++) {
        const int wc = ka.width_of(c);
        if (wc <= 0 || (wc % BK)) return cudaErrorInvalidValue;
        if (!make_map(&maps.a[c], ka.p[c], A.n_rows, wc, BM) || !make_map(&maps.b[c], kb.p[c], B.n_rows, wc, BH))
            return cudaErrorInvalidValue;
        maps.kblocks[c] = wc / BK;
    }
    p.n = a.n;
    p.r0 = a.r0;
    p.c0 = a.rect ? 0 : a.r0;
    p.rows = a.rows;
    p.kblocks = A.kb / BK;
    p.ts.gs = pair_group(a.group);
    p.ts.nbi = (a.rows + PM - 1) / PM;
    p.ts.rect = a.rect ? 1 : 0;
    p.ts.nbj = (a.n - p.c0 + BN - 1) / BN;
    const long long tiles = tiles_in(p.ts, 0, p.ts.nbi);
    if (tiles > INT32_MAX) return cudaErrorInvalidValue;
    p.num_tiles = (int)tiles;
    {
        const int gs = p.ts.gs;
        p.gt.ngroups = (p.ts.nbi + gs - 1) / gs;
        if (p.gt.ngroups > MAX_GROUPS) return cudaErrorInvalidValue;  // callers split taller stripes
        long long acc = 0;
        for (int g = 0; g < p.gt.ngroups; g++) {
            p.gt.first[g] = (int)acc;
            acc += tiles_in(p.ts, g * gs, std::min(p.ts.nbi, g * gs + gs));
        }
        p.gt.first[p.gt.ngroups] = (int)acc;
    }
    p.rdense = R;
    p.ldr = ldr;
    p.out = a.out;
    p.ldo = a.ldo;
    p.vec_store = ((a.ldo & 7) == 0 && ((uintptr_t)a.out & 15) == 0) ? 1 : 0;
    p.err = a.err;
    p.jobs = nullptr;
    p.jmaps = nullptr;
    p.tiles = nullptr;
    p.first = nullptr;
    if (p.num_tiles == 0) return cudaSuccess;
    if (a.rows <= BM && one_cta(p.num_tiles, num_sms)) {
        const int grid = std::min(p.num_tiles, num_sms);
        return launch_after(a.after_counts, tc_stripe_kernel<false, false, ONE_STAGES>, dim3((unsigned)grid), THREADS,
                            smem_bytes(false, ONE_STAGES), st, maps, p);
    }
    const int grid = 2 * std::min(p.num_tiles, std::max(num_sms / 2, 1));
    const bool few = p.kblocks <= FEW_STAGES_K;
    return launch_after(a.after_counts,
                        few ? tc_stripe_kernel<false, true, FEW_STAGES> : tc_stripe_kernel<false, true, ALL_STAGES>,
                        dim3((unsigned)grid), THREADS, smem_bytes(true, few ? FEW_STAGES : ALL_STAGES), st, maps, p);
}

}  // namespace

// A batch's tiles over CTA pairs (or single CTAs): the sets with the most K stages
// per tile first, each tile to the pair with the least to do, so that the pairs end
// within one of the shortest tiles of one another and work on the same set at about
// the same time, which keeps its operand in L2 (one contiguous range of tiles per
// CTA, split by work, measured 43.1 ms against 34.1 on 512 sets).  48 sets of 57 to
// 4 576 profiles, 39 to 161 stages: 0.512 ms, with every npairs-th tile of the sets
// in turn 0.555; the stages alone take 0.437.  Returns the longest list's work, in K
// stages.
static long long spread_tiles(const std::vector<TcJob>& jobs, const std::vector<int>& tiles_of,
                              const std::vector<int>& which, int npairs, std::vector<int2>* tiles,
                              std::vector<int>* first) {
    std::vector<int> order = which;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return jobs[x].kblocks > jobs[y].kblocks; });
    typedef std::pair<long long, int> Load;  // stages so far, pair
    std::priority_queue<Load, std::vector<Load>, std::greater<Load>> least;
    for (int p = 0; p < npairs; p++) least.push(Load(0, p));
    std::vector<std::vector<int2>> mine((size_t)npairs);
    long long most = 0;
    for (int job : order)
        for (int t = 0; t < tiles_of[job]; t++) {
            Load l = least.top();
            least.pop();
            mine[l.second].push_back(make_int2(job, t));
            l.first += jobs[job].kblocks + kEpilogueStages;
            most = std::max(most, l.first);
            least.push(l);
        }
    tiles->clear();
    first->assign(1, 0);
    for (const std::vector<int2>& m : mine) {
        tiles->insert(tiles->end(), m.begin(), m.end());
        first->push_back((int)tiles->size());
    }
    return most;
}

cudaError_t tc_batch_prepare(const std::vector<TcBatchItem>& items, int num_sms, TcBatchPlan* plan, int* err) {
    std::vector<TcJob> jobs;
    std::vector<CUtensorMap> mh;
    std::vector<int> tiles_of;  // per job
    int num_tiles = 0;
    for (const TcBatchItem& it : items) {
        const Fp4Operands& A = *it.ops;
        if (it.n < 2) continue;
        const KChunks& ka = A.pos;
        const KChunks& kb = A.neg;
        if (A.kb <= 0 || (A.kb % BK) || ka.n < 1 || ka.kb != A.kb || !same_chunking(ka, kb) || (ka.width % BK))
            return cudaErrorInvalidValue;
        if ((it.ldo & 1) || ((uintptr_t)it.out & 3)) return cudaErrorInvalidValue;
        if (it.R && ((it.ldr & 7) || ((uintptr_t)it.R & 15))) return cudaErrorInvalidValue;
        TcJob jb = TcJob{};
        jb.n = it.n;
        jb.rows = it.n;
        jb.kblocks = A.kb / BK;
        jb.nchunks = ka.n;
        jb.map0 = (int)mh.size();
        for (int c = 0; c < ka.n; c++) {
            CUtensorMap m;
            if (!make_map(&m, ka.p[c], A.n_rows, ka.width_of(c), BM)) return cudaErrorInvalidValue;
            mh.push_back(m);
            jb.kbl[c] = ka.width_of(c) / BK;
        }
        for (int c = 0; c < ka.n; c++) {
            CUtensorMap m;
            if (!make_map(&m, kb.p[c], A.n_rows, kb.width_of(c), BH)) return cudaErrorInvalidValue;
            mh.push_back(m);
        }
        jb.ts.nbi = (it.n + PM - 1) / PM;
        jb.ts.nbj = (it.n + BN - 1) / BN;
        jb.ts.gs = jb.ts.nbi;
        jb.ts.rect = 0;
        jb.rdense = it.R;
        jb.ldr = it.ldr;
        jb.out = it.out;
        jb.ldo = it.ldo;
        jb.vec_store = ((it.ldo & 7) == 0 && ((uintptr_t)it.out & 15) == 0) ? 1 : 0;
        const long long tiles = tiles_in(jb.ts, 0, jb.ts.nbi);
        if ((long long)num_tiles + tiles > INT32_MAX) return cudaErrorInvalidValue;
        num_tiles += (int)tiles;
        tiles_of.push_back((int)tiles);
        jobs.push_back(jb);
    }
    tc_batch_release(plan);
    plan->err = err;
    plan->njobs = (int)jobs.size();
    plan->num_tiles = 0;
    if (jobs.empty()) return cudaSuccess;
    plan->num_tiles = num_tiles;
    // every tile on pairs, or those of the sets of one row block on CTAs by themselves
    // (see one_cta) in a launch of their own: 1 000 sets of 20 to 100 profiles 0.450 and
    // 0.359 ms with their counts, 600 of 50 to 128 0.351 and 0.292
    std::vector<int> all(jobs.size()), small, large;
    std::iota(all.begin(), all.end(), 0);
    for (int k : all) (jobs[k].n <= BM ? small : large).push_back(k);
    auto tiles_in_all = [&](const std::vector<int>& which) {
        int c = 0;
        for (int k : which) c += tiles_of[k];
        return c;
    };
    struct Part {
        std::vector<int2> tiles;
        std::vector<int> first;
    } part[2], split[2];
    auto spread = [&](const std::vector<int>& which, int at_a_time, Part* out) -> long long {
        const int c = tiles_in_all(which);
        return c ? spread_tiles(jobs, tiles_of, which, std::max(1, std::min(c, at_a_time)), &out->tiles, &out->first) : 0;
    };
    const long long pairs_only = spread(all, num_sms / 2, &part[0]);
    const long long apart = spread(large, num_sms / 2, &split[0]) + 3 * spread(small, num_sms, &split[1]) / 2 +
                            (large.empty() ? 0 : kLaunchStages);
    if (apart < pairs_only) part[0] = split[0], part[1] = split[1];
    cudaError_t e = device_alloc(&plan->d_jobs, jobs.size() * sizeof(TcJob));
    if (e == cudaSuccess) e = device_alloc(&plan->d_maps, mh.size() * sizeof(CUtensorMap));
    if (e == cudaSuccess) e = cudaMemcpy(plan->d_jobs, jobs.data(), jobs.size() * sizeof(TcJob), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(plan->d_maps, mh.data(), mh.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice);
    for (int q = 0; q < 2 && e == cudaSuccess; q++) {
        TcBatchPlan::Part& d = plan->part[q];
        d.lists = part[q].tiles.empty() ? 0 : (int)part[q].first.size() - 1;
        if (!d.lists) continue;
        e = device_alloc(&d.d_tiles, part[q].tiles.size() * sizeof(int2));
        if (e == cudaSuccess) e = device_alloc(&d.d_first, part[q].first.size() * sizeof(int));
        if (e == cudaSuccess)
            e = cudaMemcpy(d.d_tiles, part[q].tiles.data(), part[q].tiles.size() * sizeof(int2), cudaMemcpyHostToDevice);
        if (e == cudaSuccess)
            e = cudaMemcpy(d.d_first, part[q].first.data(), part[q].first.size() * sizeof(int), cudaMemcpyHostToDevice);
    }
    if (e != cudaSuccess) return e;
    static bool attrs[kMaxDevices] = {};
    const int dev = current_device();
    if (!attrs[dev]) {
        e = set_attributes<true, true, ALL_STAGES>();
        if (e == cudaSuccess) e = set_attributes<true, false, ONE_STAGES>();
        if (e != cudaSuccess) return e;
        attrs[dev] = true;
    }
    return cudaSuccess;
}

cudaError_t launch_tc_batch(const TcBatchPlan& plan, cudaStream_t st) {
    if (plan.num_tiles == 0 || plan.njobs == 0) return cudaSuccess;
    TcMaps maps;  // the batch's maps are in device memory
    maps.n = 0;
    TcParams p = TcParams{};
    p.gt.ngroups = 0;
    p.num_tiles = plan.num_tiles;
    p.err = plan.err;
    p.jobs = static_cast<const TcJob*>(plan.d_jobs);
    p.jmaps = static_cast<const CUtensorMap*>(plan.d_maps);
    // straight after the batch's rare counts; the sets of one row block after the others
    cudaError_t e = cudaSuccess;
    for (int q = 0; q < 2 && e == cudaSuccess; q++) {
        if (!plan.part[q].lists) continue;
        p.tiles = static_cast<const int2*>(plan.part[q].d_tiles);
        p.first = static_cast<const int*>(plan.part[q].d_first);
        if (q == 0)
            e = launch_after(true, tc_stripe_kernel<true, true, ALL_STAGES>, dim3((unsigned)(2 * plan.part[q].lists)),
                             THREADS, smem_bytes(true, ALL_STAGES), st, maps, p);
        else
            e = launch_after(true, tc_stripe_kernel<true, false, ONE_STAGES>, dim3((unsigned)plan.part[q].lists), THREADS,
                             smem_bytes(false, ONE_STAGES), st, maps, p);
    }
    return e;
}

void tc_batch_release(TcBatchPlan* plan) {
    if (plan->d_jobs) cudaFree(plan->d_jobs);
    if (plan->d_maps) cudaFree(plan->d_maps);
    for (TcBatchPlan::Part& d : plan->part) {
        if (d.d_tiles) cudaFree(d.d_tiles);
        if (d.d_first) cudaFree(d.d_first);
        d = TcBatchPlan::Part();
    }
    plan->d_jobs = plan->d_maps = nullptr;
    plan->njobs = plan->num_tiles = 0;
}

cudaError_t launch_tc_stripe(const Fp4Operands& ops, const Fp4Operands* bops, const uint16_t* R, size_t ldr,
                             const StripeArgs& a, int num_sms, cudaStream_t st) {
    if (a.rows <= 0 || (!a.rect && a.r0 >= a.n) || (a.rect && a.n <= 0)) return cudaSuccess;
    if (a.rect && !bops) return cudaErrorInvalidValue;
    const Fp4Operands& b = bops ? *bops : ops;
    // one launch covers at most MAX_GROUPS raster groups of rows; a taller
    // stripe runs as consecutive sub-stripes writing into the same output
    const int max_rows = MAX_GROUPS * pair_group(a.group) * PM;
    for (int done = 0; done < a.rows; done += max_rows) {
        StripeArgs s = a;
        s.r0 = a.r0 + done;
        s.rows = std::min(max_rows, a.rows - done);
        const size_t col = a.rect ? 0 : (size_t)done;  // a triangle's columns start at its first row
        s.out = a.out + (size_t)done * a.ldo + col;
        const uint16_t* Rs = R ? R + (size_t)done * ldr + col : nullptr;
        if (done) s.after_counts = false;  // the launch before is another part's
        const cudaError_t e = launch_one(ops, b, Rs, ldr, s, num_sms, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace tch
