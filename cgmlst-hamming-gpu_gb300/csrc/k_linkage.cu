// Consumers of the distance matrix on the device: the exact minimum spanning
// tree, single-linkage clusters at thresholds and every profile's nearest
// neighbours -- the uses the reference's documentation names for the matrix
// (outbreak clustering, minimum spanning trees, nearest-neighbour searches;
// docs/index.html, "The problem").  The reference stops at the matrix.
//
// Both read the full n x n u16 matrix in HBM row by row, a warp per row with
// 16-byte loads: a pass over the matrix is bound by HBM bandwidth (2 n^2 bytes).
//
// Minimum spanning tree (Borůvka).  Edges are ordered by (distance, smaller
// index, larger index), a strict order, so the tree is unique and equals
// Kruskal's under the same order.  One pass gives every row its 16 nearest
// columns; a round then needs only these lists, most of the time:
//   lists   a row's lightest edge out of its component is its first listed
//           column outside; one atomicMin folds it into the component's best
//           key.  A row whose listed columns all lie inside is exhausted: all
//           its other edges are at least as heavy as `beyond`, what its last
//           pass left out.
//   rescan  an exhausted row whose component's best so far is not below
//           `beyond` is read again, and its list becomes its nearest columns
//           outside, up to the component's best.  The largest component is left
//           out: all others hooking still halves their number, and a component
//           that takes no part this round loses nothing.
//   hook    every other component root across its best edge, recording it (of
//           two components that chose the same edge, only the larger root hooks,
//           which breaks the only cycles such a choice can make);
//   relabel pointers to the new roots, then every profile its new root.
// Each round at least halves the number of the other components, so at most
// ceil(log2 n) + 1 rounds.  No step waits on another thread.
//
// Nearest neighbours.  A warp per row reads the row once and keeps its k
// smallest (distance, column) keys in its lanes' registers.

#include <string.h>

#include <algorithm>
#include <numeric>
#include <vector>

#include "tch_internal.cuh"

namespace tch {
namespace {

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr int kNbrThreads = 256;
constexpr int kMaxNeighbors = 32;
constexpr int kIndexBits = 21;  // a profile index in an edge key
constexpr uint32_t kIndexMask = (1u << kIndexBits) - 1;
constexpr unsigned long long kNoEdge = ~0ull;
constexpr uint32_t kNoDistance = 0x10000u;  // above every u16 distance

enum LinkErr : int {
    LINKERR_EDGE = 1,     // a component's best edge does not leave it, or the edges leave profiles apart
    LINKERR_COUNT = 2,    // more than n - 1 tree edges
    LINKERR_SELECT = 4,   // the neighbour selection lost count
};

// (distance, smaller index, larger index) as one integer.
__device__ __forceinline__ unsigned long long edge_key(uint32_t w, uint32_t i, uint32_t j) {
    const uint32_t a = i < j ? i : j, b = i < j ? j : i;
    return ((unsigned long long)w << (2 * kIndexBits)) | ((unsigned long long)a << kIndexBits) | b;
}

// Value e (0..7) of eight u16 values packed in a uint4.
__device__ __forceinline__ uint32_t lane16(const uint4& h, int e) {
    const uint32_t x = e < 2 ? h.x : e < 4 ? h.y : e < 6 ? h.z : h.w;
    return (e & 1) ? x >> 16 : x & 0xFFFFu;
}

// ---- nearest neighbours: one warp per row, one pass over the row
//
// Lane r of the warp holds the r-th smallest key (distance << 32 | column) seen
// so far.  The row streams past in blocks of 1 024 columns (four 16-byte loads
// in flight per lane); eight values are tested against the k-th smallest
// distance with three packed minima, so nearly every value costs less than one
// instruction.  Hits go to a buffer of the warp in shared memory, and every 32
// of them are sorted across the lanes (bitonic) and merged into the list.
//
// Bound by the one read of the matrix.  40 009 profiles, k = 10: 0.84 ms
// for the call; the radix select before it (a CTA per row, three reads of the
// row, a warp match per value in two of them) took 9.5 ms.  In a row whose
// distances fall from column to column every value is a hit, and 32 of them cost a
// merge of about 200 instructions, so a block after a crowded one is bounded by
// its own values first: 60 000 such rows take 5.0 ms, 28.4 without that bound, 10.9
// in the radix select.

constexpr int kNbrWarps = kNbrThreads / 32;

// One compare-exchange step of a bitonic network over the lanes: the lane
// keeps the smaller (up) or larger of its key and its partner's.
__device__ __forceinline__ unsigned long long cmp_exchange(unsigned long long v, int d, bool up) {
    const unsigned long long t = __shfl_xor_sync(FULL, v, d);
    return (v < t) == up ? v : t;
}

// v sorted descending over the lanes.
__device__ __forceinline__ unsigned long long sort_descending(unsigned long long v, int lane) {
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
        for (int d = k >> 1; d; d >>= 1) v = cmp_exchange(v, d, ((lane & k) != 0) == ((lane & d) == 0));
    return v;
}

// The 32 smallest of an ascending list and 32 further keys, ascending.
__device__ __forceinline__ unsigned long long merge_keys(unsigned long long list, unsigned long long more, int lane) {
    const unsigned long long d = sort_descending(more, lane);
    unsigned long long v = d < list ? d : list;  // the smaller half, a bitonic sequence
#pragma unroll
    for (int s = 16; s; s >>= 1) v = cmp_exchange(v, s, (lane & s) == 0);
    return v;
}

// Distance of a list key, kNoDistance for an empty place.
__device__ __forceinline__ uint32_t key_distance(unsigned long long key) {
    return key == kNoEdge ? kNoDistance : (uint32_t)(key >> 32);
}

// The 32 nearest columns j != i of a row by (distance, column), in the lanes'
// order, as far as k of them (those of distance `thr` and above may be missing
// even so); with OUT only columns whose component is not `own`.
template <bool OUT>
__device__ __forceinline__ unsigned long long nearest_keys(const uint4* __restrict__ row, int n, int i, int k,
                                                           const uint32_t* __restrict__ comp, uint32_t own,
                                                           uint32_t thr, unsigned long long* buf, int lane) {
    const int nq = (n + 7) >> 3;
    unsigned long long list = kNoEdge;
    uint32_t held = 0;    // keys in the buffer
    bool crowded = true;  // bound the next block by its own values first
    for (int q0 = 0; q0 < nq; q0 += 128) {
        uint4 h[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int q = q0 + 32 * u + lane;
            h[u] = q < nq ? __ldcs(row + q) : make_uint4(FULL, FULL, FULL, FULL);
        }
        if (crowded) {
            // a bound from the block alone, in the first one and after one of many
            // hits: the k-th smallest of the 32 lanes' smallest valid values
            uint32_t m = 0xFFFFu;
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const int j = 8 * (q0 + 32 * u + lane) + e;
                    const uint32_t w = lane16(h[u], e);
                    if (w < m && j < n && j != i && (!OUT || __ldg(comp + j) != own)) m = w;
                }
            const unsigned long long s = sort_descending((unsigned long long)m, lane);
            thr = min(thr, (uint32_t)__shfl_sync(FULL, s, 32 - k) + 1u);  // at least k valid values lie below it
        }
        // every key in the list or the buffer comes from smaller columns, except
        // those of this block: a later value at the k-th distance is no hit
        const uint32_t start = thr;
        int merges = 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t m2 = __vminu2(__vminu2(h[u].x, h[u].y), __vminu2(h[u].z, h[u].w));
            if (!__any_sync(FULL, min(m2 & 0xFFFFu, m2 >> 16) < thr)) continue;
            const int j0 = 8 * (q0 + 32 * u + lane);
            uint32_t hits = 0;
#pragma unroll
            for (int e = 0; e < 8; e++)
                if (lane16(h[u], e) < thr && j0 + e < n && j0 + e != i && (!OUT || __ldg(comp + j0 + e) != own))
                    hits |= 1u << e;
            for (;;) {  // the lanes' first remaining hits, until none is left
                const unsigned who = __ballot_sync(FULL, hits != 0);
                if (!who) break;
                if (hits) {
                    const int e = __ffs(hits) - 1;
                    hits &= hits - 1;
                    uint32_t w = 0;
#pragma unroll
                    for (int f = 0; f < 8; f++) w = f == e ? lane16(h[u], f) : w;
                    buf[held + __popc(who & ((1u << lane) - 1u))] = ((unsigned long long)w << 32) | (uint32_t)(j0 + e);
                }
                held += __popc(who);
                if (held >= 32) {
                    held -= 32;
                    merges++;
                    __syncwarp();
                    list = merge_keys(list, buf[held + lane], lane);
                    __syncwarp();
                    const uint32_t kth = key_distance(__shfl_sync(FULL, list, k - 1));
                    thr = min(start, min(thr, kth + 1u));  // equal values of this block may still win on the column
                }
            }
        }
        const uint32_t kth = key_distance(__shfl_sync(FULL, list, k - 1));
        thr = min(thr, kth);
        crowded = merges > 1;
    }
    if (held) {
        __syncwarp();
        list = merge_keys(list, lane < (int)held ? buf[lane] : kNoEdge, lane);
    }
    return list;
}

// Row i's k nearest columns (j != i) by (distance, column).
__global__ void __launch_bounds__(kNbrThreads) neighbors_kernel(const uint16_t* __restrict__ H, size_t ld, int n,
                                                                int k, uint32_t* idx, uint16_t* dist, int* err) {
    __shared__ unsigned long long buffers[kNbrWarps][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * kNbrWarps + warp;
    if (i >= n) return;  // uniform over the warp; no block-wide step follows
    const unsigned long long list = nearest_keys<false>(reinterpret_cast<const uint4*>(H + (size_t)i * ld), n, i, k,
                                                        nullptr, 0, kNoDistance, buffers[warp], lane);
    if (lane < k) {
        if (list == kNoEdge) atomicOr(err, LINKERR_SELECT);
        idx[(size_t)i * k + lane] = (uint32_t)list;
        dist[(size_t)i * k + lane] = (uint16_t)(list >> 32);
    }
}

// ---- minimum spanning tree ---------------------------------------------------

// Columns listed per row.  8, 16 and 32 of them: 1.49, 1.52 and 1.64 ms for the
// tree of 30 011 profiles in clusters of about 40, 0.99, 1.03 and 1.10 ms for
// long-tail profiles, 0.57, 0.53 and 0.54 for 5 003 small ones.
constexpr int kListed = 16;

// Scalars of a run, and what the host reads after a round.
struct MstState {
    unsigned long long largest;  // size << 32 | ~root of the largest component (the first of equal ones)
    unsigned long long total;    // sum of the edges' distances
    unsigned int nedges;
    int err;
};

// Every profile its own component, and every row its list.
__global__ void __launch_bounds__(kNbrThreads)
    mst_lists_kernel(const uint16_t* __restrict__ H, size_t ld, int n, unsigned long long* lists, uint32_t* beyond,
                     uint32_t* comp, uint32_t* size) {
    __shared__ unsigned long long buffers[kNbrWarps][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * kNbrWarps + warp;
    if (i >= n) return;
    const int k = min(kListed, n - 1);
    const unsigned long long list = nearest_keys<false>(reinterpret_cast<const uint4*>(H + (size_t)i * ld), n, i, k,
                                                        nullptr, 0, kNoDistance, buffers[warp], lane);
    if (lane < kListed) lists[(size_t)i * kListed + lane] = lane < k ? list : kNoEdge;
    const uint32_t last = key_distance(__shfl_sync(FULL, list, kListed - 1));
    if (lane == 0) {
        beyond[i] = n - 1 <= kListed ? kNoDistance : last;
        comp[i] = (uint32_t)i;
        size[i] = 1;
    }
}

// best[c] = the lightest listed edge out of component c; exhausted[i] = 1 for
// a row with none; the largest component's root.
__global__ void __launch_bounds__(256)
    mst_best_kernel(int n, const unsigned long long* __restrict__ lists, const uint32_t* __restrict__ comp,
                    const uint32_t* __restrict__ size, unsigned long long* best, uint8_t* exhausted,
                    MstState* state) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const uint32_t own = comp[i];
    const unsigned long long key = lane < kListed ? lists[(size_t)i * kListed + lane] : kNoEdge;
    const bool out = key != kNoEdge && comp[(uint32_t)key] != own;
    const unsigned who = __ballot_sync(FULL, out);
    if (who && lane == __ffs(who) - 1)
        atomicMin(best + own, edge_key((uint32_t)(key >> 32), (uint32_t)i, (uint32_t)key));
    if (lane == 0) {
        exhausted[i] = who ? 0 : 1;
        if (own == (uint32_t)i) {
            const unsigned long long mine = (unsigned long long)size[i] << 32 | ~(uint32_t)i;
            if (mine > *(volatile unsigned long long*)&state->largest) atomicMax(&state->largest, mine);
        }
    }
}

// Exhausted rows that their component's best does not rule out are read again.
__global__ void __launch_bounds__(kNbrThreads)
    mst_rescan_kernel(const uint16_t* __restrict__ H, size_t ld, int n, unsigned long long* lists, uint32_t* beyond,
                      const uint32_t* __restrict__ comp, const uint8_t* __restrict__ exhausted,
                      unsigned long long* best, const MstState* state) {
    __shared__ unsigned long long buffers[kNbrWarps][64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * kNbrWarps + warp;
    if (i >= n || !exhausted[i]) return;
    const uint32_t own = comp[i], floor = beyond[i];
    if (own == ~(uint32_t)state->largest || floor >= kNoDistance) return;
    // the best only falls while rows of the component are read: any value of it
    // rules out what is heavier
    const unsigned long long b = __shfl_sync(FULL, *(volatile unsigned long long*)(best + own), 0);
    const uint32_t limit = b == kNoEdge ? kNoDistance : (uint32_t)(b >> (2 * kIndexBits)) + 1u;
    if (floor >= limit) return;  // every edge that is not listed is heavier than the best
    const unsigned long long list = nearest_keys<true>(reinterpret_cast<const uint4*>(H + (size_t)i * ld), n, i,
                                                       kListed, comp, own, limit, buffers[warp], lane);
    if (lane < kListed) lists[(size_t)i * kListed + lane] = list;
    const uint32_t last = key_distance(__shfl_sync(FULL, list, kListed - 1));
    if (lane == 0) {
        beyond[i] = min(limit, last);
        if (list != kNoEdge) atomicMin(best + own, edge_key((uint32_t)(list >> 32), (uint32_t)i, (uint32_t)list));
    }
}

// parent[c] = the root that c hooks to this round (c itself when it does not).
__global__ void mst_hook_kernel(int n, const uint32_t* __restrict__ comp, const unsigned long long* __restrict__ best,
                                uint32_t* parent, uint32_t* size, unsigned long long* edges, MstState* state) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    uint32_t p = (uint32_t)c;
    const uint32_t largest = ~(uint32_t)state->largest;
    const unsigned long long key = c < n ? best[c] : kNoEdge;
    bool hooks = false;
    if (c < n && comp[c] == (uint32_t)c && key != kNoEdge && (uint32_t)c != largest) {
        const uint32_t u = (uint32_t)(key >> kIndexBits) & kIndexMask, v = (uint32_t)key & kIndexMask;
        if (u >= (uint32_t)n || v >= (uint32_t)n) {
            atomicOr(&state->err, LINKERR_EDGE);
        } else {
            const uint32_t cu = comp[u], cv = comp[v];
            const uint32_t d = cu == (uint32_t)c ? cv : cu;
            if ((cu != (uint32_t)c && cv != (uint32_t)c) || d == (uint32_t)c || d >= (uint32_t)n) {
                atomicOr(&state->err, LINKERR_EDGE);
            } else if (!(best[d] == key && d != largest && (uint32_t)c < d)) {
                p = d;
                hooks = true;
            }
        }
    }
    const unsigned who = __ballot_sync(FULL, hooks);
    if (who) {  // one atomic per warp
        const uint32_t sum = __reduce_add_sync(FULL, hooks ? (uint32_t)(key >> (2 * kIndexBits)) : 0u);
        unsigned int slot = 0;
        if (lane == 0) {
            slot = atomicAdd(&state->nedges, (unsigned int)__popc(who));
            atomicAdd(&state->total, (unsigned long long)sum);
        }
        slot = __shfl_sync(FULL, slot, 0) + (unsigned int)__popc(who & ((1u << lane) - 1u));
        if (hooks) {
            if (slot < (unsigned int)(n - 1)) edges[slot] = key;
            else atomicOr(&state->err, LINKERR_COUNT);
        }
    }
    if (c >= n) return;
    size[c] = 0;  // counted anew by the relabelling
    parent[c] = p;
}

// Every pointer straight to its root: all threads shorten their chains at once,
// each step taking whatever the others have made of its parent so far, so a
// chain of length l takes about log2 l steps; pointers only ever move rootwards.
__global__ void mst_jump_kernel(int n, volatile uint32_t* parent) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= n) return;
    for (uint32_t p = parent[x];;) {
        const uint32_t g = parent[p];
        if (g == p) break;
        parent[x] = p = g;
    }
}

__global__ void mst_relabel_kernel(int n, uint32_t* comp, const uint32_t* __restrict__ parent, uint32_t* size) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t c = x < n ? parent[comp[x]] : FULL;
    if (x < n) comp[x] = c;
    const unsigned peers = __match_any_sync(FULL, c);
    if (x < n && (threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(size + c, (uint32_t)__popc(peers));
}

// The edges in order: counted by distance, gathered there, and placed among the
// edges of the same distance by counting the smaller keys, a warp per edge.
// (Counting against every edge took 0.13 ms for 30 010 of them, this 0.045; the
// host's sort 1.2 with its checks.)  Where more than kManyEqual edges have one
// distance, as among duplicates, that count would be quadratic: chunks of kChunk
// keys are sorted first, and an edge searches each of its distance's chunks.
// (100 000 profiles that differ by 1 along a path: 4.31 ms for the tree, 6.83 by
// counting alone.)
//
// Trees of at most kHostOrder edges are ordered on the host, which takes less than
// these launches and their copies: 100 / 1 024 profiles 0.320 / 0.368 ms, on the
// device 0.387 / 0.404; from about 1 300 profiles on the two are alike.
constexpr int kDistances = 65536;
constexpr int kChunk = 1024, kManyEqual = 4096;
constexpr size_t kHostOrder = 1024;
static_assert(kManyEqual > kChunk, "such a distance holds the first or the last key of every chunk it enters");

__global__ void mst_count_kernel(int m, const unsigned long long* __restrict__ edges, uint32_t* count) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < m) atomicAdd(count + (edges[e] >> (2 * kIndexBits)), 1u);
}

// count -> exclusive sums (kDistances + 1 of them) and a copy to fill from; one
// CTA, each warp 2 048 counts, 128 at a time.
__global__ void __launch_bounds__(1024) mst_sum_kernel(uint32_t* count, uint32_t* fill) {
    __shared__ uint32_t warp_sum[32];
    constexpr int kSteps = kDistances / 32 / 128;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4* c4 = reinterpret_cast<uint4*>(count) + warp * (kDistances / 32 / 4) + lane;
    uint4* f4 = reinterpret_cast<uint4*>(fill) + warp * (kDistances / 32 / 4) + lane;
    uint4 v[kSteps];
    uint32_t sum = 0;
#pragma unroll
    for (int q = 0; q < kSteps; q++) v[q] = c4[32 * q];
#pragma unroll
    for (int q = 0; q < kSteps; q++) sum += v[q].x + v[q].y + v[q].z + v[q].w;
    sum = __reduce_add_sync(FULL, sum);
    if (lane == 0) warp_sum[warp] = sum;
    __syncthreads();
    uint32_t before = __reduce_add_sync(FULL, lane < warp ? warp_sum[lane] : 0u);
#pragma unroll
    for (int q = 0; q < kSteps; q++) {
        const uint32_t mine = v[q].x + v[q].y + v[q].z + v[q].w;
        uint32_t inc = mine;
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t t = __shfl_up_sync(FULL, inc, d);
            if (lane >= d) inc += t;
        }
        uint4 s;
        s.x = before + inc - mine;
        s.y = s.x + v[q].x;
        s.z = s.y + v[q].y;
        s.w = s.z + v[q].z;
        c4[32 * q] = s;
        f4[32 * q] = s;
        before += __shfl_sync(FULL, inc, 31);
    }
    if (threadIdx.x == 1023) count[kDistances] = before;
}

__global__ void mst_gather_kernel(int m, const unsigned long long* __restrict__ edges, uint32_t* fill,
                                  unsigned long long* out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < m) out[atomicAdd(fill + (edges[e] >> (2 * kIndexBits)), 1u)] = edges[e];
}

// Ascending, in place: the chunks that hold keys of a distance of many edges.
__global__ void __launch_bounds__(kChunk / 2)
    mst_chunk_kernel(int m, unsigned long long* keys, const uint32_t* __restrict__ first) {
    __shared__ unsigned long long k[kChunk];
    const int begin = blockIdx.x * kChunk, end = min(m, begin + kChunk), t = threadIdx.x;
    const uint32_t a = (uint32_t)(keys[begin] >> (2 * kIndexBits)), b = (uint32_t)(keys[end - 1] >> (2 * kIndexBits));
    if (max(first[a + 1] - first[a], first[b + 1] - first[b]) <= (uint32_t)kManyEqual) return;  // uniform
    for (int e = t; e < kChunk; e += kChunk / 2) k[e] = begin + e < end ? keys[begin + e] : kNoEdge;
    for (int size = 2; size <= kChunk; size <<= 1)
        for (int d = size >> 1; d; d >>= 1) {
            __syncthreads();
            const int x = 2 * t - (t & (d - 1)), y = x + d;
            const unsigned long long kx = k[x], ky = k[y];
            if ((kx > ky) == ((x & size) == 0)) k[x] = ky, k[y] = kx;
        }
    __syncthreads();
    for (int e = t; e < kChunk; e += kChunk / 2)
        if (begin + e < end) keys[begin + e] = k[e];
}

// The edges decoded at their places.  Also checks that the relabelling left one
// component (with n - 1 edges, a tree).
__global__ void __launch_bounds__(256)
    mst_decode_kernel(int n, const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ first,
                      const uint32_t* __restrict__ comp, uint32_t* u, uint32_t* v, uint16_t* w, MstState* state) {
    const int lane = threadIdx.x & 31, e = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (e >= n) return;
    if (lane == 0 && comp[e] != comp[0]) atomicOr(&state->err, LINKERR_EDGE);
    if (e == n - 1) return;
    const unsigned long long key = keys[e];
    const uint32_t d = (uint32_t)(key >> (2 * kIndexBits)), begin = first[d], end = first[d + 1];
    uint32_t smaller = 0;
    if (end - begin <= (uint32_t)kManyEqual) {
        for (uint32_t t = begin + lane; t < end; t += 32) smaller += keys[t] < key;
    } else {  // a chunk per lane, sorted by mst_chunk_kernel
        for (uint32_t c = begin / kChunk + lane; c * kChunk < end; c += 32) {
            const uint32_t from = max(begin, c * kChunk);
            uint32_t lo = from, hi = min(end, (c + 1) * kChunk);
            while (lo < hi) {
                const uint32_t mid = (lo + hi) / 2;
                if (keys[mid] < key) lo = mid + 1; else hi = mid;
            }
            smaller += lo - from;
        }
    }
    const uint32_t at = begin + __reduce_add_sync(FULL, smaller);
    if (lane == 0) {
        u[at] = (uint32_t)(key >> kIndexBits) & kIndexMask;
        v[at] = (uint32_t)key & kIndexMask;
        w[at] = (uint16_t)d;
    }
}

// The same on the host, for small trees.
int order_on_host(int n, std::vector<unsigned long long>& keys, uint32_t* u, uint32_t* v, uint16_t* w, Err& e) {
    std::sort(keys.begin(), keys.end());
    std::vector<uint32_t> p((size_t)n);  // the edges must join every profile: n - 1 unions
    std::iota(p.begin(), p.end(), 0u);
    auto find = [&](uint32_t x) {
        while (p[x] != x) x = p[x] = p[p[x]];
        return x;
    };
    for (size_t q = 0; q < keys.size(); q++) {
        const uint32_t i = (uint32_t)(keys[q] >> kIndexBits) & kIndexMask, j = (uint32_t)keys[q] & kIndexMask;
        const uint32_t a = find(i), b = find(j);
        if (a == b) return e.set("minimum spanning tree: device check failed (code %d)", LINKERR_EDGE);
        p[std::max(a, b)] = std::min(a, b);
        if (u) u[q] = i;
        if (v) v[q] = j;
        if (w) w[q] = (uint16_t)(keys[q] >> (2 * kIndexBits));
    }
    return 0;
}

int check_matrix(const uint16_t* d_H, size_t ld, int n, Err& e) {
    if (n < 0) return e.set("n must be >= 0");
    if (n >= (1 << kIndexBits)) return e.set("n must be below %d", 1 << kIndexBits);
    if (n > 0 && !d_H) return e.set("null matrix");
    if (ld < (size_t)n || (ld & 7)) return e.set("ld must be >= n and a multiple of 8");
    if ((uintptr_t)d_H & 15) return e.set("the matrix must be 16-byte aligned");
    return 0;
}

int mst_on_device(const uint16_t* d_H, size_t ld, int n, cudaStream_t st, uint32_t* u, uint32_t* v, uint16_t* w,
                  uint64_t* total, Err& e) {
    if (total) *total = 0;
    if (check_matrix(d_H, ld, n, e)) return 1;
    if (n < 2) return 0;
    const size_t m = (size_t)n - 1;
    char* ws = nullptr;
    unsigned long long *lists, *best, *edges;
    uint32_t *comp, *parent, *size, *beyond, *d_u, *d_v, *count;
    uint16_t* d_w;
    uint8_t* exhausted;
    MstState* state;
    MstState got = {};
    int rc = 1;
    unsigned int prev = 0;
    const int steps = 32 - __builtin_clz((unsigned)(n - 1)) + 1;  // ceil(log2 n) + 1
    const unsigned rows_grid = (unsigned)((n + kNbrWarps - 1) / kNbrWarps), vgrid = (unsigned)((n + 255) / 256);
    const size_t n8 = up((size_t)n, 8);
    // the lists' room (128 bytes a profile) serves the gathered edges afterwards
    const size_t bytes = sizeof(MstState) + n8 * (8 * kListed + 8 + 8 + 4 * 4 + 4 + 4 + 2 + 1) + 16 +
                         ((size_t)2 * kDistances + 4) * 4;
    TCH_CK(e, pool_alloc(&ws, bytes, nullptr, st));
    lists = reinterpret_cast<unsigned long long*>(ws);
    best = lists + n8 * kListed;
    edges = best + n8;
    state = reinterpret_cast<MstState*>(edges + n8);
    comp = reinterpret_cast<uint32_t*>(state + 1);
    parent = comp + n8;
    size = parent + n8;
    beyond = size + n8;
    d_u = beyond + n8;
    d_v = d_u + n8;
    d_w = reinterpret_cast<uint16_t*>(d_v + n8);
    exhausted = reinterpret_cast<uint8_t*>(d_w + n8);
    count = reinterpret_cast<uint32_t*>(ws + up((size_t)(reinterpret_cast<char*>(exhausted + n8) - ws), 16));
    TCH_CK(e, cudaMemsetAsync(state, 0, sizeof(MstState), st));
    mst_lists_kernel<<<rows_grid, kNbrThreads, 0, st>>>(d_H, ld, n, lists, beyond, comp, size);
    TCH_CK(e, cudaGetLastError());
    // each round at least halves the other components: ceil(log2 n) + 1 rounds at most
    for (int round = 0; got.nedges < m; round++) {
        if (round > steps) {
            e.set("minimum spanning tree: %u of %zu edges after %d rounds", got.nedges, m, round);
            goto fail;
        }
        TCH_CK(e, cudaMemsetAsync(best, 0xFF, (size_t)n * 8, st));
        TCH_CK(e, cudaMemsetAsync(&state->largest, 0, 8, st));
        mst_best_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(n, lists, comp, size, best, exhausted, state);
        mst_rescan_kernel<<<rows_grid, kNbrThreads, 0, st>>>(d_H, ld, n, lists, beyond, comp, exhausted, best, state);
        mst_hook_kernel<<<vgrid, 256, 0, st>>>(n, comp, best, parent, size, edges, state);
        mst_jump_kernel<<<vgrid, 256, 0, st>>>(n, parent);
        mst_relabel_kernel<<<vgrid, 256, 0, st>>>(n, comp, parent, size);
        TCH_CK(e, cudaGetLastError());
        TCH_CK(e, cudaMemcpyAsync(&got, state, sizeof(got), cudaMemcpyDeviceToHost, st));
        TCH_CK(e, cudaStreamSynchronize(st));
        if (got.err) {
            e.set("minimum spanning tree: device check failed (code %d)", got.err);
            goto fail;
        }
        if (got.nedges == prev) {
            e.set("minimum spanning tree: no edge added in round %d", round);
            goto fail;
        }
        prev = got.nedges;
    }
    if (m <= kHostOrder) {
        std::vector<unsigned long long> keys(m);
        TCH_CK(e, cudaMemcpyAsync(keys.data(), edges, m * 8, cudaMemcpyDeviceToHost, st));
        TCH_CK(e, cudaStreamSynchronize(st));
        if (order_on_host(n, keys, u, v, w, e)) goto fail;
        if (total) *total = got.total;
        rc = 0;
        goto fail;  // the workspace goes back
    }
    {
        uint32_t* fill = count + kDistances + 4;
        unsigned long long* keys = lists;
        TCH_CK(e, cudaMemsetAsync(count, 0, (size_t)kDistances * 4, st));
        mst_count_kernel<<<vgrid, 256, 0, st>>>((int)m, edges, count);
        mst_sum_kernel<<<1, 1024, 0, st>>>(count, fill);
        mst_gather_kernel<<<vgrid, 256, 0, st>>>((int)m, edges, fill, keys);
        mst_chunk_kernel<<<(unsigned)((m + kChunk - 1) / kChunk), kChunk / 2, 0, st>>>((int)m, keys, count);
        mst_decode_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(n, keys, count, comp, d_u, d_v, d_w, state);
        TCH_CK(e, cudaGetLastError());
    }
    if (u) TCH_CK(e, cudaMemcpyAsync(u, d_u, m * 4, cudaMemcpyDeviceToHost, st));
    if (v) TCH_CK(e, cudaMemcpyAsync(v, d_v, m * 4, cudaMemcpyDeviceToHost, st));
    if (w) TCH_CK(e, cudaMemcpyAsync(w, d_w, m * 2, cudaMemcpyDeviceToHost, st));
    TCH_CK(e, cudaMemcpyAsync(&got, state, sizeof(got), cudaMemcpyDeviceToHost, st));
    TCH_CK(e, cudaStreamSynchronize(st));
    if (got.err) {
        e.set("minimum spanning tree: device check failed (code %d)", got.err);
        goto fail;
    }
    if (total) *total = got.total;
    rc = 0;
fail:
    if (ws) {
        cudaFreeAsync(ws, st);
        cudaStreamSynchronize(st);
    }
    return rc;
}

int neighbors_on_device(const uint16_t* d_H, size_t ld, int n, int k, cudaStream_t st, uint32_t* idx,
                        uint16_t* dist, Err& e) {
    if (check_matrix(d_H, ld, n, e)) return 1;
    if (k < 1 || k > kMaxNeighbors) return e.set("k must be 1-%d", kMaxNeighbors);
    if (k >= n) return e.set("k must be below n (%d)", n);
    if (!idx || !dist) return e.set("null output");
    char* ws = nullptr;
    uint32_t* d_idx;
    uint16_t* d_dist;
    int* derr;
    int rc = 1, herr = 0;
    const size_t cells = (size_t)n * k;
    TCH_CK(e, pool_alloc(&ws, cells * 6 + 64, nullptr, st));
    d_idx = reinterpret_cast<uint32_t*>(ws);
    derr = reinterpret_cast<int*>(d_idx + cells);
    d_dist = reinterpret_cast<uint16_t*>(derr + 4);
    TCH_CK(e, cudaMemsetAsync(derr, 0, 4, st));
    neighbors_kernel<<<(n + kNbrWarps - 1) / kNbrWarps, kNbrThreads, 0, st>>>(d_H, ld, n, k, d_idx, d_dist, derr);
    TCH_CK(e, cudaGetLastError());
    TCH_CK(e, cudaMemcpyAsync(idx, d_idx, cells * 4, cudaMemcpyDeviceToHost, st));
    TCH_CK(e, cudaMemcpyAsync(dist, d_dist, cells * 2, cudaMemcpyDeviceToHost, st));
    TCH_CK(e, cudaMemcpyAsync(&herr, derr, 4, cudaMemcpyDeviceToHost, st));
    TCH_CK(e, cudaStreamSynchronize(st));
    if (herr) {
        e.set("nearest neighbours: device check failed (code %d)", herr);
        goto fail;
    }
    rc = 0;
fail:
    if (ws) {
        cudaFreeAsync(ws, st);
        cudaStreamSynchronize(st);
    }
    return rc;
}

// The solver's full matrix in device memory (upper triangle, then mirrored).
int full_matrix(tch_solver* s, int* n_out, uint16_t** H, size_t* ld, cudaStream_t st, char* err, int errlen) {
    Err e{err, errlen};
    tch_info info;
    *H = nullptr;
    if (!s || tch_solver_info(s, &info)) return e.set("bad solver");
    const int n = info.n;
    *n_out = n;
    *ld = up((size_t)std::max(n, 1), 8);
    if (n < 2) return 0;
    if (device_alloc(H, (size_t)n * *ld * 2) != cudaSuccess) {
        cudaGetLastError();
        *H = nullptr;
        return e.set("the full %d x %d matrix (%.1f GB) does not fit in device memory", n, n,
                     (double)n * *ld * 2 / 1e9);
    }
    if (tch_solver_stripe(s, 0, n, *H, *ld, st, err, errlen)) goto fail;
    TCH_CK(e, launch_mirror(*H, *ld, n, st));
    TCH_CK(e, cudaStreamSynchronize(st));
    if (tch_solver_check(s, err, errlen)) goto fail;
    return 0;
fail:
    cudaStreamSynchronize(st);
    cudaFree(*H);
    *H = nullptr;
    return 1;
}

struct StreamGuard {
    cudaStream_t st = nullptr;
    bool own = false;
    int make(void* stream) {
        if (stream) {
            st = (cudaStream_t)stream;
            return 0;
        }
        own = true;
        return cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess;
    }
    ~StreamGuard() {
        if (own && st) cudaStreamDestroy(st);
    }
};

}  // namespace
}  // namespace tch

using namespace tch;

extern "C" int tch_mst_device(const uint16_t* d_H, size_t ld, int n, void* stream, uint32_t* u, uint32_t* v,
                              uint16_t* w, uint64_t* total, char* err, int errlen) {
    Err e{err, errlen};
    StreamGuard g;
    if (g.make(stream)) return e.set("could not create a stream");
    return mst_on_device(d_H, ld, n, g.st, u, v, w, total, e);
}

extern "C" int tch_neighbors_device(const uint16_t* d_H, size_t ld, int n, int k, void* stream, uint32_t* idx,
                                    uint16_t* dist, char* err, int errlen) {
    Err e{err, errlen};
    StreamGuard g;
    if (g.make(stream)) return e.set("could not create a stream");
    return neighbors_on_device(d_H, ld, n, k, g.st, idx, dist, e);
}

extern "C" int tch_solver_mst(tch_solver* s, uint32_t* u, uint32_t* v, uint16_t* w, uint64_t* total, char* err,
                              int errlen) {
    Err e{err, errlen};
    StreamGuard g;
    uint16_t* H = nullptr;
    size_t ld = 0;
    int n = 0, rc = 1;
    if (g.make(nullptr)) return e.set("could not create a stream");
    if (full_matrix(s, &n, &H, &ld, g.st, err, errlen)) return 1;
    if (n < 2) {
        if (total) *total = 0;
        rc = 0;
    } else {
        rc = mst_on_device(H, ld, n, g.st, u, v, w, total, e);
    }
    cudaFree(H);
    return rc;
}

extern "C" int tch_solver_neighbors(tch_solver* s, int k, uint32_t* idx, uint16_t* dist, char* err, int errlen) {
    Err e{err, errlen};
    tch_info info;
    StreamGuard g;
    uint16_t* H = nullptr;
    size_t ld = 0;
    int n = 0, rc;
    if (!s || tch_solver_info(s, &info)) return e.set("bad solver");
    if (k < 1 || k > kMaxNeighbors) return e.set("k must be 1-%d", kMaxNeighbors);
    if (k >= info.n) return e.set("k must be below n (%d)", info.n);
    if (g.make(nullptr)) return e.set("could not create a stream");
    if (full_matrix(s, &n, &H, &ld, g.st, err, errlen)) return 1;
    rc = neighbors_on_device(H, ld, n, k, g.st, idx, dist, e);
    cudaFree(H);
    return rc;
}

extern "C" int tch_mst_clusters(int n, const uint32_t* u, const uint32_t* v, const uint16_t* w, size_t m,
                                const uint32_t* thresholds, int nt, uint32_t* labels, char* err, int errlen) {
    Err e{err, errlen};
    if (n < 0 || nt < 0) return e.set("n and nt must be >= 0");
    if (nt > 0 && n > 0 && (!thresholds || !labels)) return e.set("null thresholds or labels");
    if (m > 0 && (!u || !v || !w)) return e.set("null edges");
    for (size_t q = 0; q < m; q++)
        if (u[q] >= (uint32_t)n || v[q] >= (uint32_t)n || u[q] == v[q])
            return e.set("edge %zu (%u, %u) is not between two of the %d profiles", q, u[q], v[q], n);
    std::vector<size_t> by_w(m);
    std::iota(by_w.begin(), by_w.end(), (size_t)0);
    std::stable_sort(by_w.begin(), by_w.end(), [&](size_t a, size_t b) { return w[a] < w[b]; });
    std::vector<int> by_t((size_t)nt);
    std::iota(by_t.begin(), by_t.end(), 0);
    std::stable_sort(by_t.begin(), by_t.end(), [&](int a, int b) { return thresholds[a] < thresholds[b]; });
    // union by the smaller root: a set's root is its smallest profile index
    std::vector<uint32_t> p((size_t)n);
    std::iota(p.begin(), p.end(), 0u);
    auto find = [&](uint32_t x) {
        while (p[x] != x) x = p[x] = p[p[x]];
        return x;
    };
    size_t q = 0;
    for (int t : by_t) {
        for (; q < m && w[by_w[q]] <= thresholds[t]; q++) {
            const uint32_t a = find(u[by_w[q]]), b = find(v[by_w[q]]);
            if (a != b) p[std::max(a, b)] = std::min(a, b);
        }
        uint32_t* out = labels + (size_t)t * n;
        for (int i = 0; i < n; i++) out[i] = find((uint32_t)i);
    }
    return 0;
}

extern "C" int tch_solver_clusters(tch_solver* s, const uint32_t* thresholds, int nt, uint32_t* labels, char* err,
                                   int errlen) {
    Err e{err, errlen};
    tch_info info;
    if (!s || tch_solver_info(s, &info)) return e.set("bad solver");
    const int n = info.n;
    const size_t m = n > 1 ? (size_t)n - 1 : 0;
    std::vector<uint32_t> u(m), v(m);
    std::vector<uint16_t> w(m);
    if (tch_solver_mst(s, u.data(), v.data(), w.data(), nullptr, err, errlen)) return 1;
    return tch_mst_clusters(n, u.data(), v.data(), w.data(), m, thresholds, nt, labels, err, errlen);
}
