// Counting the members of rare groups in shared memory, 16 bytes of members per
// lane: shared by the rare counts of a set's own rows (k_rare.cu) and of new
// profiles (serve.cu).
#pragma once

#include <stdint.h>

#include "tch_internal.cuh"

namespace tch {
namespace {

// A row's partners are runs of consecutive members; a run covers whole 16-byte
// pieces of the member array but for its first and last one (8 members of two
// bytes when every row index fits them, else 4 of four).  The pieces of a row's
// runs, laid end to end, are cut into one equal part per warp, and a lane takes
// a whole piece: finding its run, the load and the two end masks cost about 30
// instructions per piece, and each member five and its shared atomic.  Walking
// the members one by one, every one with its own look at the run cursor, took
// 26 instructions per atomic.

template <class M>
constexpr int kPiece = 16 / (int)sizeof(M);  // members per piece

// Shared add under a predicate (as an `if` each one became a branch: 19
// instructions per atomic).
__device__ __forceinline__ void red_add_if(uint32_t cond, uint32_t addr, uint32_t v) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p red.shared.add.u32 [%1], %2;\n\t}\n" ::"r"(cond),
                 "r"(addr), "r"(v)
                 : "memory");
}

// Where column j's u16 counter lies: half (j - odd) & 1 of the word at base +
// (2 (j - odd) & mask), odd = 1 when the counters start at an odd column.
struct Counters {
    uint32_t base;
    uint32_t odd;
    uint32_t mask;
};
__device__ __forceinline__ Counters counters_at(const void* cnt, int first_col) {
    Counters c;
    c.odd = (uint32_t)first_col & 1u;
    c.base = (uint32_t)__cvta_generic_to_shared(cnt) - 2u * ((uint32_t)first_col - c.odd);
    c.mask = 0x1FFFCu;
    return c;
}
// Counters of one window of kQueryWindow columns; members in two bytes, modulo
// 65 536, of which the window's width is a divisor.
__device__ __forceinline__ Counters window_counters(const void* cnt) {
    Counters c;
    c.odd = 0;
    c.base = (uint32_t)__cvta_generic_to_shared(cnt);
    c.mask = 2u * kQueryWindow - 4u;
    return c;
}

// The members of a piece that `mask` names, counted.
__device__ __forceinline__ void count_piece(const Counters& c, const uint4& v, uint32_t mask, uint16_t) {
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const uint32_t base = c.base;
    if (c.odd) {
#pragma unroll
        for (int q = 0; q < 4; q++) w[q] = __vsub2(w[q], 0x00010001u);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        red_add_if(mask & (1u << (2 * q)), base + ((w[q] << 1) & c.mask), (w[q] & 1u) * 0xFFFFu + 1u);
        red_add_if(mask & (2u << (2 * q)), base + ((w[q] >> 15) & c.mask), max(w[q] & 0x10000u, 1u));
    }
}
__device__ __forceinline__ void count_piece(const Counters& c, const uint4& v, uint32_t mask, uint32_t) {
    const uint32_t w[4] = {v.x - c.odd, v.y - c.odd, v.z - c.odd, v.w - c.odd};
#pragma unroll
    for (int q = 0; q < 4; q++)
        red_add_if(mask & (1u << q), c.base + ((w[q] << 1) & ~3u), (w[q] & 1u) * 0xFFFFu + 1u);
}

// Pieces [e_begin, e_end) of nr staged runs, by one warp.  run[q].x = (first piece
// of run q among the row's) << 3 | place of its last member in its last piece,
// run[nr].x >> 3 bounds the last run; run[q].y = its first member.
template <class M>
__device__ __forceinline__ void walk_pieces(const Counters& c, const uint2* run, int nr, uint32_t e_begin,
                                            uint32_t e_end, const M* __restrict__ members,
                                            int lane) {
    constexpr int G = kPiece<M>;
    if (e_begin >= e_end) return;
    int p = 0;  // the run holding e_begin
    for (int hi = nr; hi - p > 1;) {
        const int m = (p + hi) >> 1;
        if ((run[m].x >> 3) <= e_begin) p = m; else hi = m;
    }
    uint2 cur = run[p], next = run[p + 1];  // this lane's current run and the one after it
    for (uint32_t e0 = e_begin; e0 < e_end; e0 += 64) {
        uint4 v[2];
        uint32_t mask[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {  // both loads before the first atomic
            const uint32_t e = e0 + (uint32_t)(32 * u + lane);
            mask[u] = 0;
            v[u] = make_uint4(0, 0, 0, 0);
            if (e < e_end) {
                while (e >= next.x >> 3) {  // next run (run[nr].x >> 3 = the end of all > e bounds it)
                    cur = next;
                    next = run[++p + 1];
                }
                const uint32_t k = e - (cur.x >> 3);
                mask[u] = (1u << G) - 1u;
                if (k == 0) mask[u] &= ~0u << (cur.y % G);
                if (e + 1 == next.x >> 3) mask[u] &= (2u << (cur.x & 7u)) - 1u;
                v[u] = __ldg(reinterpret_cast<const uint4*>(members) + (cur.y / G + k));
            }
        }
        count_piece(c, v[0], mask[0], M());
        if (e0 + 32 < e_end) count_piece(c, v[1], mask[1], M());
    }
}

}  // namespace
}  // namespace tch
