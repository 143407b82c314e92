// The distance matrix as TSV text, formatted on the GPU (the reference's
// write_matrix, tensorcore/rs/src/main.rs:224-265: a header line, then per
// sample its id and n distances, layout mask then cap, decimal, separator
// before every value, newline).
//
// The whole upper triangle is computed into HBM by the solver; a tiled
// transpose mirrors it into the lower half when the layout shows it.  Rows are
// then formatted in blocks: a warp per row sums the field lengths, one CTA
// scans them into offsets, and a warp per row writes its text, 32 values at a
// time (lane = value; a warp scan of the field lengths gives every lane its
// position).  Each block's text goes to pinned host memory on a stream of its own
// while the next block is formatted and the caller's callback takes the one
// before: formatting runs at about 210 GB/s of text with its length pass, the link
// at 193, and on one stream they took turns.  Device buffers come from the kept
// working pool.

#include <string.h>

#include <mutex>
#include <string>
#include <vector>

#include "tch_internal.cuh"

namespace tch {
namespace {

constexpr unsigned FULL = 0xFFFFFFFFu;
constexpr int TT = 64;  // transpose tile

// H[i][j] = H[j][i] for j < i (i, j < n): the lower half from the upper.  A CTA
// moves a tile of 64 x 64: 16-byte loads of the source rows, words of two rows out
// of shared memory (33 to a row: neither side meets a bank twice), 16-byte stores.
// Tile rows y and T - 1 - y, T + 1 tiles together, share a grid row.
//
// Bound by HBM, 2 bytes read and written per pair: 63 005 profiles in 1.22 ms (6.5
// TB/s); with 32 x 32 tiles, two bytes per access, the spanning tree from a solver
// took 17.5 ms, now 14.5.
__global__ void __launch_bounds__(256) mirror_kernel(uint16_t* H, size_t ld, int n) {
    __shared__ uint32_t t[TT][TT / 2 + 1];
    const int nt = (n + TT - 1) / TT, y = blockIdx.y, x = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (x > y && nt - 1 - y == y) return;
    const int ti = x <= y ? y : nt - 1 - y, tj = x <= y ? x : x - (y + 1);  // destination: rows ti, columns tj <= ti
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int row = 32 * u + 4 * warp + (lane >> 3), r = tj * TT + row, q = lane & 7, c = ti * TT + 8 * q;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (r < n && c < n) v = *reinterpret_cast<const uint4*>(H + (size_t)r * ld + c);
        uint32_t* w = &t[row][4 * q];
        w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
    }
    __syncthreads();
    // rows 2 p and 2 p + 1 of the destination, 8 columns
    const int p = 8 * (warp & 3) + (lane >> 2), q = 4 * (warp >> 2) + (lane & 3);
    uint32_t w[8], even[4], odd[4];
#pragma unroll
    for (int e = 0; e < 8; e++) w[e] = t[8 * q + e][p];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        even[e] = __byte_perm(w[2 * e], w[2 * e + 1], 0x5410);
        odd[e] = __byte_perm(w[2 * e], w[2 * e + 1], 0x7632);
    }
    const int c = tj * TT + 8 * q;
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const int r = ti * TT + 2 * p + u;
        const uint32_t* v = u ? odd : even;
        uint16_t* dst = H + (size_t)r * ld + c;
        if (r >= n) continue;
        if (c + 7 < r) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 8; e++)
                if (c + e < r) dst[e] = (uint16_t)(v[e / 2] >> (16 * (e & 1)));
        }
    }
}

__device__ __forceinline__ int digits(uint32_t v) { return v < 10 ? 1 : v < 100 ? 2 : v < 1000 ? 3 : v < 10000 ? 4 : 5; }

// The value printed at (i, j): layout mask (0 full, 1 lower-tri, 2 upper-tri),
// zero diagonal, then the cap.
__device__ __forceinline__ uint32_t cell(const uint16_t* H, size_t ld, int i, int j, int layout, int cap) {
    uint32_t v = 0;
    if (i != j && !(layout == 1 && j > i) && !(layout == 2 && j < i)) v = H[(size_t)i * ld + j];
    if (cap > 0 && v > (uint32_t)cap) v = (uint32_t)cap;
    return v;
}

__global__ void row_length_kernel(const uint16_t* H, size_t ld, int n, int r0, int rows, int layout, int cap,
                                  const uint64_t* id_off, int seplen, uint64_t* len) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x % 32;
    const int nw = gridDim.x * blockDim.x / 32;
    for (int r = warp; r < rows; r += nw) {
        const int i = r0 + r;
        uint64_t s = 0;
        for (int j = lane; j < n; j += 32) s += (uint64_t)(seplen + digits(cell(H, ld, i, j, layout, cap)));
#pragma unroll
        for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(FULL, s, d);
        if (lane == 0) len[r] = (id_off[i + 1] - id_off[i]) + s + 1;
    }
}

// Exclusive scan of len[0..rows) into off[0..rows], one CTA.
__global__ void scan_kernel(const uint64_t* len, int rows, uint64_t* off) {
    __shared__ uint64_t part[1024];
    const int t = threadIdx.x, T = blockDim.x;
    const int per = (rows + T - 1) / T, a = min(rows, t * per), b = min(rows, a + per);
    uint64_t s = 0;
    for (int r = a; r < b; r++) s += len[r];
    part[t] = s;
    __syncthreads();
    if (t == 0) {
        uint64_t acc = 0;
        for (int q = 0; q < T; q++) {
            const uint64_t v = part[q];
            part[q] = acc;
            acc += v;
        }
        off[rows] = acc;
    }
    __syncthreads();
    uint64_t acc = part[t];
    for (int r = a; r < b; r++) {
        off[r] = acc;
        acc += len[r];
    }
}

__global__ void row_write_kernel(const uint16_t* H, size_t ld, int n, int r0, int rows, int layout, int cap,
                                 const char* ids, const uint64_t* id_off, const char* sep, int seplen,
                                 const uint64_t* off, char* out) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x % 32;
    const int nw = gridDim.x * blockDim.x / 32;
    for (int r = warp; r < rows; r += nw) {
        const int i = r0 + r;
        char* p = out + off[r];
        const uint64_t il = id_off[i + 1] - id_off[i];
        for (uint64_t c = lane; c < il; c += 32) p[c] = ids[id_off[i] + c];
        uint64_t pos = il;
        for (int j0 = 0; j0 < n; j0 += 32) {
            const int j = j0 + lane;
            uint32_t v = 0;
            int w = 0;
            if (j < n) {
                v = cell(H, ld, i, j, layout, cap);
                w = seplen + digits(v);
            }
            int x = w;  // inclusive scan of the field widths
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int t = __shfl_up_sync(FULL, x, d);
                if (lane >= d) x += t;
            }
            if (j < n) {
                char* q = p + pos + (x - w);
                for (int c = 0; c < seplen; c++) q[c] = sep[c];
                q += seplen;
                for (int c = w - seplen - 1; c >= 0; c--) {
                    q[c] = (char)('0' + v % 10);
                    v /= 10;
                }
            }
            pos += (uint64_t)__shfl_sync(FULL, x, 31);
        }
        if (lane == 0) p[pos] = '\n';
    }
}

// Page-locked text buffers cost far more to allocate than to fill, so the pair
// of the previous call is kept for the next (one pair per process; a call that
// finds it in use allocates its own).
std::mutex g_text_mu;
char* g_text[2] = {nullptr, nullptr};
size_t g_text_bytes = 0;
bool g_text_busy = false;

bool text_acquire(size_t bytes, char* out[2]) {
    std::lock_guard<std::mutex> lk(g_text_mu);
    if (g_text_busy) return false;
    if (g_text_bytes < bytes) {
        for (int b = 0; b < 2; b++) {
            if (g_text[b]) cudaFreeHost(g_text[b]);
            g_text[b] = nullptr;
        }
        g_text_bytes = 0;
        for (int b = 0; b < 2; b++)
            if (cudaMallocHost(&g_text[b], bytes) != cudaSuccess) return false;
        g_text_bytes = bytes;
    }
    g_text_busy = true;
    out[0] = g_text[0];
    out[1] = g_text[1];
    return true;
}

void text_release() {
    std::lock_guard<std::mutex> lk(g_text_mu);
    g_text_busy = false;
}

}  // namespace

cudaError_t launch_mirror(uint16_t* H, size_t ld, int n, cudaStream_t st) {
    if (n < 2) return cudaSuccess;
    if ((ld & 7) || ((uintptr_t)H & 15)) return cudaErrorInvalidValue;
    const int nt = (n + TT - 1) / TT;
    mirror_kernel<<<dim3(nt + 1, (nt + 1) / 2), 256, 0, st>>>(H, ld, n);
    return cudaGetLastError();
}

}  // namespace tch

using namespace tch;

extern "C" int tch_solver_write_tsv(tch_solver* s, const char* const* ids, const char* osep, const char* index_name,
                                    int layout, int cap, int block_rows, tch_text_cb cb, void* ctx, char* err,
                                    int errlen) {
    Err e{err, errlen};
    tch_info info;
    uint16_t* H = nullptr;
    char *d_ids = nullptr, *d_sep = nullptr, *d_text[2] = {nullptr, nullptr}, *h_text[2] = {nullptr, nullptr};
    uint64_t *d_idoff = nullptr, *d_len = nullptr, *d_off[2] = {nullptr, nullptr};
    cudaStream_t st = nullptr, cs = nullptr;  // kernels, copies
    cudaEvent_t done[2] = {nullptr, nullptr}, ready[2] = {nullptr, nullptr};
    cudaMemPool_t pool = nullptr;
    int dev = 0, sms = 0, rc = 1, blocks = 0;
    std::vector<uint64_t> idoff;
    std::string head;
    size_t cap_bytes = 0;
    bool pooled = false;
    uint64_t lens[2] = {0, 0};
    if (!s || !ids || !osep || !index_name || !cb) return e.set("null argument");
    if (layout < 0 || layout > 2) return e.set("layout must be 0 (full), 1 (lower-tri) or 2 (upper-tri)");
    if (tch_solver_info(s, &info)) return e.set("bad solver");
    const int n = info.n;
    const int seplen = (int)strlen(osep);
    if (seplen < 1 || seplen > 16) return e.set("output separator must be 1-16 bytes");
    if (block_rows <= 0) block_rows = 2048;
    block_rows = std::min(block_rows, std::max(n, 1));
    // header (host)
    head = index_name;
    idoff.assign((size_t)n + 1, 0);
    for (int i = 0; i < n; i++) {
        head += osep;
        head += ids[i];
        idoff[i + 1] = idoff[i] + strlen(ids[i]);
    }
    head += '\n';
    cb(ctx, head.data(), head.size());
    if (n == 0) return 0;
    const size_t ld = up((size_t)n, 8);
    TCH_CK(e, cudaGetDevice(&dev));
    TCH_CK(e, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TCH_CK(e, cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    TCH_CK(e, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    TCH_CK(e, working_pool(dev, &pool));
    TCH_CK(e, pool_alloc(&H, (size_t)n * ld * 2, pool, st));
    if (n > 1) {
        if (tch_solver_stripe(s, 0, n, H, ld, st, err, errlen)) goto fail;
        TCH_CK(e, cudaStreamSynchronize(st));
        if (tch_solver_check(s, err, errlen)) goto fail;
        if (layout != 2) TCH_CK(e, launch_mirror(H, ld, n, st));
    }
    {
        std::string all_ids;
        for (int i = 0; i < n; i++) all_ids += ids[i];
        TCH_CK(e, pool_alloc(&d_ids, std::max<size_t>(all_ids.size(), 1), pool, st));
        TCH_CK(e, pool_alloc(&d_idoff, ((size_t)n + 1) * 8, pool, st));
        TCH_CK(e, pool_alloc(&d_sep, 16, pool, st));
        if (!all_ids.empty())
            TCH_CK(e, cudaMemcpyAsync(d_ids, all_ids.data(), all_ids.size(), cudaMemcpyHostToDevice, st));
        TCH_CK(e, cudaMemcpyAsync(d_idoff, idoff.data(), ((size_t)n + 1) * 8, cudaMemcpyHostToDevice, st));
        TCH_CK(e, cudaMemcpyAsync(d_sep, osep, seplen, cudaMemcpyHostToDevice, st));
        TCH_CK(e, cudaStreamSynchronize(st));  // all_ids goes out of scope
    }
    // text buffers: the longest block of rows (longest ids x widest values)
    {
        size_t maxid = 0;
        for (int i = 0; i < n; i++) maxid = std::max<size_t>(maxid, idoff[i + 1] - idoff[i]);
        cap_bytes = (size_t)block_rows * (maxid + (size_t)n * (seplen + 5) + 1);
    }
    TCH_CK(e, pool_alloc(&d_len, (size_t)block_rows * 8, pool, st));
    pooled = text_acquire(cap_bytes, h_text);
    for (int b = 0; b < 2; b++) {
        TCH_CK(e, pool_alloc(&d_off[b], ((size_t)block_rows + 1) * 8, pool, st));
        TCH_CK(e, pool_alloc(&d_text[b], cap_bytes, pool, st));
        if (!pooled) TCH_CK(e, cudaMallocHost(&h_text[b], cap_bytes));
        TCH_CK(e, cudaEventCreateWithFlags(&done[b], cudaEventDisableTiming));
        TCH_CK(e, cudaEventCreateWithFlags(&ready[b], cudaEventDisableTiming));
    }
    blocks = (n + block_rows - 1) / block_rows;
    // step k: block k is formatted, block k - 1 copied, block k - 2 handed over;
    // two buffers of each kind
    for (int k = 0; k < blocks + 2; k++) {
        if (k >= 1 && k <= blocks) {  // block k - 1's length is known when it is formatted
            const int b = (k - 1) & 1;
            TCH_CK(e, cudaEventSynchronize(ready[b]));
            TCH_CK(e, cudaMemcpyAsync(h_text[b], d_text[b], lens[b], cudaMemcpyDeviceToHost, cs));
            TCH_CK(e, cudaEventRecord(done[b], cs));
        }
        if (k < blocks) {
            const int r0 = k * block_rows, rows = std::min(block_rows, n - r0), b = k & 1;
            const int grid = std::max(1, std::min(sms * 8, (rows * 32 + 255) / 256));
            if (k >= 2) TCH_CK(e, cudaStreamWaitEvent(st, done[b], 0));  // block k - 2 has left the buffer
            row_length_kernel<<<grid, 256, 0, st>>>(H, ld, n, r0, rows, layout, cap, d_idoff, seplen, d_len);
            scan_kernel<<<1, 1024, 0, st>>>(d_len, rows, d_off[b]);
            row_write_kernel<<<grid, 256, 0, st>>>(H, ld, n, r0, rows, layout, cap, d_ids, d_idoff, d_sep, seplen,
                                                   d_off[b], d_text[b]);
            TCH_CK(e, cudaGetLastError());
        }
        if (k >= 2) {
            const int b = k & 1;
            TCH_CK(e, cudaEventSynchronize(done[b]));
            cb(ctx, h_text[b], lens[b]);
        }
        if (k < blocks) {  // after block k - 2's length has been used
            const int rows = std::min(block_rows, n - k * block_rows), b = k & 1;
            TCH_CK(e, cudaMemcpyAsync(&lens[b], d_off[b] + rows, 8, cudaMemcpyDeviceToHost, st));
            TCH_CK(e, cudaEventRecord(ready[b], st));
        }
    }
    rc = 0;
fail:
    if (cs) cudaStreamSynchronize(cs);
    for (void* q : {(void*)H, (void*)d_ids, (void*)d_sep, (void*)d_idoff, (void*)d_len, (void*)d_off[0], (void*)d_off[1],
                    (void*)d_text[0], (void*)d_text[1]})
        if (q) cudaFreeAsync(q, st);
    if (st) cudaStreamSynchronize(st);
    for (int b = 0; b < 2; b++) {
        if (h_text[b] && !pooled) cudaFreeHost(h_text[b]);
        if (done[b]) cudaEventDestroy(done[b]);
        if (ready[b]) cudaEventDestroy(ready[b]);
    }
    if (st) cudaStreamDestroy(st);
    if (cs) cudaStreamDestroy(cs);
    if (pooled) text_release();
    return rc;
}
