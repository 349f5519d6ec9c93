// split12 packer on the device, bit-identical to the reference's CPU packer
// (split12_pack.c:18-128): exponent histogram for the base_exp window search,
// sm / gr arrays, and the CSR escape list in ascending column order per row.
//
// The reference packs on one CPU core (two passes over the tensor); a
// 70B-parameter model takes minutes.  Here a tensor is packed at HBM speed:
//   1. histogram256      - one pass, per-CTA shared histograms
//   2. window search over the 256 counts -> base_exp: on the host, or by the
//                          histogram's last CTA (s12_pack_auto_async)
//   3. pack              - 16 elements per thread: 32 B in, 16 B sm + 8 B gr out,
//                          per-row escape counts by atomics into row_off[r+1]
//   4. scan              - in-place inclusive scan of row_off (single CTA)
//   5. fill              - one warp per row finds the escapes once more, in the
//                          gr nibbles (a quarter of the bytes, still in L2) or in
//                          the bf16 values, and writes cols / correct / wrong in
//                          ascending column order
#include "common.cuh"
#include <algorithm>

namespace s12 {

// What s12_pack_auto_async adds to a histogram: its CTAs count themselves in `done`, and the last one searches the window.
struct HistWindow { unsigned int* done; int* base_exp; };

// first window of 15 consecutive exponents with the largest count; starts 0..241.  All threads of a CTA of 256 or more.
__device__ void find_window(const unsigned long long* hist, int* base_exp)
{
    __shared__ unsigned long long best[32];
    __shared__ int best_at[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned long long win = 0;
    int at = 0x7FFFFFFF;
    if (t <= 241) {
        for (int i = 0; i < 15; i++) win += __ldcg(hist + t + i);
        at = t;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long ow = __shfl_xor_sync(0xFFFFFFFFu, win, off);
        const int oa = __shfl_xor_sync(0xFFFFFFFFu, at, off);
        if (ow > win || (ow == win && oa < at)) { win = ow; at = oa; }
    }
    if (lane == 0) { best[warp] = win; best_at[warp] = at; }
    __syncthreads();
    if (t == 0) {
        for (int i = 1; i < 8; i++)
            if (best[i] > win || (best[i] == win && best_at[i] < at)) { win = best[i]; at = best_at[i]; }
        *base_exp = at - 1;
    }
}

// kCopies shared histograms, lane l adds to copy l % kCopies, so that the lanes of a warp, whose exponents fall into a
// handful of bins, do not queue up on one counter.  Bound by those shared-memory additions, four clocks per 32 values:
// 26.8 us on 14336 x 4096 (18 us to read it).  kVec: 16-byte loads of eight values (16-byte aligned input), two in
// flight; else one value at a time.  kWindow: with the search behind it.  Small tensors, a few values a thread, have one copy: clearing and adding up 32 is
// most of their time (64 x 64, with the clearing of the counts, 6.0 us with 32 copies, 4.9 with one).
template <bool kVec, int kCopies, bool kWindow>
__global__ void __launch_bounds__(512)
hist_kernel(const uint16_t* __restrict__ w, int64_t n, unsigned long long* __restrict__ hist, const HistWindow W)
{
    __shared__ unsigned int sh[256 * kCopies];
    __shared__ bool last;
    for (int i = threadIdx.x; i < 256 * kCopies; i += blockDim.x) sh[i] = 0;
    grid_dependency_wait();                    // inputs and outputs may belong to the predecessor kernel
    __syncthreads();
    unsigned int* mine = sh + (threadIdx.x & (kCopies - 1));
    auto count = [&](uint32_t h) { atomicAdd(mine + ((h >> 7) & 0xFFu) * kCopies, 1u); };
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    if (kVec) {
        const uint4* w8 = reinterpret_cast<const uint4*>(w);
        const int64_t n8 = n / 8;
        for (int64_t i = first; i < n8; i += 2 * stride) {
            const bool two = i + stride < n8;
            const uint4 a = __ldg(w8 + i), b = two ? __ldg(w8 + i + stride) : make_uint4(0, 0, 0, 0);
            const uint32_t va[4] = {a.x, a.y, a.z, a.w}, vb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int j = 0; j < 4; j++) { count(va[j]); count(va[j] >> 16); }
            if (two) {
#pragma unroll
                for (int j = 0; j < 4; j++) { count(vb[j]); count(vb[j] >> 16); }
            }
        }
        if (first < n - n8 * 8) count(w[n8 * 8 + first]);
    } else {
        for (int64_t i = first; i < n; i += stride) count(w[i]);
    }
    __syncthreads();
    for (int b = threadIdx.x; b < 256; b += blockDim.x) {
        unsigned int sum = 0;
        for (int c = 0; c < kCopies; c++) sum += sh[b * kCopies + ((c + b) & (kCopies - 1))];
        if (sum) atomicAdd(&hist[b], (unsigned long long)sum);
    }
    if (!kWindow) return;
    __threadfence();                           // this CTA's counts before its arrival
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(W.done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    find_window(hist, W.base_exp);
}

// base_exp by value, or where the histogram left it
struct BaseExp { int value; const int* at; };
__device__ __forceinline__ int read_base_exp(const BaseExp& b) { return b.at ? *b.at : b.value; }

// One thread packs 16 consecutive elements (K % 16 == 0, so they share a row).  The blocks walk the tensor from its end:
// the histogram's pass has just left that part in L2.  Bound by HBM (3.5 bytes a weight) once the integer work is done on
// pairs: with the scan 50.7 us one element at a time, 44.4 us on pairs (14336 x 4096; 31 us for the bytes).
__global__ void __launch_bounds__(256)
pack16_kernel(const uint16_t* __restrict__ w, int64_t num_chunks, int K, const BaseExp be,
              uint8_t* __restrict__ sm, uint8_t* __restrict__ gr, int32_t* __restrict__ row_off)
{
    grid_dependency_wait();
    const int64_t c = (int64_t)(gridDim.x - 1 - blockIdx.x) * 256 + threadIdx.x;
    if (c >= num_chunks) return;
    const int base_exp = read_base_exp(be);
    const uint4* src = reinterpret_cast<const uint4*>(w + c * 16);
    const uint4 v0 = __ldg(src), v1 = __ldg(src + 1);
    const uint32_t in[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    uint32_t smw[4], grw[2] = {0, 0};
    int esc = 0;
    if (base_exp >= -1 && base_exp <= 240) {
        // two elements per word, eleven instructions a pair
        const uint32_t bias = (uint32_t)(255 - base_exp) * 0x00010001u;
        uint32_t s[8], nib[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            s[i] = (in[i] & 0x007F007Fu) | ((in[i] >> 8) & ~0x007F007Fu);           // bytes 0 and 2: sign << 7 | mantissa
            // per half 255 + exponent - base_exp, 256 .. 270 for groups 1 .. 15: no carry between the halves
            const uint32_t x = (((in[i] >> 7) & 0x00FF00FFu) + bias) ^ 0x01000100u; // 0 .. 14 there, 15 or more elsewhere
            nib[i] = ((__vminu2(x, 0x000F000Fu) + 0x00010001u) & 0x000F000Fu) * 0x00010010u;   // byte 2: both nibbles
        }
#pragma unroll
        for (int i = 0; i < 4; i++) smw[i] = prmt(s[2 * i], s[2 * i + 1], 0x6420u);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            grw[i] = prmt(prmt(nib[4 * i], nib[4 * i + 1], 0x0062u), prmt(nib[4 * i + 2], nib[4 * i + 3], 0x0062u), 0x5410u);
            const uint32_t t = grw[i] | (grw[i] >> 1);
            esc += __popc(~(t | (t >> 2)) & 0x11111111u);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) smw[i] = 0;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const uint32_t h = (in[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu;
            const uint32_t s = ((h >> 15) << 7) | (h & 0x7Fu);
            const int grp = (int)((h >> 7) & 0xFFu) - base_exp;
            const bool ok = grp >= 1 && grp <= 15;
            esc += !ok;
            smw[i >> 2] |= s << ((i & 3) * 8);
            grw[i >> 3] |= (ok ? (uint32_t)grp : 0u) << ((i & 7) * 4);
        }
    }
    *reinterpret_cast<uint4*>(sm + c * 16) = make_uint4(smw[0], smw[1], smw[2], smw[3]);
    *reinterpret_cast<uint2*>(gr + c * 8) = make_uint2(grw[0], grw[1]);
    if (esc) atomicAdd(&row_off[(c * 16) / K + 1], esc);
}

// General path: any even K, one thread per pair of elements.
__global__ void __launch_bounds__(256)
pack2_kernel(const uint16_t* __restrict__ w, int64_t num_pairs, int K, const BaseExp be,
             uint8_t* __restrict__ sm, uint8_t* __restrict__ gr, int32_t* __restrict__ row_off)
{
    grid_dependency_wait();
    const int64_t pr = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (pr >= num_pairs) return;
    const int base_exp = read_base_exp(be);
    uint32_t gb = 0;
#pragma unroll
    for (int h2 = 0; h2 < 2; h2++) {
        const int64_t i = pr * 2 + h2;
        const uint32_t h = w[i];
        sm[i] = (uint8_t)(((h >> 15) << 7) | (h & 0x7Fu));
        const int grp = (int)((h >> 7) & 0xFFu) - base_exp;
        const bool ok = grp >= 1 && grp <= 15;
        if (ok) gb |= (uint32_t)grp << (4 * h2);
        else atomicAdd(&row_off[i / K + 1], 1);
    }
    gr[pr] = (uint8_t)gb;
}

// In-place inclusive scan of row_off[1..M] (row_off[0] == 0), one CTA; the sum also goes to *total when it is given.
// A round takes 1024 x kRows rows: each thread loads kRows, 1024 apart (coalesced, and one latency for all), the warps scan
// their kRows x 32 pieces, one warp scans the pieces' sums.  kRows is the smallest with which one round will do, up to
// eight: with eight for all, the scan of up to 1024 rows took 1-2 us longer (pack + scan of 512 x 512 6.3 -> 8.2 us).
template <int kRows>
__global__ void __launch_bounds__(1024)
scan_kernel(int32_t* __restrict__ row_off, int M, int* __restrict__ total)
{
    grid_dependency_wait();                    // the per-row counts come from the pack kernel before
    __shared__ int piece[kRows * 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    for (int64_t base = 1; base <= M; base += kRows * 1024) {   // 64 bits: M may lie within a round of 2^31
        int v[kRows];
#pragma unroll
        for (int j = 0; j < kRows; j++) {
            const int64_t i = base + j * 1024 + threadIdx.x;
            v[j] = i <= M ? row_off[i] : 0;
        }
#pragma unroll
        for (int j = 0; j < kRows; j++) {
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int t = __shfl_up_sync(0xFFFFFFFFu, v[j], off);
                if (lane >= off) v[j] += t;
            }
            if (lane == 31) piece[j * 32 + warp] = v[j];
        }
        __syncthreads();
        if (warp == 0) {                                         // exclusive scan of the sums, kRows a lane
            int s[kRows], sum = 0;
#pragma unroll
            for (int k = 0; k < kRows; k++) { s[k] = sum; sum += piece[lane * kRows + k]; }
            int before = sum;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int t = __shfl_up_sync(0xFFFFFFFFu, before, off);
                if (lane >= off) before += t;
            }
            before -= sum;
#pragma unroll
            for (int k = 0; k < kRows; k++) piece[lane * kRows + k] = before + s[k];
        }
        __syncthreads();
        int last = 0;
#pragma unroll
        for (int j = 0; j < kRows; j++) {
            const int64_t i = base + j * 1024 + threadIdx.x;
            v[j] += piece[j * 32 + warp] + carry;
            if (i <= M) row_off[i] = v[j];
            last = v[j];
        }
        __syncthreads();
        if (threadIdx.x == 1023) piece[0] = last;                // sum so far (rows past M count nothing)
        __syncthreads();
        carry = piece[0];
        __syncthreads();
    }
    if (total != nullptr && threadIdx.x == 0) *total = carry;
}

// One warp per row writes the row's list in ascending column order.
__device__ __forceinline__ void emit_escape(uint32_t h, int col, int pos, int base_exp, int32_t* __restrict__ cols,
                                            int16_t* __restrict__ correct, int16_t* __restrict__ wrong)
{
    cols[pos] = col;
    correct[pos] = (int16_t)h;
    wrong[pos] = (int16_t)((((h >> 15) << 15) | ((uint32_t)base_exp << 7) | (h & 0x7Fu)) & 0xFFFFu);
}

// a row, 32 columns at a time, for any K
constexpr int kFillFlight = 4;                 // loads in flight
__device__ __forceinline__ void fill_row(const uint16_t* __restrict__ wr, int K, int base_exp, int pos, int32_t* __restrict__ cols,
                                         int16_t* __restrict__ correct, int16_t* __restrict__ wrong)
{
    const int lane = threadIdx.x & 31;
    for (uint32_t c0 = 0; c0 < (uint32_t)K; c0 += kFillFlight * 32) {   // no end at a complete list: later loads would wait for it
        uint32_t h[kFillFlight];
#pragma unroll
        for (int u = 0; u < kFillFlight; u++) { const uint32_t c = c0 + u * 32 + lane; h[u] = c < (uint32_t)K ? wr[c] : 0u; }
#pragma unroll
        for (int u = 0; u < kFillFlight; u++) {
            const uint32_t c = c0 + u * 32 + lane;
            const int grp = (int)((h[u] >> 7) & 0xFFu) - base_exp;
            const bool esc = c < (uint32_t)K && !(grp >= 1 && grp <= 15);
            const unsigned m = __ballot_sync(0xFFFFFFFFu, esc);
            if (esc) emit_escape(h[u], (int)c, pos + __popc(m & ((1u << lane) - 1u)), base_exp, cols, correct, wrong);
            pos += __popc(m);
        }
    }
}

// K % 8 == 0: a lane looks at eight columns at a time -- kGroups: one word of gr nibbles (zero = escape), and the exact
// values are fetched one by one; else one 16-byte load of bf16 -- with four loads in flight.  Escapes are rare, so a
// step is the load, the test and one vote.  Bound by latency and L2: 8.3 us from groups, 16.5 us from bf16 (14336 x 4096).
// A row with a third or more escapes is written 32 columns at a time, where each lane's own list would scatter the stores
// (half of 14336 x 4096 escapes: 227 -> 119 us from groups, 95 %: 583 -> 175); with a quarter of them the two ways are equal.
// Rows of less than 256 columns leave lanes without work here, and take fill_kernel (64 x 64: 1.9 -> 1.6 us).
template <bool kGroups>
__global__ void __launch_bounds__(256)
fill8_kernel(const uint16_t* __restrict__ w, const uint8_t* __restrict__ gr, int M, int K, int base_exp,
             const int32_t* __restrict__ row_off, int32_t* __restrict__ cols,
             int16_t* __restrict__ correct, int16_t* __restrict__ wrong)
{
    grid_dependency_wait();                    // row_off comes from the scan kernel before
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= M) return;
    int pos = row_off[row];
    const int end = row_off[row + 1];
    if (end == pos) return;
    const uint16_t* wr = w + (size_t)row * K;
    if ((int64_t)(end - pos) * 3 >= K) {
        fill_row(wr, K, base_exp, pos, cols, correct, wrong);
        return;
    }
    const int words = K / 8;
    for (int i0 = 0; i0 < words && pos < end; i0 += 4 * 32) {    // the rest of a row whose list is complete has none
        uint32_t esc[4];                                         // bit 4 e: column e of the eight is an escape
        if (kGroups) {
            const uint32_t* g = reinterpret_cast<const uint32_t*>(gr + (size_t)row * (K / 2));
            uint32_t x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) { const int i = i0 + u * 32 + lane; x[u] = i < words ? __ldg(g + i) : 0xFFFFFFFFu; }
#pragma unroll
            for (int u = 0; u < 4; u++) { const uint32_t t = x[u] | (x[u] >> 1); esc[u] = ~(t | (t >> 2)) & 0x11111111u; }
        } else {
            uint4 x[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = i0 + u * 32 + lane;
                if (i < words) x[u] = __ldg(reinterpret_cast<const uint4*>(wr) + i);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                esc[u] = 0;
                if (i0 + u * 32 + lane < words) {
                    const uint32_t v[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const int grp = (int)((v[e >> 1] >> ((e & 1) * 16 + 7)) & 0xFFu) - base_exp;
                        if (!(grp >= 1 && grp <= 15)) esc[u] |= 1u << (4 * e);
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (!__any_sync(0xFFFFFFFFu, esc[u])) continue;
            int before = __popc(esc[u]);
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int t = __shfl_up_sync(0xFFFFFFFFu, before, off);
                if (lane >= off) before += t;
            }
            const int all = __shfl_sync(0xFFFFFFFFu, before, 31);
            int p = pos + before - __popc(esc[u]);
            for (uint32_t m = esc[u]; m; m &= m - 1) {
                const int c = (i0 + u * 32 + lane) * 8 + (__ffs(m) - 1) / 4;
                emit_escape(wr[c], c, p++, base_exp, cols, correct, wrong);
            }
            pos += all;
        }
    }
}

// any K
__global__ void __launch_bounds__(256)
fill_kernel(const uint16_t* __restrict__ w, int M, int K, int base_exp,
            const int32_t* __restrict__ row_off, int32_t* __restrict__ cols,
            int16_t* __restrict__ correct, int16_t* __restrict__ wrong)
{
    grid_dependency_wait();                    // row_off comes from the scan kernel before
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= M) return;
    int pos = row_off[row];
    if (row_off[row + 1] == pos) return;
    fill_row(w + (size_t)row * K, K, base_exp, pos, cols, correct, wrong);
}

static int hist_launch(const void* bf16, int64_t count, unsigned long long* hist, const HistWindow& W, void* stream, const char* who)
{
    const bool vec = (reinterpret_cast<uintptr_t>(bf16) & 15) == 0, small = count < 65536;
    const int threads = small ? 256 : 512;
    const int64_t per = (int64_t)threads * (small ? 4 : vec ? 16 : 64);
    const int64_t cap = (int64_t)sm_count() * 4;                 // all resident: 32 KB of shared memory each
    const int64_t blocks = std::min(cap, (count + per - 1) / per);
    typedef void (*Kern)(const uint16_t*, int64_t, unsigned long long*, const HistWindow);
    const Kern plain = small ? hist_kernel<false, 1, false> : vec ? hist_kernel<true, 32, false> : hist_kernel<false, 32, false>;
    const Kern window = small ? hist_kernel<false, 1, true> : vec ? hist_kernel<true, 32, true> : hist_kernel<false, 32, true>;
    return launch(W.done ? window : plain, dim3((unsigned)blocks), dim3(threads), 0, stream, who, (const uint16_t*)bf16, count, hist, W);
}

// pack + scan; `total` (device, may be null) receives the number of escapes
static int pack_launch(const void* bf16, int M, int K, const BaseExp& be, void* sm, void* gr, void* row_off, int* total, void* stream,
                       const char* who)
{
    const int64_t n = (int64_t)M * K;
    const bool vec = (K % 16) == 0 && (reinterpret_cast<uintptr_t>(bf16) % 16) == 0 &&
                     (reinterpret_cast<uintptr_t>(sm) % 16) == 0 && (reinterpret_cast<uintptr_t>(gr) % 8) == 0;
    const int64_t items = vec ? n / 16 : n / 2, blocks = (items + 255) / 256;
    if (blocks > 0x7FFFFFFF) return fail(S12_ERR_TOO_LARGE, "%s: tensor too large", who);
    const int rc = launch(vec ? pack16_kernel : pack2_kernel, dim3((unsigned)blocks), dim3(256), 0, stream, who,
                          (const uint16_t*)bf16, items, K, be, (uint8_t*)sm, (uint8_t*)gr, (int32_t*)row_off);
    if (rc) return rc;
    return launch(M <= 1024 ? scan_kernel<1> : M <= 2048 ? scan_kernel<2> : M <= 4096 ? scan_kernel<4> : scan_kernel<8>, dim3(1), dim3(1024), 0,
                  stream, who, (int32_t*)row_off, M, total);
}

static int fill_launch(const void* bf16, const void* gr, int M, int K, int base_exp, const void* row_off, void* cols, void* correct,
                       void* wrong, void* stream, const char* who)
{
    const dim3 grid((M + 7) / 8), block(256);
    const bool eight = K % 8 == 0 && K >= 256, groups = eight && gr != nullptr && (reinterpret_cast<uintptr_t>(gr) & 3) == 0;
    if (groups || (eight && (reinterpret_cast<uintptr_t>(bf16) & 15) == 0))
        return launch(groups ? fill8_kernel<true> : fill8_kernel<false>, grid, block, 0, stream, who, (const uint16_t*)bf16,
                      (const uint8_t*)gr, M, K, base_exp, (const int32_t*)row_off, (int32_t*)cols, (int16_t*)correct, (int16_t*)wrong);
    return launch(fill_kernel, grid, block, 0, stream, who, (const uint16_t*)bf16, M, K, base_exp, (const int32_t*)row_off,
                  (int32_t*)cols, (int16_t*)correct, (int16_t*)wrong);
}

}  // namespace s12

extern "C" {

int s12_pack_histogram_async(const void* bf16, int64_t count, void* hist256, void* stream)
{
    using namespace s12;
    if (count < 0 || !hist256 || (count > 0 && !bf16)) return fail(S12_ERR_BAD_ARG, "s12_pack_histogram_async: bad argument");
    int rc = check_cuda(cudaMemsetAsync(hist256, 0, 256 * sizeof(unsigned long long), (cudaStream_t)stream), "s12_pack_histogram_async");
    if (rc || count == 0) return rc;
    return hist_launch(bf16, count, (unsigned long long*)hist256, HistWindow{}, stream, "s12_pack_histogram_async");
}

int s12_pack_find_base_exp_host(const uint64_t* hist256)
{
    // first window of 15 consecutive exponents with the largest count; starts 0..241
    if (!hist256) return -1;
    uint64_t win = 0, best = 0;
    int best_start = 0;
    for (int j = 0; j < 15; j++) win += hist256[j];
    for (int start = 0; start <= 241; start++) {
        if (win > best) { best = win; best_start = start; }
        if (start < 241) win += hist256[start + 15] - hist256[start];
    }
    return best_start - 1;
}

int s12_pack_async(const void* bf16, int M, int K, int base_exp, void* sm, void* gr, void* row_off, void* stream)
{
    using namespace s12;
    if (M < 0 || K < 0 || (K & 1)) return fail(S12_ERR_BAD_ARG, "s12_pack_async: M=%d K=%d (K must be even)", M, K);
    if (!row_off) return fail(S12_ERR_BAD_ARG, "s12_pack_async: null row_off");
    int rc = check_cuda(cudaMemsetAsync(row_off, 0, sizeof(int32_t) * ((size_t)M + 1), (cudaStream_t)stream), "s12_pack_async");
    if (rc || M == 0 || K == 0) return rc;
    if (!bf16 || !sm || !gr) return fail(S12_ERR_BAD_ARG, "s12_pack_async: null pointer");
    return pack_launch(bf16, M, K, BaseExp{base_exp, nullptr}, sm, gr, row_off, nullptr, stream, "s12_pack_async");
}

int s12_pack_auto_async(const void* bf16, int M, int K, void* scratch, void* meta, void* sm, void* gr, void* row_off, void* stream)
{
    using namespace s12;
    const char* who = "s12_pack_auto_async";
    if (M < 1 || K < 1 || (K & 1)) return fail(S12_ERR_BAD_ARG, "%s: M=%d K=%d (K must be even)", who, M, K);
    if (!bf16 || !scratch || !meta || !sm || !gr || !row_off) return fail(S12_ERR_BAD_ARG, "%s: null pointer", who);
    cudaStream_t st = (cudaStream_t)stream;
    int rc = check_cuda(cudaMemsetAsync(scratch, 0, S12_PACK_SCRATCH_BYTES, st), who);
    if (!rc) rc = check_cuda(cudaMemsetAsync(row_off, 0, sizeof(int32_t) * ((size_t)M + 1), st), who);
    if (rc) return rc;
    unsigned long long* hist = (unsigned long long*)scratch;
    int* base_exp = (int*)meta;
    rc = hist_launch(bf16, (int64_t)M * K, hist, HistWindow{(unsigned int*)(hist + 256), base_exp}, stream, who);
    if (rc) return rc;
    return pack_launch(bf16, M, K, BaseExp{0, base_exp}, sm, gr, row_off, base_exp + 1, stream, who);
}

int s12_pack_fill_async(const void* bf16, int M, int K, int base_exp, const void* row_off,
                        void* cols, void* correct, void* wrong, void* stream)
{
    using namespace s12;
    if (M < 0 || K < 0) return fail(S12_ERR_BAD_ARG, "s12_pack_fill_async: M=%d K=%d", M, K);
    if (M == 0 || K == 0) return S12_OK;
    if (!bf16 || !row_off || !cols || !correct || !wrong) return fail(S12_ERR_BAD_ARG, "s12_pack_fill_async: null pointer");
    return fill_launch(bf16, nullptr, M, K, base_exp, row_off, cols, correct, wrong, stream, "s12_pack_fill_async");
}

int s12_pack_fill_groups_async(const void* bf16, const void* gr, int M, int K, int base_exp, const void* row_off,
                               void* cols, void* correct, void* wrong, void* stream)
{
    using namespace s12;
    const char* who = "s12_pack_fill_groups_async";
    if (M < 0 || K < 0 || (K & 1)) return fail(S12_ERR_BAD_ARG, "%s: M=%d K=%d", who, M, K);
    if (M == 0 || K == 0) return S12_OK;
    if (!bf16 || !gr || !row_off || !cols || !correct || !wrong) return fail(S12_ERR_BAD_ARG, "%s: null pointer", who);
    return fill_launch(bf16, gr, M, K, base_exp, row_off, cols, correct, wrong, stream, who);
}

}  // extern "C"
