// The small kernels either side of the split12 projections in a decode step:
// embedding lookup, RMSNorm (with the residual add) to bf16, RoPE + INT8
// per-head KV store, decode attention over the INT8 cache (GQA), SiLU(gate)*up
// to bf16, residual add, greedy argmax.  Same entry-point names, argument order
// and layouts as the engine's own launchers (engine/kernels.hip:127-160,
// 306-336, 461-493, 588-603, 694-714, 847-880), so the engine's forward loop
// (engine/inference.cpp:198-366, 572-666) links against this library unchanged.
// The launchers return int (0 = ok) where the engine's return void; a caller
// that ignores the value is unaffected.
//
// Written for this part rather than translated: every kernel takes part in
// programmatic dependent launch (so the chain GEMV -> norm -> GEMV replays
// from one CUDA graph without full kernel boundaries), loads are 16-byte
// vectors where the layout allows, and the B=1 RoPE + KV store is one launch
// instead of two.  Floating-point results agree with the engine's kernels to
// rounding (different reduction trees, accurate sincosf instead of the fast
// intrinsic); tests/test_gpu_step.py states the tolerances.
#include "common.cuh"
#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>

namespace s12 {

__device__ __forceinline__ float bf16_raw_to_float(int16_t raw)
{
    return __uint_as_float(((uint32_t)(uint16_t)raw) << 16);
}
// round to nearest even, as engine/kernels.hip:22-28
__device__ __forceinline__ int16_t float_to_bf16_rne(float v)
{
    const uint32_t u = __float_as_uint(v);
    return (int16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
}

// block-wide sum over up to 32 warps; every thread gets the result.  One barrier: every warp adds up the warps' sums
// itself.  `scratch` serves one call of a kernel.
__device__ __forceinline__ float block_sum(float v, float* scratch /* 32 floats */)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, off);
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float w = lane < nwarps ? scratch[lane] : 0.f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) w += __shfl_xor_sync(0xFFFFFFFFu, w, off);
    return w;
}

// ---------------------------------------------------------------------------
// embedding lookup (engine/kernels.hip:57-73): bf16 table row -> fp32; a token
// outside [0, n_vocab) gives a zero row
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
embed_kernel(const int16_t* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ out,
             int n_embd, int batch, int n_vocab)
{
    grid_launch_dependents();
    grid_dependency_wait();
    const int seq = blockIdx.y, idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (seq >= batch || idx >= n_embd) return;
    const int tok = tokens[seq];
    out[(size_t)seq * n_embd + idx] =
        (tok < 0 || tok >= n_vocab) ? 0.f : bf16_raw_to_float(table[(size_t)tok * n_embd + idx]);
}

// ---------------------------------------------------------------------------
// RMSNorm -> bf16, optionally after x += residual written back in place
// (engine/kernels.hip:355-393, 399-442).  One CTA per sequence.
// ---------------------------------------------------------------------------
// Bound by latency: rows that fit the CTA's registers (two 16-byte pieces a thread) are read once, together with their
// weights.  Rows of 4096 with the residual, in a chain of launches: 2.6 -> 1.9 us at B = 1, 3.7 -> 3.1 us at B = 256.  kLong:
// the row is longer than that; without the other branch beside it, 64 rows of 16384 take 4.5 us instead of 4.7.
template <bool kAdd, bool kLong = false>
__device__ __forceinline__ void rms_norm_row(float* __restrict__ x, const float* __restrict__ residual, const float* __restrict__ weight,
                                             int16_t* __restrict__ y, int n, float eps)
{
    __shared__ float scratch[32];
    grid_launch_dependents();
    const size_t off = (size_t)blockIdx.x * n;
    const bool vec = (n & 3) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(weight) |
                                       (kAdd ? reinterpret_cast<uintptr_t>(residual) : 0)) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(y) & 7) == 0;
    float4* x4 = reinterpret_cast<float4*>(x + off);
    const float4* r4 = reinterpret_cast<const float4*>(residual + (kAdd ? off : 0));
    const float4* w4 = reinterpret_cast<const float4*>(weight);
    auto emit = [&](int i, const float4& v, const float4& w, float rms) {
        const uint32_t lo = (uint16_t)float_to_bf16_rne(v.x * rms * w.x) | ((uint32_t)(uint16_t)float_to_bf16_rne(v.y * rms * w.y) << 16);
        const uint32_t hi = (uint16_t)float_to_bf16_rne(v.z * rms * w.z) | ((uint32_t)(uint16_t)float_to_bf16_rne(v.w * rms * w.w) << 16);
        reinterpret_cast<uint2*>(y + off)[i] = make_uint2(lo, hi);
    };
    float ss = 0.f;
    grid_dependency_wait();
    if (!kLong && vec && n / 4 <= 2 * (int)blockDim.x) {
        float4 v[2], w[2], r[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int i = threadIdx.x + j * blockDim.x;
            if (i >= n / 4) continue;
            v[j] = x4[i]; w[j] = w4[i];
            if (kAdd) r[j] = r4[i];
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int i = threadIdx.x + j * blockDim.x;
            if (i >= n / 4) continue;
            if (kAdd) { v[j].x += r[j].x; v[j].y += r[j].y; v[j].z += r[j].z; v[j].w += r[j].w; x4[i] = v[j]; }
            ss += v[j].x * v[j].x + v[j].y * v[j].y + v[j].z * v[j].z + v[j].w * v[j].w;
        }
        ss = block_sum(ss, scratch);
        const float rms = rsqrtf(ss / (float)n + eps);
#pragma unroll
        for (int j = 0; j < 2; j++) { const int i = threadIdx.x + j * blockDim.x; if (i < n / 4) emit(i, v[j], w[j], rms); }
        return;
    }
    if (vec) {                                                    // 16-byte aligned rows: four elements per load
        for (int i = threadIdx.x; i < n / 4; i += blockDim.x) {
            float4 v = x4[i];
            if (kAdd) { const float4 r = r4[i]; v.x += r.x; v.y += r.y; v.z += r.z; v.w += r.w; x4[i] = v; }
            ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
        ss = block_sum(ss, scratch);
        const float rms = rsqrtf(ss / (float)n + eps);
        for (int i = threadIdx.x; i < n / 4; i += blockDim.x) emit(i, x4[i], w4[i], rms);   // a thread re-reads only what it wrote
        return;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        float v = x[off + i];
        if (kAdd) { v += residual[off + i]; x[off + i] = v; }
        ss += v * v;
    }
    ss = block_sum(ss, scratch);
    const float rms = rsqrtf(ss / (float)n + eps);
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        y[off + i] = float_to_bf16_rne(x[off + i] * rms * weight[i]);    // a thread re-reads only what it wrote
}
template <bool kAdd, bool kLong = false>
__global__ void __launch_bounds__(1024)
rms_norm_kernel(float* __restrict__ x, const float* __restrict__ residual, const float* __restrict__ weight,
                int16_t* __restrict__ y, int n, float eps)
{
    rms_norm_row<kAdd, kLong>(x, residual, weight, y, n, eps);
}
// With the residual a thread takes 48 registers, and an SM one CTA of 1024 threads.  Up to a row per SM that is the faster
// form (64 rows of 4096: 2.1 us, 2.7 with 32 registers); above, a second CTA has to fit: 32 registers.  256 rows of 1024 /
// 4096 / 16384: 2.8 / 3.8 / 9.2 -> 2.3 / 3.1 / 7.4 us.
__global__ void __launch_bounds__(1024, 2)
add_rms_norm_two_kernel(float* __restrict__ x, const float* __restrict__ residual, const float* __restrict__ weight,
                        int16_t* __restrict__ y, int n, float eps)
{
    rms_norm_row<true>(x, residual, weight, y, n, eps);
}

// SiLU(gate) * up -> bf16 (engine/kernels.hip:447-458), residual add (engine/kernels.hip:340-349)
__global__ void __launch_bounds__(256)
silu_mul_kernel(const float* __restrict__ gate, const float* __restrict__ up, int16_t* __restrict__ out, long long total)
{
    grid_launch_dependents();
    grid_dependency_wait();
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;   // four elements per thread
    if (i >= total) return;
    const bool vec = i + 3 < total && ((reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(up)) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(out) & 7) == 0;
    if (vec) {
        const float4 g = *reinterpret_cast<const float4*>(gate + i), u = *reinterpret_cast<const float4*>(up + i);
        const uint32_t lo = (uint16_t)float_to_bf16_rne(g.x / (1.0f + expf(-g.x)) * u.x) |
                            ((uint32_t)(uint16_t)float_to_bf16_rne(g.y / (1.0f + expf(-g.y)) * u.y) << 16);
        const uint32_t hi = (uint16_t)float_to_bf16_rne(g.z / (1.0f + expf(-g.z)) * u.z) |
                            ((uint32_t)(uint16_t)float_to_bf16_rne(g.w / (1.0f + expf(-g.w)) * u.w) << 16);
        *reinterpret_cast<uint2*>(out + i) = make_uint2(lo, hi);
        return;
    }
    for (long long j = i; j < total && j < i + 4; j++) {
        const float g = gate[j];
        out[j] = float_to_bf16_rne(g / (1.0f + expf(-g)) * up[j]);
    }
}
__global__ void __launch_bounds__(256)
add_kernel(float* __restrict__ y, const float* __restrict__ x, long long total)
{
    grid_launch_dependents();
    grid_dependency_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < total) y[i] += x[i];
}

// ---------------------------------------------------------------------------
// RoPE on q and k (rotate-half form, engine/kernels.hip:174-215, 717-756) and
// INT8 KV store with one scale per (position, kv head): scale = absmax/127,
// value = clamp(rint(v * 127/absmax), -127, 127) (engine/kernels.hip:220-303,
// 760-845).  One launch: warp (h, seq) with h < n_head rotates q head h;
// n_head <= h < n_head + n_head_kv rotates k head (written back, as the engine
// does) and stores it; the last n_head_kv warps store v.  store == 0: rotation
// only (launch_rope_batch); rope == 0: store only (launch_store_kv_batch).
// ---------------------------------------------------------------------------
struct RopeFreqs { float f[128]; };                              // head_dim <= 256

struct RopeKvParams {
    float* q; float* k; const float* v;
    int8_t* kv_k; int8_t* kv_v; float* sc_k; float* sc_v;
    const int* positions;       // null: every sequence uses `position`
    int position;
    int head_dim, n_head, n_head_kv;
    int q_stride, k_stride;     // floats between sequences in q and k/v
    long long kv_stride;        // int8 elements between the sequences' caches (0: one shared cache)
    int store;
    int cta_slots;              // groups of warps of a CTA, each with heads of its own
};

constexpr int kRopeWarps = 4;
__host__ __device__ constexpr int rope_head_warps(int head_dim) { return (head_dim / 2 + 31) / 32; }

__device__ __forceinline__ int8_t quantise(float v, float inv) { return (int8_t)(int)fminf(fmaxf(rintf(v * inv), -127.f), 127.f); }
// where a kv head of this sequence's position lies in the caches
struct KvSlot { int8_t* dst; float* scale; };
__device__ __forceinline__ KvSlot kv_slot(const RopeKvParams& P, int seq, int pos, int kvh, bool is_v)
{
    return {(is_v ? P.kv_v : P.kv_k) + (size_t)seq * P.kv_stride + ((size_t)pos * P.n_head_kv + kvh) * P.head_dim,
            (is_v ? P.sc_v : P.sc_k) + (size_t)seq * (P.kv_stride / P.head_dim) + (size_t)pos * P.n_head_kv + kvh};
}

// The store alone: a warp per head, no shared memory; a lane owns elements d and d + half for d = lane, lane + 32, ...
// Bound by latency.  32 kv heads of 128 at B = 256: 5.4 us (a thread per pair, as below: 8.6); 8 at B = 1: 1.3 us.
__global__ void __launch_bounds__(kRopeWarps * 32)
store_kv_kernel(const __grid_constant__ RopeKvParams P)
{
    grid_launch_dependents();
    const int lane = threadIdx.x & 31, h = blockIdx.x * kRopeWarps + (threadIdx.x >> 5), seq = blockIdx.y;
    const int hd = P.head_dim, half = hd >> 1;
    if (h >= 2 * P.n_head_kv) return;
    const bool is_v = h >= P.n_head_kv;
    const int kvh = h - (is_v ? P.n_head_kv : 0);
    const float* p = (is_v ? P.v : P.k) + (size_t)seq * P.k_stride + (size_t)kvh * hd;
    grid_dependency_wait();
    const int pos = P.positions ? P.positions[seq] : P.position;
    float lo[4], hi[4], amax = 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int d = i * 32 + lane;
        lo[i] = d < half ? p[d] : 0.f;
        hi[i] = d < half ? p[d + half] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) amax = fmaxf(amax, fmaxf(fabsf(lo[i]), fabsf(hi[i])));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, off));
    const float inv = amax > 0.f ? 127.0f / amax : 0.f;
    const KvSlot at = kv_slot(P, seq, pos, kvh, is_v);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int d = i * 32 + lane;
        if (d < half) { at.dst[d] = quantise(lo[i], inv); at.dst[d + half] = quantise(hi[i], inv); }
    }
    if (lane == 0) *at.scale = amax / 127.0f;
}

// A thread owns elements d and d + half of kHeads neighbouring heads, whose angles are the same, and runs sincosf once; a
// head lies over ceil(half / 32) neighbouring warps of a CTA.  Bound by latency: the addresses are there before the wait
// for the launch before.  In a chain of launches, 32 + 8 heads of 128, us at B = 1 / 64 / 256: a CTA per head with two
// block reductions 2.0 / 4.4 / 13.1; a warp per head, two sines a lane one after the other, 2.3 / 4.2 / 8.1; this way with
// one head a thread 1.75 / 3.8 / 8.8, with two 1.95 / 2.9 / 6.0.
template <int kHeads>
__global__ void __launch_bounds__(kRopeWarps * 32)
rope_kv_kernel(const __grid_constant__ RopeKvParams P, const __grid_constant__ RopeFreqs F)
{
    __shared__ float top[kHeads][kRopeWarps];
    grid_launch_dependents();
    const int hd = P.head_dim, half = hd >> 1, wph = rope_head_warps(hd), slots = P.cta_slots;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, seq = blockIdx.y;
    const int slot = slots == 4 ? warp : slots == 2 ? warp >> 1 : 0, d = (warp - slot * wph) * 32 + lane;
    const int h0 = (blockIdx.x * slots + slot) * kHeads, first_v = P.n_head + P.n_head_kv, end = first_v + (P.store ? P.n_head_kv : 0);
    float* p[kHeads];
    bool live[kHeads];
#pragma unroll
    for (int j = 0; j < kHeads; j++) {
        const int h = h0 + j;
        live[j] = d < half && h < end;
        p[j] = (h < P.n_head ? P.q + (size_t)seq * P.q_stride + (size_t)h * hd
                             : (h < first_v ? P.k + (size_t)(h - P.n_head) * hd : const_cast<float*>(P.v) + (size_t)(h - first_v) * hd) + (size_t)seq * P.k_stride) + d;
    }
    grid_dependency_wait();
    const int pos = P.positions ? P.positions[seq] : P.position;
    float lo[kHeads], hi[kHeads];
#pragma unroll
    for (int j = 0; j < kHeads; j++) {
        lo[j] = live[j] ? p[j][0] : 0.f;
        hi[j] = live[j] ? p[j][half] : 0.f;
    }
    if (d < half && h0 < first_v) {
        float s, c;
        sincosf((float)pos * F.f[d], &s, &c);
#pragma unroll
        for (int j = 0; j < kHeads; j++) {
            if (h0 + j >= first_v) break;
            const float x0 = lo[j], x1 = hi[j];
            lo[j] = x0 * c - x1 * s; hi[j] = x0 * s + x1 * c;
            p[j][0] = lo[j]; p[j][half] = hi[j];
        }
    }
    if (!P.store || (int)(blockIdx.x + 1) * slots * kHeads <= P.n_head) return;   // the whole CTA
    float amax[kHeads];
#pragma unroll
    for (int j = 0; j < kHeads; j++) {
        amax[j] = fmaxf(fabsf(lo[j]), fabsf(hi[j]));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) amax[j] = fmaxf(amax[j], __shfl_xor_sync(0xFFFFFFFFu, amax[j], off));
        if (lane == 0) top[j][warp] = amax[j];
    }
    if (wph > 1) {
        __syncthreads();
        for (int i = 0; i < wph; i++)
#pragma unroll
            for (int j = 0; j < kHeads; j++) amax[j] = fmaxf(amax[j], top[j][slot * wph + i]);
    }
#pragma unroll
    for (int j = 0; j < kHeads; j++) {
        const int h = h0 + j;
        if (d >= half || h < P.n_head || h >= end) continue;
        const bool is_v = h >= first_v;
        const float inv = amax[j] > 0.f ? 127.0f / amax[j] : 0.f;
        const KvSlot at = kv_slot(P, seq, pos, h - (is_v ? first_v : P.n_head), is_v);
        at.dst[d] = quantise(lo[j], inv);
        at.dst[d + half] = quantise(hi[j], inv);
        if (d == 0) *at.scale = amax[j] / 127.0f;
    }
}

// ---------------------------------------------------------------------------
// Decode attention over the INT8 cache (engine/kernels.hip:499-586, 606-692):
// scores[t] = scale * sum_d q[d] * (k[t][d] * sk[t]); softmax over t <= pos;
// out[d] = sum_t p[t] * (v[t][d] * sv[t]) -> bf16.
// CTA = (kv head, sequence, slice of the positions), 8 warps: the key and value
// rows of a kv head are read once for all the query heads that share it (GQA).
// Both passes walk the positions one warp per position, a lane reading four
// consecutive int8 of the row (128 contiguous bytes per warp for head_dim 128),
// eight positions in flight per warp; a lane keeps its four q values of every
// query head in registers.  The round's 8 x heads partial dot products are summed
// over the lanes by a halving butterfly (31 shuffles per 32 sums; the kernel is
// bound by instruction issue at large batch, and 5 shuffles per sum were half of it).  Softmax statistics are per query head and per
// slice (one warp per head, shuffles only).  With few sequences the positions
// are cut into slices that run as one thread-block cluster, and the slices'
// (max, sum, weighted values) are merged over distributed shared memory --
// split-KV decoding without a second kernel or a workspace.
// ---------------------------------------------------------------------------
struct AttnParams {
    const float* q; const int8_t* kc; const int8_t* vc; const float* sk; const float* sv;
    int16_t* out;
    const int* positions;       // null: seq_len for every sequence
    int seq_len;
    int n_head, n_head_kv, head_dim;
    long long kv_stride;
    float scale;
    int score_stride;           // floats between the score rows of two query heads in shared memory
    int nsplit;                 // CTAs (= cluster size) that share the positions of one (kv head, sequence)
    int t_limit;                // the caller's bound: positions a launch may read, whatever `positions` holds
    int stages;                 // attention_mma_kernel: chunks of a warp's ring in shared memory
};

constexpr int kAttnThreads = 256;
constexpr int kAttnWarps = kAttnThreads / 32;
constexpr int kAttnFlight = 8;           // positions in flight per warp
// exponentials of softmax weights use the fast intrinsic: arguments are <= 0 and the result feeds a bf16 output

__device__ __forceinline__ void unpack_s8x4(int w, float (&f)[4])
{
    f[0] = (float)(int8_t)(w & 0xFF); f[1] = (float)(int8_t)((w >> 8) & 0xFF);
    f[2] = (float)(int8_t)((w >> 16) & 0xFF); f[3] = (float)(int8_t)(w >> 24);
}
__device__ __forceinline__ float ld_dsmem_f32(uint32_t addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_dsmem_f32x4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t dsmem_addr(const void* p, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_barrier()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int kGqa, int kChunks>         // kChunks: 128-element pieces of a head (head_dim <= 128 * kChunks)
// four CTAs per SM (64 registers) up to four query heads per kv head: measured +1.3 % on a B=256 step over three
__global__ void __launch_bounds__(kAttnThreads, kGqa <= 4 ? 4 : 1)
attention_kernel(const __grid_constant__ AttnParams P)
{
    // scores[kGqa][score_stride], acc[warps][kGqa][head_dim] (reused as the slice's sum [kGqa][head_dim]), stats[2][kGqa]
    extern __shared__ float att_smem[];
    grid_launch_dependents();
    grid_dependency_wait();
    const int kvh = blockIdx.x, seq = blockIdx.y, split = blockIdx.z, nsplit = P.nsplit;
    const int hd = P.head_dim;
    const int Tw = P.positions ? P.positions[seq] + 1 : P.seq_len;
    const int T = Tw < P.t_limit ? Tw : P.t_limit;                 // never past the caller's bound
    const int per = (T + nsplit - 1) / nsplit;
    const int t_lo = split * per, t_hi = t_lo + per < T ? t_lo + per : T;       // this CTA's positions
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t kv_dim = (size_t)P.n_head_kv * hd;
    const int8_t* kc = P.kc + (size_t)seq * P.kv_stride + (size_t)kvh * hd;
    const int8_t* vc = P.vc + (size_t)seq * P.kv_stride + (size_t)kvh * hd;
    const float* sk = P.sk + (size_t)seq * (P.kv_stride / hd) + kvh;
    const float* sv = P.sv + (size_t)seq * (P.kv_stride / hd) + kvh;
    const float* q = P.q + ((size_t)seq * P.n_head + (size_t)kvh * kGqa) * hd;
    const int ss = P.score_stride;
    float* scores = att_smem;
    float* accs = att_smem + (size_t)kGqa * ss;
    float* stats = accs + (size_t)kAttnWarps * kGqa * hd;        // [0][h]: slice maximum, [1][h]: slice sum of exp
    float* sk_s = stats + 2 * kGqa;                               // this slice's key and value scales (strided in memory)
    float* sv_s = sk_s + ss;
    for (int i = threadIdx.x; i < t_hi - t_lo; i += kAttnThreads) {
        sk_s[i] = sk[(size_t)(t_lo + i) * P.n_head_kv];
        sv_s[i] = sv[(size_t)(t_lo + i) * P.n_head_kv];
    }

    // a lane owns elements [128*c + 4*lane, +4) of the head, c < kChunks
    bool live[kChunks];
    float qv[kGqa][kChunks][4];
#pragma unroll
    for (int c = 0; c < kChunks; c++) {
        live[c] = c * 128 + lane * 4 < hd;                        // head_dim is a multiple of 4
#pragma unroll
        for (int h = 0; h < kGqa; h++)
#pragma unroll
            for (int e = 0; e < 4; e++) qv[h][c][e] = live[c] ? q[(size_t)h * hd + c * 128 + lane * 4 + e] : 0.f;
    }
    __syncthreads();
    // ---- scores of this slice (indexed from t_lo in shared memory)
    for (int t0 = t_lo + warp; t0 < t_hi; t0 += kAttnFlight * kAttnWarps) {
        int w[kAttnFlight][kChunks];
#pragma unroll
        for (int u = 0; u < kAttnFlight; u++) {
            const int t = t0 + u * kAttnWarps;
#pragma unroll
            for (int c = 0; c < kChunks; c++)
                w[u][c] = (t < t_hi && live[c]) ? *reinterpret_cast<const int*>(kc + (size_t)t * kv_dim + c * 128 + lane * 4) : 0;
        }
        // partial dot products of the round: value v = u * kGqa + h (position u of the round, query head h)
        constexpr int V = kAttnFlight * kGqa;
        float dot[V];
#pragma unroll
        for (int v = 0; v < V; v++) dot[v] = 0.f;
#pragma unroll
        for (int u = 0; u < kAttnFlight; u++) {
#pragma unroll
            for (int c = 0; c < kChunks; c++) {
                float kf[4];
                unpack_s8x4(w[u][c], kf);
#pragma unroll
                for (int h = 0; h < kGqa; h++)
                    dot[u * kGqa + h] += qv[h][c][0] * kf[0] + qv[h][c][1] * kf[1] + qv[h][c][2] * kf[2] + qv[h][c][3] * kf[3];
            }
        }
        if (V % 32 == 0) {
            // Sums over the 32 lanes of 32 values at a time by a butterfly that halves the values a lane carries at
            // every step (31 shuffles for 32 sums instead of 5 each); lane l ends with the sum of value 32 g + l.
#pragma unroll
            for (int g = 0; g < V / 32; g++) {
                float r16[16], r8[8], r4[4], r2[2];
                const bool b16 = lane & 16, b8 = lane & 8, b4 = lane & 4, b2 = lane & 2, b1 = lane & 1;
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float keep = b16 ? dot[g * 32 + 16 + i] : dot[g * 32 + i], send = b16 ? dot[g * 32 + i] : dot[g * 32 + 16 + i];
                    r16[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 16);
                }
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float keep = b8 ? r16[8 + i] : r16[i], send = b8 ? r16[i] : r16[8 + i];
                    r8[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 8);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float keep = b4 ? r8[4 + i] : r8[i], send = b4 ? r8[i] : r8[4 + i];
                    r4[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 4);
                }
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float keep = b2 ? r4[2 + i] : r4[i], send = b2 ? r4[i] : r4[2 + i];
                    r2[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 2);
                }
                const float keep = b1 ? r2[1] : r2[0], send = b1 ? r2[0] : r2[1];
                const float total = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 1);
                const int v = g * 32 + lane, u = v / kGqa, h = v - u * kGqa;
                const int t = t0 + u * kAttnWarps;
                if (t < t_hi) scores[h * ss + (t - t_lo)] = total * sk_s[t - t_lo] * P.scale;
            }
        } else {
#pragma unroll
            for (int u = 0; u < kAttnFlight; u++) {
                const int t = t0 + u * kAttnWarps;
                if (t >= t_hi) break;
#pragma unroll
                for (int h = 0; h < kGqa; h++)
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) dot[u * kGqa + h] += __shfl_xor_sync(0xFFFFFFFFu, dot[u * kGqa + h], off);
                if (lane < kGqa) {
                    float mine = dot[u * kGqa];
#pragma unroll
                    for (int h = 1; h < kGqa; h++) mine = lane == h ? dot[u * kGqa + h] : mine;
                    scores[lane * ss + (t - t_lo)] = mine * sk_s[t - t_lo] * P.scale;
                }
            }
        }
    }
    __syncthreads();
    // ---- slice softmax, warp h for query head h; the value scale is folded into the weight
    const int n_loc = t_hi > t_lo ? t_hi - t_lo : 0;
    for (int h = warp; h < kGqa; h += kAttnWarps) {
        float m = -1e30f;
        for (int i = lane; i < n_loc; i += 32) m = fmaxf(m, scores[h * ss + i]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, off));
        float sum = 0.f;
        for (int i = lane; i < n_loc; i += 32) {
            const float e = __expf(scores[h * ss + i] - m);
            scores[h * ss + i] = e * sv_s[i];
            sum += e;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, off);
        if (lane == 0) { stats[h] = m; stats[kGqa + h] = sum; }
    }
    __syncthreads();
    // ---- weighted values of this slice
    float acc[kGqa][kChunks][4];
#pragma unroll
    for (int h = 0; h < kGqa; h++)
#pragma unroll
        for (int c = 0; c < kChunks; c++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[h][c][e] = 0.f;
    for (int t0 = t_lo + warp; t0 < t_hi; t0 += kAttnFlight * kAttnWarps) {
        int w[kAttnFlight][kChunks];
#pragma unroll
        for (int u = 0; u < kAttnFlight; u++) {
            const int t = t0 + u * kAttnWarps;
#pragma unroll
            for (int c = 0; c < kChunks; c++)
                w[u][c] = (t < t_hi && live[c]) ? *reinterpret_cast<const int*>(vc + (size_t)t * kv_dim + c * 128 + lane * 4) : 0;
        }
#pragma unroll
        for (int u = 0; u < kAttnFlight; u++) {
            const int t = t0 + u * kAttnWarps;
            if (t >= t_hi) break;
            float p[kGqa];
#pragma unroll
            for (int h = 0; h < kGqa; h++) p[h] = scores[h * ss + (t - t_lo)];
#pragma unroll
            for (int c = 0; c < kChunks; c++) {
                float vf[4];
                unpack_s8x4(w[u][c], vf);
#pragma unroll
                for (int h = 0; h < kGqa; h++)
#pragma unroll
                    for (int e = 0; e < 4; e++) acc[h][c][e] += p[h] * vf[e];
            }
        }
    }
#pragma unroll
    for (int h = 0; h < kGqa; h++)
#pragma unroll
        for (int c = 0; c < kChunks; c++)
            if (live[c])
                *reinterpret_cast<float4*>(accs + ((size_t)warp * kGqa + h) * hd + c * 128 + lane * 4) =
                    make_float4(acc[h][c][0], acc[h][c][1], acc[h][c][2], acc[h][c][3]);
    __syncthreads();
    // the slice's sums over its warps, in place in the first warp's rows
    for (int i = threadIdx.x; i < kGqa * hd; i += kAttnThreads) {
        float a = 0.f;
#pragma unroll
        for (int wv = 0; wv < kAttnWarps; wv++) a += accs[(size_t)wv * kGqa * hd + i];
        accs[i] = a;                                               // element i of warp 0's rows: read above by this thread only
    }
    if (nsplit == 1) {
        __syncthreads();
        for (int i = threadIdx.x; i < kGqa * hd; i += kAttnThreads) {
            const int h = i / hd, d = i - h * hd;
            P.out[((size_t)seq * P.n_head + (size_t)kvh * kGqa + h) * hd + d] = float_to_bf16_rne(accs[i] / stats[kGqa + h]);
        }
        return;
    }
    // ---- merge the slices of the cluster: rank r finishes the output elements i = r, r + nsplit, ...
    cluster_barrier();                                            // every slice's sums and statistics are in place
    for (int i = split * kAttnThreads + threadIdx.x; i < kGqa * hd; i += nsplit * kAttnThreads) {
        const int h = i / hd, d = i - h * hd;
        float m = -1e30f;
        for (int r = 0; r < nsplit; r++) m = fmaxf(m, ld_dsmem_f32(dsmem_addr(stats + h, r)));
        float num = 0.f, den = 0.f;
        for (int r = 0; r < nsplit; r++) {
            const float wgt = __expf(ld_dsmem_f32(dsmem_addr(stats + h, r)) - m);   // an empty slice has max -1e30: weight 0
            num += wgt * ld_dsmem_f32(dsmem_addr(accs + i, r));
            den += wgt * ld_dsmem_f32(dsmem_addr(stats + kGqa + h, r));
        }
        P.out[((size_t)seq * P.n_head + (size_t)kvh * kGqa + h) * hd + d] = float_to_bf16_rne(num / den);
    }
    cluster_barrier();                                            // nobody reads this CTA's shared memory any more
}

// ---------------------------------------------------------------------------
// The same attention on the tensor cores, for head_dim 64 / 96 / 128 and 16-byte aligned caches.
// Bound: the cache, 2 * head_dim + 8 bytes a position and kv head (11 clocks of an SM's share of HBM at head_dim 128).
// The kernel above needs ~60 clocks for them (an int8 -> float conversion per element on the quarter-rate pipe, a
// multiply-add per element and query head, the shuffles of the dot products): 0.8 TB/s at 24 sequences of 2-4 k
// positions, 195 us.  Here both products are mma.m16n8k16 with the cache as the B operand, one kv head's query heads in
// the A rows.  The operands are exact: an int8 is exact in bf16, and a 32-bit q (or softmax weight times value scale) is
// cut into three bf16 pieces of 8 significant bits, which are exact together.  With up to four query heads the pieces
// sit in rows 0-3, 4-7 and 8-11 of one MMA; with eight, in rows 0-7 and 8-15 of one and rows 8-15 of a second.
// The sums are 32-bit.  An MMA cuts off what does not fit its accumulator, which is a bias that grows with the number of
// MMAs chained on it: so the low pieces never share a row with the high ones (their additions would cut the large sum
// once more), and the weighted values of a chunk start from zero and are added to the sums rounded to nearest.  Outputs
// that are not the bf16 value nearest to the 64-bit result, of 10^4, general kernel / chained accumulators / as here:
// 56 sequences of 3.5-7 k positions 5.8 / 9.2 / 4.1, with eight query heads per kv head 4.8 / 19.9 / 3.4; 256 of 8-16
// positions, one query head 1.24 / 1.51 / 1.05.  The times are the same (752 / 215 / 210 us, 14.3 / 12.7 / 12.3 us).
// A warp walks chunks of 16 positions with a running maximum; cp.async keeps two or three chunks (8-12 KB) in flight per
// warp, sixteen warps per SM (128 registers: q is read from shared memory again for every chunk; with q in registers
// twelve warps were resident: 31 against 30 us on 256 x 192 positions, 51 against 53 on 24 x 4096).  The partial results
// of a CTA's warps meet in shared memory, those of a cluster's CTAs over distributed shared memory as above.
// Measured, 32/8 heads of 128: 24 sequences of 2-4 k positions 195 -> 54 us (2.9 TB/s); bound now by instruction issue
// (about 620 instructions a chunk, the ALU pipe half busy with the int8 conversions) and the CTAs' dependent start.
// ---------------------------------------------------------------------------
constexpr int kMmaWarps = 8;             // most warps of a CTA
constexpr int kMmaPos = 16;              // positions of a chunk
constexpr int kMmaStages = 3;
constexpr int kMmaHeads = 8;             // most query heads per kv head
__host__ __device__ constexpr int mma_stage_bytes(int hd) { return 2 * kMmaPos * hd + 2 * kMmaPos * 4; }   // K, V, scales
// A warp's weighted values in shared memory: the kHD / 8 consecutive dims that a lane holds of a column, padded so that
// the 16-byte stores of a quarter warp (two heads, four columns two apart) meet different banks.
__host__ __device__ constexpr int mma_acc_col(int hd) { return hd == 64 ? 12 : 20; }
__host__ __device__ constexpr int mma_acc_row(int hd) { return 8 * mma_acc_col(hd) + 4; }
__host__ __device__ constexpr int mma_smem_bytes(int hd, int warps, int stages, int heads)
{
    return warps * stages * mma_stage_bytes(hd) + (2 * kMmaWarps + 2) * kMmaHeads * 4 + 3 * heads * (hd / 4 + 1) * 8;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ float exp2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// int8 in the low byte of each half of x (the high bytes are ignored) -> two bf16, exact:
// the seven magnitude bits above 128, minus 128, or minus 256 where the sign bit is set.
__device__ __forceinline__ uint32_t s8_pair_to_bf16(uint32_t x)
{
    uint32_t v;
    const uint32_t mag = and_or(x, 0x007F007Fu, 0x43004300u), off = and_or(x, 0x00800080u, 0xC300C300u);
    asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(v) : "r"(mag), "r"(off));
    return v;
}
// x = hi + mid + lo, each with at most 8 significant bits (in the upper half of a register).  An infinity stays in hi
// alone; a NaN stays a NaN in hi whatever its payload.
__device__ __forceinline__ void split_bf16x3(float x, float& hi, float& mid, float& lo)
{
    const uint32_t u = __float_as_uint(x);
    hi = __uint_as_float(x == x ? u & 0xFFFF0000u : 0x7FFF0000u);
    const float r = hi == x ? 0.f : x - hi;
    mid = __uint_as_float(__float_as_uint(r) & 0xFFFF0000u);
    lo = r == mid ? 0.f : r - mid;
}
// the upper halves of two registers as one bf16 pair (a in the low half)
__device__ __forceinline__ uint32_t pack_hi16(float a, float b) { return prmt(__float_as_uint(a), __float_as_uint(b), 0x7632u); }

// the same for the product of two floats, whose NaN the hardware makes canonical
__device__ __forceinline__ void split_product_bf16x3(float x, float& hi, float& mid, float& lo)
{
    hi = __uint_as_float(__float_as_uint(x) & 0xFFFF0000u);
    const float r = hi == x ? 0.f : x - hi;
    mid = __uint_as_float(__float_as_uint(r) & 0xFFFF0000u);
    lo = r - mid;
}

template <int kHD, bool kWide>           // kWide: eight query heads per kv head, else up to four
__global__ void __launch_bounds__(kMmaWarps * 32, 2)
attention_mma_kernel(const __grid_constant__ AttnParams P)
{
    constexpr int kSteps = kHD / 16;     // MMA steps of the QK product
    constexpr int kTiles = kHD / 8;      // MMA column tiles of the PV product = dims per lane group
    constexpr int kRowPieces = kHD / 16; // 16-byte pieces of a cache row
    constexpr int kStage = mma_stage_bytes(kHD);
    extern __shared__ __align__(16) uint8_t mma_smem[];
    const int nwarps = blockDim.x >> 5;
    float* part_stats = reinterpret_cast<float*>(mma_smem + nwarps * P.stages * kStage);   // [warp][max, sum][head]
    float* stats = part_stats + 2 * kMmaWarps * kMmaHeads;                                      // the CTA's [max, sum][head]
    grid_launch_dependents();
    grid_dependency_wait();
    const int kvh = blockIdx.x, seq = blockIdx.y, split = blockIdx.z, nsplit = P.nsplit;
    const int gqa = kWide ? 8 : P.n_head / P.n_head_kv;
    const int Tw = P.positions ? P.positions[seq] + 1 : P.seq_len;
    const int T = Tw < P.t_limit ? Tw : P.t_limit;
    const int per = ((T + nsplit - 1) / nsplit + kMmaPos - 1) & ~(kMmaPos - 1);
    const int t_lo = split * per, t_hi = t_lo + per < T ? t_lo + per : T;       // this CTA's positions
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const size_t kv_dim = (size_t)P.n_head_kv * kHD;
    const int8_t* kc = P.kc + (size_t)seq * P.kv_stride + (size_t)kvh * kHD;
    const int8_t* vc = P.vc + (size_t)seq * P.kv_stride + (size_t)kvh * kHD;
    const float* scales = (lane < kMmaPos ? P.sk : P.sv) + (size_t)seq * (P.kv_stride / kHD) + kvh;
    const float* q = P.q + ((size_t)seq * P.n_head + (size_t)kvh * gqa) * kHD;
    // P.stages < kMmaStages: no warp has more chunks than that, and every chunk keeps a stage of its own
    const int ring_bytes = P.stages * kStage;
    uint8_t* ring = mma_smem + warp * ring_bytes;
    const uint32_t ring_s = smem_addr(ring);

    // A chunk in shared memory: K rows, V rows, 16 + 16 scales.  The 16-byte pieces of a row are permuted so that the
    // lanes of a load phase meet different banks: K is read four pieces of two neighbouring rows at a time, V two (one
    // and a half) pieces of four rows that lie two apart.
    auto k_piece = [](int r, int c) { return kHD == 128 ? c ^ ((r & 1) << 2) : c; };
    auto v_piece = [](int r, int c) { return kHD == 128 ? c ^ (((r >> 1) & 3) << 1) : kHD == 64 ? c ^ (((r >> 1) & 1) << 1) : c; };
    const int first = t_lo + warp * kMmaPos, stride = nwarps * kMmaPos;
    const int n = first < t_hi ? (t_hi - first + stride - 1) / stride : 0;      // this warp's chunks
    // what a lane copies of a chunk: pieces j * 32 + lane of its rows, the same in every chunk
    uint32_t src_off[kRowPieces / 2], dst_k[kRowPieces / 2], dst_v[kRowPieces / 2];
#pragma unroll
    for (int j = 0; j < kRowPieces / 2; j++) {
        const int p = j * 32 + lane, r = p / kRowPieces, c = p - r * kRowPieces;
        src_off[j] = (uint32_t)r * (uint32_t)kv_dim + c * 16;
        dst_k[j] = r * kHD + k_piece(r, c) * 16;
        dst_v[j] = (kMmaPos + r) * kHD + v_piece(r, c) * 16;
    }
    const int8_t* k_next = kc + (size_t)first * kv_dim;
    const int8_t* v_next = vc + (size_t)first * kv_dim;
    const float* s_next = scales + (size_t)first * P.n_head_kv;
    const uint32_t s_off = (uint32_t)(lane & (kMmaPos - 1)) * P.n_head_kv;
    auto fetch = [&](int i) {
        if (i < n) {
            const int left = t_hi - (first + i * stride);          // positions of this chunk, 16 or more except in the last
            const uint32_t dst = ring_s + (uint32_t)(i % kMmaStages) * kStage;
            if (left >= kMmaPos) {
#pragma unroll
                for (int j = 0; j < kRowPieces / 2; j++) {
                    cp_async16(dst + dst_k[j], k_next + src_off[j]);
                    cp_async16(dst + dst_v[j], v_next + src_off[j]);
                }
                cp_async4(dst + 2 * kMmaPos * kHD + lane * 4, s_next + s_off);
            } else {                                               // rows past the end: the last one again
#pragma unroll
                for (int j = 0; j < kRowPieces / 2; j++) {
                    const int r = (j * 32 + lane) / kRowPieces;
                    const uint32_t off = src_off[j] - (r < left ? 0u : (uint32_t)(r - left + 1) * (uint32_t)kv_dim);
                    cp_async16(dst + dst_k[j], k_next + off);
                    cp_async16(dst + dst_v[j], v_next + off);
                }
                const int r = lane & (kMmaPos - 1);
                cp_async4(dst + 2 * kMmaPos * kHD + lane * 4, s_next + (r < left ? r : left - 1) * P.n_head_kv);
            }
            k_next += (size_t)stride * kv_dim; v_next += (size_t)stride * kv_dim; s_next += stride * P.n_head_kv;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < kMmaStages - 1; i++) fetch(i);

    // q as A operand, cut once per CTA: pieces[piece][head][four dims], the four in the order 0, 2, 1, 3 (the bytes that
    // one mask of a cache word leaves side by side).  MMA step s, lane t4 stands for four consecutive dims.
    constexpr int kHeads = kWide ? 8 : 4;
    uint2* pieces = reinterpret_cast<uint2*>(stats + 2 * kMmaHeads);
    constexpr int kPieceRow = kHD / 4 + 1;                         // one more: the rows of a load phase on different banks
    for (int i = threadIdx.x; i < kHeads * kHD / 4; i += blockDim.x) {
        float hi[4], mid[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; e++) split_bf16x3(i * 4 < gqa * kHD ? q[i * 4 + e] : 0.f, hi[e], mid[e], lo[e]);
        uint2* at = pieces + i / (kHD / 4) * kPieceRow + i % (kHD / 4);
        at[0] = make_uint2(pack_hi16(hi[0], hi[2]), pack_hi16(hi[1], hi[3]));
        at[kHeads * kPieceRow] = make_uint2(pack_hi16(mid[0], mid[2]), pack_hi16(mid[1], mid[3]));
        at[2 * kHeads * kPieceRow] = make_uint2(pack_hi16(lo[0], lo[2]), pack_hi16(lo[1], lo[3]));
    }
    __syncthreads();
    const int head = kWide ? g : g & 3;                            // query head of this lane's rows (g and g + 8)
    const uint2* q_row = pieces + head * kPieceRow + (kHD == 96 ? t4 * 2 : t4 * 4) + (kWide || g < 4 ? 0 : kHeads * kPieceRow);
    const float to_log2 = P.scale * 1.4426950408889634f;           // weights are powers of two of the scaled scores

    float acc[kTiles][2];
#pragma unroll
    for (int j = 0; j < kTiles; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) acc[j][e] = 0.f;
    float m = -1e30f, l = 0.f;
#pragma unroll 1
    for (int i = 0; i < n; i++) {
        cp_async_wait<kMmaStages - 2>();
        __syncwarp();                                              // this chunk has landed; the one before has been read
        fetch(i + kMmaStages - 1);
        const uint8_t* K = ring + (i % kMmaStages) * kStage;
        const uint8_t* V = K + kMmaPos * kHD;
        const float* sc = reinterpret_cast<const float*>(V + kMmaPos * kHD);
        const int t0 = first + i * stride + 2 * t4;                // this lane's positions: t0 + 8 u + {0, 1}
        float dot[2][2], to_w[2][2];                               // a score is their product
        float mx = -1e30f;
        uint32_t kw[2][kSteps];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int r = u * 8 + g;
            if (kHD == 96) {
#pragma unroll
                for (int b = 0; b < 3; b++) {
                    const uint2 x = *reinterpret_cast<const uint2*>(K + r * kHD + b * 32 + t4 * 8);
                    kw[u][2 * b] = x.x; kw[u][2 * b + 1] = x.y;
                }
            } else {
#pragma unroll
                for (int b = 0; b < kSteps / 4; b++) {
                    const uint4 x = *reinterpret_cast<const uint4*>(K + r * kHD + k_piece(r, b * 4 + t4) * 16);
                    kw[u][4 * b] = x.x; kw[u][4 * b + 1] = x.y; kw[u][4 * b + 2] = x.z; kw[u][4 * b + 3] = x.w;
                }
            }
        }
        // q is read again for every chunk: its 32 registers would cost a quarter of the resident warps
        float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int s = 0; s < kSteps; s++) {
            const uint2* at = q_row + (kHD == 96 ? (s >> 1) * 8 + (s & 1) : (s >> 2) * 16 + (s & 3));
            const uint2 x0 = at[0];
            const uint2 x1 = kWide ? at[kHeads * kPieceRow] : g < 4 ? at[2 * kHeads * kPieceRow] : make_uint2(0u, 0u);
            const uint2 x2 = kWide ? at[2 * kHeads * kPieceRow] : make_uint2(0u, 0u);
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const uint32_t b0 = s8_pair_to_bf16(kw[u][s]), b1 = s8_pair_to_bf16(kw[u][s] >> 8);
                mma_bf16_16816(c[u], x0.x, x1.x, x0.y, x1.y, b0, b1);
                if (kWide) mma_bf16_16816(c[u], 0u, x2.x, 0u, x2.y, b0, b1);
            }
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                float x = c[u][e] + c[u][2 + e];
                if (!kWide) x += __shfl_xor_sync(0xFFFFFFFFu, x, 16);
                dot[u][e] = x;
                to_w[u][e] = sc[u * 8 + 2 * t4 + e] * to_log2;
                if (t0 + u * 8 + e < t_hi) mx = fmaxf(mx, x * to_w[u][e]);
            }
        }
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 2));
        // Weights are 2^(score - m), the difference rounded once.  m is at least the maximum so far: two above a new one,
        // so that the sums are rarely rescaled, and a whole number, so that rescaling is exact.
        if (__any_sync(0xFFFFFFFFu, mx > m)) {
            const float mn = mx > m ? ceilf(mx) + 2.f : m, f = exp2_approx(m - mn);
            m = mn;
            if (i > 0) {
                l *= f;
#pragma unroll
                for (int j = 0; j < kTiles; j++)
#pragma unroll
                    for (int e = 0; e < 2; e++) acc[j][e] *= f;
            }
        }
        uint32_t ap[4], apl[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            float hi[2], mid[2], lo[2];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const bool live = t0 + u * 8 + e < t_hi;
                const float p = live ? exp2_approx(fmaf(dot[u][e], to_w[u][e], -m)) : 0.f;
                l += p;
                split_product_bf16x3(live ? p * sc[kMmaPos + u * 8 + 2 * t4 + e] : 0.f, hi[e], mid[e], lo[e]);
            }
            if (kWide) {
                ap[2 * u] = pack_hi16(hi[0], hi[1]); ap[2 * u + 1] = pack_hi16(mid[0], mid[1]);
                apl[u] = pack_hi16(lo[0], lo[1]);
            } else {
                ap[2 * u] = g < 4 ? pack_hi16(hi[0], hi[1]) : pack_hi16(mid[0], mid[1]);
                ap[2 * u + 1] = g < 4 ? pack_hi16(lo[0], lo[1]) : 0u;
            }
        }
        // column g of value tile j stands for dim kTiles * g + j
        uint32_t vw[4][kTiles / 4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int r = 2 * t4 + (e & 1) + (e >> 1) * 8;
            if (kHD == 128) {
                const uint4 x = *reinterpret_cast<const uint4*>(V + r * kHD + v_piece(r, g) * 16);
                vw[e][0] = x.x; vw[e][1] = x.y; vw[e][kTiles / 4 - 2] = x.z; vw[e][kTiles / 4 - 1] = x.w;
            } else if (kHD == 64) {
                const uint2 x = *reinterpret_cast<const uint2*>(V + r * kHD + v_piece(r, g >> 1) * 16 + (g & 1) * 8);
                vw[e][0] = x.x; vw[e][1] = x.y;
            } else {
#pragma unroll
                for (int b = 0; b < kTiles / 4; b++) vw[e][b] = *reinterpret_cast<const uint32_t*>(V + r * kHD + g * kTiles + b * 4);
            }
        }
#pragma unroll
        for (int b = 0; b < kTiles / 4; b++)
#pragma unroll
            for (int h = 0; h < 2; h++) {                          // dims 4 b + 2 h and the next: halves {row, row + 1}
                const uint32_t sel = h ? 0x7632u : 0x5410u;
                const uint32_t x0 = prmt(vw[0][b], vw[1][b], sel), x1 = prmt(vw[2][b], vw[3][b], sel);
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const uint32_t b0 = s8_pair_to_bf16(e ? x0 >> 8 : x0), b1 = s8_pair_to_bf16(e ? x1 >> 8 : x1);
                    float c[4] = {0.f, 0.f, 0.f, 0.f}, (&sum)[2] = acc[4 * b + 2 * h + e];
                    mma_bf16_16816(c, ap[0], ap[1], ap[2], ap[3], b0, b1);
                    if (kWide) mma_bf16_16816(c, 0u, apl[0], 0u, apl[1], b0, b1);
                    sum[0] += c[0] + c[2]; sum[1] += c[1] + c[3];
                }
            }
    }
    cp_async_wait<0>();
    __syncwarp();                                                  // the ring is the warp's own: its partial result goes there
    l += __shfl_xor_sync(0xFFFFFFFFu, l, 1);
    l += __shfl_xor_sync(0xFFFFFFFFu, l, 2);
    float* mine = reinterpret_cast<float*>(ring);                  // [head][column], padded: mma_acc_row, mma_acc_col
    const bool owner = kWide || (g < 4 && head < gqa);
#pragma unroll
    for (int j = 0; j < kTiles; j += 4)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            float x[4];
#pragma unroll
            for (int d = 0; d < 4; d++) {
                x[d] = acc[j + d][e];
                if (!kWide) x[d] += __shfl_xor_sync(0xFFFFFFFFu, x[d], 16);
            }
            if (owner) *reinterpret_cast<float4*>(mine + head * mma_acc_row(kHD) + (2 * t4 + e) * mma_acc_col(kHD) + j) = make_float4(x[0], x[1], x[2], x[3]);
        }
    if (owner && t4 == 0) {
        part_stats[(2 * warp) * kMmaHeads + head] = m;
        part_stats[(2 * warp + 1) * kMmaHeads + head] = l;
    }
    __syncthreads();
    // the CTA's sums over its warps, four dims a thread, in place in the first warp's ring
    float* accs = reinterpret_cast<float*>(mma_smem);
    const int ring_floats = ring_bytes / 4;
    int16_t* out = P.out + ((size_t)seq * P.n_head + (size_t)kvh * gqa) * kHD;
    auto finish = [&](int i, const float4& num, float den) {       // output elements 4 i .. 4 i + 3
        const uint32_t lo = (uint16_t)float_to_bf16_rne(num.x / den) | (uint32_t)(uint16_t)float_to_bf16_rne(num.y / den) << 16;
        const uint32_t hi = (uint16_t)float_to_bf16_rne(num.z / den) | (uint32_t)(uint16_t)float_to_bf16_rne(num.w / den) << 16;
        int16_t* o = out + i * 4;
        if ((reinterpret_cast<uintptr_t>(o) & 7) == 0) {
            *reinterpret_cast<uint2*>(o) = make_uint2(lo, hi);
        } else {
            o[0] = (int16_t)lo; o[1] = (int16_t)(lo >> 16); o[2] = (int16_t)hi; o[3] = (int16_t)(hi >> 16);
        }
    };
    for (int i = threadIdx.x; i < gqa * kHD / 4; i += blockDim.x) {
        const int h = i / (kHD / 4), d = (i - h * (kHD / 4)) * 4, at = h * mma_acc_row(kHD) + d / kTiles * mma_acc_col(kHD) + d % kTiles;
        float mm = -1e30f, den = 0.f;
        float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int wv = 0; wv < nwarps; wv++) mm = fmaxf(mm, part_stats[2 * wv * kMmaHeads + h]);
        for (int wv = 0; wv < nwarps; wv++) {
            const float f = exp2_approx(part_stats[2 * wv * kMmaHeads + h] - mm);   // a warp without positions: 0
            const float4 x = *reinterpret_cast<const float4*>(accs + wv * ring_floats + at);
            num.x += f * x.x; num.y += f * x.y; num.z += f * x.z; num.w += f * x.w;
            den += f * part_stats[(2 * wv + 1) * kMmaHeads + h];
        }
        if (nsplit == 1) {
            finish(i, num, den);
        } else {
            *reinterpret_cast<float4*>(accs + at) = num;           // read above by this thread only
            if (d == 0) { stats[h] = mm; stats[kMmaHeads + h] = den; }
        }
    }
    if (nsplit == 1) return;
    // ---- merge the slices of the cluster: rank r finishes the output elements r * threads, ..., one a thread, or four
    // where one would not do: a thread's rounds wait for the remote memory one after the other.  Eight query heads of 128,
    // two slices: 8 sequences of 100-200 positions 7.4 -> 6.1 us (general kernel 6.3), one of 64-128 6.5 -> 5.1 (6.2);
    // four a thread wherever there is a cluster: 32/8 heads, one sequence of 256, 4.4 -> 4.6.
    cluster_barrier();
    const bool four = gqa * kHD > nsplit * (int)blockDim.x;
    for (int i = split * blockDim.x + threadIdx.x; i < gqa * kHD / (four ? 4 : 1); i += nsplit * blockDim.x) {
        const int o = four ? i * 4 : i, h = o / kHD, d = o - h * kHD, at = h * mma_acc_row(kHD) + d / kTiles * mma_acc_col(kHD) + d % kTiles;
        float mm = -1e30f;
        for (int r = 0; r < nsplit; r++) mm = fmaxf(mm, ld_dsmem_f32(dsmem_addr(stats + h, r)));
        float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
        float den = 0.f;
        for (int r = 0; r < nsplit; r++) {
            const float f = exp2_approx(ld_dsmem_f32(dsmem_addr(stats + h, r)) - mm);   // an empty slice has max -1e30: weight 0
            if (four) {
                const float4 x = ld_dsmem_f32x4(dsmem_addr(accs + at, r));
                num.x += f * x.x; num.y += f * x.y; num.z += f * x.z; num.w += f * x.w;
            } else {
                num.x += f * ld_dsmem_f32(dsmem_addr(accs + at, r));
            }
            den += f * ld_dsmem_f32(dsmem_addr(stats + kMmaHeads + h, r));
        }
        if (four) finish(i, num, den);
        else out[o] = float_to_bf16_rne(num.x / den);
    }
    cluster_barrier();                                             // nobody reads this CTA's shared memory any more
}

// ---------------------------------------------------------------------------
// Greedy argmax, one CTA per sequence.  Ties resolve as in the engine's kernel
// (engine/kernels.hip:90-122: 256 threads scan i = tid, tid + 256, ... with a
// strict ">", then a halving tree in which slot t meets slot t + s and keeps its
// own value on equality).  After the level with stride s, slot t holds the
// winner among the threads congruent to t modulo s, so the last comparison is
// even against odd threads, the one before 0 against 2 modulo 4, ...: among the
// maxima the thread whose 8-bit index read backwards is smallest wins, and
// inside a thread the smallest i.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool argmax_better(float v, int i, float bv, int bi)
{
    if (v > bv) return true;
    if (v < bv || !(v == bv)) return false;
    const unsigned r = __brev((unsigned)i & 255u), br = __brev((unsigned)bi & 255u);
    return r < br || (r == br && i < bi);
}
// With `pairs` given (tensor-parallel output projection: this rank holds `n` of the vocabulary's rows, starting at
// index_offset) the winner is not stored as a token but as the pair {value, global index as float} in this rank's
// slot of pairs[slot][sequence][2], and the other ranks' slots are zeroed, so that a sum over ranks collects every
// rank's pair.  Ties are decided on the GLOBAL index, so the merged result equals the argmax over the whole vocabulary.
__global__ void __launch_bounds__(1024)
argmax_kernel(const float* __restrict__ logits, int* __restrict__ result, int n, int index_offset, float* __restrict__ pairs,
              int pair_slot, int pair_slots)
{
    __shared__ float sv[32];
    __shared__ int si[32];
    grid_launch_dependents();
    grid_dependency_wait();
    const float* row = logits + (size_t)blockIdx.x * n;
    float bv = -INFINITY;
    int bi = index_offset;
    if ((n & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) {   // 16-byte aligned rows: four elements per load, two in flight
        const float4* r4 = reinterpret_cast<const float4*>(row);
        for (int i = threadIdx.x; i < n / 4; i += 2 * blockDim.x) {
            const int j = i + blockDim.x;
            const float4 a = r4[i];
            const float4 b = j < n / 4 ? r4[j] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            const float va[4] = {a.x, a.y, a.z, a.w}, vb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int e = 0; e < 4; e++) if (argmax_better(va[e], index_offset + 4 * i + e, bv, bi)) { bv = va[e]; bi = index_offset + 4 * i + e; }
            if (j < n / 4) {
#pragma unroll
                for (int e = 0; e < 4; e++) if (argmax_better(vb[e], index_offset + 4 * j + e, bv, bi)) { bv = vb[e]; bi = index_offset + 4 * j + e; }
            }
        }
    } else {
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float v = row[i];
            if (argmax_better(v, index_offset + i, bv, bi)) { bv = v; bi = index_offset + i; }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, off);
        const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, off);
        if (argmax_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
    }
    if (lane == 0) { sv[warp] = bv; si[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        bv = lane < nw ? sv[lane] : -INFINITY;
        bi = lane < nw ? si[lane] : 0x7FFFFFFF;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, off);
            const int oi = __shfl_xor_sync(0xFFFFFFFFu, bi, off);
            if (argmax_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
        }
        if (bi == 0x7FFFFFFF) bi = index_offset;
        if (pairs == nullptr) {
            if (lane == 0) result[blockIdx.x] = bi;
        } else if (lane < pair_slots) {
            float2 pr = make_float2(0.f, 0.f);
            if (lane == pair_slot) pr = make_float2(bv, (float)bi);
            reinterpret_cast<float2*>(pairs)[(size_t)lane * gridDim.x + blockIdx.x] = pr;
        }
    }
}

// Picks, per sequence, the best of the ranks' {value, index} pairs (same order as argmax_kernel).
__global__ void __launch_bounds__(256)
argmax_merge_kernel(const float* __restrict__ pairs, int world, int batch, int* __restrict__ result)
{
    grid_launch_dependents();
    grid_dependency_wait();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= batch) return;
    float bv = -INFINITY;
    int bi = 0x7FFFFFFF;
    for (int r = 0; r < world; r++) {
        const float2 pr = reinterpret_cast<const float2*>(pairs)[(size_t)r * batch + b];
        const int i = (int)pr.y;
        if (bi == 0x7FFFFFFF || argmax_better(pr.x, i, bv, bi)) { bv = pr.x; bi = i; }
    }
    result[b] = bi;
}

// frequencies as the engine computes them on the host (engine/kernels.hip:129-140)
static void rope_freqs(int head_dim, float theta, RopeFreqs& F)
{
    static std::mutex mu;
    static RopeFreqs cached;
    static int c_dim = 0;
    static float c_theta = 0.f;
    std::lock_guard<std::mutex> lk(mu);
    if (c_dim != head_dim || c_theta != theta) {
        for (int d = 0; d < head_dim / 2 && d < 128; d++) cached.f[d] = 1.0f / powf(theta, (float)(2 * d) / (float)head_dim);
        c_dim = head_dim; c_theta = theta;
    }
    F = cached;
}

static int rope_kv_launch(RopeKvParams P, bool rope, float theta, int batch, void* stream, const char* who)
{
    if (P.head_dim < 2 || P.head_dim > 256 || (P.head_dim & 1) || P.n_head < 0 || P.n_head_kv < 1 || batch < 1)
        return fail(S12_ERR_UNSUPPORTED, "%s: head_dim must be even and <= 256, n_head_kv >= 1, batch >= 1", who);
    if (!rope) return launch(store_kv_kernel, dim3((2 * P.n_head_kv + kRopeWarps - 1) / kRopeWarps, batch), dim3(kRopeWarps * 32), 0, stream, who, P);
    RopeFreqs F;
    rope_freqs(P.head_dim, theta, F);
    const int wph = rope_head_warps(P.head_dim), heads = P.n_head + P.n_head_kv * (P.store ? 2 : 1);
    P.cta_slots = kRopeWarps / wph;
    const int ctas = (heads + P.cta_slots - 1) / P.cta_slots;
    // two heads a thread from three CTAs per SM on: 64 + 8 heads at B = 8 (320 CTAs) 2.2 us either way, at B = 16 3.0 -> 2.4
    const int two = (long long)ctas * batch > 3ll * sm_count() ? 2 : 1;
    return launch(two == 2 ? rope_kv_kernel<2> : rope_kv_kernel<1>, dim3((ctas + two - 1) / two, batch), dim3(P.cta_slots * wph * 32), 0, stream,
                  who, P, F);
}

// Launches attention_mma_kernel when it takes the shape (returns its status, 0 or negative), else returns 1.
// It takes head_dim 64 / 96 / 128 with rows of the caches on 16-byte boundaries, whatever the number of query heads (with
// one per kv head 3 of the 16 MMA rows are used).  General kernel / this one over 576 sizes (1, 2, 8 kv heads with 1-8 query
// heads each, 1-256 sequences, 16-16000 positions): at least as fast everywhere, in the middle 1.6x with one query head,
// 2.0 / 1.8 / 1.7x with heads of 64 / 96 / 128, 1.65x up to 48 positions; nearest at 8 sequences of 100-200 positions with one
// kv head of 128 (4.9 / 4.9 us).
static int attention_mma_launch(AttnParams P, int gqa, int max_len, int batch, void* stream, const char* who)
{
    const int hd = P.head_dim;
    if ((hd != 64 && hd != 96 && hd != 128) || P.kv_stride % 16 != 0 ||
        ((reinterpret_cast<uintptr_t>(P.kc) | reinterpret_cast<uintptr_t>(P.vc)) & 15) != 0)
        return 1;
    // Slices while three CTAs per SM (four are resident) are not there, of 64 positions or more: a CTA costs ~6 us of
    // dependent loads and merging whatever its length.  32/8 heads of 128, us with 1 / 2 / 4 / 8 slices (as first built,
    // with chained accumulators; within 4 % of now): 24 sequences of
    // 4096 77 / 67 / 53 / 53; 64 of 1000 36 / 37 / 42 / 60; 256 of 192 30 / 53 / 84 / 168; one of 8000 100 / 54 / 29 / 17.
    int nsplit = 1;
    const long long pairs = (long long)P.n_head_kv * batch;
    while (nsplit < 8 && pairs * nsplit < 3ll * sm_count() && max_len / (nsplit * 2) >= 64) nsplit *= 2;
    P.nsplit = nsplit;
    // Eight warps instead of four where all CTAs are resident at once even so: one sequence of 8000 positions
    // 16.9 -> 13.9 us, four of them with 64 query heads 34 -> 26 us; otherwise (256 of 192: 30 -> 41 us) or with two
    // chunks a warp or fewer the larger CTA only waits longer.
    const int warps = pairs * nsplit <= 2ll * sm_count() && max_len / nsplit >= 256 ? 8 : 4;
    typedef void (*Kern)(const AttnParams);
    static const Kern table[3][2] = {{attention_mma_kernel<64, false>, attention_mma_kernel<64, true>},
                                     {attention_mma_kernel<96, false>, attention_mma_kernel<96, true>},
                                     {attention_mma_kernel<128, false>, attention_mma_kernel<128, true>}};
    const int hi = hd == 64 ? 0 : hd == 96 ? 1 : 2, wi = gqa == 8 ? 1 : 0;
    Kern kern = table[hi][wi];
    // short contexts keep little shared memory: the projections' kernels either side hold most of an SM's, and this
    // kernel starts early only beside them
    const int per = ((P.t_limit + nsplit - 1) / nsplit + kMmaPos - 1) / kMmaPos;
    const int least = (gqa * mma_acc_row(hd) * 4 + mma_stage_bytes(hd) - 1) / mma_stage_bytes(hd);   // the partial result's room
    P.stages = std::min(kMmaStages, std::max(least, (per + warps - 1) / warps));
    const int smem = mma_smem_bytes(hd, warps, P.stages, gqa == 8 ? 8 : 4);
    static std::atomic<bool> attr_set[64][3][2];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr_set[dev][hi][wi].load(std::memory_order_relaxed)) {
        const int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, mma_smem_bytes(hd, kMmaWarps, kMmaStages, gqa == 8 ? 8 : 4)), who);
        if (rc) return rc;
        if (dev >= 0 && dev < 64) attr_set[dev][hi][wi].store(true, std::memory_order_relaxed);
    }
    return launch_clustered_z(kern, dim3(P.n_head_kv, batch, nsplit), dim3(warps * 32), (size_t)smem, stream, who, nsplit, P);
}

static int attention_launch(AttnParams& P, int max_len, int batch, void* stream, const char* who)
{
    if (P.head_dim < 4 || P.head_dim > 256 || (P.head_dim & 3) || P.n_head_kv < 1 || P.n_head < P.n_head_kv ||
        P.n_head % P.n_head_kv != 0 || max_len < 1 || batch < 1)
        return fail(S12_ERR_UNSUPPORTED, "%s: needs head_dim %% 4 == 0 and <= 256, n_head a multiple of n_head_kv, seq_len >= 1", who);
    const int gqa = P.n_head / P.n_head_kv;
    if (gqa != 1 && gqa != 2 && gqa != 4 && gqa != 8)
        return fail(S12_ERR_UNSUPPORTED, "%s: %d query heads per kv head (supported: 1, 2, 4, 8)", who, gqa);
    // few (kv head, sequence) pairs: cut the positions into slices, one CTA each, merged inside a cluster
    int nsplit = 1;
    const long long pairs = (long long)P.n_head_kv * batch;
    while (nsplit < 8 && pairs * nsplit * 2 <= sm_count() && max_len / (nsplit * 2) >= kAttnWarps) nsplit *= 2;
    auto smem_for = [&](int ns) {
        const int per = (max_len + ns - 1) / ns;
        return ((size_t)(gqa + 2) * ((per + 3) & ~3) + (size_t)kAttnWarps * gqa * P.head_dim + 2 * gqa) * sizeof(float);
    };
    // long contexts: more slices (also with many sequences) until one slice's scores fit a CTA's shared memory
    while (nsplit < 8 && smem_for(nsplit) > 200 * 1024) nsplit *= 2;
    P.nsplit = nsplit;
    const int per = (max_len + nsplit - 1) / nsplit;
    P.score_stride = (per + 3) & ~3;
    const size_t smem = smem_for(nsplit);
    if (smem > 200 * 1024) return fail(S12_ERR_TOO_LARGE, "%s: seq_len %d needs more shared memory than one CTA has", who, max_len);
    P.t_limit = max_len;
    const int mma = attention_mma_launch(P, gqa, max_len, batch, stream, who);
    if (mma <= 0) return mma;
    typedef void (*Kern)(const AttnParams);
    static const Kern table[4][2] = {{attention_kernel<1, 1>, attention_kernel<1, 2>}, {attention_kernel<2, 1>, attention_kernel<2, 2>},
                                     {attention_kernel<4, 1>, attention_kernel<4, 2>}, {attention_kernel<8, 1>, attention_kernel<8, 2>}};
    const int gi = gqa == 1 ? 0 : gqa == 2 ? 1 : gqa == 4 ? 2 : 3, ci = P.head_dim > 128 ? 1 : 0;
    Kern kern = table[gi][ci];
    static bool attr_set[64][4][2];
    if (smem > 48 * 1024) {
        int dev = 0;
        cudaGetDevice(&dev);
        dev = (dev < 0 || dev >= 64) ? 0 : dev;
        if (!attr_set[dev][gi][ci]) {
            int rc = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024), who);
            if (rc) return rc;
            attr_set[dev][gi][ci] = true;
        }
    }
    return launch_clustered_z(kern, dim3(P.n_head_kv, batch, nsplit), dim3(kAttnThreads), smem, stream, who, nsplit, P);
}

}  // namespace s12

using namespace s12;

extern "C" {

int launch_embed_lookup(const int16_t* embd_table, const int* token_ids, float* output, int n_embd, int batch_size,
                        int n_vocab, void* stream)
{
    if (!embd_table || !token_ids || !output || n_embd < 1 || batch_size < 1) return fail(S12_ERR_BAD_ARG, "launch_embed_lookup: bad argument");
    return launch(embed_kernel, dim3((n_embd + 255) / 256, batch_size), dim3(256), 0, stream, "launch_embed_lookup",
                  embd_table, token_ids, output, n_embd, batch_size, n_vocab);
}

int launch_argmax_batch(const float* logits, int* results, int n_vocab, int batch_size, void* stream)
{
    if (!logits || !results || n_vocab < 1 || batch_size < 1) return fail(S12_ERR_BAD_ARG, "launch_argmax: bad argument");
    return launch(argmax_kernel, dim3(batch_size), dim3(1024), 0, stream, "launch_argmax", logits, results, n_vocab, 0, (float*)nullptr, 0, 0);
}
int s12_tp_argmax_partial_async(const float* logits, int n_local, int index_offset, int batch, int rank, int world, float* pairs,
                                void* stream)
{
    if (!logits || !pairs || n_local < 1 || batch < 1 || world < 1 || world > 32 || rank < 0 || rank >= world || index_offset < 0 ||
        (long long)index_offset + n_local > (1 << 24))
        return fail(S12_ERR_BAD_ARG, "s12_tp_argmax_partial_async: bad argument (indices must stay below 2^24)");
    return launch(argmax_kernel, dim3(batch), dim3(1024), 0, stream, "s12_tp_argmax_partial_async", logits, (int*)nullptr, n_local,
                  index_offset, pairs, rank, world);
}
int s12_tp_argmax_merge_async(const float* pairs, int world, int batch, int* result, void* stream)
{
    if (!pairs || !result || world < 1 || batch < 1) return fail(S12_ERR_BAD_ARG, "s12_tp_argmax_merge_async: bad argument");
    return launch(argmax_merge_kernel, dim3((batch + 255) / 256), dim3(256), 0, stream, "s12_tp_argmax_merge_async", pairs, world,
                  batch, result);
}
int launch_argmax(const float* logits, int* result, int n, void* stream) { return launch_argmax_batch(logits, result, n, 1, stream); }

int launch_rms_norm_bf16_batch(const float* x, const float* weight, int16_t* y, int n, float eps, int batch_size, void* stream)
{
    if (!x || !weight || !y || n < 1 || batch_size < 1) return fail(S12_ERR_BAD_ARG, "launch_rms_norm_bf16_batch: bad argument");
    const int threads = n >= 1024 ? 1024 : ((n + 31) / 32) * 32;
    return launch(n > 8192 ? rms_norm_kernel<false, true> : rms_norm_kernel<false>, dim3(batch_size), dim3(threads), 0, stream, "launch_rms_norm_bf16_batch",
                  const_cast<float*>(x), (const float*)nullptr, weight, y, n, eps);
}
int launch_add_rms_norm_bf16_batch(float* x, const float* residual, const float* weight, int16_t* y, int n, float eps,
                                   int batch_size, void* stream)
{
    if (!x || !residual || !weight || !y || n < 1 || batch_size < 1) return fail(S12_ERR_BAD_ARG, "launch_add_rms_norm_bf16_batch: bad argument");
    const int threads = n >= 1024 ? 1024 : ((n + 31) / 32) * 32;
    return launch(threads == 1024 && batch_size > sm_count() ? add_rms_norm_two_kernel : rms_norm_kernel<true>, dim3(batch_size), dim3(threads), 0, stream, "launch_add_rms_norm_bf16_batch",
                  x, residual, weight, y, n, eps);
}
int launch_silu_mul_bf16_batch(const float* gate, const float* up, int16_t* out, int n, int batch_size, void* stream)
{
    if (!gate || !up || !out || n < 1 || batch_size < 1) return fail(S12_ERR_BAD_ARG, "launch_silu_mul_bf16_batch: bad argument");
    const long long total = (long long)n * batch_size;
    return launch(silu_mul_kernel, dim3((unsigned)((total + 1023) / 1024)), dim3(256), 0, stream, "launch_silu_mul_bf16_batch",
                  gate, up, out, total);
}
int launch_add_batch(float* y, const float* x, int n, int batch_size, void* stream)
{
    if (!y || !x || n < 1 || batch_size < 1) return fail(S12_ERR_BAD_ARG, "launch_add_batch: bad argument");
    const long long total = (long long)n * batch_size;
    return launch(add_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, "launch_add_batch", y, x, total);
}

int launch_rope_store_kv(float* q, float* k, const float* v, int8_t* kv_k, int8_t* kv_v, float* kv_scale_k, float* kv_scale_v,
                         int head_dim, int n_head, int n_head_kv, int position, int max_seq, float theta, void* stream)
{
    if (!q || !k || !v || !kv_k || !kv_v || !kv_scale_k || !kv_scale_v) return fail(S12_ERR_BAD_ARG, "launch_rope_store_kv: null argument");
    if (position < 0 || position >= max_seq) return fail(S12_ERR_BAD_ARG, "launch_rope_store_kv: position %d outside the cache of %d", position, max_seq);
    RopeKvParams P = {};
    P.q = q; P.k = k; P.v = v; P.kv_k = kv_k; P.kv_v = kv_v; P.sc_k = kv_scale_k; P.sc_v = kv_scale_v;
    P.position = position; P.head_dim = head_dim; P.n_head = n_head; P.n_head_kv = n_head_kv;
    P.q_stride = n_head * head_dim; P.k_stride = n_head_kv * head_dim; P.store = 1;
    return rope_kv_launch(P, true, theta, 1, stream, "launch_rope_store_kv");
}
int launch_rope_batch(float* q, float* k, const int* positions, int head_dim, int n_head, int n_head_kv, int q_stride,
                      int k_stride, float theta, int batch_size, void* stream)
{
    if (!q || !k || !positions) return fail(S12_ERR_BAD_ARG, "launch_rope_batch: null argument");
    RopeKvParams P = {};
    P.q = q; P.k = k; P.positions = positions; P.head_dim = head_dim; P.n_head = n_head; P.n_head_kv = n_head_kv;
    P.q_stride = q_stride; P.k_stride = k_stride; P.store = 0;
    return rope_kv_launch(P, true, theta, batch_size, stream, "launch_rope_batch");
}
// The engine's batched store writes every sequence into ONE cache at its position
// (engine/kernels.hip:784-788); s12_store_kv_batch below adds the per-sequence stride.
int s12_store_kv_batch(const float* k, const float* v, int8_t* kv_k, int8_t* kv_v, float* kv_scale_k, float* kv_scale_v,
                       const int* positions, int n_head_kv, int head_dim, long long kv_stride, int batch_size, void* stream)
{
    if (!k || !v || !kv_k || !kv_v || !kv_scale_k || !kv_scale_v || !positions) return fail(S12_ERR_BAD_ARG, "store_kv_batch: null argument");
    RopeKvParams P = {};
    P.k = const_cast<float*>(k); P.v = v; P.kv_k = kv_k; P.kv_v = kv_v; P.sc_k = kv_scale_k; P.sc_v = kv_scale_v;
    P.positions = positions; P.head_dim = head_dim; P.n_head = 0; P.n_head_kv = n_head_kv;
    P.k_stride = n_head_kv * head_dim; P.kv_stride = kv_stride; P.store = 1;
    return rope_kv_launch(P, false, 0.f, batch_size, stream, "store_kv_batch");
}
// launch_rope_batch and s12_store_kv_batch as one launch.
int s12_rope_store_kv_batch(float* q, float* k, const float* v, int8_t* kv_k, int8_t* kv_v, float* kv_scale_k, float* kv_scale_v,
                            const int* positions, int head_dim, int n_head, int n_head_kv, long long kv_stride, float theta,
                            int batch_size, void* stream)
{
    if (!q || !k || !v || !kv_k || !kv_v || !kv_scale_k || !kv_scale_v || !positions)
        return fail(S12_ERR_BAD_ARG, "s12_rope_store_kv_batch: null argument");
    RopeKvParams P = {};
    P.q = q; P.k = k; P.v = v; P.kv_k = kv_k; P.kv_v = kv_v; P.sc_k = kv_scale_k; P.sc_v = kv_scale_v;
    P.positions = positions; P.head_dim = head_dim; P.n_head = n_head; P.n_head_kv = n_head_kv;
    P.q_stride = n_head * head_dim; P.k_stride = n_head_kv * head_dim; P.kv_stride = kv_stride; P.store = 1;
    return rope_kv_launch(P, true, theta, batch_size, stream, "s12_rope_store_kv_batch");
}
int launch_store_kv_batch(const float* k, const float* v, int8_t* kv_k, int8_t* kv_v, float* kv_scale_k, float* kv_scale_v,
                          const int* positions, int kv_dim, int max_seq, int n_head_kv, int head_dim, int batch_size, void* stream)
{
    (void)kv_dim; (void)max_seq;
    return s12_store_kv_batch(k, v, kv_k, kv_v, kv_scale_k, kv_scale_v, positions, n_head_kv, head_dim, 0, batch_size, stream);
}

int launch_attention_all_heads(const float* q, const int8_t* k_cache, const int8_t* v_cache, const float* kv_scale_k,
                               const float* kv_scale_v, int16_t* output, int n_head, int n_head_kv, int head_dim, int seq_len,
                               int max_seq, float scale, void* stream)
{
    (void)max_seq;
    if (!q || !k_cache || !v_cache || !kv_scale_k || !kv_scale_v || !output) return fail(S12_ERR_BAD_ARG, "launch_attention_all_heads: null argument");
    AttnParams P = {};
    P.scale = scale;
    P.q = q; P.kc = k_cache; P.vc = v_cache; P.sk = kv_scale_k; P.sv = kv_scale_v; P.out = output;
    P.seq_len = seq_len; P.n_head = n_head; P.n_head_kv = n_head_kv; P.head_dim = head_dim;
    return attention_launch(P, seq_len, 1, stream, "launch_attention_all_heads");
}
int launch_attention_all_heads_batch(const float* q, const int8_t* kv_k, const int8_t* kv_v, const float* kv_scale_k,
                                     const float* kv_scale_v, int16_t* output, const int* positions, int n_head, int n_head_kv,
                                     int head_dim, int max_seq, float scale, int batch_size, int kv_stride, void* stream)
{
    if (!q || !kv_k || !kv_v || !kv_scale_k || !kv_scale_v || !output || !positions)
        return fail(S12_ERR_BAD_ARG, "launch_attention_all_heads_batch: null argument");
    AttnParams P = {};
    P.scale = scale;
    P.q = q; P.kc = kv_k; P.vc = kv_v; P.sk = kv_scale_k; P.sv = kv_scale_v; P.out = output; P.positions = positions;
    P.n_head = n_head; P.n_head_kv = n_head_kv; P.head_dim = head_dim; P.kv_stride = kv_stride;
    return attention_launch(P, max_seq, batch_size, stream, "launch_attention_all_heads_batch");   // max_seq: largest position + 1
}

// The engine switches to these two names from position 1024 on (engine/inference.cpp:285,432,505,627); same
// arguments as the two launchers above, same kernels here (they have no 1024-position limit).
int launch_flash_attention(const float* q, const int8_t* k_cache, const int8_t* v_cache, const float* kv_scale_k,
                           const float* kv_scale_v, int16_t* output, int n_head, int n_head_kv, int head_dim, int seq_len,
                           int max_seq, float scale, void* stream)
{
    return launch_attention_all_heads(q, k_cache, v_cache, kv_scale_k, kv_scale_v, output, n_head, n_head_kv, head_dim, seq_len,
                                      max_seq, scale, stream);
}
int launch_flash_attention_batch(const float* q, const int8_t* kv_k, const int8_t* kv_v, const float* kv_scale_k,
                                 const float* kv_scale_v, int16_t* output, const int* positions, int n_head, int n_head_kv,
                                 int head_dim, int max_seq, float scale, int batch_size, int kv_stride, void* stream)
{
    return launch_attention_all_heads_batch(q, kv_k, kv_v, kv_scale_k, kv_scale_v, output, positions, n_head, n_head_kv, head_dim,
                                            max_seq, scale, batch_size, kv_stride, stream);
}

}  // extern "C"
