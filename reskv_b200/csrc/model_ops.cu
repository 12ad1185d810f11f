// Small fused kernels of a decoder layer's decode step around the attention call: RMS norm,
// "split the fused QKV projection, rotate, append to the dense window", and SiLU(gate) * up.
//
// A decode step is launch-bound at small batch: in plain tensor ops these three pieces are ~30
// launches per layer, here they are three.  All of them read the decode position / window count
// from the device-side step state, so they can sit in the same captured graph as the attention.
#include <initializer_list>

#include "common.cuh"

namespace reskv {
namespace {

constexpr int kNormThreads = 256;

// one CTA per row: out = fp16( fp32(x) * rsqrt(mean(x^2) + eps) * fp32(w) ).  A decode step has one row per sequence, so
// this is latency: rows of up to kNormRegs pieces per thread are requested at once, weights included, and stay in
// registers (4 rows of 4096: 3.0 -> 2.0 us).
constexpr int kNormRegs = 4;  // 16-byte pieces per thread: up to 8192 values
__global__ void __launch_bounds__(kNormThreads) rms_norm_kernel(const __half* x, const __half* w, __half* out, int dim, float eps) {
    __shared__ float part[kNormThreads / 32];
    const size_t row = blockIdx.x;
    const uint4* xr = reinterpret_cast<const uint4*>(x + row * dim);
    const uint4* wr = reinterpret_cast<const uint4*>(w);
    uint4* orow = reinterpret_cast<uint4*>(out + row * dim);
    const int chunks = dim / 8;
    const bool fits = chunks <= kNormRegs * kNormThreads;
    let_next_launch_start();
    wait_for_previous_launch();
    uint4 xv[kNormRegs], wv[kNormRegs];
    if (fits) {
#pragma unroll
        for (int k = 0; k < kNormRegs; ++k)
            if (const int c = threadIdx.x + k * kNormThreads; c < chunks) xv[k] = xr[c], wv[k] = wr[c];
    }
    float acc = 0.f;
    auto add_squares = [&](const uint4& v) {
        const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h[i]);
            acc = fmaf(f.x, f.x, acc);
            acc = fmaf(f.y, f.y, acc);
        }
    };
    if (fits) {
#pragma unroll
        for (int k = 0; k < kNormRegs; ++k)
            if (threadIdx.x + k * kNormThreads < chunks) add_squares(xv[k]);
    } else {
        for (int c = threadIdx.x; c < chunks; c += kNormThreads) add_squares(xr[c]);
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < kNormThreads / 32; ++i) total += part[i];
    const float inv = rsqrtf(total / static_cast<float>(dim) + eps);
    auto scaled = [&](const uint4& v, const uint4& g) {
        const __half2* h = reinterpret_cast<const __half2*>(&v);
        const __half2* gh = reinterpret_cast<const __half2*>(&g);
        uint4 o;
        __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __half22float2(h[i]), gw = __half22float2(gh[i]);
            oh[i] = __floats2half2_rn(f.x * inv * gw.x, f.y * inv * gw.y);
        }
        return o;
    };
    if (fits) {
#pragma unroll
        for (int k = 0; k < kNormRegs; ++k)
            if (const int c = threadIdx.x + k * kNormThreads; c < chunks) orow[c] = scaled(xv[k], wv[k]);
    } else {
        for (int c = threadIdx.x; c < chunks; c += kNormThreads) orow[c] = scaled(xr[c], wr[c]);
    }
}

// grid (q_heads + 2 kv_heads, batch), 64 threads: thread i owns the RoPE pair (i, i + 64) of one
// head of the fused projection row [q heads | k heads | v heads].  Position = step_state[0].
__global__ void __launch_bounds__(64) rope_split_kernel(const __half* qkv, int q_heads, int kv_heads,
                                                        const float* inv_freq, const int32_t* step_state, __half* q_raw,
                                                        __half* q_rot, __half* k_rot, __half* v_out, __half* win_k,
                                                        __half* win_raw, __half* win_v, int capacity) {
    const int head = blockIdx.x, b = blockIdx.y, i = threadIdx.x;
    const int heads = q_heads + 2 * kv_heads;
    const __half* src = qkv + (static_cast<size_t>(b) * heads + head) * kHeadDim;
    let_next_launch_start();
    wait_for_previous_launch();
    const __half lo = src[i], hi = src[i + 64];
    if (head >= q_heads + kv_heads) {  // value head: copy
        const int h = head - q_heads - kv_heads;
        const size_t unit = static_cast<size_t>(b) * kv_heads + h;
        if (v_out) v_out[unit * kHeadDim + i] = lo, v_out[unit * kHeadDim + i + 64] = hi;
        if (win_v) {
            const int slot = min(max(step_state[1] - 1, 0), capacity - 1);
            __half* dst = win_v + (unit * capacity + slot) * kHeadDim;
            dst[i] = lo, dst[i + 64] = hi;
        }
        return;
    }
    float s, c;
    sincosf(static_cast<float>(step_state[0]) * inv_freq[i], &s, &c);
    const float a = __half2float(lo), bb = __half2float(hi);
    const __half rlo = __float2half_rn(a * c - bb * s), rhi = __float2half_rn(bb * c + a * s);
    if (head < q_heads) {
        const size_t row = (static_cast<size_t>(b) * q_heads + head) * kHeadDim;
        if (q_raw) q_raw[row + i] = lo, q_raw[row + i + 64] = hi;
        q_rot[row + i] = rlo, q_rot[row + i + 64] = rhi;
        return;
    }
    const int h = head - q_heads;
    const size_t unit = static_cast<size_t>(b) * kv_heads + h;
    if (k_rot) k_rot[unit * kHeadDim + i] = rlo, k_rot[unit * kHeadDim + i + 64] = rhi;
    if (win_k) {
        const int slot = min(max(step_state[1] - 1, 0), capacity - 1);
        __half* dk = win_k + (unit * capacity + slot) * kHeadDim;
        __half* dr = win_raw + (unit * capacity + slot) * kHeadDim;
        dk[i] = rlo, dk[i + 64] = rhi;
        dr[i] = lo, dr[i + 64] = hi;
    }
}

// A prompt's projection rows [batch, tokens, (q | k | v heads) * 128] -> rotated queries, raw keys, rotated keys and
// values, each [batch, heads, tokens, 128].  One pass of 16-byte loads and stores in place of the ~20 elementwise
// kernels of the same step in tensor operations (FP32 copies of both halves, products, concatenations, casts): bound by
// memory, 4096 tokens x 48 heads move 126 MB in ~30 us where those took ~650 us.  Eight threads per row, thread p owns
// the RoPE pairs (8 p + u, 64 + 8 p + u); the angles come from a [tokens, 64] table of cosines and sines.
constexpr int kRopeThreads = 256;
__global__ void __launch_bounds__(kRopeThreads) rope_prompt_kernel(const uint4* __restrict__ qkv, int tokens, int q_heads,
                                                                   int kv_heads, const float4* __restrict__ cos_t,
                                                                   const float4* __restrict__ sin_t, uint4* q_rot, uint4* k_raw,
                                                                   uint4* k_rot, uint4* v_out, long long rows) {
    const long long at = static_cast<long long>(blockIdx.x) * (kRopeThreads / 8) + (threadIdx.x >> 3);
    if (at >= rows) return;
    const int p = threadIdx.x & 7, heads = q_heads + 2 * kv_heads;
    const int head = static_cast<int>(at % heads);
    const long long bt = at / heads;
    const int t = static_cast<int>(bt % tokens);
    const long long b = bt / tokens;
    const uint4 lo = qkv[at * 16 + p], hi = qkv[at * 16 + 8 + p];
    if (head >= q_heads + kv_heads) {
        uint4* dst = v_out + ((b * kv_heads + head - q_heads - kv_heads) * tokens + t) * 16;
        dst[p] = lo, dst[8 + p] = hi;
        return;
    }
    float c[8], s[8];
    *reinterpret_cast<float4*>(c) = cos_t[t * 16 + 2 * p], *reinterpret_cast<float4*>(c + 4) = cos_t[t * 16 + 2 * p + 1];
    *reinterpret_cast<float4*>(s) = sin_t[t * 16 + 2 * p], *reinterpret_cast<float4*>(s + 4) = sin_t[t * 16 + 2 * p + 1];
    const __half2 *l2 = reinterpret_cast<const __half2*>(&lo), *h2 = reinterpret_cast<const __half2*>(&hi);
    uint4 rl, rh;
    __half2 *ol = reinterpret_cast<__half2*>(&rl), *oh = reinterpret_cast<__half2*>(&rh);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const float2 a = __half22float2(l2[u]), e = __half22float2(h2[u]);
        // products and sums rounded one by one, as the tensor operations do
        ol[u] = __floats2half2_rn(__fsub_rn(__fmul_rn(a.x, c[2 * u]), __fmul_rn(e.x, s[2 * u])),
                                  __fsub_rn(__fmul_rn(a.y, c[2 * u + 1]), __fmul_rn(e.y, s[2 * u + 1])));
        oh[u] = __floats2half2_rn(__fadd_rn(__fmul_rn(e.x, c[2 * u]), __fmul_rn(a.x, s[2 * u])),
                                  __fadd_rn(__fmul_rn(e.y, c[2 * u + 1]), __fmul_rn(a.y, s[2 * u + 1])));
    }
    if (head < q_heads) {
        uint4* dst = q_rot + ((b * q_heads + head) * tokens + t) * 16;
        dst[p] = rl, dst[8 + p] = rh;
        return;
    }
    const long long row = ((b * kv_heads + head - q_heads) * tokens + t) * 16;
    k_raw[row + p] = lo, k_raw[row + 8 + p] = hi;
    k_rot[row + p] = rl, k_rot[row + 8 + p] = rh;
}

// out[r][j] = fp16( fp16(silu(gate[r][j])) * up[r][j] ), gate_up = [rows, gate | up]
__global__ void silu_mul_kernel(const __half* gate_up, __half* out, int ffn, long long total) {
    let_next_launch_start();
    wait_for_previous_launch();
    const long long idx = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) * 2;
    if (idx >= total) return;
    const long long r = idx / ffn;
    const int j = static_cast<int>(idx % ffn);
    const __half2 g = *reinterpret_cast<const __half2*>(gate_up + r * 2 * ffn + j);
    const __half2 u = *reinterpret_cast<const __half2*>(gate_up + r * 2 * ffn + ffn + j);
    const float2 gf = __half22float2(g), uf = __half22float2(u);
    const __half2 act = __floats2half2_rn(gf.x / (1.f + expf(-gf.x)), gf.y / (1.f + expf(-gf.y)));
    const float2 af = __half22float2(act);
    *reinterpret_cast<__half2*>(out + idx) = __floats2half2_rn(af.x * uf.x, af.y * uf.y);
}

}  // namespace
}  // namespace reskv

using namespace reskv;

extern "C" int reskv_rms_norm(const void* x, const void* weight, void* out, int rows, int dim, float eps, void* stream) {
    if (!x || !weight || !out) return fail(RESKV_ERR_INVALID, "rms_norm: null pointer");
    if (rows < 1 || dim < 8 || dim % 8) return fail(RESKV_ERR_INVALID, "rms_norm: rows must be positive and dim a positive multiple of 8");
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(out)) & 15)
        return fail(RESKV_ERR_INVALID, "rms_norm: pointers must be 16-byte aligned");
    return check_cuda(launch_overlapped(rms_norm_kernel, dim3(rows), kNormThreads, 0, static_cast<cudaStream_t>(stream), true,
                                        static_cast<const __half*>(x), static_cast<const __half*>(weight),
                                        static_cast<__half*>(out), dim, eps),
                      "rms_norm launch");
}

extern "C" int reskv_rope_split(const void* qkv, int batch, int q_heads, int kv_heads, const float* inv_freq,
                                const int32_t* step_state, void* q_raw, void* q_rot, void* k_rot, void* v_out,
                                void* window_k, void* window_raw, void* window_v, int window_capacity, void* stream) {
    if (!qkv || !inv_freq || !step_state || !q_rot) return fail(RESKV_ERR_INVALID, "rope_split: null pointer");
    if (batch < 1 || q_heads < 1 || kv_heads < 1) return fail(RESKV_ERR_INVALID, "rope_split: batch and head counts must be positive");
    const bool window = window_k || window_raw || window_v;
    if (window && (!window_k || !window_raw || !window_v || window_capacity < 1))
        return fail(RESKV_ERR_INVALID, "rope_split: a window needs its three buffers and a positive capacity");
    if (!window && (!k_rot || !v_out)) return fail(RESKV_ERR_INVALID, "rope_split: nowhere to write keys and values");
    const dim3 grid(q_heads + 2 * kv_heads, batch);
    return check_cuda(launch_overlapped(rope_split_kernel, grid, 64, 0, static_cast<cudaStream_t>(stream), true,
                                        static_cast<const __half*>(qkv), q_heads, kv_heads, inv_freq, step_state,
                                        static_cast<__half*>(q_raw), static_cast<__half*>(q_rot), static_cast<__half*>(k_rot),
                                        static_cast<__half*>(v_out), static_cast<__half*>(window_k),
                                        static_cast<__half*>(window_raw), static_cast<__half*>(window_v), window_capacity),
                      "rope_split launch");
}

extern "C" int reskv_rope_prompt(const void* qkv, int batch, int tokens, int q_heads, int kv_heads, const float* cos_table,
                                 const float* sin_table, void* q_rot, void* k_raw, void* k_rot, void* v, void* stream) {
    if (!qkv || !cos_table || !sin_table || !q_rot || !k_raw || !k_rot || !v) return fail(RESKV_ERR_INVALID, "rope_prompt: null pointer");
    if (batch < 1 || tokens < 1 || q_heads < 1 || kv_heads < 1)
        return fail(RESKV_ERR_INVALID, "rope_prompt: batch, tokens and head counts must be positive");
    for (const void* p : {qkv, static_cast<const void*>(cos_table), static_cast<const void*>(sin_table), static_cast<const void*>(q_rot),
                          static_cast<const void*>(k_raw), static_cast<const void*>(k_rot), static_cast<const void*>(v)})
        if (!aligned16(p)) return fail(RESKV_ERR_INVALID, "rope_prompt: pointers must be 16-byte aligned");
    const long long rows = static_cast<long long>(batch) * tokens * (q_heads + 2 * kv_heads);
    const long long blocks = (rows + kRopeThreads / 8 - 1) / (kRopeThreads / 8);
    rope_prompt_kernel<<<static_cast<unsigned>(blocks), kRopeThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint4*>(qkv), tokens, q_heads, kv_heads, reinterpret_cast<const float4*>(cos_table),
        reinterpret_cast<const float4*>(sin_table), static_cast<uint4*>(q_rot), static_cast<uint4*>(k_raw),
        static_cast<uint4*>(k_rot), static_cast<uint4*>(v), rows);
    return check_cuda(cudaGetLastError(), "rope_prompt launch");
}

extern "C" int reskv_silu_mul(const void* gate_up, void* out, int rows, int ffn, void* stream) {
    if (!gate_up || !out) return fail(RESKV_ERR_INVALID, "silu_mul: null pointer");
    if (rows < 1 || ffn < 2 || ffn % 2) return fail(RESKV_ERR_INVALID, "silu_mul: rows must be positive and ffn a positive even number");
    const long long total = static_cast<long long>(rows) * ffn;
    const int threads = 256;
    const long long blocks = (total / 2 + threads - 1) / threads;
    return check_cuda(launch_overlapped(silu_mul_kernel, dim3(static_cast<unsigned>(blocks)), threads, 0,
                                        static_cast<cudaStream_t>(stream), true, static_cast<const __half*>(gate_up),
                                        static_cast<__half*>(out), ffn, total),
                      "silu_mul launch");
}
