// Lloyd clustering of pre-RoPE K or V per (sequence, KV head): fused assignment +
// centroid accumulation, centroid update, and the decode-time incremental step.
//
// Assignment is the exact nearest centre in FP32 (squared differences summed in
// a fixed order), lowest index on ties.  The bulk of it runs on the tensor cores:
// |c|^2 - 2 x.c for 16 tokens x 8 centres per mma.sync (centres split into FP16
// hi + lo so the products are exact), which ranks the centres up to an error far
// below the FP32 sum's own; a token whose two best candidates are closer than a
// conservative bound on that error is re-ranked by the exact FP32 sum, so the
// ids are those of the exact computation.  Cluster sums are accumulated *exactly*:
// an FP16 value is an integer multiple of 2^-24, so tokens are added as 2^24-
// scaled integers (split into two 32-bit shared-memory counters per CTA, flushed
// with 64-bit integer atomics).  Integer addition is associative, which makes
// the new centres independent of scheduling and equal to the correctly rounded
// mean -- results are reproducible run to run.
//
// That exact accumulation costs ~100 warp instructions per token (128 coordinates x two shared-memory atomics).
// The default for up to 32 centres is therefore a second form that keeps the exact *assignment* but forms the
// cluster sums on the tensor cores as onehot(ids)^T . X (the token rows are already in registers as MMA
// operands; movmatrix turns them into the other operand), FP32 accumulators per warp, warps added in index
// order, and the CTA's FP32 partial sums flushed as 2^24-scaled integers.  Every step has a fixed order or is
// an integer addition, so results are still reproducible run to run; the means can differ from the correctly
// rounded ones by FP32 rounding of the partial sums (checked: within one FP16 unit in the last place).
//
// K flavour: FP32 centres, an empty cluster keeps its centre.
// V flavour: centres rounded to FP16 after every update, an empty cluster becomes 0.

#include <initializer_list>

#include "common.cuh"
#include "tensor_map.cuh"
#include "tmem.cuh"

namespace reskv {
namespace {

constexpr uint32_t kFull = 0xffffffffu;
constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kChunk = 512;  // tokens per CTA, exact accumulation: keeps the split 32-bit counters from overflowing
constexpr int kChunkFastMax = 4096;  // most tokens per CTA with tensor-core accumulation
constexpr int kRedStride = 132;   // floats per cluster row of the cross-warp reduction buffer
constexpr int kXsRow = 2 * kHeadDim + 16;  // bytes per staged token row (16-byte loads of eight lanes in distinct banks)
constexpr float kFix = 16777216.0f;  // 2^24

struct KmeansParams {
    const __half* x;       // [units, x_stride, 128]
    float* centres;        // [units, C, 128] working centres (FP32 values)
    long long* sums;       // [units, C, 128] 2^24-scaled integer sums, zero on entry
    int* counts;           // [units, C], zero on entry
    int32_t* ids;          // [units, tokens]
    uint32_t* status;      // RESKV_STATUS_* bits (a bounded wait that ran out); cleared by the init kernel
    int64_t x_stride;
    int units, tokens, clusters;
};

struct InitIndex {
    int idx[kMaxClusters];
};

// The tcgen05 form, one launch for all Lloyd iterations, over one or two tensors (sides) of the same shape.
struct UmmaParams {
    const __half* x[2];   // [units, x_stride, 128]
    int64_t x_stride[2];
    int32_t* ids[2];      // [units, tokens]
    int8_t* ids8[2];      // the same as int8, or null
    int value[2];         // flavour of a side
    // State over all sides' units: the centres an iteration used (two generations), the 2^24-scaled sums and the counts
    // it formed (three generations: the last one is read, this one's added to, the next one's zeroed).
    float* centres[2];    // [sides * units, C, 128]
    long long* sums[3];
    int* counts[3];
    int* arrived;         // [sides * units] segments flushed so far, zero on entry
    uint32_t* status;
    __half* out[2];       // [units, C, 128] the centres after the last iteration
    int sides, units, tokens, clusters, iterations;
    InitIndex init;       // tokens that are the first centres
};

__global__ void kmeans_init_kernel(KmeansParams p, InitIndex init, int value) {
    const int unit = blockIdx.x;
    for (int i = threadIdx.x; i < p.clusters * kHeadDim; i += blockDim.x) {
        const int c = i / kHeadDim, d = i % kHeadDim;
        const float v = __half2float(p.x[(static_cast<size_t>(unit) * p.x_stride + init.idx[c]) * kHeadDim + d]);
        p.centres[(static_cast<size_t>(unit) * p.clusters + c) * kHeadDim + d] = v;
        p.sums[(static_cast<size_t>(unit) * p.clusters + c) * kHeadDim + d] = 0;
    }
    for (int c = threadIdx.x; c < p.clusters; c += blockDim.x) p.counts[unit * p.clusters + c] = 0;
    if (unit == 0 && threadIdx.x == 0) *p.status = 0u;
    (void)value;
}

// Squared distance of the warp's token to each centre, reduced so that lane c
// holds the total for centre cbase + c; returns (best distance, best index) in
// every lane.  `xv` are the lane's coordinates {lane + 32 i}.
__device__ __forceinline__ void nearest(const float* cen_s, int clusters, const float (&xv)[4], int lane, float& best,
                                        int& best_c) {
    best = INFINITY, best_c = 0;
    for (int cbase = 0; cbase < clusters; cbase += 32) {
        float part[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) {
            float acc = 0.f;
            if (cbase + c < clusters) {
                const float* row = cen_s + (cbase + c) * kHeadDim;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float df = xv[i] - row[lane + 32 * i];
                    acc = fmaf(df, df, acc);
                }
            }
            part[c] = acc;
        }
        // transposing butterfly: after the step with offset `off`, a lane keeps the
        // half of its values whose centre index has the same `off` bit as the lane
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const bool up = lane & off;
#pragma unroll
            for (int c = 0; c < off; ++c) {
                const float send = up ? part[c] : part[c + off];
                const float keep = up ? part[c + off] : part[c];
                part[c] = keep + __shfl_xor_sync(kFull, send, off);
            }
        }
        float dist = (cbase + lane < clusters) ? part[0] : INFINITY;
        int idx = cbase + lane;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float od = __shfl_xor_sync(kFull, dist, off);
            const int oi = __shfl_xor_sync(kFull, idx, off);
            if (od < dist || (od == dist && oi < idx)) dist = od, idx = oi;
        }
        if (dist < best) best = dist, best_c = idx;  // earlier block wins ties
    }
}

constexpr int kCenHalfStride = 132;  // FP16 centre rows: stride = 2 banks mod 32, so B-fragment loads do not collide
constexpr float kTieBound = 1.0f / 32768.0f;  // re-rank when (d2 - d1) <= kTieBound * (|x|^2 + max |c|^2)

// Offset (in coordinates) of MMA k-step `ks` for quad lane `q`: a lane owns coordinates
// [16 q, 16 q + 16) and [64 + 16 q, 64 + 16 q + 16), four per k-step.
__device__ __forceinline__ int kstep_offset(int ks, int q) { return (ks < 4 ? 0 : 48) + 16 * q + 4 * ks; }

// grid (chunks, units).  Tensor-core assignment of the chunk's tokens (see the file header), then
// exact accumulation of sums and counts.  HILO = centres are FP32 (key flavour): use hi + lo FP16.
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}

// Sixteen bytes from an address that is only on a 2-byte boundary.
__device__ __forceinline__ uint4 load_halves(const uint4* p) {
    const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __ldg(h + 2 * i) | static_cast<uint32_t>(__ldg(h + 2 * i + 1)) << 16;
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// FAST: cluster sums on the tensor cores (needs padded <= 32 and x on a 16-byte boundary), else exact integer accumulation.
template <bool HILO, bool FAST>
__global__ void __launch_bounds__(kThreads) kmeans_assign_mma_kernel(const KmeansParams p, int padded, int chunk) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* cen_s = reinterpret_cast<float*>(smem);                              // [C][128] FP32 centres (exact path)
    int* lo_s = reinterpret_cast<int*>(cen_s + p.clusters * kHeadDim);          // [C][128] low 20 bits
    int* hi_s = lo_s + p.clusters * kHeadDim;                                   // [C][128] the rest
    // FAST uses the counter arrays' place for its FP32 reduction slabs [warps][32][kRedStride] (sized by the host)
    const int counter_ints = FAST ? kWarps * 32 * kRedStride : 2 * p.clusters * kHeadDim;
    int* cnt_s = lo_s + counter_ints;                                           // [C]
    float* cn_s = reinterpret_cast<float*>(cnt_s + kMaxClusters);               // [padded] |c|^2, +inf for padding
    __half* ch_s = reinterpret_cast<__half*>(cn_s + kMaxClusters);              // [padded][132] FP16 hi
    __half* cl_s = ch_s + padded * kCenHalfStride;                              // [padded][132] FP16 lo (HILO)
    __shared__ float cmax_s;
    const int unit = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
    const int t_begin = blockIdx.x * chunk, t_end = min(p.tokens, t_begin + chunk);
    const float* cen_g = p.centres + static_cast<size_t>(unit) * p.clusters * kHeadDim;
    for (int i = tid; i < p.clusters * kHeadDim; i += kThreads) {
        cen_s[i] = cen_g[i];
        lo_s[i] = 0;
        hi_s[i] = 0;
    }
    for (int i = tid; i < padded * kHeadDim; i += kThreads) {
        const int c = i / kHeadDim, d = i % kHeadDim;
        const float v = c < p.clusters ? cen_g[i] : 0.f;
        const __half h = __float2half_rn(v);
        ch_s[c * kCenHalfStride + d] = h;
        if (HILO) cl_s[c * kCenHalfStride + d] = __float2half_rn(v - __half2float(h));
    }
    for (int c = tid; c < kMaxClusters; c += kThreads) cnt_s[c] = 0;
    __syncthreads();
    // |c|^2 of the value the MMA actually sees (hi + lo), one warp per centre
    for (int c = warp; c < padded; c += kWarps) {
        float acc = 0.f;
        if (c < p.clusters) {
            for (int d = lane; d < kHeadDim; d += 32) {
                float v = __half2float(ch_s[c * kCenHalfStride + d]);
                if (HILO) v += __half2float(cl_s[c * kCenHalfStride + d]);
                acc = fmaf(v, v, acc);
            }
            for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(kFull, acc, off);
        } else {
            acc = INFINITY;
        }
        if (lane == 0) cn_s[c] = acc;
    }
    __syncthreads();
    if (tid == 0) {
        float m = 0.f;
        for (int c = 0; c < p.clusters; ++c) m = fmaxf(m, cn_s[c]);
        cmax_s = m;
    }
    __syncthreads();
    const float cmax = cmax_s;
    const __half* xu = p.x + static_cast<size_t>(unit) * p.x_stride * kHeadDim;
    const bool wide = FAST || (reinterpret_cast<uintptr_t>(xu) & 15u) == 0;  // a view may start anywhere
    // FAST: sums[cluster 16 mb + g (+8)][coordinate kstep_offset(ks, q) + 2 h + (0, 1)] of this warp's tokens,
    // n-block nb = 2 ks + h
    float acc_s[FAST ? 2 : 1][FAST ? 16 : 1][4];
    if constexpr (FAST) {
#pragma unroll
        for (int mb = 0; mb < 2; ++mb)
#pragma unroll
            for (int nb = 0; nb < 16; ++nb) acc_s[mb][nb][0] = acc_s[mb][nb][1] = acc_s[mb][nb][2] = acc_s[mb][nb][3] = 0.f;
    }

    // FAST: the warp's next 16 token rows travel to shared memory (16-byte asynchronous copies, rows 16 bytes
    // apart from dense) while the current block is being processed; the block is read into registers at the
    // top of the loop, which frees the buffer for the copy of the one after
    unsigned char* xs_w = reinterpret_cast<unsigned char*>(cl_s + (HILO ? padded * kCenHalfStride : 0)) + warp * 16 * kXsRow;
    auto stage_rows = [&](int t0) {
        const int n = min(16, t_end - t0);
        const unsigned char* src = reinterpret_cast<const unsigned char*>(xu + static_cast<size_t>(t0) * kHeadDim);
        for (int i = lane; i < n * 16; i += 32) cp_async16(xs_w + (i >> 4) * kXsRow + (i & 15) * 16, src + i * 16);
    };
    if constexpr (FAST) {
        if (t_begin + warp * 16 < t_end) stage_rows(t_begin + warp * 16);
    }

    for (int t0 = t_begin + warp * 16; t0 < t_end; t0 += kWarps * 16) {
        // A fragments: rows t0 + g and t0 + g + 8, the lane's 32 coordinates of each
        const int r0 = t0 + g, r1 = t0 + g + 8;
        uint32_t a[8][4];
        {
            uint4 v[2][4];
            if constexpr (FAST) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int row = r ? r1 : r0;
                const uint4* src = FAST ? reinterpret_cast<const uint4*>(xs_w + (g + 8 * r) * kXsRow)
                                        : reinterpret_cast<const uint4*>(xu + static_cast<size_t>(row) * kHeadDim);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4* at = src + (k < 2 ? 0 : 8) + 2 * q + (k & 1);
                    v[r][k] = row >= t_end ? make_uint4(0, 0, 0, 0) : FAST ? *at : wide ? __ldg(at) : load_halves(at);
                }
            }
            if constexpr (FAST) {
                __syncwarp();  // every lane has its rows in registers
                if (t0 + kWarps * 16 < t_end) stage_rows(t0 + kWarps * 16);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                a[2 * k][0] = v[0][k].x, a[2 * k][1] = v[1][k].x, a[2 * k][2] = v[0][k].y, a[2 * k][3] = v[1][k].y;
                a[2 * k + 1][0] = v[0][k].z, a[2 * k + 1][1] = v[1][k].z, a[2 * k + 1][2] = v[0][k].w, a[2 * k + 1][3] = v[1][k].w;
            }
        }
        // |x|^2 of the 16 rows: diagonal of X X^T (B fragments are the A registers themselves)
        float xn0, xn1;
        {
            float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                mma_16816(s0, a[ks][0], a[ks][1], a[ks][2], a[ks][3], a[ks][0], a[ks][2]);
                mma_16816(s1, a[ks][0], a[ks][1], a[ks][2], a[ks][3], a[ks][1], a[ks][3]);
            }
            // row g x token g sits in lane (g, g / 2), element g % 2; row g + 8 x token g + 8 likewise in s1[2..3]
            const float mine0 = (g & 1) ? s0[1] : s0[0], mine1 = (g & 1) ? s1[3] : s1[2];
            xn0 = __shfl_sync(kFull, mine0, 4 * g + (g >> 1));
            xn1 = __shfl_sync(kFull, mine1, 4 * g + (g >> 1));
        }
        float d1[2] = {INFINITY, INFINITY}, d2[2] = {INFINITY, INFINITY};
        int c1[2] = {0, 0};
        // four centre blocks at a time: their accumulation chains are independent, which keeps the tensor pipe fed
        // with few resident warps (blocks beyond the padded count repeat the last one and are ignored)
        constexpr int kChains = 4;
        for (int nb0 = 0; nb0 < padded / 8; nb0 += kChains) {
            float acc[kChains][4];
            const __half* hrow[kChains];
            const __half* lrow[kChains];
#pragma unroll
            for (int h = 0; h < kChains; ++h) {
                acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.f;
                const int nb = min(nb0 + h, padded / 8 - 1);
                hrow[h] = ch_s + (nb * 8 + g) * kCenHalfStride;
                lrow[h] = cl_s + (nb * 8 + g) * kCenHalfStride;
            }
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
#pragma unroll
                for (int h = 0; h < kChains; ++h) {
                    const uint2 bh = *reinterpret_cast<const uint2*>(hrow[h] + kstep_offset(ks, q));
                    mma_16816(acc[h], a[ks][0], a[ks][1], a[ks][2], a[ks][3], bh.x, bh.y);
                }
                if (HILO) {
#pragma unroll
                    for (int h = 0; h < kChains; ++h) {
                        const uint2 bl = *reinterpret_cast<const uint2*>(lrow[h] + kstep_offset(ks, q));
                        mma_16816(acc[h], a[ks][0], a[ks][1], a[ks][2], a[ks][3], bl.x, bl.y);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < kChains; ++h) {
                if (nb0 + h >= padded / 8) break;
                const int col = (nb0 + h) * 8 + 2 * q;
                const float n0 = cn_s[col], n1 = cn_s[col + 1];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int r = e >> 1, c = col + (e & 1);
                    const float d = fmaf(-2.f, acc[h][e], (e & 1) ? n1 : n0);
                    if (d < d1[r]) {
                        d2[r] = d1[r], d1[r] = d, c1[r] = c;
                    } else if (d < d2[r]) {
                        d2[r] = d;
                    }
                }
            }
        }
#pragma unroll
        for (int off = 1; off <= 2; off <<= 1) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float od1 = __shfl_xor_sync(kFull, d1[r], off), od2 = __shfl_xor_sync(kFull, d2[r], off);
                const int oc1 = __shfl_xor_sync(kFull, c1[r], off);
                if (od1 < d1[r] || (od1 == d1[r] && oc1 < c1[r])) {
                    d2[r] = fminf(d1[r], od2), d1[r] = od1, c1[r] = oc1;
                } else {
                    d2[r] = fminf(d2[r], od1);
                }
            }
        }
        // near-ties: re-rank with the exact FP32 sum (all lanes of the warp take part)
        const bool tie0 = r0 < t_end && (d2[0] - d1[0]) <= kTieBound * (xn0 + cmax);
        const bool tie1 = r1 < t_end && (d2[1] - d1[1]) <= kTieBound * (xn1 + cmax);
        uint32_t redo0 = __ballot_sync(kFull, tie0 && q == 0), redo1 = __ballot_sync(kFull, tie1 && q == 0);
        for (int half = 0; half < 2; ++half) {
            uint32_t redo = half ? redo1 : redo0;
            while (redo) {
                const int src = __ffs(redo) - 1;
                redo &= redo - 1;
                const int row = t0 + (src >> 2) + 8 * half;
                const __half* xr = xu + static_cast<size_t>(row) * kHeadDim;
                float xv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) xv[i] = __half2float(xr[lane + 32 * i]);
                float best;
                int c;
                nearest(cen_s, p.clusters, xv, lane, best, c);
                if ((lane >> 2) == (src >> 2)) c1[half] = c;
            }
        }
        if (q == 0) {
            if (r0 < t_end) p.ids[static_cast<size_t>(unit) * p.tokens + r0] = c1[0];
            if (r1 < t_end) p.ids[static_cast<size_t>(unit) * p.tokens + r1] = c1[1];
        }
        if constexpr (FAST) {
            // onehot(ids)^T . X: A = one-hot rows (cluster x token) from a packed FP16 compare of the ids, B = the
            // token rows transposed (movmatrix of the A fragments of the distance step); rows beyond the end are 0
            const int v0 = r0 < t_end ? c1[0] : -1, v1 = r1 < t_end ? c1[1] : -1;
            const int w0 = __shfl_sync(kFull, v0, 8 * q), w1 = __shfl_sync(kFull, v0, 8 * q + 4);
            const int w2 = __shfl_sync(kFull, v1, 8 * q), w3 = __shfl_sync(kFull, v1, 8 * q + 4);
            const __half2 gg = __half2half2(__int2half_rn(g));
            const __half2 d01 = __hsub2(__halves2half2(__int2half_rn(w0), __int2half_rn(w1)), gg);
            const __half2 d23 = __hsub2(__halves2half2(__int2half_rn(w2), __int2half_rn(w3)), gg);
            uint32_t oh[2][4];
#pragma unroll
            for (int mb = 0; mb < 2; ++mb) {
                const __half2 lo = __float2half2_rn(16.f * mb), hi = __float2half2_rn(16.f * mb + 8.f);
                const __half2 e0 = __heq2(d01, lo), e1 = __heq2(d01, hi), e2 = __heq2(d23, lo), e3 = __heq2(d23, hi);
                oh[mb][0] = *reinterpret_cast<const uint32_t*>(&e0), oh[mb][1] = *reinterpret_cast<const uint32_t*>(&e1);
                oh[mb][2] = *reinterpret_cast<const uint32_t*>(&e2), oh[mb][3] = *reinterpret_cast<const uint32_t*>(&e3);
            }
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                const uint32_t b00 = movmatrix_trans(a[ks][0]), b01 = movmatrix_trans(a[ks][1]);
                const uint32_t b10 = movmatrix_trans(a[ks][2]), b11 = movmatrix_trans(a[ks][3]);
#pragma unroll
                for (int mb = 0; mb < 2; ++mb) {
                    if (16 * mb < padded) {
                        mma_16816(acc_s[mb][2 * ks], oh[mb][0], oh[mb][1], oh[mb][2], oh[mb][3], b00, b01);
                        mma_16816(acc_s[mb][2 * ks + 1], oh[mb][0], oh[mb][1], oh[mb][2], oh[mb][3], b10, b11);
                    }
                }
            }
            if (q == 0) {
                if (r0 < t_end) atomicAdd(&cnt_s[c1[0]], 1);
                if (r1 < t_end) atomicAdd(&cnt_s[c1[1]], 1);
            }
            continue;
        }
        // exact accumulation, one token at a time with the warp across its coordinates
        const int rows = min(16, t_end - t0);
        for (int r = 0; r < rows; ++r) {
            const int c = __shfl_sync(kFull, (r & 8) ? c1[1] : c1[0], 4 * (r & 7));
            const __half* xr = xu + static_cast<size_t>(t0 + r) * kHeadDim;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                // x * 2^24 is an integer below 2^41: split it, exactly, into hi * 2^20 + lo with both
                // parts carrying the sign of x (|lo| < 2^20, |hi| < 2^21)
                const float fx = __half2float(xr[lane + 32 * i]) * kFix;
                const float hi = truncf(fx * (1.0f / 1048576.0f));
                const float lo = fmaf(hi, -1048576.0f, fx);
                atomicAdd(&lo_s[c * kHeadDim + lane + 32 * i], __float2int_rz(lo));
                atomicAdd(&hi_s[c * kHeadDim + lane + 32 * i], __float2int_rz(hi));
            }
            if (lane == 0) atomicAdd(&cnt_s[c], 1);
        }
    }
    __syncthreads();
    long long* sums_g = p.sums + static_cast<size_t>(unit) * p.clusters * kHeadDim;
    if constexpr (FAST) {
        // every warp stores its partial sums in a slab of its own (the integer counters' memory, unused in this
        // form, enlarged by the host); the slabs are added in warp order and the CTA's sums go out as 2^24-scaled
        // integers
        float* red = reinterpret_cast<float*>(lo_s);  // [warps][32][kRedStride]
        {
            float* mine = red + warp * 32 * kRedStride;
#pragma unroll
            for (int mb = 0; mb < 2; ++mb)
#pragma unroll
                for (int nb = 0; nb < 16; ++nb)
#pragma unroll
                    for (int e = 0; e < 4; e += 2) {
                        const int cl = 16 * mb + g + 8 * (e >> 1);
                        const int d = kstep_offset(nb >> 1, q) + 2 * (nb & 1);
                        *reinterpret_cast<float2*>(mine + cl * kRedStride + d) = make_float2(acc_s[mb][nb][e], acc_s[mb][nb][e + 1]);
                    }
        }
        __syncthreads();
        for (int i = tid; i < p.clusters * kHeadDim; i += kThreads) {
            const int cl = i / kHeadDim, d = i % kHeadDim;
            if (cnt_s[cl] > 0) {
                float sum = 0.f;
#pragma unroll
                for (int w = 0; w < kWarps; ++w) sum += red[(w * 32 + cl) * kRedStride + d];  // fixed order
                atomicAdd(reinterpret_cast<unsigned long long*>(sums_g + i),
                          static_cast<unsigned long long>(__float2ll_rn(sum * kFix)));
            }
        }
        for (int c = tid; c < p.clusters; c += kThreads)
            if (cnt_s[c] > 0) atomicAdd(&p.counts[unit * p.clusters + c], cnt_s[c]);
        return;
    }
    for (int i = tid; i < p.clusters * kHeadDim; i += kThreads) {
        if (cnt_s[i / kHeadDim] > 0) {
            const long long v = static_cast<long long>(hi_s[i]) * 1048576LL + lo_s[i];
            atomicAdd(reinterpret_cast<unsigned long long*>(sums_g + i), static_cast<unsigned long long>(v));
        }
    }
    for (int c = tid; c < p.clusters; c += kThreads)
        if (cnt_s[c] > 0) atomicAdd(&p.counts[unit * p.clusters + c], cnt_s[c]);
}

// ---- tcgen05 form of the assignment kernel (up to 32 centres) ---------------------------------------------------
// One CTA per SM; the 128-token tiles of all units are laid end to end and every CTA streams an equal share of them,
// segment by segment (a segment = consecutive tiles of one unit).  A tile arrives by two tensor-map copies
// (TMA, 128-byte swizzle: coordinates 0..63 and 64..127 of 128 rows) and is used three times without ever
// passing through registers:
//   * distances: D[128 tokens x 64] = X . [c_hi | c_lo]^T, X as the K-major A operand of tcgen05.mma, the centre
//     halves as a K-major B operand written once per unit and CTA; accumulator in TMEM, triple buffered;
//   * ranking: one thread per token (TMEM lane = token row) reads its row of D with tcgen05.ld, ranks the centres,
//     re-ranks near-ties exactly - only the centres inside the bound, with the arithmetic and order of the exact
//     path of the mma.sync form -, writes the id and sets one element of a one-hot operand
//     onehot[32 clusters x 128 tokens]; three groups of four warps take the tiles in turn, so each has three tile
//     periods for its chain of dependent steps;
//   * sums: S^T[128 coordinates x 32 clusters] += X^T . onehot^T, the same tile now read as the MN-major A operand,
//     accumulated in TMEM (four accumulators in turn) over the segment and flushed at its end as 2^24-scaled
//     integers.
// Three more warps issue the asynchronous work (distance MMAs, sum MMAs, copies); they stay converged (descriptor
// arithmetic on the uniform datapath) and elect one lane per instruction.  The roles run concurrently on
// different tiles and hand over through mbarriers only (triple-buffered distances and one-hot operands); every
// wait is bounded.
//
// One cooperative launch for all iterations, over K and V together when both are wanted.  A CTA keeps its segments; between
// iterations it waits for the other CTAs of its units only (a counter of flushed segments per unit), and not at all for a
// unit that is its own, whose sums it writes without atomic additions.  The new centres are formed at the start of the next
// iteration from the sums of the last one (three generations of them, so nothing has to be cleared in between).  The ring of
// copies runs on across iterations, and every second iteration takes the tiles backwards: what the last one read at its end
// is still in L2.  Where a unit's iteration begins, the loads of all sums are in flight together, and the next segment is
// worked out by a thread that waits anyway.
//
// Two segments of a unit in a row are taken without a stop, with accumulators of their own, and flushed together.
//
// Measured, clustering of one layer's K and V, 10 iterations, us, one launch per iteration -> now: 64 units x 8128 tokens
// 578 -> 486, 128 x 3000 517 -> 417, 64 x 2000 221 -> 162, 8 x 1152 105 -> 97, 8 x 8128 164 -> 133, 24 x 4870 262 -> 229.
// Of that at 64 x 8128 the single launch by itself gives 2 %, the order of the tiles 3, the loads together 1, stores in place
// of atomics and the next segment worked out ahead 6, two segments without a stop 4 (at 8 x 8128 20).
constexpr int kUGroups = 3;                    // token-owning groups; group g takes the tiles i = g (mod 3)
constexpr int kUGroupWarps = 4;                // a group: one warp per 32 token rows (TMEM lane quarter)
constexpr int kUThreads = (kUGroups * kUGroupWarps + 3) * 32;  // + three issuing warps: distance MMAs, sum MMAs, copies
constexpr int kUTile = 128;
constexpr int kUStages = 5;
constexpr int kUBoxBytes = kUTile * 128;       // 128 rows x 64 coordinates
constexpr int kUTileBytes = 2 * kUBoxBytes;
constexpr int kUOneHotBytes = 2 * 32 * 128;    // [2 token halves][32 clusters][64 tokens] FP16
constexpr uint32_t kUTmemCols = 512;           // distances 3 x 64 columns, sums 2 x 4 x 32 columns; a power of two
constexpr uint32_t kUColD = 0, kUColS = 192;
constexpr int kUSumBuffers = 4;                // tile i of a segment adds to accumulator i % 4: shorter FP32 chains, no MMA-to-MMA dependency
constexpr int kURun = 2;                       // segments of a unit that a CTA takes without a stop, accumulators of their own
constexpr int kUChunkMax = 8192;               // most tokens per CTA (2048 per accumulator)

// Shared-memory matrix descriptor, 128-byte swizzle, address bits [4, 18), leading / stride byte offsets.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) | (static_cast<uint64_t>(lbo_bytes >> 4) << 16) |
           (static_cast<uint64_t>(sbo_bytes >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// FP16 x FP16 -> FP32, M = 128, N = n; a_mn: A is MN-major (the token tile read transposed).
__host__ __device__ constexpr uint32_t umma_idesc(int n, bool a_mn) {
    return (1u << 4) | (a_mn ? (1u << 15) : 0u) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// One arrival on `bar` once every MMA issued so far by the calling thread has completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Byte offset of 16-byte piece `piece` (0..7) of row `row` in a [rows][128 B] block with the 128-byte swizzle.
__device__ __forceinline__ uint32_t sw128(int row, int piece) { return row * 128 + ((piece ^ (row & 7)) << 4); }

// True in exactly one lane of a converged warp (the same lane every time).
__device__ __forceinline__ bool elect_one() {
    uint32_t chosen;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(chosen));
    return chosen != 0;
}

constexpr int kUWorkers = kUThreads - 32;  // everyone but the copying warp: these meet at the segment boundaries

__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kUWorkers) : "memory"); }

// Four coordinates of a centre after iteration `from`: the mean of the tokens assigned then, the old centre (K) or zero
// (V) where there were none; V's centres are rounded to FP16.  In two parts, so that a thread has all its loads in flight
// together (the sums requested behind the count: two trips to L2 per centre, 7000 instead of 2500 cycles for the tables).
struct CentreSums {
    int n;
    longlong2 a, b;
};
__device__ __forceinline__ CentreSums load_sums(const UmmaParams& p, int from, size_t row, int i4) {
    const longlong2* s = reinterpret_cast<const longlong2*>(p.sums[from % 3] + row * kHeadDim) + 2 * i4;
    return {__ldcg(p.counts[from % 3] + row), __ldcg(s), __ldcg(s + 1)};  // through L2: written by other CTAs
}
__device__ __forceinline__ float4 new_centre(const UmmaParams& p, const CentreSums& cs, int from, bool value, size_t row, int i4) {
    float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
    if (cs.n > 0) {
        const double scale = __drcp_rn(static_cast<double>(cs.n)) * (1.0 / 16777216.0);
        c = make_float4(static_cast<float>(static_cast<double>(cs.a.x) * scale), static_cast<float>(static_cast<double>(cs.a.y) * scale),
                        static_cast<float>(static_cast<double>(cs.b.x) * scale), static_cast<float>(static_cast<double>(cs.b.y) * scale));
    } else if (!value) {
        c = __ldcg(reinterpret_cast<const float4*>(p.centres[from & 1] + row * kHeadDim) + i4);
    }
    if (value) {
        const float2 lo = __half22float2(__floats2half2_rn(c.x, c.y)), hi = __half22float2(__floats2half2_rn(c.z, c.w));
        c = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    return c;
}

// Where the tiles of a launch are cut.  The tiles of a side's units lie end to end; they are cut where a unit ends and at
// every multiple of `piece` tiles of the side, and a piece longer than kUChunkMax tokens into segments of that many.  A
// segment is one set of FP32 partial sums, so the centres depend on the cuts and on nothing else: not on which CTA takes a
// piece, and not on whether K and V share a launch.
struct Cuts {
    int tiles_unit, tiles_side, tiles, piece;  // tiles: of all sides
};
struct Segment {
    int unit, tile0, tiles;
};
// First cut at or behind tile w (the end of all tiles if there is none).
__host__ __device__ inline int cut_from(const Cuts& c, int w) {
    if (w >= c.tiles) return c.tiles;
    const int side = w / c.tiles_side * c.tiles_side, in_side = w - side;
    const int by_piece = (in_side + c.piece - 1) / c.piece * c.piece, by_unit = (in_side + c.tiles_unit - 1) / c.tiles_unit * c.tiles_unit;
    return side + (by_piece < by_unit ? by_piece : by_unit);
}
// The segment that starts at tile w.
__host__ __device__ inline Segment segment_at(const Cuts& c, int w) {
    Segment sg;
    sg.unit = w / c.tiles_unit, sg.tile0 = w - sg.unit * c.tiles_unit;
    const int in_unit = c.tiles_unit - sg.tile0, in_piece = c.piece - w % c.tiles_side % c.piece;
    const int n = in_unit < in_piece ? in_unit : in_piece;
    sg.tiles = n < kUChunkMax / kUTile ? n : kUChunkMax / kUTile;
    return sg;
}

// The segment that ends in front of tile w (w > 0, a cut or the end of a segment).
__host__ __device__ inline Segment segment_before(const Cuts& c, int w) {
    constexpr int kMost = kUChunkMax / kUTile;
    const int last = w - 1, unit = last / c.tiles_unit, side = last / c.tiles_side * c.tiles_side;
    const int by_piece = side + (last - side) / c.piece * c.piece, by_unit = unit * c.tiles_unit;
    const int from = by_piece > by_unit ? by_piece : by_unit;  // the cut in front
    const int start = from + (last - from) / kMost * kMost;
    return Segment{unit, start - by_unit, w - start};
}
// What a CTA takes without a stop: the segment that comes at tile w in its order of the iteration and, if it belongs to the
// same unit, the one behind it.  Their sums are kept apart and meet as integers, so the cuts decide them as before.
struct Run {
    int unit, tile0, tiles, first_tiles;  // first_tiles: of the segment taken first
};
template <bool PAIRS>
__device__ inline Run run_at(const Cuts& c, int w, bool back, int work_begin, int work_end) {
    const Segment a = back ? segment_before(c, w) : segment_at(c, w);
    Run r{a.unit, a.tile0, a.tiles, a.tiles};
    const int next = back ? w - a.tiles : w + a.tiles, unit0 = a.unit * c.tiles_unit;
    if (PAIRS && (back ? next > work_begin && next > unit0 : next < work_end && next < unit0 + c.tiles_unit)) {
        const Segment b = back ? segment_before(c, next) : segment_at(c, next);
        r.tile0 = back ? b.tile0 : a.tile0, r.tiles += b.tiles;
    }
    return r;
}
// Segments of a unit.
__host__ __device__ inline int segments_of(const Cuts& c, int unit) {
    const int begin = unit * c.tiles_unit, in_side = begin % c.tiles_side;
    if (c.piece <= kUChunkMax / kUTile) return 1 + (in_side + c.tiles_unit - 1) / c.piece - in_side / c.piece;
    int n = 0;
    for (int w = begin; w < begin + c.tiles_unit; ++n) w += segment_at(c, w).tiles;
    return n;
}

// Waits until `count` segments of a unit have been flushed, by one thread.  Every CTA of the launch is resident and takes
// its segments iteration by iteration, so the wait ends; it gives up after 2^22 looks (seconds) all the same.
__device__ __forceinline__ bool wait_for_segments(const int* arrived, int count) {
    for (uint32_t spin = 0; spin < (1u << 22); ++spin) {
        int n;
        asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(n) : "l"(arrived) : "memory");
        if (n >= count) return true;
    }
    return false;
}

// PAIRS: CTAs may have two segments of a unit in a row (a launch that has none is 5 % faster without).
template <bool PAIRS>
__global__ void __launch_bounds__(kUThreads, 1) kmeans_assign_umma_kernel(const UmmaParams p, const __grid_constant__ CUtensorMap map0,
                                                                           const __grid_constant__ CUtensorMap map1, const Cuts cuts,
                                                                           int share) {
    extern __shared__ unsigned char smem_u[];
    constexpr int kN = 64;  // rows of the centre operand: hi halves, then lo halves (K's FP32 centres; V's are FP16)
    unsigned char* base = smem_u + ((1024u - (smem_u32(smem_u) & 1023u)) & 1023u);  // swizzled blocks: 1024-byte aligned
    unsigned char* xs = base;                                   // [stages][2 halves][128 tokens][128 B]
    unsigned char* cop = xs + kUStages * kUTileBytes;           // [2 halves][kN rows][128 B]
    unsigned char* oh = cop + 2 * kN * 128;                     // [groups][2 token halves][32 clusters][128 B]
    float* cen_s = reinterpret_cast<float*>(oh + kUGroups * kUOneHotBytes);  // [32][128] FP32 centres (exact re-ranking)
    float* cn_s = cen_s + 32 * kHeadDim;                        // [32] |c|^2, +inf for padding
    int* cnt_s = reinterpret_cast<int*>(cn_s + 32);             // [kURun][32]
    // full: tile landed (TMA bytes).  dist / sums: MMAs complete (tcgen05.commit); empty: the same event as sums,
    // counted per stage for the copying warp (a barrier of its own: no later completion can overtake its wait).
    // dist_free: the 128 threads of a group have read their distance buffer.  onehot: they have written their one-hot
    // operand.
    __shared__ uint64_t bar_full[kUStages], bar_empty[kUStages], bar_dist[kUGroups], bar_dist_free[kUGroups], bar_onehot[kUGroups],
        bar_sums[kUGroups];
    __shared__ uint32_t tmem_base_s;
    __shared__ Run runs_s[2];  // the run in work and the next one, in turn

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // CTA c takes the pieces that start in [c * share, (c + 1) * share) of all tiles and walks them segment by segment.
    // Tiles are numbered q = 0, 1, ... through the CTA's whole range: stage q % 5, group / distance buffer / one-hot
    // buffer q % 3, sum accumulator q % 4, and every barrier's phase follows from q, so the ring keeps turning across
    // segment boundaries (the copies of the next segment are in flight while this one drains and flushes).
    const int work_begin = cut_from(cuts, static_cast<int>(blockIdx.x) * share), work_end = cut_from(cuts, (static_cast<int>(blockIdx.x) + 1) * share);
    bool lost = false;

    if (tid == 0) {
        for (int s = 0; s < kUStages; ++s) mbar_init(&bar_full[s], 1), mbar_init(&bar_empty[s], 1);
        for (int b = 0; b < kUGroups; ++b) {
            mbar_init(&bar_dist[b], 1), mbar_init(&bar_sums[b], 1);
            mbar_init(&bar_dist_free[b], kUGroupWarps * 32), mbar_init(&bar_onehot[b], kUGroupWarps * 32);
        }
        mbar_fence_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(kUTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < kUGroups * kUOneHotBytes / 16; i += kUThreads) reinterpret_cast<uint4*>(oh)[i] = make_uint4(0, 0, 0, 0);
    tc_fence_before();
    __syncthreads();  // barriers initialised, TMEM allocated, one-hot buffers empty
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    constexpr int kWarpDist = kUGroups * kUGroupWarps, kWarpCopy = kWarpDist + 2;  // kWarpDist + 1 issues the sum MMAs

    if (warp == kWarpCopy) {
        // ---- copies, through all segments without a stop: the stage of tile q is free once the sums of tile
        // q - 5 have run (whole warp, one elected lane per tile) --------------------------------------------------
        int q = 0;
        for (int it = 0; it < p.iterations; ++it) {
            const bool back = it & 1;
            for (int w = back ? work_end : work_begin; back ? w > work_begin : w < work_end;) {
                const Segment sg = back ? segment_before(cuts, w) : segment_at(cuts, w);
                for (int i = 0; i < sg.tiles; ++i, ++q) {
                    const int row = (sg.tile0 + (back ? sg.tiles - 1 - i : i)) * kUTile;
                    if (q >= kUStages) lost |= !mbar_wait(&bar_empty[q % kUStages], (q / kUStages - 1) & 1);
                    unsigned char* dst = xs + (q % kUStages) * kUTileBytes;
                    uint64_t* bar = &bar_full[q % kUStages];
                    if (elect_one()) {
                        const CUtensorMap* xmap = sg.unit < p.units ? &map0 : &map1;
                        const int unit = sg.unit < p.units ? sg.unit : sg.unit - p.units;
                        mbar_arrive_expect_tx(bar, kUTileBytes);
                        tma_load_3d(dst, xmap, 0, row, unit, bar);
                        tma_load_3d(dst + kUBoxBytes, xmap, 64, row, unit, bar);
                    }
                    __syncwarp();
                }
                w += back ? -sg.tiles : sg.tiles;
            }
        }
    } else {
        int q0 = 0;     // tiles of the earlier segments of this CTA
        int prev = -1;  // byte offset of the element this thread set in its group's one-hot buffer
        int unit_in_tables = -1, segments = 0;  // unit of the tables, its segments
        int turn = 0;
        if (tid == (kWarpDist + 1) * 32 && work_begin < work_end) runs_s[0] = run_at<PAIRS>(cuts, work_begin, false, work_begin, work_end);
        workers_sync();
        for (int it = 0; it < p.iterations; ++it) {
            const bool first = it == 0, last = it + 1 == p.iterations, back = it & 1;
            bool stale = true;  // the tables are those of the iteration before
            for (int w = back ? work_end : work_begin; back ? w > work_begin : w < work_end;) {
                const int unit = runs_s[turn].unit, n_tiles = runs_s[turn].tiles, tile0 = runs_s[turn].tile0;
                const int first_tiles = PAIRS ? runs_s[turn].first_tiles : n_tiles, w_next = back ? w - n_tiles : w + n_tiles;
                const bool two = PAIRS && first_tiles < n_tiles;  // segments
                const int t_begin = tile0 * kUTile, t_end = min(p.tokens, t_begin + n_tiles * kUTile);
                const int side = unit < p.units ? 0 : 1, local = unit - side * p.units;
                const bool value = p.value[side] != 0;
                const __half* xu = p.x[side] + static_cast<size_t>(local) * p.x_stride[side] * kHeadDim;
                const size_t row0 = static_cast<size_t>(unit) * p.clusters;  // first centre of the unit
                const bool opens_unit = unit * cuts.tiles_unit >= work_begin;  // this CTA also keeps the unit's centres and zeroes its next sums
                // the whole unit is this CTA's: its first segment writes the sums instead of adding to zeros (a 64-bit atomic
                // addition costs eight times a store: 2300 cycles a segment), and no other CTA is waited for
                const bool owned = opens_unit && (unit + 1) * cuts.tiles_unit <= work_end;
                const bool writes = owned && (back ? tile0 + n_tiles == cuts.tiles_unit : tile0 == 0);
                // ---- per unit: centre operand (FP16 hi | lo rows, swizzled), FP32 centres, |c|^2 ----------------------
                if (stale || unit != unit_in_tables) {
                    if (unit != unit_in_tables && !owned) segments = segments_of(cuts, unit);
                    stale = false, unit_in_tables = unit;
                    // the sums of the iteration before are complete (a unit of one segment: this CTA has made them)
                    if (!first && !owned) {
                        if (tid == 0) lost |= !wait_for_segments(p.arrived + unit, it * segments);
                        workers_sync();
                    }
                    // four coordinates per thread and step, all loads of a thread in flight together
                    constexpr int kMakers = kUWorkers - 32;  // not the last worker warp, which may still announce the segment before
                    constexpr int kSteps = (32 * kHeadDim / 4 + kMakers - 1) / kMakers;
                    if (tid < kMakers) {
                        float4 v[kSteps];
                        CentreSums sums[kSteps];
                        if (!first) {
#pragma unroll
                            for (int k = 0; k < kSteps; ++k) {
                                const int i4 = min(tid + k * kMakers, p.clusters * (kHeadDim / 4) - 1);
                                sums[k] = load_sums(p, it - 1, row0 + i4 / (kHeadDim / 4), i4 % (kHeadDim / 4));
                            }
                        }
#pragma unroll
                        for (int k = 0; k < kSteps; ++k) {
                            const int i4 = tid + k * kMakers;
                            const int c = i4 / (kHeadDim / 4), d4 = i4 % (kHeadDim / 4);
                            v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                            if (i4 >= 32 * kHeadDim / 4 || c >= p.clusters) continue;
                            if (first) {
                                const uint2 raw = __ldg(reinterpret_cast<const uint2*>(xu + static_cast<size_t>(p.init.idx[c]) * kHeadDim) + d4);
                                const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
                                v[k] = make_float4(lo.x, lo.y, hi.x, hi.y);
                            } else {
                                v[k] = new_centre(p, sums[k], it - 1, value, row0 + c, d4);
                            }
                            if (opens_unit) {
                                reinterpret_cast<float4*>(p.centres[it & 1] + row0 * kHeadDim)[i4] = v[k];
                                if (owned) continue;
                                const longlong2 zero = make_longlong2(0, 0);
                                longlong2* ahead = reinterpret_cast<longlong2*>(p.sums[(it + 1) % 3] + row0 * kHeadDim) + 2 * i4;
                                ahead[0] = zero, ahead[1] = zero;
                                if (d4 == 0) p.counts[(it + 1) % 3][row0 + c] = 0;
                            }
                        }
#pragma unroll
                        for (int k = 0; k < kSteps; ++k) {
                            const int i4 = tid + k * kMakers;
                            if (i4 >= 32 * kHeadDim / 4) break;
                            const int c = i4 / (kHeadDim / 4), d = (i4 % (kHeadDim / 4)) * 4;
                            reinterpret_cast<float4*>(cen_s)[i4] = v[k];
                            const __half2 h01 = __floats2half2_rn(v[k].x, v[k].y), h23 = __floats2half2_rn(v[k].z, v[k].w);
                            unsigned char* at = cop + (d >> 6) * (kN * 128) + ((d & 7) << 1);
                            *reinterpret_cast<uint2*>(at + sw128(c, (d & 63) >> 3)) =
                                make_uint2(*reinterpret_cast<const uint32_t*>(&h01), *reinterpret_cast<const uint32_t*>(&h23));
                            float2 f01 = __half22float2(h01), f23 = __half22float2(h23);  // what the MMA sees: hi (+ lo)
                            if (!value) {
                                const __half2 l01 = __floats2half2_rn(v[k].x - f01.x, v[k].y - f01.y);
                                const __half2 l23 = __floats2half2_rn(v[k].z - f23.x, v[k].w - f23.y);
                                *reinterpret_cast<uint2*>(at + sw128(32 + c, (d & 63) >> 3)) =
                                    make_uint2(*reinterpret_cast<const uint32_t*>(&l01), *reinterpret_cast<const uint32_t*>(&l23));
                                const float2 g01 = __half22float2(l01), g23 = __half22float2(l23);
                                f01.x += g01.x, f01.y += g01.y, f23.x += g23.x, f23.y += g23.y;
                            }
                            // |c|^2: the 32 threads of a warp hold one centre (the worker count is a multiple of 32)
                            float sq = fmaf(f01.x, f01.x, fmaf(f01.y, f01.y, fmaf(f23.x, f23.x, f23.y * f23.y)));
#pragma unroll
                            for (int off = 16; off > 0; off >>= 1) sq += __shfl_xor_sync(kFull, sq, off);
                            if (lane == 0) cn_s[c] = c < p.clusters ? sq : INFINITY;
                        }
                    }
                }
                if (tid < (PAIRS ? 64 : 32)) cnt_s[tid] = 0;
                proxy_fence();  // the operands written above are read by the tensor core (async proxy)
                workers_sync();
                // the next run, by a thread whose first tile is the farthest; a handful of divisions, unless the CTA has only
                // this one, which it then takes the other way round
                if (tid == (kWarpDist + 1) * 32) {
                    const bool more = back ? w_next > work_begin : w_next < work_end;
                    if (!more && n_tiles == work_end - work_begin)
                        runs_s[turn ^ 1] = Run{unit, tile0, n_tiles, two ? n_tiles - first_tiles : n_tiles};
                    else if (more || !last)
                        runs_s[turn ^ 1] = more ? run_at<PAIRS>(cuts, w_next, back, work_begin, work_end)
                                                : run_at<PAIRS>(cuts, back ? work_begin : work_end, !back, work_begin, work_end);
                }
                float cmax = lane < p.clusters ? cn_s[lane] : 0.f;  // largest |c|^2, in every thread
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) cmax = fmaxf(cmax, __shfl_xor_sync(kFull, cmax, off));

                if (warp < kWarpDist) {
                    // ---- ranking: one thread per token; group g takes the tiles with q = g (mod 3), distance buffer g
                    // and one-hot buffer g ---------------------------------------------------------------------------
                    const int g = warp / kUGroupWarps, quarter = warp % kUGroupWarps, row_in_tile = quarter * 32 + lane;
                    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
                    // |x|^2 of a token is the same in every Lloyd iteration: the first one forms it and stores it (as FP32
                    // bits) where the token's id goes, the following ones read it from there one tile of the group ahead,
                    // the last one writes the id
                    int32_t* ids_u = p.ids[side] + static_cast<size_t>(local) * p.tokens;
                    int8_t* ids8_u = p.ids8[side] ? p.ids8[side] + static_cast<size_t>(local) * p.tokens : nullptr;
                    const int i_first = (g + kUGroups - q0 % kUGroups) % kUGroups;
                    const auto row_of = [&](int i) { return t_begin + (back ? n_tiles - 1 - i : i) * kUTile + row_in_tile; };
                    float xn_next = 0.f;
                    if (!first && i_first < n_tiles && row_of(i_first) < t_end) xn_next = __int_as_float(ids_u[row_of(i_first)]);
                    for (int i = i_first; i < n_tiles; i += kUGroups) {
                        const int q = q0 + i, use = q / kUGroups, st = q % kUStages;
                        const int row = row_of(i), tile_row = row - row_in_tile;
                        const bool live = row < t_end;
                        float xn = xn_next;
                        if (!first && i + kUGroups < n_tiles && row_of(i + kUGroups) < t_end) xn_next = __int_as_float(ids_u[row_of(i + kUGroups)]);
                        lost |= !mbar_wait(&bar_dist[g], use & 1);
                        tc_fence_after();
                        float d[32];
                        tmem_ld32(tmem + lane_base + kUColD + g * 64, d);
                        if (!value) {
                            float lo[32];
                            tmem_ld32(tmem + lane_base + kUColD + g * 64 + 32, lo);
                            tmem_ld_wait();
#pragma unroll
                            for (int c = 0; c < 32; ++c) d[c] += lo[c];
                        } else {
                            tmem_ld_wait();
                        }
                        tc_fence_before();
                        mbar_arrive(&bar_dist_free[g]);  // the next distances of this group may be issued
                        float d1 = INFINITY, d2 = INFINITY;
                        int c1 = 0;
#pragma unroll
                        for (int c = 0; c < 32; ++c) {  // branch-free: best, second best, index of the best
                            d[c] = fmaf(-2.f, d[c], cn_s[c]);
                            d2 = fminf(d2, fmaxf(d[c], d1));
                            c1 = d[c] < d1 ? c : c1;  // a strict comparison keeps the lower index on ties
                            d1 = fminf(d1, d[c]);
                        }
                        if (first) {
                            // |x|^2 for the near-tie bound: packed FP16 products, eight at a time (an overflow gives +inf:
                            // re-rank)
                            lost |= !mbar_wait(&bar_full[st], (q / kUStages) & 1);
                            const unsigned char* xt = xs + st * kUTileBytes;
                            xn = 0.f;
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const uint4 v = *reinterpret_cast<const uint4*>(xt + (j >> 3) * kUBoxBytes + sw128(row_in_tile, j & 7));
                                const __half2* h = reinterpret_cast<const __half2*>(&v);
                                __half2 s = __hmul2(h[0], h[0]);
                                s = __hfma2(h[1], h[1], s), s = __hfma2(h[2], h[2], s), s = __hfma2(h[3], h[3], s);
                                const float2 f = __half22float2(s);
                                xn += f.x + f.y;
                            }
                        }
                        // near-ties: only a centre whose distance lies inside the bound can win; the warp forms the exact
                        // FP32 sums of those few (same arithmetic, same order as `nearest`), one tied token at a time
                        const float bound = kTieBound * (1.01f * xn + cmax);
                        uint32_t inside = 0u;
                        if (live && !((d2 - d1) > bound)) {
#pragma unroll
                            for (int c = 0; c < 32; ++c) inside |= !((d[c] - d1) > bound) ? 1u << c : 0u;
                        }
                        uint32_t redo = __ballot_sync(kFull, inside != 0u);
                        while (redo) {
                            const int src = __ffs(redo) - 1;
                            redo &= redo - 1;
                            uint32_t cands = __shfl_sync(kFull, inside, src) & (p.clusters >= 32 ? 0xffffffffu : (1u << p.clusters) - 1u);
                            const __half* xr = xu + static_cast<size_t>(tile_row + quarter * 32 + src) * kHeadDim;
                            float xv[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k) xv[k] = __half2float(xr[lane + 32 * k]);
                            float best = INFINITY;
                            int bc = 0;
                            while (cands) {  // ascending centre index: the lower one wins ties
                                const int c = __ffs(cands) - 1;
                                cands &= cands - 1;
                                const float* crow = cen_s + c * kHeadDim;
                                float acc = 0.f;
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const float df = xv[e] - crow[lane + 32 * e];
                                    acc = fmaf(df, df, acc);
                                }
#pragma unroll
                                for (int off = 16; off > 0; off >>= 1) acc = acc + __shfl_xor_sync(kFull, acc, off);
                                if (acc < best) best = acc, bc = c;
                            }
                            if (lane == src) c1 = bc;
                        }
                        if (live) {
                            if (last) {
                                ids_u[row] = c1;
                                if (ids8_u) ids8_u[row] = static_cast<int8_t>(c1);
                            } else if (first) {
                                ids_u[row] = __float_as_int(xn);
                            }
                            atomicAdd(&cnt_s[(!PAIRS || i < first_tiles ? 0 : 32) + c1], 1);
                        }
                        // one-hot buffer g was last read by the sums of tile q - 3
                        if (q >= kUGroups) lost |= !mbar_wait(&bar_sums[g], (use - 1) & 1);
                        unsigned char* ob = oh + g * kUOneHotBytes;
                        if (prev >= 0) *reinterpret_cast<unsigned short*>(ob + prev) = 0;
                        prev = -1;
                        if (live) {
                            prev = (row_in_tile >> 6) * (32 * 128) + sw128(c1, (row_in_tile & 63) >> 3) + ((row_in_tile & 7) << 1);
                            *reinterpret_cast<unsigned short*>(ob + prev) = 0x3C00;  // 1.0
                        }
                        proxy_fence();  // the tensor core (async proxy) reads what this thread wrote
                        mbar_arrive(&bar_onehot[g]);
                    }
                } else if (warp == kWarpDist) {
                    // ---- distance MMAs (whole warp, one elected lane per tile): tile q goes to buffer q % 3 as soon as
                    // the group has read tile q - 3 out of it ----------------------------------------------------------
                    const uint64_t a0 = umma_desc(smem_u32(xs), 16, 1024), b0 = umma_desc(smem_u32(cop), 16, 1024);
                    const uint32_t idesc = value ? umma_idesc(32, false) : umma_idesc(64, false);  // V's centres have no lo half
                    for (int i = 0; i < n_tiles; ++i) {
                        const int q = q0 + i, buf = q % kUGroups;
                        if (q >= kUGroups) lost |= !mbar_wait(&bar_dist_free[buf], (q / kUGroups - 1) & 1);
                        lost |= !mbar_wait(&bar_full[q % kUStages], (q / kUStages) & 1);
                        tc_fence_after();
                        const uint64_t a = a0 + static_cast<uint64_t>(((q % kUStages) * kUTileBytes) >> 4);
                        const uint32_t d = tmem + kUColD + buf * 64;
                        if (elect_one()) {  // the eight MMAs and their commit in one elected stretch
#pragma unroll
                            for (int ks = 0; ks < 8; ++ks) {  // 16 coordinates per step: 32 bytes inside the swizzled 128-byte row
                                const uint64_t ak = a + static_cast<uint64_t>(((ks >> 2) * kUBoxBytes + (ks & 3) * 32) >> 4);
                                const uint64_t bk = b0 + static_cast<uint64_t>(((ks >> 2) * (kN * 128) + (ks & 3) * 32) >> 4);
                                umma_f16(d, ak, bk, idesc, ks > 0);
                            }
                            umma_commit(&bar_dist[buf]);
                        }
                        __syncwarp();
                    }
                } else {
                    // ---- sum MMAs: the first four tiles of a segment start the four accumulators ----------------------
                    const uint64_t a0 = umma_desc(smem_u32(xs), kUBoxBytes, 1024);  // MN-major: other half of the coordinates at LBO
                    const uint64_t b0 = umma_desc(smem_u32(oh), 16, 1024);
                    for (int i = 0; i < n_tiles; ++i) {
                        const int q = q0 + i, buf = q % kUGroups;
                        const uint64_t a = a0 + static_cast<uint64_t>(((q % kUStages) * kUTileBytes) >> 4);
                        const uint64_t o = b0 + static_cast<uint64_t>((buf * kUOneHotBytes) >> 4);
                        const int in_segment = !PAIRS || i < first_tiles ? i : i - first_tiles;
                        const uint32_t d = tmem + kUColS + ((!PAIRS || i < first_tiles ? 0 : kUSumBuffers) + in_segment % kUSumBuffers) * 32;
                        lost |= !mbar_wait(&bar_onehot[buf], (q / kUGroups) & 1);
                        tc_fence_after();
                        if (elect_one()) {
#pragma unroll
                            for (int ks = 0; ks < 8; ++ks) {  // 16 tokens per step: two 8-row groups of the tile = 2048 bytes
                                const uint64_t ak = a + static_cast<uint64_t>((ks * 2048) >> 4);
                                const uint64_t bk = o + static_cast<uint64_t>(((ks >> 2) * (32 * 128) + (ks & 3) * 32) >> 4);
                                umma_f16(d, ak, bk, umma_idesc(32, true), (in_segment >= kUSumBuffers || ks > 0) ? 1u : 0u);
                            }
                            umma_commit(&bar_sums[buf]);
                            umma_commit(&bar_empty[q % kUStages]);
                        }
                        __syncwarp();
                    }
                }
                // ---- end of the segment: its sums go out (the commit of the last sum MMAs covers all of them) -----------
                // The wait stands behind the barrier: a parity tells two neighbouring phases apart, and only once the last tile's
                // group has come this far is the phase before the awaited one over for sure.
                const bool flusher = warp < 2 * kUGroupWarps;  // groups 0 and 1: coordinate row_in_tile, sixteen clusters each
                workers_sync();
                if (flusher) {
                    const int q_last = q0 + n_tiles - 1;
                    lost |= !mbar_wait(&bar_sums[q_last % kUGroups], (q_last / kUGroups) & 1);
                    tc_fence_after();
                    const int half = warp / kUGroupWarps, quarter = warp % kUGroupWarps, row_in_tile = quarter * 32 + lane;
                    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
                    long long* sums_g = p.sums[it % 3] + row0 * kHeadDim;
                    const auto put = [&](int c, long long sum) {
                        long long* at = sums_g + c * kHeadDim + row_in_tile;
                        if (writes)
                            *at = sum;
                        else
                            atomicAdd(reinterpret_cast<unsigned long long*>(at), static_cast<unsigned long long>(sum));
                    };
                    if (two) {
#pragma unroll
                        for (int part = 0; part < 2; ++part) {  // eight clusters at a time
                            const int c0 = 16 * half + 8 * part;
                            float acc[2 * kUSumBuffers][8];
#pragma unroll
                            for (int a = 0; a < 2 * kUSumBuffers; ++a) tmem_ld8(tmem + lane_base + kUColS + a * 32 + c0, acc[a]);
#pragma unroll
                            for (int a = 0; a < 2 * kUSumBuffers; ++a) tmem_ld_wait(acc[a]);
#pragma unroll
                            for (int a = 1; a < kUSumBuffers; ++a) {  // added in the order they were started
#pragma unroll
                                for (int k = 0; k < 8; ++k) {
                                    if (a < first_tiles) acc[0][k] += acc[a][k];
                                    if (a < n_tiles - first_tiles) acc[kUSumBuffers][k] += acc[kUSumBuffers + a][k];
                                }
                            }
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const int c = c0 + k, n0 = cnt_s[c], n1 = cnt_s[32 + c];
                                if (c >= p.clusters || (!writes && n0 + n1 == 0)) continue;
                                put(c, (n0 > 0 ? __float2ll_rn(acc[0][k] * kFix) : 0) + (n1 > 0 ? __float2ll_rn(acc[kUSumBuffers][k] * kFix) : 0));
                            }
                        }
                    } else {
                        float acc[kUSumBuffers][16];  // all requested together
#pragma unroll
                        for (int a = 0; a < kUSumBuffers; ++a)  // one that no tile has used is read and not added
                            tmem_ld16(tmem + lane_base + kUColS + a * 32 + 16 * half, acc[a]);
#pragma unroll
                        for (int a = 0; a < kUSumBuffers; ++a) tmem_ld_wait(acc[a]);
#pragma unroll
                        for (int a = 1; a < kUSumBuffers; ++a)  // added in the order they were started
                            if (a < n_tiles) {
#pragma unroll
                                for (int k = 0; k < 16; ++k) acc[0][k] += acc[a][k];
                            }
#pragma unroll
                        for (int k = 0; k < 16; ++k) {
                            const int c = 16 * half + k, n = cnt_s[c];
                            if (c >= p.clusters || (!writes && n == 0)) continue;
                            put(c, n > 0 ? __float2ll_rn(acc[0][k] * kFix) : 0);
                        }
                    }
                }
                if (tid < p.clusters) {
                    int* at = &p.counts[it % 3][row0 + tid];
                    const int n = cnt_s[tid] + (PAIRS ? cnt_s[32 + tid] : 0);
                    if (writes)
                        *at = n;
                    else if (n > 0)
                        atomicAdd(at, n);
                }
                tc_fence_before();
                workers_sync();  // accumulators, counters and the centre tables are free for the next segment
                tc_fence_after();
                if (warp == kWarpDist + 1 && lane == 0 && !owned) {  // (the warp whose next step is the farthest)
                    __threadfence();
                    atomicAdd(p.arrived + unit, two ? 2 : 1);
                }
                q0 += n_tiles;
                w = w_next;
                turn ^= 1;
            }
        }
        // ---- FP16 centres of the units that begin here; a warp per centre --------------------------------------------
        for (int w = work_begin; w < work_end;) {
            const int unit = w / cuts.tiles_unit, begin = unit * cuts.tiles_unit;
            w = begin + cuts.tiles_unit;
            if (begin < work_begin) continue;  // the CTA that has its first tile writes them
            if (w > work_end) {
                if (tid == 0) lost |= !wait_for_segments(p.arrived + unit, p.iterations * segments_of(cuts, unit));
                workers_sync();
            }
            const int side = unit < p.units ? 0 : 1;
            for (int c = warp; c < p.clusters; c += kUWorkers / 32) {
                const size_t row = static_cast<size_t>(unit) * p.clusters + c;
                const float4 v = new_centre(p, load_sums(p, p.iterations - 1, row, lane), p.iterations - 1, p.value[side] != 0, row, lane);
                const __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
                reinterpret_cast<uint2*>(p.out[side] + (row - static_cast<size_t>(side) * p.units * p.clusters) * kHeadDim)[lane] =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            }
        }
    }
    if (lost) atomicOr(p.status, RESKV_STATUS_WAIT_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kUTmemCols) : "memory");
}

// New centres from the exact sums; clears sums and counts for the next round.
// `final_out` (FP16 [units, C, 128]) is written when non-null.
__global__ void kmeans_update_kernel(KmeansParams p, int value, __half* final_out) {
    const int unit = blockIdx.x;
    for (int i = threadIdx.x; i < p.clusters * kHeadDim; i += blockDim.x) {
        const size_t g = static_cast<size_t>(unit) * p.clusters * kHeadDim + i;
        const int n = p.counts[unit * p.clusters + i / kHeadDim];
        float c = p.centres[g];
        if (n > 0) {
            // exact integer sum / count, one rounding to FP32
            c = static_cast<float>(static_cast<double>(p.sums[g]) * (1.0 / 16777216.0) / static_cast<double>(n));
        } else if (value) {
            c = 0.f;
        }
        if (value) c = __half2float(__float2half_rn(c));
        p.centres[g] = c;
        p.sums[g] = 0;
        if (final_out) final_out[g] = __float2half_rn(c);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < p.clusters; c += blockDim.x) p.counts[unit * p.clusters + c] = 0;
}

// Decode-time step: grid (units, parts).  Optionally appends the mean of the group's tokens as centre
// `old_clusters`, then assigns the tokens.  Every CTA of a unit forms the same mean (the same additions in the
// same order); part 0 writes the new table; the tokens are assigned in `parts` contiguous slices, so that a
// small batch still fills the machine.
__global__ void __launch_bounds__(kThreads) kmeans_incremental_kernel(const __half* x, int64_t x_stride,
                                                                      const __half* old_cen, int old_clusters,
                                                                      __half* new_cen, int new_clusters, int tokens,
                                                                      int32_t* ids) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* cen_s = reinterpret_cast<float*>(smem);  // [new_clusters][128]
    const int unit = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool writer = blockIdx.y == 0;
    const __half* xg = x + static_cast<size_t>(unit) * x_stride * kHeadDim;
    for (int i = tid; i < old_clusters * kHeadDim; i += kThreads) {
        const __half v = old_cen[static_cast<size_t>(unit) * old_clusters * kHeadDim + i];
        cen_s[i] = __half2float(v);
        if (writer) new_cen[static_cast<size_t>(unit) * new_clusters * kHeadDim + i] = v;
    }
    if (new_clusters > old_clusters && tid < kHeadDim) {
        // mean of the group, FP32 accumulation in token order, rounded to FP16; the loads of eight tokens are
        // requested together, the additions stay sequential
        float s = 0.f;
        int t = 0;
        for (; t + 8 <= tokens; t += 8) {
            __half v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = xg[static_cast<size_t>(t + u) * kHeadDim + tid];
#pragma unroll
            for (int u = 0; u < 8; ++u) s += __half2float(v[u]);
        }
        for (; t < tokens; ++t) s += __half2float(xg[static_cast<size_t>(t) * kHeadDim + tid]);
        const __half m = __float2half_rn(s / static_cast<float>(tokens));
        cen_s[old_clusters * kHeadDim + tid] = __half2float(m);
        if (writer) new_cen[(static_cast<size_t>(unit) * new_clusters + old_clusters) * kHeadDim + tid] = m;
    }
    __syncthreads();
    const int per = (tokens + gridDim.y - 1) / gridDim.y;
    const int t_end = min(tokens, static_cast<int>(blockIdx.y + 1) * per);
    for (int t = blockIdx.y * per + warp; t < t_end; t += kWarps) {
        float xv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) xv[i] = __half2float(xg[static_cast<size_t>(t) * kHeadDim + lane + 32 * i]);
        float best;
        int c;
        nearest(cen_s, new_clusters, xv, lane, best, c);
        if (lane == 0) ids[static_cast<size_t>(unit) * tokens + t] = c;
    }
}

// torch.linspace(0, t-1, count).long(): float32 steps formed with a fused
// multiply-add, symmetric about the midpoint, truncated.
void linspace_indices(int t, int count, int* out) {
    if (count == 1) {
        out[0] = 0;
        return;
    }
    const float step = static_cast<float>(t - 1) / static_cast<float>(count - 1);
    for (int i = 0; i < count; ++i) {
        const double v = i < count / 2 ? static_cast<double>(step) * i
                                       : static_cast<double>(t - 1) - static_cast<double>(step) * (count - 1 - i);
        out[i] = static_cast<int>(static_cast<float>(v));
    }
}

// 256 bytes whose first word is the status word, flushed segments per unit, then three generations of counts, three of sums,
// two of centres (the mma.sync form uses the first of each).  What a call starts from as zeros lies in front.
constexpr size_t round16(size_t bytes) { return (bytes + 15) / 16 * 16; }
size_t kmeans_ws_bytes(int units, int clusters) {
    const size_t per = static_cast<size_t>(units) * clusters;
    return 256 + round16(units * sizeof(int)) + 3 * round16(per * sizeof(int)) + per * kHeadDim * (3 * sizeof(long long) + 2 * sizeof(float));
}

// x as (coordinate, token, unit): boxes of 64 coordinates x 128 tokens, 128-byte swizzle, zeros beyond the last token of
// a unit
int token_map(CUtensorMap* map, const __half* x, int tokens, int units, int64_t x_stride) {
    const cuuint64_t dims[3] = {kHeadDim, static_cast<cuuint64_t>(tokens), static_cast<cuuint64_t>(units)};
    const cuuint64_t strides[2] = {kHeadDim * sizeof(__half), static_cast<cuuint64_t>(x_stride) * kHeadDim * sizeof(__half)};
    const cuuint32_t box[3] = {64, kUTile, 1};
    return encode_tensor_map(map, x, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B, "kmeans");
}

// The workspace's arrays for `units` units (all sides together).
void place_state(UmmaParams& p, void* workspace, int units, int clusters) {
    const size_t per = static_cast<size_t>(units) * clusters;
    unsigned char* at = static_cast<unsigned char*>(workspace) + 256;
    p.status = static_cast<uint32_t*>(workspace);
    p.arrived = reinterpret_cast<int*>(at), at += round16(units * sizeof(int));
    p.counts[0] = reinterpret_cast<int*>(at), at += round16(per * sizeof(int));
    for (int i = 0; i < 3; ++i, at += per * kHeadDim * sizeof(long long)) p.sums[i] = reinterpret_cast<long long*>(at);
    for (int i = 0; i < 2; ++i, at += per * kHeadDim * sizeof(float)) p.centres[i] = reinterpret_cast<float*>(at);
    for (int i = 1; i < 3; ++i, at += round16(per * sizeof(int))) p.counts[i] = reinterpret_cast<int*>(at);
}

// Tiles per CTA of a call for one side, which is also where its tiles are cut.  One CTA per SM, every CTA an equal share of
// all units' tiles, at least four.  A segment is charged ten tile times (pipeline drain, flush, new centre tables, refill),
// what it cost with a launch per iteration; in the present form, where runs, owned units and early requests have made it
// cheaper, it was not measured again.  The share is chosen - between the even split and half as much again - for the
// shortest slowest CTA under that charge: one that divides the units evenly often beats the smallest one, but may leave SMs
// without work (64 units x 8128 tokens: 64 tiles on each of 128 CTAs, an even split would be 55.4 on 148).
int side_share(int tiles_side, int tiles_unit) {
    constexpr int kLeast = 4, seg_max = kUChunkMax / kUTile;
    const int even = (tiles_side + sm_count() - 1) / sm_count();
    const int low = even < kLeast ? kLeast : even;
    int share = low, best_cost = -1;
    for (int cand = low; cand <= low + low / 2 + 1; ++cand) {
        int worst = 0;
        int in_unit = tiles_unit;  // tiles left in the unit
        for (int left = tiles_side; left > 0 && (best_cost < 0 || worst < best_cost);) {
            const int work = cand < left ? cand : left;
            int segments = 0;
            for (int rest = work; rest > 0; ++segments) {  // same walk as the kernel's
                int n = in_unit < rest ? in_unit : rest;
                if (n > seg_max) n = seg_max;
                rest -= n, in_unit -= n;
                if (in_unit == 0) in_unit = tiles_unit;
            }
            if (work + 10 * segments > worst) worst = work + 10 * segments;
            left -= work;
        }
        if (best_cost < 0 || worst < best_cost) best_cost = worst, share = cand;
    }
    return share;
}

// Tiles per CTA when K and V share the launches.  They are cut as a call for one side cuts them, so that ids and centres
// are those of two such calls bit for bit; only how many of the pieces a CTA takes is chosen here, again for the shortest
// slowest CTA.  A segment of the unit whose tables a CTA already has is counted as four tile times, one of another unit as
// ten, measured with a launch per iteration like side_share's (there 7 and 1, 7 and 3, 14 and 2 chose shares of the same
// time, 8 units x 1152 to 64 x 8128 tokens).  About `kTries` shares are looked at (host time).
int pair_share(const Cuts& c) {
    constexpr int kNewUnit = 10, kSameUnit = 4, kTries = 16, seg_max = kUChunkMax / kUTile;
    const int low = (c.tiles + sm_count() - 1) / sm_count();
    int share = low, best_cost = -1;
    for (int cand = low; cand <= low + low / 2 + 1; cand += low / (2 * kTries) + 1) {
        int worst = 0, cost = 0, unit_of_cta = -1;
        int unit = 0, in_unit = c.tiles_unit, in_side = c.tiles_side, in_piece = c.piece;  // tiles left
        long long next_cta = cand;
        for (int w = 0; w < c.tiles && (best_cost < 0 || worst < best_cost);) {
            if (w >= next_cta) {
                do next_cta += cand; while (w >= next_cta);
                cost = 0, unit_of_cta = -1;
            }
            const int n = in_unit < in_piece ? in_unit : in_piece;
            cost += n + (unit == unit_of_cta ? kSameUnit : kNewUnit) + (n - 1) / seg_max * kSameUnit;
            unit_of_cta = unit;
            if (cost > worst) worst = cost;
            w += n, in_unit -= n, in_side -= n, in_piece -= n;
            if (in_unit == 0) in_unit = c.tiles_unit, ++unit;
            if (in_side == 0) in_side = c.tiles_side, in_piece = c.piece;
            if (in_piece == 0) in_piece = c.piece;
        }
        if (best_cost < 0 || worst < best_cost) best_cost = worst, share = cand;
    }
    return share;
}

int launch_umma(UmmaParams& p, void* centroids0, void* centroids1, cudaStream_t s) {
    CUtensorMap maps[2];
    for (int i = 0; i < 2; ++i)  // one side: the second map repeats the first and is not used
        if (int rc = token_map(&maps[i], p.x[i < p.sides ? i : 0], p.tokens, p.units, p.x_stride[i < p.sides ? i : 0])) return rc;
    p.out[0] = static_cast<__half*>(centroids0), p.out[1] = static_cast<__half*>(centroids1);
    // status, flushed segments, and what the first iteration adds to; every iteration zeroes the next one's
    const size_t per = static_cast<size_t>(p.sides) * p.units * p.clusters;
    const size_t zeros = reinterpret_cast<unsigned char*>(p.sums[0] + per * kHeadDim) - reinterpret_cast<unsigned char*>(p.status);
    if (int rc = check_cuda(cudaMemsetAsync(p.status, 0, zeros, s), "kmeans: memset")) return rc;
    constexpr int kN = 64;
    const size_t smem = 1024 + static_cast<size_t>(kUStages) * kUTileBytes + 2 * kN * 128 + kUGroups * kUOneHotBytes +
                        32 * kHeadDim * sizeof(float) + 32 * (sizeof(float) + kURun * sizeof(int));
    Cuts cuts{};
    cuts.tiles_unit = (p.tokens + kUTile - 1) / kUTile;
    cuts.tiles_side = p.units * cuts.tiles_unit, cuts.tiles = p.sides * cuts.tiles_side;
    cuts.piece = side_share(cuts.tiles_side, cuts.tiles_unit);
    int share = p.sides == 2 ? pair_share(cuts) : cuts.piece;
    const bool pairs = share > cuts.piece && cuts.piece % cuts.tiles_unit != 0;
    const auto kern = pairs ? kmeans_assign_umma_kernel<true> : kmeans_assign_umma_kernel<false>;
    static std::atomic<unsigned long long> done[2];
    if (int rc = allow_smem(kern, smem, done[pairs], "cudaFuncSetAttribute(kmeans_assign_umma)")) return rc;
    // cooperative: CTAs wait for one another between iterations, so all of them have to be resident, and the launch starts
    // only once every one of them has its place: beside a long kernel of another stream later than an ordinary launch, which
    // could begin on the SMs that are free.  A context that has only a part of the SMs takes fewer CTAs with more pieces
    // each; the cuts, and with them the results, stay.
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kUThreads), cfg.dynamicSmemBytes = smem, cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr, cfg.numAttrs = 1;
    for (;; share *= 2) {
        cfg.gridDim = dim3(static_cast<unsigned>((cuts.tiles + share - 1) / share));
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p, maps[0], maps[1], cuts, share);
        if (e != cudaErrorCooperativeLaunchTooLarge || cfg.gridDim.x == 1) return check_cuda(e, "kmeans launch");
        cudaGetLastError();  // the refused launch must not poison later calls
    }
}

}  // namespace
}  // namespace reskv

using namespace reskv;

extern "C" size_t reskv_kmeans_workspace_bytes(int batch, int kv_heads, int clusters) {
    if (batch < 1 || kv_heads < 1 || clusters < 1 || clusters > kMaxClusters) return 0;
    return kmeans_ws_bytes(batch * kv_heads, clusters);
}

extern "C" int reskv_kmeans(const void* x, int batch, int kv_heads, int tokens, int64_t x_tok_stride, int clusters,
                            int iterations, int value, void* workspace, size_t workspace_bytes, void* centroids,
                            int32_t* ids, void* stream) {
    if (!x || !centroids || !ids) return fail(RESKV_ERR_INVALID, "kmeans: null tensor pointer");
    if (batch < 1 || kv_heads < 1 || tokens < 1) return fail(RESKV_ERR_INVALID, "kmeans: batch, heads and tokens must be positive");
    if (clusters < 1 || clusters > kMaxClusters) return fail(RESKV_ERR_INVALID, "kmeans: cluster count must be in [1,64], got %d", clusters);
    if (iterations < 1) return fail(RESKV_ERR_INVALID, "kmeans: iterations must be positive");
    if (x_tok_stride < tokens) return fail(RESKV_ERR_INVALID, "kmeans: token stride smaller than token count");
    const int units = batch * kv_heads;
    const size_t need = kmeans_ws_bytes(units, clusters);
    if (!workspace || workspace_bytes < need)
        return fail(RESKV_ERR_WORKSPACE, "kmeans: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
    if (int rc = check_device_pointer(x, "kmeans", "x")) return rc;
    if (int rc = check_device_pointer(centroids, "kmeans", "centroids")) return rc;
    KmeansParams p{};
    p.x = static_cast<const __half*>(x);
    UmmaParams u{};
    place_state(u, workspace, units, clusters);
    p.sums = u.sums[0], p.centres = u.centres[0], p.counts = u.counts[0], p.status = u.status;
    p.ids = ids;
    p.x_stride = x_tok_stride;
    p.units = units, p.tokens = tokens, p.clusters = clusters;
    InitIndex init{};
    if (tokens >= clusters) {
        linspace_indices(tokens, clusters, init.idx);
    } else {
        // fewer tokens than centres: every token once, then tokens repeated in order
        for (int c = 0; c < clusters; ++c) init.idx[c] = c % tokens;
    }
    // `value`: bit 0 = V flavour, bit 1 = exact (integer) accumulation of the cluster sums, bit 2 = the mma.sync
    // form of the tensor-core sums instead of the tcgen05 one
    const bool exact = (value & 2) != 0, warp_mma = (value & 4) != 0;
    value &= 1;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int padded = (clusters + 7) / 8 * 8;
    // the integer-counter arrays double as the FP32 reduction buffer [32][kRedStride] of the tensor-core form
    size_t counters = static_cast<size_t>(clusters) * kHeadDim * 2 * sizeof(int);
    const bool fast = !exact && padded <= 32 && aligned16(x);  // the row staging copies 16-byte pieces
    if (fast && !warp_mma && aligned16(workspace) && aligned16(centroids)) {
        u.x[0] = p.x, u.x_stride[0] = x_tok_stride, u.ids[0] = ids, u.value[0] = value, u.sides = 1;
        u.units = units, u.tokens = tokens, u.clusters = clusters, u.iterations = iterations, u.init = init;
        return launch_umma(u, centroids, nullptr, s);
    }
    kmeans_init_kernel<<<units, 256, 0, s>>>(p, init, value);
    if (fast) counters = static_cast<size_t>(kWarps) * 32 * kRedStride * sizeof(float);
    const size_t smem = static_cast<size_t>(clusters) * kHeadDim * sizeof(float) + counters +
                        kMaxClusters * (sizeof(int) + sizeof(float)) +
                        static_cast<size_t>(padded) * kCenHalfStride * sizeof(__half) * (value ? 1 : 2) +
                        (fast ? static_cast<size_t>(kWarps) * 16 * kXsRow : 0);
    void (*kernel)(const KmeansParams, int, int) =
        fast ? (value ? kmeans_assign_mma_kernel<false, true> : kmeans_assign_mma_kernel<true, true>)
             : (value ? kmeans_assign_mma_kernel<false, false> : kmeans_assign_mma_kernel<true, false>);
    if (smem > 48 * 1024) {
        if (int rc = check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                                "cudaFuncSetAttribute(kmeans_assign)"))
            return rc;
    }
    // tensor-core form: as many tokens per CTA as still leave about two CTAs per SM (set-up and the final
    // reduction are per CTA), between kChunk and kChunkFastMax
    int chunk = kChunk;
    if (fast) {
        const long long want = static_cast<long long>(units) * tokens / (2ll * sm_count());
        chunk = static_cast<int>(want < kChunk ? kChunk : want > kChunkFastMax ? kChunkFastMax : (want + 127) / 128 * 128);
    }
    const dim3 grid((tokens + chunk - 1) / chunk, units);
    for (int it = 0; it < iterations; ++it) {
        kernel<<<grid, kThreads, smem, s>>>(p, padded, chunk);
        kmeans_update_kernel<<<units, 256, 0, s>>>(p, value, it + 1 == iterations ? static_cast<__half*>(centroids) : nullptr);
    }
    return check_cuda(cudaGetLastError(), "kmeans launch");
}

extern "C" int reskv_kmeans_pair(const void* x_k, const void* x_v, int batch, int kv_heads, int tokens, int64_t k_tok_stride,
                                 int64_t v_tok_stride, int clusters, int iterations, void* workspace, size_t workspace_bytes,
                                 void* k_centroids, void* v_centroids, int32_t* k_ids, int32_t* v_ids, void* k_ids8, void* v_ids8,
                                 void* stream) {
    if (!x_k || !x_v || !k_centroids || !v_centroids || !k_ids || !v_ids) return fail(RESKV_ERR_INVALID, "kmeans_pair: null tensor pointer");
    if (batch < 1 || kv_heads < 1 || tokens < 1) return fail(RESKV_ERR_INVALID, "kmeans_pair: batch, heads and tokens must be positive");
    if (clusters < 1 || clusters > 32 || clusters > tokens)
        return fail(RESKV_ERR_INVALID, "kmeans_pair: cluster count must be in [1,32] and at most the token count, got %d", clusters);
    if (iterations < 1) return fail(RESKV_ERR_INVALID, "kmeans_pair: iterations must be positive");
    if (k_tok_stride < tokens || v_tok_stride < tokens) return fail(RESKV_ERR_INVALID, "kmeans_pair: token stride smaller than token count");
    const int units = batch * kv_heads;
    const size_t need = kmeans_ws_bytes(2 * units, clusters);
    if (!workspace || workspace_bytes < need)
        return fail(RESKV_ERR_WORKSPACE, "kmeans_pair: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
    for (const void* ptr : {x_k, x_v, static_cast<const void*>(workspace), static_cast<const void*>(k_centroids), static_cast<const void*>(v_centroids)})
        if (!aligned16(ptr)) return fail(RESKV_ERR_INVALID, "kmeans_pair: x, workspace and centroids must be 16-byte aligned");
    if (int rc = check_device_pointer(x_k, "kmeans_pair", "x_k")) return rc;
    if (int rc = check_device_pointer(x_v, "kmeans_pair", "x_v")) return rc;
    UmmaParams u{};
    place_state(u, workspace, 2 * units, clusters);
    u.x[0] = static_cast<const __half*>(x_k), u.x[1] = static_cast<const __half*>(x_v);
    u.x_stride[0] = k_tok_stride, u.x_stride[1] = v_tok_stride;
    u.ids[0] = k_ids, u.ids[1] = v_ids, u.ids8[0] = static_cast<int8_t*>(k_ids8), u.ids8[1] = static_cast<int8_t*>(v_ids8);
    u.value[0] = 0, u.value[1] = 1;
    u.sides = 2, u.units = units, u.tokens = tokens, u.clusters = clusters, u.iterations = iterations;
    linspace_indices(tokens, clusters, u.init.idx);
    return launch_umma(u, k_centroids, v_centroids, static_cast<cudaStream_t>(stream));
}

extern "C" int reskv_kmeans_status(const void* workspace, int batch, int kv_heads, int clusters, uint32_t* status, void* stream) {
    if (!workspace || !status) return fail(RESKV_ERR_INVALID, "kmeans_status: null pointer");
    if (batch < 1 || kv_heads < 1 || clusters < 1 || clusters > kMaxClusters) return fail(RESKV_ERR_INVALID, "kmeans_status: bad sizes");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (int rc = check_cuda(cudaMemcpyAsync(status, workspace, sizeof(uint32_t),
                                            cudaMemcpyDeviceToHost, s),
                            "kmeans_status copy"))
        return rc;
    return check_cuda(cudaStreamSynchronize(s), "kmeans_status synchronize");
}

extern "C" int reskv_kmeans_incremental(const void* x, int batch, int kv_heads, int tokens, int64_t x_tok_stride,
                                        const void* old_centroids, int old_clusters, void* new_centroids,
                                        int new_clusters, int32_t* ids, void* stream) {
    if (!x || !old_centroids || !new_centroids || !ids) return fail(RESKV_ERR_INVALID, "kmeans_incremental: null tensor pointer");
    if (int rc = check_device_pointer(x, "kmeans_incremental", "x")) return rc;
    if (int rc = check_device_pointer(new_centroids, "kmeans_incremental", "new_centroids")) return rc;
    if (batch < 1 || kv_heads < 1 || tokens < 1) return fail(RESKV_ERR_INVALID, "kmeans_incremental: batch, heads and tokens must be positive");
    if (old_clusters < 1 || new_clusters > kMaxClusters || (new_clusters != old_clusters && new_clusters != old_clusters + 1))
        return fail(RESKV_ERR_INVALID, "kmeans_incremental: centre counts must satisfy 1 <= old <= new <= old + 1 <= 64");
    if (x_tok_stride < tokens) return fail(RESKV_ERR_INVALID, "kmeans_incremental: token stride smaller than token count");
    const size_t smem = static_cast<size_t>(new_clusters) * kHeadDim * sizeof(float);
    // slices of the group per unit: enough CTAs for one per SM, at least one warp-load of tokens each
    int parts = 1;
    while (parts < 8 && batch * kv_heads * parts < sm_count() && tokens >= 2 * kWarps * parts) parts *= 2;
    kmeans_incremental_kernel<<<dim3(batch * kv_heads, parts), kThreads, smem, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __half*>(x), x_tok_stride, static_cast<const __half*>(old_centroids), old_clusters,
        static_cast<__half*>(new_centroids), new_clusters, tokens, ids);
    return check_cuda(cudaGetLastError(), "kmeans_incremental launch");
}
