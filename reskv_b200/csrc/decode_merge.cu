// Second kernel of a decode call: reduces the split-K partial results of a unit, applies the value centroids and folds
// the dense recent window into the same softmax.  Also serves the stand-alone merges of a finished compressed result
// with a window.
//
// What bounds it: memory latency, not bytes (a unit reads a few KB of partials and at most 48 KB of window).  A CTA of
// eight warps takes one, two or four query heads of a (sequence, KV head); a warp takes every eighth partial slot and
// every eighth block of 16 window tokens, with all loads of a pass requested before anything waits, and keeps a running
// softmax over both in registers: one trip to memory, two barriers.  (The form before it staged keys and values through
// shared memory in chunks of 32 tokens with barriers in between and read the partials after their maxima: 7.5 us at 192
// tokens and 12-17 us with the ~40 slots per unit of a batch-1 call at 8K.)  Scores of the window are MMAs on the FP16
// operands (exact products, FP32 sums); probabilities and the weighted sum stay FP32.
// Measured, calls back to back: without any merge 7.8 us at batch 1, 192 tokens, 15.2 us at 8128 tokens, 23.3 us at batch
// 3 with eight heads per KV head; with this kernel 11.4, 19.9 and 28.3 us (12.0, 22.4 and 30.2 with four heads per CTA always).
// Merging in the partial kernel's last CTA of a unit instead was slower (14.6, 24.1, 33.2 us): this launch's first half
// runs beside the partial kernel.
#include "decode_common.cuh"

namespace reskv {
namespace {

constexpr int kMergeWarps = 8;
constexpr int kMergeThreads = kMergeWarps * 32;
constexpr int kBlock = 16;                      // window tokens a warp takes at a time
constexpr int kPart = kHeadDim + kMaxClusters;  // floats per (warp, head): numerator, cluster masses

// value centroids, a block of window values per warp, partial results, (joint max, max, sum, window sum) and weight per
// warp and head, probabilities per warp, cluster masses and sum per head
template <int G>
constexpr size_t merge_smem_bytes(int cv) {
    return (static_cast<size_t>(cv) + kMergeWarps * kBlock) * kHeadDim * sizeof(__half) +
           (static_cast<size_t>(kMergeWarps) * G * (kPart + 4 + 1 + kBlock) + G * (kMaxClusters + 4)) * sizeof(float);
}

// 2^(a - b) for a <= b, 0 when a is -inf (b may be, too)
__device__ __forceinline__ float rel_exp2(float a, float b) { return a == -INFINITY ? 0.f : fast_exp2(a - b); }

// A CTA merges the heads [G blockIdx.y, G blockIdx.y + G) of unit blockIdx.x (those the unit has).
template <int G>
__global__ void __launch_bounds__(kMergeThreads, 2) decode_merge_kernel(const MergeParams p, int cv, int recent_max) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int unit = blockIdx.x, head0 = blockIdx.y * G, used = p.splits;
    const int gqa = p.nh / p.kh, heads = min(G, gqa - head0);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, q = lane & 3;
    const int fq0 = unit * gqa + head0;  // first query head row of the group
    __half* vc_s = reinterpret_cast<__half*>(smem);
    unsigned char* mine = smem + static_cast<size_t>(cv) * kHeadDim * sizeof(__half);
    // may run while the partial kernel drains: the window, the query and the value centroids are older than that kernel
    let_next_launch_start();
    __half* rv_s = reinterpret_cast<__half*>(mine) + warp * kBlock * kHeadDim;                       // [16][128] of this warp
    float* part_s = reinterpret_cast<float*>(mine + kMergeWarps * kBlock * kHeadDim * sizeof(__half));  // [warps][G][kPart]
    float* stat_s = part_s + kMergeWarps * G * kPart;                                                    // [warps][G][4]
    float* beta_s = stat_s + kMergeWarps * G * 4;                                                        // [G][64]
    float* prob_s = beta_s + G * kMaxClusters + warp * kBlock * G;                                       // [16][G] of this warp
    float* weight_s = beta_s + G * kMaxClusters + kMergeWarps * kBlock * G;                              // [warps][G]
    float* total_s = weight_s + kMergeWarps * G;                                                         // [G]
    const int counted = p.dyn ? __ldcg(p.dyn + 1) : p.tr;
    const int tr = p.dyn ? max(min(counted, recent_max), 0) : counted;
    for (int i = tid; i < cv * (kHeadDim / 8); i += kMergeThreads)
        cp_async16(vc_s + i * 8, p.vc + static_cast<size_t>(unit) * p.cv * kHeadDim + i * 8);

    // ---- requests of the window's first block and of the rotated query ----------------------------------------------
    const __half* rk_g = p.rk ? p.rk + static_cast<size_t>(unit) * p.recent_cap * kHeadDim : nullptr;
    const __half* rv_g = p.rv ? p.rv + static_cast<size_t>(unit) * p.recent_cap * kHeadDim : nullptr;
    const bool dot = !p.rscores;
    uint4 kf[2][4];        // keys of tokens g and g + 8: coordinates [16 q, 16 q + 16) and [64 + 16 q, ...)
    auto piece = [&](int k) { return (k < 2 ? 0 : 8) + 2 * q + (k & 1); };  // 16-byte piece of a row
    auto load_keys = [&](int base) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = base + g + 8 * r;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                kf[r][k] = t < tr ? __ldcg(reinterpret_cast<const uint4*>(rk_g + static_cast<size_t>(t) * kHeadDim) + piece(k))
                                  : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    auto load_values = [&](int base) {  // this warp's block, asynchronously
        const int n = min(kBlock, tr - base) * (kHeadDim / 8);
        for (int i = lane; i < n; i += 32) cp_async16(rv_s + i * 8, rv_g + static_cast<size_t>(base) * kHeadDim + i * 8);
    };
    uint4 qf[4];
    if (warp * kBlock < tr) {
        if (dot) {
            load_keys(warp * kBlock);
            const __half* qrow = p.rq + static_cast<size_t>(fq0 + (g < heads ? g : 0)) * kHeadDim;
            const bool wide = (reinterpret_cast<uintptr_t>(p.rq) & 15u) == 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (wide) {
                    qf[k] = __ldcg(reinterpret_cast<const uint4*>(qrow) + piece(k));
                } else {
                    const unsigned short* h = reinterpret_cast<const unsigned short*>(qrow) + 8 * piece(k);
                    qf[k] = make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
                }
                if (g >= heads) qf[k] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        load_values(warp * kBlock);
    }

    wait_for_previous_launch();
    // a window count beyond the buffers is cut (the newest tokens are then missing from the result): tell the host
    if (p.dyn && p.status && tid == 0 && unit == 0 && head0 == 0 && counted != tr) atomicOr(p.status, RESKV_STATUS_STATE_RANGE);

    // ---- compressed part: this warp's slots ---------------------------------------------------------------------------
    // per head: running maximum (log2 domain) and sum of the compressed tokens; numerator and cluster masses
    float mc[G], lc[G], acc[G][4], bet[G][4];
#pragma unroll
    for (int h = 0; h < G; ++h) {
        mc[h] = -INFINITY, lc[h] = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[h][i] = bet[h][i] = 0.f;
    }
    if (p.splits == 0 && warp == 0) {  // one finished result: numerator = result x sum
#pragma unroll
        for (int h = 0; h < G; ++h) {
            if (h >= heads) continue;
            mc[h] = p.ws_m[fq0 + h] * kLog2e, lc[h] = p.ws_l[fq0 + h];
            const __half* row = p.comp_out + static_cast<size_t>(fq0 + h) * kHeadDim + 4 * lane;
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[h][i] = __half2float(row[i]) * lc[h];
        }
    }
    constexpr int kAhead = 4 / G;  // slots requested together
    for (int first = warp; first < used; first += kAhead * kMergeWarps) {
        float pm[kAhead], pl[kAhead];
        float4 dv[kAhead][G], bv[kAhead][G];  // rows of an empty slot were never written: read, but not used
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const int s = min(first + k * kMergeWarps, used - 1);
            const bool have = lane < heads && first + k * kMergeWarps < used;
            pm[k] = have ? __ldcg(p.ws_m + static_cast<size_t>(fq0 + lane) * used + s) : -INFINITY;
            pl[k] = have ? __ldcg(p.ws_l + static_cast<size_t>(fq0 + lane) * used + s) : 0.f;
#pragma unroll
            for (int h = 0; h < G; ++h) {
                const size_t row = static_cast<size_t>(fq0 + (h < heads ? h : 0)) * used + s;
                dv[k][h] = __ldcg(reinterpret_cast<const float4*>(p.ws_delta + row * kHeadDim + 4 * lane));
                bv[k][h] = __ldcg(reinterpret_cast<const float4*>(p.ws_beta + row * kMaxClusters + 4 * (lane & 15)));
            }
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
#pragma unroll
            for (int h = 0; h < G; ++h) {
                const float m = __shfl_sync(0xffffffffu, pm[k], h), l = __shfl_sync(0xffffffffu, pl[k], h);
                if (m == -INFINITY) continue;
                const float mn = fmaxf(mc[h], m), a = rel_exp2(mc[h], mn), w = fast_exp2(m - mn);
                mc[h] = mn, lc[h] = lc[h] * a + l * w;
                const float d[4] = {dv[k][h].x, dv[k][h].y, dv[k][h].z, dv[k][h].w}, e[4] = {bv[k][h].x, bv[k][h].y, bv[k][h].z, bv[k][h].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[h][i] = acc[h][i] * a + d[i] * w, bet[h][i] = bet[h][i] * a + e[i] * w;
            }
        }
    }

    // ---- this warp's blocks of window tokens ----------------------------------------------------------------------------
    float mj[G], lr[G];  // joint maximum, sum of the window's terms relative to it
#pragma unroll
    for (int h = 0; h < G; ++h) mj[h] = mc[h], lr[h] = 0.f;
    const float mul = p.scaling * kLog2e;
    for (int base = warp * kBlock; base < tr; base += kMergeWarps * kBlock) {
        if (base != warp * kBlock) {
            if (dot) load_keys(base);
            load_values(base);
        }
        // sc: (token g, heads 2q, 2q + 1), (token g + 8, same heads), log2 domain
        float sc[4] = {0.f, 0.f, 0.f, 0.f};
        if (dot) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                mma_16816(sc, kf[0][k].x, kf[1][k].x, kf[0][k].y, kf[1][k].y, qf[k].x, qf[k].y);
                mma_16816(sc, kf[0][k].z, kf[1][k].z, kf[0][k].w, kf[1][k].w, qf[k].z, qf[k].w);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) sc[e] *= mul;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int h = 2 * q + (e & 1), t = base + g + 8 * (e >> 1);
                if (h < heads && t < tr) sc[e] = p.rscores[static_cast<size_t>(fq0 + h) * tr + t] * kLog2e;
            }
        }
        if (base + g >= tr) sc[0] = sc[1] = -INFINITY;
        if (base + g + 8 >= tr) sc[2] = sc[3] = -INFINITY;
        float mb[2] = {fmaxf(sc[0], sc[2]), fmaxf(sc[1], sc[3])}, lb[2];
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            mb[0] = fmaxf(mb[0], __shfl_xor_sync(0xffffffffu, mb[0], off));
            mb[1] = fmaxf(mb[1], __shfl_xor_sync(0xffffffffu, mb[1], off));
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[e] = rel_exp2(sc[e], mb[e & 1]);
        lb[0] = sc[0] + sc[2], lb[1] = sc[1] + sc[3];
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            lb[0] += __shfl_xor_sync(0xffffffffu, lb[0], off);
            lb[1] += __shfl_xor_sync(0xffffffffu, lb[1], off);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int h = 2 * q + (e & 1);
            if (h < G) prob_s[(g + 8 * (e >> 1)) * G + h] = sc[e];
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();  // probabilities and values of the block in place
        float sum[G][4];
#pragma unroll
        for (int h = 0; h < G; ++h) sum[h][0] = sum[h][1] = sum[h][2] = sum[h][3] = 0.f;
        const int n = min(kBlock, tr - base);
#pragma unroll 4
        for (int t = 0; t < n; ++t) {
            const uint2 v = *reinterpret_cast<const uint2*>(rv_s + t * kHeadDim + 4 * lane);
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
#pragma unroll
            for (int h = 0; h < G; ++h) {
                const float pr = prob_s[t * G + h];
                sum[h][0] = fmaf(pr, a.x, sum[h][0]), sum[h][1] = fmaf(pr, a.y, sum[h][1]);
                sum[h][2] = fmaf(pr, b.x, sum[h][2]), sum[h][3] = fmaf(pr, b.y, sum[h][3]);
            }
        }
        __syncwarp();  // the buffers may be filled with the next block
#pragma unroll
        for (int h = 0; h < G; ++h) {
            const float m = __shfl_sync(0xffffffffu, mb[h & 1], h >> 1), l = __shfl_sync(0xffffffffu, lb[h & 1], h >> 1);
            const float mn = fmaxf(mj[h], m), a = rel_exp2(mj[h], mn), w = rel_exp2(m, mn);
            mj[h] = mn, lr[h] = lr[h] * a + l * w;
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[h][i] = acc[h][i] * a + sum[h][i] * w, bet[h][i] *= a;
        }
    }

    // ---- the results of the warps that had any --------------------------------------------------------------------------
    const int busy = min(kMergeWarps, max(max(used, (tr + kBlock - 1) / kBlock), 1));
    if (warp < busy) {
#pragma unroll
        for (int h = 0; h < G; ++h) {
            float* slot = part_s + (warp * G + h) * kPart;
            *reinterpret_cast<float4*>(slot + 4 * lane) = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
            if (lane < 16) *reinterpret_cast<float4*>(slot + kHeadDim + 4 * lane) = make_float4(bet[h][0], bet[h][1], bet[h][2], bet[h][3]);
            if (lane == 0) *reinterpret_cast<float4*>(stat_s + (warp * G + h) * 4) = make_float4(mj[h], mc[h], lc[h], lr[h]);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int i = tid; i < heads * kMaxClusters; i += kMergeThreads) {
        const int h = i / kMaxClusters, c = i % kMaxClusters;
        float m = -INFINITY, total = 0.f, sum = 0.f;
        for (int k = 0; k < busy; ++k) m = fmaxf(m, stat_s[(k * G + h) * 4]);
#pragma unroll 4
        for (int k = 0; k < busy; ++k) {
            const float4 st = *reinterpret_cast<const float4*>(stat_s + (k * G + h) * 4);
            const float w = rel_exp2(st.x, m);
            total += st.z * rel_exp2(st.y, m) + st.w * w;
            sum += part_s[(k * G + h) * kPart + kHeadDim + c] * w;
            if (c == 0) weight_s[k * G + h] = w;
        }
        beta_s[i] = sum;
        if (c == 0) total_s[h] = fmaxf(total, 1e-20f);
    }
    if ((p.out_m || p.out_l) && tid < heads) {  // statistics of the compressed tokens alone
        float m = -INFINITY, l = 0.f;
        for (int i = 0; i < busy; ++i) m = fmaxf(m, stat_s[(i * G + tid) * 4 + 1]);
        for (int i = 0; i < busy; ++i) l += stat_s[(i * G + tid) * 4 + 2] * rel_exp2(stat_s[(i * G + tid) * 4 + 1], m);
        if (p.out_m) p.out_m[fq0 + tid] = m * kLn2;
        if (p.out_l) p.out_l[fq0 + tid] = l;
    }
    __syncthreads();
    // two coordinates per thread
    for (int i = tid; i < heads * (kHeadDim / 2); i += kMergeThreads) {
        const int h = i / (kHeadDim / 2), d = 2 * (i % (kHeadDim / 2));
        float2 num = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int k = 0; k < busy; ++k) {
            const float2 v = *reinterpret_cast<const float2*>(part_s + (k * G + h) * kPart + d);
            const float w = weight_s[k * G + h];
            num.x += v.x * w, num.y += v.y * w;
        }
#pragma unroll 8
        for (int c = 0; c < cv; ++c) {
            const float2 v = __half22float2(*reinterpret_cast<const __half2*>(vc_s + c * kHeadDim + d));
            num.x = fmaf(beta_s[h * kMaxClusters + c], v.x, num.x), num.y = fmaf(beta_s[h * kMaxClusters + c], v.y, num.y);
        }
        const float total = total_s[h];
        __half* dst = p.out + static_cast<size_t>(fq0 + h) * kHeadDim + d;
        dst[0] = __float2half_rn(num.x / total), dst[1] = __float2half_rn(num.y / total);
    }
}

template <int G>
int launch(const MergeParams& mp, int units, int heads, int recent_max, cudaStream_t s) {
    const int cv = mp.splits > 0 ? mp.cv : 0;
    const size_t smem = merge_smem_bytes<G>(cv);
    if (smem > 48 * 1024) {
        static std::atomic<unsigned long long> done{0};
        if (int rc = allow_smem(decode_merge_kernel<G>, merge_smem_bytes<G>(kMaxClusters), done, "cudaFuncSetAttribute(decode_merge)"))
            return rc;
    }
    // on its own (no partial kernel of this library in front) it starts when what is in front has ended
    return check_cuda(launch_overlapped(decode_merge_kernel<G>, dim3(units, (heads + G - 1) / G), kMergeThreads, smem, s, mp.splits > 0, mp, cv,
                                        recent_max),
                      "decode_merge launch");
}

}  // namespace

int launch_merge(const MergeParams& mp, int units, int recent_max, cudaStream_t s) {
    const int gqa = mp.nh / mp.kh;
    if (gqa < 1 || gqa > 8) return fail(RESKV_ERR_INVALID, "merge: at most 8 query heads per KV head");
    // as few heads per CTA as let all CTAs run at once, two to an SM: batch 12 (96 units of four heads) 86.9, 85.7 and
    // 88.5 us per call with four, two and one, batch 32 229.9, 232.9 and 239.8 us
    const int at_once = 2 * sm_count();
    return gqa == 1 || units * gqa <= at_once   ? launch<1>(mp, units, gqa, recent_max, s)
           : units * ((gqa + 1) / 2) <= at_once ? launch<2>(mp, units, gqa, recent_max, s)
                                                : launch<4>(mp, units, gqa, recent_max, s);
}

}  // namespace reskv
