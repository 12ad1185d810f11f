// Residual packers, one THREAD per token: the layouts that keep the globally largest residuals of a token
// (unstructured FP16 bitmap; unstructured and compact INT4 / INT2), the layouts that keep the largest of every
// 16-coordinate tile (tiled masks, 4:16 indices) and the 1-of-4 INT4 layout.
//
// With a whole token in one thread nothing crosses lanes (a warp per token spends most of its instructions on warp
// reductions, votes and popcounts):
//
//   * a warp stages the rows of 32 consecutive tokens in shared memory with 16-byte asynchronous copies
//     (rows 16 bytes apart from dense, so the 16-byte loads of eight lanes fall into distinct banks), the
//     unit's centroid table is staged once per CTA; warps meet only when the table changes;
//   * fp16(r) of two neighbouring coordinates is one packed subtraction: rounding x - c once to FP16 equals rounding it to
//     FP32 first (24 >= 2 * 11 + 2 bits).  The 128 selection keys |fp16(r)| stay in registers as 64 packed pairs;
//   * the k-th largest key is found by bisection on its 15 bits: a round is 64 packed comparisons (1.0 / 0.0
//     per half, integer pipe) summed by packed FP16 additions (floating-point pipe), two instructions per key
//     pair and round on two different pipes;
//   * ties at the threshold keep the lower coordinates; the kept FP16 residuals are compacted in place in
//     the thread's own row (one predicated store per coordinate: a loop over the set bits waits for shared memory
//     at every step) and the warp writes the 32 rows out with 16-byte stores.
//
// The tiled layouts take their thresholds from a sorting network, two tiles at a time in the two halves of the packed
// operations, and look for NaNs beside it (1 % of the time); the 1-of-4 layout compares four keys per group.
//
// What bounds it: the integer pipe, then the time a warp waits for its rows.  Microseconds per side of 64 units x 8128
// tokens (133 MB of x), and what the same layouts took with FP32 keys, a bisection of both halves apart and a compaction
// loop: bitmap 87 for 32 and 90 for 64 of 128 values (112, 126), INT4 110 (128), INT2 110 (126), tiled 67 (91), 4:16 52
// (73), 1-of-4 INT4 48 (79), compact INT4 127 to 138 (320).
//
// Rounding points are those of compress.cu (they decide bit-exactness): selection key |fp16(r)|, FP16 layouts
// store fp16(r), the quantisers divide the FP32 r with the approximate division of the reference's build.
#include <cuda_fp16.h>

#include "compress_common.cuh"

namespace reskv {
namespace {

constexpr int kTopkWarps = 4;                 // warps per CTA
constexpr int kTopkThreads = kTopkWarps * 32;
constexpr int kRowBytes = 2 * kHeadDim + 16;  // shared-memory row of one token / one centroid
constexpr int kChunkTokens = kTopkThreads;    // tokens a CTA takes per pass (32 per warp)

enum class TopkMode { kBitmapFp16, kQuant4, kQuant2, kCompact4, kCompact2, kTiledFp16, kStructFp16, kStructInt4 };

__device__ __forceinline__ float half_lo(uint32_t v) {
    return __half2float(__ushort_as_half(static_cast<unsigned short>(v & 0xffffu)));
}
__device__ __forceinline__ float half_hi(uint32_t v) {
    return __half2float(__ushort_as_half(static_cast<unsigned short>(v >> 16)));
}
__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t*>(&v); }

// a - fp32(b): one mixed-precision multiply-add (b * -1 + a), rounded once like the subtraction
__device__ __forceinline__ float sub_f16(float a, unsigned short b) {
    float d;
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d) : "h"(b), "h"(static_cast<unsigned short>(0xbc00)), "f"(a));
    return d;
}

// r[q] = fp32(x[32 p + q]) - fp32(c[32 p + q]), q = 0..31, from the token's and its centroid's shared-memory rows
__device__ __forceinline__ void residual_piece(const unsigned char* xrow, const unsigned char* crow, int p,
                                               float (&r)[32]) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const uint4 xv = *reinterpret_cast<const uint4*>(xrow + 64 * p + 16 * m);
        const uint4 cv = *reinterpret_cast<const uint4*>(crow + 64 * p + 16 * m);
        const uint32_t xs[4] = {xv.x, xv.y, xv.z, xv.w}, cs[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            r[8 * m + 2 * i] = sub_f16(half_lo(xs[i]), static_cast<unsigned short>(cs[i] & 0xffffu));
            r[8 * m + 2 * i + 1] = sub_f16(half_hi(xs[i]), static_cast<unsigned short>(cs[i] >> 16));
        }
    }
}

// Even coordinates' bits (high half) and odd ones' (low half) interleaved: bit i of the halves -> bits 2 i + 1 and 2 i.
__device__ __forceinline__ uint32_t interleave16(uint32_t x) {
    uint32_t t = (x ^ (x >> 8)) & 0x0000ff00u;
    x ^= t ^ (t << 8);
    t = (x ^ (x >> 4)) & 0x00f000f0u;
    x ^= t ^ (t << 4);
    t = (x ^ (x >> 2)) & 0x0c0c0c0cu;
    x ^= t ^ (t << 2);
    t = (x ^ (x >> 1)) & 0x22222222u;
    return x ^ t ^ (t << 1);
}

// Keep-mask of the `k` largest keys, lower coordinate first among equal keys.  key[16 p + j] holds coordinate
// 32 p + 2 j in its low and 32 p + 2 j + 1 in its high half; keep[p] has coordinate 32 p + q at bit 31 - q.  True when
// nothing is above the threshold and not everything at it is kept (the largest key itself is cut).
__device__ __forceinline__ bool select_topk_thread(const uint32_t (&key)[64], int k, uint32_t (&keep)[4]) {
    // largest v with count(key >= v) >= k
    uint32_t v = 0;
#pragma unroll 1
    for (int bit = 14; bit >= 0; --bit) {
        const uint32_t cand = v | (1u << bit);
        const __half2 c2 = as_half2(cand | (cand << 16));
        // the comparisons (1.0 / 0.0 per half) issue on the integer pipe, their sums on the FP16 pipe; counts up
        // to 128 are exact in FP16; four accumulators keep the addition chains short
        __half2 acc[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] = __hge2(as_half2(key[u]), c2);
#pragma unroll
        for (int j = 4; j < 64; ++j) acc[j & 3] = __hadd2(acc[j & 3], __hge2(as_half2(key[j]), c2));
        const __half2 total = __hadd2(__hadd2(acc[0], acc[1]), __hadd2(acc[2], acc[3]));
        const int cnt = __half2int_rn(__hadd(__low2half(total), __high2half(total)));
        if (cnt >= k) v = cand;
    }
    const __half2 v2 = as_half2(v | (v << 16));
    uint32_t ge[4] = {0u, 0u, 0u, 0u};
    int kept = 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
#pragma unroll
        for (int j = 0; j < 16; ++j) ge[p] |= __hge2_mask(as_half2(key[16 * p + j]), v2) & ((0x80000000u >> j) | (0x8000u >> j));
        kept += __popc(ge[p]);
        keep[p] = interleave16(__byte_perm(ge[p], 0u, 0x1032));  // even coordinates to the high half
    }
    if (kept == k) return false;
    // more keys equal to the threshold than places left: the lowest coordinates among them stay
    int need = k;
    uint32_t gt[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int p = 0; p < 4; ++p) {
#pragma unroll
        for (int j = 0; j < 16; ++j) gt[p] |= __hgt2_mask(as_half2(key[16 * p + j]), v2) & ((0x80000000u >> j) | (0x8000u >> j));
        need -= __popc(gt[p]);
        gt[p] = interleave16(__byte_perm(gt[p], 0u, 0x1032));
    }
    const bool cut_largest = need == k;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        uint32_t eq = keep[p] ^ gt[p], stay = gt[p];
        while (eq != 0u && need > 0) {
            const uint32_t first = 0x80000000u >> __clz(eq);
            eq ^= first, stay |= first, --need;
        }
        keep[p] = stay;
    }
    return cut_largest;
}

// Packed 16-bit keys: larger ones to `a`, smaller ones to `b`, in either half.
__device__ __forceinline__ void order2(uint32_t& a, uint32_t& b) {
    const uint32_t hi = __vmaxu2(a, b);
    b = __vminu2(a, b);
    a = hi;
}
__device__ __forceinline__ void sort4(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {  // descending
    order2(a, b), order2(c, d), order2(a, c), order2(b, d), order2(b, c);
}
// The four largest of two descending quadruples, descending, in `a`.
__device__ __forceinline__ void top4(uint32_t (&a)[4], const uint32_t (&b)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = __vmaxu2(a[i], b[3 - i]);
    order2(a[0], a[2]), order2(a[1], a[3]), order2(a[0], a[1]), order2(a[2], a[3]);
}
// M-th largest of 16 keys (M = 4 or 8), in either half: sorted runs, then the smallest of the pairwise maxima of one run
// and the other one reversed.  Bit patterns are ordered: a NaN key comes out above every number, and `largest` turns NaN then
// (one FP16 operation on the largest keys of both halves; infinity times zero does so too, which costs time only).
template <int M>
__device__ __forceinline__ uint32_t mth_of_16(const uint32_t* key, __half2& largest) {
    uint32_t a[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) a[i][j] = key[4 * i + j];
        sort4(a[i][0], a[i][1], a[i][2], a[i][3]);
    }
    if constexpr (M == 4) {
        top4(a[0], a[1]), top4(a[2], a[3]);
        largest = __hfma2(as_half2(a[0][0]), as_half2(a[2][0]), largest);
        uint32_t t = __vmaxu2(a[0][0], a[2][3]);
#pragma unroll
        for (int i = 1; i < 4; ++i) t = __vminu2(t, __vmaxu2(a[0][i], a[2][3 - i]));
        return t;
    } else {
        uint32_t run[2][8];  // two bitonic merges of a descending and a reversed descending quadruple
#pragma unroll
        for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int i = 0; i < 4; ++i) run[r][i] = a[2 * r][i], run[r][4 + i] = a[2 * r + 1][3 - i];
#pragma unroll
            for (int step = 4; step > 0; step >>= 1)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (!(i & step)) order2(run[r][i], run[r][i + step]);
        }
        largest = __hfma2(as_half2(run[0][0]), as_half2(run[1][0]), largest);
        uint32_t t = __vmaxu2(run[0][0], run[1][7]);
#pragma unroll
        for (int i = 1; i < 8; ++i) t = __vminu2(t, __vmaxu2(run[0][i], run[1][7 - i]));
        return t;
    }
}

// Per half, of 16 packed keys: the largest v with count(key >= v) >= m, 0 when there are fewer than m numbers.
__device__ __forceinline__ uint32_t mth_by_bisection(const uint32_t* key, int m) {
    const __half2 m2 = __float2half2_rn(static_cast<float>(m));
    uint32_t v2 = 0;
#pragma unroll 1
    for (int bit = 14; bit >= 0; --bit) {
        const uint32_t both = (1u << bit) | (1u << (bit + 16));
        const __half2 c2 = as_half2(v2 | both);
        __half2 a0 = __hge2(as_half2(key[0]), c2), a1 = __hge2(as_half2(key[1]), c2);
#pragma unroll
        for (int j = 2; j < 16; j += 2) {
            a0 = __hadd2(a0, __hge2(as_half2(key[j]), c2));
            a1 = __hadd2(a1, __hge2(as_half2(key[j + 1]), c2));
        }
        v2 |= both & __hge2_mask(__hadd2(a0, a1), m2);  // each half accepts the bit on its own count (exact in FP16)
    }
    return v2;
}

// Keys of two tiles from fp16(r) of their 32 coordinates (two a word): coordinate j of the first tile in the low, of the
// second one in the high half.
__device__ __forceinline__ void tile_keys(const uint32_t (&r2)[16], uint32_t* key) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        key[2 * j] = __byte_perm(r2[j], r2[8 + j], 0x5410) & 0x7fff7fffu;
        key[2 * j + 1] = __byte_perm(r2[j], r2[8 + j], 0x7632) & 0x7fff7fffu;
    }
}

// Keep-mask of the `m` largest keys of every 16-coordinate tile, lower coordinate first among equal keys; NaN keys come
// behind all numbers, so a tile always keeps exactly m.
// key[16 p + j] holds coordinate 32 p + j (tile 2 p) in its LOW and 32 p + 16 + j (tile 2 p + 1) in its HIGH half;
// keep[p] has coordinate 32 p + q at bit q (the tiled metadata word of the reference, compression.cu:126-139).
// M of the two plans that have this layout: thresholds from a sorting network (71 and 95 packed instructions per pair of
// tiles), false when the token has a NaN key and `keep` is not to be used; M = 0, any m: bisection (480).
template <int M>
__device__ __forceinline__ bool select_tiles_thread(const uint32_t (&key)[64], int m, uint32_t (&keep)[4]) {
    __half2 largest = __float2half2_rn(0.f);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const uint32_t* k16 = key + 16 * p;
        uint32_t v2;  // per half: the m-th largest key
        if constexpr (M != 0) v2 = mth_of_16<M>(k16, largest); else v2 = mth_by_bisection(k16, m);
        uint32_t ge = 0u;
#pragma unroll
        for (int j = 0; j < 16; ++j) ge |= __hge2_mask(as_half2(k16[j]), as_half2(v2)) & ((1u << j) | (0x10000u << j));
        uint32_t kept = ge;
        // in all, as each tile has at least m unless there are NaNs
        if (M != 0 ? __popc(ge) != 2 * m : __popc(ge & 0xffffu) != m || __popc(ge >> 16) != m) {
            uint32_t gt = 0u;
#pragma unroll
            for (int j = 0; j < 16; ++j) gt |= __hgt2_mask(as_half2(k16[j]), as_half2(v2)) & ((1u << j) | (0x10000u << j));
            kept = gt;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t half = 0xffffu << (16 * h);
                int need = m - __popc(gt & half);
                // more keys equal to the threshold than places left: the lowest coordinates stay; fewer than m numbers:
                // the lowest of the NaNs as well
#pragma unroll
                for (int fill = 0; fill < (M != 0 ? 1 : 2); ++fill) {
                    uint32_t from = (fill ? ~ge : ge ^ gt) & half;
                    while (from != 0u && need > 0) {
                        const uint32_t first = from & (0u - from);
                        from ^= first, kept |= first, --need;
                    }
                }
            }
        }
        keep[p] = kept;
    }
    return M == 0 || !(__hisnan(__low2half(largest)) || __hisnan(__high2half(largest)));
}

// Code of residual r: the quotient by the FP16 scale s, rounded and clamped.  A scale that underflowed to 0 gives what the
// reference's (int)lrintf(r / 0) gives: -1 for positive residuals, 0 otherwise (see lrint_low32); every other quotient of
// a kept residual is small, so the 32-bit conversion equals the 64-bit one.
template <int QMAX>
__device__ __forceinline__ int code_of(float r, float s, bool no_scale) {
    const int q = max(-QMAX, min(QMAX, __float2int_rn(div_fast(r, s))));
    return no_scale ? (r > 0.f ? -1 : 0) : q;
}

template <TopkMode MODE>
__global__ void __launch_bounds__(kTopkThreads, 5) encode_topk_kernel(const EncodeParams p) {
    extern __shared__ __align__(16) unsigned char topk_smem[];
    constexpr bool kTiles = MODE == TopkMode::kTiledFp16 || MODE == TopkMode::kStructFp16;
    constexpr bool kFp16Rows = MODE == TopkMode::kBitmapFp16 || kTiles;  // the row becomes the FP16 payload
    constexpr bool kCompact = MODE == TopkMode::kCompact4 || MODE == TopkMode::kCompact2;
    unsigned char* cen_s = topk_smem;                                                 // [clusters][kRowBytes]
    unsigned char* rows_s = topk_smem + static_cast<size_t>(p.clusters) * kRowBytes;  // [warps][32][kRowBytes]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char* my_rows = rows_s + static_cast<size_t>(warp) * 32 * kRowBytes;
    unsigned char* xrow = my_rows + lane * kRowBytes;
    const int chunks_per_unit = (p.tokens + kChunkTokens - 1) / kChunkTokens;
    const long long chunks = static_cast<long long>(p.units) * chunks_per_unit;
    int staged_unit = -1;
    for (long long c = blockIdx.x; c < chunks; c += gridDim.x) {
        const int unit = static_cast<int>(c / chunks_per_unit);
        const int t0 = static_cast<int>(c % chunks_per_unit) * kChunkTokens + warp * 32;
        const int ntok = max(0, min(32, p.tokens - t0));
        const bool new_table = unit != staged_unit;  // uniform over the CTA
        if (new_table) {
            __syncthreads();  // nobody still reads the previous table
            const unsigned char* src = reinterpret_cast<const unsigned char*>(p.cen + static_cast<size_t>(unit) * p.clusters * kHeadDim);
            for (int i = tid; i < p.clusters * 16; i += kTopkThreads) cp_async16(cen_s + (i >> 4) * kRowBytes + (i & 15) * 16, src + i * 16);
            staged_unit = unit;
        }
        int id = 0;
        if (lane < ntok) id = min(max(p.ids[static_cast<size_t>(unit) * p.tokens + t0 + lane], 0), p.clusters - 1);
        {
            const unsigned char* src = reinterpret_cast<const unsigned char*>(p.x + (static_cast<size_t>(unit) * p.x_stride + t0) * kHeadDim);
            for (int i = lane; i < ntok * 16; i += 32) cp_async16(my_rows + (i >> 4) * kRowBytes + (i & 15) * 16, src + i * 16);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (new_table) __syncthreads(); else __syncwarp();  // table and this warp's rows in place

        const size_t orow = static_cast<size_t>(unit) * p.out_stride + t0 + lane;
        const unsigned char* crow = cen_s + id * kRowBytes;
        // fp16(r) of coordinates 8 m .. 8 m + 7, two per word
        auto residual8 = [&](int m) {
            const uint4 xv = *reinterpret_cast<const uint4*>(xrow + 16 * m), cv = *reinterpret_cast<const uint4*>(crow + 16 * m);
            return make_uint4(as_u32(__hsub2(as_half2(xv.x), as_half2(cv.x))), as_u32(__hsub2(as_half2(xv.y), as_half2(cv.y))),
                              as_u32(__hsub2(as_half2(xv.z), as_half2(cv.z))), as_u32(__hsub2(as_half2(xv.w), as_half2(cv.w))));
        };
        if constexpr (MODE == TopkMode::kStructInt4) {
            // one residual of every four consecutive coordinates: the largest |fp16(r)|, lowest index on ties;
            // FP32 scale amax / 7, codes with the approximate division (compression.cu:153-239)
            if (lane < ntok) {
                const __half *xh = reinterpret_cast<const __half*>(xrow), *ch = reinterpret_cast<const __half*>(crow);
                uint32_t which[2] = {0u, 0u};  // 2-bit in-group index of group g at bit 2 (g % 16) of word g / 16
                float best[32], amax = 0.f;
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    const uint4 v = residual8(m);
                    const uint32_t r2[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        // key and reversed index in one number: equal keys leave the lowest index on top
                        const uint32_t lo = r2[2 * h] & 0x7fff7fffu, hi = r2[2 * h + 1] & 0x7fff7fffu;
                        const uint32_t k0 = (lo & 0xffffu) * 4u + 3u, k1 = (lo >> 16) * 4u + 2u, k2 = (hi & 0xffffu) * 4u + 1u, k3 = (hi >> 16) * 4u;
                        const int g = 2 * m + h, e = static_cast<int>(~max(max(k0, k1), max(k2, k3)) & 3u);
                        which[g >> 4] |= static_cast<uint32_t>(e) << (2 * (g & 15));
                        best[g] = __half2float(xh[4 * g + e]) - __half2float(ch[4 * g + e]);
                        amax = fmaxf(amax, fabsf(best[g]));
                    }
                }
                const float s = amax > 0.f ? amax * (1.0f / 7.0f) : 1.0f;
                uint32_t out[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int g = 0; g < 32; ++g) {
                    const int q = max(-7, min(7, __float2int_rn(div_fast(best[g], s))));
                    out[g >> 3] |= (static_cast<uint32_t>(q) & 15u) << (4 * (g & 7));
                }
                static_cast<uint4*>(p.payload)[orow] = make_uint4(out[0], out[1], out[2], out[3]);
                static_cast<uint2*>(p.meta)[orow] = make_uint2(which[0], which[1]);
                p.scale[orow] = __float2half_rn(s);
            }
        } else if (lane < ntok) {
            uint32_t keep[4], key[64];
            bool cut_largest = false;
#pragma unroll
            for (int pc = 0; pc < 4; ++pc) {
                uint32_t r2[16];  // fp16(r) of coordinates 32 pc + 2 j (low half), + 1
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const uint4 v = residual8(4 * pc + m);
                    r2[4 * m] = v.x, r2[4 * m + 1] = v.y, r2[4 * m + 2] = v.z, r2[4 * m + 3] = v.w;
                    if constexpr (kFp16Rows) *reinterpret_cast<uint4*>(xrow + 64 * pc + 16 * m) = v;  // replaces the consumed x
                }
                if constexpr (kTiles) {
                    tile_keys(r2, key + 16 * pc);
                } else {
#pragma unroll
                    for (int j = 0; j < 16; ++j) key[16 * pc + j] = r2[j] & 0x7fff7fffu;
                }
            }
            if constexpr (kTiles) {
                const int m = p.nnz / 8;
                bool done = false;
                if (MODE == TopkMode::kStructFp16)
                    done = select_tiles_thread<4>(key, 4, keep);
                else if (m == 8)
                    done = select_tiles_thread<8>(key, 8, keep);
                if (!done) {
                    // another count, or NaNs; the keys once more from the row, so that they are not held until here
#pragma unroll
                    for (int pc = 0; pc < 4; ++pc) {
                        uint32_t r2[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) r2[j] = reinterpret_cast<const uint32_t*>(xrow)[16 * pc + j];
                        tile_keys(r2, key + 16 * pc);
                    }
                    select_tiles_thread<0>(key, m, keep);
                }
            } else {
                cut_largest = select_topk_thread(key, p.nnz, keep);
            }

            uint32_t code[4] = {0u, 0u, 0u, 0u};  // 4:16 form: four 4-bit in-tile indices per tile, rank r at bit 4 r
            const bool whole_tiles = MODE == TopkMode::kStructFp16 || (MODE == TopkMode::kTiledFp16 && p.nnz == 64);
            if (kTiles && whole_tiles) {
                // a fixed number per tile: the kept values are fetched by index and packed in registers, two tiles at a time
                constexpr int kPerTile = MODE == TopkMode::kStructFp16 ? 4 : 8;
#pragma unroll
                for (int pc = 0; pc < 4; ++pc) {
                    uint32_t left[2] = {keep[pc] & 0xffffu, keep[pc] >> 16}, out[kPerTile];
#pragma unroll
                    for (int r = 0; r < kPerTile; ++r) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int q = __ffs(left[h]) - 1;
                            left[h] &= left[h] - 1u;
                            const uint32_t v = *reinterpret_cast<const unsigned short*>(xrow + 64 * pc + 32 * h + 2 * q);
                            uint32_t& w = out[h * (kPerTile / 2) + (r >> 1)];
                            w = r & 1 ? __byte_perm(w, v, 0x5410) : v;
                            if constexpr (MODE == TopkMode::kStructFp16) code[pc] |= static_cast<uint32_t>(q) << (4 * r + 16 * h);
                        }
                    }
#pragma unroll
                    for (int w = 0; w < kPerTile; w += 4)  // behind the read position throughout
                        *reinterpret_cast<uint4*>(xrow + 4 * kPerTile * pc + 4 * w) = make_uint4(out[w], out[w + 1], out[w + 2], out[w + 3]);
                }
            } else if constexpr (kFp16Rows && MODE != TopkMode::kStructFp16) {
                // kept values to the front of the row, ascending coordinates (write position <= read position throughout)
                uint32_t to = smem_u32(xrow);
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    const uint4 v = *reinterpret_cast<const uint4*>(xrow + 16 * m);
                    const uint32_t r2[4] = {v.x, v.y, v.z, v.w}, w = keep[m >> 2];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int q = 8 * (m & 3) + i;
                        const bool kept = kTiles ? (w >> q) & 1u : w & (0x80000000u >> q);
                        if (kept) {
                            asm volatile("st.shared.u16 [%0], %1;" ::"r"(to), "h"(static_cast<unsigned short>(i & 1 ? r2[i >> 1] >> 16 : r2[i >> 1])) : "memory");
                            to += 2;
                        }
                    }
                }
            }
            if constexpr (MODE == TopkMode::kBitmapFp16) {
                // bitmap words: coordinate d at bit 63 - d % 64 of word d / 64
                static_cast<uint4*>(p.meta)[orow] = make_uint4(keep[1], keep[0], keep[3], keep[2]);
            } else if constexpr (MODE == TopkMode::kTiledFp16) {
                static_cast<uint4*>(p.meta)[orow] = make_uint4(keep[0], keep[1], keep[2], keep[3]);
            } else if constexpr (MODE == TopkMode::kStructFp16) {
                static_cast<uint4*>(p.meta)[orow] = make_uint4(code[0], code[1], code[2], code[3]);
            } else {
                constexpr int kBits = MODE == TopkMode::kQuant4 || MODE == TopkMode::kCompact4 ? 4 : 2;
                constexpr int kQmax = (1 << (kBits - 1)) - 1;
                constexpr int kPer = 32 / kBits;  // codes per word
                // Two more passes over the residuals (largest kept magnitude, then the codes); the pieces are
                // taken one at a time (no unrolling over pc) so that only 32 residuals are live at once.  The largest
                // magnitude of all is a kept one unless the largest keys themselves were cut.
                float amax = 0.f;
#pragma unroll 1
                for (int pc = 0; pc < 4; ++pc) {
                    float r[32];
                    residual_piece(xrow, crow, pc, r);
                    if (cut_largest) {
                        const uint32_t kw = pc == 0 ? keep[0] : pc == 1 ? keep[1] : pc == 2 ? keep[2] : keep[3];
#pragma unroll
                        for (int q = 0; q < 32; ++q)
                            if (kw & (0x80000000u >> q)) amax = fmaxf(amax, fabsf(r[q]));
                    } else {
#pragma unroll
                        for (int q = 0; q < 32; ++q) amax = fmaxf(amax, fabsf(r[q]));
                    }
                }
                const __half hs = quant_scale<kQmax>(amax);
                const float s = __half2float(hs);
                const bool no_scale = s == 0.f;
                uint32_t* words = reinterpret_cast<uint32_t*>(p.payload) + orow * (kCompact ? p.nnz / kPer : 4 * kBits);
                uint32_t to = smem_u32(xrow);
#pragma unroll 1
                for (int pc = 0; pc < 4; ++pc) {
                    const uint32_t kw = pc == 0 ? keep[0] : pc == 1 ? keep[1] : pc == 2 ? keep[2] : keep[3];
                    float r[32];
                    residual_piece(xrow, crow, pc, r);
                    if constexpr (kCompact) {
                        // one byte per kept code to the front of the row (behind the read position throughout)
#pragma unroll
                        for (int q = 0; q < 32; ++q) {
                            if (kw & (0x80000000u >> q)) {
                                asm volatile("st.shared.u8 [%0], %1;" ::"r"(to), "r"(code_of<kQmax>(r[q], s, no_scale)) : "memory");
                                ++to;
                            }
                        }
                    } else {
                        uint32_t out[32 / kPer];
#pragma unroll
                        for (int w = 0; w < 32 / kPer; ++w) {
                            uint32_t word = 0u;
#pragma unroll
                            for (int i = 0; i < kPer; ++i) {
                                const int q = w * kPer + i;
                                const int code = code_of<kQmax>(r[q], s, no_scale);
                                if (kw & (0x80000000u >> q)) word |= (static_cast<uint32_t>(code) & ((1u << kBits) - 1u)) << (i * kBits);
                            }
                            out[w] = word;
                        }
                        // coordinates 32 pc .. 32 pc + 31 = words (32 / kPer) pc ...
                        if constexpr (kBits == 4) {
                            *reinterpret_cast<uint4*>(words + 4 * pc) = make_uint4(out[0], out[1], out[2], out[3]);
                        } else {
                            *reinterpret_cast<uint2*>(words + 2 * pc) = make_uint2(out[0], out[1]);
                        }
                    }
                }
                if constexpr (kCompact) {
                    // the bytes' low bits side by side, 16 bytes of codes at a time
                    for (int w4 = 0; w4 < p.nnz / (4 * kPer); ++w4) {
                        uint32_t out[4];
#pragma unroll
                        for (int w = 0; w < 4; ++w) {
                            uint32_t word = 0u;
#pragma unroll
                            for (int i = 0; i < kPer / 4; ++i) {
                                uint32_t four = *reinterpret_cast<const uint32_t*>(xrow + (4 * w4 + w) * kPer + 4 * i);
                                if constexpr (kBits == 4) {
                                    four &= 0x0f0f0f0fu;
                                    four |= four >> 4;
                                    word |= __byte_perm(four, 0u, 0x4420) << (16 * i);
                                } else {
                                    four &= 0x03030303u;
                                    four |= four >> 6;
                                    word |= ((four & 15u) | ((four >> 12) & 0xf0u)) << (8 * i);
                                }
                            }
                            out[w] = word;
                        }
                        reinterpret_cast<uint4*>(words)[w4] = make_uint4(out[0], out[1], out[2], out[3]);
                    }
                    static_cast<uint4*>(p.meta)[orow] = make_uint4(keep[1], keep[0], keep[3], keep[2]);
                }
                p.scale[orow] = hs;
            }
        }
        __syncwarp();
        if constexpr (kFp16Rows) {
            // the warp's rows are consecutive in the output: 16-byte pieces when the row length allows it
            unsigned char* dst = reinterpret_cast<unsigned char*>(static_cast<__half*>(p.payload) +
                                                                  (static_cast<size_t>(unit) * p.out_stride + t0) * p.nnz);
            if (p.nnz == 32 || p.nnz == 64) {
                const int shift = p.nnz == 32 ? 2 : 3, mask = (1 << shift) - 1;
                for (int i = lane; i < ntok << shift; i += 32)
                    reinterpret_cast<uint4*>(dst)[i] = *reinterpret_cast<const uint4*>(my_rows + (i >> shift) * kRowBytes + (i & mask) * 16);
            } else {
                for (int i = lane; i < ntok * p.nnz; i += 32) {
                    const int row = i / p.nnz, e = i % p.nnz;
                    reinterpret_cast<unsigned short*>(dst)[i] =
                        *reinterpret_cast<const unsigned short*>(my_rows + row * kRowBytes + e * 2);
                }
            }
            __syncwarp();  // rows are rewritten by the next pass
        }
    }
}

size_t topk_smem_bytes(int clusters) {
    return static_cast<size_t>(clusters + kTopkWarps * 32) * kRowBytes;
}

template <TopkMode MODE>
int launch_topk(const EncodeParams& p, cudaStream_t stream, const char* what) {
    auto kern = encode_topk_kernel<MODE>;
    static std::atomic<unsigned long long> done{0};
    // for the largest centroid table
    if (int rc = allow_smem(kern, topk_smem_bytes(kMaxClusters), done, what)) return rc;
    const long long chunks = static_cast<long long>(p.units) * ((p.tokens + kChunkTokens - 1) / kChunkTokens);
    const long long cap = static_cast<long long>(sm_count()) * 5;
    const int grid = static_cast<int>(chunks < cap ? chunks : cap);
    kern<<<grid, kTopkThreads, topk_smem_bytes(p.clusters), stream>>>(p);
    return check_cuda(cudaGetLastError(), what);
}

}  // namespace

int launch_topk_bitmap_fp16(const EncodeParams& p, cudaStream_t stream) {
    return launch_topk<TopkMode::kBitmapFp16>(p, stream, "encode_bitmap_fp16 launch");
}

int launch_topk_tiled_fp16(const EncodeParams& p, bool indexed, cudaStream_t stream) {
    return indexed ? launch_topk<TopkMode::kStructFp16>(p, stream, "encode_tiled_fp16 launch")
                   : launch_topk<TopkMode::kTiledFp16>(p, stream, "encode_tiled_fp16 launch");
}

int launch_topk_structured_int4(const EncodeParams& p, cudaStream_t stream) {
    return launch_topk<TopkMode::kStructInt4>(p, stream, "encode_structured_int4 launch");
}

int launch_topk_compact(const EncodeParams& p, int bits, cudaStream_t stream) {
    return bits == 4 ? launch_topk<TopkMode::kCompact4>(p, stream, "encode_compact launch")
                     : launch_topk<TopkMode::kCompact2>(p, stream, "encode_compact launch");
}

int launch_topk_quantized(const EncodeParams& p, int bits, cudaStream_t stream) {
    return bits == 4 ? launch_topk<TopkMode::kQuant4>(p, stream, "encode_quantized launch")
                     : launch_topk<TopkMode::kQuant2>(p, stream, "encode_quantized launch");
}

}  // namespace reskv
