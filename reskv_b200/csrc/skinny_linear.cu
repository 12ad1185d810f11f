// Linear layers of a decode step: y = x . W^T for one to eight rows of x.
//
// What bounds it: the weights, read once (436 MB per layer of a 4096-wide model), so everything is arranged around a stream
// of them that does not stop.  One CTA per SM; its copying warp keeps a ring of stages (16 weight rows x 512 columns, two
// tensor-map boxes of 8 KB; sixteen 1 KB bulk copies per stage reach half the rate) full through all output rows that the
// CTA has, and begins before the kernel in front has ended: the kernels of a step do not write weights, only x is waited
// for.  Eight warps take a stage's columns in eight slices, weights as the A operand of mma.sync (16 output rows x 16
// columns), x as the B operand (eight rows, missing ones zero); the order of a contraction is free, so a lane's fragments
// are 16 contiguous bytes of a row.  The warps' sums meet in shared memory once per 16 output rows.  In the same launch: RMS
// norm of x (every CTA forms it, x comes from L2), the residual added to the result, or SiLU(gate) * up, whose gate and up
// rows lie in one box.
//
// Measured, us per call back to back, 4 rows (cuBLAS, without the norm, SiLU and split sums' kernels): 6144 x 4096 with norm
// 12.2 (15.9), 4096 x 4096 with residual 9.3 (14.5), 2 x 14336 x 4096 with norm and SiLU 38.1 (39.0), 4096 x 14336 with
// residual 21.5 (26.3), 32000 x 4096 with norm 42.6 (47.2); one row 11.0, 12.0, 37.2, 19.3, 41.3, i.e. up to 6.35 TB/s.  A
// captured step runs faster than their sum, because a layer's weights arrive while the attention kernels in front run: prompt
// of 4 x 1024 tokens and 72 steps on two layers 26.6 -> 23.7 ms.
#include "tensor_map.cuh"

namespace reskv {
namespace {

constexpr int kLinRows = 16;                      // weight rows of a stage
constexpr int kLinCols = 512;                     // and columns
constexpr int kLinBox = 256;                      // columns of one copy (a tensor map's most)
constexpr int kLinBoxBytes = kLinRows * kLinBox * 2;
constexpr int kLinStage = kLinCols / kLinBox * kLinBoxBytes;
constexpr int kLinWarps = 8;                      // consumers
constexpr int kLinThreads = (kLinWarps + 1) * 32;
constexpr int kLinBatch = 8;                      // most rows of x
constexpr int kLinSmem = 216 * 1024;              // dynamic shared memory of a CTA

enum LinearMode { kLinPlain = 0, kLinAdd = 1, kLinSiluMul = 2, kLinFloat = 3 };

__device__ uint32_t g_linear_status;  // RESKV_STATUS_* bits: a bounded wait that ran out

struct LinearParams {
    const __half* x;       // [rows, k]
    const __half* norm;    // [k] weights of an RMS norm of x, or null
    void* out;             // [rows, n] FP16, kLinFloat: FP32; kLinAdd: also the residual
    float eps;
    int rows, n, k, mode, stages;
};

__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kLinWarps * 32) : "memory"); }

__global__ void __launch_bounds__(kLinThreads, 1) skinny_linear_kernel(const LinearParams p, const __grid_constant__ CUtensorMap map) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t bar_full[16], bar_empty[16], bar_x;
    __shared__ float red[2][kLinWarps][kLinRows * kLinBatch], squares[kLinWarps][kLinBatch];
    unsigned char* xs = smem + p.stages * kLinStage;  // [rows][x_pitch bytes]
    const int x_pitch = 2 * p.k + 64;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool pairs = p.mode == kLinSiluMul;
    const int per_unit = pairs ? kLinRows / 2 : kLinRows, units = p.n / per_unit, steps = p.k / kLinCols;
    if (tid == 0) {
        for (int s = 0; s < p.stages; ++s) mbar_init(&bar_full[s], 1), mbar_init(&bar_empty[s], kLinWarps);
        mbar_init(&bar_x, 1);
        mbar_fence_init();
    }
    let_next_launch_start();
    __syncthreads();
    bool lost = false;

    if (warp == kLinWarps) {
        // ---- copies ---------------------------------------------------------------------------------------------------
        int slot = 0, round = 0;
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            for (int s = 0; s < steps; ++s) {
                // the ring is full: nothing is given back before the kernel in front has ended, and however long that takes is
                // no part of the bounded wait
                if (round == 1 && slot == 0) wait_for_previous_launch();
                if (round > 0) lost |= !mbar_wait(&bar_empty[slot], (round - 1) & 1);
                if (lane == 0) {
                    mbar_arrive_expect_tx(&bar_full[slot], kLinStage);
#pragma unroll
                    for (int i = 0; i < kLinCols / kLinBox; ++i)
                        tma_load_3d(smem + slot * kLinStage + i * kLinBoxBytes, &map, s * kLinCols + i * kLinBox, u * per_unit, 0, &bar_full[slot]);
                }
                __syncwarp();
                if (++slot == p.stages) slot = 0, ++round;
            }
        }
    } else {
        // ---- x into shared memory, normalised if wanted ----------------------------------------------------------------
        wait_for_previous_launch();
        if (!p.norm) {  // as it is: a copy per row
            if (tid == 0) {
                mbar_arrive_expect_tx(&bar_x, p.rows * p.k * 2);
                for (int b = 0; b < p.rows; ++b) bulk_g2s(xs + b * x_pitch, p.x + static_cast<size_t>(b) * p.k, p.k * 2, &bar_x);
            }
            lost |= !mbar_wait(&bar_x, 0);
        } else {
            const int pieces = p.k / 8;  // 16 bytes each; a thread requests its piece of all rows together
            float sq[kLinBatch];
#pragma unroll
            for (int b = 0; b < kLinBatch; ++b) sq[b] = 0.f;
            for (int i = tid; i < pieces; i += kLinWarps * 32) {
                uint4 v[kLinBatch];
#pragma unroll
                for (int b = 0; b < kLinBatch; ++b)
                    if (b < p.rows) v[b] = reinterpret_cast<const uint4*>(p.x + static_cast<size_t>(b) * p.k)[i];
#pragma unroll
                for (int b = 0; b < kLinBatch; ++b) {
                    if (b >= p.rows) break;
                    *reinterpret_cast<uint4*>(xs + b * x_pitch + 16 * i) = v[b];
                    const __half2* h = reinterpret_cast<const __half2*>(&v[b]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __half22float2(h[e]);
                        sq[b] = fmaf(f.x, f.x, sq[b]), sq[b] = fmaf(f.y, f.y, sq[b]);
                    }
                }
            }
#pragma unroll
            for (int b = 0; b < kLinBatch; ++b) {
                if (b < p.rows) {
#pragma unroll
                    for (int off = 16; off > 0; off >>= 1) sq[b] += __shfl_xor_sync(0xffffffffu, sq[b], off);
                    if (lane == 0) squares[warp][b] = sq[b];
                }
            }
            uint4 weights = reinterpret_cast<const uint4*>(p.norm)[tid < pieces ? tid : 0];
            consumers_sync();
            float inv[kLinBatch];
#pragma unroll
            for (int b = 0; b < kLinBatch; ++b) {
                float total = 0.f;
#pragma unroll
                for (int w = 0; w < kLinWarps; ++w) total += b < p.rows ? squares[w][b] : 0.f;
                inv[b] = rsqrtf(total / static_cast<float>(p.k) + p.eps);
            }
            for (int i = tid; i < pieces; i += kLinWarps * 32) {  // the pieces that this thread has stored
                const uint4 now = weights;
                if (i + kLinWarps * 32 < pieces) weights = reinterpret_cast<const uint4*>(p.norm)[i + kLinWarps * 32];
                const __half2* gh = reinterpret_cast<const __half2*>(&now);
#pragma unroll
                for (int b = 0; b < kLinBatch; ++b) {
                    if (b >= p.rows) break;
                    uint4* at = reinterpret_cast<uint4*>(xs + b * x_pitch + 16 * i);
                    const uint4 v = *at;
                    const __half2* h = reinterpret_cast<const __half2*>(&v);
                    uint4 o;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __half22float2(h[e]), gw = __half22float2(gh[e]);
                        reinterpret_cast<__half2*>(&o)[e] = __floats2half2_rn(f.x * inv[b] * gw.x, f.y * inv[b] * gw.y);
                    }
                    *at = o;
                }
            }
            consumers_sync();
        }

        // ---- the product: warp w takes the columns [64 w, 64 w + 64) of every stage ------------------------------------
        const int g = lane >> 2, q = lane & 3;
        const bool has_row = g < p.rows;
        const unsigned char* x_lane = xs + (has_row ? g : 0) * x_pitch + 128 * warp + 16 * q;
        const uint32_t keep = has_row ? 0xffffffffu : 0u;
        int slot = 0, round = 0, turn = 0;
        for (int u = blockIdx.x; u < units; u += gridDim.x, turn ^= 1) {
            float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
            for (int s = 0; s < steps; ++s) {
                uint4 b[2], lo[2], hi[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    b[j] = *reinterpret_cast<const uint4*>(x_lane + s * (kLinCols * 2) + 64 * j);
                    b[j].x &= keep, b[j].y &= keep, b[j].z &= keep, b[j].w &= keep;
                }
                lost |= !mbar_wait(&bar_full[slot], round & 1);
                const unsigned char* at = smem + slot * kLinStage + (warp >> 2) * kLinBoxBytes + g * (kLinBox * 2) + 128 * (warp & 3) + 16 * q;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    lo[j] = *reinterpret_cast<const uint4*>(at + 64 * j);
                    hi[j] = *reinterpret_cast<const uint4*>(at + 8 * (kLinBox * 2) + 64 * j);
                }
                mma_16816(c0, lo[0].x, hi[0].x, lo[0].y, hi[0].y, b[0].x, b[0].y);
                mma_16816(c1, lo[0].z, hi[0].z, lo[0].w, hi[0].w, b[0].z, b[0].w);
                mma_16816(c0, lo[1].x, hi[1].x, lo[1].y, hi[1].y, b[1].x, b[1].y);
                mma_16816(c1, lo[1].z, hi[1].z, lo[1].w, hi[1].w, b[1].z, b[1].w);
                __syncwarp();
                if (lane == 0) mbar_arrive(&bar_empty[slot]);
                if (++slot == p.stages) slot = 0, ++round;
            }
            // sums of the eight slices: [row of the unit][row of x]; the buffer of the unit before is still being read
            float* mine = red[turn][warp];
            *reinterpret_cast<float2*>(mine + g * kLinBatch + 2 * q) = make_float2(c0[0] + c1[0], c0[1] + c1[1]);
            *reinterpret_cast<float2*>(mine + (g + 8) * kLinBatch + 2 * q) = make_float2(c0[2] + c1[2], c0[3] + c1[3]);
            consumers_sync();
            const int r = tid % kLinRows, bx = tid / kLinRows;  // output row of the unit, row of x
            if (bx < p.rows && bx < kLinBatch) {
                const auto total = [&](int row) {
                    float t = 0.f;
#pragma unroll
                    for (int w = 0; w < kLinWarps; ++w) t += red[turn][w][row * kLinBatch + bx];
                    return t;
                };
                if (pairs) {
                    if (r < per_unit) {  // the projections are rounded to FP16 first, as separate tensors would be
                        const float gate = __half2float(__float2half_rn(total(r))), up = __half2float(__float2half_rn(total(r + per_unit)));
                        const float act = __half2float(__float2half_rn(gate / (1.f + expf(-gate))));
                        static_cast<__half*>(p.out)[static_cast<size_t>(bx) * p.n + u * per_unit + r] = __float2half_rn(act * up);
                    }
                } else {
                    const size_t at = static_cast<size_t>(bx) * p.n + u * per_unit + r;
                    const float t = total(r);
                    if (p.mode == kLinFloat) {
                        static_cast<float*>(p.out)[at] = __half2float(__float2half_rn(t));
                    } else {
                        __half* out = static_cast<__half*>(p.out);
                        out[at] = __float2half_rn(p.mode == kLinAdd ? __half2float(out[at]) + t : t);
                    }
                }
            }
        }
    }
    if (lost) atomicOr(&g_linear_status, RESKV_STATUS_WAIT_TIMEOUT);
}

// Taken: up to eight rows, the columns of one MMA (at eight rows still 12.3 and 38.9 us for the two with a norm, cuBLAS 12.7
// and 39.1 without), as long as the rows of x leave room for four stages: with fewer the stream waits for the copies'
// latency.  14336 columns leave 11, 9, 8, 6 and 4 stages for one to five rows and are not taken for six to eight.
// stages of the ring beside `rows` rows of x (0: they do not fit)
int linear_stages(int rows, int k) {
    const int s = (kLinSmem - rows * (2 * k + 64)) / kLinStage;
    return s < 4 ? 0 : s > 12 ? 12 : s;
}
bool linear_fits(int rows, int n, int k, int mode) {
    if (rows < 1 || rows > kLinBatch || n < 1 || k < kLinCols || k % kLinCols || mode < kLinPlain || mode > kLinFloat) return false;
    return n % (mode == kLinSiluMul ? kLinRows / 2 : kLinRows) == 0 && linear_stages(rows, k) > 0;
}
}  // namespace
}  // namespace reskv

using namespace reskv;

extern "C" int reskv_skinny_linear_fits(int rows, int n, int k, int mode) { return linear_fits(rows, n, k, mode) ? 1 : 0; }

extern "C" int reskv_skinny_linear(const void* x, const void* norm_weight, float eps, const void* weight, void* out, int rows, int n,
                                   int k, int mode, void* stream) {
    if (!x || !weight || !out) return fail(RESKV_ERR_INVALID, "skinny_linear: null pointer");
    if (!linear_fits(rows, n, k, mode))
        return fail(RESKV_ERR_LIMIT, "skinny_linear: %d rows, %d x %d weights, mode %d are not taken", rows, n, k, mode);
    for (const void* ptr : {x, norm_weight, weight, static_cast<const void*>(out)})
        if (reinterpret_cast<uintptr_t>(ptr) & 15u) return fail(RESKV_ERR_INVALID, "skinny_linear: pointers must be 16-byte aligned");
    LinearParams p{};
    p.x = static_cast<const __half*>(x), p.norm = static_cast<const __half*>(norm_weight);
    p.out = out, p.eps = eps, p.rows = rows, p.n = n, p.k = k, p.mode = mode, p.stages = linear_stages(rows, k);
    // weights as (column, row, gate or up): a unit's rows in one box
    const bool two = mode == kLinSiluMul;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(n), two ? 2u : 1u};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(k) * 2, static_cast<cuuint64_t>(n) * k * 2};
    const cuuint32_t box[3] = {kLinBox, static_cast<cuuint32_t>(two ? kLinRows / 2 : kLinRows), two ? 2u : 1u};
    CUtensorMap map;
    if (int rc = encode_tensor_map(&map, weight, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE, "skinny_linear")) return rc;
    static std::atomic<unsigned long long> done{0};
    if (int rc = allow_smem(skinny_linear_kernel, kLinSmem, done, "cudaFuncSetAttribute(skinny_linear)")) return rc;
    const int units = n / (two ? kLinRows / 2 : kLinRows);
    const size_t smem = static_cast<size_t>(p.stages) * kLinStage + static_cast<size_t>(rows) * (2 * k + 64);
    return check_cuda(launch_overlapped(skinny_linear_kernel, dim3(static_cast<unsigned>(units < sm_count() ? units : sm_count())), kLinThreads,
                                        smem, static_cast<cudaStream_t>(stream), true, p, map), "skinny_linear launch");
}

extern "C" int reskv_skinny_linear_status(uint32_t* status, void* stream) {
    if (!status) return fail(RESKV_ERR_INVALID, "skinny_linear_status: null destination");
    if (int rc = check_cuda(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "skinny_linear_status synchronize")) return rc;
    return check_cuda(cudaMemcpyFromSymbol(status, g_linear_status, sizeof(uint32_t)), "skinny_linear_status copy");
}
