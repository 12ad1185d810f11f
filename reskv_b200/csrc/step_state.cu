// Device-resident decode-step state and the dense-window append that goes with it.
//
// A decode step of a model touches, per layer, the dense window (append the new token) and the
// fused attention (query position, number of window tokens).  When those two numbers live in
// device memory -- step_state = {query position, window tokens} -- the whole step can be captured
// in one CUDA graph and replayed: the append and the decode kernels read them, and one tiny kernel
// advances them at the end of the step.
#include <initializer_list>

#include "common.cuh"

namespace reskv {
namespace {

// grid = units, block = 128 threads: copy the new token's rotated key, raw key and value rows
// into the last counted slot, step_state[1] - 1, of every unit's window (the caller advances the
// window count first, so that the attention of the same step already sees the new token).
__global__ void window_append_kernel(__half* win_k, __half* win_raw, __half* win_v, const __half* k_rot,
                                     const __half* k_raw, const __half* v, int capacity,
                                     const int32_t* __restrict__ step_state) {
    const int unit = blockIdx.x, d = threadIdx.x;
    const int slot = min(max(step_state[1] - 1, 0), capacity - 1);
    const size_t dst = (static_cast<size_t>(unit) * capacity + slot) * kHeadDim + d;
    const size_t src = static_cast<size_t>(unit) * kHeadDim + d;
    win_k[dst] = k_rot[src];
    win_raw[dst] = k_raw[src];
    win_v[dst] = v[src];
}

// Same copy with the slot given by the host (eager callers that track the window length themselves).
__global__ void window_write_kernel(__half* win_k, __half* win_raw, __half* win_v, const __half* k_rot,
                                    const __half* k_raw, const __half* v, int capacity, int slot) {
    const int unit = blockIdx.x, d = threadIdx.x;
    const size_t dst = (static_cast<size_t>(unit) * capacity + slot) * kHeadDim + d;
    const size_t src = static_cast<size_t>(unit) * kHeadDim + d;
    let_next_launch_start();
    wait_for_previous_launch();
    win_k[dst] = k_rot[src];
    win_raw[dst] = k_raw[src];
    win_v[dst] = v[src];
}

// grid (units, 3): tokens [first, first + count) of a prompt's rotated keys, raw keys or values -> slots from `slot` on, in
// 16-byte pieces.  One launch in place of three strided copies: 13.4 -> 4 us behind a prompt of 8 x 8192 tokens.
struct WindowSources {
    const uint4* x[3];
    int64_t stride[3];  // tokens between units
};
__global__ void __launch_bounds__(256) window_fill_kernel(uint4* win_k, uint4* win_raw, uint4* win_v, const WindowSources src, int capacity,
                                                          int slot, int first, int count) {
    constexpr int kPieces = kHeadDim / 8;
    const int unit = blockIdx.x, side = blockIdx.y;
    const uint4* from = src.x[side] + (unit * src.stride[side] + first) * kPieces;
    uint4* to = (side == 0 ? win_k : side == 1 ? win_raw : win_v) + (static_cast<size_t>(unit) * capacity + slot) * kPieces;
#pragma unroll 4
    for (int i = threadIdx.x; i < count * kPieces; i += blockDim.x) to[i] = from[i];
}

__global__ void step_advance_kernel(int32_t* step_state, int pos_inc, int live_inc) {
    let_next_launch_start();
    wait_for_previous_launch();
    if (threadIdx.x == 0) {
        step_state[0] += pos_inc;
        step_state[1] += live_inc;
    }
}

}  // namespace
}  // namespace reskv

using namespace reskv;

extern "C" int reskv_window_append(void* window_k, void* window_raw, void* window_v, const void* k_rot,
                                   const void* k_raw, const void* v, int batch, int kv_heads, int window_capacity,
                                   const int32_t* step_state, void* stream) {
    if (!window_k || !window_raw || !window_v || !k_rot || !k_raw || !v || !step_state)
        return fail(RESKV_ERR_INVALID, "window_append: null pointer");
    if (batch < 1 || kv_heads < 1 || window_capacity < 1)
        return fail(RESKV_ERR_INVALID, "window_append: batch, heads and capacity must be positive");
    window_append_kernel<<<batch * kv_heads, kHeadDim, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<__half*>(window_k), static_cast<__half*>(window_raw), static_cast<__half*>(window_v),
        static_cast<const __half*>(k_rot), static_cast<const __half*>(k_raw), static_cast<const __half*>(v),
        window_capacity, step_state);
    return check_cuda(cudaGetLastError(), "window_append launch");
}

extern "C" int reskv_window_write(void* window_k, void* window_raw, void* window_v, const void* k_rot,
                                  const void* k_raw, const void* v, int batch, int kv_heads, int window_capacity,
                                  int slot, void* stream) {
    if (!window_k || !window_raw || !window_v || !k_rot || !k_raw || !v)
        return fail(RESKV_ERR_INVALID, "window_write: null pointer");
    if (batch < 1 || kv_heads < 1 || window_capacity < 1)
        return fail(RESKV_ERR_INVALID, "window_write: batch, heads and capacity must be positive");
    if (slot < 0 || slot >= window_capacity)
        return fail(RESKV_ERR_INVALID, "window_write: slot %d outside the window of %d tokens", slot, window_capacity);
    if (int rc = check_device_pointer(window_k, "window_write", "window_k")) return rc;
    return reskv_window_put(window_k, window_raw, window_v, k_rot, k_raw, v, batch, kv_heads, window_capacity, slot, stream);
}

extern "C" int reskv_window_put(void* window_k, void* window_raw, void* window_v, const void* k_rot, const void* k_raw,
                                const void* v, int batch, int kv_heads, int window_capacity, int slot, void* stream) {
    if (slot < 0 || slot >= window_capacity)
        return fail(RESKV_ERR_INVALID, "window_put: slot %d outside the window of %d tokens", slot, window_capacity);
    return check_cuda(launch_overlapped(window_write_kernel, dim3(batch * kv_heads), kHeadDim, 0, static_cast<cudaStream_t>(stream), true,
                                        static_cast<__half*>(window_k), static_cast<__half*>(window_raw), static_cast<__half*>(window_v),
                                        static_cast<const __half*>(k_rot), static_cast<const __half*>(k_raw),
                                        static_cast<const __half*>(v), window_capacity, slot),
                      "window_write launch");
}

extern "C" int reskv_window_fill(void* window_k, void* window_raw, void* window_v, const void* k_rot, const void* k_raw, const void* v,
                                 int batch, int kv_heads, int window_capacity, int slot, int64_t k_rot_stride, int64_t k_raw_stride,
                                 int64_t v_stride, int first, int count, void* stream) {
    if (batch < 1 || kv_heads < 1 || window_capacity < 1) return fail(RESKV_ERR_INVALID, "window_fill: batch, heads and capacity must be positive");
    if (slot < 0 || first < 0 || count < 0 || slot + static_cast<int64_t>(count) > window_capacity)
        return fail(RESKV_ERR_INVALID, "window_fill: %d tokens from slot %d on do not fit a window of %d", count, slot, window_capacity);
    const int64_t least = static_cast<int64_t>(first) + count;
    if (k_rot_stride < least || k_raw_stride < least || v_stride < least)
        return fail(RESKV_ERR_INVALID, "window_fill: token stride smaller than the tokens read");
    if (count == 0) return RESKV_OK;
    for (const void* ptr : {static_cast<const void*>(window_k), static_cast<const void*>(window_raw), static_cast<const void*>(window_v), k_rot, k_raw, v}) {
        if (!ptr) return fail(RESKV_ERR_INVALID, "window_fill: null pointer");
        if (!aligned16(ptr)) return fail(RESKV_ERR_INVALID, "window_fill: pointers must be 16-byte aligned");
    }
    if (int rc = check_device_pointer(window_k, "window_fill", "window_k")) return rc;
    const WindowSources src{{static_cast<const uint4*>(k_rot), static_cast<const uint4*>(k_raw), static_cast<const uint4*>(v)},
                            {k_rot_stride, k_raw_stride, v_stride}};
    window_fill_kernel<<<dim3(batch * kv_heads, 3), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<uint4*>(window_k), static_cast<uint4*>(window_raw), static_cast<uint4*>(window_v), src, window_capacity, slot, first, count);
    return check_cuda(cudaGetLastError(), "window_fill launch");
}

extern "C" int reskv_step_advance(int32_t* step_state, int position_increment, int window_increment, void* stream) {
    if (!step_state) return fail(RESKV_ERR_INVALID, "step_advance: null step state");
    return check_cuda(launch_overlapped(step_advance_kernel, dim3(1), 32, 0, static_cast<cudaStream_t>(stream), true, step_state,
                                        position_increment, window_increment),
                      "step_advance launch");
}
