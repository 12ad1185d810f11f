// Error reporting and device queries shared by every entry point.
#include <cstring>

#include "tensor_map.cuh"

namespace reskv {
namespace {
thread_local char g_error[512] = "";
}

int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
    return code;
}

int check_cuda(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return RESKV_OK;
    return fail(RESKV_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

int check_device_pointer(const void* ptr, const char* who, const char* what) {
    cudaPointerAttributes attr{};
    const cudaError_t e = cudaPointerGetAttributes(&attr, ptr);
    if (e != cudaSuccess) {
        cudaGetLastError();  // the failed query must not poison later calls
        return fail(RESKV_ERR_INVALID, "%s: %s is not memory a CUDA device can be asked about (%s)", who, what,
                    cudaGetErrorString(e));
    }
    if (attr.type == cudaMemoryTypeManaged) return RESKV_OK;
    if (attr.type != cudaMemoryTypeDevice)
        return fail(RESKV_ERR_INVALID, "%s: %s must be device memory, got a host pointer", who, what);
    int dev = -1;
    if (int rc = check_cuda(cudaGetDevice(&dev), "cudaGetDevice")) return rc;
    if (attr.device != dev)
        return fail(RESKV_ERR_INVALID,
                    "%s: %s lives on device %d but device %d is current; make the tensors' device current "
                    "(cudaSetDevice) before the call",
                    who, what, attr.device, dev);
    return RESKV_OK;
}

int sm_count() {
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

namespace {
using TensorMapEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                       const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up once through the runtime (no link against libcuda).
TensorMapEncodeFn tensor_map_encoder() {
    static const TensorMapEncodeFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<TensorMapEncodeFn>(f);
    }();
    return fn;
}
}  // namespace

int encode_tensor_map(CUtensorMap* map, const void* x, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
                      CUtensorMapSwizzle swizzle, const char* who) {
    TensorMapEncodeFn encode = tensor_map_encoder();
    if (!encode) return fail(RESKV_ERR_CUDA, "%s: the driver offers no cuTensorMapEncodeTiled", who);
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    const CUresult made = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, static_cast<cuuint32_t>(rank), const_cast<void*>(x), dims, strides,
                                 box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (made != CUDA_SUCCESS) return fail(RESKV_ERR_CUDA, "%s: cuTensorMapEncodeTiled failed with code %d", who, static_cast<int>(made));
    return RESKV_OK;
}
}  // namespace reskv

extern "C" const char* reskv_last_error(void) { return reskv::g_error; }

extern "C" int reskv_version(void) { return 100; }
