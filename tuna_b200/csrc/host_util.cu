// Host-side helpers shared by the pipeline kernels' launchers: the per-device status word that
// bounded waits report into, and TMA tensor-map construction through the driver entry point
// (resolved at run time, so the library does not link against libcuda).
#include <mutex>
#include "common.cuh"
#include "launchers.h"
#include "sm100_ptx.cuh"

namespace tuna {

// File scope and not cudaMalloc: the first call on a device may come while a stream is being captured.
static __device__ __align__(8) DeviceStatus g_device_status;

DeviceStatus *device_status_word()
{
    static DeviceStatus *ptrs[64] = {nullptr};
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!ptrs[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_device_status) != cudaSuccess) return nullptr;
        ptrs[dev] = (DeviceStatus *)p;
    }
    return ptrs[dev];
}

int read_device_status(cudaStream_t stream)
{
    DeviceStatus *d = device_status_word();
    if (!d) return TUNA_ERR_NO_DEVICE;
    DeviceStatus h;
    if (cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, stream) != cudaSuccess) return TUNA_ERR_LAUNCH;
    if (cudaStreamSynchronize(stream) != cudaSuccess) return TUNA_ERR_LAUNCH;
    if (h.code != 0) {
        cudaMemsetAsync(d, 0, sizeof(DeviceStatus), stream);
        return TUNA_ERR_DEVICE_TIMEOUT;
    }
    return TUNA_OK;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)ptr;
    });
    return fn;
}

bool make_tensor_map_2d(CUtensorMap *map, CUtensorMapDataType dt, const void *base, uint64_t inner, uint64_t outer,
                        uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swizzle)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {row_stride_bytes};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, dt, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Three dimensions, innermost first: extents d0, d1, d2; byte strides of d1 and d2 (any order).
bool make_tensor_map_3d(CUtensorMap *map, CUtensorMapDataType dt, const void *base, uint64_t d0, uint64_t d1, uint64_t d2,
                        uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t box0, uint32_t box1, uint32_t box2,
                        CUtensorMapSwizzle swizzle)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {d0, d1, d2};
    cuuint64_t strides[2] = {stride1_bytes, stride2_bytes};
    cuuint32_t box[3] = {box0, box1, box2};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, dt, 3, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Any rank up to 5, innermost dimension first; `strides` are the byte strides of dimensions 1 .. rank-1.
bool make_tensor_map_nd(CUtensorMap *map, CUtensorMapDataType dt, const void *base, int rank, const uint64_t *dims,
                        const uint64_t *strides, const uint32_t *box, CUtensorMapSwizzle swizzle)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn || rank < 1 || rank > 5) return false;
    cuuint64_t d[5], s[4];
    cuuint32_t b[5], e[5];
    for (int i = 0; i < rank; ++i) { d[i] = dims[i]; b[i] = box[i]; e[i] = 1; }
    for (int i = 0; i + 1 < rank; ++i) s[i] = strides[i];
    return fn(map, dt, (cuuint32_t)rank, const_cast<void *>(base), d, s, b, e, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool weight_map_has_runs(int m, int k) { return m % 32 == 0 && k % 64 == 0; }

// Tensor map of the packed weights for stages of `steps` 32-column steps x 128 rows (a row group is 4k bytes = k 32-bit
// words; word index = column index), 128-byte swizzled.
//   *w_mode 1: 32-row blocks x pairs of steps, [m/32][k/64][4 row groups][2 steps][32 words] with strides 16k, 256, 4k
//              and 128 bytes; a stage is one box of 4 x steps/2 x 4 x 2 x 32 words (256-byte runs of global memory);
//   *w_mode 0: where k is a multiple of 32 the 3-D view [k/32 steps][m/8 row groups][32 words] (strides 128 bytes and
//              4k bytes; *q3d = 1), a stage being one box of steps x 16 x 32; otherwise, or if the driver refuses that
//              view, the 2-D view and one box of 16 row groups x 32 words per step.
// A refused 5-D view sets *w_mode to 0.  Rows, columns and steps past the matrix are zero-filled by the copy.
bool make_weight_map(CUtensorMap *map, const void *q, int m, int k, int steps, int *w_mode, int *q3d)
{
    *q3d = 0;
    if (*w_mode == 1) {
        const uint64_t dims[5] = {32, 2, 4, (uint64_t)k / 64, (uint64_t)m / 32};
        const uint64_t strides[4] = {128, (uint64_t)k * 4, 256, (uint64_t)k * 16};
        const uint32_t box[5] = {32, 2, 4, (uint32_t)steps / 2, 4};
        if (weight_map_has_runs(m, k) && make_tensor_map_nd(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, q, 5, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
            return true;
        *w_mode = 0;
    }
    if (k % 32 == 0 && make_tensor_map_3d(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, q, 32, (uint64_t)m / 8, (uint64_t)k / 32, (uint64_t)k * 4, 128, 32, 16,
                                          (uint32_t)steps, CU_TENSOR_MAP_SWIZZLE_128B)) {
        *q3d = 1;
        return true;
    }
    return make_tensor_map_2d(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, q, (uint64_t)k, (uint64_t)m / 8, (uint64_t)k * 4, 32, 16, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace tuna

// ------------------------------------------------------------------ self-test of the bounded waits
//
// Every mbarrier wait of the pipeline kernels gives up after a time limit, records where in the
// device status word and lets the kernel unwind (tuna_check_device_status then reports
// TUNA_ERR_DEVICE_TIMEOUT).  This entry point exercises exactly that path without a real failure:
// one warp waits, with a limit of about a millisecond, on a barrier that nothing ever arrives at.
namespace tuna {
__global__ void bounded_wait_selftest_kernel(DeviceStatus *status, long long limit_cycles)
{
    __shared__ __align__(8) uint64_t bar;
    __shared__ int s_abort;
    if (threadIdx.x == 0) {
        s_abort = 0;
        mbar_init(smem_u32(&bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    // phase 0 of a barrier that expects one arrival and never gets it
    if (!mbar_try_wait(smem_u32(&bar), 0)) mbar_wait_slow(smem_u32(&bar), 0, &s_abort, status, 99, limit_cycles);
}
}  // namespace tuna

extern "C" int tuna_selftest_bounded_wait(void *stream)
{
    tuna::DeviceStatus *d = tuna::device_status_word();
    if (!d) return TUNA_ERR_NO_DEVICE;
    tuna::bounded_wait_selftest_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(d, 2000000ll);  // ~1 ms
    return cudaGetLastError() == cudaSuccess ? TUNA_OK : TUNA_ERR_LAUNCH;
}
