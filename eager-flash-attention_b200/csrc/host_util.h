// Host-side helpers shared by the translation units of the library: per-thread error string,
// CUDA error capture, driver entry points fetched at run time (the library does not link libcuda,
// so it can be loaded and its symbols inspected on a machine without a driver).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdarg>
#include <cstdio>

namespace efa {

void set_error(const char* fmt, ...) __attribute__((format(printf, 1, 2)));
const char* last_error();

// Returns 0 when `e` is cudaSuccess; otherwise records "<what>: <cuda error string>" and returns 1.
int check_cuda(cudaError_t e, const char* what, const char* file, int line);
int check_cu(CUresult r, const char* what, const char* file, int line);

#define EFA_CUDA(call) do { if (::efa::check_cuda((call), #call, __FILE__, __LINE__)) return 1; } while (0)
#define EFA_CU(call)   do { if (::efa::check_cu((call), #call, __FILE__, __LINE__)) return 1; } while (0)

// Driver API entry points (resolved through cudaGetDriverEntryPoint on first use).
struct DriverApi {
    CUresult (*cuTensorMapEncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                       const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                       const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    CUresult (*cuStreamBatchMemOp)(CUstream, unsigned int, CUstreamBatchMemOpParams*, unsigned int);
    CUresult (*cuStreamWriteValue32)(CUstream, CUdeviceptr, cuuint32_t, unsigned int);
    CUresult (*cuGetErrorString)(CUresult, const char**);
    CUresult (*cuMemGetAddressRange)(CUdeviceptr*, size_t*, CUdeviceptr);
    // virtual memory management and NVLink multicast objects (nvls_reduce.cu)
    CUresult (*cuCtxGetDevice)(CUdevice*);
    CUresult (*cuDeviceGetAttribute)(int*, CUdevice_attribute, CUdevice);
    CUresult (*cuMemGetAllocationGranularity)(size_t*, const CUmemAllocationProp*, CUmemAllocationGranularity_flags);
    CUresult (*cuMemCreate)(CUmemGenericAllocationHandle*, size_t, const CUmemAllocationProp*, unsigned long long);
    CUresult (*cuMemRelease)(CUmemGenericAllocationHandle);
    CUresult (*cuMemAddressReserve)(CUdeviceptr*, size_t, size_t, CUdeviceptr, unsigned long long);
    CUresult (*cuMemAddressFree)(CUdeviceptr, size_t);
    CUresult (*cuMemMap)(CUdeviceptr, size_t, size_t, CUmemGenericAllocationHandle, unsigned long long);
    CUresult (*cuMemUnmap)(CUdeviceptr, size_t);
    CUresult (*cuMemSetAccess)(CUdeviceptr, size_t, const CUmemAccessDesc*, size_t);
    CUresult (*cuMemExportToShareableHandle)(void*, CUmemGenericAllocationHandle, CUmemAllocationHandleType, unsigned long long);
    CUresult (*cuMemImportFromShareableHandle)(CUmemGenericAllocationHandle*, void*, CUmemAllocationHandleType);
    CUresult (*cuMulticastCreate)(CUmemGenericAllocationHandle*, const CUmulticastObjectProp*);
    CUresult (*cuMulticastAddDevice)(CUmemGenericAllocationHandle, CUdevice);
    CUresult (*cuMulticastBindMem)(CUmemGenericAllocationHandle, size_t, CUmemGenericAllocationHandle, size_t, size_t, unsigned long long);
    CUresult (*cuMulticastUnbind)(CUmemGenericAllocationHandle, CUdevice, size_t, size_t);
    CUresult (*cuMulticastGetGranularity)(size_t*, const CUmulticastObjectProp*, CUmulticastGranularity_flags);
};
// nullptr (with the error recorded) when the driver is not available.
const DriverApi* driver_api();

// Device-side status word (int[4]) of the current device, allocated on first use.
int* kernel_status_word();

// A device int for one launch (work distribution of persistent kernels): slots of a small per-device
// ring handed out round-robin; the caller clears its slot on the launch stream.
int* work_counter_slot();

// Number of SMs of the current device (148, a B200, where there is none: plans are also made on machines without a GPU).
int device_sms();

// Whether p is memory of the current device itself: not mapped host memory, managed memory or another GPU's.
bool own_device_memory(const void* p);

#ifdef __CUDACC__
// A launch whose blocks may start while the kernel before it in the stream still runs, as soon as all blocks of that one have
// said so or ended: its set-up (barriers, tensor memory, descriptors) and the launch itself then cost nothing. For kernels
// that wait (pdl_wait) before they touch memory, and that read it with ordinary loads or TMA only: what the kernel before it
// writes is not read-only for as long as such a kernel is on the GPU, so no __ldg, no ld.global.nc and no __restrict__ parameter, which
// lets the compiler choose them and move them ahead of the wait. Call after call: projection 4160 x 512 x 4096 24.6 -> 23.2 us, attention of
// 4032 rows, eight heads of 32, 61.5 -> 59.5 us, of 16384 rows, four heads of 64 in four splits with the merge 266 -> 262 us. A call of several
// kernels gains by itself (on an idle GPU with a cold L2: the same attention with its merge 272 -> 269 us, a block of 1024 rows with four
// projections 77 -> 55); a single kernel on an idle GPU has nothing ahead of it to start under and pays 0.2 to 0.3 us of host time for the
// attribute and as much for the wait (projection 2496 x 576 x 512 16.4 -> 17.0 us from call to completion, 4160 x 512 x 4096 29.9 -> 30.4).
// cluster > 1: the blocks along the grid's third dimension, all of them, are a cluster.
// early = false: an ordinary launch, behind all that is ahead of it in the stream.
template <class... P, class... A>
cudaError_t launch_kernel(bool early, int cluster, void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, const A&... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = (unsigned)cluster;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
    if (e != cudaSuccess) (void)cudaGetLastError();        // reported here: not once more by whoever asks next
    return e;
}
template <class... P, class... A>
cudaError_t launch_early_cluster(int cluster, void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, const A&... args)
{
    return launch_kernel(true, cluster, kernel, grid, threads, smem, stream, args...);
}
template <class... P, class... A>
cudaError_t launch_early(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, const A&... args)
{
    return launch_early_cluster(1, kernel, grid, threads, smem, stream, args...);
}
#endif

// fp16 tensor map over a row-major tensor viewed as up to 3 dimensions (dim 0 fastest).
// `box` rows x `box_cols` columns, swizzle chosen from box_cols * 2 bytes (32, 64 or 128).
int make_tmap_f16(CUtensorMap* out, const void* base, int rank,
                  const unsigned long long* dims, const unsigned long long* strides_bytes /* rank-1 */,
                  const unsigned* box);
// The same over fp32 data.
int make_tmap_f32(CUtensorMap* out, const void* base, int rank, const unsigned long long* dims,
                  const unsigned long long* strides_bytes, const unsigned* box);

}  // namespace efa
