// Host-side helpers shared by the .cu files of the library: error reporting, the device status word that kernels write
// when a bounded wait gives up, the tensor-map encoder (looked up from the driver at run time, so the library does not
// link libcuda), and the launch counter that the benchmark reports.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace es {

// Records `msg` as the last error of this thread and returns `code` (negative).
int set_error(int code, const char* msg);
// Address of this device's status word (0 = fine; otherwise the code of the first wait that gave up).
int* device_status_ptr();
// One more kernel launched by this library (read with es_launch_count).
void count_launch();

// Lets `kernel` use `bytes` of dynamic shared memory on the current device (once per device and kernel). 0 or an error code.
int opt_in_shared_memory(const void* kernel, int bytes);

// Asks that an SM runs `kernel` (which uses little shared memory) with the largest shared-memory share, as the attention kernels
// do: an SM changes its share only when it is empty, so kernels that agree on it may follow one another without draining it.
int prefer_shared_memory(const void* kernel);

// Whether every pointer is a multiple of `bytes` (null ones pass): a vector access to anything else faults.
template <typename... P> inline bool aligned(uintptr_t bytes, P... p) { return (((uintptr_t)p | ... | (uintptr_t)0) & (bytes - 1)) == 0; }

int encode_tensor_map(CUtensorMap* m, CUtensorMapDataType dt, uint32_t rank, void* base, const cuuint64_t* dims,
                      const cuuint64_t* strides_bytes, const cuuint32_t* box, const cuuint32_t* elem_strides,
                      CUtensorMapSwizzle swizzle);

#define ES_CHECK_LAUNCH(name)                                                     \
    do {                                                                          \
        cudaError_t e__ = cudaGetLastError();                                     \
        if (e__ != cudaSuccess) return es::set_error(-2, cudaGetErrorString(e__)); \
        es::count_launch();                                                       \
    } while (0)

// Launches a kernel that may begin before the previous one on the stream has ended: it must call wait_prerequisites() before it
// reads what that one wrote or writes what that one reads.
template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace es
