// Host-side helpers shared by the C-ABI translation units: error bookkeeping,
// device checks and TMA tensor-map encoding through the driver entry point
// (the library does not link against libcuda).
#pragma once
#include <cstdint>
#include <cstdio>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/trak_b200.h"

namespace tb {

void set_cuda_error(const char* what, const char* file, int line);

#define TB_CUDA(call)                                                        \
    do {                                                                     \
        cudaError_t e__ = (call);                                            \
        if (e__ != cudaSuccess) {                                            \
            ::tb::set_cuda_error(cudaGetErrorString(e__), __FILE__, __LINE__); \
            return TB_ERR_CUDA;                                              \
        }                                                                    \
    } while (0)

// TB_OK if `device` exists and is compute capability 10.x; sets it current.
int select_device(int device, int* sm_count);

// TB_OK, or the code tb_project returns for these arguments before it looks at workspace or device.
int validate_project_args(const void* grads, int dtype, int64_t B, int64_t F, int64_t ld, const float* out,
                          int64_t ld_out, uint32_t N, uint32_t num_feature_tiles, int proj_type);

// tb_project; with `publish` its last launch stores the status word to pinned host memory (take_note), without it the
// call takes no memory of any kind from the driver.
int project_dense(int device, void* stream, const void* grads, int dtype, int64_t B, int64_t F, int64_t ld, float* out,
                  int64_t ld_out, uint32_t N, uint32_t seed, uint32_t num_feature_tiles, int proj_type, float alpha,
                  int accumulate, void* ws, size_t ws_bytes, bool publish);

// The least workspace that project_dense takes for these (valid) sizes; tb_project_workspace_bytes is what it wants.
size_t project_least_bytes(int64_t B, int64_t F, uint32_t N, uint32_t num_feature_tiles);

// Device address of the status word of `device` (valid after select_device).
uint32_t* status_ptr(int device);

// Encodes a tiled tensor map (rank 2 or 3, zero fill; the box's inner extent must equal the
// swizzle width).
// dims / box are innermost first; strides_bytes has rank-1 entries.
int encode_tmap(CUtensorMap* map, CUtensorMapDataType dt, uint32_t rank, const void* base,
                const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box,
                CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B);

// A word in mapped host memory that a kernel stores the status word to (publish_status).
struct StatusNote {
    uint64_t* word = nullptr;  // null: nothing is stored
    uint32_t call = 0;
};
int take_note(StatusNote* note);
// To be called when the launch that stores `note` has been queued on `stream` as the last of its call: the thread's next
// tb_stream_status on that stream then reads `note`.
void arm_status(int device, cudaStream_t stream, const StatusNote& note);
#ifdef __CUDACC__
__device__ __forceinline__ void publish_status(const uint32_t* status, const StatusNote& note) {
    // one aligned store of eight bytes: the host sees both halves or neither
    if (note.word) *static_cast<volatile uint64_t*>(note.word) = (uint64_t)note.call << 32 | *status;
}
#endif

#ifdef __CUDACC__
// A launch that, where `early`, may begin while the one before it on the stream is still ending: its CTAs take the places
// that become free, set up their barriers and tensor memory (and start generating), and wait
// (cudaGridDependencySynchronize) where they first need what the earlier launch wrote.  A kernel in front of such a
// launch says when it may begin (cudaTriggerProgrammaticLaunchCompletion); behind one that does not, like reduce_kernel, it
// begins at that one's end.  Worth about 1.5 us a launch: a projection 3 to 5 us a call, scoring 1000 x 512 299 -> 270, the
// inverse of 2048 698 -> 640.  The places become free unevenly, and an SM takes as many CTAs as fit: a grid of no more CTAs
// than SMs asks for more than half of an SM's shared memory, or some SMs get two CTAs and others none.
template <typename... Params, typename... Args>
int launch_after(void (*kernel)(Params...), dim3 grid, uint32_t threads, size_t smem, cudaStream_t stream, bool early,
                 Args&&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    TB_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
    return TB_OK;
}

// First statement of a kernel between two such launches (or in front of its first use of global memory): what the earlier
// launch wrote is there, and the next launch may take the places that become free.  Not before: a launch further on would
// hold its shared memory through all of an earlier one that other streams' work should run beside.
__device__ __forceinline__ void after_earlier_launch() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}
#endif

// Lets `kernel` use all of an SM's shared memory on `device` (the current one); once per kernel and device.
constexpr int SMEM_PER_CTA = 227 * 1024;
int set_smem_limit(const void* kernel, int device);

// Events armed by tb_profile_events for this thread (null when not armed); taking clears them.
void take_profile_events(cudaEvent_t* before, cudaEvent_t* after);

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace tb
