// Library-wide pieces of the C ABI: version, error text, device selection,
// the per-device status word and tensor-map encoding.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "host_util.h"
#include "ptx.cuh"

namespace tb {

// Written by kernels when a bounded wait runs out (record_status).
__device__ __align__(8) uint32_t g_status[STATUS_LEN];

static thread_local char t_cuda_error[512] = "";

void set_cuda_error(const char* what, const char* file, int line) {
    snprintf(t_cuda_error, sizeof(t_cuda_error), "%s (%s:%d)", what, file, line);
}

static thread_local cudaEvent_t t_ev_before = nullptr, t_ev_after = nullptr;

void take_profile_events(cudaEvent_t* before, cudaEvent_t* after) {
    *before = t_ev_before;
    *after = t_ev_after;
    t_ev_before = t_ev_after = nullptr;
}

static std::mutex g_mu;
static constexpr int MAX_DEV = 64;
static int g_dev_state[MAX_DEV];  // 0 unknown, 1 ok, -1 unsupported
static int g_dev_sms[MAX_DEV];
static uint32_t* g_dev_status_ptr[MAX_DEV];

// The last launch of a call may publish the status word itself (arm_status); then a status read by the same thread on
// the same stream, with no other call in between, only has to wait.
static thread_local struct {
    int device = -1;
    cudaStream_t stream = nullptr;
    StatusNote note;
} t_armed;

int select_device(int device, int* sm_count) {
    t_armed.device = -1;
    if (device < 0 || device >= MAX_DEV) return TB_ERR_BAD_ARG;
    TB_CUDA(cudaSetDevice(device));
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_dev_state[device] == 0) {
        cudaDeviceProp prop;
        TB_CUDA(cudaGetDeviceProperties(&prop, device));
        g_dev_sms[device] = prop.multiProcessorCount;
        if (prop.major != 10) {
            g_dev_state[device] = -1;
        } else {
            void* p = nullptr;
            TB_CUDA(cudaGetSymbolAddress(&p, g_status));
            g_dev_status_ptr[device] = static_cast<uint32_t*>(p);
            TB_CUDA(cudaMemset(p, 0, sizeof(uint32_t) * STATUS_LEN));
            g_dev_state[device] = 1;
        }
    }
    if (g_dev_state[device] < 0) return TB_ERR_UNSUPPORTED;
    if (sm_count) *sm_count = g_dev_sms[device];
    return TB_OK;
}

uint32_t* status_ptr(int device) { return g_dev_status_ptr[device]; }

// One CTA waits, with the kernels' own bounded wait, on an mbarrier that nothing will ever arrive
// at; when the limit runs out it records the failure exactly as the pipelines do and returns.
__global__ void selftest_wait_kernel(uint32_t* status, uint64_t limit_ns) {
    __shared__ uint64_t bar;
    __shared__ uint32_t abort_word;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        abort_word = 0;
        fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        volatile uint32_t* abort_flag = &abort_word;
        if (!mbar_wait(smem_u32(&bar), 0u, abort_flag, limit_ns)) {
            if (record_status(status, (uint32_t)ST_TIMEOUT_EMPTY)) {
                status[1] = 0xFFFFFFFFu;  // marks the self-test
                status[2] = 0;
            }
        }
    }
    __syncthreads();
}

// Where kernels store the status word for the host: one ring of pinned words per process, made on first use and never
// given up, handed out in turn.  A word carries the number of the call it was handed out for beside the status, so it
// needs no owner: when it has been handed out again and a kernel of either call stores to it late (a thread that ended
// without waiting, the replay of a captured call), the reader sees a number that is not its own and asks the device.
constexpr uint32_t STATUS_WORDS = 1024;
static std::mutex g_words_mu;
static uint64_t* g_words = nullptr;
static std::atomic<uint32_t> g_calls{0};

int take_note(StatusNote* note) {
    uint64_t* words;
    {
        std::lock_guard<std::mutex> lk(g_words_mu);
        if (!g_words) {
            // a capture of any thread forbids allocations that are not told to be relaxed
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            TB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
            void* p = nullptr;
            const cudaError_t e = cudaHostAlloc(&p, STATUS_WORDS * sizeof(uint64_t), cudaHostAllocPortable | cudaHostAllocMapped);
            TB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
            TB_CUDA(e);
            memset(p, 0, STATUS_WORDS * sizeof(uint64_t));
            g_words = static_cast<uint64_t*>(p);
        }
        words = g_words;
    }
    do note->call = g_calls.fetch_add(1, std::memory_order_relaxed) + 1u;
    while (note->call == 0);  // 0 is what a word holds that nothing has been stored to
    note->word = words + note->call % STATUS_WORDS;
    return TB_OK;
}
// After the kernel that stores it has ended: false where a later call has the word by now, or may have (reads that need no word
// take a number as well, so that an answer does not outlast a round of calls and reads).
static bool read_note(const StatusNote& note, uint32_t* status) {
    const uint64_t v = *static_cast<volatile uint64_t*>(note.word);
    *status = (uint32_t)v;
    return (uint32_t)(v >> 32) == note.call && g_calls.load(std::memory_order_relaxed) - note.call < STATUS_WORDS;
}

// A word of mapped host memory per device that a kernel stores the code to beside the device's own (record_status), so that a
// status read behind work that publishes nothing has only to wait for it: the kernel that stored the word to the host behind
// every such call took 4 us of the caller's time and 3 of the device's, three times in a chain of 270 (scoring 1000 x 512).
// Made by the first read on a device and never given up.
static std::mutex g_mirror_mu;
static std::atomic<uint32_t*> g_mirror[MAX_DEV];
static int status_mirror(int device, uint32_t** word) {
    if ((*word = g_mirror[device].load(std::memory_order_acquire))) return TB_OK;
    std::lock_guard<std::mutex> lk(g_mirror_mu);
    if ((*word = g_mirror[device].load(std::memory_order_acquire))) return TB_OK;
    // a capture of any thread forbids what is not told to be relaxed, and its stream may not be waited for: a stream apart
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    TB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    uint32_t* p = nullptr;
    cudaStream_t apart = nullptr;
    cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&p), 2 * sizeof(uint32_t), cudaHostAllocPortable | cudaHostAllocMapped);
    if (e == cudaSuccess) {
        p[0] = p[1] = 0;
        e = cudaStreamCreateWithFlags(&apart, cudaStreamNonBlocking);
    }
    // from here on kernels repeat what they record; then what had been recorded before
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(g_dev_status_ptr[device] + STATUS_MIRROR, &p, sizeof(p), cudaMemcpyHostToDevice, apart);
    if (e == cudaSuccess) e = cudaMemcpyAsync(p + 1, g_dev_status_ptr[device], sizeof(uint32_t), cudaMemcpyDeviceToHost, apart);
    if (e == cudaSuccess) e = cudaStreamSynchronize(apart);
    if (apart) cudaStreamDestroy(apart);
    TB_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
    TB_CUDA(e);
    volatile uint32_t* v = p;
    if (v[1] != 0) v[0] = v[1];
    g_mirror[device].store(*word = p, std::memory_order_release);
    return TB_OK;
}

void arm_status(int device, cudaStream_t stream, const StatusNote& note) {
    t_armed.device = device;
    t_armed.stream = stream;
    t_armed.note = note;
}

int set_smem_limit(const void* kernel, int device) {
    static std::mutex mu;
    static std::vector<std::pair<const void*, uint64_t>> done;  // devices on which the kernel's limit has been raised
    std::lock_guard<std::mutex> lk(mu);
    auto it = std::find_if(done.begin(), done.end(), [&](const auto& d) { return d.first == kernel; });
    if (it != done.end() && (it->second >> device & 1u)) return TB_OK;
    cudaFuncAttributes attr;
    TB_CUDA(cudaFuncGetAttributes(&attr, kernel));
    TB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(SMEM_PER_CTA - attr.sharedSizeBytes)));
    if (it == done.end()) it = done.insert(done.end(), {kernel, 0});
    it->second |= 1ull << device;
    return TB_OK;
}

typedef CUresult (*encode_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);
static encode_fn g_encode = nullptr;

int encode_tmap(CUtensorMap* map, CUtensorMapDataType dt, uint32_t rank, const void* base,
                const uint64_t* dims, const uint64_t* strides_bytes, const uint32_t* box,
                CUtensorMapSwizzle swizzle) {
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_encode) {
            void* fn = nullptr;
            cudaDriverEntryPointQueryResult qres;
            TB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
            if (!fn || qres != cudaDriverEntryPointSuccess) {
                set_cuda_error("cuTensorMapEncodeTiled not available", __FILE__, __LINE__);
                return TB_ERR_CUDA;
            }
            g_encode = reinterpret_cast<encode_fn>(fn);
        }
    }
    cuuint64_t gdim[5];
    cuuint64_t gstr[5];
    cuuint32_t bdim[5], estr[5];
    for (uint32_t i = 0; i < rank; ++i) {
        gdim[i] = dims[i];
        bdim[i] = box[i];
        estr[i] = 1;
        if (i + 1 < rank) gstr[i] = strides_bytes[i];
    }
    CUresult r = g_encode(map, dt, rank, const_cast<void*>(base), gdim, gstr, bdim, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        char msg[96];
        snprintf(msg, sizeof(msg), "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        set_cuda_error(msg, __FILE__, __LINE__);
        return TB_ERR_CUDA;
    }
    return TB_OK;
}

}  // namespace tb

extern "C" {

int tb_version(void) { return 100; }

const char* tb_strerror(int code) {
    switch (code) {
    case TB_OK: return "ok";
    case TB_ERR_BAD_DTYPE: return "unsupported dtype (expected fp16, bf16 or fp32)";
    case TB_ERR_BAD_SHAPE: return "invalid shape or leading dimension";
    case TB_ERR_BAD_PROJ_DIM: return "Invalid Number of JL dimensions it has to be a multiple of 512";
    case TB_ERR_BAD_ARG: return "invalid argument";
    case TB_ERR_WORKSPACE: return "workspace missing, misaligned or too small";
    case TB_ERR_CUDA: return "CUDA error";
    case TB_ERR_DEVICE_TIMEOUT: return "a bounded wait inside a kernel ran out";
    case TB_ERR_UNSUPPORTED: return "unsupported device or size";
    case TB_ERR_NOT_SPD: return "matrix is not positive definite (non-positive Cholesky pivot)";
    case TB_ERR_SCRATCH_LIMIT:
        return "shape needs more scratch than tb_project_static's built-in array; use tb_project with a workspace";
    default: return "unknown error code";
    }
}

const char* tb_last_cuda_error(void) { return tb::t_cuda_error; }

int tb_profile_events(void* before, void* after) {
    tb::t_ev_before = static_cast<cudaEvent_t>(before);
    tb::t_ev_after = static_cast<cudaEvent_t>(after);
    return TB_OK;
}

int tb_selftest_wait_timeout(int device, void* stream, uint32_t limit_ms) {
    if (limit_ms == 0 || limit_ms > 2000) return TB_ERR_BAD_ARG;
    int rc = tb::select_device(device, nullptr);
    if (rc != TB_OK) return rc;
    tb::selftest_wait_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(tb::status_ptr(device),
                                                                              (uint64_t)limit_ms * 1000000ull);
    TB_CUDA(cudaGetLastError());
    return TB_OK;
}

int tb_device_status(int device, uint32_t* detail) {
    int rc = tb::select_device(device, nullptr);
    if (rc != TB_OK) return rc;
    uint32_t host[tb::STATUS_MIRROR] = {};
    TB_CUDA(cudaDeviceSynchronize());
    // first the host's word: a kernel of another thread that records something from here on sets both
    if (uint32_t* mirror = tb::g_mirror[device].load(std::memory_order_acquire)) *static_cast<volatile uint32_t*>(mirror) = 0;
    TB_CUDA(cudaMemcpy(host, tb::status_ptr(device), sizeof(host), cudaMemcpyDeviceToHost));
    if (detail) *detail = host[0];
    if (host[0] != 0) {
        TB_CUDA(cudaMemset(tb::status_ptr(device), 0, sizeof(host)));
        return host[0] == 6u ? TB_ERR_NOT_SPD : TB_ERR_DEVICE_TIMEOUT;
    }
    return TB_OK;
}

int tb_stream_status(int device, void* stream_, uint32_t* detail) {
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    const bool armed = tb::t_armed.device == device && tb::t_armed.stream == stream;
    int rc = tb::select_device(device, nullptr);
    if (rc != TB_OK) return rc;
    const tb::StatusNote note = tb::t_armed.note;
    uint32_t code = 0, *mirror = nullptr;
    if (!armed) {
        if ((rc = tb::status_mirror(device, &mirror)) != TB_OK) return rc;
        tb::g_calls.fetch_add(1, std::memory_order_relaxed);
    }
    TB_CUDA(cudaStreamSynchronize(stream));
    // A call that has published its status answers for itself: what another stream's kernels have recorded since is for their
    // caller, and asking the device would take it from them.
    if (armed ? !tb::read_note(note, &code) || code != 0 : *static_cast<volatile uint32_t*>(mirror) != 0)
        return tb_device_status(device, detail);
    if (detail) *detail = 0;
    return TB_OK;
}

}  // extern "C"
