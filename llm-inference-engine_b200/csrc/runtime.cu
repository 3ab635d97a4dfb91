// runtime.cu -- error plumbing, device queries and the library workspace of libb200llm.so.
#include "common.cuh"

#include <cuda.h>  // CUtensorMap: types only, the encoder comes through cudaGetDriverEntryPoint (no libcuda to link)
#include <atomic>
#include <algorithm>
#include <mutex>
#include <unordered_set>

#ifndef B200_NO_NVTX
#include <nvtx3/nvToolsExt.h>
#endif

namespace b200 {

#ifndef B200_NO_NVTX
NvtxRange::NvtxRange(const char *name) { nvtxRangePushA(name); }
NvtxRange::~NvtxRange() { nvtxRangePop(); }
#endif


static thread_local char g_err[512] = "";

void set_error(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int cuda_status(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return wait_status(what);
    set_error("%s: %s", what, cudaGetErrorString(e));
    return B200_ERR_CUDA;
}

// The wait word of the process, made by the first launch that needs it.
static std::atomic<unsigned int *> g_wait_word{nullptr};
static thread_local unsigned int t_wait_clocks = kWaitClocks;
static unsigned int *wait_word() {
    static std::once_flag once;
    std::call_once(once, [] {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // (the launch may be one that is being captured)
        cudaThreadExchangeStreamCaptureMode(&mode);
        void *p = nullptr;
        if (cudaHostAlloc(&p, sizeof(unsigned int), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
            *static_cast<unsigned int *>(p) = 0;
            g_wait_word.store(static_cast<unsigned int *>(p), std::memory_order_release);
        } else {
            cudaGetLastError();
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
    });
    return g_wait_word.load(std::memory_order_acquire);
}
WaitGuard wait_guard() { return {wait_word(), t_wait_clocks}; }  // (one address for host and devices: unified addressing)

static unsigned int wait_code() {
    unsigned int *w = g_wait_word.load(std::memory_order_acquire);
    return w ? *reinterpret_cast<volatile unsigned int *>(w) : 0u;
}
int wait_status(const char *what) {
    const unsigned int code = wait_code();
    if (code == 0) return B200_OK;
    static const char *const names[] = {"", "the streaming GEMV", "the CTA-pair GEMM", "the prompt attention", "the wait probe", "the one-CTA GEMM"};
    set_error("%s: a wait inside %s ran out; results since then are not valid (b200_wait_error(1) clears this)", what, code <= kWaitGemm ? names[code] : "a kernel");
    return B200_ERR_CUDA;
}

// a barrier that nothing arrives at: what is left of a kernel whose producer never comes
__global__ void wait_probe_kernel(WaitGuard wait) {
    __shared__ __align__(8) unsigned long long bar;
    const uint32_t addr = (uint32_t)__cvta_generic_to_shared(&bar);
    if (threadIdx.x == 0) {
        cta_gave_up() = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(addr) : "memory");
    }
    __syncthreads();
    mbar_wait_guarded(addr, 0, wait, kWaitProbe);
}

int sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

bool allow_smem(const void *kernel, size_t most, size_t per_sm) {
    static std::mutex mu;
    static std::unordered_set<const void *> raised[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    static thread_local std::unordered_set<const void *> seen[64];  // (what this thread has found raised: no lock on a hot path)
    dev &= 63;
    if (seen[dev].count(kernel)) return true;
    std::lock_guard<std::mutex> lk(mu);
    if (!raised[dev].count(kernel)) {
        if (most == 0) {
            int all = 0;
            cudaFuncAttributes own;
            if (cudaDeviceGetAttribute(&all, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || cudaFuncGetAttributes(&own, kernel) != cudaSuccess) return false;
            most = (size_t)all - own.sharedSizeBytes;
        }
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess) return false;
        if (per_sm > 0 && cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)std::min<size_t>(100, (per_sm * 100 + (228 << 10) - 1) / (228 << 10))) != cudaSuccess) return false;
        raised[dev].insert(kernel);
    }
    seen[dev].insert(kernel);
    return true;
}

bool tile_map(CUtensorMap *map, const void *ptr, size_t rows, int cols, int box_rows, bool bf16) {
    typedef CUresult (*Encode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &found) != cudaSuccess) cudaGetLastError(), sym = nullptr;
        return sym && found == cudaDriverEntryPointSuccess ? reinterpret_cast<Encode>(sym) : nullptr;
    }();
    if (!encode) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows}, steps[2] = {1, 1};
    auto make = [&] {
        return encode(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, steps,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    if (make() == CUDA_SUCCESS) return true;
    // The encoder is the driver's and wants a current context, which the runtime binds to a thread with its first call that needs one: in a thread whose first
    // call is this one there is none yet.
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess && make() == CUDA_SUCCESS;
}

// One workspace per device: [tickets (kTickets x u32, zeroed once, self-resetting) | scratch].
static constexpr size_t kTickets = 16384;
struct WsSlot {
    void *base = nullptr;
    size_t bytes = 0;
    bool owned = false;
};
static WsSlot g_ws[64];
static std::mutex g_ws_mu;

bool get_workspace(Workspace *ws) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_ws_mu);
    WsSlot &s = g_ws[dev & 63];
    if (!s.base) {
        set_error("library workspace not set: call b200_workspace_ensure() or b200_workspace_set() first");
        return false;
    }
    ws->tickets = reinterpret_cast<unsigned int *>(s.base);
    ws->n_tickets = kTickets;
    ws->scratch = reinterpret_cast<char *>(s.base) + kTickets * sizeof(unsigned int);
    ws->scratch_bytes = s.bytes - kTickets * sizeof(unsigned int);
    return true;
}

}  // namespace b200

using namespace b200;

extern "C" {

const char *b200_last_error_string(void) { return g_err; }
int b200_abi_version(void) { return B200LLM_ABI_VERSION; }
int b200_sm_count(void) { return sm_count(); }

int b200_wait_error(int clear) {
    const unsigned int code = wait_code();
    if (clear && code) *reinterpret_cast<volatile unsigned int *>(g_wait_word.load(std::memory_order_acquire)) = 0;
    return (int)code;
}
void b200_wait_limit(unsigned int clocks) { t_wait_clocks = clocks < kWaitClocks ? clocks : kWaitClocks; }
int b200_wait_probe(b200_stream_t stream) {
    wait_probe_kernel<<<1, 64, 0, as_stream(stream)>>>(wait_guard());
    return cuda_status("wait_probe launch");
}

size_t b200_workspace_default_bytes(void) { return (size_t)64 << 20; }

int b200_workspace_set(void *ptr, size_t bytes) {
    B200_REQUIRE(ptr != nullptr && aligned16(ptr), "workspace pointer must be non-null and 16-byte aligned");
    B200_REQUIRE(bytes >= ((size_t)1 << 20), "workspace must be at least 1 MiB");
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaMemset(ptr, 0, kTickets * sizeof(unsigned int)) != cudaSuccess) return cuda_status("workspace memset");
    std::lock_guard<std::mutex> lk(g_ws_mu);
    WsSlot &s = g_ws[dev & 63];
    if (s.owned && s.base) cudaFree(s.base);
    s.base = ptr;
    s.bytes = bytes;
    s.owned = false;
    return B200_OK;
}

int b200_workspace_ensure(size_t bytes) {
    if (bytes == 0) bytes = b200_workspace_default_bytes();
    int dev = 0;
    cudaGetDevice(&dev);
    {
        std::lock_guard<std::mutex> lk(g_ws_mu);
        WsSlot &s = g_ws[dev & 63];
        if (s.base && s.bytes >= bytes) return B200_OK;
    }
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        set_error("workspace cudaMalloc(%zu) failed", bytes);
        return B200_ERR_WORKSPACE;
    }
    if (cudaMemset(p, 0, kTickets * sizeof(unsigned int)) != cudaSuccess) return cuda_status("workspace memset");
    std::lock_guard<std::mutex> lk(g_ws_mu);
    WsSlot &s = g_ws[dev & 63];
    if (s.owned && s.base) cudaFree(s.base);
    s.base = p;
    s.bytes = bytes;
    s.owned = true;
    return B200_OK;
}

}  // extern "C"
