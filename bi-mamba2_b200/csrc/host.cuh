// Host-side helpers shared by the library's translation units: error notes, tracing, launches, device queries.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <tuple>
#include <utility>
#include <vector>

#include "common.cuh"

namespace bissd {

extern thread_local char g_cuda_err[256];

inline int note_cuda(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return BISSD_OK;
    snprintf(g_cuda_err, sizeof(g_cuda_err), "%s: %s", what, cudaGetErrorString(e));
    return BISSD_ERR_LAUNCH;
}

// ---- tracing: optional CUDA-event brackets around every kernel launch, and a launch counter -------------
struct TraceRec {
    const char *name;
    cudaEvent_t e0, e1;
};
extern std::mutex g_trace_mu;
extern std::vector<TraceRec> g_trace;
extern std::atomic<int> g_trace_on;
extern std::atomic<unsigned long long> g_launches;

struct TraceScope {
    const char *name;
    cudaStream_t s;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    TraceScope(const char *n, cudaStream_t st) : name(n), s(st) {
        if (g_trace_on.load(std::memory_order_relaxed)) {
            if (cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess) cudaEventRecord(e0, s);
            else e0 = e1 = nullptr;
        }
    }
    void end() {
        g_launches.fetch_add(1, std::memory_order_relaxed);
        if (e0 && e1) {
            cudaEventRecord(e1, s);
            std::lock_guard<std::mutex> lk(g_trace_mu);
            g_trace.push_back(TraceRec{name, e0, e1});
        }
    }
};

// Launch `...` (a full kernel<<<>>>() expression) on stream `s`, count it, bracket it with events when tracing.
// Launch with programmatic stream serialisation: the kernel may be scheduled while its predecessor drains and
// waits for it in pdl_begin().  Only kernels that open with pdl_begin() go through here.  BISSD_NO_PDL=1 turns
// the attribute off (plain stream order).
inline bool no_pdl() {
    static const bool v = std::getenv("BISSD_NO_PDL") != nullptr;
    return v;
}
template <class... Exp, class... Act>
inline cudaError_t launch_cluster(void (*kernel)(Exp...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, unsigned cluster_x, Act &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (!no_pdl()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster_x > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster_x;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
}
template <class... Exp, class... Act>
inline cudaError_t launch_pdl(void (*kernel)(Exp...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Act &&...args) {
    return launch_cluster(kernel, grid, block, smem, s, 1, std::forward<Act>(args)...);
}

#define BISSD_LAUNCH_ON(stream, name, ...)                        \
    do {                                                          \
        TraceScope ts_(name, stream);                             \
        __VA_ARGS__;                                              \
        ts_.end();                                                \
        int rc_ = note_cuda(cudaGetLastError(), name);            \
        if (rc_ != BISSD_OK) return rc_;                          \
    } while (0)
#define BISSD_LAUNCH(name, ...) BISSD_LAUNCH_ON(s, name, __VA_ARGS__)

// Raise a kernel's dynamic shared-memory limit.  The attribute is per (function, device) and sticks, so it is set the
// first time a kernel needs `bytes` on a device and remembered (the driver call costs a microsecond or two per launch
// otherwise - a tenth of the host time of a whole pass).
inline std::mutex g_smem_mu;
inline std::map<std::pair<const void *, int>, size_t> g_smem_granted;   // (kernel, device) -> bytes already allowed
template <class K> inline int allow_smem(K kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return BISSD_OK;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
    const std::pair<const void *, int> key(reinterpret_cast<const void *>(kernel), dev);
    if (dev >= 0) {
        std::lock_guard<std::mutex> lk(g_smem_mu);
        auto it = g_smem_granted.find(key);
        if (it != g_smem_granted.end() && it->second >= bytes) return BISSD_OK;
    }
    int rc = note_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes),
                       "cudaFuncSetAttribute");
    if (rc == BISSD_OK && dev >= 0) {
        std::lock_guard<std::mutex> lk(g_smem_mu);
        size_t &g = g_smem_granted[key];
        g = std::max(g, bytes);
    }
    return rc;
}

inline int sm_count() {
    static int n[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (!n[dev]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
        n[dev] = v;
    }
    return n[dev];
}

// Kernels that deal their registers anew (setmaxnreg) wait for ever if they were launched with fewer than the sum of the shares:
// has the compiler given `kernel` that many a thread?
template <class K> inline int check_registers(K kernel, int regs) {
    static std::mutex mu;
    static std::map<const void *, int> known;
    std::lock_guard<std::mutex> lk(mu);
    int &n = known[reinterpret_cast<const void *>(kernel)];
    if (n == 0) {
        cudaFuncAttributes at;
        const int rc = note_cuda(cudaFuncGetAttributes(&at, kernel), "cudaFuncGetAttributes");
        if (rc != BISSD_OK) return rc;
        n = at.numRegs;
    }
    return n >= regs ? BISSD_OK : note_cuda(cudaErrorLaunchOutOfResources, "registers of a kernel that deals them anew");
}

// Blocks of `kernel` an SM holds at once.  Asked once per form of a launch.
template <class K> inline int resident_blocks(K kernel, int threads, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<const void *, int, size_t>, int> known;
    std::lock_guard<std::mutex> lk(mu);
    int &n = known[{reinterpret_cast<const void *>(kernel), threads, smem}];
    if (n == 0 && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem) != cudaSuccess) n = 0;
    return std::max(n, 1);
}

#define BISSD_ALLOW(kernel, bytes)                  \
    do {                                             \
        int rc_ = allow_smem(kernel, bytes);         \
        if (rc_ != BISSD_OK) return rc_;             \
    } while (0)

inline int check_device() {
    static std::atomic<int> major_of[64];                        // 0 = not asked yet
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return BISSD_ERR_LAUNCH;
    int major = (dev >= 0 && dev < 64) ? major_of[dev].load(std::memory_order_relaxed) : 0;
    if (!major) {
        if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess) return BISSD_ERR_LAUNCH;
        if (dev >= 0 && dev < 64) major_of[dev].store(major, std::memory_order_relaxed);
    }
    return major == 10 ? BISSD_OK : BISSD_ERR_ARCH;
}

static inline size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

}  // namespace bissd
