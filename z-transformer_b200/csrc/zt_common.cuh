// Shared host/device helpers of libztattn: refusal reporting, launch accounting,
// per-device facts.  Nothing here computes attention.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

namespace zt {

// ---- refusals --------------------------------------------------------------
// The reference prints a reason to stderr and returns 1
// (src/cuda/attn_kernels.cu:21-37).  The same, plus a per-thread copy of the text.
inline thread_local char g_last_error[768] = "";
inline thread_local const char *g_last_path = "none";
inline std::atomic<int> g_verbose{1};
inline std::atomic<int> g_path{0};
inline std::atomic<unsigned long long> g_launches{0};

inline int refuse(const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
    va_end(ap);
    if (g_verbose.load(std::memory_order_relaxed)) fprintf(stderr, "zt_attn: %s\n", g_last_error);
    return 1;
}

// Checked after every launch, as the reference does between its two backward
// kernels (src/cuda/attn_kernels.cu:1025-1034): a failed launch is a refusal,
// never a dead process, and the error is cleared so a later call cannot inherit it.
inline int launch_failed(const char *what) {
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) {
        g_launches.fetch_add(1, std::memory_order_relaxed);
        return 0;
    }
    return refuse("%s failed: %s", what, cudaGetErrorString(e));
}

// ---- optional per-kernel timing ------------------------------------------------
// When switched on (zt_attn_profile), every launch is bracketed by two CUDA events on
// the launching stream; zt_attn_profile_read waits for them and reports, per kernel
// name, the launches and the summed device time.  Off by default: no events exist.
struct ProfEntry {
    const char *name;
    cudaEvent_t start, stop;
};
inline std::atomic<int> g_profile{0};
inline std::mutex g_prof_mu;
inline std::vector<ProfEntry> g_prof;

inline int prof_begin(cudaStream_t stream) {
    if (!g_profile.load(std::memory_order_relaxed)) return -1;
    ProfEntry e{nullptr, nullptr, nullptr};
    if (cudaEventCreate(&e.start) != cudaSuccess || cudaEventCreate(&e.stop) != cudaSuccess) {
        cudaGetLastError();
        return -1;
    }
    cudaEventRecord(e.start, stream);
    std::lock_guard<std::mutex> lock(g_prof_mu);
    g_prof.push_back(e);
    return (int)g_prof.size() - 1;
}

inline void prof_end(int idx, const char *name, cudaStream_t stream) {
    if (idx < 0) return;
    std::lock_guard<std::mutex> lock(g_prof_mu);
    if (idx >= (int)g_prof.size()) return;
    g_prof[idx].name = name;
    cudaEventRecord(g_prof[idx].stop, stream);
}

// Launch `...` (a <<<>>> statement), time it when profiling is on, and turn a failed
// launch into a refusal.  Evaluates to 0 on success, 1 on failure.
#define ZT_LAUNCH(name, stream, ...)                          \
    ([&]() -> int {                                           \
        const int zt_pi_ = ::zt::prof_begin(stream);          \
        __VA_ARGS__;                                          \
        ::zt::prof_end(zt_pi_, name, stream);                 \
        return ::zt::launch_failed(name " launch");           \
    }())

// ---- launches that overlap the end of the kernel before them -------------------------------------
// Programmatic dependent launch: the grid may be set up while the kernel before it in the stream still runs.  Every
// kernel launched this way calls pdl_wait() in every block before it touches global memory -- it returns once the
// kernel before has completed and its writes are visible, so the stream's order is what it always was -- and
// pdl_launch() as soon as its own successor may be set up.  On a chain of 5-10 us kernels this takes 1-2 us off
// each gap.  What the kernel before has written is read by plain loads only: __ldg, and pointers that are const and
// __restrict__, promise that the data does not change while the kernel runs, which lets the compiler move them ahead of
// the wait.  (Data of earlier launches is older than the kernel: the one before lets it be set up only after its own wait.)
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- per-device facts, asked once per device --------------------------------
struct DeviceInfo {
    int known = 0;
    int sm_count = 0;
    int cc_major = 0, cc_minor = 0;
    size_t smem_optin = 0;
};

inline const DeviceInfo *device_info() {
    static DeviceInfo table[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return nullptr;
    }
    DeviceInfo &d = table[dev];
    if (d.known) return &d;
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return nullptr;
    d.sm_count = v;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return nullptr;
    d.smem_optin = (size_t)v;
    cudaDeviceGetAttribute(&d.cc_major, cudaDevAttrComputeCapabilityMajor, dev);
    cudaDeviceGetAttribute(&d.cc_minor, cudaDevAttrComputeCapabilityMinor, dev);
    d.known = 1;
    return &d;
}

// Function attributes are set once per (kernel, device, value): asking the driver on every launch costs more host time
// than the launch's own bookkeeping.  Returns whether `value` is already known to hold.
inline bool attribute_known(const void *fn, int attr, size_t value, bool record) {
    struct Entry { const void *fn; int dev, attr; size_t value; };
    static std::vector<Entry> known;
    static std::mutex mu;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> lock(mu);
    for (Entry &e : known)
        if (e.fn == fn && e.dev == dev && e.attr == attr) {
            if (record && value > e.value) e.value = value;
            return value <= e.value;
        }
    if (record) known.push_back(Entry{fn, dev, attr, value});
    return record;
}

// Opt a kernel into more than 46 KiB of dynamic shared memory (the static kind counts against the 48 too); a refusal, not an exit
// (src/cuda/attn_kernels.cu:822-830).
inline int optin_smem(const void *fn, size_t bytes) {
    if (bytes <= 46u * 1024u || attribute_known(fn, (int)cudaFuncAttributeMaxDynamicSharedMemorySize, bytes, false)) return 0;
    const cudaError_t e =
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) {
        attribute_known(fn, (int)cudaFuncAttributeMaxDynamicSharedMemorySize, bytes, true);
        return 0;
    }
    return refuse("the device would not grant %zu bytes of shared memory per block: %s", bytes,
                  cudaGetErrorString(e));
}

template <typename... P, typename... A>
inline int launch_pdl(const char *name, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                      const A &...args) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = stream;
    cfg.attrs = attr, cfg.numAttrs = 1;
    const int pi = prof_begin(stream);
    cudaLaunchKernelEx(&cfg, kernel, args...);
    prof_end(pi, name, stream);
    return launch_failed(name);
}

// The same for a grid of thread-block clusters of `cluster` blocks along x.
template <typename... P, typename... A>
inline int launch_pdl_cluster(const char *name, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              int cluster, const A &...args) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster, attr[1].val.clusterDim.y = 1, attr[1].val.clusterDim.z = 1;
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = stream;
    cfg.attrs = attr, cfg.numAttrs = 2;
    const int pi = prof_begin(stream);
    cudaLaunchKernelEx(&cfg, kernel, args...);
    prof_end(pi, name, stream);
    return launch_failed(name);
}

// The same for the tensor-core kernels, which take whole SMs: overlapped only where every block finds an SM of its own.
// A longer grid set up early starts as the SMs fall free, one by one, and its blocks then walk their tiles out of step
// with the neighbours they share them with in L2: forward and backward at T 32768 took 4 % longer that way, and
// batch 8, T 512, heads of 64 still 1.6 %.
// `per_sm`: blocks that an SM holds.
template <typename... P, typename... A>
inline int launch_after(const char *name, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int per_sm,
                        const A &...args) {
    const DeviceInfo *d = device_info();
    if (d && (long long)grid.x * grid.y * grid.z <= (long long)per_sm * d->sm_count) return launch_pdl(name, kernel, grid, block, smem, stream, args...);
    const int pi = prof_begin(stream);
    kernel<<<grid, block, smem, stream>>>(args...);
    prof_end(pi, name, stream);
    return launch_failed(name);
}

// ---- in-kernel negative controls (the harness build only) ---------------------------------------
// The reference compiles defects into its kernels as template variants and requires its parity gates
// to catch every one of them (src/cuda/attn_kernels.cu:150-158,592-599,622-624; src/cuda/run-attn.sh:126-177).
// The same here, for the defects that live INSIDE a kernel: built with -DZT_DEFECTS the kernels consult a
// device word that zt_attn_set_defect writes; every defect computes wrong numbers from valid addresses.
//   1  the causal mask is dropped in the forward (a query reads the keys after it in its diagonal tiles)
//   3  the forward's running-maximum correction is skipped (sum and accumulator are never rescaled)
//   11 the causal mask is dropped in the backward
//   13 the softmax Jacobian is dropped in the backward (dS = P dP)
// The shipped library is built without the macro: ZT_DEFECT(n) is then the constant false and no kernel
// carries a switch.
#ifdef ZT_DEFECTS
static __device__ int g_defect;
#define ZT_DEFECT(n) (g_defect == (n))
#else
#define ZT_DEFECT(n) false
#endif

// Copies of an output tensor in other GPUs' memory (peer device pointers, mapped into this process): a kernel that
// is given them stores every output element there as well as locally, so the all-gather of that output happens
// inside the kernel, element by element over NVLink, instead of as a collective after it.
constexpr int kMaxPeers = 7;
struct PeerList {
    float *ptr[kMaxPeers];
    int n;
};

// ---- thread-block clusters ----------------------------------------------------------------------
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();  // (.aligned: the whole warp together, also where what lies before it was a single thread's)
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A float of block `rank`'s shared memory, at the place that `addr` has in this block's.
__device__ __forceinline__ float ld_cluster(uint32_t addr, int rank) {
    float v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}\n"
                 : "=f"(v) : "r"(addr), "r"(rank) : "memory");
    return v;
}

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// 16 bytes into shared memory, asynchronously; `in` false fills them with zeros and reads nothing.
__device__ __forceinline__ void copy16_async(uint32_t dst, const void *src, bool in) {
    const int bytes = in ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// The same from a source on a 4-byte boundary only.
__device__ __forceinline__ void copy16_async_by4(uint32_t dst, const void *src, bool in) {
    const int bytes = in ? 4 : 0;
#pragma unroll
    for (int i = 0; i < 16; i += 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + i), "l"(static_cast<const char *>(src) + i), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>  // all but the PENDING latest groups of this thread have landed
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

}  // namespace zt
