// Shared device/host helpers for the KDA kernels (sm_100a).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include <atomic>

#include "../../include/kda_b200.h"

namespace kda {

constexpr int kChunk = 64;   // tokens per chunk
constexpr int kLD = 68;      // padded leading dimension (floats) of a 64x64 shared-memory tile

__device__ __forceinline__ float ld_io(const void* p, size_t i, int bf16) {
    return bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i])
                : reinterpret_cast<const float*>(p)[i];
}
__device__ __forceinline__ void st_io(void* p, size_t i, int bf16, float x) {
    if (bf16) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16(x);
    else reinterpret_cast<float*>(p)[i] = x;
}

// Two float32 in a 64-bit register pair.  sm_100a executes one packed instruction for both at the same rate per value, so
// kernels bound by instruction issue halve that part of their count; each half rounds like the scalar instruction.
struct f2 {
    unsigned long long v;
};
__device__ __forceinline__ f2 f2_make(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2_get(f2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}
__device__ __forceinline__ f2 f2_all(float a) { return f2_make(a, a); }
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// a bf16 pair in one word <-> two float32
__device__ __forceinline__ f2 f2_from_bf16(unsigned u) { return f2_make(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
__device__ __forceinline__ unsigned f2_to_bf16(f2 a) {
    const float2 x = f2_get(a);
    const __nv_bfloat162 h = __floats2bfloat162_rn(x.x, x.y);
    return *reinterpret_cast<const unsigned*>(&h);
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// A kernel that may start while the one before it in its stream still runs (programmatic dependent launch), and while those run that that
// one started beside.  Kernels launched this way wait (dependency_wait) before they touch anything these write; convolutions and gate
// activations, which share nothing with them, wait at their own end, so that whatever is launched the usual way finds all of them done.
// None of them holds tensor memory.
template <class... P, class... A>
inline cudaError_t launch_early(void (*kern)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, bool early, int cluster, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    unsigned n = 0;
    if (early) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)cluster;
        at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}
// All of the kernel this one depends on has ended and its writes are visible; at once in a kernel launched the usual way.
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// What the kernel before may have written is read behind dependency_wait() by these: a load the compiler takes for one of constant
// memory (__ldg, or through a const __restrict__ pointer) may be moved ahead of the wait, and was.
__device__ __forceinline__ uint4 ld_after16(const void* p) {
    uint4 r;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ uint2 ld_after8(const void* p) {
    uint2 r;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p) : "memory");
    return r;
}
__device__ __forceinline__ float ld_after_bf16(const void* p, size_t i) {
    unsigned short r;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(r) : "l"(static_cast<const __nv_bfloat16*>(p) + i) : "memory");
    return __uint_as_float((unsigned)r << 16);
}
// All blocks of the cluster have come here, and what they wrote to shared memory, each other's included, is there.
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// *p = x in block `rank` of the cluster
__device__ __forceinline__ void st_cluster(float* p, int rank, float x) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(x) : "memory");
}
__device__ __forceinline__ float ld_after_f32(const float* p) {
    float r;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(p) : "memory");
    return r;
}
// The kernel after this one may start once every block has said so or ended.
__device__ __forceinline__ void dependents_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// One output of a 128-wide product: lane holds x[4 lane .. 4 lane + 3] (u) in xv; weights (float32 masters are rounded to
// bf16, as a cast of the matrix would) start at w[base].  Every lane gets the sum.
__device__ __forceinline__ void narrow_x(uint2 u, float (&xv)[4]) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    xv[0] = a.x; xv[1] = a.y; xv[2] = b.x; xv[3] = b.y;
}
template <bool F32W>
__device__ __forceinline__ void narrow_w(const void* w, size_t base, int lane, float (&wv)[4]) {
    if (F32W) {
        const float4 f = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(w) + base) + lane);
        wv[0] = __bfloat162float(__float2bfloat16(f.x)); wv[1] = __bfloat162float(__float2bfloat16(f.y));
        wv[2] = __bfloat162float(__float2bfloat16(f.z)); wv[3] = __bfloat162float(__float2bfloat16(f.w));
    } else {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(w) + base) + lane);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
        wv[0] = a.x; wv[1] = a.y; wv[2] = b.x; wv[3] = b.y;
    }
}
__device__ __forceinline__ float narrow_sum(const float (&xv)[4], const float (&wv)[4]) {
    float y = xv[0] * wv[0];
    y = fmaf(xv[1], wv[1], y);
    y = fmaf(xv[2], wv[2], y);
    y = fmaf(xv[3], wv[3], y);
    return warp_sum(y);
}

__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

// Device status of a workspace: int 0 is the status word, ints 2 and 3 hold the address of a page-locked host word that
// mirrors it (null: none), left there by the forward's first kernel.  Only a failure writes either, so a call that goes
// well pays nothing for being watched: the host reads its own memory at the next call.
// Out of line: inlined at every wait it cost the intra-chunk kernels registers (forward 56 bytes of spills, now 24).
static __device__ __noinline__ void raise_status(int* status, int code) {
    // The thread that sets the word tells the host, nobody else: an expired wait is met by hundreds of threads over a long
    // time, and one that came after the host had read and cleared its word would blame the next, healthy call.
    if (atomicCAS(status, 0, code) != 0) return;
    volatile int* mirror = *reinterpret_cast<int* const*>(status + 2);
    if (mirror != nullptr) {
        *mirror = code;
        __threadfence_system();
    }
}
int* status_mirror();      // host: the mirror word registered for the current device, or null (kda_api.cu)

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Launch accounting (implemented in kda_api.cu): every kernel launch of the library goes through
// KDA_LAUNCH, which counts it and, when profiling is enabled, brackets it with CUDA events on the
// launching stream so a caller can read per-kernel device time.
namespace prof {
extern std::atomic<unsigned long long> launches;
extern std::atomic<bool> enabled;
void begin(const char* name, cudaStream_t st);
void end(cudaStream_t st);
}  // namespace prof
#define KDA_LAUNCH(name, st, ...)                                                        \
    do {                                                                                 \
        ::kda::prof::launches.fetch_add(1, std::memory_order_relaxed);                   \
        const bool timed_ = ::kda::prof::enabled.load(std::memory_order_relaxed);        \
        if (timed_) ::kda::prof::begin(name, st);                                        \
        __VA_ARGS__;                                                                     \
        if (timed_) ::kda::prof::end(st);                                                \
    } while (0)

// Dynamic shared memory limit of a kernel: the attribute is a driver call, so it is set once per kernel and device.
// Kernels that share a signature share this function's statics; one past their number pays the driver calls every time.
constexpr int kSmemKernels = 64;
template <class Kern>
inline int set_smem_limit(Kern kern, size_t bytes) {
    constexpr int kDevices = 64, kKernels = kSmemKernels;
    static std::atomic<const void*> done[kDevices][kKernels];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return KDA_ERR_CUDA;
    const void* key = reinterpret_cast<const void*>(kern);
    if (dev < kDevices)
        for (int i = 0; i < kKernels; ++i)
            if (done[dev][i].load(std::memory_order_acquire) == key) return KDA_OK;
    int most = 0;
    if (cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return KDA_ERR_CUDA;
    cudaFuncAttributes at;
    if (cudaFuncGetAttributes(&at, key) != cudaSuccess) return KDA_ERR_CUDA;
    // the most the kernel may ask for, so that one call covers every size it is launched with
    const int limit = most - (int)at.sharedSizeBytes;
    if ((size_t)limit < bytes || cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess)
        return KDA_ERR_CUDA;
    if (dev < kDevices)
        for (int i = 0; i < kKernels; ++i) {
            const void* none = nullptr;
            if (done[dev][i].compare_exchange_strong(none, key, std::memory_order_release)) break;
        }
    return KDA_OK;
}

// Host-side launch check: returns a KDA_ERR_* code instead of throwing.
// Takes the error of a failed launch away as it reports it, so whoever asks has to pass the answer on.
[[nodiscard]] inline int launch_status() {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess && getenv("KDA_B200_VERBOSE")) fprintf(stderr, "libkda_b200: CUDA error: %s\n", cudaGetErrorString(e));
    return e == cudaSuccess ? KDA_OK : KDA_ERR_CUDA;
}

}  // namespace kda
