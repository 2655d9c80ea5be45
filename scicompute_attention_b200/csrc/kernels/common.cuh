// Shared device/host helpers for the sm_100a kernels: error reporting behind the C ABI, 16-byte
// async copies, warp-level tensor-core wrappers used by the bandwidth kernels, and softmax math.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include <atomic>
#include <cstdint>
#include <string>

#include "sca_b200.h"

namespace sca_b200 {

// ---- error plumbing (host) --------------------------------------------------------------------
// Stores the message for sca_last_error() and returns `code` so call sites can `return Fail(...)`.
int Fail(int code, const std::string& message);
void ClearError();
// Maps a cudaError_t to SCA_CUDA_ERROR / SCA_CUDA_OOM with "<what>: <cudaGetErrorName>: <string>".
int FailCuda(cudaError_t err, const char* what);
// cudaGetLastError() right after a launch (reference behaviour: src/runtime/launcher.cu:94-100);
// honours SCI_ATTENTION_DEBUG_SYNC=1 by synchronising the stream and reporting the async error.
int CheckLaunch(const char* kernel_name, cudaStream_t stream);
// True when SCI_ATTENTION_DEBUG_SYNC=1 (CheckLaunch then synchronises the stream after every launch).
bool DebugSyncEnabled();
// Opt-in to > 48 KiB of dynamic shared memory once per kernel symbol.
int EnsureDynamicSmem(const void* kernel, size_t bytes, const char* kernel_name);
// Cached SM count of the current device.
int SmCount();
// Sends `bytes` of host memory that may go away on return to the device, in the order of the stream.
int SendToDevice(void* device, const void* host, size_t bytes, cudaStream_t stream, const char* what);

// Launches `kernel` as a programmatic dependent of the kernel ahead of it on the stream (cluster > 1: on clusters of that many
// CTAs): its CTAs may be set up while that one still runs. So the kernel calls one of the two functions below ahead of its first
// access to global memory, reads and writes alike, in every CTA - its end then says that all kernels before it have ended.
// It also reads global memory with ordinary loads only: the kernel ahead may write while this one is already there, and the
// loads of __ldg and of const __restrict__ pointers are for memory that nobody writes while the kernel lives; neither the
// wait nor its memory clobber holds such a load back.
// Back to back on one stream, without / with: decode of one sequence 8.2 / 5.8 us a call, append + paged decode of 6 sequences
// 14.3 / 10.3, a prompt of 203 tokens 10.3 / 8.1, KV append + two gathers + reset 115.7 / 109.
template <typename... Params, typename... Args>
void LaunchDependent(void (*kernel)(Params...), int64_t grid, int block, size_t smem, cudaStream_t stream, int cluster, Args&&... args) {
    cudaLaunchAttribute attrs[2]{};
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = static_cast<unsigned>(cluster);
    attrs[1].val.clusterDim.y = 1;
    attrs[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(static_cast<unsigned>(block));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attrs;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);  // CheckLaunch reports a failure
}

// The answer of an occupancy query, kept per device. `ask` returns a negative number when the device cannot say; that is
// not kept. Threads that ask at the same time store the same number.
class PerDevice {
public:
    template <typename Ask>
    int Get(Ask ask) {
        int device = 0;
        const bool kept = cudaGetDevice(&device) == cudaSuccess && device >= 0 && device < kMaxDevices;
        if (kept) {
            if (const int n = answers_[device].load(std::memory_order_relaxed); n != 0) return n - 1;
        }
        const int n = ask();
        if (kept && n >= 0) answers_[device].store(n + 1, std::memory_order_relaxed);
        return n;
    }

private:
    static constexpr int kMaxDevices = 64;
    std::atomic<int> answers_[kMaxDevices] = {};  // answer + 1, 0 = not asked yet
};

inline bool Aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// ---- device helpers -----------------------------------------------------------------------------
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// Kernels launched by LaunchDependent: waits until the kernel ahead on the stream has ended and its writes are visible (at
// once where there is none).
__device__ __forceinline__ void WaitForPredecessor() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
// The same, and lets the next kernel on the stream be set up from here on.
__device__ __forceinline__ void BeginAfterPredecessor() {
    WaitForPredecessor();
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

__device__ __forceinline__ uint32_t ClusterRank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void ClusterBarrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// A float in the shared memory of CTA `rank` of this cluster, at this CTA's address `addr`.
__device__ __forceinline__ float LoadFromRank(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}
__device__ __forceinline__ float2 LoadFromRank2(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    float2 v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(remote) : "memory");
    return v;
}
__device__ __forceinline__ float4 LoadFromRank4(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    float4 v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
    return v;
}

__device__ __forceinline__ uint32_t SmemAddr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 16-byte global->shared async copy; src_bytes == 0 zero-fills the destination without reading.
__device__ __forceinline__ void CpAsync16(uint32_t smem_dst, const void* gmem_src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_dst), "l"(gmem_src),
                 "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void CpAsyncCommit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void CpAsyncWait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ uint4 LdsV4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}

// D(16x8, f32) += A(16x16) * B(16x8); A row-major, B column-major fragments, 16-bit inputs.
template <typename T>
__device__ __forceinline__ void MmaM16N8K16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                            uint32_t a3, uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void MmaM16N8K16<__half>(float (&c)[4], uint32_t a0, uint32_t a1,
                                                    uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void MmaM16N8K16<__nv_bfloat16>(float (&c)[4], uint32_t a0, uint32_t a1,
                                                           uint32_t a2, uint32_t a3, uint32_t b0,
                                                           uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Packs two floats into one 32-bit register of 16-bit values (lo in bits 0..15), round-to-nearest.
template <typename T>
__device__ __forceinline__ uint32_t Pack2(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t Pack2<__half>(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t Pack2<__nv_bfloat16>(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ float Exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}

// Two fp32 lanes per instruction (sm_100 packed arithmetic): halves the issue slots of FMA chains.
__device__ __forceinline__ float2 Fma2(float2 a, float2 b, float2 c) {
    uint64_t ra, rb, rc, rd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rc) : "f"(c.x), "f"(c.y));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(ra), "l"(rb), "l"(rc));
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
    return d;
}
__device__ __forceinline__ float Max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float2 Add2(float2 a, float2 b) {
    uint64_t ra, rb, rd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
    return d;
}

__device__ __forceinline__ float ToFloat(float v) { return v; }
__device__ __forceinline__ float ToFloat(__half v) { return __half2float(v); }
__device__ __forceinline__ float ToFloat(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T>
__device__ __forceinline__ T FromFloat(float v);
template <>
__device__ __forceinline__ float FromFloat<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half FromFloat<__half>(float v) { return __float2half_rn(v); }
template <>
__device__ __forceinline__ __nv_bfloat16 FromFloat<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

}  // namespace sca_b200
