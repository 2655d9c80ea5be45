// Prefill problems of fewer query tiles than SMs: the kernels in which the CTAs of a cluster share the KV tiles of an item
// (kSplit in flash_kernel.cuh).
#include "flash_kernel.cuh"

namespace sca_b200 {
namespace flash {

template <typename T, int DP, int QT, int BN>
int ResidentClusters(int cluster) {
    static PerDevice resident[kMaxSplit + 1];  // per instantiation
    const int n = resident[cluster].Get([cluster] {
        auto kernel = flash_fwd_sm100_kernel<T, DP, QT, BN, false, false, true>;
        // the query answers for the shared memory the kernel is allowed at that point
        if (EnsureDynamicSmem(reinterpret_cast<const void*>(kernel), FlashGeom<DP, QT, BN>::kSmemBytes, "flash_fwd_sm100_kernel") != SCA_OK) return -1;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = static_cast<unsigned>(cluster);
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(static_cast<unsigned>(cluster));
        cfg.blockDim = dim3(FlashThreads<T, DP, QT>());
        cfg.dynamicSmemBytes = FlashGeom<DP, QT, BN>::kSmemBytes;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return -1;
        }
        return clusters;
    });
    return n > 0 ? n : 0;
}

template <typename T, int DP, int QT, int BN, bool kVarlen, bool kPaged>
int LaunchSplit(int64_t items, cudaStream_t stream, const CUtensorMap& map_q, const CUtensorMap& map_k, const CUtensorMap& map_v,
                const FlashKernelParams& p) {
    auto kernel = flash_fwd_sm100_kernel<T, DP, QT, BN, kVarlen, kPaged, true>;
    constexpr int kSmem = FlashGeom<DP, QT, BN>::kSmemBytes;
    if (int rc = EnsureDynamicSmem(reinterpret_cast<const void*>(kernel), kSmem, "flash_fwd_sm100_kernel")) return rc;
    LaunchDependent(kernel, items * p.cluster, FlashThreads<T, DP, QT>(), kSmem, stream, p.cluster, map_q, map_k, map_v, p);
    return SCA_OK;
}

#define SCA_SPLIT(T, DP, QT)                                                                                                       \
    template int ResidentClusters<T, DP, QT, 128>(int);                                                                            \
    template int LaunchSplit<T, DP, QT, 128, false, false>(int64_t, cudaStream_t, const CUtensorMap&, const CUtensorMap&,          \
                                                           const CUtensorMap&, const FlashKernelParams&);                          \
    template int LaunchSplit<T, DP, QT, 128, true, false>(int64_t, cudaStream_t, const CUtensorMap&, const CUtensorMap&,           \
                                                          const CUtensorMap&, const FlashKernelParams&);                           \
    template int LaunchSplit<T, DP, QT, 128, true, true>(int64_t, cudaStream_t, const CUtensorMap&, const CUtensorMap&,            \
                                                         const CUtensorMap&, const FlashKernelParams&);
SCA_SPLIT(__half, 64, 2)
SCA_SPLIT(__half, 128, 2)
SCA_SPLIT(__half, 256, 1)
SCA_SPLIT(__nv_bfloat16, 64, 2)
SCA_SPLIT(__nv_bfloat16, 128, 2)
SCA_SPLIT(__nv_bfloat16, 256, 1)
#undef SCA_SPLIT

}  // namespace flash
}  // namespace sca_b200
