// Launches of the resident path (prop_resident.cuh): one cooperative launch per set of shots.
#include <mutex>

#include "prop_resident.cuh"

namespace fwi {

namespace {

template <typename Args> using ResKernel = void (*)(Batch<float>, ResidentGrid, Args);

template <int ST> ResKernel<ResFwdArgs> fwd_kernel(int pitch)
{
    switch (pitch) {
    case 96: return k_resident_fwd<ST, 96>;
    case 160: return k_resident_fwd<ST, 160>;
    case 224: return k_resident_fwd<ST, 224>;
    case 320: return k_resident_fwd<ST, 320>;
    case 400: return k_resident_fwd<ST, 400>;
    default: return nullptr;
    }
}
template <int ST> ResKernel<ResAdjArgs> adj_kernel(int pitch)
{
    switch (pitch) {
    case 96: return k_resident_adj<ST, 96>;
    case 160: return k_resident_adj<ST, 160>;
    case 224: return k_resident_adj<ST, 224>;
    case 320: return k_resident_adj<ST, 320>;
    case 400: return k_resident_adj<ST, 400>;
    case 512: return k_resident_adj<ST, 512>;
    case 640: return k_resident_adj<ST, 640>;
    default: return nullptr;
    }
}
ResKernel<ResFwdArgs> fwd_kernel(int store_type, int pitch)
{
    return store_type == kStoreHalf ? fwd_kernel<kStoreHalf>(pitch)
           : store_type == kStoreBf16 ? fwd_kernel<kStoreBf16>(pitch) : fwd_kernel<kStoreNative>(pitch);
}
ResKernel<ResAdjArgs> adj_kernel(int store_type, int pitch)
{
    return store_type == kStoreHalf ? adj_kernel<kStoreHalf>(pitch)
           : store_type == kStoreBf16 ? adj_kernel<kStoreBf16>(pitch) : adj_kernel<kStoreNative>(pitch);
}

// Cooperative: every CTA of the launch is resident before any of them waits on another.
template <typename Args>
cudaError_t launch(ResKernel<Args> k, const Batch<float> &b, const ResidentSet &set, const Args &a, cudaStream_t st)
{
    if (!k) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(set.grid.n);
    cfg.blockDim = dim3(set.threads);
    cfg.dynamicSmemBytes = set.smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, b, set.grid, a);
}

}  // namespace

// Dynamic shared memory of a CTA on the current device (0: the kernels cannot run there): the
// device's opt-in limit less their static shared memory; the function attributes are set once.
size_t resident_smem_limit()
{
    static std::mutex mu;
    static size_t limit[256] = {};
    static bool done[256] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) {
        cudaGetLastError();
        return 0;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (done[dev]) return limit[dev];
    int optin = 0, coop = 0;
    bool ok = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
              cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop && optin > 1024;
    const int lim = optin - 1024;
    for (int st : {(int)kStoreNative, (int)kStoreHalf, (int)kStoreBf16}) {
        for (int p : kResPitches)
            for (const void *k : {(const void *)fwd_kernel(st, p), (const void *)adj_kernel(st, p)})
                ok = ok && (!k || cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) == cudaSuccess);
    }
    if (!ok) cudaGetLastError();
    limit[dev] = ok ? (size_t)lim : 0;
    done[dev] = true;
    return limit[dev];
}

cudaError_t launch_resident_forward(const Batch<float> &b, const ResidentSet &set, const ResFwdArgs &a, cudaStream_t st)
{
    return launch(fwd_kernel(b.store_type, set.pitch), b, set, a, st);
}

cudaError_t launch_resident_adjoint(const Batch<float> &b, const ResidentSet &set, const ResAdjArgs &a, cudaStream_t st)
{
    return launch(adj_kernel(b.store_type, set.pitch), b, set, a, st);
}

}  // namespace fwi
