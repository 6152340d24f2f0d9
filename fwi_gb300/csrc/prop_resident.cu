// Launches of the resident path (prop_resident.cuh): one cooperative launch per set of shots.  The
// reference-mode adjoint's kernels are in prop_resident_ref.cu.
#include <mutex>

#include "prop_resident.cuh"

namespace fwi {

namespace {

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
ResKernel<ResFwdArgs> fwd_kernel(int store_type, int pitch)
{
    return store_type == kStoreHalf ? fwd_kernel<kStoreHalf>(pitch)
           : store_type == kStoreBf16 ? fwd_kernel<kStoreBf16>(pitch) : fwd_kernel<kStoreNative>(pitch);
}

}  // namespace

bool resident_allow_ref(int smem);  // prop_resident_ref.cu

// fwi_check_bounded_wait, the resident kernels' wait: a pair of words that nothing writes is polled, given up
// after `polls`, and the status word says so; the waits after it end at their first poll.
__device__ __align__(16) uint64_t g_unwritten[2];
__global__ void k_check_resident_wait(unsigned *status, long polls, int *waits)
{
    __shared__ int dead;
    if (threadIdx.x == 0) dead = 0;
    __syncthreads();
    for (int w = 0; w < 2; w++) {
        int k = 0;
        for (ResPair q;; k++) {
            q.load(g_unwritten);
            if (q.is(1) || res_give_up(k, &dead, status, polls)) break;
        }
        __syncthreads();
        if (threadIdx.x == 0) waits[w] = k;
    }
}
cudaError_t launch_resident_wait_check(unsigned *status, long polls, int *waits, cudaStream_t st)
{
    k_check_resident_wait<<<1, 128, 0, st>>>(status, polls, waits);
    return cudaGetLastError();
}

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
    ok = ok && res_allow([](int st, int p) { return fwd_kernel(st, p); }, lim) &&
         res_allow([](int st, int p) { return res_adj_kernel<false>(st, p); }, lim) && resident_allow_ref(lim);
    if (!ok) cudaGetLastError();
    limit[dev] = ok ? (size_t)lim : 0;
    done[dev] = true;
    return limit[dev];
}

cudaError_t launch_resident_forward(const Batch<float> &b, const ResidentSet &set, const ResFwdArgs &a, cudaStream_t st)
{
    return res_launch(fwd_kernel(b.store_type, set.pitch), b, set, a, st);
}

cudaError_t launch_resident_adjoint(const Batch<float> &b, const ResidentSet &set, const ResAdjArgs &a, cudaStream_t st)
{
    return res_launch(res_adj_kernel<false>(b.store_type, set.pitch), b, set, a, st);
}

}  // namespace fwi
