// The reference-mode adjoint on the resident path (prop_resident.cuh).
#include "prop_resident.cuh"

namespace fwi {

bool resident_allow_ref(int smem)
{
    return res_allow([](int st, int p) { return res_adj_kernel<true>(st, p); }, smem);
}

cudaError_t launch_resident_ref_adjoint(const Batch<float> &b, const ResidentSet &set, const ResAdjArgs &a, cudaStream_t st)
{
    return res_launch(res_adj_kernel<true>(b.store_type, set.pitch), b, set, a, st);
}

}  // namespace fwi
