// nbl_trav_fill64.cu -- the fill pass (with the plain FP64 test),
// every launch shape (warps per CTA x cutoff kind).
#include "nbl_traverse.cuh"

namespace nbl {
namespace {

template <int K, int W>
TravKernel pick_w(size_t &smem) {
    smem = fill_smem_bytes<false>(W);
    return k_fill<false, K, false, W, false>;
}

template <int K>
TravKernel pick_k(const TravShape &s, size_t &smem) {
    if (s.warps == 2) return pick_w<K, 2>(smem);
    if (s.warps == 8) return pick_w<K, 8>(smem);
    return pick_w<K, 4>(smem);
}

TravKernel kernel_for(int kind, const TravShape &s, size_t &smem) {
    if (kind == kCutPerAtom) return pick_k<kCutPerAtom>(s, smem);
    if (kind == kCutPerType) return pick_k<kCutPerType>(s, smem);
    return pick_k<kCutScalar>(s, smem);
}

}  // namespace

cudaError_t launch_fill_fp64(int kind, const TraverseArgs &a, int grid, cudaStream_t st,
                             const TravShape &shape) {
    size_t smem = 0;
    const TravKernel k = kernel_for(kind, shape, smem);
    return launch_kernel(k, smem, shape.warps, a, grid, st);
}

int occupancy_fill_fp64(int kind, const TravShape &shape) {
    size_t smem = 0;
    const TravKernel k = kernel_for(kind, shape, smem);
    return occupancy_kernel(k, smem, shape.warps);
}

}  // namespace nbl
