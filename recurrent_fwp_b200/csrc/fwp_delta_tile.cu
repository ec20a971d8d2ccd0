// Launch of the delta rule's tiled step-by-step backward: kernel in fwp_delta_tile.cuh.
#include "fwp_delta_tile.cuh"

namespace fwp {

int launch_bwd_tile32(const DeltaBwdParams& p, int nseq, cudaStream_t st) {
    constexpr int TC = 8;
    const int slots = spread_slots(4, nseq);
    const size_t bytes = (size_t)DeltaTileSmem<TC>::kFloats * sizeof(float) * slots;
    const bool aligned = rows_16B_aligned(p);
    const auto kern = slots == 4 ? (aligned ? delta_bwd_tile32_kernel<TC, 4, false> : delta_bwd_tile32_kernel<TC, 4, true>)
                                 : (aligned ? delta_bwd_tile32_kernel<TC, 2, false> : delta_bwd_tile32_kernel<TC, 2, true>);
    return launch_dependent(kern, p, nseq / slots, 128 * slots, bytes, st, "delta_bwd_tile32_kernel");
}

}  // namespace fwp
