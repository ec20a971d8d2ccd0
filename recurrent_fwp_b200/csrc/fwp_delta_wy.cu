// Launches of the chunkwise (WY) plan of the delta and sum rules: kernels in fwp_delta_wy.cuh.
#include "fwp_delta_wy.cuh"

namespace fwp {

// 1 if a bounded wait of these kernels ran out on the current device since the last call (reading clears it)
int wy_fault_read_clear() { return flag_read_clear(wy::g_wy_fault); }

template <int E, int M, int NB, int CTAS, typename T, bool SUM>
static int run_fwd(const DeltaFwdParams& p, int nseq, cudaStream_t st) {
    return launch_dependent(wy::delta_fwd_wy_kernel<E, M, NB, CTAS, T, SUM>, p, nseq, (M / 16 + NB) * 32,
                            NB * sizeof(wy::FwdBuf<E, wy::stream_parts<T>()>), st, "delta_fwd_wy_kernel");
}
// How many preparing warps a sequence gets and how many sequences an SM holds.  With no more sequences than SMs
// (FEW_CTAS = 1; two per SM where registers and shared memory allow it without spilling) four warps keep a chain
// supplied; with more, shared latency replaces them and residency counts.
template <int E, int M, int FEW_CTAS, int MANY_HELPERS, int MANY_CTAS, typename T, bool SUM>
static int pick_fwd(const DeltaFwdParams& p, int nseq, cudaStream_t st) {
    const int force = tune_get(T_DELTA_WY_HELPERS, 0);
    if (force ? force == 4 : nseq <= FEW_CTAS * sm_count()) return run_fwd<E, M, 4, FEW_CTAS, T, SUM>(p, nseq, st);
    return run_fwd<E, M, MANY_HELPERS, MANY_CTAS, T, SUM>(p, nseq, st);
}

// Head sizes are padded to the next instance; a state that is much wider one way keeps its own two sizes.
template <typename T, bool SUM>
int launch_fwd_wy(const DeltaFwdParams& p, int nseq, cudaStream_t st) {
    const int d = p.E > p.M ? p.E : p.M;
    if constexpr (sizeof(T) == 4) {
        const int rc = launch_fwd_wy_few<SUM>(p, nseq, st);
        if (rc >= 0) return rc;
    }
    if (d <= 16) {
        return run_fwd<16, 16, 2, 5, T, SUM>(p, nseq, st);
    }
    if (d <= 32) return pick_fwd<32, 32, 2, 2, 4, T, SUM>(p, nseq, st);
    if (d <= 48) return pick_fwd<48, 48, 1, 4, 2, T, SUM>(p, nseq, st);
    if (d <= 64) return pick_fwd<64, 64, 1, 4, 2, T, SUM>(p, nseq, st);
    if (p.E <= 32 && p.M <= 112) return run_fwd<32, 112, 4, 1, T, SUM>(p, nseq, st);
    if (p.E <= 96 && p.M <= 16) return pick_fwd<96, 16, 1, 4, 2, T, SUM>(p, nseq, st);
    if (p.E <= 96 && p.M <= 32) return pick_fwd<96, 32, 1, 4, 2, T, SUM>(p, nseq, st);
    if (p.E <= 96 && p.M <= 64) return run_fwd<96, 64, 4, 1, T, SUM>(p, nseq, st);
    if (p.E <= 128 && p.M <= 16) return pick_fwd<128, 16, 1, 4, 2, T, SUM>(p, nseq, st);
    if (p.E <= 128 && p.M <= 32) return pick_fwd<128, 32, 1, 4, 2, T, SUM>(p, nseq, st);
    if (p.E <= 128 && p.M <= 64) return run_fwd<128, 64, 4, 1, T, SUM>(p, nseq, st);
    if (p.E <= 128 && p.M <= 128) return run_fwd<128, 128, 4, 1, T, SUM>(p, nseq, st);
    return -1;
}
template int launch_fwd_wy<float, false>(const DeltaFwdParams&, int, cudaStream_t);
template int launch_fwd_wy<float, true>(const DeltaFwdParams&, int, cudaStream_t);
template int launch_fwd_wy<__nv_bfloat16, false>(const DeltaFwdParams&, int, cudaStream_t);
template int launch_fwd_wy<__nv_bfloat16, true>(const DeltaFwdParams&, int, cudaStream_t);

}  // namespace fwp
