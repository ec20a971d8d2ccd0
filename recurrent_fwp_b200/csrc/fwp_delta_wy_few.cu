// Launches of the chunkwise (WY) forward for few sequences, fp32: kernels in fwp_delta_wy.cuh.
#include "fwp_delta_wy.cuh"

namespace fwp {

// 1 if a bounded wait of these kernels ran out on the current device since the last call (reading clears it)
int wy_few_fault_read_clear() { return flag_read_clear(wy::g_wy_fault); }

template <int E, int M, int NB, int CTAS, bool SUM>
static int run_fwd_few(const DeltaFwdParams& p, int nseq, cudaStream_t st) {
    return launch_dependent(wy::delta_fwd_wy_few_kernel<E, M, NB, CTAS, float, SUM>, p, nseq, (M / 16 + NB) * 32, NB * sizeof(wy::FewBuf<E, M, 3>),
                            st, "delta_fwd_wy_few_kernel");
}

template <bool SUM>
int launch_fwd_wy_few(const DeltaFwdParams& p, int nseq, cudaStream_t st) {
    const int d = p.E > p.M ? p.E : p.M, force = tune_get(T_DELTA_WY_HELPERS, 0);
    if (d <= 16) {
        // at d = 16 a chain waits more than it works: up to two sequences per SM the form with the short chain wins once
        // its longer start (about 5 us) is paid for: 11.6 against 14.5 us at 16 sequences of 256 steps, 7.7 against 3.9 at 20 steps
        const bool few = force ? force == 4 : p.E == 16 && p.M == 16 && p.L >= 7 * wy::C;
        if (few && nseq <= sm_count()) return run_fwd_few<16, 16, 6, 2, SUM>(p, nseq, st);
        if (few && (force || nseq <= 2 * sm_count())) return run_fwd_few<16, 16, 4, 2, SUM>(p, nseq, st);
        return -1;
    }
    // One sequence per SM (evaluation, us; the other form -> this one): d = 32, 64 sequences: 20 steps 8.4 -> 9.9, 64 10.4 -> 10.6, 112 13.2 -> 12.7,
    // 512 41 -> 31; 40 x 243, rows of 20 in any layout 26.8 -> 22.9; 144 x 512, rows of 24 46 -> 40.  E, M = 96, 32, 128 x 256: 64 -> 50; 80, 32 64 -> 50;
    // 77, 32 64 -> 57; 80, 32 x 64 18.7 -> 20.7, x 128 28.9 -> 28.9; 96, 16 52 -> 41.  Buffers of larger sizes leave too few helpers: d = 48 51 -> 78,
    // 64 63 -> 88, E, M = 128, 32 64 -> 78
    if constexpr (!SUM) {
        const bool few = force ? force == 6 : nseq <= sm_count();
        if (d <= 32 && few && (force || p.L >= 7 * wy::C)) return run_fwd_few<32, 32, 6, 1, SUM>(p, nseq, st);
        if (d > 64 && d <= 96 && p.M <= 32 && few && (force || p.L >= 9 * wy::C))
            return p.M <= 16 ? run_fwd_few<96, 16, 3, 1, SUM>(p, nseq, st) : run_fwd_few<96, 32, 3, 1, SUM>(p, nseq, st);
    }
    return -1;
}
template int launch_fwd_wy_few<false>(const DeltaFwdParams&, int, cudaStream_t);
template int launch_fwd_wy_few<true>(const DeltaFwdParams&, int, cudaStream_t);

}  // namespace fwp
