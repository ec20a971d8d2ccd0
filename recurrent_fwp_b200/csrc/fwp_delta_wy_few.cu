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
    // Up to one sequence per SM, evaluation, time of this form over the other's (packed rows, rows as layers slice them; 1 to 148 sequences):
    //   E = M = 32     96 steps 1.00-1.05, 112 0.96-1.02, 128 0.91-0.98, 256 0.84-0.90
    //   other sizes up to 32 (17, 20, 24; 25, 31; 16, 32; 32, 12)   112 1.00-1.12, 120 0.94-1.02, 128 0.94-1.03, 160 0.90-1.00, 256 0.84-0.94
    //   E up to 96, M = 12, 16     128 0.71-0.96, 144 0.66-0.92, 384 0.52-0.88
    //   E, M = 66, 32; 77, 30; 80, 32; 96, 20; 96, 32, from 144 steps: up to 64 sequences 0.99-1.19, 96 0.89-1.07, 128 0.76-0.97, 148 0.70-0.93.
    //     There the other form's loops, unrolled, are fetched by many SMs at once; with few it has the shorter chunk
    // Buffers of larger sizes leave too few helpers: 128 x 256, d = 48 51 -> 78 us, 64 63 -> 88, E, M = 128, 32 64 -> 78
    if constexpr (!SUM) {
        const int sms = sm_count(), least = d > 32 ? 9 * wy::C : p.E == 32 && p.M == 32 ? 7 * wy::C : 7 * wy::C + 1;
        if (force ? force != 6 : nseq > sms || p.L < least) return -1;
        if (d <= 32) return run_fwd_few<32, 32, 6, 1, SUM>(p, nseq, st);
        if (d <= 64 || d > 96 || p.M > 32) return -1;
        if (p.M <= 16) return run_fwd_few<96, 16, 3, 1, SUM>(p, nseq, st);
        if (force || nseq >= sms * 3 / 4) return run_fwd_few<96, 32, 3, 1, SUM>(p, nseq, st);
    }
    return -1;
}
template int launch_fwd_wy_few<false>(const DeltaFwdParams&, int, cudaStream_t);
template int launch_fwd_wy_few<true>(const DeltaFwdParams&, int, cudaStream_t);

}  // namespace fwp
