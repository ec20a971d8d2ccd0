// Launches of the sum rule's backward as three sum-rule forwards (SumBwdForwards in fwp_delta_wy.cuh).
#include "fwp_delta_wy.cuh"

namespace fwp {

// 1 if a bounded wait of these kernels ran out on the current device since the last call (reading clears it)
int sum_wy_fault_read_clear() { return flag_read_clear(wy::g_wy_fault); }

template <int E, int NB, int CTAS, typename T>
static int run(const wy::SumBwdForwards& a, int nseq, cudaStream_t st) {
    return launch_dependent(wy::sum_bwd_wy_kernel<E, E, NB, CTAS, T, true>, a, dim3(nseq, 3), (E / 16 + NB) * 32,
                            NB * sizeof(wy::FwdBuf<E, wy::stream_parts<T>()>), st, "sum_bwd_wy_kernel");
}
template <int NB, typename T>
static int run_few(const wy::SumBwdForwards& a, int nseq, cudaStream_t st) {
    return launch_dependent(wy::sum_bwd_wy_few_kernel<16, 16, NB, T, true>, a, dim3(nseq, 3), (1 + NB) * 32,
                            NB * sizeof(wy::FewBuf<16, 16, wy::stream_parts<T>()>), st, "sum_bwd_wy_few_kernel");
}
static Row4 reversed(Row4 r, int L, int elem_bytes) {
    r.p = const_cast<char*>(reinterpret_cast<const char*>(r.p) + (L - 1) * r.sL * elem_bytes);
    r.sL = -r.sL;
    return r;
}

// The instances are those of the forward, picked for three times the sequences; -1 where there is none.
template <typename T>
int launch_sum_bwd_wy(const SumBwdParams& p, int nseq, cudaStream_t st) {
    wy::SumBwdForwards a = {};
    const int eb = sizeof(T);
    auto set = [&](int i, const Row4& q, const Row4& k, const Row4& v, const Row4& out, int E, int M) {
        DeltaFwdParams& f = a.p[i];
        f.q = q; f.k = k; f.v = v; f.out = out;
        f.H = p.H; f.L = p.L; f.E = E; f.M = M; f.NH = p.NH;
    };
    auto rev = [&](const Row4& r) { return reversed(r, p.L, eb); };
    set(0, p.gy, p.v, p.k, p.gq, p.M, p.E);
    set(1, rev(p.k), rev(p.q), rev(p.gy), rev(p.gv), p.E, p.M);
    set(2, rev(p.v), rev(p.gy), rev(p.q), rev(p.gk), p.M, p.E);
    const int d = p.E > p.M ? p.E : p.M, chains = 3 * nseq, sms = sm_count();
    if (d <= 16) {
        if constexpr (sizeof(T) == 4) {
            const bool few = p.E == 16 && p.M == 16 && p.L >= 7 * wy::C;
            if (few && chains <= sms) return run_few<6, T>(a, nseq, st);
            if (few && chains <= 2 * sms) return run_few<4, T>(a, nseq, st);
        }
        return run<16, 2, 5, T>(a, nseq, st);
    }
    if (d <= 32) return chains <= 2 * sms ? run<32, 4, 2, T>(a, nseq, st) : run<32, 2, 4, T>(a, nseq, st);
    if (d <= 48) return chains <= sms ? run<48, 4, 1, T>(a, nseq, st) : run<48, 4, 2, T>(a, nseq, st);
    if (d <= 64) return chains <= sms ? run<64, 4, 1, T>(a, nseq, st) : run<64, 4, 2, T>(a, nseq, st);
    return -1;
}
template int launch_sum_bwd_wy<float>(const SumBwdParams&, int, cudaStream_t);
template int launch_sum_bwd_wy<__nv_bfloat16>(const SumBwdParams&, int, cudaStream_t);

}  // namespace fwp
