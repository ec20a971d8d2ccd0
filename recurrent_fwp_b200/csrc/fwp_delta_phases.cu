// Host side of the three-launch backward of the delta rule: kernels in fwp_delta_phases.cuh.
#include "fwp_delta_phases.cuh"

namespace fwp {

// Workspace of one segment: small enough to stay in the 126 MB L2 cache between the launches.
static constexpr size_t kSegmentBytes = 64u << 20;

struct Segments {
    int nc;                 // chunks per segment
    size_t chunk, carry;    // bytes per chunk and sequence, and of G between segments per sequence
};
template <int E, int M, typename T>
static Segments segments(int nseq, int L) {
    using Sp = wy::BwdSpace<E, M, wy::stream_parts<T>()>;
    Segments s;
    s.chunk = (size_t)Sp::kSize * 16;
    s.carry = (size_t)E * M * 4;
    const int nchunks = (L + wy::C - 1) / wy::C;
    const size_t fit = kSegmentBytes / (s.chunk * (size_t)nseq);
    s.nc = fit >= (size_t)nchunks ? nchunks : fit < 1 ? 1 : (int)fit;
    return s;
}

template <int E, int M, int KG, typename T>
static int run_bwd(const DeltaBwdParams& p, int nseq, float* scratch, cudaStream_t st) {
    constexpr int KS = E / 16, MS = M / 16, NP = wy::stream_parts<T>();
    constexpr int WARPS = E <= 64 ? 4 : 2, DEPTH = E <= 32 ? 4 : 3;
    const Segments sg = segments<E, M, T>(nseq, p.L);
    wy::BwdPhase a;
    a.p = p;
    a.ws = reinterpret_cast<uint4*>(scratch);
    a.carry = a.ws + (size_t)nseq * sg.nc * (sg.chunk / 16);
    a.again = reinterpret_cast<int*>(a.carry + (size_t)nseq * (sg.carry / 16));
    const int nchunks = (p.L + wy::C - 1) / wy::C;
    for (int end = nchunks; end > 0; end -= sg.nc) {
        a.c0 = end > sg.nc ? end - sg.nc : 0;
        a.nc = end - a.c0;
        a.first = end == nchunks;
        const long long units = (long long)nseq * a.nc, tasks = units * ((KS + KG - 1) / KG);
        if ((tasks + WARPS - 1) / WARPS > 0x7fffffffLL) return FWP_ERR_SHAPE;
        int rc = launch_dependent(wy::delta_bwd_prepare_kernel<E, M, WARPS, T>, a, (int)((units + WARPS - 1) / WARPS), WARPS * 32,
                                  WARPS * sizeof(wy::PrepareSmem<E, NP>), st, "delta_bwd_prepare_kernel");
        if (rc) return rc;
        rc = launch_dependent(wy::delta_bwd_chain_kernel<E, M, DEPTH, T>, a, nseq * MS, 64, wy::ChainRing<E, M, DEPTH, T>::kBytes, st,
                              "delta_bwd_chain_kernel");
        if (rc) return rc;
        rc = launch_dependent(wy::delta_bwd_finish_kernel<E, M, KG, WARPS, T>, a, (int)((tasks + WARPS - 1) / WARPS), WARPS * 32, 0, st,
                              "delta_bwd_finish_kernel");
        if (rc) return rc;
    }
    return FWP_OK;
}

// One list of instances for both questions: floats of scratch (run = false), or the launches.
template <int E, int M, int KG, typename T>
static int64_t one(bool run, const DeltaBwdParams& p, int nseq, float* scratch, cudaStream_t st) {
    if (run) return run_bwd<E, M, KG, T>(p, nseq, scratch, st);
    const Segments sg = segments<E, M, T>(nseq, p.L);
    return (int64_t)((sg.chunk * sg.nc + sg.carry + sizeof(int)) / 4 * (size_t)nseq);
}
template <typename T>
int64_t bwd_phases(bool run, const DeltaBwdParams& p, int nseq, float* scratch, cudaStream_t st) {
    const int d = p.E > p.M ? p.E : p.M;
    if (d <= 16) return one<16, 16, 1, T>(run, p, nseq, scratch, st);
    if (d <= 32) return one<32, 32, 2, T>(run, p, nseq, scratch, st);
    if (d <= 48) return one<48, 48, 3, T>(run, p, nseq, scratch, st);
    if (d <= 64) return one<64, 64, 2, T>(run, p, nseq, scratch, st);
    if (p.E <= 32 && p.M <= 112) return one<32, 112, 2, T>(run, p, nseq, scratch, st);
    if (p.E <= 96 && p.M <= 16) return one<96, 16, 3, T>(run, p, nseq, scratch, st);
    if (p.E <= 96 && p.M <= 32) return one<96, 32, 3, T>(run, p, nseq, scratch, st);
    if (p.E <= 96 && p.M <= 64) return one<96, 64, 3, T>(run, p, nseq, scratch, st);
    if (p.E <= 128 && p.M <= 16) return one<128, 16, 2, T>(run, p, nseq, scratch, st);
    if (p.E <= 128 && p.M <= 32) return one<128, 32, 2, T>(run, p, nseq, scratch, st);
    if (p.E <= 128 && p.M <= 64) return one<128, 64, 2, T>(run, p, nseq, scratch, st);
    if (p.E <= 128 && p.M <= 128) return one<128, 128, 2, T>(run, p, nseq, scratch, st);
    return -1;
}
template int64_t bwd_phases<float>(bool, const DeltaBwdParams&, int, float*, cudaStream_t);
template int64_t bwd_phases<__nv_bfloat16>(bool, const DeltaBwdParams&, int, float*, cudaStream_t);

}  // namespace fwp
