// Host side of the three-launch backward of the delta rule: kernels in fwp_delta_phases.cuh.
#include "fwp_delta_phases.cuh"

namespace fwp {

// Bound on the workspace: small enough to stay in the 126 MB L2 cache between the launches.
static constexpr size_t kWorkspaceBytes = 64u << 20;
// A call larger than that is cut into segments of time and, where not even one chunk of all its sequences fits, into
// groups of sequences that fit with kGroupChunks chunks each: fewer make the chain kernels' launches short, more leave them
// short of sequences.  Training pass of 1024 sequences x 256 steps, ms at 1 / 2 / 4 / 8 / 16 chunks (all sequences together at one
// chunk each, 180 MB of workspace: in brackets): E, M = 128, 128 7.6 / 5.7 / 5.8 / 5.9 / 6.0 (6.5), bf16 8.9 / 7.8 / 6.7 / 6.7 / 6.6
// (7.4); 128, 64 4.0 / 3.1 / 2.9 / 2.7 / 3.3 (3.7); 2048 x 96, 64 5.7 / 4.8 / 4.4 / 4.5 / 4.6 (5.7).
static constexpr int kGroupChunks = 4;
struct Cut {
    int ns, nc;                 // sequences per group, chunks per segment
    size_t chunk, carry;        // bytes per sequence: of a chunk, and of G between segments
    size_t bytes() const { return (chunk * nc + carry + sizeof(int)) * ns; }
};
template <int E, int M, typename T>
static Cut cut(int nseq, int L) {
    using Sp = wy::BwdSpace<E, M, wy::stream_parts<T>()>;
    Cut s;
    s.chunk = (size_t)Sp::kSize * 16;
    s.carry = (size_t)E * M * 4;
    const size_t nchunks = (L + wy::C - 1) / wy::C, fixed = s.carry + sizeof(int);
    auto fit = [&](size_t n) { const size_t each = kWorkspaceBytes / n; return each < fixed + s.chunk ? 0 : (each - fixed) / s.chunk; };
    size_t ns = nseq;
    if (!fit(ns)) {
        const size_t most = kWorkspaceBytes / (fixed + s.chunk * (nchunks < kGroupChunks ? nchunks : kGroupChunks)), groups = (nseq + most - 1) / most;
        ns = (nseq + groups - 1) / groups;
    }
    s.ns = (int)ns;
    s.nc = (int)(fit(ns) < nchunks ? fit(ns) : nchunks);
    return s;
}

template <int E, int M, int KG, typename T>
static int run_bwd(const DeltaBwdParams& p, int nseq, float* scratch, cudaStream_t st) {
    constexpr int KS = E / 16, MS = M / 16, NP = wy::stream_parts<T>();
    constexpr int WARPS = E <= 64 ? 4 : 2, DEPTH = E <= 32 ? 4 : 3;
    const Cut sg = cut<E, M, T>(nseq, p.L);
    wy::BwdPhase a;
    a.p = p;
    a.ws = reinterpret_cast<uint4*>(scratch);
    a.carry = a.ws + (size_t)sg.ns * sg.nc * (sg.chunk / 16);
    a.again = reinterpret_cast<int*>(a.carry + (size_t)sg.ns * (sg.carry / 16));
    const int nchunks = (p.L + wy::C - 1) / wy::C;
    for (a.s0 = 0; a.s0 < nseq; a.s0 += sg.ns) {
        a.ns = nseq - a.s0 < sg.ns ? nseq - a.s0 : sg.ns;
        for (int end = nchunks; end > 0; end -= sg.nc) {
            a.c0 = end > sg.nc ? end - sg.nc : 0;
            a.nc = end - a.c0;
            a.first = end == nchunks;
            const int units = a.ns * a.nc, tasks = units * ((KS + KG - 1) / KG);    // bounded by the workspace that holds them
            int rc = launch_dependent(wy::delta_bwd_prepare_kernel<E, M, WARPS, T>, a, (units + WARPS - 1) / WARPS, WARPS * 32,
                                      WARPS * sizeof(wy::PrepareSmem<E, NP>), st, "delta_bwd_prepare_kernel");
            if (rc) return rc;
            rc = launch_dependent(wy::delta_bwd_chain_kernel<E, M, DEPTH, T>, a, a.ns * MS, 64, wy::ChainRing<E, M, DEPTH, T>::kBytes, st,
                                  "delta_bwd_chain_kernel");
            if (rc) return rc;
            rc = launch_dependent(wy::delta_bwd_finish_kernel<E, M, KG, WARPS, T>, a, (tasks + WARPS - 1) / WARPS, WARPS * 32, 0, st,
                                  "delta_bwd_finish_kernel");
            if (rc) return rc;
        }
    }
    return FWP_OK;
}

// One list of instances for both questions: floats of scratch (run = false), or the launches.
template <int E, int M, int KG, typename T>
static int64_t one(bool run, const DeltaBwdParams& p, int nseq, float* scratch, cudaStream_t st) {
    if (run) return run_bwd<E, M, KG, T>(p, nseq, scratch, st);
    return (int64_t)(cut<E, M, T>(nseq, p.L).bytes() / 4);
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
