// Kernel parameter blocks of the delta rule, shared by the translation units that hold its plans.
#pragma once
#include "fwp_core.cuh"

namespace fwp {

struct DeltaFwdParams {
    Row4 q, k, v, beta, v_old, v_ins, out;
    float* W; long long wN, wH, wE;
    int H, L, E, M;
    int NH;     // number of sequences (N*H)
};

struct DeltaBwdParams {
    Row4 q, k, v, beta, v_old, gy, gq, gk, gv, gb;
    float* W; long long wN, wH, wE;
    int H, L, E, M;
    int NH;     // number of sequences (N*H)
    int bulk = 1;           // stage contiguous chunks with bulk copies where the kernel supports it
};

struct SumBwdParams {
    Row4 q, k, v, gy, gq, gk, gv;
    int H, L, E, M;
    int NH;     // number of sequences (N*H)
};

// chunkwise plan for bf16 streams with E = M = 64 (fwp_delta_chunk_bf16.cuh): applies when every row is 16-byte aligned
bool chunk_bf16_applies(const DeltaFwdParams& p);
int launch_fwd_chunk_bf16(const DeltaFwdParams& p, int nseq, cudaStream_t st);
bool chunk_bf16_applies(const DeltaBwdParams& p);
int launch_bwd_chunk_bf16(const DeltaBwdParams& p, int nseq, cudaStream_t st);
// chunkwise plan on split fp32 products (fwp_delta_wy.cuh); -1 when the sizes have no instance
int wy_fault_read_clear();
int wy_few_fault_read_clear();
int sum_wy_fault_read_clear();
// its form for few sequences, fp32; -1 where the other is the better one or has the only instance
template <bool SUM> int launch_fwd_wy_few(const DeltaFwdParams& p, int nseq, cudaStream_t st);
template <typename T, bool SUM> int launch_fwd_wy(const DeltaFwdParams& p, int nseq, cudaStream_t st);
// three-launch backward over a workspace (fwp_delta_phases.cuh): floats of scratch it needs (run = false) or the launches; -1
// when the sizes have no instance
template <typename T> int64_t bwd_phases(bool run, const DeltaBwdParams& p, int nseq, float* scratch, cudaStream_t st);
static inline bool rows_16B_aligned(const DeltaBwdParams& p) {        // of fp32 streams
    return rows_16B_aligned(p.k) && rows_16B_aligned(p.q) && rows_16B_aligned(p.v) && rows_16B_aligned(p.v_old) && rows_16B_aligned(p.gy);
}
// step by step over four warps a sequence, E = M = 32, fp32 streams (fwp_delta_tile.cuh)
int launch_bwd_tile32(const DeltaBwdParams& p, int nseq, cudaStream_t st);
int tc_fault_read_clear();
int launch_wait_probe(int polls, cudaStream_t st);
// the sum rule's backward as three forwards of the plan above; -1 when the sizes have no instance
template <typename T> int launch_sum_bwd_wy(const SumBwdParams& p, int nseq, cudaStream_t st);

}  // namespace fwp
