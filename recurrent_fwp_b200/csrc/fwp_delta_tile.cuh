// Delta rule backward at E = M = 32, fp32 streams, step by step with the work of a sequence over four warps (sm_100a).
//
// Time reversed, a step is
//   G += q (x) gy;  r = G^T k;  dv = beta r;  dbeta = r . w;  dq = S gy;  S -= k (x) u;  dk = G u - S dv;  G -= k (x) dv
// with w = v - v_old and u = beta w.  Only G and dv go round from step to step; what S takes part in follows.
//   warps A0, A1    sixteen columns of G each, pieces of eight rows and two columns per lane: r, the G part of dk.  Columns do not
//                   meet, so the two never wait for one another;
//   warps B0, B1    one chunk of steps behind, sixteen rows of S each, pieces of four rows and four columns: dq, the S part of dk,
//                   the rewind, dv and dbeta.  And one chunk ahead they turn v and v_old of a chunk into w and -u.
// The four meet once per chunk of eight steps.  A lane reads 4 to 8 operands per product where a line per lane takes 32; its sums
// over other lanes are reduce-scatters.  Bound by the latency of an A step with one sequence per SM (39 us for 128 sequences x
// 256 steps, 75 for x 512), by issue and shared memory with more (256 x 512: 101 us; 512 x 256: 88).  The four-step blocked kernel took
// 66, 126, 132 and 136 us.  Other splits were slower where it counts: G over four warps or S over four 11 and 22 % (128 and 512 x
// 256), three chunks in flight instead of one the same.
#pragma once
#include "fwp_delta_params.cuh"
#include "fwp_trail.cuh"

namespace fwp {

template <int TC>
struct DeltaTileSmem {
    static constexpr int D = 32;
    static constexpr int kStage = 5 * TC * D + r4(TC);      // k, q, v (then w), v_old (then -u), gy; beta
    static constexpr int kStages = 4;                       // chunk j + 1 in flight, w and -u of j, A on j - 1, B on j - 2
    static constexpr int kR = TC * D;                       // r of a chunk
    static constexpr int kDk = 2 * TC * D;                  // -G u in two parts
    static constexpr int kTable = (sizeof(StageTable) + 15) / 16 * 4;
    static constexpr int kFloats = kStages * kStage + 2 * (kR + kDk) + kTable;
};

template <int TC, int SLOTS, bool WORDS>
__global__ void __launch_bounds__(128 * SLOTS, 1) delta_bwd_tile32_kernel(const __grid_constant__ DeltaBwdParams p) {
    constexpr int D = 32, NT = 128;
    using SM = DeltaTileSmem<TC>;
    const int nslots = blockDim.x / NT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp % nslots, role = warp / nslots;       // 0, 1: A; 2, 3: B
    const int stid = role * 32 + lane;
    const int seq = blockIdx.x * nslots + slot;
    const int n = seq / p.H, h = seq - n * p.H;
    extern __shared__ __align__(16) float smem_all[];
    float* smem = smem_all + (size_t)slot * SM::kFloats;
    float* const rss = smem + SM::kStages * SM::kStage;     // [chunk parity] each
    float* const dks = rss + 2 * SM::kR;
    StageTable* tb = reinterpret_cast<StageTable*>(dks + 2 * SM::kDk);
    griddep_wait();               // launched as a dependent: global memory is touched from here on
    griddep_launch_dependents();
    if (stid == 0) {
        stage_table_set(tb, 0, p.k, n, h);
        stage_table_set(tb, 1, p.q, n, h);
        stage_table_set(tb, 2, p.v, n, h);
        stage_table_set(tb, 3, p.v_old, n, h);
        stage_table_set(tb, 4, p.gy, n, h);
        stage_table_set_col(tb, 0, p.beta, n, h);
    }
    slot_barrier(slot, NT);
    const int nchunks = (p.L + TC - 1) / TC;
    RowStager<TC, 4, 5, WORDS> rows_in(tb, (nchunks - 1) * TC, stid);
    auto issue = [&](int j) {           // called for j = 0, 1, 2, ...
        rows_in.issue(smem + (j % SM::kStages) * SM::kStage, min(TC, p.L - (nchunks - 1 - j) * TC));
    };
    auto advance = [&](int j) {
        cp_async_wait<0>();
        slot_barrier(slot, NT);
        if (j + 1 < nchunks) issue(j + 1);
    };
    issue(0);
    auto stream = [&](const Row4& r) { return reinterpret_cast<float*>(r.p) + n * r.sN + h * r.sH; };

    if (role < 2) {
        // ---------------------------------------------------------------- A: G
        // lane (eg, mg) = (lane >> 3, lane & 7): rows 8 eg .. 8 eg + 7 (the four that it keeps in a sum over columns first), columns
        // 16 role + 2 mg, + 1.  r of column `own` comes out in two lanes.
        const int row0 = 8 * (lane >> 3) + (lane & 4), row1 = row0 ^ 4, col = 16 * role + 2 * (lane & 7), own = col + (lane >> 4);
        const bool b4 = lane & 16, b1 = lane & 2, b0 = lane & 1;
        f2 G[2][4];
#pragma unroll
        for (int i = 0; i < 4; i++) { G[0][i] = 0ull; G[1][i] = 0ull; }
        for (int j = 0; j <= nchunks + 1; j++) {
            advance(j);
            if (j == 0 || j > nchunks) continue;
            const float* st = smem + ((j - 1) % SM::kStages) * SM::kStage;
            const float *ks = st, *qs = st + TC * D, *us = st + 3 * TC * D + col, *ys = st + 4 * TC * D + col, *bs = st + 5 * TC * D;
            const int nt = min(TC, p.L - (nchunks - j) * TC), par = (j - 1) & 1;
            float* const rp = rss + par * SM::kR;
            float* const dkp = dks + par * SM::kDk + role * TC * D + lane;
#pragma unroll TC
            for (int t = nt - 1; t >= 0; t--) {
                auto rows = [&](f2 (&x)[4], const float* at) {
                    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(at + t * D + row0), b = *reinterpret_cast<const ulonglong2*>(at + t * D + row1);
                    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
                };
                f2 q[4], k[4], x[4];
                rows(q, qs);
                rows(k, ks);
                const float2 y2 = *reinterpret_cast<const float2*>(ys + t * D), u2 = *reinterpret_cast<const float2*>(us + t * D);
                const f2 y[2] = {f2_dup(y2.x), f2_dup(y2.y)}, u[2] = {f2_dup(u2.x), f2_dup(u2.y)};
                const float nb = -bs[t];
                float rr[2];
#pragma unroll
                for (int c = 0; c < 2; c++) {
#pragma unroll
                    for (int i = 0; i < 4; i++) G[c][i] = ffma2(q[i], y[c], G[c][i]);
                    rr[c] = f2_hsum(fadd2(ffma2(G[c][2], k[2], fmul2(G[c][0], k[0])), ffma2(G[c][3], k[3], fmul2(G[c][1], k[1]))));
                }
                float r = (b4 ? rr[1] : rr[0]) + __shfl_xor_sync(0xffffffffu, b4 ? rr[0] : rr[1], 16);
                r += __shfl_xor_sync(0xffffffffu, r, 8);
                rp[t * D + own] = r;
#pragma unroll
                for (int i = 0; i < 4; i++) x[i] = ffma2(G[1][i], u[1], fmul2(G[0][i], u[0]));
                __syncwarp();
                const float2 d2 = *reinterpret_cast<const float2*>(rp + t * D + col);
                const f2 d[2] = {f2_dup(nb * d2.x), f2_dup(nb * d2.y)};         // -dv
#pragma unroll
                for (int c = 0; c < 2; c++)
#pragma unroll
                    for (int i = 0; i < 4; i++) G[c][i] = ffma2(k[i], d[c], G[c][i]);
                x[0] = fadd2(x[0], shfl_xor2(x[2], 4));
                x[1] = fadd2(x[1], shfl_xor2(x[3], 4));
                const f2 sum = fadd2(b1 ? x[1] : x[0], shfl_xor2(b1 ? x[0] : x[1], 2));
                float lo, hi;
                f2_unpack(sum, lo, hi);
                dkp[t * D] = (b0 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b0 ? lo : hi, 1);
            }
        }
        return;
    }
    // -------------------------------------------------------------------- B: S
    // lane (rg, mg) = (lane >> 3, lane & 7): rows 16 part + 4 rg .. + 3 (the pair that it keeps first), columns 2 mg, + 1 and
    // 16 + 2 mg, + 1 in pairs.  Of the two lanes that end up with a row one stores dq, the other dk.
    const int part = role - 2, mg = lane & 7, row0 = 16 * part + 4 * (lane >> 3) + ((lane >> 1) & 2), row1 = row0 ^ 2;
    const bool b0 = lane & 1, b1 = lane & 2;
    const int own = row0 + ((lane >> 1) & 1);
    float* const W = p.W + n * p.wN + h * p.wH;
    auto at = [&](int i, int c) { return W + (long long)((i < 2 ? row0 : row1) + (i & 1)) * p.wE + 2 * mg + 16 * c; };
    f2 S[4][2];                 // [row][pair of columns]
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < 2; c++) S[i][c] = f2_pack(at(i, c)[0], at(i, c)[1]);
    const long long last = p.L - 1, sg = b0 ? p.gk.sL : p.gq.sL;
    float* pg = (b0 ? stream(p.gk) : stream(p.gq)) + own + last * sg;
    float* const pgv = stream(p.gv) + lane;
    float* const pgb = stream(p.gb);
    for (int j = 0; j <= nchunks + 1; j++) {
        advance(j);
        if (j < nchunks) {                          // w and -u of the chunk that A takes next
            float* const st = smem + (j % SM::kStages) * SM::kStage;
            float *vs = st + 2 * TC * D + lane, *os = st + 3 * TC * D + lane;
            const float* bs = st + 5 * TC * D;
            const int nt = min(TC, p.L - (nchunks - 1 - j) * TC);
#pragma unroll
            for (int i = 0; i < TC / 2; i++) {
                const int t = 2 * i + part;
                if (t < nt) {
                    const float w = vs[t * D] - os[t * D];
                    vs[t * D] = w;
                    os[t * D] = -bs[t] * w;
                }
            }
        }
        if (j < 2) continue;
        const float* st = smem + ((j - 2) % SM::kStages) * SM::kStage;
        const float *ks = st, *ws = st + 2 * TC * D, *us = st + 3 * TC * D + 2 * mg, *ys = st + 4 * TC * D + 2 * mg, *bs = st + 5 * TC * D;
        const int t0 = (nchunks + 1 - j) * TC, nt = min(TC, p.L - t0), par = j & 1;
        const float* const rp = rss + par * SM::kR;
        const float* const dkp = dks + par * SM::kDk + own;
#pragma unroll TC
        for (int t = nt - 1; t >= 0; t--) {
            auto cols = [&](f2 (&x)[2], const float* src) {
                x[0] = *reinterpret_cast<const f2*>(src + t * D);
                x[1] = *reinterpret_cast<const f2*>(src + t * D + 16);
            };
            const float2 k0 = *reinterpret_cast<const float2*>(ks + t * D + row0), k1 = *reinterpret_cast<const float2*>(ks + t * D + row1);
            const f2 k[4] = {f2_dup(k0.x), f2_dup(k0.y), f2_dup(k1.x), f2_dup(k1.y)}, nb = f2_dup(-bs[t]);
            f2 y[2], u[2], d[2];
            cols(y, ys);
            cols(u, us);
            cols(d, rp + 2 * mg);
            d[0] = fmul2(d[0], nb);                     // -dv
            d[1] = fmul2(d[1], nb);
            float dq[4], ds[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                dq[i] = f2_hsum(ffma2(S[i][1], y[1], fmul2(S[i][0], y[0])));
                S[i][0] = ffma2(u[0], k[i], S[i][0]);           // S_{t-1}
                S[i][1] = ffma2(u[1], k[i], S[i][1]);
                ds[i] = f2_hsum(ffma2(S[i][1], d[1], fmul2(S[i][0], d[0])));
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                dq[i] += __shfl_xor_sync(0xffffffffu, dq[i + 2], 4);
                ds[i] += __shfl_xor_sync(0xffffffffu, ds[i + 2], 4);
            }
            // one lane of a pair goes on with dq, the other with dk
            const float g0 = (b0 ? ds[0] : dq[0]) + __shfl_xor_sync(0xffffffffu, b0 ? dq[0] : ds[0], 1);
            const float g1 = (b0 ? ds[1] : dq[1]) + __shfl_xor_sync(0xffffffffu, b0 ? dq[1] : ds[1], 1);
            float g = (b1 ? g1 : g0) + __shfl_xor_sync(0xffffffffu, b1 ? g0 : g1, 2);
            const float kg = dkp[t * D] + dkp[(TC + t) * D];
            g -= b0 ? kg : 0.f;
            *pg = g;
            pg -= sg;
        }
        // dv and dbeta = r . w of half the chunk's steps: eight lanes to a step of dbeta
        static_assert(TC == 8, "four steps of a chunk to a warp");
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int t = 4 * part + i;
            if (t < nt) pgv[(t0 + t) * p.gv.sL] = bs[t] * rp[t * D + lane];
        }
        const int t = 4 * part + (lane >> 3);
        const float4 r4 = *reinterpret_cast<const float4*>(rp + t * D + 4 * (lane & 7)), w4 = *reinterpret_cast<const float4*>(ws + t * D + 4 * (lane & 7));
        float db = fmaf(r4.x, w4.x, r4.y * w4.y) + fmaf(r4.z, w4.z, r4.w * w4.w);
#pragma unroll
        for (int o = 4; o >= 1; o >>= 1) db += __shfl_xor_sync(0xffffffffu, db, o);
        if ((lane & 7) == 0 && t < nt) pgb[(t0 + t) * p.gb.sL] = db;
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int c = 0; c < 2; c++) {
            float* w = at(i, c);
            f2_unpack(S[i][c], w[0], w[1]);
        }
}

}  // namespace fwp
