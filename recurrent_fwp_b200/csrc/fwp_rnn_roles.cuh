// Backward of the delta RNN (v2 and v1) at d = 32: a chain warp and a trailing warp per sequence.
//
// The backward of one step (time reversed) is  g = gy + g_h;  dz = g (v2) or h .* (g - <h, g>) (v1);  G += s (x) dz;
// r = G^T k;  dv = beta r;  dbeta = r . w;  dk = G u - S dv;  G -= k (x) dv;  g_h = S_t dz, in v2 through the softmax.
// What one step hands to the next is g_h alone, and it needs S_t only, never G: the three gradients hang off dz.  A
// hand-off between two warps costs about 140 cycles on this machine, four times an exchange inside a warp, so the chain
// stays inside one warp and everything else follows it a chunk of steps at a time:
//   warp X (chain)      S, two rows and half the columns per lane: dz, w = v - v_old and -u of every step into a ring;
//   warp T (one chunk behind)  the other gradients, from G and its own S (fwp_trail.cuh), the chunk unrolled.
// The two meet once per chunk on a named barrier; that is also where staged input tiles change hands.  Each alone would take
// about 490 (X) and 600 (T) cycles per step with four sequences per SM; a scheduler with one sequence issues for both.
// 512 sequences x 512 steps: 167 us, 180 with one stream whose rows are not 16-byte aligned (194 when a loop over single pieces
// staged the tiles); 32 sequences x 256 65 and 70 us, against 222 us with T's work in two warps that held G by columns and by rows, and 222 us with T's columns split
// over two warps (a third more instructions).
#pragma once
#include "fwp_trail.cuh"

namespace fwp {

template <int TC, bool V1>
struct RnnRolesSmem {
    static constexpr int D = 32;
    using Stage = RnnBwdStage<D, TC, V1>;
    static constexpr int kStages = 3;                 // X on chunk j, T on j - 1, chunk j + 1 in flight
    static constexpr int kStep = 3 * D;               // per step: dz, -u, w
    static constexpr int kRing = TC * kStep;
    static constexpr int kOwn = 2 * D + TC * (D + 4); // T: dv of two steps, r w of a chunk
    static constexpr int kTable = (sizeof(StageTable) + 15) / 16 * 4;
    static constexpr int kFloats = kStages * Stage::kFloats + 2 * kRing + kOwn + kTable;
};

template <int TC, bool V1, bool WORDS>
__global__ void __launch_bounds__(256, 1) rnn_bwd_roles32_kernel(const RnnBwdParams p) {
    griddep_wait();               // launched as a dependent: global memory is touched from here on
    griddep_launch_dependents();
    constexpr int D = 32, NT = 64;
    using SM = RnnRolesSmem<TC, V1>;
    using Stage = typename SM::Stage;
    const int nslots = blockDim.x / NT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp % nslots, role = warp / nslots;       // the warps of a sequence share a scheduler
    const int stid = role * 32 + lane;
    const int seq = blockIdx.x * nslots + slot;
    const int n = seq / p.H, h = seq - n * p.H;
    extern __shared__ __align__(16) float smem_all[];
    float* smem = smem_all + (size_t)slot * SM::kFloats;
    float* ring = smem + SM::kStages * Stage::kFloats;
    float* xch = ring + 2 * SM::kRing;
    float* pw = xch + 2 * D;
    StageTable* tb = reinterpret_cast<StageTable*>(xch + SM::kOwn);
    if (stid == 0) {                // tile order of RnnBwdStage: k, v, gy, v_old, od, (out)
        stage_table_set(tb, 0, p.k, n, h);
        stage_table_set(tb, 1, p.v, n, h);
        stage_table_set(tb, 2, p.gy, n, h);
        stage_table_set(tb, 3, p.v_old, n, h);
        if (V1 && !p.od.p) stage_table_set_lagging(tb, 4, p.out, p.start, n, h);
        else stage_table_set(tb, 4, p.od, n, h);
        if (V1) stage_table_set(tb, 5, p.out, n, h);
        stage_table_set_col(tb, 0, p.beta, n, h);
    }
    float* W = p.W + n * p.wN + h * p.wH;
    slot_barrier(slot, NT);         // the table is in place

    const int nchunks = (p.L + TC - 1) / TC;
    constexpr int TILES = V1 ? 6 : 5;
    RowStager<TC, 2, TILES, WORDS> rows_in(tb, (nchunks - 1) * TC, stid);
    auto issue = [&](int j) {           // called for j = 0, 1, 2, ...
        const int t0 = (nchunks - 1 - j) * TC, nt = min(TC, p.L - t0);
        float* const st = smem + (j % SM::kStages) * Stage::kFloats;
        if (V1 && t0 == 0) stage_table_issue<TC, NT>(st, tb, TILES, 1, t0, nt, stid);
        else rows_in.issue(st, nt);
    };
    // top of the loop both warps run: chunk j's tiles have landed, X is through chunk j - 1, T through j - 2
    auto advance = [&](int j) {
        cp_async_wait<0>();
        slot_barrier(slot, NT);
        if (j + 1 < nchunks) issue(j + 1);
    };
    issue(0);
    if (role == 0) {
        // ---------------------------------------------------------------- X: the chain
        // lane (half, lp): rows 2 lp + half (finished here) and 2 lp + 1 - half (given away), columns 16 half .. 16 half + 15
        const int half = lane >> 4, lp = lane & 15, own = 2 * lp + half, other = 2 * lp + 1 - half;
        f2 M[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float* w = W + (long long)(i < 8 ? own : other) * p.wE + 16 * half + 2 * (i & 7);
            M[i] = f2_pack(w[0], w[1]);
        }
        float* pgz = reinterpret_cast<float*>(p.gz.p) + n * p.gz.sN + h * p.gz.sH + (p.L - 1) * p.gz.sL + own;
        float gh = 0.f;             // the gradient handed back through the recurrence (of feature `own`)
        for (int j = 0; j <= nchunks; j++) {
            advance(j);
            if (j == nchunks) break;
            Stage s; s.bind(smem + (j % SM::kStages) * Stage::kFloats);
            const int nt = min(TC, p.L - (nchunks - 1 - j) * TC);
            float* rg = ring + (j & 1) * SM::kRing;
            float nb, k0, k1, se, gy, hm, w;
            auto fetch = [&](int t) {               // what step t does not wait for, one step early
                nb = -s.b.f[t];
                k0 = s.k.f[t * D + own];
                k1 = s.k.f[t * D + other];
                se = V1 ? 0.f : s.od.f[t * D + own];
                hm = V1 ? s.out.f[t * D + own] : 0.f;
                gy = s.gy.f[t * D + own];
                w = s.v.f[t * D + own] - s.vo.f[t * D + own];
            };
            fetch(nt - 1);
#pragma unroll 2
            for (int t = nt - 1; t >= 0; t--) {
                float* e = rg + t * SM::kStep;
                const f2 kd0 = f2_dup(k0), kd1 = f2_dup(k1);
                const float st = se;
                float g = gy + gh;
                if constexpr (V1) {
                    const float dotp = warp_sum_idx<1>(hm * g);
                    g = hm * (g - dotp);
                }
                e[own] = g;
                e[D + own] = nb * w;
                e[2 * D + own] = w;
                *pgz = g;
                pgz -= p.gz.sL;
                __syncwarp();
                f2 vg[8], vw[8];
                lds_slice<16>(vg, e + 16 * half);
                lds_slice<16>(vw, e + D + 16 * half);
                fetch(t > 0 ? t - 1 : 0);
                f2 a0 = 0ull, a1 = 0ull, b0 = 0ull, b1 = 0ull;
#pragma unroll
                for (int i = 0; i < 8; i += 2) {
                    b0 = ffma2(M[8 + i], vg[i], b0);
                    b1 = ffma2(M[9 + i], vg[i + 1], b1);
                    a0 = ffma2(M[i], vg[i], a0);
                    a1 = ffma2(M[i + 1], vg[i + 1], a1);
                }
                const float gs = f2_hsum(fadd2(a0, a1)) + __shfl_xor_sync(0xffffffffu, f2_hsum(fadd2(b0, b1)), 16);
                if constexpr (V1) {
                    gh = gs;
                } else {
                    const float dotp = warp_sum_idx<1>(st * gs);
                    gh = st * (gs - dotp);
                }
#pragma unroll
                for (int i = 0; i < 8; i++) {       // S_{t-1} = S_t - k (x) u: in the shadow of the reduction
                    M[i] = ffma2(vw[i], kd0, M[i]);
                    M[8 + i] = ffma2(vw[i], kd1, M[8 + i]);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 16; i++) {
            float* w = W + (long long)(i < 8 ? own : other) * p.wE + 16 * half + 2 * (i & 7);
            f2_unpack(M[i], w[0], w[1]);
        }
        return;
    }
    // -------------------------------------------------------------------- T: one chunk behind
    Trail32 tr(lane, W, p.wE);
    const long long last = p.L - 1;
    float* pgk = reinterpret_cast<float*>(p.gk.p) + n * p.gk.sN + h * p.gk.sH + lane + last * p.gk.sL;
    float* pgv = reinterpret_cast<float*>(p.gv.p) + n * p.gv.sN + h * p.gv.sH + tr.own + last * p.gv.sL;
    float* const pgb = reinterpret_cast<float*>(p.gb.p) + n * p.gb.sN + h * p.gb.sH;
    for (int j = 0; j <= nchunks; j++) {
        advance(j);
        if (j == 0) continue;
        const int jj = j - 1, t0 = (nchunks - 1 - jj) * TC, nt = min(TC, p.L - t0);
        Stage s; s.bind(smem + (jj % SM::kStages) * Stage::kFloats);
        const float* rg = ring + (jj & 1) * SM::kRing;
#pragma unroll TC   // a step waits for the one before through dv alone: the rest of the others fills in
        for (int t = nt - 1; t >= 0; t--) {
            const float* e = rg + t * SM::kStep;
            float r, dv, dk;
            tr.step(s.od.f + t * D, s.k.f + t * D, e, e + D, s.b.f[t], xch + (t & 1) * D, r, dv, dk);
            pw[t * (D + 4) + lane] = r * e[2 * D + tr.own];
            *pgv = dv;
            *pgk = dk;
            pgk -= p.gk.sL; pgv -= p.gv.sL;
        }
        trail_dbeta<TC>(pw, pgb + t0 * p.gb.sL, p.gb.sL, nt, lane);
    }
}

}  // namespace fwp
