// Backward of the recurrent delta net at d = 32: three warps per sequence.
//
// Everything but the parameter gradients sits on the chain here: the gradient handed back through tanh(y_{t-1})
// needs dq, dk (both matrices G and S), their softmax backward and the three products with the rows of R.  What G takes part
// in, though, is known a step early but for a rank-one term, so G lives in a warp of its own:
//   warp P   holds G (8 x 4 pieces, fwp_trail.cuh).  For step t it posts  r0 = G^T k,  G u  and  q . k  before g_t is known,
//            then takes g_t and dv_t:  G += q (x) g - k (x) dv;
//   warp X   the chain, two rows and half the columns of S and of the three R per lane:  r = r0 + (q.k) g,  dv = beta r,
//            dq = S_{t-1} g + k (u.g),  dk = G u + q (u.g) - S_{t-1} dv,  softmax backward, the products with R, tanh.
//            Two of the sums over features come from products of vectors that the lane reads anyway: u.g = beta (w.g) and
//            db = (w.dv) (1 - beta).  Those of the softmax, q . dq and k . dk, are taken over the dq and dk that they are subtracted from:
//            y . g and w.dv - v_old.dv are the same numbers by the forward's saved values, but those and the rewound S part by the
//            rewind's rounding, and the gradients through the softmax then sum to that instead of to zero;
//   warp Y   turns v into w = v - v_old (and the outputs into their tanh) for the chunk that X takes next, and two chunks later accumulates the three parameter
//            gradients (8 x 4 pieces) and stores.
// X and P hand over twice per step at named barriers: P has X's step to answer in.  The warps meet once per chunk of steps.
// 512 sequences x 256 steps take 161 us, 32 sequences 105, and 171 and 105 where gy's rows are off a 16-byte boundary (320 bytes of
// spills with four sequences per SM) (230 us for 512 with one warp for all but the parameter gradients; 10 more when
// all three ran a loop over single pieces instead of Y staging by running pointers).  X alone took 131 -- 250 instructions a step, 128 of
// them packed multiply-adds at 2.7 cycles -- and P alone 160, when q . dq and k . dk came from the saved values: that form's seventh tile
// cost 6 us of 167 with 512 sequences, its shorter chain gave 10 of 105 with 32.  Not worth its instructions: P posting from a G one step
// older, corrected by scalars, and the two sums over the parts of dq and dk before the halves of the warp meet (164 us and 104).
// With four sequences per SM (504 of 512 registers of a scheduler's four threads: 208 X, 120 P, 176 Y) 512 sequences are resident.
#pragma once
#include "fwp_trail.cuh"

namespace fwp {

template <int TC>
struct RecRolesSmem {
    static constexpr int D = 32;
    using Stage = RecBwdStage<D, TC>;
    static constexpr int kTiles = 6;
    static constexpr int kStages = 4;                 // chunk j + 1 in flight, w of chunk j, X and P on j - 1, Y on j - 2
    static constexpr int kStep = 4 * D + 4;           // per step: g, dv, dq~, dk~, db~
    static constexpr int kRing = TC * kStep;
    static constexpr int kMail = 2 * D + 4;           // r0, G u, q.k
    static constexpr int kTable = (sizeof(StageTable) + 15) / 16 * 4;
    static constexpr int kFloats = kStages * Stage::kFloats + 2 * kRing + 2 * kMail + kTable;
};

// registers a thread of X, P and Y with four sequences per SM (a warpgroup each)
struct RecRolesRegs {
    static constexpr int X = 208, P = 120, Y = 176, kSum = X + P + Y;
};

template <int TC, int SLOTS, bool OUT, bool WORDS>
__global__ void __launch_bounds__(96 * SLOTS, 1) rec_bwd_roles32_kernel(const RecBwdParams p) {
    griddep_wait();               // launched as a dependent: global memory is touched from here on
    griddep_launch_dependents();
    constexpr int D = 32, NT = 96;
    using SM = RecRolesSmem<TC>;
    using Stage = typename SM::Stage;
    const int nslots = SLOTS == 4 ? 4 : blockDim.x / NT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp % nslots, role = warp / nslots;       // 0: X, 1: P, 2: Y
    const int stid = role * 32 + lane;
    const int seq = blockIdx.x * nslots + slot;
    const int n = seq / p.H, h = seq - n * p.H;
    extern __shared__ __align__(16) float smem_all[];
    float* smem = smem_all + (size_t)slot * SM::kFloats;
    float* ring = smem + SM::kStages * Stage::kFloats;
    float* mail = ring + 2 * SM::kRing;
    StageTable* tb = reinterpret_cast<StageTable*>(mail + 2 * SM::kMail);
    if (stid == 0) {                // tile order: q, k, v, v_old, od, gy
        stage_table_set(tb, 0, p.q, n, h);
        stage_table_set(tb, 1, p.k, n, h);
        stage_table_set(tb, 2, p.v, n, h);
        stage_table_set(tb, 3, p.v_old, n, h);
        if constexpr (OUT) stage_table_set_lagging(tb, 4, p.out, p.start, n, h);
        else stage_table_set(tb, 4, p.od, n, h);
        stage_table_set(tb, 5, p.gy, n, h);
        stage_table_set_col(tb, 0, p.beta, n, h);
    }
    slot_barrier(slot, NT);         // the table is in place

    const int nchunks = (p.L + TC - 1) / TC;
    // top of the loop that every warp runs; Y stages the tiles
    auto issue = [&](int) {};
    auto advance = [&](int j, auto&& issue) {
        cp_async_wait<0>();
        slot_barrier(slot, NT);
        if (j + 1 < nchunks) issue(j + 1);
    };
    // hand-overs between X and P: one side arrives, the other waits, in strict alternation
    auto arrive = [&](int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); };
    auto await = [&](int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); };
    const int given = 5 + slot, posted = 9 + slot;
    float* const W = p.W + n * p.wN + h * p.wH;
    if (role == 0) {
        // ---------------------------------------------------------------- X: the chain
        if constexpr (SLOTS == 4) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(RecRolesRegs::X));
        // lane (half, lp): rows 2 lp + half (finished here) and 2 lp + 1 - half (given away), columns 16 half .. 16 half + 15
        const int half = lane >> 4, lp = lane & 15, own = 2 * lp + half, other = 2 * lp + 1 - half;
        auto at = [&](int i) { return (i < 8 ? own : other); };
        f2 S[16], Rq[16], Rk[16], Rv[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int c = 16 * half + 2 * (i & 7);
            const float* w = W + (long long)at(i) * p.wE + c;
            S[i] = f2_pack(w[0], w[1]);
            const long long r = h * p.rH + (long long)at(i) * p.rE + c;
            Rq[i] = f2_pack(p.Rq[r], p.Rq[r + 1]);
            Rk[i] = f2_pack(p.Rk[r], p.Rk[r + 1]);
            Rv[i] = f2_pack(p.Rv[r], p.Rv[r + 1]);
        }
        const float rbl = p.rb[h * p.rbH + own];
        // a0 + a1, b0 + b1: M x for the rows `own` and `other`
        auto dots = [&](const f2 (&M)[16], const f2 (&x)[8], f2& a, f2& b) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                a = ffma2(M[i], x[i], a);
                b = ffma2(M[8 + i], x[i], b);
            }
        };
        auto dot = [&](const f2 (&x)[8], const f2 (&y)[8]) {
            f2 a = fmul2(x[0], y[0]), b = fmul2(x[1], y[1]);
#pragma unroll
            for (int i = 2; i < 8; i += 2) {
                a = ffma2(x[i], y[i], a);
                b = ffma2(x[i + 1], y[i + 1], b);
            }
            return f2_hsum(fadd2(a, b));
        };
        auto swap_halves = [&](float x) { return __shfl_xor_sync(0xffffffffu, x, 16); };
        float gh = 0.f;
        for (int j = 0; j <= nchunks + 1; j++) {
            advance(j, issue);
            if (j == 0 || j > nchunks) continue;
            Stage s; s.bind(smem + ((j - 1) % SM::kStages) * Stage::kFloats);
            const int nt = min(TC, p.L - (nchunks - j) * TC);
            float* rg = ring + ((j - 1) & 1) * SM::kRing;
            f2 w[8];
            float nbeta, nqe, nke;
            auto rewind = [&](int t, float live) {      // S_{t-1} = S_t - beta k (x) w; what step t does not wait for
                nbeta = s.b.f[t];
                nqe = s.q.f[t * D + own];
                nke = s.k.f[t * D + own];
                lds_slice<16>(w, s.v.f + t * D + 16 * half);
                const float nb = -nbeta * live;
                const f2 k0 = f2_dup(nb * nke), k1 = f2_dup(nb * s.k.f[t * D + other]);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    S[i] = ffma2(w[i], k0, S[i]);
                    S[8 + i] = ffma2(w[i], k1, S[8 + i]);
                }
            };
            rewind(nt - 1, 1.f);
#pragma unroll 1
            for (int t = nt - 1; t >= 0; t--) {
                float* e = rg + t * SM::kStep;
                const float beta = nbeta, qe = nqe, ke = nke;
                const float* mb = mail + (t & 1) * SM::kMail;
                const float gcol = s.gy.f[t * D + own] + gh, hte = s.od.f[t * D + own];
                await(posted);
                const float r = fmaf(mb[2 * D], gcol, mb[own]), gu = mb[D + own];
                e[own] = gcol;
                e[D + own] = beta * r;
                __syncwarp();
                arrive(given);
                f2 x[8], y[8];
                lds_slice<16>(x, e + 16 * half);
                lds_slice<16>(y, e + D + 16 * half);
                float wg = dot(w, x), wdv = dot(w, y);
                f2 a = 0ull, b = 0ull, c = 0ull, d = 0ull;
                dots(S, x, a, b);
                dots(S, y, c, d);
                const float sg = f2_hsum(a) + swap_halves(f2_hsum(b));
                const float sdv = f2_hsum(c) + swap_halves(f2_hsum(d));
                wg += swap_halves(wg);
                wdv += swap_halves(wdv);
                const float ug = beta * wg;
                const float dq = fmaf(ke, ug, sg), dk = fmaf(qe, ug, gu) - sdv;
                const float dbh = wdv * (1.f - beta);
                float pq = qe * dq, pk = ke * dk;       // both softmax sums in one shuffle sequence
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) {
                    pq += __shfl_xor_sync(0xffffffffu, pq, o);
                    pk += __shfl_xor_sync(0xffffffffu, pk, o);
                }
                a = b = 0ull;
                dots(Rv, y, a, b);                      // beside the sums: the part of the feedback that needs dv only, and
                rewind(t > 0 ? t - 1 : 0, t > 0 ? 1.f : 0.f);       // the next step's state (at t = 0 nothing is subtracted: no branch)
                const float dqh = qe * (dq - pq), dkh = ke * (dk - pk);
                e[2 * D + own] = dqh;
                e[3 * D + own] = dkh;
                if (lane == 0) e[4 * D] = dbh;
                __syncwarp();
                lds_slice<16>(x, e + 2 * D + 16 * half);
                lds_slice<16>(y, e + 3 * D + 16 * half);
                c = d = 0ull;
                dots(Rq, x, a, b);
                dots(Rk, y, c, d);
                gh = (1.f - hte * hte) * (fmaf(rbl, dbh, f2_hsum(fadd2(a, c))) + swap_halves(f2_hsum(fadd2(b, d))));
            }
        }
#pragma unroll
        for (int i = 0; i < 16; i++) {
            float* w = W + (long long)at(i) * p.wE + 16 * half + 2 * (i & 7);
            f2_unpack(S[i], w[0], w[1]);
        }
        return;
    }
    if (role == 1) {
        // ---------------------------------------------------------------- P: G
        if constexpr (SLOTS == 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(RecRolesRegs::P));
        const Tile32 tile(lane);
        f2 G[16];
#pragma unroll
        for (int i = 0; i < 16; i++) G[i] = 0ull;
        for (int j = 0; j <= nchunks + 1; j++) {
            advance(j, issue);
            if (j == 0 || j > nchunks) continue;
            Stage s; s.bind(smem + ((j - 1) % SM::kStages) * Stage::kFloats);
            const int nt = min(TC, p.L - (nchunks - j) * TC);
            const float* rg = ring + ((j - 1) & 1) * SM::kRing;
#pragma unroll 1
            for (int t = nt - 1; t >= 0; t--) {
                float* mb = mail + (t & 1) * SM::kMail;
                f2 qq[4], kk[4], x[4], acc[4];
                tile.rows(qq, s.q.f + t * D);
                tile.rows(kk, s.k.f + t * D);
                tile.cols(x, s.v.f + t * D);            // w
                float r[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    f2 d = 0ull;
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        d = i == 0 ? fmul2(G[4 * c], kk[0]) : ffma2(G[4 * c + i], kk[i], d);
                        acc[i] = c == 0 ? fmul2(G[i], x[0]) : ffma2(G[4 * c + i], x[c], acc[i]);
                    }
                    r[c] = f2_hsum(d);
                }
                f2 d = fmul2(qq[0], kk[0]);
#pragma unroll
                for (int i = 1; i < 4; i++) d = ffma2(qq[i], kk[i], d);
                float qk = f2_hsum(d);
                qk += __shfl_xor_sync(0xffffffffu, qk, 8);
                qk += __shfl_xor_sync(0xffffffffu, qk, 16);
                mb[tile.own] = tile.sum_rows(r);
                mb[D + lane] = s.b.f[t] * tile.sum_cols(acc);
                if (lane == 0) mb[2 * D] = qk;
                __syncwarp();
                arrive(posted);
                await(given);
                const float* e = rg + t * SM::kStep;
                f2 y[4];
                tile.cols(x, e);
                {
                    const float2 a = *reinterpret_cast<const float2*>(e + D + tile.col0), b = *reinterpret_cast<const float2*>(e + D + tile.col1);
                    y[0] = f2_dup(-a.x); y[1] = f2_dup(-a.y); y[2] = f2_dup(-b.x); y[3] = f2_dup(-b.y);
                }
#pragma unroll
                for (int c = 0; c < 4; c++)
#pragma unroll
                    for (int i = 0; i < 4; i++) G[4 * c + i] = ffma2(kk[i], y[c], ffma2(qq[i], x[c], G[4 * c + i]));
            }
        }
        return;
    }
    // -------------------------------------------------------------------- Y: w for X and P, then parameter gradients and stores
    if constexpr (SLOTS == 4) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(RecRolesRegs::Y));
    const Tile32 tile(lane);
    f2 A[16], B[16], C[16];             // the partial gradients of Rq, Rk, Rv
#pragma unroll
    for (int i = 0; i < 16; i++) { A[i] = 0ull; B[i] = 0ull; C[i] = 0ull; }
    float arb = 0.f;
    const long long last = p.L - 1;
    float* pgq = reinterpret_cast<float*>(p.gq.p) + n * p.gq.sN + h * p.gq.sH + lane + last * p.gq.sL;
    float* pgk = reinterpret_cast<float*>(p.gk.p) + n * p.gk.sN + h * p.gk.sH + lane + last * p.gk.sL;
    float* pgv = reinterpret_cast<float*>(p.gv.p) + n * p.gv.sN + h * p.gv.sH + lane + last * p.gv.sL;
    float* pgb = reinterpret_cast<float*>(p.gb.p) + n * p.gb.sN + h * p.gb.sH + last * p.gb.sL;
    RowStager<TC, 1, SM::kTiles, WORDS> rows_in(tb, (nchunks - 1) * TC, lane);
    auto stage = [&](int j) {           // called for j = 0, 1, 2, ...
        const int t0 = (nchunks - 1 - j) * TC, nt = min(TC, p.L - t0);
        float* const st = smem + (j % SM::kStages) * Stage::kFloats;
        if (OUT && t0 == 0) stage_table_issue<TC, 32>(st, tb, SM::kTiles, 1, t0, nt, lane);
        else rows_in.issue(st, nt);
    };
    stage(0);
    for (int j = 0; j <= nchunks + 1; j++) {
        advance(j, stage);
        if (j < nchunks) {
            Stage s; s.bind(smem + (j % SM::kStages) * Stage::kFloats);
            const int nt = min(TC, p.L - (nchunks - 1 - j) * TC);
#pragma unroll 4
            for (int t = 0; t < nt; t++) {
                s.v.f[t * D + lane] -= s.vo.f[t * D + lane];
                if constexpr (OUT) s.od.f[t * D + lane] = tanhf(s.od.f[t * D + lane]);       // the accuracy of fwp_delayed
            }
        }
        if (j < 2) continue;
        Stage s; s.bind(smem + ((j - 2) % SM::kStages) * Stage::kFloats);
        const int nt = min(TC, p.L - (nchunks + 1 - j) * TC);
        const float* rg = ring + (j & 1) * SM::kRing;
#pragma unroll 2
        for (int t = nt - 1; t >= 0; t--) {
            const float* e = rg + t * SM::kStep;
            f2 hs[4], x[4], y[4], z[4];
            tile.rows(hs, s.od.f + t * D);
            tile.cols(x, e + 2 * D);
            tile.cols(y, e + 3 * D);
            tile.cols(z, e + D);
#pragma unroll
            for (int c = 0; c < 4; c++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    A[4 * c + i] = ffma2(hs[i], x[c], A[4 * c + i]);
                    B[4 * c + i] = ffma2(hs[i], y[c], B[4 * c + i]);
                    C[4 * c + i] = ffma2(hs[i], z[c], C[4 * c + i]);
                }
            const float dbh = e[4 * D];
            arb += s.od.f[t * D + lane] * dbh;
            *pgq = e[2 * D + lane]; *pgk = e[3 * D + lane]; *pgv = e[D + lane];
            if (lane == 0) *pgb = dbh;
            pgq -= p.gq.sL; pgk -= p.gk.sL; pgv -= p.gv.sL; pgb -= p.gb.sL;
        }
    }
    // partial parameter gradients of this (n, h): [3][d][d] then [d]; element (e, m) at e d + m
    float* out = p.scratch + (long long)seq * (3 * D * D + D);
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float* o = out + tile.row(i) * D + tile.col(c);
            f2_unpack(A[4 * c + i], o[0], o[D]);
            f2_unpack(B[4 * c + i], o[D * D], o[D * D + D]);
            f2_unpack(C[4 * c + i], o[2 * D * D], o[2 * D * D + D]);
        }
    out[3 * D * D + lane] = arb;
}

}  // namespace fwp
