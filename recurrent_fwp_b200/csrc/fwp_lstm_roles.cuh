// Backward of the delta LSTM (v1..v4) at d = 32: a chain warp and one trailing warp per gate.
//
// Time reversed, the only quantities one step hands to the next are the gradient of the fed-back output g_h and
// the cell gradient g_c.  The chain is  g_h, g_c -> dz[3] (element-wise) -> sum over the gates of S^q_t dz^q ->
// (softmax backward) -> g_h;  the value, key and beta gradients of the three delta rules hang off dz but feed
// nothing back.  So per sequence
//   warp X      holds S^i, S^u, S^o by rows (two rows and half the columns per lane), runs the chain, rewinds the matrices
//               (that needs inputs only) and leaves dz[3], w[3] = v - v_old, -u[3] = -beta w and the z-gradient of the update gate in a ring;
//   warp H_q    (q = i, u, o) runs one chunk of steps behind X and produces the gate's value, key, beta and z gradients
//               (fwp_trail.cuh).
// The four warps of a sequence meet once per chunk on a named barrier (that is also where staged input tiles
// change hands); nothing else crosses warps, because a hand-off costs about 140 cycles on this machine against 33
// for an exchange inside a warp.  SLOTS sequences share a CTA: four fill an SM with chunks of four steps (152 registers for the
// X warps, 120 for the others, out of the 128 a thread of the launch), so that 512 sequences are resident at once.  Bound by
// issue slots and the fp32 pipe (65 and 55 % on an SM with four sequences, 1200 warp instructions per sequence and step).
// 512 sequences x 512 steps: 520 us against 720 us for the form whose H warps held G twice (by columns and by rows, 208
// registers a thread), two sequences per SM and so two waves.
#pragma once
#include "fwp_trail.cuh"

namespace fwp {

template <int TC>
struct LstmRolesSmem {
    static constexpr int D = 32;
    using Stage = LstmBwdStage<D, TC>;
    static constexpr int kStages = 3;                 // X on chunk j, the H warps on chunk j - 1, chunk j + 1 in flight
    static constexpr int kStep = 10 * D;              // per step: dz[3], -u[3], w[3], z-gradient of gate u (variant 3)
    static constexpr int kRing = TC * kStep;
    static constexpr int kOwn = 2 * D + TC * (D + 4); // per H warp: dv of two steps, r w of a chunk
    static constexpr int kTable = (sizeof(StageTable) + 15) / 16 * 4;
    static constexpr int kFloats = kStages * Stage::kFloats + 2 * kRing + 3 * kOwn + kTable;
};

// registers a thread of X and of each H_q with four sequences per SM (a warpgroup each)
struct LstmRolesRegs {
    static constexpr int X = 152, H = 120, kSum = X + 3 * H;
};

template <int TC, int VAR, int SLOTS>
__global__ void __launch_bounds__(128 * SLOTS, 1) lstm_bwd_roles32_kernel(const LstmBwdParams p) {
    griddep_wait();               // launched as a dependent: global memory is touched from here on
    griddep_launch_dependents();
    constexpr int D = 32, NT = 128;
    using SM = LstmRolesSmem<TC>;
    using Stage = typename SM::Stage;
    const int nslots = SLOTS == 4 ? 4 : blockDim.x / NT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp % nslots, role = warp / nslots;       // role 0: X, 1..3: H of gate role - 1
    const int stid = role * 32 + lane;
    const int seq = blockIdx.x * nslots + slot;
    const int n = seq / p.H, h = seq - n * p.H;
    extern __shared__ __align__(16) float smem_all[];
    float* smem = smem_all + (size_t)slot * SM::kFloats;
    for (int i = stid; i < SM::kFloats - SM::kTable; i += NT) smem[i] = 0.f;
    float* ring = smem + SM::kStages * Stage::kFloats;
    float* hown = ring + 2 * SM::kRing;

    const bool lagging = !p.umc.p;      // tile 16 has the cell of the step before instead of u - that cell
    StageTable* tb = reinterpret_cast<StageTable*>(hown + 3 * SM::kOwn);
    if (stid == 0) {                // tile order of LstmBwdStage: k, v, v_old, gate of each gate, then gy, out, od, cell, umc
        for (int a = 0; a < 3; a++) {
            stage_table_set(tb, 4 * a + 0, p.k[a], n, h);
            stage_table_set(tb, 4 * a + 1, p.v[a], n, h);
            stage_table_set(tb, 4 * a + 2, p.v_old[a], n, h);
            stage_table_set(tb, 4 * a + 3, p.gate[a], n, h);
            stage_table_set_col(tb, a, p.beta[a], n, h);
        }
        stage_table_set(tb, 12, p.gy, n, h);
        stage_table_set(tb, 13, p.out, n, h);
        if (VAR != 1) tb->src[13] = nullptr;
        if (VAR == 1 && !p.od.p) stage_table_set_lagging(tb, 14, p.out, p.start, n, h);
        else stage_table_set(tb, 14, p.od, n, h);
        stage_table_set(tb, 15, p.cell, n, h);
        if (lagging) stage_table_set_lagging(tb, 16, p.cell, p.cell_start, n, h);
        else stage_table_set(tb, 16, p.umc, n, h);
    }
    slot_barrier(slot, NT);      // the zero fill is complete before the first copies land

    const int nchunks = (p.L + TC - 1) / TC;
    // top of the loop that every warp runs: chunk j's tiles have landed, X is through chunk j - 1, the H warps through j - 2,
    // and chunk j + 1 goes into the stage the H warps have just left
    auto issue = [&](int j) {
        const int c = nchunks - 1 - j;
        const int t0 = c * TC, nt = min(TC, p.L - t0);
        stage_table_issue<TC, NT>(smem + (j % SM::kStages) * Stage::kFloats, tb, 17, 3, t0, nt, stid);
    };
    auto advance = [&](int j) {
        cp_async_wait<0>();
        slot_barrier(slot, NT);
        if (j + 1 < nchunks) issue(j + 1);
    };
    issue(0);

    if (role == 0) {
        // ---------------------------------------------------------------- X: the chain
        if constexpr (SLOTS == 4) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(LstmRolesRegs::X));
        // lane (half, lp): rows 2 lp + half (finished here) and 2 lp + 1 - half (given away), columns 16 half .. 16 half + 15
        const int half = lane >> 4, lp = lane & 15, own = 2 * lp + half, other = 2 * lp + 1 - half;
        f2 M[3][16];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const float* W = p.W[q] + n * p.wN[q] + h * p.wH[q] + 16 * half;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const float* w = W + (long long)(i < 8 ? own : other) * p.wE[q] + 2 * (i & 7);
                M[q][i] = f2_pack(w[0], w[1]);
            }
        }
        float gh = 0.f, gc = 0.f;       // gradients handed back through the output and the cell
        for (int j = 0; j <= nchunks; j++) {
            advance(j);
            if (j == nchunks) break;
            Stage s; s.bind(smem + (j % SM::kStages) * Stage::kFloats);
            const int nt = min(TC, p.L - (nchunks - 1 - j) * TC);
            float* rg = ring + (j & 1) * SM::kRing;
#pragma unroll 1
            for (int t = nt - 1; t >= 0; t--) {
                const int o = t * D + own;
                float* e = rg + t * SM::kStep;
                // what the rewind and the trailing warps need and the chain does not
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const float w = s.v[q].f[o] - s.vo[q].f[o];
                    e[(3 + q) * D + own] = -s.b[q].f[t] * w;
                    e[(6 + q) * D + own] = w;
                }
                const float gsum = s.gy.f[o] + gh;
                float a = gsum;
                if constexpr (VAR == 1) {
                    const float hm = s.out.f[o];
                    const float dotp = warp_sum_idx<1>(hm * gsum);
                    a = hm * (gsum - dotp);
                }
                const float gi = s.gate[0].f[o], uu = s.gate[1].f[o], go = s.gate[2].f[o];
                float dz[3];
                dz[2] = (s.cell.f[o] * a) * (1.f - go) * go;
                gc += go * a;
                const float before = s.umc.f[o];
                dz[0] = (gc * (lagging ? uu - before : before)) * (1.f - gi) * gi;
                dz[1] = gc * gi;
                if constexpr (VAR != 4) dz[1] = dz[1] * (1.f - uu) * uu;
                gc *= (1.f - gi);
#pragma unroll
                for (int q = 0; q < 3; q++) e[q * D + own] = dz[q];
                if constexpr (VAR == 3) e[9 * D + own] = dz[1] + gsum;
                __syncwarp();
                f2 a0 = 0ull, a1 = 0ull, b0 = 0ull, b1 = 0ull;
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    f2 x[8];
                    lds_slice<16>(x, e + q * D + 16 * half);
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        a0 = ffma2(M[q][i], x[i], a0);
                        b0 = ffma2(M[q][8 + i], x[i], b0);
                        a1 = ffma2(M[q][i + 1], x[i + 1], a1);
                        b1 = ffma2(M[q][9 + i], x[i + 1], b1);
                    }
                }
                const float ghn = f2_hsum(fadd2(a0, a1)) + __shfl_xor_sync(0xffffffffu, f2_hsum(fadd2(b0, b1)), 16);
                if constexpr (VAR != 1) {
                    const float xe = s.od.f[o];
                    const float dotp = warp_sum_idx<1>(xe * ghn);
                    gh = xe * (ghn - dotp);
                } else {
                    gh = ghn;
                }
                // S^q_{t-1} = S^q_t - k (x) u, beside the reduction
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    f2 x[8];
                    lds_slice<16>(x, e + (3 + q) * D + 16 * half);
                    const f2 k0 = f2_dup(s.k[q].f[o]), k1 = f2_dup(s.k[q].f[t * D + other]);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        M[q][i] = ffma2(x[i], k0, M[q][i]);
                        M[q][8 + i] = ffma2(x[i], k1, M[q][8 + i]);
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 3; q++) {
            float* W = p.W[q] + n * p.wN[q] + h * p.wH[q] + 16 * half;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                float* w = W + (long long)(i < 8 ? own : other) * p.wE[q] + 2 * (i & 7);
                f2_unpack(M[q][i], w[0], w[1]);
            }
        }
        return;
    }

    // -------------------------------------------------------------------- H_q: one chunk behind
    if constexpr (SLOTS == 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(LstmRolesRegs::H));
    const int q = role - 1;
    // this gate's gradient streams, picked once (by value: a reference chosen at run time would make every
    // later field access an indexed load from the parameter bank)
    const Row4 rk = q == 0 ? p.gk[0] : (q == 1 ? p.gk[1] : p.gk[2]);
    const Row4 rz = q == 0 ? p.gz[0] : (q == 1 ? p.gz[1] : p.gz[2]);
    const Row4 rv = q == 0 ? p.gv[0] : (q == 1 ? p.gv[1] : p.gv[2]);
    const Row4 rb = q == 0 ? p.gb[0] : (q == 1 ? p.gb[1] : p.gb[2]);
    float* const W = (q == 0 ? p.W[0] : (q == 1 ? p.W[1] : p.W[2])) + n * (q == 0 ? p.wN[0] : (q == 1 ? p.wN[1] : p.wN[2])) +
                     h * (q == 0 ? p.wH[0] : (q == 1 ? p.wH[1] : p.wH[2]));
    Trail32 tr(lane, W, q == 0 ? p.wE[0] : (q == 1 ? p.wE[1] : p.wE[2]));
    const long long last = p.L - 1;
    float* pgk = reinterpret_cast<float*>(rk.p) + n * rk.sN + h * rk.sH + lane + last * rk.sL;
    float* pgz = reinterpret_cast<float*>(rz.p) + n * rz.sN + h * rz.sH + lane + last * rz.sL;
    float* pgv = reinterpret_cast<float*>(rv.p) + n * rv.sN + h * rv.sH + tr.own + last * rv.sL;
    float* const pgb = reinterpret_cast<float*>(rb.p) + n * rb.sN + h * rb.sH;
    float* const xch = hown + q * SM::kOwn;
    float* const pw = xch + 2 * D;
    for (int j = 0; j <= nchunks; j++) {
        advance(j);
        if (j == 0) continue;
        const int jj = j - 1, t0 = (nchunks - 1 - jj) * TC, nt = min(TC, p.L - t0);
        const float* stage = smem + (jj % SM::kStages) * Stage::kFloats;
        const float* rg = ring + (jj & 1) * SM::kRing;
        const float* kt = stage + 4 * q * r4(TC * D);
        const float* st = stage + 14 * r4(TC * D);
        const float* bt = stage + 17 * r4(TC * D) + q * r4(TC);
#pragma unroll 1
        for (int t = nt - 1; t >= 0; t--) {
            const float* e = rg + t * SM::kStep;
            float r, dv, dk;
            tr.step(st + t * D, kt + t * D, e + q * D, e + (3 + q) * D, bt[t], xch + (t & 1) * D, r, dv, dk);
            pw[t * (D + 4) + lane] = r * e[(6 + q) * D + tr.own];
            *pgz = e[((VAR == 3 && q == 1) ? 9 : q) * D + lane];
            *pgv = dv;
            *pgk = dk;
            pgk -= rk.sL; pgz -= rz.sL; pgv -= rv.sL;
        }
        trail_dbeta<TC>(pw, pgb + t0 * rb.sL, rb.sL, nt, lane);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Forward of the delta LSTM at d = 32 with one warp per gate.
//
// A step has three delta-rule updates and three read-outs, one per gate, and they meet only in the element-wise
// cell update.  Warp q of a sequence holds S^q, applies its update (inputs only, so it runs beside the chain),
// forms its pre-activation S^q_t^T x + z^q, applies its gate's nonlinearity and posts the gate; after the one
// barrier of the step every warp reads the three gates and computes the cell, the output and the next fed-back
// vector for itself (the same instructions on the same numbers in all three warps, so they agree bit for bit).  One barrier per step
// (about 110 cycles) buys a chain warp of about 150 instead of 400 instructions per step.
template <int TC>
struct LstmGatesSmem {
    static constexpr int D = 32;
    using Stage = LstmFwdStage<D, TC>;
    static constexpr int kStages = 2;
    static constexpr int kX = 3 * D;                  // the fed-back vector, one private copy per warp
    static constexpr int kP = 2 * 3 * D;              // posted pre-activations, two step parities
    static constexpr int kFloats = kStages * Stage::kFloats + kX + kP;
};

// WORDS: some stream's rows are not 16-byte aligned
template <int TC, int VAR, bool WORDS>
__global__ void __launch_bounds__(384, 1) lstm_fwd_gates32_kernel(const LstmFwdParams p) {
    griddep_wait();               // launched as a dependent: global memory is touched from here on
    griddep_launch_dependents();
    constexpr int D = 32, NP = 16, NT = 96;
    using SM = LstmGatesSmem<TC>;
    using Stage = typename SM::Stage;
    constexpr int kTile = r4(TC * D);
    const int nslots = blockDim.x / NT;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp % nslots, q = warp / nslots;          // q: the gate this warp serves (0 = i, 1 = u, 2 = o)
    const int stid = q * 32 + lane;
    const int seq = blockIdx.x * nslots + slot;
    const int n = seq / p.H, h = seq - n * p.H;
    extern __shared__ __align__(16) float smem_all[];
    float* smem = smem_all + (size_t)slot * SM::kFloats;
    for (int i = stid; i < SM::kFloats; i += NT) smem[i] = 0.f;
    float* xv = smem + SM::kStages * Stage::kFloats + q * D;
    float* post = smem + SM::kStages * Stage::kFloats + SM::kX;
    // this warp's matrix and its three output streams
    // selected with compares, not with a run-time index (that would put the parameter block in local memory)
    float* const Wb = q == 0 ? p.W[0] : (q == 1 ? p.W[1] : p.W[2]);
    const long long wN = q == 0 ? p.wN[0] : (q == 1 ? p.wN[1] : p.wN[2]);
    const long long wH = q == 0 ? p.wH[0] : (q == 1 ? p.wH[1] : p.wH[2]);
    const long long wE = q == 0 ? p.wE[0] : (q == 1 ? p.wE[1] : p.wE[2]);
    const Row4& rgate = q == 0 ? p.gate[0] : (q == 1 ? p.gate[1] : p.gate[2]);
    const Row4& rvold = q == 0 ? p.v_old[0] : (q == 1 ? p.v_old[1] : p.v_old[2]);
    float* W = Wb + n * wN + h * wH;
    f2 S[NP];
    {
        float v[2];
#pragma unroll
        for (int i = 0; i < D; i++) {       // column m = lane: element (e, m)
            v[i & 1] = W[(long long)i * wE + lane];
            if (i & 1) S[i >> 1] = f2_pack(v[0], v[1]);
        }
    }
    auto colptr = [&](const Row4& r) { return reinterpret_cast<float*>(r.p) + n * r.sN + h * r.sH + lane; };
    // stores are shared out: every warp writes its gate and its v_old, and one of out / cell / fed-back vector
    float* pg = colptr(rgate);
    float* pvo = colptr(rvold);
    const Row4& third = q == 0 ? p.out : (q == 1 ? p.cell : p.nmz);
    const bool has_third = q < 2 || VAR != 1;
    float* p3 = has_third ? colptr(third) : pg;
    const long long sg = rgate.sL, svo = rvold.sL, s3 = has_third ? third.sL : 0;
    float* hp = p.h + n * p.hN + h * p.hH;
    float* cp = p.c + n * p.cN + h * p.cH;
    float hv = hp[lane], cv = cp[lane];
    slot_barrier(slot, NT);         // the zero fill is complete before the first copies land

    const int nchunks = (p.L + TC - 1) / TC;
    // a warp copies z, k, v and beta of its own gate, by running pointers: four rows at a time, a 16-byte piece per lane, or row by
    // row word by word (12 rolled iterations over a table of all nine tiles: 512 sequences x 512 steps
    // 286 us, now 255; 32 sequences 192, now 151)
    WarpRows32<TC, WORDS, true> rz, rk, rv;
    rz.init(q == 0 ? p.z[0] : (q == 1 ? p.z[1] : p.z[2]), n, h, lane);
    rk.init(q == 0 ? p.k[0] : (q == 1 ? p.k[1] : p.k[2]), n, h, lane);
    rv.init(q == 0 ? p.v[0] : (q == 1 ? p.v[1] : p.v[2]), n, h, lane);
    const Row4& rbeta = q == 0 ? p.beta[0] : (q == 1 ? p.beta[1] : p.beta[2]);
    const long long sb = rbeta.sL;
    const float* bfrom = reinterpret_cast<const float*>(rbeta.p) + n * rbeta.sN + h * rbeta.sH + lane * sb;
    auto issue = [&](int c) {           // called for c = 0, 1, 2, ...
        const int nt = min(TC, p.L - c * TC);
        float* const base = smem + (c & 1) * Stage::kFloats;
        rz.issue(base + 3 * q * kTile, nt);
        rk.issue(base + (3 * q + 1) * kTile, nt);
        rv.issue(base + (3 * q + 2) * kTile, nt);
        if (lane < nt) cp_async4(base + 9 * kTile + q * r4(TC) + lane, bfrom);
        bfrom += TC * sb;
        cp_async_commit();
    };
    issue(0);
    int par = 0;
    for (int c = 0; c < nchunks; c++) {
        cp_async_wait<0>();
        slot_barrier(slot, NT);     // chunk c has landed; everyone is through chunk c - 1
        if (c + 1 < nchunks) issue(c + 1);
        const float* base = smem + (c & 1) * Stage::kFloats;
        const float* zcol = base + (3 * q) * kTile + lane;          // z of this gate
        const float* krow = base + (3 * q + 1) * kTile;             // k of this gate
        const float* vcol = base + (3 * q + 2) * kTile + lane;      // v of this gate
        const float* zu = base + 3 * kTile + lane;                  // z of the update gate (variant 3)
        const float* brow = base + 9 * kTile + q * r4(TC);
        const int nt = min(TC, p.L - c * TC);
#pragma unroll 1
        for (int t = 0; t < nt; t++, zcol += D, krow += D, vcol += D, zu += D, brow++) {
            float* pp = post + par * (3 * D);
            par ^= 1;
            // this gate's delta update (inputs only)
            f2 kk[NP];
            lds_slice<D>(kk, krow);
            const float vo = dot2<NP>(S, kk);
            const float u = brow[0] * (vcol[0] - vo);
            axpy2<NP>(S, kk, u);
            // the fed-back vector, computed by every warp for itself
            float xe;
            if constexpr (VAR == 1) {
                xe = hv;
            } else {
                const float mx = warp_max_f32(hv);
                xe = exp_neg(hv - mx);
                xe *= rcp_approx(warp_sum_unit_scaled(xe) * (1.f / 67108864.f) + kLstmEps);
            }
            xv[lane] = xe;
            __syncwarp();
            f2 xs[NP];
            lds_slice<D>(xs, xv);
            // each warp posts its gate already activated: one sigmoid per warp and step instead of three
            const float pre = dot2<NP>(S, xs) + zcol[0];
            pp[q * D + lane] = (VAR == 4 && q == 1) ? pre : sigmoidf_(pre);
            slot_barrier(slot, NT);
            const float gi = pp[lane], uu = pp[D + lane], go = pp[2 * D + lane];
            cv = gi * uu + (1.f - gi) * cv;
            float hn = go * cv;
            if constexpr (VAR == 1) {
                const float mx = warp_max_f32(hn);
                const float ex = exp_neg(hn - mx);
                hn = ex * rcp_approx(warp_sum_unit_scaled(ex) * (1.f / 67108864.f));
            } else if constexpr (VAR == 3) {
                hn += zu[0];
            }
            hv = hn;
            *pg = q == 0 ? gi : (q == 1 ? uu : go);
            *pvo = vo;
            if (has_third) *p3 = q == 0 ? hn : (q == 1 ? cv : xe);
            pg += sg; pvo += svo; p3 += s3;
        }
    }
#pragma unroll
    for (int i = 0; i < D; i++) {
        float lo, hi;
        f2_unpack(S[i >> 1], lo, hi);
        W[(long long)i * wE + lane] = (i & 1) ? hi : lo;
    }
    if (q == 0) { hp[lane] = hv; cp[lane] = cv; }
}

}  // namespace fwp
