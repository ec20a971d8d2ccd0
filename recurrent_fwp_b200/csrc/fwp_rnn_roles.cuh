// Backward of the delta RNN (v2 and v1) at d = 32: a chain warp and two trailing warps per sequence.
//
// The backward of one step (time reversed) is  g = gy + g_h;  dz = g (v2) or h .* (g - <h, g>) (v1);  G += s (x) dz;
// r = G^T k;  dv = beta r;  dbeta = r . w;  dk = G u - S dv;  G -= k (x) dv;  g_h = S_t dz, in v2 through the softmax.
// What one step hands to the next is g_h alone, and it needs S_t only, never G: the three gradients hang off dz.  A
// hand-off between two warps costs about 140 cycles on this machine, four times an exchange inside a warp, so the chain
// stays inside one warp and everything else follows it a chunk of steps at a time:
//   warp X (chain)      S by rows: leaves dz and u = beta (v - v_old) of every step in a ring and rewinds S;
//   warp C (one chunk behind)  G by columns: r, hence the value and beta gradients and dv in the ring;
//   warp R (two chunks behind) G and S by rows: the key gradient.
// The three warps meet once per chunk on a named barrier; that is also where staged input tiles change hands.  They hold
// 32, 48 and 80 packed multiply-adds per step, so with 512 sequences the fp32 pipe (about 280 cycles per step and SM
// sub-partition) and the chain (about 250) bound the kernel alike.  The form before this one kept G by columns in the
// chain warp (96 + 80): 900 cycles per step.
#pragma once

namespace fwp {

template <int TC, bool V1>
struct RnnRolesSmem {
    static constexpr int D = 32;
    using Stage = RnnBwdStage<D, TC, V1>;
    static constexpr int kStages = 4;                 // X on chunk j, C on j - 1, R on j - 2, chunk j + 1 in flight
    static constexpr int kStep = 3 * D;               // per step: dz, u, dv
    static constexpr int kRing = TC * kStep;
    static constexpr int kSums = TC * (D + 4);        // C's r w, summed a chunk at a time
    static constexpr int kTable = (sizeof(StageTable) + 15) / 16 * 4;
    static constexpr int kFloats = kStages * Stage::kFloats + 3 * kRing + kSums + kTable;
};

template <int TC, bool V1>
__global__ void __launch_bounds__(384, 1) rnn_bwd_roles32_kernel(const RnnBwdParams p) {
    griddep_wait();               // launched as a dependent: global memory is touched from here on
    griddep_launch_dependents();
    constexpr int D = 32, NP = 16, NT = 96;
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

    float* pw = ring + 3 * SM::kRing;
    StageTable* tb = reinterpret_cast<StageTable*>(pw + SM::kSums);
    if (stid == 0) {                // tile order of RnnBwdStage: k, v, gy, v_old, od, (out)
        stage_table_set(tb, 0, p.k, n, h);
        stage_table_set(tb, 1, p.v, n, h);
        stage_table_set(tb, 2, p.gy, n, h);
        stage_table_set(tb, 3, p.v_old, n, h);
        stage_table_set(tb, 4, p.od, n, h);
        if (V1) stage_table_set(tb, 5, p.out, n, h);
        stage_table_set_col(tb, 0, p.beta, n, h);
    }
    float* W = p.W + n * p.wN + h * p.wH;
    // X: A = S[lane][.].  C and R hold a 2 x 16 piece per lane, two lines (2 lp, 2 lp + 1) and one half of the other index,
    // first line in [0, 8), second in [8, 16) -- C: A = G by columns; R: A = S, B = G by rows
    const int half = lane >> 4, lp = lane & 15, own = 2 * lp + half;       // own: the line this lane finishes and stores
    f2 A[NP], B[NP];
#pragma unroll
    for (int i = 0; i < NP; i++) {
        const float* w = role == 0 ? W + (long long)lane * p.wE + 2 * i : W + (long long)(2 * lp + (i >> 3)) * p.wE + 16 * half + 2 * (i & 7);
        A[i] = role == 1 ? 0ull : f2_pack(w[0], w[1]);
        B[i] = 0ull;
    }
    slot_barrier(slot, NT);         // the table is in place, and nobody has written W

    const int nchunks = (p.L + TC - 1) / TC;
    auto issue = [&](int j) {
        const int c = nchunks - 1 - j;
        const int t0 = c * TC, nt = min(TC, p.L - t0);
        stage_table_issue<TC, NT>(smem + (j % SM::kStages) * Stage::kFloats, tb, V1 ? 6 : 5, 1, t0, nt, stid);
    };
    issue(0);
    float gh = 0.f;                 // X: the gradient handed back through the recurrence (lane = feature index)
    for (int j = 0; j < nchunks + 2; j++) {
        cp_async_wait<0>();
        slot_barrier(slot, NT);     // chunk j's tiles have landed; X is through chunk j - 1, C through j - 2, R through j - 3
        if (j + 1 < nchunks) issue(j + 1);      // into the stage R has just left
        const int jj = j - role;
        if (jj < 0 || jj >= nchunks) continue;
        Stage s; s.bind(smem + (jj % SM::kStages) * Stage::kFloats);
        const int c = nchunks - 1 - jj;
        const int t0 = c * TC, nt = min(TC, p.L - t0);
        float* rg = ring + (jj % 3) * SM::kRing;
        if (role == 0) {
            // ------------------------------------------------------------ X: the chain
            float ke, se, gy, hm, u;
            auto fetch = [&](int t) {               // what step t does not wait for, one step early
                ke = s.k.f[t * D + lane];
                se = V1 ? 0.f : s.od.f[t * D + lane];
                hm = V1 ? s.out.f[t * D + lane] : 0.f;
                gy = s.gy.f[t * D + lane];
                u = s.b.f[t] * (s.v.f[t * D + lane] - s.vo.f[t * D + lane]);
            };
            fetch(nt - 1);
#pragma unroll 2
            for (int t = nt - 1; t >= 0; t--) {
                float* e = rg + t * SM::kStep;
                const float kt = ke, st = se;
                float g = gy + gh;
                if constexpr (V1) {
                    const float dotp = warp_sum_idx<1>(hm * g);
                    g = hm * (g - dotp);
                }
                e[lane] = g;
                e[D + lane] = u;
                __syncwarp();
                f2 vg[NP], vu[NP];
                lds_slice<D>(vg, e);
                lds_slice<D>(vu, e + D);
                fetch(t > 0 ? t - 1 : 0);
                f2 acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
                for (int i = 0; i < NP; i++) acc[i & 3] = ffma2(A[i], vg[i], acc[i & 3]);
                const float gs = f2_hsum(fadd2(fadd2(acc[0], acc[1]), fadd2(acc[2], acc[3])));
                if constexpr (V1) {
                    gh = gs;
                } else {
                    const float dotp = warp_sum_idx<1>(st * gs);
                    gh = st * (gs - dotp);
                }
                axpy2<NP>(A, vu, -kt);              // S_{t-1}: in the shadow of the reduction
            }
        } else if (role == 1) {
            // ------------------------------------------------------------ C: one chunk behind
            const long long tl = t0 + nt - 1;
            float* pgz = reinterpret_cast<float*>(p.gz.p) + n * p.gz.sN + h * p.gz.sH + tl * p.gz.sL + own;
            float* pgv = reinterpret_cast<float*>(p.gv.p) + n * p.gv.sN + h * p.gv.sH + tl * p.gv.sL + own;
#pragma unroll 4
            for (int t = nt - 1; t >= 0; t--) {
                float* e = rg + t * SM::kStep;
                f2 xs[NP / 2], kk[NP / 2];
                lds_slice<D / 2>(xs, s.od.f + t * D + 16 * half);
                lds_slice<D / 2>(kk, s.k.f + t * D + 16 * half);
                const float2 g2 = *reinterpret_cast<const float2*>(e + 2 * lp);
                const float beta = s.b.f[t], w = s.v.f[t * D + own] - s.vo.f[t * D + own];
                f2 d0 = 0ull, d1 = 0ull, d2 = 0ull;
#pragma unroll
                for (int i = 0; i < NP / 2; i++) {
                    d0 = ffma2(A[i], kk[i], d0);
                    d1 = ffma2(A[8 + i], kk[i], d1);
                    d2 = ffma2(xs[i], kk[i], d2);
                }
                const float p0 = f2_hsum(d0), p1 = f2_hsum(d1);
                float xk = f2_hsum(d2);
                xk += __shfl_xor_sync(0xffffffffu, xk, 16);
                const float r0 = (half ? p1 : p0) + __shfl_xor_sync(0xffffffffu, half ? p0 : p1, 16);
                const float g = half ? g2.y : g2.x;
                const float r = fmaf(xk, g, r0);                    // (G + s (x) dz)^T k
                const float dv = beta * r, dvo = __shfl_xor_sync(0xffffffffu, dv, 16);
                e[2 * D + own] = dv;
                const f2 g0 = f2_pack(g2.x, g2.x), g1 = f2_pack(g2.y, g2.y);
                const float n0 = half ? -dvo : -dv, n1 = half ? -dv : -dvo;
                const f2 m0 = f2_pack(n0, n0), m1 = f2_pack(n1, n1);
#pragma unroll
                for (int i = 0; i < NP / 2; i++) {
                    A[i] = ffma2(kk[i], m0, ffma2(xs[i], g0, A[i]));
                    A[8 + i] = ffma2(kk[i], m1, ffma2(xs[i], g1, A[8 + i]));
                }
                pw[t * (D + 4) + lane] = r * w;
                *pgz = g; *pgv = dv;
                pgz -= p.gz.sL; pgv -= p.gv.sL;
            }
            // dbeta of the whole chunk at once: 32 / TC lanes share a step
            __syncwarp();
            constexpr int SH = 32 / TC;
            const float* q = pw + (lane / SH) * (D + 4) + (lane % SH) * (D / SH);
            float db = 0.f;
#pragma unroll
            for (int i = 0; i < D / SH; i++) db += q[i];
#pragma unroll
            for (int o = SH / 2; o > 0; o >>= 1) db += __shfl_xor_sync(0xffffffffu, db, o);
            if (lane % SH == 0 && lane / SH < nt)
                reinterpret_cast<float*>(p.gb.p)[n * p.gb.sN + h * p.gb.sH + (long long)(t0 + lane / SH) * p.gb.sL] = db;
            __syncwarp();
        } else {
            // ------------------------------------------------------------ R: two chunks behind
            float* pgk = reinterpret_cast<float*>(p.gk.p) + n * p.gk.sN + h * p.gk.sH + (long long)(t0 + nt - 1) * p.gk.sL + own;
#pragma unroll 4
            for (int t = nt - 1; t >= 0; t--) {
                const float* e = rg + t * SM::kStep;
                const float2 se = *reinterpret_cast<const float2*>(s.od.f + t * D + 2 * lp), ke = *reinterpret_cast<const float2*>(s.k.f + t * D + 2 * lp);
                f2 vg[NP / 2], vu[NP / 2], vd[NP / 2];
                lds_slice<D / 2>(vg, e + 16 * half);
                lds_slice<D / 2>(vu, e + D + 16 * half);
                lds_slice<D / 2>(vd, e + 2 * D + 16 * half);
                const f2 s0 = f2_pack(se.x, se.x), s1 = f2_pack(se.y, se.y), k0 = f2_pack(-ke.x, -ke.x), k1 = f2_pack(-ke.y, -ke.y);
                f2 d0 = 0ull, d1 = 0ull, f0 = 0ull, f1 = 0ull;
#pragma unroll
                for (int i = 0; i < NP / 2; i++) {
                    B[i] = ffma2(vg[i], s0, B[i]);
                    B[8 + i] = ffma2(vg[i], s1, B[8 + i]);
                    A[i] = ffma2(vu[i], k0, A[i]);              // S_{t-1}
                    A[8 + i] = ffma2(vu[i], k1, A[8 + i]);
                    d0 = ffma2(B[i], vu[i], d0);
                    d1 = ffma2(B[8 + i], vu[i], d1);
                    f0 = ffma2(A[i], vd[i], f0);
                    f1 = ffma2(A[8 + i], vd[i], f1);
                    B[i] = ffma2(vd[i], k0, B[i]);
                    B[8 + i] = ffma2(vd[i], k1, B[8 + i]);
                }
                const float p0 = f2_hsum(d0) - f2_hsum(f0), p1 = f2_hsum(d1) - f2_hsum(f1);
                *pgk = (half ? p1 : p0) + __shfl_xor_sync(0xffffffffu, half ? p0 : p1, 16);
                pgk -= p.gk.sL;
            }
        }
    }
    if (role == 0) {
#pragma unroll
        for (int i = 0; i < NP; i++) {
            float lo, hi;
            f2_unpack(A[i], lo, hi);
            W[(long long)lane * p.wE + 2 * i] = lo;
            W[(long long)lane * p.wE + 2 * i + 1] = hi;
        }
    }
}

}  // namespace fwp
