// Backward of the bf16 chunk plan (E = M = 64, mathematics in fwp_delta_chunk_bf16.cuh) with a role per kind of work.
//
// What a chunk hands to the one before it is G alone, and that path is short: lambda = Lt + Kt G1, then
// G0 = G1 + Q^T gY - K^T (b lambda).  Everything else either needs neither G nor S (the Gram tiles, T', X, Kt, U) or hangs
// off the path (the rewind of S, dQ, dK).  One CTA per sequence, its roles a few chunks apart:
//   prepare  PW warps, whole chunks round robin: copies, w, U = b w, B, Gram tiles, T', X = Aqk T', Kt = T'^T K;
//   chain    four warps, sixteen value columns each: G, held transposed (rows m, columns e).  Its fragments, rounded to
//            bf16, are the left operand of G^T Kt^T, and those of (b lambda)^T the left operand of the update, so the
//            chain crosses neither lanes nor warps; the warps leave G1 (two bf16 parts) and b lambda in shared memory;
//   state    four warps, sixteen key rows each: S, its rewind, dQ, and the part of dK that S enters;
//   key      four warps, sixteen key columns each: the rest of dK, dv and dbeta.
// The roles meet at mbarriers, one arrival per warp, every wait bounded.  The kernel before this one ran chain, state and
// key in the same four warps between CTA-wide barriers: 4900 cycles per chunk alone on an SM and 2500 with three sequences
// per SM, against 1120 cycles of tensor pipe (542 products of 16 x 8 x 16) and about as many of shared memory.  Measured,
// 1024 steps: 128 sequences 165 -> 86 us, 256 206 -> 169, 432 271 -> 252 (chain and trail as two roles of two or four warps, two
// CTAs per SM: 106, 167, 273; their 128 registers a thread spill).
#pragma once
#include "fwp_delta_chunk_bf16.cuh"
#include "fwp_delta_tc.cuh"

namespace fwp {
namespace cb {

struct BwdStage {
    __nv_bfloat16 k[C * LDT], q[C * LDT], gy[C * LDT];      // inputs, [t][.]
    __nv_bfloat16 v[C * LDT];           // v, then Kt, [t][e]
    float vo[C * LDO];                  // v_old, [t][m]; becomes w = v - v_old in place
    uint4 fx[32];                       // X = Aqk T' as right-operand fragments
    __nv_bfloat16 uh[C * LDT], ul[C * LDT];     // U = b w as two bf16 parts, [t][m]
    __nv_bfloat16 bm[C * LDQ];          // B = lower(gY U^T), [t][i]
    float b[C];
};
template <int R>
struct BwdSmem {
    BwdStage stage[R];
    __nv_bfloat16 gh[D * LDT], gl[D * LDT];     // G1^T as two bf16 parts, [m][e]
    __nv_bfloat16 bl[2][C * LDT];       // b lambda = dv, [t][m]
    float4 dk[2][4][2][32];             // -(b lambda) S0^T, a fragment per key warp
    float dbp[2][4][C];                 // partial sums of dbeta over sixteen value columns each
    unsigned long long full[R], empty[R], gfull, gempty, blfull[2], dkfull[2];
};

__device__ __forceinline__ void bwd_wait(unsigned long long* bar, unsigned parity) {
    if (!mbar_wait_bounded(bar, parity)) atomicExch(&g_tc_fault, 1);
}
// one arrival per warp, after everything its lanes have done
__device__ __forceinline__ void bwd_arrive(unsigned long long* bar, int lane) {
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace cb

template <int PW, int R>
__global__ void __launch_bounds__((12 + PW) * 32, 1) delta_bwd_chunk_bf16_pipe_kernel(const DeltaBwdParams p) {
    using namespace cb;
    using bf16 = __nv_bfloat16;
    using SM = BwdSmem<R>;
    extern __shared__ __align__(16) unsigned char cb_smem[];
    SM& s = *reinterpret_cast<SM*>(cb_smem);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int seq = blockIdx.x, n = seq / p.H, h = seq - n * p.H;
    const int nchunks = (p.L + C - 1) / C;
    if (threadIdx.x == 0) {
        for (int i = 0; i < R; i++) {
            mbar_init(&s.full[i], 1);
            mbar_init(&s.empty[i], 12);
        }
        mbar_init(&s.gfull, 4);
        mbar_init(&s.gempty, 4);            // the key warps, who have by then seen the state warps finish the chunk before
        for (int i = 0; i < 2; i++) {
            mbar_init(&s.blfull[i], 4);
            mbar_init(&s.dkfull[i], 4);
        }
    }
    __syncthreads();
    griddep_wait();
    griddep_launch_dependents();

    if (warp >= 12) {
        // ------------------------------------------------------------ prepare
        const int first = warp - 12;
        const int r8 = lane >> 3, r16 = lane >> 4;      // rows of the first 16-byte piece this lane copies, bf16 and fp32 tiles
        const int o8 = r8 * LDT + (lane & 7) * 8, o16 = r16 * LDO + (lane & 15) * 4;
        const long long row = (long long)(nchunks - 1 - first) * C;
        auto at = [&](const Row4& r, int rr, int part) { return n * r.sN + h * r.sH + (row + rr) * r.sL + part; };
        const bf16* qp = reinterpret_cast<const bf16*>(p.q.p) + at(p.q, r8, (lane & 7) * 8);
        const bf16* kp = reinterpret_cast<const bf16*>(p.k.p) + at(p.k, r8, (lane & 7) * 8);
        const bf16* vp = reinterpret_cast<const bf16*>(p.v.p) + at(p.v, r8, (lane & 7) * 8);
        const bf16* yp = reinterpret_cast<const bf16*>(p.gy.p) + at(p.gy, r8, (lane & 7) * 8);
        const float* op = reinterpret_cast<const float*>(p.v_old.p) + at(p.v_old, r16, (lane & 15) * 4);
        const bf16* bp = reinterpret_cast<const bf16*>(p.beta.p) + at(p.beta, lane & 15, 0);
        float bnext = 0.f;
        auto stage_in = [&](int it) {       // all copies of the chunk processed it-th, by this warp; the pointers move on to its next
            BwdStage& d = s.stage[it % R];
            const int nt = min(C, p.L - (nchunks - 1 - it) * C);
            bwd_wait(&s.empty[it % R], ((it / R) & 1) ^ 1);     // passes at once the first time round
            auto tile = [&](bf16* dst, const bf16*& src, long long sL) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (nt == C || r8 + 4 * i < nt) cp_async16(dst + o8 + 4 * i * LDT, src + 4 * i * sL);
                    else *reinterpret_cast<uint4*>(dst + o8 + 4 * i * LDT) = make_uint4(0u, 0u, 0u, 0u);
                }
                src -= PW * C * sL;
            };
            tile(d.k, kp, p.k.sL);
            tile(d.q, qp, p.q.sL);
            tile(d.v, vp, p.v.sL);
            tile(d.gy, yp, p.gy.sL);
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (nt == C || r16 + 2 * i < nt) cp_async16(d.vo + o16 + 2 * i * LDO, op + 2 * i * p.v_old.sL);
                else *reinterpret_cast<float4*>(d.vo + o16 + 2 * i * LDO) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            op -= PW * C * p.v_old.sL;
            cp_async_commit();
            bnext = (lane & 15) < nt ? __bfloat162float(*bp) : 0.f;
            bp -= PW * C * p.beta.sL;
        };
        if (first < nchunks) stage_in(first);
#pragma unroll 1
        for (int it = first; it < nchunks; it += PW) {
            BwdStage& sg = s.stage[it % R];
            cp_async_wait<0>();
            if (lane < C) sg.b[lane] = bnext;
            __syncwarp();
            const bf16* Ks = sg.k;
            const bf16* Qs = sg.q;
            const bf16* Ys = sg.gy;
            float* Ws = sg.vo;
            const float* bs = sg.b;
            // w = v - v_old in place, U = b w in two bf16 parts: four elements of a row at a time, eight lanes to half a row
#pragma unroll
            for (int ii = 0; ii < 8; ii++) {
                const int r = r8 + 4 * (ii >> 1), c0 = 4 * (lane & 7) + 32 * (ii & 1);
                const uint2 vraw = *reinterpret_cast<const uint2*>(sg.v + r * LDT + c0);
                float4 w = *reinterpret_cast<const float4*>(Ws + r * LDO + c0);
                const __nv_bfloat162 va = *reinterpret_cast<const __nv_bfloat162*>(&vraw.x), vb = *reinterpret_cast<const __nv_bfloat162*>(&vraw.y);
                w = make_float4(__low2float(va) - w.x, __high2float(va) - w.y, __low2float(vb) - w.z, __high2float(vb) - w.w);
                *reinterpret_cast<float4*>(Ws + r * LDO + c0) = w;
                const float br = bs[r];
                uint2 hi, lo;
                split_bf16(br * w.x, br * w.y, hi.x, lo.x);
                split_bf16(br * w.z, br * w.w, hi.y, lo.y);
                *reinterpret_cast<uint2*>(sg.uh + r * LDT + c0) = hi;
                *reinterpret_cast<uint2*>(sg.ul + r * LDT + c0) = lo;
            }
            __syncwarp();
            {   // B = lower(gY U^T)
                float acc[2][4] = {};
                unsigned b4[4];
#pragma unroll
                for (int ks = 0; ks < 4; ks++) {
                    unsigned ya[4], bu[4];
                    lda_rowmajor(ya, Ys + 16 * ks, LDT, lane);
                    ldb_nk(bu, sg.uh + 16 * ks, LDT, lane);
                    mm(acc, ya, bu);
                }
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (8 * (i >> 2) + 2 * t4 + (i & 1) > g + 8 * ((i >> 1) & 1)) acc[i >> 2][i & 3] = 0.f;
                a_of(b4, acc);
                stsm4(sg.bm + (lane & 15) * LDQ + 8 * (lane >> 4), b4);
            }
            if (it + PW < nchunks) stage_in(it + PW);   // half a chunk of work before it is waited for
            unsigned bX[4];
            float Y[2][4];
            {
            float akk[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            float aqk[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
                unsigned ak[4], aq[4];
                lda_rowmajor(ak, Ks + 16 * ks, LDT, lane);      // also K^T as right operand
                lda_rowmajor(aq, Qs + 16 * ks, LDT, lane);
                mma_bf16(akk[0], ak, ak[0], ak[2]);
                mma_bf16(akk[1], ak, ak[1], ak[3]);
                mma_bf16(aqk[0], aq, ak[0], ak[2]);
                mma_bf16(aqk[1], aq, ak[1], ak[3]);
            }
            float N1[2][4];
#pragma unroll
            for (int j = 0; j < 2; j++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int r = g + 8 * (i >> 1), cc = 8 * j + 2 * t4 + (i & 1);
                    N1[j][i] = cc < r ? akk[j][i] * bs[r] : 0.f;
                    aqk[j][i] = cc <= r ? aqk[j][i] : 0.f;
                    Y[j][i] = -N1[j][i];
                }
            unsigned a[4], bN[4], b2[4], b4[4];
            float N2[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            a_of(a, N1);
            b_of(bN, N1);
            mm(N2, a, bN);
            b_of(b2, N2);
            {
                float N3[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                mm(N3, a, b2);
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int i = 0; i < 4; i++) Y[j][i] += N2[j][i] - N3[j][i];
            }
            float N4[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            a_of(a, N2);
            mm(N4, a, b2);
            b_of(b4, N4);
            {
                float Z1[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                a_of(a, Y);
                mm(Z1, a, b4);
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int i = 0; i < 4; i++) Y[j][i] += N4[j][i] + Z1[j][i];
            }
            {
                float N8[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                a_of(a, N4);
                mm(N8, a, b4);
                unsigned b8[4];
                b_of(b8, N8);
                float Z2[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                a_of(a, Y);
                mm(Z2, a, b8);
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int i = 0; i < 4; i++) Y[j][i] += N8[j][i] + Z2[j][i];
            }
            {   // X = Aqk T' = Aqk + Aqk (T' - I)
                unsigned by[4];
                b_of(by, Y);
                a_of(a, aqk);
                mm(aqk, a, by);
                b_of(bX, aqk);
            }
            }
            sg.fx[lane] = make_uint4(bX[0], bX[1], bX[2], bX[3]);
            {   // Kt = T'^T K, sixteen columns at a time: the left operand is the transposed fragment, in two bf16 parts
                float T[2][4];
#pragma unroll
                for (int j = 0; j < 2; j++)
#pragma unroll
                    for (int i = 0; i < 4; i++) T[j][i] = Y[j][i] + ((8 * j + 2 * t4 + (i & 1)) == (g + 8 * (i >> 1)) ? 1.f : 0.f);
                unsigned ah[4], al[4], th2[4], tl2[4];
                split_bf16(T[0][0], T[0][1], ah[0], al[0]); split_bf16(T[0][2], T[0][3], ah[1], al[1]);
                split_bf16(T[1][0], T[1][1], ah[2], al[2]); split_bf16(T[1][2], T[1][3], ah[3], al[3]);
                th2[0] = movm(ah[0]); th2[1] = movm(ah[2]); th2[2] = movm(ah[1]); th2[3] = movm(ah[3]);
                tl2[0] = movm(al[0]); tl2[1] = movm(al[2]); tl2[2] = movm(al[1]); tl2[3] = movm(al[3]);
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    unsigned bK[4], k4[4];
                    ldb_kn(bK, Ks + 16 * w, LDT, lane);
                    float kt[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                    mm(kt, th2, bK);
                    mm(kt, tl2, bK);
                    a_of(k4, kt);
                    stsm4(sg.v + (lane & 15) * LDT + 16 * w + 8 * (lane >> 4), k4);
                }
            }
            bwd_arrive(&s.full[it % R], lane);
        }
        return;
    }

    if (warp < 4) {
        // ------------------------------------------------------------ chain
        const int m0 = 16 * warp;
        float G[8][4] = {};                 // G^T: rows m0 + g (+8), columns 8 j + 2 t4, +1
#pragma unroll 1
        for (int it = 0; it < nchunks; it++) {
            const BwdStage& sg = s.stage[it % R];
            unsigned gh[4][4], ya[4], bX[4];        // gh: G1^T rounded to bf16, left operand
            bwd_wait(&s.gempty, (it & 1) ^ 1);
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
                unsigned lo[4];
                const int o = (m0 + (lane & 15)) * LDT + 16 * ks + 8 * (lane >> 4);
#pragma unroll
                for (int i = 0; i < 4; i++)
                    split_bf16(G[2 * ks + (i >> 1)][2 * (i & 1)], G[2 * ks + (i >> 1)][2 * (i & 1) + 1], gh[ks][i], lo[i]);
                stsm4(s.gh + o, gh[ks]);
                stsm4(s.gl + o, lo);
            }
            bwd_arrive(&s.gfull, lane);
            bwd_wait(&s.full[it % R], (it / R) & 1);
            {
                const uint4 f = sg.fx[lane];
                bX[0] = f.x; bX[1] = f.y; bX[2] = f.z; bX[3] = f.w;
            }
            float lm[2][4] = {};            // lambda^T: Lt^T + G1^T Kt^T, Lt^T = gY^T X
            lda_trans(ya, sg.gy + m0, LDT, lane);
            mm(lm, ya, bX);
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
                unsigned bk[4];
                ldb_nk(bk, sg.v + 16 * ks, LDT, lane);
                mm(lm, gh[ks], bk);
            }
            // the half of G's update that does not wait for lambda
#pragma unroll
            for (int jp = 0; jp < 4; jp++) {
                unsigned bq[4];
                ldb_kn(bq, sg.q + 16 * jp, LDT, lane);
                mma_bf16(G[2 * jp], ya, bq[0], bq[1]);
                mma_bf16(G[2 * jp + 1], ya, bq[2], bq[3]);
            }
            unsigned la[4];                 // (b lambda)^T
            float db[2][2] = {};
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int t = 8 * j + 2 * t4;
                const float2 b2 = *reinterpret_cast<const float2*>(sg.b + t);
#pragma unroll
                for (int hr = 0; hr < 2; hr++) {
                    const float* w = sg.vo + t * LDO + m0 + g + 8 * hr;
                    const float l0 = lm[j][2 * hr], l1 = lm[j][2 * hr + 1];
                    db[j][0] = fmaf(l0, w[0], db[j][0]);
                    db[j][1] = fmaf(l1, w[LDO], db[j][1]);
                    la[2 * j + hr] = pack_bf16(b2.x * l0, b2.y * l1);
                }
            }
            stsm4t(s.bl[it & 1] + ((lane & 7) + 8 * (lane >> 4)) * LDT + m0 + 8 * ((lane >> 3) & 1), la);
            {   // four sums over the eight lanes that share t4: a lane gives half of its values away at a time.  Upper half of the warp
                // first: 9.05 -> 8.95 ms at 4096 sequences x 4096 steps; the other way round it took 9.17
                const bool h4 = lane & 16, h3 = lane & 8;
                const float x0 = (h4 ? db[1][0] : db[0][0]) + __shfl_xor_sync(0xffffffffu, h4 ? db[0][0] : db[1][0], 16);
                const float x1 = (h4 ? db[1][1] : db[0][1]) + __shfl_xor_sync(0xffffffffu, h4 ? db[0][1] : db[1][1], 16);
                float x = (h3 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, h3 ? x0 : x1, 8);
                x += __shfl_xor_sync(0xffffffffu, x, 4);
                if (!(lane & 4)) s.dbp[it & 1][warp][8 * (lane >> 4) + 2 * t4 + ((lane >> 3) & 1)] = x;
            }
            bwd_arrive(&s.blfull[it & 1], lane);
            neg4(la, la);
#pragma unroll
            for (int jp = 0; jp < 4; jp++) {
                unsigned bk[4];
                ldb_kn(bk, sg.k + 16 * jp, LDT, lane);
                mma_bf16(G[2 * jp], la, bk[0], bk[1]);
                mma_bf16(G[2 * jp + 1], la, bk[2], bk[3]);
            }
            bwd_arrive(&s.empty[it % R], lane);
        }
        return;
    }

    // what a state or key warp stores: its sixteen columns of dQ or dK, rows g and g + 8, four columns per lane.  Neighbouring
    // lanes swap halves so that four of them store a whole 32-byte sector (4-byte stores, two to a sector, took twice as long)
    const int e0 = 16 * (warp & 3);
    const long long last = (long long)(nchunks - 1) * C;
    auto at = [&](const Row4& r, int rr, int c) { return reinterpret_cast<bf16*>(r.p) + n * r.sN + h * r.sH + (last + rr) * r.sL + c; };
    const int col = e0 + 8 * (t4 & 1) + 4 * (t4 >> 1);
    auto put = [&](bf16* dst, long long sL, const float (&x)[2][4], int nt) {
#pragma unroll
        for (int hr = 0; hr < 2; hr++) {
            const unsigned x0 = pack_bf16(x[0][2 * hr], x[0][2 * hr + 1]), x1 = pack_bf16(x[1][2 * hr], x[1][2 * hr + 1]);
            const unsigned got = __shfl_xor_sync(0xffffffffu, (t4 & 1) ? x0 : x1, 1);
            if (g + 8 * hr < nt) *reinterpret_cast<uint2*>(dst + 8 * hr * sL) = (t4 & 1) ? make_uint2(got, x1) : make_uint2(x0, got);
        }
    };

    if (warp < 8) {
        // ------------------------------------------------------------ state: S, its rewind, dQ, and S's part of dK
        bf16* gq = at(p.gq, g, col);
        float* W = p.W + n * p.wN + h * p.wH + (long long)(e0 + g) * p.wE + 2 * t4;
        float S[8][4];                      // rows e0 + g (+8), columns 8 j + 2 t4, +1
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float2 x = *reinterpret_cast<const float2*>(W + (long long)(8 * (i & 1)) * p.wE + 8 * (i >> 1));
            S[i >> 1][2 * (i & 1)] = x.x; S[i >> 1][2 * (i & 1) + 1] = x.y;
        }
#pragma unroll 1
        for (int it = 0; it < nchunks; it++) {
            const BwdStage& sg = s.stage[it % R];
            bwd_wait(&s.full[it % R], (it / R) & 1);
            unsigned ka[4], kan[4], bh[4][4], bl[4][4];
            lda_trans(ka, sg.k + e0, LDT, lane);    // K^T, left operand; its registers are also K as right operand
            neg4(kan, ka);
#pragma unroll
            for (int jp = 0; jp < 4; jp++) {
                ldb_kn(bh[jp], sg.uh + 16 * jp, LDT, lane);
                ldb_kn(bl[jp], sg.ul + 16 * jp, LDT, lane);
            }
#pragma unroll
            for (int jp = 0; jp < 4; jp++) {        // rewind: S0 = S1 - K^T U
                mma_bf16(S[2 * jp], kan, bh[jp][0], bh[jp][1]);
                mma_bf16(S[2 * jp + 1], kan, bh[jp][2], bh[jp][3]);
            }
#pragma unroll
            for (int jp = 0; jp < 4; jp++) {
                mma_bf16(S[2 * jp], kan, bl[jp][0], bl[jp][1]);
                mma_bf16(S[2 * jp + 1], kan, bl[jp][2], bl[jp][3]);
            }
            unsigned ya[4][4], ba[4];
#pragma unroll
            for (int ks = 0; ks < 4; ks++) lda_rowmajor(ya[ks], sg.gy + 16 * ks, LDT, lane);
            lda_rowmajor(ba, sg.bm, LDQ, lane);
            bwd_arrive(&s.empty[it % R], lane);
            unsigned sh[4][4], sl[4][4];            // S0 as right operand, contraction over m
            float dq[2][4] = {}, dq2[2][4] = {};    // two sums each: half as long a chain of products
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {        // dQ = gY S0^T + B K
#pragma unroll
                for (int i = 0; i < 4; i++)
                    split_bf16(S[2 * ks + (i & 1)][2 * (i >> 1)], S[2 * ks + (i & 1)][2 * (i >> 1) + 1], sh[ks][i], sl[ks][i]);
                mm(dq, ya[ks], sh[ks]);
                mm(dq2, ya[ks], sl[ks]);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) dq[i >> 2][i & 3] += dq2[i >> 2][i & 3];
            const unsigned bK[4] = {ka[0], ka[2], ka[1], ka[3]};
            mm(dq, ba, bK);
            bwd_wait(&s.blfull[it & 1], (it >> 1) & 1);
            float dk[2][4] = {}, dk2[2][4] = {};
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
                unsigned la[4];
                lda_rowmajor(la, s.bl[it & 1] + 16 * ks, LDT, lane);
                neg4(la, la);
                mm(dk, la, sh[ks]);
                mm(dk2, la, sl[ks]);
            }
            put(gq, p.gq.sL, dq, min(C, p.L - (nchunks - 1 - it) * C));
            gq -= C * p.gq.sL;
            // this buffer was read two chunks ago, before the key warps let the chain pass to the chunk after it
#pragma unroll
            for (int j = 0; j < 2; j++)
                s.dk[it & 1][warp & 3][j][lane] = make_float4(dk[j][0] + dk2[j][0], dk[j][1] + dk2[j][1], dk[j][2] + dk2[j][2], dk[j][3] + dk2[j][3]);
            bwd_arrive(&s.dkfull[it & 1], lane);
        }
#pragma unroll
        for (int i = 0; i < 16; i++)
            *reinterpret_cast<float2*>(W + (long long)(8 * (i & 1)) * p.wE + 8 * (i >> 1)) = make_float2(S[i >> 1][2 * (i & 1)], S[i >> 1][2 * (i & 1) + 1]);
        return;
    }

    // ---------------------------------------------------------------- key: the rest of dK, dv, dbeta
    bf16* gk = at(p.gk, g, col);
    const int vrow = 4 * (warp & 3) + (lane >> 3);
    bf16* gv = at(p.gv, vrow, (lane & 7) * 8);
    bf16* gb = at(p.gb, lane & 15, 0);
#pragma unroll 1
    for (int it = 0; it < nchunks; it++) {
        const BwdStage& sg = s.stage[it % R];
        const int nt = min(C, p.L - (nchunks - 1 - it) * C);
        bwd_wait(&s.full[it % R], (it / R) & 1);
        unsigned ua[4][4], ula[4][4], bta[4], bQ[4], bK[4];
#pragma unroll
        for (int ks = 0; ks < 4; ks++) {
            lda_rowmajor(ua[ks], sg.uh + 16 * ks, LDT, lane);
            lda_rowmajor(ula[ks], sg.ul + 16 * ks, LDT, lane);
        }
        lda_trans(bta, sg.bm, LDQ, lane);
        ldb_kn(bQ, sg.q + e0, LDT, lane);
        ldb_kn(bK, sg.k + e0, LDT, lane);
        bwd_arrive(&s.empty[it % R], lane);
        bwd_wait(&s.gfull, it & 1);
        unsigned bh[4][4], bl[4][4];
#pragma unroll
        for (int ks = 0; ks < 4; ks++) {
            ldb_kn(bh[ks], s.gh + 16 * ks * LDT + e0, LDT, lane);
            ldb_kn(bl[ks], s.gl + 16 * ks * LDT + e0, LDT, lane);
        }
        bwd_arrive(&s.gempty, lane);
        float dk[2][4] = {}, dk2[2][4] = {};
#pragma unroll
        for (int ks = 0; ks < 4; ks++) {    // U G1^T + B^T Q
            mm(dk, ua[ks], bh[ks]);
            mm(dk2, ua[ks], bl[ks]);
            mm(dk2, ula[ks], bh[ks]);
        }
        mm(dk, bta, bQ);
        bwd_wait(&s.blfull[it & 1], (it >> 1) & 1);
        const bf16* lam = s.bl[it & 1];
        float Z[2][4] = {};                 // (b lambda) U^T
#pragma unroll
        for (int ks = 0; ks < 4; ks++) {
            unsigned la[4];
            lda_rowmajor(la, lam + 16 * ks, LDT, lane);
            mma_bf16(Z[0], la, ua[ks][0], ua[ks][2]);       // the left operand of U is the right operand of U^T
            mma_bf16(Z[1], la, ua[ks][1], ua[ks][3]);
        }
        if (vrow < nt) *reinterpret_cast<uint4*>(gv) = *reinterpret_cast<const uint4*>(lam + vrow * LDT + (lane & 7) * 8);
        if (warp == 8 && lane < nt) {
            const float (*db)[C] = s.dbp[it & 1];
            *gb = __float2bfloat16_rn(db[0][lane] + db[1][lane] + db[2][lane] + db[3][lane]);
        }
        unsigned za[4], zl[4];              // -(strict_lower(Z) + its mirror image)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = g + 8 * (i & 1), cc = 8 * (i >> 1) + 2 * t4;
            zl[i] = pack_bf16(cc < r ? -Z[i >> 1][2 * (i & 1)] : 0.f, cc + 1 < r ? -Z[i >> 1][2 * (i & 1) + 1] : 0.f);
        }
        za[0] = zl[0] | movm(zl[0]);
        za[1] = zl[1];
        za[2] = movm(zl[1]);
        za[3] = zl[3] | movm(zl[3]);
        mm(dk, za, bK);
        bwd_wait(&s.dkfull[it & 1], (it >> 1) & 1);
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float4 x = s.dk[it & 1][warp & 3][j][lane];
            dk[j][0] += dk2[j][0] + x.x; dk[j][1] += dk2[j][1] + x.y; dk[j][2] += dk2[j][2] + x.z; dk[j][3] += dk2[j][3] + x.w;
        }
        put(gk, p.gk.sL, dk, nt);
        gk -= C * p.gk.sL;
        gv -= C * p.gv.sL;
        gb -= C * p.gb.sL;
    }
}

}  // namespace fwp
