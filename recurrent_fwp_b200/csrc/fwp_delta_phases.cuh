// Delta rule backward in chunks of sixteen steps, as three launches over a workspace (sm_100a).
//
// In WY form almost everything of a chunk can be computed without knowing the state at its border.  A kernel that runs
// a whole sequence per CTA leaves that parallelism unused: with 16 sequences it keeps 16 SMs busy.  Here
//   prepare   one warp per chunk, all chunks at once: what the chain needs, in operand form;
//   chain     one warp per sequence and 16 state columns: two 16-deep products per chunk, nothing else (and, beside
//             it, the rewind of the state, a plain running difference);
//   finish    one warp per chunk, all chunks at once: the gradients, from the states at the chunk's borders.
// With w = V - v_old, u = diag(beta) w known from the forward, G = dL/dS after the chunk, S0 the state before it:
//   r  = Tv + X G,    X = T' K,  Tv = T' triu(K Q^T) gY,  T' = (I + striu(K K^T) diag(beta))^-1
//   G += Q^T gY - K^T diag(beta) r,     S0 = S - K^T U                                        (chain)
//   b = diag(beta) r = dV,   dbeta_i = r_i . w_i,   dQ = gY S0^T + H K,   H = tril(gY U^T)
//   dK = U G^T - b S0^T + H^T Q - R K,  R_ij = u_min(i,j) . b_max(i,j)  (i != j)               (finish)
// All products are split fp32 products (fwp_split3.cuh).  The workspace holds operands as ready fragments, 16 bytes per
// lane, so that every access to it is a coalesced 512-byte line per warp; it is meant to stay in the L2 cache, and larger
// calls are cut into segments of time, then into groups of sequences, that do.  Each kernel is short enough to stay in the instruction cache (one kernel with a
// role per phase was not: instruction fetch was its largest stall, and two sequences per SM took twice as long as one).
//
// Values that are not finite.  As in the forward (fwp_delta_wy.cuh), a chunk's products would carry a NaN or Inf to steps of
// the chunk that do not depend on it: here to gradients of later steps.  What can do so ends up in G or in the rewound
// state, and stays there (both are running sums), so the chain kernel looks at the two when it is through with a segment
// and marks the sequence; finish writes nothing for marked sequences, and in the last segment the warp of chunk 0 does
// the sequence again step by step (stepwise_backward).
#pragma once
#include "fwp_wy_common.cuh"

namespace fwp {
namespace wy {

template <int E, int M, int NP>
struct BwdSpace {                       // one chunk, in uint4
    static constexpr int KS = E / 16, MS = M / 16;
    static constexpr int X = 0;                         // T' K, right operand by rows        [KS][3][32]
    static constexpr int K = X + KS * 3 * 32;           // K, right operand by columns        [KS][NP][32]
    static constexpr int Q = K + KS * NP * 32;          // Q, the same                        [KS][NP][32]
    static constexpr int R = Q + KS * NP * 32;          // Tv, then r (transposed, fp32)      [MS][2][32]
    static constexpr int G = R + MS * 64;               // (Q^T gY)^T, then G^T after the chunk [MS][KS][2][32]
    static constexpr int S = G + MS * KS * 64;          // K^T U, then S0                     [KS][MS][2][32]
    static constexpr int B = S + MS * KS * 64;          // beta
    static constexpr int kSize = B + 4;
};

struct BwdPhase {
    DeltaBwdParams p;
    uint4* ws;                          // [sequence of the group][chunk of the segment]
    uint4* carry;                       // [sequence of the group][MS][KS][2][32]: G^T between segments
    int* again;                         // [sequence of the group]: something that is not finite turned up
    int s0, ns;                         // the group: sequences [s0, s0 + ns)
    int c0, nc;                         // the segment: chunks [c0, c0 + nc)
    int first;                          // 1: the last chunks of the sequence, G starts from zero
};

template <int NP>
__device__ __forceinline__ void put_frag(uint4* at, const Frag<NP>& f, int lane) {
#pragma unroll
    for (int i = 0; i < NP; i++) at[i * 32 + lane] = make_uint4(f.r[i][0], f.r[i][1], f.r[i][2], f.r[i][3]);
}
template <int NP>
__device__ __forceinline__ void get_frag(Frag<NP>& f, const uint4* at, int lane) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
        const uint4 v = at[i * 32 + lane];
        f.r[i][0] = v.x; f.r[i][1] = v.y; f.r[i][2] = v.z; f.r[i][3] = v.w;
    }
}
__device__ __forceinline__ void put_block(uint4* at, const float (&x)[2][4], int lane) {
#pragma unroll
    for (int i = 0; i < 2; i++)
        at[i * 32 + lane] = make_uint4(__float_as_uint(x[i][0]), __float_as_uint(x[i][1]), __float_as_uint(x[i][2]), __float_as_uint(x[i][3]));
}
__device__ __forceinline__ void get_block(float (&x)[2][4], const uint4* at, int lane) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint4 v = at[i * 32 + lane];
        x[i][0] = __uint_as_float(v.x); x[i][1] = __uint_as_float(v.y); x[i][2] = __uint_as_float(v.z); x[i][3] = __uint_as_float(v.w);
    }
}
__device__ __forceinline__ void zero(float (&x)[2][4]) {
#pragma unroll
    for (int i = 0; i < 8; i++) x[i >> 2][i & 3] = 0.f;
}
// x[.][step] *= beta[step] for a block whose columns are steps
__device__ __forceinline__ void scale_steps(float (&x)[2][4], const float (&b)[2][2]) {
#pragma unroll
    for (int i = 0; i < 8; i++) x[i >> 2][i & 3] *= b[i >> 2][i & 1];
}
template <typename T>
__device__ __forceinline__ T* stream_at(const Row4& r, int n, int h) {
    return reinterpret_cast<T*>(r.p) + n * r.sN + h * r.sH;
}
// beta of the steps a lane's columns stand for (2t, 2t+1, 2t+8, 2t+9); 0 past the end
template <typename T>
__device__ __forceinline__ void load_beta(float (&b)[2][2], const T* p, long long sL, int nt, int t) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int s = 8 * (i >> 1) + 2 * t + (i & 1);
        b[i >> 1][i & 1] = s < nt ? to_f32(p[s * sL]) : 0.f;
    }
}

template <int K>
__device__ __forceinline__ bool finite(const float (&x)[K][2][4]) {
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
        for (int i = 0; i < 8; i++) acc = fmaf(x[k][i >> 2][i & 3], 0.f, acc);
    return acc == 0.f;
}

// The recurrence of one sequence backwards as it stands, by one warp whose lanes own state columns.  W holds the rewound
// state; S is brought forward from it with the u of the forward first.  `G` and `S` hold E x M floats each and `vec` 2 M, all
// of them this warp's own (the arrays hold whole blocks of rows, so BT of them can be in flight at a time: the loop is nothing
// but latency).  Inlined, for the reason stepwise_forward is.
template <typename T>
__device__ __forceinline__ void stepwise_backward(const DeltaBwdParams& p, int n, int h, float* G, float* S, float* vec) {
    const int lane = threadIdx.x & 31, E = p.E, M = p.M;
    const T *qp = stream_at<T>(p.q, n, h), *kp = stream_at<T>(p.k, n, h), *vp = stream_at<T>(p.v, n, h), *bp = stream_at<T>(p.beta, n, h);
    const T* yp = stream_at<T>(p.gy, n, h);
    const float* op = stream_at<float>(p.v_old, n, h);
    T *gqp = stream_at<T>(p.gq, n, h), *gkp = stream_at<T>(p.gk, n, h), *gvp = stream_at<T>(p.gv, n, h), *gbp = stream_at<T>(p.gb, n, h);
    const float* W = p.W + n * p.wN + h * p.wH;
    float *us = vec, *bs = vec + M;
    constexpr int BT = 8;
    auto at = [&](const T* row, int e) { return e < E ? to_f32(row[e]) : 0.f; };
    for (int m = lane; m < M; m += 32) {
#pragma unroll 1
        for (int e = 0; e < E; e++) {
            S[e * M + m] = W[(long long)e * p.wE + m];
            G[e * M + m] = 0.f;
        }
        for (long long t = 0; t < p.L; t++) {
            const float u = to_f32(bp[t * p.beta.sL]) * (to_f32(vp[t * p.v.sL + m]) - op[t * p.v_old.sL + m]);
#pragma unroll 1
            for (int e = 0; e < E; e += BT) {
                float s[BT];
#pragma unroll
                for (int i = 0; i < BT; i++) s[i] = fmaf(at(kp + t * p.k.sL, e + i), u, S[(e + i) * M + m]);
#pragma unroll
                for (int i = 0; i < BT; i++) S[(e + i) * M + m] = s[i];
            }
        }
    }
    for (long long t = p.L - 1; t >= 0; t--) {
        const T *q = qp + t * p.q.sL, *k = kp + t * p.k.sL, *y = yp + t * p.gy.sL;
        const float beta = to_f32(bp[t * p.beta.sL]);
        float db = 0.f;
        for (int m = lane; m < M; m += 32) {
            const float gy = to_f32(y[m]), w = to_f32(vp[t * p.v.sL + m]) - op[t * p.v_old.sL + m];
            float r = 0.f;
#pragma unroll 1
            for (int e = 0; e < E; e += BT) {
                float x[BT];
#pragma unroll
                for (int i = 0; i < BT; i++) x[i] = fmaf(at(q, e + i), gy, G[(e + i) * M + m]);
#pragma unroll
                for (int i = 0; i < BT; i++) {
                    G[(e + i) * M + m] = x[i];
                    if (e + i < E) r = fmaf(x[i], to_f32(k[e + i]), r);
                }
            }
            db = fmaf(r, w, db);
            us[m] = beta * w;
            bs[m] = beta * r;
            gvp[t * p.gv.sL + m] = from_f32<T>(beta * r);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) db += __shfl_xor_sync(0xffffffffu, db, o);
        if (lane == 0) gbp[t * p.gb.sL] = from_f32<T>(db);
#pragma unroll 1
        for (int e = 0; e < E; e += BT) {
            float dq[BT] = {}, dk[BT] = {};
#pragma unroll 1
            for (int m = lane; m < M; m += 32) {
                const float u = us[m], b = bs[m], gy = to_f32(y[m]);
                float s[BT], x[BT];
#pragma unroll
                for (int i = 0; i < BT; i++) {
                    s[i] = S[(e + i) * M + m];
                    x[i] = G[(e + i) * M + m];
                }
#pragma unroll
                for (int i = 0; i < BT; i++) {
                    const float ke = at(k, e + i), s0 = fmaf(-ke, u, s[i]);
                    dq[i] = fmaf(s[i], gy, dq[i]);
                    dk[i] = fmaf(x[i], u, fmaf(-s0, b, dk[i]));
                    S[(e + i) * M + m] = s0;
                    G[(e + i) * M + m] = fmaf(-ke, b, x[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < BT; i++) {
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    dq[i] += __shfl_xor_sync(0xffffffffu, dq[i], o);
                    dk[i] += __shfl_xor_sync(0xffffffffu, dk[i], o);
                }
                if (lane == i && e + i < E) {
                    gqp[t * p.gq.sL + e + i] = from_f32<T>(dq[i]);
                    gkp[t * p.gk.sL + e + i] = from_f32<T>(dk[i]);
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------ prepare
template <int E, int NP>
struct PrepareSmem {                    // per warp
    static constexpr int P = E + 8;
    __nv_bfloat16 K[NP][C][P], Q[NP][C][P], Tt[3][C][PC];
    float A[C][C + 4];
};

template <int E, int M, int WARPS, typename T>
__global__ void __launch_bounds__(WARPS * 32) delta_bwd_prepare_kernel(const __grid_constant__ BwdPhase a) {
    constexpr int KS = E / 16, MS = M / 16, NP = stream_parts<T>();
    using Sp = BwdSpace<E, M, NP>;
    using Sm = PrepareSmem<E, NP>;
    constexpr int P = Sm::P, kPart = C * P * 2, kPartC = C * PC * 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const DeltaBwdParams& p = a.p;
    const long long unit = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
    const int seq = (int)(unit / a.nc), c = a.c0 + (int)(unit - (long long)seq * a.nc);
    griddep_wait();
    griddep_launch_dependents();
    if (seq >= a.ns) return;
    Sm& sm = reinterpret_cast<Sm*>(smem_raw)[threadIdx.x >> 5];
    const int n = (a.s0 + seq) / p.H, h = a.s0 + seq - n * p.H, t0 = c * C, nt = min(C, p.L - t0);
    if (a.first && c == a.c0 && lane == 0) a.again[seq] = 0;
    uint4* const ws = a.ws + unit * Sp::kSize;
    const unsigned at = 2 * lane_at(lane, P), atC = 2 * lane_at(lane, PC);
    const unsigned aK = smem_u32(&sm.K[0][0][0]) + at, aQ = smem_u32(&sm.Q[0][0][0]) + at;
    const T* vp = stream_at<T>(p.v, n, h) + (t0 + 2 * t) * p.v.sL + g;
    const T* yp = stream_at<T>(p.gy, n, h) + (t0 + 2 * t) * p.gy.sL + g;
    const float* op = stream_at<float>(p.v_old, n, h) + (t0 + 2 * t) * p.v_old.sL + g;
    float sy[2][4], sv[2][4], so[2][4];       // gY, V, v_old of the next slice, requested early
    auto streams = [&](int j) {
        const int width = p.M - 16 * j;
        load_block_t<T>(sy, yp + 16 * j, p.gy.sL, nt, width, g, t);
        load_block_t<T>(sv, vp + 16 * j, p.v.sL, nt, width, g, t);
        load_block_t<float>(so, op + 16 * j, p.v_old.sL, nt, width, g, t);
    };
    float bt[2][2];
    load_beta(bt, stream_at<T>(p.beta, n, h) + t0 * p.beta.sL, p.beta.sL, nt, t);
    constexpr bool kAhead = KS <= 4, kRolled = KS > 4 && KS <= 6 && MS <= 2;
    // rolled loops over the blocks: less to fetch, slower to run.  Training pass, rolled over unrolled: E up to 96, M up to 32 0.95-1.00 (4 to
    // 320 sequences); 128, 32 0.97-0.99 up to 144 sequences, 1.01 with 320; 128, 64 0.98-1.04; 128, 128 1.03-1.08
    constexpr int kUnroll = kRolled ? 1 : KS;
    if (kAhead) streams(0);
    if (g == 0) {
#pragma unroll
        for (int i = 0; i < 4; i++) reinterpret_cast<float*>(ws + Sp::B)[8 * (i >> 1) + 2 * t + (i & 1)] = bt[i >> 1][i & 1];
    }
    float kk[2][4], z[2][4];
    {
        const T* kp = stream_at<T>(p.k, n, h) + (t0 + g) * p.k.sL + 2 * t;
        const T* qp = stream_at<T>(p.q, n, h) + (t0 + g) * p.q.sL + 2 * t;
        auto even = [&](const T* q, long long sL) { return p.E == E && (reinterpret_cast<uintptr_t>(q) & (2 * sizeof(T) - 1)) == 0 && (sL & 1) == 0; };
        const bool kpair = even(kp, p.k.sL), qpair = even(qp, p.q.sL);
        constexpr int AHEAD = KS < 2 ? KS : kRolled ? 1 : 2;
        float x[AHEAD][2][4], y[AHEAD][2][4];
        auto fetch = [&](int k) {
            load_block<T>(x[k % AHEAD], kp + 16 * k, p.k.sL, nt, p.E - 16 * k, kpair, g, t);
            load_block<T>(y[k % AHEAD], qp + 16 * k, p.q.sL, nt, p.E - 16 * k, qpair, g, t);
        };
#pragma unroll
        for (int k = 0; k < AHEAD; k++) fetch(k);
        if (kRolled) {
            zero(kk);
            zero(z);
        }
#pragma unroll kUnroll
        for (int k = 0; k < KS; k++) {
            Frag<NP> fk, fq;
            from_c(fk, x[k % AHEAD][0], x[k % AHEAD][1]);
            from_c(fq, y[k % AHEAD][0], y[k % AHEAD][1]);
            if (k + AHEAD < KS) fetch(k + AHEAD);
            store(aK + 32 * k, kPart, fk);
            store(aQ + 32 * k, kPart, fq);
            sum_product<BY_ROWS>(kRolled ? 1 : k, kk, fk, fk);
            sum_product<BY_ROWS>(kRolled ? 1 : k, z, fk, fq);
        }
    }
#pragma unroll
    for (int nn = 0; nn < 2; nn++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int row = g + 8 * (i >> 1), col = 8 * nn + 2 * t + (i & 1);
            if (col < row) z[nn][i] = 0.f;
            sm.A[C - 1 - row][C - 1 - col] = col > row ? kk[nn][i] * bt[nn][i & 1] : 0.f;
        }
    __syncwarp();
    invert_lower<C + 4, true>(&sm.A[0][0], &sm.Tt[0][0][0], lane);
    __syncwarp();
    if (!kAhead) streams(0);
    Frag<3> ta, tz;
    load_left_t(ta, smem_u32(&sm.Tt[0][0][0]) + atC, kPartC);
    {
        Frag<3> fz;
        float x[2][4];
        from_c(fz, z[0], z[1]);
        product<BY_COLS>(x, ta, by_cols(fz));           // T' triu(K Q^T)
        from_c(tz, x[0], x[1]);
    }
#pragma unroll kUnroll
    for (int k = 0; k < KS; k++) {
        Frag<NP> r;
        Frag<3> f;
        float x[2][4];
        load_cols(r, aK + 32 * k, kPart);
        put_frag(ws + Sp::K + k * NP * 32, r, lane);
        product<BY_COLS>(x, ta, r);
        from_c(f, x[0], x[1]);
        put_frag(ws + Sp::X + k * 96, f, lane);
        load_cols(r, aQ + 32 * k, kPart);
        put_frag(ws + Sp::Q + k * NP * 32, r, lane);
    }
#pragma unroll 1
    for (int j = 0; j < MS; j++) {
        float x[2][4];
#pragma unroll
        for (int i = 0; i < 8; i++) sv[i >> 2][i & 3] -= so[i >> 2][i & 3];
        scale_steps(sv, bt);
        Frag<NP> fy;
        Frag<3> fu;
        from_c(fy, sy[0], sy[1]);
        from_c(fu, sv[0], sv[1]);
        if (j + 1 < MS) streams(j + 1);
        product<BY_ROWS>(x, fy, tz);                    // Tv^T = gY^T (T' Z)^T
        put_block(ws + Sp::R + j * 64, x, lane);
#pragma unroll kUnroll
        for (int k = 0; k < KS; k++) {
            Frag<NP> r;
            load_cols(r, aQ + 32 * k, kPart);
            product<BY_COLS>(x, fy, r);                 // (Q^T gY)^T
            put_block(ws + Sp::G + (j * KS + k) * 64, x, lane);
            load_left_t(r, aK + 32 * k, kPart);
            product<BY_ROWS>(x, r, fu);                 // K^T U
            put_block(ws + Sp::S + (k * MS + j) * 64, x, lane);
        }
    }
}

// -------------------------------------------------------------------------------------------------------- chain
// One CTA per sequence and 16 state columns.  Warp 0 runs the chain of G, its operands copied DEPTH - 1 chunks ahead
// (every lane copies the pieces it will read itself, so no barrier is needed); warp 1 the running difference of S.
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}
template <int E, int M, int DEPTH, typename T>
struct ChainRing {                      // pieces of 16 bytes per lane
    static constexpr int KS = E / 16, NP = stream_parts<T>();
    static constexpr int X = 0, K = X + KS * 3, R = K + KS * NP, G = R + 2, B = G + KS * 2, kPieces = B + 1;
    static constexpr size_t kBytes = (size_t)DEPTH * kPieces * 512;
};
template <int E, int M, int DEPTH, typename T>
__global__ void __launch_bounds__(64) delta_bwd_chain_kernel(const __grid_constant__ BwdPhase a) {
    constexpr int KS = E / 16, MS = M / 16, NP = stream_parts<T>();
    using Sp = BwdSpace<E, M, NP>;
    using Rg = ChainRing<E, M, DEPTH, T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const DeltaBwdParams& p = a.p;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int seq = blockIdx.x / MS, j = blockIdx.x - seq * MS;
    griddep_wait();
    griddep_launch_dependents();
    uint4* const ws = a.ws + (long long)seq * a.nc * Sp::kSize;
    if (threadIdx.x >= 32) {
        const int n = (a.s0 + seq) / p.H, h = a.s0 + seq - n * p.H;
        float* W = p.W + n * p.wN + h * p.wH;
        constexpr int AHEAD = 4;
        bool good = true;
#pragma unroll 1
        for (int k = 0; k < KS; k++) {
            uint4* at = ws + Sp::S + (k * MS + j) * 64;
            float s1[1][2][4], (&s)[2][4] = s1[0], d[AHEAD][2][4];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int e = 16 * k + g + 8 * ((i >> 1) & 1), m = 16 * j + 8 * (i >> 2) + 2 * t + (i & 1);
                s[i >> 2][i & 3] = e < p.E && m < p.M ? W[(long long)e * p.wE + m] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < AHEAD; q++)
                if (q < a.nc) get_block(d[q], at + (long long)(a.nc - 1 - q) * Sp::kSize, lane);
            for (int c = a.nc - 1; c >= 0; c -= AHEAD) {
#pragma unroll
                for (int q = 0; q < AHEAD; q++) {
                    if (c - q < 0) break;
#pragma unroll
                    for (int i = 0; i < 8; i++) s[i >> 2][i & 3] -= d[q][i >> 2][i & 3];
                    put_block(at + (long long)(c - q) * Sp::kSize, s, lane);
                    if (c - q >= AHEAD) get_block(d[q], at + (long long)(c - q - AHEAD) * Sp::kSize, lane);
                }
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int e = 16 * k + g + 8 * ((i >> 1) & 1), m = 16 * j + 8 * (i >> 2) + 2 * t + (i & 1);
                if (e < p.E && m < p.M) W[(long long)e * p.wE + m] = s[i >> 2][i & 3];
            }
            good &= finite(s1);
        }
        if (!good) a.again[seq] = 1;
        return;
    }
    uint4* const carry = a.carry + ((long long)seq * MS + j) * KS * 64;
    uint4* const ring = reinterpret_cast<uint4*>(smem_raw);
    auto issue = [&](int c) {
        if (c >= 0) {
            const uint4* s = ws + (long long)c * Sp::kSize;
            uint4* d = ring + (c % DEPTH) * Rg::kPieces * 32 + lane;
#pragma unroll
            for (int i = 0; i < KS * 3; i++) cp_async16(d + (Rg::X + i) * 32, s + Sp::X + i * 32 + lane);
#pragma unroll
            for (int i = 0; i < KS * NP; i++) cp_async16(d + (Rg::K + i) * 32, s + Sp::K + i * 32 + lane);
#pragma unroll
            for (int i = 0; i < 2; i++) cp_async16(d + (Rg::R + i) * 32, s + Sp::R + (2 * j + i) * 32 + lane);
#pragma unroll
            for (int i = 0; i < KS * 2; i++) cp_async16(d + (Rg::G + i) * 32, s + Sp::G + (j * KS * 2 + i) * 32 + lane);
            const float* b = reinterpret_cast<const float*>(s + Sp::B) + 2 * t;
            float* db = reinterpret_cast<float*>(d + Rg::B * 32);
            cp_async8(db, b);
            cp_async8(db + 2, b + 8);
        }
        cp_async_commit();
    };
    float G[KS][2][4];
#pragma unroll
    for (int k = 0; k < KS; k++) {
        if (a.first) zero(G[k]);
        else get_block(G[k], carry + k * 64, lane);
    }
#pragma unroll
    for (int q = 0; q < DEPTH - 1; q++) issue(a.nc - 1 - q);
    for (int c = a.nc - 1; c >= 0; c--) {
        issue(c - (DEPTH - 1));
        cp_async_wait<DEPTH - 1>();
        const uint4* r0 = ring + (c % DEPTH) * Rg::kPieces * 32;
        uint4* out = ws + (long long)c * Sp::kSize;
        float r[2][4];
        get_block(r, r0 + Rg::R * 32, lane);
#pragma unroll
        for (int k = 0; k < KS; k++) {
            Frag<3> s, x;
            from_c(s, G[k][0], G[k][1]);
            get_frag(x, r0 + (Rg::X + 3 * k) * 32, lane);
            add_product<BY_ROWS>(r, s, x);
        }
        const float4 b = *reinterpret_cast<const float4*>(r0 + Rg::B * 32 + lane);
        const float bt[2][2] = {{-b.x, -b.y}, {-b.z, -b.w}};
#pragma unroll
        for (int k = 0; k < KS; k++) put_block(out + Sp::G + (j * KS + k) * 64, G[k], lane);
        put_block(out + Sp::R + j * 64, r, lane);
        scale_steps(r, bt);
        Frag<3> s;
        from_c(s, r[0], r[1]);
#pragma unroll
        for (int k = 0; k < KS; k++) {
            Frag<NP> x;
            float d[2][4];
            get_block(d, r0 + (Rg::G + 2 * k) * 32, lane);
            add_to(G[k], d);
            get_frag(x, r0 + (Rg::K + NP * k) * 32, lane);
            add_product<BY_COLS>(G[k], s, x);
        }
    }
#pragma unroll
    for (int k = 0; k < KS; k++) put_block(carry + k * 64, G[k], lane);
    if (!finite(G)) a.again[seq] = 1;
}

// ------------------------------------------------------------------------------------------------------- finish
// One warp per chunk and group of KG row blocks of the state.
template <int E, int M, int KG, int WARPS, typename T>
__global__ void __launch_bounds__(WARPS * 32, M == 16 ? (E > 64 ? 5 : 4) : 0) delta_bwd_finish_kernel(const __grid_constant__ BwdPhase a) {
    constexpr int KS = E / 16, MS = M / 16, NP = stream_parts<T>(), GROUPS = (KS + KG - 1) / KG;
    using Sp = BwdSpace<E, M, NP>;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const DeltaBwdParams& p = a.p;
    const long long task = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
    const long long unit = GROUPS == 1 ? task : task / GROUPS;
    const int k0 = GROUPS == 1 ? 0 : (int)(task - unit * GROUPS) * KG;
    const int seq = (int)(unit / a.nc), c = a.c0 + (int)(unit - (long long)seq * a.nc);
    griddep_wait();
    griddep_launch_dependents();
    if (seq >= a.ns) return;
    const int n = (a.s0 + seq) / p.H, h = a.s0 + seq - n * p.H, t0 = c * C, nt = min(C, p.L - t0);
    const uint4* const ws = a.ws + unit * Sp::kSize;
    float bt[2][2];
    load_beta(bt, stream_at<T>(p.beta, n, h) + t0 * p.beta.sL, p.beta.sL, nt, t);
    const T* vp = stream_at<T>(p.v, n, h) + (t0 + 2 * t) * p.v.sL + g;
    const T* yp = stream_at<T>(p.gy, n, h) + (t0 + 2 * t) * p.gy.sL + g;
    const float* op = stream_at<float>(p.v_old, n, h) + (t0 + 2 * t) * p.v_old.sL + g;
    T* gvp = stream_at<T>(p.gv, n, h) + (t0 + 2 * t) * p.gv.sL + g;
    float dq[KG][2][4], dk[KG][2][4], hh[2][4] = {}, pp[2][4] = {}, db[2][2] = {};
#pragma unroll
    for (int k = 0; k < KG; k++) {
        zero(dq[k]);
        zero(dk[k]);
    }
    float sr[2][4], sy[2][4], sv[2][4], so[2][4], xs[2][4], xg[2][4];
    auto streams = [&](int j) {                         // r, V, v_old, gY of the next slice, requested early
        const int width = p.M - 16 * j;
        get_block(sr, ws + Sp::R + j * 64, lane);
        load_block_t<T>(sv, vp + 16 * j, p.v.sL, nt, width, g, t);
        load_block_t<float>(so, op + 16 * j, p.v_old.sL, nt, width, g, t);
        load_block_t<T>(sy, yp + 16 * j, p.gy.sL, nt, width, g, t);
    };
    auto states = [&](int j, int k) {                   // and the next blocks of S0 and G
        get_block(xs, ws + Sp::S + ((k0 + k) * MS + j) * 64, lane);
        get_block(xg, ws + Sp::G + (j * KS + k0 + k) * 64, lane);
    };
    streams(0);
    states(0, 0);
    if (__builtin_expect(a.again[seq] != 0, 0)) {
        if (c == 0 && k0 == 0) {                        // the last segment: nobody else writes to this chunk's part of the workspace
            float* const own = reinterpret_cast<float*>(a.ws + unit * Sp::kSize);
            stepwise_backward<T>(p, n, h, own + 4 * Sp::G, own + 4 * Sp::S, own + 4 * Sp::R);
        }
        return;
    }
    const int kn = KS % KG ? min(KG, KS - k0) : KG;
#pragma unroll 1
    for (int j = 0; j < MS; j++) {
        float r[2][4], w[2][4], y[2][4];
        const int width = p.M - 16 * j;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            r[i >> 2][i & 3] = sr[i >> 2][i & 3];
            y[i >> 2][i & 3] = sy[i >> 2][i & 3];
            w[i >> 2][i & 3] = sv[i >> 2][i & 3] - so[i >> 2][i & 3];
        }
        if (j + 1 < MS) streams(j + 1);
        if (k0 == 0) {
#pragma unroll
            for (int i = 0; i < 8; i++) db[i >> 2][i & 1] += r[i >> 2][i & 3] * w[i >> 2][i & 3];
        }
        scale_steps(w, bt);
        scale_steps(r, bt);
        if (k0 == 0) store_block_t<T>(r, gvp + 16 * j, p.gv.sL, nt, width, g, t);
#pragma unroll
        for (int i = 0; i < 8; i++) r[i >> 2][i & 3] = -r[i >> 2][i & 3];
        Frag<3> u, b;
        Frag<NP> gy;
        {
            Frag<3> f;
            from_c(f, w[0], w[1]);
            u = left_of_transpose(f);                   // rows of U: left operand, and right operand by rows
            from_c(f, r[0], r[1]);
            b = left_of_transpose(f);                   // rows of -b
            Frag<NP> fy;
            from_c(fy, y[0], y[1]);
            gy = left_of_transpose(fy);
        }
        add_product<BY_ROWS>(hh, gy, u);                // gY U^T
        add_product<BY_ROWS>(pp, u, b);                 // -U b^T
#pragma unroll
        for (int k = 0; k < KG; k++) {
            if (KS % KG && k >= kn) break;
            Frag<3> f, fg;
            from_c(f, xs[0], xs[1]);
            from_c(fg, xg[0], xg[1]);
            if (k + 1 < kn) states(j, k + 1);
            else if (j + 1 < MS) states(j + 1, 0);
            add_product<BY_ROWS>(dq[k], gy, f);         // gY S0^T
            add_product<BY_ROWS>(dk[k], b, f);          // -b S0^T
            add_product<BY_COLS>(dk[k], u, by_cols(fg)); // U G^T
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int row = g + 8 * ((i >> 1) & 1), col = 8 * (i >> 2) + 2 * t + (i & 1);
        if (col > row) hh[i >> 2][i & 3] = 0.f;
        else pp[i >> 2][i & 3] = 0.f;
    }
    Frag<3> fh, fht, fr;
    from_c(fh, hh[0], hh[1]);
    fht = left_of_transpose(fh);
    from_c(fr, pp[0], pp[1]);
#pragma unroll
    for (int i = 0; i < 3; i++) {                       // -R: the mirror image below the diagonal
        fr.r[i][0] |= transpose8(fr.r[i][0]);
        fr.r[i][1] = transpose8(fr.r[i][2]);
        fr.r[i][3] |= transpose8(fr.r[i][3]);
    }
    T* gqp = stream_at<T>(p.gq, n, h) + (t0 + g) * p.gq.sL + 2 * t;
    T* gkp = stream_at<T>(p.gk, n, h) + (t0 + g) * p.gk.sL + 2 * t;
    auto even = [&](const T* q, long long sL) { return (reinterpret_cast<uintptr_t>(q) & (2 * sizeof(T) - 1)) == 0 && (sL & 1) == 0; };
    const bool qpair = even(gqp, p.gq.sL), kpair = even(gkp, p.gk.sL);
#pragma unroll
    for (int k = 0; k < KG; k++) {
        if (KS % KG && k >= kn) break;
        Frag<NP> x, y;
        get_frag(x, ws + Sp::K + (k0 + k) * NP * 32, lane);
        get_frag(y, ws + Sp::Q + (k0 + k) * NP * 32, lane);
        add_product<BY_COLS>(dq[k], fh, x);             // H K
        add_product<BY_COLS>(dk[k], fr, x);             // -R K
        add_product<BY_COLS>(dk[k], fht, y);            // H^T Q
        store_block<T>(dq[k], gqp + 16 * (k0 + k), p.gq.sL, nt, p.E - 16 * (k0 + k), qpair, g, t);
        store_block<T>(dk[k], gkp + 16 * (k0 + k), p.gk.sL, nt, p.E - 16 * (k0 + k), kpair, g, t);
    }
    if (k0 == 0) {
        T* gbp = stream_at<T>(p.gb, n, h) + t0 * p.gb.sL;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float d = db[i >> 1][i & 1];
#pragma unroll
            for (int o = 4; o <= 16; o <<= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            const int s = 8 * (i >> 1) + 2 * t + (i & 1);
            if (g == 0 && s < nt) gbp[s * p.gb.sL] = from_f32<T>(d);
        }
    }
}

}  // namespace wy
}  // namespace fwp
