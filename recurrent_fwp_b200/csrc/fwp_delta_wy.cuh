// Delta rule and sum rule in chunks of sixteen steps (WY form), fp32 arithmetic on the tensor pipe (sm_100a).
//
// Within a chunk that starts from the state S (E x M),
//   w_i = v_i - v_old_i = v_i - S^T k_i - sum_{j<i} beta_j (k_i . k_j) w_j
// is a unit lower triangular system in w, the same for every column of the state.  With A_ij = beta_j k_i . k_j (j < i),
// T = (I + A)^-1 by forward substitution (sixteen steps in fp32, exact algebra, no division) and X = T K,
//   w = T V - X S,   u = diag(beta) w,   S += K^T u,   y = Q S + tril(Q K^T) u,   v_old = v - w.
// The sum rule is the same with u = V.  All products are 16 steps deep or wide and run as three-part bf16 products with
// fp32 accuracy (fwp_split3.cuh).
//
// Roles.  One CTA per sequence:
//   * chain warps own 16 state columns each and do what depends on the chunk before: X S, w, u and K^T u.  The state
//     is held transposed (rows m, columns e) as fp32 C fragments, so that it is the left operand of X S and its update
//     lands in the same registers: nothing of the chain crosses lanes;
//   * helper warps own whole chunks, round robin.  Before the chain: K, Q and V come from global memory in fragment
//     order (whole sectors at any alignment), are split, and leave as operand tiles in shared memory together with X,
//     T V and tril(Q K^T).  After it (OUT): the outputs, from the parts of S and u the chain left behind.
// The two sides meet at two mbarriers per buffer.  With many sequences of a large state the copies of S would fill
// shared memory, so there (OUT = false) the chain warps form the outputs themselves.
//
// Values that are not finite.  A chunk's products run over all sixteen steps: above the diagonal a zero meets the value of
// a later step, and zero times NaN or Inf is NaN, so one bad step would reach up to fifteen outputs before it (and a split
// Inf is Inf, NaN, NaN).  Whatever goes wrong this way -- in an input, or by overflow -- stays in the state to the end of
// the sequence (S only ever gets K^T u added); a query alone shows in its row of tril(Q K^T).  So a CTA that ends with a
// state, or meets a product of queries and keys, that is not finite does its sequence again, step by step from the state
// it started from (stepwise_forward): what a caller sees is the recurrence itself, for any value.  The end state is
// therefore stored behind a barrier of the CTA.
#pragma once
#include "fwp_wy_common.cuh"

namespace fwp {
namespace wy {

// The sum rule's three gradients are sum-rule forwards of other streams, two of them backwards in time (negative strides):
//   dq_t = sum_{i<=t} (gy_t . v_i) k_i,   dv_t = sum_{i>=t} (k_t . q_i) gy_i,   dk_t = sum_{i>=t} (v_t . gy_i) q_i
// from states that start at zero.  One launch runs the three side by side.
struct SumBwdForwards {
    DeltaFwdParams p[3];
};

static __device__ int g_wy_fault;       // a bounded wait ran out (read by fwp_delta_device_fault)

__device__ __forceinline__ void arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// one arrival per warp, after everything its lanes have done
__device__ __forceinline__ void warp_arrive(unsigned long long* bar, int lane) {
    __syncwarp();
    if (lane == 0) arrive(bar);
}
__device__ __forceinline__ void wait(unsigned long long* bar, unsigned parity) {
    if (!mbar_wait_bounded(bar, parity)) atomicExch(&g_wy_fault, 1);
}

// One stream of one sequence as a warp copies it, sixteen rows at a time, into an fp32 tile of pitch P floats.  fp32 rows
// go by cp.async (16-byte pieces where the rows allow it, else 4-byte: the layers' value slices start at odd offsets);
// bf16 rows are widened on the way.
template <int W, int P, typename T>
struct Stream {
    const T* base;
    const T* at;            // this lane's first element of row 0 of a sweep
    long long sL;
    int width, off;         // off: that element's place in the tile
    bool vec, full;         // 16-byte pieces; whole rows of W elements
    static constexpr bool kNarrow = W > 16;     // 16-byte pieces of narrower rows too (in tiles of 16 the test costs more)
    static constexpr int RS1 = W < 32 ? 32 / W : 1;                                 // 4-byte copies of whole rows: rows per sweep
    static constexpr int PPR = W / 4, RS = PPR <= 32 ? 32 / PPR : 1;                // 16-byte pieces per row, rows per sweep
    static constexpr int CS1 = (W + 31) / 32;                                       // 4-byte copies: column groups
    static constexpr bool kVec = PPR <= 32 && 32 % PPR == 0;
    __device__ __forceinline__ void init(const Row4& r, int n, int h, int w, int lane) {
        base = reinterpret_cast<const T*>(r.p) + n * r.sN + h * r.sH;
        sL = r.sL;
        width = w;
        full = kVec && w == W;
        vec = sizeof(T) == 4 && (reinterpret_cast<uintptr_t>(base) & 15) == 0 && sL % 4 == 0 && (kNarrow ? w % 4 == 0 : full);
        at = base + (vec ? (full ? (lane / PPR) * sL + (lane % PPR) * 4 : 4 * lane) : W < 32 ? (lane / W) * sL + lane % W : lane);
        off = vec ? (full ? (lane / PPR) * P + (lane % PPR) * 4 : 4 * lane) : W < 32 ? (lane / W) * P + lane % W : lane;
    }
    // rows past the end are zeroed
    __device__ __forceinline__ void copy(float* tile, int t0, int nt, int lane) const {
        if (nt < C)
            for (int i = lane; i < (C - nt) * P; i += 32) tile[nt * P + i] = 0.f;
        if constexpr (sizeof(T) == 4) {
            const T* g = at + t0 * sL;
            tile += off;
            if (vec && (full || !kNarrow) && nt == C) {
#pragma unroll
                for (int r = 0; r < C; r += RS, g += RS * sL) cp_async16(tile + r * P, g);
            } else if (W < 32 && full && nt == C) {
#pragma unroll
                for (int r = 0; r < C; r += RS1, g += RS1 * sL) cp_async4(tile + r * P, g);
            } else if (kNarrow && vec && !full) {       // a row at a time
                if (4 * lane < width)
#pragma unroll 4
                    for (int r = 0; r < nt; r++, g += sL) cp_async16(tile + r * P, g);
            } else {
                g = base + lane + t0 * sL;
                tile += lane - off;
#pragma unroll
                for (int c = 0; c < CS1; c++)
                    if (lane + 32 * c < width) {
                        const T* gc = g + 32 * c;
#pragma unroll 4
                        for (int r = 0; r < nt; r++, gc += sL) cp_async4(tile + r * P + 32 * c, gc);
                    }
            }
        } else {
            const T* g = base + t0 * sL;
#pragma unroll 4
            for (int r = 0; r < nt; r++, g += sL)
                for (int c = lane; c < width; c += 32) tile[r * P + c] = to_f32(g[c]);
        }
    }
};
// Columns [0, W) of sixteen rows of a tile back to a stream, one warp.
template <int W, int P, typename T>
__device__ __forceinline__ void flush(const float* tile, T* base, long long sL, int nt, int width, bool vec, int lane) {
    constexpr int per16 = 16 / (int)sizeof(T), PPR = W / per16 > 0 ? W / per16 : 1, RS = PPR <= 32 ? 32 / PPR : 1;
    if (vec && nt == C && width >= W && 32 % PPR == 0) {
        const float* s = tile + (lane / PPR) * P + (lane % PPR) * per16;
        T* g = base + (lane / PPR) * sL + (lane % PPR) * per16;
#pragma unroll
        for (int r = 0; r < C; r += RS, g += RS * sL) flush_piece<W, 32, T>(g, s + r * P);
    } else {
        for (int r = 0; r < nt; r++)
            for (int c = lane; c < (width < W ? width : W); c += 32) base[r * sL + c] = from_f32<T>(tile[r * P + c]);
    }
}
template <typename T>
__device__ __forceinline__ bool rows_vec(const T* base, long long sL) {
    return (reinterpret_cast<uintptr_t>(base) & 15) == 0 && sL % (16 / (int)sizeof(T)) == 0;
}

// the CTA's flag: something that is not finite turned up
__device__ __forceinline__ int& redo() {
    __shared__ int flag;
    return flag;
}
// raises it when one of a block's values is not finite: their sum times zero is NaN then
template <int K>
__device__ __forceinline__ void note(const float (&x)[K][4]) {
    f2 acc = 0ull;
#pragma unroll
    for (int i = 0; i < 2 * K; i++) acc = ffma2(f2_pack(x[i >> 1][2 * (i & 1)], x[i >> 1][2 * (i & 1) + 1]), 0ull, acc);
    if (!(f2_hsum(acc) == 0.f)) redo() = 1;
}

// The recurrence of one sequence as it stands, a thread per state column; W in place, or a zeroed E x M array of the
// caller's where the parameters name none.  It stands once at the end of a kernel, inlined: a call would cost every launch
// 0.5 to 0.9 us (the kernel then has a stack).
template <typename T, bool SUM>
__device__ __forceinline__ void stepwise_forward(const DeltaFwdParams& p, float* own) {
    const int n = blockIdx.x / p.H, h = blockIdx.x - n * p.H;
    const T* const qp = reinterpret_cast<const T*>(p.q.p) + n * p.q.sN + h * p.q.sH;
    const T* const kp = reinterpret_cast<const T*>(p.k.p) + n * p.k.sN + h * p.k.sH;
    const T* const vp = reinterpret_cast<const T*>(p.v.p) + n * p.v.sN + h * p.v.sH;
    const T* const bp = SUM ? nullptr : reinterpret_cast<const T*>(p.beta.p) + n * p.beta.sN + h * p.beta.sH;
    T* const yp = reinterpret_cast<T*>(p.out.p) + n * p.out.sN + h * p.out.sH;
    float* const vop = SUM || !p.v_old.p ? nullptr : reinterpret_cast<float*>(p.v_old.p) + n * p.v_old.sN + h * p.v_old.sH;
    float* const vip = SUM || !p.v_ins.p ? nullptr : reinterpret_cast<float*>(p.v_ins.p) + n * p.v_ins.sN + h * p.v_ins.sH;
    const long long sE = p.W ? p.wE : p.M;
    for (int m = threadIdx.x; m < p.M; m += blockDim.x) {
        float* const S = (p.W ? p.W + n * p.wN + h * p.wH : own) + m;
        if (!p.W)
            for (int e = 0; e < p.E; e++) S[e * sE] = 0.f;
        for (long long t = 0; t < p.L; t++) {
            const T *k = kp + t * p.k.sL, *q = qp + t * p.q.sL;
            float u = to_f32(vp[t * p.v.sL + m]), y = 0.f;
            if constexpr (!SUM) {
                float vo = 0.f;
#pragma unroll 1
                for (int e = 0; e < p.E; e++) vo = fmaf(S[e * sE], to_f32(k[e]), vo);
                u = to_f32(bp[t * p.beta.sL]) * (u - vo);
                if (vop) vop[t * p.v_old.sL + m] = vo;
                if (vip) vip[t * p.v_ins.sL + m] = u;
            }
#pragma unroll 1
            for (int e = 0; e < p.E; e++) {
                const float s = fmaf(to_f32(k[e]), u, S[e * sE]);
                S[e * sE] = s;
                y = fmaf(s, to_f32(q[e]), y);
            }
            yp[t * p.out.sL + m] = from_f32<T>(y);
        }
    }
}

// 16 x 16 block of a tile as C fragments: `at` is this lane's (g, 2t)
template <int P>
__device__ __forceinline__ void tile_block(float (&x)[2][4], const float* at) {
#pragma unroll
    for (int n = 0; n < 2; n++)
#pragma unroll
        for (int hi = 0; hi < 2; hi++) {
            const float2 v = *reinterpret_cast<const float2*>(at + 8 * hi * P + 8 * n);
            x[n][2 * hi] = v.x;
            x[n][2 * hi + 1] = v.y;
        }
}
// element i of the transposed block: `at` is this lane's (row 2t, column g)
template <int P>
__host__ __device__ constexpr int block_t_at(int n, int i) { return (8 * n + (i & 1)) * P + 8 * (i >> 1); }
template <int P>
__device__ __forceinline__ void tile_block_t(float (&x)[2][4], const float* at) {
#pragma unroll
    for (int n = 0; n < 2; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) x[n][i] = at[block_t_at<P>(n, i)];
}
template <int P>
__device__ __forceinline__ void put_block_t(const float (&x)[2][4], float* at) {
#pragma unroll
    for (int n = 0; n < 2; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) at[block_t_at<P>(n, i)] = x[n][i];
}

// ---------------------------------------------------------------------------------- forward, few sequences
template <int E, int M, int NP>
struct FewBuf {
    static constexpr int P = E + 8, PR = E + 8, PV = M + 4, NCW = M / 16, KS = E / 16;
    float kraw[C][PR], qraw[C][PR], v[2][C][PV], beta[2][C];      // the chunk's rows; v becomes v_old
    __nv_bfloat16 K[NP][C][P], Q[NP][C][P], X[3][C][P], Aqk[3][C][PC];
    union {
        struct {
            __nv_bfloat16 Tt[3][C][PC];
            float A[C][C + 4];
        } inv;                                                    // until X and T V are there
        float y[C][PV];
    };
    float4 tv[NCW][2][32];                                        // T V, then w, in the chain warp's fragment order
    uint4 s[NCW][KS][3][32];                                      // parts of the chunk's start state
};

template <int E, int M, int NB, typename T, bool SUM>
__device__ __forceinline__ void fwd_few(const DeltaFwdParams& p) {
    constexpr int NCW = M / 16, KS = E / 16, NP = stream_parts<T>();
    using Buf = FewBuf<E, M, NP>;
    constexpr int P = Buf::P, PR = Buf::PR, PV = Buf::PV, kPart = C * P * 2, kPartC = C * PC * 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Buf* bufs = reinterpret_cast<Buf*>(smem_raw);
    __shared__ unsigned long long filled[NB], done[NB];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n = blockIdx.x / p.H, h = blockIdx.x - n * p.H;
    const int nchunks = (p.L + C - 1) / C;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; i++) {
            mbar_init(&filled[i], 1);
            mbar_init(&done[i], NCW);
        }
        redo() = 0;
        mbar_fence_init();
    }
    if (warp >= NCW && (p.E < E || p.M < M)) {      // columns that no copy writes
        float* raw = &bufs[warp - NCW].kraw[0][0];
        for (int i = lane; i < 2 * C * PR + 2 * C * PV; i += 32) raw[i] = 0.f;
    }
    __syncthreads();
    griddep_wait();
    griddep_launch_dependents();
    T* const yp = reinterpret_cast<T*>(p.out.p) + n * p.out.sN + h * p.out.sH;
    float* const vop = SUM || !p.v_old.p ? nullptr : reinterpret_cast<float*>(p.v_old.p) + n * p.v_old.sN + h * p.v_old.sH;
    float* const vip = SUM || !p.v_ins.p ? nullptr : reinterpret_cast<float*>(p.v_ins.p) + n * p.v_ins.sN + h * p.v_ins.sH;
    const bool yvec = rows_vec(yp, p.out.sL), vovec = vop && rows_vec(vop, p.v_old.sL);
    // v_old = v - w in place of v, for one 16-column slice
    auto side = [&](Buf& buf, int st, const float (&w)[2][4], const float (&u)[2][4], int m0, int t0, int nt) {
        float* at = &buf.v[st][2 * t][m0 + g];
#pragma unroll
        for (int i = 0; i < 8; i++) at[block_t_at<PV>(i >> 2, i & 3)] -= w[i >> 2][i & 3];
        if (vip) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int s = 8 * (i >> 2) + 2 * t + (i & 1), m = m0 + g + 8 * ((i >> 1) & 1);
                if (s < nt && m < p.M) vip[(t0 + s) * p.v_ins.sL + m] = u[i >> 2][i & 3];
            }
        }
    };
    auto scale = [&](float (&u)[2][4], const float (&w)[2][4], const float* beta) {
#pragma unroll
        for (int nn = 0; nn < 2; nn++) {
            const float2 b2 = *reinterpret_cast<const float2*>(beta + 8 * nn + 2 * t);
#pragma unroll
            for (int i = 0; i < 4; i++) u[nn][i] = w[nn][i] * ((i & 1) ? b2.y : b2.x);
        }
    };

    if (warp < NCW) {
        const int m0 = warp * 16, width = p.M - m0;
        float* W = p.W ? p.W + n * p.wN + h * p.wH + m0 : nullptr;    // none: a state that starts at zero and is not asked for
        float S[2 * KS][4];             // S[j]: state rows e = 8j + 2t, 8j + 2t + 1 of columns m = g, g + 8
#pragma unroll
        for (int j = 0; j < 2 * KS; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int e = 8 * j + 2 * t + (i & 1), m = g + 8 * (i >> 1);
                S[j][i] = W && e < p.E && m < width ? W[(long long)e * p.wE + m] : 0.f;
            }
        int b = 0, st = 0;
        unsigned phase = 0;
        for (int c = 0; c < nchunks; c++) {
            Buf& buf = bufs[b];
            const unsigned at = 2 * lane_at(lane, P);
            const unsigned aK = smem_u32(&buf.K[0][0][0]) + at, aX = smem_u32(&buf.X[0][0][0]) + at;
            wait(&filled[b], phase);
            float w[2][4], xs[2][4];
            *reinterpret_cast<float4*>(w[0]) = buf.tv[warp][0][lane];
            *reinterpret_cast<float4*>(w[1]) = buf.tv[warp][1][lane];
#pragma unroll
            for (int i = 0; i < 8; i++) xs[i >> 2][i & 3] = 0.f;
#pragma unroll
            for (int k = 0; k < KS; k++) {
                Frag<3> s;
                from_c(s, S[2 * k], S[2 * k + 1]);
                if constexpr (!SUM) {
                    Frag<3> r;
                    load_rows(r, aX + 32 * k, kPart);
                    sum_product<BY_ROWS>(k, xs, s, r);
                }
#pragma unroll
                for (int i = 0; i < 3; i++) buf.s[warp][k][i][lane] = make_uint4(s.r[i][0], s.r[i][1], s.r[i][2], s.r[i][3]);
            }
            Frag<3> us;
            if constexpr (SUM) {
                from_c(us, w[0], w[1]);
            } else {
                float u[2][4];
#pragma unroll
                for (int i = 0; i < 8; i++) w[i >> 2][i & 3] -= xs[i >> 2][i & 3];
                scale(u, w, buf.beta[st]);
                from_c(us, u[0], u[1]);
            }
            buf.tv[warp][0][lane] = make_float4(w[0][0], w[0][1], w[0][2], w[0][3]);
            buf.tv[warp][1][lane] = make_float4(w[1][0], w[1][1], w[1][2], w[1][3]);
#pragma unroll
            for (int k = 0; k < KS; k++) {          // S += K^T u
                Frag<NP> r;
                float d[2][4] = {};
                load_cols(r, aK + 32 * k, kPart);
                product<BY_COLS>(d, us, r);
#pragma unroll
                for (int i = 0; i < 8; i++) S[2 * k + (i >> 2)][i & 3] += d[i >> 2][i & 3];
            }
            warp_arrive(&done[b], lane);
            if (++b == NB) { b = 0; phase ^= 1; st ^= 1; }
        }
        note(S);
        slot_barrier(0, (NCW + NB) * 32);           // the other warps have written what they have to write
        if (redo()) return;
#pragma unroll
        for (int j = 0; j < 2 * KS; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int e = 8 * j + 2 * t + (i & 1), m = g + 8 * (i >> 1);
                if (W && e < p.E && m < width) W[(long long)e * p.wE + m] = S[j][i];
            }
        return;
    }

    // ---- helper: chunks b, b + NB, ...  Its loops over blocks stay rolled: with as many helpers as chunks in flight, each in a place of
    // its own, instruction fetch was the largest stall (E, M = 96, 32, 128 x 256: 72 us unrolled, 50 rolled)
    constexpr int kUnroll = KS == 1 ? 16 : 1;   // at d = 16 they are single blocks, and the chain waits for every instruction
    const int b = warp - NCW;
    Buf& buf = bufs[b];
    Stream<E, PR, T> sk, sq;
    Stream<M, PV, T> sv;
    sk.init(p.k, n, h, p.E, lane);
    sq.init(p.q, n, h, p.E, lane);
    sv.init(p.v, n, h, p.M, lane);
    const T* betap = SUM ? nullptr : reinterpret_cast<const T*>(p.beta.p) + n * p.beta.sN + h * p.beta.sH;
    const unsigned at = 2 * lane_at(lane, P), atC = 2 * lane_at(lane, PC);
    const unsigned aK = smem_u32(&buf.K[0][0][0]) + at, aQ = smem_u32(&buf.Q[0][0][0]) + at, aX = smem_u32(&buf.X[0][0][0]) + at;
    const unsigned aT = smem_u32(&buf.inv.Tt[0][0][0]) + atC, aA = smem_u32(&buf.Aqk[0][0][0]) + atC;
    auto issue = [&](int c, int st) {
        const int t0 = c * C, nt = min(C, p.L - t0);
        sk.copy(&buf.kraw[0][0], t0, nt, lane);
        sq.copy(&buf.qraw[0][0], t0, nt, lane);
        sv.copy(&buf.v[st][0][0], t0, nt, lane);
        if (!SUM && lane < C) {
            if (lane >= nt) buf.beta[st][lane] = 0.f;
            else if constexpr (sizeof(T) == 4) cp_async4(&buf.beta[st][lane], betap + (t0 + lane) * p.beta.sL);
            else buf.beta[st][lane] = to_f32(betap[(t0 + lane) * p.beta.sL]);
        }
        cp_async_commit();
    };
    if (b < nchunks) issue(b, 0);
    unsigned phase = 0;
    int st = 0;
    for (int c = b; c < nchunks; c += NB, phase ^= 1, st ^= 1) {
        cp_async_wait<0>();
        __syncwarp();
        float kk[2][4] = {}, qk[2][4] = {};
#pragma unroll kUnroll
        for (int k = 0; k < KS; k++) {
            Frag<NP> fk, fq;
            float x[2][4];
            tile_block<PR>(x, &buf.kraw[g][2 * t + 16 * k]);
            from_c(fk, x[0], x[1]);
            store(aK + 32 * k, kPart, fk);
            tile_block<PR>(x, &buf.qraw[g][2 * t + 16 * k]);
            from_c(fq, x[0], x[1]);
            store(aQ + 32 * k, kPart, fq);
            if (!SUM) sum_product<BY_ROWS>(KS == 1 ? 0 : 1, kk, fk, fk);
            sum_product<BY_ROWS>(KS == 1 ? 0 : 1, qk, fq, fk);
        }
#pragma unroll
        for (int nn = 0; nn < 2; nn++) {
            const float2 b2 = SUM ? make_float2(0.f, 0.f) : *reinterpret_cast<const float2*>(&buf.beta[st][8 * nn + 2 * t]);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int row = g + 8 * (i >> 1), col = 8 * nn + 2 * t + (i & 1);
                if (col > row) qk[nn][i] = 0.f;
                if (!SUM) kk[nn][i] = col < row ? kk[nn][i] * ((i & 1) ? b2.y : b2.x) : 0.f;
            }
        }
        if (!SUM) {
#pragma unroll
            for (int nn = 0; nn < 2; nn++) {
                *reinterpret_cast<float2*>(&buf.inv.A[g][8 * nn + 2 * t]) = make_float2(kk[nn][0], kk[nn][1]);
                *reinterpret_cast<float2*>(&buf.inv.A[g + 8][8 * nn + 2 * t]) = make_float2(kk[nn][2], kk[nn][3]);
            }
        }
        note(qk);
        Frag<3> f;
        from_c(f, qk[0], qk[1]);
        store(aA, kPartC, f);
        __syncwarp();
        if (c + NB < nchunks) issue(c + NB, st ^ 1);  // K and Q have been read; the other copy of V was flushed before
        Frag<3> tt;
        if constexpr (!SUM) {
            invert_lower<C + 4>(&buf.inv.A[0][0], &buf.inv.Tt[0][0][0], lane);
            __syncwarp();
            load_cols(tt, aT, kPartC);                // T^T as right operand (BY_COLS); with registers 1 and 2 swapped, T as left
            Frag<3> ta;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                ta.r[i][0] = tt.r[i][0];
                ta.r[i][1] = tt.r[i][2];
                ta.r[i][2] = tt.r[i][1];
                ta.r[i][3] = tt.r[i][3];
            }
#pragma unroll kUnroll
            for (int k = 0; k < KS; k++) {            // X = T K
                Frag<NP> r;
                float x[2][4] = {};
                load_cols(r, aK + 32 * k, kPart);
                product<BY_COLS>(x, ta, r);
                from_c(f, x[0], x[1]);
                store(aX + 32 * k, kPart, f);
            }
        }
#pragma unroll kUnroll
        for (int j = 0; j < NCW; j++) {               // (T V)^T = V^T T^T
            float x[2][4];
            tile_block_t<PV>(x, &buf.v[st][2 * t][16 * j + g]);
            if constexpr (!SUM) {
                Frag<NP> fv;
                from_c(fv, x[0], x[1]);
#pragma unroll
                for (int i = 0; i < 8; i++) x[i >> 2][i & 3] = 0.f;
                product<BY_COLS>(x, fv, tt);
            }
            buf.tv[j][0][lane] = make_float4(x[0][0], x[0][1], x[0][2], x[0][3]);
            buf.tv[j][1][lane] = make_float4(x[1][0], x[1][1], x[1][2], x[1][3]);
        }
        warp_arrive(&filled[b], lane);
        const int t0 = c * C, nt = min(C, p.L - t0);
        Frag<3> ra;
        load_rows(ra, aA, kPartC);
        wait(&done[b], phase);
#pragma unroll kUnroll
        for (int j = 0; j < NCW; j++) {
            float y[2][4], w[2][4], u[2][4];
            Frag<3> us;
            *reinterpret_cast<float4*>(w[0]) = buf.tv[j][0][lane];
            *reinterpret_cast<float4*>(w[1]) = buf.tv[j][1][lane];
            if constexpr (SUM) {
                from_c(us, w[0], w[1]);
            } else {
                scale(u, w, buf.beta[st]);
                from_c(us, u[0], u[1]);
                if (vop || vip) side(buf, st, w, u, 16 * j, t0, nt);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) y[i >> 2][i & 3] = 0.f;
            product<BY_ROWS>(y, us, ra);
#pragma unroll kUnroll
            for (int k = 0; k < KS; k++) {
                Frag<3> s;
                Frag<NP> r;
#pragma unroll
                for (int i = 0; i < 3; i++) *reinterpret_cast<uint4*>(s.r[i]) = buf.s[j][k][i][lane];
                load_rows(r, aQ + 32 * k, kPart);
                add_product<BY_ROWS>(y, s, r);
            }
            put_block_t<PV>(y, &buf.y[2 * t][16 * j + g]);
        }
        __syncwarp();
        flush<M, PV, T>(&buf.y[0][0], yp + t0 * p.out.sL, p.out.sL, nt, p.M, yvec && p.M == M, lane);
        if (vop) flush<M, PV, float>(&buf.v[st][0][0], vop + t0 * p.v_old.sL, p.v_old.sL, nt, p.M, vovec && p.M == M, lane);
        __syncwarp();
    }
    slot_barrier(0, (NCW + NB) * 32);
}
template <int E, int M, int NB, int CTAS, typename T, bool SUM>
__global__ void __launch_bounds__((M / 16 + NB) * 32, CTAS) delta_fwd_wy_few_kernel(const __grid_constant__ DeltaFwdParams p) {
    fwd_few<E, M, NB, T, SUM>(p);
    if (redo()) stepwise_forward<T, SUM>(p, nullptr);
}
template <int E, int M, int NB, typename T, bool SUM>
__global__ void __launch_bounds__((M / 16 + NB) * 32, 2) sum_bwd_wy_few_kernel(const __grid_constant__ SumBwdForwards a) {
    static_assert(E * M * sizeof(float) <= NB * sizeof(FewBuf<E, M, stream_parts<T>()>), "room for the state of stepwise_forward");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    fwd_few<E, M, NB, T, SUM>(a.p[blockIdx.y]);
    if (redo()) stepwise_forward<T, SUM>(a.p[blockIdx.y], reinterpret_cast<float*>(smem_raw));
}

// --------------------------------------------------------------------------------- forward, many sequences
// The same for many sequences: what counts is the number of resident warps, so the helpers keep nothing but operand
// tiles and the chain warps do everything that touches the state -- K S and Q S from one split of S, then T (V - K S) --
// and move V and the outputs between registers and global memory themselves.
template <int E, int NP>
struct FwdBuf {
    static constexpr int P = E + 8;
    __nv_bfloat16 K[NP][C][P], Q[NP][C][P];
    __nv_bfloat16 Tt[3][C][PC], Aqk[3][C][PC];
    float A[C][C + 4];
    float beta[C];
};

template <int E, int M, int NB, int CTAS, typename T, bool SUM>
__device__ __forceinline__ void fwd(const DeltaFwdParams& p) {
    constexpr int NCW = M / 16, KS = E / 16, NP = stream_parts<T>();
    using Buf = FwdBuf<E, NP>;
    constexpr int P = Buf::P, kPart = C * P * 2, kPartC = C * PC * 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Buf* bufs = reinterpret_cast<Buf*>(smem_raw);
    __shared__ unsigned long long filled[NB], freed[NB];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n = blockIdx.x / p.H, h = blockIdx.x - n * p.H;
    const int nchunks = (p.L + C - 1) / C;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NB; i++) {
            mbar_init(&filled[i], 1);
            mbar_init(&freed[i], NCW);
        }
        redo() = 0;
        mbar_fence_init();
    }
    __syncthreads();
    griddep_wait();
    griddep_launch_dependents();

    if (warp < NCW) {
        const int m0 = warp * 16, width = p.M - m0;
        float* W = p.W ? p.W + n * p.wN + h * p.wH + m0 : nullptr;    // none: a state that starts at zero and is not asked for
        float S[2 * KS][4];             // S[j]: state rows e = 8j + 2t, 8j + 2t + 1 of columns m = g, g + 8
#pragma unroll
        for (int j = 0; j < 2 * KS; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int e = 8 * j + 2 * t + (i & 1), m = g + 8 * (i >> 1);
                S[j][i] = W && e < p.E && m < width ? W[(long long)e * p.wE + m] : 0.f;
            }
        const T* vp = reinterpret_cast<const T*>(p.v.p) + n * p.v.sN + h * p.v.sH + m0 + 2 * t * p.v.sL + g;
        T* yp = reinterpret_cast<T*>(p.out.p) + n * p.out.sN + h * p.out.sH + m0 + 2 * t * p.out.sL + g;
        float* vop = SUM || !p.v_old.p ? nullptr : reinterpret_cast<float*>(p.v_old.p) + n * p.v_old.sN + h * p.v_old.sH + m0 + 2 * t * p.v_old.sL + g;
        float* vip = SUM || !p.v_ins.p ? nullptr : reinterpret_cast<float*>(p.v_ins.p) + n * p.v_ins.sN + h * p.v_ins.sH + m0 + 2 * t * p.v_ins.sL + g;
        float v[2][4];
        load_block_t<T>(v, vp, p.v.sL, min(C, p.L), width, g, t);
        int b = 0;
        unsigned phase = 0;
        for (int c = 0; c < nchunks; c++) {
            const int nt = min(C, p.L - c * C);
            Buf& buf = bufs[b];
            const unsigned at = 2 * lane_at(lane, P), atC = 2 * lane_at(lane, PC);
            const unsigned aK = smem_u32(&buf.K[0][0][0]) + at, aQ = smem_u32(&buf.Q[0][0][0]) + at;
            float u[2][4] = {}, y[2][4] = {};
            wait(&filled[b], phase);
#pragma unroll
            for (int k = 0; k < KS; k++) {          // K S and Q S
                Frag<3> s;
                Frag<NP> r;
                from_c(s, S[2 * k], S[2 * k + 1]);
                if (!SUM) {
                    load_rows(r, aK + 32 * k, kPart);
                    sum_product<BY_ROWS>(k, u, s, r);
                }
                load_rows(r, aQ + 32 * k, kPart);
                sum_product<BY_ROWS>(k, y, s, r);
            }
            if constexpr (SUM) {
#pragma unroll
                for (int i = 0; i < 8; i++) u[i >> 2][i & 3] = v[i >> 2][i & 3];
            } else {
#pragma unroll
                for (int i = 0; i < 8; i++) u[i >> 2][i & 3] = v[i >> 2][i & 3] - u[i >> 2][i & 3];
                Frag<3> s, r;
                from_c(s, u[0], u[1]);
                load_cols(r, smem_u32(&buf.Tt[0][0][0]) + atC, kPartC);
                float w[2][4] = {};
                product<BY_COLS>(w, s, r);          // w = T (V - K S)
                if (vop) {
#pragma unroll
                    for (int i = 0; i < 8; i++) v[i >> 2][i & 3] -= w[i >> 2][i & 3];
                    store_block_t<float>(v, vop + c * C * p.v_old.sL, p.v_old.sL, nt, width, g, t);
                }
#pragma unroll
                for (int nn = 0; nn < 2; nn++) {
                    const float2 b2 = *reinterpret_cast<const float2*>(&buf.beta[8 * nn + 2 * t]);
#pragma unroll
                    for (int i = 0; i < 4; i++) u[nn][i] = w[nn][i] * ((i & 1) ? b2.y : b2.x);
                }
                if (vip) store_block_t<float>(u, vip + c * C * p.v_ins.sL, p.v_ins.sL, nt, width, g, t);
            }
            if (c + 1 < nchunks) load_block_t<T>(v, vp + (c + 1) * C * p.v.sL, p.v.sL, min(C, p.L - (c + 1) * C), width, g, t);
            Frag<3> us;
            from_c(us, u[0], u[1]);
#pragma unroll
            for (int k = 0; k < KS; k++) {          // S += K^T u
                Frag<NP> r;
                float d[2][4] = {};
                load_cols(r, aK + 32 * k, kPart);
                product<BY_COLS>(d, us, r);
#pragma unroll
                for (int i = 0; i < 8; i++) S[2 * k + (i >> 2)][i & 3] += d[i >> 2][i & 3];
            }
            Frag<3> r;
            load_rows(r, smem_u32(&buf.Aqk[0][0][0]) + atC, kPartC);
            warp_arrive(&freed[b], lane);
            add_product<BY_ROWS>(y, us, r);         // y = Q S + tril(Q K^T) u
            store_block_t<T>(y, yp + c * C * p.out.sL, p.out.sL, nt, width, g, t);
            if (++b == NB) { b = 0; phase ^= 1; }
        }
        note(S);
        slot_barrier(0, (NCW + NB) * 32);           // the other warps have written what they have to write
        if (redo()) return;
#pragma unroll
        for (int j = 0; j < 2 * KS; j++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int e = 8 * j + 2 * t + (i & 1), m = g + 8 * (i >> 1);
                if (W && e < p.E && m < width) W[(long long)e * p.wE + m] = S[j][i];
            }
        return;
    }

    // ---- preparing warp: chunks b, b + NB, ...
    const int b = warp - NCW;
    Buf& buf = bufs[b];
    const T* kp = reinterpret_cast<const T*>(p.k.p) + n * p.k.sN + h * p.k.sH;
    const T* qp = reinterpret_cast<const T*>(p.q.p) + n * p.q.sN + h * p.q.sH;
    const T* betap = SUM ? nullptr : reinterpret_cast<const T*>(p.beta.p) + n * p.beta.sN + h * p.beta.sH;
    auto even = [&](const T* q, long long sL) {       // pairs of elements can be read in one access
        return p.E == E && (reinterpret_cast<uintptr_t>(q) & (2 * sizeof(T) - 1)) == 0 && (sL & 1) == 0;
    };
    const bool kpair = even(kp, p.k.sL), qpair = even(qp, p.q.sL);
    const unsigned at = 2 * lane_at(lane, P);
    const unsigned aK = smem_u32(&buf.K[0][0][0]) + at, aQ = smem_u32(&buf.Q[0][0][0]) + at;
    const unsigned aA = smem_u32(&buf.Aqk[0][0][0]) + 2 * lane_at(lane, PC);
    constexpr bool kAhead = KS <= 2;                  // the next chunk's K and Q wait in registers
    constexpr int KF = kAhead ? KS : 1;
    float kf[KF][2][4], qf[KF][2][4], bt = 0.f;
    auto fetch = [&](int c, int k, float (&kx)[2][4], float (&qx)[2][4]) {
        const int t0 = c * C, nt = min(C, p.L - t0);
        load_block<T>(kx, kp + (t0 + g) * p.k.sL + 16 * k + 2 * t, p.k.sL, nt, p.E - 16 * k, kpair, g, t);
        load_block<T>(qx, qp + (t0 + g) * p.q.sL + 16 * k + 2 * t, p.q.sL, nt, p.E - 16 * k, qpair, g, t);
    };
    auto fetch_beta = [&](int c) {
        if (!SUM && lane < C) bt = c * C + lane < p.L ? to_f32(betap[(c * C + lane) * p.beta.sL]) : 0.f;
    };
    if (b < nchunks) {
        fetch_beta(b);
        if (kAhead)
#pragma unroll
            for (int k = 0; k < KF; k++) fetch(b, k, kf[k], qf[k]);
    }
    unsigned phase = 1;
    for (int c = b; c < nchunks; c += NB, phase ^= 1) {
        wait(&freed[b], phase);                       // passes at once the first time round
        float kk[2][4] = {}, qk[2][4] = {};
        if (!SUM && lane < C) buf.beta[lane] = bt;
#pragma unroll
        for (int k = 0; k < KS; k++) {
            const int f = kAhead ? k : 0;
            if (!kAhead) fetch(c, k, kf[f], qf[f]);
            Frag<NP> fk, fq;
            from_c(fk, kf[f][0], kf[f][1]);
            from_c(fq, qf[f][0], qf[f][1]);
            store(aK + 32 * k, kPart, fk);
            store(aQ + 32 * k, kPart, fq);
            if (!SUM) sum_product<BY_ROWS>(k, kk, fk, fk);
            sum_product<BY_ROWS>(k, qk, fq, fk);
        }
        __syncwarp();
#pragma unroll
        for (int nn = 0; nn < 2; nn++) {
            const float2 b2 = SUM ? make_float2(0.f, 0.f) : *reinterpret_cast<const float2*>(&buf.beta[8 * nn + 2 * t]);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int row = g + 8 * (i >> 1), col = 8 * nn + 2 * t + (i & 1);
                if (col > row) qk[nn][i] = 0.f;
                if (!SUM) kk[nn][i] = col < row ? kk[nn][i] * ((i & 1) ? b2.y : b2.x) : 0.f;
            }
        }
        if (!SUM) {
#pragma unroll
            for (int nn = 0; nn < 2; nn++) {
                *reinterpret_cast<float2*>(&buf.A[g][8 * nn + 2 * t]) = make_float2(kk[nn][0], kk[nn][1]);
                *reinterpret_cast<float2*>(&buf.A[g + 8][8 * nn + 2 * t]) = make_float2(kk[nn][2], kk[nn][3]);
            }
        }
        note(qk);
        Frag<3> f;
        from_c(f, qk[0], qk[1]);
        store(aA, kPartC, f);
        if (c + NB < nchunks) {
            fetch_beta(c + NB);
            if (kAhead)
#pragma unroll
                for (int k = 0; k < KF; k++) fetch(c + NB, k, kf[k], qf[k]);
        }
        if (!SUM) {
            __syncwarp();
            invert_lower<C + 4>(&buf.A[0][0], &buf.Tt[0][0][0], lane);
        }
        warp_arrive(&filled[b], lane);
    }
    slot_barrier(0, (NCW + NB) * 32);
}
template <int E, int M, int NB, int CTAS, typename T, bool SUM>
__global__ void __launch_bounds__((M / 16 + NB) * 32, CTAS) delta_fwd_wy_kernel(const __grid_constant__ DeltaFwdParams p) {
    fwd<E, M, NB, CTAS, T, SUM>(p);
    if (redo()) stepwise_forward<T, SUM>(p, nullptr);
}
template <int E, int M, int NB, int CTAS, typename T, bool SUM>
__global__ void __launch_bounds__((M / 16 + NB) * 32, CTAS) sum_bwd_wy_kernel(const __grid_constant__ SumBwdForwards a) {
    static_assert(E * M * sizeof(float) <= NB * sizeof(FwdBuf<E, stream_parts<T>()>), "room for the state of stepwise_forward");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    fwd<E, M, NB, CTAS, T, SUM>(a.p[blockIdx.y]);
    if (redo()) stepwise_forward<T, SUM>(a.p[blockIdx.y], reinterpret_cast<float*>(smem_raw));
}

}  // namespace wy
}  // namespace fwp
