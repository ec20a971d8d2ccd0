// One delta rule's gradients at d = 32, one step at a time, by a warp that trails the chain (sm_100a).
//
// In the backward of the delta RNN and LSTM a chain warp leaves dz (the gradient of the read-out) and w = v - v_old of every
// step in shared memory; what remains, time reversed, is
//   G += s (x) dz;  r = G^T k;  dv = beta r;  dbeta = r . w;  S -= k (x) u;  dk = G u - S dv;  G -= k (x) dv     (u = beta w).
// The chain leaves -u beside w, and dv is exchanged negated, so that no vector is negated here.
// Lane (eg, mg) = (lane >> 3, lane & 7) holds an 8 x 4 piece of G and of S (Tile32): rows 8 eg .. 8 eg + 7, columns 2 mg, 2 mg + 1 and
// 16 + 2 mg, 17 + 2 mg.  Both roles of G come from the one copy, so a step is 96 packed multiply-adds against
// 128 with G held by columns and by rows, and each lane reads 8 + 8 + 4 + 4 + 4 operands where a line per
// lane takes 32 of each.  Sums over the other lanes are reduce-scatters: 3 shuffles for r, 7 for dk.  What a lane gives away
// in the first of them is always its second half, because lanes that keep the upper half hold their piece upper half first.
#pragma once
#include "fwp_core.cuh"

namespace fwp {

__device__ __forceinline__ f2 fmul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 fsub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 f2_dup(float x) { return f2_pack(x, x); }
__device__ __forceinline__ f2 shfl_xor2(f2 x, int o) {
    float lo, hi;
    f2_unpack(x, lo, hi);
    return f2_pack(__shfl_xor_sync(0xffffffffu, lo, o), __shfl_xor_sync(0xffffffffu, hi, o));
}

// Lane (eg, mg) = (lane >> 3, lane & 7) of a 32 x 32 matrix in pieces: [column][pair of rows]
struct Tile32 {
    int row0, row1;         // first of the four rows this lane keeps when a sum runs over columns, and of the four it gives away
    int col0, col1;         // first of the two columns it keeps when a sum runs over rows, and of the two it gives away
    int own;                // the column it ends up with there (the row it ends up with is its lane index)
    int lane;

    __device__ __forceinline__ explicit Tile32(int lane_) : lane(lane_) {
        const int eg = lane >> 3, mg = lane & 7, b2 = (lane >> 2) & 1, b4 = lane >> 4;
        row0 = 8 * eg + 4 * b2;
        row1 = 8 * eg + 4 * (b2 ^ 1);
        col0 = 2 * mg + 16 * b4;
        col1 = 2 * mg + 16 * (b4 ^ 1);
        own = col0 + ((lane >> 3) & 1);
    }
    __device__ __forceinline__ int row(int i) const { return (i < 2 ? row0 : row1) + 2 * (i & 1); }     // of pair i: the first
    __device__ __forceinline__ int col(int c) const { return (c < 2 ? col0 : col1) + (c & 1); }
    __device__ __forceinline__ void rows(f2 (&x)[4], const float* p) const {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p + row0), b = *reinterpret_cast<const ulonglong2*>(p + row1);
        x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
    }
    __device__ __forceinline__ void cols(f2 (&x)[4], const float* p) const {
        const float2 a = *reinterpret_cast<const float2*>(p + col0), b = *reinterpret_cast<const float2*>(p + col1);
        x[0] = f2_dup(a.x); x[1] = f2_dup(a.y); x[2] = f2_dup(b.x); x[3] = f2_dup(b.y);
    }
    // shares of the four columns, summed over the rows: the sum of column `own`
    __device__ __forceinline__ float sum_rows(float (&x)[4]) const {
        x[0] += __shfl_xor_sync(0xffffffffu, x[2], 16);
        x[1] += __shfl_xor_sync(0xffffffffu, x[3], 16);
        const bool b3 = lane & 8;
        return (b3 ? x[1] : x[0]) + __shfl_xor_sync(0xffffffffu, b3 ? x[0] : x[1], 8);
    }
    // shares of the eight rows, summed over the columns: the sum of row `lane`
    __device__ __forceinline__ float sum_cols(f2 (&x)[4]) const {
        x[0] = fadd2(x[0], shfl_xor2(x[2], 4));
        x[1] = fadd2(x[1], shfl_xor2(x[3], 4));
        const bool b1 = lane & 2, b0 = lane & 1;
        const f2 sum = fadd2(b1 ? x[1] : x[0], shfl_xor2(b1 ? x[0] : x[1], 2));
        float lo, hi;
        f2_unpack(sum, lo, hi);
        return (b0 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b0 ? lo : hi, 1);
    }
};

struct Trail32 : Tile32 {
    f2 G[16], S[16];

    __device__ __forceinline__ Trail32(int lane_, const float* W, long long wE) : Tile32(lane_) {
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float* w = W + row(i) * wE + col(c);
                S[4 * c + i] = f2_pack(w[0], w[wE]);
                G[4 * c + i] = 0ull;
            }
    }
    // s, k, dz, nu = -u: this step's vectors in shared memory; xch: 32 floats of this warp's own, another 32 in the next step.
    // Gives r and dv of column `own` and dk of row `lane`.
    __device__ __forceinline__ void step(const float* s, const float* k, const float* dz, const float* nu, float beta, float* xch,
                                         float& r, float& dv, float& dk) {
        f2 ss[4], kk[4], x[4], acc[4], neg[4];
        rows(ss, s);
        rows(kk, k);
        cols(x, dz);
        float rr[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                G[4 * c + i] = ffma2(ss[i], x[c], G[4 * c + i]);
                acc[c] = i == 0 ? fmul2(G[4 * c], kk[0]) : ffma2(G[4 * c + i], kk[i], acc[c]);
            }
            rr[c] = f2_hsum(acc[c]);
        }
        r = sum_rows(rr);
        dv = beta * r;
        xch[own] = -dv;
        // what does not wait for dv
        cols(x, nu);
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                neg[i] = c == 0 ? fmul2(G[i], x[0]) : ffma2(G[4 * c + i], x[c], neg[i]);
                S[4 * c + i] = ffma2(kk[i], x[c], S[4 * c + i]);        // S_{t-1}
            }
        __syncwarp();
        cols(x, xch);
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                acc[i] = c == 0 ? fmul2(S[i], x[0]) : ffma2(S[4 * c + i], x[c], acc[i]);
                G[4 * c + i] = ffma2(kk[i], x[c], G[4 * c + i]);
            }
#pragma unroll
        for (int i = 0; i < 4; i++) acc[i] = fsub2(acc[i], neg[i]);
        dk = sum_cols(acc);
    }
};

// dbeta of a chunk of TC steps at once from r w of every step (rows of 36 in `pw`): 32 / TC lanes share a step
template <int TC>
__device__ __forceinline__ void trail_dbeta(const float* pw, float* out, long long sL, int nt, int lane) {
    constexpr int D = 32, SH = 32 / TC;
    __syncwarp();
    const float* q = pw + (lane / SH) * (D + 4) + (lane % SH) * (D / SH);
    float db = 0.f;
#pragma unroll
    for (int i = 0; i < D / SH; i++) db += q[i];
#pragma unroll
    for (int o = SH / 2; o > 0; o >>= 1) db += __shfl_xor_sync(0xffffffffu, db, o);
    if (lane % SH == 0 && lane / SH < nt) out[(lane / SH) * sL] = db;
    __syncwarp();
}

}  // namespace fwp
