// One delta rule's gradients at d = 32, one step at a time, by a warp that trails the chain (sm_100a).
//
// In the backward of the delta RNN and LSTM a chain warp leaves dz (the gradient of the read-out) and w = v - v_old of every
// step in shared memory; what remains, time reversed, is
//   G += s (x) dz;  r = G^T k;  dv = beta r;  dbeta = r . w;  S -= beta k (x) w;  dk = beta G w - S dv;  G -= k (x) dv.
// Lane (eg, mg) = (lane >> 3, lane & 7) holds an 8 x 4 piece of G and of S: rows 8 eg .. 8 eg + 7, columns 2 mg, 2 mg + 1 and
// 16 + 2 mg, 17 + 2 mg.  Both roles of G come from the one copy, so a step is 96 packed multiply-adds and 104 with the
// scalings, against 128 with G held by columns and by rows, and each lane reads 8 + 8 + 4 + 4 + 4 operands where a line per
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
__device__ __forceinline__ f2 f2_dup(float x) { return f2_pack(x, x); }
__device__ __forceinline__ f2 shfl_xor2(f2 x, int o) {
    float lo, hi;
    f2_unpack(x, lo, hi);
    return f2_pack(__shfl_xor_sync(0xffffffffu, lo, o), __shfl_xor_sync(0xffffffffu, hi, o));
}

struct Trail32 {
    int row0, row1;         // first of the four rows this lane keeps in dk's reduction, and of the four it gives away
    int col0, col1;         // first of the two columns it keeps in r's reduction, and of the two it gives away
    int own;                // the column whose r this lane ends up with (and the row of dk it ends up with is its lane index)
    int lane;
    f2 G[16], S[16];        // [column][pair of rows]

    __device__ __forceinline__ void init(int lane_, const float* W, long long wE) {
        lane = lane_;
        const int eg = lane >> 3, mg = lane & 7, b2 = (lane >> 2) & 1, b4 = lane >> 4;
        row0 = 8 * eg + 4 * b2;
        row1 = 8 * eg + 4 * (b2 ^ 1);
        col0 = 2 * mg + 16 * b4;
        col1 = 2 * mg + 16 * (b4 ^ 1);
        own = col0 + ((lane >> 3) & 1);
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float* w = W + (long long)((i < 2 ? row0 : row1) + 2 * (i & 1)) * wE + (c < 2 ? col0 : col1) + (c & 1);
                S[4 * c + i] = f2_pack(w[0], w[wE]);
                G[4 * c + i] = 0ull;
            }
    }
    __device__ __forceinline__ void rows(f2 (&x)[4], const float* p) const {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p + row0), b = *reinterpret_cast<const ulonglong2*>(p + row1);
        x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
    }
    __device__ __forceinline__ void cols(f2 (&x)[4], const float* p) const {
        const float2 a = *reinterpret_cast<const float2*>(p + col0), b = *reinterpret_cast<const float2*>(p + col1);
        x[0] = f2_dup(a.x); x[1] = f2_dup(a.y); x[2] = f2_dup(b.x); x[3] = f2_dup(b.y);
    }
    // s, k, dz, w: this step's vectors in shared memory; xch: 32 floats of this warp's own, another 32 in the next step.
    // Gives r and dv of column `own` and dk of row `lane`.
    __device__ __forceinline__ void step(const float* s, const float* k, const float* dz, const float* w, float beta, float* xch,
                                         float& r, float& dv, float& dk) {
        f2 ss[4], kk[4], x[4], acc[4];
        rows(ss, s);
        rows(kk, k);
        cols(x, dz);
        float rr[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            acc[c] = 0ull;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                G[4 * c + i] = ffma2(ss[i], x[c], G[4 * c + i]);
                acc[c] = ffma2(G[4 * c + i], kk[i], acc[c]);
            }
            rr[c] = f2_hsum(acc[c]);
        }
        rr[0] += __shfl_xor_sync(0xffffffffu, rr[2], 16);
        rr[1] += __shfl_xor_sync(0xffffffffu, rr[3], 16);
        const bool b3 = lane & 8;
        r = (b3 ? rr[1] : rr[0]) + __shfl_xor_sync(0xffffffffu, b3 ? rr[0] : rr[1], 8);
        dv = beta * r;
        xch[own] = -dv;
        // what does not wait for dv
        f2 kb[4];
        cols(x, w);
        const f2 nb = f2_dup(-beta);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            kb[i] = fmul2(kk[i], nb);
            acc[i] = 0ull;
        }
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                acc[i] = ffma2(G[4 * c + i], x[c], acc[i]);
                S[4 * c + i] = ffma2(kb[i], x[c], S[4 * c + i]);        // S_{t-1}
            }
        const f2 pb = f2_dup(beta);
#pragma unroll
        for (int i = 0; i < 4; i++) acc[i] = fmul2(acc[i], pb);
        __syncwarp();
        cols(x, xch);
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int i = 0; i < 4; i++) {
                acc[i] = ffma2(S[4 * c + i], x[c], acc[i]);
                G[4 * c + i] = ffma2(kk[i], x[c], G[4 * c + i]);
            }
        acc[0] = fadd2(acc[0], shfl_xor2(acc[2], 4));
        acc[1] = fadd2(acc[1], shfl_xor2(acc[3], 4));
        const bool b1 = lane & 2, b0 = lane & 1;
        const f2 sum = fadd2(b1 ? acc[1] : acc[0], shfl_xor2(b1 ? acc[0] : acc[1], 2));
        float lo, hi;
        f2_unpack(sum, lo, hi);
        dk = (b0 ? hi : lo) + __shfl_xor_sync(0xffffffffu, b0 ? lo : hi, 1);
    }
};

}  // namespace fwp
