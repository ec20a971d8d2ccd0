// Input prologue and output epilogue of the delta-rule attention layer (sm_100a).
//
// Between the fused q/k/v/beta projection and the fast-weight op the reference's layers run a chain of
// separate elementwise and permute launches (language_modeling/src/utils/cuda_fast_weight_layer.py:106-125,
// algorithmic/layers.py:110-137):
//   qkvb (len, B, H, 3d+1) -> split -> sigmoid(beta) -> permute to (B, H, len, .) -> elu+1 -> sum-normalise q, k
// and after the op a scale, transpose and reshape back to (len, B, H*d) (cuda_fast_weight_layer.py:152-163).
// Here each direction is one pass: a projected row is read once and q, k, v, beta leave in the (B, H, len, .)
// layout with aligned, contiguous rows (which is also what lets the op stage them with 16-byte and bulk
// copies); the backward pass recomputes the normalisation from the same row and writes the gradient row once.
// All kernels are plain streaming kernels.  The prologue kernels give 8, 16 or 32 lanes to a (len, batch, head) row,
// visit rows in the order of the projected tensor so that reads are fully contiguous and writes are whole aligned
// rows, and issue every load before the first use; the tile forms below move the same rows by 16-byte accesses.  The
// transpose moves 16-byte pieces, four per thread.
#include "fwp_core.cuh"

namespace fwp {

constexpr int kLayerWarps = 8;          // warps per CTA
constexpr int kLayerRows = 4;           // pieces per thread of the transpose, all loads issued before the first use
constexpr int kLayerMaxD = 128;

struct LayerDims {
    int L, B, H, D;
    long long rows;     // L * B * H
};
struct PrologueParams {
    const float* qkvb;
    float *q, *k, *v, *beta;
    float scale;        // of the queries
    LayerDims d;
};
struct PrologueGradParams {
    const float *qkvb, *gq, *gk, *gv, *gbeta;
    float* gx;
    float scale;
    LayerDims d;
};
struct TransposeParams {
    const float* src;
    float* dst;
    LayerDims d;
    int per_row;
    float scale;
    int to_len_major;
};

// elu(x) + 1 = x + 1 for x > 0, exp(x) otherwise
__device__ __forceinline__ float elu_p1(float x) { return x > 0.f ? x + 1.f : expf(x); }

// row r of the projected (len, B, H, .) tensor -> row of the (B, H, len, .) tensors (rows fit 31 bits: 32-bit divisions)
__device__ __forceinline__ long long bhl_row(const LayerDims& d, long long r) {
    const unsigned r32 = (unsigned)r;
    const unsigned lb = r32 / (unsigned)d.H, h = r32 - lb * (unsigned)d.H;
    const unsigned l = lb / (unsigned)d.B, b = lb - l * (unsigned)d.B;
    return ((long long)b * d.H + h) * d.L + l;
}

// sum over the LPR consecutive lanes that share a row
template <int LPR>
__device__ __forceinline__ float row_sum(float x) {
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// LPR lanes share a row (8, 16 or 32 for D up to 32, 64, 128); lane `sub` of a row holds elements sub + LPR*j,
// j < 4, of each of q, k, v, so that one load instruction covers 32/LPR rows with contiguous 4*LPR-byte pieces.
constexpr int kLayerPer = 4;

template <int LPR, int PASSES>
__global__ void __launch_bounds__(kLayerWarps * 32) layer_prologue_fwd_kernel(const PrologueParams p) {
    griddep_wait();
    griddep_launch_dependents();
    const LayerDims& d = p.d;
    const float* __restrict__ qkvb = p.qkvb;
    float *__restrict__ q = p.q, *__restrict__ k = p.k, *__restrict__ v = p.v, *__restrict__ beta = p.beta;
    constexpr int RPW = 32 / LPR;       // rows per warp and pass
    const int lane = threadIdx.x & 31, sub = lane % LPR, D = d.D;
    const long long r0 = ((long long)blockIdx.x * kLayerWarps + (threadIdx.x >> 5)) * (RPW * PASSES) + lane / LPR;
    float xq[PASSES][kLayerPer], xk[PASSES][kLayerPer], xv[PASSES][kLayerPer], xb[PASSES];
#pragma unroll
    for (int a = 0; a < PASSES; a++) {
        const long long r = r0 + a * RPW;
        const float* x = qkvb + r * (3 * D + 1);
        const bool live = r < d.rows;
#pragma unroll
        for (int j = 0; j < kLayerPer; j++) {
            const int i = sub + LPR * j;
            const bool ok = live && i < D;
            xq[a][j] = ok ? x[i] : 0.f;
            xk[a][j] = ok ? x[D + i] : 0.f;
            xv[a][j] = ok ? x[2 * D + i] : 0.f;
        }
        xb[a] = (live && sub == 0) ? x[3 * D] : 0.f;
    }
#pragma unroll
    for (int a = 0; a < PASSES; a++) {
        const long long r = r0 + a * RPW;
        const bool live = r < d.rows;
        const long long o = live ? bhl_row(d, r) : 0;
        float sq = 0.f, sk = 0.f;
#pragma unroll
        for (int j = 0; j < kLayerPer; j++) {
            const bool ok = sub + LPR * j < D;
            xq[a][j] = ok ? elu_p1(xq[a][j]) : 0.f;
            xk[a][j] = ok ? elu_p1(xk[a][j]) : 0.f;
            sq += xq[a][j];
            sk += xk[a][j];
        }
        const float iq = p.scale / row_sum<LPR>(sq), ik = 1.f / row_sum<LPR>(sk);
        if (!live) continue;
#pragma unroll
        for (int j = 0; j < kLayerPer; j++) {
            const int i = sub + LPR * j;
            if (i < D) {
                q[o * D + i] = xq[a][j] * iq;
                k[o * D + i] = xk[a][j] * ik;
                v[o * D + i] = xv[a][j];
            }
        }
        if (sub == 0) beta[o] = 1.f / (1.f + expf(-xb[a]));
    }
}

// y = p / s with p = elu(x)+1:  dL/dx_i = (g_i - sum_j g_j y_j) / s * (x_i > 0 ? 1 : p_i);  sigmoid: g * b * (1 - b).  The
// queries are scale * y, so their gradient comes in as g / scale.
template <int LPR>
__global__ void __launch_bounds__(kLayerWarps * 32) layer_prologue_bwd_kernel(const PrologueGradParams p) {
    griddep_wait();
    griddep_launch_dependents();
    const LayerDims& d = p.d;
    const float *__restrict__ qkvb = p.qkvb, *__restrict__ gq = p.gq, *__restrict__ gk = p.gk, *__restrict__ gv = p.gv, *__restrict__ gbeta = p.gbeta;
    float* __restrict__ gx = p.gx;
    constexpr int RPW = 32 / LPR;
    const int lane = threadIdx.x & 31, sub = lane % LPR, D = d.D;
    const long long r = ((long long)blockIdx.x * kLayerWarps + (threadIdx.x >> 5)) * RPW + lane / LPR;
    const bool live = r < d.rows;
    const long long o = live ? bhl_row(d, r) : 0;
    const float* x = qkvb + r * (3 * D + 1);
    float xq[kLayerPer], xk[kLayerPer], aq[kLayerPer], ak[kLayerPer], av[kLayerPer];
#pragma unroll
    for (int j = 0; j < kLayerPer; j++) {
        const int i = sub + LPR * j;
        const bool ok = live && i < D;
        xq[j] = ok ? x[i] : 0.f;
        xk[j] = ok ? x[D + i] : 0.f;
        aq[j] = ok ? p.scale * gq[o * D + i] : 0.f;
        ak[j] = ok ? gk[o * D + i] : 0.f;
        av[j] = ok ? gv[o * D + i] : 0.f;
    }
    const float xb = (live && sub == 0) ? x[3 * D] : 0.f;
    const float ab = (live && sub == 0) ? gbeta[o] : 0.f;
    float pq[kLayerPer], pk[kLayerPer];
    float sq = 0.f, sk = 0.f, dq = 0.f, dk = 0.f;
#pragma unroll
    for (int j = 0; j < kLayerPer; j++) {
        const bool ok = sub + LPR * j < D;
        pq[j] = ok ? elu_p1(xq[j]) : 0.f;
        pk[j] = ok ? elu_p1(xk[j]) : 0.f;
        sq += pq[j];
        sk += pk[j];
        dq = fmaf(aq[j], pq[j], dq);
        dk = fmaf(ak[j], pk[j], dk);
    }
    const float iq = 1.f / row_sum<LPR>(sq), ik = 1.f / row_sum<LPR>(sk);
    dq = row_sum<LPR>(dq) * iq;     // sum_j g_j y_j
    dk = row_sum<LPR>(dk) * ik;
    if (!live) return;
    float* y = gx + r * (3 * D + 1);
#pragma unroll
    for (int j = 0; j < kLayerPer; j++) {
        const int i = sub + LPR * j;
        if (i < D) {
            y[i] = (aq[j] - dq) * iq * (xq[j] > 0.f ? 1.f : pq[j]);
            y[D + i] = (ak[j] - dk) * ik * (xk[j] > 0.f ? 1.f : pk[j]);
            y[2 * D + i] = av[j];
        }
    }
    if (sub == 0) {
        const float sg = 1.f / (1.f + expf(-xb));
        y[3 * D] = ab * sg * (1.f - sg);
    }
}

// The same two passes for D % 4 == 0 and 16-byte aligned tensors.  A warp takes a span of 32/LPR projected rows (4 or 8):
// (3D+1) * 32/LPR floats that start on a 16-byte boundary, although the rows in the span do not.  It goes to shared memory by
// 16-byte copies; LPR lanes share a row, lane `sub` holding elements 4 (sub + LPR m) + j (j < 4) of each of q, k, v, so that
// rows of the (B, H, len, .) tensors move by 16-byte accesses and with LPR = 8 a warp's reads of the span (four rows, each
// 1 mod 4 floats after the one before) meet every bank once.  What bounded the 4-byte kernels was the
// load/store unit (71 %) and issue (69 %).  The backward does not load what only the gradient of v replaces and writes the
// gradient row over the row it was computed from.  Warps never wait for one another.
template <int LPR, int MP>
struct LayerTile {
    static constexpr int kWarps = MP == 4 ? 4 : 8;
    static constexpr int kRows = 32 / LPR;                  // a warp's rows; 6 KB of shared memory for D = 128, 1.6 KB for 16, 32
    static constexpr int kThreads = kWarps * 32;
};

// the warp's rows of the projected tensor -> its part of shared memory, without the 16-byte pieces that hold nothing but
// values if SKIP_V; returns how many rows there are.  A warp past the last row has none, not a negative count: the remainder of a
// negative length would lie in the span of the last warp that has rows.
template <int ROWS, int SKIP_V>
__device__ __forceinline__ int load_span(float* xs, const float* qkvb, long long r0, const LayerDims& d) {
    const int W = 3 * d.D + 1, lane = threadIdx.x & 31;
    const int n = max(0, (int)min(d.rows - r0, (long long)ROWS)), len = n * W;
    const float* src = qkvb + r0 * W;
    for (int i = 4 * lane; i + 3 < len; i += 128) {
        if (SKIP_V) {
            int c = i;
#pragma unroll
            for (int r = 1; r < ROWS; r++) c -= i >= r * W ? W : 0;
            if (c >= 2 * d.D && c + 3 < 3 * d.D) continue;
        }
        cp_async16(xs + i, src + i);
    }
    const int rest = (len & ~3) + lane;
    if (rest < len) xs[rest] = src[rest];
    cp_async_commit();
    return n;
}

__device__ __forceinline__ float4 f4(const float* x) { return make_float4(x[0], x[1], x[2], x[3]); }

template <int LPR, int MP>
__global__ void __launch_bounds__(LayerTile<LPR, MP>::kThreads) layer_prologue_fwd_tile_kernel(const PrologueParams p) {
    using T = LayerTile<LPR, MP>;
    extern __shared__ float4 span4[];
    griddep_wait();
    griddep_launch_dependents();
    const LayerDims& d = p.d;
    const int D = d.D, W = 3 * D + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LPR, row = lane / LPR;
    const long long r0 = ((long long)blockIdx.x * T::kWarps + warp) * T::kRows;
    float* xs = reinterpret_cast<float*>(span4) + warp * T::kRows * W;
    const int n = load_span<T::kRows, 0>(xs, p.qkvb, r0, d);
    const bool live = row < n;
    const long long o = live ? bhl_row(d, r0 + row) : 0;
    cp_async_wait<0>();
    __syncwarp();
    const float* x = xs + row * W;
    float pq[MP][4], pk[MP][4];
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int m = 0; m < MP; m++) {
        const int i = 4 * (sub + LPR * m);
        const bool ok = live && i < D;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            pq[m][j] = ok ? elu_p1(x[i + j]) : 0.f;
            pk[m][j] = ok ? elu_p1(x[D + i + j]) : 0.f;
            sq += pq[m][j];
            sk += pk[m][j];
        }
    }
    const float iq = p.scale / row_sum<LPR>(sq), ik = 1.f / row_sum<LPR>(sk);
    if (!live) return;
#pragma unroll
    for (int m = 0; m < MP; m++) {
        const int i = 4 * (sub + LPR * m);
        if (i < D) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                pq[m][j] *= iq;
                pk[m][j] *= ik;
            }
            *reinterpret_cast<float4*>(p.q + o * D + i) = f4(pq[m]);
            *reinterpret_cast<float4*>(p.k + o * D + i) = f4(pk[m]);
            *reinterpret_cast<float4*>(p.v + o * D + i) = f4(x + 2 * D + i);
        }
    }
    if (sub == 0) p.beta[o] = 1.f / (1.f + expf(-x[3 * D]));
}

// D <= 16 only: a lane's piece of each tensor is one 16-byte access.
__global__ void __launch_bounds__(LayerTile<4, 1>::kThreads) layer_prologue_bwd_tile_kernel(const PrologueGradParams p) {
    using T = LayerTile<4, 1>;
    extern __shared__ float4 span4[];
    griddep_wait();
    griddep_launch_dependents();
    const LayerDims& d = p.d;
    const int D = d.D, W = 3 * D + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane & 3, row = lane >> 2, i = 4 * sub;
    const long long r0 = ((long long)blockIdx.x * T::kWarps + warp) * T::kRows;
    float* xs = reinterpret_cast<float*>(span4) + warp * T::kRows * W;
    const int n = load_span<T::kRows, 1>(xs, p.qkvb, r0, d);
    const bool live = row < n, ok = live && i < D;
    const long long o = live ? bhl_row(d, r0 + row) : 0;
    float4 gq = make_float4(0.f, 0.f, 0.f, 0.f), gk = gq, gv = gq;
    if (ok) {
        gq = *reinterpret_cast<const float4*>(p.gq + o * D + i);
        gk = *reinterpret_cast<const float4*>(p.gk + o * D + i);
        gv = *reinterpret_cast<const float4*>(p.gv + o * D + i);
    }
    const float gb = (live && sub == 0) ? p.gbeta[o] : 0.f;
    cp_async_wait<0>();
    __syncwarp();
    float* x = xs + row * W;
    const float aq[4] = {p.scale * gq.x, p.scale * gq.y, p.scale * gq.z, p.scale * gq.w};
    const float ak[4] = {gk.x, gk.y, gk.z, gk.w}, av[4] = {gv.x, gv.y, gv.z, gv.w};
    float xq[4], xk[4], pq[4], pk[4];
    float sq = 0.f, sk = 0.f, dq = 0.f, dk = 0.f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        xq[j] = ok ? x[i + j] : 0.f;
        xk[j] = ok ? x[D + i + j] : 0.f;
        pq[j] = ok ? elu_p1(xq[j]) : 0.f;
        pk[j] = ok ? elu_p1(xk[j]) : 0.f;
        sq += pq[j];
        sk += pk[j];
        dq = fmaf(aq[j], pq[j], dq);
        dk = fmaf(ak[j], pk[j], dk);
    }
    const float iq = 1.f / row_sum<4>(sq), ik = 1.f / row_sum<4>(sk);
    dq = row_sum<4>(dq) * iq;       // sum_j g_j y_j
    dk = row_sum<4>(dk) * ik;
    if (ok) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            x[i + j] = (aq[j] - dq) * iq * (xq[j] > 0.f ? 1.f : pq[j]);
            x[D + i + j] = (ak[j] - dk) * ik * (xk[j] > 0.f ? 1.f : pk[j]);
            x[2 * D + i + j] = av[j];
        }
    }
    if (live && sub == 0) {
        const float sg = 1.f / (1.f + expf(-x[3 * D]));
        x[3 * D] = gb * sg * (1.f - sg);
    }
    __syncwarp();
    const int len = n * W, rest = (len & ~3) + lane;
    float* y = p.gx + r0 * W;
    for (int e = 4 * lane; e + 3 < len; e += 128) *reinterpret_cast<float4*>(y + e) = *reinterpret_cast<const float4*>(xs + e);
    if (rest < len) y[rest] = xs[rest];
}

// (B, H, len, D) <-> (len, B, H, D) with a scale: dst row of one side = scale * src row of the other.
// One thread per 16-byte piece (4-byte piece when D is not a multiple of 4), kLayerRows pieces per thread.
template <typename V>
__global__ void __launch_bounds__(kLayerWarps * 32) layer_transpose_kernel(const TransposeParams p) {
    griddep_wait();
    griddep_launch_dependents();
    const V* __restrict__ src = reinterpret_cast<const V*>(p.src);
    V* __restrict__ dst = reinterpret_cast<V*>(p.dst);
    const LayerDims& d = p.d;
    const int per_row = p.per_row, to_len_major = p.to_len_major;
    const float scale = p.scale;
    const long long total = d.rows * per_row;
    const long long i0 = ((long long)blockIdx.x * kLayerRows) * (kLayerWarps * 32) + threadIdx.x;
    V x[kLayerRows];
    long long to[kLayerRows];
#pragma unroll
    for (int a = 0; a < kLayerRows; a++) {
        const long long i = i0 + (long long)a * (kLayerWarps * 32);      // piece index in (len, B, H, .) order
        to[a] = -1;
        if (i < total) {
            long long r;
            int c;
            if (total <= 0x7fffffffLL) {
                const unsigned q32 = (unsigned)i / (unsigned)per_row;
                r = q32;
                c = (int)((unsigned)i - q32 * (unsigned)per_row);
            } else {
                r = i / per_row;
                c = (int)(i - r * per_row);
            }
            const long long j = bhl_row(d, r) * per_row + c;
            x[a] = src[to_len_major ? j : i];
            to[a] = to_len_major ? i : j;
        }
    }
#pragma unroll
    for (int a = 0; a < kLayerRows; a++) {
        if (to[a] < 0) continue;
        if constexpr (sizeof(V) == 16) {
            x[a].x *= scale; x[a].y *= scale; x[a].z *= scale; x[a].w *= scale;
        } else {
            x[a] *= scale;
        }
        dst[to[a]] = x[a];
    }
}

// dst[n,h,t,:] = f(t == 0 ? first[n,h,0,:] : src[n,h,t-1,:]), f = identity or tanh; with a minuend, minuend - that.
// V = float4 when rows are 16-byte aligned and D % 4 == 0.
struct DelayedParams {
    const float* src; long long sN, sH, sL;
    const float* first; long long fN, fH;
    const float* minuend; long long mN, mH, mL;
    float* dst; long long dN, dH, dL;
    int H, L, per_row, op;
    long long total;
};
template <typename V>
__global__ void __launch_bounds__(256) delayed_kernel(const DelayedParams p) {
    griddep_wait();
    griddep_launch_dependents();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= p.total) return;
    constexpr int W = sizeof(V) / 4;
    const int c = (int)(i % p.per_row) * W;
    const long long row = i / p.per_row;
    const int t = (int)(row % p.L);
    const long long nh = row / p.L;
    const int h = (int)(nh % p.H);
    const long long n = nh / p.H;
    const float* sp = t == 0 ? p.first + n * p.fN + h * p.fH + c : p.src + n * p.sN + h * p.sH + (long long)(t - 1) * p.sL + c;
    V x = *reinterpret_cast<const V*>(sp);
    float* xf = reinterpret_cast<float*>(&x);
    if (p.op == 1) {
#pragma unroll
        for (int j = 0; j < W; j++) xf[j] = tanhf(xf[j]);
    }
    if (p.minuend) {
        const V m = *reinterpret_cast<const V*>(p.minuend + n * p.mN + h * p.mH + (long long)t * p.mL + c);
        const float* mf = reinterpret_cast<const float*>(&m);
#pragma unroll
        for (int j = 0; j < W; j++) xf[j] = mf[j] - xf[j];
    }
    *reinterpret_cast<V*>(p.dst + n * p.dN + h * p.dH + (long long)t * p.dL + c) = x;
}

// the tile kernels: every piece of 16 bytes lies in one row of q, k, v and on a boundary of 16
static bool layer_tile_ok(const LayerDims& d, const void* a, const void* b, const void* c, const void* e, const void* f = nullptr) {
    return d.D % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
                             reinterpret_cast<uintptr_t>(e) | reinterpret_cast<uintptr_t>(f)) & 15) == 0;
}
// Where the forward's is the faster one (us, 4-byte kernel and this, everything in L2):
//   D = 4, 8     4 rows 2.09 and 2.22, 2.02 and 2.22; 128 2.57 and 2.21; 12800 3.3 and 2.9; 65536 7.0 and 5.6;  D = 12, 16 at any size
//   D = 24       4 rows 2.4 and 2.2, 12800 3.9 and 3.3, but 25600 5.5 and 5.7, 65536 8.7 and 9.1 (a quarter of the lanes idle); D = 32 at any size
//   D = 96       4 rows 3.0 and 3.4, 3200 3.9 and 4.3; 6400 6.4 and 4.8, 25600 12.2 and 10.2;  D = 48, 64 at any size
//   D = 128      4 rows 3.2 and 3.9, 3200 4.2 and 5.1, 12800 8.3 and 8.9; 25600 13.5 and 12.6
static bool fwd_tile_pays(int D, long long rows) {
    if (D <= 8) return rows >= 128;
    if (D > 16 && D < 32) return rows < 16384;
    return D <= 64 || rows >= (D <= 96 ? 6144 : 16384);
}
template <int LPR, int MP, class K, class P>
static int launch_layer_tile(K kern, const P& p, cudaStream_t st) {
    using T = LayerTile<LPR, MP>;
    constexpr int rows = T::kWarps * T::kRows;
    return launch_dependent(kern, p, (int)((p.d.rows + rows - 1) / rows), T::kThreads, sizeof(float) * rows * (3 * p.d.D + 1), st,
                            nullptr);
}

static int layer_dims(int L, int B, int H, int D, LayerDims& d) {
    if (L <= 0 || B <= 0 || H <= 0 || D <= 0) return FWP_ERR_SHAPE;
    if (D > kLayerMaxD) return FWP_ERR_UNSUPPORTED;
    d.L = L; d.B = B; d.H = H; d.D = D;
    d.rows = (long long)L * B * H;
    if (d.rows > 0x7fffffffLL) return FWP_ERR_SHAPE;
    return FWP_OK;
}

}  // namespace fwp

using namespace fwp;

FWP_API int fwp_delta_layer_prologue_forward_scaled(int L, int B, int H, int D, const float* qkvb, float* q, float* k, float* v,
                                                    float* beta, float q_scale, void* stream, int device) {
    PrologueParams p = {qkvb, q, k, v, beta, q_scale, {}};
    if (int rc = layer_dims(L, B, H, D, p.d)) return rc;
    if (!qkvb || !q || !k || !v || !beta) return FWP_ERR_NULL;
    if ((reinterpret_cast<uintptr_t>(qkvb) | reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) |
         reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(beta)) & 3) return FWP_ERR_ALIGN;
    DeviceGuard guard(device);
    if (guard.status) return guard.status;
    cudaStream_t st = (cudaStream_t)stream;
    // L2 flushed before, 4-byte kernel and this: (512, 96, 8) rows of 16 45.8 and 32.8 us, (512, 32, 8) rows of 32 28.7 and 24.6,
    // of 64 41.8 and 39.0, (256, 32, 8) of 128 41.0 and 40.8, of 96 36.9 and 32.8.
    if (layer_tile_ok(p.d, qkvb, q, k, v) && fwd_tile_pays(D, p.d.rows)) {
        if (D <= 16) return launch_layer_tile<4, 1>(layer_prologue_fwd_tile_kernel<4, 1>, p, st);
        if (D <= 32) return launch_layer_tile<8, 1>(layer_prologue_fwd_tile_kernel<8, 1>, p, st);
        if (D <= 64) return launch_layer_tile<8, 2>(layer_prologue_fwd_tile_kernel<8, 2>, p, st);
        return launch_layer_tile<8, 4>(layer_prologue_fwd_tile_kernel<8, 4>, p, st);
    }
    auto grid = [&](int rows_per_warp) { return (int)((p.d.rows + kLayerWarps * rows_per_warp - 1) / (kLayerWarps * rows_per_warp)); };
    if (D <= 32) return launch_dependent(layer_prologue_fwd_kernel<8, 2>, p, grid(8), kLayerWarps * 32, 0, st, nullptr);
    if (D <= 64) return launch_dependent(layer_prologue_fwd_kernel<16, 2>, p, grid(4), kLayerWarps * 32, 0, st, nullptr);
    return launch_dependent(layer_prologue_fwd_kernel<32, 2>, p, grid(2), kLayerWarps * 32, 0, st, nullptr);
}

FWP_API int fwp_delta_layer_prologue_forward(int L, int B, int H, int D, const float* qkvb,
                                             float* q, float* k, float* v, float* beta, void* stream, int device) {
    return fwp_delta_layer_prologue_forward_scaled(L, B, H, D, qkvb, q, k, v, beta, 1.f, stream, device);
}

FWP_API int fwp_delta_layer_prologue_backward_scaled(int L, int B, int H, int D, const float* qkvb,
                                                     const float* grad_q, const float* grad_k, const float* grad_v,
                                                     const float* grad_beta, float* grad_qkvb, float q_scale, void* stream, int device) {
    PrologueGradParams p = {qkvb, grad_q, grad_k, grad_v, grad_beta, grad_qkvb, q_scale, {}};
    if (int rc = layer_dims(L, B, H, D, p.d)) return rc;
    if (!qkvb || !grad_q || !grad_k || !grad_v || !grad_beta || !grad_qkvb) return FWP_ERR_NULL;
    if ((reinterpret_cast<uintptr_t>(qkvb) | reinterpret_cast<uintptr_t>(grad_q) | reinterpret_cast<uintptr_t>(grad_k) |
         reinterpret_cast<uintptr_t>(grad_v) | reinterpret_cast<uintptr_t>(grad_beta) | reinterpret_cast<uintptr_t>(grad_qkvb)) & 3)
        return FWP_ERR_ALIGN;
    DeviceGuard guard(device);
    if (guard.status) return guard.status;
    cudaStream_t st = (cudaStream_t)stream;
    // L2 flushed before, 4-byte kernel and this form: (512, 96, 8) rows of 16 65.5 and 59.4 us, but (512, 32, 8) rows of 32
    // 36.8 and 40.9, of 64 58.1 and 68.2, (256, 32, 8) of 128 58.1 and 72.4.  In L2, D = 4 and 16: 4 rows 1.8 and 2.4, 1.9 and 2.5 us;
    // 12800 3.1 and 3.3, 3.4 and 4.0; 25600 4.3 and 4.4, 4.8 and 5.9; 65536 8.3 and 6.9, 9.3 and 9.1; 393216 42 and 33, 57 and 51.
    if (D <= 16 && p.d.rows >= 65536 && layer_tile_ok(p.d, qkvb, grad_q, grad_k, grad_v, grad_qkvb))
        return launch_layer_tile<4, 1>(layer_prologue_bwd_tile_kernel, p, st);
    auto grid = [&](int rows_per_warp) { return (int)((p.d.rows + kLayerWarps * rows_per_warp - 1) / (kLayerWarps * rows_per_warp)); };
    if (D <= 32) return launch_dependent(layer_prologue_bwd_kernel<8>, p, grid(4), kLayerWarps * 32, 0, st, nullptr);
    if (D <= 64) return launch_dependent(layer_prologue_bwd_kernel<16>, p, grid(2), kLayerWarps * 32, 0, st, nullptr);
    return launch_dependent(layer_prologue_bwd_kernel<32>, p, grid(1), kLayerWarps * 32, 0, st, nullptr);
}

FWP_API int fwp_delta_layer_prologue_backward(int L, int B, int H, int D, const float* qkvb,
                                              const float* grad_q, const float* grad_k, const float* grad_v,
                                              const float* grad_beta, float* grad_qkvb, void* stream, int device) {
    return fwp_delta_layer_prologue_backward_scaled(L, B, H, D, qkvb, grad_q, grad_k, grad_v, grad_beta, grad_qkvb, 1.f, stream, device);
}

FWP_API int fwp_delta_layer_transpose(int L, int B, int H, int D, const float* src, float* dst, float scale,
                                      int to_len_major, void* stream, int device) {
    LayerDims d;
    if (int rc = layer_dims(L, B, H, D, d)) return rc;
    if (!src || !dst) return FWP_ERR_NULL;
    const uintptr_t mask = (D & 3) == 0 ? 15 : 3;
    if ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & mask) return FWP_ERR_ALIGN;
    DeviceGuard guard(device);
    if (guard.status) return guard.status;
    const int per_row = (D & 3) == 0 ? D / 4 : D;
    const long long per_cta = (long long)kLayerWarps * 32 * kLayerRows;
    const long long ctas = (d.rows * per_row + per_cta - 1) / per_cta;
    if (ctas > 0x7fffffffLL) return FWP_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    const TransposeParams p = {src, dst, d, per_row, scale, to_len_major ? 1 : 0};
    if ((D & 3) == 0) return launch_dependent(layer_transpose_kernel<float4>, p, (int)ctas, kLayerWarps * 32, 0, st, nullptr);
    return launch_dependent(layer_transpose_kernel<float>, p, (int)ctas, kLayerWarps * 32, 0, st, nullptr);
}

FWP_API int fwp_delayed(int N, int H, int L, int D, const fwp_tensor* src, const fwp_tensor* first,
                        const fwp_tensor* minuend, const fwp_tensor* dst, int op, void* stream, int device) {
    if (N <= 0 || H <= 0 || L <= 0 || D <= 0) return FWP_ERR_SHAPE;
    if (op != 0 && op != 1) return FWP_ERR_UNSUPPORTED;
    int rc;
    if ((rc = check_tensor(src, 4, true)) || (rc = check_tensor(first, 4, true)) || (rc = check_tensor(dst, 4, true)) ||
        (rc = check_tensor(minuend, 4, false)))
        return rc;
    const bool sub = minuend && minuend->data;
    DeviceGuard guard(device);
    if (guard.status) return guard.status;
    DelayedParams p;
    p.src = (const float*)src->data; p.sN = src->stride[0]; p.sH = src->stride[1]; p.sL = src->stride[2];
    p.first = (const float*)first->data; p.fN = first->stride[0]; p.fH = first->stride[1];
    p.minuend = sub ? (const float*)minuend->data : nullptr;
    p.mN = sub ? minuend->stride[0] : 0; p.mH = sub ? minuend->stride[1] : 0; p.mL = sub ? minuend->stride[2] : 0;
    p.dst = (float*)dst->data; p.dN = dst->stride[0]; p.dH = dst->stride[1]; p.dL = dst->stride[2];
    p.H = H; p.L = L; p.op = op;
    auto al = [](const void* q, long long a, long long b, long long c) {
        return (reinterpret_cast<uintptr_t>(q) & 15) == 0 && a % 4 == 0 && b % 4 == 0 && c % 4 == 0;
    };
    const bool vec = D % 4 == 0 && al(p.src, p.sN, p.sH, p.sL) && al(p.first, p.fN, p.fH, 0) &&
                     al(p.dst, p.dN, p.dH, p.dL) && (!sub || al(p.minuend, p.mN, p.mH, p.mL));
    p.per_row = vec ? D / 4 : D;
    p.total = (long long)N * H * L * p.per_row;
    const long long ctas = (p.total + 255) / 256;
    if (ctas > 0x7fffffffLL) return FWP_ERR_SHAPE;
    cudaStream_t st = (cudaStream_t)stream;
    return vec ? launch_dependent(delayed_kernel<float4>, p, (int)ctas, 256, 0, st, nullptr)
               : launch_dependent(delayed_kernel<float>, p, (int)ctas, 256, 0, st, nullptr);
}
