// What the chunkwise (WY) plans share: blocks of a stream in fragment order, and the inverse of a chunk's triangular
// system.  A chunk is sixteen steps.
#pragma once
#include "fwp_delta_params.cuh"
#include "fwp_split3.cuh"

namespace fwp {
namespace wy {

using namespace s3;
constexpr int C = 16;                   // steps per chunk
constexpr int PC = C + 8;               // pitch of the 16 x 16 operand tiles

template <typename T> __host__ __device__ constexpr int stream_parts() { return sizeof(T) == 4 ? 3 : 1; }

// 16 x 16 block of rows [0, nt) of a stream straight from global memory as C fragments: element (row, col) =
// p[row * sL + col].  `at` = p + g * sL + 2t.
template <typename T>
__device__ __forceinline__ void load_block(float (&x)[2][4], const T* at, long long sL, int nt, int width, bool pairs, int g, int t) {
    if (pairs && nt == C) {
#pragma unroll
        for (int hi = 0; hi < 2; hi++)
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const T* q = at + (hi ? 8 * sL : 0) + 8 * n;
                if constexpr (sizeof(T) == 4) {
                    const float2 v = *reinterpret_cast<const float2*>(q);
                    x[n][2 * hi] = v.x;
                    x[n][2 * hi + 1] = v.y;
                } else {
                    const unsigned v = *reinterpret_cast<const unsigned*>(q);
                    x[n][2 * hi] = __uint_as_float(v << 16);
                    x[n][2 * hi + 1] = __uint_as_float(v & 0xffff0000u);
                }
            }
    } else {
#pragma unroll
        for (int hi = 0; hi < 2; hi++)
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int r = g + 8 * hi, c = 8 * n + 2 * t + i;
                    x[n][2 * hi + i] = r < nt && c < width ? to_f32(at[8 * hi * sL + 8 * n + i]) : 0.f;
                }
    }
}
template <typename T>
__device__ __forceinline__ void store_block(const float (&x)[2][4], T* at, long long sL, int nt, int width, bool pairs, int g, int t) {
    const bool whole = nt == C && width >= 16;
#pragma unroll
    for (int hi = 0; hi < 2; hi++) {
        if (!whole && g + 8 * hi >= nt) continue;
#pragma unroll
        for (int n = 0; n < 2; n++) {
            T* q = at + (hi ? 8 * sL : 0) + 8 * n;
            const float x0 = x[n][2 * hi], x1 = x[n][2 * hi + 1];
            if (whole && pairs) {
                if constexpr (sizeof(T) == 4) *reinterpret_cast<float2*>(q) = make_float2(x0, x1);
                else *reinterpret_cast<__nv_bfloat162*>(q) = __floats2bfloat162_rn(x0, x1);
            } else {
                if (8 * n + 2 * t < width) q[0] = from_f32<T>(x0);
                if (8 * n + 2 * t + 1 < width) q[1] = from_f32<T>(x1);
            }
        }
    }
}
// the same block transposed: element (m, step) = p[step * sL + m].  `at` = p + 2t * sL + g: the four rows a lane touches
// hold 8 consecutive elements each of 8 lanes, whole sectors at any alignment.
template <typename T>
__device__ __forceinline__ void load_block_t(float (&x)[2][4], const T* at, long long sL, int nt, int width, int g, int t) {
    const bool whole = nt == C && width >= 16;
#pragma unroll
    for (int n = 0; n < 2; n++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const T* q = at + (8 * n + i) * sL;
            if (whole) {
                x[n][i] = to_f32(q[0]);
                x[n][2 + i] = to_f32(q[8]);
            } else {
                const bool row = 8 * n + 2 * t + i < nt;
                x[n][i] = row && g < width ? to_f32(q[0]) : 0.f;
                x[n][2 + i] = row && g + 8 < width ? to_f32(q[8]) : 0.f;
            }
        }
}
template <typename T>
__device__ __forceinline__ void store_block_t(const float (&x)[2][4], T* at, long long sL, int nt, int width, int g, int t) {
    if (nt == C && width >= 16) {
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                T* q = at + (8 * n + i) * sL;
                q[0] = from_f32<T>(x[n][i]);
                q[8] = from_f32<T>(x[n][2 + i]);
            }
    } else {
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                if (8 * n + 2 * t + i >= nt) continue;
                T* q = at + (8 * n + i) * sL;
                if (g < width) q[0] = from_f32<T>(x[n][i]);
                if (g + 8 < width) q[8] = from_f32<T>(x[n][2 + i]);
            }
    }
}

// T = (I + A)^-1, A strictly lower triangular in rows of pitch PA floats; lane c (mod 16) finds column c and leaves it
// as row c of the operand tile `Tt` (T^T), its two copies sharing the splitting.  REVERSED: A and T belong to the system
// with its steps in reverse order; the tile gets the inverse in the original order.
template <int PA, bool REVERSED = false>
__device__ __forceinline__ void invert_lower(const float* A, __nv_bfloat16* Tt, int lane) {
    const int c = lane & 15;
    float x[C];
    f2 xp[C / 2];
#pragma unroll
    for (int p = 0; p < C / 2; p++) xp[p] = 0ull;
#pragma unroll
    for (int i = 0; i < C; i++) {
        f2 acc = 0ull;
#pragma unroll
        for (int q = 0; 4 * q < i; q++) {
            const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(A + i * PA + 4 * q);
            acc = ffma2(a.x, xp[2 * q], acc);
            if (4 * q + 2 < i) acc = ffma2(a.y, xp[2 * q + 1], acc);
        }
        x[i] = (i == c ? 1.f : 0.f) - f2_hsum(acc);
        xp[i >> 1] = (i & 1) ? f2_pack(x[i - 1], x[i]) : f2_pack(x[i], 0.f);
    }
    const bool upper = lane >= 16;
    unsigned o[3][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        unsigned s[3];
        if constexpr (REVERSED) split<3>(upper ? x[7 - 2 * j] : x[15 - 2 * j], upper ? x[6 - 2 * j] : x[14 - 2 * j], s);
        else split<3>(upper ? x[2 * j + 8] : x[2 * j], upper ? x[2 * j + 9] : x[2 * j + 1], s);
#pragma unroll
        for (int i = 0; i < 3; i++) o[i][j] = s[i];
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
        *reinterpret_cast<uint4*>(Tt + (i * C + (REVERSED ? C - 1 - c : c)) * PC + (upper ? 8 : 0)) = make_uint4(o[i][0], o[i][1], o[i][2], o[i][3]);
}

}  // namespace wy
}  // namespace fwp
