// fp32 products on the bf16 tensor pipe (warp-level mma, sm_100a).
//
// A float is the exact sum of three bf16 numbers (8 significand bits each, 24 together, same exponent range), so a
// product of two floats is the sum of nine bf16 products, all exact in the fp32 accumulator.  The three smallest
// (middle x low, low x middle, low x low) are below 2^-24 of the product and are left out, like the rounding of an fp32
// multiply; six mma.m16n8k16 per tile remain.  (G. Henry, P. Tang, A. Heinecke, "Leveraging the bfloat16 artificial
// intelligence datatype for higher-precision computations", ARITH 2019.)  Measured on B200 per SM: one such mma every 2.06 cycles, i.e. 166
// fp32-accurate multiply-adds per cycle against 128 on the fp32 pipe -- and the operands come from registers as
// fragments instead of one shared-memory broadcast per two packed multiply-adds, which is what bounds the fp32 form.
// The tensor pipe truncates when it accumulates, so sums that run through a whole sequence are kept outside: every
// product starts from zero, smallest terms first, and is added to the running fp32 value with a rounded add (H. Ootomo,
// R. Yokota, "Recovering single precision accuracy from tensor cores while surpassing the FP32 theoretical peak
// performance", 2022).
//
// Fragments of mma.m16n8k16 (lane = 4 g + t): A holds rows g, g+8 and columns 2t, 2t+1, 2t+8, 2t+9; B rows (k)
// 2t, 2t+1, 2t+8, 2t+9 of column g; C rows g, g+8 and columns 2t, 2t+1.  So the C fragments of a 16 x 16 matrix Z, packed
// in pairs, are the A fragment of Z and the two B fragments of Z^T without any exchange between lanes.
#pragma once
#include "fwp_core.cuh"

namespace fwp {
namespace s3 {

// two floats -> packed pairs of their three parts, by truncation: every remainder is exact
__device__ __forceinline__ f2 fsub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
template <int NP>
__device__ __forceinline__ void split(float x0, float x1, unsigned (&o)[NP]) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
        const unsigned u0 = __float_as_uint(x0), u1 = __float_as_uint(x1);
        o[i] = __byte_perm(u0, u1, 0x7632);
        if (i + 1 < NP) f2_unpack(fsub2(f2_pack(x0, x1), f2_pack(__uint_as_float(u0 & 0xffff0000u), __uint_as_float(u1 & 0xffff0000u))), x0, x1);
    }
}

__device__ __forceinline__ void mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// the same with a zero accumulator (no registers to clear)
__device__ __forceinline__ void mma_first(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// 16 x 16 operand in NP parts, four registers each: as A fragments, or as the B fragments of two column tiles
template <int NP>
struct Frag {
    unsigned r[NP][4];
};

// the C fragments of a 16 x 16 matrix (two column tiles) as an operand
template <int NP>
__device__ __forceinline__ void from_c(Frag<NP>& f, const float (&c0)[4], const float (&c1)[4]) {
    unsigned o[NP];
    split<NP>(c0[0], c0[1], o);
#pragma unroll
    for (int i = 0; i < NP; i++) f.r[i][0] = o[i];
    split<NP>(c0[2], c0[3], o);
#pragma unroll
    for (int i = 0; i < NP; i++) f.r[i][1] = o[i];
    split<NP>(c1[0], c1[1], o);
#pragma unroll
    for (int i = 0; i < NP; i++) f.r[i][2] = o[i];
    split<NP>(c1[2], c1[3], o);
#pragma unroll
    for (int i = 0; i < NP; i++) f.r[i][3] = o[i];
}

// How a Frag serves as the right operand: of the transpose of a matrix read by rows (column tile n: registers n, n + 2),
// or of a matrix read with the transposing load (column tile n: registers 2n, 2n + 1).
enum Right { BY_ROWS, BY_COLS };

// c[n] = A * B for the two column tiles n, kept terms in ascending order of size
template <Right R, int NA, int NB>
__device__ __forceinline__ void product(float (&c)[2][4], const Frag<NA>& a, const Frag<NB>& b) {
#pragma unroll
    for (int order = 2; order >= 0; order--)
#pragma unroll
        for (int i = NA - 1; i >= 0; i--) {
            const int j = order - i;
            if (j < 0 || j >= NB) continue;
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const unsigned b0 = R == BY_ROWS ? b.r[j][n] : b.r[j][2 * n], b1 = R == BY_ROWS ? b.r[j][n + 2] : b.r[j][2 * n + 1];
                // the first kept term: the smallest left part that pairs with a right part at this order
                if (order == (NA - 1 < 2 ? (NA - 1 + NB - 1 < 2 ? NA - 1 + NB - 1 : 2) : 2) && i == NA - 1) mma_first(c[n], a.r[i], b0, b1);
                else mma(c[n], a.r[i], b0, b1);
            }
        }
}

// Operand tiles in shared memory: NP parts of 16 rows x P bf16 (P = columns + 8: eight rows fall on eight different
// groups of four banks).  A lane's address inside a 16 x 16 block, for all four forms of access:
__device__ __forceinline__ int lane_at(int lane, int P) { return ((lane & 7) + ((lane >> 3) & 1) * 8) * P + (lane >> 4) * 8; }

__device__ __forceinline__ void stm(unsigned addr, const unsigned (&r)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void ldm(unsigned addr, unsigned (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldm_t(unsigned addr, unsigned (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stm_t(unsigned addr, const unsigned (&r)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ unsigned transpose8(unsigned x) {        // an 8 x 8 block across the warp
    unsigned r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
    return r;
}
// `addr` is this lane's address of the block in part 0, `part` the bytes between parts
template <int NP>
__device__ __forceinline__ void store(unsigned addr, int part, const Frag<NP>& f) {
#pragma unroll
    for (int i = 0; i < NP; i++) stm(addr + i * part, f.r[i]);
}
template <int NP>
__device__ __forceinline__ void load_rows(Frag<NP>& f, unsigned addr, int part) {
#pragma unroll
    for (int i = 0; i < NP; i++) ldm(addr + i * part, f.r[i]);
}
template <int NP>
__device__ __forceinline__ void load_cols(Frag<NP>& f, unsigned addr, int part) {
#pragma unroll
    for (int i = 0; i < NP; i++) ldm_t(addr + i * part, f.r[i]);
}

// stores the transpose: registers 1 and 2 change places with the blocks they hold
template <int NP>
__device__ __forceinline__ void store_t(unsigned addr, int part, const Frag<NP>& f) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
        const unsigned r[4] = {f.r[i][0], f.r[i][2], f.r[i][1], f.r[i][3]};
        stm_t(addr + i * part, r);
    }
}
// left operand: the transpose of the tile's block
template <int NP>
__device__ __forceinline__ void load_left_t(Frag<NP>& f, unsigned addr, int part) {
#pragma unroll
    for (int i = 0; i < NP; i++) {
        unsigned r[4];
        ldm_t(addr + i * part, r);
        f.r[i][0] = r[0];
        f.r[i][1] = r[2];
        f.r[i][2] = r[1];
        f.r[i][3] = r[3];
    }
}

// A Frag read by rows, read the other way: as left operand of the transpose, or as BY_COLS right operand
template <int NP>
__device__ __forceinline__ Frag<NP> left_of_transpose(const Frag<NP>& f) {
    Frag<NP> o;
#pragma unroll
    for (int i = 0; i < NP; i++) {
        o.r[i][0] = transpose8(f.r[i][0]);
        o.r[i][1] = transpose8(f.r[i][2]);
        o.r[i][2] = transpose8(f.r[i][1]);
        o.r[i][3] = transpose8(f.r[i][3]);
    }
    return o;
}
template <int NP>
__device__ __forceinline__ Frag<NP> by_cols(const Frag<NP>& f) {
    Frag<NP> o;
#pragma unroll
    for (int i = 0; i < NP; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) o.r[i][j] = transpose8(f.r[i][j]);
    return o;
}
// x += A B, the product formed from zero
__device__ __forceinline__ void add_to(float (&x)[2][4], const float (&d)[2][4]) {
#pragma unroll
    for (int i = 0; i < 8; i++) x[i >> 2][i & 3] += d[i >> 2][i & 3];
}
template <Right R, int NA, int NB>
__device__ __forceinline__ void add_product(float (&x)[2][4], const Frag<NA>& a, const Frag<NB>& b) {
    float d[2][4] = {};
    product<R>(d, a, b);
    add_to(x, d);
}

// the k-th of a sum of products
template <Right R, int NA, int NB>
__device__ __forceinline__ void sum_product(int k, float (&x)[2][4], const Frag<NA>& a, const Frag<NB>& b) {
    if (k == 0) product<R>(x, a, b);
    else add_product<R>(x, a, b);
}

}  // namespace s3
}  // namespace fwp
