// Trailing updates on the INT8 tensor cores (tcgen05.mma kind::i8, sm_100a):
// products of byte digits, accumulated exactly in 32-bit integers.
//
// The update is F -= W B^T over one panel group's K columns (W = L D, B = L,
// complex). FP64 runs at 37 TFLOP/s on this device, INT8 at over a hundred
// times that, so the FP64 operands are written as fixed-point numbers and those as
// base-256 digits (the error-free splitting of Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication", 2012):
//
//   row i of W:  w_ik 2^(62 - e_i), rounded to an integer, |.| <= 2^62, with
//   2^e_i just above the row's largest component; = sum_p d_p 256^(7 - p),
//   eight digits in [-128, 127]. Rows of B likewise, with exponents of their own.
//
// A product of two digits is at most 2^14, and every product of digits p and q
// belongs to level l = p + q, of weight 256^(14 - l). Level by level the
// products of all K columns are summed in a 32-bit accumulator (below 2^28 for
// K = 512), without any rounding. Levels 0 .. L - 1 are kept. With 2^e_i and
// 2^f_j the exponents of an entry's two rows, its errors are
//   - the operands' rounding: numbers down to 2^-9 of their row's largest are
//     exact, smaller ones off by 2^-63 2^e_i; K 2^-61 2^(e_i + f_j) over a sum;
//   - the dropped levels, seven products of 2^14 at the first of them:
//     K 2^-58 2^(e_i + f_j) (2 x 7.02 x 2^-62 per complex product);
//   - one rounding of the sum and one of the destination.
// All of it is relative to the rows, not to the entry: where the rows' large
// components meet (on the diagonal always) it is below an FP64 chain's
// rounding; where rows graded against one another give products far below
// 2^(e_i + f_j) it is not, and the FP64 arithmetic (aphi_factor_set_fp64_digits)
// keeps each number's own precision. A symmetric scaling by powers of two moves
// the exponents with the rows, so a badly scaled system loses nothing. Over 120
// systems of the cylinder (7^3 to 28^3, 50 Hz to 1 MHz, port and random
// right-hand sides) the solutions' errors against extended-precision ones are
// 0.96 times those of the DMMA form (geometric mean; 0.61 to 1.60), the
// backward errors 0.99 times; over 1,024 systems of the torus with its cut port
// (14^3 to 22^3, 50 Hz to 10 kHz, both formulations) 0.99 +- 0.01 and 0.99.
// Seven digits (2^-54) are enough for the solutions' accuracy but not for the
// smallest pivots, which are what is left of sums of much larger terms: on
// the 32^3 cylinder at 1 MHz the smallest pivot came out 2e-8 off, and 1e-10
// from the FP64 FMA chains' with eight, nearer to the reference's (2.9e-10)
// than theirs (4.0e-10).
//
// FP32 operands (the sweep's factors, which a refinement uses) take four
// digits and four levels: K 2^-29 2^(e_i + f_j) from the operands' rounding
// (2^-31 2^e_i each) and K 2^-27.4 2^(e_i + f_j) from the dropped levels,
// against 2^-22 of each number with the two TF32 pieces they took before. On the 32^3
// sweep's first six frequencies the factors' solves are 3 to 10 times more
// accurate and the refinement needs 3-8 iterations (4-13). Three digits cost
// 8 % less of the tiles' time and one or two iterations more.
//
// The pivots' magnitudes are shared out between the operands (column k of W is
// divided and of B multiplied by 2^h, h half of D_k's exponent), so that the
// columns of both have the scale of a Cholesky factor's and one exponent per
// row serves them all.
//
// Tile: 128 rows x Nc complex columns. B is staged twice per digit, [Br | Bi]
// and [-Bi | Br], so that [Cr | Ci] += Ar [Br | Bi]^T + Ai [-Bi | Br]^T; the
// digits q of B lie back to back, and their levels p + q back to back in
// TMEM, so one MMA takes digit p of A against up to four digits of B
// (N = 256): the tensor core reads each A digit once per N = 256 rather than
// once per 64 columns.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "tc_config.hpp"
#include "tc_update.cuh"

namespace aphi_b200 {

constexpr int kI8FloatShift = 17;  // see i8_combine

// S digits per operand, L levels kept, Nc complex columns per tile, Stages
// operand buffers.
template <int S_, int L_, int Nc_, int Stages_>
struct I8Shape {
    static constexpr int S = S_, L = L_, Nc = Nc_, Stages = Stages_;
    static constexpr int W = 2 * Nc;                       // accumulator columns per level: Cr, Ci
    static constexpr int blockA = S * 2 * kTcM * kI8K;     // one stage of 128 A rows: digits x (re, im)
    static constexpr int imageB = S * W * kI8K;            // one stage of Nc B rows, one image
    static constexpr int blockB = 2 * imageB;              // [Br | Bi] per digit, then [-Bi | Br] per digit
    static constexpr int stage = blockA + blockB;
    static constexpr int extra = 1024;                     // barriers and tile slots
    static constexpr int smem = Stages * stage + extra;
    static constexpr int tmem = 512;                       // columns allocated (L W of them used)
    static_assert(L * W <= tmem && L >= S && L <= 2 * S - 1, "levels must fit TMEM");
    static_assert(smem <= 227 * 1024, "operand buffers exceed shared memory");
};
using I8Fp64 = I8Shape<kI8Digits64, kI8Levels64, kI8Nc64, 2>;
using I8Fp32 = I8Shape<kI8Digits32, kI8Levels32, kI8Nc32, 3>;

// A front's region (R padded rows, nst stages of 32 columns): the A blocks
// [R / 128][nst], the B blocks [R / Nc][nst], then a scale per A row and per
// B row (doubles).
template <class C>
__device__ __forceinline__ long long i8_a_off(int nst, int r, int c) {
    return (static_cast<long long>(r / kTcM) * nst + c) * C::blockA;
}
template <class C>
__device__ __forceinline__ long long i8_b_off(int R, int nst, int r, int c) {
    return static_cast<long long>(R / kTcM) * nst * C::blockA + (static_cast<long long>(r / C::Nc) * nst + c) * C::blockB;
}
template <class C>
__device__ __forceinline__ long long i8_scale_off(int R, int nst) {
    return static_cast<long long>(R / kTcM) * nst * C::blockA + static_cast<long long>(R / C::Nc) * nst * C::blockB;
}

// Row r's 16 bytes of columns 16 h .. of a 32-column stage, in the canonical
// K-major no-swizzle layout (8-row x 16-byte core matrices; the strides of
// smem_desc).
__device__ __forceinline__ uint32_t i8_off(int r, int h) { return (r >> 3) * 256 + h * 128 + (r & 7) * 16; }

// kind::i8 instruction descriptor: S32 accumulators, signed 8-bit A and B,
// K-major, M = 128, N = n.
__device__ __forceinline__ constexpr uint32_t i8_idesc(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(kTcM >> 4) << 24);
}

__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// The MMAs of one stage (32 columns of K). first: the tile's first stage,
// whose products start the accumulators afresh.
template <class C>
__device__ __forceinline__ void i8_issue(uint32_t stage, uint32_t tmem, bool first) {
    const uint32_t B = stage + C::blockA;
    int top = -1;  // highest level written so far in this stage
#pragma unroll
    for (int p = 0; p < C::S; ++p) {
        const int q = C::L - p < C::S ? C::L - p : C::S;  // digits 0 .. q - 1 of B meet digit p of A
#pragma unroll
        for (int im = 0; im < 2; ++im) {
            const uint64_t a = smem_desc(stage + (2 * p + im) * kTcM * kI8K);
            const uint32_t b = B + im * C::imageB;
            // Columns [0, q W) of the stacked B rows, at most 256 at a time;
            // levels above `top` start afresh in the first stage.
            const int split = im == 0 && p > 0 && p + q - 1 > top ? (q - 1) * C::W : q * C::W;
#pragma unroll
            for (int n0 = 0; n0 < C::S * C::W; n0 += 256) {
                if (n0 >= q * C::W) break;
                const int n1 = n0 + 256 < q * C::W ? n0 + 256 : q * C::W;
                const bool fresh0 = first && im == 0 && p == 0;
                if (split < n1 && first) {  // [n0, split) accumulates, [split, n1) is new
                    if (split > n0)
                        mma_i8(tmem + p * C::W + n0, a, smem_desc(b + n0 * kI8K), i8_idesc(split - n0), 1);
                    const int s0 = split > n0 ? split : n0;
                    mma_i8(tmem + p * C::W + s0, a, smem_desc(b + s0 * kI8K), i8_idesc(n1 - s0), 0);
                } else {
                    mma_i8(tmem + p * C::W + n0, a, smem_desc(b + n0 * kI8K), i8_idesc(n1 - n0), fresh0 ? 0u : 1u);
                }
            }
        }
        if (p + q - 1 > top) top = p + q - 1;
    }
}

// 32 lanes x N consecutive columns of TMEM into registers.
__device__ __forceinline__ void tmem_ld(uint32_t taddr, int (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, int (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                 : "r"(taddr));
}
// The operands' arithmetic in the factor's type: bits ordered like the
// magnitude (infinities and NaN on top), biased exponents, powers of two, and
// the nearest integer.
template <class R>
struct I8Real;
template <>
struct I8Real<double> {
    // none: infinities and NaN; least: the smallest exponent told apart;
    // shift: see i8_combine.
    static constexpr int bias = 1023, none = 0x7ff, least = 200, shift = 0;
    static __device__ __forceinline__ int size(double x) { return __double2hiint(x) & 0x7fffffff; }
    static __device__ __forceinline__ int exponent(int size) { return size >> 20; }
    static __device__ __forceinline__ double pow2(int biased) { return __hiloint2double(biased << 20, 0); }
    static __device__ __forceinline__ unsigned long long integer(double x) { return __double2ll_rn(x); }
};
template <>
struct I8Real<float> {
    static constexpr int bias = 127, none = 0xff, least = 30, shift = kI8FloatShift;
    static __device__ __forceinline__ int size(float x) { return __float_as_int(x) & 0x7fffffff; }
    static __device__ __forceinline__ int exponent(int size) { return size >> 23; }
    static __device__ __forceinline__ float pow2(int biased) { return __int_as_float(biased << 23); }
    static __device__ __forceinline__ unsigned integer(float x) { return __float2int_rn(x); }
};

// sum_l a_l 256^(3 - l) of the first four levels as hi 2^16 + lo, exactly and
// in 32-bit steps: the top digits are at most 64, so a_0 is below 2^23, a_1
// below 2^25 and hi below 2^31 for K = 512.
__device__ __forceinline__ void i8_top(const int* a, int& hi, int& lo) {
    hi = (a[0] << 8) + a[1] + (a[2] >> 8);
    lo = ((a[2] & 255) << 8) + a[3];
}

// The levels' sum in units of the last one (float: times 2^(-2 kI8FloatShift),
// so that the rows' scales, larger by 2^kI8FloatShift each, multiply to about
// the size of the product itself and stay within a float's range with it). The
// accumulators are read between
// two tiles' MMAs, so this is on the critical path: the integers become
// doubles by their place in the mantissa of a power of two (minus that power),
// not by conversions, and the work is spread over the integer, multiply and
// FP64 pipes. One rounding (double), or two of parts of the sum (float).
__device__ __forceinline__ double i8_combine(const int (&a)[8]) {
    auto real32 = [](int v) { return __hiloint2double(0x43300000, v ^ 0x80000000) - 4503601774854144.0; };
    auto real51 = [](long long v) { return __longlong_as_double(v + 0x4338000000000000LL) - 6755399441055744.0; };
    int hi, lo;
    i8_top(a, hi, lo);
    // levels 4 .. 7: below 2^51
    const long long low = a[4] * 16777216LL + (a[5] * 65536LL + (a[6] * 256LL + a[7]));
    return fma(fma(real32(hi), 65536.0, real32(lo)), 4294967296.0, real51(low));
}
__device__ __forceinline__ float i8_combine(const int (&a)[4]) {
    constexpr float kUnit = 1.0f / (1LL << (2 * kI8FloatShift));
    int hi, lo;
    i8_top(a, hi, lo);
    return fmaf(__int2float_rn(hi), 65536.0f * kUnit, __int2float_rn(lo) * kUnit);
}

}  // namespace aphi_b200
