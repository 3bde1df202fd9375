// BLS12-381 base field Fp on sm_103a: 12 x 32-bit limbs, Montgomery form with
// R = 2^384.  Because 12 x 32 = 6 x 64, the Montgomery representation (and the
// little-endian byte image) is identical to the reference's 6 x u64 blst_fp
// (bindings/blst_types.h:84, scalar/fields/Fp.h:35-40), so device buffers hold
// caller bytes unchanged.
//
// Multiplication is CIOS Montgomery (Koc, Acar, Kaliski 1996) written with PTX
// carry chains (mad.lo.cc / madc.hi.cc): two accumulators of 64-bit slots, E at
// even and O at odd words, that are merged once at the end of a product.
//
// Values are kept lazily reduced in [0, 2p): 4p < 2^384 / 2, so a product of
// two values below 2p leaves CIOS below 1.41p and the final conditional
// subtraction is skipped.  add/sub reduce modulo 2p.  fp_canon() maps to
// [0, p) for output; fp_is_zero() tests congruence to zero.
#pragma once
#include <cstdint>

namespace catmsm {

struct fp { uint32_t v[12]; };

// p, 2p, R mod p (Montgomery one), R^2 mod p, -p^-1 mod 2^32
#define CATMSM_P0  0xffffaaabu
#define CATMSM_P1  0xb9feffffu
#define CATMSM_P2  0xb153ffffu
#define CATMSM_P3  0x1eabfffeu
#define CATMSM_P4  0xf6b0f624u
#define CATMSM_P5  0x6730d2a0u
#define CATMSM_P6  0xf38512bfu
#define CATMSM_P7  0x64774b84u
#define CATMSM_P8  0x434bacd7u
#define CATMSM_P9  0x4b1ba7b6u
#define CATMSM_P10 0x397fe69au
#define CATMSM_P11 0x1a0111eau
#define CATMSM_N0  0xfffcfffdu

__device__ __constant__ static const uint32_t FP_P[12] = {
    0xffffaaabu, 0xb9feffffu, 0xb153ffffu, 0x1eabfffeu, 0xf6b0f624u, 0x6730d2a0u,
    0xf38512bfu, 0x64774b84u, 0x434bacd7u, 0x4b1ba7b6u, 0x397fe69au, 0x1a0111eau};
__device__ __constant__ static const uint32_t FP_ONE[12] = {
    0x0002fffdu, 0x76090000u, 0xc40c0002u, 0xebf4000bu, 0x53c758bau, 0x5f489857u,
    0x70525745u, 0x77ce5853u, 0xa256ec6du, 0x5c071a97u, 0xfa80e493u, 0x15f65ec3u};

__device__ __forceinline__ void fp_zero(fp& r)
{
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = 0;
}

__device__ __forceinline__ void fp_set_one(fp& r)
{
#pragma unroll
    for (int i = 0; i < 12; i++) r.v[i] = FP_ONE[i];
}

// Carry chains of the Montgomery products.  Both accumulators of a product are
// arrays over absolute word positions: E holds 64-bit slots at even words, O
// at odd words, so the products a_j b_i (word i + j) of one row alternate
// between them and every slot keeps its register pair from row to row.  Row i
// adds its even-j products to A (E for even i, O for odd i) at words i .. i + 11
// with the carry in word i + 12, and its odd-j products to B at words
// i + 1 .. i + 12, which cannot carry out: E + O stays below 2^(32 (i + 13)).
#define CATMSM_CHAIN6(FIRST, LAST, HI) \
    FIRST                              \
    "madc.hi.cc.u32 %1, %13, %19, %1;\n\t"  \
    "madc.lo.cc.u32 %2, %14, %19, %2;\n\t"  \
    "madc.hi.cc.u32 %3, %14, %19, %3;\n\t"  \
    "madc.lo.cc.u32 %4, %15, %19, %4;\n\t"  \
    "madc.hi.cc.u32 %5, %15, %19, %5;\n\t"  \
    "madc.lo.cc.u32 %6, %16, %19, %6;\n\t"  \
    "madc.hi.cc.u32 %7, %16, %19, %7;\n\t"  \
    "madc.lo.cc.u32 %8, %17, %19, %8;\n\t"  \
    "madc.hi.cc.u32 %9, %17, %19, %9;\n\t"  \
    "madc.lo.cc.u32 %10, %18, %19, %10;\n\t" \
    HI LAST
#define CATMSM_FIRST "mad.lo.cc.u32  %0, %13, %19, %0;\n\t"
#define CATMSM_ACC11(w)                                                                              \
    "+r"((w)[0]), "+r"((w)[1]), "+r"((w)[2]), "+r"((w)[3]), "+r"((w)[4]), "+r"((w)[5]), "+r"((w)[6]), \
        "+r"((w)[7]), "+r"((w)[8]), "+r"((w)[9]), "+r"((w)[10])

#define CATMSM_IN6(x) "r"((x)[0]), "r"((x)[2]), "r"((x)[4]), "r"((x)[6]), "r"((x)[8]), "r"((x)[10])

// w[0 .. 11] += (the six x) * b; the carry to w[12]: assigned (New) or added.
template <bool New>
__device__ __forceinline__ void chain_carry(uint32_t* w, const uint32_t* x, uint32_t b)
{
    if (New)
        asm(CATMSM_CHAIN6(CATMSM_FIRST, "addc.u32 %12, 0, 0;", "madc.hi.cc.u32 %11, %18, %19, %11;\n\t")
            : CATMSM_ACC11(w), "+r"(w[11]), "=r"(w[12])
            : CATMSM_IN6(x), "r"(b));
    else
        asm(CATMSM_CHAIN6(CATMSM_FIRST, "addc.u32 %12, %12, 0;", "madc.hi.cc.u32 %11, %18, %19, %11;\n\t")
            : CATMSM_ACC11(w), "+r"(w[11]), "+r"(w[12])
            : CATMSM_IN6(x), "r"(b));
}

// w[0 .. 11] += (the six x) * b without a carry out; w[11] is assigned if Fresh.
template <bool Fresh>
__device__ __forceinline__ void chain_top(uint32_t* w, const uint32_t* x, uint32_t b)
{
    uint32_t unused;
    if (Fresh)
        asm(CATMSM_CHAIN6(CATMSM_FIRST, "mov.u32 %12, 0;", "madc.hi.u32 %11, %18, %19, 0;\n\t")
            : CATMSM_ACC11(w), "=r"(w[11]), "=r"(unused)
            : CATMSM_IN6(x), "r"(b));
    else
        asm(CATMSM_CHAIN6(CATMSM_FIRST, "mov.u32 %12, 0;", "madc.hi.u32 %11, %18, %19, %11;\n\t")
            : CATMSM_ACC11(w), "+r"(w[11]), "=r"(unused)
            : CATMSM_IN6(x), "r"(b));
    (void)unused;
}

// The Montgomery rows: A += m (p_0, p_2, ...) with the carry in its word 12, ...
__device__ __forceinline__ void mont_carry(uint32_t* w, uint32_t m)
{
    asm(CATMSM_CHAIN6(CATMSM_FIRST, "addc.u32 %12, %12, 0;", "madc.hi.cc.u32 %11, %18, %19, %11;\n\t")
        : CATMSM_ACC11(w), "+r"(w[11]), "+r"(w[12])
        : "n"(CATMSM_P0), "n"(CATMSM_P2), "n"(CATMSM_P4), "n"(CATMSM_P6), "n"(CATMSM_P8), "n"(CATMSM_P10), "r"(m));
}

// ... and B += m (p_1, p_3, ...) with the carry of lo_a + lo_b coming in: the
// words of A and B at this row's position add up to a multiple of 2^32, whose
// carry belongs to B's first word.
__device__ __forceinline__ void mont_top(uint32_t* w, uint32_t m, uint32_t lo_a, uint32_t lo_b)
{
    uint32_t dropped;
    asm(CATMSM_CHAIN6("add.cc.u32 %12, %20, %21;\n\tmadc.lo.cc.u32 %0, %13, %19, %0;\n\t", "",
                      "madc.hi.u32 %11, %18, %19, %11;\n\t")
        : CATMSM_ACC11(w), "+r"(w[11]), "=&r"(dropped)
        : "n"(CATMSM_P1), "n"(CATMSM_P3), "n"(CATMSM_P5), "n"(CATMSM_P7), "n"(CATMSM_P9), "n"(CATMSM_P11), "r"(m),
          "r"(lo_a), "r"(lo_b));
    (void)dropped;
}

// Row i's reduction: A, B as above.
__device__ __forceinline__ void mont_row(uint32_t* A, uint32_t* B, int i)
{
    const uint32_t lo_b = i ? B[i] : 0u;
    const uint32_t m = (A[i] + lo_b) * CATMSM_N0;
    mont_carry(A + i, m);
    mont_top(B + i + 1, m, A[i], lo_b);
}

// r = (E + O) >> 384 after the twelve rows
__device__ __forceinline__ void mont_merge(fp& r, const uint32_t* e, const uint32_t* o)
{
    asm("add.cc.u32  %0, %12, %24;\n\t"
        "addc.cc.u32 %1, %13, %25;\n\t"
        "addc.cc.u32 %2, %14, %26;\n\t"
        "addc.cc.u32 %3, %15, %27;\n\t"
        "addc.cc.u32 %4, %16, %28;\n\t"
        "addc.cc.u32 %5, %17, %29;\n\t"
        "addc.cc.u32 %6, %18, %30;\n\t"
        "addc.cc.u32 %7, %19, %31;\n\t"
        "addc.cc.u32 %8, %20, %32;\n\t"
        "addc.cc.u32 %9, %21, %33;\n\t"
        "addc.cc.u32 %10, %22, %34;\n\t"
        "addc.u32    %11, %23, %35;"
        : "=&r"(r.v[0]), "=&r"(r.v[1]), "=&r"(r.v[2]), "=&r"(r.v[3]), "=&r"(r.v[4]), "=&r"(r.v[5]),
          "=&r"(r.v[6]), "=&r"(r.v[7]), "=&r"(r.v[8]), "=&r"(r.v[9]), "=&r"(r.v[10]), "=&r"(r.v[11])
        : "r"(e[12]), "r"(e[13]), "r"(e[14]), "r"(e[15]), "r"(e[16]), "r"(e[17]),
          "r"(e[18]), "r"(e[19]), "r"(e[20]), "r"(e[21]), "r"(e[22]), "r"(e[23]),
          "r"(o[12]), "r"(o[13]), "r"(o[14]), "r"(o[15]), "r"(o[16]), "r"(o[17]),
          "r"(o[18]), "r"(o[19]), "r"(o[20]), "r"(o[21]), "r"(o[22]), "r"(o[23]));
}

// Row 0 of a product: the slots of both accumulators, and A's carry word.
__device__ __forceinline__ void row_first(uint32_t* e, uint32_t* o, const uint32_t* x, uint32_t b)
{
#pragma unroll
    for (int k = 0; k < 6; k++) {
        e[2 * k] = x[2 * k] * b;
        e[2 * k + 1] = __umulhi(x[2 * k], b);
        o[2 * k + 1] = x[2 * k + 1] * b;
        o[2 * k + 2] = __umulhi(x[2 * k + 1], b);
    }
    e[12] = 0;
}

// r = a * b * 2^-384 mod p; inputs in [0, 2p), output in [0, 2p).  The multiply
// pipe bounds it (288 wide multiply-adds at half rate); the accumulators are
// merged once, after the last row, not after every row: 396 instructions
// instead of 490.  Measured on GB300, one function called in a loop: 4 warps per
// scheduler 29.6 -> 30.3 G products/s, 2 warps 28.0 -> 29.1.
__device__ __forceinline__ void fp_mul_impl(fp& r, const fp& a, const fp& b)
{
    uint32_t e[26], o[26];
#pragma unroll
    for (int i = 0; i < 12; i++) {
        uint32_t* A = (i & 1) ? o : e;
        uint32_t* B = (i & 1) ? e : o;
        if (i == 0) {
            row_first(e, o, a.v, b.v[0]);
        } else {
            chain_carry<true>(A + i, a.v, b.v[i]);
            chain_top<true>(B + i + 1, a.v + 1, b.v[i]);
        }
        mont_row(A, B, i);
    }
    mont_merge(r, e, o);
}

// The multiplication is one out-of-line function per translation unit, called
// with its operands and result in registers.  Inlined, a group operation is
// ~10 copies of ~750 instructions and the accumulation loop outgrows the
// instruction cache (ncu: ~2 cycles of no_instruction stall per issue); out of
// line the hot loop is one body plus call sites.  Measured on GB300: the 2^20
// MSM 9.1 -> 8.0 ms, a 2^14 G1 FFT 39 -> 26 ms.  A call costs ~24 moves that the
// compiler puts on the multiply pipe, so a translation unit may inline the
// squaring (CATMSM_INLINE_SQR) and the two-product multiplication
// (CATMSM_INLINE_MUL2), which have few call sites: accumulating mixed additions
// 2.50 -> 2.45 ms (300007-point MSM without affine rounds), a 2^16 FFT 28.9 ->
// 28.3.  Inlining the multiplication as well is slower again (2.59, 33.7 ms),
// and decoding keeps the calls (300000 elements 13.8 -> 14.3 ms inlined) but for
// the loop of fp_pow, which inlines its squaring everywhere (-> 13.6).
static __device__ __noinline__ fp fp_mul_call(const fp a, const fp b)
{
    fp r;
    fp_mul_impl(r, a, b);
    return r;
}

__device__ __forceinline__ void fp_mul(fp& r, const fp& a, const fp& b) { r = fp_mul_call(a, b); }

// r = a^2 * 2^-384 mod p; input in [0, 2p), output in [0, 2p).  The rows of
// fp_mul_impl with the symmetry of a square: row i adds
// a_i * V_i, V_i = a_i 2^(32i) + 2 sum_{j>i} a_j 2^(32j) (a < 2p keeps the top word
// below 2^30, so doubling stays in 12 words), i.e. 12 - i limb products
// instead of 12: 156 product IMAD instead of 288.  Each row adds at most 4p 2^32,
// so the running value stays below 6p < 2^384 and the result below 2p.  Against
// merging E and O after every row, 4 warps per scheduler: 37.4 -> 39.0 G squares/s,
// 2 warps: 35.8 -> 38.3.  The body is the output of gen/gen_fp_sqr.py (in this
// package), checked by a CPU test.
__device__ __forceinline__ void fp_sqr_impl(fp& r, const fp& a)
{
    uint32_t e[26], o[26], d[12];
#pragma unroll
    for (int j = 1; j < 12; j++) d[j] = __funnelshift_l(a.v[j - 1], a.v[j], 1);   // (2a)_j
    {   // row 0
        const uint32_t bi = a.v[0];
        e[0] = a.v[0] * bi;
        e[1] = __umulhi(a.v[0], bi);
        e[2] = d[2] * bi;
        e[3] = __umulhi(d[2], bi);
        e[4] = d[4] * bi;
        e[5] = __umulhi(d[4], bi);
        e[6] = d[6] * bi;
        e[7] = __umulhi(d[6], bi);
        e[8] = d[8] * bi;
        e[9] = __umulhi(d[8], bi);
        e[10] = d[10] * bi;
        e[11] = __umulhi(d[10], bi);
        o[1] = (a.v[1] << 1) * bi;
        o[2] = __umulhi((a.v[1] << 1), bi);
        o[3] = d[3] * bi;
        o[4] = __umulhi(d[3], bi);
        o[5] = d[5] * bi;
        o[6] = __umulhi(d[5], bi);
        o[7] = d[7] * bi;
        o[8] = __umulhi(d[7], bi);
        o[9] = d[9] * bi;
        o[10] = __umulhi(d[9], bi);
        o[11] = d[11] * bi;
        o[12] = __umulhi(d[11], bi);
        e[12] = 0;
        mont_row(e, o, 0);
    }
    {   // row 1
        const uint32_t bi = a.v[1];
        asm("mad.lo.cc.u32  %0, %11, %16, %0;\n\t"
            "madc.hi.cc.u32 %1, %11, %16, %1;\n\t"
            "madc.lo.cc.u32 %2, %12, %16, %2;\n\t"
            "madc.hi.cc.u32 %3, %12, %16, %3;\n\t"
            "madc.lo.cc.u32 %4, %13, %16, %4;\n\t"
            "madc.hi.cc.u32 %5, %13, %16, %5;\n\t"
            "madc.lo.cc.u32 %6, %14, %16, %6;\n\t"
            "madc.hi.cc.u32 %7, %14, %16, %7;\n\t"
            "madc.lo.cc.u32 %8, %15, %16, %8;\n\t"
            "madc.hi.cc.u32 %9, %15, %16, %9;\n\t"
            "addc.u32       %10, 0, 0;"
            : "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11]), "+r"(o[12]), "=&r"(o[13])
            : "r"((a.v[2] << 1)), "r"(d[4]), "r"(d[6]), "r"(d[8]), "r"(d[10]), "r"(bi));
        // e[2..3] += a.v[1] * bi;
        // e[4..5] += d[3] * bi;
        // e[6..7] += d[5] * bi;
        // e[8..9] += d[7] * bi;
        // e[10..11] += d[9] * bi;
        // e[12..13] += d[11] * bi;
        asm("mad.lo.cc.u32  %0, %12, %18, %0;\n\t"
            "madc.hi.cc.u32 %1, %12, %18, %1;\n\t"
            "madc.lo.cc.u32 %2, %13, %18, %2;\n\t"
            "madc.hi.cc.u32 %3, %13, %18, %3;\n\t"
            "madc.lo.cc.u32 %4, %14, %18, %4;\n\t"
            "madc.hi.cc.u32 %5, %14, %18, %5;\n\t"
            "madc.lo.cc.u32 %6, %15, %18, %6;\n\t"
            "madc.hi.cc.u32 %7, %15, %18, %7;\n\t"
            "madc.lo.cc.u32 %8, %16, %18, %8;\n\t"
            "madc.hi.cc.u32 %9, %16, %18, %9;\n\t"
            "madc.lo.cc.u32 %10, %17, %18, %10;\n\t"
            "madc.hi.u32    %11, %17, %18, 0;"
            : "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12]), "=&r"(e[13])
            : "r"(a.v[1]), "r"(d[3]), "r"(d[5]), "r"(d[7]), "r"(d[9]), "r"(d[11]), "r"(bi));
        mont_row(o, e, 1);
    }
    {   // row 2
        const uint32_t bi = a.v[2];
        asm("mad.lo.cc.u32  %0, %11, %16, %0;\n\t"
            "madc.hi.cc.u32 %1, %11, %16, %1;\n\t"
            "madc.lo.cc.u32 %2, %12, %16, %2;\n\t"
            "madc.hi.cc.u32 %3, %12, %16, %3;\n\t"
            "madc.lo.cc.u32 %4, %13, %16, %4;\n\t"
            "madc.hi.cc.u32 %5, %13, %16, %5;\n\t"
            "madc.lo.cc.u32 %6, %14, %16, %6;\n\t"
            "madc.hi.cc.u32 %7, %14, %16, %7;\n\t"
            "madc.lo.cc.u32 %8, %15, %16, %8;\n\t"
            "madc.hi.cc.u32 %9, %15, %16, %9;\n\t"
            "addc.u32       %10, 0, 0;"
            : "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12]), "+r"(e[13]), "=&r"(e[14])
            : "r"(a.v[2]), "r"(d[4]), "r"(d[6]), "r"(d[8]), "r"(d[10]), "r"(bi));
        // o[5..6] += (a.v[3] << 1) * bi;
        // o[7..8] += d[5] * bi;
        // o[9..10] += d[7] * bi;
        // o[11..12] += d[9] * bi;
        // o[13..14] += d[11] * bi;
        asm("mad.lo.cc.u32  %0, %10, %15, %0;\n\t"
            "madc.hi.cc.u32 %1, %10, %15, %1;\n\t"
            "madc.lo.cc.u32 %2, %11, %15, %2;\n\t"
            "madc.hi.cc.u32 %3, %11, %15, %3;\n\t"
            "madc.lo.cc.u32 %4, %12, %15, %4;\n\t"
            "madc.hi.cc.u32 %5, %12, %15, %5;\n\t"
            "madc.lo.cc.u32 %6, %13, %15, %6;\n\t"
            "madc.hi.cc.u32 %7, %13, %15, %7;\n\t"
            "madc.lo.cc.u32 %8, %14, %15, %8;\n\t"
            "madc.hi.u32    %9, %14, %15, 0;"
            : "+r"(o[5]), "+r"(o[6]), "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11]), "+r"(o[12]), "+r"(o[13]), "=&r"(o[14])
            : "r"((a.v[3] << 1)), "r"(d[5]), "r"(d[7]), "r"(d[9]), "r"(d[11]), "r"(bi));
        mont_row(e, o, 2);
    }
    {   // row 3
        const uint32_t bi = a.v[3];
        asm("mad.lo.cc.u32  %0, %9, %13, %0;\n\t"
            "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
            "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
            "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
            "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
            "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
            "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
            "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
            "addc.u32       %8, 0, 0;"
            : "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11]), "+r"(o[12]), "+r"(o[13]), "+r"(o[14]), "=&r"(o[15])
            : "r"((a.v[4] << 1)), "r"(d[6]), "r"(d[8]), "r"(d[10]), "r"(bi));
        // e[6..7] += a.v[3] * bi;
        // e[8..9] += d[5] * bi;
        // e[10..11] += d[7] * bi;
        // e[12..13] += d[9] * bi;
        // e[14..15] += d[11] * bi;
        asm("mad.lo.cc.u32  %0, %10, %15, %0;\n\t"
            "madc.hi.cc.u32 %1, %10, %15, %1;\n\t"
            "madc.lo.cc.u32 %2, %11, %15, %2;\n\t"
            "madc.hi.cc.u32 %3, %11, %15, %3;\n\t"
            "madc.lo.cc.u32 %4, %12, %15, %4;\n\t"
            "madc.hi.cc.u32 %5, %12, %15, %5;\n\t"
            "madc.lo.cc.u32 %6, %13, %15, %6;\n\t"
            "madc.hi.cc.u32 %7, %13, %15, %7;\n\t"
            "madc.lo.cc.u32 %8, %14, %15, %8;\n\t"
            "madc.hi.u32    %9, %14, %15, 0;"
            : "+r"(e[6]), "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12]), "+r"(e[13]), "+r"(e[14]), "=&r"(e[15])
            : "r"(a.v[3]), "r"(d[5]), "r"(d[7]), "r"(d[9]), "r"(d[11]), "r"(bi));
        mont_row(o, e, 3);
    }
    {   // row 4
        const uint32_t bi = a.v[4];
        asm("mad.lo.cc.u32  %0, %9, %13, %0;\n\t"
            "madc.hi.cc.u32 %1, %9, %13, %1;\n\t"
            "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
            "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
            "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
            "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
            "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
            "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
            "addc.u32       %8, 0, 0;"
            : "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12]), "+r"(e[13]), "+r"(e[14]), "+r"(e[15]), "=&r"(e[16])
            : "r"(a.v[4]), "r"(d[6]), "r"(d[8]), "r"(d[10]), "r"(bi));
        // o[9..10] += (a.v[5] << 1) * bi;
        // o[11..12] += d[7] * bi;
        // o[13..14] += d[9] * bi;
        // o[15..16] += d[11] * bi;
        asm("mad.lo.cc.u32  %0, %8, %12, %0;\n\t"
            "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
            "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
            "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
            "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
            "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
            "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
            "madc.hi.u32    %7, %11, %12, 0;"
            : "+r"(o[9]), "+r"(o[10]), "+r"(o[11]), "+r"(o[12]), "+r"(o[13]), "+r"(o[14]), "+r"(o[15]), "=&r"(o[16])
            : "r"((a.v[5] << 1)), "r"(d[7]), "r"(d[9]), "r"(d[11]), "r"(bi));
        mont_row(e, o, 4);
    }
    {   // row 5
        const uint32_t bi = a.v[5];
        asm("mad.lo.cc.u32  %0, %7, %10, %0;\n\t"
            "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
            "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
            "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
            "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
            "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
            "addc.u32       %6, 0, 0;"
            : "+r"(o[11]), "+r"(o[12]), "+r"(o[13]), "+r"(o[14]), "+r"(o[15]), "+r"(o[16]), "=&r"(o[17])
            : "r"((a.v[6] << 1)), "r"(d[8]), "r"(d[10]), "r"(bi));
        // e[10..11] += a.v[5] * bi;
        // e[12..13] += d[7] * bi;
        // e[14..15] += d[9] * bi;
        // e[16..17] += d[11] * bi;
        asm("mad.lo.cc.u32  %0, %8, %12, %0;\n\t"
            "madc.hi.cc.u32 %1, %8, %12, %1;\n\t"
            "madc.lo.cc.u32 %2, %9, %12, %2;\n\t"
            "madc.hi.cc.u32 %3, %9, %12, %3;\n\t"
            "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
            "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
            "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
            "madc.hi.u32    %7, %11, %12, 0;"
            : "+r"(e[10]), "+r"(e[11]), "+r"(e[12]), "+r"(e[13]), "+r"(e[14]), "+r"(e[15]), "+r"(e[16]), "=&r"(e[17])
            : "r"(a.v[5]), "r"(d[7]), "r"(d[9]), "r"(d[11]), "r"(bi));
        mont_row(o, e, 5);
    }
    {   // row 6
        const uint32_t bi = a.v[6];
        asm("mad.lo.cc.u32  %0, %7, %10, %0;\n\t"
            "madc.hi.cc.u32 %1, %7, %10, %1;\n\t"
            "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
            "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
            "madc.lo.cc.u32 %4, %9, %10, %4;\n\t"
            "madc.hi.cc.u32 %5, %9, %10, %5;\n\t"
            "addc.u32       %6, 0, 0;"
            : "+r"(e[12]), "+r"(e[13]), "+r"(e[14]), "+r"(e[15]), "+r"(e[16]), "+r"(e[17]), "=&r"(e[18])
            : "r"(a.v[6]), "r"(d[8]), "r"(d[10]), "r"(bi));
        // o[13..14] += (a.v[7] << 1) * bi;
        // o[15..16] += d[9] * bi;
        // o[17..18] += d[11] * bi;
        asm("mad.lo.cc.u32  %0, %6, %9, %0;\n\t"
            "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
            "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
            "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
            "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
            "madc.hi.u32    %5, %8, %9, 0;"
            : "+r"(o[13]), "+r"(o[14]), "+r"(o[15]), "+r"(o[16]), "+r"(o[17]), "=&r"(o[18])
            : "r"((a.v[7] << 1)), "r"(d[9]), "r"(d[11]), "r"(bi));
        mont_row(e, o, 6);
    }
    {   // row 7
        const uint32_t bi = a.v[7];
        asm("mad.lo.cc.u32  %0, %5, %7, %0;\n\t"
            "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
            "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
            "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
            "addc.u32       %4, 0, 0;"
            : "+r"(o[15]), "+r"(o[16]), "+r"(o[17]), "+r"(o[18]), "=&r"(o[19])
            : "r"((a.v[8] << 1)), "r"(d[10]), "r"(bi));
        // e[14..15] += a.v[7] * bi;
        // e[16..17] += d[9] * bi;
        // e[18..19] += d[11] * bi;
        asm("mad.lo.cc.u32  %0, %6, %9, %0;\n\t"
            "madc.hi.cc.u32 %1, %6, %9, %1;\n\t"
            "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
            "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
            "madc.lo.cc.u32 %4, %8, %9, %4;\n\t"
            "madc.hi.u32    %5, %8, %9, 0;"
            : "+r"(e[14]), "+r"(e[15]), "+r"(e[16]), "+r"(e[17]), "+r"(e[18]), "=&r"(e[19])
            : "r"(a.v[7]), "r"(d[9]), "r"(d[11]), "r"(bi));
        mont_row(o, e, 7);
    }
    {   // row 8
        const uint32_t bi = a.v[8];
        asm("mad.lo.cc.u32  %0, %5, %7, %0;\n\t"
            "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
            "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
            "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
            "addc.u32       %4, 0, 0;"
            : "+r"(e[16]), "+r"(e[17]), "+r"(e[18]), "+r"(e[19]), "=&r"(e[20])
            : "r"(a.v[8]), "r"(d[10]), "r"(bi));
        // o[17..18] += (a.v[9] << 1) * bi;
        // o[19..20] += d[11] * bi;
        asm("mad.lo.cc.u32  %0, %4, %6, %0;\n\t"
            "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
            "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
            "madc.hi.u32    %3, %5, %6, 0;"
            : "+r"(o[17]), "+r"(o[18]), "+r"(o[19]), "=&r"(o[20])
            : "r"((a.v[9] << 1)), "r"(d[11]), "r"(bi));
        mont_row(e, o, 8);
    }
    {   // row 9
        const uint32_t bi = a.v[9];
        asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
            "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
            "addc.u32       %2, 0, 0;"
            : "+r"(o[19]), "+r"(o[20]), "=&r"(o[21])
            : "r"((a.v[10] << 1)), "r"(bi));
        // e[18..19] += a.v[9] * bi;
        // e[20..21] += d[11] * bi;
        asm("mad.lo.cc.u32  %0, %4, %6, %0;\n\t"
            "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
            "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
            "madc.hi.u32    %3, %5, %6, 0;"
            : "+r"(e[18]), "+r"(e[19]), "+r"(e[20]), "=&r"(e[21])
            : "r"(a.v[9]), "r"(d[11]), "r"(bi));
        mont_row(o, e, 9);
    }
    {   // row 10
        const uint32_t bi = a.v[10];
        asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
            "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
            "addc.u32       %2, 0, 0;"
            : "+r"(e[20]), "+r"(e[21]), "=&r"(e[22])
            : "r"(a.v[10]), "r"(bi));
        // o[21..22] += (a.v[11] << 1) * bi;
        asm("mad.lo.cc.u32  %0, %2, %3, %0;\n\t"
            "madc.hi.u32    %1, %2, %3, 0;"
            : "+r"(o[21]), "=&r"(o[22])
            : "r"((a.v[11] << 1)), "r"(bi));
        mont_row(e, o, 10);
    }
    {   // row 11
        const uint32_t bi = a.v[11];
        o[23] = 0;
        // e[22..23] += a.v[11] * bi;
        asm("mad.lo.cc.u32  %0, %2, %3, %0;\n\t"
            "madc.hi.u32    %1, %2, %3, 0;"
            : "+r"(e[22]), "=&r"(e[23])
            : "r"(a.v[11]), "r"(bi));
        mont_row(o, e, 11);
    }
    mont_merge(r, e, o);
}

static __device__ __noinline__ fp fp_sqr_call(const fp a)
{
    fp r;
    fp_sqr_impl(r, a);
    return r;
}

__device__ __forceinline__ void fp_sqr_inline(fp& r, const fp& a)
{
    fp t;
    fp_sqr_impl(t, a);
    r = t;
}

__device__ __forceinline__ void fp_sqr(fp& r, const fp& a)
{
#ifdef CATMSM_INLINE_SQR
    fp_sqr_inline(r, a);
#else
    r = fp_sqr_call(a);
#endif
}

// r = (a * b + c * d) * 2^-384 mod p; inputs in [0, 2p), output in [0, 2p).
// The rows of fp_mul_impl with both products added in each row
// before its single Montgomery reduction (876 IMAD against 2 x 588).  Each
// step adds at most 4p 2^32, so the running value stays below 6p < 2^384,
// and a b + c d < 8p^2 < p 2^384 leaves the result below 1.82p.
__device__ __forceinline__ void fp_mul2_impl(fp& r, const fp& a, const fp& b, const fp& c, const fp& d)
{
    uint32_t e[26], o[26];
#pragma unroll
    for (int i = 0; i < 12; i++) {
        uint32_t* A = (i & 1) ? o : e;
        uint32_t* B = (i & 1) ? e : o;
        if (i == 0) {
            row_first(e, o, a.v, b.v[0]);
        } else {
            chain_carry<true>(A + i, a.v, b.v[i]);
            chain_top<true>(B + i + 1, a.v + 1, b.v[i]);
        }
        chain_carry<false>(A + i, c.v, d.v[i]);
        chain_top<false>(B + i + 1, c.v + 1, d.v[i]);
        mont_row(A, B, i);
    }
    mont_merge(r, e, o);
}

static __device__ __noinline__ fp fp_mul2_call(const fp a, const fp b, const fp c, const fp d)
{
    fp r;
    fp_mul2_impl(r, a, b, c, d);
    return r;
}

// r = a * b + c * d (Montgomery), one reduction
__device__ __forceinline__ void fp_mul2(fp& r, const fp& a, const fp& b, const fp& c, const fp& d)
{
#ifdef CATMSM_INLINE_MUL2
    fp t;
    fp_mul2_impl(t, a, b, c, d);
    r = t;
#else
    r = fp_mul2_call(a, b, c, d);
#endif
}

// r = a + b mod 2p (inputs < 2p)
__device__ __forceinline__ void fp_add(fp& r, const fp& a, const fp& b)
{
    uint32_t s[12], d[12], borrow;
    asm("add.cc.u32  %0, %12, %24;\n\t"
        "addc.cc.u32 %1, %13, %25;\n\t"
        "addc.cc.u32 %2, %14, %26;\n\t"
        "addc.cc.u32 %3, %15, %27;\n\t"
        "addc.cc.u32 %4, %16, %28;\n\t"
        "addc.cc.u32 %5, %17, %29;\n\t"
        "addc.cc.u32 %6, %18, %30;\n\t"
        "addc.cc.u32 %7, %19, %31;\n\t"
        "addc.cc.u32 %8, %20, %32;\n\t"
        "addc.cc.u32 %9, %21, %33;\n\t"
        "addc.cc.u32 %10, %22, %34;\n\t"
        "addc.u32    %11, %23, %35;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]),
          "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
          "r"(a.v[6]), "r"(a.v[7]), "r"(a.v[8]), "r"(a.v[9]), "r"(a.v[10]), "r"(a.v[11]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
          "r"(b.v[6]), "r"(b.v[7]), "r"(b.v[8]), "r"(b.v[9]), "r"(b.v[10]), "r"(b.v[11]));
    asm("sub.cc.u32  %0, %13, 0xffff5556;\n\t"
        "subc.cc.u32 %1, %14, 0x73fdffff;\n\t"
        "subc.cc.u32 %2, %15, 0x62a7ffff;\n\t"
        "subc.cc.u32 %3, %16, 0x3d57fffd;\n\t"
        "subc.cc.u32 %4, %17, 0xed61ec48;\n\t"
        "subc.cc.u32 %5, %18, 0xce61a541;\n\t"
        "subc.cc.u32 %6, %19, 0xe70a257e;\n\t"
        "subc.cc.u32 %7, %20, 0xc8ee9709;\n\t"
        "subc.cc.u32 %8, %21, 0x869759ae;\n\t"
        "subc.cc.u32 %9, %22, 0x96374f6c;\n\t"
        "subc.cc.u32 %10, %23, 0x72ffcd34;\n\t"
        "subc.cc.u32 %11, %24, 0x340223d4;\n\t"
        "subc.u32    %12, 0, 0;"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]),
          "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]),
          "=r"(borrow)
        : "r"(s[0]), "r"(s[1]), "r"(s[2]), "r"(s[3]), "r"(s[4]), "r"(s[5]),
          "r"(s[6]), "r"(s[7]), "r"(s[8]), "r"(s[9]), "r"(s[10]), "r"(s[11]));
    // borrow == 0xffffffff iff s < 2p
#pragma unroll
    for (int k = 0; k < 12; k++) r.v[k] = borrow ? s[k] : d[k];
}

// r = a - b mod 2p (inputs < 2p)
__device__ __forceinline__ void fp_sub(fp& r, const fp& a, const fp& b)
{
    uint32_t d[12], s[12], borrow;
    asm("sub.cc.u32  %0, %13, %25;\n\t"
        "subc.cc.u32 %1, %14, %26;\n\t"
        "subc.cc.u32 %2, %15, %27;\n\t"
        "subc.cc.u32 %3, %16, %28;\n\t"
        "subc.cc.u32 %4, %17, %29;\n\t"
        "subc.cc.u32 %5, %18, %30;\n\t"
        "subc.cc.u32 %6, %19, %31;\n\t"
        "subc.cc.u32 %7, %20, %32;\n\t"
        "subc.cc.u32 %8, %21, %33;\n\t"
        "subc.cc.u32 %9, %22, %34;\n\t"
        "subc.cc.u32 %10, %23, %35;\n\t"
        "subc.cc.u32 %11, %24, %36;\n\t"
        "subc.u32    %12, 0, 0;"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]),
          "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]),
          "=r"(borrow)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
          "r"(a.v[6]), "r"(a.v[7]), "r"(a.v[8]), "r"(a.v[9]), "r"(a.v[10]), "r"(a.v[11]),
          "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]),
          "r"(b.v[6]), "r"(b.v[7]), "r"(b.v[8]), "r"(b.v[9]), "r"(b.v[10]), "r"(b.v[11]));
    asm("add.cc.u32  %0, %12, 0xffff5556;\n\t"
        "addc.cc.u32 %1, %13, 0x73fdffff;\n\t"
        "addc.cc.u32 %2, %14, 0x62a7ffff;\n\t"
        "addc.cc.u32 %3, %15, 0x3d57fffd;\n\t"
        "addc.cc.u32 %4, %16, 0xed61ec48;\n\t"
        "addc.cc.u32 %5, %17, 0xce61a541;\n\t"
        "addc.cc.u32 %6, %18, 0xe70a257e;\n\t"
        "addc.cc.u32 %7, %19, 0xc8ee9709;\n\t"
        "addc.cc.u32 %8, %20, 0x869759ae;\n\t"
        "addc.cc.u32 %9, %21, 0x96374f6c;\n\t"
        "addc.cc.u32 %10, %22, 0x72ffcd34;\n\t"
        "addc.u32    %11, %23, 0x340223d4;"
        : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]),
          "=r"(s[6]), "=r"(s[7]), "=r"(s[8]), "=r"(s[9]), "=r"(s[10]), "=r"(s[11])
        : "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]),
          "r"(d[6]), "r"(d[7]), "r"(d[8]), "r"(d[9]), "r"(d[10]), "r"(d[11]));
#pragma unroll
    for (int k = 0; k < 12; k++) r.v[k] = borrow ? s[k] : d[k];
}

__device__ __forceinline__ void fp_neg(fp& r, const fp& a)
{
    fp z;
    fp_zero(z);
    fp_sub(r, z, a);
}

// Map [0, 2p) to [0, p).
__device__ __forceinline__ void fp_canon(fp& r, const fp& a)
{
    uint32_t d[12], borrow;
    asm("sub.cc.u32  %0, %13, 0xffffaaab;\n\t"
        "subc.cc.u32 %1, %14, 0xb9feffff;\n\t"
        "subc.cc.u32 %2, %15, 0xb153ffff;\n\t"
        "subc.cc.u32 %3, %16, 0x1eabfffe;\n\t"
        "subc.cc.u32 %4, %17, 0xf6b0f624;\n\t"
        "subc.cc.u32 %5, %18, 0x6730d2a0;\n\t"
        "subc.cc.u32 %6, %19, 0xf38512bf;\n\t"
        "subc.cc.u32 %7, %20, 0x64774b84;\n\t"
        "subc.cc.u32 %8, %21, 0x434bacd7;\n\t"
        "subc.cc.u32 %9, %22, 0x4b1ba7b6;\n\t"
        "subc.cc.u32 %10, %23, 0x397fe69a;\n\t"
        "subc.cc.u32 %11, %24, 0x1a0111ea;\n\t"
        "subc.u32    %12, 0, 0;"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]),
          "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]),
          "=r"(borrow)
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
          "r"(a.v[6]), "r"(a.v[7]), "r"(a.v[8]), "r"(a.v[9]), "r"(a.v[10]), "r"(a.v[11]));
#pragma unroll
    for (int k = 0; k < 12; k++) r.v[k] = borrow ? a.v[k] : d[k];
}

// a == 0 mod p, for a in [0, 2p): a == 0 or a == p
__device__ __forceinline__ bool fp_is_zero(const fp& a)
{
    uint32_t z = 0, q = 0;
#pragma unroll
    for (int k = 0; k < 12; k++) {
        z |= a.v[k];
        q |= a.v[k] ^ FP_P[k];
    }
    return z == 0 || q == 0;
}

// exact (bitwise) zero test, for encodings where zero means "absent"
__device__ __forceinline__ bool fp_is_zero_raw(const fp& a)
{
    uint32_t z = 0;
#pragma unroll
    for (int k = 0; k < 12; k++) z |= a.v[k];
    return z == 0;
}

__device__ __forceinline__ void fp_dbl(fp& r, const fp& a) { fp_add(r, a, a); }

// r = a^e for a public exponent e > 0 given as 12 little-endian words: sliding
// windows of five bits over the odd powers a, a^3, ..., a^31 (~380 squarings and
// ~80 multiplications for a 381-bit e; bit by bit it is ~190 multiplications).
// The exponent is the same for every lane, so the windows do not diverge.
__device__ __forceinline__ void fp_pow(fp& r, const fp& a, const uint32_t* e)
{
    fp T[16], acc;
    T[0] = a;
    fp_sqr(acc, a);
#pragma unroll 1
    for (int i = 1; i < 16; i++) fp_mul(T[i], T[i - 1], acc);
    bool started = false;
    int i = 383;
    while (i >= 0) {
        if (!((e[i >> 5] >> (i & 31)) & 1)) {
            if (started) fp_sqr_inline(acc, acc);
            i--;
            continue;
        }
        int l = i < 4 ? 0 : i - 4;                    // the window: bits i .. l, l the lowest set bit in reach
        while (!((e[l >> 5] >> (l & 31)) & 1)) l++;
        uint32_t w = 0;
        for (int b = i; b >= l; b--) w = (w << 1) | ((e[b >> 5] >> (b & 31)) & 1);
        if (started) {
#pragma unroll 1
            for (int b = i; b >= l; b--) fp_sqr_inline(acc, acc);
            fp_mul(acc, acc, T[w >> 1]);
        } else {
            acc = T[w >> 1];
            started = true;
        }
        i = l - 1;
    }
    r = acc;
}

// r = a^(p-2) = a^-1 (Fermat); zero maps to zero
__device__ __forceinline__ void fp_inv(fp& r, const fp& a)
{
    uint32_t e[12];
#pragma unroll
    for (int k = 0; k < 12; k++) e[k] = FP_P[k];
    e[0] -= 2;
    fp_pow(r, a, e);
}

}  // namespace catmsm
