// mp_mont64.cuh -- arithmetic modulo an odd 64-bit n, and the BPSW primality test built on it,
// for B200 (sm_100a).  Used by the BPSW kernels (mp_bpsw.cu) and the constellation sieve
// (mp_chain.cu).
//
// What is computed follows the reference (paths inside the Mathpub project): the base-2 strong
// probable-prime test (sprp2_64, A350826/a350826.c:618), the strong Lucas test with Selfridge's
// parameters (slprp64 :766, D from selfridge :739) and their conjunction (bpsw :965).  Both
// give exact primality below 2^64, so the verdicts are the reference's.  How it is computed is
// this file's own design, from the published mathematics:
//
//  * A residue is two 32-bit limbs; each product is one PTX block of 32-bit multiply-add carry
//    chains, with the subtracting reduction of the 128-bit product t (R = 2^64): m = t n^-1 mod
//    2^64, then (t - m n) / R = t_hi - hi(m n), exact since the low halves agree, plus n when it
//    borrows.  In and out in [0, n), for any odd n.
//  * Base-2 exponentiation computes 2^-d (the strong test's conditions hold for 2^-d exactly when
//    they hold for 2^d).  In Montgomery form 2^-c is the plain power of two 2^(64 - c), so the
//    ladder starts from the top bits of d with a shift, and R mod n is not needed.  Then five
//    bits at a time: five squarings and one product by 2^-c, c = 0 .. 31, which is a shift left by
//    32 - c and one word of reduction.  Three size classes, each with its squaring:
//    n < 2^62 keeps x below 2^63 without a comparison; n < 2^63 with a subtraction of n when bit 63
//    is set; n >= 2^63 keeps x below 2^64 with a subtraction of n on a carry out.
//  * The squarings form the cross product once and keep the sums at even and odd words apart,
//    because a 64-bit multiply-add (mad.lo.cc directly followed by madc.hi.cc) lands in an aligned
//    pair of registers.  Measured on B200, clocks of an SM per warp: a 64-bit product 1.02, a low
//    32-bit product 0.51; so n < 2^62 has a floor of 8.2 a squaring and takes 9.5 (n >= 2^63: 14.3,
//    much of it carries).  A product with the subtracting reduction takes 13.6, and was run for
//    every bit here before.
//  * Lucas sequences (P = 1, Q = (1 - D)/4) run as the ladder (V_k, V_k+1, Q^k) with
//        V_2k = V_k^2 - 2 Q^k,   V_2k+1 = V_k V_k+1 - P Q^k,
//    the same four products for either exponent bit (the bit only selects operands), so the
//    lanes of a warp never diverge on the exponent.  U_d = 0 (mod n) is read off as
//    2 V_d+1 = P V_d (mod n): D U_k = 2 V_k+1 - P V_k, and gcd(D, n) = 1 when (D/n) = -1.
//  * The Jacobi symbol is the binary (shift and subtract) algorithm after one reduction n mod
//    |D|; the perfect-square check (a square has no D with (D/n) = -1) runs only after 24 values
//    of D have failed.
#pragma once
#include "mp_common.cuh"

// n^-1 mod 2^64 for odd n.  n n = 1 (mod 8), so n is its own inverse to 3 bits; each Newton
// step x (2 - n x) doubles the correct bits: 6, 12, 24, 48, 96.
__host__ __device__ __forceinline__ u64 inv64(u64 n)
{
    u64 x = n;
    x *= 2 - n * x;
    x *= 2 - n * x;
    x *= 2 - n * x;
    x *= 2 - n * x;
    x *= 2 - n * x;
    return x;
}

// the modulus with what the products need: n^-1 mod 2^64 and R mod n
struct Mod64 {
    u64 n;
    u64 ni;        // n^-1 mod 2^64 (the subtracting reduction)
    u64 one;       // R mod n, the residue of 1
};

// ---- products: t = a b (128 bits), then the reduction, result t / 2^64 ----

// the subtracting reduction of t3:t2:t1:t0 (< n R): m = (t1:t0) n^-1 mod 2^64 (i1:i0), then
// (t3:t2) - hi64(m n) + (n if it borrows).  The words of m n below 2^64 equal t1:t0, so only
// their carries into word 2 are formed.
#define MM_REDUCE_SUB                                    \
    "mul.lo.u32     m0, t0, i0;\n\t"                     \
    "mul.hi.u32     m1, t0, i0;\n\t"                     \
    "mad.lo.u32     m1, t0, i1, m1;\n\t"                 \
    "mad.lo.u32     m1, t1, i0, m1;\n\t"                 \
    "mul.hi.u32     v1, m0, n0;\n\t"                     \
    "mad.lo.cc.u32  v1, m0, n1, v1;\n\t"                 \
    "madc.hi.u32    v2, m0, n1, 0;\n\t"                  \
    "mad.lo.cc.u32  v1, m1, n0, v1;\n\t"                 \
    "madc.hi.cc.u32 v2, m1, n0, v2;\n\t"                 \
    "addc.u32       v3, 0, 0;\n\t"                       \
    "mad.lo.cc.u32  v2, m1, n1, v2;\n\t"                 \
    "madc.hi.u32    v3, m1, n1, v3;\n\t"                 \
    "sub.cc.u32     t2, t2, v2;\n\t"                     \
    "subc.cc.u32    t3, t3, v3;\n\t"                     \
    "subc.u32       bw, 0, 0;\n\t"                       \
    "and.b32        k0, n0, bw;\n\t"                     \
    "and.b32        k1, n1, bw;\n\t"                     \
    "add.cc.u32     t2, t2, k0;\n\t"                     \
    "addc.u32       t3, t3, k1;\n\t"

#define MS_REGS ".reg .u32 a0, a1, b0, b1, n0, n1, i0, i1, t0, t1, t2, t3, m0, m1, v1, v2, v3, bw, k0, k1;\n\t"

// a b / R mod n by the subtracting reduction: a, b < n (or a b < n R), result in [0, n)
__device__ __forceinline__ u64 ms_mul(u64 a, u64 b, const Mod64 &M)
{
    u64 r;
    asm("{\n\t" MS_REGS
        "mov.b64 {a0, a1}, %1;\n\t"
        "mov.b64 {b0, b1}, %2;\n\t"
        "mov.b64 {n0, n1}, %3;\n\t"
        "mov.b64 {i0, i1}, %4;\n\t"
        "mul.lo.u32     t0, a0, b0;\n\t"
        "mul.hi.u32     t1, a0, b0;\n\t"
        "mul.lo.u32     t2, a1, b1;\n\t"
        "mul.hi.u32     t3, a1, b1;\n\t"
        "mad.lo.cc.u32  t1, a0, b1, t1;\n\t"
        "madc.hi.cc.u32 t2, a0, b1, t2;\n\t"
        "addc.u32       t3, t3, 0;\n\t"
        "mad.lo.cc.u32  t1, a1, b0, t1;\n\t"
        "madc.hi.cc.u32 t2, a1, b0, t2;\n\t"
        "addc.u32       t3, t3, 0;\n\t"
        MM_REDUCE_SUB
        "mov.b64 %0, {t2, t3};\n\t}"
        : "=l"(r) : "l"(a), "l"(b), "l"(M.n), "l"(M.ni));
    return r;
}

// a^2 / R mod n by the subtracting reduction, a in [0, n)
__device__ __forceinline__ u64 ms_sqr(u64 a, const Mod64 &M)
{
    u64 r;
    asm("{\n\t" MS_REGS
        "mov.b64 {a0, a1}, %1;\n\t"
        "mov.b64 {n0, n1}, %2;\n\t"
        "mov.b64 {i0, i1}, %3;\n\t"
        "mul.lo.u32     t0, a0, a0;\n\t"
        "mul.hi.u32     t1, a0, a0;\n\t"
        "mul.lo.u32     t2, a1, a1;\n\t"
        "mul.hi.u32     t3, a1, a1;\n\t"
        "mad.lo.cc.u32  t1, a0, a1, t1;\n\t"
        "madc.hi.cc.u32 t2, a0, a1, t2;\n\t"
        "addc.u32       t3, t3, 0;\n\t"
        "mad.lo.cc.u32  t1, a0, a1, t1;\n\t"
        "madc.hi.cc.u32 t2, a0, a1, t2;\n\t"
        "addc.u32       t3, t3, 0;\n\t"
        MM_REDUCE_SUB
        "mov.b64 %0, {t2, t3};\n\t}"
        : "=l"(r) : "l"(a), "l"(M.n), "l"(M.ni));
    return r;
}

// x 2^b mod n for b in {0, 1} and x in [0, n): a funnel shift by b (the bit shifted out of 64
// is kept), then one conditional subtraction; result in [0, n)
__device__ __forceinline__ u64 mm_dbl(u64 x, u32 b, const Mod64 &M)
{
    u64 r;
        asm("{\n\t.reg .u32 x0, x1, n0, n1, y0, y1, c, d0, d1, bw;\n\t.reg .pred p;\n\t"
            "mov.b64 {x0, x1}, %1;\n\t"
            "mov.b64 {n0, n1}, %2;\n\t"
            "shl.b32         y0, x0, %3;\n\t"
            "shf.l.clamp.b32 y1, x0, x1, %3;\n\t"
            "shr.b32         c, x1, 31;\n\t"
            "and.b32         c, c, %3;\n\t"
            "sub.cc.u32      d0, y0, n0;\n\t"
            "subc.cc.u32     d1, y1, n1;\n\t"
            "subc.u32        bw, c, 0;\n\t"
            "setp.ne.u32     p, bw, 0;\n\t"
            "selp.u32        y0, y0, d0, p;\n\t"
            "selp.u32        y1, y1, d1, p;\n\t"
            "mov.b64 %0, {y0, y1};\n\t}"
            : "=l"(r) : "l"(x), "l"(M.n), "r"(b));
    return r;
}

// (a + b) mod n and (a - b) mod n for a, b in [0, n)
__device__ __forceinline__ u64 mm_add(u64 a, u64 b, u64 n)
{
    const u64 s = a + b;
    const u64 t = s - n;
    // a + b >= n exactly when the sum wrapped past 2^64 or the difference did not borrow
    return (s < a || s >= n) ? t : s;
}
__device__ __forceinline__ u64 mm_sub(u64 a, u64 b, u64 n)
{
    const u64 d = a - b;
    return a < b ? d + n : d;
}

// the modulus set-up: n^-1 mod 2^64 and R mod n.  R mod n = 2^64 mod n is reached from
// 2^(bitlen(n) - 1) < n by doublings, which are exact.
__device__ __forceinline__ Mod64 mm_setup(u64 n)
{
    Mod64 M;
    M.n = n;
    M.ni = inv64(n);
    const int top = 63 - __clzll((long long)n);
    u64 x = 1ull << top;
    for (int i = top; i < 64; i++) x = mm_dbl(x, 1u, M);
    M.one = x;
    return M;
}

// Montgomery residue of a small signed integer v (|v| < n): |v| R by double-and-add of R mod n
// over the bits of |v|, then negated
__device__ __forceinline__ u64 mm_from_small(i32 v, const Mod64 &M)
{
    const u32 a = v < 0 ? (u32)(-v) : (u32)v;
    u64 r = 0;
    for (int i = 31 - __clz(a | 1u); i >= 0; i--) {
        r = mm_dbl(r, 1u, M);
        if ((a >> i) & 1u) r = mm_add(r, M.one, M.n);
    }
    return (v < 0 && r) ? M.n - r : r;
}

// ---- base-2 strong probable-prime test ----

// size classes of the base-2 ladder: below 2^62 (no corrections), below 2^63, any n
#define SP_LAZY 1
#define SP_MID 2
#define SP_WIDE 3

// x <- x - n when x has bit 63 set
__device__ __forceinline__ void sp_below63(u32 &x0, u32 &x1, u32 n0, u32 n1)
{
    asm("{\n\t.reg .pred p;\n\t"
        "setp.lt.s32    p, %1, 0;\n\t"
        "@p sub.cc.u32  %0, %0, %2;\n\t"
        "@p subc.u32    %1, %1, %3;\n\t}"
        : "+r"(x0), "+r"(x1) : "r"(n0), "r"(n1));
}

// x <- x^2 / R (mod n), np = -n^-1 mod 2^32, by two words of adding reduction.
//   SP_LAZY: x < 2^63, n < 2^62: x^2 / R + n < 2^63, and < 2n once x < 2n
//   SP_MID:  x < 2^63, n < 2^63: x^2 / R + n < 2^62 + n, less n when that has bit 63 set
//   SP_WIDE: any x < 2^64: x^2 / R + n < 2^64 + n, less n when it reaches 2^64
template <int CLS>
__device__ __forceinline__ void sp_sqr(u32 &x0, u32 &x1, u32 n0, u32 n1, u32 np)
{
    if (CLS != SP_WIDE) {
        asm("{\n\t.reg .u32 a0, a1, a2, a3, b1, b2, e1, m;\n\t"
            "shl.b32        e1, %1, 1;\n\t"
            "mul.lo.u32     a0, %0, %0;\n\t"
            "mul.hi.u32     a1, %0, %0;\n\t"
            "mul.lo.u32     b1, %0, e1;\n\t"
            "mul.hi.u32     b2, %0, e1;\n\t"
            "mul.lo.u32     m, a0, %4;\n\t"
            "mad.lo.cc.u32  a0, m, %2, a0;\n\t"
            "madc.hi.cc.u32 a1, m, %2, a1;\n\t"
            "madc.lo.cc.u32 a2, %1, %1, 0;\n\t"
            "madc.hi.u32    a3, %1, %1, 0;\n\t"
            "add.cc.u32     b1, b1, a1;\n\t"
            "addc.u32       b2, b2, 0;\n\t"
            "mad.lo.cc.u32  b1, m, %3, b1;\n\t"
            "madc.hi.cc.u32 b2, m, %3, b2;\n\t"
            "addc.u32       a3, a3, 0;\n\t"
            "mul.lo.u32     m, b1, %4;\n\t"
            "mad.lo.cc.u32  b1, m, %2, b1;\n\t"
            "madc.hi.cc.u32 b2, m, %2, b2;\n\t"
            "addc.u32       a3, a3, 0;\n\t"
            "mad.lo.cc.u32  a2, m, %3, a2;\n\t"
            "madc.hi.u32    a3, m, %3, a3;\n\t"
            "add.cc.u32     %0, a2, b2;\n\t"
            "addc.u32       %1, a3, 0;\n\t}"
            : "+r"(x0), "+r"(x1) : "r"(n0), "r"(n1), "r"(np));
        if (CLS == SP_MID) sp_below63(x0, x1, n0, n1);
    } else {
        asm("{\n\t.reg .u32 a0, a1, a2, a3, b1, b2, k, m;\n\t.reg .pred p;\n\t"
            "mul.lo.u32     a0, %0, %0;\n\t"
            "mul.hi.u32     a1, %0, %0;\n\t"
            "mul.lo.u32     b1, %0, %1;\n\t"
            "mul.hi.u32     b2, %0, %1;\n\t"
            "mul.lo.u32     m, a0, %4;\n\t"
            "mad.lo.cc.u32  a0, m, %2, a0;\n\t"
            "madc.hi.cc.u32 a1, m, %2, a1;\n\t"
            "madc.lo.cc.u32 a2, %1, %1, 0;\n\t"
            "madc.hi.u32    a3, %1, %1, 0;\n\t"
            "mad.lo.cc.u32  b1, %0, %1, b1;\n\t"
            "madc.hi.cc.u32 b2, %0, %1, b2;\n\t"
            "addc.u32       a3, a3, 0;\n\t"                 // x^2 + m n0 < 2^128
            "add.cc.u32     b1, b1, a1;\n\t"
            "addc.cc.u32    b2, b2, 0;\n\t"
            "addc.cc.u32    a3, a3, 0;\n\t"
            "addc.u32       k, 0, 0;\n\t"
            "mad.lo.cc.u32  b1, m, %3, b1;\n\t"
            "madc.hi.cc.u32 b2, m, %3, b2;\n\t"
            "addc.cc.u32    a3, a3, 0;\n\t"
            "addc.u32       k, k, 0;\n\t"
            "mul.lo.u32     m, b1, %4;\n\t"
            "mad.lo.cc.u32  b1, m, %2, b1;\n\t"
            "madc.hi.cc.u32 b2, m, %2, b2;\n\t"
            "addc.cc.u32    a3, a3, 0;\n\t"
            "addc.u32       k, k, 0;\n\t"
            "mad.lo.cc.u32  a2, m, %3, a2;\n\t"
            "madc.hi.cc.u32 a3, m, %3, a3;\n\t"
            "addc.u32       k, k, 0;\n\t"
            "add.cc.u32     %0, a2, b2;\n\t"
            "addc.cc.u32    %1, a3, 0;\n\t"
            "addc.u32       k, k, 0;\n\t"
            "setp.ne.u32    p, k, 0;\n\t"
            "@p sub.cc.u32  %0, %0, %2;\n\t"
            "@p subc.u32    %1, %1, %3;\n\t}"
            : "+r"(x0), "+r"(x1) : "r"(n0), "r"(n1), "r"(np));
    }
}

// x <- (x 2^sh + m n) / 2^32 (mod n), sh in [0, 32]: x itself for 32, else below x / 2 + n; brought
// into the class's range
template <int CLS>
__device__ __forceinline__ void sp_shift(u32 &x0, u32 &x1, u32 sh, u32 n0, u32 n1, u32 np)
{
    u32 k;
    asm("{\n\t.reg .u32 t0, t1, t2, b1, b2, m;\n\t"
        "shl.b32         t0, %0, %6;\n\t"
        "shf.l.clamp.b32 t1, %0, %1, %6;\n\t"
        "shf.l.clamp.b32 t2, %1, 0, %6;\n\t"
        "mul.lo.u32      m, t0, %5;\n\t"
        "mul.lo.u32      b1, m, %4;\n\t"
        "mul.hi.u32      b2, m, %4;\n\t"
        "mad.lo.cc.u32   t0, m, %3, t0;\n\t"
        "madc.hi.cc.u32  t1, m, %3, t1;\n\t"
        "addc.u32        t2, t2, 0;\n\t"                    // below 2^31 + 1
        "add.cc.u32      %0, t1, b1;\n\t"
        "addc.cc.u32     %1, t2, b2;\n\t"
        "addc.u32        %2, 0, 0;\n\t}"
        : "+r"(x0), "+r"(x1), "=r"(k) : "r"(n0), "r"(n1), "r"(np), "r"(sh));
    if (CLS == SP_MID) sp_below63(x0, x1, n0, n1);
    if (CLS == SP_WIDE)
        asm("{\n\t.reg .pred p;\n\t"
            "setp.ne.u32    p, %4, 0;\n\t"
            "@p sub.cc.u32  %0, %0, %2;\n\t"
            "@p subc.u32    %1, %1, %3;\n\t}"
            : "+r"(x0), "+r"(x1) : "r"(n0), "r"(n1), "r"(k));
}

// x / R mod n in [0, n]
__device__ __forceinline__ u64 sp_leave(u32 x0, u32 x1, u32 n0, u32 n1, u32 np)
{
    u32 m = x0 * np;
    u64 c = (u64)m * n0 + x0;
    c = (u64)m * n1 + x1 + (c >> 32);
    const u32 t = (u32)c, u = (u32)(c >> 32);
    m = t * np;
    c = (u64)m * n0 + t;
    return (u64)m * n1 + u + (c >> 32);
}

// -n^-1 mod 2^32
__device__ __forceinline__ u32 sp_ninv(u32 n0)
{
    u32 v = n0;                                             // n0^-1: 3 bits, doubled four times
    v *= 2 - n0 * v;
    v *= 2 - n0 * v;
    v *= 2 - n0 * v;
    v *= 2 - n0 * v;
    return 0u - v;
}

// x = 2^-d (mod n) in Montgomery form
template <int CLS>
__device__ __forceinline__ void sp_ladder(u32 &x0, u32 &x1, u64 d, u64 n, u32 np)
{
    const u32 n0 = (u32)n, n1 = (u32)(n >> 32);
    // w digits of five bits below a top of at most seven: w from the length of n, so that the lanes of
    // a warp, whose d differ in length, walk the same digits.  The top c: 2^-c R is 2^(64 - c) to
    // c = 63, one or two more shifts above
    const int bits = 64 - __clzll((long long)n);
    int w = bits > 8 ? (bits - 4) / 5 : 0;
    while (d >> (5 * w) == 0) w--;
    u32 c = (u32)(d >> (5 * w));
    u64 x = 1ull << (64 - min(c, 63u));
    if (CLS != SP_WIDE && d == 1) x -= n;                   // 2^63, brought below 2^63
    x0 = (u32)x;
    x1 = (u32)(x >> 32);
    for (c -= min(c, 63u); c; c -= min(c, 32u)) sp_shift<CLS>(x0, x1, 32u - min(c, 32u), n0, n1, np);
    while (--w >= 0) {
#pragma unroll
        for (int i = 0; i < 5; i++) sp_sqr<CLS>(x0, x1, n0, n1, np);
        sp_shift<CLS>(x0, x1, 32u - ((u32)(d >> (5 * w)) & 31u), n0, n1, np);
    }
}

// n - 1 = d 2^s with d odd: the strong condition 2^-d = 1, or 2^(-d 2^r) = -1 for some
// 0 <= r < s (mod n).  Odd n > 2 in size class CLS.
template <int CLS>
__device__ __forceinline__ bool spsp2(u64 n)
{
    const u32 n0 = (u32)n, n1 = (u32)(n >> 32), np = sp_ninv(n0);
    const int s = __ffsll((long long)(n - 1)) - 1;
    u32 x0, x1;
    sp_ladder<CLS>(x0, x1, (n - 1) >> s, n, np);
    u64 z = sp_leave(x0, x1, n0, n1, np);
    bool pass = z == 1 || z == n - 1;
    for (int r = 1; r < s && !pass; r++) {
        if (z == 1) break;                                  // 1 before -1: not a strong probable prime
        sp_sqr<CLS>(x0, x1, n0, n1, np);
        z = sp_leave(x0, x1, n0, n1, np);
        pass = z == n - 1;
    }
    return pass;
}

// the test for any odd n > 2, in its size class
__device__ __forceinline__ bool spsp2_u64(u64 n)
{
    return n >> 62 == 0 ? spsp2<SP_LAZY>(n) : n >> 63 == 0 ? spsp2<SP_MID>(n) : spsp2<SP_WIDE>(n);
}

// ---- strong Lucas test ----

// Jacobi symbol (a/m) for odd m > 0 and 0 <= a < m: strip factors 2 of a (each flips the sign
// when m = 3, 5 mod 8), swap by reciprocity when a < m (flip when a = m = 3 mod 4), subtract
__device__ __forceinline__ int jacobi32(u32 a, u32 m)
{
    int t = 1;
    while (a) {
        const int z = __ffs((int)a) - 1;
        a >>= z;
        if ((z & 1) && ((m & 7u) == 3u || (m & 7u) == 5u)) t = -t;
        if (a < m) {
            const u32 x = a;
            a = m;
            m = x;
            if (a & m & 2u) t = -t;
        }
        a -= m;
    }
    return m == 1 ? t : 0;
}

// (D/n) for odd n > |D|, D odd: (-1/n) for the sign, then reciprocity (|D|/n) = +-(n mod |D| / |D|)
__device__ __forceinline__ int jacobi_dn(i32 D, u64 n)
{
    const u32 a = D < 0 ? (u32)(-D) : (u32)D;
    int t = 1;
    if (D < 0 && (n & 3) == 3) t = -t;
    if ((a & 3u) == 3u && (n & 3) == 3) t = -t;
    return t * jacobi32((u32)(n % a), a);
}

// exact test for a perfect square: residue filters mod 64 and 63, then the integer root by
// bits from the top
__device__ __forceinline__ bool is_square64(u64 n)
{
    if (!((0x0202021202030213ull >> (n & 63)) & 1)) return false;
    if (!((0x0402483012450293ull >> (n % 63)) & 1)) return false;
    u64 r = 0;
    for (int b = 31; b >= 0; b--) {
        const u64 c = r | (1ull << b);
        if (c * c <= n) r = c;
    }
    return r * r == n;
}

// Selfridge's method A: the first D of 5, -7, 9, -11, 13, ... with (D/n) = -1.  Returns 0 when
// n is shown composite on the way: some |D| < n shares a factor with n, or n is a perfect
// square (no D exists then).  Odd n, larger than the |D| reached.
__device__ __forceinline__ i32 selfridge_d(u64 n)
{
    for (int k = 0; k < 2048; k++) {
        const i32 a = 5 + 2 * k;
        const i32 D = (k & 1) ? -a : a;
        const int j = jacobi_dn(D, n);
        if (j < 0) return D;
        if (j == 0 && (u64)a != n) return 0;
        if (k == 23 && is_square64(n)) return 0;
    }
    return 0;
}

// strong Lucas probable prime with P = 1, Q = (1 - D)/4 (D = 1 mod 4 here, so Q is exact):
// n + 1 = d 2^s, d odd; U_d = 0, or V_(d 2^r) = 0 for some 0 <= r < s.  Odd n > 2, n < 2^64 - 1.
__device__ __forceinline__ bool lucas_strong(const Mod64 &M, i32 D)
{
    const u64 n = M.n;
    const i32 Q = (1 - D) / 4;
    const u64 q1 = mm_from_small(Q, M);
    const int s = __ffsll((long long)(n + 1)) - 1;
    const u64 d = (n + 1) >> s;
    // k = 1 (d's top bit): V_1 = P = 1, V_2 = P^2 - 2Q, Q^1
    u64 vk = M.one;
    u64 vk1 = mm_sub(M.one, mm_add(q1, q1, n), n);
    u64 qk = q1;
    for (int i = 62 - __clzll((long long)d); i >= 0; i--) {
        const bool b = (d >> i) & 1;
        const u64 w = mm_sub(ms_mul(vk, vk1, M), qk, n);               // V_2k+1
        const u64 qb = ms_mul(qk, b ? q1 : M.one, M);                  // Q^(k+b)
        const u64 sq = ms_sqr(b ? vk1 : vk, M);
        const u64 v2 = mm_sub(sq, mm_add(qb, qb, n), n);               // V_2(k+b)
        qk = ms_mul(qk, qb, M);                                        // Q^(2k+b)
        vk = b ? w : v2;
        vk1 = b ? v2 : w;
    }
    if (vk == 0 || mm_add(vk1, vk1, n) == vk) return true;             // V_d = 0 or U_d = 0
    for (int r = 1; r < s; r++) {
        vk = mm_sub(ms_sqr(vk, M), mm_add(qk, qk, n), n);               // V_(d 2^r)
        if (vk == 0) return true;
        qk = ms_sqr(qk, M);
    }
    return false;
}

// the same test for D = 5 (P = 1, Q = -1), the D of about half of all candidates: Q^k = (-1)^k is
// a sign, so a ladder step takes the two V products only.  From (V_k, V_k+1) with Q^k = sg:
// V_2k+1 = V_k V_k+1 - sg, V_2k = V_k^2 - 2 sg, V_2k+2 = V_k+1^2 + 2 sg (Q^(k+1) = -sg); k's
// parity after the step is the exponent bit.  Then Q^d = -1 (d odd), so V_2d = V_d^2 + 2 and
// V_(d 2^r) = V^2 - 2 for r >= 2.
__device__ __forceinline__ bool lucas_strong_d5(const Mod64 &M)
{
    const u64 n = M.n;
    const int s = __ffsll((long long)(n + 1)) - 1;
    const u64 d = (n + 1) >> s;
    const u64 one = M.one, two = mm_add(one, one, n);
    // k = 1: V_1 = 1, V_2 = 1 + 2 = 3, Q^1 = -1
    u64 vk = one, vk1 = mm_add(two, one, n);
    bool neg = true;                                                   // Q^k = -1
    for (int i = 62 - __clzll((long long)d); i >= 0; i--) {
        const bool b = (d >> i) & 1;
        const u64 p = ms_mul(vk, vk1, M);
        const u64 w = neg ? mm_add(p, one, n) : mm_sub(p, one, n);     // V_2k+1
        const u64 sq = ms_sqr(b ? vk1 : vk, M);
        // V_2k = sq - 2 sg; V_2k+2 = sq + 2 sg: subtract 2 exactly when (sg = +1) != b
        const bool sub2 = (!neg) != b;
        const u64 v2 = sub2 ? mm_sub(sq, two, n) : mm_add(sq, two, n);
        vk = b ? w : v2;
        vk1 = b ? v2 : w;
        neg = b;
    }
    if (vk == 0 || mm_add(vk1, vk1, n) == vk) return true;             // V_d = 0 or U_d = 0
    for (int r = 1; r < s; r++) {
        const u64 sq = ms_sqr(vk, M);
        vk = r == 1 ? mm_add(sq, two, n) : mm_sub(sq, two, n);         // V_(d 2^r)
        if (vk == 0) return true;
    }
    return false;
}

// the Lucas half of BPSW for an odd n > 2 that passed the base-2 test
__device__ __forceinline__ bool lucas_u64(u64 n)
{
    if (n == ~0ull) return false;                                      // 3 | 2^64 - 1
    const i32 D = selfridge_d(n);
    if (!D) return false;
    return lucas_strong(mm_setup(n), D);
}

// primality of an odd n > 2 with no small factor to look for first: the base-2 strong test and
// the strong Lucas test (BPSW; exact below 2^64)
__device__ __forceinline__ bool bpsw_odd(u64 n)
{
    if (n == ~0ull) return false;
    if (!spsp2_u64(n)) return false;
    const i32 D = selfridge_d(n);
    return D && lucas_strong(mm_setup(n), D);
}
