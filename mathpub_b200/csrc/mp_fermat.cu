// mp_fermat.cu -- Fermat quotients q_p(2) = (2^(p-1) mod p^2 - 1) / p on B200 (sm_100a).
//
// Reference (paths inside the Mathpub project): pctx_init / msqr / redc
// A001220/wieferich.c:546-645 (Montgomery arithmetic mod N = p^2 with R = 2^128, p^-1 by
// Newton from (3p) xor 2), fermat_quotient :939 (q = (r - 1) p^-1 mod 2^64), finish_lanes
// :1051-1075 (Fermat's little theorem check q < p, checksum mix64(q ^ p * GOLD), symmetric
// residue A).
//
// The device form keeps the same mathematics with a different number layout and exponent: N = p^2
// is held in K 32-bit limbs (K = 3, R = 2^96, for p < 2^47; K = 4, R = 2^128, for p < 2^63).
//
//  * The ladder computes 2^-(p-1), not 2^(p-1): in Montgomery form 2^-c is the plain power of two
//    2^(32K - c), so the ladder starts from the exponent's top six bits with a shift, and neither
//    R mod N nor the first six squarings are needed.  2^-(p-1) = 1 + q'p (mod p^2) exactly when
//    2^(p-1) = 1 + qp, with q = -q' (mod p).
//  * Five exponent bits at a time: five squarings, then x <- x 2^-c for a digit c = 1 .. 32, which
//    is a shift left by 32 - c and one word of Montgomery reduction.  Digits 1 .. 32 instead of
//    0 .. 31 are reached by taking 1 from every digit position beforehand (p - 1 - off).
//  * Values stay in [0, 2^(32K-1)) without a comparison: x -> (x^2 + mN) / R < x^2 / R + N, and
//    both terms are below 2^(32K-2).  Leaving Montgomery form gives the residue in [0, N].
//  * What bounds it is the multiply pipe.  Measured on B200, clocks of an SM per warp instruction:
//    32-bit low product 0.51, high product 1.0, 64-bit product with or without accumulation and
//    carry 1.02, an add with carry about 0.4.  So a product of two limbs is one 64-bit
//    multiply-add (mad.lo.cc directly followed by madc.hi.cc), and a squaring forms each cross
//    product once: 18 products at K = 3, a floor of 16.8 clocks; this form takes 17.8 (K = 4:
//    35.2 against a floor of 28.5).  Low and high halves in separate carry chains took 57
//    low-product units (29 clocks).  Sums at even and odd limb positions are kept apart until the
//    end: the pair of registers a 64-bit product lands in is aligned, and sharing one set of sums
//    between even and odd positions cost moves (23.3 clocks at K = 3, 43.4 at K = 4).
#include "mp_common.cuh"

// x <- x^2 / R (mod N): see the header for the bounds; np = -N^-1 mod 2^32
template <int K>
__device__ __forceinline__ void msqr(u32 (&x)[K], const u32 (&n)[K], u32 np);

// a0 .. hold the sums at even limb positions, b1 .. those at odd ones; a word of reduction adds m N
// with m = (lowest word) np, and the word it does not clear joins the other set.  Products that
// start a pair of sums take the carry below them (their sum cannot overflow).
template <>
__device__ __forceinline__ void msqr<3>(u32 (&x)[3], const u32 (&n)[3], u32 np)
{
    asm("{\n\t.reg .u32 a0, a1, a2, a3, a4, a5, b1, b2, b3, b4, b5, e1, e2, f2, m;\n\t"
        "shl.b32         e1, %1, 1;\n\t"                   // 2 (x1, x2) = (e1, e2), 2 x2 = f2
        "shf.l.wrap.b32  e2, %1, %2, 1;\n\t"
        "shl.b32         f2, %2, 1;\n\t"
        "mul.lo.u32      a0, %0, %0;\n\t"
        "mul.hi.u32      a1, %0, %0;\n\t"
        "mul.lo.u32      a2, %1, %1;\n\t"
        "mul.hi.u32      a3, %1, %1;\n\t"
        "mad.lo.cc.u32   a2, %0, e2, a2;\n\t"
        "madc.hi.cc.u32  a3, %0, e2, a3;\n\t"
        "madc.lo.cc.u32  a4, %2, %2, 0;\n\t"
        "madc.hi.u32     a5, %2, %2, 0;\n\t"
        "mul.lo.u32      b1, %0, e1;\n\t"
        "mul.hi.u32      b2, %0, e1;\n\t"
        "mul.lo.u32      m, a0, %6;\n\t"                   // word 0
        "mad.lo.cc.u32   b1, m, %4, b1;\n\t"
        "madc.hi.cc.u32  b2, m, %4, b2;\n\t"
        "madc.lo.cc.u32  b3, %1, f2, 0;\n\t"
        "madc.hi.u32     b4, %1, f2, 0;\n\t"
        "mad.lo.cc.u32   a0, m, %3, a0;\n\t"
        "madc.hi.cc.u32  a1, m, %3, a1;\n\t"
        "madc.lo.cc.u32  a2, m, %5, a2;\n\t"
        "madc.hi.cc.u32  a3, m, %5, a3;\n\t"
        "addc.cc.u32     a4, a4, 0;\n\t"
        "addc.u32        a5, a5, 0;\n\t"
        "add.cc.u32      b1, b1, a1;\n\t"                  // word 1
        "mul.lo.u32      m, b1, %6;\n\t"
        "madc.lo.cc.u32  a2, m, %4, a2;\n\t"
        "madc.hi.cc.u32  a3, m, %4, a3;\n\t"
        "addc.cc.u32     a4, a4, 0;\n\t"
        "addc.u32        a5, a5, 0;\n\t"
        "mad.lo.cc.u32   b1, m, %3, b1;\n\t"
        "madc.hi.cc.u32  b2, m, %3, b2;\n\t"
        "madc.lo.cc.u32  b3, m, %5, b3;\n\t"
        "madc.hi.cc.u32  b4, m, %5, b4;\n\t"
        "addc.u32        b5, 0, 0;\n\t"
        "add.cc.u32      a2, a2, b2;\n\t"                  // word 2
        "mul.lo.u32      m, a2, %6;\n\t"
        "madc.lo.cc.u32  b3, m, %4, b3;\n\t"
        "madc.hi.cc.u32  b4, m, %4, b4;\n\t"
        "addc.u32        b5, b5, 0;\n\t"
        "mad.lo.cc.u32   a2, m, %3, a2;\n\t"
        "madc.hi.cc.u32  a3, m, %3, a3;\n\t"
        "madc.lo.cc.u32  a4, m, %5, a4;\n\t"
        "madc.hi.u32     a5, m, %5, a5;\n\t"
        "add.cc.u32      %0, a3, b3;\n\t"
        "addc.cc.u32     %1, a4, b4;\n\t"
        "addc.u32        %2, a5, b5;\n\t}"
        : "+r"(x[0]), "+r"(x[1]), "+r"(x[2])
        : "r"(n[0]), "r"(n[1]), "r"(n[2]), "r"(np));
}

template <>
__device__ __forceinline__ void msqr<4>(u32 (&x)[4], const u32 (&n)[4], u32 np)
{
    asm("{\n\t.reg .u32 a0, a1, a2, a3, a4, a5, a6, a7, b1, b2, b3, b4, b5, b6, b7, e1, e2, e3, f2, g3, m;\n\t"
        "shl.b32         e1, %1, 1;\n\t"                   // 2 (x1, x2, x3) = (e1, e2, e3),
        "shf.l.wrap.b32  e2, %1, %2, 1;\n\t"               // 2 (x2, x3) = (f2, e3), 2 x3 = g3
        "shf.l.wrap.b32  e3, %2, %3, 1;\n\t"
        "shl.b32         f2, %2, 1;\n\t"
        "shl.b32         g3, %3, 1;\n\t"
        "mul.lo.u32      a0, %0, %0;\n\t"
        "mul.hi.u32      a1, %0, %0;\n\t"
        "mul.lo.u32      a2, %1, %1;\n\t"
        "mul.hi.u32      a3, %1, %1;\n\t"
        "mad.lo.cc.u32   a2, %0, e2, a2;\n\t"
        "madc.hi.cc.u32  a3, %0, e2, a3;\n\t"
        "madc.lo.cc.u32  a4, %2, %2, 0;\n\t"
        "madc.hi.u32     a5, %2, %2, 0;\n\t"
        "mul.lo.u32      b1, %0, e1;\n\t"
        "mul.hi.u32      b2, %0, e1;\n\t"
        "mul.lo.u32      b3, %0, e3;\n\t"
        "mul.hi.u32      b4, %0, e3;\n\t"
        "mul.lo.u32      m, a0, %8;\n\t"                   // word 0
        "mad.lo.cc.u32   b1, m, %5, b1;\n\t"
        "madc.hi.cc.u32  b2, m, %5, b2;\n\t"
        "madc.lo.cc.u32  b3, m, %7, b3;\n\t"
        "madc.hi.cc.u32  b4, m, %7, b4;\n\t"
        "madc.lo.cc.u32  b5, %2, g3, 0;\n\t"
        "madc.hi.u32     b6, %2, g3, 0;\n\t"
        "mad.lo.cc.u32   b3, %1, f2, b3;\n\t"
        "madc.hi.cc.u32  b4, %1, f2, b4;\n\t"
        "addc.cc.u32     b5, b5, 0;\n\t"
        "addc.u32        b6, b6, 0;\n\t"
        "mad.lo.cc.u32   a0, m, %4, a0;\n\t"
        "madc.hi.cc.u32  a1, m, %4, a1;\n\t"
        "madc.lo.cc.u32  a2, m, %6, a2;\n\t"
        "madc.hi.cc.u32  a3, m, %6, a3;\n\t"
        "madc.lo.cc.u32  a4, %1, e3, a4;\n\t"
        "madc.hi.cc.u32  a5, %1, e3, a5;\n\t"
        "madc.lo.cc.u32  a6, %3, %3, 0;\n\t"
        "madc.hi.u32     a7, %3, %3, 0;\n\t"
        "add.cc.u32      b1, b1, a1;\n\t"                  // word 1
        "mul.lo.u32      m, b1, %8;\n\t"
        "madc.lo.cc.u32  a2, m, %5, a2;\n\t"
        "madc.hi.cc.u32  a3, m, %5, a3;\n\t"
        "madc.lo.cc.u32  a4, m, %7, a4;\n\t"
        "madc.hi.cc.u32  a5, m, %7, a5;\n\t"
        "addc.cc.u32     a6, a6, 0;\n\t"
        "addc.u32        a7, a7, 0;\n\t"
        "mad.lo.cc.u32   b1, m, %4, b1;\n\t"
        "madc.hi.cc.u32  b2, m, %4, b2;\n\t"
        "madc.lo.cc.u32  b3, m, %6, b3;\n\t"
        "madc.hi.cc.u32  b4, m, %6, b4;\n\t"
        "addc.cc.u32     b5, b5, 0;\n\t"
        "addc.cc.u32     b6, b6, 0;\n\t"
        "addc.u32        b7, 0, 0;\n\t"
        "add.cc.u32      a2, a2, b2;\n\t"                  // word 2
        "mul.lo.u32      m, a2, %8;\n\t"
        "madc.lo.cc.u32  b3, m, %5, b3;\n\t"
        "madc.hi.cc.u32  b4, m, %5, b4;\n\t"
        "madc.lo.cc.u32  b5, m, %7, b5;\n\t"
        "madc.hi.cc.u32  b6, m, %7, b6;\n\t"
        "addc.u32        b7, b7, 0;\n\t"
        "mad.lo.cc.u32   a2, m, %4, a2;\n\t"
        "madc.hi.cc.u32  a3, m, %4, a3;\n\t"
        "madc.lo.cc.u32  a4, m, %6, a4;\n\t"
        "madc.hi.cc.u32  a5, m, %6, a5;\n\t"
        "addc.cc.u32     a6, a6, 0;\n\t"
        "addc.u32        a7, a7, 0;\n\t"
        "add.cc.u32      b3, b3, a3;\n\t"                  // word 3
        "mul.lo.u32      m, b3, %8;\n\t"
        "madc.lo.cc.u32  a4, m, %5, a4;\n\t"
        "madc.hi.cc.u32  a5, m, %5, a5;\n\t"
        "madc.lo.cc.u32  a6, m, %7, a6;\n\t"
        "madc.hi.u32     a7, m, %7, a7;\n\t"
        "mad.lo.cc.u32   b3, m, %4, b3;\n\t"
        "madc.hi.cc.u32  b4, m, %4, b4;\n\t"
        "madc.lo.cc.u32  b5, m, %6, b5;\n\t"
        "madc.hi.cc.u32  b6, m, %6, b6;\n\t"
        "addc.u32        b7, b7, 0;\n\t"
        "add.cc.u32      %0, a4, b4;\n\t"
        "addc.cc.u32     %1, a5, b5;\n\t"
        "addc.cc.u32     %2, a6, b6;\n\t"
        "addc.u32        %3, a7, b7;\n\t}"
        : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3])
        : "r"(n[0]), "r"(n[1]), "r"(n[2]), "r"(n[3]), "r"(np));
}

// x <- (x 2^sh + m N) / 2^32 (mod N), sh in [0, 31]: below x / 2 + N
template <int K>
__device__ __forceinline__ void mshift(u32 (&x)[K], u32 sh, const u32 (&n)[K], u32 np);

template <>
__device__ __forceinline__ void mshift<3>(u32 (&x)[3], u32 sh, const u32 (&n)[3], u32 np)
{
    asm("{\n\t.reg .u32 t0, t1, t2, t3, b1, b2, m;\n\t"
        "shl.b32         t0, %0, %7;\n\t"
        "shf.l.wrap.b32  t1, %0, %1, %7;\n\t"
        "shf.l.wrap.b32  t2, %1, %2, %7;\n\t"
        "shf.l.wrap.b32  t3, %2, 0, %7;\n\t"
        "mul.lo.u32      m, t0, %6;\n\t"
        "mul.lo.u32      b1, m, %4;\n\t"
        "mul.hi.u32      b2, m, %4;\n\t"
        "mad.lo.cc.u32   t0, m, %3, t0;\n\t"
        "madc.hi.cc.u32  t1, m, %3, t1;\n\t"
        "madc.lo.cc.u32  t2, m, %5, t2;\n\t"
        "madc.hi.u32     t3, m, %5, t3;\n\t"
        "add.cc.u32      %0, t1, b1;\n\t"
        "addc.cc.u32     %1, t2, b2;\n\t"
        "addc.u32        %2, t3, 0;\n\t}"
        : "+r"(x[0]), "+r"(x[1]), "+r"(x[2])
        : "r"(n[0]), "r"(n[1]), "r"(n[2]), "r"(np), "r"(sh));
}

template <>
__device__ __forceinline__ void mshift<4>(u32 (&x)[4], u32 sh, const u32 (&n)[4], u32 np)
{
    asm("{\n\t.reg .u32 t0, t1, t2, t3, t4, b1, b2, b3, b4, m;\n\t"
        "shl.b32         t0, %0, %9;\n\t"
        "shf.l.wrap.b32  t1, %0, %1, %9;\n\t"
        "shf.l.wrap.b32  t2, %1, %2, %9;\n\t"
        "shf.l.wrap.b32  t3, %2, %3, %9;\n\t"
        "shf.l.wrap.b32  t4, %3, 0, %9;\n\t"
        "mul.lo.u32      m, t0, %8;\n\t"
        "mul.lo.u32      b1, m, %5;\n\t"
        "mul.hi.u32      b2, m, %5;\n\t"
        "mul.lo.u32      b3, m, %7;\n\t"
        "mul.hi.u32      b4, m, %7;\n\t"
        "mad.lo.cc.u32   t0, m, %4, t0;\n\t"
        "madc.hi.cc.u32  t1, m, %4, t1;\n\t"
        "madc.lo.cc.u32  t2, m, %6, t2;\n\t"
        "madc.hi.cc.u32  t3, m, %6, t3;\n\t"
        "addc.u32        t4, t4, 0;\n\t"
        "add.cc.u32      %0, t1, b1;\n\t"
        "addc.cc.u32     %1, t2, b2;\n\t"
        "addc.cc.u32     %2, t3, b3;\n\t"
        "addc.u32        %3, t4, b4;\n\t}"
        : "+r"(x[0]), "+r"(x[1]), "+r"(x[2]), "+r"(x[3])
        : "r"(n[0]), "r"(n[1]), "r"(n[2]), "r"(n[3]), "r"(np), "r"(sh));
}

// leave Montgomery form: K words of reduction bring x / R into [0, N]
template <int K>
__device__ __forceinline__ void mleave(u32 (&x)[K], const u32 (&n)[K], u32 np)
{
#pragma unroll
    for (int i = 0; i < K; i++) {
        const u32 m = x[0] * np;
        u64 c = (u64)m * n[0] + x[0];
#pragma unroll
        for (int j = 1; j < K; j++) {
            c = (u64)m * n[j] + x[j] + (c >> 32);
            x[j - 1] = (u32)c;
        }
        x[K - 1] = (u32)(c >> 32);
    }
}

// N = p^2, -N^-1 mod 2^32 and p^-1 mod 2^64
template <int K>
__device__ __forceinline__ void fermat_modulus(u64 p, u32 (&n)[K], u32 &np, u64 &pinv)
{
    pinv = (3 * p) ^ 2;
    pinv *= 2 - p * pinv;
    pinv *= 2 - p * pinv;
    pinv *= 2 - p * pinv;
    pinv *= 2 - p * pinv;
    np = 0u - (u32)(pinv * pinv);
    const u64 N0 = p * p, N1 = __umul64hi(p, p);
    n[0] = (u32)N0; n[1] = (u32)(N0 >> 32); n[2] = (u32)N1;
    if (K == 4) n[K - 1] = (u32)(N1 >> 32);
}

struct FermOut { u64 q; bool ok; };

// the quotient's definition, q = (r - 1) p^-1 mod 2^64 and q < p with r = 2^(p-1) mod N, for a p
// that is no prime and has 2^(p-1) <> 1 (mod p): r itself, by squaring and doubling from R mod N
template <int K>
__device__ __forceinline__ u64 fermat_not_one(u64 p)
{
    u32 n[K], x[K], np;
    u64 pinv;
    fermat_modulus<K>(p, n, np, pinv);
    const auto less_n = [&](u32 (&t)[K]) {             // t - N if t >= N
        u32 d[K];
        u64 b = 0;
        for (int j = 0; j < K; j++) {
            b = (u64)t[j] - n[j] - b;
            d[j] = (u32)b;
            b = (b >> 32) & 1;
        }
        for (int j = 0; j < K; j++) t[j] = b ? t[j] : d[j];
    };
    const auto twice = [&](u32 (&t)[K]) {              // t < N, 2N < R
        for (int j = K - 1; j > 0; j--) t[j] = __funnelshift_l(t[j - 1], t[j], 1);
        t[0] <<= 1;
        less_n(t);
    };
    for (int j = 0; j < K; j++) x[j] = j == 0;
    for (int i = 0; i < 32 * K; i++) twice(x);
    const u64 e = p - 1;
    for (int b = 63 - __clzll((long long)e); b >= 0; b--) {
        msqr<K>(x, n, np);                             // below N^2 / R + N < 2N
        less_n(x);
        if ((e >> b) & 1) twice(x);
    }
    mleave<K>(x, n, np);
    less_n(x);
    const u64 q = (((u64)x[0] | ((u64)x[1] << 32)) - 1) * pinv;
    return q < p ? q : ~0ull;
}

// q_p(2) for odd p >= 3 (p < 2^47 for K = 3, p < 2^63 for K = 4); ok is false when 2^(p-1) <> 1
// (mod p), which happens for no prime
template <int K>
__device__ __forceinline__ FermOut fermat_one(u64 p)
{
    u32 n[K], np;
    u64 pinv;
    fermat_modulus<K>(p, n, np, pinv);
    // T squarings after the top six bits; w whole digits of five bits below a digit of rem bits
    const u64 e = p - 1;
    const int L = 64 - __clzll((long long)e), T = L > 6 ? L - 6 : 0;
    int w = T / 5;
    const int rem = T - 5 * w;
    const u64 ones = 0x1084210842108421ull;            // one in every five-bit digit
    const u64 d = e - ((ones & ((1ull << (5 * w)) - 1)) + (rem ? 1ull << (5 * w) : 0));
    u32 x[K];
    const u32 s0 = 32 * K - (u32)(d >> T);             // 2^-c R, c = the top (30 .. 63, or e itself)
#pragma unroll
    for (int j = 0; j < K; j++) x[j] = (s0 >> 5) == (u32)j ? 1u << (s0 & 31) : 0u;
    if (rem) {
        for (int i = 0; i < rem; i++) msqr<K>(x, n, np);
        mshift<K>(x, 31u - ((u32)(d >> (5 * w)) & ((1u << rem) - 1u)), n, np);
    }
    while (--w >= 0) {
#pragma unroll
        for (int i = 0; i < 5; i++) msqr<K>(x, n, np);
        mshift<K>(x, 31u - ((u32)(d >> (5 * w)) & 31u), n, np);
    }
    mleave<K>(x, n, np);
    const u64 r = (u64)x[0] | ((u64)x[1] << 32);
    const u64 q = (r - 1) * pinv;                      // q' with 2^-(p-1) = 1 + q'p
    FermOut o;
    // 2^-(p-1) = 1 (mod p), so that 1 + q'p is the whole residue, for every prime p
    const u64 hi = __umul64hi(q, p) + (q * p == ~0ull);
    const u64 rhi = K == 4 ? (u64)x[2] | ((u64)x[K - 1] << 32) : (u64)x[2];
    o.ok = q < p && hi == rhi;
    o.q = q ? p - q : 0;
    return o;
}

// one prime per thread (ILP = 1) or two interleaved primes per thread (ILP = 2).  The entries that
// are not ok are done again at the end, from the definition: inside the loop that code cost the
// ladder registers (5% of the kernel), and no prime needs it.  Until then such an entry holds its p
// with bit 63 set (p and every quotient are below 2^63), so that Q may be P's own array
template <int K, int ILP>
__global__ void __launch_bounds__(256) fermat_kernel(const u64 *P, u64 count, u64 *Q)
{
    const u64 stride = (u64)gridDim.x * blockDim.x * ILP, first = ((u64)blockIdx.x * blockDim.x + threadIdx.x) * ILP;
    bool again = false;
    for (u64 i = first; i < count; i += stride) {
        u64 p[ILP];
        FermOut o[ILP];
#pragma unroll
        for (int v = 0; v < ILP; v++) {
            p[v] = i + v < count ? P[i + v] : 0;
            o[v] = fermat_one<K>(p[v] >= 3 && (p[v] & 1) ? p[v] : 3);
        }
#pragma unroll
        for (int v = 0; v < ILP; v++) {
            const bool odd = p[v] >= 3 && (p[v] & 1);
            if (i + v < count) Q[i + v] = odd ? (o[v].ok ? o[v].q : p[v] | 1ull << 63) : 0;
            again |= odd && !o[v].ok;
        }
    }
    if (!again) return;
    for (u64 i = first; i < count; i += stride)
        for (int v = 0; v < ILP; v++)
            if (i + v < count && Q[i + v] >> 63) Q[i + v] = fermat_not_one<K>(Q[i + v] & ~(1ull << 63));
}

// ---- statistics: checksum, near count, FLT errors, hits, ordered hash ----

struct FermPart {
    u64 h, len;          // ordered hash over the segment and its number of terms
    u64 cks, near, flt, tests;
};

__device__ __forceinline__ u64 pow_u64(u64 b, u64 e)
{
    u64 r = 1;
    while (e) { if (e & 1) r *= b; b *= b; e >>= 1; }
    return r;
}

__device__ __forceinline__ void fp_join(FermPart &L, const FermPart &R)
{
    L.h = L.h * pow_u64(MP_FNV_PRIME, R.len) + R.h;
    L.len += R.len;
    L.cks += R.cks; L.near += R.near; L.flt += R.flt; L.tests += R.tests;
}

#define FS_THREADS 256
#define FS_PER 8                                           // consecutive entries per thread
#define FS_TILE (FS_THREADS * FS_PER)                      // entries per CTA

// the next prime p (in order) with its quotient q
__device__ __forceinline__ void fp_term(FermPart &f, u64 p, u64 q, u64 *hits, u64 *nhits)
{
    if (p < 3) return;                                     // 2 is not tested (and padding)
    f.tests++;
    if (q >= p) { f.flt++; return; }
    f.cks += mp_mix64(q ^ (p * MP_GOLD));
    const u64 A = q <= p / 2 ? q : p - q;
    f.near += A <= (p - 1) / 1000;                         // 1000 A < p
    f.h = f.h * MP_FNV_PRIME + mp_mix64(p ^ mp_mix64(q));
    f.len++;
    if (q == 0) {
        // keep the 16 smallest hits, sorted, whatever the order the threads arrive in:
        // slot j keeps the smaller of its value and the incoming one and passes the larger
        // on, so slot j ends with the (j+1)-th smallest value that ever reached it
        atomicAdd((unsigned long long *)nhits, 1ull);
        u64 v = p;
        for (int j = 0; j < 16 && v != ~0ull; j++) {
            const u64 old = atomicMin((unsigned long long *)(hits + j), (unsigned long long)v);
            v = old > v ? old : v;
        }
    }
}

// in-order join of the threads' parts; thread 0 holds the result.  s_w: one part per warp
__device__ __forceinline__ void fp_cta_join(FermPart &f, FermPart *s_w)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll 1
    for (int round = 0; round < 2; round++) {
#pragma unroll 1
        for (int d = 1; d < 32; d <<= 1) {
            FermPart r;
            r.h = __shfl_down_sync(0xffffffffu, f.h, d);
            r.len = __shfl_down_sync(0xffffffffu, f.len, d);
            r.cks = __shfl_down_sync(0xffffffffu, f.cks, d);
            r.near = __shfl_down_sync(0xffffffffu, f.near, d);
            r.flt = __shfl_down_sync(0xffffffffu, f.flt, d);
            r.tests = __shfl_down_sync(0xffffffffu, f.tests, d);
            if ((lane & (2 * d - 1)) == 0 && lane + d < 32) fp_join(f, r);
        }
        if (round) return;
        if (lane == 0) s_w[warp] = f;
        __syncthreads();
        if (warp) return;
        f = lane < nw ? s_w[lane] : FermPart{0, 0, 0, 0, 0, 0};
    }
}

// one CTA per FS_TILE entries: the tile's primes and quotients are staged in shared memory
// with coalesced loads, each thread folds its FS_PER consecutive entries in order (the ordered
// hash by Horner's rule), then the threads join in order
__global__ void __launch_bounds__(FS_THREADS) fermat_stats_kernel(const u64 *__restrict__ P, const u64 *__restrict__ Q,
                                                                  u64 count, FermPart *parts, u64 *hits, u64 *nhits)
{
    __shared__ FermPart s_w[FS_THREADS / 32];
    // entry k at k + k / FS_PER: a thread's FS_PER entries are 9 words apart from the next
    // thread's, which keeps the reads nearly free of bank conflicts
    __shared__ u64 sp[FS_TILE + FS_TILE / FS_PER], sq[FS_TILE + FS_TILE / FS_PER];
    const u64 t0 = (u64)blockIdx.x * FS_TILE;
    for (u32 k = threadIdx.x; k < FS_TILE; k += FS_THREADS) {
        const bool in = t0 + k < count;
        sp[k + k / FS_PER] = in ? __ldcs(P + t0 + k) : 0;
        sq[k + k / FS_PER] = in ? __ldcs(Q + t0 + k) : 0;
    }
    __syncthreads();
    FermPart f = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int u = 0; u < FS_PER; u++)
        fp_term(f, sp[threadIdx.x * (FS_PER + 1) + u], sq[threadIdx.x * (FS_PER + 1) + u], hits, nhits);
    fp_cta_join(f, s_w);
    if (threadIdx.x == 0) parts[blockIdx.x] = f;
}

// the quotients and their statistics in one pass, for callers that want the statistics only: one
// CTA per FS_TILE primes, each thread FS_PER consecutive ones, one after the other (ILP = 1) or
// two at a time.  The quotients stay in registers, which saves writing them and reading both
// arrays again (36.2 M primes near 1e12: 3.7 ms of kernels with the tree join below, 4.2 ms before)
template <int K, int ILP>
__global__ void __launch_bounds__(FS_THREADS) fermat_fused_kernel(const u64 *__restrict__ P, u64 count, FermPart *parts,
                                                                  u64 *hits, u64 *nhits)
{
    __shared__ FermPart s_w[FS_THREADS / 32];
    const u64 i0 = (u64)blockIdx.x * FS_TILE + (u64)threadIdx.x * FS_PER;
    FermPart f = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
    for (int u = 0; u < FS_PER; u += ILP) {
        u64 p[ILP], q[ILP];
#pragma unroll
        for (int v = 0; v < ILP; v++) {
            p[v] = i0 + u + v < count ? __ldg(P + i0 + u + v) : 0;
            const bool odd = p[v] >= 3 && (p[v] & 1);
            const FermOut o = fermat_one<K>(odd ? p[v] : 3);
            q[v] = odd ? (o.ok ? o.q : ~0ull) : 0;
        }
#pragma unroll
        for (int v = 0; v < ILP; v++) fp_term(f, p[v], q[v], hits, nhits);
    }
    fp_cta_join(f, s_w);
    if (threadIdx.x == 0) parts[blockIdx.x] = f;
}

// in-order join of the CTAs' parts: each thread a contiguous run, then the threads (0.47 ms for
// 17,672 parts when thread 0 joined the 1024 threads' results one after the other)
__global__ void __launch_bounds__(1024) fermat_final_kernel(const FermPart *parts, u64 nparts, const u64 *nhits,
                                                            const u64 *hits, mp_wief_stats *out)
{
    __shared__ FermPart s_w[32];
    const u32 tid = threadIdx.x, nth = blockDim.x;
    const u64 per = (nparts + nth - 1) / nth;
    FermPart f = {0, 0, 0, 0, 0, 0};
    for (u64 b = tid * per; b < (tid + 1) * per && b < nparts; b++) fp_join(f, parts[b]);
    fp_cta_join(f, s_w);
    if (tid == 0) {
        out->tests = f.tests;
        out->near = f.near;
        out->flt = f.flt;
        out->cks = f.cks;
        out->ordered_hash = f.h;
        out->nhits = *nhits;
        for (int k = 0; k < 16; k++) out->hits[k] = (u64)k < *nhits ? hits[k] : 0;
    }
}

// ---- host side ----

int mp_fermat_run(mp_handle *h, const u64 *d_p, u64 count, u64 *d_q, cudaStream_t st, int variant, u64 *)
{
    if (!count) return MP_OK;
    // variant: bit 0 = limbs (0: K=3, 1: K=4); bit 1 = two primes per thread
    const int k4 = variant & 1, ilp2 = (variant >> 1) & 1;
    const u64 work = ilp2 ? (count + 1) / 2 : count;
    u64 grid = (work + 255) / 256;
    const u64 gmax = (u64)h->sm_count * 64;
    if (grid > gmax) grid = gmax;
    ProfScope ps(h, PROF_FERMAT, st);
    if (!k4 && !ilp2) fermat_kernel<3, 1><<<(unsigned)grid, 256, 0, st>>>(d_p, count, d_q);
    else if (!k4 && ilp2) fermat_kernel<3, 2><<<(unsigned)grid, 256, 0, st>>>(d_p, count, d_q);
    else if (k4 && !ilp2) fermat_kernel<4, 1><<<(unsigned)grid, 256, 0, st>>>(d_p, count, d_q);
    else fermat_kernel<4, 2><<<(unsigned)grid, 256, 0, st>>>(d_p, count, d_q);
    MP_CUDA(h, cudaGetLastError());
    return MP_OK;
}

// the statistics of mp_wieferich_range over the primes d_p (variant as in mp_fermat_run)
int mp_fermat_stats(mp_handle *h, const u64 *d_p, u64 count, mp_wief_stats *d_stats, cudaStream_t st, int variant)
{
    const u64 nb = count ? (count + FS_TILE - 1) / FS_TILE : 1;
    MP_CUDA(h, h->ferm_part.ensure((size_t)nb * sizeof(FermPart) + 256));
    FermPart *parts = h->ferm_part.as<FermPart>();
    u64 *hits = (u64 *)((char *)h->ferm_part.p + nb * sizeof(FermPart));
    u64 *nhits = hits + 16;
    MP_CUDA(h, cudaMemsetAsync(hits, 0xff, 16 * 8, st));        // empty slots hold 2^64 - 1
    MP_CUDA(h, cudaMemsetAsync(nhits, 0, 8, st));
    if (count) {
        ProfScope ps(h, PROF_FERMAT, st);
        switch (variant & 3) {
        case 0: fermat_fused_kernel<3, 1><<<(unsigned)nb, FS_THREADS, 0, st>>>(d_p, count, parts, hits, nhits); break;
        case 1: fermat_fused_kernel<4, 1><<<(unsigned)nb, FS_THREADS, 0, st>>>(d_p, count, parts, hits, nhits); break;
        case 2: fermat_fused_kernel<3, 2><<<(unsigned)nb, FS_THREADS, 0, st>>>(d_p, count, parts, hits, nhits); break;
        default: fermat_fused_kernel<4, 2><<<(unsigned)nb, FS_THREADS, 0, st>>>(d_p, count, parts, hits, nhits); break;
        }
        MP_CUDA(h, cudaGetLastError());
    } else {
        MP_CUDA(h, cudaMemsetAsync(parts, 0, sizeof(FermPart), st));
    }
    ProfScope ps(h, PROF_FERMAT_STATS, st);
    fermat_final_kernel<<<1, 1024, 0, st>>>(parts, nb, nhits, hits, d_stats);
    MP_CUDA(h, cudaGetLastError());
    return MP_OK;
}

// ---------------------------------------------------------------------------------------
// mp_wieferich_stats_noalloc: the statistics of mp_wieferich_range for caller-supplied device
// arrays of primes and quotients, for callers that must not allocate device memory -- code
// that runs under a memory manager or pool that owns the whole device, inside a framework
// whose allocator may not be bypassed, or in a latency-critical loop where a cudaMalloc
// (which can synchronise the device) is not allowed.  It uses no handle (a handle allocates
// its tables and buffers) and no allocation of any kind: its scratch lives in the file-scope
// array below, which every GPU that loads this library keeps until the process exits.
// ---------------------------------------------------------------------------------------

#define NOALLOC_PARTS (MP_NOALLOC_MAX_COUNT / FS_TILE)    // one partial per stats CTA
static_assert(MP_NOALLOC_MAX_COUNT % FS_TILE == 0, "the scratch limit must be whole stats tiles");
static_assert((u64)NOALLOC_PARTS * FS_TILE >= MP_NOALLOC_MAX_COUNT, "one partial per CTA of the largest call");

struct NoallocScratch {
    FermPart parts[NOALLOC_PARTS];                          // 384 KB
    u64 hits[16];
    u64 nhits;
};

static __device__ __align__(256) NoallocScratch g_noalloc_scratch;

// The host sees g_noalloc_scratch only as a stand-in symbol: its device address is looked up
// once per device with cudaGetSymbolAddress (with that device current) and kept here.  A
// device reset between calls would move the array; that is not supported.
static std::mutex g_noalloc_mu;
static void *g_noalloc_ptr[64] = {nullptr};

// the hit list and its count carry over from the previous call: empty slots hold 2^64 - 1
__global__ void noalloc_clear_kernel(NoallocScratch *s)
{
    if (threadIdx.x < 16) s->hits[threadIdx.x] = ~0ull;
    if (threadIdx.x == 0) s->nhits = 0;
}

__global__ void noalloc_count_kernel(mp_wief_stats *out, u64 count) { out->primes = count; }

extern "C" int mp_wieferich_stats_noalloc(const uint64_t *d_p, const uint64_t *d_q, uint64_t count,
                                           mp_wief_stats *d_stats, void *stream)
{
    if (!d_stats || (count && (!d_p || !d_q))) return MP_EINVAL;
    if (count > MP_NOALLOC_MAX_COUNT) return MP_EINVAL;    // beyond the fixed scratch
    // an error already pending in this thread belongs to the caller: leave it for the caller
    // to read, and run nothing
    if (cudaPeekAtLastError() != cudaSuccess) return MP_ECUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return MP_ECUDA;
    NoallocScratch *s = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_ptr[dev]) {
            void *p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
                cudaGetLastError();                          // this call's own failure
                return MP_ECUDA;
            }
            g_noalloc_ptr[dev] = p;
        }
        s = (NoallocScratch *)g_noalloc_ptr[dev];
    }
    cudaStream_t st = (cudaStream_t)stream;
    // every launch is checked; a failure here is this call's own, so it is cleared
#define NOALLOC_CHECK()                                                                       \
    do {                                                                                      \
        if (cudaPeekAtLastError() != cudaSuccess) { cudaGetLastError(); return MP_ECUDA; }   \
    } while (0)
    noalloc_clear_kernel<<<1, 32, 0, st>>>(s);
    NOALLOC_CHECK();
    const u64 nb = count ? (count + FS_TILE - 1) / FS_TILE : 0;
    if (count) {
        fermat_stats_kernel<<<(unsigned)nb, FS_THREADS, 0, st>>>(d_p, d_q, count, s->parts, s->hits, &s->nhits);
        NOALLOC_CHECK();
    } else if (cudaMemsetAsync(s->parts, 0, sizeof(FermPart), st) != cudaSuccess) {
        cudaGetLastError();
        return MP_ECUDA;                                     // no input: one empty partial
    }
    fermat_final_kernel<<<1, 1024, 0, st>>>(s->parts, nb ? nb : 1, &s->nhits, s->hits, d_stats);
    NOALLOC_CHECK();
    noalloc_count_kernel<<<1, 1, 0, st>>>(d_stats, count);
    NOALLOC_CHECK();
#undef NOALLOC_CHECK
    return MP_OK;
}
