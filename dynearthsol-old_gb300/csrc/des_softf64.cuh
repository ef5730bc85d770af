// Exactly rounded FP64 arithmetic on the integer pipes: products, quotients,
// square roots, some sums, comparisons and conversions.
//
// GB300 retires 2 FP64 instructions per clock per SM at its nominal rate and
// 1.6 in a loop of independent FMAs (one warp instruction in 20.2 clocks),
// while its integer ALU and FMA pipes retire 64 and more lanes per clock.  A kernel bound by the
// FP64 pipe can move part of its arithmetic to these
// routines and run both pipes at once.  Each returns, bit for bit, what the
// FP64 unit returns (IEEE-754 binary64, round to nearest even, subnormals
// kept): the fast path covers normal operands with a normal result, and the
// rest (zeros, subnormals, infinities, NaN, overflow, underflow) takes an
// integer slow path.  Neither path issues an FP64 instruction: the compiler
// predicates short branches, and a predicated FP64 instruction still
// occupies the FP64 pipe.  64-bit leading-zero counts are formed from two
// 32-bit counts for the same reason (the 64-bit count is lowered through a
// conversion on the FP64 unit).
//
// The header compiles as plain C++ too, so that the host can check it
// against its own IEEE arithmetic.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define DES_SF_HD __host__ __device__ __forceinline__
#else
#define DES_SF_HD static inline
#endif

namespace des {
namespace sf {

constexpr uint64_t kAbs = 0x7fffffffffffffffull;
constexpr uint64_t kSign = 0x8000000000000000ull;
constexpr uint64_t kFrac = 0x000fffffffffffffull;
constexpr uint64_t kHidden = 0x0010000000000000ull;
constexpr uint64_t kInf = 0x7ff0000000000000ull;
constexpr uint64_t kQuiet = 0x0008000000000000ull;
constexpr uint64_t kDefaultNaN = 0x7ff8000000000000ull;

DES_SF_HD uint64_t bits(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    memcpy(&b, &x, 8);
    return b;
#endif
}

DES_SF_HD double from_bits(uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double x;
    memcpy(&x, &b, 8);
    return x;
#endif
}

DES_SF_HD float float_from_bits(uint32_t b)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float x;
    memcpy(&x, &b, 4);
    return x;
#endif
}

DES_SF_HD int clz32(uint32_t x)
{
#if defined(__CUDA_ARCH__)
    return __clz((int)x);
#else
    return x ? __builtin_clz(x) : 32;
#endif
}

// leading zeros of a 64-bit word from two 32-bit counts
DES_SF_HD int clz64(uint64_t x)
{
    const uint32_t hi = (uint32_t)(x >> 32);
    return hi ? clz32(hi) : 32 + clz32((uint32_t)x);
}

DES_SF_HD uint64_t mulhi64(uint64_t a, uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// round to nearest even on the 11 bits below a 53-bit significand held at
// the top of r (bit 63 down to 11), then pack with the biased exponent e
// (1 <= e; a carry out of the significand moves into the exponent, and
// e = 2046 with a carry gives the infinity the rounding asks for)
DES_SF_HD uint64_t round_pack(uint64_t sign, int e, uint64_t r)
{
    const uint64_t m = r >> 11, rem = r & 0x7ff;
    const uint64_t up = (uint64_t)((rem > 0x400) | ((rem == 0x400) & (uint32_t)m));
    return ((((uint64_t)(e - 1)) << 52) + m + up) | sign;
}

// the cases the fast path of mul leaves: zeros, subnormals, infinities, NaN,
// results outside the normal range
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
uint64_t mul_slow(uint64_t a, uint64_t b)
{
    const uint64_t sign = (a ^ b) & kSign;
    const uint64_t ma = a & kAbs, mb = b & kAbs;
    const int ea = (int)(ma >> 52), eb = (int)(mb >> 52);
    if (ea == 2047 || eb == 2047) {
        if (ma > kInf) return a | kQuiet;
        if (mb > kInf) return b | kQuiet;
        if (ma == 0 || mb == 0) return kDefaultNaN;
        return sign | kInf;
    }
    if (ma == 0 || mb == 0) return sign;
    uint64_t fa = (ma & kFrac) | (ea ? kHidden : 0), fb = (mb & kFrac) | (eb ? kHidden : 0);
    const int la = clz64(fa), lb = clz64(fb);
    fa <<= la;
    fb <<= lb;
    const uint64_t hi = mulhi64(fa, fb), lo = fa * fb;
    const int lz = (int)(1 - (hi >> 63));
    uint64_t r = (hi << lz) | (uint64_t)(lo != 0);
    int e = (ea ? ea : 1) + (eb ? eb : 1) - 1000 - la - lb - lz;
    if (e >= 2047) return sign | kInf;
    if (e < 1) {
        const uint32_t sh = (uint32_t)(1 - e) > 63u ? 63u : (uint32_t)(1 - e);
        uint64_t rs = r >> sh;
        rs |= (uint64_t)((rs << sh) != r);
        r = rs;
        e = 1;
    }
    return round_pack(sign, e, r);
}

// 32x32 -> 64 products with a 64-bit addend; on the device as PTX
// mul.wide.u32 / mad.wide.u32 instructions, which the compiler's IR passes
// keep as they are
DES_SF_HD uint64_t wide_mul(uint32_t x, uint32_t y)
{
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("mul.wide.u32 %0, %1, %2;" : "=l"(r) : "r"(x), "r"(y));
    return r;
#else
    return (uint64_t)x * y;
#endif
}

DES_SF_HD uint64_t wide_mad(uint32_t x, uint32_t y, uint64_t c)
{
#if defined(__CUDA_ARCH__)
    uint64_t r;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(x), "r"(y), "l"(c));
    return r;
#else
    return (uint64_t)x * y + c;
#endif
}

// An operand taken apart for products: the significand shifted left by 6
// (hi 27 bits with the hidden bit, lo 32 bits) and the word of sign and
// exponent.
struct Op {
    uint32_t lo, hi, ex;
};

// x taken apart.  far collects the largest distance of a nonzero operand's
// exponent from the bottom of [2^-510, 2^511): while in_range(far), products
// of the operands so far are zero or normal numbers.  A zero's significand is
// 0 (no hidden bit).
DES_SF_HD Op unpack(double x, uint32_t &far)
{
    const uint64_t b = bits(x);
    const uint32_t h = (uint32_t)(b >> 32), l = (uint32_t)b, h2 = h + h;
    const bool nz = (h2 | l) != 0;
    const uint32_t f = nz ? h2 - (513u << 21) : 0u;
    far = far > f ? far : f;
    const uint32_t hh = nz ? ((h & 0xfffffu) | 0x100000u) : 0u;
    Op u;
    u.lo = l << 6;
    u.hi = (hh << 6) | (l >> 26);
    u.ex = h & 0xfff00000u;
    return u;
}
DES_SF_HD bool in_range(uint32_t far) { return far < (1021u << 21); }

// a b as the FP64 unit rounds it, for operands in unpack()'s range (any
// bits otherwise).  With both significands shifted by 6, the 118-bit
// product P holds the result's 53-bit significand at bit 64 (t = 0) or 65
// (t = 1, P >= 2^117): four 32x32 -> 64 products, one shift by t, and the
// rounding as one carry chain (2^63 - 1 added to the bits below, plus the
// carry of the sticky bits and the significand's last bit: round to nearest
// even).  The signs and exponents add in their word; the sum's range is
// unpack()'s promise.  22 instructions and no branch, against 35 and a branch
// for a product that checks its own operands: operands are taken apart once,
// and a group of products is checked once.
DES_SF_HD double prod(Op a, Op b)
{
    const uint32_t ex = a.ex + b.ex - (1024u << 20);
    const uint32_t sign = (a.ex ^ b.ex) & 0x80000000u;
    uint32_t lo, hi, top;
#if defined(__CUDA_ARCH__)
    asm("{\n\t.reg .b64 p, s, m;\n\t.reg .b32 low, mid, sl, sh, m0, m1, t, r, e;\n\t"
        "mul.wide.u32 p, %3, %5;\n\t"
        "mul.wide.u32 s, %3, %6;\n\t"
        "mul.wide.u32 m, %4, %6;\n\t"
        "mad.wide.u32 s, %4, %5, s;\n\t"
        "mov.b64 {low, mid}, p;\n\t"
        "mov.b64 {sl, sh}, s;\n\t"
        "mov.b64 {m0, m1}, m;\n\t"
        "add.cc.u32 mid, mid, sl;\n\t"
        "addc.cc.u32 m0, m0, sh;\n\t"
        "addc.u32 m1, m1, 0;\n\t"
        "mov.b32 %2, m1;\n\t"
        "shr.u32 t, m1, 21;\n\t"
        "lop3.b32 low, mid, t, low, 0xEA;\n\t"      // the bit the shift drops joins the sticky bits
        "shf.r.clamp.b32 mid, mid, m0, t;\n\t"
        "shf.r.clamp.b32 m0, m0, m1, t;\n\t"
        "shr.u32 m1, m1, t;\n\t"
        "mad.lo.u32 e, t, 0x100000, %7;\n\t"
        "lop3.b32 r, m0, 1, low, 0xEA;\n\t"
        "add.cc.u32 r, r, 0xffffffff;\n\t"
        "addc.cc.u32 mid, mid, 0x7fffffff;\n\t"
        "addc.cc.u32 %0, m0, 0;\n\t"
        "addc.u32 %1, m1, e;\n\t}"
        : "=r"(lo), "=r"(hi), "=r"(top)
        : "r"(a.lo), "r"(a.hi), "r"(b.lo), "r"(b.hi), "r"(ex));
#else
    const uint64_t p = wide_mul(a.lo, b.lo), s = wide_mad(a.hi, b.lo, wide_mul(a.lo, b.hi));
    const uint64_t c = (p >> 32) + (uint32_t)s;
    uint64_t m = wide_mul(a.hi, b.hi) + (s >> 32) + (c >> 32);
    top = (uint32_t)(m >> 32);
    const uint32_t t = (uint32_t)(m >> 53);
    const uint32_t low = (uint32_t)p | ((uint32_t)c & t);
    const uint32_t mid = (uint32_t)(((m << 32) | (uint32_t)c) >> t);
    m >>= t;
    const uint64_t up = ((uint64_t)mid + 0x7fffffffu + (uint64_t)((low | ((uint32_t)m & 1)) != 0)) >> 32;
    m += up;
    lo = (uint32_t)m;
    hi = (uint32_t)(m >> 32) + ex + (t << 20);
#endif
    if (top == 0) hi = sign;     // a zero operand (a nonzero product has top >= 2^20)
    return from_bits(((uint64_t)hi << 32) | lo);
}

// x * y as the FP64 unit rounds it
DES_SF_HD double mul(double x, double y)
{
    uint32_t far = 0;
    const Op a = unpack(x, far), b = unpack(y, far);
    if (in_range(far)) return prod(a, b);
    return from_bits(mul_slow(bits(x), bits(y)));
}

// a < b (an FP64 comparison occupies the FP64 pipe like an addition)
DES_SF_HD bool less(double a, double b)
{
    const uint64_t x = bits(a), y = bits(b), mx = x & kAbs, my = y & kAbs;
    // a zero's sign does not count; NaN compares false
    const int64_t kx = (x >> 63) ? -(int64_t)mx : (int64_t)mx, ky = (y >> 63) ? -(int64_t)my : (int64_t)my;
    return kx < ky && mx <= kInf && my <= kInf;
}

// ---- sum and difference ---------------------------------------------------------
// x + y and x - y as the FP64 unit rounds them, for products of operands in
// unpack()'s range (zeros or normal numbers); rare stays false where neither
// result loses more than its 31 leading bits or falls near the subnormal
// range (any bits otherwise).  The two share their alignment: about 37
// instructions a result on the integer pipes, which take them in less time
// than the FP64 pipe takes its two.
DES_SF_HD void sum_diff(double x, double y, double &sum, double &diff, bool &rare)
{
    const uint64_t bx = bits(x), by = bits(y);
    const bool swap = (bx & kAbs) < (by & kAbs);
    const uint64_t big = swap ? by : bx, small = swap ? bx : by;
    const uint32_t hb = (uint32_t)(big >> 32), hs = (uint32_t)(small >> 32);
    const uint32_t eb = hb & 0x7ff00000u, es = hs & 0x7ff00000u;
    uint32_t d = (eb - es) >> 20;
    d = d < 63u ? d : 63u;
    // significands at bit 62, 10 zero bits below; a zero has none
    const uint64_t mb = ((big << 10) & 0x3fffffffffffffffull) | (eb ? 0x4000000000000000ull : 0);
    const uint64_t ms = ((small << 10) & 0x3fffffffffffffffull) | (es ? 0x4000000000000000ull : 0);
    uint64_t a = ms >> d;
    a |= (uint64_t)((a << d) != ms);                      // sticky
    // the magnitudes' sum, one bit up where it carries
    uint64_t s = mb + a;
    const uint32_t t = (uint32_t)(s >> 63);
    s = (s >> t) | (s & t);
    s += 0x1ff + ((uint32_t)(s >> 10) & 1);
    const uint32_t sl = (uint32_t)(s >> 10), sh = (uint32_t)(s >> 42) + eb + (t << 20) - (1u << 20);
    // their difference, shifted up to bit 62
    uint64_t f = mb - a;
    const uint32_t k = (uint32_t)clz32((uint32_t)(f >> 32)) - 1;
    const bool none = f == 0;
    rare = rare || (!none && k > 30u) || eb - 1u < (64u << 20) - 1u;
    f <<= k & 63;
    f += 0x1ff + ((uint32_t)(f >> 10) & 1);
    const uint32_t fl = (uint32_t)(f >> 10);
    const uint32_t fh = none ? 0u : (uint32_t)(f >> 42) + eb - (k << 20) - (1u << 20);
    const bool same = !((uint32_t)((bx ^ by) >> 32) & 0x80000000u);
    const uint32_t sx = (uint32_t)(bx >> 32) & 0x80000000u;
    const uint32_t sd = none ? 0u : same ? (swap ? sx ^ 0x80000000u : sx) : hb & 0x80000000u;   // the difference's sign
    const uint32_t ss = sx;                                                                   // the sum's
    const uint64_t S = ((uint64_t)((eb ? sh : 0u) | ss) << 32) | (eb ? sl : 0u);
    const uint64_t D = ((uint64_t)(fh | sd) << 32) | (none ? 0u : fl);
    sum = from_bits(same ? S : D);
    diff = from_bits(same ? D : S);
}

// x + y alone, for numbers of 2^-900 and more and a zero beside them (rare as
// above; two zeros are rare, too: N-C's walk over a node whose first x term is
// one is repeated on the FP64 unit, 95-104 us a pass on a box without jitter in
// its first steps, where most are, against 90).
DES_SF_HD double sum(double x, double y, bool &rare)
{
    const uint64_t bx = bits(x), by = bits(y);
    const bool swap = (bx & kAbs) < (by & kAbs);
    const uint64_t big = swap ? by : bx, small = swap ? bx : by;
    const uint32_t hb = (uint32_t)(big >> 32), hs = (uint32_t)(small >> 32);
    const uint32_t eb = hb & 0x7ff00000u, es = hs & 0x7ff00000u;
    uint32_t d = (eb - es) >> 20;
    d = d < 63u ? d : 63u;
    // significands at bit 61, 9 zero bits below; a zero has none
    const uint64_t mb = ((big << 9) & 0x1fffffffffffffffull) | (eb ? 0x2000000000000000ull : 0);
    const uint64_t ms = ((small << 9) & 0x1fffffffffffffffull) | (es ? 0x2000000000000000ull : 0);
    uint64_t a = ms >> d;
    a |= (uint64_t)((a << d) != ms);                      // sticky
    const uint64_t minus = (uint64_t)((int64_t)(bx ^ by) >> 63);
    uint64_t f = mb + (a ^ minus) - minus;
    const uint32_t k = (uint32_t)clz32((uint32_t)(f >> 32)) - 1;
    const bool none = f == 0;
    rare = rare || (!none && k > 30u) || eb - (123u << 20) > (1900u << 20) - (123u << 20);
    f <<= k & 63;
    f += 0x1ff + ((uint32_t)(f >> 10) & 1);
    const uint64_t w = (f >> 10) + ((uint64_t)(eb - (k << 20)) << 32);
    const uint64_t sign = none && minus ? 0 : big & kSign;
    return from_bits((none ? 0 : w) | sign);
}

// ---- quotients ----------------------------------------------------------------
// The FP64 unit's division takes about nine FP64 instructions; on the integer
// pipes the reciprocal of the denominator's significand comes from an FP32
// reciprocal and two Newton steps in fixed point (64 bits, relative error
// below 2^-58), the quotient's significand from one high product, and its
// remainder, exact in 64 bits, moves it to the nearest where the candidate is
// one off.  A quotient of two 53-bit significands is never half way between
// two of them, so the nearest is the rounded quotient.

#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
double div_slow(double a, double b) { return a / b; }

// A denominator: its significand and about 2^115 / m.
struct Den {
    uint64_t m, y;
    uint32_t ex;
};

// the reciprocal seed: about 2^31 / x for the significand x in [1, 2) whose
// top 23 fraction bits are f, within 2^-20 of it, in [2^30, 2^31)
DES_SF_HD uint32_t rcp_seed(uint32_t f)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(float_from_bits(0x3f800000u | f)));
    uint32_t b = __float_as_uint(r);
#else
    const float r = 1.0f / float_from_bits(0x3f800000u | f);
    uint32_t b;
    memcpy(&b, &r, 4);
#endif
    b = b > 0x3f000000u ? b : 0x3f000000u;
    return b >= 0x3f800000u ? 0x7fffffffu : ((b & 0x7fffffu) | 0x800000u) << 7;
}

// b as a denominator; far as in unpack (a zero is out of range here)
DES_SF_HD Den denominator(double b, uint32_t &far)
{
    const uint64_t v = bits(b);
    const uint32_t f = ((uint32_t)(v >> 32) << 1) - (513u << 21);
    far = far > f ? far : f;
    Den d;
    d.m = (v & kFrac) | kHidden;
    d.ex = (uint32_t)(v >> 32) & 0xfff00000u;
    const uint64_t M = d.m << 11;
    const uint32_t y0 = rcp_seed((uint32_t)(M >> 40) & 0x7fffffu);
    // e0 = 2^62 - M y0 / 2^32 (M y0 is near 2^94)
    const uint64_t p = wide_mad((uint32_t)(M >> 32), y0, wide_mul((uint32_t)M, y0) >> 32);
    const int32_t e0 = (int32_t)((int64_t)((1ull << 62) - p) >> 11);
    const uint64_t y1 = ((uint64_t)y0 << 32) + (uint64_t)(((int64_t)e0 * (int64_t)y0) >> 19);
    const int32_t e1 = (int32_t)((1ull << 62) - mulhi64(M, y1));
    d.y = y1 + (uint64_t)(((int64_t)e1 * (int64_t)(y1 >> 32)) >> 30);
    return d;
}

// a / b as the FP64 unit rounds it, for a in unpack's range (collected in
// far) and b from denominator()
DES_SF_HD double quotient(double a, const Den &b, uint32_t &far)
{
    const uint64_t v = bits(a);
    const uint32_t h = (uint32_t)(v >> 32), h2 = h + h;
    const bool nz = (h2 | (uint32_t)v) != 0;
    const uint32_t f = nz ? h2 - (513u << 21) : 0u;
    far = far > f ? far : f;
    const uint64_t m = (v & kFrac) | kHidden;
    const uint32_t s = (uint32_t)(m < b.m);              // a quotient below 1 takes one more bit
    const uint32_t sh = 10 - s;
    uint64_t q = (mulhi64(m << 11, b.y) + (1ull << (sh - 1))) >> sh;
    const int64_t r = (int64_t)((m << (52 + s)) - q * b.m), half = (int64_t)(b.m >> 1);
    q += (uint64_t)(r > half) - (uint64_t)(r < -half);
    const uint32_t ex = (h & 0xfff00000u) - b.ex + ((1022u - s) << 20);
    const uint64_t w = q + ((uint64_t)ex << 32);
    return from_bits(nz ? w : (uint64_t)((h ^ b.ex) & 0x80000000u) << 32);
}

// x / y as the FP64 unit rounds it
DES_SF_HD double div(double x, double y)
{
    uint32_t far = 0;
    const Den d = denominator(y, far);
    const double q = quotient(x, d, far);
    return in_range(far) ? q : div_slow(x, y);
}

// ---- square root -----------------------------------------------------------------

#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
double root_slow(double x) { return ::sqrt(x); }

// about 2^32 / sqrt(a) for a in [1, 4) given as an FP32 number, in (2^31, 2^32)
DES_SF_HD uint32_t rsqrt_seed(uint32_t fbits)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(float_from_bits(fbits)));
    uint32_t b = __float_as_uint(r);
#else
    const float r = 1.0f / ::sqrtf(float_from_bits(fbits));
    uint32_t b;
    memcpy(&b, &r, 4);
#endif
    b = b > 0x3f000000u ? b : 0x3f000000u;
    return b >= 0x3f800000u ? 0xffffffffu : ((b & 0x7fffffu) | 0x800000u) << 8;
}

// sqrt(x) as the FP64 unit rounds it (about 18 FP64 instructions there): with
// a in [1, 4) and an even exponent, an FP32 reciprocal root and two steps of
// g += (a - g g) / (2 sqrt(a)) in 62-bit fixed point, then the exact remainder
// of the nearest 53-bit candidate, which is at most one off.  A root is never
// half way between two 53-bit numbers.
DES_SF_HD double root(double x)
{
    const uint64_t v = bits(x);
    const uint32_t h = (uint32_t)(v >> 32);
    if (!(h - (1u << 20) < (2046u << 20))) return root_slow(x);      // zero, subnormal, negative, infinity, NaN
    const uint32_t e = h >> 20, odd = (e & 1) ^ 1;                   // biased 1023 is even in effect
    const uint64_t A = ((v & kFrac) | kHidden) << (10 + odd);        // a 2^62
    const uint32_t y = rsqrt_seed((0x3f800000u + (odd << 23)) | ((uint32_t)(v >> 29) & 0x7fffffu));
    uint64_t g = wide_mad((uint32_t)(A >> 32), y, wide_mul((uint32_t)A, y) >> 32);
    const int32_t r0 = (int32_t)((int64_t)((A >> 2) - mulhi64(g, g)) >> 12);
    g += (uint64_t)(((int64_t)r0 * (int64_t)y) >> 19);
    const int32_t r1 = (int32_t)((A >> 2) - mulhi64(g, g));
    g += (uint64_t)(((int64_t)r1 * (int64_t)y) >> 31);
    uint64_t s = (g + 512) >> 10;
    const int64_t r = (int64_t)((A << 42) - s * s);
    s += (uint64_t)(r > (int64_t)s) - (uint64_t)(r <= -(int64_t)s);
    const uint64_t ex = (uint64_t)((e + 1023 - odd) >> 1) - 1;
    return from_bits((ex << 52) + s);
}

// ---- sums of positive numbers ---------------------------------------------------
// A running sum of positive doubles, rounded after every addition as the FP64
// unit rounds it, with its significand at bits 62..10 of s and 10 zero bits
// below.  Terms within 2^9 of the sum (either way) lose no bit in the
// alignment and leave bit 0 clear for the carry's shift; gap collects the
// largest exponent difference and far the range of the terms, and exact()
// says whether every addition so far was one of these.  About 27 integer
// instructions an addition, which the integer pipes retire in less time than
// the FP64 unit (2 per clock per SM) takes for it, and beside it.
struct PosSum {
    uint64_t s;
    int32_t e;
    uint32_t gap, far;
};

DES_SF_HD void pos_split(double x, uint64_t &m, int32_t &e, uint32_t &far)
{
    const uint64_t b = bits(x);
    const uint32_t h = (uint32_t)(b >> 32), f = h - (64u << 20);
    far = far > f ? far : f;                 // (a negative number is far, too)
    e = (int32_t)(h >> 20);
    m = ((b & kFrac) | kHidden) << 10;
}

DES_SF_HD PosSum pos_first(double x)
{
    PosSum p;
    p.gap = 0;
    p.far = 0;
    pos_split(x, p.s, p.e, p.far);
    return p;
}

DES_SF_HD void pos_add(PosSum &p, double x)
{
    uint64_t m;
    int32_t e;
    pos_split(x, m, e, p.far);
    const int32_t d = p.e - e;
    const uint64_t big = d < 0 ? m : p.s, small = d < 0 ? p.s : m;
    const uint32_t gap = (uint32_t)(d < 0 ? -d : d);
    p.gap = p.gap > gap ? p.gap : gap;
    uint64_t r = big + (small >> (gap & 31));
    const uint32_t t = (uint32_t)(r >> 63);
    r >>= t;
    p.e = (d < 0 ? e : p.e) + (int32_t)t;
    r += 0x1ff + ((uint32_t)(r >> 10) & 1);
    p.s = r & ~0x3ffull;                     // (a carry into bit 63 is one more in the next addition's t)
}

DES_SF_HD bool exact(const PosSum &p) { return p.gap < 10 && p.far < (1900u << 20); }

DES_SF_HD double value(const PosSum &p)
{
    return from_bits((p.s >> 10) + ((uint64_t)(p.e - 1) << 52));
}

// 0.0 + x as the FP64 unit rounds it: x itself, except that -0.0 gives
// +0.0 (a NaN comes back unchanged).  The first addition of a sum that
// starts from zero.
DES_SF_HD double add0(double x)
{
    const uint64_t b = bits(x);
    return from_bits(b == kSign ? 0ull : b);
}

// 2 x and x / 2 (x * 2.0, x * 0.5) as the FP64 unit rounds them: an exponent
// step where the operand and the result are normal, the integer multiply
// otherwise (zeros, subnormals, infinities, NaN, overflow, a subnormal half)
DES_SF_HD double twice(double x)
{
    const uint64_t b = bits(x);
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ff;
    if (e - 1 < 2045u) return from_bits(b + (1ull << 52));
    if ((b & kAbs) == 0) return x;
    return from_bits(mul_slow(b, 0x4000000000000000ull));
}

DES_SF_HD double half(double x)
{
    const uint64_t b = bits(x);
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ff;
    if (e - 2 < 2045u) return from_bits(b - (1ull << 52));
    if ((b & kAbs) == 0) return x;
    return from_bits(mul_slow(b, 0x3fe0000000000000ull));
}

// x / 4 (x * 0.25) as the FP64 unit rounds it
DES_SF_HD double quarter(double x)
{
    const uint64_t b = bits(x);
    const uint32_t e = (uint32_t)(b >> 52) & 0x7ff;
    if (e - 3 < 2044u) return from_bits(b - (2ull << 52));
    if ((b & kAbs) == 0) return x;
    return from_bits(mul_slow(b, 0x3fd0000000000000ull));
}

// x / (3 2^k), k = 0 or 1, for the cases the fast path of div3k leaves:
// zeros, subnormals, operands whose quotient is subnormal, infinities, NaN
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
uint64_t div3k_slow(uint64_t a, int k)
{
    const uint64_t sign = a & kSign, ma = a & kAbs;
    int ea = (int)(ma >> 52);
    if (ea == 2047) return ma > kInf ? (a | kQuiet) : a;
    if (ma == 0) return sign;
    uint64_t m = (ma & kFrac) | (ea ? kHidden : 0);
    if (!ea) {                           // normalise a subnormal significand to bit 52
        const int s = clz64(m) - 11;
        m <<= s;
        ea = 1 - s;
    }
    const uint64_t M = m << 11, q = M / 3, r = M - 3 * q;
    const int t = (int)(q >> 62);        // the quotient's top bit is bit 61 + t
    const uint64_t rr = (q << (2 - t)) | (uint64_t)(r != 0);
    int e = ea - 2 - k + t;
    if (e < 1) {
        const uint32_t sh = (uint32_t)(1 - e) > 63u ? 63u : (uint32_t)(1 - e);
        uint64_t rs = rr >> sh;
        rs |= (uint64_t)((rs << sh) != rr);
        return round_pack(sign, 1, rs);
    }
    return round_pack(sign, e, rr);
}

// x / 3 (k = 0) and x / 6 (k = 1) as the FP64 unit's division rounds them.
// With the significand m (2^52 <= m < 2^53), the quotient of M = m 2^11 by 3
// (an integer division by a constant: a high multiply) holds 62 or 63 bits;
// its top 53 are the result's significand, and the bits below them with the
// remainder of the division (sticky) decide the rounding to nearest even.
template <int k>
DES_SF_HD double div3k(double x)
{
    const uint64_t a = bits(x);
    const uint32_t e = (uint32_t)(a >> 52) & 0x7ff;
    if (e - (3 + k) < 2044u - k) {       // the quotient is normal
        const uint64_t M = ((a & kFrac) | kHidden) << 11;
        const uint64_t q = M / 3, r = M - 3 * q;
        const uint32_t t = (uint32_t)(q >> 62);
        const uint32_t sh = 9 + t;
        const uint64_t sig = q >> sh, rem = q & ((1ull << sh) - 1), hf = 1ull << (sh - 1);
        const uint64_t up = (uint64_t)((rem > hf) | ((rem == hf) & ((r != 0) | (uint32_t)(sig & 1))));
        return from_bits(((((uint64_t)(e - 3 - k + t)) << 52) + sig + up) | (a & kSign));
    }
    return from_bits(div3k_slow(a, k));
}

DES_SF_HD double div3(double x) { return div3k<0>(x); }
DES_SF_HD double div6(double x) { return div3k<1>(x); }

// the cases the fast path of to_float leaves: zeros, subnormal FP32
// results, infinities, NaN, overflow
#if defined(__CUDACC__)
static __host__ __device__ __noinline__
#else
static
#endif
uint32_t to_float_slow(uint64_t a)
{
    const uint32_t sign = (uint32_t)(a >> 32) & 0x80000000u;
    const int e = (int)((a >> 52) & 0x7ff);
    if (e == 2047) return (a & kFrac) ? 0x7fffffffu : (sign | 0x7f800000u);
    if (e - 896 >= 255) return sign | 0x7f800000u;
    // FP32 subnormal or zero: k = round(significand / 2^(926 - e)) units of 2^-149
    const int sh = 926 - e;
    if (sh >= 54) return sign;
    const uint64_t f = (a & kFrac) | kHidden;
    const uint64_t k = f >> sh, rem = f & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    const uint64_t up = (uint64_t)((rem > half) | ((rem == half) & (uint32_t)k));
    return sign | (uint32_t)(k + up);
}

// (float)x, round to nearest even, as the FP64 unit converts it
// (10 instructions; with the rounding as comparisons and selects 15, and the FP32
// form's E-A, 17 conversions an element, 228 instead of 221 us for 2.4M elements)
DES_SF_HD float to_float(double x)
{
    const uint64_t a = bits(x);
    const uint32_t hi = (uint32_t)(a >> 32), lo = (uint32_t)a;
    if ((hi & 0x7fffffffu) - (897u << 20) < (254u << 20)) {
        // half a unit less a bit, plus the unit's parity, added below the 24
        // bits that stay; the exponent's upper bits leave with the shift
        const uint64_t r = a + (0x0fffffffu + ((lo >> 29) & 1));
        return float_from_bits((hi & 0x80000000u) | (((uint32_t)(r >> 29) - (896u << 23)) & 0x7fffffffu));
    }
    return float_from_bits(to_float_slow(a));
}

// (double)x, exact
DES_SF_HD double widen(float x)
{
#if defined(__CUDA_ARCH__)
    const uint32_t b = __float_as_uint(x);
#else
    uint32_t b;
    memcpy(&b, &x, 4);
#endif
    const uint32_t e = (b >> 23) & 0xff;
    if (e - 1 < 254u)
        return from_bits(((uint64_t)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))) << 32) |
                         ((uint64_t)(b & 7u) << 29));
    const uint64_t sign = (uint64_t)(b & 0x80000000u) << 32, f = b & 0x7fffffu;
    if (e) return from_bits(sign | (f ? 0x7fffffffe0000000ull : kInf));   // an infinity or NaN
    if (!f) return from_bits(sign);
    const int k = clz32((uint32_t)f);        // a subnormal: f 2^-149 with its top bit at 31 - k
    return from_bits(sign | ((uint64_t)(905 - k) << 52) | ((f << (k + 21)) & kFrac));
}

}  // namespace sf
}  // namespace des
