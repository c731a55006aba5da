// nx_f64.cuh -- correctly rounded binary64 quotients and square roots with
// one binary64 operation each.
//
// GB300 issues two binary64 operations per SM and cycle against 128 binary32
// ones, so a correctly rounded division or square root (about ten binary64
// operations) costs as much as hundreds of binary32 instructions, and the
// kernels that need the reference's exact binary64 results (mesh vertices,
// edge lengths, height shaping) are bound by them.  Here:
//  * the quotient or root is approximated by a pair of binary32s (a
//    reciprocal or reciprocal square root estimate and one residual step),
//    within 2^-44.5 (quotient) or 2^-43.5 (root);
//  * the pair's sum is put together as a binary64 G by integer operations;
//  * one fused multiply-add gives the residual r = a - G b or s - G^2;
//  * r / b or r / (2 G), in binary32 and in units of G's last place (below
//    2^8.5 or 2^9.5, and within 2^-21 of itself: an estimate of 2^-22, a
//    truncation to 24 bits and two products), is rounded to the integer by
//    which G's bits move.
// The result is the correctly rounded one unless that quotient lies within
// its error of a half (2^-11 and 2^-10 are kept), or a power of two lies
// between the pair's leading part, G and the result; then, and for operands outside the ranges below (zeros among
// them), the function calls the binary64 operation.
// Measured (GB300, throughput of a loop of them, 10^10 results bit for bit
// equal to the binary64 operations'): quotients 70 -> 362 G/s, roots 67 ->
// 367 G/s, pairs 134 -> 779 G/s; a binary64 product alone 392 G/s.
#pragma once

#include <cstdint>

namespace nxf {

// v's bits, by a move the compiler does not see through: it turns integer
// tests of a binary64's bits (for NaN, for the sign) back into binary64
// comparisons, which take a slot of the narrow pipe each.
__device__ __forceinline__ uint2 words(double v)
{
    uint2 w;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(w.x), "=r"(w.y) : "d"(v));
    return w;
}

__device__ __forceinline__ unsigned long long bits(double v)
{
    unsigned long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(v));
    return b;
}

// c ? a : b, word by word: a select of binary64s is moved by the compiler
// past the operation that follows, which is then carried out for both.
__device__ __forceinline__ double pick(bool c, double a, double b)
{
    const uint2 u = words(a), v = words(b);
    double r;
    asm("mov.b64 %0, {%1, %2};" : "=d"(r) : "r"(c ? u.x : v.x), "r"(c ? u.y : v.y));
    return r;
}

// |v|'s high word -> h + l, binary32s: h the top 24 bits (truncated), l the
// next 23; for 2^-80 <= |v| < 2^127.
__device__ __forceinline__ void split_abs(uint32_t ah, uint32_t lw, float &h, float &l)
{
    h = __uint_as_float(__funnelshift_l(lw, ah - (896u << 20), 3));
    const float i = __fsub_rn(__uint_as_float(0x4B000000u | ((lw >> 6) & 0x7FFFFFu)), 8388608.0f);
    l = __fmul_rn(i, __uint_as_float(((ah & 0x7FF00000u) - (942u << 20)) << 3));
}

// r as a binary32, truncated; 0 below 2^-126.
__device__ __forceinline__ float chop(double r)
{
    const uint2 w = words(r);
    const uint32_t hw = w.y, ah = hw & 0x7FFFFFFFu;
    const uint32_t f = __funnelshift_l(w.x, ah - (896u << 20), 3);
    return __uint_as_float(ah < (897u << 20) ? 0u : (f | (hw & 0x80000000u)));
}

// h + l as binary64 bits (h > 0 of 24 bits, |l| <= ulp(h)), l rounded to
// h's binary64 grid; scale = 1 / that grid's step, 2^52 / 2^exponent(h).
__device__ __forceinline__ unsigned long long join(float h, float l, float &scale)
{
    const uint32_t hb = __float_as_uint(h);
    scale = __uint_as_float((306u - (hb >> 23)) << 23);
    const unsigned long long b = ((unsigned long long)((hb >> 3) + (896u << 20)) << 32) | (hb << 29);
    return b + (unsigned long long)(long long)__float2int_rn(__fmul_rn(l, scale));
}

// G's bits moved by c steps of its grid; false when c is within `near` of a
// half or G or the result has another exponent than h (the grid is h's).
__device__ __forceinline__ bool settle(unsigned long long &g, float h, float c, float near)
{
    const float n = rintf(c);
    const unsigned long long m = g + (unsigned long long)(long long)(int)n;
    const uint32_t e = (__float_as_uint(h) >> 23) + 896u;
    const bool ok = fabsf(fabsf(__fsub_rn(c, n)) - 0.5f) > near && (uint32_t)(m >> 52) == e && (uint32_t)(g >> 52) == e;
    g = m;
    return ok;
}

// a * w, rounded to nearest even, for an integer 0 <= w < 2^31 and |a| in
// [2^-900, 2^900] or 0: the product of the 53-bit significand and w as an
// integer of at most 84 bits, rounded by hand (a binary64 product costs as
// many issue slots as three of these).
__device__ __forceinline__ double times(double a, int w)
{
    const uint2 x = words(a);
    const uint32_t sign = x.y & 0x80000000u;
    if (w == 0 || ((x.y << 1) | x.x) == 0u) return __hiloint2double((int)sign, 0);
    const unsigned long long lo = (unsigned long long)x.x * (uint32_t)w;
    const unsigned long long hi = (unsigned long long)((x.y & 0xFFFFFu) | 0x100000u) * (uint32_t)w + (lo >> 32);
    // p = hi : low word of lo, with its top bit at 52 + d, d = that of w (or one more)
    const int d = 43 - __clzll((long long)hi);              // shift of the significand, 0 .. 31
    const uint32_t l = (uint32_t)lo;
    unsigned long long m;
    if (d == 0) {
        m = (hi << 32) | l;
    } else {
        m = (hi << (32 - d)) | (l >> d);
        const uint32_t rest = l << (32 - d);
        m += rest > 0x80000000u || (rest == 0x80000000u && (m & 1ull)) ? 1ull : 0ull;
    }
    // (the implicit bit adds 1 to the exponent field; a carry out of the
    // rounding adds one more)
    const uint32_t e = ((x.y >> 20) & 0x7FFu) + (uint32_t)d - 1u;
    const unsigned long long b = m + ((unsigned long long)e << 52);
    return __longlong_as_double((long long)(b | ((unsigned long long)sign << 32)));
}

// A factor b for mul: its significand in the top 53 bits of m (0: b outside
// [2^-500, 2^500), products take the binary64 pipe).
struct Factor {
    double b;
    unsigned long long m;
    uint32_t hw;
};

__device__ __forceinline__ Factor factor(double b)
{
    const uint2 w = words(b);
    const bool in = ((w.y >> 20) & 0x7FFu) - 523u < 1000u;
    return Factor{b, in ? ((unsigned long long)((w.y & 0xFFFFFu) | 0x100000u) << 43) | ((unsigned long long)w.x << 11) : 0ull, w.y};
}

static __device__ __noinline__ double mul_slow(double a, double b) { return __dmul_rn(a, b); }

// a * F.b, correctly rounded, without the binary64 pipe: the top 64 bits of
// the significands' product round to 53 whatever the others are unless they
// end in a half exactly (one in 2^11, then and outside the ranges the
// binary64 product).  About 28 integer operations, half the pipe's 16 cycles
// of a warp where the others are free.
__device__ __forceinline__ double mul(double a, const Factor &F)
{
    const uint2 w = words(a);
    const uint32_t e = (w.y >> 20) & 0x7FFu;
    if (e - 523u < 1000u && F.m) {
        const unsigned long long A = ((unsigned long long)((w.y & 0xFFFFFu) | 0x100000u) << 43) | ((unsigned long long)w.x << 11);
        const unsigned long long hi = __umul64hi(A, F.m);            // in [2^62, 2^64)
        const uint32_t top = (uint32_t)(hi >> 63);
        const unsigned long long x = top ? hi : hi << 1;
        if (((uint32_t)x & 0x7FFu) != 0x400u) {
            const unsigned long long m = (x >> 11) + (((uint32_t)x >> 10) & 1u);
            // (m's leading bit adds 1 to the exponent field)
            const uint32_t field = e + ((F.hw >> 20) & 0x7FFu) - 1024u + top;
            const unsigned long long b = m + ((unsigned long long)(field | ((w.y ^ F.hw) >> 20 & 0x800u)) << 52);
            return __longlong_as_double((long long)b);
        }
    }
    return mul_slow(a, F.b);
}

// a * a, as mul.
__device__ __forceinline__ double square(double a)
{
    const uint2 w = words(a);
    const uint32_t e = (w.y >> 20) & 0x7FFu;
    if (e - 523u < 1000u) {
        const unsigned long long A = ((unsigned long long)((w.y & 0xFFFFFu) | 0x100000u) << 43) | ((unsigned long long)w.x << 11);
        const unsigned long long hi = __umul64hi(A, A);
        const uint32_t top = (uint32_t)(hi >> 63);
        const unsigned long long x = top ? hi : hi << 1;
        if (((uint32_t)x & 0x7FFu) != 0x400u)
            return __longlong_as_double((long long)((x >> 11) + (((uint32_t)x >> 10) & 1u) +
                                                    ((unsigned long long)(2u * e - 1024u + top) << 52)));
    }
    return mul_slow(a, a);
}

static __device__ __noinline__ double div_slow(double a, double b) { return __ddiv_rn(a, b); }
static __device__ __noinline__ double sqrt_slow(double s) { return __dsqrt_rn(s); }

// 1 / b as a pair y1 + y2 (relative error below 2^-44); y1 = 0 for b outside
// [2^-28, 2^28).
struct Recip {
    double b;
    float y1, y2;
};

__device__ __forceinline__ Recip recip(double b)
{
    Recip R;
    R.b = b;
    R.y1 = R.y2 = 0.0f;
    const uint32_t hw = words(b).y;
    if (hw < (995u << 20) || hw >= (1051u << 20)) return R;     // (a set sign bit makes hw large)
    float h, l;
    split_abs(hw, words(b).x, h, l);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(R.y1) : "f"(h));   // within 2^-23
    // 1/b = y1 (1 + t + t^2 + ...), t = 1 - b y1 below 2^-22
    const float t = __fmaf_rn(-l, R.y1, __fmaf_rn(-h, R.y1, 1.0f));
    R.y2 = __fmul_rn(R.y1, __fmaf_rn(t, t, t));
    return R;
}

// a / R.b, correctly rounded (|a| in [2^-44, 2^44) without the slow call).
__device__ __forceinline__ double div(double a, const Recip &R)
{
    const uint2 w = words(a);
    const uint32_t hw = w.y, ah = hw & 0x7FFFFFFFu, lw = w.x;
    if (ah - (979u << 20) < (88u << 20) && R.y1 > 0.0f) {
        float a1, a2;
        split_abs(ah, lw, a1, a2);
        const float p = __fmul_rn(a1, R.y1);
        const float e = __fmaf_rn(a2, R.y1, __fmaf_rn(a1, R.y2, __fmaf_rn(a1, R.y1, -p)));
        const float h = __fadd_rn(p, e), l = __fsub_rn(e, __fsub_rn(h, p));
        float scale;
        unsigned long long g = join(h, l, scale);
        const double r = __fma_rn(-__longlong_as_double((long long)g), R.b, __hiloint2double((int)ah, (int)lw));
        if (settle(g, h, __fmul_rn(__fmul_rn(chop(r), R.y1), scale), 0x1p-11f))
            return __longlong_as_double((long long)(g | ((unsigned long long)(hw & 0x80000000u) << 32)));
    }
    return div_slow(a, R.b);
}

// sqrt(s), correctly rounded (s in [2^-60, 2^60) without the slow call).
__device__ __forceinline__ double sqrt(double s)
{
    const uint32_t hw = words(s).y;
    if (hw - (963u << 20) < (120u << 20)) {
        float s1, s2, y;
        split_abs(hw, words(s).x, s1, s2);
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s1));    // within 2^-22
        const float p = __fmul_rn(s1, y), y2 = __fmul_rn(0.5f, y);
        // s - p^2 below 2^-20 s: its rounding and the neglected square of
        // the step leave 2^-42
        const float e = __fmul_rn(__fadd_rn(__fmaf_rn(-p, p, s1), s2), y2);
        const float h = __fadd_rn(p, e), l = __fsub_rn(e, __fsub_rn(h, p));
        float scale;
        unsigned long long g = join(h, l, scale);
        const double G = __longlong_as_double((long long)g);
        const double r = __fma_rn(-G, G, s);
        if (settle(g, h, __fmul_rn(__fmul_rn(chop(r), y2), scale), 0x1p-10f)) return __longlong_as_double((long long)g);
    }
    return sqrt_slow(s);
}

// d as a pair hi + lo of binary32s, both rounded to nearest (|d| in [2^-60,
// 2^60), else by conversion): hi by integer rounding of the top 24 bits, lo =
// the rest, an integer of at most 29 bits times its last place.
__device__ __forceinline__ float2 pair(double d)
{
    const uint2 w = words(d);
    const uint32_t sign = w.y & 0x80000000u, hw = w.y & 0x7FFFFFFFu, lw = w.x;
    if (hw - (963u << 20) < (120u << 20)) {
        const uint32_t t = __funnelshift_l(lw, hw - (896u << 20), 3), rem = lw & 0x1FFFFFFFu;
        const bool up = rem > 0x10000000u || (rem == 0x10000000u && (t & 1u));
        const int r = up ? (int)rem - 0x20000000 : (int)rem;
        return make_float2(__uint_as_float((t + (up ? 1u : 0u)) | sign),
                           __fmul_rn(__int2float_rn(sign ? -r : r), __uint_as_float((((hw >> 20) & 0x7FFu) - 948u) << 23)));
    }
    const float h = (float)d;
    return make_float2(h, (float)(d - (double)h));
}

}  // namespace nxf
