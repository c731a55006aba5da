// nx_noise.cu -- fused fractal OpenSimplex-3D noise (fBm) for sm_103a.
//
// Replaces terrain.sample_octaves / terrain.sample_noise (terrain.py:12-59)
// over opensimplex.noise3d (opensimplex.py:266-759).
//
// Design
//  * One thread per vertex, all octaves in registers; persistent grid of
//    (#SM x resident CTAs) walking the vertex range.
//  * The seeded tables live in shared memory as one packed word per entry
//    (perm in bits 7-14, the gradient's byte offset above), replicated 32
//    times (entry k of lane l at word 32*k + l) so the three dependent hash
//    loads of a warp never conflict on a bank; the gradients are binary32,
//    one copy per lane too.
//  * Arithmetic is binary32.  The lattice cell, the region and the two extra
//    lattice points must equal what binary64 decides.  The large-magnitude
//    part of the skew is removed exactly: x*scale is formed as a float pair,
//    split into an integer A and a fraction a in [-1/2, 1/2], and with
//    T = Ax+Ay+Az = 6q + r the skewed coordinate becomes
//    xs = (Ax - q) + (a_x - (r + a_x + a_y + a_z)/6), whose second term is
//    O(1) and carries an absolute error of at most 2.2e-7 for
//    |x*scale| < 2^16 (the bound is worked through at decide_f32).  Every
//    comparison that decides the cell or region records its margin; the
//    compared quantities combine up to three such terms with a few more
//    roundings (errors below 1.6e-6), and when the smallest margin is below
//    TAU = 4e-6 (2.5x that), or |x*scale| >= 2^16, that lane recomputes the
//    decisions in binary64 with the reference's operation order
//    (decide_f64), so the decisions always equal the reference's.
//  * The 6 or 8 contributions are evaluated branch-free as four pairs of
//    slots: a region's first four fixed corners (offsets from a table by
//    region), the octahedron's other two (masked), the two extra points
//    (offsets and hash steps from a table by case); hash prefixes of the
//    fixed slots are shared.
//  * Both kernels are bound by instruction issue (binary32: 81 % of the slots,
//    320 instructions per vertex and octave) and, in pairs, as much by the FMA
//    pipe (68 %).  Measured on 10,000,002 vertices x 12 octaves: case numbers
//    from sign bits and cases SoA 1570 -> 1385 us in binary32 and 3131 -> 2969
//    in pairs, slots by region 1385 -> 1299 (binary32), gradients by single
//    loads, tables in operand order and the rest of the shorter chain 1299 ->
//    1184 and 2965 -> 2750.  Skipping the octahedron's pair where no lane
//    needs it: 1226 and 2750 (nearly every warp has one).
#include "nx_common.cuh"

#include <vector>

#include <cmath>

namespace {

constexpr float MAGIC = 12582912.0f;   // 1.5 * 2^23: v + MAGIC rounds v to an integer, |v| < 2^22
constexpr int MAGIC_BITS = 0x4B400000;
constexpr float TAU = 4.0e-6f;         // decision margin below which binary64 decides
constexpr float PMAX = 65536.0f;       // |x*scale| bound of the binary32 decision path
constexpr float THIRD = 1.0f / 3.0f;
constexpr float SIXTH = 1.0f / 6.0f;

// opensimplex.py:51-60 (GRADIENTS_3D), used only to build the packed table.
__constant__ int c_grad3[72] = {
    -11, 4, 4, -4, 11, 4, -4, 4, 11,
    11, 4, 4, 4, 11, 4, 4, 4, 11,
    -11, -4, 4, -4, -11, 4, -4, -4, 11,
    11, -4, 4, 4, -11, 4, 4, -4, 11,
    -11, 4, -4, -4, 11, -4, -4, 4, -11,
    11, 4, -4, 4, 11, -4, 4, 4, -11,
    -11, -4, -4, -4, -11, -4, -4, -4, -11,
    11, -4, -4, 4, -11, -4, 4, -4, -11,
};

struct FbmParams {
    int n_oct;
    float s_hi[NX_MAX_OCTAVES];   // scale[o] as a binary32 pair
    float s_lo[NX_MAX_OCTAVES];
    float amp[NX_MAX_OCTAVES];    // 0.5 * strength[o] * radius / 103
    float base;                   // sum over octaves of 0.5 * strength[o] * radius
    double s[NX_MAX_OCTAVES];     // scale[o] (binary64 decision path)
};

static_assert(sizeof(nx_fbm_planet) == 960, "fBm planet descriptor layout");

constexpr int TABLE_WORDS = 256 * 32;
constexpr int TABLE_BYTES = TABLE_WORDS * 4;

// GRADIENTS_3D as binary32, a copy per lane (no bank conflicts).  Three
// single loads a slot go straight into the halves of the paired operands; one
// 16-byte load took moves to get there.  Two layouts of the same size:
//  * binary32 kernels: the table's 72 numbers in its own order, number q of a
//    lane at 32 q + lane, so that a gradient starts at any of them, as the
//    reference's GRADIENTS_3D[index], [index + 1], [index + 2] do (init() makes
//    multiples of 3 only, other tables need not);
//  * AXIS, the pair kernels: component c of gradient i at 768 c + 32 i + lane,
//    the gradients in the order of the component that is +-11, i = 8 axis +
//    (0-7) (every gradient has one +-11 and two +-4 components); indices are
//    rounded down to a multiple of 3.
__shared__ float s_gr[3 * 768];

template <bool AXIS>
__device__ __forceinline__ void init_grad_table()
{
    if (!AXIS) {
        for (int j = threadIdx.x; j < 72 * 32; j += blockDim.x) s_gr[j] = (float)c_grad3[j >> 5];
        return;
    }
    for (int j = threadIdx.x; j < 768; j += blockDim.x) {
        const int i = j >> 5, row = 3 * (i & 7) + (i >> 3);
        for (int c = 0; c < 3; ++c) s_gr[768 * c + j] = (float)c_grad3[3 * row + c];
    }
}

// The hash table (TABLE_WORDS), at the start of the block's dynamic memory.
// A lane's word of an entry: perm in bits 7-14, and from bit 18 on the byte
// offset of the entry's gradient in s_gr for this lane, 128 i + 4 lane, i the
// index itself or (AXIS) the gradient's place, whose axis is then bits 26-27.
extern __shared__ __align__(16) uint32_t smem[];

// A warp fills runs of 32 entries: each lane forms one entry's word (two
// global reads a lane, all in flight together), then the 32 words go out one
// by one to their 32 replicas, a conflict-free store each.
template <bool AXIS>
__device__ __forceinline__ void build_table(const int32_t *__restrict__ perm, const int32_t *__restrict__ pgi)
{
    const uint32_t lane = threadIdx.x & 31;
    for (int k0 = (threadIdx.x >> 5) * 32; k0 < 256; k0 += blockDim.x) {
        const uint32_t p = (uint32_t)perm[k0 + lane] & 255u;
        int g = pgi[k0 + lane];
        g = g < 0 ? 0 : (g > 69 ? 69 : g);
        if (AXIS) g = 8 * (g / 3 % 3) + g / 9;
        const uint32_t w = p << 7 | (uint32_t)g << 23;
#pragma unroll 8
        for (int j = 0; j < 32; ++j) smem[32 * (k0 + j) + lane] = __shfl_sync(0xFFFFFFFFu, w, j) | lane << 18;
    }
}

// Hash table load: bits 7-14 of a select the entry; lb = this lane's byte
// offset in an entry's 32 words.  The table's own address goes into the
// load, so an address is one three-input logic operation (19 lookups per
// vertex and octave).
__device__ __forceinline__ uint32_t lk(uint32_t lb, int a)
{
    return *reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(smem) + (((uint32_t)a & 0x7F80u) | lb));
}

// Component c of the gradient of a table word.
template <bool AXIS>
__device__ __forceinline__ float grad_of(uint32_t w, int c)
{
    return *reinterpret_cast<const float *>(reinterpret_cast<const char *>(s_gr + (AXIS ? 768 : 32) * c) + (w >> 16));
}

// Split a binary64 into hi + lo binary32 with integer operations (no FP64
// unit): hi = value truncated to 24 significant bits, lo = the next 23 bits.
// |x - (hi+lo)| <= 2^-47 |x|.  Magnitudes outside [2^-74, 2^127] give lo = 0
// (and hi = +-0 or +-inf); such lanes take the binary64 path anyway.
__device__ __forceinline__ void split_f64(double v, float &hi, float &lo)
{
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    uint32_t hw = (uint32_t)(b >> 32), lw = (uint32_t)b;
    int e = (int)((hw >> 20) & 0x7FF) - 1023;
    uint32_t sign = hw & 0x80000000u;
    if (e < -126) { hi = __uint_as_float(sign); lo = 0.0f; return; }
    if (e > 127) { hi = __uint_as_float(sign | 0x7F800000u); lo = 0.0f; return; }
    uint32_t top = ((hw & 0xFFFFFu) << 3) | (lw >> 29);
    hi = __uint_as_float(sign | ((uint32_t)(e + 127) << 23) | top);
    if (e < -74 + 6) { lo = 0.0f; return; }
    // remainder bits 28..6 of the low word, as 23-bit integer times 2^(e-46)
    uint32_t rem = (lw & 0x1FFFFFFFu) >> 6;
    float r = __uint_as_float(0x4B000000u | rem) - 8388608.0f;    // exact
    float sc = __uint_as_float((uint32_t)(e - 46 + 127) << 23);
    lo = __uint_as_float(__float_as_uint(r * sc) | sign);
}

// Decisions of noise3d (opensimplex.py:302-700) in either precision.  For
// float, `m` tracks the smallest |a-b| over the comparisons on the taken
// path; for double it is unused.  Extra-point offsets are relative to the
// cell origin (components in {-1,0,1,2}).
struct Decision {
    int region;
    float e0x, e0y, e0z, e1x, e1y, e1z;   // decide() only
    uint32_t w0, w1;                      // step words of the two extra points (pack_step)
    float E[6];                           // displacement offsets e + (ex + ey + ez) / 3 of both points
};

__device__ __forceinline__ void decide(double xins, double yins, double zins, double in_sum, Decision &D)
{
    using T = double;
    const T one = (T)1, two = (T)2, three = (T)3;
    if (in_sum <= one) {
        // tetrahedron at (0,0,0): closest two of (1,0,0), (0,1,0), (0,0,1)
        D.region = 0;
        int ap = 1, bp = 2;
        T as = xins, bs = yins;
        if (as >= bs) {
            if (zins > bs) { bs = zins; bp = 4; }
        } else {
            if (zins > as) { as = zins; ap = 4; }
        }
        T wins = one - in_sum;
        bool near0 = wins > as;
        if (!near0) near0 = wins > bs;
        if (near0) {
            int c = (bs > as) ? bp : ap;
            if ((c & 1) == 0) { D.e0x = -1.f; D.e1x = 0.f; } else { D.e0x = 1.f; D.e1x = 1.f; }
            if ((c & 2) == 0) {
                D.e0y = 0.f; D.e1y = 0.f;
                if ((c & 1) == 0) D.e1y = -1.f; else D.e0y = -1.f;
            } else { D.e0y = 1.f; D.e1y = 1.f; }
            if ((c & 4) == 0) { D.e0z = 0.f; D.e1z = -1.f; } else { D.e0z = 1.f; D.e1z = 1.f; }
        } else {
            int c = ap | bp;
            if ((c & 1) == 0) { D.e0x = 0.f; D.e1x = -1.f; } else { D.e0x = 1.f; D.e1x = 1.f; }
            if ((c & 2) == 0) { D.e0y = 0.f; D.e1y = -1.f; } else { D.e0y = 1.f; D.e1y = 1.f; }
            if ((c & 4) == 0) { D.e0z = 0.f; D.e1z = -1.f; } else { D.e0z = 1.f; D.e1z = 1.f; }
        }
    } else if (in_sum >= two) {
        // tetrahedron at (1,1,1): closest two of (1,1,0), (1,0,1), (0,1,1)
        D.region = 1;
        int ap = 6, bp = 5;
        T as = xins, bs = yins;
        if (as <= bs) {
            if (zins < bs) { bs = zins; bp = 3; }
        } else {
            if (zins < as) { as = zins; ap = 3; }
        }
        T wins = three - in_sum;
        bool near1 = wins < as;
        if (!near1) near1 = wins < bs;
        if (near1) {
            int c = (bs < as) ? bp : ap;
            if ((c & 1) != 0) { D.e0x = 2.f; D.e1x = 1.f; } else { D.e0x = 0.f; D.e1x = 0.f; }
            if ((c & 2) != 0) {
                D.e0y = 1.f; D.e1y = 1.f;
                if ((c & 1) != 0) D.e1y = 2.f; else D.e0y = 2.f;
            } else { D.e0y = 0.f; D.e1y = 0.f; }
            if ((c & 4) != 0) { D.e0z = 1.f; D.e1z = 2.f; } else { D.e0z = 0.f; D.e1z = 0.f; }
        } else {
            int c = ap & bp;
            if ((c & 1) != 0) { D.e0x = 1.f; D.e1x = 2.f; } else { D.e0x = 0.f; D.e1x = 0.f; }
            if ((c & 2) != 0) { D.e0y = 1.f; D.e1y = 2.f; } else { D.e0y = 0.f; D.e1y = 0.f; }
            if ((c & 4) != 0) { D.e0z = 1.f; D.e1z = 2.f; } else { D.e0z = 0.f; D.e1z = 0.f; }
        }
    } else {
        // octahedron between them
        D.region = 2;
        T as, bs, score;
        int ap, bp;
        bool af, bf;
        T p1 = xins + yins;
        if (p1 > one) { as = p1 - one; ap = 3; af = true; }
        else { as = one - p1; ap = 4; af = false; }
        T p2 = xins + zins;
        if (p2 > one) { bs = p2 - one; bp = 5; bf = true; }
        else { bs = one - p2; bp = 2; bf = false; }
        T p3 = yins + zins;
        bool t3 = p3 > one;
        score = t3 ? p3 - one : one - p3;
        if (as <= bs) {
            if (as < score) { ap = t3 ? 6 : 1; af = t3; }
        } else {
            if (bs < score) { bp = t3 ? 6 : 1; bf = t3; }
        }
        if (af == bf) {
            if (af) {
                D.e0x = 1.f; D.e0y = 1.f; D.e0z = 1.f;
                int c = ap & bp;
                if (c & 1) { D.e1x = 2.f; D.e1y = 0.f; D.e1z = 0.f; }
                else if (c & 2) { D.e1x = 0.f; D.e1y = 2.f; D.e1z = 0.f; }
                else { D.e1x = 0.f; D.e1y = 0.f; D.e1z = 2.f; }
            } else {
                D.e0x = 0.f; D.e0y = 0.f; D.e0z = 0.f;
                int c = ap | bp;
                if ((c & 1) == 0) { D.e1x = -1.f; D.e1y = 1.f; D.e1z = 1.f; }
                else if ((c & 2) == 0) { D.e1x = 1.f; D.e1y = -1.f; D.e1z = 1.f; }
                else { D.e1x = 1.f; D.e1y = 1.f; D.e1z = -1.f; }
            }
        } else {
            int c1 = af ? ap : bp;
            int c2 = af ? bp : ap;
            if ((c1 & 1) == 0) { D.e0x = -1.f; D.e0y = 1.f; D.e0z = 1.f; }
            else if ((c1 & 2) == 0) { D.e0x = 1.f; D.e0y = -1.f; D.e0z = 1.f; }
            else { D.e0x = 1.f; D.e0y = 1.f; D.e0z = -1.f; }
            D.e1x = 0.f; D.e1y = 0.f; D.e1z = 0.f;
            if (c2 & 1) D.e1x = 2.f;
            else if (c2 & 2) D.e1y = 2.f;
            else D.e1z = 2.f;
        }
    }
}


// The extra points' offsets of a case, o[0..2] and o[3..5], from the signs of
// the comparisons' differences (1: negative).  Octahedron (opensimplex.py:
// 535-700): bit 5 p1 - 1, 4 p2 - 1, 3 p3 - 1, 2 |p1-1| - |p2-1|, 1 |p1-1| -
// |p3-1|, 0 |p2-1| - |p3-1|.  Offsets are in {-1, 0, 1, 2}; a block tabulates
// every case once (s_extra) and the per-lane decision looks its case up.
__device__ __forceinline__ void octa_case(int b, float *o)
{
    const bool g1 = !(b & 32), g2 = !(b & 16), t3 = !(b & 8), ale = b & 4, a_lt = b & 2, b_lt = b & 1;
    const bool swa = ale && a_lt, swb = !ale && b_lt;
    const int oap = swa ? (t3 ? 6 : 1) : (g1 ? 3 : 4);
    const int obp = swb ? (t3 ? 6 : 1) : (g2 ? 5 : 2);
    const bool af = swa ? t3 : g1, bf = swb ? t3 : g2;
    float o0x, o0y, o0z, o1x, o1y, o1z;
    if (af == bf) {
        const int c = af ? (oap & obp) : (oap | obp);
        const float b = af ? 1.f : 0.f;
        o0x = b; o0y = b; o0z = b;
        // af: the single bit of c picks the axis that gets 2; otherwise the
        // first axis whose bit is clear gets -1 and the others 1
        const bool c1 = (c & 1) != 0, c2 = (c & 2) != 0;
        const bool ax = af ? c1 : !c1, ay = af ? (!c1 && c2) : (c1 && !c2);
        const bool az = !ax && !ay;
        const float hit = af ? 2.f : -1.f, miss = af ? 0.f : 1.f;
        o1x = ax ? hit : miss; o1y = ay ? hit : miss; o1z = az ? hit : miss;
    } else {
        const int c1 = af ? oap : obp, c2 = af ? obp : oap;
        const bool bx = (c1 & 1) == 0, by = !bx && (c1 & 2) == 0;
        const bool bz = !bx && !by;
        o0x = bx ? -1.f : 1.f; o0y = by ? -1.f : 1.f; o0z = bz ? -1.f : 1.f;
        const bool qx = (c2 & 1) != 0, qy = !qx && (c2 & 2) != 0;
        const bool qz = !qx && !qy;
        o1x = qx ? 2.f : 0.f; o1y = qy ? 2.f : 0.f; o1z = qz ? 2.f : 0.f;
    }
    o[0] = o0x; o[1] = o0y; o[2] = o0z; o[3] = o1x; o[4] = o1y; o[5] = o1z;
}

// Tetrahedra (opensimplex.py:302-533): bit 4 in_sum - 2 (clear: region 1), 3
// x - y, 2 y - z, 1 x - z, 0 wins - the middle one of x, y, z.  The two scores
// the reference compares with wins are the two largest (region 1: smallest),
// so one of them is passed where the middle one is, and which of the two is
// the larger (smaller) follows from the order.  Region 1's comparisons are
// region 0's with both sides negated and its offsets t become 1 - t.
__device__ __forceinline__ void tetra_case(int b, float *o)
{
    const bool r1 = !(b & 16);
    const bool xy = r1 == ((b & 8) != 0), zb = r1 != ((b & 4) != 0), za = r1 != ((b & 2) != 0);   // x >= y, z > y, z > x
    const bool near = r1 == ((b & 1) != 0);
    const bool repb = xy && zb, repa = !xy && za;
    const bool cnb = repb ? za : (repa ? !zb : !xy);
    const int ap = repa ? 4 : 1, bp = repb ? 4 : 2;
    const int cn = cnb ? bp : ap;
    const int cf = ap | bp;
    const bool cn1 = (cn & 1) != 0, cn2 = (cn & 2) != 0, cn4 = (cn & 4) != 0;
    float t[6];
    t[0] = near ? (cn1 ? 1.f : -1.f) : ((cf & 1) ? 1.f : 0.f);
    t[3] = near ? (cn1 ? 1.f : 0.f) : ((cf & 1) ? 1.f : -1.f);
    t[1] = near ? (cn2 ? 1.f : (cn1 ? -1.f : 0.f)) : ((cf & 2) ? 1.f : 0.f);
    t[4] = near ? (cn2 ? 1.f : (cn1 ? 0.f : -1.f)) : ((cf & 2) ? 1.f : -1.f);
    t[2] = near ? (cn4 ? 1.f : 0.f) : ((cf & 4) ? 1.f : 0.f);
    t[5] = near ? (cn4 ? 1.f : -1.f) : ((cf & 4) ? 1.f : -1.f);
    for (int k = 0; k < 6; ++k) o[k] = r1 ? 1.f - t[k] : t[k];
}

// Cases: [0, 64) octahedron, [64, 96) tetrahedra.
constexpr int CASES = 96;
__device__ __forceinline__ void extra_case(int i, float *o)
{
    if (i < 64) octa_case(i, o); else tetra_case(i - 64, o);
}

// An extra point's offsets + 1 as steps of a hash address (bits 7-14): x at
// bit 7, y at bit 16, z at bit 25, so that w, w >> 9 and w >> 18 each have
// theirs at bit 7, nothing below it, and the rest above bit 14, which the
// lookup masks away.
__device__ __forceinline__ uint32_t pack_step(float ox, float oy, float oz)
{
    return (uint32_t)((int)ox + 1) << 7 | (uint32_t)((int)oy + 1) << 16 | (uint32_t)((int)oz + 1) << 25;
}

__device__ __forceinline__ int step_offset(uint32_t w, int axis)
{
    return (int)((w >> (7 + 9 * axis)) & 3u) - 1;
}

// The displacement offsets of an extra point o: o + (ox + oy + oz) / 3
// per component (the point's skewed position relative to the cell
// origin's), rounded step by step.
__device__ __forceinline__ void extra_disp(float ox, float oy, float oz, float *E)
{
    const float s = __fmul_rn(__fadd_rn(__fadd_rn(ox, oy), oz), THIRD);
    E[0] = __fadd_rn(ox, s);
    E[1] = __fadd_rn(oy, s);
    E[2] = __fadd_rn(oz, s);
}

// Step words and displacement offsets of a decision from its six offsets
// (the binary64 path).
__device__ __forceinline__ void pack_extra(Decision &D)
{
    D.w0 = pack_step(D.e0x, D.e0y, D.e0z);
    D.w1 = pack_step(D.e1x, D.e1y, D.e1z);
    extra_disp(D.e0x, D.e0y, D.e0z, D.E);
    extra_disp(D.e1x, D.e1y, D.e1z, D.E + 3);
}

// Extra-point table of a block: case i's two float4s at i and CASES + i (so
// that the lanes' different cases spread over the banks): the six displacement
// offsets (E0x, E1x, E0y, E1y), (E0z, E1z, the two step words as bits),
// in the order the paired operands take them.
__shared__ float4 s_extra[2 * CASES];

// Fill s_extra (the caller synchronises the block before use).
__device__ __forceinline__ void init_extra_table()
{
    for (int i = threadIdx.x; i < CASES; i += blockDim.x) {
        float o[6], E[6];
        extra_case(i, o);
        extra_disp(o[0], o[1], o[2], E);
        extra_disp(o[3], o[4], o[5], E + 3);
        s_extra[i] = make_float4(E[0], E[3], E[1], E[4]);
        s_extra[CASES + i] = make_float4(E[2], E[5], __uint_as_float(pack_step(o[0], o[1], o[2])),
                                         __uint_as_float(pack_step(o[3], o[4], o[5])));
    }
}

// (bits << 1) | sign of d: one funnel shift per comparison.
__device__ __forceinline__ uint32_t push_sign(uint32_t bits, float d)
{
    return __funnelshift_l(__float_as_uint(d), bits, 1);
}

// The same decision for the binary32 path without data-dependent branches
// (lanes of a warp sit in different regions at high octaves): the sign of
// each comparison's difference becomes a bit of the case number, for the
// tetrahedra and the octahedron, and the region selects.  Every difference
// is a margin (a superset of those the branching form compares), and a lane
// keeps its binary32 decision only when all of them clear TAU, so ties and
// the sign of a zero do not matter.  `m` is the smallest margin so far.
// About 45 operations; comparisons, selects and masks of each outcome took 85.
__device__ __forceinline__ int decide_sel(float x, float y, float z, float in_sum, float &m, int &region)
{
    const float mn = fminf(x, y), mx = fmaxf(x, y);
    const float mid = fmaxf(mn, fminf(mx, z));
    m = fminf(m, fminf(fminf(mn, z), 1.0f - fmaxf(mx, z)));      // the cell: 0 < x, y, z < 1
    const float e1 = in_sum - 1.0f, e2 = in_sum - 2.0f;
    const bool r0 = e1 < 0.0f, r1 = e2 >= 0.0f;
    const float dxy = x - y, dyz = y - z, dxz = x - z;
    const float dw = ((r1 ? 3.0f : 1.0f) - in_sum) - mid;
    const float d1 = e1 - z, d2 = e1 - y, d3 = e1 - x;            // x + y - 1, x + z - 1, y + z - 1
    const float q12 = fabsf(d1) - fabsf(d2), q13 = fabsf(d1) - fabsf(d3), q23 = fabsf(d2) - fabsf(d3);
    m = fminf(m, fminf(fabsf(e1), fabsf(e2)));
    m = fminf(m, fminf(fabsf(dxy), fabsf(dyz)));
    m = fminf(m, fminf(fabsf(dxz), fabsf(dw)));
    m = fminf(m, fminf(fabsf(d1), fabsf(d2)));
    m = fminf(m, fminf(fabsf(d3), fabsf(q12)));
    m = fminf(m, fminf(fabsf(q13), fabsf(q23)));
    uint32_t tt = push_sign(2u, e2), ot = push_sign(0u, d1);    // 2 << 5 = 64: the tetrahedra's cases
    tt = push_sign(push_sign(push_sign(push_sign(tt, dxy), dyz), dxz), dw);
    ot = push_sign(push_sign(push_sign(push_sign(push_sign(ot, d2), d3), q12), q13), q23);
    region = r0 ? 0 : (r1 ? 1 : 2);
    return (int)(r0 || r1 ? tt : ot);
}

// Decision of a binary32-path lane from its case-table entry.
__device__ __forceinline__ void case_decision(int ci, int region, Decision &D)
{
    const float4 a = s_extra[ci], b = s_extra[CASES + ci];
    D.region = region;
    D.w0 = __float_as_uint(b.z);
    D.w1 = __float_as_uint(b.w);
    D.E[0] = a.x; D.E[3] = a.y; D.E[1] = a.z; D.E[4] = a.w; D.E[2] = b.x; D.E[5] = b.y;
}

// opensimplex.py:18-21 in binary64
__device__ __forceinline__ long long fastfloor64(double x)
{
    long long xi = __double2ll_rz(x);
    return x < (double)xi ? xi - 1 : xi;
}

// The cell state the contributions need.
struct Cell {
    float dx0, dy0, dz0;
    int xb7, yb7, zb7;       // cell origin << 7 (hash base)
    int xsb, ysb, zsb;       // cell origin (trace only)
    Decision D;
    double dxd, dyd, dzd;    // binary64 path only: the displacement before rounding to binary32
};

// Binary64 decisions with the reference's operation order (opensimplex.py:
// 270-300 and the region code).  No FMA contraction: explicit _rn ops.
// Returns the cell by value: a cell passed by reference would be
// address-taken in the caller, which then keeps it in local memory on the
// common binary32 path too.
__device__ __noinline__ Cell decide_f64(double X, double Y, double Z, double s)
{
    Cell c;
    double x = __dmul_rn(X, s), y = __dmul_rn(Y, s), z = __dmul_rn(Z, s);
    double so = __dmul_rn(__dadd_rn(__dadd_rn(x, y), z), -1.0 / 6);
    double xs = __dadd_rn(x, so), ys = __dadd_rn(y, so), zs = __dadd_rn(z, so);
    long long xsb = fastfloor64(xs), ysb = fastfloor64(ys), zsb = fastfloor64(zs);
    double sq = __dmul_rn((double)(xsb + ysb + zsb), 1.0 / 3);
    double xb = __dadd_rn((double)xsb, sq), yb = __dadd_rn((double)ysb, sq), zb = __dadd_rn((double)zsb, sq);
    double xins = __dsub_rn(xs, (double)xsb), yins = __dsub_rn(ys, (double)ysb), zins = __dsub_rn(zs, (double)zsb);
    double in_sum = __dadd_rn(__dadd_rn(xins, yins), zins);
    decide(xins, yins, zins, in_sum, c.D);
    pack_extra(c.D);
    c.dxd = __dsub_rn(x, xb);
    c.dyd = __dsub_rn(y, yb);
    c.dzd = __dsub_rn(z, zb);
    c.dx0 = (float)c.dxd;
    c.dy0 = (float)c.dyd;
    c.dz0 = (float)c.dzd;
    c.xsb = (int)xsb; c.ysb = (int)ysb; c.zsb = (int)zsb;
    c.xb7 = (int)((unsigned)xsb << 7);
    c.yb7 = (int)((unsigned)ysb << 7);
    c.zb7 = (int)((unsigned)zsb << 7);
    return c;
}

// What the decision from a coordinate split leaves for the displacement:
// the floors f of the skewed fractions and G = r + fx + fy + fz, so that
// dx0 = a_x - (3 fx + G) / 3 (and likewise y, z), and the case-table index.
struct Core {
    int xsb, ysb, zsb;
    int xb7, yb7, zb7;
    float fx, fy, fz, G;
    int region, ci;
};

// The decision from the split of x*scale into integers A (binary32, |A| <
// 2^22; M = A + MAGIC) and fractions a (|a| < 1) for each axis; `big` = max |x*scale|.
// Returns false when binary64 must decide.  The error analysis is at
// decide_f32 (a within 3.1e-8 of x*scale - A).
__device__ __forceinline__ bool decide_core(float Mx, float Ax, float ax, float My, float Ay, float ay, float Mz, float Az,
                                            float az, float big, Core &o)
{
    const float T = __fadd_rn(__fadd_rn(Ax, Ay), Az);
    const float q = floorf(__fmaf_rn(T, SIXTH, 1.0f / 12.0f));
    const float r = __fmaf_rn(-6.0f, q, T);
    const float u = __fadd_rn(r, __fadd_rn(__fadd_rn(ax, ay), az));
    const float bx = __fmaf_rn(-u, SIXTH, ax), by = __fmaf_rn(-u, SIXTH, ay), bz = __fmaf_rn(-u, SIXTH, az);
    const float fx = floorf(bx), fy = floorf(by), fz = floorf(bz);
    const float xins = __fsub_rn(bx, fx), yins = __fsub_rn(by, fy), zins = __fsub_rn(bz, fz);
    // the cell's integers stay on MAGIC's grid (|A| < 2^22: exact)
    const int xi = __float_as_int(__fadd_rn(__fsub_rn(Mx, q), fx)), yi = __float_as_int(__fadd_rn(__fsub_rn(My, q), fy)),
              zi = __float_as_int(__fadd_rn(__fsub_rn(Mz, q), fz));
    o.xsb = xi - MAGIC_BITS; o.ysb = yi - MAGIC_BITS; o.zsb = zi - MAGIC_BITS;
    o.xb7 = xi << 7; o.yb7 = yi << 7; o.zb7 = zi << 7;
    o.fx = fx; o.fy = fy; o.fz = fz;
    o.G = __fadd_rn(r, __fadd_rn(__fadd_rn(fx, fy), fz));
    const float in_sum = __fadd_rn(__fadd_rn(xins, yins), zins);
    float m = 1.0f;
    o.ci = decide_sel(xins, yins, zins, in_sum, m, o.region);
    return m >= TAU && big < PMAX;
}

// Binary32 path.  Returns false when binary64 must decide.
//
// Error of b = a - u/6 (the skewed coordinate less its integer part Ax - q)
// for |x*scale| < 2^16, each step's rounding in absolute terms:
//  * p + e = x*scale within 2^-45 |x*scale| < 2e-9: the coordinate and the
//    scale are binary32 pairs (2^-47 and 2^-48 relative), the lo*lo term is
//    dropped and the three cross terms are fused;
//  * A = round(p) and p - A are exact; a = (p - A) + e rounds once,
//    |a| < 1: <= 2^-25 (3.0e-8);
//  * T = Ax + Ay + Az is an exact integer and q = floor(T/6 + 1/12) is exact
//    (T/6 + 1/12 lies at least 1/12 from an integer; the fused product's
//    error is below |T| 2^-24 < 0.02), so r = T - 6q in 0..5 is exact;
//  * the sum of the three a (two roundings, values < 1.5): <= 1.2e-7,
//    entering b divided by 6: 2.0e-8; u = r + that, |u| < 8: 2.4e-7 / 6 =
//    4.0e-8; the errors of the a themselves: 3.0e-8 * (5/6 + 2/6) = 3.5e-8;
//  * SIXTH = 1/6 rounded, off by 5.0e-9, times |u| <= 6.5: 3.2e-8; the
//    fused b = a - u*SIXTH, |b| < 2: <= 2^-24 (6.0e-8).
// Total <= 1.9e-7 (checked by simulating these operations on random
// coordinates and scales: largest 1.3e-7).  xins = b - floor(b) is exact.
__device__ __forceinline__ bool decide_f32(float xh, float xl, float yh, float yl, float zh, float zl,
                                           float sh, float sl, Cell &c)
{
    float px = xh * sh, py = yh * sh, pz = zh * sh;
    float ex = fmaf(xh, sh, -px), ey = fmaf(yh, sh, -py), ez = fmaf(zh, sh, -pz);
    ex = fmaf(xh, sl, ex); ey = fmaf(yh, sl, ey); ez = fmaf(zh, sl, ez);
    ex = fmaf(xl, sh, ex); ey = fmaf(yl, sh, ey); ez = fmaf(zl, sh, ez);
    float big = fmaxf(fabsf(px), fmaxf(fabsf(py), fabsf(pz)));
    const float Mx = px + MAGIC, My = py + MAGIC, Mz = pz + MAGIC;
    const float Ax = Mx - MAGIC, Ay = My - MAGIC, Az = Mz - MAGIC;
    float ax = (px - Ax) + ex, ay = (py - Ay) + ey, az = (pz - Az) + ez;
    Core o;
    const bool ok = decide_core(Mx, Ax, ax, My, Ay, ay, Mz, Az, az, big, o);
    c.xsb = o.xsb; c.ysb = o.ysb; c.zsb = o.zsb;
    c.xb7 = o.xb7; c.yb7 = o.yb7; c.zb7 = o.zb7;
    const float g = __fmul_rn(o.G, THIRD);
    c.dx0 = __fsub_rn(__fsub_rn(ax, o.fx), g);
    c.dy0 = __fsub_rn(__fsub_rn(ay, o.fy), g);
    c.dz0 = __fsub_rn(__fsub_rn(az, o.fz), g);
    case_decision(o.ci, o.region, c.D);
    return ok;
}

// The table's word at an extra point (base: the cell's hash bases less one
// step, w its step word).
__device__ __forceinline__ uint32_t lk_extra(uint32_t lb, int xm, int ym, int zm, uint32_t w)
{
    const uint32_t hx = lk(lb, (int)((uint32_t)xm + w));
    const uint32_t hy = lk(lb, (int)(hx + (uint32_t)ym + (w >> 9)));
    return lk(lb, (int)(hy + (uint32_t)zm + (w >> 18)));
}

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }

// Two lattice contributions at once in paired binary32 arithmetic (one
// FFMA2/FMUL2/FADD2 does both): acc += attn^4 * (grad . d) for slots a and
// b; ON (1 or 0) masks slots outside the region (MASK).  -attn = |d|^2 - 2
// is clamped at 0 before squaring, so only attn > 0 counts.
template <bool MASK>
__device__ __forceinline__ float2 contrib2(uint32_t wa, uint32_t wb, float2 DX, float2 DY, float2 DZ, float2 ON,
                                           float2 acc)
{
    float2 na = __ffma2_rn(DZ, DZ, f2(-2.0f, -2.0f));
    na = __ffma2_rn(DY, DY, na);
    na = __ffma2_rn(DX, DX, na);
    na = f2(fminf(na.x, 0.0f), fminf(na.y, 0.0f));
    if (MASK) na = __fmul2_rn(na, ON);
    const float2 a2 = __fmul2_rn(na, na);
    const float2 a4 = __fmul2_rn(a2, a2);
    const float2 gx = f2(grad_of<false>(wa, 0), grad_of<false>(wb, 0)), gy = f2(grad_of<false>(wa, 1), grad_of<false>(wb, 1)),
                 gz = f2(grad_of<false>(wa, 2), grad_of<false>(wb, 2));
    float2 dot = __fmul2_rn(gz, DZ);
    dot = __ffma2_rn(gy, DY, dot);
    dot = __ffma2_rn(gx, DX, dot);
    return __ffma2_rn(a4, dot, acc);
}

// The fixed corners that a lane of region g evaluates first: corner 0 | A1,
// A2, A3 = (1,0,0), (0,1,0), (0,0,1) | B1, B2, B3 = (1,1,0), (1,0,1), (0,1,1).
// Region 0: 0, A1, A2, A3; region 1: corner 0 (there (1,1,1)), B1, B2, B3; the
// octahedron: A1, A2, A3, B1 (its B2 and B3 are a slot pair of their own).
__device__ __forceinline__ int region_corner(int g, int x)
{
    return g == 2 ? x + 1 : (x == 0 ? 0 : (g == 1 ? 3 + x : x));
}

// Three times component a of corner c's displacement offset in region g.
__device__ __forceinline__ int corner_thirds(int g, int c, int a)
{
    if (c == 0) return g == 1 ? 6 : 0;
    if (c <= 3) return a == c - 1 ? 4 : 1;     // (4,1,1), (1,4,1), (1,1,4)
    return a == 6 - c ? 2 : 5;                 // (5,5,2), (5,2,5), (2,5,5)
}

// Displacement offsets o + (ox + oy + oz)/3, negated, of the fixed corners
// that a lane of each region evaluates (slots X1..X4 of noise_raw): entry
// 4 q + region, q = 0: (X1x, X2x, X1y, X2y), 1: (X1z, X2z, X3x, X4x), 2: (X3y,
// X4y, X3z, X4z).
__shared__ float4 s_corner32[12];

__device__ __forceinline__ void init_corner32_table(int g)
{
    if (g >= 3) return;
    float v[4][3];
    for (int x = 0; x < 4; ++x) {
        const int c = region_corner(g, x);
        for (int a = 0; a < 3; ++a) {
            const int m = corner_thirds(g, c, a);
            v[x][a] = m == 6 ? -2.0f : (m == 5 ? -(1.0f + 2.0f * THIRD) : (m == 4 ? -(1.0f + THIRD) : (m == 2 ? -(2.0f * THIRD) : (m == 1 ? -THIRD : 0.0f))));
        }
    }
    s_corner32[g] = make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
    s_corner32[4 + g] = make_float4(v[0][2], v[1][2], v[2][0], v[3][0]);
    s_corner32[8 + g] = make_float4(v[2][1], v[3][1], v[2][2], v[3][2]);
}

// noise3d(x*s) * 103 for one vertex and octave.  A lane evaluates its
// region's four or six fixed corners and the two extra points in four slot
// pairs (X1..X4, the octahedron's X5 and X6, the extra points).
template <bool TRACE>
__device__ __forceinline__ float noise_raw(float xh, float xl, float yh, float yl, float zh, float zl,
                                           float sh, float sl, double X, double Y, double Z, double s,
                                           uint32_t lb, unsigned &nfb, int32_t *tr, int32_t *sl9)
{
    Cell c;
    if (!decide_f32(xh, xl, yh, yl, zh, zl, sh, sl, c)) {
        c = decide_f64(X, Y, Z, s);
        ++nfb;
    }
    const int r = c.D.region;
    // hash prefixes of the fixed slots
    uint32_t h0 = lk(lb, c.xb7), h1 = lk(lb, c.xb7 + 128);
    uint32_t h00 = lk(lb, (int)h0 + c.yb7), h01 = lk(lb, (int)h0 + c.yb7 + 128);
    uint32_t h10 = lk(lb, (int)h1 + c.yb7), h11 = lk(lb, (int)h1 + c.yb7 + 128);
    const int z0 = c.zb7, z1 = c.zb7 + 128;
    const float dx0 = c.dx0, dy0 = c.dy0, dz0 = c.dz0;
    // corner 0: (0,0,0) in region 0, (1,1,1) in region 1
    const bool r1 = r == 1, r2 = r == 2;
    const uint32_t w0 = lk(lb, r1 ? (int)h11 + z1 : (int)h00 + z0);
    const uint32_t w100 = lk(lb, (int)h10 + z0), w010 = lk(lb, (int)h01 + z0), w001 = lk(lb, (int)h00 + z1);
    const uint32_t w110 = lk(lb, (int)h11 + z0), w101 = lk(lb, (int)h10 + z1), w011 = lk(lb, (int)h01 + z1);
    // extra points
    const Decision &D = c.D;
    const uint32_t ew0 = D.w0, ew1 = D.w1;
    const int xm = c.xb7 - 128, ym = c.yb7 - 128, zm = c.zb7 - 128;
    const uint32_t we0 = lk_extra(lb, xm, ym, zm, ew0), we1 = lk_extra(lb, xm, ym, zm, ew1);
    const uint32_t wX1 = r2 ? w100 : w0, wX2 = r2 ? w010 : (r1 ? w110 : w100);
    const uint32_t wX3 = r2 ? w001 : (r1 ? w101 : w010), wX4 = r2 ? w110 : (r1 ? w011 : w001);
    const float4 k0 = s_corner32[r], k1 = s_corner32[4 + r], k2 = s_corner32[8 + r];
    const float2 X0 = f2(dx0, dx0), Y0 = f2(dy0, dy0), Z0 = f2(dz0, dz0);
    const float fr2 = r2 ? 1.0f : 0.0f;
    const float2 none = f2(1.0f, 1.0f);
    const float c2 = 2.0f * THIRD, c3 = 1.0f + 2.0f * THIRD;   // displacement d = d0 - o - sum(o)/3
    float2 acc = f2(0.0f, 0.0f);
    acc = contrib2<false>(wX1, wX2, __fadd2_rn(X0, f2(k0.x, k0.y)), __fadd2_rn(Y0, f2(k0.z, k0.w)),
                          __fadd2_rn(Z0, f2(k1.x, k1.y)), none, acc);
    acc = contrib2<false>(wX3, wX4, __fadd2_rn(X0, f2(k1.z, k1.w)), __fadd2_rn(Y0, f2(k2.x, k2.y)),
                          __fadd2_rn(Z0, f2(k2.z, k2.w)), none, acc);
    acc = contrib2<true>(w101, w011, __fadd2_rn(X0, f2(-c3, -c2)), __fadd2_rn(Y0, f2(-c2, -c3)),
                         __fadd2_rn(Z0, f2(-c3, -c3)), f2(fr2, fr2), acc);
    acc = contrib2<false>(we0, we1, __fadd2_rn(X0, f2(-D.E[0], -D.E[3])), __fadd2_rn(Y0, f2(-D.E[1], -D.E[4])),
                          __fadd2_rn(Z0, f2(-D.E[2], -D.E[5])), none, acc);
    const float v = acc.x + acc.y;
    if (TRACE) {
        tr[0] = c.xsb; tr[1] = c.ysb; tr[2] = c.zsb; tr[3] = r;
        int e[6];
        for (int k = 0; k < 6; ++k) e[k] = step_offset(k < 3 ? ew0 : ew1, k % 3);
        tr[4] = c.xsb + e[0]; tr[5] = c.ysb + e[1]; tr[6] = c.zsb + e[2];
        tr[7] = c.xsb + e[3]; tr[8] = c.ysb + e[4]; tr[9] = c.zsb + e[5];
        const int o[9][3] = {{r == 1, r == 1, r == 1}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 0},
                             {1, 0, 1}, {0, 1, 1}, {e[0], e[1], e[2]}, {e[3], e[4], e[5]}};
        const uint32_t w[9] = {w0, w100, w010, w001, w110, w101, w011, we0, we1};
        const bool on0 = r != 2, onA = r != 1, onB = r != 0;
        const bool on[9] = {on0, onA, onA, onA, onB, onB, onB, true, true};
        for (int k = 0; k < 9; ++k) {
            int32_t *q = sl9 + 5 * k;
            q[0] = c.xsb + o[k][0]; q[1] = c.ysb + o[k][1]; q[2] = c.zsb + o[k][2];
            q[3] = 0;
            for (int a = 0; a < 3; ++a) q[3] |= ((int)grad_of<false>(w[k], a) + 16) << (8 * a);
            q[4] = on[k] ? 1 : 0;
        }
    }
    return v;
}


// ---------------------------------------------------------------------------
// Pair-precision noise (the batched, plain and served planet paths).
//
// Eroded planets need elevations much closer to binary64 than binary32
// gives: the erosion update branches on the sign of every neighbour height
// difference, and starting heights off by binary32 rounding (3e-7 relative)
// flip near-ties, after which water, sediment and heights leave the binary64
// trajectory (0.4 % of max |h| after 30 iterations, 13 % after 60, on a
// 100,002-vertex sphere; random errors of 1e-11 in the raw fBm sum flipped
// nothing in 100 iterations on 900,002 vertices, 1e-10 did).  This path
// takes the same decisions as the binary32 one and carries every
// continuous quantity as an unevaluated pair hi + lo of binary32s:
//  * x*scale = A + a1 + a2 + a3 exactly (A an integer): for a power-of-two
//    scale the vertex's binary32 triple scaled, otherwise the product of
//    the vertex and scale triples to ~2^-70 relative;
//  * dx0 = a - (3f + G)/3 (f, G from the decision) and every slot's offset
//    K = m/3 are anchored: hi on the 2^-21 grid, so the hi part of d =
//    dx0 - K is exact and only the lo parts round (~2^-46); d is then
//    renormalised (|lo| <= ulp(hi)/2), which keeps the cross terms 2 hi lo
//    of |d|^2 small enough to sum to ~2^-46;
//  * attn = 2 - |d|^2, attn^4, grad . d and their product with error-free
//    transforms (fma-exact products, two-sums; the running 2 - dx^2 - dy^2
//    - dz^2 uses fast two-sums, exact whenever attn > 0), two slots at a
//    time in paired binary32 lanes;
//  * for the octaves below 1/8 of the largest amplitude, whose displacements
//    are not renormalised, the squares are summed on a fixed grid and the
//    two-sums ordered by a bias, 50 paired operations per two slots instead
//    of 64; attn^2, attn^4 and the product keep the low parts' squares, which
//    puts the error below that of the longer form without them (12 octaves:
//    1.16e-14 of the field's norm against 1.44e-14);
//  * the contributions, the division by 103 and the octave's
//    (noise + 1) * 0.5 * strength * radius term are summed in pairs; the
//    running sum over octaves is renormalised after every octave, so a
//    vertex gives the same bits whether its octaves run in one launch or
//    one launch each.

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Knuth's two-sum per lane: s + e == a + b exactly.
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2 &s, float2 &e)
{
    s = add2(a, b);
    const float2 bb = sub2(s, a);
    e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}

__device__ __forceinline__ void two_sum1(float a, float b, float &s, float &e)
{
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Anchored thirds m/3, m = 0..6: hi = rint(m 2^21 / 3) 2^-21, lo = m/3 - hi
// (+-1/(3 2^21) or 0).
constexpr float ANC = 6.0f;                         // (v + 6) - 6 rounds v in [-2, 2) to the 2^-21 grid
constexpr float T1H = 699051.0f / 2097152.0f;       // 1/3
constexpr float T2H = 1398101.0f / 2097152.0f;      // 2/3
constexpr float T4H = 2796203.0f / 2097152.0f;      // 4/3
constexpr float T5H = 3495253.0f / 2097152.0f;      // 5/3
constexpr float C3L = (float)(1.0 / (3.0 * 2097152.0));   // 2^-21 / 3: |lo| of the thirds above
constexpr float C3L2 = 2.0f * C3L;

// Anchored m/3 for an integer m (|m| < 2^9): hi on the 2^-21 grid, lo.
__device__ __forceinline__ void anchor_third(int m, float &H, float &L)
{
    const int N = m * 2097152;
    const int q = N >= 0 ? (N + 1) / 3 : -((1 - N) / 3);
    H = __fmul_rn((float)q, 1.0f / 2097152.0f);
    L = __fmul_rn((float)(N - 3 * q), C3L);
}

// anchor_third(m) and its doubled lo part for m = -8..7 at entry m & 15.
__shared__ float2 s_third[16];

__device__ __forceinline__ void init_third_table(int i)
{
    if (i >= 0 && i < 16) {
        float H, L;
        anchor_third(i < 8 ? i : i - 16, H, L);
        s_third[i] = make_float2(H, 2.0f * L);
    }
}

// Pair case table of a block: case i (as s_extra) has four float4s, CASES
// apart: the two extra points' offsets e + (ex + ey + ez)/3 anchored, hi parts
// (E0x, E1x, E0y, E1y), (E0z, E1z, the two step words), doubled lo parts
// (E0x, E1x, E0y, E1y), (E0z, E1z, 0, 0).
__shared__ float4 s_extra_p[4 * CASES];

__device__ __forceinline__ void anchored_offsets(uint32_t w0, uint32_t w1, float *H, float *L)
{
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const uint32_t w = p ? w1 : w0;
        const int ox = step_offset(w, 0), oy = step_offset(w, 1), oz = step_offset(w, 2);
        const int t = ox + oy + oz;
        anchor_third(3 * ox + t, H[3 * p], L[3 * p]);
        anchor_third(3 * oy + t, H[3 * p + 1], L[3 * p + 1]);
        anchor_third(3 * oz + t, H[3 * p + 2], L[3 * p + 2]);
    }
}

__device__ __forceinline__ void init_extra_table_pair(int i)
{
    if (i >= 0 && i < CASES) {
        float o[6];
        extra_case(i, o);
        const uint32_t w0 = pack_step(o[0], o[1], o[2]), w1 = pack_step(o[3], o[4], o[5]);
        float H[6], L[6];
        anchored_offsets(w0, w1, H, L);
        s_extra_p[i] = make_float4(H[0], H[3], H[1], H[4]);
        s_extra_p[CASES + i] = make_float4(H[2], H[5], __uint_as_float(w0), __uint_as_float(w1));
        s_extra_p[2 * CASES + i] = make_float4(2.0f * L[0], 2.0f * L[3], 2.0f * L[1], 2.0f * L[4]);
        s_extra_p[3 * CASES + i] = make_float4(2.0f * L[2], 2.0f * L[5], 0.0f, 0.0f);
    }
}

// d = dx0 - K for one axis of two slots, from the anchored dx0 (hi X0H,
// doubled lo X0L2) and offsets (K, doubled lo KL2): the hi part dx0 - K is
// exact (both on the 2^-21 grid); then renormalised by a fast two-sum
// (|hi| >= 2^-21 > |lo| or hi = 0), H + L2/2 == d with |L2/2| <=
// ulp(H)/2.  L2 = 2 lo (exact: twice the fast two-sum's exact error).
// Without NORM the anchored pair is used as it is (|lo| up to 2^-20): the
// cross terms then carry ~2^-42 of error, which octaves of small amplitude
// can afford (see noise_pair).
template <bool NORM>
__device__ __forceinline__ void slot_disp(float X0H, float X0L2, float2 K, float2 KL2, float2 &H, float2 &L2)
{
    const float2 h0 = sub2(f2(X0H, X0H), K);
    const float2 l2 = sub2(f2(X0L2, X0L2), KL2);
    if (NORM) {
        H = fma2(f2(0.5f, 0.5f), l2, h0);
        L2 = fma2(f2(-2.0f, -2.0f), sub2(H, h0), l2);
    } else {
        H = h0;
        L2 = l2;
    }
}

// v times the sign of g.
__device__ __forceinline__ float with_sign(float v, float g)
{
    return __uint_as_float(__float_as_uint(v) ^ (__float_as_uint(g) & 0x80000000u));
}

// The component that the gradient of a table word has its +-11 in.
__device__ __forceinline__ float of_axis(uint32_t w, float x, float y, float z)
{
    return (w & (2u << 26)) ? z : ((w & (1u << 26)) ? y : x);
}

// Two lattice contributions (slots a, b in the lanes) in pair arithmetic,
// added to the pair accumulator (AH, AL).  X0H, X0L2: the anchored dx0 (hi,
// 2 lo); KX/KXL2 the slots' anchored offsets (hi, 2 lo); MASK: ON 1/0 masks.
// Without NORM the accumulator starts at ACC_BIAS, which keeps it larger than
// any contribution, so that fast two-sums do.
constexpr float ACC_BIAS = 48.0f;      // a contribution's quarter is below 14.7, four of them below 26
template <bool NORM, bool MASK>
__device__ __forceinline__ void contrib2_pair(uint32_t wa, uint32_t wb, float X0H, float X0L2, float Y0H, float Y0L2,
                                              float Z0H, float Z0L2, float2 KX, float2 KXL2, float2 KY, float2 KYL2,
                                              float2 KZ, float2 KZL2, float2 ON, float2 &AH, float2 &AL)
{
    float2 Xh, X2, Yh, Y2, Zh, Z2;
    slot_disp<NORM>(X0H, X0L2, KX, KXL2, Xh, X2);
    slot_disp<NORM>(Y0H, Y0L2, KY, KYL2, Yh, Y2);
    slot_disp<NORM>(Z0H, Z0L2, KZ, KZL2, Zh, Z2);
    // attn = 2 - |d|^2 = r3 + al
    float2 r3, al;
    if (NORM) {
        // squares of the hi parts exact as p + pe, plus the cross terms 2 hi lo
        const float2 px = mul2(Xh, Xh), py = mul2(Yh, Yh), pz = mul2(Zh, Zh);
        const float2 pxe = fma2(Xh, Xh, f2(-px.x, -px.y)), pye = fma2(Yh, Yh, f2(-py.x, -py.y)),
                     pze = fma2(Zh, Zh, f2(-pz.x, -pz.y));
        float2 L = add2(pxe, add2(pye, pze));
        L = fma2(Xh, X2, L);
        L = fma2(Yh, Y2, L);
        L = fma2(Zh, Z2, L);
        const float2 r0 = f2(2.0f, 2.0f);
        const float2 r1 = sub2(r0, px), r2 = sub2(r1, py);
        r3 = sub2(r2, pz);
        const float2 e1 = sub2(sub2(r0, r1), px), e2 = sub2(sub2(r1, r2), py), e3 = sub2(sub2(r2, r3), pz);
        al = sub2(add2(add2(e1, e2), e3), L);
    } else {
        // the squares added to 2 one by one: while the sum stays below 4 (where
        // attn > 0) each step rounds to the 2^-22 grid, its increment is exact
        // and the square's rest (below 2^-22, on the 2^-42 grid) comes exact
        // from one fma; 15 operations against 23 above, and no less exact
        // beside the cross terms, which reach 2^-19 without NORM
        const float2 t0 = f2(2.0f, 2.0f), t1 = fma2(Xh, Xh, t0), t2 = fma2(Yh, Yh, t1), t3 = fma2(Zh, Zh, t2);
        const float2 d1 = sub2(t1, t0), d2 = sub2(t2, t1), d3 = sub2(t3, t2);
        const float2 e1 = fma2(Xh, Xh, f2(-d1.x, -d1.y)), e2 = fma2(Yh, Yh, f2(-d2.x, -d2.y)),
                     e3 = fma2(Zh, Zh, f2(-d3.x, -d3.y));
        float2 L = add2(add2(e1, e2), e3);
        L = fma2(Xh, X2, L);
        L = fma2(Yh, Y2, L);
        L = fma2(Zh, Z2, L);
        r3 = sub2(f2(4.0f, 4.0f), t3);
        al = f2(-L.x, -L.y);
    }
    // only attn > 0 counts, and only in the region (ah = 0 zeroes the rest)
    float2 ah = f2(fmaxf(r3.x, 0.0f), fmaxf(r3.y, 0.0f));
    if (MASK) ah = mul2(ah, ON);
    // attn^2, attn^4 as pairs (with the squares of the low parts: without NORM
    // al reaches 2^-19, and its square would show)
    const float2 two = f2(2.0f, 2.0f);
    const float2 h2 = mul2(ah, ah);
    float2 l2 = fma2(ah, ah, f2(-h2.x, -h2.y));
    l2 = fma2(fma2(two, ah, al), al, l2);
    const float2 h4 = mul2(h2, h2);
    float2 l4 = fma2(h2, h2, f2(-h4.x, -h4.y));
    l4 = fma2(fma2(two, h2, l2), l2, l4);
    // grad . d as a pair (dh, dl), times DSC (see below)
    const float2 gx = f2(grad_of<true>(wa, 0), grad_of<true>(wb, 0)), gy = f2(grad_of<true>(wa, 1), grad_of<true>(wb, 1)),
                 gz = f2(grad_of<true>(wa, 2), grad_of<true>(wb, 2));
    float2 dh, dl;
    if (NORM) {
        // products exact as q + qe, summed with two-sums; DSC = 1
        const float2 qx = mul2(gx, Xh), qy = mul2(gy, Yh), qz = mul2(gz, Zh);
        const float2 qxe = fma2(gx, Xh, f2(-qx.x, -qx.y)), qye = fma2(gy, Yh, f2(-qy.x, -qy.y)),
                     qze = fma2(gz, Zh, f2(-qz.x, -qz.y));
        float2 s1, t1, t2;
        two_sum2(qx, qy, s1, t1);
        two_sum2(s1, qz, dh, t2);
        const float2 gl = fma2(gx, X2, fma2(gy, Y2, mul2(gz, Z2)));     // 2 (grad . lo)
        dl = fma2(f2(0.5f, 0.5f), gl, add2(add2(add2(qxe, qye), qze), add2(t1, t2)));
    } else {
        // hi parts on the 2^-21 grid (|d| < sqrt 2 wherever attn > 0): with
        // g_i = s_i (4 + 7 [i == a]), grad . hi = 4 (U + V) exactly, U =
        // sum s_i hi_i + 2 s_a hi_a (|U| < 8 on the grid: exact), V =
        // -s_a hi_a / 4; the lo parts' product in binary32.  DSC = 1/4.
        const float2 sx = f2(with_sign(Xh.x, gx.x), with_sign(Xh.y, gx.y)), sy = f2(with_sign(Yh.x, gy.x), with_sign(Yh.y, gy.y)),
                     sz = f2(with_sign(Zh.x, gz.x), with_sign(Zh.y, gz.y));
        const float2 s_a = f2(of_axis(wa, sx.x, sy.x, sz.x), of_axis(wb, sx.y, sy.y, sz.y));
        const float2 U = fma2(f2(2.0f, 2.0f), s_a, add2(add2(sx, sy), sz));
        const float2 V = mul2(f2(-0.25f, -0.25f), s_a);
        // a fast two-sum: where |U| < |V| (below 3/8) the sum, on the 2^-23
        // grid and below 1, is exact
        dh = add2(U, V);
        const float2 e = sub2(V, sub2(dh, U));
        const float2 gl = fma2(gx, X2, fma2(gy, Y2, mul2(gz, Z2)));     // 2 (grad . lo)
        dl = fma2(f2(0.125f, 0.125f), gl, e);
    }
    // attn^4 * (grad . d)
    const float2 ch = mul2(h4, dh);
    float2 cl = fma2(h4, dh, f2(-ch.x, -ch.y));
    cl = fma2(add2(h4, l4), dl, fma2(l4, dh, cl));
    float2 s, e;
    if (NORM) {
        two_sum2(AH, ch, s, e);
    } else {
        s = add2(AH, ch);
        e = sub2(ch, sub2(s, AH));
    }
    AH = s;
    AL = add2(AL, add2(e, cl));
}

// Offsets of the fixed corners that a lane of each region evaluates (slots
// X1..X4 of noise_pair), anchored: entry 4 q + region, q = 0: (X1x, X2x, X1y,
// X2y), 1: (X1z, X2z, X1 2lo, X2 2lo), 2 and 3 the same of X3, X4.  Four
// shared loads (the regions' entries on different banks) instead of 27
// selects per vertex and octave.
__shared__ float4 s_corner[16];

__device__ __forceinline__ void init_corner_table(int i)
{
    // X1..X4 per region in thirds m / 3 (hi), and the sign of the lo part
    if (i >= 0 && i < 12) {
        const int q = i / 3, g = i % 3;
        float v[2][4];
        for (int u = 0; u < 2; ++u) {
            const int x = 2 * (q / 2) + u;                   // slot X1..X4
            const int c = region_corner(g, x);
            for (int a = 0; a < 3; ++a) {
                const int m = corner_thirds(g, c, a);
                v[u][a] = m == 6 ? 2.0f : (m == 5 ? T5H : (m == 4 ? T4H : (m == 2 ? T2H : (m == 1 ? T1H : 0.0f))));
            }
            v[u][3] = c == 0 ? 0.0f : (c <= 3 ? -C3L2 : C3L2);
        }
        s_corner[4 * q + g] = (q & 1) ? make_float4(v[0][2], v[1][2], v[0][3], v[1][3])
                                      : make_float4(v[0][0], v[1][0], v[0][1], v[1][1]);
    }
}

// x*scale = A + a1 + a2 + a3 for one axis: x = x1 + x2 + x3 and scale =
// s1 + s2 + s3 exact binary32 triples; |x*scale| < 2^22 for A to be exact.
__device__ __forceinline__ void coord_split(float x1, float x2, float x3, float s1, float s2, float s3, bool pow2,
                                            float &p, float &M, float &A, float &a1, float &a2, float &a3)
{
    p = __fmul_rn(x1, s1);
    M = __fadd_rn(p, MAGIC);
    A = __fsub_rn(M, MAGIC);
    a1 = __fsub_rn(p, A);
    if (pow2) {                       // scale = s1, a power of two: exact scaling
        a2 = __fmul_rn(x2, s1);
        a3 = __fmul_rn(x3, s1);
        return;
    }
    const float e11 = __fmaf_rn(x1, s1, -p);
    const float p12 = __fmul_rn(x1, s2), e12 = __fmaf_rn(x1, s2, -p12);
    const float p21 = __fmul_rn(x2, s1), e21 = __fmaf_rn(x2, s1, -p21);
    const float q = __fmaf_rn(x1, s3, __fmaf_rn(x2, s2, __fmul_rn(x3, s1)));
    float b, c, b2, c2;
    two_sum1(p12, p21, b, c);
    two_sum1(b, e11, b2, c2);
    a2 = b2;
    a3 = __fadd_rn(__fadd_rn(c, c2), __fadd_rn(__fadd_rn(e12, e21), q));
}

// Anchor a pair (h, l) with h in [-2, 2): hi on the 2^-21 grid, lo.
__device__ __forceinline__ void anchor_pair(float h, float l, float &H, float &L)
{
    H = __fsub_rn(__fadd_rn(h, ANC), ANC);
    L = __fadd_rn(__fsub_rn(h, H), l);
}

// A displacement anchored (binary64 decision path).  It lies in [-2, 2) unless
// the coordinate is past binary64's integers; beyond 4 no lattice point of the
// cell is near and 4 does as well, while larger ones' low parts are not small
// and their squares (contrib2_pair) would stay where attn is 0.
__device__ __forceinline__ void anchor_f64(double d, float &H, float &L)
{
    const float h = __double2float_rn(d), l = __double2float_rn(__dsub_rn(d, (double)h));
    const bool far = fabsf(h) > 4.0f && fabsf(h) < 0x1p66f;       // (an infinite coordinate stays no number)
    anchor_pair(far ? copysignf(4.0f, h) : h, far ? 0.0f : l, H, L);
}

// Per-octave constants of the pair path.
struct OctP {
    float s1, s2, s3;     // scale as a binary32 triple
    float amph, ampl;     // 0.5 * strength * radius as a pair
    double s;             // scale (binary64 decision path)
    bool norm;            // renormalise the displacements (noise_pair<true>)
};

// noise3d(x * s) as a pair (vh, vl) of 103 * noise, for one vertex and
// octave.  x1..z3: the vertex's binary32 triples (x1 + x2 + x3 == x).
//
// A lane evaluates at most 8 lattice points: its region's fixed corners
// (tetrahedra: the corner at 0 or 1 and its three neighbours; octahedron:
// the six mixed corners) and the two extra points.  The corners are
// assigned to lanes per region (selects), so a warp runs four slot pairs:
// X1..X4 (every region), X5/X6 (octahedron only) and the extra points.
//
// NORM: renormalise the slots' displacements.  Without it the value carries
// up to ~1.5e-13 * (0.5 strength radius) of extra error, so the planet
// paths skip it only for octaves whose amplitude is at most 1/8 of the
// first one's (|error| <= 2e-14 of a field whose range is ~2 amp_0).
template <bool NORM>
__device__ __forceinline__ void noise_pair(float x1, float x2, float x3, float y1, float y2, float y3, float z1,
                                           float z2, float z3, const OctP &O, bool pow2, uint32_t lb, unsigned &nfb,
                                           float &vh, float &vl)
{
    float px, Mx, Ax, ax1, ax2, ax3, py, My, Ay, ay1, ay2, ay3, pz, Mz, Az, az1, az2, az3;
    coord_split(x1, x2, x3, O.s1, O.s2, O.s3, pow2, px, Mx, Ax, ax1, ax2, ax3);
    coord_split(y1, y2, y3, O.s1, O.s2, O.s3, pow2, py, My, Ay, ay1, ay2, ay3);
    coord_split(z1, z2, z3, O.s1, O.s2, O.s3, pow2, pz, Mz, Az, az1, az2, az3);
    const float ax = __fadd_rn(ax1, ax2), ay = __fadd_rn(ay1, ay2), az = __fadd_rn(az1, az2);
    const float big = fmaxf(fabsf(px), fmaxf(fabsf(py), fabsf(pz)));
    Core o;
    int region, xb7, yb7, zb7;
    uint32_t ew0, ew1;
    float X0H, X0L2, Y0H, Y0L2, Z0H, Z0L2;
    float EH[6], EL2[6];
    if (decide_core(Mx, Ax, ax, My, Ay, ay, Mz, Az, az, big, o)) {
        region = o.region;
        xb7 = o.xb7; yb7 = o.yb7; zb7 = o.zb7;
        // the fraction anchored, then dx0 = a - (f + G/3)
        // (-6 <= G <= 5: |a| < 0.51 here, so the skewed fractions a - (r + ax +
        // ay + az) / 6 lie in (-1.6, 0.8) and their floors in -2..0, r in 0..5)
        const float2 third = s_third[__float_as_uint(__fadd_rn(o.G, MAGIC)) & 15u];
        const float GH = third.x, GL2 = third.y;
        const float FXH = __fsub_rn(__fadd_rn(ax, ANC), ANC), FYH = __fsub_rn(__fadd_rn(ay, ANC), ANC),
                    FZH = __fsub_rn(__fadd_rn(az, ANC), ANC);
        const float FXL = __fadd_rn(__fadd_rn(__fsub_rn(ax1, FXH), ax2), ax3);
        const float FYL = __fadd_rn(__fadd_rn(__fsub_rn(ay1, FYH), ay2), ay3);
        const float FZL = __fadd_rn(__fadd_rn(__fsub_rn(az1, FZH), az2), az3);
        X0H = __fsub_rn(FXH, __fadd_rn(o.fx, GH));
        Y0H = __fsub_rn(FYH, __fadd_rn(o.fy, GH));
        Z0H = __fsub_rn(FZH, __fadd_rn(o.fz, GH));
        X0L2 = __fmaf_rn(2.0f, FXL, -GL2);
        Y0L2 = __fmaf_rn(2.0f, FYL, -GL2);
        Z0L2 = __fmaf_rn(2.0f, FZL, -GL2);
        const float4 *t = s_extra_p + o.ci;
        const float4 t0 = t[0], t1 = t[CASES], t2 = t[2 * CASES], t3 = t[3 * CASES];
        EH[0] = t0.x; EH[3] = t0.y; EH[1] = t0.z; EH[4] = t0.w; EH[2] = t1.x; EH[5] = t1.y;
        ew0 = __float_as_uint(t1.z);
        ew1 = __float_as_uint(t1.w);
        EL2[0] = t2.x; EL2[3] = t2.y; EL2[1] = t2.z; EL2[4] = t2.w; EL2[2] = t3.x; EL2[5] = t3.y;
    } else {
        // the vertex as binary64 (the triple's sum is exact)
        const double X = (double)x1 + (double)x2 + (double)x3, Y = (double)y1 + (double)y2 + (double)y3,
                     Z = (double)z1 + (double)z2 + (double)z3;
        const Cell c = decide_f64(X, Y, Z, O.s);
        ++nfb;
        region = c.D.region;
        xb7 = c.xb7; yb7 = c.yb7; zb7 = c.zb7;
        float L;
        anchor_f64(c.dxd, X0H, L);
        X0L2 = __fmul_rn(2.0f, L);
        anchor_f64(c.dyd, Y0H, L);
        Y0L2 = __fmul_rn(2.0f, L);
        anchor_f64(c.dzd, Z0H, L);
        Z0L2 = __fmul_rn(2.0f, L);
        ew0 = c.D.w0;
        ew1 = c.D.w1;
        float EL[6];
        anchored_offsets(ew0, ew1, EH, EL);
        for (int k = 0; k < 6; ++k) EL2[k] = __fmul_rn(2.0f, EL[k]);
    }
    const bool r1 = region == 1, r2 = region == 2;
    uint32_t h0 = lk(lb, xb7), h1 = lk(lb, xb7 + 128);
    uint32_t h00 = lk(lb, (int)h0 + yb7), h01 = lk(lb, (int)h0 + yb7 + 128);
    uint32_t h10 = lk(lb, (int)h1 + yb7), h11 = lk(lb, (int)h1 + yb7 + 128);
    const int zo0 = zb7, zo1 = zb7 + 128;
    const uint32_t w0 = lk(lb, r1 ? (int)h11 + zo1 : (int)h00 + zo0);
    const uint32_t w100 = lk(lb, (int)h10 + zo0), w010 = lk(lb, (int)h01 + zo0), w001 = lk(lb, (int)h00 + zo1);
    const uint32_t w110 = lk(lb, (int)h11 + zo0), w101 = lk(lb, (int)h10 + zo1), w011 = lk(lb, (int)h01 + zo1);
    const int xm = xb7 - 128, ym = yb7 - 128, zm = zb7 - 128;
    const uint32_t we0 = lk_extra(lb, xm, ym, zm, ew0), we1 = lk_extra(lb, xm, ym, zm, ew1);
    // fixed corners per lane (offsets o + (ox + oy + oz)/3 in thirds: A1 =
    // (1,0,0) -> (4,1,1)/3, A2 (1,4,1)/3, A3 (1,1,4)/3, B1 = (1,1,0) ->
    // (5,5,2)/3, B2 (5,2,5)/3, B3 (2,5,5)/3; corner 0: (0,0,0) or (2,2,2));
    // A-corners' anchored lo is -C3L, B-corners' +C3L, the corner's 0
    const float pL2 = C3L2;
    //   X1: r2 ? A1 : corner 0       X2: r2 ? A2 : (r1 ? B1 : A1)
    //   X3: r2 ? A3 : (r1 ? B2 : A2) X4: r2 ? B1 : (r1 ? B3 : A3)
    //   X5: B2, X6: B3 (octahedron only)
    const uint32_t wX1 = r2 ? w100 : w0, wX2 = r2 ? w010 : (r1 ? w110 : w100);
    const uint32_t wX3 = r2 ? w001 : (r1 ? w101 : w010), wX4 = r2 ? w110 : (r1 ? w011 : w001);
    const float4 c0 = s_corner[region], c1 = s_corner[4 + region], c2 = s_corner[8 + region], c3 = s_corner[12 + region];
    const float fr2 = r2 ? 1.0f : 0.0f;
    const float bias = NORM ? 0.0f : ACC_BIAS;
    float2 AH = f2(bias, bias), AL = f2(0.0f, 0.0f);
    const float2 none = f2(1.0f, 1.0f), l12 = f2(c1.z, c1.w), l34 = f2(c3.z, c3.w);
    contrib2_pair<NORM, false>(wX1, wX2, X0H, X0L2, Y0H, Y0L2, Z0H, Z0L2, f2(c0.x, c0.y), l12, f2(c0.z, c0.w), l12,
                               f2(c1.x, c1.y), l12, none, AH, AL);
    contrib2_pair<NORM, false>(wX3, wX4, X0H, X0L2, Y0H, Y0L2, Z0H, Z0L2, f2(c2.x, c2.y), l34, f2(c2.z, c2.w), l34,
                               f2(c3.x, c3.y), l34, none, AH, AL);
    contrib2_pair<NORM, true>(w101, w011, X0H, X0L2, Y0H, Y0L2, Z0H, Z0L2, f2(T5H, T2H), f2(pL2, pL2), f2(T2H, T5H),
                              f2(pL2, pL2), f2(T5H, T5H), f2(pL2, pL2), f2(fr2, fr2), AH, AL);
    contrib2_pair<NORM, false>(we0, we1, X0H, X0L2, Y0H, Y0L2, Z0H, Z0L2, f2(EH[0], EH[3]), f2(EL2[0], EL2[3]),
                               f2(EH[1], EH[4]), f2(EL2[1], EL2[4]), f2(EH[2], EH[5]), f2(EL2[2], EL2[5]), none, AH, AL);
    if (!NORM) AH = f2(__fsub_rn(AH.x, ACC_BIAS), __fsub_rn(AH.y, ACC_BIAS));     // exact
    float e;
    two_sum1(AH.x, AH.y, vh, e);
    vl = __fadd_rn(e, __fadd_rn(AL.x, AL.y));
    if (NORM) {                       // without NORM the dot products carry a factor 1/4 (exact)
        vh = __fmul_rn(vh, 0.25f);
        vl = __fmul_rn(vl, 0.25f);
    }
}

// The octave's term (v/103 + 1) * amp added to the running pair (rh, rl),
// then renormalised (|rl| <= ulp(rh)/2).
__device__ __forceinline__ void octave_accumulate(float vh, float vl, float amph, float ampl, float &rh, float &rl)
{
    constexpr float R103 = 4.0f / 103.0f;
    const float wq = __fmul_rn(vh, R103);
    const float rem = __fmaf_rn(-wq, 25.75f, vh);                 // exact
    const float wl = __fmul_rn(__fadd_rn(rem, vl), R103);
    const float s = __fadd_rn(1.0f, wq);                          // |wq| <= 1: fast two-sum
    const float lo = __fadd_rn(__fadd_rn(__fsub_rn(1.0f, s), wq), wl);
    const float th = __fmul_rn(s, amph);
    float tl = __fmaf_rn(s, amph, -th);
    tl = __fmaf_rn(s, ampl, __fmaf_rn(lo, amph, tl));
    float sh, se;
    two_sum1(rh, th, sh, se);
    const float sl = __fadd_rn(rl, __fadd_rn(se, tl));
    rh = __fadd_rn(sh, sl);
    rl = __fsub_rn(sl, __fsub_rn(rh, sh));
}

// Split a binary64 into three binary32s x1 + x2 + x3 == v exactly, with
// integer operations (GB300's binary64 pipe is narrow): x1 = the top 24
// significant bits, x2 = the next 23 as an integer times 2^(e-46), x3 = the
// last 6 times 2^(e-52).  Needs 2^-74 <= |v| < 2^128 (the scales stay
// normal binary32s); v = 0 gives zeros.  Other magnitudes give x1 =
// (float)v and zeros: outside what the planet paths use (unit or
// radius-scaled vertices), and such a coordinate only loses its low bits.
__device__ __forceinline__ void split3_f64(double v, float &x1, float &x2, float &x3)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const uint32_t hw = (uint32_t)(b >> 32), lw = (uint32_t)b;
    const int e = (int)((hw >> 20) & 0x7FF) - 1023;
    const uint32_t sign = hw & 0x80000000u;
    if (e < -74 || e > 127) {
        x1 = (float)v;
        x2 = 0.0f;
        x3 = 0.0f;
        return;
    }
    // top 24 bits: the implicit one and 23 fraction bits (bits 51-29)
    x1 = __uint_as_float(sign | ((uint32_t)(e + 127) << 23) | ((hw & 0xFFFFFu) << 3) | (lw >> 29));
    // next 23 bits (28-6) and last 6 (5-0), as exact integers scaled by 2^(e-46) and 2^(e-52)
    const uint32_t m2 = (lw >> 6) & 0x7FFFFFu, m3 = lw & 0x3Fu;
    const float i2 = __fsub_rn(__uint_as_float(0x4B000000u | m2), 8388608.0f);
    const float i3 = __fsub_rn(__uint_as_float(0x4B000000u | m3), 8388608.0f);
    const float t2 = __fmul_rn(i2, __uint_as_float((uint32_t)(e + 81) << 23));
    const float t3 = __fmul_rn(i3, __uint_as_float((uint32_t)(e + 75) << 23));
    x2 = __uint_as_float(__float_as_uint(t2) | sign);
    x3 = __uint_as_float(__float_as_uint(t3) | sign);
}

// Ordered-key transform: unsigned comparisons of keys follow float order.
__device__ __forceinline__ uint32_t fkey(float f)
{
    uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b ^ 0x80000000u);
}

// Ordered 64-bit key of a normalised pair: unsigned key order = value order.
__device__ __forceinline__ unsigned long long pair_key(float h, float l)
{
    return ((unsigned long long)fkey(h) << 32) | (unsigned long long)fkey(l);
}

__device__ __forceinline__ uint32_t lane_base() { return (threadIdx.x & 31u) << 2; }

__global__ void __launch_bounds__(256) fbm_kernel(const double *__restrict__ xyz, int64_t n,
                                                  const int32_t *__restrict__ perm,
                                                  const int32_t *__restrict__ pgi, FbmParams P,
                                                  double *__restrict__ out64, float *__restrict__ out32,
                                                  int accumulate, unsigned long long *nfb_out)
{
    build_table<false>(perm, pgi);
    init_grad_table<false>();
    init_extra_table();
    init_corner32_table((int)threadIdx.x);
    __syncthreads();
    const uint32_t lb = lane_base();
    unsigned nfb = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        double X = xyz[3 * i], Y = xyz[3 * i + 1], Z = xyz[3 * i + 2];
        float xh, xl, yh, yl, zh, zl;
        split_f64(X, xh, xl);
        split_f64(Y, yh, yl);
        split_f64(Z, zh, zl);
        float acc = 0.0f;
        for (int o = 0; o < P.n_oct; ++o) {
            float v = noise_raw<false>(xh, xl, yh, yl, zh, zl, P.s_hi[o], P.s_lo[o], X, Y, Z, P.s[o], lb,
                                       nfb, nullptr, nullptr);
            // (noise + 1) * 0.5 * strength * radius, noise = v / 103
            acc = fmaf(v, P.amp[o], acc);
        }
        acc += P.base;
        if (out64) out64[i] = accumulate ? out64[i] + (double)acc : (double)acc;
        if (out32) out32[i] = accumulate ? out32[i] + acc : acc;
    }
    if (nfb_out) {
        unsigned tot = __reduce_add_sync(0xFFFFFFFFu, nfb);
        if ((threadIdx.x & 31) == 0 && tot) atomicAdd(nfb_out, (unsigned long long)tot);
    }
}

__global__ void __launch_bounds__(256) trace_kernel(const double *__restrict__ xyz, int64_t n,
                                                    const int32_t *__restrict__ perm,
                                                    const int32_t *__restrict__ pgi, double s,
                                                    float *__restrict__ value, int32_t *__restrict__ trace,
                                                    int32_t *__restrict__ slots,
                                                    unsigned long long *nfb_out)
{
    build_table<false>(perm, pgi);
    init_grad_table<false>();
    init_extra_table();
    init_corner32_table((int)threadIdx.x);
    __syncthreads();
    const uint32_t lb = lane_base();
    float sh, sl;
    split_f64(s, sh, sl);
    unsigned nfb = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        double X = xyz[3 * i], Y = xyz[3 * i + 1], Z = xyz[3 * i + 2];
        float xh, xl, yh, yl, zh, zl;
        split_f64(X, xh, xl);
        split_f64(Y, yh, yl);
        split_f64(Z, zh, zl);
        int32_t tr[10], s9[45];
        float v = noise_raw<true>(xh, xl, yh, yl, zh, zl, sh, sl, X, Y, Z, s, lb, nfb, tr, s9);
        value[i] = v * (1.0f / 103.0f);
        if (trace)
            for (int k = 0; k < 10; ++k) trace[10 * i + k] = tr[k];
        if (slots)
            for (int k = 0; k < 45; ++k) slots[45 * i + k] = s9[k];
    }
    if (nfb_out) {
        unsigned tot = __reduce_add_sync(0xFFFFFFFFu, nfb);
        if ((threadIdx.x & 31) == 0 && tot) atomicAdd(nfb_out, (unsigned long long)tot);
    }
}


constexpr int CHUNK = 2048;   // vertices per work item of the batched kernel

__device__ __forceinline__ int chunk_planet(const nx_fbm_planet *P, int np, int c)
{
    int lo = 0, hi = np - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (P[mid].chunk0 <= c) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Threads of a pair block: one block of 512 per SM (128 registers a thread).
// Measured (GB300, 12 octaves of 10,000,002 vertices, before the shorter
// chains above, which take 2.75 ms now): 3.13 ms, against 3.38 ms for two
// blocks of 256 (each with a table of its own), 3.63 ms for three
// of 192, 3.74 ms for one of 640 and 3.90 ms for two of 320 (96 registers:
// more warps, but longer dependent stretches).
constexpr int PAIR_THREADS = 512;
constexpr int PAIR_WARPS = PAIR_THREADS / 32;

// A block's step: PAIR_THREADS / S vertices, their octaves dealt out to S
// groups of warps (S a power of two up to 16).  S = 1 where there are vertices
// for every warp; small spheres and the remainder of large ones are split, so
// that they fill the GPU with fewer octaves each: a warp's octave takes ~6 us
// however few there are.  Measured (GB300, 12 octaves): 1,442 vertices 47.5
// -> 14.9 us, 19,456 48.4 -> 21.7 us, 77,824 59.2 -> 55.3 us.
constexpr int SPLIT_MAX = 16;

// Shared memory of the octaves' values of a split step.
static size_t split_bytes(int S, int n_oct) { return S > 1 ? sizeof(float2) * (size_t)(PAIR_THREADS / S) * (size_t)n_oct : 0; }

// The largest split with which `vertices` make no more than `blocks` steps.
static int split_for(int64_t vertices, int blocks, int n_oct)
{
    int S = 1;
    while (2 * S <= SPLIT_MAX && S < n_oct && (vertices * 2 * S + PAIR_THREADS - 1) / PAIR_THREADS <= blocks) S *= 2;
    return S;
}

// Steps of a batched launch: block b takes steps [first[b], first[b + 1]) in
// order, the ranges cut so that each block gets an equal share of the
// estimated cost (vertices x octaves, renormalised octaves weighted 9/8).
constexpr int FBM_SPLIT_MAX = 2048;
struct FbmSplit {
    int S;                              // octave split
    int first[FBM_SPLIT_MAX + 1];
};

// Fold the ordered keys (kmn, kmx) of the block's sums of planet P into its
// min/max (a block barrier; the whole block calls it).
__device__ __forceinline__ void fold_minmax(const nx_fbm_planet &P, unsigned long long kmn, unsigned long long kmx,
                                            unsigned long long (*s_mm)[PAIR_WARPS])
{
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long a = __shfl_xor_sync(0xFFFFFFFFu, kmn, o);
        const unsigned long long b = __shfl_xor_sync(0xFFFFFFFFu, kmx, o);
        kmn = a < kmn ? a : kmn;
        kmx = b > kmx ? b : kmx;
    }
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) { s_mm[0][w] = kmn; s_mm[1][w] = kmx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long a0 = s_mm[0][0], a1 = s_mm[1][0];
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) {
            a0 = s_mm[0][k] < a0 ? s_mm[0][k] : a0;
            a1 = s_mm[1][k] > a1 ? s_mm[1][k] : a1;
        }
        atomicMin(&P.minmax[0], a0);
        atomicMax(&P.minmax[1], a1);
    }
    __syncthreads();
}

// One vertex's binary32 triples.
struct Triples {
    float x1, x2, x3, y1, y2, y3, z1, z2, z3;
};

__device__ __forceinline__ Triples load_triples(const double *__restrict__ xyz, int64_t i)
{
    Triples t;
    split3_f64(xyz[3 * i], t.x1, t.x2, t.x3);
    split3_f64(xyz[3 * i + 1], t.y1, t.y2, t.y3);
    split3_f64(xyz[3 * i + 2], t.z1, t.z2, t.z3);
    return t;
}

__device__ __forceinline__ void octave_value(const Triples &t, const OctP &O, bool norm, bool pow2, uint32_t lb,
                                             unsigned &nfb, float &vh, float &vl)
{
    if (norm) noise_pair<true>(t.x1, t.x2, t.x3, t.y1, t.y2, t.y3, t.z1, t.z2, t.z3, O, pow2, lb, nfb, vh, vl);
    else noise_pair<false>(t.x1, t.x2, t.x3, t.y1, t.y2, t.y3, t.z1, t.z2, t.z3, O, pow2, lb, nfb, vh, vl);
}

// The block's constant tables, by its upper warps (the hash table's words are
// filled by the lower ones meanwhile).
__device__ __forceinline__ void init_pair_tables()
{
    static_assert(PAIR_THREADS == 512, "threads 256-351, 448-459 and 480-495 fill the small tables");
    init_grad_table<true>();
    init_extra_table_pair((int)threadIdx.x - 256);
    init_corner_table((int)threadIdx.x - 448);
    init_third_table((int)threadIdx.x - 480);
}

// Octave o's constants of a planet descriptor or a launch's parameters.
__device__ __forceinline__ OctP oct_of(const nx_fbm_planet &P, int o)
{
    OctP O;
    O.s1 = P.s1[o]; O.s2 = P.s2[o]; O.s3 = P.s3[o];
    O.amph = P.amp_hi[o]; O.ampl = P.amp_lo[o]; O.s = P.s[o];
    return O;
}

// The sum over P's octaves at one vertex, added to (rh, rl).
template <typename P_t>
__device__ __forceinline__ void sum_octaves(const P_t &P, int n_oct, const Triples &t, bool pow2, uint32_t lb,
                                            unsigned &nfb, float &rh, float &rl)
{
    for (int o = 0; o < n_oct; ++o) {
        const OctP O = oct_of(P, o);
        float vh, vl;
        octave_value(t, O, (P.norm_mask >> o) & 1u, pow2, lb, nfb, vh, vl);
        octave_accumulate(vh, vl, O.amph, O.ampl, rh, rl);
    }
}

// The same by a whole block for one step's PAIR_THREADS / S vertices from
// `first` on: the sum is valid in threads below PAIR_THREADS / S (vertex first +
// thread), the octaves summed there in order, so the bits do not depend on S.
template <typename P_t>
__device__ __forceinline__ void sum_split(const P_t &P, int n_oct, const double *__restrict__ xyz, int64_t first,
                                          int64_t last, int S, bool pow2, uint32_t lb, float2 *part, unsigned &nfb,
                                          float &rh, float &rl)
{
    const int U = PAIR_THREADS / S, q = threadIdx.x % U;
    const int64_t i = first + q;
    // (past the end: the last vertex again, so that warps stay whole)
    const Triples t = load_triples(xyz, i < last ? i : last - 1);
    unsigned extra = 0;
    for (int o = threadIdx.x / U; o < n_oct; o += S) {
        const OctP O = oct_of(P, o);
        float vh, vl;
        octave_value(t, O, (P.norm_mask >> o) & 1u, pow2, lb, extra, vh, vl);
        part[o * U + q] = make_float2(vh, vl);
    }
    if (i < last) nfb += extra;
    __syncthreads();
    if ((int)threadIdx.x < U)
        for (int o = 0; o < n_oct; ++o) {
            const OctP O = oct_of(P, o);
            const float2 v = part[o * U + q];
            octave_accumulate(v.x, v.y, O.amph, O.ampl, rh, rl);
        }
    __syncthreads();
}

// Many planets in one persistent launch: work items are steps of
// PAIR_THREADS / S vertices of one planet (CHUNK vertices hold S CHUNK /
// PAIR_THREADS of them); each block walks its contiguous range of steps
// (so it meets few planets), rebuilding its shared table when the planet
// changes.  Sums are pairs (pair path above); the ordered keys of a block's
// sums of a planet are folded into the planet's min/max once, when the
// block leaves the planet (for the rescale to metres that follows).
template <bool SPLIT>
__global__ void __launch_bounds__(PAIR_THREADS, 1) fbm_batch_kernel(const nx_fbm_planet *__restrict__ planets, int np,
                                                                    const __grid_constant__ FbmSplit split,
                                                                    unsigned long long *nfb_out)
{
    __shared__ unsigned long long s_mm[2][PAIR_WARPS];
    init_pair_tables();
    __syncthreads();
    const uint32_t lb = lane_base();
    float2 *part = reinterpret_cast<float2 *>(smem + TABLE_WORDS);
    const int S = SPLIT ? split.S : 1, U = PAIR_THREADS / S, per = CHUNK / U;
    const int u0 = split.first[blockIdx.x], u1 = split.first[blockIdx.x + 1];
    int cur = -1;
    unsigned nfb = 0;
    unsigned long long kmn = ~0ull, kmx = 0ull;
    for (int u = u0; u < u1; ++u) {
        const int c = u / per;
        int p = cur < 0 ? chunk_planet(planets, np, c) : cur;
        while (p + 1 < np && planets[p + 1].chunk0 <= c) ++p;
        if (p != cur) {
            if (cur >= 0 && planets[cur].minmax) fold_minmax(planets[cur], kmn, kmx, s_mm);
            kmn = ~0ull;
            kmx = 0ull;
            __syncthreads();
            build_table<true>(planets[p].perm, planets[p].pgi);
            __syncthreads();
            cur = p;
        }
        const nx_fbm_planet &P = planets[p];
        const int64_t first = (int64_t)(c - P.chunk0) * CHUNK + (int64_t)(u - c * per) * U;
        if (first >= P.n) continue;
        const bool pow2 = P.pow2 != 0;
        float rh = 0.0f, rl = 0.0f;
        const int64_t i = first + threadIdx.x;
        bool mine = i < P.n;
        if (!SPLIT) {
            if (mine) sum_octaves(P, P.n_octaves, load_triples(P.xyz, i), pow2, lb, nfb, rh, rl);
        } else {
            sum_split(P, P.n_octaves, P.xyz, first, P.n, S, pow2, lb, part, nfb, rh, rl);
            mine = mine && (int)threadIdx.x < U;
        }
        if (mine) {
            reinterpret_cast<float2 *>(P.out)[i] = make_float2(rh, rl);
            const unsigned long long k = pair_key(rh, rl);
            kmn = k < kmn ? k : kmn;
            kmx = k > kmx ? k : kmx;
        }
    }
    if (cur >= 0 && planets[cur].minmax) fold_minmax(planets[cur], kmn, kmx, s_mm);
    if (nfb_out) {
        unsigned tot = __reduce_add_sync(0xFFFFFFFFu, nfb);
        if ((threadIdx.x & 31) == 0 && tot) atomicAdd(nfb_out, (unsigned long long)tot);
    }
}

// Per-octave constants of a single-planet pair launch.
struct FbmPairParams {
    int n_oct;
    int pow2;
    uint32_t norm_mask;   // bit o: octave o renormalises its displacements
    float s1[NX_MAX_OCTAVES], s2[NX_MAX_OCTAVES], s3[NX_MAX_OCTAVES];
    float amph[NX_MAX_OCTAVES], ampl[NX_MAX_OCTAVES];
    double s[NX_MAX_OCTAVES];
};

// One planet, the pair path: the octaves of P (any subset of a planet's
// octaves: the plain path launches NX_MAX_OCTAVES at a time, accumulate = 1
// after the first) added to the running pair sums in out2 (float2 per vertex),
// and/or written as binary64 (out64, = hi + lo exactly; accumulate adds to
// it).  minmax (optional): ordered keys of the resulting pair sums.
//
// Vertices [begin, n): a thread a vertex, or (SPLIT) a step of S octave
// groups to a block.
__device__ __forceinline__ OctP oct_of(const FbmPairParams &P, int o)
{
    OctP O;
    O.s1 = P.s1[o]; O.s2 = P.s2[o]; O.s3 = P.s3[o];
    O.amph = P.amph[o]; O.ampl = P.ampl[o]; O.s = P.s[o];
    return O;
}

template <bool SPLIT>
__global__ void __launch_bounds__(PAIR_THREADS, 1) fbm_pair_kernel(const double *__restrict__ xyz, int64_t begin,
                                                                   int64_t n, int S, const int32_t *__restrict__ perm,
                                                                   const int32_t *__restrict__ pgi,
                                                                   const __grid_constant__ FbmPairParams P,
                                                                   float2 *__restrict__ out2,
                                                                   double *__restrict__ out64, int accumulate,
                                                                   unsigned long long *minmax,
                                                                   unsigned long long *nfb_out)
{
    __shared__ unsigned long long s_mm[2][PAIR_WARPS];
    build_table<true>(perm, pgi);
    init_pair_tables();
    __syncthreads();
    const uint32_t lb = lane_base();
    float2 *part = reinterpret_cast<float2 *>(smem + TABLE_WORDS);
    unsigned nfb = 0;
    unsigned long long kmn = ~0ull, kmx = 0ull;
    const bool pow2 = P.pow2 != 0;
    auto put = [&](int64_t i, float rh, float rl) {
        if (out2) out2[i] = make_float2(rh, rl);
        if (out64) {
            const double v = (double)rh + (double)rl;
            out64[i] = (accumulate && !out2) ? out64[i] + v : v;
        }
        const unsigned long long k = pair_key(rh, rl);
        kmn = k < kmn ? k : kmn;
        kmx = k > kmx ? k : kmx;
    };
    const bool running = accumulate && out2;
    if (!SPLIT) {
        for (int64_t i = begin + (int64_t)blockIdx.x * PAIR_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * PAIR_THREADS) {
            const float2 v = running ? out2[i] : make_float2(0.0f, 0.0f);
            float rh = v.x, rl = v.y;
            sum_octaves(P, P.n_oct, load_triples(xyz, i), pow2, lb, nfb, rh, rl);
            put(i, rh, rl);
        }
    } else {
        const int U = PAIR_THREADS / S;
        const int64_t first = begin + (int64_t)blockIdx.x * U, i = first + threadIdx.x;
        const bool mine = i < n && (int)threadIdx.x < U;
        const float2 v = running && mine ? out2[i] : make_float2(0.0f, 0.0f);
        float rh = v.x, rl = v.y;
        if (first < n) sum_split(P, P.n_oct, xyz, first, n, S, pow2, lb, part, nfb, rh, rl);
        if (mine) put(i, rh, rl);
    }
    if (minmax) {
        nx_fbm_planet out;
        out.minmax = minmax;
        fold_minmax(out, kmn, kmx, s_mm);
    }
    if (nfb_out) {
        unsigned tot = __reduce_add_sync(0xFFFFFFFFu, nfb);
        if ((threadIdx.x & 31) == 0 && tot) atomicAdd(nfb_out, (unsigned long long)tot);
    }
}

int grid_for(int64_t n, int block, const void *kernel, int smem)
{
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem);
    if (per_sm < 1) per_sm = 1;
    int64_t need = (n + block - 1) / block;
    int64_t g = (int64_t)nx::sm_count() * per_sm;
    if (need < g) g = need;
    return (int)(g < 1 ? 1 : g);
}

bool smem_configured = false;

int configure_smem()
{
    if (smem_configured) return NX_OK;
    NX_CHECK_CUDA(cudaFuncSetAttribute(fbm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TABLE_BYTES));
    NX_CHECK_CUDA(cudaFuncSetAttribute(trace_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TABLE_BYTES));
    const int pair_bytes = TABLE_BYTES + (int)split_bytes(2, NX_MAX_OCTAVES);
    NX_CHECK_CUDA(cudaFuncSetAttribute(fbm_batch_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_bytes));
    NX_CHECK_CUDA(cudaFuncSetAttribute(fbm_batch_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TABLE_BYTES));
    NX_CHECK_CUDA(cudaFuncSetAttribute(fbm_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_bytes));
    NX_CHECK_CUDA(cudaFuncSetAttribute(fbm_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TABLE_BYTES));
    smem_configured = true;
    return NX_OK;
}

}  // namespace

namespace nx {
void note_launch(int k);
}

NX_EXPORT int nx_fbm(const double *xyz_dev, int64_t n, const int32_t *perm_dev, const int32_t *pgi_dev,
                     int n_octaves, const double *scale, const double *strength, double radius,
                     double *elev_f64_dev, float *elev_f32_dev, int accumulate,
                     unsigned long long *n_fallback_dev, void *stream)
{
    if (n < 0) return nx::fail(NX_EINVAL, "nx_fbm: n < 0");
    if (n_octaves < 0 || n_octaves > NX_MAX_OCTAVES)
        return nx::fail(NX_EINVAL, "nx_fbm: n_octaves must be in [0, %d]", NX_MAX_OCTAVES);
    if (n == 0) return NX_OK;
    if (!xyz_dev || !perm_dev || !pgi_dev || (n_octaves > 0 && (!scale || !strength)))
        return nx::fail(NX_EINVAL, "nx_fbm: null pointer");
    if (!elev_f64_dev && !elev_f32_dev) return nx::fail(NX_EINVAL, "nx_fbm: no output");
    FbmParams P;
    P.n_oct = n_octaves;
    double base = 0.0;
    for (int o = 0; o < n_octaves; ++o) {
        double s = scale[o];
        float hi = (float)s;
        float lo = (float)(s - (double)hi);
        P.s_hi[o] = hi;
        P.s_lo[o] = lo;
        P.s[o] = s;
        P.amp[o] = (float)(0.5 * strength[o] * radius / 103.0);
        base += 0.5 * strength[o] * radius;
    }
    P.base = (float)base;
    int rc = configure_smem();
    if (rc) return rc;
    int grid = grid_for(n, 256, (const void *)fbm_kernel, TABLE_BYTES);
    fbm_kernel<<<grid, 256, TABLE_BYTES, (cudaStream_t)stream>>>(xyz_dev, n, perm_dev, pgi_dev, P, elev_f64_dev,
                                                                 elev_f32_dev, accumulate, n_fallback_dev);
    NX_CHECK_LAUNCH("fbm_kernel");
    nx::note_launch(1);
    return NX_OK;
}

NX_EXPORT int nx_sample_octaves(const double *xyz_dev, int64_t n, const int32_t *perm_dev,
                                const int32_t *pgi_dev, int n_octaves, double n_init_roughness,
                                double n_init_strength, double n_roughness, double n_persistence,
                                double world_radius, double *elev_f64_dev, float *elev_f32_dev,
                                int accumulate, void *stream)
{
    if (n_octaves < 0 || n_octaves > NX_MAX_OCTAVES)
        return nx::fail(NX_EINVAL, "nx_sample_octaves: n_octaves must be in [0, %d]", NX_MAX_OCTAVES);
    double scale[NX_MAX_OCTAVES], strength[NX_MAX_OCTAVES];
    // terrain.py:35-46: the per-octave arguments, in binary64 as the reference
    double f = n_init_roughness, a = n_init_strength;
    for (int o = 0; o < n_octaves; ++o) {
        scale[o] = f / world_radius;
        strength[o] = a / world_radius;
        f *= n_roughness;
        a *= n_persistence;
    }
    return nx_fbm(xyz_dev, n, perm_dev, pgi_dev, n_octaves, scale, strength, world_radius, elev_f64_dev,
                  elev_f32_dev, accumulate, nullptr, stream);
}

NX_EXPORT int nx_noise3d_trace(const double *xyz_dev, int64_t n, const int32_t *perm_dev,
                               const int32_t *pgi_dev, double scale, float *value_dev, int32_t *trace_dev,
                               int32_t *slots_dev, unsigned long long *n_fallback_dev, void *stream)
{
    if (n < 0) return nx::fail(NX_EINVAL, "nx_noise3d_trace: n < 0");
    if (n == 0) return NX_OK;
    if (!xyz_dev || !perm_dev || !pgi_dev || !value_dev)
        return nx::fail(NX_EINVAL, "nx_noise3d_trace: null pointer");
    int rc = configure_smem();
    if (rc) return rc;
    int grid = grid_for(n, 256, (const void *)trace_kernel, TABLE_BYTES);
    trace_kernel<<<grid, 256, TABLE_BYTES, (cudaStream_t)stream>>>(xyz_dev, n, perm_dev, pgi_dev, scale,
                                                                   value_dev, trace_dev, slots_dev,
                                                                   n_fallback_dev);
    NX_CHECK_LAUNCH("trace_kernel");
    nx::note_launch(1);
    return NX_OK;
}

// scale as an exact triple of binary32s and whether it is a power of two
static void split_scale(double v, float &a, float &b, float &c)
{
    a = (float)v;
    const double r = v - (double)a;      // exact
    b = (float)r;
    c = (float)(r - (double)b);          // exact (the few bits left)
}

static bool is_pow2(double v)
{
    int e = 0;
    return v > 0.0 && std::frexp(v, &e) == 0.5;
}

// Octaves whose displacements are renormalised (bit o): those with
// |0.5 strength radius| >= ref / 8, ref = amp_ref if positive, else the
// largest amplitude among the given octaves.
static uint32_t norm_mask(int n_octaves, const double *strength, double radius, double amp_ref)
{
    double ref = amp_ref;
    if (!(ref > 0.0))
        for (int o = 0; o < n_octaves; ++o) ref = std::fmax(ref, std::fabs(0.5 * strength[o] * radius));
    uint32_t m = 0;
    for (int o = 0; o < n_octaves; ++o)
        if (std::fabs(0.5 * strength[o] * radius) >= ref / 8.0) m |= 1u << o;
    return m;
}

static int check_octaves(int n_octaves, const double *scale, const double *strength, const char *who)
{
    if (n_octaves < 0 || n_octaves > NX_MAX_OCTAVES)
        return nx::fail(NX_EINVAL, "%s: n_octaves must be in [0, %d]", who, NX_MAX_OCTAVES);
    if (n_octaves && (!scale || !strength)) return nx::fail(NX_EINVAL, "%s: null scale or strength", who);
    for (int o = 0; o < n_octaves; ++o)
        if (!std::isfinite(scale[o]) || !std::isfinite(strength[o]) || std::fabs(scale[o]) > 1e30)
            return nx::fail(NX_EINVAL, "%s: octave %d: scale and strength must be finite", who, o);
    return NX_OK;
}

NX_EXPORT int nx_fbm_planet_fill(nx_fbm_planet *planet, int n_octaves, const double *scale, const double *strength,
                                 double radius)
{
    if (!planet) return nx::fail(NX_EINVAL, "nx_fbm_planet_fill: null planet");
    int rc = check_octaves(n_octaves, scale, strength, "nx_fbm_planet_fill");
    if (rc) return rc;
    planet->n_octaves = n_octaves;
    bool pow2 = true;
    for (int o = 0; o < NX_MAX_OCTAVES; ++o) {
        const double sc = o < n_octaves ? scale[o] : 0.0;
        split_scale(sc, planet->s1[o], planet->s2[o], planet->s3[o]);
        planet->s[o] = sc;
        const double amp = o < n_octaves ? 0.5 * strength[o] * radius : 0.0;
        planet->amp_hi[o] = (float)amp;
        planet->amp_lo[o] = (float)(amp - (double)planet->amp_hi[o]);
        if (o < n_octaves && !is_pow2(sc)) pow2 = false;
    }
    planet->pow2 = pow2 ? 1 : 0;
    planet->norm_mask = norm_mask(n_octaves, strength, radius, 0.0);
    return NX_OK;
}

NX_EXPORT int nx_fbm_pair(const double *xyz_dev, int64_t n, const int32_t *perm_dev, const int32_t *pgi_dev,
                          int n_octaves, const double *scale, const double *strength, double radius, double amp_ref,
                          float *pair_dev, double *elev_f64_dev, int accumulate, unsigned long long *minmax_dev,
                          unsigned long long *n_fallback_dev, void *stream)
{
    if (n < 0) return nx::fail(NX_EINVAL, "nx_fbm_pair: n < 0");
    int rc = check_octaves(n_octaves, scale, strength, "nx_fbm_pair");
    if (rc) return rc;
    if (n == 0) return NX_OK;
    if (!xyz_dev || !perm_dev || !pgi_dev) return nx::fail(NX_EINVAL, "nx_fbm_pair: null pointer");
    if (!pair_dev && !elev_f64_dev) return nx::fail(NX_EINVAL, "nx_fbm_pair: no output");
    if (pair_dev && ((uintptr_t)pair_dev & 7u)) return nx::fail(NX_EINVAL, "nx_fbm_pair: pair output must be 8-byte aligned");
    FbmPairParams P;
    P.n_oct = n_octaves;
    bool pow2 = true;
    for (int o = 0; o < NX_MAX_OCTAVES; ++o) {
        const double sc = o < n_octaves ? scale[o] : 0.0;
        split_scale(sc, P.s1[o], P.s2[o], P.s3[o]);
        P.s[o] = sc;
        const double amp = o < n_octaves ? 0.5 * strength[o] * radius : 0.0;
        P.amph[o] = (float)amp;
        P.ampl[o] = (float)(amp - (double)P.amph[o]);
        if (o < n_octaves && !is_pow2(sc)) pow2 = false;
    }
    P.pow2 = pow2 ? 1 : 0;
    P.norm_mask = norm_mask(n_octaves, strength, radius, amp_ref);
    rc = configure_smem();
    if (rc) return rc;
    // whole rounds of one block per SM, then the remainder by octaves (a
    // round of its own, however few its vertices, would take as long as a
    // warp's octaves one after the other)
    const int sms = nx::sm_count();
    const int64_t round = (int64_t)sms * PAIR_THREADS, rest = n % round;
    const int S = split_for(rest, sms, n_octaves);
    const int64_t main = S > 1 ? n - rest : n;
    if (main > 0) {
        const int64_t blocks = (main + PAIR_THREADS - 1) / PAIR_THREADS;
        fbm_pair_kernel<false><<<(int)(blocks < sms ? blocks : sms), PAIR_THREADS, TABLE_BYTES, (cudaStream_t)stream>>>(
            xyz_dev, 0, main, 1, perm_dev, pgi_dev, P, (float2 *)pair_dev, elev_f64_dev, accumulate, minmax_dev,
            n_fallback_dev);
        NX_CHECK_LAUNCH("fbm_pair_kernel");
        nx::note_launch(1);
    }
    if (main < n) {
        const int64_t steps = (rest * S + PAIR_THREADS - 1) / PAIR_THREADS;
        fbm_pair_kernel<true><<<(int)steps, PAIR_THREADS, TABLE_BYTES + split_bytes(S, n_octaves), (cudaStream_t)stream>>>(
            xyz_dev, main, n, S, perm_dev, pgi_dev, P, (float2 *)pair_dev, elev_f64_dev, accumulate, minmax_dev,
            n_fallback_dev);
        NX_CHECK_LAUNCH("fbm_pair_kernel");
        nx::note_launch(1);
    }
    return NX_OK;
}

NX_EXPORT int nx_fbm_batch(const nx_fbm_planet *planets_dev, const nx_fbm_planet *planets_host, int nplanets,
                           unsigned long long *n_fallback_dev, void *stream)
{
    if (nplanets <= 0) return NX_OK;
    if (!planets_dev || !planets_host) return nx::fail(NX_EINVAL, "nx_fbm_batch: null pointer");
    int total = 0;
    for (int p = 0; p < nplanets; ++p) {
        const nx_fbm_planet &P = planets_host[p];
        if (P.n < 0 || (P.n > 0 && (!P.xyz || !P.perm || !P.pgi || !P.out)))
            return nx::fail(NX_EINVAL, "nx_fbm_batch: planet %d incomplete", p);
        if ((uintptr_t)P.out & 7u) return nx::fail(NX_EINVAL, "nx_fbm_batch: planet %d: out must be 8-byte aligned", p);
        if (P.n_octaves < 0 || P.n_octaves > NX_MAX_OCTAVES) return nx::fail(NX_EINVAL, "nx_fbm_batch: octaves");
        if (P.chunk0 != total)
            return nx::fail(NX_EINVAL, "nx_fbm_batch: planet %d chunk0 must be %d (chunks of %d vertices)", p, total,
                            CHUNK);
        total += (int)((P.n + CHUNK - 1) / CHUNK);
    }
    if (total == 0) return NX_OK;
    int rc = configure_smem();
    if (rc) return rc;
    int64_t vertices = 0;
    int max_oct = 0;
    for (int p = 0; p < nplanets; ++p) {
        vertices += planets_host[p].n;
        if (planets_host[p].n > 0 && planets_host[p].n_octaves > max_oct) max_oct = planets_host[p].n_octaves;
    }
    const int sms = nx::sm_count() < FBM_SPLIT_MAX ? nx::sm_count() : FBM_SPLIT_MAX;
    FbmSplit split;
    split.S = split_for(vertices, sms, max_oct);
    const int U = PAIR_THREADS / split.S, per_chunk = CHUNK / U;
    if ((int64_t)total * per_chunk > 0x7FFFFFFF) return nx::fail(NX_EINVAL, "nx_fbm_batch: too many vertices");
    const int steps = total * per_chunk;
    const int grid = steps < sms ? steps : sms;
    // cut the steps into grid ranges of equal estimated cost: a planet's
    // step costs its vertices x (8 per octave + 1 per renormalised octave)
    std::vector<int64_t> wchunk(nplanets), cum(nplanets + 1, 0);
    for (int p = 0; p < nplanets; ++p) {
        const nx_fbm_planet &P = planets_host[p];
        const uint32_t live = P.n_octaves >= 32 ? ~0u : ((1u << P.n_octaves) - 1u);
        wchunk[p] = 8 * (int64_t)P.n_octaves + (int64_t)__builtin_popcount(P.norm_mask & live);
        cum[p + 1] = cum[p] + wchunk[p] * P.n;
    }
    const int64_t tot = cum[nplanets];
    int p = 0;
    split.first[0] = 0;
    for (int b = 1; b <= grid; ++b) {
        if (b == grid || tot == 0) { split.first[b] = steps; continue; }
        // first step whose cost prefix reaches b * tot / grid
        const int64_t t = (int64_t)((__int128)tot * b / grid);
        while (p + 1 < nplanets && cum[p + 1] <= t) ++p;
        const nx_fbm_planet &P = planets_host[p];
        const int64_t per = wchunk[p] * U;
        int64_t k = per > 0 ? (t - cum[p] + per - 1) / per : 0;
        const int64_t nst = (P.n + CHUNK - 1) / CHUNK * per_chunk;
        if (k > nst) k = nst;
        int c = P.chunk0 * per_chunk + (int)k;
        if (c < split.first[b - 1]) c = split.first[b - 1];
        split.first[b] = c;
    }
    const auto kernel = split.S > 1 ? fbm_batch_kernel<true> : fbm_batch_kernel<false>;
    kernel<<<grid, PAIR_THREADS, TABLE_BYTES + split_bytes(split.S, max_oct), (cudaStream_t)stream>>>(
        planets_dev, nplanets, split, n_fallback_dev);
    NX_CHECK_LAUNCH("fbm_batch_kernel");
    nx::note_launch(1);
    return NX_OK;
}

NX_EXPORT int nx_fbm_chunk_size(void) { return CHUNK; }
