// nx_insolation.cu -- per-vertex insolation accumulated over sun positions.
//
// Replaces the loop of climate.sample_insolation calls (climate.py:415-444;
// driven over rotations as in brute_daily_insolation, climate.py:450-489).
// For one sun position (rotation theta about z, tilt tau about y) the
// reference adds, per vertex,
//   max(cos|lat|, 0) * max(cos lon, 0)
// with lat, lon of the rotated and tilted point (util.xyz2latlon,
// util.py:59-75).  For a vertex on the sphere of the given radius r this
// equals max(t, 0) / r with
//   t = A cos(theta) + B sin(theta) + C,  A = x cos(tau), B = -y cos(tau),
//   C = z sin(tau)
// (cos lat = sqrt(tx^2+ty^2)/r, cos lon = tx/sqrt(tx^2+ty^2)).  When the
// rotations come in pairs theta, theta + 180 degrees (every even uniform
// schedule, e.g. 24 hours of 15 degrees), the pair contributes
//   max(C+u, 0) + max(C-u, 0) = C + max(|C|, |u|),  u = A cos + B sin,
// i.e. two operations per sun position.  Vertices off that sphere
// (| |v|^2 - r^2 | > 1e-12 r^2) take the reference's general formula.
//
// With u = cos(tau) U(theta), U = x cos(theta) - y sin(theta) the same on
// every day, a day's pairs sum to n C + |cos tau| sum_h max(c, |U_h|),
// c = |z| |tan tau|.  Schedules of up to SORT_MAX days are then summed by
// breakpoints: each max picks one side, so over the year the sum is
// sum_h [ |U_h| (sum of |cos| over days with c < |U_h|) + |z| (sum of
// |cos| |tan| over the other days) ], both inner sums read from prefix /
// suffix sums over the days sorted by |tan tau| (built once per block).  A
// pair's value is a convex piecewise linear function of |U_h|, so a bucket
// table of line pairs gives it as the larger of two lines: twelve table
// reads per vertex for a year of hourly positions.  Longer schedules sum day
// by day (paired lanes, groups of 8 days, Kahan across groups).
//
// Schedules of many rotations (a day in one-degree steps) are summed by
// arcs: U(theta) + const > 0 holds on one arc of rotation angles, so a tilt
// costs one arc (an arc cosine, two searches in the sorted angles) and the
// difference of two prefix sums of (cos, sin) instead of a max per rotation.
//
// The vertices come in binary64; GB300 issues two binary64 operations per
// SM and cycle, so the kernels split them into binary32 pairs with integer
// operations and test ||v|^2 - r^2| in pairs: with the test in binary64 (8
// operations and 3 conversions per vertex) it alone took longer than the
// reading of the vertices.
#include "nx_common.cuh"

namespace nx {
void note_launch(int k);
}

namespace {

struct InsoArgs {
    const double *xyz;
    int64_t n;
    double r;
    float inv_r;
    float r2h, r2l;        // r^2 as a pair; r2h = 0: r outside [2^-20, 2^60] (binary64 test)
    float zmin;            // 1e-20 r: |z| of the breakpoint form is kept off 0
    const float2 *tilt;    // (cos tau, sin tau) per tilt
    int n_tilt;
    const float2 *rot;     // (cos theta, sin theta): all rotations, or the first half in pair mode
    int n_rot;             // number of entries in rot
    int pairs;             // 1: each rot entry stands for theta and theta + 180
    float *out;
    int accumulate;
    float scale;           // of the sums (1: none)
};

__host__ __device__ __forceinline__ void radius_pair(double r, float &h, float &l)
{
    h = l = 0.0f;
    if (!(r >= 0x1p-20 && r <= 0x1p60)) return;
    const double r2 = r * r;
    h = (float)r2;
    l = (float)(r2 - (double)h);
}

// |v| as h + l2 / 2, binary32s, by integer operations, for 2^-40 <= |v| <
// 2^61: h = the top 24 bits (truncated), l2 / 2 the next 23.  ah = the high
// word of |v|.
__device__ __forceinline__ void split_abs(uint32_t ah, uint32_t lw, float &h, float &l2)
{
    h = __uint_as_float(__funnelshift_l(lw, ah - (896u << 20), 3));
    const float i = __fsub_rn(__uint_as_float(0x4B000000u | ((lw >> 6) & 0x7FFFFFu)), 8388608.0f);
    l2 = __fmul_rn(i, __uint_as_float(((ah & 0x7FF00000u) - (941u << 20)) << 3));
}

__device__ __forceinline__ float signed_sum(float h, float l2, uint32_t hw)
{
    return __uint_as_float(__float_as_uint(__fmaf_rn(0.5f, l2, h)) | (hw & 0x80000000u));
}

// s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e)
{
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// A vertex in binary32 and whether it lies on the sphere of radius r
// (| |v|^2 - r^2 | <= 1e-12 r^2): yes where the difference in pairs, within
// 2^-44 (6e-14) of r^2, is below 8e-13 r^2; otherwise, and for a radius or
// coordinate outside the pairs' range (a coordinate of 0 among them), as
// binary64 has it.  JOIN: the answer is hidden as well (in the kernel by
// breakpoints it costs 3 us of a year's 106 on 10,000,002 vertices).
template <bool JOIN>
__device__ __forceinline__ bool load_vertex(double X, double Y, double Z, double r, float r2h, float r2l, float &x,
                                            float &y, float &z)
{
    const uint32_t hx = (uint32_t)__double2hiint(X), hy = (uint32_t)__double2hiint(Y), hz = (uint32_t)__double2hiint(Z);
    const uint32_t ax = hx & 0x7FFFFFFFu, ay = hy & 0x7FFFFFFFu, az = hz & 0x7FFFFFFFu;
    bool on = false;
    if (min(ax, min(ay, az)) >= (983u << 20) && max(ax, max(ay, az)) < (1084u << 20) && r2h > 0.0f) {
        float xh, xl, yh, yl, zh, zl;
        split_abs(ax, (uint32_t)__double2loint(X), xh, xl);
        split_abs(ay, (uint32_t)__double2loint(Y), yh, yl);
        split_abs(az, (uint32_t)__double2loint(Z), zh, zl);
        const float px = __fmul_rn(xh, xh), py = __fmul_rn(yh, yh), pz = __fmul_rn(zh, zh);
        const float ex = __fmaf_rn(xh, xl, __fmaf_rn(xh, xh, -px)), ey = __fmaf_rn(yh, yl, __fmaf_rn(yh, yh, -py)),
                    ez = __fmaf_rn(zh, zl, __fmaf_rn(zh, zh, -pz));
        float s1, e1, s2, e2;
        two_sum(px, py, s1, e1);
        two_sum(s1, pz, s2, e2);
        const float low = __fsub_rn(__fadd_rn(__fadd_rn(e1, e2), __fadd_rn(__fadd_rn(ex, ey), ez)), r2l);
        x = signed_sum(xh, xl, hx);
        y = signed_sum(yh, yl, hy);
        z = signed_sum(zh, zl, hz);
        on = fabsf(__fadd_rn(__fsub_rn(s2, r2h), low)) <= 8e-13f * r2h;
    }
    if (!on) {
        x = (float)X;
        y = (float)Y;
        z = (float)Z;
        const double rho2 = X * X + Y * Y + Z * Z, r2 = r * r;
        on = fabs(rho2 - r2) <= 1e-12 * r2;
    }
    // One way out, which the compiler does not see behind.  With two it made
    // the loops over a schedule twice, with half the loads in flight (2,500 days
    // of 9,002 vertices 605 us instead of 317); without the coordinates here it
    // made the loop of vertices off the sphere half as fast again (24 positions
    // of 10 tilts on 400,002 of them 171 us instead of 128).
    if (JOIN) {
        int o = on;
        asm volatile("" : "+f"(x), "+f"(y), "+f"(z), "+r"(o));
        return o != 0;
    }
    asm volatile("" : "+f"(x), "+f"(y), "+f"(z));
    return on;
}

// climate.py:419-442 for a vertex off the sphere of radius r (binary32),
// turned to (rx, ry, z).
__device__ __forceinline__ float general_term(float rx, float ry, float z, float inv_r, float ct, float st)
{
    float tx = rx * ct + z * st;
    float ty = ry;
    float tz = z * ct - rx * st;
    float q = fminf(fmaxf(tz * inv_r, -1.0f), 1.0f);
    float clat = sqrtf(fmaxf(1.0f - q * q, 0.0f));
    float h2 = tx * tx + ty * ty;
    float clon = h2 > 0.0f ? tx * rsqrtf(h2) : 1.0f;    // atan2(0, 0) = 0 -> cos = 1
    return clat * fmaxf(clon, 0.0f);
}

__device__ __forceinline__ float approx_sqrt(float v)
{
    float w;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(w) : "f"(v));
    return w;
}

__device__ __forceinline__ float approx_rcp(float v)
{
    float w;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(w) : "f"(v));
    return w;
}

// Tilts whose per-day constants a block stages in shared memory (16 B each).
constexpr int TILT_STAGE_MAX = 2048;

// Per-day constants of the factored pair sum, (|cos tau|, |sin tau| / |cos
// tau|, HP sin tau, 0); days with |cos tau| < 2^-20 (the direct form) get
// zeros, which add nothing to the factored sum, and are listed after the
// days (day indices as ints, their count in entry n_tilt.y); entry n_tilt.x
// holds the sum of HP sin tau over the factored days (binary64, rounded
// once; a lane per 32nd day, so that a block is not held up by one thread's
// chain of additions), so a vertex adds its days' C terms as one product.
// Shared memory: tilt_smem(a).
template <int HP>
__device__ __forceinline__ void stage_tilts(const InsoArgs &a, float4 *tt)
{
    for (int d = threadIdx.x; d < a.n_tilt; d += blockDim.x) {
        const float2 t = a.tilt[d];
        const float ak = fabsf(t.x);
        tt[d] = ak >= 0x1p-20f ? make_float4(ak, __fdiv_rn(fabsf(t.y), ak), (float)HP * t.y, 0.0f)
                               : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncthreads();
    // warp 0: the sum and, in day order, the list of direct days
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int *direct = reinterpret_cast<int *>(tt + a.n_tilt + 1);
        double sc = 0.0;
        int nd = 0;
        for (int d0 = 0; d0 < a.n_tilt; d0 += 32) {
            const int d = d0 + lane;
            const float4 k = d < a.n_tilt ? tt[d] : make_float4(1.0f, 0.0f, 0.0f, 0.0f);
            const bool dir = !(k.x > 0.0f);
            if (!dir) sc += (double)k.z;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, dir);
            if (dir) direct[nd + __popc(m & ((1u << lane) - 1u))] = d;
            nd += __popc(m);
        }
        for (int o = 16; o > 0; o >>= 1) sc += __shfl_xor_sync(0xFFFFFFFFu, sc, o);
        if (lane == 0) tt[a.n_tilt] = make_float4((float)sc, __int_as_float(nd), 0.0f, 0.0f);
    }
    __syncthreads();
}

// Days per group of the staged sum: a group's days accumulate in paired
// lanes (one FFMA2 per day), the groups are added with compensation.
constexpr int DAY_GROUP = 8;

// Schedules of up to SORT_MAX days are also summed by breakpoints.  With
// c_d = |z| tan_d (tan_d = |tan tau_d|, cos_d = |cos tau_d|) and a_h = |U_h|,
// the factored days' part of the year is
//   sum_d cos_d sum_h max(c_d, a_h)
//     = sum_h [ a_h sum_{d: c_d < a_h} cos_d + |z| sum_{d: c_d >= a_h} cos_d tan_d ],
// exactly (each max picks one side).  With the days sorted by tan_d, both
// inner sums are a prefix sum P0 and a suffix sum Q1 of the sorted days,
// read at the count B_h of days with tan_d < a_h / |z|.  As a function of
// a_h this is the line P0[B] a_h + Q1[B] |z|, its slope P0 growing with B at
// the breakpoints T: convex, so near a breakpoint it is the larger of the
// two lines that meet there, and no comparison with T is needed.  With t =
// a_h / |z| a value is |z| (P0 t + Q1).
// Shared memory after the staged constants: the bucket table of NB + 1
// float4s (bucket_count), the lines L[nf + 1] = (P0,
// Q1) (exact sums rounded once), K[SP] (SP a power of two > the days) the
// sorted tan_d, padded with +inf,
// with their cos_d.  Bucket b holds the t nearest to tmax (1 - (b /
// NB)^2), tmax the largest tan_d: seasonal tilts go as a sine, so the
// breakpoints crowd at tmax as those t do, and hardly a bucket gets two
// (with buckets of equal width in t the crowded ones held up to 14, and the
// walk through them was a third of the instructions).  Bucket 0 takes all t
// beyond tmax.  An entry is the lines of the bucket's two ends (p0, p0', q1,
// q1') where its breakpoints lie within 2e-6 of each other (or 1e-9 tmax); otherwise p0 is
// NaN, the two ends' line numbers follow, and a vertex takes the largest of
// the lines between.  A bucket number one off by rounding changes a value by
// no more than its rounding does, as the lines meet there.
// Measured (GB300, a year of hourly positions, 10,000,002 vertices): 289 ->
// 137 us with the tables and the test in pairs, 111 us in a kernel of its own
// (BREAK_THREADS); a month 224 -> 101 us with 256 buckets instead of 32;
// 9,002 vertices 63.6 -> 16.6 us (the blocks' start).
constexpr int SORT_MAX = 512;

__host__ __device__ __forceinline__ int sort_pad(int n)
{
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

// Buckets of a schedule's table: as many as the padded days, 256 at least
// (a month's breakpoints are spread over t, not crowded at tmax: with 32
// buckets several share one).
__host__ __device__ __forceinline__ int bucket_count(int n_tilt)
{
    const int sp = sort_pad(n_tilt + 1);
    return sp < 256 ? 256 : sp;
}

// Exclusive prefix sums over the block of 64-bit integers (two per thread),
// and their totals.  Sums of cosines are kept as integers of 2^-44: exact,
// and without chains of binary64 additions, which took most of a block's
// start (40 of 64 us from launch to end on a sphere of 9,002 vertices).
__device__ __forceinline__ void block_scan2(long long &u, long long &v, long long &tu, long long &tv)
{
    __shared__ long long s_sum[2][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const long long u0 = u, v0 = v;
    for (int o = 1; o < 32; o <<= 1) {
        const long long a = __shfl_up_sync(0xFFFFFFFFu, u, o), b = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if (lane >= o) { u += a; v += b; }
    }
    if (lane == 31) { s_sum[0][w] = u; s_sum[1][w] = v; }
    __syncthreads();
    u -= u0;
    v -= v0;
    tu = tv = 0;
    for (int k = 0; k < nw; ++k) {
        if (k == w) { u += tu; v += tv; }
        tu += s_sum[0][k];
        tv += s_sum[1][k];
    }
    __syncthreads();
}

__device__ __forceinline__ long long to_fixed(float v) { return __float2ll_rn(v * 0x1p44f); }
__device__ __forceinline__ float from_fixed(long long v) { return __ll2float_rn(v) * 0x1p-44f; }

// Breakpoint tables of a block (stage_breakpoints).
struct Breaks {
    const float2 *L = nullptr;
    const float4 *rot = nullptr;   // the rotations, two to an entry
    uint32_t bucket = 0;       // shared address of the table less what a bucket number's binary32 exponent adds
    float nb = 0.0f;           // buckets
    float inv = 0.0f;          // 1 / tmax
    bool crowded = false;      // some bucket holds distinct breakpoints
};

// Builds the tables from the staged constants (after stage_tilts).  Called
// by the whole block.
__device__ __forceinline__ Breaks stage_breakpoints(const InsoArgs &a, const float4 *tt, uint2 *K, float2 *L,
                                                    float4 *bucket)
{
    const int nd = __float_as_int(tt[a.n_tilt].y);
    const int nf = a.n_tilt - nd;
    const int sp = sort_pad(a.n_tilt + 1), nb = bucket_count(a.n_tilt);
    // bitonic sort of the factored days by tan (direct days, padding: +inf),
    // the cosine alongside
    for (int d = threadIdx.x; d < sp; d += blockDim.x) {
        const bool day = d < a.n_tilt && tt[d].x > 0.0f;
        K[d] = day ? make_uint2(__float_as_uint(tt[d].y), __float_as_uint(tt[d].x)) : make_uint2(0x7F800000u, 0u);
    }
    __syncthreads();
    for (int size = 2; size <= sp; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int q = threadIdx.x; q < sp / 2; q += blockDim.x) {
                const int i = 2 * q - (q & (stride - 1)), j = i + stride;
                const uint2 u = K[i], v = K[j];
                if ((u.x > v.x) == ((i & size) == 0)) { K[i] = v; K[j] = u; }
            }
            __syncthreads();
        }
    auto tan_of = [&](int j) { return __uint_as_float(K[j].x); };
    const float tmax = nf > 0 ? tan_of(nf - 1) : 0.0f;
    // prefix sums of cos (2^-20 at least: exact in units of 2^-44) and of cos *
    // tan, whose unit is 2^-53 of the power of two above the largest of them (so
    // 512 of them stay below 2^63): each thread a run of the days
    const int top = (int)(__float_as_uint(fminf(tmax, 1.0f)) >> 23) - 126, up = min(53 - top, 126);
    const float in = __uint_as_float((uint32_t)(127 + up) << 23), out = __uint_as_float((uint32_t)(127 - up) << 23);
    const int per = (sp + (int)blockDim.x - 1) / (int)blockDim.x;
    const int j0 = min(nf, (int)threadIdx.x * per), j1 = min(nf, j0 + per);
    auto term = [&](int j, long long &u, long long &v) {
        const float c = __uint_as_float(K[j].y), t = tan_of(j), p = __fmul_rn(c, t);
        u += to_fixed(c);
        v += __float2ll_rn(p * in) + __float2ll_rn(__fmaf_rn(c, t, -p) * in);
    };
    long long u = 0, v = 0, tu, tv;
    for (int j = j0; j < j1; ++j) term(j, u, v);
    block_scan2(u, v, tu, tv);
    for (int j = j0; j < j1; ++j) {
        L[j] = make_float2(from_fixed(u), __ll2float_rn(tv - v) * out);
        term(j, u, v);
    }
    if (threadIdx.x == 0) L[nf] = make_float2(from_fixed(tu), 0.0f);
    __syncthreads();
    Breaks bk;
    bk.L = L;
    bk.bucket = (uint32_t)__cvta_generic_to_shared(bucket) - (0x4B000000u << 4);
    bk.nb = (float)nb;
    bk.inv = tmax > 0.0f ? 1.0f / tmax : 0.0f;
    auto below = [&](float t) {
        int c = 0;
        for (int step = sp >> 1; step > 0; step >>= 1) c += tan_of(c + step - 1) < t ? step : 0;
        return c;
    };
    bool crowded = false;
    for (int b = threadIdx.x; b <= nb; b += blockDim.x) {
        const float w0 = ((float)b - 0.5f) / bk.nb, w1 = ((float)b + 0.5f) / bk.nb;
        const int k0 = below(tmax * (1.0f - w1 * w1)), k1 = b > 0 && tmax > 0.0f ? below(tmax * (1.0f - w0 * w0)) : nf;
        const float2 l0 = L[k0], l1 = L[k1];
        const float gap = k1 - k0 <= 1 ? 0.0f : tan_of(k1 - 1) - tan_of(k0);
        const bool simple = gap <= 2e-6f * tan_of(max(k1 - 1, 0)) || gap <= 1e-9f * tmax;   // (or all at t = 0)
        bucket[b] = simple ? make_float4(l0.x, l1.x, l0.y, l1.y)
                           : make_float4(__int_as_float(0x7FFFFFFF), __int_as_float(k0), __int_as_float(k1), 0.0f);
        crowded = crowded || !simple;
    }
    // (the rotations from shared memory: read through the global pointer they
    // cost each vertex twelve loads, as its result might overwrite them)
    __shared__ float4 s_rot[8];
    if (threadIdx.x < a.n_rot && threadIdx.x < 16) reinterpret_cast<float2 *>(s_rot)[threadIdx.x] = a.rot[threadIdx.x];
    bk.rot = s_rot;
    bk.crowded = __syncthreads_or(crowded) != 0;
    return bk;
}

// The year's sum of the factored days for one rotation pair of a = |U|, c =
// |z|: the larger of the two lines of the bucket of a / c (ti = 1 / (c
// tmax), rounded).
template <bool CROWDED>
__device__ __forceinline__ float pair_value(const Breaks &bk, float a, float c, float ti)
{
    // the bucket number, rounded to nearest, in the low bits of a binary32
    const float w = approx_sqrt(__saturatef(fmaf(-a, ti, 1.0f)));
    const uint32_t at = (__float_as_uint(fmaf(w, bk.nb, 8388608.0f)) << 4) + bk.bucket;
    float4 e;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(e.x), "=f"(e.y), "=f"(e.z), "=f"(e.w) : "r"(at));
    const float2 v2 = __ffma2_rn(make_float2(a, a), make_float2(e.x, e.y),
                                 __fmul2_rn(make_float2(c, c), make_float2(e.z, e.w)));
    float v = fmaxf(v2.x, v2.y);
    if (CROWDED && e.x != e.x) {
        const int k1 = __float_as_int(e.z);
        v = 0.0f;
        for (int k = __float_as_int(e.y); k <= k1; ++k) {
            const float2 l = bk.L[k];
            v = fmaxf(v, fmaf(a, l.x, c * l.y));
        }
    }
    return v;
}

template <int HP, bool CROWDED>
__device__ __forceinline__ float pair_sum(const Breaks &bk, float x, float y, float c, float ti)
{
    // (four short sums: with two of six each the roundings were as large as the
    // values' own)
    float2 s[2];
#pragma unroll
    for (int h = 0; h < HP; h += 2) {
        const float4 q = bk.rot[h / 2];
        const float2 u = make_float2(pair_value<CROWDED>(bk, fabsf(fmaf(x, q.x, -(y * q.y))), c, ti),
                                     pair_value<CROWDED>(bk, fabsf(fmaf(x, q.z, -(y * q.w))), c, ti));
        s[h / 2 % 2] = h < 4 ? u : __fadd2_rn(s[h / 2 % 2], u);
    }
    const float2 t = __fadd2_rn(s[0], s[1]);
    return t.x + t.y;
}

// Arcs (HP = ARCS).  x cos(theta) - y sin(theta) = rho cos(theta + phi), phi
// = atan2(y, x), so a tilt's terms max(k rho cos(theta + phi) + C, 0), k =
// cos tau, are positive on the arc of half width acos(-C / (|k| rho)) about
// -phi (about -phi + pi for k < 0), and their sum over it is k (x sum cos -
// y sum sin) + C count: a difference of prefix sums of the rotations sorted
// by angle.  A rotation put on the wrong side of an end of the arc by
// rounding has a term of that rounding's size, so the searches need not be
// exact.  Rotations come in any order; up to ARC_MAX of them.
// Shared memory: the prefix sums P[n + 1] (exact sums rounded once), the
// angles less the smallest one, ascending, an index F of NB = a power of two
// >= n buckets (F[b] = angles below b 2 pi / NB), the rotations' order.
// Measured (GB300, one tilt, 360 rotations): 110.8 -> 35 us for 2,500,002
// vertices, 420 -> 100 us for 10,000,002 (2.8 TB/s of the 28 B per vertex;
// instruction issue and the two gathers bound it; see INSO_THREADS).
// From ARC_MIN rotations on, for ARC_VERTICES vertices or ARC_TERMS positions:
// a sum by arcs has a few roundings whatever its rotations (5e-8 of the norm
// for one-degree days, 5e-7 by maxima), and its time hardly depends on them,
// but a block's sorting and prefix sums take ~5 us.  By arcs / by maxima, us
// (GB300, 9,002, 256,002, 625,002 and 2,500,002 vertices): 128 rotations 7.0 /
// 2.8, 11.5 / 6.4, 14.9 / 11.1, 31.1 / 36.2; 360 8.0 / 3.7, 12.1 / 10.3, 15.6 /
// 21.3, 31.8 / 75.9; 700 12.4 / 21.8, 16.4 / 48.7, 19.5 / 104, 35.8 / 372; of 48
// rotations, 30 tilts, 20.3 / 9.5, 43.3 / 37.8, 88.2 / 87.9, 249 / 331.  So large
// spheres and long days gain time by arcs, a one-degree day on a small one
// pays 4 us for the smaller error, and fewer rotations than ARC_MIN have
// little error to lose.
constexpr int ARCS = -1;
constexpr int ARC_MIN = 128;
constexpr int64_t ARC_VERTICES = 1 << 18;
constexpr int ARC_TERMS = 360;
constexpr int ARC_MAX = 1024;
constexpr float TWO_PI = 6.28318531f;

// Rotations without pairs keep their prefix sums as the integers they are formed
// as, and a vertex's products with their rest: a difference of rounded sums is
// off by what the largest sum is, which a vertex lit in a few rotations would
// show (129 to 1,023 rotations, up to 40 of them lit: 4-30 times the error of
// those terms added one by one; as integers no more than theirs).  The maxima of
// pairs cancel in the same way as rounded sums do, so pairs keep those.
struct Arcs {
    const float2 *P = nullptr;     // pairs
    const longlong2 *Q = nullptr;  // no pairs: units of 2^-44
    const float *ang = nullptr;
    const int *F = nullptr;
    int n = 0, nb = 0;
    float base = 0.0f, scale = 0.0f;
};

__host__ __device__ __forceinline__ size_t arc_smem(int n, int pairs)
{
    return (pairs ? sizeof(float2) : sizeof(longlong2)) * ((size_t)n + 1) + sizeof(float) * (2 * (size_t)n + 1) + sizeof(int) * (size_t)(sort_pad(n) + n + 1);
}

__device__ __forceinline__ Arcs stage_arcs(const InsoArgs &a, void *smem)
{
    Arcs A;
    const int n = a.pairs ? 2 * a.n_rot : a.n_rot, nb = sort_pad(n);
    float2 *P = reinterpret_cast<float2 *>(smem);
    longlong2 *Q = reinterpret_cast<longlong2 *>(smem);
    float *ang = a.pairs ? reinterpret_cast<float *>(P + n + 1) : reinterpret_cast<float *>(Q + n + 1), *raw = ang + n;
    int *order = reinterpret_cast<int *>(raw + n + 1), *F = order + n;
    auto rot = [&](int i) {
        const float2 q = a.rot[i < a.n_rot ? i : i - a.n_rot];
        return i < a.n_rot ? q : make_float2(-q.x, -q.y);
    };
    // (an angle that is no number has no place in the order, and a tilt that is
    // none no arc: none of the tables, and the vertices go through the rotations
    // one by one)
    bool number = true;
    for (int d = threadIdx.x; d < a.n_tilt; d += blockDim.x) number = number && a.tilt[d].x == a.tilt[d].x;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float2 q = rot(i);
        raw[i] = atan2f(q.y, q.x);
        number = number && raw[i] == raw[i];
    }
    if (!__syncthreads_and(number)) return A;
    bool ascending = true;
    for (int i = threadIdx.x; i + 1 < n; i += blockDim.x) ascending = ascending && raw[i] <= raw[i + 1];
    if (__syncthreads_and(ascending)) {
        for (int i = threadIdx.x; i < n; i += blockDim.x) order[i] = i;
    } else {
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const float v = raw[i];
            int rank = 0;
            for (int j = 0; j < n; ++j) rank += raw[j] < v || (raw[j] == v && j < i) ? 1 : 0;
            order[rank] = i;
        }
    }
    __syncthreads();
    const float base = raw[order[0]];
    for (int i = threadIdx.x; i < n; i += blockDim.x) ang[i] = raw[order[i]] - base;
    const int per = (n + (int)blockDim.x - 1) / (int)blockDim.x;
    const int j0 = min(n, (int)threadIdx.x * per), j1 = min(n, j0 + per);
    long long u = 0, v = 0, tu, tv;
    for (int j = j0; j < j1; ++j) {
        const float2 q = rot(order[j]);
        u += to_fixed(q.x);
        v += to_fixed(q.y);
    }
    block_scan2(u, v, tu, tv);
    for (int j = j0; j < j1; ++j) {
        const float2 q = rot(order[j]);
        if (a.pairs) P[j] = make_float2(from_fixed(u), from_fixed(v));
        else Q[j] = make_longlong2(u, v);
        u += to_fixed(q.x);
        v += to_fixed(q.y);
    }
    if (threadIdx.x == 0) {
        if (a.pairs) P[n] = make_float2(from_fixed(tu), from_fixed(tv));
        else Q[n] = make_longlong2(tu, tv);
    }
    __syncthreads();
    for (int b = threadIdx.x; b <= nb; b += blockDim.x) {
        const float edge = (float)b * (TWO_PI / (float)nb);
        int lo = 0, hi = n;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (ang[mid] < edge) lo = mid + 1;
            else hi = mid;
        }
        F[b] = lo;
    }
    __syncthreads();
    A.P = P;
    A.Q = Q;
    A.ang = ang;
    A.F = F;
    A.n = n;
    A.nb = nb;
    A.base = base;
    A.scale = (float)nb / TWO_PI;
    return A;
}

// How many of the sorted angles lie below v (0 <= v <= 2 pi).
__device__ __forceinline__ int arc_find(const Arcs &A, float v)
{
    int c = A.F[min((int)(v * A.scale), A.nb)];
    while (c < A.n && A.ang[c] < v) ++c;
    return c;
}

__device__ __forceinline__ float arc_sum(const InsoArgs &a, const Arcs &A, float x, float y, float z)
{
    const float phi = atan2f(-y, x), rho = sqrtf(fmaf(x, x, y * y));
    float tot = 0.0f, comp = 0.0f;          // Kahan over tilts
    for (int d = 0; d < a.n_tilt; ++d) {
        const float2 t = a.tilt[d];
        const float C = z * t.y, den = fabsf(t.x) * rho;
        int lo = 0, hi = 0, turns = 0;         // rotations [lo, hi), and all of them once more
        if (C >= den) {
            hi = A.n;
        } else if (C > -den) {
            const float alpha = acosf(__fdividef(-C, den));
            float a0 = (t.x < 0.0f ? phi + 0.5f * TWO_PI : phi) - alpha - A.base;
            a0 -= TWO_PI * floorf(a0 * (1.0f / TWO_PI));
            const float a1 = a0 + 2.0f * alpha;
            turns = a1 >= TWO_PI ? 1 : 0;
            lo = arc_find(A, a0);
            hi = arc_find(A, turns ? a1 - TWO_PI : a1);
        }
        const float cnt = (float)(hi - lo + turns * A.n);
        float s;
        if (a.pairs) {
            const float2 l = A.P[lo], h = A.P[hi];
            float2 S = make_float2(h.x - l.x, h.y - l.y);
            if (turns) {
                const float2 w = A.P[A.n];
                S.x += w.x;
                S.y += w.y;
            }
            s = fmaf(t.x, fmaf(x, S.x, -(y * S.y)), C * cnt);
        } else {
            const longlong2 l = A.Q[lo], h = A.Q[hi];
            long long u = h.x - l.x, v = h.y - l.y;
            if (turns) {
                const longlong2 w = A.Q[A.n];
                u += w.x;
                v += w.y;
            }
            // t.x (x Sx - y Sy) + z t.y cnt in pairs
            const float Sx = from_fixed(u), Sy = -from_fixed(v);
            const float px = __fmul_rn(x, Sx), py = __fmul_rn(y, Sy), p = __fmul_rn(C, cnt);
            float q, qe, r, re;
            two_sum(px, py, q, qe);
            qe += __fmaf_rn(x, Sx, -px) + __fmaf_rn(y, Sy, -py);
            const float g = __fmul_rn(t.x, q);
            two_sum(g, p, r, re);
            re += __fmaf_rn(t.x, q, -g) + __fmaf_rn(C, cnt, -p);
            s = r + fmaf(t.x, qe, fmaf(__fmaf_rn(z, t.y, -C), cnt, re));
        }
        s = fmaxf(s, 0.0f);
        const float yk = s - comp;
        const float tk = tot + yk;
        comp = (tk - tot) - yk;
        tot = tk;
    }
    return tot;
}

template <int HP, bool BREAKS>
__device__ __forceinline__ float inso_vertex(const InsoArgs &a, double X, double Y, double Z, double r, float r2h,
                                             float r2l, float zmin, float inv_r, const float4 *tt = nullptr,
                                             const Breaks &bk = Breaks(), const Arcs &arc = Arcs())
{
    float x, y, z;
    const bool on_sphere = load_vertex<!BREAKS>(X, Y, Z, r, r2h, r2l, x, y, z);
    if (HP == ARCS && on_sphere) return arc_sum(a, arc, x, y, z) * inv_r;
    float tot = 0.0f, comp = 0.0f;          // Kahan over tilts
    const int nr = HP > 0 ? HP : a.n_rot;
    if constexpr (HP > 0) {
    if (on_sphere) {
        // u = A cos(theta) + B sin(theta) = k U(theta) with k = cos(tau) and
        // U = x cos(theta) - y sin(theta) the same for every day, so per day
        //   sum_h max(|C|, |u_h|) = |k| sum_h max(|C| / |k|, |U_h|)
        // (exact in real arithmetic): |U_h| is formed once per vertex and a
        // day costs a max and an add per rotation pair.  Days with |k| near 0
        // take the direct form.
        float au[HP];
        if (!BREAKS) {
#pragma unroll
            for (int h = 0; h < HP; ++h) {
                const float2 q = a.rot[h];
                au[h] = fabsf(fmaf(x, q.x, -(y * q.y)));
            }
        }
        if (BREAKS || tt) {
            // constants staged by the block: per day a shared load, one
            // multiply for the threshold, the max / add of each pair and one
            // paired multiply-add into the group's lanes; the days' C terms
            // come in at the end as z times their staged sum, the (rare)
            // direct-form days after the others
            const float az = fabsf(z);
            auto add = [&](float s) {
                const float yk = s - comp;
                const float tk = tot + yk;
                comp = (tk - tot) - yk;
                tot = tk;
            };
            if constexpr (BREAKS) {
                // each pair's line pair from its bucket of t = a_h / |z|
                // (|z| kept off 0: 1e-20 r in its place changes no value)
                const float ti = approx_rcp(fmaxf(az, zmin)) * bk.inv;
                tot = bk.crowded ? pair_sum<HP, true>(bk, x, y, az, ti) : pair_sum<HP, false>(bk, x, y, az, ti);
            } else {
            auto day = [&](int d, float2 g) {
                const float4 k = tt[d];
                const float c = az * k.y;
                float2 acc = make_float2(fmaxf(c, au[0]), fmaxf(c, au[1]));
#pragma unroll
                for (int h = 2; h < HP; h += 2)
                    acc = __fadd2_rn(acc, make_float2(fmaxf(c, au[h]), fmaxf(c, au[h + 1])));
                return __ffma2_rn(make_float2(k.x, k.x), acc, g);
            };
            const int full = a.n_tilt - a.n_tilt % DAY_GROUP;
            for (int d0 = 0; d0 < full; d0 += DAY_GROUP) {
                float2 g = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int j = 0; j < DAY_GROUP; ++j) g = day(d0 + j, g);
                add(g.x + g.y);
            }
            if (full < a.n_tilt) {
                float2 g = make_float2(0.0f, 0.0f);
                for (int d = full; d < a.n_tilt; ++d) g = day(d, g);
                add(g.x + g.y);
            }
            }   // days one by one
            const float4 e = tt[a.n_tilt];
            const int nd = __float_as_int(e.y);
            const int *direct = reinterpret_cast<const int *>(tt + a.n_tilt + 1);
            for (int i = 0; i < nd; ++i) {
                const float2 t = a.tilt[direct[i]];
                const float A = x * t.x, B = -(y * t.x), C = z * t.y, aC = fabsf(C);
                float s = 0.0f;
#pragma unroll
                for (int h = 0; h < HP; ++h) {
                    const float2 q = a.rot[h];
                    s += fmaxf(aC, fabsf(fmaf(A, q.x, B * q.y)));
                }
                add(fmaf((float)HP, C, s));
            }
            add(z * e.x);
            return tot * inv_r;
        }
        for (int d = 0; d < a.n_tilt; ++d) {
            const float2 t = a.tilt[d];
            const float C = z * t.y, aC = fabsf(C), ak = fabsf(t.x);
            float s;
            if (ak >= 0x1p-20f) {
                const float c = __fdividef(aC, ak);
                float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int h = 0; h < HP; h += 2)
                    acc = __fadd2_rn(acc, make_float2(fmaxf(c, au[h]), fmaxf(c, au[h + 1])));
                s = fmaf(ak, acc.x + acc.y, (float)HP * C);
            } else {
                const float A = x * t.x, B = -(y * t.x);
                s = 0.0f;
#pragma unroll
                for (int h = 0; h < HP; ++h) {
                    const float2 q = a.rot[h];
                    s += fmaxf(aC, fabsf(fmaf(A, q.x, B * q.y)));
                }
                s = fmaf((float)HP, C, s);
            }
            float yk = s - comp;
            float tk = tot + yk;
            comp = (tk - tot) - yk;
            tot = tk;
        }
        return tot * inv_r;
    }
    } else if (on_sphere) {
        for (int d = 0; d < a.n_tilt; ++d) {
            const float2 t = a.tilt[d];
            const float A = x * t.x, B = -(y * t.x), C = z * t.y;
            float s = 0.0f;
            if (a.pairs) {
                const float aC = fabsf(C);
                for (int h = 0; h < nr; ++h) {
                    float2 q = a.rot[h];
                    float u = fmaf(A, q.x, B * q.y);
                    s += fmaxf(aC, fabsf(u));
                }
                s = fmaf((float)nr, C, s);
            } else {
                for (int h = 0; h < nr; ++h) {
                    float2 q = a.rot[h];
                    s += fmaxf(fmaf(A, q.x, fmaf(B, q.y, C)), 0.0f);
                }
            }
            float yk = s - comp;
            float tk = tot + yk;
            comp = (tk - tot) - yk;
            tot = tk;
        }
        return tot * inv_r;
    }
    for (int d = 0; d < a.n_tilt; ++d) {
        const float2 t = a.tilt[d];
        float s = 0.0f;
#pragma unroll 6
        for (int h = 0; h < nr; ++h) {
            // (a pair's other rotation turns to the opposite point)
            const float2 q = a.rot[h];
            const float rx = x * q.x - y * q.y, ry = x * q.y + y * q.x;
            s += general_term(rx, ry, z, inv_r, t.x, t.y);
            if (HP > 0 || a.pairs) s += general_term(-rx, -ry, z, inv_r, t.x, t.y);
        }
        float yk = s - comp;
        float tk = tot + yk;
        comp = (tk - tot) - yk;
        tot = tk;
    }
    return tot;
}

// The block's breakpoint tables after the staged constants (see SORT_MAX).
template <int HP>
__device__ __forceinline__ Breaks stage_all(const InsoArgs &a, float4 *s_tilt)
{
    stage_tilts<HP>(a, s_tilt);
    // 16-byte units: the bucket table first, then the lines, then the rest
    float4 *bucket = s_tilt + a.n_tilt + 1 + (a.n_tilt + 3) / 4;
    float2 *L = reinterpret_cast<float2 *>(bucket + bucket_count(a.n_tilt) + 1);
    uint2 *K = reinterpret_cast<uint2 *>(L + a.n_tilt + 1);
    return stage_breakpoints(a, s_tilt, K, L, bucket);
}

// Threads of a block: two of 512 per SM for the breakpoints' tables (half as
// many tables to build as with 256), in a kernel without the other forms,
// whose registers it spilled: a year on 10,000,002 vertices 142 -> 111 us (2.5
// TB/s of the 28 B per vertex), 40,000,002 521 -> 355 us.  One block of 768
// is as fast on large spheres, 106 instead of 97 us where a bucket is crowded.
constexpr int BREAK_THREADS = 512, BREAK_BLOCKS = 2;
// By arcs: one block of 1,024 per SM where there are vertices for all of them,
// blocks of 512 otherwise (a day of 360 rotations, with blocks of 256, 512
// and 1,024: 10,000,002 vertices 119, 107, 103 us; 2,500,002 43.6, 39.6, 37.5;
// 9,002 12.9, 12.9, 15.0).
template <bool BREAKS, int HP>
constexpr int INSO_THREADS = BREAKS ? BREAK_THREADS : (HP == ARCS ? 1024 : 256);

template <int HP, bool BREAKS, bool AHEAD>
__device__ __forceinline__ void insolation_body(const InsoArgs &a)
{
    extern __shared__ float4 s_tilt[];
    const bool staged = BREAKS || (HP > 0 && a.n_tilt <= TILT_STAGE_MAX);
    Breaks bk;
    Arcs arc;
    if constexpr (BREAKS) bk = stage_all<HP>(a, s_tilt);
    else if (HP > 0 && staged) stage_tilts<HP>(a, s_tilt);
    if constexpr (HP == ARCS) arc = stage_arcs(a, s_tilt);
    // AHEAD: the next vertex is read while this one is summed (32 warps' 768
    // bytes each are too few in flight per SM for the memory's latency: one
    // position on 10,000,002 vertices 74 -> 62 us); sums over more positions
    // than a launch's arguments hold are better off with the registers (2,500
    // days of 2,500,002 vertices 9.36 -> 8.98 ms)
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    // the scale here instead of in a pass of its own over the sums (11 us for
    // 10 M vertices)
    auto put = [&](int64_t at, float sum) {
        const float v = __fmul_rn(sum, a.scale);
        a.out[at] = a.accumulate ? a.out[at] + v : v;
    };
    if (HP == ARCS && arc.n == 0) {
        for (; i < a.n; i += step)
            put(i, inso_vertex<0, false>(a, a.xyz[3 * i], a.xyz[3 * i + 1], a.xyz[3 * i + 2], a.r, a.r2h, a.r2l, a.zmin, a.inv_r));
        return;
    }
    double X = 0.0, Y = 0.0, Z = 0.0;
    if (AHEAD && i < a.n) { X = a.xyz[3 * i]; Y = a.xyz[3 * i + 1]; Z = a.xyz[3 * i + 2]; }
    for (; i < a.n; i += step) {
        if (!AHEAD) { X = a.xyz[3 * i]; Y = a.xyz[3 * i + 1]; Z = a.xyz[3 * i + 2]; }
        const double cx = X, cy = Y, cz = Z;
        const int64_t j = i + step;
        if (AHEAD && j < a.n) { X = a.xyz[3 * j]; Y = a.xyz[3 * j + 1]; Z = a.xyz[3 * j + 2]; }
        put(i, inso_vertex<HP, BREAKS>(a, cx, cy, cz, a.r, a.r2h, a.r2l, a.zmin, a.inv_r, staged ? s_tilt : nullptr, bk, arc));
    }
}

template <int HP, bool BREAKS = false>
__global__ void __launch_bounds__(INSO_THREADS<BREAKS, HP>, BREAKS ? BREAK_BLOCKS : (HP == ARCS ? 1 : (HP == 12 ? 3 : 4))) insolation_kernel(InsoArgs a)
{
    insolation_body<HP, BREAKS, BREAKS || HP == ARCS>(a);
}

// A short schedule's table as a kernel argument (a table of its own on the
// device takes another launch, ~3 us).
constexpr int ARG_POSITIONS = 496;
struct InsoTable {
    float2 t[ARG_POSITIONS];
};

template <int HP, bool BREAKS = false>
__global__ void __launch_bounds__(INSO_THREADS<BREAKS, HP>, BREAKS ? BREAK_BLOCKS : (HP == ARCS ? 1 : (HP == 12 ? 3 : 4)))
    insolation_args_kernel(InsoArgs a, const __grid_constant__ InsoTable table)
{
    a.rot = table.t;
    a.tilt = table.t + a.n_rot;
    insolation_body<HP, BREAKS, true>(a);
}

// Many planets: planet p's vertices fill packed rows [vbeg, vbeg + n)
// (vbeg a multiple of 256); one block covers 256 rows of one planet.
template <int HP, bool BREAKS = false>
__global__ void __launch_bounds__(256, HP == 12 && !BREAKS ? 3 : 4) insolation_batch_kernel(InsoArgs a, const nx_inso_planet *__restrict__ P, int np,
                                                               int64_t total_rows)
{
    extern __shared__ float4 s_tilt[];
    const bool staged = BREAKS || (HP > 0 && a.n_tilt <= TILT_STAGE_MAX);
    Breaks bk;
    Arcs arc;
    if constexpr (BREAKS) bk = stage_all<HP>(a, s_tilt);
    else if (HP > 0 && staged) stage_tilts<HP>(a, s_tilt);
    if constexpr (HP == ARCS) arc = stage_arcs(a, s_tilt);
    auto rows = [&](auto vertex) {
        // rows only go up: walk to the next planet, and form a planet's radius
        // constants (binary64) once
        int p = -1;
        int64_t beg = 0, next = 0;
        double r = 1.0;
        float r2h = 0.0f, r2l = 0.0f, zmin = 0.0f, inv_r = 1.0f;
        for (int64_t blk = blockIdx.x; blk * 256 < total_rows; blk += gridDim.x) {
            if (p < 0 || blk * 256 >= next) {
                do {
                    ++p;
                    next = p + 1 < np ? P[p + 1].vbeg : INT64_MAX;
                } while (blk * 256 >= next);
                beg = P[p].vbeg;
                r = P[p].radius;
                radius_pair(r, r2h, r2l);
                inv_r = (float)(1.0 / r);
                zmin = (float)(1e-20 * r);
            }
            const int64_t i = blk * 256 + threadIdx.x - beg;
            if (i < 0 || i >= P[p].n) continue;
            const double *v = P[p].xyz + 3 * i;
            a.out[beg + i] = vertex(v[0], v[1], v[2], r, r2h, r2l, zmin, inv_r);
        }
    };
    if (HP == ARCS && arc.n == 0)
        rows([&](double x, double y, double z, double r, float r2h, float r2l, float zmin, float inv_r) {
            return inso_vertex<0, false>(a, x, y, z, r, r2h, r2l, zmin, inv_r);
        });
    else
        rows([&](double x, double y, double z, double r, float r2h, float r2l, float zmin, float inv_r) {
            return inso_vertex<HP, BREAKS>(a, x, y, z, r, r2h, r2l, zmin, inv_r, staged ? s_tilt : nullptr, bk, arc);
        });
}

// ---------------------------------------------------------------------------
// Latitude-table path (climate.py:503-597): per tilt, a table of 181
// latitudes (entry i = latitude i for i <= 90, i - 181 above), each the
// binary32 running sum over 360 rotations of 1 degree from -180 of the
// reference's binary64 term at (lat, lon 0) (calc_insolation_slice with
// sample_insolation's formula); then per vertex a linear
// interpolation between floor(lat) and ceil(lat), summed in binary32 over
// the tables (calc_yearly_insolation adds 360 daily tables).

constexpr double DEG = 3.141592653589793 / 180;

// One block per table, one thread per latitude entry.  The table's points
// lie on the sphere of the given radius at longitude 0 (y = 0), so the
// reference's term equals max(tx, 0) / radius with tx = x cos(theta)
// cos(tau) + z sin(tau) (the identity at the top of this file); it is
// evaluated in binary64 and summed in binary32 over the 360 rotations
// (-180, -179, ..., 179 degrees: the running sum of 1.0 steps is exact) as
// the reference sums its binary64 terms.  The rotations' cosines are
// computed once per block into shared memory.
__global__ void __launch_bounds__(192) slice_kernel(const double *__restrict__ tilts, int n_tilts, double radius,
                                                    float *__restrict__ tables)
{
    __shared__ double rc[360];
    const int d = blockIdx.x, i = threadIdx.x;
    for (int j = i; j < 360; j += blockDim.x) rc[j] = cos((-180.0 + (double)j) * 3.141592653589793 / 180);
    __syncthreads();
    if (d >= n_tilts || i >= 181) return;
    const double lat = (double)(i <= 90 ? i : i - 181);
    // util.latlon2xyz (util.py:79-88) at lon 0
    const double x = radius * cos(lat * DEG) * cos(0.0 * DEG);
    const double z = radius * sin(lat * DEG);
    const double tilt = tilts[d];
    const double ct = cos(tilt * 3.141592653589793 / 180), st = sin(tilt * 3.141592653589793 / 180);
    const double xc = x * ct, zs = z * st, inv_r = 1.0 / radius;
    float acc = 0.0f;
    for (int j = 0; j < 360; ++j) {
        const double tx = __fma_rn(xc, rc[j], zs);
        acc = __double2float_rn(__dadd_rn((double)acc, __dmul_rn(fmax(tx, 0.0), inv_r)));
    }
    tables[181 * d + i] = acc;
}

// One interpolation of climate.py:575, round32(tl + frac * (tu - tl)) with
// tu - tl rounded to binary32 and the product and sum rounded to binary64,
// computed in binary32 pairs.  frac = fh + fl (+ a remainder below 2^-48
// frac); with M = max(|tl|, |tu|) the pair value v' = sh + t is within
// 2^-45 M of the exact tl + frac (tu - tl), and the reference's binary64
// value within 2^-52 M of it.  When v' lies more than 2^-43 M from every
// binary32 rounding boundary both round to the same binary32 value r;
// otherwise (about one evaluation in 2^19) the binary64 formula is used.
__device__ __forceinline__ float interp_one(float tl, float tu, float fh, float fl, double frac)
{
    const float dd = __fsub_rn(tu, tl);
    const float ph = __fmul_rn(fh, dd);
    const float pl = __fmaf_rn(fl, dd, __fmaf_rn(fh, dd, -ph));   // fh*dd = ph + (fh*dd - ph) exactly
    // two-sum tl + ph = sh + se
    const float sh = __fadd_rn(tl, ph);
    const float bb = __fsub_rn(sh, tl);
    const float se = __fadd_rn(__fsub_rn(tl, __fsub_rn(sh, bb)), __fsub_rn(ph, bb));
    const float t = __fadd_rn(se, pl);
    // two-sum sh + t = r + e: v' - r = e exactly
    const float r = __fadd_rn(sh, t);
    const float b2 = __fsub_rn(r, sh);
    const float e = __fadd_rn(__fsub_rn(sh, __fsub_rn(r, b2)), __fsub_rn(t, b2));
    const float M = fmaxf(fabsf(tl), fabsf(tu));
    const uint32_t rb = __float_as_uint(r) & 0x7FFFFFFFu;
    const uint32_t ex = rb >> 23;
    if (ex > 24 && ex < 255) {
        // half an ulp of |r| away from zero, and toward zero (a quarter ulp
        // below a power of two)
        const float hu = __uint_as_float((ex - 24) << 23);
        const float hd = (rb & 0x7FFFFFu) ? hu : 0.5f * hu;
        const float ea = __float_as_uint(r) >> 31 ? -e : e;     // e measured away from zero
        const float dist = ea >= 0.0f ? __fsub_rn(hu, ea) : __fadd_rn(hd, ea);
        if (dist > 0x1p-43f * M) return r;
    } else if (M == 0.0f) {
        return r;                                                // tl = tu = 0
    }
    return __double2float_rn(__dadd_rn((double)tl, __dmul_rn(frac, (double)dd)));
}

// climate.py:551-577 per vertex and table, summed in binary32 over tables.
// The reference divides the table difference by upper - lower, which is
// exactly 1.0 whenever lower != upper, so no division is issued.
__global__ void __launch_bounds__(256) interp_kernel(const double *__restrict__ xyz, int64_t n, double radius,
                                                     const float *__restrict__ tables, int n_tables,
                                                     float *__restrict__ out, int accumulate)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const double q = fmin(fmax(xyz[3 * v + 2] / radius, -1.0), 1.0);
        const double lat = asin(q) * (180.0 / 3.141592653589793);
        const double fl = floor(lat), cl = ceil(lat);
        const int lower = (int)fl, upper = (int)cl;
        const int il = (lower + 181) % 181, iu = (upper + 181) % 181;
        const double frac = lat - fl;
        const float fh = __double2float_rn(frac);
        const float fr = __double2float_rn(__dsub_rn(frac, (double)fh));
        float acc = accumulate ? out[v] : 0.0f;
        for (int d = 0; d < n_tables; ++d) {
            const float tl = __ldg(tables + 181 * d + il), tu = __ldg(tables + 181 * d + iu);
            const float val = lower != upper ? interp_one(tl, tu, fh, fr, frac) : tl;
            acc = (n_tables == 1 && !accumulate) ? val : __fadd_rn(acc, val);
        }
        out[v] = acc;
    }
}

// climate.assign_surface_temp (climate.py:345-411) per vertex: latitude as
// util.xyz2latlon (util.py:59-75), then max(cos(|lat - tilt| * pi / 180), 0)
// in binary64 with the reference's operation order, stored as binary32.
// The reference's altitude term h2 = rescale(altitudes, 0, 0) is 0 (NaN for
// a constant field) at every vertex, so its h2 > 0 branch is never taken.
__global__ void __launch_bounds__(256) surface_temp_kernel(const double *__restrict__ xyz, int64_t n, double radius,
                                                           double tilt, float *__restrict__ out)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const double q = fmin(fmax(__ddiv_rn(xyz[3 * v + 2], radius), -1.0), 1.0);
        const double lat = __dmul_rn(asin(q), 180.0 / 3.141592653589793);
        const double a = __ddiv_rn(__dmul_rn(fabs(__dsub_rn(lat, tilt)), 3.141592653589793), 180.0);
        const double c = cos(a);
        out[v] = __double2float_rn(0.0 > c ? 0.0 : c);     // Python max(c, 0): c unless 0 > c
    }
}

// Dynamic shared memory of the 12-pair kernels: the staged tilt constants.
size_t tilt_smem(const InsoArgs &a)
{
    if (!a.pairs || a.n_tilt > TILT_STAGE_MAX) return 0;
    size_t b = sizeof(float4) * ((size_t)a.n_tilt + 1) + sizeof(int) * (size_t)a.n_tilt;
    if (a.n_tilt <= SORT_MAX) {    // the list rounded to 16 bytes, bucket table, lines, sorted days
        const size_t sp = (size_t)sort_pad(a.n_tilt + 1), nb = (size_t)bucket_count(a.n_tilt), nt = (size_t)a.n_tilt;
        b = sizeof(float4) * (nt + 1 + (nt + 3) / 4 + nb + 1) + sizeof(float2) * (nt + 1 + sp);
    }
    return b;
}

int grid_for(int64_t n, int per_sm = 8)
{
    int64_t g = (n + 255) / 256;
    int64_t cap = (int64_t)nx::sm_count() * per_sm;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

// Whether a schedule is summed by breakpoints (short ones as kernel arguments
// always are: 12 pairs leave room for 484 days).
static_assert(ARG_POSITIONS - 12 <= SORT_MAX, "no args kernel for longer schedules of 12 pairs");
bool breaks(const InsoArgs &a) { return a.pairs && a.n_rot == 12 && a.n_tilt <= SORT_MAX; }

// A block that sums by breakpoints sorts the schedule first, so the grid is the
// resident blocks and each takes many vertices.
int grid_breaks(int64_t n)
{
    const int64_t g = (n + BREAK_THREADS - 1) / BREAK_THREADS, cap = (int64_t)nx::sm_count() * BREAK_BLOCKS;
    return (int)(g < cap ? g : cap);
}

int arc_threads(int64_t n) { return n >= (int64_t)nx::sm_count() * 1024 ? 1024 : 512; }

int grid_arcs(int64_t n)
{
    const int t = arc_threads(n);
    const int64_t g = (n + t - 1) / t, cap = (int64_t)nx::sm_count() * (1024 / t);
    return (int)(g < cap ? g : cap);
}

// Whether a schedule is summed by arcs (radius: on spheres whose squares are
// binary32 numbers, 2^-20 to 2^60).
bool use_arcs(const InsoArgs &a, int64_t vertices, bool radius)
{
    const int n = a.pairs ? 2 * a.n_rot : a.n_rot;
    return radius && n >= ARC_MIN && n <= ARC_MAX && (vertices >= ARC_VERTICES || n * a.n_tilt >= ARC_TERMS);
}

}  // namespace

// Degrees -> (cos, sin) as the reference computes them (climate.py:423-436:
// cos(angle * pi / 180) in binary64), rounded to binary32.
static void trig_table(const double *deg, int n, float *out)
{
    const double PI = 3.141592653589793;
    for (int i = 0; i < n; ++i) {
        double a = deg[i] * PI / 180;
        out[2 * i] = (float)cos(a);
        out[2 * i + 1] = (float)sin(a);
    }
}

NX_EXPORT int nx_insolation_plan(const double *rot_deg, int n_rot, const double *tilt_deg, int n_tilt,
                                 float *table_host, int *n_rot_entries, int *pairs)
{
    if (n_rot < 0 || n_tilt < 0 || !table_host || !n_rot_entries || !pairs || (n_rot && !rot_deg) ||
        (n_tilt && !tilt_deg))
        return nx::fail(NX_EINVAL, "nx_insolation_plan: bad arguments");
    // pair mode: rotation h + n/2 is rotation h + 180 degrees exactly
    int pr = 0;
    if (n_rot > 0 && n_rot % 2 == 0) {
        pr = 1;
        for (int h = 0; h < n_rot / 2; ++h)
            if (rot_deg[h + n_rot / 2] != rot_deg[h] + 180.0) { pr = 0; break; }
    }
    int nr = pr ? n_rot / 2 : n_rot;
    trig_table(rot_deg, nr, table_host);
    trig_table(tilt_deg, n_tilt, table_host + 2 * nr);
    *n_rot_entries = nr;
    *pairs = pr;
    return NX_OK;
}

static int insolation_sums(const double *xyz_dev, int64_t n, double radius, const float *table_dev, int n_rot_entries,
                           int pairs, int n_tilt, float scale, float *out_dev, int accumulate, void *stream, const float *table_host = nullptr)
{
    if (n < 0 || n_rot_entries < 0 || n_tilt < 0) return nx::fail(NX_EINVAL, "nx_insolation: negative size");
    if (n == 0) return NX_OK;
    if (!xyz_dev || !out_dev || ((n_rot_entries || n_tilt) && !table_dev && !table_host))
        return nx::fail(NX_EINVAL, "nx_insolation: null pointer");
    if (!(radius > 0.0)) return nx::fail(NX_EINVAL, "nx_insolation: radius must be > 0");
    cudaStream_t s = (cudaStream_t)stream;
    if (n_rot_entries == 0 || n_tilt == 0) {
        if (!accumulate) NX_CHECK_CUDA(cudaMemsetAsync(out_dev, 0, sizeof(float) * (size_t)n, s));
        return NX_OK;
    }
    InsoArgs a;
    a.xyz = xyz_dev;
    a.n = n;
    a.r = radius;
    a.inv_r = (float)(1.0 / radius);
    radius_pair(radius, a.r2h, a.r2l);
    a.zmin = (float)(1e-20 * radius);
    a.rot = (const float2 *)table_dev;
    a.n_rot = n_rot_entries;
    a.pairs = pairs ? 1 : 0;
    a.tilt = (const float2 *)table_dev + n_rot_entries;
    a.n_tilt = n_tilt;
    a.out = out_dev;
    a.accumulate = accumulate;
    a.scale = scale;
    const size_t arcs = arc_smem(a.pairs ? 2 * a.n_rot : a.n_rot, a.pairs);
    if (table_host) {
        InsoTable T;
        memcpy(T.t, table_host, sizeof(float2) * (size_t)(n_rot_entries + n_tilt));
        if (breaks(a))
            insolation_args_kernel<12, true><<<grid_breaks(n), BREAK_THREADS, tilt_smem(a), s>>>(a, T);
        else if (use_arcs(a, n, a.r2h > 0.0f))
            insolation_args_kernel<ARCS><<<grid_arcs(n), arc_threads(n), arcs, s>>>(a, T);
        else
            insolation_args_kernel<0><<<grid_for(n), 256, 0, s>>>(a, T);
    } else if (breaks(a)) {
        insolation_kernel<12, true><<<grid_breaks(n), BREAK_THREADS, tilt_smem(a), s>>>(a);
    } else if (a.pairs && n_rot_entries == 12) {
        insolation_kernel<12><<<grid_for(n), 256, tilt_smem(a), s>>>(a);
    } else if (use_arcs(a, n, a.r2h > 0.0f)) {
        insolation_kernel<ARCS><<<grid_arcs(n), arc_threads(n), arcs, s>>>(a);
    } else {
        insolation_kernel<0><<<grid_for(n), 256, 0, s>>>(a);
    }
    NX_CHECK_LAUNCH("insolation_kernel");
    nx::note_launch(1);
    return NX_OK;
}

NX_EXPORT int nx_insolation(const double *xyz_dev, int64_t n, double radius, const float *table_dev, int n_rot_entries,
                            int pairs, int n_tilt, float *out_dev, int accumulate, void *stream)
{
    return insolation_sums(xyz_dev, n, radius, table_dev, n_rot_entries, pairs, n_tilt, 1.0f, out_dev, accumulate, stream);
}

NX_EXPORT int nx_insolation_positions(const double *xyz_dev, int64_t n, double radius, const double *rot_deg, int n_rot,
                                      const double *tilt_deg, int n_tilt, double scale, float *table_dev, float *out_dev,
                                      int accumulate, void *stream)
{
    if (n < 0 || n_rot < 0 || n_tilt < 0 || n_rot + (int64_t)n_tilt > NX_MAX_POSITIONS)
        return nx::fail(NX_EINVAL, "nx_insolation_positions: bad sizes");
    if (n == 0) return NX_OK;
    if (n_rot && n_tilt && !table_dev) return nx::fail(NX_EINVAL, "nx_insolation_positions: null pointer");
    float table[2 * NX_MAX_POSITIONS];
    int entries = 0, pairs = 0;
    int rc = nx_insolation_plan(rot_deg, n_rot, tilt_deg, n_tilt, table, &entries, &pairs);
    if (rc) return rc;
    const bool args = entries + n_tilt <= ARG_POSITIONS;
    if (n_rot && n_tilt && !args) {
        rc = nx_upload(table_dev, table, (int64_t)sizeof(float) * 2 * (entries + n_tilt), stream);
        if (rc) return rc;
    }
    return insolation_sums(xyz_dev, n, radius, table_dev, entries, pairs, n_tilt, (float)scale, out_dev, accumulate, stream,
                           args ? table : nullptr);
}

// climate.calculate_seasonal_tilt(axial, climate.day2deg(year, d)) for days
// d = 0..days-1, in the reference's order of operations (climate.py:171,
// 201) with the C library's sine, the one Python's math.sin calls.
NX_EXPORT int nx_seasonal_tilts(double axial_tilt, double year_length, int days, double *tilt_deg)
{
    if (days < 0 || (days && !tilt_deg)) return nx::fail(NX_EINVAL, "nx_seasonal_tilts: bad arguments");
    const double PI = 3.141592653589793;
    for (int d = 0; d < days; ++d) {
        const double deg = (double)d / year_length * 360.0;
        tilt_deg[d] = sin(deg * PI / 180) * axial_tilt;
    }
    return NX_OK;
}

NX_EXPORT int nx_insolation_batch(const nx_inso_planet *planets_dev, const nx_inso_planet *planets_host, int nplanets,
                                  const float *table_dev, int n_rot_entries, int pairs, int n_tilt, float *out_dev,
                                  void *stream)
{
    if (nplanets <= 0) return NX_OK;
    if (!planets_dev || !planets_host || !out_dev || !table_dev || n_rot_entries <= 0 || n_tilt <= 0)
        return nx::fail(NX_EINVAL, "nx_insolation_batch: bad arguments");
    int64_t total = 0;
    bool radius = true;
    for (int p = 0; p < nplanets; ++p) {
        const nx_inso_planet &P = planets_host[p];
        if (P.vbeg % 256 || P.n < 0 || (P.n > 0 && !P.xyz) || !(P.radius > 0) || P.vbeg < total)
            return nx::fail(NX_EINVAL, "nx_insolation_batch: planet %d: rows must be packed, 256-aligned", p);
        total = P.vbeg + P.n;
        float h, l;
        radius_pair(P.radius, h, l);
        radius = radius && h > 0.0f;
    }
    InsoArgs a;
    a.xyz = nullptr;
    a.n = 0;
    a.r = 1.0;
    a.inv_r = 1.0f;
    a.r2h = a.r2l = a.zmin = 0.0f;
    a.rot = (const float2 *)table_dev;
    a.n_rot = n_rot_entries;
    a.pairs = pairs ? 1 : 0;
    a.tilt = (const float2 *)table_dev + n_rot_entries;
    a.n_tilt = n_tilt;
    a.out = out_dev;
    a.accumulate = 0;
    a.scale = 1.0f;
    cudaStream_t s = (cudaStream_t)stream;
    if (breaks(a))
        insolation_batch_kernel<12, true><<<grid_for(total, 4), 256, tilt_smem(a), s>>>(a, planets_dev, nplanets, total);
    else if (a.pairs && n_rot_entries == 12)
        insolation_batch_kernel<12><<<grid_for(total), 256, tilt_smem(a), s>>>(a, planets_dev, nplanets, total);
    else if (use_arcs(a, total, radius))
        insolation_batch_kernel<ARCS><<<grid_for(total, 4), 256, arc_smem(a.pairs ? 2 * a.n_rot : a.n_rot, a.pairs), s>>>(
            a, planets_dev, nplanets, total);
    else
        insolation_batch_kernel<0><<<grid_for(total), 256, 0, s>>>(a, planets_dev, nplanets, total);
    NX_CHECK_LAUNCH("insolation_batch_kernel");
    nx::note_launch(1);
    return NX_OK;
}

// Daily latitude tables for n_tilts tilts (degrees, device array):
// tables_dev float[n_tilts * 181].
NX_EXPORT int nx_insolation_slices(const double *tilts_dev, int n_tilts, double radius, float *tables_dev,
                                   void *stream)
{
    if (n_tilts <= 0 || !tilts_dev || !tables_dev || !(radius > 0.0))
        return nx::fail(NX_EINVAL, "nx_insolation_slices: bad arguments");
    slice_kernel<<<n_tilts, 192, 0, (cudaStream_t)stream>>>(tilts_dev, n_tilts, radius, tables_dev);
    NX_CHECK_LAUNCH("slice_kernel");
    nx::note_launch(1);
    return NX_OK;
}

// Interpolated insolation of every vertex from n_tables tables, summed in
// binary32 in table order (accumulate = 1 adds to out_dev; with one table
// and accumulate = 0 the value is written as interpolate_insolation does).
NX_EXPORT int nx_interpolate_insolation(const double *xyz_dev, int64_t n, double radius, const float *tables_dev,
                                        int n_tables, float *out_dev, int accumulate, void *stream)
{
    if (n < 0 || n_tables <= 0 || (n > 0 && (!xyz_dev || !tables_dev || !out_dev)) || !(radius > 0.0))
        return nx::fail(NX_EINVAL, "nx_interpolate_insolation: bad arguments");
    if (n == 0) return NX_OK;
    interp_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(xyz_dev, n, radius, tables_dev, n_tables, out_dev,
                                                                 accumulate);
    NX_CHECK_LAUNCH("interp_kernel");
    nx::note_launch(1);
    return NX_OK;
}

// climate.assign_surface_temp: out_dev float[n] for the vertices xyz_dev.
NX_EXPORT int nx_surface_temp(const double *xyz_dev, int64_t n, double radius, double tilt, float *out_dev,
                              void *stream)
{
    if (n < 0 || (n > 0 && (!xyz_dev || !out_dev)) || !(radius > 0.0))
        return nx::fail(NX_EINVAL, "nx_surface_temp: bad arguments");
    if (n == 0) return NX_OK;
    surface_temp_kernel<<<grid_for(n), 256, 0, (cudaStream_t)stream>>>(xyz_dev, n, radius, tilt, out_dev);
    NX_CHECK_LAUNCH("surface_temp_kernel");
    nx::note_launch(1);
    return NX_OK;
}
