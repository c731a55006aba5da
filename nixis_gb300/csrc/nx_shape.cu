// nx_shape.cu -- the post-noise height shaping of nixis.py:330-364 on the GPU:
// util.rescale (util.py:110-176, all of its forms), util.find_percent_val
// (util.py:556-566), terrain.make_bool_elevation_mask (terrain.py:61-72) and
// util.power_rescale (util.py:179-250), in binary64 with the reference's
// operation order.
//
// Reductions are exact and order independent: min and max as atomics on
// ordered 64-bit keys.  power_rescale finds the masked range with a running
// update, `if x < lo: lo = x  elif x > hi: hi = x` from lo = max(x),
// hi = min(x) (util.py:203-214); a value that is a new running minimum (a
// record) is never considered for the maximum.  So hi = max(min(x), max of
// the selected values that are no records).  A run of values is summed up
// by its first value, its minimum and the largest value that is no record
// within the run; two adjacent runs join into one, because the second's
// records are records of the whole only while they lie below the first's
// minimum, and its first value is the largest of them.  One pass leaves a
// summary per chunk, and the last block to finish joins the chunks'.
//
// All scalars (ranges, the ocean level) stay in the workspace on the device:
// a shaping run makes no host round trip.
//
// What bounds it: binary64 operations (two per SM and cycle on GB300), not
// memory.  A division or square root costs one of them (nx_f64.cuh) instead
// of about ten, comparisons and keys none (integers), operations of the
// reference that change nothing (* 1.0, / 1.0, + 0.0) are left out, and the
// whole shaping is four passes, ~11 binary64 operations a vertex: the two
// masked ranges come from one pass over h1 (the land's values are the same
// before and after the ocean's power curve), and the extremes of a monotone
// map are the map of the extremes, so neither needs a pass of its own.
// Measured (GB300, shape_heights of 6,400,002 heights): 975 -> 268 us (20
// passes before); with the products put together from integers as well
// (nxf::mul) 280 -> 250 us on another machine, a rescale 84 -> 67: the
// binary64 pipe is then busy for 49-77 % of a pass, the integer one for 58-62.
#include "nx_common.cuh"
#include "nx_f64.cuh"

namespace nx {
void note_launch(int k);
}

namespace {

typedef unsigned long long u64;

constexpr int THREADS = 256;
constexpr int PER_THREAD = 8;
constexpr int CHUNK = THREADS * PER_THREAD;   // elements per summary
constexpr u64 NONE = ~0ull;

__device__ __forceinline__ u64 umin(u64 a, u64 b) { return a < b ? a : b; }

// Ordered key of a binary64, below NONE: -0 taken as +0, as the reference's
// comparisons see them equal.  A NaN with its sign bit set, as 0 / 0 gives, is
// smaller than all numbers, so the minimum is NaN with it; any other NaN comes
// right below 0, so in a field on both sides of 0 it is neither extreme.  -0 and
// NaNs are found by the high word and leave the others the two operations of the
// sign (shape_heights of 6,400,002 heights 246.4 us; with 64-bit comparisons for
// every key 251.5).
constexpr u64 KEY_SIGN = 0x8000000000000000ull, KEY_NAN = 0x7FF7FFFFFFFFFFFFull;

__device__ __forceinline__ u64 dkey(double v)
{
    const u64 b = nxf::bits(v);
    const unsigned hi = (unsigned)(b >> 32);
    u64 k = b ^ ((u64)((long long)b >> 63) | KEY_SIGN);
    if (hi == 0x80000000u || (hi < 0x80000000u && hi >= 0x7FF00000u)) {
        if (b == KEY_SIGN) k = KEY_SIGN;
        if ((long long)b > 0x7FF0000000000000ll) k = KEY_NAN;
    }
    return k;
}

__device__ __forceinline__ double dunkey(u64 k)
{
    const u64 b = (k & KEY_SIGN) ? (k & ~KEY_SIGN) : ~k;
    return __longlong_as_double((long long)b);
}

__device__ __forceinline__ u64 umax(u64 a, u64 b) { return a > b ? a : b; }
__device__ __forceinline__ bool is_nan(double v) { return (nxf::bits(v) << 1) > 0xFFE0000000000000ull; }

// Minimum and maximum keys, the minimum inverted so that both start at 0.
struct Extremes {
    u64 nmin, max;
};

// A masked range and its map's constants.
struct Range {
    double lo, hi;
};

// util.rescale.  form: 0 plain, 1 with mid, 2 mode 'lower', 3 mode 'upper'.
// u_min / u_max widen the input range (util.py:128-131).
struct RescaleArgs {
    double lower, upper, mid, u_min, u_max;
    int form, has_umin, has_umax;
};

// One linear map ((v - from) / span) * width + to.
struct Linear {
    double from, to;
    nxf::Factor width;
    nxf::Recip span;
    __device__ __forceinline__ double operator()(double v) const
    {
        return __dadd_rn(nxf::mul(nxf::div(__dsub_rn(v, from), span), width), to);
    }
};

__device__ __forceinline__ Linear rescale_low(const RescaleArgs &a, double x_min, double x_max)
{
    const double end = a.form == 0 ? x_max : a.mid, top = a.form == 0 ? a.upper : a.mid;
    return Linear{x_min, a.lower, nxf::factor(__dsub_rn(top, a.lower)), nxf::recip(__dsub_rn(end, x_min))};
}

// find_percent_val (util.py:556-566)
__device__ __forceinline__ double percent_val(double mn, double mx, double percent)
{
    if (!(0.0 < percent && percent < 100.0)) percent = 50.0;
    return __dadd_rn(mn, __ddiv_rn(__dmul_rn(__dsub_rn(mx, mn), percent), 100.0));
}

// Workspace (zeroed before a run), then the chunks' summaries.
struct Ws {
    Extremes in, shifted;      // of the input; of the heights less the ocean level
    double level;              // ocean level (find_percent_val)
    Range range[2];            // power_rescale's, by mode (shape_heights: [1] the ocean's, [0] the land's)
    Linear base;               // shape_heights: the first rescale, and its image's extremes (keys)
    u64 kmin, kmax;
    unsigned blocks, done;     // blocks done with the pass over the input; with the pass that writes summaries
    u64 pad;
};

__device__ __forceinline__ double ext_min(const Extremes &e) { return dunkey(~e.nmin); }
__device__ __forceinline__ double ext_max(const Extremes &e) { return dunkey(e.max); }

// Fold every thread's keys into e: one pair of atomics per block.
__device__ __forceinline__ void fold_extremes(u64 nmin, u64 max, Extremes *e)
{
    __shared__ u64 s_e[2][THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) {
        nmin = umax(nmin, __shfl_xor_sync(0xFFFFFFFFu, nmin, o));
        max = umax(max, __shfl_xor_sync(0xFFFFFFFFu, max, o));
    }
    if ((threadIdx.x & 31) == 0) { s_e[0][threadIdx.x >> 5] = nmin; s_e[1][threadIdx.x >> 5] = max; }
    __syncthreads();
    if (threadIdx.x < 2) {
        u64 m = s_e[threadIdx.x][0];
        for (int k = 1; k < THREADS / 32; ++k) m = umax(m, s_e[threadIdx.x][k]);
        atomicMax(threadIdx.x ? &e->max : &e->nmin, m);
    }
}

// Last block to get here (what all of them wrote before is then visible).
__device__ __forceinline__ bool last_block(unsigned *count)
{
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(count, 1u) + 1 == gridDim.x;
        __threadfence();
    }
    __syncthreads();
    return s_last;
}

// The workspace's words, zeroed before each use.  A memset on the stream is 2 us
// dearer between two kernels than this one: the rescale of 4,002 heights 8.6 us
// with it, 6.7 without (GB300).
static_assert(sizeof(Ws) % 8 == 0, "zeroed by words");
__global__ void zero_ws_kernel(u64 *__restrict__ w)
{
    for (int i = threadIdx.x; i < (int)(sizeof(Ws) / 8); i += 32) w[i] = 0;
}

// np.min / np.max (util.py:125-126, 195-196)
// For shape_heights (SHAPE) the last block leaves the first rescale, h1's
// extremes (the map of h's: each of its steps is monotone) and the ocean
// level.
template <bool SHAPE>
__global__ void __launch_bounds__(THREADS) minmax_kernel(const double *__restrict__ x, int64_t n, RescaleArgs a,
                                                         double percent, double *__restrict__ level_out, Ws *w)
{
    u64 nmin = 0, max = 0;
    const int64_t step = (int64_t)gridDim.x * THREADS;
    int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x;
    for (; i + 3 * step < n; i += 4 * step) {
        double v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = x[i + k * step];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const u64 q = dkey(v[k]);
            nmin = umax(nmin, ~q);
            max = umax(max, q);
        }
    }
    for (; i < n; i += step) {
        const u64 q = dkey(x[i]);
        nmin = umax(nmin, ~q);
        max = umax(max, q);
    }
    fold_extremes(nmin, max, &w->in);
    if (!SHAPE || !last_block(&w->blocks) || threadIdx.x) return;
    const volatile Extremes *e = &w->in;
    const double x_min = dunkey(~e->nmin), x_max = dunkey(e->max);
    w->base = rescale_low(a, x_min, x_max);
    const u64 p = dkey(w->base(x_min)), q = dkey(w->base(x_max));
    w->kmin = umin(p, q);
    w->kmax = umax(p, q);
    w->level = percent_val(dunkey(w->kmin), dunkey(w->kmax), percent);
    if (level_out) *level_out = w->level;
}

template <int FORM>
__global__ void __launch_bounds__(THREADS) rescale_kernel(const double *__restrict__ x, int64_t n, const Extremes *e,
                                                          RescaleArgs a, double *__restrict__ out)
{
    double x_min = ext_min(*e), x_max = ext_max(*e);
    if (a.has_umin && a.u_min < x_min) x_min = a.u_min;
    if (a.has_umax && a.u_max > x_max) x_max = a.u_max;
    const Linear low = rescale_low(a, x_min, x_max);
    const Linear high{a.mid, a.mid, nxf::factor(__dsub_rn(a.upper, a.mid)), nxf::recip(__dsub_rn(x_max, a.mid))};
    // v <= mid and v >= mid by keys (false for a NaN on either side)
    const bool no_mid = is_nan(a.mid);
    const u64 kmid = dkey(a.mid);
    for (int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * THREADS) {
        const double v = x[i];
        if (FORM == 0) {
            out[i] = low(v);
            continue;
        }
        const u64 k = dkey(v);
        const bool none = no_mid || is_nan(v), below = !none && k <= kmid;
        if (FORM == 1) {
            // the operands selected, so that warps on both sides run one path
            const Linear both{nxf::pick(below, low.from, high.from), nxf::pick(below, low.to, high.to),
                              nxf::Factor{nxf::pick(below, low.width.b, high.width.b),
                                          below ? low.width.m : high.width.m, below ? low.width.hw : high.width.hw},
                              nxf::Recip{nxf::pick(below, low.span.b, high.span.b), below ? low.span.y1 : high.span.y1,
                                         below ? low.span.y2 : high.span.y2}};
            out[i] = both(v);
        } else if (FORM == 2) {
            out[i] = below ? low(v) : v;
        } else {
            out[i] = !none && k >= kmid ? high(v) : v;
        }
    }
}

// make_bool_elevation_mask (terrain.py:61-72): height <= level
// One binary64 comparison to eight bytes read: comparing keys instead measured
// 4.9 against 4.2 us (GB300, 900,002 heights).
__global__ void __launch_bounds__(THREADS) mask_kernel(const double *__restrict__ h, int64_t n, double level,
                                                       uint8_t *__restrict__ mask)
{
    for (int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * THREADS)
        mask[i] = h[i] <= level ? 1 : 0;
}

// A run of selected values: the first one's key, the smallest key, the
// largest key that is no record of the run (0: none); min = NONE: empty.
struct Run {
    u64 first, min, rest;
};

__device__ __forceinline__ Run empty_run() { return Run{NONE, NONE, 0ull}; }

__device__ __forceinline__ void append(Run &r, u64 k)
{
    if (r.min == NONE) r.first = r.min = k;
    else if (k < r.min) r.min = k;
    else r.rest = umax(r.rest, k);
}

// a followed by b
__device__ __forceinline__ Run join(const Run &a, const Run &b)
{
    if (a.min == NONE) return b;
    if (b.min == NONE) return a;
    u64 rest = umax(a.rest, b.rest);
    if (b.first >= a.min) rest = umax(rest, b.first);
    return Run{a.first, umin(a.min, b.min), rest};
}

// The runs of a block's threads (in thread order), joined; valid in thread 0.
__device__ __forceinline__ Run join_block(Run r)
{
    __shared__ Run s_run[32];
    for (int o = 1; o < 32; o <<= 1) {
        const Run b = {__shfl_down_sync(0xFFFFFFFFu, r.first, o), __shfl_down_sync(0xFFFFFFFFu, r.min, o),
                       __shfl_down_sync(0xFFFFFFFFu, r.rest, o)};
        r = join(r, b);                 // lanes at multiples of 2 o hold 2 o threads
    }
    __syncthreads();                    // (s_run may still be read from a call before)
    if ((threadIdx.x & 31) == 0) s_run[threadIdx.x >> 5] = r;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int k = 1; k < (int)(blockDim.x >> 5); ++k) r = join(r, s_run[k]);
    return r;
}

// power_rescale's range from the whole run and np.min / np.max of the field
// (keys).
__device__ __forceinline__ Range range_of(const Run &r, u64 kmin, u64 kmax)
{
    u64 hi = umax(kmin, r.rest);
    if (r.min != NONE && r.first >= kmax) hi = umax(hi, r.first);
    return Range{dunkey(umin(kmax, r.min)), dunkey(hi)};
}

// The map of power_rescale (util.py:223-248): ((v - lo) / range) ** power,
// back to the range.
struct Curve {
    double lo, power;
    nxf::Factor range;
    nxf::Recip span;
    __device__ __forceinline__ double operator()(double v) const
    {
        double t = nxf::div(__dsub_rn(v, lo), span);
        if (power == 2.0) t = __dmul_rn(t, t);
        else if (power == 0.5) t = nxf::sqrt(t);
        else if (power != 1.0) t = pow(__dadd_rn(t, 0.0), power);
        return __dadd_rn(nxf::mul(t, range), lo);
    }
};

__device__ __forceinline__ Curve curve_of(const Range &r, double power)
{
    const double range = __dsub_rn(r.hi, r.lo);
    return Curve{r.lo, power, nxf::factor(range), nxf::recip(range)};
}

// All chunks' runs joined by one block; valid in thread 0.
__device__ __forceinline__ Run join_chunks(const Run *runs, int64_t nchunks)
{
    const int64_t per = (nchunks + THREADS - 1) / THREADS;
    const int64_t b = (int64_t)threadIdx.x * per, e = b + per < nchunks ? b + per : nchunks;
    Run r = empty_run();
    for (int64_t c = b; c < e; ++c) {
        const volatile Run *q = runs + c;
        r = join(r, Run{q->first, q->min, q->rest});
    }
    return join_block(r);
}

// Key k of a chunk in shared memory: a thread's consecutive ones without
// bank conflicts.
__device__ __forceinline__ int slot(int k) { return k + k / PER_THREAD; }

// power_rescale: the masked range.
__global__ void __launch_bounds__(THREADS) range_kernel(const double *__restrict__ x, const uint8_t *__restrict__ mask,
                                                        int64_t n, int mode, Run *runs, Ws *w)
{
    __shared__ u64 s_key[CHUNK + CHUNK / PER_THREAD];
    const int64_t b = (int64_t)blockIdx.x * CHUNK;
    for (int k = threadIdx.x; k < CHUNK; k += THREADS) {
        const int64_t i = b + k;
        s_key[slot(k)] = i < n && (mask[i] != 0) == (mode == 1) ? dkey(x[i]) : NONE;
    }
    __syncthreads();
    Run r = empty_run();
    for (int k = 0; k < PER_THREAD; ++k) {
        const u64 q = s_key[slot(threadIdx.x * PER_THREAD + k)];
        if (q != NONE) append(r, q);
    }
    r = join_block(r);
    if (threadIdx.x == 0) runs[blockIdx.x] = r;
    if (!last_block(&w->done)) return;
    r = join_chunks(runs, gridDim.x);
    if (threadIdx.x == 0) w->range[mode] = range_of(r, ~w->in.nmin, w->in.max);
}

__global__ void __launch_bounds__(THREADS) power_map_kernel(const double *__restrict__ x, const uint8_t *__restrict__ mask,
                                                            int64_t n, int mode, double power, const Ws *w,
                                                            double *__restrict__ out)
{
    const Curve curve = curve_of(w->range[mode < 0 ? 0 : mode], power);
    for (int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * THREADS) {
        const double v = x[i];
        out[i] = mode >= 0 && (mask[i] != 0) == (mode == 1) ? curve(v) : v;
    }
}

// shape_heights, pass 2: h1 = rescale(h), the ocean mask, and the runs of
// the ocean's and the land's values; the last block leaves both ranges.
__global__ void __launch_bounds__(THREADS) shape_base_kernel(const double *__restrict__ h, int64_t n,
                                                             double *__restrict__ h1, uint8_t *__restrict__ mask,
                                                             Run *runs, Ws *w)
{
    __shared__ u64 s_key[CHUNK + CHUNK / PER_THREAD];
    const Linear low = w->base;
    const bool dry = is_nan(w->level);
    const u64 klev = dkey(w->level);
    const int64_t b = (int64_t)blockIdx.x * CHUNK;
    for (int k = threadIdx.x; k < CHUNK; k += THREADS) {
        const int64_t i = b + k;
        u64 q = NONE;
        if (i < n) {
            const double v = low(h[i]);
            h1[i] = v;
            q = dkey(v);
            mask[i] = !dry && q <= klev && q != KEY_NAN ? 1 : 0;
        }
        s_key[slot(k)] = q;
    }
    __syncthreads();
    Run sea = empty_run(), land = empty_run();
    for (int k = 0; k < PER_THREAD; ++k) {
        const u64 q = s_key[slot(threadIdx.x * PER_THREAD + k)];
        if (q == NONE) continue;
        if (!dry && q <= klev && q != KEY_NAN) append(sea, q);
        else append(land, q);
    }
    sea = join_block(sea);
    land = join_block(land);
    if (threadIdx.x == 0) {
        runs[2 * (int64_t)blockIdx.x] = sea;
        runs[2 * (int64_t)blockIdx.x + 1] = land;
    }
    if (!last_block(&w->done)) return;
    // the chunks' runs, sea and land alternating
    const int64_t nc = gridDim.x, per = (nc + THREADS - 1) / THREADS;
    const int64_t cb = (int64_t)threadIdx.x * per, ce = cb + per < nc ? cb + per : nc;
    Run all[2] = {empty_run(), empty_run()};
    for (int64_t c = cb; c < ce; ++c)
        for (int m = 0; m < 2; ++m) {
            const volatile Run *q = runs + 2 * c + m;
            all[m] = join(all[m], Run{q->first, q->min, q->rest});
        }
    sea = join_block(all[0]);
    land = join_block(all[1]);
    if (threadIdx.x) return;
    const Range r1 = range_of(sea, w->kmin, w->kmax);
    w->range[1] = r1;
    // np.min / np.max of h2: the land as it is, the ocean's ends through the
    // curve (monotone for a positive range; otherwise it gives NaN)
    u64 k2min = land.min, k2max = land.min == NONE ? 0ull : umax(land.rest, land.first);
    if (sea.min != NONE) {
        const Curve curve = curve_of(r1, 0.5);
        const u64 p = dkey(curve(dunkey(sea.min))), q = dkey(curve(dunkey(umax(sea.rest, sea.first))));
        k2min = umin(k2min, umin(p, q));
        k2max = umax(k2max, umax(p, q));
    }
    w->range[0] = range_of(land, k2min, k2max);
}

// pass 3: the ocean's and the land's power curves, less the ocean level
__global__ void __launch_bounds__(THREADS) shape_curve_kernel(const double *__restrict__ h1, int64_t n, Ws *w,
                                                              double *__restrict__ h4)
{
    const Curve sea = curve_of(w->range[1], 0.5), land = curve_of(w->range[0], 2.0);
    const double level = w->level;
    const bool dry = is_nan(level);
    const u64 klev = dkey(level);
    u64 nmin = 0, max = 0;
    for (int64_t i = (int64_t)blockIdx.x * THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * THREADS) {
        const double v = h1[i];
        // the operands selected, so that a coast's warps run one path
        const u64 k = dkey(v);
        const bool wet = !dry && k <= klev && k != KEY_NAN;
        const double lo = nxf::pick(wet, sea.lo, land.lo);
        const nxf::Factor range{nxf::pick(wet, sea.range.b, land.range.b), wet ? sea.range.m : land.range.m,
                                wet ? sea.range.hw : land.range.hw};
        double t = nxf::div(__dsub_rn(v, lo), nxf::Recip{range.b, wet ? sea.span.y1 : land.span.y1, wet ? sea.span.y2 : land.span.y2});
        if (wet) t = nxf::sqrt(t);
        else t = nxf::mul(t, nxf::factor(t));
        const double r = __dsub_rn(__dadd_rn(nxf::mul(t, range), lo), level);
        h4[i] = r;
        const u64 q = dkey(r);
        nmin = umax(nmin, ~q);
        max = umax(max, q);
    }
    fold_extremes(nmin, max, &w->shifted);
}

int grid_for(int64_t n)
{
    int64_t g = (n + THREADS - 1) / THREADS;
    const int64_t cap = (int64_t)nx::sm_count() * 8;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

int64_t nchunks_of(int64_t n) { return (n + CHUNK - 1) / CHUNK; }

int launch_minmax(const double *x, int64_t n, Ws *w, cudaStream_t s)
{
    zero_ws_kernel<<<1, 32, 0, s>>>((u64 *)w);
    NX_CHECK_LAUNCH("zero_ws_kernel");
    nx::note_launch(1);
    minmax_kernel<false><<<grid_for(n), THREADS, 0, s>>>(x, n, RescaleArgs(), 0.0, nullptr, w);
    NX_CHECK_LAUNCH("minmax_kernel");
    nx::note_launch(1);
    return NX_OK;
}

int launch_rescale(const double *x, int64_t n, const RescaleArgs &a, const Extremes *e, double *out, cudaStream_t s)
{
    const int g = grid_for(n);
    if (a.form == 0) rescale_kernel<0><<<g, THREADS, 0, s>>>(x, n, e, a, out);
    else if (a.form == 1) rescale_kernel<1><<<g, THREADS, 0, s>>>(x, n, e, a, out);
    else if (a.form == 2) rescale_kernel<2><<<g, THREADS, 0, s>>>(x, n, e, a, out);
    else rescale_kernel<3><<<g, THREADS, 0, s>>>(x, n, e, a, out);
    NX_CHECK_LAUNCH("rescale_kernel");
    nx::note_launch(1);
    return NX_OK;
}

int check_ws(void *ws, size_t ws_bytes, int64_t n, const char *who);

}  // namespace

NX_EXPORT size_t nx_shape_workspace_size(int64_t n)
{
    return sizeof(Ws) + 2 * sizeof(Run) * (size_t)(nchunks_of(n > 0 ? n : 1)) + 64;
}

namespace {
int check_ws(void *ws, size_t ws_bytes, int64_t n, const char *who)
{
    if (!ws) return nx::fail(NX_EINVAL, "%s: null workspace", who);
    if (((uintptr_t)ws) % 16) return nx::fail(NX_EINVAL, "%s: workspace must be 16-byte aligned", who);
    if (ws_bytes < nx_shape_workspace_size(n)) return nx::fail(NX_EINVAL, "%s: workspace too small", who);
    return NX_OK;
}
}  // namespace

NX_EXPORT int nx_rescale(const double *x_dev, int64_t n, double lower, double upper, double mid, int form,
                         double u_min, int has_umin, double u_max, int has_umax, double *out_dev, void *ws,
                         size_t ws_bytes, void *stream)
{
    if (n <= 0) return nx::fail(NX_EINVAL, "nx_rescale: n must be > 0");
    if (!x_dev || !out_dev) return nx::fail(NX_EINVAL, "nx_rescale: null pointer");
    if (form < 0 || form > 3) return nx::fail(NX_EINVAL, "nx_rescale: form must be 0-3");
    int rc = check_ws(ws, ws_bytes, n, "nx_rescale");
    if (rc) return rc;
    RescaleArgs a;
    a.lower = lower; a.upper = upper; a.mid = mid; a.u_min = u_min; a.u_max = u_max;
    a.form = form; a.has_umin = has_umin != 0; a.has_umax = has_umax != 0;
    cudaStream_t s = (cudaStream_t)stream;
    Ws *w = (Ws *)ws;
    rc = launch_minmax(x_dev, n, w, s);
    if (rc) return rc;
    return launch_rescale(x_dev, n, a, &w->in, out_dev, s);
}

NX_EXPORT int nx_power_rescale(const double *x_dev, int64_t n, const uint8_t *mask_dev, int mode, double power,
                               double *out_dev, void *ws, size_t ws_bytes, void *stream)
{
    if (n <= 0) return nx::fail(NX_EINVAL, "nx_power_rescale: n must be > 0");
    if (!x_dev || !out_dev) return nx::fail(NX_EINVAL, "nx_power_rescale: null pointer");
    if (mode != -1 && mode != 0 && mode != 1) return nx::fail(NX_EINVAL, "nx_power_rescale: mode must be -1, 0 or 1");
    if (mode >= 0 && !mask_dev) return nx::fail(NX_EINVAL, "nx_power_rescale: mode %d needs a mask", mode);
    int rc = check_ws(ws, ws_bytes, n, "nx_power_rescale");
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    Ws *w = (Ws *)ws;
    rc = launch_minmax(x_dev, n, w, s);
    if (rc) return rc;
    if (mode >= 0) {
        range_kernel<<<(unsigned)nchunks_of(n), THREADS, 0, s>>>(x_dev, mask_dev, n, mode, (Run *)(w + 1), w);
        NX_CHECK_LAUNCH("range_kernel");
        nx::note_launch(1);
    }
    power_map_kernel<<<grid_for(n), THREADS, 0, s>>>(x_dev, mask_dev, n, mode, power, w, out_dev);
    NX_CHECK_LAUNCH("power_map_kernel");
    nx::note_launch(1);
    return NX_OK;
}

NX_EXPORT int nx_elevation_mask(const double *h_dev, int64_t n, double level, uint8_t *mask_dev, void *stream)
{
    if (n < 0 || (n > 0 && (!h_dev || !mask_dev))) return nx::fail(NX_EINVAL, "nx_elevation_mask: bad arguments");
    if (n == 0) return NX_OK;
    mask_kernel<<<grid_for(n), THREADS, 0, (cudaStream_t)stream>>>(h_dev, n, level, mask_dev);
    NX_CHECK_LAUNCH("mask_kernel");
    nx::note_launch(1);
    return NX_OK;
}

// nixis.py:332-364 with h1..h5 as there: h1 = rescale(h, min_alt, max_alt);
// level = find_percent_val(min h1, max h1, ocean_percent); ocean = h1 <= level;
// h2 = power_rescale(h1, ocean, 1, 0.5); h3 = power_rescale(h2, ocean, 0, 2.0);
// h5 = rescale(h3 - level, min_alt, max_alt, mid=0).  out_dev gets h5,
// mask_dev (optional) the ocean mask, level_dev (optional) the level.
// tmp_dev: a second array of n doubles.
NX_EXPORT int nx_shape_heights(const double *h_dev, int64_t n, double min_alt, double max_alt, double ocean_percent,
                               double *out_dev, double *tmp_dev, uint8_t *mask_dev, double *level_dev, void *ws,
                               size_t ws_bytes, void *stream)
{
    if (n <= 0) return nx::fail(NX_EINVAL, "nx_shape_heights: n must be > 0");
    if (!h_dev || !out_dev || !tmp_dev || !mask_dev) return nx::fail(NX_EINVAL, "nx_shape_heights: null pointer");
    int rc = check_ws(ws, ws_bytes, n, "nx_shape_heights");
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    Ws *w = (Ws *)ws;
    RescaleArgs a;
    a.lower = min_alt; a.upper = max_alt; a.mid = 0.0; a.u_min = 0.0; a.u_max = 0.0;
    a.form = 0; a.has_umin = 0; a.has_umax = 0;
    zero_ws_kernel<<<1, 32, 0, s>>>((u64 *)w);
    NX_CHECK_LAUNCH("zero_ws_kernel");
    nx::note_launch(1);
    minmax_kernel<true><<<grid_for(n), THREADS, 0, s>>>(h_dev, n, a, ocean_percent, level_dev, w);
    NX_CHECK_LAUNCH("minmax_kernel");
    shape_base_kernel<<<(unsigned)nchunks_of(n), THREADS, 0, s>>>(h_dev, n, out_dev, mask_dev, (Run *)(w + 1), w);   // h1 -> out
    NX_CHECK_LAUNCH("shape_base_kernel");
    shape_curve_kernel<<<grid_for(n), THREADS, 0, s>>>(out_dev, n, w, tmp_dev);            // h4 -> tmp
    NX_CHECK_LAUNCH("shape_curve_kernel");
    nx::note_launch(3);
    a.form = 1;
    return launch_rescale(tmp_dev, n, a, &w->shifted, out_dev, s);                         // h5 -> out
}
