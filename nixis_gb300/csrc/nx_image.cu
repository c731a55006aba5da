// nx_image.cu -- equirectangular map sampling (util.py:290-366, nixis.py:270-302):
// the pixel positions of make_ll_arr and the inverse-distance weighting of
// make_gray_array, in binary64 with the reference's operation order.  The
// three nearest vertices of each pixel come from nx_nearest3 (nx_mesh.cu).
#include "nx_common.cuh"
#include "nx_f64.cuh"

namespace nx {
void note_launch(int k);
}

namespace {

constexpr double PI = 3.141592653589793;

// make_ll_arr (util.py:290-310): row h at latitude max(90 - h*180/(height-1),
// -90), column w at longitude max(-180 + w*360/width, -180), through
// util.latlon2xyz (util.py:79-88).  A block takes LL_ROWS rows of 256 columns:
// a column's sine and cosine are computed once per block, a row's once per
// block row, instead of all four per pixel (binary64 sines and cosines, ~40
// operations each on a pipe of two per SM and cycle).  32 rows, or 4 where 32
// would leave three SMs in four without a block.  PART: rows from `base` on.
// Measured (GB300): 1,024 x 512 pixels 103 -> 14.4 us; 256 x 128 pixels 8.9 us
// one by one, 13.4 in blocks of 32 rows and 8.1 of 4, 400 x 200 24.2, 14.3, 8.1.
template <int LL_ROWS, bool PART>
__global__ void __launch_bounds__(256) make_ll_kernel(int width, int height, int base, double radius, double *__restrict__ out)
{
    __shared__ double s_rc[LL_ROWS], s_z[LL_ROWS];           // radius cos(lat), radius sin(lat)
    const int h0 = (PART ? base : 0) + blockIdx.y * LL_ROWS;
    if (threadIdx.x < LL_ROWS) {
        const double latpercent = 180.0 / (double)(height - 1);
        const double lat = fmax(__dsub_rn(90.0, __dmul_rn((double)(h0 + (int)threadIdx.x), latpercent)), -90.0);
        const double a = __dmul_rn(lat, PI / 180);
        s_rc[threadIdx.x] = __dmul_rn(radius, cos(a));
        s_z[threadIdx.x] = __dmul_rn(radius, sin(a));
    }
    __syncthreads();
    const int w = blockIdx.x * 256 + threadIdx.x;
    if (w >= width) return;
    const double lonpercent = 360.0 / (double)width;
    const double lon = fmax(__dadd_rn(-180.0, __dmul_rn((double)w, lonpercent)), -180.0);
    const double b = __dmul_rn(lon, PI / 180);
    const double cb = cos(b), sb = sin(b);
    const int rows = min(LL_ROWS, height - h0);
    for (int r = 0; r < rows; ++r) {
        double *o = out + 3 * ((int64_t)(h0 + r) * width + w);
        o[0] = __dmul_rn(s_rc[r], cb);
        o[1] = __dmul_rn(s_rc[r], sb);
        o[2] = s_z[r];
    }
}

// make_gray_array (util.py:342-366) per pixel: weights 1 / ((d + 1e-5) / sum d)
// normalised by their sum, the weighted colours summed in slot order and
// truncated toward zero (Python int()).  Quotients with one binary64 operation
// each (nx_f64.cuh); measured (GB300, 1024 x 512 pixels): 77 -> 32 us.
__global__ void __launch_bounds__(256) gray_kernel(const double *__restrict__ dist, const int64_t *__restrict__ idx,
                                                   int64_t np, const double *__restrict__ colors, int64_t nc,
                                                   double *__restrict__ out, int *__restrict__ err)
{
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < np; p += (int64_t)gridDim.x * blockDim.x) {
        const double *d = dist + 3 * p;
        const nxf::Recip sd = nxf::recip(__dadd_rn(__dadd_rn(d[0], d[1]), d[2]));
        double ws[3];
        for (int k = 0; k < 3; ++k) ws[k] = nxf::div(1.0, nxf::recip(nxf::div(__dadd_rn(d[k], 0.00001), sd)));
        const nxf::Recip t = nxf::recip(__dadd_rn(__dadd_rn(ws[0], ws[1]), ws[2]));
        double acc = 0.0;
        for (int k = 0; k < 3; ++k) {
            const int64_t v = idx[3 * p + k];
            if (v < 0 || v >= nc) {
                atomicOr(err, 1);
                continue;
            }
            acc = __dadd_rn(acc, __dmul_rn(colors[v], nxf::div(ws[k], t)));
        }
        out[p] = trunc(acc);
    }
}

int grid_for(int64_t n)
{
    int64_t g = (n + 255) / 256;
    const int64_t cap = (int64_t)nx::sm_count() * 8;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

}  // namespace

NX_EXPORT int nx_make_ll(int width, int height, double radius, double *out_dev, void *stream)
{
    if (width < 1 || height < 2 || !out_dev) return nx::fail(NX_EINVAL, "nx_make_ll: bad arguments");
    const cudaStream_t s = (cudaStream_t)stream;
    const int64_t xb = (width + 255LL) / 256;
    auto grid = [&](int64_t h, int rows) { return dim3((unsigned)xb, (unsigned)((h + rows - 1) / rows)); };
    // (a grid's y is at most 65,535 blocks: taller maps in parts)
    const int64_t part = 65535LL * 32;
    for (int64_t base = 0; base < height; base += part) {
        const int64_t h = height - base < part ? height - base : part;
        if (height > part)
            make_ll_kernel<32, true><<<grid(h, 32), 256, 0, s>>>(width, height, (int)base, radius, out_dev);
        else if (xb * ((h + 31) / 32) < nx::sm_count() / 4)
            make_ll_kernel<4, false><<<grid(h, 4), 256, 0, s>>>(width, height, 0, radius, out_dev);
        else
            make_ll_kernel<32, false><<<grid(h, 32), 256, 0, s>>>(width, height, 0, radius, out_dev);
        NX_CHECK_LAUNCH("make_ll_kernel");
        nx::note_launch(1);
    }
    return NX_OK;
}

NX_EXPORT int nx_sample_gray(const double *dist_dev, const int64_t *idx_dev, int64_t npix, const double *colors_dev,
                             int64_t ncolors, double *out_dev, int *err_dev, void *stream)
{
    if (npix < 0 || (npix > 0 && (!dist_dev || !idx_dev || !colors_dev || !out_dev || !err_dev)))
        return nx::fail(NX_EINVAL, "nx_sample_gray: bad arguments");
    if (npix == 0) return NX_OK;
    gray_kernel<<<grid_for(npix), 256, 0, (cudaStream_t)stream>>>(dist_dev, idx_dev, npix, colors_dev, ncolors, out_dev,
                                                                  err_dev);
    NX_CHECK_LAUNCH("gray_kernel");
    nx::note_launch(1);
    return NX_OK;
}
