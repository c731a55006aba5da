// nx_mesh.cu -- icosphere generation, adjacency and per-slot edge lengths.
//
// The reference gets its sphere from meshzoo.icosa_sphere (util.py:43) and
// its neighbour table from build_adjacency + sort_adjacency (util.py:591-662).
// meshzoo is not available, so the vertex layout here is this project's own
// (documented in nixis_gb300/icosphere.py); the adjacency kernels implement
// the reference's two functions for any consistently wound triangle mesh, so
// the neighbour table equals what the reference computes from the same
// triangles.
#include <algorithm>
#include <climits>
#include <cmath>

#include "nx_common.cuh"
#include "nx_f64.cuh"

namespace nx {
void note_launch(int k);
}

namespace {

struct IcoTables {
    double corner[12][3];
    int face[20][3];
    int fedge[20][3][2];   // per face side (AB, AC, BC): edge id, 1 if it runs low->high corner
    int edge[30][2];
    double inv[20][3][3];  // per face: inverse of the matrix with columns A, B, C
};

__constant__ IcoTables c_ico;

// Home face of every corner and edge (the lowest-numbered face containing
// it), used to give every vertex one (face, i, j) grid position for tiling.
struct IcoHome {
    int corner_face[12], corner_which[12];        // which: 0 = A, 1 = B, 2 = C of that face
    int edge_face[30], edge_side[30], edge_fwd[30];  // side: 0 = AB, 1 = AC, 2 = BC
};

__constant__ IcoHome c_home;

// Point = normalise(w0*A + w1*B + w2*C), sums in the written order, no FMA.
// GB300's two binary64 operations per SM and cycle bound the vertices: the
// integer multiples and the squares come from integer products, the norm and
// the quotients from one binary64 operation each (nx_f64.cuh), which leaves 12
// a vertex of about 58.  Measured (GB300, 4,900,002 vertices): 506 -> 173 us;
// with the squares, 10,000,002 vertices 363 -> 304.
__device__ __forceinline__ void normalise(const double *p, double *out)
{
    const double r = nxf::sqrt(
        __dadd_rn(__dadd_rn(nxf::square(p[0]), nxf::square(p[1])), nxf::square(p[2])));
    const nxf::Recip R = nxf::recip(r);
    for (int c = 0; c < 3; ++c) out[c] = nxf::div(p[c], R);
}

__device__ __forceinline__ void blend3(const double *A, const double *B, const double *C, int w0, int w1, int w2,
                                       double *out)
{
    double p[3];
    for (int c = 0; c < 3; ++c)
        p[c] = __dadd_rn(__dadd_rn(nxf::times(A[c], w0), nxf::times(B[c], w1)), nxf::times(C[c], w2));
    normalise(p, out);
}

__device__ __forceinline__ void blend2(const double *A, const double *B, int w0, int w1, double *out)
{
    double p[3];
    for (int c = 0; c < 3; ++c) p[c] = __dadd_rn(nxf::times(A[c], w0), nxf::times(B[c], w1));
    normalise(p, out);
}

// Face-interior offset q -> (face, i, j): rows i = 1..k-2 hold k-1-i points.
__device__ __forceinline__ void interior_fij(int64_t q, int k, int &f, int &i, int &j)
{
    const int64_t npf = (int64_t)(k - 1) * (k - 2) / 2;
    f = (int)(q / npf);
    const int64_t off = q - (int64_t)f * npf;
    // binary32 estimate of the row; the loops below make it exact
    const float kk = (float)k;
    const float disc = (2.0f * kk - 3.0f) * (2.0f * kk - 3.0f) - 8.0f * (float)off;
    int ii = (int)floorf(((2.0f * kk - 3.0f) - sqrtf(fmaxf(disc, 0.0f))) * 0.5f) + 1;
    if (ii < 1) ii = 1;
    if (ii > k - 2) ii = k - 2;
    auto start = [&](int a) -> int64_t { return (int64_t)(a - 1) * (k - 1) - (int64_t)(a - 1) * a / 2; };
    while (ii > 1 && start(ii) > off) --ii;
    while (ii < k - 2 && start(ii + 1) <= off) ++ii;
    i = ii;
    j = (int)(off - start(ii)) + 1;
}

__global__ void ico_vertices_kernel(int k, int64_t nv, double *__restrict__ xyz)
{
    const int64_t ne = (int64_t)30 * (k - 1);
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
        double out[3];
        if (v < 12) {
            for (int c = 0; c < 3; ++c) out[c] = c_ico.corner[v][c];
        } else if (v < 12 + ne) {
            int64_t q = v - 12;
            int e = (int)(q / (k - 1));
            int t = (int)(q - (int64_t)e * (k - 1)) + 1;
            blend2(c_ico.corner[c_ico.edge[e][0]], c_ico.corner[c_ico.edge[e][1]], k - t, t, out);
        } else {
            int f, i, j;
            interior_fij(v - 12 - ne, k, f, i, j);
            const int *F = c_ico.face[f];
            blend3(c_ico.corner[F[0]], c_ico.corner[F[1]], c_ico.corner[F[2]], k - i - j, i, j, out);
        }
        xyz[3 * v] = out[0];
        xyz[3 * v + 1] = out[1];
        xyz[3 * v + 2] = out[2];
    }
}

// Vertex id of face point (i, j); layout in icosphere.py.
__device__ __forceinline__ int32_t face_vid(int f, int i, int j, int k)
{
    const int *F = c_ico.face[f];
    if (i == 0 && j == 0) return F[0];
    if (i == k && j == 0) return F[1];
    if (i == 0 && j == k) return F[2];
    int side, pos;
    if (j == 0) { side = 0; pos = i; }
    else if (i == 0) { side = 1; pos = j; }
    else if (i + j == k) { side = 2; pos = j; }
    else {
        int64_t npf = (int64_t)(k - 1) * (k - 2) / 2;
        int64_t off = (int64_t)(i - 1) * (k - 1) - (int64_t)(i - 1) * i / 2 + (j - 1);
        return (int32_t)(12 + (int64_t)30 * (k - 1) + (int64_t)f * npf + off);
    }
    int e = c_ico.fedge[f][side][0];
    int t = c_ico.fedge[f][side][1] ? pos : k - pos;
    return (int32_t)(12 + (int64_t)e * (k - 1) + t - 1);
}

// Triangles of one face row-pair: triangle index within the face for
// (i, j): rows before i hold sum_{i'<i} (2(k-i') - 1) = i(2k - i) triangles.
__global__ void ico_triangles_kernel(int k, int64_t nt, int32_t *__restrict__ tris)
{
    const int64_t per_face = (int64_t)k * k;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += (int64_t)gridDim.x * blockDim.x) {
        int f = (int)(t / per_face);
        int64_t q = t - (int64_t)f * per_face;
        // find row i with i(2k-i) <= q < (i+1)(2k-i-1)
        double kk = (double)k;
        int i = (int)floor(kk - sqrt(kk * kk - (double)q));
        if (i < 0) i = 0;
        if (i > k - 1) i = k - 1;
        while (i > 0 && (int64_t)i * (2 * k - i) > q) --i;
        while (i < k - 1 && (int64_t)(i + 1) * (2 * k - i - 1) <= q) ++i;
        int64_t r = q - (int64_t)i * (2 * k - i);   // 0 .. 2(k-i)-2
        int j = (int)(r / 2);
        bool down = (r & 1) != 0;
        int32_t a, b, c;
        if (!down) {
            a = face_vid(f, i, j, k); b = face_vid(f, i + 1, j, k); c = face_vid(f, i, j + 1, k);
        } else {
            a = face_vid(f, i + 1, j, k); b = face_vid(f, i + 1, j + 1, k); c = face_vid(f, i, j + 1, k);
        }
        tris[3 * t] = a;
        tris[3 * t + 1] = b;
        tris[3 * t + 2] = c;
    }
}

// build_adjacency (util.py:591-613): every triangle t appends t1 to t0's row,
// t2 to t1's, t0 to t2's, in triangle order.  Records (t, neighbour) are
// gathered with an atomic slot per vertex, then each row is ordered by t.
__global__ void adj_records_kernel(const int32_t *__restrict__ tris, int64_t nt, int64_t nv,
                                   unsigned *__restrict__ cnt, unsigned long long *__restrict__ rec,
                                   int *__restrict__ err)
{
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += (int64_t)gridDim.x * blockDim.x) {
        for (int e = 0; e < 3; ++e) {
            int32_t a = tris[3 * t + e], b = tris[3 * t + (e + 1) % 3];
            if ((uint64_t)(uint32_t)a >= (uint64_t)nv || (uint64_t)(uint32_t)b >= (uint64_t)nv) {
                atomicOr(err, 1);
                continue;
            }
            unsigned s = atomicAdd(&cnt[a], 1u);
            if (s >= 6) {
                atomicOr(err, 2);
                continue;
            }
            rec[6 * (int64_t)a + s] = ((unsigned long long)t << 32) | (uint32_t)b;
        }
    }
}

__device__ __forceinline__ void cswap(unsigned long long &a, unsigned long long &b)
{
    const unsigned long long lo = a < b ? a : b, hi = a < b ? b : a;
    a = lo;
    b = hi;
}

__global__ void adj_rows_kernel(int64_t nv, const unsigned *__restrict__ cnt,
                                const unsigned long long *__restrict__ rec, int32_t *__restrict__ adj)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
        unsigned c = cnt[v];
        if (c > 6) c = 6;
        unsigned long long r[6];
#pragma unroll
        for (int s = 0; s < 6; ++s) r[s] = s < (int)c ? rec[6 * v + s] : ~0ull;
        // by triangle index: a 12-comparator sorting network for 6 keys
        // (fixed indices, so the keys stay in registers)
        cswap(r[0], r[5]); cswap(r[1], r[3]); cswap(r[2], r[4]);
        cswap(r[1], r[2]); cswap(r[3], r[4]);
        cswap(r[0], r[3]); cswap(r[2], r[5]);
        cswap(r[0], r[1]); cswap(r[2], r[3]); cswap(r[4], r[5]);
        cswap(r[1], r[2]); cswap(r[3], r[4]);
#pragma unroll
        for (int s = 0; s < 6; ++s) adj[6 * v + s] = s < (int)c ? (int32_t)(uint32_t)r[s] : -1;
    }
}

__device__ __forceinline__ bool row_has(const int32_t *row, int32_t v)
{
    bool f = false;
    for (int s = 0; s < 6; ++s) f |= row[s] == v;
    return f;
}

// sort_adjacency (util.py:638-662) with next_vert (util.py:623-629): walk the
// neighbours of each vertex into a ring starting at slot 0.  Reads the
// unsorted rows `in`, writes `out` (membership tests do not depend on order).
__global__ void adj_sort_kernel(int64_t nv, const int32_t *__restrict__ in, int32_t *__restrict__ out)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
        int32_t row[6], vis[6];
        for (int s = 0; s < 6; ++s) { row[s] = in[6 * v + s]; vis[s] = -1; }
        int deg = v < 12 ? 5 : 6;
        int32_t pv = (int32_t)v, cur = row[0];
        for (int i = 0; i < deg - 1; ++i) {
            vis[i] = cur;
            int32_t nxt = -1;
            if (cur >= 0 && (int64_t)cur < nv) {
                const int32_t *other = in + 6 * (int64_t)cur;
                int32_t o[6];
                for (int s = 0; s < 6; ++s) o[s] = other[s];
                for (int s = 0; s < 6; ++s) {
                    int32_t c = row[s];
                    if (row_has(o, c) && c != pv) { nxt = c; break; }
                }
            }
            cur = nxt;
            pv = vis[i];
        }
        vis[deg - 1] = cur;
        for (int s = 0; s < 6; ++s) out[6 * v + s] = vis[s];
    }
}

__device__ __forceinline__ double edge_len(const double *xyz, int64_t v, int64_t j)
{
    const double dx = __dsub_rn(xyz[3 * v], xyz[3 * j]);
    const double dy = __dsub_rn(xyz[3 * v + 1], xyz[3 * j + 1]);
    const double dz = __dsub_rn(xyz[3 * v + 2], xyz[3 * j + 2]);
    return nxf::sqrt(__dadd_rn(__dadd_rn(nxf::square(dx), nxf::square(dy)), nxf::square(dz)));
}

__device__ __forceinline__ float2 edge_pair(double d) { return nxf::pair(d); }

// erosion.py:38-40 in binary64 (squares by multiplication), split into a
// pair hi + lo of binary32s: el[2q] = hi, el[2q+1] = lo.  |v_i - v_j| and
// |v_j - v_i| are the same number (the differences only change sign), so
// the binary64 arithmetic -- slow at GB300's binary64 rate -- runs once per
// edge: this pass fills the slots whose neighbour has the larger id (or is
// the vertex itself), edge_mirror_kernel copies them into the reverse slots.
// Each warp takes 64 consecutive slots at a time and gathers the ones that
// need a distance (about half) into consecutive lanes through shared
// memory, so the binary64 instructions run with the warp's lanes busy
// instead of half of them masked off.
__global__ void __launch_bounds__(256) edge_len_kernel(const double *__restrict__ xyz, const int32_t *__restrict__ nbr,
                                                       int64_t nv, float2 *__restrict__ el, int *__restrict__ err)
{
    __shared__ int64_t s_q[8][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t nq = 6 * nv;
    const int64_t wid = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = wid * 64; base < nq; base += nw * 64) {
        int cnt = 0;
        for (int h = 0; h < 2; ++h) {
            const int64_t q = base + 32 * h + lane;
            bool work = false;
            if (q < nq) {
                const int32_t j = nbr[q];
                if (j >= 0 && (int64_t)j < nv) {
                    work = (int64_t)j >= q / 6;                  // j < v: filled by the mirror pass
                } else {
                    if (j != -1 && err) atomicOr(err, 1);
                    el[q] = make_float2(0.0f, 0.0f);
                }
            }
            const unsigned m = __ballot_sync(0xFFFFFFFFu, work);
            if (work) s_q[w][cnt + __popc(m & ((1u << lane) - 1u))] = q;
            cnt += __popc(m);
        }
        __syncwarp();
        for (int r = lane; r < cnt; r += 32) {
            const int64_t q = s_q[w][r];
            el[q] = edge_pair(edge_len(xyz, q / 6, nbr[q]));
        }
        __syncwarp();
    }
}

// Slots whose neighbour j has the smaller id take the pair of j's slot that
// points back; a table that is not symmetric gets the distance computed.
__global__ void edge_mirror_kernel(const double *__restrict__ xyz, const int32_t *__restrict__ nbr, int64_t nv,
                                   float2 *__restrict__ el)
{
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < 6 * nv; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t v = q / 6;
        const int32_t j = nbr[q];
        if (j < 0 || (int64_t)j >= nv || (int64_t)j >= v) continue;
        int m = -1;
        for (int s = 0; s < 6; ++s)
            if (nbr[6 * (int64_t)j + s] == (int32_t)v) { m = s; break; }
        el[q] = m >= 0 ? el[6 * (int64_t)j + m] : edge_pair(edge_len(xyz, v, j));
    }
}

// The icosphere's own neighbour rows, as build_adjacency and sort_adjacency
// make them of its triangles (checked against those), without the triangles:
// a triangle (v, b, c) of v's gives the ring's step b -> c, a row starts at
// the b of v's first triangle and goes round the ring to whichever of that
// b's two neighbours belongs to an earlier triangle.  Inside a face that is
// the same six steps everywhere; vertices of edges and corners collect their
// triangles from the faces around them.  Measured (GB300, 4,900,002
// vertices): 54 us (2.2 TB/s of rows written), against 510 us for the
// triangles, their records, the rows' sorting and the ring walk.
struct Tri {
    int64_t t;
    int32_t b, c;
};

// A vertex on an edge or a corner: its place(s), in face f at (i, j).
__device__ __forceinline__ bool border_place(int64_t v, int k, int f, int &i, int &j)
{
    if (v < 12) {
        const int *F = c_ico.face[f];
        i = F[1] == (int)v ? k : 0;
        j = F[2] == (int)v ? k : 0;
        return F[0] == (int)v || i || j;
    }
    const int e = (int)((v - 12) / (k - 1)), t = (int)((v - 12) - (int64_t)e * (k - 1)) + 1;
    for (int s = 0; s < 3; ++s) {
        if (c_ico.fedge[f][s][0] != e) continue;
        const int pos = c_ico.fedge[f][s][1] ? t : k - t;
        i = s == 0 ? pos : (s == 1 ? 0 : k - pos);
        j = s == 0 ? 0 : pos;
        return true;
    }
    return false;
}

__device__ __noinline__ void border_row(int64_t v, int k, int32_t *__restrict__ row)
{
    Tri tri[6];
    int n = 0;
    for (int f = 0; f < 20; ++f) {
        int i, j;
        if (!border_place(v, k, f, i, j)) continue;
        // the six triangles about (i, j): the upward ones at (i, j), (i-1, j),
        // (i, j-1) with the vertex first, second, third, the downward ones at
        // (i-1, j), (i-1, j-1), (i, j-1) likewise
        for (int q = 0; q < 6; ++q) {
            const bool down = q >= 3;
            const int a = q % 3;
            const int ti = down ? (a == 2 ? i : i - 1) : (a == 1 ? i - 1 : i);
            const int tj = down ? (a == 0 ? j : j - 1) : (a == 2 ? j - 1 : j);
            if (ti < 0 || tj < 0 || ti + tj > k - 1 - (down ? 1 : 0)) continue;
            int32_t id[3];
            if (down) {
                id[0] = face_vid(f, ti + 1, tj, k); id[1] = face_vid(f, ti + 1, tj + 1, k); id[2] = face_vid(f, ti, tj + 1, k);
            } else {
                id[0] = face_vid(f, ti, tj, k); id[1] = face_vid(f, ti + 1, tj, k); id[2] = face_vid(f, ti, tj + 1, k);
            }
            const Tri x = {(int64_t)f * k * k + (int64_t)ti * (2 * k - ti) + 2 * tj + (down ? 1 : 0), id[(a + 1) % 3], id[(a + 2) % 3]};
            int at = n++;
            for (; at > 0 && tri[at - 1].t > x.t; --at) tri[at] = tri[at - 1];
            tri[at] = x;
        }
    }
    // the first triangle's b, then towards its ring neighbour of the earlier
    // triangle: forward (its own c) or backward (the b whose c it is)
    int fwd = n, bwd = n;
    for (int q = 0; q < n; ++q) {
        if (tri[q].b == tri[0].c) fwd = q;
        if (tri[q].c == tri[0].b) bwd = q;
    }
    int32_t cur = tri[0].b;
    for (int s = 0; s < 6; ++s) {
        row[s] = s < n ? cur : -1;
        for (int q = 0; q < n; ++q) {
            if (fwd < bwd ? tri[q].b == cur : tri[q].c == cur) { cur = fwd < bwd ? tri[q].c : tri[q].b; break; }
        }
    }
}

// Ids of a face-interior vertex's six neighbours in slot order, and which of
// them are face-interior themselves (bit per slot).
__device__ __forceinline__ unsigned interior_row(int64_t v, int f, int i, int j, int k, int32_t *row)
{
    const int len = k - 1 - i;                       // points of row i
    row[0] = (int32_t)(v - len - 1);                 // (i-1, j): row i-1 has len + 1 points
    row[1] = (int32_t)(v - len);                     // (i-1, j+1)
    row[2] = (int32_t)(v + 1);                       // (i, j+1)
    row[3] = (int32_t)(v + len);                     // (i+1, j)
    row[4] = (int32_t)(v + len - 1);                 // (i+1, j-1)
    row[5] = (int32_t)(v - 1);                       // (i, j-1)
    if (i > 1 && j > 1 && j < len) return 63u;
    unsigned in = 0;
    const int di[6] = {-1, -1, 0, 1, 1, 0}, dj[6] = {0, 1, 1, 0, -1, -1};
#pragma unroll
    for (int s = 0; s < 6; ++s) {
        const int a = i + di[s], b = j + dj[s];
        if (a >= 1 && b >= 1 && a + b <= k - 1) in |= 1u << s;
        else row[s] = face_vid(f, a, b, k);
    }
    return in;
}

__global__ void __launch_bounds__(256) ico_neighbours_kernel(int k, int64_t nv, int32_t *__restrict__ nbr)
{
    const int64_t inner = 12 + (int64_t)30 * (k - 1);
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
        int32_t row[6];
        if (v < inner) {
            border_row(v, k, row);
        } else {
            int f, i, j;
            interior_fij(v - inner, k, f, i, j);
            interior_row(v, f, i, j, k, row);
        }
        int2 *o = reinterpret_cast<int2 *>(nbr + 6 * v);
        o[0] = make_int2(row[0], row[1]);
        o[1] = make_int2(row[2], row[3]);
        o[2] = make_int2(row[4], row[5]);
    }
}

// Edge length pairs of the icosphere.  Two face-interior neighbours share
// one distance: a vertex computes its slots 2-4, (i, j+1), (i+1, j) and
// (i+1, j-1), and writes each into its own row and the neighbour's opposite
// slot (s + 3) mod 6.  Distances to vertices of edges and corners are
// computed by both sides.  So 6 binary64 operations an edge (the squares come
// from integer products), each edge once, and no search for the reverse slot.
// Measured (GB300, 4,900,002 vertices): ~880 us for the general pair of
// passes, 359 us here, 289 us with the squares from integers, 220 us with the
// three distances side by side and slots 2 and 3 in one store (WIDE: rows
// 16-byte aligned); the binary64 pipe is then busy for 82 % of it.
template <bool WIDE>
__global__ void __launch_bounds__(256) ico_edges_kernel(int k, int64_t nv, const double *__restrict__ xyz,
                                                        const int32_t *__restrict__ nbr, float2 *__restrict__ el,
                                                        int *__restrict__ info)
{
    const int64_t inner = 12 + (int64_t)30 * (k - 1);
    float longest = 0.0f;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
        if (v < inner) {
            for (int s = 0; s < 6; ++s) {
                const int32_t j = nbr[6 * v + s];
                const bool on = j >= 0 && (int64_t)j < nv;
                if (!on && j != -1 && info) atomicOr(info, 1);
                const float2 d = on ? edge_pair(edge_len(xyz, v, j)) : make_float2(0.0f, 0.0f);
                longest = fmaxf(longest, d.x);
                el[6 * v + s] = d;
            }
            continue;
        }
        int f, i, j;
        interior_fij(v - inner, k, f, i, j);
        int32_t row[6];
        const unsigned in = interior_row(v, f, i, j, k, row);
        const float2 d2 = edge_pair(edge_len(xyz, v, row[2])), d3 = edge_pair(edge_len(xyz, v, row[3])),
                     d4 = edge_pair(edge_len(xyz, v, row[4]));
        longest = fmaxf(longest, fmaxf(d2.x, fmaxf(d3.x, d4.x)));
        if (WIDE) {
            *reinterpret_cast<float4 *>(el + 6 * v + 2) = make_float4(d2.x, d2.y, d3.x, d3.y);
        } else {
            el[6 * v + 2] = d2;
            el[6 * v + 3] = d3;
        }
        el[6 * v + 4] = d4;
        if (in & 4u) el[6 * (int64_t)row[2] + 5] = d2;
        if (in & 8u) el[6 * (int64_t)row[3]] = d3;
        if (in & 16u) el[6 * (int64_t)row[4] + 1] = d4;
        if ((in & 35u) != 35u) {
            // (counted here too: a border vertex's row need not name this vertex)
            auto border = [&](int slot) {
                const float2 d = edge_pair(edge_len(xyz, v, row[slot]));
                longest = fmaxf(longest, d.x);
                el[6 * v + slot] = d;
            };
            if (!(in & 1u)) border(0);
            if (!(in & 2u)) border(1);
            if (!(in & 32u)) border(5);
        }
    }
    if (!info) return;
    for (int o = 16; o > 0; o >>= 1) longest = fmaxf(longest, __shfl_xor_sync(0xFFFFFFFFu, longest, o));
    if ((threadIdx.x & 31) == 0) atomicMax(info + 1, __float_as_int(longest));     // (not negative: ordered as integers)
}

// Whether a table's rows of face-interior vertices are the icosphere's own
// (differ: set to 1 where not).
__global__ void __launch_bounds__(256) ico_like_kernel(int k, int64_t nv, const int32_t *__restrict__ nbr, int *__restrict__ differ)
{
    const int64_t inner = 12 + (int64_t)30 * (k - 1);
    bool same = true;
    for (int64_t v = inner + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
        int f, i, j;
        interior_fij(v - inner, k, f, i, j);
        int32_t row[6];
        interior_row(v, f, i, j, k, row);
        const int2 *o = reinterpret_cast<const int2 *>(nbr + 6 * v);
        const int2 a = o[0], b = o[1], c = o[2];
        same = same && a.x == row[0] && a.y == row[1] && b.x == row[2] && b.y == row[3] && c.x == row[4] && c.y == row[5];
    }
    if (!same) *differ = 1;
}

int grid1d(int64_t n, int block = 256)
{
    int64_t g = (n + block - 1) / block;
    int64_t cap = (int64_t)nx::sm_count() * 16;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

bool g_tables_ready[64] = {false};

int upload_tables(const double *corners, const int *faces, const int *fedge, const int *edges)
{
    int dev = 0;
    NX_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && g_tables_ready[dev]) return NX_OK;
    IcoTables t;
    for (int i = 0; i < 12; ++i)
        for (int c = 0; c < 3; ++c) t.corner[i][c] = corners[3 * i + c];
    for (int f = 0; f < 20; ++f)
        for (int c = 0; c < 3; ++c) {
            t.face[f][c] = faces[3 * f + c];
            t.fedge[f][c][0] = fedge[6 * f + 2 * c];
            t.fedge[f][c][1] = fedge[6 * f + 2 * c + 1];
        }
    for (int e = 0; e < 30; ++e) {
        t.edge[e][0] = edges[2 * e];
        t.edge[e][1] = edges[2 * e + 1];
    }
    for (int f = 0; f < 20; ++f) {
        // M = [A B C] (columns); inverse by cofactors
        double m[3][3];
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) m[r][c] = t.corner[t.face[f][c]][r];
        const double c00 = m[1][1] * m[2][2] - m[1][2] * m[2][1], c01 = m[1][2] * m[2][0] - m[1][0] * m[2][2],
                     c02 = m[1][0] * m[2][1] - m[1][1] * m[2][0];
        const double det = m[0][0] * c00 + m[0][1] * c01 + m[0][2] * c02;
        t.inv[f][0][0] = c00 / det;
        t.inv[f][1][0] = c01 / det;
        t.inv[f][2][0] = c02 / det;
        t.inv[f][0][1] = (m[0][2] * m[2][1] - m[0][1] * m[2][2]) / det;
        t.inv[f][1][1] = (m[0][0] * m[2][2] - m[0][2] * m[2][0]) / det;
        t.inv[f][2][1] = (m[0][1] * m[2][0] - m[0][0] * m[2][1]) / det;
        t.inv[f][0][2] = (m[0][1] * m[1][2] - m[0][2] * m[1][1]) / det;
        t.inv[f][1][2] = (m[0][2] * m[1][0] - m[0][0] * m[1][2]) / det;
        t.inv[f][2][2] = (m[0][0] * m[1][1] - m[0][1] * m[1][0]) / det;
    }
    NX_CHECK_CUDA(cudaMemcpyToSymbol(c_ico, &t, sizeof(t)));
    IcoHome h;
    for (int c = 0; c < 12; ++c) {
        h.corner_face[c] = -1;
        for (int f = 0; f < 20 && h.corner_face[c] < 0; ++f)
            for (int w = 0; w < 3; ++w)
                if (t.face[f][w] == c) { h.corner_face[c] = f; h.corner_which[c] = w; break; }
    }
    for (int e = 0; e < 30; ++e) {
        h.edge_face[e] = -1;
        for (int f = 0; f < 20 && h.edge_face[e] < 0; ++f)
            for (int sd = 0; sd < 3; ++sd)
                if (t.fedge[f][sd][0] == e) { h.edge_face[e] = f; h.edge_side[e] = sd; h.edge_fwd[e] = t.fedge[f][sd][1]; break; }
    }
    NX_CHECK_CUDA(cudaMemcpyToSymbol(c_home, &h, sizeof(h)));
    if (dev >= 0 && dev < 64) g_tables_ready[dev] = true;
    return NX_OK;
}

}  // namespace

NX_EXPORT int nx_icosphere_tables(const double *corners, const int32_t *faces, const int32_t *face_edges,
                                  const int32_t *edges)
{
    if (!corners || !faces || !face_edges || !edges) return nx::fail(NX_EINVAL, "nx_icosphere_tables: null pointer");
    int dev = 0;
    NX_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64) g_tables_ready[dev] = false;
    return upload_tables(corners, faces, face_edges, edges);
}

NX_EXPORT int nx_icosphere(int k, double *xyz_dev, int32_t *tris_dev, void *stream)
{
    if (k < 1 || (int64_t)10 * k * k + 2 > 0x7FFFFFFFLL) return nx::fail(NX_EINVAL, "nx_icosphere: bad divisions %d", k);
    int dev = 0;
    NX_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !g_tables_ready[dev])
        return nx::fail(NX_EINVAL, "nx_icosphere: call nx_icosphere_tables first on this device");
    int64_t nv = (int64_t)10 * k * k + 2, nt = (int64_t)20 * k * k;
    cudaStream_t s = (cudaStream_t)stream;
    if (xyz_dev) {
        ico_vertices_kernel<<<grid1d(nv), 256, 0, s>>>(k, nv, xyz_dev);
        NX_CHECK_LAUNCH("ico_vertices_kernel");
        nx::note_launch(1);
    }
    if (tris_dev) {
        ico_triangles_kernel<<<grid1d(nt), 256, 0, s>>>(k, nt, tris_dev);
        NX_CHECK_LAUNCH("ico_triangles_kernel");
        nx::note_launch(1);
    }
    return NX_OK;
}

static int check_rows(int k, const void *nbr, const void *edge, const char *who)
{
    if (k < 2 || (int64_t)10 * k * k + 2 > 0x7FFFFFFFLL) return nx::fail(NX_EINVAL, "%s: bad divisions %d", who, k);
    if (!nbr) return nx::fail(NX_EINVAL, "%s: null pointer", who);
    if (((uintptr_t)nbr & 7u) || ((uintptr_t)edge & 7u)) return nx::fail(NX_EINVAL, "%s: rows must be 8-byte aligned", who);
    int dev = 0;
    NX_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !g_tables_ready[dev])
        return nx::fail(NX_EINVAL, "%s: call nx_icosphere_tables first on this device", who);
    return NX_OK;
}

NX_EXPORT int nx_icosphere_rows(int k, int32_t *nbr_dev, void *stream)
{
    int rc = check_rows(k, nbr_dev, nullptr, "nx_icosphere_rows");
    if (rc) return rc;
    const int64_t nv = (int64_t)10 * k * k + 2;
    ico_neighbours_kernel<<<grid1d(nv), 256, 0, (cudaStream_t)stream>>>(k, nv, nbr_dev);
    NX_CHECK_LAUNCH("ico_neighbours_kernel");
    nx::note_launch(1);
    return NX_OK;
}

NX_EXPORT int nx_icosphere_like(int k, const int32_t *nbr_dev, int *differ_dev, void *stream)
{
    int rc = check_rows(k, nbr_dev, nullptr, "nx_icosphere_like");
    if (rc) return rc;
    if (!differ_dev) return nx::fail(NX_EINVAL, "nx_icosphere_like: null pointer");
    const int64_t nv = (int64_t)10 * k * k + 2;
    ico_like_kernel<<<grid1d(nv), 256, 0, (cudaStream_t)stream>>>(k, nv, nbr_dev, differ_dev);
    NX_CHECK_LAUNCH("ico_like_kernel");
    nx::note_launch(1);
    return NX_OK;
}

NX_EXPORT int nx_icosphere_edges(int k, const double *xyz_dev, const int32_t *nbr_dev, float *edge_dev, int *info_dev,
                                 void *stream)
{
    int rc = check_rows(k, nbr_dev, edge_dev, "nx_icosphere_edges");
    if (rc) return rc;
    if (!xyz_dev || !edge_dev) return nx::fail(NX_EINVAL, "nx_icosphere_edges: null pointer");
    const int64_t nv = (int64_t)10 * k * k + 2;
    if (((uintptr_t)edge_dev & 15u) == 0)
        ico_edges_kernel<true><<<grid1d(nv), 256, 0, (cudaStream_t)stream>>>(k, nv, xyz_dev, nbr_dev, (float2 *)edge_dev, info_dev);
    else
        ico_edges_kernel<false><<<grid1d(nv), 256, 0, (cudaStream_t)stream>>>(k, nv, xyz_dev, nbr_dev, (float2 *)edge_dev, info_dev);
    NX_CHECK_LAUNCH("ico_edges_kernel");
    nx::note_launch(1);
    return NX_OK;
}

NX_EXPORT size_t nx_adjacency_workspace_size(int64_t nv)
{
    return (size_t)nv * (6 * sizeof(unsigned long long) + sizeof(unsigned)) + 256;
}

NX_EXPORT int nx_build_adjacency(const int32_t *tris_dev, int64_t nt, int64_t nv, int32_t *adj_dev, void *workspace,
                                 size_t ws_bytes, int *err_dev, void *stream)
{
    if (nt < 0 || nv < 0 || (nt + 4) / 2 != nv) return nx::fail(NX_EINVAL, "nx_build_adjacency: need nv = (nt+4)/2");
    if (nv == 0) return NX_OK;
    if (!tris_dev || !adj_dev || !workspace || !err_dev) return nx::fail(NX_EINVAL, "nx_build_adjacency: null pointer");
    if (ws_bytes < nx_adjacency_workspace_size(nv)) return nx::fail(NX_EINVAL, "nx_build_adjacency: workspace too small");
    cudaStream_t s = (cudaStream_t)stream;
    unsigned long long *rec = (unsigned long long *)workspace;
    unsigned *cnt = (unsigned *)(rec + 6 * nv);
    NX_CHECK_CUDA(cudaMemsetAsync(cnt, 0, sizeof(unsigned) * (size_t)nv, s));
    adj_records_kernel<<<grid1d(nt), 256, 0, s>>>(tris_dev, nt, nv, cnt, rec, err_dev);
    NX_CHECK_LAUNCH("adj_records_kernel");
    adj_rows_kernel<<<grid1d(nv), 256, 0, s>>>(nv, cnt, rec, adj_dev);
    NX_CHECK_LAUNCH("adj_rows_kernel");
    nx::note_launch(2);
    return NX_OK;
}

NX_EXPORT int nx_sort_adjacency(const int32_t *adj_in_dev, int32_t *adj_out_dev, int64_t nv, void *stream)
{
    if (nv < 0) return nx::fail(NX_EINVAL, "nx_sort_adjacency: nv < 0");
    if (nv == 0) return NX_OK;
    if (!adj_in_dev || !adj_out_dev || adj_in_dev == adj_out_dev)
        return nx::fail(NX_EINVAL, "nx_sort_adjacency: need distinct input and output rows");
    adj_sort_kernel<<<grid1d(nv), 256, 0, (cudaStream_t)stream>>>(nv, adj_in_dev, adj_out_dev);
    NX_CHECK_LAUNCH("adj_sort_kernel");
    nx::note_launch(1);
    return NX_OK;
}

NX_EXPORT int nx_edge_lengths(const double *xyz_dev, const int32_t *nbr_dev, int64_t nv, float *edge_dev,
                              int *err_dev, void *stream)
{
    if (nv < 0) return nx::fail(NX_EINVAL, "nx_edge_lengths: nv < 0");
    if (nv == 0) return NX_OK;
    if (!xyz_dev || !nbr_dev || !edge_dev) return nx::fail(NX_EINVAL, "nx_edge_lengths: null pointer");
    edge_len_kernel<<<grid1d(3 * nv), 256, 0, (cudaStream_t)stream>>>(xyz_dev, nbr_dev, nv, (float2 *)edge_dev, err_dev);
    NX_CHECK_LAUNCH("edge_len_kernel");
    edge_mirror_kernel<<<grid1d(6 * nv), 256, 0, (cudaStream_t)stream>>>(xyz_dev, nbr_dev, nv, (float2 *)edge_dev);
    NX_CHECK_LAUNCH("edge_mirror_kernel");
    nx::note_launch(1);
    nx::note_launch(1);
    return NX_OK;
}


// ---------------------------------------------------------------------------
// Tiling for temporally blocked erosion.
//
// Every vertex gets one grid position (face, i, j) in its home face (corners
// and edge vertices belong to the lowest-numbered face containing them);
// tile (f, i / B, j / B) holds it, and finds it there.  For each tile a
// block collects the R rings of neighbours around it (breadth first over the neighbour
// table, with a shared-memory hash set), numbers them locally (members,
// ring 1, ..., ring R) and stores, for every vertex that a pass can update
// (members and rings 1..R-1), its six neighbours as local indices and its
// six edge lengths.

namespace {

__device__ __forceinline__ void home_of(int64_t v, int k, int &f, int &i, int &j)
{
    const int64_t ne = (int64_t)30 * (k - 1);
    if (v < 12) {
        f = c_home.corner_face[v];
        const int w = c_home.corner_which[v];
        i = w == 1 ? k : 0;
        j = w == 2 ? k : 0;
    } else if (v < 12 + ne) {
        const int64_t q = v - 12;
        const int e = (int)(q / (k - 1));
        const int t = (int)(q - (int64_t)e * (k - 1)) + 1;
        f = c_home.edge_face[e];
        const int pos = c_home.edge_fwd[e] ? t : k - t;
        const int sd = c_home.edge_side[e];
        if (sd == 0) { i = pos; j = 0; }
        else if (sd == 1) { i = 0; j = pos; }
        else { i = k - pos; j = pos; }
    } else {
        interior_fij(v - 12 - ne, k, f, i, j);
    }
}

// Square tile number t -> (face, row, column): row ti of a face holds M + 1 -
// ti tiles, M = k / B.
__device__ __forceinline__ void tile_place(int64_t t, int M, int &f, int &ti, int &tj)
{
    const int64_t tpf = (int64_t)(M + 1) * (M + 2) / 2;
    f = (int)(t / tpf);
    const int q = (int)(t - (int64_t)f * tpf);
    auto start = [&](int a) { return a * (M + 1) - (int)((int64_t)a * (a - 1) / 2); };
    const float b = 2.0f * (float)M + 3.0f;
    ti = (int)((b - sqrtf(fmaxf(b * b - 8.0f * (float)q, 0.0f))) * 0.5f);
    ti = ti < 0 ? 0 : (ti > M ? M : ti);
    while (ti > 0 && start(ti) > q) --ti;
    while (ti < M && start(ti + 1) <= q) ++ti;
    tj = q - start(ti);
}

}  // namespace

// Hexagonal tiles.  On the face grid's lattice (neighbours (+-1, 0),
// (0, +-1), (+1, -1), (-1, +1)) the vertices within graph distance rho of a
// point c, max(|i - ci|, |j - cj|, |i + j - ci - cj|) <= rho, form a hexagon
// of N = 3 rho^2 + 3 rho + 1 points, and these hexagons tile the lattice
// exactly with centres c = m a + n b, a = (2 rho + 1, -rho), b = (rho,
// rho + 1) (det [a b] = N).  A hexagon is the set with the fewest vertices
// within R of it for its size, so hexagonal tiles carry fewer halo vertices
// per member than squares.  Per face the tiles are the (m, n) whose hexagon
// meets the face triangle {i, j >= 0, i + j <= k}; for each m these form one
// run of n, numbered row by row.
constexpr int HEX_ROWS_MAX = 1024;
struct HexRows {
    int rho, N;
    int m0, nrows;          // rows m = m0 .. m0 + nrows - 1
    int per_face;           // tiles per face
    int nlo[HEX_ROWS_MAX];  // first n of each row
    int base[HEX_ROWS_MAX + 1];   // local index of each row's first tile; base[nrows] = per_face
};

static inline int hex_points(int r) { return 3 * r * r + 3 * r + 1; }

// Whether the hexagon of radius rho centred at (ci, cj) holds a point of
// the face triangle: integer i, j with |i - ci|, |j - cj|, |i + j - ci - cj|
// <= rho and i, j >= 0, i + j <= k.  Every sum between ilo + jlo and
// ihi + jhi is reachable, so the box and the sum band must overlap.
static bool hex_meets_face(long long ci, long long cj, int rho, int k)
{
    const long long ilo = std::max(ci - rho, 0LL), ihi = std::min(ci + rho, (long long)k);
    const long long jlo = std::max(cj - rho, 0LL), jhi = std::min(cj + rho, (long long)k);
    const long long slo = std::max(ci + cj - rho, 0LL), shi = std::min(ci + cj + rho, (long long)k);
    return ilo <= ihi && jlo <= jhi && slo <= shi && std::max(slo, ilo + jlo) <= std::min(shi, ihi + jhi);
}

// Host: the row table of hexagonal tiles of radius rho on divisions k.
static int hex_rows(int k, int rho, HexRows &H)
{
    H.rho = rho;
    H.N = hex_points(rho);
    // lattice coordinates of a grid point: (m, n) = [a b]^-1 (i, j) =
    // ((rho + 1) i - rho j, rho i + (2 rho + 1) j) / N; over the triangle's
    // corners, widened by one centre on every side
    const double N = H.N;
    const double cm[3] = {0.0, (rho + 1.0) * k / N, -(double)rho * k / N};
    const double cn[3] = {0.0, (double)rho * k / N, (2.0 * rho + 1.0) * k / N};
    const int mlo = (int)std::floor(std::min(cm[0], std::min(cm[1], cm[2]))) - 2;
    const int mhi = (int)std::ceil(std::max(cm[0], std::max(cm[1], cm[2]))) + 2;
    const int nlo = (int)std::floor(std::min(cn[0], std::min(cn[1], cn[2]))) - 2;
    const int nhi = (int)std::ceil(std::max(cn[0], std::max(cn[1], cn[2]))) + 2;
    H.nrows = 0;
    H.m0 = 0;
    int total = 0;
    for (int m = mlo; m <= mhi; ++m) {
        int first = INT_MAX, last = INT_MIN;
        for (int n = nlo; n <= nhi; ++n) {
            const long long ci = (long long)m * (2 * rho + 1) + (long long)n * rho;
            const long long cj = -(long long)m * rho + (long long)n * (rho + 1);
            if (hex_meets_face(ci, cj, rho, k)) {
                if (first == INT_MAX) first = n;
                else if (n != last + 1)
                    return nx::fail(NX_EINVAL, "hexagonal tiling: row %d of divisions %d is not one run", m, k);
                last = n;
            }
        }
        if (first == INT_MAX) {
            if (H.nrows > 0) break;      // past the last row
            continue;
        }
        if (H.nrows == 0) H.m0 = m;
        else if (m != H.m0 + H.nrows)
            return nx::fail(NX_EINVAL, "hexagonal tiling: rows of divisions %d are not contiguous", k);
        if (H.nrows >= HEX_ROWS_MAX)
            return nx::fail(NX_EINVAL, "hexagonal tiling: more than %d rows (divisions %d, radius %d)", HEX_ROWS_MAX, k, rho);
        H.nlo[H.nrows] = first;
        H.base[H.nrows] = total;
        total += last - first + 1;
        ++H.nrows;
    }
    H.base[H.nrows] = total;
    H.per_face = total;
    return total > 0 ? NX_OK : nx::fail(NX_EINVAL, "hexagonal tiling: no tiles");
}

namespace {

__device__ __forceinline__ int floor_div(int a, int b) { return a >= 0 ? a / b : -((b - 1 - a) / b); }

// Tile of a grid point: the centre within rho is one of the four lattice
// points at the floors of its lattice coordinates and their +1 neighbours.
__device__ __forceinline__ int64_t hex_tile_of(int f, int i, int j, const HexRows &H)
{
    const int rho = H.rho;
    const int m0 = floor_div((rho + 1) * i - rho * j, H.N), n0 = floor_div(rho * i + (2 * rho + 1) * j, H.N);
    for (int q = 0; q < 4; ++q) {
        const int m = m0 + (q & 1), n = n0 + (q >> 1);
        const int di = i - (m * (2 * rho + 1) + n * rho), dj = j - (-m * rho + n * (rho + 1));
        if (max(abs(di), max(abs(dj), abs(di + dj))) <= rho) {
            const int r = m - H.m0;
            if (r < 0 || r >= H.nrows) return -1;
            const int loc = H.base[r] + n - H.nlo[r];
            if (n < H.nlo[r] || loc >= H.base[r + 1]) return -1;
            return (int64_t)f * H.per_face + loc;
        }
    }
    return -1;
}

__global__ void tile_assign_hex_kernel(int k, int64_t nv, int R, int nmax, int32_t *__restrict__ counts,
                                       int32_t *__restrict__ ids, int *__restrict__ err,
                                       const __grid_constant__ HexRows H)
{
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += (int64_t)gridDim.x * blockDim.x) {
        int f, i, j;
        home_of(v, k, f, i, j);
        const int64_t t = hex_tile_of(f, i, j, H);
        if (t < 0) {
            atomicOr(err, 2);
            continue;
        }
        const int pos = atomicAdd(&counts[t * (R + 1)], 1);
        if (pos < nmax) ids[t * nmax + pos] = (int32_t)v;
        else atomicOr(err, 1);
    }
}

// Per-tile hash set of vertex ids in shared memory: 2^bits entries, the
// smallest power of two with at least twice the tile's local bound (load
// factor <= 1/2), linear probing.
struct HashSet {
    int bits;
    uint32_t mask;
};

__host__ __device__ __forceinline__ int hash_bits_for(int nmax)
{
    int b = 6;
    while ((1 << b) < 2 * nmax) ++b;
    return b;
}

__device__ __forceinline__ uint32_t hslot(const HashSet &H, int32_t v)
{
    return ((uint32_t)v * 2654435761u) >> (32 - H.bits);
}

// Insert v (bounded probing); returns its local index, assigning the next
// one if v is new.  -1 if the set or the list is full.
__device__ __forceinline__ int hinsert(const HashSet &H, int32_t *key, int32_t *val, int32_t *list, int *cnt, int nmax,
                                       int32_t v)
{
    uint32_t h = hslot(H, v);
    for (uint32_t probe = 0; probe <= H.mask; ++probe) {
        // (most are there already: a read costs less than an exchange)
        const int32_t seen = *reinterpret_cast<volatile int32_t *>(key + h);
        const int32_t old = seen == -1 ? atomicCAS(&key[h], -1, v) : seen;
        if (old == -1) {
            const int idx = atomicAdd(cnt, 1);
            if (idx >= nmax) { val[h] = -1; return -1; }
            list[idx] = v;
            val[h] = idx;
            return idx;
        }
        if (old == v) return 0;       // present (its index is read after a barrier)
        h = (h + 1) & H.mask;
    }
    return -1;
}

__device__ __forceinline__ int hfind(const HashSet &H, const int32_t *key, const int32_t *val, int32_t v)
{
    uint32_t h = hslot(H, v);
    for (uint32_t probe = 0; probe <= H.mask; ++probe) {
        const int32_t kk = key[h];
        if (kk == v) return val[h];
        if (kk == -1) return -1;
        h = (h + 1) & H.mask;
    }
    return -1;
}

// Graph distance, on a face's grid, of a point from the B x B square that
// starts at its origin: steps (+1, -1) and (-1, +1) mend both coordinates at
// once where they lie off on opposite sides.
__device__ __forceinline__ int square_distance(int i, int j, int B)
{
    const int di = i < 0 ? i : (i >= B ? i - B + 1 : 0), dj = j < 0 ? j : (j >= B ? j - B + 1 : 0);
    return (di < 0) == (dj < 0) || di == 0 || dj == 0 ? abs(di) + abs(dj) : max(abs(di), abs(dj));
}

// A square tile that lies, with its R rings, inside one face: rings, orders
// and neighbours follow from the grid, without a search.  The points of the
// widened square are ranked within their ring by counting (row by row is the
// order of the ids), and a map of the square gives the local neighbours.
// About two thirds of divisions 800's tiles, four fifths of 2000's.  A
// neighbour table that differs from the icosphere's in these rows is left to
// the search (false).  Measured (GB300, divisions 700, 5,060 tiles of side 32
// with 4 rings): the build 640 -> 290 us with the members found by the tiles
// themselves.  Bound by issue (69 % of the slots) and by the searched tiles
// (about a third); rows by reciprocal, keys read before they are exchanged
// and slots stored two at a time 329 -> 289 us on a slower machine, divisions
// 1,000 585 -> 508.
__device__ bool inner_tile(int k, int B, int R, int f, int i0, int j0, int nmax, const int32_t *__restrict__ nbr,
                           const float *__restrict__ edge, int32_t *__restrict__ tc, int32_t *__restrict__ tid,
                           uint32_t *__restrict__ lnbr, float4 *__restrict__ ledge, int *__restrict__ err, int32_t *sh)
{
    const int W = B + 2 * R, np = W * W, nchunk = (np + 31) / 32;
    int32_t *list = sh;                                                    // ids by local index
    uint16_t *at = reinterpret_cast<uint16_t *>(list + nmax);              // grid position by local index
    uint16_t *map = at + ((nmax + 1) & ~1);                                // local index by grid position
    int32_t *cnt = reinterpret_cast<int32_t *>(map + ((np + 1) & ~1));     // [ring][chunk]
    __shared__ int s_base[10];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t inv = 0xFFFFFFFFu / (uint32_t)W + 1u;
    auto row_of = [&](int p) { return (int)__umulhi((uint32_t)p, inv); };     // p / W (p < 2^16)
    auto ring_of = [&](int p) {
        const int a = row_of(p), d = p < np ? square_distance(a - R, p - a * W - R, B) : 99;
        return d <= R ? d : 99;
    };
    const int64_t inner = 12 + (int64_t)30 * (k - 1) + (int64_t)f * ((int64_t)(k - 1) * (k - 2) / 2);
    auto id_of = [&](int p) {
        const int a = row_of(p);
        const int64_t i = i0 + a - R, j = j0 + p - a * W - R;
        return (int32_t)(inner + (i - 1) * (k - 1) - (i - 1) * i / 2 + j - 1);
    };
    bool same = true;
    for (int p = threadIdx.x; p < np; p += blockDim.x) {
        if (ring_of(p) >= R) continue;
        const int32_t v = id_of(p), len = k - 1 - (i0 + row_of(p) - R);
        const int2 *row = reinterpret_cast<const int2 *>(nbr + 6 * (int64_t)v);
        const int2 a = row[0], b = row[1], c = row[2];
        same = same && a.x == v - len - 1 && a.y == v - len && b.x == v + 1 && b.y == v + len && c.x == v + len - 1 && c.y == v - 1;
    }
    if (!__syncthreads_and(same)) return false;
    for (int c = warp; c < nchunk; c += nw) {
        const int d = ring_of(32 * c + lane);
        for (int r = 0; r <= R; ++r) {
            const unsigned m = __ballot_sync(0xFFFFFFFFu, d == r);
            if (lane == 0) cnt[r * nchunk + c] = __popc(m);
        }
    }
    __syncthreads();
    // exclusive prefix over the chunks, a warp per ring
    for (int r = warp; r <= R; r += nw) {
        int run = 0;
        for (int c0 = 0; c0 < nchunk; c0 += 32) {
            const int c = c0 + lane, v = c < nchunk ? cnt[r * nchunk + c] : 0;
            int inc = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += u;
            }
            if (c < nchunk) cnt[r * nchunk + c] = run + inc - v;
            run += __shfl_sync(0xFFFFFFFFu, inc, 31);
        }
        if (lane == 0) s_base[r + 1] = run;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        s_base[0] = 0;
        for (int r = 0; r <= R; ++r) {
            tc[r] = s_base[r + 1];
            s_base[r + 1] += s_base[r];
        }
        atomicMax(&err[1], s_base[R + 1]);
        atomicMax(&err[2], s_base[R]);
    }
    __syncthreads();
    for (int c = warp; c < nchunk; c += nw) {
        const int p = 32 * c + lane, d = ring_of(p);
        for (int r = 0; r <= R; ++r) {
            const unsigned m = __ballot_sync(0xFFFFFFFFu, d == r);
            if (d != r) continue;
            const int l = s_base[r] + cnt[r * nchunk + c] + __popc(m & ((1u << lane) - 1u));
            const int32_t v = id_of(p);
            list[l] = v;
            at[l] = (uint16_t)p;
            map[p] = (uint16_t)l;
            tid[l] = v;
        }
    }
    __syncthreads();
    const int C0 = s_base[R];                  // members and rings below R
    for (int w = threadIdx.x; w < 3 * C0; w += blockDim.x) {
        const int l = w / 3, q = w - 3 * l, p = at[l];
        // slots 2q, 2q + 1 of (-1, 0), (-1, 1), (0, 1), (1, 0), (1, -1), (0, -1)
        const int s0 = q == 0 ? -W : (q == 1 ? 1 : W - 1), s1 = q == 0 ? 1 - W : (q == 1 ? W : -1);
        lnbr[tile_unit(l) + 32 * q] = (uint32_t)map[p + s0] | ((uint32_t)map[p + s1] << 16);
        const float4 *e = reinterpret_cast<const float4 *>(edge) + 3 * (int64_t)list[l];
        ledge[tile_unit(l) + 32 * q] = e[q];
    }
    return true;
}

// squares: tile t is (face, row, column) of the face grids' B x B squares,
// its members found here; otherwise (B = 0) the members come in ids.
__global__ void __launch_bounds__(512) tile_rings_kernel(int k, int B, bool aligned, const int32_t *__restrict__ nbr,
                                                         const float *__restrict__ edge, int64_t nv, int R, int nmax, int cmax, int32_t *__restrict__ counts,
                                                         int32_t *__restrict__ ids, uint16_t *__restrict__ lnbr,
                                                         float *__restrict__ ledge, int *__restrict__ err)
{
    extern __shared__ int32_t sh[];
    HashSet H;
    H.bits = hash_bits_for(nmax);
    H.mask = (1u << H.bits) - 1u;
    const int hcap = 1 << H.bits;
    int32_t *key = sh;                      // hcap
    int32_t *val = key + hcap;              // hcap
    int32_t *list = val + hcap;             // local vertices; list + nmax: sort scratch
    __shared__ int s_cnt, s_bad;
    __shared__ int s_ring[16];
    const int64_t tile = blockIdx.x;
    int32_t *tc = counts + tile * (R + 1);
    int32_t *tid = ids + tile * nmax;
    int T;
    if (B > 0) {
        int f, i0, j0;
        tile_place(tile, k / B, f, i0, j0);
        i0 *= B;
        j0 *= B;
        if (aligned && i0 > R && j0 > R && i0 + j0 + 2 * (B - 1) + R <= k - 1 &&
            inner_tile(k, B, R, f, i0, j0, nmax, nbr, edge, tc, tid, reinterpret_cast<uint32_t *>(lnbr) + tile * cmax * 3,
                       reinterpret_cast<float4 *>(ledge) + tile * cmax * 3, err, sh))
            return;
        // members in ascending id order: the square's vertices on edges and
        // corners (of this home face), ranked, then the interior ones row by
        // row
        __shared__ int s_edge, s_in;
        if (threadIdx.x == 0) { s_edge = 0; s_cnt = 0; s_bad = 0; }
        for (int q = threadIdx.x; q < hcap; q += blockDim.x) key[q] = -1;
        __syncthreads();
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
        const int nchunk = (B * B + 31) / 32;
        const int64_t base = 12 + (int64_t)30 * (k - 1) + (int64_t)f * ((int64_t)(k - 1) * (k - 2) / 2);
        int32_t *border = list + nmax;           // scratch
        for (int c = warp; c < nchunk; c += nw) {
            const int p = 32 * c + lane, i = i0 + p / B, j = j0 + p % B;
            const bool on = p < B * B && i + j <= k, in = on && i >= 1 && j >= 1 && i + j <= k - 1;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, in);
            if (lane == 0) val[c] = __popc(m);
            if (on && !in) {
                const int32_t v = face_vid(f, i, j, k);
                int f2, i2, j2;
                home_of(v, k, f2, i2, j2);
                if (f2 == f && i2 == i && j2 == j) border[atomicAdd(&s_edge, 1)] = v;
            }
        }
        __syncthreads();
        const int ne = s_edge;
        if (threadIdx.x == 0) {
            int run = ne;
            for (int c = 0; c < nchunk; ++c) { const int n = val[c]; val[c] = run; run += n; }
            s_in = run;
        }
        for (int q = threadIdx.x; q < ne; q += blockDim.x) {
            const int32_t v = border[q];
            int rank = 0;
            for (int x = 0; x < ne; ++x) rank += border[x] < v ? 1 : 0;
            list[rank] = v;
        }
        __syncthreads();
        for (int c = warp; c < nchunk; c += nw) {
            const int p = 32 * c + lane, i = i0 + p / B, j = j0 + p % B;
            const bool in = p < B * B && i >= 1 && j >= 1 && i + j <= k - 1;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, in);
            if (in) list[val[c] + __popc(m & ((1u << lane) - 1u))] = (int32_t)(base + (int64_t)(i - 1) * (k - 1) - (int64_t)(i - 1) * i / 2 + j - 1);
        }
        T = s_in;
        __syncthreads();
    } else {
        T = tc[0];
        if (T > nmax) T = nmax;
        int P2 = 1;
        while (P2 < T) P2 <<= 1;
        for (int q = threadIdx.x; q < hcap; q += blockDim.x) key[q] = -1;
        for (int q = threadIdx.x; q < P2; q += blockDim.x) list[q] = q < T ? tid[q] : 0x7FFFFFFF;
        if (threadIdx.x == 0) { s_cnt = 0; s_bad = 0; }
        __syncthreads();
        // members in ascending id order (row segments -> coalesced accesses)
        for (int size = 2; size <= P2; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int q = threadIdx.x; q < P2; q += blockDim.x) {
                    const int o = q ^ stride;
                    if (o > q) {
                        const bool up = (q & size) == 0;
                        const int32_t a = list[q], b = list[o];
                        if ((a > b) == up) { list[q] = b; list[o] = a; }
                    }
                }
                __syncthreads();
            }
    }
    for (int q = threadIdx.x; q < T; q += blockDim.x) {
        // members take local indices 0..T-1 in sorted order
        const int32_t v = list[q];
        uint32_t h = hslot(H, v);
        for (uint32_t probe = 0; probe <= H.mask; ++probe) {
            if (atomicCAS(&key[h], -1, v) == -1) { val[h] = q; break; }
            h = (h + 1) & H.mask;
        }
    }
    if (threadIdx.x == 0) s_cnt = T;
    __syncthreads();
    int beg = 0, end = T;
    for (int r = 1; r <= R; ++r) {
        const int nwork = (end - beg) * 6;
        // two slots per thread per round, both reads issued first (the
        // ring's order is fixed by the sort below, not by insertion order)
        for (int w0 = threadIdx.x; w0 < nwork; w0 += 2 * blockDim.x) {
            int32_t jv[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int w = w0 + u * blockDim.x;
                jv[u] = w < nwork ? nbr[6 * (int64_t)list[beg + w / 6] + (w % 6)] : -1;
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int32_t j = jv[u];
                if (j < 0) continue;
                if ((int64_t)j >= nv) { s_bad = 1; continue; }
                if (hinsert(H, key, val, list, &s_cnt, nmax, j) < 0) s_bad = 1;
            }
        }
        __syncthreads();
        beg = end;
        end = min(s_cnt, nmax);
        if (threadIdx.x == 0) s_ring[r] = end - beg;
        __syncthreads();
    }
    const int NL = end;
    // each ring in ascending id order too (neighbouring vertices get nearby
    // local indices: fewer shared-memory bank conflicts in the erosion pass),
    // then the hash values follow the new positions
    {
        int32_t *scr = list + nmax;        // scratch of nmax entries
        int rb = T;
        for (int r = 1; r <= R; ++r) {
            const int re = rb + s_ring[r];
            const int ln = re - rb;
            // rank sort (the ids of a ring are distinct): each entry's
            // position is the number of smaller ids, read as broadcasts
            for (int q = threadIdx.x; q < ln; q += blockDim.x) {
                const int32_t v = list[rb + q];
                int rank = 0;
                for (int x = 0; x < ln; ++x) rank += list[rb + x] < v ? 1 : 0;
                scr[rank] = v;
            }
            __syncthreads();
            for (int q = threadIdx.x; q < ln; q += blockDim.x) {
                const int32_t v = scr[q];
                list[rb + q] = v;
                uint32_t h = hslot(H, v);
                for (uint32_t probe = 0; probe <= H.mask; ++probe) {
                    if (key[h] == v) { val[h] = rb + q; break; }
                    h = (h + 1) & H.mask;
                }
            }
            __syncthreads();
            rb = re;
        }
    }
    int C0 = T;
    for (int r = 1; r < R; ++r) C0 += s_ring[r];
    if (C0 > cmax) { if (threadIdx.x == 0) s_bad = 1; C0 = cmax; }
    __syncthreads();
    for (int q = threadIdx.x; q < NL; q += blockDim.x) tid[q] = list[q];
    // a missing neighbour (-1, pentagon slot) points at the vertex itself: the
    // erosion update then sees equal heights and adds nothing
    auto local = [&](int q, int32_t j) {
        if (j < 0) return q;
        const int loc = hfind(H, key, val, j);
        if (loc < 0) { s_bad = 1; return q; }
        return loc;
    };
    if (aligned) {
        // two slots at a time, the global reads of two rounds issued before any
        // hash probe
        uint32_t *nb = reinterpret_cast<uint32_t *>(lnbr) + tile * 3 * cmax;
        float4 *ed = reinterpret_cast<float4 *>(ledge) + tile * 3 * cmax;
        constexpr int U = 2;
        for (int w0 = threadIdx.x; w0 < 3 * C0; w0 += U * blockDim.x) {
            int2 jv[U];
            float4 ev[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int w = w0 + u * blockDim.x;
                if (w < 3 * C0) {
                    const int64_t g = 3 * (int64_t)list[w / 3] + w % 3;
                    jv[u] = reinterpret_cast<const int2 *>(nbr)[g];
                    ev[u] = reinterpret_cast<const float4 *>(edge)[g];
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int w = w0 + u * blockDim.x;
                if (w < 3 * C0) {
                    const int q = w / 3, at = tile_unit(q) + 32 * (w % 3);
                    nb[at] = (uint32_t)local(q, jv[u].x) | ((uint32_t)local(q, jv[u].y) << 16);
                    ed[at] = ev[u];
                }
            }
        }
    } else {
        for (int w = threadIdx.x; w < 6 * C0; w += blockDim.x) {
            const int q = w / 6, sl = w % 6;
            const int64_t g = 6 * (int64_t)list[q] + sl, at = 2 * (tile * 3 * cmax + tile_unit(q) + 32 * (sl >> 1)) + (sl & 1);
            lnbr[at] = (uint16_t)local(q, nbr[g]);
            reinterpret_cast<float2 *>(ledge)[at] = reinterpret_cast<const float2 *>(edge)[g];
        }
    }
    if (threadIdx.x == 0) {
        tc[0] = T;
        for (int r = 1; r <= R; ++r) tc[r] = s_ring[r];
        atomicMax(&err[1], NL);
        atomicMax(&err[2], C0);
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_bad) atomicOr(err, 2);
}

}  // namespace

static_assert(sizeof(nx_tiling) == 48, "tiling descriptor layout");

// Local and updatable capacities of tiles whose members lie within graph
// distance `reach` of a point or square (see nx_tiling_shape).
static int tile_caps(int64_t nm, int64_t cm, int32_t *nmax, int32_t *cmax)
{
    cm = (cm + 31) & ~(int64_t)31;                   // whole groups of rows (tile_unit)
    if (nm > 4096) return nx::fail(NX_EINVAL, "nx_tiling_shape: tile too large (%lld local vertices)", (long long)nm);
    *nmax = (int32_t)nm;
    *cmax = (int32_t)cm;
    return NX_OK;
}

NX_EXPORT int nx_tiling_shape(int k, int tile, int rings, int32_t *ntiles, int32_t *nmax, int32_t *cmax)
{
    if (k < 1 || rings < 1 || rings > 8 || !ntiles || !nmax || !cmax || (tile >= 0 && tile < 2) || tile < -64 ||
        tile == -1)
        return nx::fail(NX_EINVAL, "nx_tiling_shape: bad arguments");
    if (tile < 0) {
        // hexagons of radius rho: the vertices within R of a tile lie within
        // rho + R of its centre (on the flat lattice of a face and across an
        // edge onto the next face; around the twelve five-neighbour corners
        // the count only drops), at most hex_points(rho + R); 6(rho + R) of
        // slack as for squares
        const int rho = -tile;
        HexRows H;
        int rc = hex_rows(k, rho, H);
        if (rc) return rc;
        const int64_t nt = (int64_t)20 * H.per_face;
        if (nt > 0x7FFFFFFF) return nx::fail(NX_EINVAL, "nx_tiling_shape: too many tiles");
        rc = tile_caps(hex_points(rho + rings) + 6 * (rho + rings), hex_points(rho + rings - 1) + 6 * (rho + rings - 1),
                       nmax, cmax);
        if (rc) return rc;
        *ntiles = (int32_t)nt;
        return NX_OK;
    }
    const int M = k / tile;
    const int64_t nt = (int64_t)20 * (M + 1) * (M + 2) / 2;
    // A tile holds at most B x B members of one face grid.  On the lattice
    // of the face grids (six neighbours: (+-1, 0), (0, +-1), (+1, -1),
    // (-1, +1)) the vertices within graph distance R of a B x B square form
    // the square widened by R on every side less two corners, fewer than
    // (B + 2R)^2; at the twelve five-neighbour corners the count only drops.
    // The bounds keep 4(B + 2R) of slack (overflow is still detected and
    // reported by the build); the updatable set (rings below R) uses R - 1.
    const int64_t B = tile, D = B + 2 * (int64_t)rings, Dc = D - 2;
    if (nt > 0x7FFFFFFF) return nx::fail(NX_EINVAL, "nx_tiling_shape: too many tiles");
    const int rc = tile_caps(D * D + 4 * D, Dc * Dc + 4 * Dc, nmax, cmax);
    if (rc) return rc;
    *ntiles = (int32_t)nt;
    return NX_OK;
}

NX_EXPORT int nx_tiling_build(int k, int tile, int rings, const int32_t *nbr_dev, const float *edge_dev,
                              int32_t *counts_dev, int32_t *ids_dev, uint16_t *lnbr_dev, float *ledge_dev, int *err_dev,
                              void *stream)
{
    int32_t nt = 0, nmax = 0, cmax = 0;
    int rc = nx_tiling_shape(k, tile, rings, &nt, &nmax, &cmax);
    if (rc) return rc;
    if (!nbr_dev || !edge_dev || !counts_dev || !ids_dev || !lnbr_dev || !ledge_dev || !err_dev)
        return nx::fail(NX_EINVAL, "nx_tiling_build: null pointer");
    int dev = 0;
    NX_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !g_tables_ready[dev]) return nx::fail(NX_EINVAL, "nx_tiling_build: call nx_icosphere_tables first");
    const int64_t nv = (int64_t)10 * k * k + 2;
    cudaStream_t s = (cudaStream_t)stream;
    if (tile < 0) {
        HexRows H;
        rc = hex_rows(k, -tile, H);
        if (rc) return rc;
        NX_CHECK_CUDA(cudaMemsetAsync(counts_dev, 0, sizeof(int32_t) * (size_t)nt * (rings + 1), s));
        tile_assign_hex_kernel<<<grid1d(nv), 256, 0, s>>>(k, nv, rings, nmax, counts_dev, ids_dev, err_dev, H);
        NX_CHECK_LAUNCH("tile_assign_hex_kernel");
        nx::note_launch(1);
    }
    int P2 = 1;
    while (P2 < nmax) P2 <<= 1;
    // hash keys + values, the local list (padded for sorting) and a scratch
    const size_t smem = sizeof(int32_t) * (2 * ((size_t)1 << hash_bits_for(nmax)) + 2 * (size_t)P2);
    NX_CHECK_CUDA(cudaFuncSetAttribute(tile_rings_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const bool aligned = (((uintptr_t)edge_dev | (uintptr_t)ledge_dev) & 15u) == 0 && ((uintptr_t)nbr_dev & 7u) == 0 &&
                         ((uintptr_t)lnbr_dev & 3u) == 0;
    tile_rings_kernel<<<nt, 512, smem, s>>>(k, tile > 0 ? tile : 0, aligned, nbr_dev, edge_dev, nv, rings, nmax, cmax,
                                            counts_dev, ids_dev, lnbr_dev, ledge_dev, err_dev);
    NX_CHECK_LAUNCH("tile_rings_kernel");
    nx::note_launch(1);
    return NX_OK;
}

// ---------------------------------------------------------------------------
// Nearest three vertices of query points (the reference's KD-tree
// query(k=3), nixis.py:278-283), by point location in the icosphere's own
// structure: the face whose corner matrix gives the query direction the
// largest smallest barycentric weight, the grid triangle of the flat face
// point (the spherical triangles are radial projections of the flat ones),
// then the exact distances to that triangle's vertices and all their
// neighbours.  On the icosphere's near-equilateral triangles the three
// nearest vertices of a point are always among them (checked against brute
// force in the tests).  Distances sqrt((dx*dx + dy*dy) + dz*dz), ascending,
// ties by vertex id.
//
// Binary64 bounds a direct evaluation (180 operations for the faces, 16 for
// each of 21 candidates, on a pipe of two per SM and cycle).  The location
// needs no more than binary32: a point within its error of another face or
// triangle has the same three among either's candidates.  The candidates are
// ranked in binary32 as well; the four best are compared exactly, and only
// where a fifth is not clearly farther than the third (the poles' rows, whose
// neighbours are all alike) all of them.  Measured (GB300, 1024 x 512 queries,
// 256,002 vertices): 636 -> 107 us.

namespace {

struct Best {
    double d[3];
    int64_t i[3];
};

__device__ __forceinline__ void best_take(Best &b, const double *xyz, int64_t v, double qx, double qy, double qz)
{
    if (v == b.i[0] || v == b.i[1] || v == b.i[2]) return;
    const double dx = __dsub_rn(qx, xyz[3 * v]), dy = __dsub_rn(qy, xyz[3 * v + 1]), dz = __dsub_rn(qz, xyz[3 * v + 2]);
    const double d = nxf::sqrt(__dadd_rn(__dadd_rn(nxf::square(dx), nxf::square(dy)), nxf::square(dz)));
#pragma unroll
    for (int m = 0; m < 3; ++m) {
        if (!(d < b.d[m] || (d == b.d[m] && v < b.i[m]))) continue;
#pragma unroll
        for (int r = 2; r > m; --r) { b.d[r] = b.d[r - 1]; b.i[r] = b.i[r - 1]; }
        b.d[m] = d;
        b.i[m] = v;
        return;
    }
}

__device__ __noinline__ void best_of_all(Best &b, const int32_t *tri, const double *xyz, const int32_t *nbr, int64_t nv, double qx,
                                         double qy, double qz)
{
    for (int m = 0; m < 3; ++m) { b.d[m] = INFINITY; b.i[m] = -1; }
    for (int c = 0; c < 21; ++c) {
        const int32_t v = c < 3 ? tri[c] : nbr[6 * (int64_t)tri[(c - 3) / 6] + (c - 3) % 6];
        if (v < 0 || (int64_t)v >= nv) continue;
        best_take(b, xyz, v, qx, qy, qz);
    }
}

// v * 2^-e as a binary32 (truncated), e the exponent that brings the query to
// [1, 2); 0 below 2^-60 of it.
__device__ __forceinline__ float scaled_chop(double v, uint32_t e20)
{
    const uint2 w = nxf::words(v);
    const uint32_t a = (w.y & 0x7FFFFFFFu);
    if (a + (60u << 20) < e20) return 0.0f;
    if (a > e20 + (60u << 20)) return __int_as_float(0x7F800000);
    const uint32_t s = a + (1023u << 20) - e20;
    return __uint_as_float(__funnelshift_l(w.x, s - (896u << 20), 3) | (w.y & 0x80000000u));
}

__global__ void __launch_bounds__(256) nearest3_kernel(int k, const double *__restrict__ xyz,
                                                       const int32_t *__restrict__ nbr, int64_t nv,
                                                       const double *__restrict__ q, int64_t nq,
                                                       double *__restrict__ dist, int64_t *__restrict__ idx)
{
    __shared__ float s_inv[20][9];
    for (int x = threadIdx.x; x < 180; x += blockDim.x) s_inv[x / 9][x % 9] = (float)c_ico.inv[x / 9][x % 9 / 3][x % 3];
    __syncthreads();
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nq; p += (int64_t)gridDim.x * blockDim.x) {
        const double qx = q[3 * p], qy = q[3 * p + 1], qz = q[3 * p + 2];
        // the query scaled to its largest component's binade (below the smallest
        // binade by a power of two, which only serves the location)
        const uint32_t ex = nxf::words(qx).y & 0x7FF00000u, ey = nxf::words(qy).y & 0x7FF00000u, ez = nxf::words(qz).y & 0x7FF00000u;
        const uint32_t e20 = max(ex, max(ey, ez));
        float x = scaled_chop(qx, e20), y = scaled_chop(qy, e20), z = scaled_chop(qz, e20);
        if (e20 == 0) {
            x = (float)(qx * 0x1p1022);
            y = (float)(qy * 0x1p1022);
            z = (float)(qz * 0x1p1022);
        }
        int bf = 0;
        float bw0 = 0.0f, bw1 = 0.0f, bw2 = 0.0f, bs = -INFINITY;
        for (int f = 0; f < 20; ++f) {
            const float *m = s_inv[f];
            const float w0 = fmaf(m[0], x, fmaf(m[1], y, m[2] * z)), w1 = fmaf(m[3], x, fmaf(m[4], y, m[5] * z)),
                        w2 = fmaf(m[6], x, fmaf(m[7], y, m[8] * z));
            const float sc = fminf(w0, fminf(w1, w2));
            if (sc > bs) { bs = sc; bf = f; bw0 = w0; bw1 = w1; bw2 = w2; }
        }
        const float tot = bw0 + bw1 + bw2;
        const float fi = fminf(fmaxf(bw1 / tot, 0.0f), 1.0f) * (float)k, fj = fminf(fmaxf(bw2 / tot, 0.0f), 1.0f) * (float)k;
        int i0 = (int)floorf(fi), j0 = (int)floorf(fj);
        if (i0 > k - 1) i0 = k - 1;
        if (i0 < 0) i0 = 0;
        if (j0 > k - 1 - i0) j0 = k - 1 - i0;
        if (j0 < 0) j0 = 0;
        const bool up = (fi - i0) + (fj - j0) <= 1.0f || i0 + j0 == k - 1;
        int32_t tri[3];
        if (up) {
            tri[0] = face_vid(bf, i0, j0, k); tri[1] = face_vid(bf, i0 + 1, j0, k); tri[2] = face_vid(bf, i0, j0 + 1, k);
        } else {
            tri[0] = face_vid(bf, i0 + 1, j0, k); tri[1] = face_vid(bf, i0 + 1, j0 + 1, k);
            tri[2] = face_vid(bf, i0, j0 + 1, k);
        }
        // the four smallest binary32 squared distances, and the smallest left out
        float a[4] = {INFINITY, INFINITY, INFINITY, INFINITY}, out = INFINITY;
        int32_t id[4] = {-1, -1, -1, -1};
        for (int c = 0; c < 21; ++c) {
            const int t = (c - 3) / 6;
            const int32_t v = c < 3 ? (c == 0 ? tri[0] : (c == 1 ? tri[1] : tri[2]))
                                    : nbr[6 * (int64_t)(t == 0 ? tri[0] : (t == 1 ? tri[1] : tri[2])) + (c - 3) % 6];
            if (v < 0 || (int64_t)v >= nv || v == id[0] || v == id[1] || v == id[2] || v == id[3]) continue;
            const float dx = x - scaled_chop(xyz[3 * (int64_t)v], e20), dy = y - scaled_chop(xyz[3 * (int64_t)v + 1], e20),
                        dz = z - scaled_chop(xyz[3 * (int64_t)v + 2], e20);
            float d = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            int32_t w = v;
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (d < a[m]) {
                    const float td = a[m];
                    const int32_t ti = id[m];
                    a[m] = d; id[m] = w;
                    d = td; w = ti;
                }
            // (a vertex pushed out earlier may come again: it only lowers out to
            // what it was)
            out = fminf(out, d);
        }
        // A scaled query's components are below 2 and off by less than 2^-23, a
        // vertex's by less than 2^-23 of itself, the vertex no longer than |q| +
        // d; the subtraction, the three roundings of d^2 and the root add 3.5
        // 2^-24 d: a distance is within 2^-23 (5.2 + 2.75 d), two of them within
        // 1.3e-6 + 6.6e-7 d5 (a vertex left out at a larger distance than d5 is
        // farther still by more than its own error grows).
        const float d3 = sqrtf(a[2]), d5 = sqrtf(out);
        Best b;
        if (d5 > d3 + __fmaf_rn(7e-7f, d5, 4e-6f) && a[3] < INFINITY && e20 != 0) {
            for (int m = 0; m < 3; ++m) { b.d[m] = INFINITY; b.i[m] = -1; }
#pragma unroll
            for (int m = 0; m < 4; ++m) best_take(b, xyz, id[m], qx, qy, qz);
        } else {
            best_of_all(b, tri, xyz, nbr, nv, qx, qy, qz);
        }
        for (int m = 0; m < 3; ++m) {
            dist[3 * p + m] = b.d[m];
            idx[3 * p + m] = b.i[m];
        }
    }
}

}  // namespace

NX_EXPORT int nx_nearest3(int k, const double *xyz_dev, const int32_t *nbr_dev, int64_t nv, const double *q_dev,
                          int64_t nq, double *dist_dev, int64_t *idx_dev, void *stream)
{
    if (k < 1 || nv != 10 * (int64_t)k * k + 2 || nq < 0) return nx::fail(NX_EINVAL, "nx_nearest3: bad sizes");
    if (nq == 0) return NX_OK;
    if (!xyz_dev || !nbr_dev || !q_dev || !dist_dev || !idx_dev) return nx::fail(NX_EINVAL, "nx_nearest3: null pointer");
    int dev = 0;
    NX_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !g_tables_ready[dev]) return nx::fail(NX_EINVAL, "nx_nearest3: icosphere tables not set");
    nearest3_kernel<<<grid1d(nq), 256, 0, (cudaStream_t)stream>>>(k, xyz_dev, nbr_dev, nv, q_dev, nq, dist_dev, idx_dev);
    NX_CHECK_LAUNCH("nearest3_kernel");
    nx::note_launch(1);
    return NX_OK;
}
