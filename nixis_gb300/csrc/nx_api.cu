// nx_api.cu -- error reporting, device queries and host-side table setup.
#include "nx_common.cuh"

#include <atomic>
#include <cstdarg>
#include <cstring>
#include <mutex>

namespace nx {

static thread_local char g_err[512] = "";
static std::atomic<unsigned long long> g_launches{0};

void set_error(const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int fail(int code, const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

int check_cuda(cudaError_t e, const char *what)
{
    if (e == cudaSuccess) return NX_OK;
    set_error("%s: %s", what, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? NX_ENOMEM : NX_ECUDA;
}

int sm_count()
{
    static int cache[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    if (!cache[dev]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v < 1) v = 1;
        cache[dev] = v;
    }
    return cache[dev];
}

void note_launch(int k) { g_launches.fetch_add((unsigned long long)k, std::memory_order_relaxed); }

}  // namespace nx

NX_EXPORT const char *nx_last_error(void) { return nx::g_err; }

NX_EXPORT int nx_version(void) { return 10200; }

NX_EXPORT unsigned long long nx_launch_count(void) { return nx::g_launches.load(); }

// opensimplex.init (opensimplex.py:90-107).  `over` (opensimplex.py:110-112)
// is compiled by numba with signature int32(int32): each LCG state is cut to
// its low 32 bits, sign-extended; the 64-bit multiply-add itself wraps.
// The index r is a floor-mod, non-negative for the positive modulus.
NX_EXPORT int nx_perm_init(int64_t seed, int32_t *perm, int32_t *pgi)
{
    if (!perm || !pgi) return nx::fail(NX_EINVAL, "nx_perm_init: null pointer");
    auto step = [](int64_t state) -> int64_t {
        uint64_t v = (uint64_t)state * 6364136223846793005ULL + 1442695040888963407ULL;
        return (int64_t)(int32_t)(uint32_t)(v & 0xFFFFFFFFu);
    };
    int32_t pool[256];
    for (int i = 0; i < 256; ++i) pool[i] = i;
    int64_t st = step(step(step(seed)));
    for (int i = 255; i >= 0; --i) {
        st = step(st);
        int64_t m = (int64_t)i + 1;
        int64_t r = (st + 31) % m;
        if (r < 0) r += m;
        perm[i] = pool[r];
        pgi[i] = (perm[i] % 24) * 3;   // int((perm % 24.0) * 3) for perm in [0, 255]
        pool[r] = pool[i];
    }
    return NX_OK;
}

// ---------------------------------------------------------------------------
// Small host tables (permutations, sun positions) to the device as kernel
// arguments: the bytes are taken when the call is made, so the host may reuse
// them at once, nothing waits, and a captured launch carries them.  A copy
// through pinned memory took 24 us for 60 KB and 25 us for 1 KB (allocation,
// event, copy engine), a pageable one waits for the stream; this is a launch.
// ---------------------------------------------------------------------------
struct UploadChunk {
    unsigned w[1000];      // 4,000 bytes: within the argument space of every launch
};

static __global__ void upload_kernel(UploadChunk c, unsigned char *dst, int bytes)
{
    const unsigned char *src = reinterpret_cast<const unsigned char *>(c.w);
    for (int i = threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
}

static __global__ void upload_words_kernel(UploadChunk c, unsigned *dst, int words)
{
    for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = c.w[i];
}

NX_EXPORT int nx_upload(void *dst_dev, const void *src_host, int64_t bytes, void *stream)
{
    if (bytes < 0 || bytes > NX_UPLOAD_MAX || (bytes && (!dst_dev || !src_host)))
        return nx::fail(NX_EINVAL, "nx_upload: bad arguments");
    for (int64_t o = 0; o < bytes; o += (int64_t)sizeof(UploadChunk)) {
        const int64_t left = bytes - o;
        const int take = (int)(left < (int64_t)sizeof(UploadChunk) ? left : (int64_t)sizeof(UploadChunk));
        UploadChunk c;
        memcpy(c.w, (const unsigned char *)src_host + o, (size_t)take);
        unsigned char *d = (unsigned char *)dst_dev + o;
        if (take % 4 == 0 && (uintptr_t)d % 4 == 0)
            upload_words_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(c, (unsigned *)d, take / 4);
        else
            upload_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(c, d, take);
        NX_CHECK_LAUNCH("upload_kernel");
        nx::note_launch(1);
    }
    return NX_OK;
}

// (the question is one that a capture on another thread forbids by default: the
// calling thread's interaction with captures is relaxed meanwhile)
NX_EXPORT int nx_stream_idle(void *stream)
{
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    bool idle = cudaStreamIsCapturing((cudaStream_t)stream, &capture) == cudaSuccess &&
                capture == cudaStreamCaptureStatusNone;
    if (idle && cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess) {
        idle = cudaStreamQuery((cudaStream_t)stream) == cudaSuccess;
        cudaThreadExchangeStreamCaptureMode(&mode);
    } else {
        idle = false;
    }
    if (!idle) cudaGetLastError();
    return idle ? 1 : 0;
}
