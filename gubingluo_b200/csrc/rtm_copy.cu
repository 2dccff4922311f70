// rtm_copy.cu — results from the device into the caller's (pageable) host memory.
//
// A plain cudaMemcpy into pageable memory goes through the driver's staging buffers on one host
// thread, which also takes the page faults of a freshly allocated destination: 2 GB/s for the
// four 2.4 MB images of a 1701 x 351 model (4.6 ms), and fp64 images were copied whole and
// narrowed on the host (95 ms for four 4001 x 1201 images).  Here up to kLanes host threads each
// move chunks through a page-locked buffer and stream of their own, so copies, page faults and
// host writes overlap, and fp64 images are narrowed by a kernel that writes the page-locked
// buffer (half the bytes over the bus).  Measured: 1.1 ms and 7 ms.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <string>

#include "rtm_internal.h"

namespace rtm {

namespace {

constexpr size_t kChunk = (size_t)1 << 20;   // bytes of a lane's page-locked buffer
constexpr int kLanes = 4;                    // lanes of a copy, and those kept per device (4 MB page-locked)
constexpr int kMaxDevices = 64;              // (lanes of devices beyond are not kept)

struct Lane {
    void *buf = nullptr;
    cudaStream_t st = nullptr;
    int dev = -1;
    unsigned long long ctx = 0;   // the context they were made in
};
// Lanes not in use, per device: lanes of one device must not take the places of another's, whose every
// copy would then allocate and free its own.
std::mutex g_mu;
Lane g_free[kMaxDevices][kLanes];
int g_kept[kMaxDevices];

void drop(Lane &l)
{
    if (l.st) cudaStreamDestroy(l.st);
    if (l.buf) cudaFreeHost(l.buf);
    l = Lane();
}
// Number of the current context, different for every context that the process ever makes (0 where the driver
// has no such call): a cudaDeviceReset takes the kept lanes' buffers and streams with it, and the
// device's next context has another number.
unsigned long long context_id()
{
    typedef CUresult (*Fn)(CUcontext, unsigned long long *);
    static const Fn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (Fn)p;
    }();
    unsigned long long id = 0;
    return fn && fn(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}
bool take(int dev, unsigned long long ctx, Lane &l)
{
    {
        std::lock_guard<std::mutex> lock(g_mu);
        while (dev < kMaxDevices && g_kept[dev] > 0) {
            l = g_free[dev][--g_kept[dev]];
            if (l.ctx == ctx) return true;
            l = Lane();   // gone with its context
        }
    }
    l.dev = dev;
    l.ctx = ctx;
    if (cudaHostAlloc(&l.buf, kChunk, cudaHostAllocDefault) != cudaSuccess ||
        cudaStreamCreateWithFlags(&l.st, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        drop(l);
        return false;
    }
    return true;
}
void give(Lane &l)
{
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (l.dev < kMaxDevices && g_kept[l.dev] < kLanes) {
            g_free[l.dev][g_kept[l.dev]++] = l;
            return;
        }
    }
    drop(l);
}

__global__ void k_narrow(const double *__restrict__ src, float *__restrict__ dst, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = (float)src[i];
}

// The narrowing copy without a lane: n doubles through a buffer on the stack.
cudaError_t plain_narrow(float *dst, const double *src, size_t n)
{
    double part[4096];
    for (size_t i = 0; i < n; i += 4096) {
        const size_t m = std::min<size_t>(4096, n - i);
        cudaError_t e = cudaMemcpy(part, src + i, m * sizeof(double), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return e;
        for (size_t k = 0; k < m; k++) dst[i + k] = (float)part[k];
    }
    return cudaSuccess;
}

}  // namespace

// dst (packed rows of row_bytes) <- rows of the device array src, src_pitch bytes apart, on the
// current device, whose writers have finished: unlike a plain cudaMemcpy, the lanes' streams do not wait for
// the default stream.  narrow: src holds doubles (contiguous), dst floats.
int copy_out(void *dst, const void *src, size_t src_pitch, size_t row_bytes, size_t rows, bool narrow)
{
    if (src_pitch == row_bytes || rows == 1) {   // contiguous: rows of a chunk
        const size_t total = row_bytes * rows;
        if (total < kChunk / 4 && !narrow) {
            cudaError_t e = cudaMemcpy(dst, src, total, cudaMemcpyDeviceToHost);
            return e == cudaSuccess ? RTM_OK : fail(RTM_ERR_CUDA, std::string("copy to host: ") + cudaGetErrorString(e));
        }
        row_bytes = 1;
        src_pitch = 1;
        rows = total;
    } else if (row_bytes > kChunk) {
        for (size_t r = 0; r < rows; r++)
            if (int rc = copy_out((char *)dst + r * row_bytes, (const char *)src + r * src_pitch, row_bytes, row_bytes, 1, false))
                return rc;
        return RTM_OK;
    }
    const size_t per = kChunk / row_bytes, n = (rows + per - 1) / per;   // rows per chunk, chunks
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(RTM_ERR_CUDA, std::string("copy to host: ") + cudaGetErrorString(e));
    std::atomic<size_t> next{0};
    std::atomic<int> err{(int)cudaSuccess};
    const unsigned long long ctx = context_id();   // (the library runs in the device's primary context only)
    const int nt = (int)std::min<size_t>(kLanes, n);
    const bool team = host_team();
#pragma omp parallel num_threads(nt) if (team)
    {
        Lane l;
        cudaError_t e = cudaSetDevice(dev);
        const bool lane = e == cudaSuccess && take(dev, ctx, l);   // without one this thread copies nothing
        while (lane && e == cudaSuccess) {
            const size_t c = next.fetch_add(1);
            if (c >= n) break;
            const size_t r0 = c * per, nr = std::min(per, rows - r0), bytes = nr * row_bytes;
            if (narrow) {
                k_narrow<<<64, 256, 0, l.st>>>((const double *)src + r0 / 4, (float *)l.buf, (int)(bytes / 4));
                e = cudaGetLastError();
            } else if (row_bytes == 1) {
                e = cudaMemcpyAsync(l.buf, (const char *)src + r0, bytes, cudaMemcpyDeviceToHost, l.st);
            } else {
                e = cudaMemcpy2DAsync(l.buf, row_bytes, (const char *)src + r0 * src_pitch, src_pitch, row_bytes, nr,
                                      cudaMemcpyDeviceToHost, l.st);
            }
            if (e == cudaSuccess) e = cudaStreamSynchronize(l.st);
            if (e == cudaSuccess) std::memcpy((char *)dst + r0 * row_bytes, l.buf, bytes);
        }
        if (l.buf) {
            if (e == cudaSuccess) give(l);
            else drop(l);
        }
        if (e != cudaSuccess) err.store((int)e);
    }
    e = (cudaError_t)err.load();
    const size_t r0 = std::min(next.load() * per, rows);
    if (e == cudaSuccess && r0 < rows) {
        // what no lane took (no page-locked memory or stream to be had): plain copies
        void *to = (char *)dst + r0 * row_bytes;
        const void *from = (const char *)src + r0 * src_pitch;
        if (narrow) e = plain_narrow((float *)to, (const double *)src + r0 / 4, (rows - r0) / 4);
        else if (row_bytes == 1) e = cudaMemcpy(to, from, rows - r0, cudaMemcpyDeviceToHost);
        else e = cudaMemcpy2D(to, row_bytes, from, src_pitch, row_bytes, rows - r0, cudaMemcpyDeviceToHost);
    }
    if (e != cudaSuccess) return fail(RTM_ERR_CUDA, std::string("copy to host: ") + cudaGetErrorString(e));
    return RTM_OK;
}

}  // namespace rtm
