// sp_upload.cu — caller-supplied Wiener increments, host -> device.
//
// The caller's array is [S][M][n] doubles in pageable memory; the step kernels read
// [S][M][Np] Real.  A few host threads copy it piece by piece into pinned buffers, two each,
// while the copy engine empties the other one; a kernel spreads the rows to their padded
// pitch and converts them where the layouts differ (FP32, or n not a multiple of kPad).  The
// host therefore touches every increment once.  16384 particles, 250 steps (98 MB) on
// a B200 host: 3.6-4.8 ms; building the padded array on the host first and handing the driver
// a pageable copy of it took 53-55 ms.  The first upload of a context also allocates the pieces and
// grows the pool: whole call 22-37 ms there, 4 ms after, 59 and 55 the old way.  865 MB: 23 ms.  Below 4 MB one thread is as fast.
#include <algorithm>
#include <cstring>
#include <numeric>
#include <system_error>
#include <thread>
#include <vector>

#include "sp_runtime.h"

namespace sp {

namespace {

constexpr int kThreads = 4;                           // host threads
constexpr size_t kPiece = size_t(2) << 20;            // bytes of a pinned buffer
constexpr size_t kPieceDoubles = kPiece / 8;
constexpr size_t kFewBytes = size_t(4) << 20;         // below this one thread is enough

// doubles [first, first + count) of the caller's array to their places
template <class R>
__global__ void spread_kernel(const double* __restrict__ src, R* __restrict__ dst, unsigned long long first,
                              unsigned long long count, unsigned long long n, unsigned long long Np) {
    for (unsigned long long i = static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < count;
         i += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
        const unsigned long long g = first + i, row = g / n;
        dst[row * Np + (g - row * n)] = static_cast<R>(src[i]);
    }
}

struct Range {
    const double* src;
    size_t begin, end;  // doubles
};

// one thread's share; returns the first CUDA error, adds the kernels it launched to `launched`
cudaError_t upload_range(int device, const Range& r, void* dst, bool direct, int real, size_t n, size_t Np,
                         double* const* pinned, cudaMemPool_t pool, unsigned long long& launched) {
    if (r.begin >= r.end) return cudaSuccess;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return e;
    cudaStream_t s = nullptr;
    cudaEvent_t free_ev[2] = {nullptr, nullptr};
    double* raw[2] = {nullptr, nullptr};
    const auto ok = [&](cudaError_t x) {
        if (e == cudaSuccess) e = x;
        return e == cudaSuccess;
    };
    ok(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    for (int b = 0; b < 2 && e == cudaSuccess; ++b) {
        ok(cudaEventCreateWithFlags(&free_ev[b], cudaEventDisableTiming));
        if (!direct && e == cudaSuccess) ok(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&raw[b]), kPiece, pool, s));
    }
    int b = 0;
    for (size_t at = r.begin; at < r.end && e == cudaSuccess; at += kPieceDoubles, b ^= 1) {
        const size_t count = std::min(kPieceDoubles, r.end - at);
        if (!ok(cudaEventSynchronize(free_ev[b]))) break;  // the buffer's previous copy has left it
        const double* from = r.src + at;  // pageable, where there is no pinned buffer
        if (pinned[b]) from = static_cast<const double*>(std::memcpy(pinned[b], from, count * 8));
        if (direct) {
            ok(cudaMemcpyAsync(static_cast<double*>(dst) + at, from, count * 8, cudaMemcpyHostToDevice, s));
        } else {
            ok(cudaMemcpyAsync(raw[b], from, count * 8, cudaMemcpyHostToDevice, s));
            const unsigned grid = static_cast<unsigned>((count + 255) / 256);
            if (real == 8) spread_kernel<double><<<grid, 256, 0, s>>>(raw[b], static_cast<double*>(dst), at, count, n, Np);
            else spread_kernel<float><<<grid, 256, 0, s>>>(raw[b], static_cast<float*>(dst), at, count, n, Np);
            if (ok(cudaGetLastError())) ++launched;
        }
        ok(cudaEventRecord(free_ev[b], s));
    }
    for (double* p : raw)
        if (p) cudaFreeAsync(p, s);
    if (s) ok(cudaStreamSynchronize(s));
    for (cudaEvent_t ev : free_ev)
        if (ev) cudaEventDestroy(ev);
    if (s) cudaStreamDestroy(s);
    return e;
}

}  // namespace

// returns when the increments are on the device.  dst was allocated in stream order on s.
unsigned long long upload_increments(sp_context* ctx, const double* src, void* dst, int real, size_t rows, size_t n,
                                     size_t Np, cudaStream_t s) {
    const size_t total = rows * n;
    const bool direct = real == 8 && n == Np;
    if (!direct) check_cuda(cudaMemsetAsync(dst, 0, rows * Np * real, s), "clear dW");
    check_cuda(cudaStreamSynchronize(s), "dW buffer");
    // the pinned buffers belong to the context and serve one upload at a time
    std::lock_guard<std::mutex> lk(ctx->dw_mu);
    const int threads = total * 8 < kFewBytes ? 1 : kThreads;
    while (ctx->dw_pinned.size() < static_cast<size_t>(2 * threads)) {
        double* p = nullptr;
        if (cudaMallocHost(reinterpret_cast<void**>(&p), kPiece) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        ctx->dw_pinned.push_back(p);
    }
    const size_t share = ((total + threads - 1) / threads + 511) / 512 * 512;
    cudaError_t errors[kThreads] = {};
    unsigned long long launched[kThreads] = {};
    const auto work = [&](int t) {
        const Range r{src, std::min(total, t * share), std::min(total, (t + 1) * share)};
        errors[t] = upload_range(ctx->device, r, dst, direct, real, n, Np, &ctx->dw_pinned[2 * t], ctx->pool,
                                 launched[t]);
    };
    std::vector<std::thread> helpers;
    int started = 1;
    try {
        helpers.reserve(threads);
        for (; started < threads; ++started) helpers.emplace_back(work, started);
    } catch (const std::exception&) {
        // no more threads to be had: this one does the rest
    }
    work(0);
    for (int t = started; t < threads; ++t) work(t);
    for (std::thread& h : helpers) h.join();
    for (int t = 0; t < threads; ++t) check_cuda(errors[t], "upload dW");
    return std::accumulate(launched, launched + threads, 0ull);
}

}  // namespace sp
