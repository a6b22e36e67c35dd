// What follows the last distance layer of a classifier while it trains: margins of the interval [dist - eps, dist + eps], and
// the hinge loss on them.
//
// Both are a few KB, so the launches are all they cost: as torch operators they are 18 forward and 20 backward, each behind 4
// to 10 us of host work, which a small network's step waits for (256 x 3072 -> 1024 -> 1024 -> 1024 -> 10, p = inf, forward,
// loss and gradients: 780 us, of which the device is busy for 371).  Here they are two kernels forward and two backward: the step
// takes 585 us where it took 1018 on one machine.
#include "ldn_b200.h"
#include "ldn_common.cuh"

namespace ldn {
namespace {

constexpr int kHingeThreads = 1024;

// logits = -dist; margin_j = (upper bound of the target's distance) - (lower bound of j's), 0 for the target, times `inv`.  The
// roundings are those of -(dist - eps) - (-(dist_target + eps)) in 32 bits.
__global__ void __launch_bounds__(kThreads) margins_kernel(const float* dist, const float* dist_target, const long long* targets,
                                                           unsigned n, unsigned classes, float eps, float inv, float* logits,
                                                           float* margin) {
    stream_order_begin();
    for (unsigned i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        const unsigned b = i / classes, j = i - b * classes;
        const float d = dist[i];
        const float v = __fsub_rn(-__fsub_rn(d, eps), -__fadd_rn(dist_target[b], eps));
        logits[i] = -d;
        margin[i] = __fmul_rn(static_cast<long long>(j) == targets[b] ? 0.0f : v, inv);
    }
}

// A warp per row: grad_j = -(grad_logits_j) - inv grad_margin_j, and the target collects what the others give up.
__global__ void __launch_bounds__(kThreads) margins_backward_kernel(const float* grad_logits, const float* grad_margin,
                                                                    const long long* targets, int rows, int classes, float inv,
                                                                    float* grad) {
    stream_order_begin();
    const int lane = threadIdx.x & 31;
    for (int b = (blockIdx.x * kThreads + threadIdx.x) >> 5; b < rows; b += gridDim.x * kThreads >> 5) {
        const long long at = static_cast<long long>(b) * classes, target = targets[b];
        float sum = 0.0f;
        for (int j = lane; j < classes; j += 32) {
            const float m = grad_margin && j != target ? __fmul_rn(grad_margin[at + j], inv) : 0.0f;
            sum += m;
            if (j != target) grad[at + j] = -m - (grad_logits ? grad_logits[at + j] : 0.0f);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
        if (lane == 0 && target >= 0 && target < classes)
            grad[at + target] = sum - (grad_logits ? grad_logits[at + target] : 0.0f);
    }
}

// a in front of b as the larger value: NaN first, equal values by their place
__device__ __forceinline__ bool in_front(float a, int ia, float b, int ib) {
    if (isnan(a) != isnan(b)) return isnan(a);
    return isnan(a) || a == b ? ia < ib : a > b;
}

// loss = (1 - mix) mean over rows of max_j pos + mix mean of pos, pos = max(margin, 0); first[b] = where the row's maximum
// stands first.  One block: the rows are few.
__global__ void __launch_bounds__(kHingeThreads) hinge_kernel(const float* margin, int rows, int classes, double mix, float* loss,
                                                              int* first) {
    stream_order_begin();
    __shared__ double totals[2][kHingeThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double largest = 0.0, all = 0.0;
    for (int b = warp; b < rows; b += kHingeThreads / 32) {
        const float* row = margin + static_cast<long long>(b) * classes;
        float top = -1.0f;  // below every clamped value
        int where = 0x7fffffff;
        for (int j = lane; j < classes; j += 32) {
            const float v = row[j], pos = v < 0.0f ? 0.0f : v;  // (a NaN stays)
            all += pos;
            if (in_front(pos, j, top, where)) {
                top = pos;
                where = j;
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            const float t = __shfl_xor_sync(0xffffffffu, top, d);
            const int w = __shfl_xor_sync(0xffffffffu, where, d);
            if (in_front(t, w, top, where)) {
                top = t;
                where = w;
            }
        }
        if (lane == 0) {
            largest += top;
            first[b] = where;
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) all += __shfl_xor_sync(0xffffffffu, all, d);
    if (lane == 0) {
        totals[0][warp] = largest;
        totals[1][warp] = all;
    }
    __syncthreads();
    if (warp == 0) {
        largest = totals[0][lane];
        all = totals[1][lane];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            largest += __shfl_xor_sync(0xffffffffu, largest, d);
            all += __shfl_xor_sync(0xffffffffu, all, d);
        }
        if (lane == 0) *loss = static_cast<float>((1.0 - mix) * (largest / rows) + mix * (all / (static_cast<double>(rows) * classes)));
    }
}

__global__ void __launch_bounds__(kThreads) hinge_backward_kernel(const float* grad_loss, const float* margin, const int* first,
                                                                  unsigned n, unsigned classes, float largest, float each,
                                                                  float* grad) {
    stream_order_begin();
    const float g = *grad_loss;
    for (unsigned i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        const unsigned b = i / classes, j = i - b * classes;
        const float v = g * each + (static_cast<int>(j) == first[b] ? g * largest : 0.0f);
        grad[i] = margin[i] >= 0.0f ? v : 0.0f;
    }
}

constexpr int kMostElements = 1 << 24;
bool few(int rows, int classes) {
    return rows > 0 && classes > 0 && static_cast<long long>(rows) * classes <= kMostElements;
}
unsigned blocks(long long threads) {
    const long long n = (threads + kThreads - 1) / kThreads;
    return static_cast<unsigned>(n < 1184 ? n : 1184);
}

}  // namespace
}  // namespace ldn

using namespace ldn;

extern "C" LDN_API int ldn_margins(const float* dist, const float* dist_target, const long long* targets, int B, int classes,
                                   float eps, float inv, float* logits, float* margin, ldn_stream_t stream) {
    if (!few(B, classes) || !dist || !dist_target || !targets || !logits || !margin) return kBadArgument;
    const unsigned n = static_cast<unsigned>(B) * classes;
    return launch_after(margins_kernel, blocks(n), kThreads, 0, reinterpret_cast<cudaStream_t>(stream), dist, dist_target, targets,
                        n, static_cast<unsigned>(classes), eps, inv, logits, margin);
}

extern "C" LDN_API int ldn_margins_backward(const float* grad_logits, const float* grad_margin, const long long* targets, int B,
                                            int classes, float inv, float* grad, ldn_stream_t stream) {
    if (!few(B, classes) || !targets || !grad) return kBadArgument;
    return launch_after(margins_backward_kernel, blocks(32LL * B), kThreads, 0, reinterpret_cast<cudaStream_t>(stream), grad_logits,
                        grad_margin, targets, B, classes, inv, grad);
}

extern "C" LDN_API int ldn_hinge(const float* margin, int B, int classes, double mix, float* loss, int* first,
                                 ldn_stream_t stream) {
    if (!few(B, classes) || !margin || !loss || !first) return kBadArgument;
    return launch_after(hinge_kernel, 1, kHingeThreads, 0, reinterpret_cast<cudaStream_t>(stream), margin, B, classes, mix, loss,
                        first);
}

extern "C" LDN_API int ldn_hinge_backward(const float* grad_loss, const float* margin, const int* first, int B, int classes,
                                          double mix, float* grad, ldn_stream_t stream) {
    if (!few(B, classes) || !grad_loss || !margin || !first || !grad) return kBadArgument;
    const unsigned n = static_cast<unsigned>(B) * classes;
    return launch_after(hinge_backward_kernel, blocks(n), kThreads, 0, reinterpret_cast<cudaStream_t>(stream), grad_loss, margin,
                        first, n, static_cast<unsigned>(classes), static_cast<float>((1.0 - mix) / B),
                        static_cast<float>(mix / (static_cast<double>(B) * classes)), grad);
}
