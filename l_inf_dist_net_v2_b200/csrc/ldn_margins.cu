// What follows the last distance layer of a classifier while it trains: margins of the interval [dist - eps, dist + eps], and
// the hinge loss on them.
//
// Both are a few KB, so the launches are all they cost: as torch operators they are 18 forward and 20 backward, each behind 4
// to 10 us of host work, which a small network's step waits for (256 x 3072 -> 1024 -> 1024 -> 1024 -> 10, p = inf, forward,
// loss and gradients: 780 us, of which the device is busy for 371).  Here they are two kernels forward and two backward: the step
// takes 585 us where it took 1018 on one machine.
#include <cooperative_groups.h>

#include "ldn_b200.h"
#include "ldn_common.cuh"

namespace ldn {
namespace {

constexpr int kHingeThreads = 1024;
constexpr int kHingeRows = 4;    // rows in flight per group of lanes
constexpr int kHingeBlocks = 8;  // (the largest cluster that every device of the kind takes)

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
// stands first.  Latency bounds it: a row is a load and a shuffle tree.  So LANES lanes have a row (as many as there are classes,
// up to a warp) and kHingeRows rows at a time, and up to eight blocks work as a cluster, whose first adds up the sums of all in
// shared memory: one launch, sums in a fixed order.  On the device, forward, with one block and a warp per row ->
// this, in us (torch operators): 64 x 10 4 -> 6 (14), 512 x 10 14 -> 6 (14), 4096 x 10 96 -> 8 (19), 16384 x 10 372 -> 23 (25),
// 1000 x 1000 153 -> 29 (27).
template <int LANES>
__global__ void __launch_bounds__(kHingeThreads) hinge_kernel(const float* margin, int rows, int classes, double mix, float* loss,
                                                              int* first) {
    stream_order_begin();
    __shared__ double totals[2][kHingeThreads / 32];
    __shared__ double cluster_totals[kHingeBlocks][2];
    constexpr int kGroups = kHingeThreads / LANES;  // of a block
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = threadIdx.x % LANES;
    const int step = gridDim.x * kGroups;  // (the grid is one cluster)
    double largest = 0.0, all = 0.0;
    // (a warp's groups take part in its shuffles whether they have a row or not)
    const int warp_first = blockIdx.x * kGroups + warp * (32 / LANES);
    for (long long base = warp_first; base < rows; base += static_cast<long long>(step) * kHingeRows) {
        const long long b0 = base + lane / LANES;
        float top[kHingeRows];
        int where[kHingeRows];
#pragma unroll
        for (int u = 0; u < kHingeRows; ++u) {
            top[u] = -1.0f;  // below every clamped value
            where[u] = 0x7fffffff;
        }
        for (int j = sub; j < classes; j += LANES) {
            float v[kHingeRows];
#pragma unroll
            for (int u = 0; u < kHingeRows; ++u) {
                const long long b = b0 + static_cast<long long>(u) * step;
                v[u] = b < rows ? margin[b * classes + j] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < kHingeRows; ++u) {
                const float pos = v[u] < 0.0f ? 0.0f : v[u];  // (a NaN stays; rows that are not there add 0)
                all += pos;
                if (in_front(pos, j, top[u], where[u])) {
                    top[u] = pos;
                    where[u] = j;
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kHingeRows; ++u) {
#pragma unroll
            for (int d = LANES / 2; d > 0; d >>= 1) {
                const float t = __shfl_xor_sync(0xffffffffu, top[u], d);
                const int w = __shfl_xor_sync(0xffffffffu, where[u], d);
                if (in_front(t, w, top[u], where[u])) {
                    top[u] = t;
                    where[u] = w;
                }
            }
            const long long b = b0 + static_cast<long long>(u) * step;
            if (sub == 0 && b < rows) {
                largest += top[u];
                first[b] = where[u];
            }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        largest += __shfl_xor_sync(0xffffffffu, largest, d);
        all += __shfl_xor_sync(0xffffffffu, all, d);
    }
    if (lane == 0) {
        totals[0][warp] = largest;
        totals[1][warp] = all;
    }
    __syncthreads();
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    if (warp == 0) {
        largest = totals[0][lane];
        all = totals[1][lane];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            largest += __shfl_xor_sync(0xffffffffu, largest, d);
            all += __shfl_xor_sync(0xffffffffu, all, d);
        }
        if (lane == 0) {
            double* to = cluster.map_shared_rank(&cluster_totals[blockIdx.x][0], 0);
            to[0] = largest;
            to[1] = all;
        }
    }
    cluster.sync();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        largest = all = 0.0;
        for (unsigned i = 0; i < gridDim.x; ++i) {
            largest += cluster_totals[i][0];
            all += cluster_totals[i][1];
        }
        *loss = static_cast<float>((1.0 - mix) * (largest / rows) + mix * (all / (static_cast<double>(rows) * classes)));
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

template <int LANES>
int launch_hinge(const float* margin, int rows, int classes, double mix, float* loss, int* first, cudaStream_t st) {
    // a block more for every pass over rows that it saves
    int blocks = 1;
    while (blocks < kHingeBlocks && static_cast<long long>(blocks) * (kHingeThreads / LANES) * kHingeRows < rows) blocks *= 2;
    return launch_after_in_clusters(hinge_kernel<LANES>, blocks, blocks, kHingeThreads, 0, st, margin, rows, classes, mix, loss, first);
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
    const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (classes <= 2) return launch_hinge<2>(margin, B, classes, mix, loss, first, st);
    if (classes <= 4) return launch_hinge<4>(margin, B, classes, mix, loss, first, st);
    if (classes <= 8) return launch_hinge<8>(margin, B, classes, mix, loss, first, st);
    if (classes <= 16) return launch_hinge<16>(margin, B, classes, mix, loss, first, st);
    return launch_hinge<32>(margin, B, classes, mix, loss, first, st);
}

extern "C" LDN_API int ldn_hinge_backward(const float* grad_loss, const float* margin, const int* first, int B, int classes,
                                          double mix, float* grad, ldn_stream_t stream) {
    if (!few(B, classes) || !grad_loss || !margin || !first || !grad) return kBadArgument;
    const unsigned n = static_cast<unsigned>(B) * classes;
    return launch_after(hinge_backward_kernel, blocks(n), kThreads, 0, reinterpret_cast<cudaStream_t>(stream), grad_loss, margin,
                        first, n, static_cast<unsigned>(classes), static_cast<float>((1.0 - mix) / B),
                        static_cast<float>(mix / (static_cast<double>(B) * classes)), grad);
}
