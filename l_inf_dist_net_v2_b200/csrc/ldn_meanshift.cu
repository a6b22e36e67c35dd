// Training-mode MeanShift of a fully connected distance layer in one kernel: per-channel batch mean, update of
// the running mean, subtraction.  The reference does this with separate torch operators
// (core/modules/basic_modules.py:104-135: x.mean(dim=[0, 2]), running_mean.mul_(1 - m).add_(mean, alpha = m),
// x - mean); the same kernel without a running mean is its backward pass (grad - mean over the batch of grad).
// Convolution layers (x[B][C][HW], mean over samples and positions): mean_shift_planes_kernel.
#include <cooperative_groups.h>

#include "ldn_b200.h"
#include "ldn_common.cuh"

namespace ldn {
namespace {
constexpr int kCols = 32;      // channels per CTA (one 128-byte row segment per warp-wide load)
constexpr int kRowLanes = 32;  // row groups per CTA (1024 threads: 8 of them took 20 us at 512 x 5120, latency bound)

// x, out: [B][C] row-major.  Thread (lane = channel in the CTA's 32, rl = row group) sums rows rl, rl + 8, ...;
// the 8 partial sums of a channel are folded in shared memory in a fixed order, so the result is deterministic.
__global__ void __launch_bounds__(kCols * kRowLanes)
mean_shift_rows_kernel(const float* x, float* out, float* running_mean,
                       float* mean_out, float momentum, int B, int C) {
    stream_order_begin();
    __shared__ float part[kRowLanes][kCols];
    const int lane = threadIdx.x & (kCols - 1);
    const int rl = threadIdx.x / kCols;
    const int col = blockIdx.x * kCols + lane;
    const bool live = col < C;
    float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
    if (live) {
        int r = rl;
        for (; r + 3 * kRowLanes < B; r += 4 * kRowLanes) {
            s0 += x[static_cast<size_t>(r) * C + col];
            s1 += x[static_cast<size_t>(r + kRowLanes) * C + col];
            s2 += x[static_cast<size_t>(r + 2 * kRowLanes) * C + col];
            s3 += x[static_cast<size_t>(r + 3 * kRowLanes) * C + col];
        }
        for (; r < B; r += kRowLanes) s0 += x[static_cast<size_t>(r) * C + col];
    }
    part[rl][lane] = (s0 + s1) + (s2 + s3);
    __syncthreads();
    float mean = 0.0f;
#pragma unroll
    for (int q = 0; q < kRowLanes; ++q) mean += part[q][lane];
    mean /= static_cast<float>(B);
    if (!live) return;
    if (rl == 0) {
        if (running_mean) running_mean[col] = running_mean[col] * (1.0f - momentum) + momentum * mean;
        if (mean_out) mean_out[col] = mean;
    }
    for (int r = rl; r < B; r += kRowLanes) {
        const size_t i = static_cast<size_t>(r) * C + col;
        out[i] = x[i] - mean;
    }
}

// x, out: [B][C][HW].  Bound by the bytes of x and out, so x is read once: a cluster of 8 CTAs owns a channel, every CTA
// sums its eighth of the channel's B HW elements and keeps them in registers (up to kKeep 16-byte pieces per thread, 64 K
// elements per channel; what lies beyond is read again), the eight sums are exchanged through distributed shared memory and
// added in rank order (deterministic).  Sums are 64 bits wide beyond a thread's 16-byte piece: in 32 bits the mean of a
// channel of 32768 elements was further off than torch's, by up to 1.6 times behind the subtraction, which takes most of the
// value away.  V = elements per piece: 4 where planes are whole aligned pieces, else 1.
// (Mean, running mean and subtraction by torch operators were five launches forward and four backward, 50 us of a
// 128 x 64 x 16 x 16 layer step; with this kernel and the fold by rows that step takes 310 us instead of 388.)
constexpr int kCluster = 8;
constexpr int kPlaneThreads = 256;
constexpr int kKeep = 8;

template <int V>
__global__ void __launch_bounds__(kPlaneThreads)
mean_shift_planes_kernel(const float* x, float* out, float* running_mean, float momentum, int B, int C, int HW) {
    stream_order_begin();
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    __shared__ double warp_sums[kPlaneThreads / 32];
    __shared__ double total;
    const int c = blockIdx.x / kCluster, rank = blockIdx.x % kCluster;
    const long long row = HW / V, n = B * row;  // pieces per plane and per channel
    const long long first = n * rank / kCluster + threadIdx.x, last = n * (rank + 1) / kCluster;
    auto offset = [&](long long t) {
        const long long b = t / row;
        return (b * C + c) * HW + (t - b * row) * V;
    };
    float keep[kKeep][V];
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kKeep; ++k) {
        const long long t = first + k * kPlaneThreads;
#pragma unroll
        for (int e = 0; e < V; ++e) keep[k][e] = 0.0f;
        if (t < last) {
            if constexpr (V == 4) {
                const float4 v = *reinterpret_cast<const float4*>(x + offset(t));
                keep[k][0] = v.x; keep[k][1] = v.y; keep[k][2] = v.z; keep[k][3] = v.w;
            } else {
                keep[k][0] = x[offset(t)];
            }
        }
    }
    auto piece_sum = [](const float* v) { return V == 4 ? (v[0] + v[1]) + (v[2] + v[3]) : v[0]; };
#pragma unroll
    for (int k = 0; k < kKeep; ++k) s += piece_sum(keep[k]);
    for (long long t = first + kKeep * kPlaneThreads; t < last; t += kPlaneThreads) s += piece_sum(x + offset(t));
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x / 32] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        s = 0.0;
        for (int w = 0; w < kPlaneThreads / 32; ++w) s += warp_sums[w];
        total = s;
    }
    cluster.sync();
    s = 0.0;
#pragma unroll
    for (int q = 0; q < kCluster; ++q) s += *cluster.map_shared_rank(&total, q);
    const float mean = static_cast<float>(s / (static_cast<double>(B) * HW));
    cluster.sync();  // every rank has read the others' sums before one of them may exit
    if (running_mean && rank == 0 && threadIdx.x == 0)
        running_mean[c] = running_mean[c] * (1.0f - momentum) + momentum * mean;
    auto store = [&](long long t, const float* v) {
        if constexpr (V == 4)
            *reinterpret_cast<float4*>(out + offset(t)) = make_float4(v[0] - mean, v[1] - mean, v[2] - mean, v[3] - mean);
        else
            out[offset(t)] = v[0] - mean;
    };
#pragma unroll
    for (int k = 0; k < kKeep; ++k)
        if (first + k * kPlaneThreads < last) store(first + k * kPlaneThreads, keep[k]);
    for (long long t = first + kKeep * kPlaneThreads; t < last; t += kPlaneThreads) {
        float v[V];
#pragma unroll
        for (int e = 0; e < V; ++e) v[e] = x[offset(t) + e];
        store(t, v);
    }
}
}  // namespace
}  // namespace ldn

using namespace ldn;

extern "C" LDN_API int ldn_mean_shift_rows(const float* x, int B, int C, float* running_mean, float momentum,
                                           float* out, float* mean_out, ldn_stream_t stream) {
    if (B < 0 || C <= 0) return kBadArgument;
    if (B == 0) return kOk;
    if (!x || !out) return kBadArgument;
    const DeviceCtx* ctx;
    int r = get_device_ctx(&ctx);
    if (r != kOk) return r;
    const unsigned blocks = static_cast<unsigned>((C + kCols - 1) / kCols);
    return launch_after(mean_shift_rows_kernel, blocks, kCols * kRowLanes, 0, reinterpret_cast<cudaStream_t>(stream),
                        x, out, running_mean, mean_out, momentum, B, C);
}

extern "C" LDN_API int ldn_mean_shift_planes(const float* x, int B, int C, int HW, float* running_mean, float momentum,
                                             float* out, ldn_stream_t stream) {
    if (B < 0 || C <= 0 || HW < 0 || C > 0x7fffffff / kCluster) return kBadArgument;
    if (B == 0 || HW == 0) return kOk;
    if (!x || !out) return kBadArgument;
    const bool vec = (HW & 3) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const unsigned grid = static_cast<unsigned>(C) * kCluster;
    return vec ? launch_after_in_clusters(mean_shift_planes_kernel<4>, kCluster, grid, kPlaneThreads, 0, st, x, out,
                                          running_mean, momentum, B, C, HW)
               : launch_after_in_clusters(mean_shift_planes_kernel<1>, kCluster, grid, kPlaneThreads, 0, st, x, out,
                                          running_mean, momentum, B, C, HW);
}
