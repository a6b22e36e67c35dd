// Work that follows a backward tile kernel beside its fold and needs nothing from the fold: the reduction of the fused
// backward's per-row-tile column sums, and the coefficients of the guard's second form.  Device functions over a range of
// blocks, so that they can share a launch with tile_fixup_kernel (ldn_tile.cuh): the integer-p backward pass takes 6 launches
// instead of 9 (64 x 784 -> 1024, p = 8, forward + backward: 104 -> 95 us; 512 x 3072 -> 5120: 3118 -> 3093 us, where the
// reduction, 60 us of it, also got 16-byte loads and four row tiles in flight).
#pragma once
#include "ldn_common.cuh"

namespace ldn {

constexpr int kPostBlock = 256;  // threads per block of every kernel that runs these jobs

// gw[i] = -sum_t part[t * count + i], t < tiles (added to gw when `accumulate`); runs only if gate is null or
// (*gate != 0) == run_if_nonzero
struct SideJob {
    const float* part;
    float* gw;
    long long count;
    int tiles;
    bool accumulate, vec;  // vec: count is a multiple of 4 and both arrays are 16-byte aligned
    bool wide;             // vec only: the warps of a block share the row tiles
    const int* gate;
    bool run_if_nonzero;
    int blocks;  // 0: no such job
};

// Coefficients of the general-p kernels, padded to whole tiles: a[g][row][c] = -q lg2 y (fold) or 1 / y, b = go.  Padding
// gets the offset -1e30 (folded form) or the factor 0 (1 / y form), which sends the power to (almost) zero whatever |t| the
// zero-filled partner operand produces, and a zero gradient factor.  Runs only if gate is null or *gate != 0.
struct CoefJob {
    const float* go;
    const float* y;
    float* a;
    float* b;
    Shape s;
    int pitch;
    long long rows_pad;
    float q;
    bool fold, flat;  // flat: source and destination have the same element order and whole, aligned vectors
    const int* gate;
    int blocks;       // 0: no such job
};

// index helpers -------------------------------------------------------------------------------
// canonical arrays are [g][m][pitch]; thread index runs over (g, m, c) with c fastest
struct CanonIdx {
    int g, c;
    long long m;
};
__device__ __forceinline__ CanonIdx canon_idx(long long i, int inner, long long M) {
    CanonIdx r;
    r.c = static_cast<int>(i % inner);
    const long long t = i / inner;
    r.m = t % M;
    r.g = static_cast<int>(t / M);
    return r;
}
// thread index runs over (g, m, o) with o fastest; source offset in output layout
__device__ __forceinline__ long long y_offset(const Shape& s, const CanonIdx& q) {
    const long long b = q.m / s.HW, hw = q.m % s.HW;
    if (s.co_src != s.CO) return (b * s.co_src + s.co_off + q.c) * s.HW + hw;  // channel range, G == 1
    return ((b * s.G + q.g) * s.COg + q.c) * s.HW + hw;
}

__device__ __forceinline__ void side_reduce_block(const SideJob& J, unsigned block, unsigned blocks) {
    if (J.gate && (*J.gate != 0) != J.run_if_nonzero) return;
    const long long first = block * (long long)kPostBlock + threadIdx.x, step = (long long)blocks * kPostBlock;
    if (J.wide) {
        __shared__ float4 sums[kPostBlock];
        const long long n4 = J.count / 4;
        const float4* part = reinterpret_cast<const float4*>(J.part);
        float4* gw = reinterpret_cast<float4*>(J.gw);
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        for (long long i0 = block * 32LL; i0 < n4; i0 += blocks * 32LL) {
            const long long i = i0 + lane;
            float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (i < n4) {
#pragma unroll 4
                for (int t = w; t < J.tiles; t += kPostBlock / 32) {
                    const float4 v = part[t * n4 + i];
                    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
                }
            }
            sums[threadIdx.x] = s;
            __syncthreads();
            if (w == 0 && i < n4) {
                for (int k = 1; k < kPostBlock / 32; ++k) {
                    const float4 v = sums[k * 32 + lane];
                    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
                }
                const float4 o = J.accumulate ? gw[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                gw[i] = make_float4(o.x - s.x, o.y - s.y, o.z - s.z, o.w - s.w);
            }
            __syncthreads();
        }
        return;
    }
    if (J.vec) {
        // bound by HBM / L2 reads: 16-byte loads, four row tiles in flight
        const long long n4 = J.count / 4;
        const float4* part = reinterpret_cast<const float4*>(J.part);
        float4* gw = reinterpret_cast<float4*>(J.gw);
        for (long long i = first; i < n4; i += step) {
            float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            int t = 0;
            for (; t + 4 <= J.tiles; t += 4) {
                float4 v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = part[(t + u) * n4 + i];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    s.x += v[u].x; s.y += v[u].y; s.z += v[u].z; s.w += v[u].w;
                }
            }
            for (; t < J.tiles; ++t) {
                const float4 v = part[t * n4 + i];
                s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
            }
            if (J.accumulate) {
                const float4 o = gw[i];
                gw[i] = make_float4(o.x - s.x, o.y - s.y, o.z - s.z, o.w - s.w);
            } else {
                gw[i] = make_float4(-s.x, -s.y, -s.z, -s.w);
            }
        }
        return;
    }
    for (long long i = first; i < J.count; i += step) {
        float s = 0.0f;
        for (int t = 0; t < J.tiles; ++t) s += J.part[t * J.count + i];
        J.gw[i] = J.accumulate ? J.gw[i] - s : -s;
    }
}

__device__ __forceinline__ void coef_gen_block(const CoefJob& J, unsigned block, unsigned blocks) {
    if (J.gate && *J.gate == 0) return;
    const long long first = block * (long long)kPostBlock + threadIdx.x, step = (long long)blocks * kPostBlock;
    if (J.flat) {
        const float4* y4 = reinterpret_cast<const float4*>(J.y);
        const float4* g4 = reinterpret_cast<const float4*>(J.go);
        const long long n4 = J.s.M * J.s.COg / 4;
        for (long long i = first; i < n4; i += step) {
            const float4 yv = y4[i];
            reinterpret_cast<float4*>(J.a)[i] =
                J.fold ? make_float4(-J.q * log2f(yv.x), -J.q * log2f(yv.y), -J.q * log2f(yv.z), -J.q * log2f(yv.w))
                       : make_float4(1.0f / yv.x, 1.0f / yv.y, 1.0f / yv.z, 1.0f / yv.w);
            reinterpret_cast<float4*>(J.b)[i] = g4[i];
        }
        return;
    }
    const long long total = static_cast<long long>(J.s.G) * J.rows_pad * J.pitch;
    for (long long i = first; i < total; i += step) {
        const CanonIdx ci = canon_idx(i, J.pitch, J.rows_pad);
        float off = J.fold ? -1e30f : 0.0f, gv = 0.0f;
        if (ci.m < J.s.M && ci.c < J.s.COg) {
            const long long src = y_offset(J.s, ci);
            off = J.fold ? -J.q * log2f(J.y[src]) : 1.0f / J.y[src];
            gv = J.go[src];
        }
        J.a[i] = off;
        J.b[i] = gv;
    }
}

}  // namespace ldn
