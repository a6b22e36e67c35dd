// Patches of an image batch as columns, and the adjoint sum: what NormDistConv does in front of and behind the distance
// operator (the reference calls torch's unfold there, core/modules/norm_dist.py:84-97).
//
//   unfold: cols[b, (c, ki, kj), (oh, ow)] = x[b, c, oh s - pad + ki d, ow s - pad + kj d]   (0 outside the image)
//   fold:   x[b, c, h, w] = sum of the column elements that unfold copies from that pixel, in ascending (oh, ow) order
//
// Both are bound by the bytes of `cols` (9 times the image for a 3 x 3 kernel): unfold writes them once, four
// neighbouring positions per thread and store where a row's length allows, fold reads them once, neighbouring threads
// reading neighbouring positions.  torch launches one unfold kernel per sample, so a batch of 128 small images costs 128
// launches: 128 x 64 channels of 16 x 16, 3 x 3 (75.5 MB of columns): unfold 767 us, fold 252 us there, and a layer step
// around them 1656 us instead of 413; three unfolds of 64 x 32 channels of 14 x 14 take 1099 us there (192 launches), the
// certification of that layer 1533 us instead of 133.
#include "ldn_b200.h"
#include "ldn_common.cuh"

namespace ldn {
namespace {

constexpr int kBlock = 256;

// n / d for 0 <= n < 2^31 by a multiplication and a shift (Granlund and Montgomery, PLDI 1994, section 4)
struct Divider {
    unsigned d, mul, shift;
};
Divider make_divider(unsigned d) {
    Divider r{d, 0, 0};
    while (r.shift < 32 && (1ull << r.shift) < d) ++r.shift;
    r.mul = static_cast<unsigned>(((1ull << 32) * ((1ull << r.shift) - d)) / d + 1);
    return r;
}
__device__ __forceinline__ unsigned quotient(unsigned n, const Divider& v) {
    return (__umulhi(n, v.mul) + n) >> v.shift;
}

struct Patches {
    int H, W, OH, OW, kh, kw, stride, pad, dil;
    Divider by_row;   // cols: vectors of positions in one row (b, c, ki, kj); x: pixels of one image plane
    Divider by_ow, by_kw, by_khkw, by_w, by_stride;
};

// Thread = V neighbouring positions of one row of `cols`; blockIdx.y splits the planes so that every index fits 31 bits.
template <int V>
__global__ void __launch_bounds__(kBlock) unfold_kernel(const float* x, float* cols, Patches P,
                                                        long long planes, unsigned planes_per_slice) {
    stream_order_begin();
    const long long plane0 = static_cast<long long>(blockIdx.y) * planes_per_slice;
    const unsigned here = static_cast<unsigned>(planes - plane0 < planes_per_slice ? planes - plane0 : planes_per_slice);
    const unsigned n = here * P.by_khkw.d * P.by_row.d;
    x += plane0 * (static_cast<long long>(P.H) * P.W);
    cols += plane0 * (static_cast<long long>(P.by_khkw.d) * P.by_row.d * V);
    for (unsigned i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
        const unsigned row = quotient(i, P.by_row);
        const unsigned l = (i - row * P.by_row.d) * V;
        const unsigned plane = quotient(row, P.by_khkw);
        const unsigned kk = row - plane * P.by_khkw.d;
        const unsigned ki = quotient(kk, P.by_kw), kj = kk - ki * P.by_kw.d;
        unsigned oh = quotient(l, P.by_ow), ow = l - oh * P.by_ow.d;
        const float* src = x + static_cast<long long>(plane) * P.H * P.W;
        float v[V];
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const int h = static_cast<int>(oh) * P.stride - P.pad + static_cast<int>(ki) * P.dil;
            const int w = static_cast<int>(ow) * P.stride - P.pad + static_cast<int>(kj) * P.dil;
            const bool in = h >= 0 && h < P.H && w >= 0 && w < P.W;
            v[e] = in ? src[h * P.W + w] : 0.0f;
            if (++ow == static_cast<unsigned>(P.OW)) {
                ow = 0;
                ++oh;
            }
        }
        float* dst = cols + static_cast<long long>(i) * V;
        if constexpr (V == 4) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        else dst[0] = v[0];
    }
}

// Thread = one pixel of one plane (b, c).
__global__ void __launch_bounds__(kBlock) fold_kernel(const float* cols, float* x, Patches P,
                                                      long long planes, unsigned planes_per_slice) {
    stream_order_begin();
    const long long plane0 = static_cast<long long>(blockIdx.y) * planes_per_slice;
    const unsigned n =
        static_cast<unsigned>(planes - plane0 < planes_per_slice ? planes - plane0 : planes_per_slice) * P.by_row.d;
    const int L = P.OH * P.OW;
    for (unsigned i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
        const unsigned pl = quotient(i, P.by_row);
        const unsigned pix = i - pl * P.by_row.d;
        const int h = static_cast<int>(quotient(pix, P.by_w)), w = static_cast<int>(pix) - h * P.W;
        const float* src = cols + (plane0 + pl) * (static_cast<long long>(P.kh) * P.kw * L);
        float s = 0.0f;
        // descending patch offsets are ascending output positions
        for (int ki = P.kh - 1; ki >= 0; --ki) {
            const int hs = h + P.pad - ki * P.dil;
            if (hs < 0) continue;
            const int oh = static_cast<int>(quotient(static_cast<unsigned>(hs), P.by_stride));
            if (oh >= P.OH || oh * P.stride != hs) continue;
            for (int kj = P.kw - 1; kj >= 0; --kj) {
                const int ws = w + P.pad - kj * P.dil;
                if (ws < 0) continue;
                const int ow = static_cast<int>(quotient(static_cast<unsigned>(ws), P.by_stride));
                if (ow >= P.OW || ow * P.stride != ws) continue;
                s += src[static_cast<long long>(ki * P.kw + kj) * L + oh * P.OW + ow];
            }
        }
        x[(plane0 + pl) * P.by_row.d + pix] = s;
    }
}

// The same at stride 1 for rows of whole 16-byte pieces: a thread sums four neighbouring pixels, so the index arithmetic of a
// patch offset serves four loads, which are in flight together (32 x 64 x 32 x 32, 3 x 3: 17 us instead of 52).
__global__ void __launch_bounds__(kBlock) fold_row_kernel(const float* cols, float* x, Patches P, long long planes,
                                                          unsigned planes_per_slice) {
    stream_order_begin();
    const long long plane0 = static_cast<long long>(blockIdx.y) * planes_per_slice;
    const unsigned n =
        static_cast<unsigned>(planes - plane0 < planes_per_slice ? planes - plane0 : planes_per_slice) * P.by_row.d;
    const int L = P.OH * P.OW;
    for (unsigned i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) {
        const unsigned pl = quotient(i, P.by_row);
        const unsigned pix = (i - pl * P.by_row.d) * 4;
        const int h = static_cast<int>(quotient(pix, P.by_w)), w = static_cast<int>(pix) - h * P.W;
        const float* src = cols + (plane0 + pl) * (static_cast<long long>(P.kh) * P.kw * L);
        float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int ki = P.kh - 1; ki >= 0; --ki) {
            const int oh = h + P.pad - ki * P.dil;
            if (oh < 0 || oh >= P.OH) continue;
#pragma unroll 3
            for (int kj = P.kw - 1; kj >= 0; --kj) {
                const int ow = w + P.pad - kj * P.dil;
                const float* row = src + static_cast<long long>(ki * P.kw + kj) * L + oh * P.OW + ow;
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (ow + e >= 0 && ow + e < P.OW) s[e] += row[e];
            }
        }
        *reinterpret_cast<float4*>(x + (plane0 + pl) * P.by_row.d * 4 + pix) = make_float4(s[0], s[1], s[2], s[3]);
    }
}

// Checks the geometry and fills it in.
int fill(Patches* P, int B, int C, int H, int W, int kh, int kw, int stride, int pad, int dil) {
    if (B < 0 || C <= 0 || H <= 0 || W <= 0 || kh <= 0 || kw <= 0 || stride <= 0 || pad < 0 || dil <= 0) return kBadArgument;
    constexpr long long kMax = (1LL << 30) - 1;
    const long long eh = H + 2LL * pad - dil * (kh - 1LL) - 1, ew = W + 2LL * pad - dil * (kw - 1LL) - 1;
    if (eh < 0 || ew < 0) return kBadArgument;
    const long long OH = eh / stride + 1, OW = ew / stride + 1;
    if (1LL * H * W > kMax || OH * OW > kMax || 1LL * kh * kw > kMax || OH * OW * kh * kw > kMax || H + 2LL * pad > kMax ||
        W + 2LL * pad > kMax)
        return kBadArgument;
    *P = Patches{H, W, static_cast<int>(OH), static_cast<int>(OW), kh, kw, stride, pad, dil, {}, {}, {}, {}, {}, {}};
    P->by_ow = make_divider(static_cast<unsigned>(OW));
    P->by_kw = make_divider(kw);
    P->by_khkw = make_divider(static_cast<unsigned>(kh) * kw);
    P->by_w = make_divider(W);
    P->by_stride = make_divider(stride);
    return kOk;
}

// Planes of `each` work items in slices of less than 2^30 items.
struct Slices {
    unsigned per_slice, count, blocks;
};
int slice(long long planes, unsigned each, Slices* s) {
    const long long per = ((1LL << 30) - 1) / each;  // at least 1: fill() bounds a plane
    const long long count = (planes + per - 1) / per;
    if (count > 65535) return kBadArgument;
    s->per_slice = static_cast<unsigned>(planes < per ? planes : per);
    s->count = static_cast<unsigned>(count);
    const long long blocks = (static_cast<long long>(s->per_slice) * each + kBlock - 1) / kBlock;
    s->blocks = static_cast<unsigned>(blocks < (1 << 20) ? blocks : (1 << 20));
    return kOk;
}

}  // namespace
}  // namespace ldn

using namespace ldn;

extern "C" {

LDN_API int ldn_unfold(const float* x, int B, int C, int H, int W, int kh, int kw, int stride, int pad, int dil, float* cols,
                       ldn_stream_t stream) {
    Patches P;
    int r = fill(&P, B, C, H, W, kh, kw, stride, pad, dil);
    if (r != kOk) return r;
    if (B == 0) return kOk;
    if (!x || !cols) return kBadArgument;
    const int L = P.OH * P.OW;
    const bool vec = (L & 3) == 0 && (reinterpret_cast<uintptr_t>(cols) & 15u) == 0;
    P.by_row = make_divider(static_cast<unsigned>(vec ? L / 4 : L));
    const long long planes = static_cast<long long>(B) * C;
    Slices s;
    if ((r = slice(planes, P.by_khkw.d * P.by_row.d, &s)) != kOk) return r;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const dim3 grid(s.blocks, s.count);
    if (vec) return launch_after(unfold_kernel<4>, grid, kBlock, 0, st, x, cols, P, planes, s.per_slice);
    return launch_after(unfold_kernel<1>, grid, kBlock, 0, st, x, cols, P, planes, s.per_slice);
}

LDN_API int ldn_fold(const float* cols, int B, int C, int H, int W, int kh, int kw, int stride, int pad, int dil, float* x,
                     ldn_stream_t stream) {
    Patches P;
    int r = fill(&P, B, C, H, W, kh, kw, stride, pad, dil);
    if (r != kOk) return r;
    if (B == 0) return kOk;
    if (!x || !cols) return kBadArgument;
    const bool vec = stride == 1 && (W & 3) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    P.by_row = make_divider(static_cast<unsigned>(vec ? H * W / 4 : H * W));
    const long long planes = static_cast<long long>(B) * C;
    Slices s;
    if ((r = slice(planes, P.by_row.d, &s)) != kOk) return r;
    const dim3 grid(s.blocks, s.count);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (vec) return launch_after(fold_row_kernel, grid, kBlock, 0, st, cols, x, P, planes, s.per_slice);
    return launch_after(fold_kernel, grid, kBlock, 0, st, cols, x, P, planes, s.per_slice);
}

}  // extern "C"
