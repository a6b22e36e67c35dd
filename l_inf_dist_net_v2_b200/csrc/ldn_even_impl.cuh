// Even integer exponents on the tensor cores.
//
// For even p the distance is a polynomial:
//   y^p            = sum_c x^p + sum_c w^p + sum_{j=1}^{p-1} (-1)^j C(p, j) sum_c x^j w^(p-j)
//   grad_x[b, c]   = sum_j (-1)^j C(p-1, j) d^(p-1-j) sum_o A[b, o] u[o, c]^j,      A = go / y^(p-1)
//   grad_w[o, c]   = sum_j (-1)^j C(p-1, j) d^(p-1-j) sum_b A[b, o] u[b, c]^j
// with u = w - m, d = x - m for grad_x and u = x - m, d = w - m for grad_w, m[c] about the mean of the channel in the operand
// that is summed over.  That is p - 1 matrix products each.  Every factor is split into two 11-bit halves, v = hi + lo in fp16 (lo holds what hi
// rounds off, so the pair keeps 22 - 23 bits), and a product is hi hi + hi lo + lo hi with fp32 accumulators (and lo lo for
// p = 2): 3 x 7 multiply-adds per pair on the tensor cores for p = 8, against 4 (forward) and 8 (backward) FP32 instructions of
// the direct kernels.  In the forward pass the terms do not cancel where it matters: large |x - w| come from x and w of opposite
// sign, for which all terms of the expansion have one sign (a guard looks at every output).  In the backward pass the errors go
// with E = sum |A| (|d| + |u|)^(p-1) and the direct kernels' with D = sum |A| |d - u|^(p-1).  Around the mean the two are close
// whatever the channel holds: |m - x| <= ||d - u|| in the (p-1)-norm over the rows, so ||d| + |u|| <= 3 ||d - u|| at worst, and
// E is about 2 D for channels of any offset or spread, a few of the rows far from the others, or values that hardly differ.
// (Around zero, p = 8: entries of grad_w at pixels 0.5 +- 0.02 were wrong by 1.3e-2 at the 90th percentile, channels of offset
// 1.5 by 4e-3 in 2-norm.)  What may still go wrong is that the coefficients prefer rows near x: the guards below.
//
// What is kept as precise as in the direct kernels, and how:
//   * the tensor core's accumulator drops the bits below the largest summand instead of rounding, so it takes one stage
//     at a time and the sums are added up in registers.  What 64 elements' products lose that way is 2.0e-7 - 2.8e-7 of
//     their sum in the forward pass (p = 4 and 8, 128 - 3072 channels, images and zero-mean activations, against 64 bits),
//     always towards zero: kTruncation gives it back there.  What is left of it in the values, on average: between -5e-9 and 1.5e-8
//     of them for p = 2, 4, 6 and 8, 256 - 3000 channels, pairs' tiles and split ones, images, activations and operands of opposite
//     signs.  (Root mean square errors 2.0e-8 - 4.3e-8, direct kernels 4e-8 - 4e-7; the largest of one output of 4 M 1.1e-6 at
//     p = 8 and 256 channels, where direct ones have 2.6e-7, 1e-7 - 6e-7 from 576 channels on, 2e-7 - 2.3e-6.)  (The backward pass's sums, whose terms have either sign, show no
//     such drift.)
//   * powers are scaled into fp16's range: by one power of two for both operands in the forward pass (all terms of the sum
//     share it), by one per channel and one per coefficient row in the backward pass;
//   * forward: an output for which the terms could cancel, y^p < r (|x|_p + |w|_p)^p (least_of_norms says with which r), or that is
//     small on the common scale, y^p < 2^-10 M^p with the largest magnitude M, goes to a list and is summed directly; too many of
//     them, or a value that is not finite, and the direct kernels behind this path run instead.  Where that is to be expected it is
//     known before the products: from sampled outputs, and from rows whose norms are small on the common scale;
//   * backward: the direct kernels run if the coefficients of a row (of x, or of w) sit on few of its terms, sum |A| < 4 max |A|;
//     if they prefer small differences in all channels at once, as within clusters: an output below kLeastOfSpread (by p) of
//     (sum_c s^p)^(1/p), s[c] the root mean square of x - w over all pairs; if an output is below a third of the largest |d| + |u|
//     of a channel (rows of different scales: powers of the small ones would leave fp16's range); or if a channel's u are
//     below 2^-12 of its d without being 0.
//     Errors against 64 bits, 512 x 1536 -> 2048, p = 8, products / direct kernels, 2-norm (99th percentile of the entries'
//     relative errors): grad_x of images 2.4e-7 / 7.6e-7 (1.2e-5 / 2.6e-5), grad_w 2.4e-7 / 2.8e-7 (1.2e-5 / 1.7e-5), of pixels
//     0.5 +- 0.02 2.3e-7 / 2.7e-7 (1.1e-5 / 1.7e-5), both operands in [1, 2) 2.4e-7 / 2.3e-7 (1.4e-5 / 1.4e-5).  Two clusters of
//     Gaussian rows, as far apart as they are wide, lie at 1.03 (sum_c s^p)^(1/p) and would have 6.2e-7 / 2.9e-7; at half that width,
//     0.59, 3.0e-6 / 3.4e-7.  Rows whose channels are independent of one another lie at 1.24 and above (1.14, 1.0, 0.78 at
//     p = 6, 4, 2; 192 - 1024 channels, uniform, normal, of zeros and ones).
#pragma once
#include <float.h>
#include <math.h>

#include "ldn_even.cuh"

namespace ldn {
namespace {

constexpr int kMRows = 128;                 // rows of A per CTA = TMEM lanes
constexpr int kNRows = 224;                 // widest B tile: 7 powers of 32 channels, or 224 rows
constexpr int kBlockK = 32;                 // reduction elements of a block: a row of one is 32 hi | 32 lo, 128 bytes
constexpr int kABytes = kMRows * 128;       // a block of A as shared memory holds it (128-byte swizzle)
constexpr int kEpiWarps = 8, kConvWarps = 7;
constexpr int kEvenThreads = 32 * (kEpiWarps + kConvWarps + 1);
constexpr float kScaleB = 32768.0f;         // backward: powers of values below 1 as fp16 holds them best
constexpr float kTruncation = 1.0f + 1.0f / (1 << 22);
constexpr int kListCap = 1 << 16;
constexpr int kGuardSamples = 64;  // sampled outputs of the forward form, and how many of them below the line say that the list
constexpr int kMostBelow = 8;      // will not do (it holds a 40th of 512 x 5120 outputs: 8 of 64 then by chance 3 times in 10^4)
// guards of the backward form
constexpr float kLeastSpread = 4.0f;       // sum of |A| over its largest, per row
__device__ __forceinline__ double least_of_spread(int p) { return p == 8 ? 1.1 : (p == 6 ? 1.05 : (p == 4 ? 0.7 : 0.5)); }
constexpr float kMostOfOutput = 3.0f;      // largest |d| + |u| of a channel over y
constexpr float kLeastChannel = 1.0f / 4096;   // largest |u| over largest |d|
constexpr float kChannelFloor = 1.0f / 512;    // scales: d stays below 512, d^7 times the sums below 2^127

// A tile is the work of a pair of CTAs: 256 rows of A, kNRows of B, half of either in each CTA.
constexpr int kBlocks = 2;                             // blocks of 32 reduction elements per stage
constexpr int kStageK = kBlocks * kBlockK;
constexpr int kStages = 3;
constexpr int kRowsB = kNRows / 2;                     // rows of B in a CTA
// bytes of a block of B in a CTA; of a stage: all blocks of A, then all blocks of B
__host__ __device__ constexpr int b_bytes(bool fwd, int np);
__host__ __device__ constexpr int stage_bytes(bool fwd, int np) { return kBlocks * (kABytes + b_bytes(fwd, np)); }
// backward: the resident operand of a tile (32 kEpiWarps threads, half of the tile's channels each), the channels' scales and shifts
__host__ __device__ constexpr int resident_bytes(int ct) { return 32 * kEpiWarps * (ct / 2) * 4; }
__host__ __device__ constexpr int even_smem(bool fwd, int np);

// Channels per tile of the backward form: (p - 1) * channels rows of B, at most kNRows
__host__ __device__ constexpr int channels_of(int np) { return np >= 5 ? 32 : (np == 3 ? 64 : 128); }

__host__ __device__ constexpr int b_bytes(bool fwd, int np) { return (fwd ? kRowsB : np * channels_of(np) / 2) * 128; }
__host__ __device__ constexpr int even_smem(bool fwd, int np) {
    return kStages * stage_bytes(fwd, np) + 1024 + 256 + (fwd ? 0 : resident_bytes(channels_of(np)) + kEpiWarps * (channels_of(np) / 2) * 8);
}

__host__ __device__ constexpr float binomial(int n, int k) {
    float r = 1.0f;
    for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
    return r;
}

// An fp32 operand as the converters read it.  Element (row, k) of group g:
//   kind 0 / 1: p[g * s_g + row * s_row + k] (s_k = 1), 0: in aligned 16-byte pieces
//   kind 2:     p[g * s_g + (row / hw) * s_b + (row % hw) * s_row + k * s_k], without the division where hw is 0
//   kind 3 / 4: p[g * s_g + row * s_row + (k / hw) * s_b + k % hw], 4: in aligned 16-byte pieces
struct Source {
    const float* p;
    int kind, rows, k, hw;
    long long s_row, s_k, s_b, s_g;
};

struct EvenParams {
    int M, N, G;                    // per group: rows of A, rows of B (forward) or channels (backward)
    int tiles_m, tiles_n, kt;       // kt: stages per tile
    int blocks;                     // forward: blocks of 32 channels times powers, in this order
    int total;                      // stages in all
    const char* images;             // A: [g][block of rows][block of the reduction ([power], forward)], kABytes each
    Source src;                     // B
    OutAddr out;
    bool split;                     // at most 128 rows of A: the pair's first CTA has their hi, the second their lo
    int slots;                      // partial sums that a CTA may have to keep (split: one per tile that its range touches)
    bool swap;                      // forward: the output's row is the tile's column
    bool vec;                       // columns n .. n + 3 (n a multiple of 4) of an output row are one aligned 16-byte piece
    bool accumulate;
    float* out_f;
    // forward
    const float *sum_a, *norm_a, *sum_b, *norm_b;  // row sums of p-th powers on the common scale and their p-th roots
    const unsigned* scale_word;     // bits of the largest magnitude
    float least;                    // of the guard on the norms (least_of_norms)
    int* list;                      // outputs to be summed directly
    int* list_count;
    int* dense;
    // backward
    const float* resident;          // the operand with the output's layout
    const float *col_down, *col_shift; // [g][channel, padded to whole tiles]: v = (value - m) 2^-e = value * down + shift
    const int* row_exp;             // [g][row]: coefficients are scaled by 2^exp
    const float* row_sum;           // [g][row]: sum of the scaled coefficients
    const int *gate0, *gate1;       // run only while both words are 0 (may be null)
    float* partials;                // [cta][slots][columns][kMRows]
    int* status;
};

// ---- tcgen05 ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* slot) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(base) : "memory");
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t desc, bool add) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(desc), "r"(static_cast<uint32_t>(add))
        : "memory");
}
// arrival on the barrier of both CTAs when the products issued so far are done
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
        "h"(static_cast<uint16_t>(3))
        : "memory");
}
__device__ __forceinline__ void tmem_load16(uint32_t addr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// (the registers are operands, so that nothing that uses them moves in front of the wait)
__device__ __forceinline__ void tmem_load_wait(float (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]), "+f"(v[8]),
                   "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]), "+f"(v[15])
                 :
                 : "memory");
}
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// arrival on the same barrier of the pair's first CTA
__device__ __forceinline__ void mbar_arrive_first(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\t"
        "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}" ::"r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// K-major operand, rows of 128 bytes in groups of 8 (1024 bytes apart), 128-byte swizzle
__device__ __forceinline__ uint64_t smem_desc(const void* p) {
    return static_cast<uint64_t>((smem_u32(p) & 0x3ffffu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// fp16 x fp16 -> fp32, both operands K-major
__host__ __device__ constexpr uint32_t mma_desc(int m, int n) {
    return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// ---- splitting -------------------------------------------------------------------------------------------------------
// eight values as 16 bytes of hi and 16 bytes of lo
__device__ __forceinline__ void split8(const float2 (&v)[4], uint4* hi, uint4* lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h[i]) : "f"(v[i].y), "f"(v[i].x));
        float2 f;
        asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.f32.f16 %0, a;\n\tcvt.f32.f16 %1, b;\n\t}"
            : "=f"(f.x), "=f"(f.y)
            : "r"(h[i]));
        const float2 d = __ffma2_rn(f, make_float2(-1.0f, -1.0f), v[i]);
        asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(l[i]) : "f"(d.y), "f"(d.x));
    }
    *hi = make_uint4(h[0], h[1], h[2], h[3]);
    *lo = make_uint4(l[0], l[1], l[2], l[3]);
}
__device__ __forceinline__ float2 scale2(float2 v, float s) { return __fmul2_rn(v, make_float2(s, s)); }
template <int P>
__device__ __forceinline__ float power(float v) {
    if constexpr (P == 1) return v;
    else if constexpr (P % 2 == 0) {
        const float h = power<P / 2>(v);
        return h * h;
    } else {
        return power<P - 1>(v) * v;
    }
}
// v^(1/P), rounded (almost) once: what a square root's rounding took is carried on to the next
template <int P>
__device__ __forceinline__ float root(float v) {
    if constexpr (P == 6) return cbrtf(sqrtf(v));
    float low = 0.0f;  // v + low is the value so far
#pragma unroll
    for (int i = P; i > 1; i /= 2) {
        const float inv = rsqrtf(v), r = v * inv;
        low = 0.5f * (fmaf(-r, r, v) + low) * inv;
        v = r;
    }
    return v + low;
}
// 2^e, |e| <= 126
__device__ __forceinline__ float pow2i(int e) { return __int_as_float((e + 127) << 23); }
// 2^(n e) from 2^-e, |n e| <= 126
template <int N>
__device__ __forceinline__ float up_of(float down) {
    return pow2i(N * (127 - (__float_as_int(down) >> 23)));
}
// smallest e with 2^e > v, from the bits of |v|
__device__ __forceinline__ int exponent_above(unsigned bits) { return static_cast<int>(bits >> 23) - 126; }

__device__ __forceinline__ const float* source_row(const Source& S, int g, int row) {
    if (row >= S.rows) return nullptr;
    const float* p = S.p + g * S.s_g;
    if (S.kind == 2 && S.hw > 0) {
        const int b = row / S.hw;
        return p + b * S.s_b + (row - b * S.hw) * S.s_row;
    }
    return p + row * S.s_row;
}
// Loads into registers that hold 0 where there is nothing to load.  (As predicated instructions on the destination itself: a
// conditional in C++ ends in moves behind the loads, and those wait for them, a thousand cycles per prefetch.)
__device__ __forceinline__ void load1(float* v, const float* p, bool there) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.global.f32 %0, [%1];\n\t}"
                 : "+f"(*v)
                 : "l"(p), "r"(static_cast<uint32_t>(there)));
}
__device__ __forceinline__ void load4(float2* v, const float* p, bool there) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t@q ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "+f"(v[0].x), "+f"(v[0].y), "+f"(v[1].x), "+f"(v[1].y)
                 : "l"(p), "r"(static_cast<uint32_t>(there)));
}
// elements k0 .. k0 + 7 of a row (k0 a multiple of 8); 0 outside
__device__ __forceinline__ void fetch8(const Source& S, const float* row, int k0, float2 (&v)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = make_float2(0.0f, 0.0f);
    const int left = row == nullptr ? 0 : S.k - k0;
    if (S.kind == 1 || S.kind == 2) {
        const float* p = row + k0 * S.s_k;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            load1(i % 2 ? &v[i / 2].y : &v[i / 2].x, p, left > i);
            p += S.s_k;
        }
    } else if (S.kind == 0) {
        load4(v, row + k0, left > 0);
        load4(v + 2, row + k0 + 4, left > 4);
    } else if (S.kind == 4) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int k = k0 + 4 * i, b = k / S.hw;
            load4(v + 2 * i, row + b * S.s_b + (k - b * S.hw), left > 4 * i);
        }
    } else {
        const int b = k0 / S.hw;
        int r = k0 - b * S.hw;
        const float* p = row + b * S.s_b + r;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            load1(i % 2 ? &v[i / 2].y : &v[i / 2].x, p, left > i);
            ++p;
            if (++r == S.hw) {
                r = 0;
                p += S.s_b - S.hw;
            }
        }
    }
}

// ---- where results go ------------------------------------------------------------------------------------------------
__device__ __forceinline__ long long even_offset(const EvenParams& P, int g, int m, int n) {
    const int r = P.swap ? n : m, c = P.swap ? m : n;
    const int q = P.out.hw_div == 1 ? r : r / P.out.hw_div;
    return q * P.out.s_b + (r - q * P.out.hw_div) * P.out.s_hw + g * P.out.s_g + c * P.out.s_n;
}

// Scales of the forward form, from the largest magnitude M of both operands.  With unit = 2^e > M and values v = value / unit,
// the factors of term j are C(p, j) x^j 2^a(j) and w^(p-j) 2^b(j), both below 2^16, with a(j) + b(j) = total for all j.
template <int PW>
struct ForwardScale {
    int e, total;
    float bits, top;  // bits = log2(unit / M), top = M / unit in [0.5, 1)
    __device__ __forceinline__ explicit ForwardScale(unsigned word) {
        e = exponent_above(word);
        top = __uint_as_float((word & 0x7fffffu) | 0x3f000000u);
        bits = -log2f(top) * 0.9999f;
        total = 1000;
#pragma unroll
        for (int j = 1; j < PW; ++j)
            total = min(total, static_cast<int>(floorf(15.9f + j * bits - log2f(binomial(PW, j)))) + b(PW - j));
    }
    __device__ __forceinline__ int b(int exponent) const { return 15 + static_cast<int>(exponent * bits); }
    __device__ __forceinline__ int a(int j) const { return total - b(PW - j); }
};

// A sum of the forward form -> the output value; outputs that may have lost bits go to the list.
struct ForwardEnd {
    float from_acc, least, unit;  // accumulated units -> sums; smallest sum that is large enough on the common scale
};
template <int PW>
__device__ __forceinline__ ForwardEnd forward_end(const EvenParams& P) {
    const ForwardScale<PW> f(*P.scale_word);
    return ForwardEnd{pow2i(-f.total) * kTruncation, power<PW>(f.top) * (1.0f / 1024), pow2i(f.e)};
}
template <int PW>
__device__ __forceinline__ float forward_value(const EvenParams& P, const ForwardEnd& E, float acc, float sa, float na, float sb,
                                               float nb, int off) {
    const float s = fmaf(acc, E.from_acc, sa + sb);
    const float least = fmaxf(E.least, power<PW>(na + nb) * P.least);
    if (!(s >= least) && *static_cast<volatile int*>(P.dense) == 0) {
        const int at = atomicAdd(P.list_count, 1);
        if (at < kListCap) P.list[at] = off;
        else *P.dense = 1;
    }
    return root<PW>(s) * E.unit;
}

struct Span {
    int g, tm, tn, kt0, kt1;  // stages [kt0, kt1) of one tile
};
__device__ __forceinline__ Span span_at(const EvenParams& P, int it, int end) {
    Span s;
    const int t = it / P.kt;
    s.kt0 = it - t * P.kt;
    s.kt1 = min(P.kt, s.kt0 + end - it);
    const int per_group = P.tiles_m * P.tiles_n;
    s.g = t / per_group;
    const int r = t - s.g * per_group;
    s.tn = r / P.tiles_m;
    s.tm = r - s.tn * P.tiles_m;
    return s;
}
// first stage of unit (CTA or pair) i of n
__device__ __forceinline__ int even_begin(const EvenParams& P, int n, int i) {
    return static_cast<int>(static_cast<long long>(P.total) * i / n);
}

// The blocks of A of stage kt of a tile, for CTA `rank` of its pair.
__device__ __forceinline__ const char* a_blocks(const EvenParams& P, const Span& s, int kt, int rank) {
    const int row_block = (s.g * P.tiles_m + s.tm) * 2 + rank;  // (split: of the same rows, with hi and lo exchanged)
    return P.images + (static_cast<long long>(row_block) * P.kt + kt) * static_cast<long long>(kBlocks * kABytes);
}

struct Bars {
    uint64_t full[kStages], empty[kStages];
    uint64_t peer_full[kStages];  // of the pair's first CTA: the second CTA's part of the stage is there
    uint64_t acc_full[2], acc_empty[2];
    uint32_t tmem;
    int abort;
};

template <bool CLUSTER>
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, int* abort, int* status) {
    for (uint32_t i = 0; i < kMaxPolls; ++i) {
        if (CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity)) return true;
        if (i >= kFastPolls) {
            if (*static_cast<volatile int*>(abort)) return false;
            __nanosleep(64);
        }
    }
    *static_cast<volatile int*>(abort) = 1;
    *status = kDeviceTimeout;
    return false;
}

// FWD: powers run along the reduction (all powers of 32 channels, then of the next 32; a stage = kBlocks of these blocks),
// B = rows of the larger operand.
// !FWD: powers run along the tile's columns, a stage = kBlocks * 32 rows of the operand.  The columns are two halves (the rows
// of B of the two CTAs of a pair), each p - 1 powers of CT / 2 channels.
//
// 16 warps and one CTA per SM, every pair with an equal share of all tiles' stages (a tile that is shared leaves partial sums
// for the fold).  Warps 0 - 7 add up accumulators and finalise, warps 8 - 14 turn fp32 values into the powers' hi and lo and
// ask for the blocks of A, warp 15 issues the products in the pair's first CTA (its second CTA's passes on that its part of
// a stage is there).
//
// Problems of at most 128 rows of A (128 output channels of a convolution, small batches) are split otherwise: both CTAs take the
// same rows, the first their hi, the second their lo, so that a product is two passes, A hi and lo times B lo and B hi, instead
// of three with half of the rows empty; both leave partial sums, which the fold adds.
//
// What bounds it: the products, 1344 cycles per stage at 224 columns (alone, on random data: 2.0 PFLOP/s at the clock that
// the power limit leaves).  Measured in the middle of a tile: 1550 cycles per stage.  Why a pair: the products of one CTA read
// 1056 x 128 bytes of shared memory per 1344 cycles, beside 256 of copies of A and 448 of stores of B; of a pair, whose CTAs
// hold half of B each, 720, 256 and 224 (512 x 3072 -> 5120, p = 8, forward / grad_x / grad_w: 488 / 331 / 369 us with single
// CTAs, 374 / 300 / 370 with pairs).  What made the difference after that (now 232 / 222 / 286): a remote arrival without
// cluster-wide release (1150 cycles each), prefetching loads that nothing behind them waits for (950 cycles), loops that stay
// in the instruction cache, forward powers from one another instead of from the value (248 -> 232).  The forward form's
// converters, 2080 cycles per stage, are what bounds it now; 222 us are 1.5 PFLOP/s.
template <int PW, bool FWD>
__global__ void __launch_bounds__(kEvenThreads, 1) even_kernel(const EvenParams P) {
    constexpr int NP = PW - 1;
    constexpr int CT = channels_of(NP);
    constexpr int COLS = FWD ? kNRows : NP * CT;    // columns of the accumulator
    constexpr int NC = COLS / 2;                    // of which a warp adds up
    constexpr int CW = CT / 2;                      // !FWD: channels of a half, which one CTA converts
    constexpr int kBBytes = b_bytes(FWD, NP), kStageBytes = stage_bytes(FWD, NP);
    constexpr int UNITS = CW * kBlocks / 8;         // !FWD: converter units (32 items of 8 reduction elements) per stage
    // (A barrier's parity tells a phase from its neighbours only: a converter warp's units have to lie less than kStages stages
    // apart, or it may take the phase before for the one that it waits for.)
    static_assert(FWD || kConvWarps < kStages * UNITS, "units of a warp too far apart");
    extern __shared__ __align__(16) char raw[];
    char* smem = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
    Bars* B = reinterpret_cast<Bars*>(smem + kStages * kStageBytes);
    stream_order_begin();
    if ((P.gate0 && *P.gate0 != 0) || (P.gate1 && *P.gate1 != 0)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1;
    const int workers = gridDim.x / 2, worker = blockIdx.x / 2;
    const int it0 = even_begin(P, workers, worker), it1 = even_begin(P, workers, worker + 1);
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&B->full[i], 1 + (FWD ? kConvWarps : UNITS));
            mbar_init(&B->peer_full[i], 1);
            mbar_init(&B->empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&B->acc_full[i], 1);
            mbar_init(&B->acc_empty[i], kEpiWarps * 2);
        }
        B->abort = 0;
        mbar_fence_init();
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(&B->tmem);
    tmem_fence_before();
    cluster_sync();
    tmem_fence_after();
    const uint32_t tmem = B->tmem;

    if (warp < kEpiWarps) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 160;");
        const int quad = warp & 3, half = warp >> 2, row = quad * 32 + lane;
        const uint32_t taddr = tmem + (static_cast<uint32_t>(quad * 32) << 16) + half * NC;
        const int first_tile = it0 / P.kt;
        [[maybe_unused]] char* resident = reinterpret_cast<char*>(B) + 256;  // [piece of 4 channels][thread], 16 bytes each
        [[maybe_unused]] char* scales = resident + resident_bytes(CT) + warp * CW * 8;  // 2^-e, then shifts
        int buf = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int it = it0; it < it1 && ok;) {
            const Span s = span_at(P, it, it1);
            float2 acc[NC / 2];
#pragma unroll
            for (int i = 0; i < NC / 2; ++i) acc[i] = make_float2(0.0f, 0.0f);
            const int m = (P.split ? s.tm : s.tm * 2 + rank) * kMRows + row;
            const bool in = m < P.M;
            [[maybe_unused]] const int n0 = s.tn * CT + half * CW;  // backward: first channel
            [[maybe_unused]] long long off = 0;
            [[maybe_unused]] float q0 = 0.0f, row_exp = 0.0f;
            if constexpr (!FWD) {
                // what the end of the tile needs, fetched meanwhile (each thread reads back what it copied, a warp its scales)
                off = even_offset(P, s.g, in ? m : 0, n0);
                __syncwarp();
#pragma unroll
                for (int c = 0; c < CW; c += 4) {
                    if (P.vec) {
                        copy_async<16>(resident + (c / 4 * 32 * kEpiWarps + threadIdx.x) * 16, P.resident + off + c, in && n0 + c < P.N ? 16 : 0);
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            copy_async<4>(resident + (c / 4 * 32 * kEpiWarps + threadIdx.x) * 16 + 4 * i, P.resident + off + (c + i) * P.out.s_n,
                                          in && n0 + c + i < P.N ? 4 : 0);
                    }
                }
                if (lane < CW / 2) {
                    const int q = lane % (CW / 4);
                    copy_async<16>(scales + lane * 16, (lane < CW / 4 ? P.col_down : P.col_shift) + s.g * P.tiles_n * CT + n0 + 4 * q, 16);
                }
                load1(&row_exp, reinterpret_cast<const float*>(P.row_exp) + s.g * P.M + m, in);
                load1(&q0, P.row_sum + s.g * P.M + m, s.kt0 == 0 && in && !(P.split && rank == 1));
            }
            for (int kt = s.kt0; kt < s.kt1; ++kt) {
                ok = __all_sync(0xffffffffu, wait_or_abort<false>(&B->acc_full[buf], phase, &B->abort, P.status));
                if (!ok) break;
                tmem_fence_after();
#pragma unroll
                for (int q = 0; q < NC; q += 32) {
                    float v[2][16];
                    const bool two = q + 16 < NC;
                    tmem_load16(taddr + buf * 256 + q, v[0]);
                    if (two) tmem_load16(taddr + buf * 256 + q + 16, v[1]);
                    tmem_load_wait(v[0]);
                    if (two) tmem_load_wait(v[1]);
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (i < 8 || two) {
                            const float2 sum = make_float2(v[i / 8][2 * (i % 8)], v[i / 8][2 * (i % 8) + 1]);
                            if constexpr (FWD) {
                                acc[q / 2 + i] = __fadd2_rn(acc[q / 2 + i], sum);
                            } else {  // the power's coefficient (-1)^j C(p - 1, j) in the same instruction
                                const int j = (q + 2 * i) / CW + 1;
                                const float k = j % 2 ? -binomial(NP, j) : binomial(NP, j);
                                acc[q / 2 + i] = __ffma2_rn(sum, make_float2(k, k), acc[q / 2 + i]);
                            }
                        }
                }
                tmem_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_first(&B->acc_empty[buf]);
                buf ^= 1;
                if (buf == 0) phase ^= 1;
            }
            if (!ok) break;
            const bool whole = s.kt0 == 0 && s.kt1 == P.kt && !P.split;
            const int slot = P.split ? it / P.kt - first_tile : (it / P.kt == first_tile ? 0 : 1);
            float* part = P.partials + (static_cast<size_t>(blockIdx.x) * P.slots + slot) * static_cast<size_t>(FWD ? kNRows : CT) * kMRows + row;
            if constexpr (FWD) {
                if (!whole) {
#pragma unroll
                    for (int i = 0; i < NC / 2; ++i) {
                        part[(half * NC + 2 * i) * kMRows] = acc[i].x;
                        part[(half * NC + 2 * i + 1) * kMRows] = acc[i].y;
                    }
                } else if (in) {
                    // the sums as they are; even_fold_kernel makes values of them (the roots and guards of a tile here would
                    // hold its CTA up for as long as ten stages)
#pragma unroll
                    for (int q = 0; q < NC; q += 4) {
                        const int n = s.tn * kNRows + half * NC + q;
                        if (P.vec) {
                            if (n < P.N)
                                *reinterpret_cast<float4*>(P.out_f + even_offset(P, s.g, m, n)) =
                                    make_float4(acc[q / 2].x, acc[q / 2].y, acc[q / 2 + 1].x, acc[q / 2 + 1].y);
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (n + i < P.N)
                                    P.out_f[even_offset(P, s.g, m, n + i)] = i % 2 ? acc[q / 2 + i / 2].y : acc[q / 2 + i / 2].x;
                        }
                    }
                }
            } else {
                // Horner's scheme over the powers.  The next tile's products run on meanwhile, but only for two accumulators, 2700
                // cycles, so a tile's end has to be short: the coefficients came with the sums, the resident operand waits in
                // shared memory.  (512 x 3072 -> 5120, weight gradient, tiles of 8 stages: 7500 cycles and 297 us with a rolled
                // loop that loaded and multiplied them here, 5400 and 286 now.)
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
                const float row_scale = pow2i(-15 - __float_as_int(row_exp));
                const float2 start = scale2(make_float2(q0, q0), kScaleB);
                float* out = P.out_f + off;
#pragma unroll
                for (int c = 0; c < CW; c += 4) {
                    const float4 u = *reinterpret_cast<const float4*>(resident + (c / 4 * 32 * kEpiWarps + threadIdx.x) * 16);
                    const float4 d = *reinterpret_cast<const float4*>(scales + c * 4);
                    const float4 t = *reinterpret_cast<const float4*>(scales + (CW + c) * 4);
                    const float2 x0 = __ffma2_rn(make_float2(u.x, u.y), make_float2(d.x, d.y), make_float2(t.x, t.y));
                    const float2 x1 = __ffma2_rn(make_float2(u.z, u.w), make_float2(d.z, d.w), make_float2(t.z, t.w));
                    float2 h0 = start, h1 = start;
#pragma unroll
                    for (int j = 0; j < NP; ++j) {
                        h0 = __ffma2_rn(h0, x0, acc[(j * CW + c) / 2]);
                        h1 = __ffma2_rn(h1, x1, acc[(j * CW + c) / 2 + 1]);
                    }
                    if (!whole) {
                        float* o = part + (half * CW + c) * kMRows;
                        o[0] = h0.x; o[kMRows] = h0.y; o[2 * kMRows] = h1.x; o[3 * kMRows] = h1.y;
                    } else if (in && n0 + c < P.N) {
                        h0 = __fmul2_rn(scale2(h0, row_scale), make_float2(up_of<NP>(d.x), up_of<NP>(d.y)));
                        h1 = __fmul2_rn(scale2(h1, row_scale), make_float2(up_of<NP>(d.z), up_of<NP>(d.w)));
                        if (P.vec) {
                            float4* o = reinterpret_cast<float4*>(out + c);
                            const float4 old = P.accumulate ? *o : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                            *o = make_float4(old.x + h0.x, old.y + h0.y, old.z + h1.x, old.w + h1.y);
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (n0 + c + i < P.N) {
                                    float* o = out + (c + i) * P.out.s_n;
                                    const float h = i == 0 ? h0.x : (i == 1 ? h0.y : (i == 2 ? h1.x : h1.y));
                                    *o = P.accumulate ? *o + h : h;
                                }
                        }
                    }
                }
            }
            it += s.kt1 - s.kt0;
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
        if (warp == kEpiWarps + kConvWarps) {
            uint32_t slot = 0, phase = 0, acc_phase = 1;
            bool ok = true;
            if (rank == 1) {
                const int count = it1 - it0;
                for (int i = 0; i < count; ++i) {
                    if (!(ok = wait_or_abort<false>(&B->full[slot], phase, &B->abort, P.status))) break;
                    if (lane == 0) mbar_arrive_first(&B->peer_full[slot]);
                    __syncwarp();
                    if (++slot == kStages) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
            } else {
                // (warp-uniform code, one elected lane issues: operands stay in uniform registers)
                const bool lead = elect_one();
                constexpr uint32_t desc = mma_desc(kMRows * 2, COLS);
                const uint64_t first_slot = smem_desc(smem);
                int buf = 0;
                for (int it = it0; it < it1 && ok;) {
                    const Span s = span_at(P, it, it1);
                    const int count = s.kt1 - s.kt0;
                    for (int i = 0; i < count; ++i) {
                        // (a fresh barrier counts as having completed the phase before its first)
                        if (!(ok = wait_or_abort<true>(&B->acc_empty[buf], acc_phase, &B->abort, P.status))) break;
                        if (!(ok = wait_or_abort<false>(&B->full[slot], phase, &B->abort, P.status))) break;
                        if (!(ok = wait_or_abort<true>(&B->peer_full[slot], phase, &B->abort, P.status))) break;
                        tmem_fence_after();
                        if (lead) {
                            const uint64_t a = first_slot + slot * (kStageBytes >> 4), b = a + (kBlocks * kABytes >> 4);
                            const uint32_t d = tmem + buf * 256;
                            auto at = [](int k, int step) { return (k / 2) * (step >> 4) + 2 * (k % 2); };
                            // the small products first, while the accumulator is small
#pragma unroll
                            for (int k = 0; k < 2 * kBlocks; ++k) {
                                const uint64_t ak = a + at(k, kABytes), bk = b + at(k, kBBytes);
                                mma_f16(d, ak, bk + 4, desc, k > 0);
                                if (!P.split) mma_f16(d, ak + 4, bk, desc, true);
                                if (PW == 2 && !P.split) mma_f16(d, ak + 4, bk + 4, desc, true);
                            }
#pragma unroll
                            for (int k = 0; k < 2 * kBlocks; ++k) mma_f16(d, a + at(k, kABytes), b + at(k, kBBytes), desc, true);
                            mma_commit(&B->empty[slot]);
                            mma_commit(&B->acc_full[buf]);
                        }
                        __syncwarp();
                        buf ^= 1;
                        if (buf == 0) acc_phase ^= 1;
                        if (++slot == kStages) {
                            slot = 0;
                            phase ^= 1;
                        }
                    }
                    it += count;
                }
            }
        } else if constexpr (FWD) {
            // Item i of a thread: 8 channels of a row of a block.  Rows contiguous in memory: four lanes for the four pieces of
            // a row, and lanes that store together have rows that differ in bit 2, which the swizzle turns into the other half
            // of the banks.  Channels contiguous over rows: a lane per row.
            constexpr int ITEMS = kRowsB * 4 / (32 * kConvWarps);
            const int t = threadIdx.x - 32 * kEpiWarps;
            const bool lanes_are_rows = P.src.kind == 2;
            const int row0 = lanes_are_rows ? t % kRowsB : (t >> 4) * 8 + ((t >> 3) & 1) * 2 + ((t >> 2) & 1) * 4;
            const int piece0 = lanes_are_rows ? t / kRowsB * ITEMS : t & 3;
            auto row_of = [&](int i) { return lanes_are_rows ? row0 : row0 + i; };
            const ForwardScale<PW> scales(*P.scale_word);
            const float factor = pow2i(-scales.e);
            float2 base[ITEMS][4], cur[ITEMS][4], nxt[ITEMS][4];  // values, their power of this block, values of the next channels
            uint32_t slot = 0, phase = 1;  // (a fresh barrier counts as having completed the phase before its first)
            bool ok = true;
            for (int it = it0; it < it1 && ok;) {
                const Span s = span_at(P, it, it1);
                const int n0 = s.tn * kNRows + rank * kRowsB;
                const int last = min(P.blocks, s.kt1 * kBlocks);  // block behind the last one of the span
                auto load = [&](int kb) {
#pragma unroll
                    for (int i = 0; i < ITEMS; ++i)
                        fetch8(P.src, source_row(P.src, s.g, n0 + row_of(i)), kb * kBlockK + 8 * (lanes_are_rows ? piece0 + i : piece0), nxt[i]);
                };
                // (scaled when they are needed, not when they are asked for: the loads are still under way then)
                auto first_power = [&]() {
                    const float lift = pow2i(scales.b(1));
#pragma unroll
                    for (int i = 0; i < ITEMS; ++i)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            base[i][e] = scale2(nxt[i][e], factor);
                            cur[i][e] = scale2(base[i][e], lift);
                        }
                };
                auto next_power = [&](int exponent) {
                    const float step = pow2i(scales.b(exponent) - scales.b(exponent - 1));
#pragma unroll
                    for (int i = 0; i < ITEMS; ++i)
#pragma unroll
                        for (int e = 0; e < 4; ++e) cur[i][e] = __fmul2_rn(cur[i][e], scale2(base[i][e], step));
                };
                int kb = s.kt0 * kBlocks / NP, j = s.kt0 * kBlocks - kb * NP;  // block: channels 32 kb .., exponent j + 1
                load(kb);
                first_power();
                for (int e = 2; e <= j + 1; ++e) next_power(e);
                if ((kb + 1) * NP < last) load(kb + 1);
                for (int kt = s.kt0; kt < s.kt1; ++kt) {
                    ok = __all_sync(0xffffffffu, wait_or_abort<false>(&B->empty[slot], phase, &B->abort, P.status));
                    if (!ok) break;
                    char* stage = smem + slot * kStageBytes;
                    if (t == 0) {
                        mbar_expect_tx(&B->full[slot], kBlocks * kABytes);
                        bulk_load(stage, a_blocks(P, s, kt, rank), kBlocks * kABytes, &B->full[slot]);
                    }
#pragma unroll 1
                    for (int bl = 0; bl < kBlocks; ++bl) {
                        char* b = stage + kBlocks * kABytes + bl * kBBytes;
#pragma unroll
                        for (int i = 0; i < ITEMS; ++i) {
                            uint4 hi, lo;
                            split8(cur[i], &hi, &lo);
                            const int row = row_of(i), piece = lanes_are_rows ? piece0 + i : piece0;
                            const uint32_t at = row * 128 + ((piece ^ (row & 7)) << 4);
                            *reinterpret_cast<uint4*>(b + at) = hi;
                            *reinterpret_cast<uint4*>(b + (at ^ 64)) = lo;
                        }
                        // (behind the last block of all there may be one that only fills the stage: A is 0 there, B finite)
                        if (++j < NP) {
                            next_power(j + 1);
                        } else {
                            j = 0;
                            ++kb;
                            if (kb * NP < last) first_power();
                            if ((kb + 1) * NP < last) load(kb + 1);
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&B->full[slot]);
                    if (++slot == kStages) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
                it += s.kt1 - s.kt0;
            }
        } else {
            // unit u of the CTA's range: stage u / UNITS, 32 items of it; dealt to the warps in turn.  An item is a channel
            // and 8 rows; neighbouring lanes have neighbouring channels.
            const int cw = warp - kEpiWarps;
            const int units = (it1 - it0) * UNITS;
            Span s{};
            int span_first = 0, span_end = 0;  // the stages of the range that s describes
            float2 nxt[4];
            float nxt_down = 0.0f, nxt_shift = 0.0f;
            int nxt_left = 0;  // elements of the item that there are
            const char* nxt_a = nullptr;
            auto fetch = [&](int u) {
                const int n = u / UNITS, item = (u % UNITS) * 32 + lane, cl = item % CW, chunk = item / CW;
                while (n >= span_end) {
                    s = span_at(P, it0 + span_end, it1);
                    span_first = span_end;
                    span_end += s.kt1 - s.kt0;
                }
                const int c = s.tn * CT + rank * CW + cl, kt = s.kt0 + n - span_first;
                fetch8(P.src, source_row(P.src, s.g, c), kt * kStageK + 8 * chunk, nxt);
                nxt_left = P.src.k - kt * kStageK - 8 * chunk;
                load1(&nxt_down, P.col_down + s.g * P.tiles_n * CT + c, true);
                load1(&nxt_shift, P.col_shift + s.g * P.tiles_n * CT + c, true);
                if (u % UNITS == 0) nxt_a = a_blocks(P, s, kt, rank);
            };
            if (cw < units) fetch(cw);
            for (int u = cw; u < units; u += kConvWarps) {
                const int n = u / UNITS, slot = n % kStages;
                if (!__all_sync(0xffffffffu, wait_or_abort<false>(&B->empty[slot], (n / kStages & 1) ^ 1, &B->abort, P.status))) break;
                char* stage = smem + slot * kStageBytes;
                if (u % UNITS == 0 && lane == 0) {
                    mbar_expect_tx(&B->full[slot], kBlocks * kABytes);
                    bulk_load(stage, nxt_a, kBlocks * kABytes, &B->full[slot]);
                }
                float2 v[4], cur[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = __ffma2_rn(nxt[e], make_float2(nxt_down, nxt_down), make_float2(nxt_shift, nxt_shift));
                if (nxt_left < 8) {  // (the powers of a shift alone could leave fp16's range)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (nxt_left <= 2 * e) v[e].x = 0.0f;
                        if (nxt_left <= 2 * e + 1) v[e].y = 0.0f;
                    }
                }
                if (u + kConvWarps < units) fetch(u + kConvWarps);
                // row of B: power, channel of the half
                const int item = (u % UNITS) * 32 + lane, cl = item % CW, chunk = item / CW;
                char* b = stage + kBlocks * kABytes + (chunk / 4) * kBBytes;
                const uint32_t at = cl * 128 + (((chunk & 3) ^ (cl & 7)) << 4);
#pragma unroll
                for (int e = 0; e < 4; ++e) cur[e] = scale2(v[e], kScaleB);
#pragma unroll 1
                for (int j = 0; j < NP; ++j) {  // (rolled: the body stays in the instruction cache)
                    uint4 hi, lo;
                    split8(cur, &hi, &lo);
                    *reinterpret_cast<uint4*>(b + j * CW * 128 + at) = hi;
                    *reinterpret_cast<uint4*>(b + j * CW * 128 + (at ^ 64)) = lo;
#pragma unroll
                    for (int e = 0; e < 4; ++e) cur[e] = __fmul2_rn(cur[e], v[e]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&B->full[slot]);
            }
        }
    }
    // (every copy has landed when its stage's products were issued; after a wait that gave up they get a while)
    if (*static_cast<volatile int*>(&B->abort))
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    tmem_fence_before();
    __syncwarp();
    cluster_sync();
    tmem_fence_after();
    __syncwarp();
    if (warp == 0) tmem_free(tmem);
}

// Adds up the partial sums of tiles that are shared between pairs (or by the CTAs of one, split).  blockIdx.y: eight columns,
// blockIdx.z: CTA of the pair (one block for both where they have the same rows).  Forward and split: a tile per blockIdx.x, and
// in the forward pass the values are made here, of tiles that one pair had from the sums in the output array.  Backward: a shared
// tile holds the end of some pair's range; the first boundary inside it stands for it.
template <int PW, bool FWD>
__global__ void __launch_bounds__(kMRows) even_fold_kernel(const EvenParams P, const int workers) {
    constexpr int NP = PW - 1;
    constexpr int CT = channels_of(NP);
    constexpr int COLS = FWD ? kNRows : CT;
    stream_order_begin();
    if ((P.gate0 && *P.gate0 != 0) || (P.gate1 && *P.gate1 != 0)) return;
    const int rank = blockIdx.z, row = threadIdx.x, col0 = blockIdx.y * 8;
    int c0, t0;
    if (FWD || P.split) {
        t0 = blockIdx.x * P.kt;
        c0 = static_cast<int>((static_cast<long long>(t0 + 1) * workers - 1) / P.total);
    } else {
        c0 = blockIdx.x;
        const int cut = even_begin(P, workers, c0 + 1);
        t0 = cut / P.kt * P.kt;
        if (cut == t0 || even_begin(P, workers, c0) > t0) return;
    }
    const int c1 = static_cast<int>((static_cast<long long>(t0 + P.kt) * workers - 1) / P.total);
    const Span s = span_at(P, t0, P.total);
    const int m = (P.split ? s.tm : s.tm * 2 + rank) * kMRows + row, n0 = s.tn * COLS + col0;
    if (m >= P.M || n0 >= P.N) return;
    float v[8];
    const bool parts = P.split || !FWD || c0 != c1;
    if (parts) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = 0.0f;
        // a worker's slot of this tile is its first, unless it began in an earlier one, as only c0 can have
        int slot = t0 / P.kt - even_begin(P, workers, c0) / P.kt;
        if (!P.split) slot = min(slot, 1);
        const size_t size = static_cast<size_t>(COLS) * kMRows, step = P.slots * size;  // of a partial sum, of a CTA's
        const float* part = P.partials + (P.split ? 2 * c0 : 2 * c0 + rank) * step + static_cast<size_t>(col0) * kMRows + row;
        auto add = [&](const float* p) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] += p[i * kMRows];
        };
        add(part + slot * size);
        if (P.split) add(part + step + slot * size);
#pragma unroll 4
        for (int c = c0 + 1; c <= c1; ++c) {
            add(part + static_cast<size_t>(c - c0) * 2 * step);
            if (P.split) add(part + (static_cast<size_t>(c - c0) * 2 + 1) * step);
        }
    }
    if constexpr (FWD) {
        const ForwardEnd end = forward_end<PW>(P);
        const float sa = P.sum_a[s.g * P.M + m], na = P.norm_a[s.g * P.M + m];
        const float *sb = P.sum_b + s.g * P.N + n0, *nb = P.norm_b + s.g * P.N + n0;
#pragma unroll
        for (int q = 0; q < 8; q += 4) {
            if (n0 + q >= P.N) break;
            long long off[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) off[i] = i > 0 && P.vec ? off[0] + i : even_offset(P, s.g, m, min(n0 + q + i, P.N - 1));
            if (!parts) {
                if (P.vec) {
                    const float4 r = *reinterpret_cast<const float4*>(P.out_f + off[0]);
                    v[q] = r.x; v[q + 1] = r.y; v[q + 2] = r.z; v[q + 3] = r.w;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[q + i] = P.out_f[off[i]];
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (n0 + q + i < P.N)
                    v[q + i] = forward_value<PW>(P, end, v[q + i], sa, na, sb[q + i], nb[q + i], static_cast<int>(off[i]));
            if (P.vec) {
                *reinterpret_cast<float4*>(P.out_f + off[0]) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (n0 + q + i < P.N) P.out_f[off[i]] = v[q + i];
            }
        }
    } else {
        const float row_scale = pow2i(-15 - P.row_exp[s.g * P.M + m]);
        const float* down = P.col_down + s.g * P.tiles_n * CT + n0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (n0 + i < P.N) {
                float* o = P.out_f + even_offset(P, s.g, m, n0 + i);
                const float h = v[i] * row_scale * up_of<NP>(down[i]);
                *o = P.accumulate ? *o + h : h;
            }
    }
}

// ---- preparation -----------------------------------------------------------------------------------------------------
// One item of a block of A: eight reduction elements of a row, hi and lo where the swizzle puts them.
// twin: not 0 if the block of the pair's second CTA, which takes lo for hi, is that many bytes behind this one.
__device__ __forceinline__ void put_item(char* block, int row, int chunk, const float2 (&v)[4], long long twin) {
    uint4 hi, lo;
    split8(v, &hi, &lo);
    const uint32_t at = row * 128 + ((chunk ^ (row & 7)) << 4);
    *reinterpret_cast<uint4*>(block + at) = hi;
    *reinterpret_cast<uint4*>(block + (at ^ 64)) = lo;
    if (twin != 0) {
        *reinterpret_cast<uint4*>(block + twin + at) = lo;
        *reinterpret_cast<uint4*>(block + twin + (at ^ 64)) = hi;
    }
}
constexpr int kPrep = 256;
__device__ __forceinline__ void item_of(const Source& S, int i, int* row, int* chunk) {
    const bool lanes_are_rows = S.kind == 2;  // neighbouring rows are neighbours in memory
    *row = lanes_are_rows ? i & (kMRows - 1) : i >> 2;
    *chunk = lanes_are_rows ? i >> 7 : i & 3;
}
__device__ __forceinline__ unsigned magnitude(float v) { return __float_as_uint(v) & 0x7fffffffu; }

// Sums of p-th powers of every row of both operands (64 bits: 4 us of arithmetic at 512 x 3072 -> 5120, and no error of
// theirs reaches the result) and the largest magnitude of all.  Rows contiguous in memory: a warp per row; else 32 rows per
// block, its warps sharing the reduction.
template <int PW>
__device__ __forceinline__ void row_power_sums(const Source& S, int G, int block, double* sums, unsigned* scale_word) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned top = 0;
    double sum = 0.0;
    auto take = [&](float v) {
        top = max(top, magnitude(v));
        double d = v;
        d *= d;
        double q = d;
#pragma unroll
        for (int i = 1; i < PW / 2; ++i) q *= d;
        sum += q;
    };
    if (S.kind != 2) {
        const long long r = static_cast<long long>(block) * 8 + warp;
        if (r < static_cast<long long>(G) * S.rows) {
            const int g = static_cast<int>(r / S.rows);
            const float* p = source_row(S, g, static_cast<int>(r - static_cast<long long>(g) * S.rows));
            if (S.kind == 0) {
#pragma unroll 4
                for (int k = 4 * lane; k < S.k; k += 128) {
                    const float4 v = *reinterpret_cast<const float4*>(p + k);
                    take(v.x); take(v.y); take(v.z); take(v.w);
                }
            } else {
#pragma unroll 8
                for (int k = lane; k < S.k; k += 32) take(p[k]);
            }
            for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
            if (lane == 0) sums[r] = sum;
        }
    } else {
        __shared__ double part[8][32];
        const int per_group = (S.rows + 31) / 32, g = block / per_group, row = (block - g * per_group) * 32 + lane;
        const float* p = source_row(S, g, row);
        if (p)
#pragma unroll 4
            for (int k = warp; k < S.k; k += 8) take(p[k * S.s_k]);
        part[warp][lane] = sum;
        __syncthreads();
        if (warp == 0 && p) {
            for (int i = 1; i < 8; ++i) sum += part[i][lane];
            sums[static_cast<long long>(g) * S.rows + row] = sum;
        }
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if (lane == 0 && top > *static_cast<volatile unsigned*>(scale_word)) atomicMax(scale_word, top);
}
// One of the sampled outputs: whether it is below the guard's line.  The last block to know decides.  counts: outputs below, blocks.
// It runs beside the kernel in front of it, whose results it does not need, and waits for that at its end (in one kernel with the
// row sums these took 72 us instead of 31 for 32 images of 576 x 1024; behind them it would add 9).
// That kernel starts behind a memset, which nothing overtakes: whatever was queued before the memset is done when blocks of either
// kernel start, so that only the kernels behind this one depend on the wait.
template <int PW>
__global__ void __launch_bounds__(kPrep) even_sample_kernel(const Source a, const Source b, int G, float least, int* counts, int* dense) {
    stream_order_release();
    const int sample = blockIdx.x;
    __shared__ double part[3][8];
    const int g = sample % G;
    // (spread over both operands; coprime strides)
    const float* pa = source_row(a, g, static_cast<int>(static_cast<long long>(sample) * a.rows / kGuardSamples));
    const float* pb = source_row(b, g, static_cast<int>((sample * 7919LL + 13) % b.rows));
    double sum[3] = {};
#pragma unroll 4
    for (int k = threadIdx.x; k < a.k; k += kPrep) {
        const double v[3] = {pa[k * a.s_k], pb[k * b.s_k], static_cast<double>(pa[k * a.s_k]) - pb[k * b.s_k]};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double d = v[i] * v[i];
            double q = d;
#pragma unroll
            for (int e = 1; e < PW / 2; ++e) q *= d;
            sum[i] += q;
        }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        for (int d = 16; d > 0; d >>= 1) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], d);
        if ((threadIdx.x & 31) == 0) part[i][threadIdx.x >> 5] = sum[i];
    }
    __syncthreads();
    if (threadIdx.x != 0) {
        stream_order_wait();
        return;
    }
    for (int w = 1; w < kPrep / 32; ++w)
        for (int i = 0; i < 3; ++i) sum[i] += part[i][w];
    const double most = fmax(sum[0], sum[1]);
    const float na = static_cast<float>(sum[0] / most), nb = static_cast<float>(sum[1] / most);
    if (static_cast<float>(sum[2] / most) < least * power<PW>(powf(na, 1.0f / PW) + powf(nb, 1.0f / PW))) atomicAdd(counts, 1);
    __threadfence();
    if (atomicAdd(counts + 1, 1) == kGuardSamples - 1 && atomicAdd(counts, 0) >= kMostBelow) *dense = 1;
    stream_order_wait();
}
template <int PW>
__global__ void __launch_bounds__(kPrep) even_rows_kernel(const Source a, const Source b, int G, int blocks_a, double* sums_a,
                                                         double* sums_b, unsigned* scale_word) {
    stream_order_begin();
    if (static_cast<int>(blockIdx.x) < blocks_a) row_power_sums<PW>(a, G, blockIdx.x, sums_a, scale_word);
    else row_power_sums<PW>(b, G, blockIdx.x - blocks_a, sums_b, scale_word);
}

// The blocks of A of the forward form, C(p, j) x^j split, j = 1 .. p - 1 (seq blocks per block of rows: zeros behind the last
// where stages need an even number); the blocks behind those put the row sums on the common scale.
template <int PW>
__global__ void __launch_bounds__(kPrep) even_powers_kernel(const Source a, int G, int tiles_m, int kb, int seq, bool split, char* images,
                                                           const double* sums_a, const double* sums_b, int rows_b,
                                                           float* sum_a, float* norm_a, float* sum_b, float* norm_b,
                                                           const unsigned* scale_word, int* dense, int* small) {
    constexpr int NP = PW - 1;
    stream_order_begin();
    const unsigned top = *scale_word;
    const int e = exponent_above(top);
    if (*static_cast<volatile int*>(dense) != 0) return;
    if (top >= 0x7f800000u || e < -100 || e > 100) {  // not finite, all zero, or hardly a number
        if (blockIdx.x == 0 && threadIdx.x == 0) *dense = 1;
        return;
    }
    const int images_blocks = G * tiles_m * kb, block = blockIdx.x;
    if (block >= images_blocks) {
        // An output is at most the sum of its rows' norms.  Where rows of either operand lie below half of what an output has to
        // reach (ForwardEnd::least), their outputs go to the list for certain: more of them than it holds, and there is no
        // point in the products (512 x 3072 -> 5120, p = 8, one value of 100: 1594 -> 1089 us; the
        // direct kernels take 1045).  small: rows of a, rows of b, blocks done.
        const int i = (block - images_blocks) * kPrep + threadIdx.x, rows = G * (a.rows + rows_b);
        const float half = 0.5f * __uint_as_float((top & 0x7fffffu) | 0x3f000000u) * exp2f(-10.0f / PW);
        bool small_a = false, small_b = false;
        if (i < rows) {
            const bool is_a = i < G * a.rows;
            const int r = is_a ? i : i - G * a.rows;
            const float v = static_cast<float>((is_a ? sums_a : sums_b)[r] * exp2(-static_cast<double>(PW) * e));
            const float norm = v > 0.0f ? root<PW>(v) : 0.0f;
            (is_a ? sum_a : sum_b)[r] = v;
            (is_a ? norm_a : norm_b)[r] = norm;
            (is_a ? small_a : small_b) = norm < 0.999f * half;
        }
        const int count_a = __syncthreads_count(small_a), count_b = __syncthreads_count(small_b);
        if (threadIdx.x == 0) {
            if (count_a) atomicAdd(small, count_a);
            if (count_b) atomicAdd(small + 1, count_b);
            __threadfence();
            if (atomicAdd(small + 2, 1) == (rows + kPrep - 1) / kPrep - 1) {
                const double pairs = static_cast<double>(atomicAdd(small, 0)) * atomicAdd(small + 1, 0);
                if (pairs > static_cast<double>(kListCap) * G) *dense = 1;  // (of G groups: as many on average)
            }
        }
        return;
    }
    const ForwardScale<PW> scales(top);
    const float factor = pow2i(-e);
    const int k = block % kb, t = block / kb, tm = t % tiles_m, g = t / tiles_m;
    const long long first_block = (static_cast<long long>(g) * tiles_m + tm) * (split ? 2 : 1);  // block of rows in the images
    const long long twin = split ? static_cast<long long>(seq) * kABytes : 0;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        int row, chunk;
        item_of(a, threadIdx.x + n * kPrep, &row, &chunk);
        float2 v[4], cur[4];
        fetch8(a, source_row(a, g, tm * kMRows + row), k * kBlockK + 8 * chunk, v);
#pragma unroll
        for (int i = 0; i < 4; ++i) cur[i] = v[i] = scale2(v[i], factor);
#pragma unroll
        for (int j = 0; j < NP; ++j) {
            float2 term[4];
            const float c = (j % 2 == 0 ? -binomial(PW, j + 1) : binomial(PW, j + 1)) * pow2i(scales.a(j + 1));
#pragma unroll
            for (int i = 0; i < 4; ++i) term[i] = scale2(cur[i], c);
            // (in the order in which B's exponent, p less this one, rises)
            put_item(images + (first_block * seq + k * NP + NP - 1 - j) * static_cast<long long>(kABytes), row, chunk, term, twin);
#pragma unroll
            for (int i = 0; i < 4; ++i) cur[i] = __fmul2_rn(cur[i], v[i]);
        }
        if (k == kb - 1 && seq > kb * NP) {
            const float2 zero[4] = {};
            put_item(images + (first_block * seq + kb * NP) * static_cast<long long>(kABytes), row, chunk, zero, twin);
        }
    }
}

// The listed outputs, summed directly: a warp each.
template <int PW>
__global__ void __launch_bounds__(kPrep) even_direct_kernel(const float* x, const float* w, Shape s, float* y, const int* list,
                                                           const int* list_count, const int* dense) {
    stream_order_begin();
    if (*dense != 0) return;
    const int count = min(*list_count, kListCap), lane = threadIdx.x & 31;
    for (int i = blockIdx.x * (kPrep / 32) + (threadIdx.x >> 5); i < count; i += gridDim.x * (kPrep / 32)) {
        const int off = list[i], t = off / s.HW, hw = off - t * s.HW, b = t / s.CO, o = t - b * s.CO, g = o / s.COg;
        const float* xr = x + (static_cast<long long>(b) * s.CI + static_cast<long long>(g) * s.CIg) * s.HW + hw;
        const float* wr = w + static_cast<long long>(o) * s.CIg;
        float sum = 0.0f;
#pragma unroll 8
        for (int c = lane; c < s.CIg; c += 32) sum += power<PW>(xr[static_cast<long long>(c) * s.HW] - wr[c]);
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
        if (lane == 0) y[off] = powf(fmaxf(sum, FLT_MIN), 1.0f / PW);
    }
}

constexpr int kColumnRows = 128;  // least rows per block of the column jobs
constexpr int kMaxRanges = 64;
constexpr int kMaxSplits = 64;    // row ranges of the coefficients' column sums
constexpr int kMaxChannelExp = 17;  // channels of values beyond 2^17 or below 2^-17: 2^(7 * 17) is still a number

struct BackwardStats {
    Shape s;
    const float *coef, *x, *w, *y;
    int pitch;
    int *row_exp, *out_exp;                           // rows of the coefficients, output channels
    float *row_sum, *out_sum;
    // [g][channel_pitch], of the two operands that are summed over (w: grad_x, x: grad_w): 2^-e, -m 2^-e
    float *down_w, *down_x, *shift_w, *shift_x;
    int channel_pitch;
    unsigned *x_top, *x_low, *w_top, *w_low;          // per channel: codes of the largest value and of the largest negative
    double2 *x_part, *w_part;                         // [range of rows][channel]: sums of values and of squares
    int x_ranges, w_ranges, x_rows, w_rows;           // ranges, and rows (samples, of images) in each
    unsigned *y_low, *most;                           // code of the largest -y, bits of the largest |d| + |u| of a channel
    double* spread_part;                              // [channel block]: sum of s^p
    double per_x, per_w;                              // 1 / rows
    int p;
    unsigned* part_top;                               // [split][CO]
    double* part_sum;
    float* part_abs;
    int splits, rows_per_split;
    bool need_x, need_w;                              // grad_x / grad_w is wanted
    int blocks_rows, blocks_cols, blocks_w, blocks_x, blocks_y; // blocks of each job, in this order
    int blocks_channels;                              // of the second kernel
    int* bad;                                         // data that the expansion does not suit
    const int* range;
    int* cond;
};

__device__ __forceinline__ void add_moments(double2* sum, float v) {
    const double d = v;
    sum->x += d;
    sum->y += d * d;
}

// column extremes and sums of rows [r0, r1) of a matrix whose columns are contiguous: 32 columns per block
__device__ __forceinline__ void column_extremes(const float* p, long long pitch, int r0, int r1, int col, int cols, unsigned* top,
                                                unsigned* low, double2* part) {
    __shared__ unsigned tops[8][32], lows[8][32];
    __shared__ double2 sums[8][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned t = 0, l = 0;
    double2 sum = make_double2(0.0, 0.0);
    if (col + lane < cols)
#pragma unroll 8
        for (int r = r0 + warp; r < r1; r += 8) {
            const float v = p[r * pitch + col + lane];
            t = max(t, ordered(v));
            l = max(l, ordered(-v));
            add_moments(&sum, v);
        }
    tops[warp][lane] = t;
    lows[warp][lane] = l;
    sums[warp][lane] = sum;
    __syncthreads();
    if (warp == 0) {
        for (int i = 1; i < 8; ++i) {
            t = max(t, tops[i][lane]);
            l = max(l, lows[i][lane]);
            sum.x += sums[i][lane].x;
            sum.y += sums[i][lane].y;
        }
        if (col + lane < cols) {
            atomicMax(top + col + lane, t);
            atomicMax(low + col + lane, l);
            part[col + lane] = sum;
        }
    }
}

__device__ __forceinline__ int row_scale(unsigned top) {
    return top == 0 ? 0 : max(-100, min(100, 15 - exponent_above(top)));
}

// What the backward form needs to know of its operands: largest coefficient and sums of every row (over the output channels)
// and of every output channel (over the rows, in ranges), range and mean of the values of every channel of x and w.
__global__ void __launch_bounds__(kPrep) even_stats_kernel(const BackwardStats A) {
    stream_order_begin();
    const Shape& s = A.s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int block = blockIdx.x;
    if (block < A.blocks_rows) {
        const long long r = static_cast<long long>(block) * 8 + warp;
        if (r >= static_cast<long long>(s.G) * s.M) return;
        const float* p = A.coef + r * A.pitch;
        unsigned top = 0;
        double sum = 0.0;
        float abs = 0.0f;
#pragma unroll 4
        for (int o = lane; o < s.COg; o += 32) {
            top = max(top, magnitude(p[o]));
            sum += p[o];
            abs += fabsf(p[o]);
        }
        top = __reduce_max_sync(0xffffffffu, top);
        for (int d = 16; d > 0; d >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, d);
            abs += __shfl_xor_sync(0xffffffffu, abs, d);
        }
        if (lane == 0) {
            const int e = row_scale(top);
            A.row_exp[r] = e;
            A.row_sum[r] = static_cast<float>(sum * pow2i(e));
            if (top >= 0x7f800000u || (A.need_x && !(abs >= kLeastSpread * __uint_as_float(top)))) *A.bad = 1;
        }
        return;
    }
    block -= A.blocks_rows;
    if (block < A.blocks_cols) {
        __shared__ unsigned tops[8][32];
        __shared__ double sums[8][32];
        __shared__ float abses[8][32];
        const int per_group = (s.COg + 31) / 32;
        const int split = block / (per_group * s.G), rest = block - split * per_group * s.G, g = rest / per_group;
        const int o = (rest - g * per_group) * 32 + lane;
        const long long r0 = static_cast<long long>(split) * A.rows_per_split;
        const long long r1 = r0 + A.rows_per_split < s.M ? r0 + A.rows_per_split : s.M;
        unsigned top = 0;
        double sum = 0.0;
        float abs = 0.0f;
        if (o < s.COg) {
            const float* p = A.coef + static_cast<long long>(g) * s.M * A.pitch + o;
#pragma unroll 8
            for (long long r = r0 + warp; r < r1; r += 8) {
                const float v = p[r * A.pitch];
                top = max(top, magnitude(v));
                sum += v;
                abs += fabsf(v);
            }
        }
        tops[warp][lane] = top;
        sums[warp][lane] = sum;
        abses[warp][lane] = abs;
        __syncthreads();
        if (warp == 0 && o < s.COg) {
            for (int i = 1; i < 8; ++i) {
                top = max(top, tops[i][lane]);
                sum += sums[i][lane];
                abs += abses[i][lane];
            }
            const long long at = static_cast<long long>(split) * s.CO + g * s.COg + o;
            A.part_top[at] = top;
            A.part_sum[at] = sum;
            A.part_abs[at] = abs;
        }
        return;
    }
    block -= A.blocks_cols;
    const int col_blocks = (s.CIg + 31) / 32;
    if (block < A.blocks_w) {
        const int cb = block % col_blocks, t = block / col_blocks, g = t % s.G, range = t / s.G, r0 = range * A.w_rows;
        column_extremes(A.w + static_cast<long long>(g) * s.COg * s.CIg, s.CIg, r0, min(s.COg, r0 + A.w_rows), cb * 32, s.CIg,
                        A.w_top + g * s.CIg, A.w_low + g * s.CIg, A.w_part + static_cast<long long>(range) * s.CI + g * s.CIg);
        return;
    }
    block -= A.blocks_w;
    if (block >= A.blocks_x) {
        const long long total = s.M * s.CO, step = static_cast<long long>(A.blocks_y) * kPrep;
        unsigned l = 0;
#pragma unroll 4
        for (long long i = static_cast<long long>(block - A.blocks_x) * kPrep + threadIdx.x; i < total; i += step) l = max(l, ordered(-A.y[i]));
        l = __reduce_max_sync(0xffffffffu, l);
        if (lane == 0 && l > *static_cast<volatile unsigned*>(A.y_low)) atomicMax(A.y_low, l);
        return;
    }
    if (s.HW == 1) {
        const int cols = (s.CI + 31) / 32, cb = block % cols, range = block / cols, r0 = range * A.x_rows;
        column_extremes(A.x, s.CI, r0, min(s.B, r0 + A.x_rows), cb * 32, s.CI, A.x_top, A.x_low, A.x_part + static_cast<long long>(range) * s.CI);
        return;
    }
    const long long r = static_cast<long long>(block) * 8 + warp;  // (range of samples, channel)
    if (r >= static_cast<long long>(A.x_ranges) * s.CI) return;
    const int range = static_cast<int>(r / s.CI), c = static_cast<int>(r - static_cast<long long>(range) * s.CI);
    unsigned t = 0, l = 0;
    double2 sum = make_double2(0.0, 0.0);
    for (int b = range * A.x_rows; b < min(s.B, (range + 1) * A.x_rows); ++b) {
        const float* p = A.x + (static_cast<long long>(b) * s.CI + c) * s.HW;
#pragma unroll 4
        for (int i = lane; i < s.HW; i += 32) {
            t = max(t, ordered(p[i]));
            l = max(l, ordered(-p[i]));
            add_moments(&sum, p[i]);
        }
    }
    t = __reduce_max_sync(0xffffffffu, t);
    l = __reduce_max_sync(0xffffffffu, l);
    for (int d = 16; d > 0; d >>= 1) {
        sum.x += __shfl_xor_sync(0xffffffffu, sum.x, d);
        sum.y += __shfl_xor_sync(0xffffffffu, sum.y, d);
    }
    if (lane == 0) {
        atomicMax(A.x_top + c, t);
        atomicMax(A.x_low + c, l);
        A.x_part[r] = sum;
    }
}

// What a channel is taken relative to: its mean, to a sixteenth of half its range (the value itself where there is but one).  With
// so few bits the other operand less the centre is exact for all but small values of it, and zero-mean channels are left as they
// are; the mean itself, with its rounding in every d, made gradients 10 % worse (3.0e-7 -> 3.3e-7, p = 8).
__device__ __forceinline__ float center_of(double mean, float least, float most) {
    const float half = 0.5f * most - 0.5f * least;
    if (!(half > 0.0f)) return most;
    const int e = max(-120, min(120, exponent_above(__float_as_uint(half)) - 4));
    return static_cast<float>(rint(mean * pow2i(-e)) * pow2i(e));
}

// 2^-e and shift of a channel that is summed over, its values in [u_low, u_top], the other operand's in [d_low, d_top]; the largest
// |d| + |u|.
__device__ __forceinline__ float channel_scale(float center, float u_low, float u_top, float d_low, float d_top, float* down, float* shift,
                                               bool* bad) {
    const float u = fmaxf(u_top - center, center - u_low), d = fmaxf(d_top - center, center - d_low);
    const float m = u > 0.0f ? fmaxf(u, d * kChannelFloor) : d;
    const int e = m > 0.0f ? exponent_above(__float_as_uint(m)) : 0;
    *bad |= abs(e) > kMaxChannelExp || (u > 0.0f && !(u >= d * kLeastChannel));
    *down = pow2i(-max(-kMaxChannelExp, min(kMaxChannelExp, e)));
    *shift = -center * *down;
    return u + d;
}

// Scales of the channels and of the output channels' coefficients; guards on both.  Blocks of channels: 32 of a group, whose
// warps share the ranges of rows.
__global__ void __launch_bounds__(kPrep) even_scales_kernel(const BackwardStats A) {
    stream_order_begin();
    const Shape& s = A.s;
    bool bad = false;
    if (static_cast<int>(blockIdx.x) < A.blocks_channels) {
        __shared__ double2 parts[2][8][32];
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int per_group = (s.CIg + 31) / 32, g = blockIdx.x / per_group, c = (blockIdx.x - g * per_group) * 32 + lane, i = g * s.CIg + c;
        double2 sx = make_double2(0.0, 0.0), sw = sx;
        unsigned codes[4] = {};
        if (warp == 0 && c < s.CIg) {
            codes[0] = A.x_top[i]; codes[1] = A.x_low[i]; codes[2] = A.w_top[i]; codes[3] = A.w_low[i];
        }
        if (c < s.CIg) {
#pragma unroll 4
            for (int k = warp; k < A.x_ranges; k += 8) {
                const double2 v = A.x_part[static_cast<long long>(k) * s.CI + i];
                sx.x += v.x;
                sx.y += v.y;
            }
#pragma unroll 4
            for (int k = warp; k < A.w_ranges; k += 8) {
                const double2 v = A.w_part[static_cast<long long>(k) * s.CI + i];
                sw.x += v.x;
                sw.y += v.y;
            }
        }
        parts[0][warp][lane] = sx;
        parts[1][warp][lane] = sw;
        __syncthreads();
        if (warp != 0) return;
        float most = 0.0f;
        double spread = 0.0;
        if (c < s.CIg) {
            for (int k = 1; k < 8; ++k) {
                sx.x += parts[0][k][lane].x;
                sx.y += parts[0][k][lane].y;
                sw.x += parts[1][k][lane].x;
                sw.y += parts[1][k][lane].y;
            }
            const float xt = from_ordered(codes[0]), xl = -from_ordered(codes[1]);
            const float wt = from_ordered(codes[2]), wl = -from_ordered(codes[3]);
            bad = !(fmaxf(fabsf(xt), fabsf(wt)) < INFINITY) || !(fmaxf(fabsf(xl), fabsf(wl)) < INFINITY) || isnan(xt + xl + wt + wl);
            const double ex = sx.x * A.per_x, ew = sw.x * A.per_w;
            const double square = fmax(sx.y * A.per_x - ex * ex, 0.0) + fmax(sw.y * A.per_w - ew * ew, 0.0) + (ex - ew) * (ex - ew);
            spread = square;
            for (int k = 1; k < A.p / 2; ++k) spread *= square;
            const int at = g * A.channel_pitch + c;
            bool bad_x = false, bad_w = false;
            const float most_x = channel_scale(center_of(ew, wl, wt), wl, wt, xl, xt, A.down_w + at, A.shift_w + at, &bad_x);
            const float most_w = channel_scale(center_of(ex, xl, xt), xl, xt, wl, wt, A.down_x + at, A.shift_x + at, &bad_w);
            bad |= (A.need_x && bad_x) || (A.need_w && bad_w);
            most = bad ? 0.0f : fmaxf(A.need_x ? most_x : 0.0f, A.need_w ? most_w : 0.0f);
        }
        for (int d = 16; d > 0; d >>= 1) spread += __shfl_xor_sync(0xffffffffu, spread, d);
        const unsigned bits = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
        if (lane == 0) {
            A.spread_part[blockIdx.x] = spread;
            atomicMax(A.most, bits);
            bad |= blockIdx.x == 0 && *A.bad != 0;
        }
        if (bad && *A.range == 0) *A.cond = 1;
        return;
    }
    if (static_cast<int>(blockIdx.x) >= A.blocks_channels) {  // a warp per output channel
        const int o = (static_cast<int>(blockIdx.x) - A.blocks_channels) * (kPrep / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
        unsigned top = 0;
        double sum = 0.0;
        float abs = 0.0f;
        for (int k = lane; k < A.splits && o < s.CO; k += 32) {
            top = max(top, A.part_top[static_cast<long long>(k) * s.CO + o]);
            sum += A.part_sum[static_cast<long long>(k) * s.CO + o];
            abs += A.part_abs[static_cast<long long>(k) * s.CO + o];
        }
        top = __reduce_max_sync(0xffffffffu, top);
        for (int d = 16; d > 0; d >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, d);
            abs += __shfl_xor_sync(0xffffffffu, abs, d);
        }
        if (lane == 0 && o < s.CO) {
            if (A.need_w && !(abs >= kLeastSpread * __uint_as_float(top)) && *A.range == 0) *A.cond = 1;
            const int e = row_scale(top);
            A.out_exp[o] = e;
            A.out_sum[o] = static_cast<float>(sum * pow2i(e));
        }
    }
}

// The guards on the smallest output, by one warp.
__device__ __forceinline__ void guard_outputs(const BackwardStats& A) {
    const int lane = threadIdx.x & 31, per_group = (A.s.CIg + 31) / 32;
    double most = 0.0;
    for (int g = 0; g < A.s.G; ++g) {
        double sum = 0.0;
        for (int k = lane; k < per_group; k += 32) sum += A.spread_part[g * per_group + k];
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
        most = fmax(most, sum);
    }
    const float y = -from_ordered(*A.y_low);
    const double scaled = y / least_of_spread(A.p), square = scaled * scaled;
    double power = square;
    for (int k = 1; k < A.p / 2; ++k) power *= square;
    if (lane == 0 && (!(kMostOfOutput * y >= __uint_as_float(*A.most)) || !(power >= most))) *A.cond = 1;
}

// Blocks of A of the backward form: the coefficients with rows = positions (grad_x) and with rows = output channels (grad_w).
struct CoefImages {
    Source src;
    const int* exp;
    char* images;
    int tiles_m, kb, blocks;
    bool split;
};
// (and, in a block behind theirs, the last guard: the products, not the images, wait for it)
__global__ void __launch_bounds__(kPrep) even_coef_kernel(const BackwardStats A, const CoefImages X, const CoefImages W) {
    stream_order_begin();
    if (*A.range != 0 || *A.cond != 0) return;
    if (static_cast<int>(blockIdx.x) == X.blocks + W.blocks) {
        if (threadIdx.x < 32) guard_outputs(A);
        return;
    }
    const bool first = static_cast<int>(blockIdx.x) < X.blocks;
    const CoefImages& J = first ? X : W;
    const int block = first ? blockIdx.x : blockIdx.x - X.blocks;
    const int k = block % J.kb, t = block / J.kb, tm = t % J.tiles_m, g = t / J.tiles_m;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        int row, chunk;
        item_of(J.src, threadIdx.x + n * kPrep, &row, &chunk);
        const int r = tm * kMRows + row;
        float2 v[4];
        fetch8(J.src, source_row(J.src, g, r), k * kBlockK + 8 * chunk, v);
        const float f = r < J.src.rows ? pow2i(J.exp[g * J.src.rows + r]) : 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = scale2(v[i], f);
        put_item(J.images + (static_cast<long long>(t) * (J.split ? 2 : 1) * J.kb + k) * kABytes, row, chunk, v,
                 J.split ? static_cast<long long>(J.kb) * kABytes : 0);
    }
}

// ---- host ------------------------------------------------------------------------------------------------------------
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline int div_up(long long a, long long b) { return static_cast<int>((a + b - 1) / b); }

// x as rows = positions, reduction = channels; w as rows = output channels
Source rows_of_x(const float* x, const Shape& s) {
    if (s.HW == 1) return Source{x, s.CIg % 4 == 0 && aligned16(x) ? 0 : 1, static_cast<int>(s.M), s.CIg, 0, s.CI, 1, 0, s.CIg};
    return Source{x, 2, static_cast<int>(s.M), s.CIg, s.HW, 1, s.HW, static_cast<long long>(s.CI) * s.HW,
                  static_cast<long long>(s.CIg) * s.HW};
}
Source rows_of_w(const float* w, const Shape& s) {
    return Source{w, s.CIg % 4 == 0 && aligned16(w) ? 0 : 1, s.COg, s.CIg, 0, s.CIg, 1, 0, static_cast<long long>(s.COg) * s.CIg};
}
// rows = channels, reduction = output channels (w) or positions (x)
Source channels_of_w(const float* w, const Shape& s) {
    return Source{w, 2, s.CIg, s.COg, 0, 1, s.CIg, 0, static_cast<long long>(s.COg) * s.CIg};
}
Source channels_of_x(const float* x, const Shape& s) {
    if (s.HW == 1) return Source{x, 2, s.CIg, s.B, 0, 1, s.CI, 0, s.CIg};
    return Source{x, s.HW % 4 == 0 && aligned16(x) ? 4 : 3, s.CIg, static_cast<int>(s.M), s.HW, s.HW, 1,
                  static_cast<long long>(s.CI) * s.HW, static_cast<long long>(s.CIg) * s.HW};
}

// Tiles along m rows of A, and blocks of kMRows rows in them that are prepared; stages along k reduction elements.
// Split tiles take two passes per product instead of three: worth it up to 128 rows, where a pair would be half empty (32 x 64 x
// 32 x 32 convolution to 128 channels, p = 8, forward and weight gradient: 172 and 133 us with half-empty pairs, 162 and 129
// split, all else equal: the converters bound the forward form there, 2200 cycles per stage against 896 of products).
bool split_rows(long long m) { return m <= kMRows; }
int row_tiles(long long m) { return div_up(m, 2 * kMRows); }
int row_blocks(long long m) { return split_rows(m) ? 1 : 2 * row_tiles(m); }
// partial sums that a CTA may have to keep: of the tiles that its range touches (split), or of its first and last
int part_slots(long long m, long long total, int kt, int workers) {
    return split_rows(m) ? static_cast<int>(((total + workers - 1) / workers + kt - 2) / kt) + 1 : 2;
}
int workers_of(long long total, int cap) { return static_cast<int>(total < cap / 2 ? total : cap / 2); }
size_t part_floats(long long m, long long total, int kt, int cap, int cols) {
    const int workers = workers_of(total, cap);
    return 2 * static_cast<size_t>(workers) * part_slots(m, total, kt, workers) * cols * kMRows;
}
int stages_of(long long k) { return div_up(k, kStageK); }

// Which operand's powers are written out as A: the one for which products on padding plus the bytes of its powers take less
// time, at 1.2 PFLOP/s and 4 TB/s.
struct ForwardPlan {
    bool swap;  // A = w
    int M, N, row_blocks, tiles_n, stages;
    size_t image_bytes;
    long long total;
};
ForwardPlan plan_forward(const Shape& s, int np) {
    ForwardPlan best{};
    double least = 0.0;
    for (int swap = 0; swap < 2; ++swap) {
        ForwardPlan f;
        f.swap = swap != 0;
        f.M = swap ? s.COg : static_cast<int>(s.M);
        f.N = swap ? static_cast<int>(s.M) : s.COg;
        f.row_blocks = row_blocks(f.M);
        f.tiles_n = div_up(f.N, kNRows);
        f.stages = stages_of(static_cast<long long>(div_up(s.CIg, kBlockK)) * np * kBlockK);
        f.total = static_cast<long long>(s.G) * row_tiles(f.M) * f.tiles_n * f.stages;
        f.image_bytes = static_cast<size_t>(s.G) * 2 * row_tiles(f.M) * f.stages * kBlocks * kABytes;
        // (split: four operations per pair of halves and row of the pair instead of six)
        const double flops = (split_rows(f.M) ? 4.0 : 6.0) * f.total * kStageK * (2.0 * kMRows) * kNRows;
        const double t = flops / 1.2e15 + 2.0 * f.image_bytes / 4e12;
        if (swap == 0 || t < least) {
            least = t;
            best = f;
        }
    }
    return best;
}

template <int PW, bool FWD>
int launch_even(const EvenParams& P, int cap, cudaStream_t st) {
    static OncePerDevice once;
    constexpr int smem = even_smem(FWD, PW - 1);
    int r = once([] { return allow_smem(even_kernel<PW, FWD>, smem); });
    if (r != kOk) return r;
    const int workers = workers_of(P.total, cap);
    timing_before(st);
    r = launch_after_in_clusters(even_kernel<PW, FWD>, 2, workers * 2, kEvenThreads, smem, st, P);
    timing_after(st);
    if (r != kOk) return r;
    constexpr unsigned pieces = (FWD ? kNRows : channels_of(PW - 1)) / 8;
    if (FWD || P.split)
        return launch_after(even_fold_kernel<PW, FWD>, dim3(P.total / P.kt, pieces, P.split ? 1 : 2), kMRows, 0, st, P, workers);
    if (workers < 2 || (P.total % workers == 0 && (P.total / workers) % P.kt == 0)) return kOk;
    return launch_after(even_fold_kernel<PW, FWD>, dim3(workers - 1, pieces, 2), kMRows, 0, st, P, workers);
}

// r of the forward guard: what an output may be, to the p-th power, of its rows' norms.  The expansion's error of a value goes with
// 1 / (p r), the direct kernels' with the root of the channels.  Measured with r = 2^-6 for all, operands with a common offset,
// products / direct kernels, in 1e-8 of the values: root mean square at p = 2 133 / 26 (1536 channels) and 93 / 12 (256), p = 4 17 / 16
// and 19 / 6.5; the largest at p = 6 and 8 and 256 channels 103 / 27 and 111 / 26, from 576 channels on 40 - 65 / 36.  With these
// of what passes at most 26 / 30 and 14 / 11, 6 / 16 and 5 / 7; the largest 63 / 27 (p = 6, 256 channels).  Images and activations
// with N(0, 1) weights lie at 2^-0.9 (p = 2) to 2^-3.4 (p = 8), their smallest outputs at 2^-5.5 and above from 576 channels on.
inline float least_of_norms(int p, int channels) {
    const float base = p == 2 ? 0.0625f : (p == 4 ? 0.0221f : 0.015625f);
    return channels < 1024 ? base * sqrtf(1024.0f / channels) : base;
}

template <int PW>
int forward_power(const float* x, const float* w, const Shape& s, float* y, int cap, Bump* bump, int* status, const int** dense,
                  cudaStream_t st) {
    constexpr int NP = PW - 1;
    const ForwardPlan f = plan_forward(s, NP);
    const int rows_x = static_cast<int>(s.G * s.M), rows_w = s.CO;
    const int rows_a = f.swap ? rows_w : rows_x, rows_b = f.swap ? rows_x : rows_w;
    char* images = bump->take<char>(f.image_bytes);
    double* sums = bump->take<double>(static_cast<size_t>(rows_a) + rows_b);
    float* floats = bump->take<float>(2 * (static_cast<size_t>(rows_a) + rows_b));
    int* list = bump->take<int>(kListCap);
    int* words = bump->take<int>(8);  // largest magnitude, list length, dense, three counts of even_powers_kernel, two of samples
    float* partials = bump->take<float>(part_floats(f.M, f.total, f.stages, cap, kNRows));
    if (!images || !sums || !floats || !list || !words || !partials) return kWorkspace;
    *dense = words + 2;
    const cudaError_t e = cudaMemsetAsync(words, 0, 8 * sizeof(int), st);
    if (e != cudaSuccess) return cuda_status(e);
    const Source xs = rows_of_x(x, s), ws = rows_of_w(w, s);
    const Source a = f.swap ? ws : xs, b = f.swap ? xs : ws;
    unsigned* scale = reinterpret_cast<unsigned*>(words);
    auto sum_blocks = [&](const Source& S) { return S.kind == 2 ? s.G * div_up(S.rows, 32) : div_up(static_cast<long long>(s.G) * S.rows, 8); };
    const int blocks_a = sum_blocks(a);
    int r = launch_after(even_rows_kernel<PW>, blocks_a + sum_blocks(b), kPrep, 0, st, a, b, s.G, blocks_a, sums, sums + rows_a, scale);
    const float least = least_of_norms(PW, s.CIg);
    if (r == kOk && static_cast<double>(s.M) * s.CO * kMostBelow > 2.0 * kListCap * kGuardSamples)
        r = launch_after(even_sample_kernel<PW>, kGuardSamples, kPrep, 0, st, a, b, s.G, least, words + 6, words + 2);
    if (r != kOk) return r;
    float *sum_a = floats, *norm_a = sum_a + rows_a, *sum_b = norm_a + rows_a, *norm_b = sum_b + rows_b;
    const int kb = div_up(s.CIg, kBlockK);
    const int prep = s.G * f.row_blocks * kb + div_up(static_cast<long long>(rows_a) + rows_b, kPrep);
    r = launch_after(even_powers_kernel<PW>, prep, kPrep, 0, st, a, s.G, f.row_blocks, kb, f.stages * kBlocks, split_rows(f.M), images, sums,
                     sums + rows_a, b.rows, sum_a, norm_a, sum_b, norm_b, scale, words + 2, words + 3);
    if (r != kOk) return r;
    EvenParams P{};
    P.M = f.M; P.N = f.N; P.G = s.G;
    P.tiles_m = row_tiles(f.M); P.tiles_n = f.tiles_n; P.kt = f.stages; P.blocks = kb * NP;
    P.total = static_cast<int>(f.total);
    P.split = split_rows(f.M);
    P.slots = part_slots(f.M, f.total, P.kt, workers_of(f.total, cap));
    P.images = images;
    P.src = b;
    P.out = OutAddr{static_cast<long long>(s.CO) * s.HW, 1, static_cast<long long>(s.COg) * s.HW, s.HW, s.HW};
    P.swap = f.swap;
    // rows of four neighbours: output channels of a fully connected layer, or positions of an image
    P.vec = aligned16(y) && (f.swap ? s.HW > 1 && s.HW % 4 == 0 : s.HW == 1 && s.COg % 4 == 0);
    P.out_f = y;
    P.sum_a = sum_a; P.norm_a = norm_a; P.sum_b = sum_b; P.norm_b = norm_b;
    P.scale_word = scale;
    P.least = least;
    P.list = list; P.list_count = words + 1; P.dense = words + 2;
    P.gate0 = words + 2;
    P.partials = partials;
    P.status = status;
    if ((r = launch_even<PW, true>(P, cap, st)) != kOk) return r;
    return launch_after(even_direct_kernel<PW>, 148, kPrep, 0, st, x, w, s, y, static_cast<const int*>(list),
                        static_cast<const int*>(words + 1), static_cast<const int*>(words + 2));
}

// one gradient: rows of A (positions for grad_x, output channels for grad_w), reduction length
struct GradientPlan {
    int M, K, kt;
    long long total;
    size_t image_bytes;
};
GradientPlan plan_gradient(const Shape& s, bool weights, int ct) {
    GradientPlan g;
    g.M = weights ? s.COg : static_cast<int>(s.M);
    g.K = weights ? static_cast<int>(s.M) : s.COg;
    g.kt = stages_of(g.K);
    g.total = static_cast<long long>(s.G) * row_tiles(g.M) * div_up(s.CIg, ct) * g.kt;
    g.image_bytes = static_cast<size_t>(s.G) * 2 * row_tiles(g.M) * kBlocks * g.kt * kABytes;
    return g;
}
size_t gradient_part_floats(const Shape& s, bool gx, bool gw, int ct, int cap) {
    size_t most = 0;
    for (int k = 0; k < 2; ++k) {
        if (!(k == 0 ? gx : gw)) continue;
        const GradientPlan g = plan_gradient(s, k == 1, ct);
        const size_t n = part_floats(g.M, g.total, g.kt, cap, ct);
        most = n > most ? n : most;
    }
    return most;
}

// ranges of rows for the coefficients' column sums
int row_splits(const Shape& s) {
    const int n = div_up(s.M, 128);
    return n < kMaxSplits ? n : kMaxSplits;
}

// words that a backward call clears: codes of the extremes of the channels of x and w, and single ones
inline size_t channel_words(const Shape& s) { return 4 * static_cast<size_t>(s.CI) + 8; }
// ranges of rows for the channels' sums: at most kMaxRanges, of kColumnRows rows or more (images: of any number of samples)
inline void channel_ranges(int rows, bool columns, int* ranges, int* in_each) {
    *in_each = div_up(rows, kMaxRanges);
    if (columns && *in_each < kColumnRows) *in_each = kColumnRows;
    *ranges = div_up(rows, *in_each);
}

template <int PW>
int backward_power(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx, float* gw,
                   bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond, cudaStream_t st) {
    constexpr int NP = PW - 1;
    constexpr int CT = channels_of(NP);
    const size_t rows = static_cast<size_t>(s.G) * s.M;
    const int splits = row_splits(s);
    BackwardStats A{};
    A.s = s;
    A.coef = coef; A.x = x; A.w = w; A.y = y; A.pitch = pitch;
    A.row_exp = bump->take<int>(rows);
    A.row_sum = bump->take<float>(rows);
    A.out_exp = bump->take<int>(s.CO);
    A.out_sum = bump->take<float>(s.CO);
    A.channel_pitch = div_up(s.CIg, CT) * CT;
    const size_t scales = static_cast<size_t>(s.G) * A.channel_pitch;
    float* channels = bump->take<float>(4 * scales);
    const size_t words_size = channel_words(s);
    unsigned* words = bump->take<unsigned>(words_size);
    A.part_top = bump->take<unsigned>(static_cast<size_t>(splits) * s.CO);
    A.part_sum = bump->take<double>(static_cast<size_t>(splits) * s.CO);
    A.part_abs = bump->take<float>(static_cast<size_t>(splits) * s.CO);
    channel_ranges(s.B, s.HW == 1, &A.x_ranges, &A.x_rows);
    channel_ranges(s.COg, true, &A.w_ranges, &A.w_rows);
    A.x_part = bump->take<double2>(static_cast<size_t>(A.x_ranges) * s.CI);
    A.w_part = bump->take<double2>(static_cast<size_t>(A.w_ranges) * s.CI);
    A.blocks_channels = s.G * div_up(s.CIg, 32);
    A.spread_part = bump->take<double>(A.blocks_channels);
    const GradientPlan px = plan_gradient(s, false, CT), pw = plan_gradient(s, true, CT);
    char* images_x = gx ? bump->take<char>(px.image_bytes) : nullptr;
    char* images_w = gw ? bump->take<char>(pw.image_bytes) : nullptr;
    float* partials = bump->take<float>(gradient_part_floats(s, gx != nullptr, gw != nullptr, CT, cap));
    if (!A.row_exp || !A.row_sum || !A.out_exp || !A.out_sum || !channels || !words || !A.part_top || !A.part_sum || !A.part_abs ||
        !A.x_part || !A.w_part || !A.spread_part || (gx && !images_x) || (gw && !images_w) || !partials)
        return kWorkspace;
    A.p = PW;
    A.per_x = 1.0 / static_cast<double>(s.M);
    A.per_w = 1.0 / s.COg;
    A.down_w = channels; A.down_x = channels + scales;
    A.shift_w = channels + 2 * scales; A.shift_x = channels + 3 * scales;
    A.x_top = words; A.x_low = A.x_top + s.CI; A.w_top = A.x_low + s.CI; A.w_low = A.w_top + s.CI;
    unsigned* single = A.w_low + s.CI;
    A.bad = reinterpret_cast<int*>(single);
    A.cond = A.bad + 1;
    A.y_low = single + 2; A.most = single + 3;
    A.range = range;
    A.need_x = gx != nullptr;
    A.need_w = gw != nullptr;
    *cond = A.cond;
    cudaError_t e = cudaMemsetAsync(words, 0, words_size * sizeof(unsigned), st);
    // (scales and shifts of the padding channels are multiplied with zeros: they only have to be numbers)
    if (e == cudaSuccess && A.channel_pitch != s.CIg) e = cudaMemsetAsync(channels, 0, 4 * scales * sizeof(float), st);
    if (e != cudaSuccess) return cuda_status(e);
    A.splits = splits;
    A.rows_per_split = div_up(s.M, splits);
    A.blocks_rows = div_up(static_cast<long long>(rows), 8);
    A.blocks_cols = splits * s.G * div_up(s.COg, 32);
    A.blocks_w = div_up(s.CIg, 32) * s.G * A.w_ranges;
    A.blocks_x = s.HW == 1 ? div_up(s.CI, 32) * A.x_ranges : div_up(static_cast<long long>(A.x_ranges) * s.CI, 8);
    A.blocks_y = div_up(s.M * s.CO, 16 * kPrep);
    if (A.blocks_y > 1184) A.blocks_y = 1184;
    int r = launch_after(even_stats_kernel, A.blocks_rows + A.blocks_cols + A.blocks_w + A.blocks_x + A.blocks_y, kPrep, 0, st, A);
    if (r != kOk) return r;
    if ((r = launch_after(even_scales_kernel, A.blocks_channels + div_up(s.CO, kPrep / 32), kPrep, 0, st, A)) != kOk) return r;
    CoefImages X{}, W{};
    const long long group = static_cast<long long>(s.M) * pitch;
    X.src = Source{coef, s.COg % 4 == 0 ? 0 : 1, static_cast<int>(s.M), s.COg, 0, pitch, 1, 0, group};
    auto blocks_of = [&](CoefImages& J, const GradientPlan& g, char* images) {
        J.images = images;
        J.split = split_rows(g.M);
        J.tiles_m = row_blocks(g.M);
        J.kb = kBlocks * g.kt;
        J.blocks = images ? s.G * J.tiles_m * J.kb : 0;
    };
    blocks_of(X, px, images_x);
    X.exp = A.row_exp;
    W.src = Source{coef, 2, s.COg, static_cast<int>(s.M), 0, 1, pitch, 0, group};
    blocks_of(W, pw, images_w);
    W.exp = A.out_exp;
    if ((r = launch_after(even_coef_kernel, X.blocks + W.blocks + 1, kPrep, 0, st, A, X, W)) != kOk) return r;
    EvenParams P{};
    P.G = s.G;
    P.N = s.CIg;
    P.tiles_n = div_up(s.CIg, CT);
    P.gate0 = range;
    P.gate1 = A.cond;
    P.partials = partials;
    P.status = status;
    auto rows_of = [&](const GradientPlan& g) {
        P.M = g.M;
        P.kt = g.kt;
        P.tiles_m = row_tiles(g.M);
        P.total = static_cast<int>(g.total);
        P.split = split_rows(g.M);
        P.slots = part_slots(g.M, g.total, g.kt, workers_of(g.total, cap));
    };
    if (gx) {
        rows_of(px);
        P.images = images_x;
        P.src = channels_of_w(w, s);
        P.out = OutAddr{static_cast<long long>(s.CI) * s.HW, 1, static_cast<long long>(s.CIg) * s.HW, s.HW, s.HW};
        P.vec = s.HW == 1 && s.CIg % 4 == 0 && aligned16(x) && aligned16(gx);
        P.out_f = gx;
        P.resident = x;
        P.col_down = A.down_w; P.col_shift = A.shift_w; P.row_exp = A.row_exp; P.row_sum = A.row_sum;
        if ((r = launch_even<PW, false>(P, cap, st)) != kOk) return r;
    }
    if (gw) {
        rows_of(pw);
        P.images = images_w;
        P.src = channels_of_x(x, s);
        P.out = OutAddr{s.CIg, 0, static_cast<long long>(s.COg) * s.CIg, 1, 1};
        P.vec = s.CIg % 4 == 0 && aligned16(w) && aligned16(gw);
        P.out_f = gw;
        P.resident = w;
        P.accumulate = accumulate_gw;
        P.col_down = A.down_x; P.col_shift = A.shift_x; P.row_exp = A.out_exp; P.row_sum = A.out_sum;
        if ((r = launch_even<PW, false>(P, cap, st)) != kOk) return r;
    }
    return kOk;
}

}  // namespace
}  // namespace ldn
