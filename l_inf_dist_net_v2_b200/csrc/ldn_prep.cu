#include "ldn_prep.cuh"

namespace ldn {

namespace {
constexpr int kBlock = kPostBlock;
constexpr int kRescanInplaceMaxSmem = 200 * 1024;  // input slab of rescan_inplace_kernel
constexpr int kColumnWarps = 4;                       // warps of a block of the scatters by columns
constexpr int kColumnMaxChannels = 224;               // channels of a column: two blocks of four warps per SM
constexpr long long kColumnLeastOutputs = 16384;      // (below, the launch more costs as much as the atomics)
constexpr int kRescanIlp = 4;                         // outputs in flight per lane group of rescan_kernel
constexpr int kRescanStep = kRescanIlp * kBlock / 4;  // outputs a block of rescan_kernel handles in one step
constexpr long long kRescanBlocks = 148 * 32;         // its blocks beyond which each takes several steps of one input row
// grid of a kernel that usually returns at once (gated): small, the grid-stride loops cover the rest when it runs
inline unsigned gated_blocks(unsigned blocks, const int* gate) { return (gate && blocks > 592u) ? 592u : blocks; }
inline unsigned blocks_for(long long n) {
    long long b = (n + kBlock - 1) / kBlock;
    if (b < 1) b = 1;
    if (b > 1184 * 8) b = 1184 * 8;  // grid-stride beyond this
    return static_cast<unsigned>(b);
}

// Copies that only gated kernels read run when one of those will (gates: either word not 0; null, null: always).
__device__ __forceinline__ bool copy_wanted(const CopyGate& g) {
    return (g.a == nullptr && g.b == nullptr) || (g.a && *g.a != 0) || (g.b && *g.b != 0);
}

__global__ void canon_x_kernel(const float* x, float* xc, Shape s, int pitch, CopyGate gate) {
    stream_order_begin();
    if (!copy_wanted(gate)) return;
    const long long total = static_cast<long long>(s.G) * s.M * s.CIg;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const CanonIdx q = canon_idx(i, s.CIg, s.M);
        const long long b = q.m / s.HW, hw = q.m % s.HW;
        xc[(static_cast<long long>(q.g) * s.M + q.m) * pitch + q.c] = x[((b * s.G + q.g) * s.CIg + q.c) * s.HW + hw];
    }
}

__global__ void canon_bounds_kernel(const float* xl, const float* xu, float* lc,
                                    float* uc, Shape s, int pitch) {
    stream_order_begin();
    const long long total = static_cast<long long>(s.G) * s.M * s.CIg;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const CanonIdx q = canon_idx(i, s.CIg, s.M);
        const long long b = q.m / s.HW, hw = q.m % s.HW;
        const long long src = ((b * s.G + q.g) * s.CIg + q.c) * s.HW + hw;
        float lo = xl[src], up = xu[src];
        if (lo > up) lo = up = (lo + up) * 0.5f;
        const long long dst = (static_cast<long long>(q.g) * s.M + q.m) * pitch + q.c;
        lc[dst] = lo;
        uc[dst] = up;
    }
}

// HW > 1: tiled transpose through shared memory.  Source rows (b, g, c, :) are contiguous in hw, destination
// rows (g, m = b HW + hw, :) are contiguous in c; a 32 x 32 tile makes both sides coalesced.  grid = (ceil(HW/32),
// ceil(CIg/32), B*G).  With `second` non-null the pair (x, second) is treated as interval bounds and sanitised.
__global__ void canon_transpose_kernel(const float* x, const float* second,
                                       float* xc, float* sc, Shape s, int pitch, CopyGate gate) {
    stream_order_begin();
    if (!copy_wanted(gate)) return;
    __shared__ float t0[32][33], t1[32][33];
    const int bg = blockIdx.z, b = bg / s.G, g = bg % s.G;
    const int hw0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
    const float* src = x + (static_cast<long long>(bg) * s.CIg) * s.HW;
    const float* src2 = second ? second + (static_cast<long long>(bg) * s.CIg) * s.HW : nullptr;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int c = c0 + r, hw = hw0 + threadIdx.x;
        if (c < s.CIg && hw < s.HW) {
            float lo = src[static_cast<long long>(c) * s.HW + hw];
            if (src2) {
                float up = src2[static_cast<long long>(c) * s.HW + hw];
                if (lo > up) lo = up = (lo + up) * 0.5f;
                t1[r][threadIdx.x] = up;
            }
            t0[r][threadIdx.x] = lo;
        }
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int hw = hw0 + r, c = c0 + threadIdx.x;
        if (c < s.CIg && hw < s.HW) {
            const long long dst = (static_cast<long long>(g) * s.M + static_cast<long long>(b) * s.HW + hw) * pitch + c;
            xc[dst] = t0[threadIdx.x][r];
            if (src2) sc[dst] = t1[threadIdx.x][r];
        }
    }
}

__global__ void canon_w_kernel(const float* w, float* wc, Shape s, int pitch, CopyGate gate) {
    stream_order_begin();
    if (!copy_wanted(gate)) return;
    const long long total = static_cast<long long>(s.CO) * s.CIg;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long row = i / s.CIg;
        const int c = static_cast<int>(i - row * s.CIg);
        wc[row * pitch + c] = w[i];
    }
}

// Range guard of the integer-q coefficient g / y^q: *flag is raised when some y^-q is outside [kRqMin, kRqMax]
// (beyond: y^-q overflows or |t|^q <= y^q goes denormal; below: the coefficient loses its bits).  The caller clears
// the word beforehand; flag may be null (q = 0).
constexpr float kRqMin = 1e-30f, kRqMax = 1e24f;
__device__ __forceinline__ bool rq_unsafe(float rq) { return !(rq >= kRqMin && rq <= kRqMax); }

__global__ void coef_int_kernel(const float* go, const float* y, float* coef,
                                Shape s, int pitch, int iq, int* flag) {
    stream_order_begin();
    const long long total = static_cast<long long>(s.G) * s.M * s.COg;
    bool bad = false;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const CanonIdx q = canon_idx(i, s.COg, s.M);
        const long long src = y_offset(s, q);
        const float r = 1.0f / y[src];
        float rq = 1.0f;
        for (int k = 0; k < iq; ++k) rq *= r;
        bad |= rq_unsafe(rq);
        coef[(static_cast<long long>(q.g) * s.M + q.m) * pitch + q.c] = go[src] * rq;
    }
    if (flag && bad) *flag = 1;
}

// HW > 1: the same through shared memory.  Rows (b, g, o, :) of go / y are contiguous in hw, rows (g, m, :) of the coefficients
// contiguous in o; a 32 x 32 tile makes both sides coalesced (one thread per coefficient read 4 bytes from every 4 HW).  grid =
// (ceil(HW/32), ceil(COg/32), B*G).
__global__ void __launch_bounds__(kBlock) coef_int_transpose_kernel(const float* go, const float* y, float* coef, Shape s,
                                                                    int pitch, int iq, int* flag) {
    stream_order_begin();
    __shared__ float tile[32][33];
    const int bg = blockIdx.z, b = bg / s.G, g = bg - b * s.G;
    const int hw0 = blockIdx.x * 32, o0 = blockIdx.y * 32;
    const long long src = s.co_src != s.CO ? (static_cast<long long>(b) * s.co_src + s.co_off) * s.HW
                                           : static_cast<long long>(bg) * s.COg * s.HW;
    bool bad = false;
#pragma unroll
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int o = o0 + r, hw = hw0 + threadIdx.x;
        if (o < s.COg && hw < s.HW) {
            const long long i = src + static_cast<long long>(o) * s.HW + hw;
            const float inv = 1.0f / y[i];
            float rq = 1.0f;
            for (int k = 0; k < iq; ++k) rq *= inv;
            bad |= rq_unsafe(rq);
            tile[r][threadIdx.x] = go[i] * rq;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int hw = hw0 + r, o = o0 + threadIdx.x;
        if (o < s.COg && hw < s.HW)
            coef[(g * s.M + static_cast<long long>(b) * s.HW + hw) * pitch + o] = tile[threadIdx.x][r];
    }
    if (flag && bad) *flag = 1;
}

// flat fast paths (HW == 1, G == 1, pitch == COg: source and destination have the same element order)
__global__ void coef_int_flat_kernel(const float4* go, const float4* y,
                                     float4* coef, long long n4, int iq, int* flag) {
    stream_order_begin();
    bool bad = false;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
        const float4 yv = y[i];
        const float4 gv = go[i];
        const float4 r = make_float4(1.0f / yv.x, 1.0f / yv.y, 1.0f / yv.z, 1.0f / yv.w);
        float4 rq = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        for (int k = 0; k < iq; ++k) {
            rq.x *= r.x; rq.y *= r.y; rq.z *= r.z; rq.w *= r.w;
        }
        bad |= rq_unsafe(rq.x) | rq_unsafe(rq.y) | rq_unsafe(rq.z) | rq_unsafe(rq.w);
        coef[i] = make_float4(gv.x * rq.x, gv.y * rq.y, gv.z * rq.z, gv.w * rq.w);
    }
    if (flag && bad) *flag = 1;
}
__global__ void __launch_bounds__(kBlock) coef_gen_kernel(const CoefJob job) {
    stream_order_begin();
    coef_gen_block(job, blockIdx.x, gridDim.x);
}

// Four lanes per output element, kRescanIlp outputs per lane group in flight: lane q of a group loads the 16-byte pieces q
// and q + 4 of the recorded 32-channel stage of each operand row (one full 128-byte line per output and operand: operand
// views are 16-byte aligned with row pitches that are multiples of 4 floats), finds the lowest matching channel among its
// eight, and a minimum over the group's lanes keeps the lowest channel of the stage -- the index a strictly-greater scan in
// ascending order ends with.  The search is a chain of two dependent loads (stage id, then the pieces), so it is bound by
// their latency unless several outputs are in flight per lane, and then by the L2 reads of the weight pieces (128 bytes
// per output) and by its instructions (hence four lanes with two pieces rather than eight with one).
// (512 x 5120 -> 5120 forward + backward 1149 -> 1116 us, of which the search was 99 with one output in flight.)
// blockIdx.x = (sample, group); blockIdx.y walks that pair's CO/G * HW outputs in steps of kRescanStep, so the index
// arithmetic per output is one division by HW (none for fully connected layers) and, for those, a block keeps rereading
// one input row, which stays in the L1 cache: only the weight pieces come from L2.
template <int mode>
__global__ void __launch_bounds__(kBlock) rescan_kernel(Operand a0, Operand a1, Operand b, const float* y,
                                                        int* pos, Shape s, long long a_stride_k, const int* gate) {
    stream_order_begin();
    if (gate && *gate == 0) return;
    constexpr int U = kRescanIlp;
    const int kpad = (s.CIg + 3) & ~3;
    const int q = threadIdx.x & 3;
    const int group_in_block = threadIdx.x >> 2;
    const unsigned cohw = static_cast<unsigned>(s.COg) * static_cast<unsigned>(s.HW);  // < 2^31, checked by the launcher
    const long long bg = blockIdx.x;
    const int bi = static_cast<int>(bg / s.G), g = static_cast<int>(bg - static_cast<long long>(bi) * s.G);
    const float* arow = a0.ptr + g * a0.stride_group;
    const float* urow = a1.ptr + g * a1.stride_group;
    const float* brow = b.ptr + g * b.stride_group;
    // (the trip counts are the same for all lanes of a warp: its eight groups handle consecutive outputs)
    for (unsigned j0 = blockIdx.y * kRescanStep; j0 < cohw; j0 += gridDim.y * kRescanStep) {
        int stage[U];
        float yv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned j = j0 + u * (kBlock / 4) + group_in_block;
            const bool valid = j < cohw;
            stage[u] = valid ? pos[bg * cohw + j] : -1;
            yv[u] = valid ? y[bg * cohw + j] : 0.0f;
        }
        int best[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            best[u] = 0x7fffffff;
            const unsigned j = j0 + u * (kBlock / 4) + group_in_block;
            if (stage[u] >= 0) {
                const unsigned o = s.HW == 1 ? j : j / static_cast<unsigned>(s.HW);
                const unsigned hw = j - o * s.HW;
                const long long m = static_cast<long long>(bi) * s.HW + hw;
#pragma unroll
                for (int h = 1; h >= 0; --h) {
                    const int k = stage[u] * 32 + 16 * h + 4 * q;
                    if (k < kpad) {
                        float4 av;
                        if (a_stride_k == 1) {
                            av = *reinterpret_cast<const float4*>(arow + m * a0.stride_row + k);
                        } else {
                            // input read in place (channels HW apart, no padding behind the last one)
                            const float* ap = a0.ptr + bg * a0.stride_group + hw * a0.stride_row + k * a_stride_k;
                            av.x = ap[0];
                            av.y = k + 1 < s.CIg ? ap[a_stride_k] : 0.0f;
                            av.z = k + 2 < s.CIg ? ap[2 * a_stride_k] : 0.0f;
                            av.w = k + 3 < s.CIg ? ap[3 * a_stride_k] : 0.0f;
                        }
                        const float4 bv = *reinterpret_cast<const float4*>(brow + o * b.stride_row + k);
                        float4 uv = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (mode != 0) uv = *reinterpret_cast<const float4*>(urow + m * a1.stride_row + k);
                        const float ae[4] = {av.x, av.y, av.z, av.w};
                        const float be[4] = {bv.x, bv.y, bv.z, bv.w};
                        const float ue[4] = {uv.x, uv.y, uv.z, uv.w};
#pragma unroll
                        for (int e = 3; e >= 0; --e) {
                            bool hit, flag;
                            if (mode == 0) {
                                const float d = ae[e] - be[e];
                                hit = fabsf(d) == yv[u];
                                flag = d < 0.0f;
                            } else {
                                const float t1 = be[e] - ae[e], t2v = ue[e] - be[e];
                                hit = (mode == 1) ? (fminf(t1, t2v) == -yv[u]) : (fmaxf(t1, t2v) == yv[u]);
                                flag = !(t1 <= t2v);
                            }
                            if (hit && k + e < s.CIg) best[u] = ((k + e) << 1) | (flag ? 1 : 0);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            best[u] = min(best[u], __shfl_xor_sync(0xffffffffu, best[u], 1));
            best[u] = min(best[u], __shfl_xor_sync(0xffffffffu, best[u], 2));
            const unsigned j = j0 + u * (kBlock / 4) + group_in_block;
            if (j < cohw && q == 0) {
                int result = (mode == 1) ? static_cast<int>(0xffffffffu) : 0;
                if (best[u] != 0x7fffffff) result = (best[u] >> 1) | ((best[u] & 1) ? static_cast<int>(0x80000000u) : 0);
                pos[bg * cohw + j] = result;
            }
        }
    }
}

// The same search for inputs read in place (x[B, C, HW]: the channels of an output are HW floats apart, so the
// kernel above pulls one 32-byte sector per channel and output from L2).  Here a block owns P neighbouring
// positions of one (sample, group): it copies their CI/G x P input values to shared memory once (rows of P floats,
// coalesced), then every thread scans the 32 channels of its output's stage there; a warp holds P consecutive
// positions of 32 / P outputs, so y / pos are read and written coalesced and the shared-memory reads are
// conflict-free whatever the lanes' stages.  The weight pieces (one 128-byte run per output and stage) come from L1 / L2.
template <int P>
__global__ void __launch_bounds__(kBlock) rescan_inplace_kernel(Operand a0, Operand b, const float* y,
                                                                int* pos, Shape s) {
    stream_order_begin();
    extern __shared__ float4 xs4[];
    float* xs = reinterpret_cast<float*>(xs4);  // [CI/G][P]
    constexpr int V = P / 4;
    const long long bg = blockIdx.x;
    const int g = static_cast<int>(bg % s.G);
    const int hw0 = blockIdx.y * P;
    const float* xsrc = a0.ptr + bg * a0.stride_group;
    for (int idx = threadIdx.x; idx < s.CIg * V; idx += kBlock) {
        const int c = idx / V, v = idx - c * V;
        const int hw = hw0 + 4 * v;
        float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
        if (hw < s.HW) val = *reinterpret_cast<const float4*>(xsrc + static_cast<long long>(c) * s.HW + hw);
        xs4[idx] = val;
    }
    __syncthreads();
    const int hl = threadIdx.x % P;
    const int hw = hw0 + hl;
    if (hw >= s.HW) return;
    const int kpad = (s.CIg + 3) & ~3;
    const float* brow = b.ptr + g * b.stride_group;
    const long long base = bg * (static_cast<long long>(s.COg) * s.HW) + hw;
    for (int o = threadIdx.x / P; o < s.COg; o += kBlock / P) {
        const long long i = base + static_cast<long long>(o) * s.HW;
        const int stage = pos[i];
        int result = 0;
        if (stage >= 0) {
            const float yv = y[i];
            const int k0 = stage * 32;
            const float* wr = brow + o * b.stride_row + k0;
            int best = -1;
            bool neg = false;
#pragma unroll
            for (int c4 = 7; c4 >= 0; --c4) {
                const int k = k0 + 4 * c4;
                if (k < kpad) {
                    const float4 wv = *reinterpret_cast<const float4*>(wr + 4 * c4);
                    const float we[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                    for (int e = 3; e >= 0; --e) {
                        if (k + e < s.CIg) {
                            const float d = xs[(k + e) * P + hl] - we[e];
                            if (fabsf(d) == yv) {
                                best = k + e;
                                neg = d < 0.0f;
                            }
                        }
                    }
                }
            }
            if (best >= 0) result = best | (neg ? static_cast<int>(0x80000000u) : 0);
        }
        pos[i] = result;
    }
}

template <int P>
int launch_rescan_inplace(Operand a0, Operand b, const float* y, int* pos, const Shape& s, cudaStream_t st) {
    static OncePerDevice once;
    const int smem = s.CIg * P * static_cast<int>(sizeof(float));
    const int r = once([] { return allow_smem(rescan_inplace_kernel<P>, kRescanInplaceMaxSmem); });
    if (r != kOk) return r;
    const dim3 grid(static_cast<unsigned>(static_cast<long long>(s.B) * s.G), static_cast<unsigned>((s.HW + P - 1) / P));
    return launch_after(rescan_inplace_kernel<P>, grid, kBlock, smem, st, a0, b, y, pos, s);
}

// out[g * rows + r] = max_k |v[g][r][k]|.  Contiguous k: one warp per row; k `stride_k` apart with neighbouring rows
// contiguous (inputs read in place): one thread per row.  clear (may be null): a flag word the first thread resets.
__global__ void row_absmax_kernel(Operand v, long long rows, int inner, int groups, float* out, int* clear) {
    stream_order_begin();
    if (clear && blockIdx.x == 0 && threadIdx.x == 0) *clear = 0;
    const int lane = threadIdx.x & 31;
    const long long warps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
    const long long total = rows * groups;
    for (long long i = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; i < total; i += warps) {
        const long long g = i / rows, r = i - g * rows;
        const float* src = v.ptr + g * v.stride_group + r * v.stride_row;
        float m = 0.0f;
        for (int k = lane; k < inner; k += 32) m = fmaxf(m, fabsf(src[k]));
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
        if (lane == 0) out[i] = m;
    }
}
__global__ void row_absmax_strided_kernel(Operand v, long long rows, int inner, int groups, long long stride_k,
                                          float* out, int* clear) {
    stream_order_begin();
    if (clear && blockIdx.x == 0 && threadIdx.x == 0) *clear = 0;
    const long long total = rows * groups;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const long long g = i / rows, r = i - g * rows;
        const float* src = v.ptr + g * v.stride_group + r * v.stride_row;
        float m = 0.0f;
        for (int k = 0; k < inner; ++k) m = fmaxf(m, fabsf(src[k * stride_k]));
        out[i] = m;
    }
}

// The gradients a scatter adds into, cleared in one launch (a memset per gradient costs a launch each, and the scatter could
// not be set up behind it: bounds of 100 x 1023 -> 500, forward + backward, 100 -> 95 us).
struct ZeroArgs {
    float* p[3];
    long long n[3];
};
__global__ void __launch_bounds__(kBlock) zero_kernel(const ZeroArgs A) {
    stream_order_begin();
    const long long first = blockIdx.x * (long long)kBlock + threadIdx.x, step = (long long)gridDim.x * kBlock;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float* p = A.p[k];
        if (p == nullptr) continue;
        const long long n4 = (reinterpret_cast<uintptr_t>(p) & 15u) == 0 ? A.n[k] / 4 : 0;
        for (long long i = first; i < n4; i += step) reinterpret_cast<float4*>(p)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (long long i = 4 * n4 + first; i < A.n[k]; i += step) p[i] = 0.0f;
    }
}

// One thread per output element, in output-layout order (coalesced reads of go / pos).
__global__ void inf_scatter_kernel(const float* go, const int* pos, float* gx, float* gw,
                                   Shape s) {
    stream_order_begin();
    const long long total = static_cast<long long>(s.B) * s.CO * s.HW;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int hw = static_cast<int>(i % s.HW);
        const long long t = i / s.HW;
        const int o = static_cast<int>(t % s.COg);
        const long long t2 = t / s.COg;
        const int g = static_cast<int>(t2 % s.G);
        const long long b = t2 / s.G;
        const int ps = pos[i];
        const int idx = ps & 0x7fffffff;
        const float v = ps >= 0 ? go[i] : -go[i];
        if (gx) atomicAdd(&gx[((b * s.G + g) * s.CIg + idx) * s.HW + hw], v);
        if (gw) atomicAdd(&gw[(static_cast<long long>(g) * s.COg + o) * s.CIg + idx], -v);
    }
}

// The same two gradients where an output has many positions (convolutions).  The kernel above is bound by its atomics there:
// every position adds into the same CO x CI/G weight gradient (128 x 1024 positions of 64 channels -> 64: 218 us for both
// gradients, 162 of them the weight's), and the input gradient is cleared first and then read and written by pieces of 4
// bytes.  Here a lane owns one position and its own column of a shared-memory tile [channels][32 lanes] (bank = lane, whatever
// the channels the lanes add to), so nothing on the way is atomic and no lane waits for another: 47 us (columns 28, of which
// reading and writing 101 MB are 15; weights 19).  4 groups of 144 channels -> 16 over 128 x 256 positions: 75 -> 32 us.
// The weight's sums are closer to 64 bits too (relative error 9e-7 -> 1.4e-7): a column adds up a 32nd of the positions.
//
// Input gradient: one lane per (sample, position, group) adds its CO/G outputs into its column and writes all the column's
// channels, zeros included.  It also clears the weight gradient (gw, may be null) for the kernel behind it.
__global__ void __launch_bounds__(kColumnWarps * 32) inf_scatter_columns_kernel(const float* go, const int* pos, float* gx,
                                                                                float* gw, long long nw, Shape s) {
    stream_order_begin();
    extern __shared__ float columns[];
    if (gw) {
        const long long step = static_cast<long long>(gridDim.x) * gridDim.y * blockDim.x;
        const long long block = blockIdx.y * static_cast<long long>(gridDim.x) + blockIdx.x;
        for (long long i = block * blockDim.x + threadIdx.x; i < nw; i += step) gw[i] = 0.0f;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long m = (blockIdx.x * (long long)kColumnWarps + warp) * 32 + lane;
    if (m >= s.M) return;
    float* col = columns + warp * s.CIg * 32 + lane;
    const int g = blockIdx.y;
    const long long b = m / s.HW;
    const int hw = static_cast<int>(m - b * s.HW);
    for (int c = 0; c < s.CIg; ++c) col[c * 32] = 0.0f;
    const long long out = (b * s.G + g) * s.COg * (long long)s.HW + hw;
    constexpr int U = 8;  // outputs in flight
    for (int o0 = 0; o0 < s.COg; o0 += U) {
        int ps[U];
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const bool valid = o0 + u < s.COg;
            const long long i = out + static_cast<long long>(o0 + u) * s.HW;
            ps[u] = valid ? pos[i] : 0x7fffffff;
            v[u] = valid ? go[i] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = ps[u] & 0x7fffffff;
            if (c < s.CIg) col[c * 32] += ps[u] >= 0 ? v[u] : -v[u];
        }
    }
    float* dst = gx + (b * s.G + g) * s.CIg * (long long)s.HW + hw;
#pragma unroll 4
    for (int c = 0; c < s.CIg; ++c) dst[static_cast<long long>(c) * s.HW] = col[c * 32];
}

// Weight gradient: a warp owns one output channel and a range of positions, and adds its columns' sums to the gradient at
// the end.
__global__ void __launch_bounds__(kColumnWarps * 32) inf_scatter_weight_kernel(const float* go, const int* pos, float* gw,
                                                                               Shape s, int splits) {
    stream_order_begin();
    extern __shared__ float columns[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long job = blockIdx.x * (long long)kColumnWarps + warp;
    if (job >= static_cast<long long>(s.CO) * splits) return;
    const int channel = static_cast<int>(job / splits), split = static_cast<int>(job - static_cast<long long>(channel) * splits);
    float* tile = columns + warp * s.CIg * 32;
    for (int c = 0; c < s.CIg; ++c) tile[c * 32 + lane] = 0.0f;
    const unsigned hws = static_cast<unsigned>(s.HW);
    const unsigned first = static_cast<unsigned>(s.M * split / splits), last = static_cast<unsigned>(s.M * (split + 1) / splits);
    const long long plane = static_cast<long long>(s.CO) * s.HW, at = static_cast<long long>(channel) * s.HW;
    constexpr int U = 8;  // positions in flight per lane
    for (unsigned m0 = first; m0 < last; m0 += 32 * U) {
        int ps[U];
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned m = m0 + u * 32 + lane;
            const bool valid = m < last;
            const unsigned b = m / hws;
            const long long i = b * plane + at + (m - b * hws);
            ps[u] = valid ? pos[i] : 0x7fffffff;
            v[u] = valid ? go[i] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = ps[u] & 0x7fffffff;
            if (c < s.CIg) tile[c * 32 + lane] += ps[u] >= 0 ? v[u] : -v[u];
        }
    }
    __syncwarp();
    // a lane adds up one channel's 32 columns, each lane from another column on (no bank conflicts)
    float* dst = gw + static_cast<long long>(channel) * s.CIg;
    for (int c = lane; c < s.CIg; c += 32) {
        float sum = 0.0f;
#pragma unroll
        for (int j = 0; j < 32; ++j) sum += tile[c * 32 + ((j + lane) & 31)];
        if (sum != 0.0f) atomicAdd(&dst[c], -sum);
    }
}

__global__ void bound_scatter_kernel(const float* gol, const float* gou,
                                     const int* posl, const int* posu, float* gxl, float* gxu,
                                     float* gw, Shape s) {
    stream_order_begin();
    const long long total = static_cast<long long>(s.B) * s.CO * s.HW;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int hw = static_cast<int>(i % s.HW);
        const long long t = i / s.HW;
        const int o = static_cast<int>(t % s.COg);
        const long long t2 = t / s.COg;
        const int g = static_cast<int>(t2 % s.G);
        const long long b = t2 / s.G;
        const int pl = posl[i], pu = posu[i];
        const int il = pl & 0x7fffffff, iu = pu & 0x7fffffff;
        const float vl = pl >= 0 ? gol[i] : -gol[i];
        const float vu = pu >= 0 ? gou[i] : -gou[i];
        const long long xrow = ((b * s.G + g) * s.CIg) * (long long)s.HW + hw;
        const long long wrow = (static_cast<long long>(g) * s.COg + o) * s.CIg;
        if (pl != static_cast<int>(0xffffffffu)) {
            float* dst = pl >= 0 ? gxl : gxu;
            atomicAdd(&dst[xrow + static_cast<long long>(il) * s.HW], vl);
            if (gw) atomicAdd(&gw[wrow + il], -vl);
        }
        float* dst = pu >= 0 ? gxu : gxl;
        atomicAdd(&dst[xrow + static_cast<long long>(iu) * s.HW], vu);
        if (gw) atomicAdd(&gw[wrow + iu], -vu);
    }
}
}  // namespace



static bool transpose_grid(const Shape& s, int channels, dim3* grid) {
    const long long bg = static_cast<long long>(s.B) * s.G;
    if (s.HW < 8 || bg > 65535 || (channels + 31) / 32 > 65535) return false;
    *grid = dim3((s.HW + 31) / 32, (channels + 31) / 32, static_cast<unsigned>(bg));
    return true;
}

int launch_canon_x(const float* x, float* xc, const Shape& s, int pitch, CopyGate gate, cudaStream_t st) {
    dim3 grid;
    if (transpose_grid(s, s.CIg, &grid)) {
        return launch_after(canon_transpose_kernel, grid, dim3(32, 8), 0, st, x, nullptr, xc, nullptr, s, pitch, gate);
    }
    return launch_after(canon_x_kernel, blocks_for((long long)s.G * s.M * s.CIg), kBlock, 0, st, x, xc, s, pitch, gate);
}
int launch_canon_bounds(const float* xl, const float* xu, float* lc, float* uc, const Shape& s, int pitch,
                        cudaStream_t st) {
    dim3 grid;
    if (transpose_grid(s, s.CIg, &grid)) {
        return launch_after(canon_transpose_kernel, grid, dim3(32, 8), 0, st, xl, xu, lc, uc, s, pitch, CopyGate{});
    }
    return launch_after(canon_bounds_kernel, blocks_for((long long)s.G * s.M * s.CIg), kBlock, 0, st, xl, xu, lc, uc,
                        s, pitch);
}
int launch_canon_w(const float* w, float* wc, const Shape& s, int pitch, CopyGate gate, cudaStream_t st) {
    return launch_after(canon_w_kernel, blocks_for((long long)s.CO * s.CIg), kBlock, 0, st, w, wc, s, pitch, gate);
}
static bool flat_ok(const Shape& s, int pitch, const void* a, const void* b) {
    return s.HW == 1 && s.G == 1 && s.co_src == s.CO && pitch == s.COg && (s.COg & 3) == 0 &&
           ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15u) == 0;
}

int launch_coef_int(const float* go, const float* y, float* coef, const Shape& s, int pitch, int iq, int* flag,
                    cudaStream_t st) {
    if (flat_ok(s, pitch, go, y)) {
        const long long n4 = static_cast<long long>(s.M) * s.COg / 4;
        return launch_after(coef_int_flat_kernel, blocks_for(n4), kBlock, 0, st, reinterpret_cast<const float4*>(go),
                            reinterpret_cast<const float4*>(y), reinterpret_cast<float4*>(coef), n4, iq, flag);
    }
    dim3 grid;
    if (transpose_grid(s, s.COg, &grid))
        return launch_after(coef_int_transpose_kernel, grid, dim3(32, 8), 0, st, go, y, coef, s, pitch, iq, flag);
    return launch_after(coef_int_kernel, blocks_for((long long)s.G * s.M * s.COg), kBlock, 0, st, go, y, coef, s,
                        pitch, iq, flag);
}
CoefJob coef_gen_job(const float* go, const float* y, float* rinv, float* gcp, const Shape& s, int pitch,
                     long long rows_pad, float q, bool fold, const int* gate) {
    const bool flat = flat_ok(s, pitch, go, y) && rows_pad == s.M;
    const long long items = flat ? s.M * s.COg / 4 : static_cast<long long>(s.G) * rows_pad * pitch;
    return CoefJob{go, y, rinv, gcp, s, pitch, rows_pad, q, fold, flat, gate,
                   static_cast<int>(gated_blocks(blocks_for(items), gate))};
}
int launch_coef_gen(const CoefJob& job, cudaStream_t st) {
    return launch_after(coef_gen_kernel, job.blocks, kBlock, 0, st, job);
}

int launch_rescan(int mode, Operand a0, Operand a1, Operand b, const float* y, int* pos, const Shape& s,
                  cudaStream_t st, long long a_stride_k, const int* gate) {
    if (a_stride_k != 1 && mode != 0) return kBadArgument;
    const long long cohw = static_cast<long long>(s.COg) * s.HW;
    const long long bg = static_cast<long long>(s.B) * s.G;
    if (cohw > 0x7fffffffLL || bg > 0x7fffffffLL) return kBadArgument;
    if (mode == 0 && a_stride_k != 1 && a_stride_k == s.HW && a0.stride_row == 1 && (s.HW & 3) == 0 &&
        (reinterpret_cast<uintptr_t>(a0.ptr) & 15u) == 0 && (s.HW + 7) / 8 <= 65535) {
        // inputs read in place: the largest slab of positions that leaves room for two blocks per SM, else the
        // largest that fits at all; beyond that (CI/G > 6400) the general kernel
        const long long row = static_cast<long long>(s.CIg) * sizeof(float);
        for (int pass = 0; pass < 2; ++pass) {
            const long long limit = pass == 0 ? 96 * 1024 : kRescanInplaceMaxSmem;
            if (row * 32 <= limit) return launch_rescan_inplace<32>(a0, b, y, pos, s, st);
            if (row * 16 <= limit) return launch_rescan_inplace<16>(a0, b, y, pos, s, st);
            if (row * 8 <= limit) return launch_rescan_inplace<8>(a0, b, y, pos, s, st);
        }
    }
    long long chunks = (cohw + kRescanStep - 1) / kRescanStep;
    const long long most = kRescanBlocks / bg > 1 ? kRescanBlocks / bg : 1;
    if (chunks > most) chunks = most;  // the kernel strides over the rest
    if (chunks > 65535) chunks = 65535;
    const dim3 grid(static_cast<unsigned>(bg), static_cast<unsigned>(chunks));
    if (mode == 0) return launch_after(rescan_kernel<0>, grid, kBlock, 0, st, a0, a1, b, y, pos, s, a_stride_k, gate);
    if (mode == 1) return launch_after(rescan_kernel<1>, grid, kBlock, 0, st, a0, a1, b, y, pos, s, a_stride_k, gate);
    return launch_after(rescan_kernel<2>, grid, kBlock, 0, st, a0, a1, b, y, pos, s, a_stride_k, gate);
}

int launch_row_absmax(Operand v, long long rows, int inner, int groups, long long stride_k, float* out, int* clear,
                      cudaStream_t st) {
    if (stride_k == 1)
        return launch_after(row_absmax_kernel, blocks_for(rows * groups * 32), kBlock, 0, st, v, rows, inner, groups, out,
                            clear);
    return launch_after(row_absmax_strided_kernel, blocks_for(rows * groups), kBlock, 0, st, v, rows, inner, groups,
                        stride_k, out, clear);
}

SideJob side_reduce_job(const float* part, float* gw, long long count, int tiles, bool accumulate, const int* gate,
                        bool run_if_nonzero) {
    const bool vec = (count & 3) == 0 && ((reinterpret_cast<uintptr_t>(part) | reinterpret_cast<uintptr_t>(gw)) & 15u) == 0;
    // many row tiles of a small weight (convolutions): with a thread per piece 512 blocks' worth of threads would not exist,
    // so the 8 warps of a block share the tiles of 32 pieces (256 tiles of 128 x 576: 40 us with a thread per piece; with this
    // and the coefficients by tiles, 46 us before, the fold by rows and the mean by planes the step went 1377 -> 1242 us)
    const bool wide = vec && tiles >= 32 && count / 4 < 512LL * kPostBlock;
    const long long threads = (vec ? count / 4 : count) * (wide ? 8 : 1);
    return SideJob{part, gw, count, tiles, accumulate, vec, wide, gate, run_if_nonzero,
                   static_cast<int>(gated_blocks(blocks_for(threads), run_if_nonzero ? gate : nullptr))};
}

static int launch_zero(const ZeroArgs& A, cudaStream_t st) {
    long long most = 0;
    for (int k = 0; k < 3; ++k)
        if (A.p[k] && A.n[k] > most) most = A.n[k];
    return most > 0 ? launch_after(zero_kernel, blocks_for(most / 4), kBlock, 0, st, A) : kOk;
}

template <class Kernel>
static int allow_columns(Kernel* kernel) {
    // (set on every call: it is cheap, and the setting belongs to the current device)
    return cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            kColumnWarps * kColumnMaxChannels * 32 * static_cast<int>(sizeof(float))));
}

// Columns for convolutions of at most kColumnMaxChannels channels per group: with longer rows a tile leaves an SM too few
// warps, and a tile per piece of the channels reads all outputs once per piece (576 channels -> 128 over 32 x 1024 positions in
// three pieces: 168 us against 82 with atomics, which spread over more addresses the longer the rows are).
int launch_inf_scatter(const float* go, const int* pos, float* gx, float* gw, const Shape& s, cudaStream_t st) {
    const long long nx = static_cast<long long>(s.B) * s.CI * s.HW, nw = static_cast<long long>(s.CO) * s.CIg;
    const long long outputs = static_cast<long long>(s.B) * s.CO * s.HW;
    int r;
    if (s.HW > 1 && s.CIg <= kColumnMaxChannels && outputs >= kColumnLeastOutputs && s.M < (1LL << 30) && s.G <= 65535) {
        const int block_smem = kColumnWarps * s.CIg * 32 * static_cast<int>(sizeof(float));
        if (gx) {
            if ((r = allow_columns(inf_scatter_columns_kernel)) != kOk) return r;
            const dim3 grid(static_cast<unsigned>((s.M + 32 * kColumnWarps - 1) / (32 * kColumnWarps)), s.G);
            r = launch_after(inf_scatter_columns_kernel, grid, kColumnWarps * 32, block_smem, st, go, pos, gx, gw, nw, s);
        } else {
            r = launch_zero(ZeroArgs{{gw, nullptr, nullptr}, {nw, 0, 0}}, st);
        }
        if (r != kOk || !gw) return r;
        if ((r = allow_columns(inf_scatter_weight_kernel)) != kOk) return r;
        // as many warps as the chip holds at once (a block keeps 1 KB of an SM's 228 to itself), each with 256 positions or more
        const int resident = min(8, 228 * 1024 / (block_smem + 1024)) * kColumnWarps * 148;
        long long splits = resident / s.CO;
        if (splits > s.M / 256) splits = s.M / 256;
        if (splits < 1) splits = 1;
        const long long blocks = (s.CO * splits + kColumnWarps - 1) / kColumnWarps;
        return launch_after(inf_scatter_weight_kernel, static_cast<unsigned>(blocks), kColumnWarps * 32, block_smem, st, go, pos,
                            gw, s, static_cast<int>(splits));
    }
    if ((r = launch_zero(ZeroArgs{{gx, gw, nullptr}, {nx, nw, 0}}, st)) != kOk) return r;
    return launch_after(inf_scatter_kernel, blocks_for(outputs), kBlock, 0, st, go, pos, gx, gw, s);
}

int launch_bound_scatter(const float* gol, const float* gou, const int* posl, const int* posu, float* gxl, float* gxu,
                         float* gw, const Shape& s, cudaStream_t st) {
    const long long nx = static_cast<long long>(s.B) * s.CI * s.HW, nw = static_cast<long long>(s.CO) * s.CIg;
    const int r = launch_zero(ZeroArgs{{gxl, gxu, gw}, {nx, nx, nw}}, st);
    if (r != kOk) return r;
    return launch_after(bound_scatter_kernel, blocks_for((long long)s.B * s.CO * s.HW), kBlock, 0, st, gol, gou, posl,
                        posu, gxl, gxu, gw, s);
}

}  // namespace ldn
