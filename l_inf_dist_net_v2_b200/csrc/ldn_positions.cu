// The p = inf forward pass over inputs with many positions per sample (convolutions): values, indices, interval bounds.
//
// What bounds it: the ALU's minima and maxima (one per pair and 64 a clock and SM; bounds: four), then the copy of the input.
// The general path (tile kernels, then a search for the indices) loses on these shapes to outputs that do not fill its tiles
// (16 of a group in a 32-wide tile), reductions of a few stages per tile, a second launch that reads inputs and results again,
// and transposed copies for bounds.  Measured, before and after, in us (index / value / bounds):
//   128 x 256 positions, 4 groups of 144 channels -> 16:  152 / 91 / 563  ->  65 / 42 / 112
//   32 x 1024 positions, 200 channels -> 128:             243 / 89 / 240  ->  120 / 84 / 217
//   64 x 49 positions, 288 channels -> 64:                 30 / 20 /  46  ->  14 / 11 /  22
// Tried and left: weights straight from global memory (109 / 84 / 166 on the first line: the stream of inputs pushes them out
// of the L1 cache), and warps with outputs of their own only (70 / 42 / 112; the channels of 576 -> 128 value 270 against 213).
#include "ldn_ops.cuh"
#include "ldn_positions.cuh"

namespace ldn {

namespace {
constexpr int kTile = 64;     // positions of a block, two per lane
constexpr int kOuts = 8;      // outputs of a warp in one pass over the channels
constexpr int kBatch = 8;     // channels whose batch the maximum is remembered by (kIndex)
constexpr int kStage = 16;    // channels of a stage of a warp's weight ring: one 16-byte copy per lane
constexpr int kRing = 4;      // stages of the ring
constexpr int kMaxWarps = 16;
constexpr int kMaxSmem = 226 * 1024;
constexpr int kRingFloats = kRing * kStage * kOuts;  // of one warp
constexpr int kPartFloats = kOuts * kTile;           // of one warp and array

enum Mode { kValue, kIndex, kBounds };

inline int tile_floats(const Shape& s, bool bounds) {
    return (s.CIg + kStage - 1) / kStage * kStage * kTile * (bounds ? 2 : 1);
}
inline int smem_bytes(const Shape& s, int warps, int mode) {
    return (tile_floats(s, mode == kBounds) + warps * (kRingFloats + kPartFloats * (mode == kValue ? 1 : 2))) *
           static_cast<int>(sizeof(float));
}

__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// Copies [channels][kTile] of the input at positions m0 ... (positions beyond the last repeat it, channels beyond it are zero).
// V positions per copy.
template <int V>
__device__ __forceinline__ void copy_tile(float* tile, const float* x, const Shape& s, int g, long long m0, int channels) {
    constexpr int kPieces = kTile / V;
    const int threads = blockDim.x / kTile * kTile, tid = threadIdx.x;
    if (tid >= threads) return;
    const int piece = tid % kPieces, step = threads / kPieces;
    const long long m = min(m0 + piece * V, s.M - V);
    const long long b = m / s.HW;
    const float* src = x + (b * s.G + g) * s.CIg * (long long)s.HW + (m - b * s.HW);
    const long long stride = s.HW;
#pragma unroll 4
    for (int c = tid / kPieces; c < channels; c += step)
        copy_async<4 * V>(tile + c * kTile + piece * V, src + min(c, s.CIg - 1) * stride, c < s.CIg ? 4 * V : 0);
}

// A block owns kTile positions of one group and keeps their channels in shared memory; a warp owns kOuts outputs and one of
// `parts` ranges of the channels, reads two positions per lane from there and its weights, which all lanes share, from a ring
// that it fills for itself (no block-wide wait in the loop).  The ranges' results meet in shared memory, where every warp
// finishes a part of the outputs.
template <int MODE>
__global__ void __launch_bounds__(kMaxWarps * 32) inf_positions_kernel(const float* x, const float* xu, Operand w, Shape s,
                                                                       int parts, int block_outs, int splits, int vec, float* y,
                                                                       float* yu, int* pos, const float* sub, const float* add) {
    stream_order_begin();
    extern __shared__ float4 shared4[];
    float* const tile = reinterpret_cast<float*>(shared4);
    const int stages = (s.CIg + kStage - 1) / kStage, channels = stages * kStage;
    float* const tile_u = tile + channels * kTile;  // kBounds: the upper inputs
    float* const rings = tile + (MODE == kBounds ? 2 : 1) * channels * kTile;
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* const part_f = rings + warps * kRingFloats;  // [warp][output][position]: maxima (kBounds: of the upper bound)
    float* const part_2 = part_f + warps * kPartFloats;  // kBounds: minima; kIndex: batches (as integers)
    int* const part_i = reinterpret_cast<int*>(part_2);

    const int g = blockIdx.y / splits, o_first = (blockIdx.y - g * splits) * block_outs;
    const int o_end = min(s.COg, o_first + block_outs);
    const long long m0 = blockIdx.x * (long long)kTile;

    if (vec) copy_tile<4>(tile, x, s, g, m0, channels);
    else copy_tile<1>(tile, x, s, g, m0, channels);
    if (MODE == kBounds) {
        if (vec) copy_tile<4>(tile_u, xu, s, g, m0, channels);
        else copy_tile<1>(tile_u, xu, s, g, m0, channels);
    }
    copy_commit();
    copy_wait<0>();
    __syncthreads();
    if (MODE == kBounds) {
        for (int i = threadIdx.x; i < channels * kTile; i += blockDim.x) {
            const float lo = tile[i], up = tile_u[i];
            if (lo > up) tile[i] = tile_u[i] = (lo + up) * 0.5f;
        }
        __syncthreads();
    }

    const int groups = warps / parts;  // warps with different outputs
    const int part = warp / groups;
    float* const ring = rings + warp * kRingFloats;
    const int first = stages * part / parts, last = stages * (part + 1) / parts;
    // (the trip count is the same for all warps)
    for (int o_pass = o_first; o_pass < o_end; o_pass += groups * kOuts) {
        const int o0 = o_pass + (warp - part * groups) * kOuts;
        // this lane's piece of a stage: four channels of one output
        const float* const from = w.ptr + g * w.stride_group + min(o0 + (lane >> 2), o_end - 1) * w.stride_row;
        auto fetch = [&](int stage) {
            if (stage < last) {
                const int c = stage * kStage + 4 * (lane & 3);
                const int n = max(0, min(4, s.CIg - c));
                copy_async<16>(ring + (stage & (kRing - 1)) * (kStage * kOuts) + 4 * lane, n > 0 ? from + c : from, 4 * n);
            }
            copy_commit();
        };
        __syncwarp();  // the ring's last readers are done
#pragma unroll
        for (int i = 0; i < kRing - 1; ++i) fetch(first + i);

        float top[kOuts][2];   // running maximum (kBounds: of the upper bound)
        float low[kOuts][2];   // kBounds: running minimum
        int batch[kOuts][2];   // kIndex: the batch that raised the maximum last
#pragma unroll
        for (int j = 0; j < kOuts; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                top[j][h] = kEps;
                low[j][h] = -kEps;
                batch[j][h] = -1;
            }
#pragma unroll 1
        for (int stage = first; stage < last; ++stage) {
            copy_wait<kRing - 2>();
            __syncwarp();  // all lanes' pieces of this stage have arrived; all lanes are done with the stage before
            fetch(stage + kRing - 1);
            const float4* ws = reinterpret_cast<const float4*>(ring + (stage & (kRing - 1)) * (kStage * kOuts));
            const float* xs = tile + stage * (kStage * kTile) + lane;
            const float* us = tile_u + stage * (kStage * kTile) + lane;
#pragma unroll
            for (int k = 0; k < kStage / kBatch; ++k) {
                float before[kOuts][2];
#pragma unroll
                for (int j = 0; j < kOuts; ++j) {
                    before[j][0] = top[j][0];
                    before[j][1] = top[j][1];
                }
#pragma unroll
                for (int q = k * (kBatch / 4); q < (k + 1) * (kBatch / 4); ++q) {
                    float a[2][4], c[2][4];
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            a[h][e] = xs[(4 * q + e) * kTile + 32 * h];
                            if (MODE == kBounds) c[h][e] = us[(4 * q + e) * kTile + 32 * h];
                        }
#pragma unroll
                    for (int j = 0; j < kOuts; ++j) {
                        const float4 v = ws[j * (kStage / 4) + q];
                        const float2 w0 = make_float2(v.x, v.y), w1 = make_float2(v.z, v.w);
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const float2 a0 = make_float2(a[h][0], a[h][1]), a1 = make_float2(a[h][2], a[h][3]);
                            if (MODE == kBounds) {
                                const float2 s0 = pk_sub(w0, a0), s1 = pk_sub(w1, a1);
                                const float2 t0 = pk_sub(make_float2(c[h][0], c[h][1]), w0);
                                const float2 t1 = pk_sub(make_float2(c[h][2], c[h][3]), w1);
                                float lo = low[j][h], up = top[j][h];
                                lo = fminf(fminf(lo, s0.x), t0.x);
                                up = fmaxf(fmaxf(up, s0.x), t0.x);
                                lo = fminf(fminf(lo, s0.y), t0.y);
                                up = fmaxf(fmaxf(up, s0.y), t0.y);
                                lo = fminf(fminf(lo, s1.x), t1.x);
                                up = fmaxf(fmaxf(up, s1.x), t1.x);
                                lo = fminf(fminf(lo, s1.y), t1.y);
                                up = fmaxf(fmaxf(up, s1.y), t1.y);
                                low[j][h] = lo;
                                top[j][h] = up;
                            } else {
                                const float2 d0 = pk_sub(a0, w0), d1 = pk_sub(a1, w1);
                                float t = top[j][h];
                                t = fmaxf(fmaxf(t, fabsf(d0.x)), fabsf(d0.y));
                                t = fmaxf(fmaxf(t, fabsf(d1.x)), fabsf(d1.y));
                                top[j][h] = t;
                            }
                        }
                    }
                }
                if (MODE == kIndex) {
#pragma unroll
                    for (int j = 0; j < kOuts; ++j)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            if (top[j][h] > before[j][h]) batch[j][h] = stage * (kStage / kBatch) + k;
                }
            }
        }

        __syncthreads();  // the last pass's partial results have been read
#pragma unroll
        for (int j = 0; j < kOuts; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = warp * kPartFloats + j * kTile + 32 * h + lane;
                part_f[i] = top[j][h];
                if (MODE == kBounds) part_2[i] = low[j][h];
                if (MODE == kIndex) part_i[i] = batch[j][h];
            }
        __syncthreads();
        // a warp finishes 64 positions of every (warps)th of the pass's outputs
        for (int j = warp; j < groups * kOuts && o_pass + j < o_end; j += warps) {
            const int o = o_pass + j, slot = (j / kOuts) * kPartFloats + (j % kOuts) * kTile;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int p = 32 * h + lane;
                float up = part_f[slot + p], lo = MODE == kBounds ? part_2[slot + p] : 0.0f;
                int where = MODE == kIndex ? part_i[slot + p] : -1;
                for (int r = 1; r < parts; ++r) {
                    const int i = slot + r * groups * kPartFloats + p;
                    const float v = part_f[i];
                    if (MODE == kIndex && v > up) where = part_i[i];  // (channels ascend: an equal maximum comes later)
                    up = fmaxf(up, v);
                    if (MODE == kBounds) lo = fminf(lo, part_2[i]);
                }
                int found = 0;
                if (MODE == kIndex && where >= 0) {
                    // the first channel of the batch that reaches the maximum
                    const float* row = w.ptr + g * w.stride_group + o * w.stride_row;
                    int best = -1;
                    bool negative = false;
#pragma unroll
                    for (int q = kBatch / 4 - 1; q >= 0; --q) {
                        const int c = where * kBatch + 4 * q;
                        if (c < s.CIg) {
                            const float4 v = *reinterpret_cast<const float4*>(row + c);
                            const float we[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int e = 3; e >= 0; --e) {
                                const float d = tile[(c + e) * kTile + p] - we[e];
                                if (fabsf(d) == up && c + e < s.CIg) {
                                    best = c + e;
                                    negative = d < 0.0f;
                                }
                            }
                        }
                    }
                    if (best >= 0) found = best | (negative ? kSignBit : 0);
                }
                const long long m = m0 + p;
                if (m >= s.M) continue;
                const long long b = m / s.HW;
                const long long i = ((b * s.G + g) * s.COg + o) * (long long)s.HW + (m - b * s.HW);
                float v = MODE == kBounds ? -lo : up;
                if (MODE != kIndex) {
                    const int ch = g * s.COg + o;
                    if (sub) {
                        v = __fsub_rn(v, sub[ch]);
                        up = __fsub_rn(up, sub[ch]);
                    }
                    if (add) {
                        v = __fadd_rn(v, add[ch]);
                        up = __fadd_rn(up, add[ch]);
                    }
                }
                y[i] = v;
                if (MODE == kBounds) yu[i] = up;
                if (MODE == kIndex) pos[i] = found;
            }
        }
    }
}

template <int MODE>
int launch(const float* x, const float* xu, Operand w, const Shape& s, float* y, float* yu, int* pos, const float* sub,
           const float* add, cudaStream_t st) {
    const cudaError_t e =
        cudaFuncSetAttribute(inf_positions_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return cuda_status(e);
    const long long tiles = (s.M + kTile - 1) / kTile;
    const int passes = (s.COg + kOuts - 1) / kOuts, stages = (s.CIg + kStage - 1) / kStage;
    // fewer tiles than SMs: the outputs are split over blocks (each copies its input)
    long long splits = 148 / (tiles * s.G);
    if (splits > passes) splits = passes;
    if (splits < 1) splits = 1;
    const int block_passes = static_cast<int>((passes + splits - 1) / splits);
    splits = (passes + block_passes - 1) / block_passes;
    const long long per_sm = (tiles * s.G * splits + 147) / 148;
    // warps with outputs of their own, up to eight; while an SM would hold fewer than 12 (bounds, whose inputs take twice the
    // shared memory: 8), they share the channels
    const int rounds = (block_passes + 7) / 8;
    const int groups = (block_passes + rounds - 1) / rounds;
    int parts = 1;
    while (parts < 8 && parts * 2 <= stages && groups * parts * 2 <= kMaxWarps && smem_bytes(s, groups * parts * 2, MODE) <= kMaxSmem) {
        const long long resident = min(per_sm, static_cast<long long>(kMaxSmem / smem_bytes(s, groups * parts, MODE)));
        if (groups * parts >= 2 && groups * parts * resident >= (MODE == kBounds ? 8 : 12)) break;
        parts *= 2;
    }
    const int warps = groups * parts;
    const int vec = s.HW % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(xu)) & 15u) == 0;
    const dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>(s.G * splits));
    return launch_after(inf_positions_kernel<MODE>, grid, (warps < 2 ? 2 : warps) * 32, smem_bytes(s, warps < 2 ? 2 : warps, MODE),
                        st, x, xu, w, s, parts, block_passes * kOuts, static_cast<int>(splits), vec, y, yu, pos, sub, add);
}
}  // namespace

// The tile kernels of the general path make the channels of many outputs an outer loop and take groups of outputs 32, 64 or 128
// wide; they find indices in a second launch and need inputs of other than whole 16-byte pieces copied.  Here the input of a
// block stays in shared memory, which bounds the channels (704 per group, bounds 352), and outputs come in eights.  Both sides
// over 32 shapes from 8 x 4 x 49 to 128 x 800 x 256: indices 1.2 to 7.7 times as fast, bounds 0.97 to 5, values 1.05 to 2.7
// except where the lines below lie: whole 128-wide tiles of long rows (32 x 1024 positions of 576 channels -> 128: 213 us
// here, 196 there), and long rows of fewer blocks than half the SMs (16 x 81 positions of 300 channels -> 24: 14.3 and 13.3).
bool inf_positions_apply(const Shape& s, bool index, bool bounds) {
    if (s.HW <= 1 || s.M >= (1LL << 31) || static_cast<long long>(s.COg) * s.HW >= (1LL << 31) ||
        static_cast<long long>(s.B) * s.G >= (1LL << 31) || s.G > 8192 || s.co_src != s.CO)
        return false;
    if (s.CIg > 1024 || smem_bytes(s, 8, bounds ? kBounds : kIndex) > kMaxSmem) return false;
    if (index || bounds) return true;
    const long long blocks = (s.M + kTile - 1) / kTile * s.G * ((s.COg + kOuts - 1) / kOuts);
    return !(s.COg % 128 == 0 && s.CIg > 384) && !(blocks < 148 / 2 && s.CIg > 256);
}

int launch_inf_positions(const float* x, const float* upper, Operand w, const Shape& s, float* y, float* y_upper, int* pos,
                         const float* sub, const float* add, cudaStream_t st) {
    if (upper) return launch<kBounds>(x, upper, w, s, y, y_upper, nullptr, sub, add, st);
    if (pos) return launch<kIndex>(x, nullptr, w, s, y, nullptr, pos, nullptr, nullptr, st);
    return launch<kValue>(x, nullptr, w, s, y, nullptr, nullptr, sub, add, st);
}

}  // namespace ldn
