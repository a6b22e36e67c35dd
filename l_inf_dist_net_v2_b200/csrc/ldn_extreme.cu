// p = inf forward of large fully connected layers: max_c |x[b, c] - w[o, c]| without visiting most channels.
//
// A channel can only be the maximum of output (b, o) where |x| or |w| is large.  So every row of either operand gets a list
// of its extreme channels (|w| >= tau, |x| >= sigma) and the largest magnitude that is NOT in the list, rest_o and rest_b.
// The maximum over the two lists' channels, M, is compared with fl(rest_o + rest_b): a channel in neither list has
// |w| <= rest_o and |x| <= rest_b, hence |fl(x - w)| <= fl(rest_o + rest_b) (rounding is monotonic), so
// M > fl(rest_o + rest_b) proves that M is the maximum over all channels and that no other channel equals it: value and
// first channel are those of the dense kernel, bit for bit.  Outputs without the proof ("hard") are searched over all
// channels.  All arithmetic is the dense kernel's fp32 subtraction and comparison.
//
// tau and sigma come from the data: a sample of outputs is searched in full, tau + sigma is a low quantile of their maxima,
// and the split between the two is the one with the fewest list entries by the magnitudes' histograms.  With weights
// N(0, 1) about 60 of 3072 channels are visited for images in [0, 1], 170 of 5120 for activations of deviation 0.5.  Where
// the lists would not be a small part of a row, anything is not finite, or too many outputs turn out hard, a device word
// makes the dense kernels behind it run instead.
// 512 x 5120 -> 5120 forward + backward 1105 -> 567 us, certification of 512 x 3072 -> 5120 (value and bounds) 1971 -> 443.
//
// What bounds it: the gathers x[b, c] for a list's channels.  A block keeps S rows of one operand in shared memory as
// [channel][S], so a lane gathers four rows' values of a channel with one 16-byte read; a warp holds 32 / (S / 4) lists at
// once, whose entries lie [entry][list] in groups of 16 so that one step reads whole 128-byte lines.  Random channels meet
// bank conflicts of about two, i.e. 16 pairs per clock and SM.  The maximum is taken over batches of 8 entries and compared
// once per batch (2.4 instructions per pair); the channel is found at the end in the batch that last raised it.
#include <float.h>

#include "ldn_extreme.cuh"

namespace ldn {
namespace {

constexpr float kFloor = 1e-10f;   // value floor of the p = inf family
constexpr int kListW = 256;        // entries of a weight row's list, at most
constexpr int kListX = 128;        // of a sample's
constexpr int kGroup = 16;         // lists whose entries are interleaved
constexpr int kListThreads = 256;
constexpr int kMaxChannels = 6144;
constexpr int kListKeep = kMaxChannels / kListThreads;  // channels a thread of extreme_lists_kernel holds
constexpr int kScanThreads = 1024;
constexpr int kSampleBlocks = 148;
constexpr int kSamples = kSampleBlocks * 8;
constexpr int kQuantile = 4;       // tau + sigma: this smallest of the samples' maxima (0.3 %)
constexpr int kMaxTile = 224 * 1024;
// a gathered pair costs about 4 of the dense kernel's, and the samples' lists another pass over the weights
constexpr int kDenseShare = 8;     // dense where the lists hold more than 1 / kDenseShare of a row
constexpr int kSecondPass = 60;    // entries that pass costs

// device words (cleared by every call): 0 dense gate, 1 finished sampling blocks, 2 hard outputs
constexpr int kThresholdWord = 4;  // tau, sigma
constexpr int kHistWord = 8;

// magnitude histograms: 32 bins per octave from 2^-10 to 2^6 (what lies outside counts in the first / last bin)
constexpr int kBins = 512;
constexpr int kBinShift = 18;
constexpr int kBinBase = (127 - 10) << (23 - kBinShift);
__device__ __forceinline__ int bin_of(float m) {
    return min(kBins - 1, max(0, (__float_as_int(m) >> kBinShift) - kBinBase));
}
__device__ __forceinline__ float bin_edge(int i) { return __int_as_float((i + kBinBase) << kBinShift); }

// an entry: the value (bounds: lower and upper) and its channel
struct Entry1 {
    float v;
    int c;
};
struct Entry2 {
    float lo, up;
    int c, unused;
};
template <bool PAIR>
struct EntryOf {
    using type = Entry1;
};
template <>
struct EntryOf<true> {
    using type = Entry2;
};

__host__ __device__ inline long long groups_of(long long rows) { return (rows + kGroup - 1) / kGroup; }
__device__ __forceinline__ long long entry_index(long long row, int k, int cap) {
    return (row / kGroup * cap + k) * kGroup + row % kGroup;
}
__device__ __forceinline__ float block_max(float v, float* warps, int n_warps) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
    __syncthreads();
    v = warps[0];
    for (int k = 1; k < n_warps; ++k) v = fmaxf(v, warps[k]);
    return v;
}

// One block per row: the channels whose magnitude reaches the threshold, in ascending order; the row is read once, into
// registers, with all loads in flight.  Channels beyond `cap` entries count as not listed.
template <bool PAIR>
__global__ void __launch_bounds__(kListThreads)
extreme_lists_kernel(Operand v, Operand second, int C, int cap, const float* threshold, typename EntryOf<PAIR>::type* list,
                     int* len, float* rest, int* words) {
    stream_order_begin();
    // (one decision per block: another block of this very kernel may set the word between two threads' reads)
    if (__syncthreads_or(words[0] != 0)) return;
    __shared__ float warps[kListThreads / 32];
    __shared__ int counts[kListThreads / 32];
    const long long row = blockIdx.x;
    const float* src = v.ptr + row * v.stride_row;
    const float* src2 = second.ptr + row * second.stride_row;
    const float limit = *threshold;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // a warp takes a run of channels
    const int per = (C + kListThreads - 1) / kListThreads * 32;
    const int c0 = warp * per, c1 = min(C, c0 + per);
    float a[kListKeep], b[PAIR ? kListKeep : 1];
#pragma unroll
    for (int k = 0; k < kListKeep; ++k) {
        const int c = c0 + 32 * k + lane;
        a[k] = c < c1 ? src[c] : 0.0f;
        if (PAIR) b[k] = c < c1 ? src2[c] : 0.0f;
    }
    int n = 0;
    bool finite = true;
#pragma unroll
    for (int k = 0; k < kListKeep; ++k) {
        const float m = PAIR ? fmaxf(fabsf(a[k]), fabsf(b[k])) : fabsf(a[k]);
        finite &= fabsf(a[k]) <= FLT_MAX && (!PAIR || fabsf(b[k]) <= FLT_MAX);
        n += __popc(__ballot_sync(0xffffffffu, c0 + 32 * k + lane < c1 && m >= limit));
    }
    if (!finite) words[0] = 1;  // dense
    if (lane == 0) counts[warp] = n;
    __syncthreads();
    int at = 0, total = 0;
#pragma unroll
    for (int k = 0; k < kListThreads / 32; ++k) {
        if (k < warp) at += counts[k];
        total += counts[k];
    }
    float left = 0.0f;
#pragma unroll
    for (int k = 0; k < kListKeep; ++k) {
        const int c = c0 + 32 * k + lane;
        const float m = PAIR ? fmaxf(fabsf(a[k]), fabsf(b[k])) : fabsf(a[k]);
        const bool in = c < c1 && m >= limit;
        const unsigned who = __ballot_sync(0xffffffffu, in);
        const int slot = at + __popc(who & ((1u << lane) - 1));
        if (in && slot < cap) {
            if constexpr (PAIR) list[entry_index(row, slot, cap)] = Entry2{a[k], b[k], c, 0};
            else list[entry_index(row, slot, cap)] = Entry1{a[k], c};
        } else {
            left = fmaxf(left, m);
        }
        at += __popc(who);
    }
    left = block_max(left, warps, kListThreads / 32);
    if (threadIdx.x == 0) {
        len[row] = min(total, cap);
        rest[row] = left;
    }
}

struct Problem {
    Operand x, xu, w;
    long long B;
    int CO, C;
    float* y;   // BOUND: lower bounds
    float* yu;
    int* pos;   // may be null
    const float* sub;
    const float* add;
    ExtremeScratch t;
};

// Whether the outputs found from the lists are proven (see the head of this file).
__device__ __forceinline__ bool proven(float value, float rest_o, float rest_b) { return value > __fadd_rn(rest_o, rest_b); }

template <bool BOUND>
__device__ __forceinline__ void visit(float lo, float up, float w, float& best_lo, float& best_up) {
    if (BOUND) {
        const float d1 = lo - w, d2 = w - up;  // (w - lo and up - w are their exact negatives)
        best_lo = fmaxf(best_lo, fmaxf(d1, d2));
        best_up = fmaxf(best_up, fmaxf(-d1, -d2));
    } else {
        best_lo = fmaxf(best_lo, fabsf(lo - w));
    }
}

// A warp per sampled output: its maximum over all channels, and every fourth magnitude of its two rows into the histograms.
// The last block to finish chooses tau and sigma, or the dense kernels.
template <bool BOUND>
__global__ void __launch_bounds__(256) extreme_sample_kernel(const Problem P) {
    stream_order_begin();
    __shared__ int hist[2 * kBins];  // weights, inputs
    __shared__ float warps[8];
    __shared__ bool last;
    const int tid = threadIdx.x, lane = tid & 31;
    for (int i = tid; i < 2 * kBins; i += 256) hist[i] = 0;
    __syncthreads();
    const unsigned id = blockIdx.x * 8 + (tid >> 5);
    {
        // samples on a lattice that visits rows and outputs evenly (fractions of the golden ratio and of the square root of 2)
        const long long b = static_cast<long long>((static_cast<unsigned long long>(id * 2654435769u) * P.B) >> 32);
        const int o = static_cast<int>((static_cast<unsigned long long>(id * 1779033703u) * P.CO) >> 32);
        const float* xrow = P.x.ptr + b * P.x.stride_row;
        const float* urow = P.xu.ptr + b * P.xu.stride_row;
        const float* wrow = P.w.ptr + o * P.w.stride_row;
        float lo = kFloor, up = kFloor;
#pragma unroll 4
        for (int c = 4 * lane; c < P.C; c += 128) {
            const float4 x4 = *reinterpret_cast<const float4*>(xrow + c);  // (rows are whole 16-byte pieces)
            const float4 u4 = BOUND ? *reinterpret_cast<const float4*>(urow + c) : x4;
            const float4 w4 = *reinterpret_cast<const float4*>(wrow + c);
            const float xv[4] = {x4.x, x4.y, x4.z, x4.w}, uv[4] = {u4.x, u4.y, u4.z, u4.w}, wv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (c + e < P.C) visit<BOUND>(xv[e], uv[e], wv[e], lo, up);
            atomicAdd(&hist[bin_of(fabsf(w4.x))], 1);
            atomicAdd(&hist[kBins + bin_of(BOUND ? fmaxf(fabsf(x4.x), fabsf(u4.x)) : fabsf(x4.x))], 1);
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            lo = fmaxf(lo, __shfl_xor_sync(0xffffffffu, lo, d));
            up = fmaxf(up, __shfl_xor_sync(0xffffffffu, up, d));
        }
        if (lane == 0) P.t.samples[id] = BOUND ? fminf(lo, up) : lo;
    }
    __syncthreads();
    for (int i = tid; i < 2 * kBins; i += 256)
        if (hist[i]) atomicAdd(&P.t.words[kHistWord + i], hist[i]);
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(&P.t.words[1], 1) == kSampleBlocks - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the kQuantile-th smallest maximum
    float mine[(kSamples + 255) / 256];
#pragma unroll
    for (int k = 0; k < (kSamples + 255) / 256; ++k)
        mine[k] = tid + 256 * k < kSamples ? __ldcg(&P.t.samples[tid + 256 * k]) : FLT_MAX;
    float total = 0.0f;
    for (int round = 0; round < kQuantile; ++round) {
        float low = FLT_MAX;
#pragma unroll
        for (int k = 0; k < (kSamples + 255) / 256; ++k) low = fminf(low, mine[k]);
        total = -block_max(-low, warps, 8);
        // one thread that holds it drops one copy
        __syncthreads();
        if (tid == 0) hist[0] = 256;
        __syncthreads();
        if (low == total) atomicMin(&hist[0], tid);
        __syncthreads();
        if (tid == hist[0]) {
            bool dropped = false;
#pragma unroll
            for (int k = 0; k < (kSamples + 255) / 256; ++k)
                if (!dropped && mine[k] == total) {
                    mine[k] = FLT_MAX;
                    dropped = true;
                }
        }
        __syncthreads();
    }
    for (int i = tid; i < 2 * kBins; i += 256) hist[i] = __ldcg(&P.t.words[kHistWord + i]);
    __syncthreads();
    // suffix sums: values in this bin and above
    for (int d = 1; d < kBins; d <<= 1) {
        int add[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = tid + 256 * k;
            add[k] = i % kBins + d < kBins ? hist[i + d] : 0;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) hist[tid + 256 * k] += add[k];
        __syncthreads();
    }
    const float per_row = 4.0f / kSamples;
    float best = FLT_MAX, tau = 0.0f, sigma = 0.0f;
    for (int i = tid; i < kBins; i += 256) {
        const float t = bin_edge(i);
        if (!(t < total)) continue;
        const int j = bin_of(total - t);
        const float nw = hist[i] * per_row, nx = hist[kBins + j] * per_row;
        // (bin 0 holds everything below its edge too: a threshold there would be no bound)
        if (i == 0 || j == 0 || nw > 0.75f * kListW || nx > 0.75f * kListX) continue;
        const float cost = nw + (hist[kBins + j] > 0 ? nx + kSecondPass : 0.0f);
        if (cost < best) {
            best = cost;
            tau = t;
            sigma = bin_edge(j);
        }
    }
    const float least = -block_max(-best, warps, 8);
    if (tid == 0) hist[0] = 256;
    __syncthreads();
    if (best == least && best < FLT_MAX) atomicMin(&hist[0], tid);
    __syncthreads();
    if (hist[0] == 256 || least * kDenseShare > P.C) {
        if (tid == 0) P.t.words[0] = 1;
    } else if (tid == hist[0]) {
        P.t.words[kThresholdWord] = __float_as_int(tau);
        P.t.words[kThresholdWord + 1] = __float_as_int(sigma);
    }
}

// The maximum over one operand's lists.  WSIDE: S samples in shared memory, the weight rows' lists walked (sets y and pos);
// else: S weight rows in shared memory, the samples' lists walked (merged into y and pos).
template <bool BOUND, bool WSIDE, int S>
__global__ void __launch_bounds__(kScanThreads) extreme_scan_kernel(const Problem P, int splits) {
    stream_order_begin();
    if (P.t.words[0] != 0) return;
    extern __shared__ float4 tile4[];
    constexpr int Q = S / 4;           // lanes that share a list
    constexpr int LISTS = 32 / Q;      // lists of a warp
    constexpr bool PAIR_TILE = BOUND && WSIDE, PAIR_LIST = BOUND && !WSIDE;
    constexpr int CAP = WSIDE ? kListW : kListX;
    constexpr int kBatch = PAIR_LIST ? 4 : 8;  // entries in flight beside those being worked on
    using E = typename EntryOf<PAIR_LIST>::type;
    const int C4 = (P.C + 3) / 4;      // (rows of the operands are whole 16-byte pieces)
    const long long block = blockIdx.x / splits;
    const int split = static_cast<int>(blockIdx.x - block * splits);
    const long long tile_rows = WSIDE ? P.B : P.CO, list_rows = WSIDE ? P.CO : P.B;
    const int* len = WSIDE ? P.t.w_len : P.t.x_len;
    const E* list = static_cast<const E*>(WSIDE ? P.t.w_list : P.t.x_list);
    const long long row0 = block * S;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* tile = reinterpret_cast<float*>(tile4);
    float* tile_up = tile + static_cast<size_t>(C4) * 4 * S;
    if (!WSIDE) {
        // nothing to do where none of the samples kept a list (then the weights are not even read)
        int any = 0;
        for (long long r = threadIdx.x; r < list_rows; r += kScanThreads) any |= len[r];
        if (!__syncthreads_or(any)) return;
    }
    auto fill = [&](const Operand& v, float* dst) {
        for (int i = threadIdx.x; i < C4 * S; i += kScanThreads) {
            const int r = i % S, c = i / S;
            float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row0 + r < tile_rows) q = *reinterpret_cast<const float4*>(v.ptr + (row0 + r) * v.stride_row + 4 * c);
            dst[(4 * c + 0) * S + r] = q.x;
            dst[(4 * c + 1) * S + r] = q.y;
            dst[(4 * c + 2) * S + r] = q.z;
            dst[(4 * c + 3) * S + r] = q.w;
        }
    };
    fill(WSIDE ? P.x : P.w, tile);
    if (PAIR_TILE) fill(P.xu, tile_up);
    __syncthreads();
    const int q = lane % Q;
    const long long chunks = (list_rows + LISTS - 1) / LISTS;
    for (long long chunk = static_cast<long long>(split) * (kScanThreads / 32) + warp; chunk < chunks;
         chunk += static_cast<long long>(splits) * (kScanThreads / 32)) {
        const long long l = chunk * LISTS + lane / Q;
        const int n = l < list_rows ? len[l] : 0;
        int most = n;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, d));
        float best[4], best_up[4];
        int batch[4];  // first entry of the batch that last raised the maximum
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            best[e] = best_up[e] = kFloor;
            batch[e] = -1;
        }
        const E* entries = list + (l / kGroup * CAP) * kGroup + l % kGroup;
        auto load = [&](E (&en)[kBatch], int k0) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                en[u] = E{};
                if (k0 + u < n) en[u] = entries[(k0 + u) * kGroup];
            }
        };
        auto gather = [&](const float* from, int c, float (&v)[4]) {
            const float4 t = *reinterpret_cast<const float4*>(from + c * S + 4 * q);
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        };
        E now[kBatch];
        load(now, 0);
        for (int k0 = 0; k0 < most; k0 += kBatch) {
            E next[kBatch];
            load(next, k0 + kBatch);
            float top[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) top[e] = 0.0f;
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                if (k0 + u < n) {
                    float tv[4], sv[4];
                    gather(tile, now[u].c, tv);
                    if constexpr (PAIR_TILE) gather(tile_up, now[u].c, sv);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if constexpr (PAIR_TILE) visit<true>(tv[e], sv[e], now[u].v, best[e], best_up[e]);
                        else if constexpr (PAIR_LIST) visit<true>(now[u].lo, now[u].up, tv[e], best[e], best_up[e]);
                        else top[e] = fmaxf(top[e], fabsf(now[u].v - tv[e]));
                    }
                }
            }
            if constexpr (!BOUND) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (top[e] > best[e]) {  // channels ascend: the first batch of equal ones stays
                        best[e] = top[e];
                        batch[e] = k0;
                    }
            }
#pragma unroll
            for (int u = 0; u < kBatch; ++u) now[u] = next[u];
        }
        int at[4] = {0, 0, 0, 0};
        if (!BOUND && P.pos) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (batch[e] >= 0) {
#pragma unroll
                    for (int u = kBatch - 1; u >= 0; --u) {
                        if (batch[e] + u < n) {
                            const E en = entries[(batch[e] + u) * kGroup];
                            float lv, tv = tile[en.c * S + 4 * q + e];
                            if constexpr (PAIR_LIST) lv = en.lo;
                            else lv = en.v;
                            const float d = WSIDE ? tv - lv : lv - tv;  // x - w
                            if (fabsf(d) == best[e]) at[e] = en.c | (d < 0.0f ? static_cast<int>(0x80000000u) : 0);
                        }
                    }
                }
            }
        }
        if (l >= list_rows) continue;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const long long r = row0 + 4 * q + e;
            if (r >= tile_rows) continue;
            const long long i = WSIDE ? r * P.CO + l : l * P.CO + r;
            if (BOUND) {
                P.y[i] = WSIDE ? best[e] : fmaxf(P.y[i], best[e]);
                P.yu[i] = WSIDE ? best_up[e] : fmaxf(P.yu[i], best_up[e]);
            } else if (WSIDE) {
                P.y[i] = best[e];
                if (P.pos) P.pos[i] = at[e];
            } else {
                const float old = P.y[i];
                if (P.pos) {
                    const int c = at[e] & 0x7fffffff;
                    if (best[e] > old || (best[e] == old && best[e] > kFloor && c < (P.pos[i] & 0x7fffffff))) P.pos[i] = at[e];
                }
                if (best[e] > old) P.y[i] = best[e];
            }
        }
    }
}

__device__ __forceinline__ float epilogue(float v, int o, const Problem& P) {
    if (P.sub) v = __fsub_rn(v, P.sub[o]);
    if (P.add) v = __fadd_rn(v, P.add[o]);
    return v;
}

// The proof for every output; proven ones get the layer's epilogue, the others are put down for the full search.
template <bool BOUND>
__global__ void __launch_bounds__(256) extreme_check_kernel(const Problem P, unsigned most_hard) {
    stream_order_begin();
    if (P.t.words[0] != 0) return;
    const bool shift = P.sub != nullptr || P.add != nullptr;
    for (long long b = blockIdx.y; b < P.B; b += gridDim.y) {
        const float rest_b = P.t.x_rest[b];
        for (int o = blockIdx.x * 256 + threadIdx.x; o < P.CO; o += gridDim.x * 256) {
            const long long i = b * P.CO + o;
            const float lo = P.y[i], up = BOUND ? P.yu[i] : lo;
            if (proven(fminf(lo, up), P.t.w_rest[o], rest_b)) {
                if (shift) {
                    P.y[i] = epilogue(lo, o, P);
                    if (BOUND) P.yu[i] = epilogue(up, o, P);
                }
            } else {
                const unsigned h = atomicAdd(reinterpret_cast<unsigned*>(&P.t.words[2]), 1u);
                if (h < most_hard) P.t.hard[h] = static_cast<unsigned>(i);
                else P.t.words[0] = 1;  // dense (it overwrites every output)
            }
        }
    }
}

// A warp per hard output: all channels.
template <bool BOUND>
__global__ void __launch_bounds__(256) extreme_resolve_kernel(const Problem P) {
    stream_order_begin();
    if (P.t.words[0] != 0) return;
    const int lane = threadIdx.x & 31;
    const unsigned n = static_cast<unsigned>(P.t.words[2]);
    for (unsigned h = blockIdx.x * 8 + (threadIdx.x >> 5); h < n; h += gridDim.x * 8) {
        const unsigned i = P.t.hard[h];
        const unsigned b = i / static_cast<unsigned>(P.CO), o = i - b * static_cast<unsigned>(P.CO);
        const float* xr = P.x.ptr + b * P.x.stride_row;
        const float* ur = P.xu.ptr + b * P.xu.stride_row;
        const float* wr = P.w.ptr + o * P.w.stride_row;
        float lo = kFloor, up = kFloor;
        int at = 0x7fffffff, sign = 0;
#pragma unroll 4
        for (int c = lane; c < P.C; c += 32) {
            if (BOUND) {
                visit<true>(xr[c], ur[c], wr[c], lo, up);
            } else {
                const float d = xr[c] - wr[c];
                if (fabsf(d) > lo) {
                    lo = fabsf(d);
                    at = c;
                    sign = d < 0.0f ? static_cast<int>(0x80000000u) : 0;
                }
            }
        }
        float top = lo, top_up = up;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
            top_up = fmaxf(top_up, __shfl_xor_sync(0xffffffffu, top_up, d));
        }
        if (!BOUND && P.pos) {
            int first = lo == top ? at : 0x7fffffff;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, d));
            if (first == 0x7fffffff) {
                if (lane == 0) P.pos[i] = 0;
            } else if (lo == top && at == first) {
                P.pos[i] = at | sign;
            }
        }
        if (lane == 0) {
            P.y[i] = epilogue(top, static_cast<int>(o), P);
            if (BOUND) P.yu[i] = epilogue(top_up, static_cast<int>(o), P);
        }
    }
}

unsigned most_hard_of(long long B, int CO) {
    // a full search costs about 20 times an output's share of the dense kernel
    const long long n = B * CO / 64;
    return static_cast<unsigned>(n > 4096 ? n : 4096);
}

int round4(int c) { return (c + 3) & ~3; }
// samples (weight rows) a scan block holds: 8 where they fit, else 4
int tile_rows_of(int C, int arrays) { return static_cast<long long>(round4(C)) * 8 * 4 * arrays <= kMaxTile ? 8 : 4; }

template <class K>
int allow_smem(K kernel, bool (&configured)[64], int bytes) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 64 && configured[dev]) return kOk;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return cuda_status(e);
    if (dev < 64) configured[dev] = true;
    return kOk;
}

template <bool BOUND, bool WSIDE, int S>
int launch_scan_s(const Problem& P, cudaStream_t st) {
    static bool configured[64] = {};
    int r = allow_smem(extreme_scan_kernel<BOUND, WSIDE, S>, configured, kMaxTile);
    if (r != kOk) return r;
    const int smem = round4(P.C) * S * 4 * (BOUND && WSIDE ? 2 : 1);
    const long long tiles = ((WSIDE ? P.B : P.CO) + S - 1) / S;
    const long long chunks = ((WSIDE ? P.CO : P.B) + 32 / (S / 4) - 1) / (32 / (S / 4));
    // blocks that share a tile's lists: as few as fill the chip's last wave well (each fills its own tile)
    const int resident = 148 * (2 * (smem + 1024) <= 227 * 1024 ? 2 : 1);
    int splits = 1;
    double best = 0.0;
    for (int k = 1; k <= 16 && k * (kScanThreads / 32) <= chunks + kScanThreads / 32 - 1; ++k) {
        const long long blocks = tiles * k;
        const double waves = static_cast<double>((blocks + resident - 1) / resident);
        const double use = blocks / (waves * resident) - 0.02 * k;
        if (use > best) {
            best = use;
            splits = k;
        }
    }
    return launch_after(extreme_scan_kernel<BOUND, WSIDE, S>, static_cast<unsigned>(tiles * splits), kScanThreads, smem, st, P,
                        splits);
}
template <bool BOUND, bool WSIDE>
int launch_scan(const Problem& P, cudaStream_t st) {
    return tile_rows_of(P.C, BOUND && WSIDE ? 2 : 1) == 8 ? launch_scan_s<BOUND, WSIDE, 8>(P, st)
                                                          : launch_scan_s<BOUND, WSIDE, 4>(P, st);
}

template <bool BOUND>
int run(const Problem& P, cudaStream_t st) {
    using EX = typename EntryOf<BOUND>::type;
    const cudaError_t e = cudaMemsetAsync(P.t.words, 0, kExtremeWords * sizeof(int), st);
    if (e != cudaSuccess) return cuda_status(e);
    const float* thresholds = reinterpret_cast<const float*>(P.t.words + kThresholdWord);
    int r = launch_after(extreme_sample_kernel<BOUND>, kSampleBlocks, 256, 0, st, P);
    if (r == kOk)
        r = launch_after(extreme_lists_kernel<false>, static_cast<unsigned>(P.CO), kListThreads, 0, st, P.w, P.w, P.C, kListW,
                         thresholds, static_cast<Entry1*>(P.t.w_list), P.t.w_len, P.t.w_rest, P.t.words);
    if (r == kOk)
        r = launch_after(extreme_lists_kernel<BOUND>, static_cast<unsigned>(P.B), kListThreads, 0, st, P.x, P.xu, P.C, kListX,
                         thresholds + 1, static_cast<EX*>(P.t.x_list), P.t.x_len, P.t.x_rest, P.t.words);
    if (r == kOk) r = launch_scan<BOUND, true>(P, st);
    if (r == kOk) r = launch_scan<BOUND, false>(P, st);
    if (r == kOk) {
        const dim3 grid(static_cast<unsigned>((P.CO + 255) / 256), static_cast<unsigned>(P.B < 65535 ? P.B : 65535));
        r = launch_after(extreme_check_kernel<BOUND>, grid, 256, 0, st, P, most_hard_of(P.B, P.CO));
    }
    if (r == kOk) r = launch_after(extreme_resolve_kernel<BOUND>, 148 * 8, 256, 0, st, P);
    return r;
}

}  // namespace

// Lines of the rule.  Below 2048 channels the lists are not a small part of a row.  Below 6.4 G pairs (values; bounds, which
// cost the dense kernel 2.6 times as much: 2.5 G) what the path gains is not sure to cover its fixed cost, 100 us of sample,
// lists and nine launches, and the 45 us it costs where the sample decides for dense: 128 x 3072 -> 5500 (2.2 G) takes 261 us
// for hidden activations with index against 198 dense, 512 x 3072 -> 5120 (8.1 G) 446 against 672.  Beyond 6144 channels a
// row no longer fits a list block's registers and four rows of both bounds no longer shared memory; narrow sides leave the
// scan's blocks idle.
bool extreme_applies(long long B, int CO, int C, bool bound) {
    return C >= 2048 && C <= kMaxChannels && B >= 128 && CO >= 512 && B * CO < (1LL << 31) &&
           B * CO * C >= (bound ? 2500000000LL : 6400000000LL);
}

size_t extreme_scratch_bytes(long long B, int CO, bool bound) {
    const size_t ex = bound ? sizeof(Entry2) : sizeof(Entry1);
    return pad256(groups_of(B) * kGroup * kListX * ex) + pad256(groups_of(CO) * kGroup * kListW * sizeof(Entry1)) +
           2 * pad256(B * sizeof(int)) + 2 * pad256(static_cast<size_t>(CO) * sizeof(int)) +
           pad256(static_cast<size_t>(most_hard_of(B, CO)) * sizeof(unsigned)) + pad256(kExtremeWords * sizeof(int)) +
           pad256(kSamples * sizeof(float));
}

bool extreme_take_scratch(Bump* bump, long long B, int CO, bool bound, ExtremeScratch* t) {
    const size_t ex = bound ? sizeof(Entry2) : sizeof(Entry1);
    t->x_list = bump->take<char>(groups_of(B) * kGroup * kListX * ex);
    t->w_list = bump->take<char>(groups_of(CO) * kGroup * kListW * sizeof(Entry1));
    t->x_len = bump->take<int>(B);
    t->w_len = bump->take<int>(CO);
    t->x_rest = bump->take<float>(B);
    t->w_rest = bump->take<float>(CO);
    t->hard = bump->take<unsigned>(most_hard_of(B, CO));
    t->words = bump->take<int>(kExtremeWords);
    t->samples = bump->take<float>(kSamples);
    return t->samples && t->x_list && t->w_list && t->x_len && t->w_len && t->x_rest && t->w_rest && t->hard && t->words;
}

int launch_extreme(Operand x, Operand xu, Operand w, long long B, int CO, int C, bool bound, float* y, float* yu, int* pos,
                   const float* sub, const float* add, const ExtremeScratch& t, const int** dense_gate, cudaStream_t st) {
    const Problem P{x, xu, w, B, CO, C, y, yu, pos, sub, add, t};
    *dense_gate = t.words;
    return bound ? run<true>(P, st) : run<false>(P, st);
}

}  // namespace ldn
