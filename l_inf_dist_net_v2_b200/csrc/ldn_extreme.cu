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
// 512 x 5120 -> 5120 forward + backward: dense 1105 us, this path 505; certification of 512 x 3072 -> 5120 (value and bounds):
// 1971 and 335.
//
// What bounds it: the gathers x[b, c] for a list's channels.  A block keeps S rows of one operand in shared memory as
// [channel][S]; a lane owns a list, gathers four rows' values of a channel with one 16-byte read, and a warp's 32 lists lie
// [entry][list] in groups of 16, so that a step reads whole 128-byte lines, in an order that keeps the lists of a step on
// different banks (extreme_lists_kernel).  The maximum is taken over batches of 8 entries and compared once per batch; the
// channel is found at the end in the batch that last raised it, or in the whole list where a later batch reached the same
// value.
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
constexpr int kScanThreads = 512;
constexpr int kBatch = 8;          // entries a scan works on at a time (lists are whole batches long)
constexpr int kSampleBlocks = 148;
constexpr int kSamples = kSampleBlocks * 8;
constexpr int kQuantile = 2;       // tau + sigma: this smallest of the samples' maxima (0.2 %)
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

// One block per row: the channels whose magnitude reaches the threshold; the row is read once, into registers, with all loads
// in flight (KEEP channels per thread), and magnitudes are compared as integers (a sign bit less, not-a-numbers on top).
//
// Order of a list.  A scan step reads one channel of each of a warp's lists from shared memory, 32 bytes at bank
// 8 (channel % 4) (tiles of 8 rows), so four neighbouring lists read without conflicts if their channels differ modulo 4.
// Entry k of row r's list therefore has channel % 4 == (k + r) % 4: four interleaved sub-lists, the shorter ones filled up
// with entries that change nothing (NaN), so that a list is a whole number of batches, at least one.  A lane's channels are
// all of class lane % 4, so places come from one count per lane.  Channels beyond `cap` entries count as not listed.
template <bool PAIR, int KEEP>
__global__ void __launch_bounds__(kListThreads, KEEP <= 12 ? 3 : 2)
extreme_lists_kernel(Operand v, Operand second, int C, int cap, const float* threshold, typename EntryOf<PAIR>::type* list,
                     int* len, float* rest, int* words) {
    stream_order_begin();
    // (one decision per block: another block of this very kernel may set the word between two threads' reads)
    if (__syncthreads_or(words[0] != 0)) return;
    using E = typename EntryOf<PAIR>::type;
    constexpr int WARPS = kListThreads / 32;
    __shared__ int counts[WARPS][4], lefts[WARPS];
    const long long row = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int limit = __float_as_int(*threshold);
    const float* src = v.ptr + row * v.stride_row + threadIdx.x;
    const float* src2 = second.ptr + row * second.stride_row + threadIdx.x;
    float a[KEEP], b[PAIR ? KEEP : 1];
    const int mine_n = C - static_cast<int>(threadIdx.x);  // this thread's channels: threadIdx.x + 256 k < C
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
        a[k] = kListThreads * k < mine_n ? src[kListThreads * k] : 0.0f;
        if (PAIR) b[k] = kListThreads * k < mine_n ? src2[kListThreads * k] : 0.0f;
    }
    auto magnitude = [&](int k) {
        const int m = __float_as_int(a[k]) & 0x7fffffff;
        return PAIR ? max(m, __float_as_int(b[k]) & 0x7fffffff) : m;
    };
    int n = 0, top = 0;
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
        const int m = magnitude(k);
        top = max(top, m);
        n += m >= limit ? 1 : 0;  // (the threshold is above 0, padding is not)
    }
    if (top >= 0x7f800000) words[0] = 1;  // infinite or not a number: dense
    // places: exclusive sums over the lanes of a class, then over the warps
    int at = n;
#pragma unroll
    for (int d = 4; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, at, d);
        if (lane >= d) at += o;
    }
    if (lane >= 28) counts[warp][lane & 3] = at;
    at -= n;
    __syncthreads();
    int longest = 0, here = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        int total = 0;
#pragma unroll
        for (int k = 0; k < WARPS; ++k) {
            if (q == (lane & 3) && k < warp) at += counts[k][q];
            total += counts[k][q];
        }
        longest = max(longest, total);
        if (q == (lane & 3)) here = total;
    }
    longest = min(longest, cap / 4);
    const int slots = max((longest + 1) & ~1, 2);  // of a sub-list, fillers included: kBatch entries are two slots
    static_assert(kBatch == 8 && kListW % kBatch == 0 && kListX % kBatch == 0, "lists are whole batches");
    // entry of class lane % 4 at sub-list position `slot`
    E* dst = list + entry_index(row, ((lane & 3) - static_cast<int>(row & 3)) & 3, cap);
    int left = 0;
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
        const int m = magnitude(k);
        if (m >= limit && at < cap / 4) {
            const int c = static_cast<int>(threadIdx.x) + kListThreads * k;
            E e;
            if constexpr (PAIR) e = E{a[k], b[k], c, 0};
            else e = E{a[k], c};
            dst[at * 4 * kGroup] = e;
            ++at;
        } else {
            left = max(left, m);
        }
    }
    if (threadIdx.x < 4) {
        const float none = __int_as_float(0x7fc00000);
        E e;
        if constexpr (PAIR) e = E{none, none, static_cast<int>(threadIdx.x), 0};
        else e = E{none, static_cast<int>(threadIdx.x)};
        for (int slot = here; slot < slots; ++slot) dst[slot * 4 * kGroup] = e;
    }
    left = __reduce_max_sync(0xffffffffu, left);
    if (lane == 0) lefts[warp] = left;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 1; k < WARPS; ++k) left = max(left, lefts[k]);
        len[row] = longest > 0 ? 4 * slots : 0;
        rest[row] = __int_as_float(left);
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
#pragma unroll 8
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
//
// A lane owns a list and S outputs.  What bounds the walk is the load / store pipe: a step of 32 lists costs 4 S / 4 wavefronts
// of shared memory and about 4.5 of list entries, hence as many rows per list as fit (S = 8) where the lists are long; the
// samples' lists are short, and four rows leave room for two blocks, one filling its tile while the other walks.
template <bool BOUND, bool WSIDE, int S>
__global__ void __launch_bounds__(kScanThreads, S == 4 ? 2 : 1) extreme_scan_kernel(const Problem P, int splits) {
    stream_order_begin();
    if (P.t.words[0] != 0) return;
    extern __shared__ float4 tile4[];
    constexpr int H = S / 4;
    constexpr bool PAIR_TILE = BOUND && WSIDE, PAIR_LIST = BOUND && !WSIDE;
    constexpr int CAP = WSIDE ? kListW : kListX;
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
#pragma unroll 5
        for (int i = threadIdx.x; i < C4 * S; i += kScanThreads) {
            const int r = i % S, c = i / S;
            float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row0 + r < tile_rows) t = *reinterpret_cast<const float4*>(v.ptr + (row0 + r) * v.stride_row + 4 * c);
            // the four stores of neighbouring pieces start at different channels: no two lanes of a store on one bank
            if (c & 1) t = make_float4(t.y, t.z, t.w, t.x);
            if (c & 2) t = make_float4(t.z, t.w, t.x, t.y);
            dst[(4 * c + (c & 3)) * S + r] = t.x;
            dst[(4 * c + ((c + 1) & 3)) * S + r] = t.y;
            dst[(4 * c + ((c + 2) & 3)) * S + r] = t.z;
            dst[(4 * c + ((c + 3) & 3)) * S + r] = t.w;
        }
    };
    fill(WSIDE ? P.x : P.w, tile);
    if (PAIR_TILE) fill(P.xu, tile_up);
    __syncthreads();
    // of a channel's two 16-byte halves a lane reads first the one that its neighbours four lists on do not (H = 2)
    const int swap = H == 2 ? (lane >> 2) & 1 : 0;
    const long long chunks = (list_rows + 31) / 32;
    for (long long chunk = static_cast<long long>(split) * (kScanThreads / 32) + warp; chunk < chunks;
         chunk += static_cast<long long>(splits) * (kScanThreads / 32)) {
        const long long l = chunk * 32 + lane;
        const long long row = l < list_rows ? l : list_rows - 1;  // (lanes beyond the last list repeat it)
        const int n = max(len[row], kBatch);
        const int most = __reduce_max_sync(0xffffffffu, n);
        float best[S], best_up[S];
        int batch[S];  // first entry of the batch that last raised the maximum; kTie: a later batch reached it too
        constexpr int kTie = 1 << 30;
#pragma unroll
        for (int e = 0; e < S; ++e) {
            best[e] = best_up[e] = kFloor;
            batch[e] = 0;
        }
        const E* entries = list + (row / kGroup * CAP) * kGroup + row % kGroup;
        auto gather = [&](const float* from, int c, float (&v)[S]) {
#pragma unroll
            for (int h = 0; h < H; ++h) {
                const float4 t = *reinterpret_cast<const float4*>(from + c * S + 4 * (h ^ swap));
                v[4 * h] = t.x; v[4 * h + 1] = t.y; v[4 * h + 2] = t.z; v[4 * h + 3] = t.w;
            }
        };
        // (lanes whose list has ended keep their last batch and work on it again without taking the result)
        auto load = [&](E (&en)[kBatch], int k0) {
            if (k0 < n) {
#pragma unroll
                for (int u = 0; u < kBatch; ++u) en[u] = entries[(k0 + u) * kGroup];
            }
        };
        auto work = [&](const E (&en)[kBatch], int k0) {
            float top[S];
#pragma unroll
            for (int e = 0; e < S; ++e) top[e] = 0.0f;
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                float tv[S], sv[S];
                gather(tile, en[u].c, tv);
                if constexpr (PAIR_TILE) gather(tile_up, en[u].c, sv);
#pragma unroll
                for (int e = 0; e < S; ++e) {
                    if constexpr (PAIR_TILE) visit<true>(tv[e], sv[e], en[u].v, best[e], best_up[e]);
                    else if constexpr (PAIR_LIST) visit<true>(en[u].lo, en[u].up, tv[e], best[e], best_up[e]);
                    else top[e] = fmaxf(top[e], fabsf(en[u].v - tv[e]));
                }
            }
            if constexpr (!BOUND) {
                if (k0 < n) {
#pragma unroll
                    for (int e = 0; e < S; ++e)
                        if (top[e] >= best[e]) {
                            batch[e] = top[e] > best[e] ? k0 : batch[e] | kTie;
                            best[e] = top[e];
                        }
                }
            }
        };
        if constexpr (S == 4) {
            E en[kBatch];
            for (int k0 = 0; k0 < most; k0 += kBatch) {
                load(en, k0);
                work(en, k0);
            }
        } else {
            E even[kBatch], odd[kBatch];
            load(even, 0);
#pragma unroll
            for (int u = 0; u < kBatch; ++u) odd[u] = even[u];
            for (int k0 = 0; k0 < most; k0 += 2 * kBatch) {
                load(odd, k0 + kBatch);
                work(even, k0);
                load(even, k0 + 2 * kBatch);
                if (k0 + kBatch < most) work(odd, k0 + kBatch);
            }
        }
        if (l >= list_rows) continue;
#pragma unroll
        for (int e = 0; e < S; ++e) {
            const int in_tile = 4 * ((e / 4) ^ swap) + e % 4;
            const long long r = row0 + in_tile;
            if (r >= tile_rows) continue;
            const long long i = WSIDE ? r * P.CO + l : l * P.CO + r;
            if constexpr (BOUND) {
                P.y[i] = WSIDE ? best[e] : fmaxf(P.y[i], best[e]);
                P.yu[i] = WSIDE ? best_up[e] : fmaxf(P.yu[i], best_up[e]);
            } else {
                const float old = WSIDE ? kFloor : P.y[i];
                int at = 0;
                if (P.pos && best[e] > kFloor && best[e] >= old) {
                    // the lowest channel that attains the maximum: in the batch that raised it, or anywhere after a tie
                    const bool tie = (batch[e] & kTie) != 0;
                    const int from = tie ? 0 : batch[e], to = tie ? n : from + kBatch;
                    int first = 0x7fffffff;
                    for (int k = from; k < to; k += kBatch) {
                        E en[kBatch];
#pragma unroll
                        for (int u = 0; u < kBatch; ++u) en[u] = entries[(k + u) * kGroup];
#pragma unroll
                        for (int u = 0; u < kBatch; ++u) {
                            float lv;
                            const float tv = tile[en[u].c * S + in_tile];
                            if constexpr (PAIR_LIST) lv = en[u].lo;
                            else lv = en[u].v;
                            const float d = WSIDE ? tv - lv : lv - tv;  // x - w
                            if (fabsf(d) == best[e] && en[u].c < first) {
                                first = en[u].c;
                                at = en[u].c | (d < 0.0f ? static_cast<int>(0x80000000u) : 0);
                            }
                        }
                    }
                    if (!WSIDE && (best[e] > old || first < (P.pos[i] & 0x7fffffff))) P.pos[i] = at;
                }
                if (WSIDE) {
                    P.y[i] = best[e];
                    if (P.pos) P.pos[i] = at;
                } else if (best[e] > old) {
                    P.y[i] = best[e];
                }
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
    for (long long b0 = blockIdx.y * 4LL; b0 < P.B; b0 += gridDim.y * 4LL) {
        const int o = blockIdx.x * 256 + threadIdx.x;
        if (o >= P.CO) continue;
        const float rest_o = P.t.w_rest[o];
        float lo[4], up[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (b0 + k < P.B) {
                lo[k] = P.y[(b0 + k) * P.CO + o];
                up[k] = BOUND ? P.yu[(b0 + k) * P.CO + o] : lo[k];
            }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (b0 + k >= P.B) break;
            const long long i = (b0 + k) * P.CO + o;
            if (proven(fminf(lo[k], up[k]), rest_o, P.t.x_rest[b0 + k])) {
                if (shift) {
                    P.y[i] = epilogue(lo[k], o, P);
                    if (BOUND) P.yu[i] = epilogue(up[k], o, P);
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
    const long long chunks = ((WSIDE ? P.CO : P.B) + 31) / 32;
    // blocks that share a tile's lists: as few as fill the chip's last wave well (each fills its own tile)
    const int resident = 148 * (S == 4 && 2 * (smem + 1024) <= 227 * 1024 ? 2 : 1);
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
    if constexpr (WSIDE)
        if (static_cast<long long>(round4(P.C)) * 8 * 4 * (BOUND ? 2 : 1) <= kMaxTile) return launch_scan_s<BOUND, WSIDE, 8>(P, st);
    return launch_scan_s<BOUND, WSIDE, 4>(P, st);
}

template <bool PAIR>
int launch_lists(const Operand& v, const Operand& second, long long rows, int C, int cap, const float* threshold,
                 typename EntryOf<PAIR>::type* list, int* len, float* rest, int* words, cudaStream_t st) {
    const unsigned grid = static_cast<unsigned>(rows);
    if (C <= 12 * kListThreads)
        return launch_after(extreme_lists_kernel<PAIR, 12>, grid, kListThreads, 0, st, v, second, C, cap, threshold, list, len,
                            rest, words);
    if (C <= 20 * kListThreads)
        return launch_after(extreme_lists_kernel<PAIR, 20>, grid, kListThreads, 0, st, v, second, C, cap, threshold, list, len,
                            rest, words);
    static_assert(kListKeep == 24, "the longest row");
    return launch_after(extreme_lists_kernel<PAIR, 24>, grid, kListThreads, 0, st, v, second, C, cap, threshold, list, len,
                        rest, words);
}

template <bool BOUND>
int run(const Problem& P, cudaStream_t st) {
    using EX = typename EntryOf<BOUND>::type;
    const cudaError_t e = cudaMemsetAsync(P.t.words, 0, kExtremeWords * sizeof(int), st);
    if (e != cudaSuccess) return cuda_status(e);
    const float* thresholds = reinterpret_cast<const float*>(P.t.words + kThresholdWord);
    int r = launch_after(extreme_sample_kernel<BOUND>, kSampleBlocks, 256, 0, st, P);
    if (r == kOk)
        r = launch_lists<false>(P.w, P.w, P.CO, P.C, kListW, thresholds, static_cast<Entry1*>(P.t.w_list), P.t.w_len, P.t.w_rest,
                                P.t.words, st);
    if (r == kOk)
        r = launch_lists<BOUND>(P.x, P.xu, P.B, P.C, kListX, thresholds + 1, static_cast<EX*>(P.t.x_list), P.t.x_len,
                                P.t.x_rest, P.t.words, st);
    if (r == kOk) r = launch_scan<BOUND, true>(P, st);
    if (r == kOk) r = launch_scan<BOUND, false>(P, st);
    if (r == kOk) {
        const long long rows4 = (P.B + 3) / 4;
        const dim3 grid(static_cast<unsigned>((P.CO + 255) / 256), static_cast<unsigned>(rows4 < 65535 ? rows4 : 65535));
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
