// p = inf forward of large fully connected layers: max_c |x[b, c] - w[o, c]| without visiting most channels.
//
// A channel can only be the maximum of output (b, o) where |x| or |w| is large.  So every row of either operand gets a list
// of its extreme channels and the largest magnitude that is NOT in the list, rest_o and rest_b.  The maximum over the two
// lists' channels, M, is compared with fl(rest_o + rest_b): a channel in neither list has |w| <= rest_o and |x| <= rest_b, hence
// |fl(x - w)| <= fl(rest_o + rest_b) (rounding is monotonic), so M > fl(rest_o + rest_b) proves that M is the maximum over all
// channels and that no other channel equals it: value and first channel are those of the dense kernel, bit for bit.  Outputs
// without the proof ("hard") are searched over all channels.  All arithmetic is the dense kernel's fp32 subtraction and
// comparison.
//
// A list holds the same number of channels in every row, the row's own largest ones, so rows may have any scale and a list
// never overflows (with one threshold for all rows, rows whose scales differ by a tenth overflowed their lists: the walks ran
// for nothing in front of the dense kernels).  The two lengths are chosen by trial on 592 outputs: their full maxima, and
// what the rests of their two rows would be after lists of any length, tell how many of them each pair of lengths leaves
// hard; the cheapest pair is taken, before anything is listed or walked.  Where no pair is cheaper than the dense kernels, or
// anything is not finite, or far more outputs turn out hard than the samples said, a device word makes the dense kernels behind
// run instead.
// Forward with index / bounds in us, against the dense kernels' 1048 / 2349 (512 x 5120 -> 5120) and 677 / 1426 (512 x 3072 ->
// 5120), w = N(0, 1) with rows scaled by exp(s N(0, 1)); one threshold for all rows in parentheses (+: dense behind the walks):
//                           s = 0                    s = 0.05                 s = 0.1                   s = 0.4
//   5120, x = N(0, 0.5^2)   373 / 701 (429 / 780)    359 / 696 (1531+/3240+)  369 / 699 (1091 / 2392)   416 / 768 (1091 / 2389)
//   5120, x in [0, 1)       203 / 262 (220 / 326)    201 / 263 (308 / 556)    195 / 271 (1089 / 2392)   206 / 339 (1089 / 2393)
//   3072, x = N(0, 0.5^2)   293 / 500 (341 / 541)    297 / 512 (396 / 637)    297 / 523 (1206+/1468)    344 / 543 (716 / 1468)
//   3072, x in [0, 1)       162 / 209 (183 / 205)    162 / 211 (218 / 264)    162 / 187 (978+/1804+)    175 / 228 (715 / 1468)
// Signs (w, x = +-1: nothing can be proven, the samples choose dense) 1083 / 2378 and 709 / 1461.  512 x 5120 -> 5120 layer,
// forward + backward: dense 1105 us, one threshold 496, now 430; certification of 512 x 3072 -> 5120 (value and bounds): 1971,
// 335 and 298.
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
constexpr int kListWarps = kListThreads / 32;
constexpr int kMaxChannels = 6144;
constexpr int kScanThreads = 512;
constexpr int kBatch = 8;          // entries a scan works on at a time (lists are whole batches long)
constexpr int kSamples = 148 * 4;
constexpr int kMaxTile = 224 * 1024;

// Lengths that are tried: kBatch (a + 1) entries of the weights' lists, kBatch b of the samples' (none at b = 0).
constexpr int kLevelsW = kListW / kBatch, kLevelsX = kListX / kBatch + 1;
// What a pair of lengths costs, in the walk of one entry of the weights' lists in tiles of eight rows (0.5 us of
// 512 x 5120 -> 5120, bounds 0.8), fitted to lengths of 40 to 256 and 0 to 128 at 3072 and 5120 channels:
//   the samples' lists at all, another pass over the weights and over the outputs: 52 - 54 us there, bounds 240;
//   an entry of theirs (four rows per step of a list instead of eight) 1.0 us, bounds 1.2;
//   one output in a hundred hard: 75 - 87 us at 5120 channels, 49 at 3072, bounds 100 and 63;
//   filling the tiles and reading the outputs 45 us, and the lists themselves 56 us (in proportion to rows, not to outputs).
// The dense kernels take a channel in 0.17 us there (without index), bounds 0.46.
struct Costs {
    float second_pass, second_entry, hard_channel, dense_channel;
};
template <bool BOUND>
__device__ constexpr Costs costs() {
    return BOUND ? Costs{290.0f, 1.7f, 2.5f, 1.0f / 2.5f} : Costs{100.0f, 2.0f, 3.2f, 1.0f / 3.5f};
}
constexpr float kFixedCost = 90.0f, kListCost = 11.0f;  // the latter per channel and row of the weights
constexpr int kMostFailed = 6;  // hard samples, at most: 1 % (3 % of the outputs are more than can be searched in full)

__host__ __device__ constexpr int round4(int c) { return (c + 3) & ~3; }
// whether a tile of the weights' lists' walk holds eight samples (with both bounds), not four
template <bool BOUND>
__host__ __device__ constexpr bool eight_rows(int C) {
    return round4(C) * 8 * 4 * (BOUND ? 2 : 1) <= kMaxTile;
}

// device words (cleared by every call): 0 dense gate, 1 finished sampling blocks, 2 hard outputs
constexpr int kLengthWord = 4;  // entries of a weight row's list, of a sample's
constexpr int kTrialWord = 8;   // [level a][first level b that proves the sample, kLevelsX: none], counts of samples
static_assert(kTrialWord + kLevelsW * (kLevelsX + 1) == kExtremeWords, "");

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
__device__ __forceinline__ float block_max(float v, float* warps) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
    __syncthreads();
    v = warps[0];
    for (int k = 1; k < kListWarps; ++k) v = fmaxf(v, warps[k]);
    return v;
}

// Magnitudes in order.  A block holds a row, thread t channels t + 256 k, magnitudes as integers (a sign bit less,
// not-a-numbers on top); padding has magnitude 0.  The channels of a class (channel % 4, so lane % 4) are put in the order of
// the bins of a histogram, 64 per octave and two octaves from half of a magnitude near the row's top (the fourth largest of
// the warps' maxima: outliers do not move it, nor runs of zeros), higher ones first, any order within a bin.  emit(k, m, place)
// is called for the places below `keep`; the return value is the largest magnitude of this thread's that got none, `top` the
// largest of all.  Magnitudes below the last bin get no place.
constexpr int kBins = 128;
constexpr int kBinShift = 23 - 6;
struct RankShared {
    int bins[4 * kBins];  // [bin][class]: counts, then the next place
    int warps[kListWarps];
    int upper[4], stop[4], total[4];
};
template <int KEEP, class Magnitude, class Emit>
__device__ __forceinline__ int rank_row(RankShared& sh, int keep, Magnitude magnitude, int& top, Emit emit) {
    static_assert(kListThreads == 2 * kBins, "a thread scans two bins of a class");
    const int t = threadIdx.x, lane = t & 31;
    top = 0;
#pragma unroll
    for (int k = 0; k < KEEP; ++k) top = max(top, magnitude(k));
    const int mine = __reduce_max_sync(0xffffffffu, top);
    __syncthreads();  // (the arrays may still be read from an earlier call)
    if (lane == 0) sh.warps[t >> 5] = mine;
    sh.bins[t] = sh.bins[t + kListThreads] = 0;
    __syncthreads();
    const int v = sh.warps[lane & 7];
    int above = 0;
#pragma unroll
    for (int j = 0; j < kListWarps; ++j) {
        const int o = sh.warps[j];
        above += (o > v || (o == v && j < (lane & 7))) ? 1 : 0;
    }
    const int near_top = __shfl_sync(0xffffffffu, v, __ffs(__ballot_sync(0xffffffffu, above == 3)) - 1);
    // (finite: then no sum below overflows; rows with infinities go to the dense kernels)
    const int cut = max(min(near_top, 0x7f7fffff) - (1 << 23), 1);
    auto bin_of = [&](int m) { return min((m - cut) >> kBinShift, kBins - 1) * 4 + (lane & 3); };
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
        const int m = magnitude(k);
        if (m >= cut) atomicAdd(&sh.bins[bin_of(m)], 1);
    }
    __syncthreads();
    // places: of class q, 64 threads with two bins each
    const int q = t >> 6, lower_bin = 2 * (t & 63);
    const int n0 = sh.bins[lower_bin * 4 + q], n1 = sh.bins[(lower_bin + 1) * 4 + q];
    int sum = n0 + n1;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_down_sync(0xffffffffu, sum, d);
        if (lane + d < 32) sum += o;
    }
    if ((t & 63) == 32) sh.upper[q] = sum;
    __syncthreads();
    if ((t & 32) == 0) sum += sh.upper[q];  // magnitudes in these two bins and above
    const int first1 = sum - n0 - n1, first0 = first1 + n1;
    sh.bins[(lower_bin + 1) * 4 + q] = first1;
    sh.bins[lower_bin * 4 + q] = first0;
    if (lower_bin == 0) sh.total[q] = sum;
    // the lowest bin that has a place below `keep`
    if (first0 < keep ? (lower_bin == 0 || sum >= keep) : first1 < keep) sh.stop[q] = first0 < keep ? lower_bin : lower_bin + 1;
    __syncthreads();
    const int limit = keep > 0 ? cut + (sh.stop[lane & 3] << kBinShift) : 0x7fffffff;
    int left = 0;
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
        const int m = magnitude(k);
        bool listed = false;
        if (m >= limit) {
            const int place = atomicAdd(&sh.bins[bin_of(m)], 1);
            if (place < keep) {
                emit(k, m, place);
                listed = true;
            }
        }
        if (!listed) left = max(left, m);
    }
    return left;
}
__device__ __forceinline__ int magnitude_of(float v) { return __float_as_int(v) & 0x7fffffff; }
constexpr int kInfinite = 0x7f800000;

// One block per row: its list and its rest; the row is read once, into registers, with all loads in flight (KEEP channels per
// thread).
//
// Order of a list.  A scan step reads one channel of each of a warp's lists from shared memory, 32 bytes at bank
// 8 (channel % 4) (tiles of 8 rows), so four neighbouring lists read without conflicts if their channels differ modulo 4.
// Entry k of row r's list therefore has channel % 4 == (k + r) % 4: four interleaved sub-lists with a quarter of the entries
// each, filled up with entries that change nothing (NaN) where a class has fewer magnitudes near the row's top.
template <bool PAIR, int KEEP>
__global__ void __launch_bounds__(kListThreads, KEEP <= 12 ? 4 : (PAIR && KEEP > 20 ? 2 : 3))
extreme_lists_kernel(Operand v, Operand second, int C, int cap, int length_word, typename EntryOf<PAIR>::type* list,
                     float* rest, int* words) {
    stream_order_begin();
    // (one decision per block: another block of this very kernel may set the word between two threads' reads)
    if (__syncthreads_or(words[0] != 0)) return;
    using E = typename EntryOf<PAIR>::type;
    __shared__ RankShared sh;
    const long long row = blockIdx.x;
    const int t = threadIdx.x, lane = t & 31;
    const int keep = words[length_word] / 4;
    const float* src = v.ptr + row * v.stride_row + t;
    const float* src2 = second.ptr + row * second.stride_row + t;
    float a[KEEP], b[PAIR ? KEEP : 1];
    const int mine_n = C - t;  // this thread's channels: t + 256 k < C
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
        a[k] = kListThreads * k < mine_n ? src[kListThreads * k] : 0.0f;
        if (PAIR) b[k] = kListThreads * k < mine_n ? src2[kListThreads * k] : 0.0f;
    }
    auto magnitude = [&](int k) {
        if constexpr (PAIR) return max(magnitude_of(a[k]), magnitude_of(b[k]));
        else return magnitude_of(a[k]);
    };
    int left = 0, top = 0;
    if (keep == 0) {
#pragma unroll
        for (int k = 0; k < KEEP; ++k) top = max(top, magnitude(k));
        left = top;
    } else {
        // entry of class q at place `p`
        auto entry_at = [&](int q, int p) { return list + entry_index(row, ((q - static_cast<int>(row & 3)) & 3) + 4 * p, cap); };
        left = rank_row<KEEP>(sh, keep, magnitude, top, [&](int k, int, int place) {
            const int c = t + kListThreads * k;
            E e;
            if constexpr (PAIR) e = E{a[k], b[k], c, 0};
            else e = E{a[k], c};
            *entry_at(lane & 3, place) = e;
        });
        const int q = t >> 6;
        for (int p = sh.total[q] + (t & 63); p < keep; p += 64) {
            const float none = __int_as_float(0x7fc00000);
            E e;
            if constexpr (PAIR) e = E{none, none, q, 0};
            else e = E{none, q};
            *entry_at(q, p) = e;
        }
    }
    if (top >= kInfinite) words[0] = 1;  // infinite or not a number: dense
    left = __reduce_max_sync(0xffffffffu, left);
    if (lane == 0) sh.warps[t >> 5] = left;
    __syncthreads();
    if (t == 0) {
#pragma unroll
        for (int k = 1; k < kListWarps; ++k) left = max(left, sh.warps[k]);
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

// A block per sampled output: its maximum over all channels, and for every length of the weights' list the shortest list of
// the sample's that would prove it.  The last block to finish chooses the two lengths, or the dense kernels.
template <bool BOUND, int KEEP>
__global__ void __launch_bounds__(kListThreads, KEEP <= 12 ? 3 : 2) extreme_sample_kernel(const Problem P) {
    stream_order_begin();
    __shared__ RankShared sh;
    __shared__ float warps[kListWarps];
    __shared__ int level_w[kLevelsW + 1], level_x[kLevelsX];  // largest magnitude among the places of a batch; last: without
    __shared__ int trials[kLevelsW * (kLevelsX + 1)];
    __shared__ unsigned long long best;
    __shared__ bool last;
    const int t = threadIdx.x, lane = t & 31;
    const unsigned id = blockIdx.x;
    // samples on a lattice that visits rows and outputs evenly (fractions of the golden ratio and of the square root of 2)
    const long long b = static_cast<long long>((static_cast<unsigned long long>(id * 2654435769u) * P.B) >> 32);
    const int o = static_cast<int>((static_cast<unsigned long long>(id * 1779033703u) * P.CO) >> 32);
    const float* xrow = P.x.ptr + b * P.x.stride_row + t;
    const float* urow = P.xu.ptr + b * P.xu.stride_row + t;
    const float* wrow = P.w.ptr + o * P.w.stride_row + t;
    float x[KEEP], u[BOUND ? KEEP : 1], w[KEEP];
    const int mine_n = P.C - t;
#pragma unroll
    for (int k = 0; k < KEEP; ++k) {
        const bool in = kListThreads * k < mine_n;
        x[k] = in ? xrow[kListThreads * k] : 0.0f;
        if (BOUND) u[k] = in ? urow[kListThreads * k] : 0.0f;
        w[k] = in ? wrow[kListThreads * k] : 0.0f;
    }
    if (t <= kLevelsW) level_w[t] = 0;
    if (t < kLevelsX) level_x[t] = 0;
    float lo = kFloor, up = kFloor;
#pragma unroll
    for (int k = 0; k < KEEP; ++k) visit<BOUND>(x[k], BOUND ? u[k] : x[k], w[k], lo, up);
    lo = block_max(lo, warps);
    if (BOUND) up = block_max(up, warps);
    const float value = BOUND ? fminf(lo, up) : lo;
    auto put = [&](int* level) { return [=](int, int m, int place) { atomicMax(&level[4 * place / kBatch], m); }; };
    int top_w, top_x;
    const int left_w = rank_row<KEEP>(sh, kListW / 4, [&](int k) { return magnitude_of(w[k]); }, top_w, put(level_w));
    const int left_x = rank_row<KEEP>(sh, kListX / 4, [&](int k) {
        return BOUND ? max(magnitude_of(x[k]), magnitude_of(u[k])) : magnitude_of(x[k]);
    }, top_x, put(level_x));
    const int worst_w = __reduce_max_sync(0xffffffffu, left_w), worst_x = __reduce_max_sync(0xffffffffu, left_x);
    if (lane == 0) {
        atomicMax(&level_w[kLevelsW], worst_w);
        atomicMax(&level_x[kLevelsX - 1], worst_x);
    }
    if (max(top_w, top_x) >= kInfinite) P.t.words[0] = 1;
    __syncthreads();
    if (t < kLevelsW) {
        int rest_o = 0, rest_b = 0, tries = 0;
        for (int k = t + 1; k <= kLevelsW; ++k) rest_o = max(rest_o, level_w[k]);
        for (int k = kLevelsX - 1; k >= 0; --k) {
            rest_b = max(rest_b, level_x[k]);
            tries += proven(value, __int_as_float(rest_o), __int_as_float(rest_b)) ? 0 : 1;
        }
        atomicAdd(&P.t.words[kTrialWord + t * (kLevelsX + 1) + tries], 1);
    }
    __threadfence();
    __syncthreads();
    if (t == 0) {
        last = atomicAdd(&P.t.words[1], 1) == kSamples - 1;
        best = ~0ull;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int i = t; i < kLevelsW * (kLevelsX + 1); i += kListThreads) trials[i] = __ldcg(&P.t.words[kTrialWord + i]);
    __syncthreads();
    constexpr Costs unit = costs<BOUND>();
    const float entry = BOUND && !eight_rows<BOUND>(P.C) ? 2.0f : 1.0f;
    const float most = unit.dense_channel * P.C - kFixedCost - kListCost * P.C / P.B;
    for (int i = t; i < kLevelsW * kLevelsX; i += kListThreads) {
        const int lw = i / kLevelsX, lx = i % kLevelsX;
        int failed = 0;
        for (int k = lx + 1; k <= kLevelsX; ++k) failed += trials[lw * (kLevelsX + 1) + k];
        const float cost = entry * kBatch * (lw + 1) +
                           (lx > 0 ? unit.second_pass + unit.second_entry * kBatch * lx : 0.0f) +
                           unit.hard_channel * P.C / kSamples * failed;
        if (failed <= kMostFailed && cost <= most)
            atomicMin(&best, (static_cast<unsigned long long>(__float_as_int(cost)) << 32) | i);
    }
    __syncthreads();
    if (t != 0) return;
    if (best == ~0ull) {
        P.t.words[0] = 1;
    } else {
        const int i = static_cast<int>(best & 0xffffffffu);
        P.t.words[kLengthWord] = kBatch * (i / kLevelsX + 1);
        P.t.words[kLengthWord + 1] = kBatch * (i % kLevelsX);
    }
}

// The maximum over one operand's lists.  WSIDE: S samples in shared memory, the weight rows' lists walked (sets y and pos);
// else: S weight rows in shared memory, the samples' lists walked (merged into y and pos).
//
// A lane owns a list and S outputs.  What bounds the walk is the load / store pipe: a step of 32 lists costs 4 S / 4 wavefronts
// of shared memory and about 4.5 of list entries, hence as many rows per list as fit (S = 8) where the lists are long; the
// samples' lists are short, and four rows leave room for two blocks, one filling its tile while the other walks.  (Times at
// 512 x 5120 -> 5120 with index, n entries: weights' lists 44 + 0.51 n us, samples' lists 44 + 1.0 n.)
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
    const int n = P.t.words[WSIDE ? kLengthWord : kLengthWord + 1];  // entries of every list
    if (n == 0) return;
    const E* list = static_cast<const E*>(WSIDE ? P.t.w_list : P.t.x_list);
    const long long row0 = block * S;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* tile = reinterpret_cast<float*>(tile4);
    float* tile_up = tile + static_cast<size_t>(C4) * 4 * S;
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
        auto load = [&](E (&en)[kBatch], int k0) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u) en[u] = entries[(k0 + u) * kGroup];
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
#pragma unroll
                for (int e = 0; e < S; ++e)
                    if (top[e] >= best[e]) {
                        batch[e] = top[e] > best[e] ? k0 : batch[e] | kTie;
                        best[e] = top[e];
                    }
            }
        };
        if constexpr (S == 4) {
            E en[kBatch];
            for (int k0 = 0; k0 < n; k0 += kBatch) {
                load(en, k0);
                work(en, k0);
            }
        } else {
            E even[kBatch], odd[kBatch];
            load(even, 0);
            for (int k0 = 0; k0 < n; k0 += 2 * kBatch) {
                const bool more = k0 + kBatch < n;
                if (more) load(odd, k0 + kBatch);
                work(even, k0);
                if (k0 + 2 * kBatch < n) load(even, k0 + 2 * kBatch);
                if (more) work(odd, k0 + kBatch);
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
    // a full search costs about 20 times an output's share of the dense kernels: 1 / 32 of them more than half of all those
    const long long n = B * CO / 32;
    return static_cast<unsigned>(n > 4096 ? n : 4096);
}

template <bool BOUND, bool WSIDE, int S>
int launch_scan_s(const Problem& P, cudaStream_t st) {
    static OncePerDevice once;
    int r = once([] { return allow_smem(extreme_scan_kernel<BOUND, WSIDE, S>, kMaxTile); });
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
        if (eight_rows<BOUND>(P.C)) return launch_scan_s<BOUND, WSIDE, 8>(P, st);
    return launch_scan_s<BOUND, WSIDE, 4>(P, st);
}

// KEEP channels per thread, in steps of four: the smallest that holds a row.
template <template <int> class Launch, class... A>
int by_row_length(int C, const A&... args) {
    switch ((C + 4 * kListThreads - 1) / (4 * kListThreads)) {
        case 1: case 2: return Launch<8>::run(args...);
        case 3: return Launch<12>::run(args...);
        case 4: return Launch<16>::run(args...);
        case 5: return Launch<20>::run(args...);
        default: break;
    }
    static_assert(kMaxChannels == 24 * kListThreads, "the longest row");
    return Launch<24>::run(args...);
}
template <bool PAIR>
struct Lists {
    template <int KEEP>
    struct Launch {
        static int run(const Operand& v, const Operand& second, long long rows, int C, int cap, int length_word,
                       typename EntryOf<PAIR>::type* list, float* rest, int* words, cudaStream_t st) {
            return launch_after(extreme_lists_kernel<PAIR, KEEP>, static_cast<unsigned>(rows), kListThreads, 0, st, v, second, C,
                                cap, length_word, list, rest, words);
        }
    };
};
template <bool BOUND>
struct Sample {
    template <int KEEP>
    struct Launch {
        static int run(const Problem& P, cudaStream_t st) {
            return launch_after(extreme_sample_kernel<BOUND, KEEP>, kSamples, kListThreads, 0, st, P);
        }
    };
};

template <bool BOUND>
int run(const Problem& P, cudaStream_t st) {
    using EX = typename EntryOf<BOUND>::type;
    const cudaError_t e = cudaMemsetAsync(P.t.words, 0, kExtremeWords * sizeof(int), st);
    if (e != cudaSuccess) return cuda_status(e);
    int r = by_row_length<Sample<BOUND>::template Launch>(P.C, P, st);
    if (r == kOk)
        r = by_row_length<Lists<false>::template Launch>(P.C, P.w, P.w, static_cast<long long>(P.CO), P.C, kListW, kLengthWord,
                                                         static_cast<Entry1*>(P.t.w_list), P.t.w_rest, P.t.words, st);
    if (r == kOk)
        r = by_row_length<Lists<BOUND>::template Launch>(P.C, P.x, P.xu, P.B, P.C, kListX, kLengthWord + 1,
                                                         static_cast<EX*>(P.t.x_list), P.t.x_rest, P.t.words, st);
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

// Lines of the rule.  Below 2048 channels the lists are not a small part of a row.  What a call pays whose data can prove
// nothing (samples, and the launches behind them that return at once) is 35 - 45 us: under 7 % of the dense kernels' time from
// 6.4 G pairs on (values; 512 x 3072 -> 5120, 8.1 G: 588 against 552), under 9 % of the bounds', which take them 2.6 times as
// long, from 2.5 G on (128 x 6144 -> 3300: 519 against 474), but 11 - 25 % below (values of 512 x 2048 -> 5120, 5.4 G: 418 against
// 378; 128 x 3072 -> 5500, 2.2 G: 195 against 163).  Data that it can be proven on gains there too: hidden activations 209
// against 380 and 152 against 165.  Beyond 6144 channels a row no longer fits a list block's registers and four rows of both
// bounds no longer shared memory; narrow sides leave the scan's blocks idle.
bool extreme_applies(long long B, int CO, int C, bool bound) {
    return C >= 2048 && C <= kMaxChannels && B >= 128 && CO >= 512 && B * CO < (1LL << 31) &&
           B * CO * C >= (bound ? 2500000000LL : 6400000000LL);
}

size_t extreme_scratch_bytes(long long B, int CO, bool bound) {
    const size_t ex = bound ? sizeof(Entry2) : sizeof(Entry1);
    return pad256(groups_of(B) * kGroup * kListX * ex) + pad256(groups_of(CO) * kGroup * kListW * sizeof(Entry1)) +
           pad256(B * sizeof(float)) + pad256(static_cast<size_t>(CO) * sizeof(float)) +
           pad256(static_cast<size_t>(most_hard_of(B, CO)) * sizeof(unsigned)) + pad256(kExtremeWords * sizeof(int));
}

bool extreme_take_scratch(Bump* bump, long long B, int CO, bool bound, ExtremeScratch* t) {
    const size_t ex = bound ? sizeof(Entry2) : sizeof(Entry1);
    t->x_list = bump->take<char>(groups_of(B) * kGroup * kListX * ex);
    t->w_list = bump->take<char>(groups_of(CO) * kGroup * kListW * sizeof(Entry1));
    t->x_rest = bump->take<float>(B);
    t->w_rest = bump->take<float>(CO);
    t->hard = bump->take<unsigned>(most_hard_of(B, CO));
    t->words = bump->take<int>(kExtremeWords);
    return t->x_list && t->w_list && t->x_rest && t->w_rest && t->hard && t->words;
}

int launch_extreme(Operand x, Operand xu, Operand w, long long B, int CO, int C, bool bound, float* y, float* yu, int* pos,
                   const float* sub, const float* add, const ExtremeScratch& t, const int** dense_gate, cudaStream_t st) {
    const Problem P{x, xu, w, B, CO, C, y, yu, pos, sub, add, t};
    *dense_gate = t.words;
    return bound ? run<true>(P, st) : run<false>(P, st);
}

}  // namespace ldn
