// General exponents, forward: y = (sum_c |x - w|^p)^(1/p) from the channels whose terms count.
//
// At p = 37.5 a term below 0.6 of the largest |t| is below 2^-27 of the sum: of 3072 channels all but a few hundred could be
// left out without a trace in fp32.  Which ones can is known from one operand at a time.  Every weight row lists its channels
// with |w - c| > tau_o (c: the middle of x's range), largest first in 64 levels; where the samples' values spread widely, every
// sample lists its channels with |x - c| > sigma.  A channel in neither list has |t| <= |w - c| + sigma, so all that is left out
// of an output's sum S is bounded by numbers of the weight row alone: its channels per level.  The output is done when
//     sum over the levels not looked at of channels * (upper end of the level + sigma)^p  <=  p * 2^-26 * S,
// a relative error of the value below 2^-26, and a walk along a row's list stops as soon as that holds for the samples of its
// tile.  Outputs that come to the end of the lists without it are summed directly.  tau_o is a fraction of the row's largest
// |w - c|, so that rows of different scales have lists of like length; that fraction and sigma come from sampled outputs, summed
// in full: the cheapest pair that would do for all but one of them, or the dense kernels if no pair is clearly cheaper.
//
// The walks hold a tile of one operand in shared memory as [channel][rows of the tile] and run along the lists of the other;
// each lane has a row of the tile, the groups of lanes take channels of different classes modulo kClasses, whose rows lie in
// different banks.  They are bound by the logarithm / exponential mix of the dense kernel (one MUFU logarithm per term, two
// exponentials in three as a polynomial) beside one shared-memory load and half a list load per term.
#include <float.h>
#include <math.h>

#include "ldn_ops.cuh"
#include "ldn_power_lists.cuh"

namespace ldn {
namespace {

constexpr int kBlock = 256;
constexpr int kSamples = 148;
constexpr int kLevels = 64;     // fractions of a weight row's largest |w - c|
constexpr int kSigmas = 8;      // fractions of the largest |x - c|
constexpr int kTrip = 6;        // entries per lane and trip of the walks
constexpr int kWalkWarps = 24;
constexpr int kCheck = 4;       // trips between two looks at whether a sum is done
constexpr float kEarly = 0.75f; // of a weight row's list, what is walked on average
constexpr int kDirectCap = 1 << 16;
constexpr int kMaxWide = 3500;  // channels up to which 16 rows of a tile fit shared memory (8 beyond)
constexpr int kMaxChannels = 7000;

__device__ __forceinline__ float sigma_fraction(int k) {
    const float f[kSigmas] = {1.0f, 0.85f, 0.7f, 0.6f, 0.5f, 0.4f, 0.3f, 0.2f};
    return f[k];
}

struct Entry {
    unsigned at;  // byte offset of the channel's row in the tile
    float v;
};

// Device words.
struct Words {
    unsigned x_top, x_low;       // ordered codes of the largest x and of the largest -x
    unsigned spread;             // bits of the largest |x - c|
    int samples_done;
    int direct_count;
    int dense;                   // read by the caller's kernels as their gate
    int x_listed;                // samples list channels at all
    float fraction, sigma;
    int hist_w[kLevels];         // of sampled weight rows: channels by |w - c| / largest
    int hist_x[kSigmas];         // of sampled samples: channels with |x - c| beyond each sigma
    float needed[kSigmas][kSamples];  // per sampled output: the largest fraction that proves it
};

struct ListParams {
    const float *x, *w;
    int B, CO, CI;
    float p;
    Words* words;
    float *x_abs, *x_mid, *w_abs, *w_mid;  // per row: largest magnitude, largest |v - c|
    Entry *w_lists, *x_lists;              // [row][class][cap]
    int *w_counts, *x_counts;              // entries per class (a multiple of kTrip)
    float* w_tails;                        // [row][trip]: log2 of the bound of all that trip and those behind it have, and the rest
    float* w_left;                         // [row]: the same of the channels not listed
    int w_cap, x_cap;
    int* direct;
    float* y;
};

__device__ __forceinline__ float center_of(const Words* W) { return 0.5f * (from_ordered(W->x_top) - from_ordered(W->x_low)); }

__global__ void __launch_bounds__(kBlock) lists_range_kernel(const ListParams P) {
    stream_order_begin();
    const long long total = static_cast<long long>(P.B) * P.CI;
    unsigned t = 0, l = 0;
#pragma unroll 4
    for (long long i = blockIdx.x * static_cast<long long>(kBlock) + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * kBlock) {
        const float v = P.x[i];
        t = max(t, ordered(v));
        l = max(l, ordered(-v));
    }
    t = __reduce_max_sync(0xffffffffu, t);
    l = __reduce_max_sync(0xffffffffu, l);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&P.words->x_top, t);
        atomicMax(&P.words->x_low, l);
    }
}

// Largest |v| and |v - c| of every row of both operands, a warp per row; values that are not finite send the call to the dense
// kernels.
__global__ void __launch_bounds__(kBlock) lists_rows_kernel(const ListParams P) {
    stream_order_begin();
    const int r = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= P.B + P.CO) return;
    const float c = center_of(P.words);
    const bool is_x = r < P.B;
    const float* row = is_x ? P.x + static_cast<long long>(r) * P.CI : P.w + static_cast<long long>(r - P.B) * P.CI;
    unsigned a = 0, m = 0;
#pragma unroll 8
    for (int k = lane; k < P.CI; k += 32) {
        const float v = row[k];
        a = max(a, __float_as_uint(v) & 0x7fffffffu);
        m = max(m, __float_as_uint(v - c) & 0x7fffffffu);
    }
    a = __reduce_max_sync(0xffffffffu, a);
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane != 0) return;
    (is_x ? P.x_abs[r] : P.w_abs[r - P.B]) = __uint_as_float(a);
    (is_x ? P.x_mid[r] : P.w_mid[r - P.B]) = __uint_as_float(m);
    if (is_x) atomicMax(&P.words->spread, m);
    if (max(a, m) >= 0x7f800000u) P.words->dense = 1;
}

// Level of |v - c| in a row whose largest is top: per = levels_per(top).
__device__ __forceinline__ float levels_per(float top) { return top > 0.0f ? kLevels / top : 0.0f; }
__device__ __forceinline__ int level_of(float distance, float per) { return min(kLevels - 1, static_cast<int>(distance * per)); }
// smallest distance of level `first` or above, by the same arithmetic (a row without levels has none)
__device__ __forceinline__ float least_of(int first, float per) {
    if (!(per > 0.0f)) return INFINITY;
    float d = first / per;
    while (level_of(d, per) >= first) d = nextafterf(d, 0.0f);
    while (level_of(d, per) < first) d = nextafterf(d, INFINITY);
    return d;
}

// What the channels that are left out may add to a sum, relative to it.
__device__ __forceinline__ float allowance(float p) { return p * (1.0f / (1 << 26)); }

// One sampled output per block, summed in full: the largest tau + sigma that would prove it, and how long lists would be.  The
// last block chooses.
__global__ void __launch_bounds__(kBlock) lists_sample_kernel(const ListParams P, float dense_share) {
    __shared__ float red[kBlock / 32];
    __shared__ int hist[kLevels], past[kSigmas];
    __shared__ bool last;
    stream_order_begin();
    Words* W = P.words;
    if (W->dense != 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, s = blockIdx.x;
    // (spread over both operands; coprime strides)
    const int o = static_cast<int>((static_cast<long long>(s) * P.CO) / kSamples), b = static_cast<int>((s * 7919ll + 13) % P.B);
    const float *xr = P.x + static_cast<long long>(b) * P.CI, *wr = P.w + static_cast<long long>(o) * P.CI;
    const float c = center_of(W), spread = __uint_as_float(W->spread), wm = P.w_mid[o];
    if (tid < kLevels) hist[tid] = 0;
    if (tid < kSigmas) past[tid] = 0;
    __syncthreads();
    const float per = levels_per(wm);
    float top = 0.0f;
    int over[kSigmas] = {};
    for (int k = tid; k < P.CI; k += kBlock) {
        top = fmaxf(top, fabsf(xr[k] - wr[k]));
        const float ax = fabsf(xr[k] - c);
        atomicAdd(&hist[level_of(fabsf(wr[k] - c), per)], 1);
#pragma unroll
        for (int q = 0; q < kSigmas; ++q) over[q] += ax > sigma_fraction(q) * spread;
    }
#pragma unroll
    for (int q = 0; q < kSigmas; ++q) atomicAdd(&past[q], over[q]);
    for (int d = 16; d > 0; d >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
    if (lane == 0) red[warp] = top;
    __syncthreads();
    for (int i = 0; i < kBlock / 32; ++i) top = fmaxf(top, red[i]);
    __syncthreads();
    float sum = 0.0f;
    if (top > 0.0f)
        for (int k = tid; k < P.CI; k += kBlock) sum += exp2f(P.p * log2f(fabsf(xr[k] - wr[k]) / top));
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (lane == 0) red[warp] = sum;
    __syncthreads();
    sum = 0.0f;
    for (int i = 0; i < kBlock / 32; ++i) sum += red[i];
    if (tid < kSigmas) {
        // levels from below, as long as what they have may be left out
        const float sigma = sigma_fraction(tid) * spread, room = allowance(P.p) * sum;
        float left = 0.0f;
        int level = 0;
        if (wm > 0.0f && top > 0.0f)
            for (; level < kLevels; ++level) {
                if (hist[level]) left += hist[level] * exp2f(P.p * log2f((wm * (level + 1) / kLevels + sigma) / top));
                if (!(left <= room)) break;
            }
        W->needed[tid][s] = static_cast<float>(level) / kLevels;
        if (past[tid]) atomicAdd(&W->hist_x[tid], past[tid]);
    }
    if (tid < kLevels && hist[tid]) atomicAdd(&W->hist_w[tid], hist[tid]);
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(&W->samples_done, 1) == kSamples - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    __shared__ float needed[kSigmas][kSamples];
    __shared__ int counts_w[kLevels], counts_x[kSigmas];
    for (int i = tid; i < kSigmas * kSamples; i += kBlock)
        needed[i / kSamples][i % kSamples] = *static_cast<volatile float*>(&W->needed[i / kSamples][i % kSamples]);
    if (tid < kLevels) counts_w[tid] = *static_cast<volatile int*>(&W->hist_w[tid]);
    if (tid < kSigmas) counts_x[tid] = *static_cast<volatile int*>(&W->hist_x[tid]);
    __syncthreads();
    __shared__ float best_cost[kBlock / 32];
    __shared__ int best_at[kBlock / 32];
    float cost = FLT_MAX;
    int at = -1;
    for (int i = tid; i < kSigmas * kLevels; i += kBlock) {
        const int q = i / kLevels, level = i % kLevels;
        if (level == 0) continue;
        const float f = static_cast<float>(level) / kLevels;
        int failed = 0;
        for (int k = 0; k < kSamples; ++k) failed += !(needed[q][k] >= f);
        if (failed > 1) continue;
        int nw = 0;
        for (int k = level; k < kLevels; ++k) nw += counts_w[k];
        const int nx = counts_x[q];
        // (without samples' lists most walks stop early; a term of the second walk also looks its weight's list up, and the walk
        // needs tiles of the weights)
        const float t = q == 0 ? kEarly * nw / kSamples : (nw + 1.2f * nx) / kSamples + 0.04f * P.CI;
        if (t < cost) {
            cost = t;
            at = i;
        }
    }
    for (int d = 16; d > 0; d >>= 1) {
        const float t = __shfl_xor_sync(0xffffffffu, cost, d);
        const int i = __shfl_xor_sync(0xffffffffu, at, d);
        if (t < cost || (t == cost && i > at)) {
            cost = t;
            at = i;
        }
    }
    if (lane == 0) {
        best_cost[warp] = cost;
        best_at[warp] = at;
    }
    __syncthreads();
    if (tid != 0) return;
    for (int i = 1; i < kBlock / 32; ++i)
        if (best_cost[i] < cost) {
            cost = best_cost[i];
            at = best_at[i];
        }
    if (at < 0 || !(cost < dense_share * P.CI)) {
        W->dense = 1;
        return;
    }
    W->fraction = static_cast<float>(at % kLevels) / kLevels;
    W->sigma = sigma_fraction(at / kLevels) * spread;
    W->x_listed = at / kLevels != 0;
}

// Lists of both operands, a warp per row: by level, largest first, in channel order within one (samples' lists have one level).
// The ends of a row's lists are filled up to equal lengths, multiples of kTrip, with entries of a row of zeros behind the tile's
// last channel: a term of 0.
template <int ROWS>
__global__ void __launch_bounds__(kBlock) lists_build_kernel(const ListParams P) {
    constexpr int CLASSES = 32 / ROWS;
    constexpr int AHEAD = 8;
    __shared__ int at_all[kBlock / 32][kLevels * CLASSES];
    stream_order_begin();
    Words* W = P.words;
    if (W->dense != 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = blockIdx.x * (kBlock / 32) + warp;
    if (r >= P.B + P.CO) return;
    const bool is_x = r < P.B;
    if (is_x && !W->x_listed) {
        if (lane == 0) P.x_counts[r] = 0;
        return;
    }
    int* at = at_all[warp];  // [level][class]: entries, then the next entry's place
    const int row = is_x ? r : r - P.B, cap = is_x ? P.x_cap : P.w_cap, cls = lane % CLASSES;
    const float c = center_of(W), top = is_x ? 0.0f : P.w_mid[row], sigma = W->sigma;
    const float per = levels_per(top);
    const int first = static_cast<int>(W->fraction * kLevels + 0.5f);  // lowest level that is listed
    const float* src = (is_x ? P.x : P.w) + static_cast<long long>(row) * P.CI;
    Entry* dst = (is_x ? P.x_lists : P.w_lists) + static_cast<long long>(row) * CLASSES * cap;
    auto level = [&](float v) {
        const float a = fabsf(v - c);
        return is_x ? (a > sigma ? kLevels - 1 : 0) : level_of(a, per);
    };
    const int lowest = is_x ? kLevels - 1 : first;
    for (int i = lane; i < kLevels * CLASSES; i += 32) at[i] = 0;
    __syncwarp();
    // twice along the row: entries per level, then the entries
    auto along = [&](auto take) {
        for (int k0 = 0; k0 < P.CI; k0 += 32 * AHEAD) {
            float v[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) v[i] = k0 + 32 * i + lane < P.CI ? src[k0 + 32 * i + lane] : 0.0f;
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) take(k0 + 32 * i + lane, v[i]);
        }
    };
    along([&](int k, float v) {
        if (k < P.CI) atomicAdd(&at[level(v) * CLASSES + cls], 1);
    });
    __syncwarp();
    // bounds of what is left behind each level, on the scale of the largest
    float left[kLevels / 32] = {};  // lane: levels 2 lane, 2 lane + 1: all of that level and below
    const float scale = top + sigma;
    if (!is_x) {
        float below = 0.0f;
#pragma unroll
        for (int i = 0; i < kLevels / 32; ++i) {
            const int l = lane * (kLevels / 32) + i;
            int n = 0;
#pragma unroll
            for (int k = 0; k < CLASSES; ++k) n += at[l * CLASSES + k];
            below += n > 0 ? n * exp2f(P.p * log2f((top * (l + 1) / kLevels + sigma) / scale)) : 0.0f;
            left[i] = below;
        }
        float sum = below;
        for (int d = 1; d < 32; d <<= 1) {
            const float t = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= d) sum += t;
        }
        sum -= below;  // of the lanes in front
#pragma unroll
        for (int i = 0; i < kLevels / 32; ++i) left[i] = P.p * log2f(scale) + log2f((left[i] + sum) * 1.0001f);
    }
    auto left_at = [&](int l) {  // (warp-uniform or not: every lane asks)
        float v = 0.0f;
#pragma unroll
        for (int i = 0; i < kLevels / 32; ++i) {
            const float t = __shfl_sync(0xffffffffu, left[i], l / (kLevels / 32));
            if (l % (kLevels / 32) == i) v = t;
        }
        return v;
    };
    // places: classes side by side, levels from above
    int n = 0;
    if (lane < CLASSES)
        for (int l = kLevels - 1; l >= lowest; --l) {
            const int here = at[l * CLASSES + lane];
            at[l * CLASSES + lane] = n;
            n += here;
        }
    n = __shfl_sync(0xffffffffu, n, cls);
    int longest = static_cast<int>(__reduce_max_sync(0xffffffffu, static_cast<unsigned>(n)));
    longest = (longest + kTrip - 1) / kTrip * kTrip;
    if (longest > cap) {  // (cap is a multiple of kTrip)
        if (lane == 0) W->dense = 1;
        return;
    }
    __syncwarp();
    along([&](int k, float v) {
        const int l = level(v);
        const bool listed = k < P.CI && l >= lowest;
        const int key = listed ? l * CLASSES + cls : -1;
        const unsigned same = __match_any_sync(0xffffffffu, key);
        int place = listed ? at[key] : 0;
        __syncwarp();
        if (listed && (same & ((1u << lane) - 1)) == 0) at[key] = place + __popc(same);
        __syncwarp();
        place += __popc(same & ((1u << lane) - 1));
        if (listed) dst[cls * cap + place] = Entry{static_cast<unsigned>(k) * (ROWS * 4), v};
    });
    // zero rows: one of each class behind the last channel
    const unsigned zero = static_cast<unsigned>((P.CI + CLASSES - 1) / CLASSES * CLASSES + cls) * (ROWS * 4);
    for (int i = n + lane / CLASSES; i < longest; i += 32 / CLASSES) dst[cls * cap + i] = Entry{zero, 0.0f};
    if (lane == 0) (is_x ? P.x_counts : P.w_counts)[row] = longest;
    if (is_x) return;
    // of each trip: the bound of its highest level (at[] now holds where each level ends)
    __syncwarp();
    const int trips = longest / kTrip;
    for (int t0 = 0; t0 < trips; t0 += 32) {
        const int t = t0 + lane;
        int l = first - 1;
        for (int q = kLevels - 1; q >= first; --q) {
            bool here = false;
#pragma unroll
            for (int k = 0; k < CLASSES; ++k) here |= at[q * CLASSES + k] > t * kTrip;
            if (here) {
                l = q;
                break;
            }
        }
        const float v = left_at(max(l, 0));
        if (t < trips) P.w_tails[static_cast<long long>(row) * (P.w_cap / kTrip) + t] = l < 0 ? -INFINITY : v;
    }
    const float rest = left_at(max(first - 1, 0));
    if (lane == 0) P.w_left[row] = first > 0 ? rest : -INFINITY;
}

// The value of a sum, or a place on the list of outputs to be summed directly.  left: log2 of the bound of what the sum leaves out.
__device__ __forceinline__ float finish_value(const ListParams& P, float s, float norm, float left, bool done, long long off) {
    Words* W = P.words;
    const float scale = log2f(norm);
    if ((!(done || left - P.p * scale <= log2f(allowance(P.p) * s)) || !(s >= kNormGuard)) && *static_cast<volatile int*>(&W->dense) == 0) {
        const int at = atomicAdd(&W->direct_count, 1);
        if (at < kDirectCap) P.direct[at] = static_cast<int>(off);
        else W->dense = 1;
    }
    return norm * powf(s + exp2f(P.p * (log2f(kEps) - scale)), 1.0f / P.p);
}

// One walk.  !SECOND: tile = ROWS samples, lists = weight rows; makes the values if no sample lists anything, else leaves sums in
// y[b][o].  SECOND: tile = ROWS weight rows, lists = samples; channels that the weight row lists itself are skipped, and the values
// are made of both sums.
template <int ROWS, bool SECOND>
__global__ void __launch_bounds__(32 * kWalkWarps, 1) lists_walk_kernel(const ListParams P) {
    constexpr int CLASSES = 32 / ROWS;
    constexpr int GROUP = 8;               // lists whose sums are stored at once
    constexpr int OWN = GROUP / CLASSES;   // of which a lane makes the values
    extern __shared__ __align__(16) char tile[];
    stream_order_begin();
    Words* W = P.words;
    if (__syncthreads_or(W->dense != 0)) return;  // (as one: a walk may set it while other blocks begin)
    const bool x_listed = W->x_listed != 0;
    if (SECOND && !x_listed) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lr = lane % ROWS, cls = lane / ROWS;
    const float c = center_of(W), log_allowance = log2f(allowance(P.p));
    const int tile_rows = SECOND ? P.CO : P.B, lists = SECOND ? P.B : P.CO;
    const float* tile_src = SECOND ? P.w : P.x;
    const Entry* entries = SECOND ? P.x_lists : P.w_lists;
    const int* counts = SECOND ? P.x_counts : P.w_counts;
    const int cap = SECOND ? P.x_cap : P.w_cap;
    const float *tile_abs = SECOND ? P.w_abs : P.x_abs, *list_abs = SECOND ? P.x_abs : P.w_abs;
    const int tiles = (tile_rows + ROWS - 1) / ROWS, groups = (lists + GROUP - 1) / GROUP;
    const long long units = static_cast<long long>(tiles) * groups;
    const long long u0 = units * blockIdx.x / gridDim.x, u1 = units * (blockIdx.x + 1) / gridDim.x;
    const int zero_from = (P.CI + CLASSES - 1) / CLASSES * CLASSES;
    for (long long u = u0; u < u1;) {
        const int t = static_cast<int>(u / groups), g0 = static_cast<int>(u - static_cast<long long>(t) * groups);
        const int g1 = static_cast<int>(u1 - u < groups - g0 ? g0 + (u1 - u) : groups);
        __syncthreads();
        // the tile, [channel][row]: lanes along the channels, four rows per thread and store
        for (int i = tid; i < P.CI * (ROWS / 4); i += 32 * kWalkWarps) {
            const int q = i / P.CI, k = i - q * P.CI;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const int r = t * ROWS + 4 * q;
            const float* src = tile_src + static_cast<long long>(r) * P.CI + k;
            if (r < tile_rows) v.x = src[0];
            if (r + 1 < tile_rows) v.y = src[P.CI];
            if (r + 2 < tile_rows) v.z = src[2 * static_cast<long long>(P.CI)];
            if (r + 3 < tile_rows) v.w = src[3 * static_cast<long long>(P.CI)];
            *reinterpret_cast<float4*>(tile + k * (ROWS * 4) + q * 16) = v;
        }
        for (int i = tid; i < CLASSES * ROWS; i += 32 * kWalkWarps) reinterpret_cast<float*>(tile)[zero_from * ROWS + i] = 0.0f;
        __syncthreads();
        const int row = t * ROWS + lr;
        const bool in = row < tile_rows;
        const float own = in ? tile_abs[row] : 1.0f;
        // from where on the weight row's own lists have a channel
        const float listed_from =
            SECOND && in ? least_of(static_cast<int>(W->fraction * kLevels + 0.5f), levels_per(P.w_mid[row])) : INFINITY;
        const char* base = tile + lr * 4;
        for (int g = g0 + warp; g < g1; g += kWalkWarps) {
            float sums[OWN];
            unsigned done = 0;  // lists whose walk ended because every sum of the tile was complete
#pragma unroll 1
            for (int i = 0; i < GROUP; ++i) {
                const int l = g * GROUP + i;
                float s = 0.0f;
                if (l < lists) {
                    const int n = counts[l];
                    const float norm = fmaxf(own + list_abs[l], kEps), off = -P.p * log2f(norm);
                    const float2 pp = make_float2(P.p, P.p), off2 = make_float2(off, off);
                    const uint4* e = reinterpret_cast<const uint4*>(entries + (static_cast<long long>(l) * CLASSES + cls) * cap);
                    const float* tails = P.w_tails + static_cast<long long>(l) * (P.w_cap / kTrip);
                    float2 acc = make_float2(0.0f, 0.0f);
                    uint4 q[kTrip / 2];
                    if (n > 0)
#pragma unroll
                        for (int k = 0; k < kTrip / 2; ++k) q[k] = e[k];
                    const int trips = n / kTrip;
                    for (int trip = 0; trip < trips; ++trip) {
                        float2 tv[kTrip / 2];
#pragma unroll
                        for (int k = 0; k < kTrip / 2; ++k) {
                            const float v0 = *reinterpret_cast<const float*>(base + q[k].x), v1 = *reinterpret_cast<const float*>(base + q[k].z);
                            tv[k] = __fadd2_rn(make_float2(v0, v1), make_float2(-__uint_as_float(q[k].y), -__uint_as_float(q[k].w)));
                            if (SECOND) {
                                if (fabsf(v0 - c) >= listed_from) tv[k].x = 0.0f;
                                if (fabsf(v1 - c) >= listed_from) tv[k].y = 0.0f;
                            }
                        }
                        e += kTrip / 2;
                        const bool more = trip + 1 < trips, look = !SECOND && !x_listed && more && trip % kCheck == kCheck - 1;
                        const float tail = look ? tails[trip + 1] : 0.0f;
                        if (more)
#pragma unroll
                            for (int k = 0; k < kTrip / 2; ++k) q[k] = e[k];
#pragma unroll
                        for (int k = 0; k < kTrip / 2; ++k) {
                            const float2 lg = make_float2(lg2_approx(fabsf(tv[k].x)), lg2_approx(fabsf(tv[k].y)));
                            acc = __fadd2_rn(acc, ex2_mixed2<4, kMufuEveryFwd>(__ffma2_rn(pp, lg, off2), k));
                        }
                        if (look) {
                            float part = acc.x + acc.y;
#pragma unroll
                            for (int d = ROWS; d < 32; d <<= 1) part += __shfl_xor_sync(0xffffffffu, part, d);
                            if (__all_sync(0xffffffffu, !in || tail + off <= log_allowance + lg2_approx(part) - 0.01f)) {
                                done |= 1u << i;
                                break;
                            }
                        }
                    }
                    s = acc.x + acc.y;
                }
#pragma unroll
                for (int d = ROWS; d < 32; d <<= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
#pragma unroll
                for (int k = 0; k < OWN; ++k)
                    if (cls * OWN + k == i) sums[k] = s;
            }
            if (!in) continue;
#pragma unroll
            for (int k = 0; k < OWN; ++k) {
                const int i = cls * OWN + k, l = g * GROUP + i;
                if (l >= lists) continue;
                const float norm = fmaxf(own + list_abs[l], kEps);
                const int b = SECOND ? l : row, o = SECOND ? row : l;
                const long long at = static_cast<long long>(b) * P.CO + o;
                if (SECOND) P.y[at] = finish_value(P, sums[k] + P.y[at], norm, P.w_left[o], false, at);
                else P.y[at] = x_listed ? sums[k] : finish_value(P, sums[k], norm, P.w_left[o], (done >> i & 1) != 0, at);
            }
        }
        u += g1 - g0;
    }
}

// The outputs that could not be proven, a block each: largest difference first, then the sum, as the dense kernels have it.
__global__ void __launch_bounds__(kBlock) lists_direct_kernel(const ListParams P) {
    __shared__ float red[2][kBlock / 32];
    stream_order_begin();
    if (P.words->dense != 0) return;
    const int count = min(P.words->direct_count, kDirectCap), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int off = P.direct[i], b = off / P.CO, o = off - b * P.CO;
        const float *xr = P.x + static_cast<long long>(b) * P.CI, *wr = P.w + static_cast<long long>(o) * P.CI;
        float top = kEps;
#pragma unroll 4
        for (int k = threadIdx.x; k < P.CI; k += kBlock) top = fmaxf(top, fabsf(xr[k] - wr[k]));
        for (int d = 16; d > 0; d >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
        if (lane == 0) red[0][warp] = top;
        __syncthreads();
        for (int k = 0; k < kBlock / 32; ++k) top = fmaxf(top, red[0][k]);
        const float off2 = -P.p * log2f(top);
        float s = 0.0f;
#pragma unroll 4
        for (int k = threadIdx.x; k < P.CI; k += kBlock) s += ex2_approx(fmaf(P.p, lg2_approx(fabsf(xr[k] - wr[k])), off2));
        for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (lane == 0) red[1][warp] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            s = 0.0f;
            for (int k = 0; k < kBlock / 32; ++k) s += red[1][k];
            P.y[off] = top * powf(s + exp2f(P.p * (log2f(kEps) - log2f(top))), 1.0f / P.p);
        }
        __syncthreads();
    }
}

// ---- host ------------------------------------------------------------------------------------------------------------
inline int tile_rows_of(int channels) { return channels <= kMaxWide ? 16 : 8; }
inline int whole_trips(double n) { return static_cast<int>(ceil(n / kTrip)) * kTrip; }
// Room for lists of 0.65 (weights) and 0.35 (samples) of the channels: longer ones would not be cheaper than the dense kernels.
inline int w_cap_of(const Shape& s) { return whole_trips(0.65 * s.CI / (32 / tile_rows_of(s.CI))); }
inline int x_cap_of(const Shape& s) { return whole_trips(0.35 * s.CI / (32 / tile_rows_of(s.CI))); }

template <int ROWS>
int launch_lists(const ListParams& P, int sm_count, cudaStream_t st) {
    static OncePerDevice once;
    constexpr int classes = 32 / ROWS;
    const int smem = ((P.CI + classes - 1) / classes * classes + classes) * ROWS * 4;
    int r = once([] {
        constexpr int most = ((ROWS == 16 ? kMaxWide : kMaxChannels) + 2 * (32 / ROWS)) * ROWS * 4;
        const cudaError_t e = allow_smem(lists_walk_kernel<ROWS, false>, most);
        return e == cudaSuccess ? allow_smem(lists_walk_kernel<ROWS, true>, most) : e;
    });
    if (r != kOk) return r;
    const int row_blocks = (P.B + P.CO + kBlock / 32 - 1) / (kBlock / 32);
    r = launch_after(lists_range_kernel, 2 * sm_count, kBlock, 0, st, P);
    if (r == kOk) r = launch_after(lists_rows_kernel, row_blocks, kBlock, 0, st, P);
    if (r == kOk) r = launch_after(lists_sample_kernel, kSamples, kBlock, 0, st, P, 0.5f);
    if (r == kOk) r = launch_after(lists_build_kernel<ROWS>, row_blocks, kBlock, 0, st, P);
    if (r == kOk) r = launch_after(lists_walk_kernel<ROWS, false>, sm_count, 32 * kWalkWarps, smem, st, P);
    if (r == kOk) r = launch_after(lists_walk_kernel<ROWS, true>, sm_count, 32 * kWalkWarps, smem, st, P);
    if (r == kOk) r = launch_after(lists_direct_kernel, 8 * sm_count, kBlock, 0, st, P);
    return r;
}

}  // namespace

// Forward pass, us, dense -> this path, images in [0, 1] / zero-mean activations of deviation 0.5, N(0, 1) weights:
//     512 x 3072 -> 5120   p = 28    3053 -> 1143 / 3088        512 x 1024 -> 2048   p = 28    454 -> 293 / 487
//                          p = 37.5  3050 ->  726 / 1726                             p = 37.5  454 -> 224 / 417
//                          p = 100   3052 ->  352, 6674 -> 832                       p = 100   453 -> 125, 993 -> 266
// (p = 100, activations: the dense path has to find the largest differences first).  Where the samples choose the dense kernels
// the call takes 30 us more than it did: 1 % at 8 G pairs, 7 % at 1 G, so the line is drawn at 2 G; and at p = 32, below which
// activations no longer gain.
bool power_lists_apply(const Shape& s, float p) {
    return s.G == 1 && s.HW == 1 && p >= 32.0f && p <= 100.0f && s.CI >= 512 && s.CI <= kMaxChannels && s.M >= 16 && s.CO >= 64 &&
           s.M * s.CO <= (1LL << 30) && static_cast<double>(s.M) * s.CO * s.CI >= 2e9;
}

size_t power_lists_bytes(const Shape& s) {
    const size_t classes = 32 / tile_rows_of(s.CI), rows = static_cast<size_t>(s.M) + s.CO;
    return pad256(sizeof(Words)) + 4 * pad256(rows * 4) + 2 * pad256(rows * 4) + pad256(kDirectCap * 4) +
           pad256(static_cast<size_t>(s.CO) * (w_cap_of(s) / kTrip) * 4) + pad256(static_cast<size_t>(s.CO) * 4) +
           pad256(static_cast<size_t>(s.CO) * classes * w_cap_of(s) * sizeof(Entry)) +
           pad256(static_cast<size_t>(s.M) * classes * x_cap_of(s) * sizeof(Entry));
}

int launch_power_lists(const float* x, const float* w, const Shape& s, float* y, float p, int sm_count, Bump* bump, PowerLists* out,
                       cudaStream_t st) {
    const size_t classes = 32 / tile_rows_of(s.CI), B = static_cast<size_t>(s.M), CO = s.CO;
    ListParams P{};
    P.x = x; P.w = w; P.y = y; P.p = p;
    P.B = static_cast<int>(s.M); P.CO = s.CO; P.CI = s.CI;
    P.w_cap = w_cap_of(s);
    P.x_cap = x_cap_of(s);
    P.words = bump->take<Words>(1);
    P.x_abs = bump->take<float>(B);
    P.x_mid = bump->take<float>(B);
    P.w_abs = bump->take<float>(CO);
    P.w_mid = bump->take<float>(CO);
    P.x_counts = bump->take<int>(B);
    P.w_counts = bump->take<int>(CO);
    P.direct = bump->take<int>(kDirectCap);
    P.w_tails = bump->take<float>(CO * (P.w_cap / kTrip));
    P.w_left = bump->take<float>(CO);
    P.w_lists = bump->take<Entry>(CO * classes * P.w_cap);
    P.x_lists = bump->take<Entry>(B * classes * P.x_cap);
    if (!P.words || !P.x_abs || !P.x_mid || !P.w_abs || !P.w_mid || !P.x_counts || !P.w_counts || !P.direct || !P.w_tails || !P.w_left || !P.w_lists || !P.x_lists)
        return kWorkspace;
    const cudaError_t e = cudaMemsetAsync(P.words, 0, sizeof(Words), st);
    if (e != cudaSuccess) return cuda_status(e);
    *out = PowerLists{P.x_abs, P.w_abs, &P.words->dense};
    return s.CI <= kMaxWide ? launch_lists<16>(P, sm_count, st) : launch_lists<8>(P, sm_count, st);
}

}  // namespace ldn
