// Even integer exponents: which path, which scratch, and the calls of the instantiations (ldn_even_impl.cuh says how they work).
#include "ldn_even_impl.cuh"

namespace ldn {

namespace {
// Which path is the faster one: estimated times in microseconds, from fits to measured calls of either (32 - 512 rows or 8 -
// 128 images, 256 - 4096 channels, 256 - 5120 outputs; they are within 15 % of most).  The matrix products take a fixed time
// for preparation and launches and one per stage of 64 reduction elements, the backward pass also one per tile; the direct
// kernels a time per pair, padding of their 128-wide tiles included.  Either runs on the CTAs it may have: the fits' times per
// stage and per pair go up as those go down (512 x 1536 -> 2048, p = 8, 37 of 148: 842 / 1614 us direct,
// 212 / 434 on the products).  Measured, direct -> this path, p = 8, forward / both
// gradients: 512 x 3072 -> 5120 1045 / 2019 -> 285 / 640, 256 x 1024 -> 2048 81 / 161 -> 70 / 128, 256 x 1024 -> 1024 50 / 103
// -> 52 / 102 (here the line lies), 64 x 784 -> 1024 20 / 71 -> 47 / 97; 32 images of 576 x 1024 -> 128 340 / 878 -> 232 / 426.
constexpr double kMargin = 1.1;         // the estimate has to win by this factor
constexpr int kLeastChannels = 192;     // below, an output's error is a few terms' error: no smaller than the direct sum's

double padded(double n, double tile) { return ceil(n / tile) * tile; }
double direct_rows(const Shape& s) { return s.M <= 64 ? 64.0 : padded(static_cast<double>(s.M), 128.0); }
// elements of x, w and the output that preparation reads and writes, at the rate it does
double prepare_us(const Shape& s) {
    const double x = static_cast<double>(s.M) * s.CI, w = static_cast<double>(s.CO) * s.CIg, y = static_cast<double>(s.M) * s.CO;
    return (x + w + 4.0 * y) * 4.0 / 2.5e6;
}
bool in_range(const Shape& s, double stages) {
    return s.CIg >= kLeastChannels && s.M * s.CO <= (1LL << 30) && s.G * s.M <= (1LL << 30) && stages < 1e9;
}

}  // namespace

bool even_forward_applies(const Shape& s, float p, int cap, int sm_count) {
    const int i = static_cast<int>(p) / 2 - 1;
    constexpr double per_stage[4] = {2.3, 1.35, 1.2, 1.15}, per_pair[4] = {80e-9, 100e-9, 138e-9, 130e-9};
    const ForwardPlan f = plan_forward(s, 2 * i + 1);
    const double stages = static_cast<double>(f.total);
    const double products = 38.0 + prepare_us(s) + per_stage[i] * ceil(stages / (cap / 2));
    const double narrow = i == 3 && s.COg <= 64 ? (s.COg <= 32 ? 32.0 : 64.0) : 128.0;
    const double direct = 12.0 + per_pair[i] * direct_rows(s) * padded(s.COg, narrow) * s.G * s.CIg * sm_count / (cap > 0 ? cap : 1);
    return cap >= 2 && in_range(s, stages) && products * kMargin < direct;
}

bool even_backward_applies(const Shape& s, float p, bool gx, bool gw, int cap, int sm_count) {
    const int i = static_cast<int>(p) / 2 - 1, ct = channels_of(2 * i + 1);
    constexpr double per_stage[4] = {2.4, 1.3, 0.92, 1.05}, per_tile = 2.7;
    constexpr double both[4] = {139e-9, 195e-9, 223e-9, 248e-9}, one[4] = {85e-9, 134e-9, 162e-9, 190e-9};
    const double columns = div_up(s.CIg, ct), workers = cap / 2 > 0 ? cap / 2 : 1;
    double products = (gx && gw ? 70.0 : 58.0) + prepare_us(s), most = 0.0;
    for (int k = 0; k < 2; ++k) {
        if (!(k == 0 ? gx : gw)) continue;
        const double tiles = s.G * columns * row_tiles(k == 0 ? s.M : s.COg), stages = tiles * stages_of(k == 0 ? s.COg : s.M);
        products += per_stage[i] * ceil(stages / workers) + per_tile * ceil(tiles / workers);
        most = stages > most ? stages : most;
    }
    // tiles of the direct kernels: rows x channels, over the outputs; for grad_w alone outputs x channels, over the rows
    const double columns_d = s.G * padded(s.CIg, 128.0), out_rows = s.COg <= 64 ? 64.0 : padded(s.COg, 128.0);
    double pairs = columns_d * (gx ? direct_rows(s) * padded(s.COg, 32.0) : out_rows * padded(static_cast<double>(s.M), 32.0));
    pairs *= static_cast<double>(sm_count) / (cap > 0 ? cap : 1);
    const double direct = gx && gw ? 35.0 + both[i] * pairs : 30.0 + one[i] * pairs;
    return cap >= 2 && in_range(s, most) && products * kMargin < direct;
}

size_t even_forward_bytes(const Shape& s, float p, int cap) {
    const size_t rows = static_cast<size_t>(s.G) * s.M + s.CO;
    const ForwardPlan f = plan_forward(s, static_cast<int>(p) - 1);
    return pad256(f.image_bytes) + pad256(rows * sizeof(double)) +
           pad256(2 * rows * sizeof(float)) + pad256(kListCap * sizeof(int)) + 256 +
           pad256(part_floats(f.M, f.total, f.stages, cap, kNRows) * sizeof(float));
}

int launch_even_forward(const float* x, const float* w, const Shape& s, float* y, float p, int cap, Bump* bump, int* status,
                        const int** dense, cudaStream_t st) {
    switch (static_cast<int>(p)) {
        case 2: return even_forward_2(x, w, s, y, cap, bump, status, dense, st);
        case 4: return even_forward_4(x, w, s, y, cap, bump, status, dense, st);
        case 6: return even_forward_6(x, w, s, y, cap, bump, status, dense, st);
        default: return even_forward_8(x, w, s, y, cap, bump, status, dense, st);
    }
}

size_t even_backward_bytes(const Shape& s, float p, bool gx, bool gw, int cap) {
    const int ct = channels_of(static_cast<int>(p) - 1);
    const int splits = row_splits(s);
    const size_t rows = static_cast<size_t>(s.G) * s.M;
    int x_ranges, w_ranges, in_each;
    channel_ranges(s.B, s.HW == 1, &x_ranges, &in_each);
    channel_ranges(s.COg, true, &w_ranges, &in_each);
    return 2 * pad256(rows * 4) + 2 * pad256(4 * static_cast<size_t>(s.CO)) + pad256(4 * 4 * static_cast<size_t>(s.G) * (s.CIg + 128)) +
           pad256(channel_words(s) * sizeof(unsigned)) + 2 * pad256(static_cast<size_t>(splits) * s.CO * 4) +
           pad256(static_cast<size_t>(splits) * s.CO * sizeof(double)) + pad256(x_ranges * static_cast<size_t>(s.CI) * sizeof(double2)) +
           pad256(w_ranges * static_cast<size_t>(s.CI) * sizeof(double2)) + pad256(s.G * static_cast<size_t>(div_up(s.CIg, 32)) * sizeof(double)) +
           (gx ? pad256(plan_gradient(s, false, ct).image_bytes) : 0) + (gw ? pad256(plan_gradient(s, true, ct).image_bytes) : 0) +
           pad256(gradient_part_floats(s, gx, gw, ct, cap) * sizeof(float));
}

int launch_even_backward(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx, float* gw,
                         float p, bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond,
                         cudaStream_t st) {
    switch (static_cast<int>(p)) {
        case 2: return even_backward_2(coef, pitch, x, w, y, s, gx, gw, accumulate_gw, range, cap, bump, status, cond, st);
        case 4: return even_backward_4(coef, pitch, x, w, y, s, gx, gw, accumulate_gw, range, cap, bump, status, cond, st);
        case 6: return even_backward_6(coef, pitch, x, w, y, s, gx, gw, accumulate_gw, range, cap, bump, status, cond, st);
        default: return even_backward_8(coef, pitch, x, w, y, s, gx, gw, accumulate_gw, range, cap, bump, status, cond, st);
    }
}

}  // namespace ldn
