// Forward pass of general exponents from the channels whose terms count (ldn_power_lists.cu).
#pragma once
#include "ldn_common.cuh"

namespace ldn {

// Fully connected, ungrouped problems for which it can win (whether it does, the data decides on the device).
bool power_lists_apply(const Shape& s, float p);
size_t power_lists_bytes(const Shape& s);

struct PowerLists {
    const float *norm_rows, *norm_cols;  // largest |x| of every row, largest |w| of every row
    const int* dense;                    // not 0 when the launches have run: the caller's dense kernels, gated by it, have to
};
// y = (sum_c |x - w|^p)^(1/p), 10 < p <= 100.
int launch_power_lists(const float* x, const float* w, const Shape& s, float* y, float p, int sm_count, Bump* bump, PowerLists* out,
                       cudaStream_t st);

}  // namespace ldn
