// p = inf forward of convolutions (many positions per sample) in one launch (ldn_positions.cu).
#pragma once
#include "ldn_common.cuh"

namespace ldn {

// Whether the problem runs as one launch: the value, with the index, or the interval bounds.
bool inf_positions_apply(const Shape& s, bool index, bool bounds);
// y[b][o][hw] = max_c |x - w| (at least 1e-10) and, with pos, the first channel that reaches it and the sign of its
// difference; with `upper` (x and upper are interval bounds) the bounds of the value in y and y_upper.  w: rows of whole 16-byte
// pieces.  sub / add (may be null; not with pos): (v - sub[o]) + add[o] in the store.
int launch_inf_positions(const float* x, const float* upper, Operand w, const Shape& s, float* y, float* y_upper, int* pos,
                         const float* sub, const float* add, cudaStream_t st);

}  // namespace ldn
