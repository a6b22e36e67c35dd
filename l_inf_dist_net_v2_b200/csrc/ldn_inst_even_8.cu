// Matrix-product form of p = 8.
#include "ldn_even_impl.cuh"

namespace ldn {

int even_forward_8(const float* x, const float* w, const Shape& s, float* y, int cap, Bump* bump, int* status, const int** dense,
                   cudaStream_t st) {
    return forward_power<8>(x, w, s, y, cap, bump, status, dense, st);
}
int even_backward_8(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx,
                    float* gw, bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond,
                    cudaStream_t st) {
    return backward_power<8>(coef, pitch, x, w, y, s, gx, gw, accumulate_gw, range, cap, bump, status, cond, st);
}

}  // namespace ldn
