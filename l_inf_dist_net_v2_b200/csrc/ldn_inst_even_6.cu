// Matrix-product form of p = 6.
#include "ldn_even_impl.cuh"

namespace ldn {

int even_forward_6(const float* x, const float* w, const Shape& s, float* y, int cap, Bump* bump, int* status, const int** dense,
                   cudaStream_t st) {
    return forward_power<6>(x, w, s, y, cap, bump, status, dense, st);
}
int even_backward_6(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx,
                    float* gw, bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond,
                    cudaStream_t st) {
    return backward_power<6>(coef, pitch, x, w, y, s, gx, gw, accumulate_gw, range, cap, bump, status, cond, st);
}

}  // namespace ldn
