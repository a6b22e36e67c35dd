// Matrix-product form of p = 4.
#include "ldn_even_impl.cuh"

namespace ldn {

int even_forward_4(const float* x, const float* w, const Shape& s, float* y, int cap, Bump* bump, int* status, const int** dense,
                   cudaStream_t st) {
    return forward_power<4>(x, w, s, y, cap, bump, status, dense, st);
}
int even_backward_4(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx,
                    float* gw, bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond,
                    cudaStream_t st) {
    return backward_power<4>(coef, pitch, x, w, y, s, gx, gw, accumulate_gw, range, cap, bump, status, cond, st);
}

}  // namespace ldn
