// Even integer exponents (p = 2, 4, 6, 8) as contractions on the tensor cores (ldn_even.cu).
#pragma once
#include "ldn_common.cuh"

namespace ldn {

inline bool even_power(float p) { return p == 2.0f || p == 4.0f || p == 6.0f || p == 8.0f; }

// Whether a problem is large enough for this path to be the faster one, forward and backward, on `cap` of the device's CTAs.
bool even_forward_applies(const Shape& s, float p, int cap, int sm_count);
bool even_backward_applies(const Shape& s, float p, bool gx, bool gw, int cap, int sm_count);

// Scratch of a forward call; launch_even_forward takes it from the bump allocator.
size_t even_forward_bytes(const Shape& s, float p, int cap);
// y = (sum_c |x - w|^p)^(1/p).  *dense (device word, set when the launches have run): not 0 if the outputs have to be computed
// by the direct kernels, which the caller launches behind it with that word as their gate.
int launch_even_forward(const float* x, const float* w, const Shape& s, float* y, float p, int cap, Bump* bump, int* status,
                        const int** dense, cudaStream_t st);

size_t even_backward_bytes(const Shape& s, float p, bool gx, bool gw, int cap);
// Gradients from the coefficients coef[g][m][pitch] = go / y^(p-1); range: the word that the coefficient kernel raises.  *cond:
// the same for data that the expansion does not suit; neither word set: gx / gw hold the result.  (cond is left alone when
// range is set.)  gx or gw may be null; gw is added to when accumulate_gw.
int launch_even_backward(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx, float* gw,
                         float p, bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond,
                         cudaStream_t st);

// the instantiations, one translation unit each (ldn_inst_even_*.cu)
int even_forward_2(const float* x, const float* w, const Shape& s, float* y, int cap, Bump* bump, int* status, const int** dense,
                   cudaStream_t st);
int even_backward_2(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx,
                    float* gw, bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond,
                    cudaStream_t st);
int even_forward_4(const float* x, const float* w, const Shape& s, float* y, int cap, Bump* bump, int* status, const int** dense,
                   cudaStream_t st);
int even_backward_4(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx,
                    float* gw, bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond,
                    cudaStream_t st);
int even_forward_6(const float* x, const float* w, const Shape& s, float* y, int cap, Bump* bump, int* status, const int** dense,
                   cudaStream_t st);
int even_backward_6(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx,
                    float* gw, bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond,
                    cudaStream_t st);
int even_forward_8(const float* x, const float* w, const Shape& s, float* y, int cap, Bump* bump, int* status, const int** dense,
                   cudaStream_t st);
int even_backward_8(const float* coef, int pitch, const float* x, const float* w, const float* y, const Shape& s, float* gx,
                    float* gw, bool accumulate_gw, const int* range, int cap, Bump* bump, int* status, const int** cond,
                    cudaStream_t st);

}  // namespace ldn
