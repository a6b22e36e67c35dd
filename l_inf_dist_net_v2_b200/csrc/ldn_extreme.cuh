// p = inf forward of large fully connected layers from the extreme channels of both operands (ldn_extreme.cu).
#pragma once
#include "ldn_common.cuh"

namespace ldn {

// What a call needs besides its operands.  Sizes in extreme_scratch_bytes().
struct ExtremeScratch {
    void* x_list;
    void* w_list;
    float* x_rest;
    float* w_rest;
    unsigned* hard;  // outputs to be searched in full
    int* words;      // kExtremeWords device words, cleared by the call; the first is the dense gate
};
constexpr int kExtremeWords = 8 + 32 * 18;

// Whether a problem of B samples, CO outputs and C channels takes this path (bound: interval bounds).
bool extreme_applies(long long B, int CO, int C, bool bound);
size_t extreme_scratch_bytes(long long B, int CO, bool bound);
// Carves the scratch out of a bump allocator; false: it does not fit.
bool extreme_take_scratch(Bump* bump, long long B, int CO, bool bound, ExtremeScratch* out);

// Values (and channel | sign, pos not null) of all outputs into y / pos, [B][CO].  bound: x = lower, xu = upper inputs
// (lower <= upper), y / yu = lower / upper bounds, pos unused.  sub / add: the eval-mode layer epilogue per output channel.
// On return *dense_gate is a device word: not 0 means that the caller's dense kernels, launched behind this with that gate,
// have to compute all outputs.
int launch_extreme(Operand x, Operand xu, Operand w, long long B, int CO, int C, bool bound, float* y, float* yu, int* pos,
                   const float* sub, const float* add, const ExtremeScratch& t, const int** dense_gate, cudaStream_t st);

// What a call's first words say once it is done: whether the dense kernels computed the outputs, and how many the lists left
// to be searched in full.
constexpr int kExtremeOutcomeWords = 3;
inline void extreme_outcome(const int (&words)[kExtremeOutcomeWords], int outcome[2]) {
    outcome[0] = words[0] != 0 ? 1 : 0;
    outcome[1] = words[2];
}

}  // namespace ldn
