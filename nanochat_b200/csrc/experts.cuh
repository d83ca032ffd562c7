// Shared pieces of the mixture-of-experts kernels (experts.cu, experts_tc.cu).
//
// Routing leaves the (token, choice) pairs sorted by expert: position i of the sorted order belongs to
// pair slot[i] = token * top + choice with weight scale[i]; expert e has positions [offsets[e], offsets[e + 1]).
#pragma once

#include "vec_io.cuh"

namespace nckv {

// The two products of all experts.  UP: act[i] = silu(s g) * (s u) with [g; u] = W_e h[token], s = scale[i] (the
// weight multiplies the expert's input, which for a product without bias is its output).  Otherwise
// y[slot[i]] = W_e act[i].
struct ExpertParams {
    const void *a;         // UP: h (rows, K); else act (R, K)
    const void *w;         // UP: (E, 2 N, K) gate rows, then up rows; else (E, N, K)
    void *out;             // UP: act (R, N); else y (R, N) by slot
    const int32_t *offsets, *slot;  // on pairs of CTAs without offsets: one expert with all R positions
    const float *scale;             // there, null: 1
    int32_t *status;
    int R, E, top, N, K;
};

constexpr int EQ_MAX_EXPERTS = 256;
long long experts_tc_waves(bool up, int R, int E, int N, int bn);  // of tiles of bn weight rows, at an even spread of the positions
bool experts_tc_wide(bool up, int R, int E, int N);                // whether experts_tc takes the wide ones
bool experts_in_pairs(bool up, int R, int E, int N, int K);  // whether that many rows take the form on pairs of CTAs
cudaError_t experts_pair(ExpertParams p, bool up, void *sorted, cudaStream_t s, int *rc);  // sorted: UP: room for (R, K)
cudaError_t experts_tc(const ExpertParams &p, bool up, cudaStream_t s, int *rc);  // tcgen05 form, many rows

}  // namespace nckv
