// What the attention kernels with a distance bias share.
#pragma once

#define BIAS_NONE 0
#define BIAS_LOG 1
#define BIAS_LINEAR 2

__device__ __forceinline__ float awb_bias(int kind, float b1, float b2, float dist) {
    return kind == BIAS_LOG ? b1 * log1pf(b2 * dist) : (kind == BIAS_LINEAR ? b1 * dist : 0.f);
}
// the scaled score, bounded by a soft cap where there is one: cap * tanh(score / cap)
__device__ __forceinline__ float awb_cap(float score, float cap) { return cap > 0.f ? cap * tanhf(score / cap) : score; }
