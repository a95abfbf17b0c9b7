// Embedding with an additive sinusoidal position vector and an RMS norm, in one pass:
//
//   v[2i]   = table[token][2i]   * scale + sin(pos * inv_freq[i])
//   v[2i+1] = table[token][2i+1] * scale + cos(pos * inv_freq[i])
//   x = v / sqrt(mean(v^2) + eps) * w          (norm only when w is given)
//
// into the 32-bit residual stream.  Angles are 32-bit products of the position and a
// frequency the host computed in 64-bit and rounded once; sincosf is the accurate routine.
// One block per row, the row kept in shared memory between the two passes.
#include "common.cuh"

#define EMBED_THREADS 256

// The sum under the norm has one order for every number of rows, so that a row has the same bits in any step: it is formed as by
// 256 threads, a pair of entries (an entry, where there are no positions) after another to each.  A CTA of 1024 leaves it to its
// first 256, which take the row from shared memory.
template <typename TW, typename TN>
__global__ void __launch_bounds__(1024)
embed_sinusoid_norm_kernel(const int* __restrict__ tokens, const int* __restrict__ positions,
                           const TW* __restrict__ table, const float* __restrict__ inv_freq,
                           const TN* __restrict__ norm_w, float eps, float scale, float* __restrict__ x,
                           int H, int V) {
    extern __shared__ __align__(16) float row_buf[];
    __shared__ float red[32];
    const int t = blockIdx.x;
    int tok = tokens[t];
    tok = tok < 0 ? 0 : (tok >= V ? V - 1 : tok);
    const float pos = (float)positions[t];
    const TW* src = table + (size_t)tok * H;
    float ss = 0.f;
    if (inv_freq != nullptr) {
        // a sine and a cosine of one angle to a thread (a step of few rows is a chain of these)
#pragma unroll 2
        for (int p = threadIdx.x; p < H / 2; p += blockDim.x) {
            float sn, cs;
            sincosf(pos * inv_freq[p], &sn, &cs);
            const float v0 = ap_to_float(src[2 * p]) * scale + sn, v1 = ap_to_float(src[2 * p + 1]) * scale + cs;
            row_buf[2 * p] = v0;
            row_buf[2 * p + 1] = v1;
            ss = fmaf(v1, v1, fmaf(v0, v0, ss));
        }
    } else {
        for (int i = threadIdx.x; i < H; i += blockDim.x) {
            const float v = ap_to_float(src[i]) * scale;
            row_buf[i] = v;
            ss = fmaf(v, v, ss);
        }
    }
    if (blockDim.x > EMBED_THREADS && norm_w != nullptr) {
        __syncthreads();
        ss = 0.f;
        if (threadIdx.x < EMBED_THREADS) {
            if (inv_freq != nullptr) {
#pragma unroll 4
                for (int p = threadIdx.x; p < H / 2; p += EMBED_THREADS) {
                    const float2 v = *reinterpret_cast<const float2*>(row_buf + 2 * p);
                    ss = fmaf(v.y, v.y, fmaf(v.x, v.x, ss));
                }
            } else {
#pragma unroll 4
                for (int i = threadIdx.x; i < H; i += EMBED_THREADS) ss = fmaf(row_buf[i], row_buf[i], ss);
            }
        }
    }
    float inv = 1.f;
    if (norm_w != nullptr) {
        ss = ap_block_sum(ss, red);
        inv = 1.0f / sqrtf(ss / (float)H + eps);
    } else {
        __syncthreads();
    }
    float* dst = x + (size_t)t * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x)
        dst[i] = norm_w != nullptr ? row_buf[i] * inv * ap_to_float(norm_w[i]) : row_buf[i];
}

// inv_freq: [H/2] 32-bit or null (no position vector); norm_w: [H] in norm_dtype or null (no norm).
AP_EXPORT int ap_embed_sinusoid_norm(const int* tokens, const int* positions, const void* table, int table_dtype,
                                     const float* inv_freq, const void* norm_w, int norm_dtype, float eps, float scale,
                                     float* x, int T, int H, int V, cudaStream_t stream) {
    AP_REQUIRE(T >= 0 && H > 0 && V > 0, "embed_sinusoid_norm: bad sizes T=%d H=%d V=%d", T, H, V);
    AP_REQUIRE(inv_freq == nullptr || H % 2 == 0, "embed_sinusoid_norm: sine and cosine alternate, the width %d is odd", H);
    AP_REQUIRE((size_t)H * 4 <= 200 * 1024, "embed_sinusoid_norm: width %d does not fit the row buffer", H);
    if (T == 0) return AP_OK;
    const size_t smem = (size_t)H * sizeof(float);
    // A CTA of 1024, with a pair of entries to a thread, for up to a row to an SM; beyond, such CTAs wait for one another.  With 1024
    // threads and with 256, us: 1024 entries, 149 rows 3.5 and 3.5, 300 rows 4.9 and 3.7; 2048 entries, 149 rows 4.1 and 5.1, 300 rows
    // 5.7 and 5.2, 2048 rows 21 and 11; 4096 entries, 149 rows 5.0 and 8.1, 512 rows 9.0 and 8.5.  (8 rows of 2048 3.5; with two angles
    // to a pair 5.1.)
    const int threads = T <= 148 && H >= 1024 ? 1024 : EMBED_THREADS;
    // The first kernel of a step is launched in plain stream order (see ap_embed_gather).
#define LAUNCH(TW, TN)                                                                                       \
    do {                                                                                                     \
        auto kern = embed_sinusoid_norm_kernel<TW, TN>;                                                      \
        if (smem > 48 * 1024) {                                                                              \
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
            AP_REQUIRE(e == cudaSuccess, "embed_sinusoid_norm: cannot reserve %zu bytes of shared memory", smem); \
        }                                                                                                    \
        kern<<<T, threads, smem, stream>>>(tokens, positions, (const TW*)table, inv_freq, (const TN*)norm_w, eps, \
                                       scale, x, H, V);                                                      \
    } while (0)
    if (table_dtype == AP_F32 && norm_dtype == AP_F32) LAUNCH(float, float);
    else if (table_dtype == AP_BF16 && norm_dtype == AP_BF16) LAUNCH(bf16, bf16);
    else if (table_dtype == AP_BF16 && norm_dtype == AP_F32) LAUNCH(bf16, float);
    else if (table_dtype == AP_F32 && norm_dtype == AP_BF16) LAUNCH(float, bf16);
    else AP_REQUIRE(false, "embed_sinusoid_norm: unknown dtypes table=%d norm=%d", table_dtype, norm_dtype);
#undef LAUNCH
    AP_CHECK_LAUNCH("embed_sinusoid_norm");
    return AP_OK;
}
