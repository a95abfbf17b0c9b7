// Causal grouped-query attention over paged keys and values, for one head size
// fixed at compile time (-DAP_HEAD_DIM=...).  One launch serves a whole step: rows
// of prompt portions and single decode rows alike, each row with its own sequence,
// position and block table.
//
//   q, out : [T, nh, HD]
//   cache  : one layer, [page][2][nkv][P][HD]   (keys then values of a page)
//   block_table : [nseq, max_blocks] page ids, < 0 where a page was given back
//   row r attends to keys at positions <= positions[r] of sequence token_seq[r]
//   (and > positions[r] - window when window > 0).
//
// Scores, softmax and the weighted sum are 32-bit.  This file holds the general
// kernel that also is the true 32-bit path.
//
// Reference counterparts (cuda/src/kernels.cu): attention_qtile_kernel :1801 and
// attention_split_gqa_kernel :1874 with the online softmax of attn_tile_step
// :1460-1552; the causal rule :1583-1585.  The reference packs pages into a
// contiguous buffer first (crates/allpaca-core/src/kv_tier.rs:1317-1417); here the
// kernel reads the block table itself.
#include "common.cuh"
#include <float.h>

#ifndef AP_HEAD_DIM
#error "compile with -DAP_HEAD_DIM=<head size>"
#endif

#define HD AP_HEAD_DIM
#define ATT_THREADS 128
#define ATT_CHUNK 128

AP_EXPORT int ap_attention_head_dim(void) { return HD; }

// A CTA takes one row and one head, 128 keys at a time.  Latency bounds it (a decode step's keys are few): a key's page is looked up
// once, by the thread that forms its score with 16-byte loads of the key; the weighted sum of the values deals a chunk's keys to
// groups of threads, 16 bytes of the head to a thread (head size 64 eight groups, 128 four, 256 two), and adds the groups up in
// their order.
// Measured (one B200, 32-bit, head size 64, 32 heads on 8, in a step): 4 rows of some 100 keys 7.9 us, 173 rows of 20 to 90 20.8;
// a thread per column walking all keys, with a page lookup each, took 18.4 and 53.
#define VEC (HD % 4 == 0 ? 4 : 1)
#define ATT_LANES ((HD / VEC) < ATT_THREADS ? (HD / VEC) : ATT_THREADS)     // threads side by side on a value row
#define ATT_GROUPS (ATT_THREADS / ATT_LANES)                                // groups of them, each with its keys
#define ATT_COLS ((HD / VEC + ATT_LANES - 1) / ATT_LANES)                   // runs of a row to a thread

template <typename T> struct AttRun { float v[VEC]; };
template <typename T> __device__ __forceinline__ AttRun<T> att_load(const T* p, bool aligned) {
    AttRun<T> r;
    if constexpr (VEC == 4 && sizeof(T) == 4) {
        if (aligned) {
            const float4 f = *reinterpret_cast<const float4*>(p);
            r.v[0] = f.x; r.v[1] = f.y; r.v[2] = f.z; r.v[3] = f.w;
            return r;
        }
    } else if constexpr (VEC == 4) {
        if (aligned) {
            const uint2 u = *reinterpret_cast<const uint2*>(p);
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
            const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
            r.v[0] = a.x; r.v[1] = a.y; r.v[2] = b.x; r.v[3] = b.y;
            return r;
        }
    }
#pragma unroll
    for (int i = 0; i < VEC; ++i) r.v[i] = ap_to_float(p[i]);
    return r;
}

template <typename T>
__global__ void __launch_bounds__(ATT_THREADS)
attention_rows_kernel(const T* __restrict__ q, T* __restrict__ out, const T* __restrict__ cache,
                      const int* __restrict__ block_table, int max_blocks,
                      const int* __restrict__ token_seq, const int* __restrict__ positions,
                      int nh, int nkv, int P, size_t page_stride, float scale, int window) {
    __shared__ float q_s[HD];
    __shared__ float p_s[ATT_CHUNK];
    __shared__ size_t at_s[ATT_CHUNK];                     // where a key of the chunk lies
    __shared__ float red[32];
    __shared__ float part_s[ATT_GROUPS > 1 ? ATT_GROUPS * HD : 1];
    const int t = blockIdx.x, h = blockIdx.y;
    const int kvh = h / (nh / nkv);
    ap_pdl_trigger();
    ap_pdl_wait();
    const int seq = token_seq[t];
    const int qpos = positions[t];
    const int* table = block_table + (size_t)seq * max_blocks;
    const T* qr = q + ((size_t)t * nh + h) * HD;
    for (int d = threadIdx.x; d < HD; d += ATT_THREADS) q_s[d] = ap_to_float(qr[d]);
    __syncthreads();

    const bool aligned = ((uintptr_t)cache % (VEC * sizeof(T))) == 0 && page_stride % VEC == 0;
    const size_t head_off = (size_t)kvh * P * HD;          // keys of this head inside a page
    const size_t v_off = (size_t)nkv * P * HD;             // from a key to its value
    const int lane = threadIdx.x % ATT_LANES, group = threadIdx.x / ATT_LANES;
    float acc[ATT_COLS][VEC];
#pragma unroll
    for (int i = 0; i < ATT_COLS; ++i)
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[i][e] = 0.f;
    float m = -FLT_MAX, l = 0.f;

    const int kfirst = (window > 0 && qpos - window + 1 > 0) ? qpos - window + 1 : 0;
    for (int c0 = kfirst; c0 <= qpos; c0 += ATT_CHUNK) {
        const int kpos = c0 + threadIdx.x;
        float s = -FLT_MAX;
        if (kpos <= qpos) {
            const int pg = kpos / P;
            const size_t at = (size_t)table[pg] * page_stride + head_off + (size_t)(kpos - pg * P) * HD;
            at_s[threadIdx.x] = at;
            float dot = 0.f;
#pragma unroll 8
            for (int d = 0; d < HD; d += VEC) {
                const AttRun<T> k = att_load<T>(cache + at + d, aligned);
#pragma unroll
                for (int e = 0; e < VEC; ++e) dot = fmaf(q_s[d + e], k.v[e], dot);
            }
            s = dot * scale;
        }
        const float cmax = ap_block_max(s, red);
        const float m_new = fmaxf(m, cmax);
        const float p = (kpos <= qpos) ? expf(s - m_new) : 0.f;
        p_s[threadIdx.x] = p;
        const float csum = ap_block_sum(p, red);   // also publishes p_s and at_s (it synchronises)
        const float alpha = expf(m - m_new);       // 0 on the first chunk (m = -FLT_MAX)
        l = l * alpha + csum;
        m = m_new;
        const int nk = min(ATT_CHUNK, qpos - c0 + 1);
#pragma unroll
        for (int i = 0; i < ATT_COLS; ++i)
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[i][e] *= alpha;
        if (group < ATT_GROUPS) {
#pragma unroll 4
            for (int j = group; j < nk; j += ATT_GROUPS) {
                const float pj = p_s[j];
                const T* vr = cache + at_s[j] + v_off;
#pragma unroll
                for (int i = 0; i < ATT_COLS; ++i) {
                    const int d = (lane + i * ATT_LANES) * VEC;
                    if (d < HD) {
                        const AttRun<T> v = att_load<T>(vr + d, aligned);
#pragma unroll
                        for (int e = 0; e < VEC; ++e) acc[i][e] = fmaf(pj, v.v[e], acc[i][e]);
                    }
                }
            }
        }
        __syncthreads();   // p_s is rewritten by the next chunk
    }
    T* o = out + ((size_t)t * nh + h) * HD;
    const float inv = 1.0f / l;
    if constexpr (ATT_GROUPS > 1) {
        if (group < ATT_GROUPS) {
#pragma unroll
            for (int i = 0; i < ATT_COLS; ++i) {
                const int d = (lane + i * ATT_LANES) * VEC;
                if (d < HD)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) part_s[group * HD + d + e] = acc[i][e];
            }
        }
        __syncthreads();
        for (int d = threadIdx.x; d < HD; d += ATT_THREADS) {
            float a = part_s[d];
#pragma unroll
            for (int g = 1; g < ATT_GROUPS; ++g) a += part_s[g * HD + d];
            o[d] = ap_from_float<T>(a * inv);
        }
    } else {
#pragma unroll
        for (int i = 0; i < ATT_COLS; ++i) {
            const int d = (lane + i * ATT_LANES) * VEC;
            if (d < HD && group < ATT_GROUPS)
#pragma unroll
                for (int e = 0; e < VEC; ++e) o[d + e] = ap_from_float<T>(acc[i][e] * inv);
        }
    }
}

AP_EXPORT int ap_attention_rows(const void* q, void* out, const void* cache, int dtype,
                                const int* block_table, int max_blocks, const int* token_seq,
                                const int* positions, int T, int nh, int nkv, int hd, int P,
                                long long page_stride, float scale, int window, cudaStream_t stream) {
    AP_REQUIRE(hd == HD, "attention: this library was compiled for head size %d, not %d", HD, hd);
    AP_REQUIRE(T >= 0 && nh > 0 && nkv > 0 && nh % nkv == 0 && P > 0 && max_blocks > 0,
               "attention: bad sizes T=%d heads=%d kv_heads=%d page=%d", T, nh, nkv, P);
    AP_REQUIRE(nh <= 65535, "attention: %d heads exceed the grid", nh);
    if (T == 0) return AP_OK;
    dim3 grid(T, nh);
#define LAUNCH(TT)                                                                                                          \
    AP_CHECK_PDL_LAUNCH("attention_rows", ap_launch_pdl(attention_rows_kernel<TT>, grid, dim3(ATT_THREADS), 0, stream, (const TT*)q, \
                                                        (TT*)out, (const TT*)cache, block_table, max_blocks, token_seq,     \
                                                        positions, nh, nkv, P, (size_t)page_stride, scale, window))
    if (dtype == AP_F32) LAUNCH(float);
    else if (dtype == AP_BF16) LAUNCH(bf16);
    else
        AP_REQUIRE(false, "attention: unknown dtype %d", dtype);
#undef LAUNCH
    return AP_OK;
}
