// Sequences that bring one row (decoding), bfloat16 pages, behind a window or none: the attention of
// attention_window_bias.cu for keys of up to 192 and values of up to 128 numbers in whole 16-byte runs.
//
// What bounds it is latency: a window of 512 keys is 128 KB per sequence and key/value head, microseconds of traffic
// for the whole GPU, so the keys go to many warps and no warp has a long chain.  A warp takes blocks of 16 keys; all
// its loads of a block's keys AND values are independent 16-byte loads straight into the registers from which
// mma.sync.m16n8k16 takes them (no shared memory on the way):
//
// * scores: the sum over a head's coordinates may run in any order that queries and keys share, so lane (g, t) of
//   key g loads coordinates 32 b + 8 t .. + 7 at once and they serve as two steps' B operand; the queries are read the same
//   way.  All query heads of a key/value head are the 16 rows of the product (16 at a time where there are more).
// * output: likewise the columns of a block of eight may be any eight, so lane (g, t) loads columns 64 c + 8 g .. + 7 of
//   the four keys it needs, and pairs of keys are put side by side by byte permutes.
//
// The probabilities keep their 32 bits: each is the sum of three bfloat16 numbers, whose products are added in 32 bits.
// Four warps to a CTA; up to eight CTAs of a cluster share a sequence's blocks, and each finishes a part of the output.
//
// Measured (one B200, inside a decode step of a 4-layer decoder, 4 query heads to a key/value head, head size 128, window
// 512; in brackets the kernel with a key per lane): 1 row of 16 heads 9.3 us (38), 8 rows 8.0 (36), 16 rows with 64 kept
// first tokens 15.8 (54), 32 rows of 32 heads and a window of 1024 19.7 (62); 4 rows of up to 1500 keys without a window 18.3 (39).
#include "common.cuh"
#include <cooperative_groups.h>
#include <float.h>
#include "window_bias.cuh"
namespace cg = cooperative_groups;

#define AWD_WARPS 4
#define AWD_HEADS 16
#define AWD_KEYS 16

__device__ __forceinline__ void awd_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t awd_word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
// x and y as three bfloat16 pairs whose sum they are (24 significant bits)
__device__ __forceinline__ void awd_split(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        p[i] = *reinterpret_cast<const uint32_t*>(&h);
        const float2 f = __bfloat1622float2(h);
        x -= f.x;
        y -= f.y;
    }
}

// KB: blocks of 32 coordinates of a key, VB: blocks of 64 columns of a value
template <int KB, int VB>
__global__ void __launch_bounds__(AWD_WARPS * 32, 2)
attention_window_decode_kernel(const bf16* __restrict__ q, bf16* __restrict__ out, const bf16* __restrict__ cache,
                               const int* __restrict__ block_table, int max_blocks, const int* __restrict__ seq_start,
                               const int* __restrict__ positions, int nh, int nkv, int D, int VD, int P,
                               size_t page_stride, float scale, float softcap, int window, const float* __restrict__ r1,
                               const float* __restrict__ r2, int RS, int voff, int bias_kind, int keep_first,
                               const float* __restrict__ gate, long long gate_ld, const float* __restrict__ sink,
                               int nslice, int settled) {
    extern __shared__ __align__(16) float part[];            // [warps][heads here][VD], then maxima and sums of weights
    ap_pdl_trigger();
    // where the caller says so, the step's metadata and, but for the newest token, its pages are older than the kernel ahead
    if (!settled) ap_pdl_wait();
    const int seq = blockIdx.x / nslice, slice = blockIdx.x % nslice, kvh = blockIdx.y;
    const int row = seq_start[seq];
    if (seq_start[seq + 1] - row != 1) {
        ap_pdl_wait();
        return;
    }
    const int rep_all = nh / nkv, z0 = blockIdx.z * AWD_HEADS;
    const int h0 = kvh * rep_all + z0, rep = min(AWD_HEADS, rep_all - z0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int qpos = positions[row];
    const int* table = block_table + (size_t)seq * max_blocks;
    const int klo = (window > 0 && qpos - window + 1 > 0) ? qpos - window + 1 : 0;
    const int kfe = keep_first < klo ? keep_first : klo;     // kept first tokens before the window
    const int blk_win = klo / AWD_KEYS, blk_kept = min((kfe + AWD_KEYS - 1) / AWD_KEYS, blk_win);
    const int blocks = blk_kept + qpos / AWD_KEYS - blk_win + 1;

    uint4 kr[2][KB], vr[4][VB];
    // block n: the offset of key `lane` of it in the cache, or -1 where no row sees it
    auto find = [&](int n) -> long long {
        const int kp = (n < blk_kept ? n : blk_win + n - blk_kept) * AWD_KEYS + lane;
        if (lane >= AWD_KEYS || n >= blocks || !((kp >= klo || kp < kfe) && kp <= qpos)) return -1;
        const int pg = kp / P;
        return (long long)((size_t)table[pg] * page_stride + ((size_t)kvh * P + (kp - pg * P)) * RS);
    };
    auto load = [&](long long mine) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const long long at = __shfl_sync(0xffffffffu, mine, 8 * j + g);
#pragma unroll
            for (int b = 0; b < KB; ++b) {
                const int d = 32 * b + 8 * t4;
                kr[j][b] = at >= 0 && d < D ? *reinterpret_cast<const uint4*>(cache + at + d) : make_uint4(0, 0, 0, 0);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const long long at = __shfl_sync(0xffffffffu, mine, 2 * t4 + (j & 1) + 8 * (j >> 1));
#pragma unroll
            for (int c = 0; c < VB; ++c) {
                const int d = 64 * c + 8 * g;
                vr[j][c] = at >= 0 && d < VD ? *reinterpret_cast<const uint4*>(cache + at + voff + d) : make_uint4(0, 0, 0, 0);
            }
        }
    };
    const int step = AWD_WARPS * nslice;
    int n = warp + AWD_WARPS * slice;
    long long mine = find(n);
    const bool ahead = n < blocks - 1;                       // the last block holds the newest token
    if (ahead) load(mine);
    ap_pdl_wait();
    if (!ahead) load(mine);
    uint4 qa[KB], qb[KB];                                    // heads g and g + 8
#pragma unroll
    for (int b = 0; b < KB; ++b) {
        const int d = 32 * b + 8 * t4;
        const bf16* src = q + ((size_t)row * nh + h0) * D + d;
        qa[b] = g < rep && d < D ? *reinterpret_cast<const uint4*>(src + (size_t)g * D) : make_uint4(0, 0, 0, 0);
        qb[b] = g + 8 < rep && d < D ? *reinterpret_cast<const uint4*>(src + (size_t)(g + 8) * D) : make_uint4(0, 0, 0, 0);
    }
    float acc[VB * 8][4], m[2] = {-FLT_MAX, -FLT_MAX}, l[2] = {0.f, 0.f}, b1[2], b2[2];
#pragma unroll
    for (int i = 0; i < VB * 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const bool here = g + 8 * i < rep;
        b1[i] = r1 && here ? r1[h0 + g + 8 * i] : 0.f;
        b2[i] = r2 && here ? r2[h0 + g + 8 * i] : 0.f;
    }
    while (n < blocks) {
        float s[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
            for (int b = 0; b < KB; ++b) {
                awd_mma(s[j], qa[b].x, qb[b].x, qa[b].y, qb[b].y, kr[j][b].x, kr[j][b].y);
                awd_mma(s[j], qa[b].z, qb[b].z, qa[b].w, qb[b].w, kr[j][b].z, kr[j][b].w);
            }
        }
        const int k0 = (n < blk_kept ? n : blk_win + n - blk_kept) * AWD_KEYS;
        const long long next = find(n + step);
        float mx[2] = {m[0], m[1]};
        unsigned seen = 0;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = e >> 1, kp = k0 + 8 * j + 2 * t4 + (e & 1);
                const bool in = (kp >= klo || kp < kfe) && kp <= qpos;
                s[j][e] = in ? awb_cap(s[j][e] * scale, softcap) - awb_bias(bias_kind, b1[i], b2[i], (float)(qpos - kp)) : -FLT_MAX;
                seen |= (unsigned)in << (4 * j + e);
                mx[i] = fmaxf(mx[i], s[j][e]);
            }
        float alpha[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
            mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
            alpha[i] = expf(m[i] - mx[i]);
            m[i] = mx[i];
            l[i] *= alpha[i];
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[j][e] = (seen >> (4 * j + e)) & 1u ? expf(s[j][e] - m[e >> 1]) : 0.f;
                l[e >> 1] += s[j][e];                        // this lane's share; the lanes of a head meet at the end
            }
        uint32_t a0[3], a1[3], a2[3], a3[3];
        awd_split(s[0][0], s[0][1], a0);
        awd_split(s[0][2], s[0][3], a1);
        awd_split(s[1][0], s[1][1], a2);
        awd_split(s[1][2], s[1][3], a3);
#pragma unroll
        for (int c = 0; c < VB; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                float (&o)[4] = acc[8 * c + i];
                o[0] *= alpha[0];
                o[1] *= alpha[0];
                o[2] *= alpha[1];
                o[3] *= alpha[1];
                const uint32_t sel = (i & 1) ? 0x7632u : 0x5410u;
                const uint32_t v0 = __byte_perm(awd_word(vr[0][c], i >> 1), awd_word(vr[1][c], i >> 1), sel);
                const uint32_t v1 = __byte_perm(awd_word(vr[2][c], i >> 1), awd_word(vr[3][c], i >> 1), sel);
#pragma unroll
                for (int t = 2; t >= 0; --t) awd_mma(o, a0[t], a1[t], a2[t], a3[t], v0, v1);
            }
        n += step;
        if (n < blocks) load(next);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    }
    // the warps' results: head x column sums, then per warp and head the maximum and the sum of weights
    float* stat = part + (size_t)AWD_WARPS * rep * VD;       // [warps][heads][2]; then the CTA's own [heads][2]
    float* own = stat + AWD_WARPS * rep * 2;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int i = g + 8 * half;
        if (i < rep) {
            float* dst = part + ((size_t)warp * rep + i) * VD;
#pragma unroll
            for (int c = 0; c < VB; ++c)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int d = 64 * c + 8 * (2 * t4 + e);
                    if (d < VD) {
                        float4 lo, hi;
                        lo.x = acc[8 * c][2 * half + e]; lo.y = acc[8 * c + 1][2 * half + e];
                        lo.z = acc[8 * c + 2][2 * half + e]; lo.w = acc[8 * c + 3][2 * half + e];
                        hi.x = acc[8 * c + 4][2 * half + e]; hi.y = acc[8 * c + 5][2 * half + e];
                        hi.z = acc[8 * c + 6][2 * half + e]; hi.w = acc[8 * c + 7][2 * half + e];
                        *reinterpret_cast<float4*>(dst + d) = lo;
                        *reinterpret_cast<float4*>(dst + d + 4) = hi;
                    }
                }
            if (t4 == 0) {
                stat[(warp * rep + i) * 2] = m[half];
                stat[(warp * rep + i) * 2 + 1] = l[half];
            }
        }
    }
    __syncthreads();
    auto finish = [&](int i, int d, float num, float den, float mm) {
        if (sink) den += expf(sink[h0 + i] - mm);
        float res = num / den;
        if (gate) res /= 1.0f + expf(-gate[(size_t)row * gate_ld + h0 + i]);
        out[((size_t)row * nh + h0 + i) * VD + d] = __float2bfloat16_rn(res);
    };
    // the warps in their order; a warp that met no key has weight exp(-FLT_MAX - maximum) = 0
    for (int e = threadIdx.x; e < rep * VD; e += AWD_WARPS * 32) {
        const int i = e / VD, d = e - i * VD;
        float mm = -FLT_MAX, num = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < AWD_WARPS; ++w) mm = fmaxf(mm, stat[(w * rep + i) * 2]);
#pragma unroll
        for (int w = 0; w < AWD_WARPS; ++w) {
            const float f = expf(stat[(w * rep + i) * 2] - mm);
            num = fmaf(part[((size_t)w * rep + i) * VD + d], f, num);
            den = fmaf(stat[(w * rep + i) * 2 + 1], f, den);
        }
        if (nslice == 1) {
            finish(i, d, num, den, mm);
        } else {
            part[e] = num;                                   // warp 0's place, which this thread alone reads
            if (d == 0) {
                own[2 * i] = mm;
                own[2 * i + 1] = den;
            }
        }
    }
    if (nslice == 1) return;
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();                                               // every CTA's results are in its shared memory
    for (int e = threadIdx.x + slice * AWD_WARPS * 32; e < rep * VD; e += AWD_WARPS * 32 * nslice) {
        const int i = e / VD, d = e - i * VD;
        float mm = -FLT_MAX, num = 0.f, den = 0.f;
        float cm[8], cn[8], cd[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            if (c < nslice) {
                const float* o = cl.map_shared_rank(own, c);
                cm[c] = o[2 * i];
                cd[c] = o[2 * i + 1];
                cn[c] = cl.map_shared_rank(part, c)[e];
                mm = fmaxf(mm, cm[c]);
            }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {                        // in the order of the slices
            if (c < nslice) {
                const float f = expf(cm[c] - mm);
                num = fmaf(cn[c], f, num);
                den = fmaf(cd[c], f, den);
            }
        }
        finish(i, d, num, den, mm);
    }
    cl.sync();                                               // nobody leaves while others still read
}

// Whether the kernel here takes the call: whole 16-byte runs everywhere
bool attention_window_decode_takes(const void* q, const void* cache, int D, int VD, long long page_stride, int RS, int voff) {
    return D % 8 == 0 && VD % 8 == 0 && D <= 192 && VD <= 128 && RS % 8 == 0 && voff % 8 == 0 && page_stride % 8 == 0 &&
           (((uintptr_t)q | (uintptr_t)cache) & 15) == 0;
}

int attention_window_decode(const void* q, void* out, const void* cache, const int* block_table, int max_blocks,
                            const int* seq_start, const int* positions, int nseq, int nh, int nkv, int D, int VD, int P,
                            long long page_stride, float scale, float softcap, int window, const float* r1, const float* r2,
                            int RS, int voff, int bias_kind, int keep_first, const float* gate, long long gate_ld,
                            const float* sink, int max_context, int settled, cudaStream_t stream) {
    const int rep = nh / nkv, nz = (rep + AWD_HEADS - 1) / AWD_HEADS;
    AP_REQUIRE(nkv <= 65535 && nz <= 65535, "attention_window_bias: %d key/value heads exceed the grid", nkv);
    // a CTA walks 64 keys at a time: shared by more CTAs while that shortens the walk and two of them fit every SM
    // (a context that is not known counts as a window's, or as 1024 keys)
    const int context = max_context > 0 ? max_context : 1024;
    const int keys = window > 0 && window < context ? window + keep_first : context;
    int nslice = 1;
    while (nslice < 8 && keys > 64 * nslice && (long long)nseq * nkv * nz * nslice < 148) nslice *= 2;
    const int here = rep < AWD_HEADS ? rep : AWD_HEADS;
    const size_t smem = ((size_t)AWD_WARPS * here * VD + (size_t)(AWD_WARPS + 1) * here * 2) * sizeof(float);
    auto kern = D <= 64 && VD <= 64 ? attention_window_decode_kernel<2, 1>
                : D <= 128          ? attention_window_decode_kernel<4, 2>
                                    : attention_window_decode_kernel<6, 2>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        AP_REQUIRE(e == cudaSuccess, "attention_window_bias: cannot reserve %zu bytes of shared memory", smem);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nseq * nslice), (unsigned)nkv, (unsigned)nz);
    cfg.blockDim = dim3(AWD_WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (nslice > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)nslice;
        attr[n].val.clusterDim.y = 1;
        attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (ap_pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    AP_CHECK_PDL_LAUNCH("attention_window_decode",
                        cudaLaunchKernelEx(&cfg, kern, (const bf16*)q, (bf16*)out, (const bf16*)cache, block_table, max_blocks,
                                           seq_start, positions, nh, nkv, D, VD, P, (size_t)page_stride, scale, softcap, window,
                                           r1, r2, RS, voff, bias_kind, keep_first, gate, gate_ld, sink, nslice, settled));
    return AP_OK;
}
