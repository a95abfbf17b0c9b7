// The products of routed experts on the tensor cores, all experts in one launch:
//     out[p, n] = A[p, :] . W[e(p)][n, :]      for the rows p of every expert e, first[e] <= p < first[e + 1]
// bfloat16 operands, 32-bit sums.  GATED: W[e] is [2 N, K], gate rows, then up rows, and out[p, n] = act(gate, up) of
// the 32-bit sums; else W[e] is [N, K] and out[p, n] is the sum or an activation of it.
//
// How many rows an expert has is known on the device only.  Every CTA reads first[], cuts each expert's rows into equal
// tiles of at most BN and walks the items (expert, weight tile, row tile) round robin, the row tiles of a weight tile side by
// side (they share it in L2).  The weight is the M side of the instruction.  Operands come by TMA into a ring that
// runs on across items; accumulators are two deep, so an item's sums are written while the next one's are formed.
//
// * SUB 1: 128 weight rows (64 gate and 64 up rows where GATED) to an item, 16, 32 or 64 rows of A, two CTAs to an SM:
//   decoding, where the time goes into streaming the weights of the chosen experts once.  Twice the rows that an
//   expert has on average, so that a second tile (which reads the weight again, from L2) is rare.
// * SUB 2: 256 weight rows and 128 rows of A: prompts, where 256 x 128 of arithmetic per 48 KB of operands is what an SM
//   can be fed.  The rows are as wide as the tile needs (a multiple of 16), so small experts waste little.
//
// Measured (one B200, 16 experts of 2048 x 1024 with gates, first and second product, us; bytes of the weights alone 20 and 10):
// 32 pairs 29 and 17, 128 pairs 35 and 21, 1024 37 and 21, 8192 80 (860 TFLOP/s) and 46; 32 experts of 4096 x 2048 without gates
// 8192 pairs 185 (743 TFLOP/s) and 168.  What was before: on the CUDA cores 41 and 21, 76 and 39; prompts a launch per expert and product
// behind a copy of first[] to the host, 37 and 29 us per expert of the latter.
//
// A shared expert that all rows use (rows, sizes, matrix and result of its own) may ride along: its items follow the routed
// ones, so it costs its bytes and no launch (4 rows, 10 of 16 experts of 2048 x 1024 with gates and a shared one of the same size: 21.4 and
// 12.8 us; 20.1 and 12.5 without it, whose own two products took 4.4 and 3.9).
//
// A row's sums run over K in one order whatever tile it lies in: its result does not depend on the other rows.
//
// Every barrier wait has a time limit; on expiry the status word is raised, loads in flight are let land, tensor memory is
// freed and the CTA returns.
#include "common.cuh"
#include "gated_activation.cuh"
#include "tcgen05.cuh"
#include <float.h>

#define MT_K 64                        // elements of K per stage: one 128-byte swizzled row
#define MT_BOX (64 * MT_K * 2)         // bytes of a box of 64 weight rows
#define MT_MAX_EXPERTS 256
#define MT_THREADS 192

static __device__ int g_moe_tc_status;

template <int BN, int SUB> struct MoeTile {
    static constexpr int kABox = BN < 32 ? BN : 32;                      // rows of A per load
    static constexpr int kWBytes = SUB * 2 * MT_BOX;
    static constexpr int kABytes = BN * MT_K * 2;
    static constexpr int kStageBytes = kWBytes + kABytes;
    static constexpr int kExchange = SUB == 1 ? 16 * 64 * 4 : 0;         // up sums on their way to the gate's lanes
    static constexpr int kTail = 512 + (2 * MT_MAX_EXPERTS + 2) * 4 + 16 + kExchange;
    static constexpr int kStages = ((SUB == 1 ? 232448 / 2 - 1024 : 232448) - 1024 - kTail) / kStageBytes;
    static constexpr int kSmem = 1024 + kStages * kStageBytes + kTail;
    static constexpr int kTmem = 2 * SUB * BN < 32 ? 32 : 2 * SUB * BN;
    static_assert(kStages >= 3 && kStages <= 8 && kTmem <= 512, "the ring or the accumulators do not fit");
};

struct MoeTcArgs {
    const int* first;          // [experts + 1]
    const float* pair_scale;   // or nullptr: the pair's input row counts that many times, pair_scale[perm[p]]
    const int* perm;
    int experts, NT, N, K, act;
    long long ldc;
    float limit, alpha, shift;
    int x_rows, x_NT, x_N, x_K;        // the shared expert (x_rows 0: none); its results are x_N wide
};

struct MoeItem {
    int e, j, p0, rows, width;  // expert (-1: the shared one), weight tile, first row, rows, rows rounded up to 16
};

// item `it` of the walk; first[] and the experts' row tiles before each (cum) lie in shared memory
template <int BN> __device__ __forceinline__ MoeItem moe_item(const int* first, const int* cum, const MoeTcArgs& g, int it) {
    const int experts = g.experts, NT = g.NT;
    MoeItem w;
    if (it >= cum[experts] * NT) {
        const int x = it - cum[experts] * NT, tiles = (g.x_rows + BN - 1) / BN;
        w.e = -1;
        w.j = x / tiles;
        w.width = ((g.x_rows + tiles - 1) / tiles + 15) & ~15;
        w.p0 = (x - w.j * tiles) * w.width;
        w.rows = min(w.width, g.x_rows - w.p0);
        return w;
    }
    int lo = 0, hi = experts;                    // cum[lo] NT <= it < cum[hi] NT
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (cum[mid] * NT <= it) lo = mid;
        else hi = mid;
    }
    w.e = lo;
    const int tiles = cum[lo + 1] - cum[lo], local = it - cum[lo] * NT;
    w.j = local / tiles;
    const int all = first[lo + 1] - first[lo];
    w.width = ((all + tiles - 1) / tiles + 15) & ~15;
    const int r0 = (local - w.j * tiles) * w.width;
    w.p0 = first[lo] + r0;
    w.rows = min(w.width, all - r0);
    return w;
}

// whether `mine` holds for all threads of the four epilogue warps (barrier 1)
__device__ __forceinline__ bool mt_all(bool mine) {
    uint32_t all;
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"((uint32_t)mine)
        : "memory");
    return all != 0;
}

// x / (1 + exp(-z)): an approximate quotient and one Newton step for its remainder (Markstein, IBM J. Res. Dev. 34, 1990), with divisors
// beyond the approximate reciprocal's range scaled down.  The error is that of the general division (2.9 units of 2^-24 at most over
// -86 .. 40), which the epilogue waits for: 16 experts of 2048 x 1024 with gates under silu, 1024 and 8192 pairs, 29.9 and 81 us here, 33.5 and
// 84 with the general division, 29.0 and 78 with the approximate quotient alone (3.5 units; zero for divisors from 2^126 on).
__device__ __forceinline__ float mt_sigmoid_times(float x, float z) {
    const float scale = z < -80.f ? 0x1p-40f : 1.0f;
    const float d = (1.0f + expf(-z)) * scale, r = __fdividef(1.0f, d);
    x *= scale;
    const float q = x * r;
    return d <= FLT_MAX && fabsf(q) <= FLT_MAX ? fmaf(fmaf(-q, d, x), r, q) : q;            // (what is infinite has no remainder)
}

// Sixteen finished sums under their activation.  The switch stands outside the loops: with all activations in the body of
// an unrolled loop the code of an item ran to hundreds of KB and the epilogue waited for instructions (8192 rows x 2048 x
// 1024: 127 us).  GATED: x = act(x, y); else x (and y, a second set of sums) under it by themselves.
template <bool GATED, bool TWO>
__device__ __forceinline__ void mt_activate(float (&x)[16], float (&y)[16], const MoeTcArgs& g) {
    if (g.act < 0) return;
#define EACH(EXPR_X, EXPR_Y)                                      \
    _Pragma("unroll") for (int i = 0; i < 16; ++i) {              \
        x[i] = EXPR_X;                                            \
        if (TWO && !GATED) y[i] = EXPR_Y;                         \
    }
    auto silu = [](float v) { return mt_sigmoid_times(v, v); };
    if (g.act == ACT_RELU2) {
        EACH((fmaxf(x[i], 0.f) * fmaxf(x[i], 0.f) * (GATED ? y[i] : 1.0f)), (fmaxf(y[i], 0.f) * fmaxf(y[i], 0.f)))
    } else if (g.act == ACT_RELU) {
        EACH((fmaxf(x[i], 0.f) * (GATED ? y[i] : 1.0f)), (fmaxf(y[i], 0.f)))
    } else if (g.act == ACT_SILU) {
        EACH((silu(x[i]) * (GATED ? y[i] : 1.0f)), (silu(y[i])))
    } else if (GATED && g.act == ACT_CLAMPED) {
        const float limit = g.limit, alpha = g.alpha, shift = g.shift;
        EACH((mt_sigmoid_times(fminf(x[i], limit), alpha * fminf(x[i], limit)) *
              (fminf(fmaxf(y[i], -limit), limit) + shift)), y[i])
    } else {
        _Pragma("unroll 1") for (int i = 0; i < 16; ++i) {
            // (selected by a chain, so that the arrays stay in registers)
            float a = 0.f, b = 0.f;
            _Pragma("unroll") for (int k = 0; k < 16; ++k) if (k == i) { a = x[k]; b = y[k]; }
            const float fa = gated_activation(a, GATED ? b : 1.0f, g.act, g.limit, g.alpha, g.shift);
            const float fb = TWO && !GATED ? gated_activation(b, 1.0f, g.act, g.limit, g.alpha, g.shift) : b;
            _Pragma("unroll") for (int k = 0; k < 16; ++k) if (k == i) { x[k] = fa; y[k] = fb; }
        }
    }
#undef EACH
}

// one lane's results of up to sixteen rows
template <typename TO> __device__ __forceinline__ void mt_store(TO* o, long long ld, const float (&x)[16], int rows) {
    if (rows >= 16) {
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i * ld] = ap_from_float<TO>(x[i]);
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (i < rows) o[i * ld] = ap_from_float<TO>(x[i]);
    }
}

template <int BN, int SUB, bool GATED, typename TO>
__global__ void __launch_bounds__(MT_THREADS)
moe_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
              const __grid_constant__ CUtensorMap tmap_xw, const __grid_constant__ CUtensorMap tmap_xa, TO* __restrict__ out,
              TO* __restrict__ x_out, const MoeTcArgs g) {
    using Cfg = MoeTile<BN, SUB>;
    constexpr int STAGES = Cfg::kStages;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* tail = smem + STAGES * Cfg::kStageBytes;
    uint64_t* full = (uint64_t*)tail;
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;         // [2]
    uint64_t* acc_empty = acc_full + 2;          // [2]
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    int* first = (int*)(tail + 512);
    int* cum = first + MT_MAX_EXPERTS + 1;
    float* exchange = (float*)(tail + 512 + (2 * MT_MAX_EXPERTS + 2) * 4 + 8);   // [16][64]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&acc_full[b], 1);
            tc::mbar_init(&acc_empty[b], 4);
        }
        *abort_flag = *(volatile int*)&g_moe_tc_status != 0;
        tc::fence_barrier_init();
        tc::prefetch_tensormap(&tmap_w);
        tc::prefetch_tensormap(&tmap_a);
    }
    if (warp == 1) tc::tmem_alloc(tmem_slot, Cfg::kTmem);
    ap_pdl_wait();
    if (g.experts > 0)
        for (int e = threadIdx.x; e <= g.experts; e += MT_THREADS) first[e] = g.first[e];
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) {
        // row tiles before every expert: a running sum, 32 experts at a time
        int before = 0;
        for (int e0 = 0; e0 < g.experts; e0 += 32) {
            const int e = e0 + lane;
            int n = e < g.experts ? (first[e + 1] - first[e] + BN - 1) / BN : 0, sum = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += up;
            }
            if (e < g.experts) cum[e + 1] = before + sum;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) cum[0] = 0;
    }
    __syncthreads();
    const uint32_t tmem_base = *tmem_slot;
    const int items = *abort_flag ? 0 : cum[g.experts] * g.NT + (g.x_rows + BN - 1) / BN * g.x_NT;
    if (SUB == 1) ap_pdl_trigger();

    if (warp == 0) {
        if (lane == 0) {
            int b = 0;                           // blocks asked for so far
            for (int it = blockIdx.x; it < items && !*abort_flag; it += gridDim.x) {
                const MoeItem w = moe_item<BN>(first, cum, g, it);
                const bool shared = w.e < 0;
                const int N = shared ? g.x_N : g.N, nkb = ((shared ? g.x_K : g.K) + MT_K - 1) / MT_K;
                const CUtensorMap *mw = shared ? &tmap_xw : &tmap_w, *ma = shared ? &tmap_xa : &tmap_a;
                const int w_rows = shared ? 0 : GATED ? 2 * N : N;
                int row[2 * SUB];
#pragma unroll
                for (int s = 0; s < 2 * SUB; ++s) {
                    if (GATED) row[s] = SUB == 1 ? w.j * 64 + s * N : w.j * 128 + (s >> 1) * N + (s & 1) * 64;
                    else row[s] = w.j * 128 * SUB + s * 64;
                    row[s] += (shared ? 0 : w.e) * w_rows;
                }
                const int boxes = (w.width + Cfg::kABox - 1) / Cfg::kABox;
                const uint32_t bytes = Cfg::kWBytes + boxes * Cfg::kABox * MT_K * 2;
                for (int k = 0; k < nkb; ++k, ++b) {
                    const int s = b % STAGES;
                    if (*abort_flag) break;
                    if (!tc::mbar_wait(&empty[s], ((b / STAGES) & 1) ^ 1)) {
                        *abort_flag = 1;
                        atomicCAS(&g_moe_tc_status, 0, 1);
                        break;
                    }
                    uint8_t* stage = smem + s * Cfg::kStageBytes;
                    tc::mbar_expect_tx(&full[s], bytes);
#pragma unroll
                    for (int i = 0; i < 2 * SUB; ++i) tc::tma_load_2d(stage + i * MT_BOX, mw, k * MT_K, row[i], &full[s]);
                    for (int i = 0; i < boxes; ++i)
                        tc::tma_load_2d(stage + Cfg::kWBytes + i * Cfg::kABox * MT_K * 2, ma, k * MT_K,
                                        w.p0 + i * Cfg::kABox, &full[s]);
                }
            }
            // nothing is left in flight when this CTA's shared memory passes on
            for (int i = max(0, b - STAGES); i < b; ++i) tc::mbar_wait(&full[i % STAGES], (i / STAGES) & 1, 200000000LL);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            int b = 0, n = 0;
            for (int it = blockIdx.x; it < items && !*abort_flag; it += gridDim.x, ++n) {
                const MoeItem w = moe_item<BN>(first, cum, g, it);
                const int nkb = ((w.e < 0 ? g.x_K : g.K) + MT_K - 1) / MT_K;
                const uint32_t idesc = tc::instr_desc_bf16_f32(128, w.width);
                const int buf = n & 1;
                const uint32_t acc = tmem_base + (uint32_t)(buf * SUB * BN);
                if (!tc::mbar_wait(&acc_empty[buf], ((n >> 1) & 1) ^ 1)) {
                    *abort_flag = 1;
                    atomicCAS(&g_moe_tc_status, 0, 3);
                    break;
                }
                tc::fence_after_sync();
                bool ok = true;
                for (int k = 0; k < nkb; ++k, ++b) {
                    const int s = b % STAGES;
                    if (*abort_flag || !tc::mbar_wait(&full[s], (b / STAGES) & 1)) {
                        if (!*abort_flag) {
                            *abort_flag = 1;
                            atomicCAS(&g_moe_tc_status, 0, 2);
                        }
                        ok = false;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint8_t* stage = smem + s * Cfg::kStageBytes;
                    const uint64_t ad = tc::smem_desc_k_major_sw128(stage + Cfg::kWBytes);
#pragma unroll
                    for (int i = 0; i < SUB; ++i) {
                        const uint64_t wd = tc::smem_desc_k_major_sw128(stage + i * 2 * MT_BOX);
#pragma unroll
                        for (int kk = 0; kk < MT_K / 16; ++kk)
                            tc::mma_bf16(acc + (uint32_t)(i * BN), wd + 2 * kk, ad + 2 * kk, idesc, (k > 0 || kk > 0) ? 1u : 0u);
                    }
                    tc::mma_commit(&empty[s]);
                }
                if (!ok) break;
                tc::mma_commit(&acc_full[buf]);
            }
        }
    } else {
        const int q = warp & 3, row = q * 32 + lane;
        int n = 0;
        for (int it = blockIdx.x; it < items; it += gridDim.x, ++n) {
            const MoeItem w = moe_item<BN>(first, cum, g, it);
            const int buf = n & 1;
            const bool have = !*abort_flag && tc::mbar_wait(&acc_full[buf], (n >> 1) & 1);
            if (!have && !*abort_flag) {
                *abort_flag = 1;
                atomicCAS(&g_moe_tc_status, 0, 3);
            }
            if (!mt_all(have)) break;                                 // all four warps agree, as they meet at barriers below
            tc::fence_after_sync();
            const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * SUB * BN);
            const int N = w.e < 0 ? g.x_N : g.N;
            const long long ldc = w.e < 0 ? g.x_N : g.ldc;
            TO* to = w.e < 0 ? x_out : out;
            const bool scaled = g.pair_scale != nullptr && w.e >= 0;
#pragma unroll 1
            for (int c = 0; c < w.rows; c += 16) {
                float scale = 1.0f;                                  // of row c + lane % 16
                if (scaled && c + (lane & 15) < w.rows) scale = g.pair_scale[g.perm[w.p0 + c + (lane & 15)]];
                uint32_t v[16], u[16];
                tc::tmem_ld_x16(acc + (uint32_t)c, v);
                if (SUB == 2) tc::tmem_ld_x16(acc + (uint32_t)(BN + c), u);
                tc::tmem_ld_wait();
                if constexpr (SUB == 1 && GATED) {
                    // lanes 0..63 hold gate rows, lanes 64..127 up rows
                    if (row >= 64) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) exchange[i * 64 + row - 64] = __uint_as_float(v[i]);
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (row < 64) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) u[i] = __float_as_uint(exchange[i * 64 + row]);
                    }
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                }
                float x[16], y[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    x[i] = __uint_as_float(v[i]);
                    y[i] = SUB == 2 || GATED ? __uint_as_float(u[i]) : 1.0f;
                }
                if (scaled) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float sc = __shfl_sync(0xffffffffu, scale, i);
                        x[i] *= sc;
                        y[i] *= sc;
                    }
                }
                mt_activate<GATED, SUB == 2>(x, y, g);
                const int left = w.rows - c;
                if constexpr (GATED) {
                    const int n0 = SUB == 1 ? w.j * 64 + row : w.j * 128 + row;
                    if ((SUB == 2 || row < 64) && n0 < N) mt_store(to + (size_t)(w.p0 + c) * ldc + n0, ldc, x, left);
                } else {
                    const int n0 = w.j * 128 * SUB + row;
                    TO* o = to + (size_t)(w.p0 + c) * ldc + n0;
                    if (n0 < N) mt_store(o, ldc, x, left);
                    if (SUB == 2 && n0 + 128 < N) mt_store(o + 128, ldc, y, left);
                }
            }
            tc::fence_before_sync();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncwarp();
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 1) tc::tmem_dealloc(tmem_base, Cfg::kTmem);
}

// ---- host side ---------------------------------------------------------------------------
typedef CUresult (*MoeEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// rows x K, contiguous, box = box_rows x 64; what lies outside reads as zero
static bool moe_map(CUtensorMap* map, const void* base, long long rows, long long K, int box_rows) {
    static MoeEncodeFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return false;
        fn = (MoeEncodeFn)p;
    }
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    cuuint32_t box[2] = {MT_K, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, int SUB, bool GATED, typename TO>
static int moe_launch(const void* a, const void* w, void* out, const MoeTcArgs& args, int pairs, const void* x_a,
                      const void* x_w, void* x_out, cudaStream_t stream) {
    using Cfg = MoeTile<BN, SUB>;
    CUtensorMap tw, ta, txw, txa;
    AP_REQUIRE(args.experts == 0 || (moe_map(&tw, w, (long long)args.experts * (GATED ? 2 : 1) * args.N, args.K, 64) &&
                                     moe_map(&ta, a, pairs, args.K, Cfg::kABox)),
               "moe_tc: cannot encode the tensor maps");
    AP_REQUIRE(args.x_rows == 0 || (moe_map(&txw, x_w, (long long)(GATED ? 2 : 1) * args.x_N, args.x_K, 64) &&
                                    moe_map(&txa, x_a, args.x_rows, args.x_K, Cfg::kABox)),
               "moe_tc: cannot encode the shared expert's tensor maps");
    // what is not there is not loaded from
    if (args.experts == 0) { tw = txw; ta = txa; }
    if (args.x_rows == 0) { txw = tw; txa = ta; }
    auto kern = moe_tc_kernel<BN, SUB, GATED, TO>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
    AP_REQUIRE(e == cudaSuccess, "moe_tc: cannot reserve %d bytes of shared memory: %s", Cfg::kSmem, cudaGetErrorString(e));
    MoeTcArgs g = args;
    const int cols = (GATED ? 64 : 128) * SUB;                // results per weight tile
    g.NT = (g.N + cols - 1) / cols;
    g.x_NT = (g.x_N + cols - 1) / cols;
    const long long most = (long long)((pairs < g.experts ? pairs : g.experts) + pairs / BN) * g.NT +
                           (long long)((g.x_rows + BN - 1) / BN) * g.x_NT;
    AP_REQUIRE(most < 0x7fffffffLL, "moe_tc: too many tiles");
    const long long room = SUB == 1 ? 2 * 148 : 148;
    AP_CHECK_PDL_LAUNCH("moe_tc", ap_launch_pdl(kern, dim3((unsigned)(most < room ? most : room)), dim3(MT_THREADS), Cfg::kSmem,
                                                stream, tw, ta, txw, txa, (TO*)out, (TO*)x_out, g));
    return AP_OK;
}

// Whether a step's experts run here: operands that TMA can address, and work enough.  The kernel on the CUDA cores gives 16
// columns to a CTA, so a few pairs of small experts have more CTAs there; it slows down with the multiply-adds.  Measured,
// both products and the gathering of the rows against both products there, us (N rows of the first matrix, K, pairs):
//   2048 x 1024:  16 pairs 34 against 31,  32 36 against 35,  64 38 against 49
//   2048 x 2048:   8 pairs 41 against 41,  12 46 against 47,  16 50 against 59,  32 59 against 74,  128 69 against 127
//   1024 x 2048:  16 pairs 44 against 43,  32 51 against 55
//   2048 x 4096:   4 pairs 61 against 64,   8 83 against 100, 128 214 against 354
// so it is from about 50 million multiply-adds of the first product on.
AP_EXPORT int ap_moe_tc_takes(const void* a, const void* w, int pairs, int E, int N, int K) {
    return pairs > 0 && E > 0 && E <= MT_MAX_EXPERTS && N > 0 && K > 0 && K % 8 == 0 &&
           (((uintptr_t)a | (uintptr_t)w) & 15) == 0 && (long long)pairs * N * K >= (48ll << 20) &&
           (long long)E * N < 0x7fffffffLL;
}

// a: [pairs, K] in grouped order; w: [E, 2 N, K] (gated) or [E, N, K]; out: [pairs, N]; first: [E + 1]; act: -1 for none.
// x_rows > 0: the shared expert, x_a [x_rows, x_K], x_w [2 x_N or x_N, x_K], x_out [x_rows, x_N], the same activation, unscaled
AP_EXPORT int ap_moe_tc(const void* a, const void* w, void* out, int out_dtype, const int* first, int pairs, int E, int N,
                        int K, int gated, int act, float limit, float alpha, float shift, const float* pair_scale,
                        const int* perm, const void* x_a, const void* x_w, void* x_out, int x_rows, int x_N, int x_K,
                        cudaStream_t stream) {
    AP_REQUIRE(x_rows == 0 || (x_rows > 0 && x_a && x_w && x_out && x_N > 0 && x_K > 0 && x_K % 8 == 0 &&
                               (((uintptr_t)x_a | (uintptr_t)x_w) & 15) == 0),
               "moe_tc: bad shared expert of %d rows, %d x %d", x_rows, x_N, x_K);
    AP_REQUIRE(pairs >= 0 && E > 0 && E <= MT_MAX_EXPERTS && N > 0 && K > 0 && K % 8 == 0, "moe_tc: bad sizes pairs=%d experts=%d N=%d K=%d",
               pairs, E, N, K);
    AP_REQUIRE(act >= (gated ? 0 : -1) && act <= ACT_RELU2 && (gated || act != ACT_CLAMPED), "moe_tc: activation %d", act);
    AP_REQUIRE((((uintptr_t)a | (uintptr_t)w) & 15) == 0, "moe_tc: operands must be 16-byte aligned");
    AP_REQUIRE(pair_scale == nullptr || perm != nullptr, "moe_tc: scales go by the permutation");
    AP_REQUIRE((long long)E * (gated ? 2 : 1) * N < 0x7fffffffLL, "moe_tc: too many weight rows");
    if (pairs == 0 && x_rows == 0) return AP_OK;
    if (pairs == 0) E = 0;                     // the shared expert alone: first[] is not looked at
    const MoeTcArgs g{first, pair_scale, perm, E, 0, N, K, act, (long long)N, limit, alpha, shift, x_rows, 0, x_N, x_K};
    const int mean = E > 0 ? (pairs + E - 1) / E : x_rows;
#define LAUNCH(BN, SUB)                                                                                                \
    do {                                                                                                               \
        if (gated && out_dtype == AP_BF16) return moe_launch<BN, SUB, true, bf16>(a, w, out, g, pairs, x_a, x_w, x_out, stream);        \
        if (!gated && out_dtype == AP_BF16) return moe_launch<BN, SUB, false, bf16>(a, w, out, g, pairs, x_a, x_w, x_out, stream);      \
        if (!gated && out_dtype == AP_F32) return moe_launch<BN, SUB, false, float>(a, w, out, g, pairs, x_a, x_w, x_out, stream);      \
        AP_REQUIRE(false, "moe_tc: unsupported out dtype %d", out_dtype);                                              \
    } while (0)
    // Tiles of about twice the average, so that a second tile of an expert is rare; 256 weight rows by 128 where a weight tile's
    // bytes are no longer the cost.  Both products, us, tiles of 16, 32, 64 and 2 x 128 rows, pairs dealt at random.  16 experts of
    // 2048 x 1024 with gates: 8 pairs to an expert 41, 41, 41, 43; 16 54, 42, 42, 44; 32 62, 52, 44, 46; 48 76, 49, 46, 47; 64 77, 65, 58, 49; 256
    // 262, 148, 99, 102.  32 of 4096 x 2048 without: 8 176, 176, 176, 182; 16 181, 180, 179, 184; 32 240, 195, 188, 198; 49 312, 215, 186, 194; 64 360, 239,
    // 208, 206; 256 1248, 705, 465, 411.
    if (2 * mean <= 16) LAUNCH(16, 1);
    if (2 * mean <= 32) LAUNCH(32, 1);
    if (mean <= 48) LAUNCH(64, 1);
    LAUNCH(128, 2);
#undef LAUNCH
}

// 0 when every product here so far ran to its end; else the wait that expired (1 a free stage, 2 operands, 3 accumulator)
AP_EXPORT int ap_moe_tc_status(void) {
    int v = -1;
    if (cudaMemcpyFromSymbol(&v, g_moe_tc_status, sizeof(int)) != cudaSuccess) return -1;
    return v;
}
