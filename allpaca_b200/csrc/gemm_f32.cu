// C[M,N] = A[M,K] * W[N,K]^T in true 32-bit (fused multiply-adds of the CUDA cores) for rows of whole 16-byte runs.
//
// One order of sums for every number of rows, so that a row has the same bits in any batch: K is cut into SEGS runs of
// whole blocks of 32; a run is one thread's chain in ascending k from zero, and the runs are added in their order.
// Two kernels keep that order:
//
// * up to 32 rows (decoding) the time goes into reading the weight once.  A CTA takes 128 weight rows; TMA brings
//   blocks of 128 x 32 into a ring of shared memory, a thread owns four weight rows and up to eight rows of A, so that a
//   16-byte read serves 16 to 32 multiply-adds.  Where the 128-row tiles do not fill the GPU, the runs of a tile go to
//   the eight CTAs of a cluster, which add up through distributed shared memory; else a CTA walks all of K and keeps
//   the finished runs' sum beside the current one.
// * beyond, tiles of 64 to 176 rows x 96, 112 or 128 columns, always a cluster of eight per tile: up to 11 x 14 outputs to a thread (a
//   number read from shared memory serves 6.2 multiply-adds, at 8 x 8, where the reads take as long as the arithmetic, 4).
//
// Measured (one B200, weights rotating over more than L2; in brackets the 64 x 64 tiles of gemm_simt.cu, which load 4 bytes
// at a time), us:
//
//   rows    3072 x 2048    2048 x 2048    16384 x 2048    2048 x 8192    128256 x 2048
//      1     7.5 (152)      6.5 (153)      31.4 (210)     18.1 (621)
//      4     9.7 (152)      8.6 (153)      39.1 (211)     25.7 (625)     189 (1168): 5.6 TB/s
//     32    20.8 (157)     19.8 (156)      83.7 (222)     69.0 (640)     549 (1261)
//    173    62.6 (151)     50.0 (148)       353 (674)      176 (591)
//    300     113            99             615            350
//    512     183 (303)      122 (208)       968 (1357)     434 (852): 40 TFLOP/s of the CUDA cores' 74
//
// The relative error against 64 bits is 2.9e-7 at K = 2048 and 5.7e-7 at 8192 (8.1e-7 and 1.6e-6 for one chain over K).
//
// Every barrier wait has a time limit; on expiry the status word is raised, loads in flight are let land, and the CTA
// walks to the barriers at the end.
#include <type_traits>

#include "tcgen05.cuh"
#include "common.cuh"

#define F32_SEGS 8
#define F32_BK 32
#define F32_BN 128
#define F32_W_BYTES (F32_BN * F32_BK * 4)
#define F32_FEW_ROWS 32
#define F32_FEW_STAGES 4
#define F32_TILE_STAGES 3

static __device__ int g_f32_status;

// 16 bytes of row `row`, columns 4 chunk .. 4 chunk + 3, of a [rows][32] block as TMA writes it with the 128-byte swizzle
__device__ __forceinline__ float4 f32_block_read(const uint8_t* block, int row, int chunk) {
    return *reinterpret_cast<const float4*>(block + row * 128 + ((chunk ^ (row & 7)) << 4));
}

struct F32Ring {
    uint64_t* full;
    uint64_t* empty;
    volatile int* abort_flag;
};

// The producer's part of the few-rows kernel: blocks [kb0, kb1) of a weight tile and of the rows' tile.  Weight blocks of the
// first round are asked for before the kernels that produce the rows have finished.
template <int STAGES>
__device__ __forceinline__ void f32_produce(const CUtensorMap* tw, const CUtensorMap* ta, uint8_t* w_ring, uint8_t* a_ring,
                                            uint32_t a_bytes, const F32Ring& r, int kb0, int kb1, int n0, int m0) {
    const int blocks = kb1 - kb0, pre = min(STAGES, blocks);
    for (int i = 0; i < pre; ++i) {
        tc::mbar_expect_tx(&r.full[i], F32_W_BYTES + a_bytes);
        tc::tma_load_2d(w_ring + i * F32_W_BYTES, tw, (kb0 + i) * F32_BK, n0, &r.full[i]);
    }
    ap_pdl_wait();
    for (int i = 0; i < pre; ++i) tc::tma_load_2d(a_ring + i * a_bytes, ta, (kb0 + i) * F32_BK, m0, &r.full[i]);
    int issued = pre;
    for (int b = pre; b < blocks; ++b) {
        const int s = b % STAGES;
        if (*r.abort_flag || !tc::mbar_wait(&r.empty[s], (uint32_t)((b / STAGES - 1) & 1))) {
            if (!*r.abort_flag) {
                *r.abort_flag = 1;
                atomicCAS(&g_f32_status, 0, 1);
            }
            break;
        }
        tc::mbar_expect_tx(&r.full[s], F32_W_BYTES + a_bytes);
        tc::tma_load_2d(w_ring + s * F32_W_BYTES, tw, (kb0 + b) * F32_BK, n0, &r.full[s]);
        tc::tma_load_2d(a_ring + s * a_bytes, ta, (kb0 + b) * F32_BK, m0, &r.full[s]);
        issued = b + 1;
    }
    // nothing is left in flight when this CTA's shared memory passes on
    for (int b = max(0, issued - STAGES); b < issued; ++b) tc::mbar_wait(&r.full[b % STAGES], (uint32_t)((b / STAGES) & 1));
}

// whether block b has landed (all lanes of the warp agree)
template <int STAGES>
__device__ __forceinline__ bool f32_landed(const F32Ring& r, int b) {
    const bool ok = !*r.abort_flag && tc::mbar_wait(&r.full[b % STAGES], (uint32_t)((b / STAGES) & 1));
    if (__all_sync(0xffffffffu, ok)) return true;
    if (!*r.abort_flag) {
        *r.abort_flag = 1;
        atomicCAS(&g_f32_status, 0, 2);
    }
    return false;
}

// Up to 32 rows.  Warp 0 loads; warp 1 + w owns rows w RPT .. w RPT + RPT - 1.  CLUSTER: this CTA's rank is its run of K.
template <int RPT, bool CLUSTER>
__global__ void __launch_bounds__(160)
gemm_f32_few_kernel(const __grid_constant__ CUtensorMap tw, const __grid_constant__ CUtensorMap ta, float* __restrict__ C,
                    int M, int N, int K, long long ldc, int a_rows) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t a_bytes = (uint32_t)a_rows * F32_BK * 4;
    uint8_t* w_ring = smem;
    uint8_t* a_ring = smem + F32_FEW_STAGES * F32_W_BYTES;
    uint64_t* bars = (uint64_t*)(a_ring + F32_FEW_STAGES * F32_FEW_ROWS * F32_BK * 4);
    F32Ring ring{bars, bars + F32_FEW_STAGES, (volatile int*)(bars + 2 * F32_FEW_STAGES)};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row_warps = blockDim.x / 32 - 1;
    const int n0 = (CLUSTER ? blockIdx.x / F32_SEGS : blockIdx.x) * F32_BN;
    const int rank = CLUSTER ? (int)tc::cluster_ctarank() : 0;
    const int nkb = (K + F32_BK - 1) / F32_BK, run = (nkb + F32_SEGS - 1) / F32_SEGS;
    const int kb0 = min(nkb, rank * run), kb1 = CLUSTER ? min(nkb, kb0 + run) : nkb;
    ap_pdl_trigger();
    if (threadIdx.x == 0) {
        for (int s = 0; s < F32_FEW_STAGES; ++s) {
            tc::mbar_init(&ring.full[s], 1);
            tc::mbar_init(&ring.empty[s], row_warps);
        }
        *ring.abort_flag = *(volatile int*)&g_f32_status != 0;
        tc::fence_barrier_init();
    }
    __syncthreads();
    float acc[RPT][4], sum[CLUSTER ? 1 : RPT][4];
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = 0.f;
            if constexpr (!CLUSTER) sum[i][j] = 0.f;
        }
    const int r0 = (warp - 1) * RPT;
    if (warp == 0) {
        if (lane == 0 && !*ring.abort_flag)
            f32_produce<F32_FEW_STAGES>(&tw, &ta, w_ring, a_ring, a_bytes, ring, kb0, kb1, n0, 0);
        ap_pdl_wait();
    } else {
        ap_pdl_wait();                   // C may still be read by an earlier kernel
        int left = run;                  // blocks until the current run of K ends
        for (int b = 0; b < kb1 - kb0; ++b) {
            if (!f32_landed<F32_FEW_STAGES>(ring, b)) break;
            const uint8_t* wb = w_ring + (b % F32_FEW_STAGES) * F32_W_BYTES;
            const uint8_t* ab = a_ring + (size_t)(b % F32_FEW_STAGES) * a_bytes;
#pragma unroll
            for (int c = 0; c < F32_BK / 4; ++c) {
                float4 w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) w[j] = f32_block_read(wb, lane + 32 * j, c);
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const float4 a = f32_block_read(ab, r0 + i, c);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
                        acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
                        acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
                        acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&ring.empty[b % F32_FEW_STAGES]);
            if constexpr (!CLUSTER) {
                if (--left == 0 || b + 1 == nkb) {
                    left = run;
#pragma unroll
                    for (int i = 0; i < RPT; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            sum[i][j] += acc[i][j];
                            acc[i][j] = 0.f;
                        }
                }
            }
        }
        if constexpr (!CLUSTER) {
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int n = n0 + lane + 32 * j;
                    if (r0 + i < M && n < N) C[(size_t)(r0 + i) * ldc + n] = sum[i][j];
                }
        }
    }
    if constexpr (CLUSTER) {
        float* part = reinterpret_cast<float*>(smem);           // [row][128]: the ring is idle now
        __syncthreads();
        if (warp > 0) {
#pragma unroll
            for (int i = 0; i < RPT; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) part[(r0 + i) * F32_BN + lane + 32 * j] = acc[i][j];
        }
        tc::cluster_sync();
        // each CTA finishes 16 of the tile's columns
        constexpr int COLS = F32_BN / F32_SEGS;
        for (int e = threadIdx.x; e < M * COLS; e += blockDim.x) {
            const int m = e / COLS, c = rank * COLS + e % COLS;
            const uint32_t at = tc::smem_addr(part + m * F32_BN + c);
            float p[F32_SEGS], v = 0.f;
#pragma unroll
            for (int s = 0; s < F32_SEGS; ++s) p[s] = tc::ld_cluster_f32(tc::map_to_rank(at, (uint32_t)s));
#pragma unroll
            for (int s = 0; s < F32_SEGS; ++s) v += p[s];
            if (n0 + c < N) C[(size_t)m * ldc + n0 + c] = v;
        }
        tc::cluster_sync();
    }
}

// Tiles of 16 RM rows x 8 CN columns.  Thread (ty, tx) owns rows ty + 16 i and columns tx + 8 j; the first thread also
// loads (a fifth warp would leave 168 registers to a thread); the CTA's rank in its cluster is its run of K.
template <int RM, int CN>
__global__ void __launch_bounds__(128, 2)
gemm_f32_tile_kernel(const __grid_constant__ CUtensorMap tw, const __grid_constant__ CUtensorMap ta, float* __restrict__ C,
                     int M, int N, int K, long long ldc) {
    constexpr int BM = 16 * RM;
    constexpr int BN = 8 * CN;
    constexpr uint32_t A_BYTES = BM * F32_BK * 4, W_BYTES = BN * F32_BK * 4;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* w_ring = smem;
    uint8_t* a_ring = smem + F32_TILE_STAGES * W_BYTES;
    uint64_t* bars = (uint64_t*)(a_ring + F32_TILE_STAGES * A_BYTES);
    F32Ring ring{bars, bars + F32_TILE_STAGES, (volatile int*)(bars + 2 * F32_TILE_STAGES)};
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (int)(blockIdx.x / F32_SEGS) * BN, m0 = (int)blockIdx.y * BM;
    const int rank = (int)tc::cluster_ctarank();
    const int nkb = (K + F32_BK - 1) / F32_BK, run = (nkb + F32_SEGS - 1) / F32_SEGS;
    const int kb0 = min(nkb, rank * run), blocks = min(nkb, kb0 + run) - kb0;
    ap_pdl_trigger();
    if (threadIdx.x == 0) {
        for (int s = 0; s < F32_TILE_STAGES; ++s) {
            tc::mbar_init(&ring.full[s], 1);
            tc::mbar_init(&ring.empty[s], 4);
        }
        *ring.abort_flag = *(volatile int*)&g_f32_status != 0;
        tc::fence_barrier_init();
    }
    __syncthreads();
    auto ask_w = [&](int b) {
        tc::mbar_expect_tx(&ring.full[b % F32_TILE_STAGES], W_BYTES + A_BYTES);
        tc::tma_load_2d(w_ring + (b % F32_TILE_STAGES) * W_BYTES, &tw, (kb0 + b) * F32_BK, n0, &ring.full[b % F32_TILE_STAGES]);
    };
    auto ask_a = [&](int b) {
        tc::tma_load_2d(a_ring + (b % F32_TILE_STAGES) * A_BYTES, &ta, (kb0 + b) * F32_BK, m0, &ring.full[b % F32_TILE_STAGES]);
    };
    const bool loads = threadIdx.x == 0 && !*ring.abort_flag;
    int asked = loads ? min(F32_TILE_STAGES, blocks) : 0;
    for (int b = 0; b < asked; ++b) ask_w(b);           // does not depend on earlier kernels
    ap_pdl_wait();
    for (int b = 0; b < asked; ++b) ask_a(b);

    const int tx = lane & 7, ty = warp * 4 + (lane >> 3);
    float acc[RM][CN];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < CN; ++j) acc[i][j] = 0.f;
    for (int b = 0; b < blocks; ++b) {
        if (!f32_landed<F32_TILE_STAGES>(ring, b)) break;
        const uint8_t* wb = w_ring + (b % F32_TILE_STAGES) * W_BYTES;
        const uint8_t* ab = a_ring + (b % F32_TILE_STAGES) * A_BYTES;
#pragma unroll 1
        for (int c = 0; c < F32_BK / 4; ++c) {
            float4 a[RM];
#pragma unroll
            for (int i = 0; i < RM; ++i) a[i] = f32_block_read(ab, ty + 16 * i, c);
#pragma unroll
            for (int j = 0; j < CN; ++j) {
                const float4 w = f32_block_read(wb, tx + 8 * j, c);
#pragma unroll
                for (int i = 0; i < RM; ++i) {
                    acc[i][j] = fmaf(a[i].x, w.x, acc[i][j]);
                    acc[i][j] = fmaf(a[i].y, w.y, acc[i][j]);
                    acc[i][j] = fmaf(a[i].z, w.z, acc[i][j]);
                    acc[i][j] = fmaf(a[i].w, w.w, acc[i][j]);
                }
            }
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&ring.empty[b % F32_TILE_STAGES]);
        if (loads && b + F32_TILE_STAGES < blocks) {
            // the other warps are at most a block behind
            if (*ring.abort_flag || !tc::mbar_wait(&ring.empty[b % F32_TILE_STAGES], (uint32_t)((b / F32_TILE_STAGES) & 1))) {
                if (!*ring.abort_flag) {
                    *ring.abort_flag = 1;
                    atomicCAS(&g_f32_status, 0, 1);
                }
            } else {
                asked = b + F32_TILE_STAGES + 1;
                ask_w(asked - 1);
                ask_a(asked - 1);
            }
        }
    }
    // nothing is left in flight when the ring takes the sums
    for (int b = max(0, asked - F32_TILE_STAGES); b < asked; ++b)
        tc::mbar_wait(&ring.full[b % F32_TILE_STAGES], (uint32_t)((b / F32_TILE_STAGES) & 1));
    float* part = reinterpret_cast<float*>(smem);                // [row][BN]: the ring is idle now
    static_assert(BM * BN * 4 <= F32_TILE_STAGES * ((int)W_BYTES + (int)A_BYTES), "the ring holds a tile of sums");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < CN; ++j) part[(ty + 16 * i) * BN + tx + 8 * j] = acc[i][j];
    tc::cluster_sync();
    // each CTA finishes BM / 8 of the tile's rows
    constexpr int ROWS = BM / F32_SEGS;
    for (int e = threadIdx.x; e < ROWS * BN; e += blockDim.x) {
        const int m = rank * ROWS + e / BN, c = e % BN;
        const uint32_t at = tc::smem_addr(part + m * BN + c);
        float p[F32_SEGS], v = 0.f;
#pragma unroll
        for (int s = 0; s < F32_SEGS; ++s) p[s] = tc::ld_cluster_f32(tc::map_to_rank(at, (uint32_t)s));
#pragma unroll
        for (int s = 0; s < F32_SEGS; ++s) v += p[s];
        if (m0 + m < M && n0 + c < N) C[(size_t)(m0 + m) * ldc + n0 + c] = v;
    }
    tc::cluster_sync();
}

// ---- host side ---------------------------------------------------------------------------
typedef CUresult (*F32EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// rows x K 32-bit matrix with leading dimension ld (elements), box = box_rows x 32; what lies outside reads as zero
static bool f32_make_map(CUtensorMap* map, const void* base, long long rows, long long K, long long ld, int box_rows) {
    static F32EncodeFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return false;
        fn = (F32EncodeFn)p;
    }
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {F32_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename Kern>
static int f32_launch(Kern kern, dim3 grid, int threads, size_t smem, bool cluster, cudaStream_t stream, const CUtensorMap& tw,
                      const CUtensorMap& ta, float* C, int M, int N, int K, long long ldc, int a_rows) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    AP_REQUIRE(e == cudaSuccess, "gemm_f32: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (cluster) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = F32_SEGS;
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
    if constexpr (std::is_invocable_v<Kern, CUtensorMap, CUtensorMap, float*, int, int, int, long long, int>) {
        AP_CHECK_PDL_LAUNCH("gemm_f32", cudaLaunchKernelEx(&cfg, kern, tw, ta, C, M, N, K, ldc, a_rows));
    } else {
        AP_CHECK_PDL_LAUNCH("gemm_f32", cudaLaunchKernelEx(&cfg, kern, tw, ta, C, M, N, K, ldc));
    }
    return AP_OK;
}

// Whether the kernels here take a 32-bit product: rows that TMA can address.  (The rule asks nothing of M: all batches of
// one weight go the same way.)
bool gemm_f32_takes(const void* a, const void* w, long long K, long long lda, long long ldw) {
    return K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0;
}

// The tile of a product of more than 32 rows, by what its clusters take (one B200, tenths of a us at K = 2048; the same ratios at K = 512 and 8192).
// 33 clusters of 8 run at once, two CTAs to an SM (the last of them often only in the next round), and a round takes `full`; up to 10 clusters have an SM to a CTA and take
// `alone`, up to 14 something between.  Of 4 x 16 outputs a thread 48 clusters run at once, three to an SM, and a last round that is not full
// takes as much less as one alone.  The tile that leaves the fewest rows empty (the larger of two equals) is taken unless another is 2 %
// cheaper: 173 rows x 3072 one round of 11 x 12 in place of two of 6 x 16 (63 us against 99), x 16384 five of 11 x 14 in place of eight (354 against
// 397); 448 rows x 16384 stay with 4 x 16 (888 us; 6 x 16 983), 144 rows x 1024 take it (39; 6 x 16 49).  Of 1213 products measured (33 to 2048 rows,
// 256 to 16384 columns, K of 512 to 8192) the tile so chosen takes 0.3 % longer than the best one on average, 10 % at most; 15 take 3 to 10 %
// longer than with the fewest empty rows, all of them together 8 % less.  Every tile gives the same bits.
struct F32Tile { int rm, cn, full, alone; };
static const F32Tile f32_tiles[] = {{8, 16, 615, 390}, {6, 16, 500, 330}, {4, 16, 0, 0},    {8, 12, 485, 325},
                                    {10, 12, 585, 375}, {11, 12, 640, 400}, {11, 14, 715, 450}};

static long long f32_tile_cost(long long M, long long N, const F32Tile& t) {
    const long long clusters = ((M + 16 * t.rm - 1) / (16 * t.rm)) * ((N + 8 * t.cn - 1) / (8 * t.cn));
    if (t.rm == 4) {
        const int rest = (int)(clusters % 48);
        return clusters / 48 * 500 + (rest == 0 ? 0 : rest <= 10 ? 280 : rest <= 14 ? 300 : rest <= 17 ? 380 : rest <= 24 ? 410 : rest <= 33 ? 530 : 540);
    }
    return clusters <= 10 ? t.alone : clusters <= 14 ? t.full * 85 / 100 : t.full * (clusters / 33 + 1);
}

static const F32Tile& f32_tile(int M, int N) {
    int pick = 0;
    for (int i = 1; i < 3; ++i) {
        const auto rows = [M](const F32Tile& t) { return ((long long)M + 16 * t.rm - 1) / (16 * t.rm) * (16 * t.rm); };
        if (rows(f32_tiles[i]) < rows(f32_tiles[pick])) pick = i;
    }
    long long least = f32_tile_cost(M, N, f32_tiles[pick]) * 98 / 100;
    for (int i = 0; i < 7; ++i) {
        const long long cost = f32_tile_cost(M, N, f32_tiles[i]);
        if (cost < least && ((long long)M + 16 * f32_tiles[i].rm - 1) / (16 * f32_tiles[i].rm) <= 65535) {
            least = cost;
            pick = i;
        }
    }
    return f32_tiles[pick];
}

// the outputs to a thread of the tile that a product of M rows and N columns takes (rows x 100 + columns); 0: the few-rows kernel's
AP_EXPORT int ap_gemm_f32_tile(int M, int N) {
    if (M <= F32_FEW_ROWS || N <= 0) return 0;
    const F32Tile& t = f32_tile(M, N);
    return t.rm * 100 + t.cn;
}

int gemm_f32(const float* a, const float* w, float* out, int M, int N, int K, long long lda, long long ldw, long long ldc,
             cudaStream_t stream) {
    const int tiles_n = (N + F32_BN - 1) / F32_BN;
    CUtensorMap tw, ta;
    if (M <= F32_FEW_ROWS) {
        AP_REQUIRE(f32_make_map(&tw, w, N, K, ldw, F32_BN), "gemm_f32: cannot encode the weight's tensor map");
        const int a_rows = (M + 7) / 8 * 8;
        AP_REQUIRE(f32_make_map(&ta, a, M, K, lda, a_rows), "gemm_f32: cannot encode the rows' tensor map");
        const size_t smem = F32_FEW_STAGES * (size_t)(F32_W_BYTES + F32_FEW_ROWS * F32_BK * 4) + 2 * F32_FEW_STAGES * 8 + 16 + 1024;
        const bool cluster = tiles_n < 2 * 148;
        const dim3 grid((unsigned)(cluster ? tiles_n * F32_SEGS : tiles_n));
#define FEW(RPT)                                                                                                             \
    do {                                                                                                                     \
        const int threads = 32 * (1 + (M + RPT - 1) / RPT);                                                                  \
        return cluster ? f32_launch(gemm_f32_few_kernel<RPT, true>, grid, threads, smem, true, stream, tw, ta, out, M, N, K, \
                                    ldc, a_rows)                                                                             \
                       : f32_launch(gemm_f32_few_kernel<RPT, false>, grid, threads, smem, false, stream, tw, ta, out, M, N,  \
                                    K, ldc, a_rows);                                                                         \
    } while (0)
        if (M <= 4) FEW(1);
        if (M <= 8) FEW(2);
        if (M <= 16) FEW(4);
        FEW(8);
#undef FEW
    }
    const int rm = f32_tile(M, N).rm, cn = f32_tile(M, N).cn;
    const dim3 grid((unsigned)((N + 8 * cn - 1) / (8 * cn)) * F32_SEGS, (unsigned)((M + 16 * rm - 1) / (16 * rm)));
    AP_REQUIRE(grid.y <= 65535, "gemm: %d rows exceed the grid of the CUDA-core kernel", M);
    AP_REQUIRE(f32_make_map(&tw, w, N, K, ldw, 8 * cn), "gemm_f32: cannot encode the weight's tensor map");
    AP_REQUIRE(f32_make_map(&ta, a, M, K, lda, 16 * rm), "gemm_f32: cannot encode the rows' tensor map");
    const size_t smem = F32_TILE_STAGES * (size_t)((8 * cn + 16 * rm) * F32_BK * 4) + 2 * F32_TILE_STAGES * 8 + 16 + 1024;
#define TILE(RM, CN) \
    if (rm == RM && cn == CN) return f32_launch(gemm_f32_tile_kernel<RM, CN>, grid, 128, smem, true, stream, tw, ta, out, M, N, K, ldc, 0)
    TILE(8, 16);
    TILE(6, 16);
    TILE(4, 16);
    TILE(8, 12);
    TILE(10, 12);
    TILE(11, 12);
    TILE(11, 14);
#undef TILE
    ap_set_error("gemm_f32: no kernel of %d x %d outputs", rm, cn);
    return AP_ERR_UNSUPPORTED;
}

// 0 when every product here so far ran to its end; else the wait that expired (1 a free stage, 2 operands)
AP_EXPORT int ap_gemm_f32_status(void) {
    int v = -1;
    if (cudaMemcpyFromSymbol(&v, g_f32_status, sizeof(int)) != cudaSuccess) return -1;
    return v;
}
