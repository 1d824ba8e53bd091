// Learned impulse-response surrogate: a Fourier-feature MLP trained and
// evaluated with hand-written tcgen05 BF16 GEMMs (FP32 accumulation in
// TMEM) on sm_100a. No counterpart in the reference; the FDTD engine of
// this library generates its training data and measures its error.
//
// Network: x (n_in values in [0, 1]) -> [sin(2 pi x B), cos(2 pi x B)]
// (B: n_in x n_freq, N(0, sigma^2)) -> (n_layers - 1) x [Linear + ReLU] ->
// Linear -> n_out samples. Weights kept in FP32 (Adam) with BF16 copies in
// both orientations for the GEMMs; activations and their gradients in BF16.
//
// GEMM: C[M][N] = A[M][K] * B[N][K]^T, both operands K-major BF16, K in
// steps of 64 through a ring of TMA stages. Warp 0 streams tiles, warp 1
// allocates TMEM, issues tcgen05.mma (K = 16 per instruction) and commits stage
// releases, warps 2-5 read the accumulator with tcgen05.ld and run the
// epilogue. Four forms, chosen by plan_gemm:
//   k_gemm_p  persistent, one CTA per SM looping over 128 x 256 output
//             tiles, 4-stage ring of 48 KB, two 256-column TMEM accumulators so
//             that the epilogue of one tile overlaps the MMAs of the next;
//   k_gemm_pair  the same by CTA pairs (clusters of two): 256 x 256 tiles, each
//             CTA loading 128 rows of A and 128 rows of B per k-step (32 KB,
//             6-stage ring) and the even CTA issuing tcgen05.mma.cta_group::2 M
//             256 N 256 over both CTAs' shared memory, so a CTA pulls a third
//             less from L2 per FLOP;
//   k_gemm    one 128 x 128 tile per CTA, 3-stage ring, two CTAs per SM;
//   k_gemm_tile  one 128 x {32, 64, 128} tile per CTA with a deep ring, of one
//             or several GEMMs in a launch, K split over a cluster where even
//             32-column tiles are too few.
// Every wait is bounded; on expiry the kernel records it in the error flag,
// drains and frees TMEM.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <random>
#include <stdexcept>
#include <string>
#include <vector>

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/afd_surrogate.h"
#include "gemm_plan.hpp"
#include "tc.cuh"
#include "wait_flags.hpp"

namespace afd {
namespace mlp {

using bf16 = __nv_bfloat16;

struct Err : std::runtime_error {
    int code;
    Err(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define MCK(call)                                                                                  \
    do {                                                                                           \
        cudaError_t e__ = (call);                                                                  \
        if (e__ != cudaSuccess) throw Err(AFD_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e__)); \
    } while (0)

constexpr int NST = 3;
constexpr int A_BYTES = TM * TK * 2, B_BYTES = TN * TK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int GEMM_THREADS = 192;
constexpr size_t GEMM_SMEM = 1024 + (size_t)NST * STAGE_BYTES + 256;
// persistent form
constexpr int PNST = 4;
constexpr int PSTAGE = A_BYTES + 2 * B_BYTES;  // A 128 x 64, B 256 x 64
constexpr size_t PGEMM_SMEM = 1024 + (size_t)PNST * PSTAGE + 256;
// pair form
constexpr int QNST = 6;
constexpr int QSTAGE = A_BYTES + B_BYTES;  // 128 rows of A and 128 rows of B, 64 deep
constexpr size_t QGEMM_SMEM = 1024 + (size_t)QNST * QSTAGE + 256;

enum Epi : int {
    EPI_F32 = 0,   // c32[row][col] = acc (+ bias[col])
    EPI_RELU = 1,  // h = relu(acc + bias): c16[row][col] and c16t[col][row]
    EPI_MASK = 2,  // g = acc * (mask[row][col] > 0): c16[row][col] and c16t[col][row]
};

struct GemmOut {
    int M, N, K;
    const float* bias;
    float* c32;
    int ldc;
    bf16* c16;
    bf16* c16t;
    int ld16, ld16t;
    const bf16* mask;
    int ldmask;
    int* flag;  // bit 0: a wait expired
};

// 32 accumulator columns col0 .. col0+31 of output row `row` through the
// epilogue EPI.
template <int EPI>
__device__ __forceinline__ void epilogue32(const GemmOut& g, float v[32], int row, int col0) {
    if (g.bias) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] += __ldg(g.bias + col0 + j);
    }
    if constexpr (EPI == EPI_F32) {
        float4* dst = reinterpret_cast<float4*>(g.c32 + (size_t)row * g.ldc + col0);
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    } else {
        if constexpr (EPI == EPI_RELU) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.0f);
        } else {
            const uint4* mk = reinterpret_cast<const uint4*>(g.mask + (size_t)row * g.ldmask + col0);
#pragma unroll
            for (int j4 = 0; j4 < 4; ++j4) {
                const uint4 w = __ldg(mk + j4);
                const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const __nv_bfloat162 p = *reinterpret_cast<const __nv_bfloat162*>(&ws[h]);
                    if (!(__low2float(p) > 0.0f)) v[8 * j4 + 2 * h] = 0.0f;
                    if (!(__high2float(p) > 0.0f)) v[8 * j4 + 2 * h + 1] = 0.0f;
                }
            }
        }
        uint32_t packed[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const __nv_bfloat162 p = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
            packed[j] = *reinterpret_cast<const uint32_t*>(&p);
        }
        uint4* dst = reinterpret_cast<uint4*>(g.c16 + (size_t)row * g.ld16 + col0);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            dst[j] = make_uint4(packed[4 * j], packed[4 * j + 1], packed[4 * j + 2], packed[4 * j + 3]);
        if (g.c16t) {
#pragma unroll
            for (int j = 0; j < 32; ++j) g.c16t[(size_t)(col0 + j) * g.ld16t + row] = __float2bfloat16_rn(v[j]);
        }
    }
}

// Two CTAs per SM (99 KB of shared memory and 128 TMEM columns each): one
// CTA's epilogue and set-up overlap the other's MMAs.
template <int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 2)
    k_gemm(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, const GemmOut g) {
    extern __shared__ unsigned char raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + NST * STAGE_BYTES);
    uint64_t* empty = full + NST;
    uint64_t* done = empty + NST;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int KT = g.K / TK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; ++s) {
            tc::bar_init(&full[s], 1);
            tc::bar_init(&empty[s], 1);
        }
        tc::bar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tc::tmem_alloc(tslot, TN);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;

    if (warp == 0) {
        {
            int issued = 0;
            for (int kt = 0; kt < KT; ++kt) {
                const int s = kt % NST;
                if (kt >= NST && !tc::bar_wait_warp(&empty[s], ((kt / NST) - 1) & 1)) {
                    atomicOr(g.flag, 1);
                    break;
                }
                unsigned char* st = sm + s * STAGE_BYTES;
                if (tc::elect()) {
                    tc::bar_expect_tx(&full[s], STAGE_BYTES);
                    tc::tma_3d(st, &ta, m0, kt, &full[s]);
                    tc::tma_3d(st + A_BYTES, &tb, n0, kt, &full[s]);
                }
                __syncwarp();
                ++issued;
            }
            // the copies still in flight complete before the block leaves
            for (int s = 0; s < NST && s < issued; ++s) {
                const int last = issued - 1 - ((issued - 1 - s) % NST);
                tc::bar_wait(&full[s], (last / NST) & 1);
            }
        }
    } else if (warp == 1) {
        {
            const uint32_t idesc = tc::bf16_f32_idesc(TM, TN);
            const uint64_t d0 = tc::sw128_kmajor_desc(tc::smem_u32(sm));
            for (int kt = 0; kt < KT; ++kt) {
                const int s = kt % NST;
                if (!tc::bar_wait_warp(&full[s], (kt / NST) & 1)) {
                    atomicOr(g.flag, 1);
                    break;
                }
                const uint64_t da = d0 + (uint64_t)(s * (STAGE_BYTES / 16)), db = da + A_BYTES / 16;
                if (tc::elect()) {
#pragma unroll
                    for (int ks = 0; ks < TK / 16; ++ks)  // 16 BF16 = 32 bytes along K inside the swizzled row
                        tc::umma_bf16(tmem, da + 2 * ks, db + 2 * ks, idesc, (kt | ks) != 0);
                    tc::umma_commit(&empty[s]);  // stage free once these MMAs have read it
                }
                __syncwarp();
            }
            if (tc::elect()) tc::umma_commit(done);  // accumulator complete (or the issued part of it)
        }
    } else {
        // epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 = tile rows
        const int q = warp & 3;
        const int row = m0 + 32 * q + lane;
        const bool ok = __all_sync(0xffffffffu, tc::bar_wait(done, 0));  // warp-uniform for tcgen05.ld
        if (!ok && lane == 0) atomicOr(g.flag, 1);
        tc::fence_after();
        if (ok) {
#pragma unroll 1
            for (int c = 0; c < TN / 32; ++c) {
                float v[32];
                tc::tmem_ld32(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * c), v);
                epilogue32<EPI>(g, v, row, n0 + 32 * c);
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc::fence_after();
        tc::tmem_dealloc(tmem, TN);
    }
}

// Output tile t of the persistent forms and of the tile form: groups of 16 row
// panels, columns outer inside a group, so that the ~148 tiles in flight share
// their A and B panels in L2 whichever operand is the long one (with the tile
// form's tiles in plain column order every column of tiles read a tall A again:
// 11008x640x10752 175 us, 148 this way; 10880x896x12288 305 and 262).
constexpr int RASTER_M = 16;
__device__ __forceinline__ void tile_of(int t, int tiles_m, int tiles_n, int tile_h, int tile_w, int& m0, int& n0) {
    const int per_group = RASTER_M * tiles_n;
    const int first = (t / per_group) * RASTER_M;
    const int gm = min(tiles_m - first, RASTER_M);
    const int w = t % per_group;
    m0 = (first + w % gm) * tile_h;
    n0 = (w / gm) * tile_w;
}

// Persistent form, one CTA per SM (194 KB of shared memory, all 512 TMEM
// columns), tiles t = blockIdx.x + i gridDim.x placed by tile_of. Barrier
// phases count uses: stage s is used for the u-th k-step of the CTA with
// s = u mod 4, accumulator ab for the it-th tile with ab = it & 1.
template <int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    k_gemm_p(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, const GemmOut g) {
    extern __shared__ unsigned char raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + PNST * PSTAGE);
    uint64_t* empty = full + PNST;
    uint64_t* acc_full = empty + PNST;   // [2] MMAs of a tile done
    uint64_t* acc_empty = acc_full + 2;  // [2] its four epilogue warps done reading
    uint64_t* drain = acc_empty + 2;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(drain + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_m = g.M / TM, tiles_n = g.N / PTN, tiles = tiles_m * tiles_n;
    const int KT = g.K / TK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < PNST; ++s) {
            tc::bar_init(&full[s], 1);
            tc::bar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::bar_init(&acc_full[b], 1);
            tc::bar_init(&acc_empty[b], 4);
        }
        tc::bar_init(drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tc::tmem_alloc(tslot, 2 * PTN);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;

    if (warp == 0) {
        {
            uint32_t u = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
                int m0, n0;
                tile_of(t, tiles_m, tiles_n, TM, PTN, m0, n0);
                for (int kt = 0; kt < KT; ++kt, ++u) {
                    const uint32_t s = u % PNST;
                    if (u >= (uint32_t)PNST && !tc::bar_wait_warp(&empty[s], ((u / PNST) - 1) & 1)) {
                        atomicOr(g.flag, 1);
                        ok = false;
                        break;
                    }
                    unsigned char* st = sm + s * PSTAGE;
                    if (tc::elect()) {
                        tc::bar_expect_tx(&full[s], PSTAGE);
                        tc::tma_3d(st, &ta, m0, kt, &full[s]);
                        tc::tma_3d(st + A_BYTES, &tb, n0, kt, &full[s]);
                    }
                    __syncwarp();
                }
            }
            // the copies still in flight complete before the block leaves
            for (uint32_t s = 0; s < (uint32_t)PNST && s < u; ++s) {
                const uint32_t last = u - 1 - ((u - 1 - s) % PNST);
                tc::bar_wait(&full[s], (last / PNST) & 1);
            }
        }
    } else if (warp == 1) {
        {
            const uint32_t idesc = tc::bf16_f32_idesc(TM, PTN);
            const uint64_t d0 = tc::sw128_kmajor_desc(tc::smem_u32(sm));
            uint32_t u = 0;
            int it = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++it) {
                const int ab = it & 1;
                if (it >= 2 && !tc::bar_wait_warp(&acc_empty[ab], ((it >> 1) - 1) & 1)) {
                    atomicOr(g.flag, 1);
                    break;
                }
                tc::fence_after();
                const uint32_t d = tmem + (uint32_t)(ab * PTN);
                for (int kt = 0; kt < KT; ++kt, ++u) {
                    const uint32_t s = u % PNST;
                    if (!tc::bar_wait_warp(&full[s], (u / PNST) & 1)) {
                        atomicOr(g.flag, 1);
                        ok = false;
                        break;
                    }
                    const uint64_t da = d0 + (uint64_t)(s * (PSTAGE / 16)), db = da + A_BYTES / 16;
                    if (tc::elect()) {
#pragma unroll
                        for (int ks = 0; ks < TK / 16; ++ks)
                            tc::umma_bf16(d, da + 2 * ks, db + 2 * ks, idesc, (kt | ks) != 0);
                        tc::umma_commit(&empty[s]);
                    }
                    __syncwarp();
                }
                if (ok && tc::elect()) tc::umma_commit(&acc_full[ab]);
                __syncwarp();
            }
            // every MMA issued has completed once this arrives
            if (tc::elect()) tc::umma_commit(drain);
            tc::bar_wait(drain, 0);
        }
    } else {
        // epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 = tile rows
        const int q = warp & 3;
        int it = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
            const int ab = it & 1;
            const bool ok = __all_sync(0xffffffffu, tc::bar_wait(&acc_full[ab], (it >> 1) & 1));
            if (!ok) {
                if (lane == 0) atomicOr(g.flag, 1);
                break;
            }
            tc::fence_after();
            int m0, n0;
            tile_of(t, tiles_m, tiles_n, TM, PTN, m0, n0);
            const int row = m0 + 32 * q + lane;
#pragma unroll 1
            for (int c = 0; c < PTN / 32; ++c) {
                float v[32];
                tc::tmem_ld32(tmem + (uint32_t)(ab * PTN) + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * c), v);
                epilogue32<EPI>(g, v, row, n0 + 32 * c);
            }
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::bar_arrive(&acc_empty[ab]);
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc::fence_after();
        tc::tmem_dealloc(tmem, 2 * PTN);
    }
}

// Pair form: clusters of two CTAs, one per SM, over 256 x 256 tiles placed
// by tile_of (pair p takes tiles p, p + pairs, ...). Rank r loads rows
// m0 + 128 r of A and n0 + 128 r of B into its own ring; both loads count
// on rank 0's full barrier (64 KB per stage). Rank 0's MMA thread issues the
// pair's MMAs and commits every stage release, accumulator completion and
// the final drain to the barrier of the same offset in both CTAs. Each CTA's
// epilogue drains its own TMEM rows and arrives on rank 0's acc_empty
// (eight warps per use). Every path reaches both cluster barriers once.
template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
    k_gemm_pair(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, const GemmOut g) {
    extern __shared__ unsigned char raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + QNST * QSTAGE);
    uint64_t* empty = full + QNST;
    uint64_t* acc_full = empty + QNST;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* drain = acc_empty + 2;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(drain + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = tc::cluster_rank();
    const int pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    const int tiles_m = g.M / (2 * TM), tiles_n = g.N / PTN, tiles = tiles_m * tiles_n;
    const int KT = g.K / TK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < QNST; ++s) {
            tc::bar_init(&full[s], 1);
            tc::bar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::bar_init(&acc_full[b], 1);
            tc::bar_init(&acc_empty[b], 8);
        }
        tc::bar_init(drain, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tc::tmem_alloc_pair(tslot, 2 * PTN);
    tc::fence_before();
    __syncthreads();
    tc::cluster_sync();  // both CTAs' barriers initialised and TMEM allocated
    tc::fence_after();
    const uint32_t tmem = *tslot;

    if (warp == 0) {
        {
            uint32_t u = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs) {
                int m0, n0;
                tile_of(t, tiles_m, tiles_n, 2 * TM, PTN, m0, n0);
                const int am = m0 + (int)rank * TM, bn = n0 + (int)rank * TN;
                for (int kt = 0; kt < KT; ++kt, ++u) {
                    const uint32_t s = u % QNST;
                    if (u >= (uint32_t)QNST && !tc::bar_wait_warp(&empty[s], ((u / QNST) - 1) & 1)) {
                        atomicOr(g.flag, 1);
                        ok = false;
                        break;
                    }
                    unsigned char* st = sm + s * QSTAGE;
                    if (tc::elect()) {
                        if (rank == 0) tc::bar_expect_tx(&full[s], 2 * QSTAGE);
                        const uint32_t fb = tc::mapa(tc::smem_u32(&full[s]), 0);
                        tc::tma_3d_pair(st, &ta, am, kt, fb);
                        tc::tma_3d_pair(st + A_BYTES, &tb, bn, kt, fb);
                    }
                    __syncwarp();
                }
            }
            // rank 0 sees the pair's copies complete; rank 1's land on the
            // same barriers
            if (rank == 0)
                for (uint32_t s = 0; s < (uint32_t)QNST && s < u; ++s) {
                    const uint32_t last = u - 1 - ((u - 1 - s) % QNST);
                    tc::bar_wait(&full[s], (last / QNST) & 1);
                }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = tc::bf16_f32_idesc(2 * TM, PTN);
            const uint64_t d0 = tc::sw128_kmajor_desc(tc::smem_u32(sm));
            uint32_t u = 0;
            int it = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs, ++it) {
                const int ab = it & 1;
                if (it >= 2 && !tc::bar_wait_warp(&acc_empty[ab], ((it >> 1) - 1) & 1)) {
                    atomicOr(g.flag, 1);
                    break;
                }
                tc::fence_after();
                const uint32_t d = tmem + (uint32_t)(ab * PTN);
                for (int kt = 0; kt < KT; ++kt, ++u) {
                    const uint32_t s = u % QNST;
                    if (!tc::bar_wait_warp(&full[s], (u / QNST) & 1)) {
                        atomicOr(g.flag, 1);
                        ok = false;
                        break;
                    }
                    const uint64_t da = d0 + (uint64_t)(s * (QSTAGE / 16)), db = da + A_BYTES / 16;
                    if (tc::elect()) {
#pragma unroll
                        for (int ks = 0; ks < TK / 16; ++ks)
                            tc::umma_bf16_pair(d, da + 2 * ks, db + 2 * ks, idesc, (kt | ks) != 0);
                        tc::umma_commit_pair(&empty[s], 3);
                    }
                    __syncwarp();
                }
                if (ok && tc::elect()) tc::umma_commit_pair(&acc_full[ab], 3);
                __syncwarp();
            }
            if (tc::elect()) tc::umma_commit_pair(drain, 3);
        }
    } else {
        const int q = warp & 3;
        int it = 0;
        for (int t = pair; t < tiles; t += pairs, ++it) {
            const int ab = it & 1;
            const bool ok = __all_sync(0xffffffffu, tc::bar_wait(&acc_full[ab], (it >> 1) & 1));
            if (!ok) {
                if (lane == 0) atomicOr(g.flag, 1);
                break;
            }
            tc::fence_after();
            int m0, n0;
            tile_of(t, tiles_m, tiles_n, 2 * TM, PTN, m0, n0);
            const int row = m0 + (int)rank * TM + 32 * q + lane;
#pragma unroll 1
            for (int c = 0; c < PTN / 32; ++c) {
                float v[32];
                tc::tmem_ld32(tmem + (uint32_t)(ab * PTN) + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * c), v);
                epilogue32<EPI>(g, v, row, n0 + 32 * c);
            }
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::bar_arrive_cluster(tc::mapa(tc::smem_u32(&acc_empty[ab]), 0));
        }
    }
    // every MMA of the pair has completed (rank 0 commits the drain to both)
    if (warp == 1 && lane == 0) tc::bar_wait(drain, 0);
    tc::fence_before();
    __syncthreads();
    tc::cluster_sync();  // neither CTA leaves while the other may still use its memory
    if (warp == 1) {
        __syncwarp();
        tc::fence_after();
        tc::tmem_dealloc_pair(tmem, 2 * PTN);
    }
}

// Tile form: one 128 x TN tile per CTA of one or several GEMMs of a launch,
// for outputs too small to fill the chip with 256 x 256 tiles. A deep ring
// (the loop over K is bound by the latency and rate of one SM's loads, not by
// the MMAs). With a cluster of S CTAs the tile's K range is split over them:
// each accumulates its share, writes it to its own shared memory, and CTA z
// sums columns z TN / S .. in the order of the shares (EPI_F32 only).
//
// Issuing a stage costs its two warps about 300 clocks whatever its size, so a
// stage holds two 64-column blocks, fetched by one TMA box per operand:
// 128x2048x8192 as 32-column tiles fell from 43.2 us (one block a stage, the
// loops in one lane) over 30.8 (elected lane) to 24.7. The five weight
// gradients of the 512-wide network run in one launch of 120 tiles instead of
// five of 16 us each with 4 to 32 CTAs.
template <int TN_>
struct Tile {
    static constexpr int b_bytes = TN_ * TK * 2;
    static constexpr int stage = 2 * (A_BYTES + b_bytes);  // two column blocks of A, then of B
    static constexpr int stages = TN_ == 128 ? 3 : TN_ == 64 ? 4 : 5;
    static constexpr size_t smem = 1024 + (size_t)stages * stage + 256;
    static constexpr int part_ld = TN_ + 4;  // row stride of a share in shared memory (floats)
};
struct alignas(64) GemmItem {
    CUtensorMap ta, tb;
    GemmOut o;
    int epi, first;  // first tile of this GEMM in the launch; several: EPI_F32
};
template <int NG>
struct GemmGroup {
    GemmItem g[NG];
    int n;
};
template <int TN_, int NG>
__global__ void __launch_bounds__(GEMM_THREADS, 1) k_gemm_tile(const __grid_constant__ GemmGroup<NG> gg) {
    using S = Tile<TN_>;
    constexpr int NS = S::stages;
    extern __shared__ unsigned char raw[];
    unsigned char* sm = (unsigned char*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = reinterpret_cast<uint64_t*>(sm + NS * S::stage);
    uint64_t* empty = full + NS;
    uint64_t* done = empty + NS;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = (int)gridDim.y, part = (int)blockIdx.y;
    int at = 0;
    if constexpr (NG > 1)
        while (at + 1 < gg.n && (int)blockIdx.x >= gg.g[at + 1].first) ++at;
    const GemmItem& G = gg.g[at];
    const GemmOut& g = G.o;
    int m0, n0;
    tile_of((int)blockIdx.x - G.first, g.M / TM, g.N / TN_, TM, TN_, m0, n0);
    const int KT = (g.K / TK + 1) / 2;  // two column blocks a step; the last one's second may be zero fill
    const int kb = (int)((int64_t)KT * part / split), ke = (int)((int64_t)KT * (part + 1) / split);
    tc::launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < NS; ++i) {
            tc::bar_init(&full[i], 1);
            tc::bar_init(&empty[i], 1);
        }
        tc::bar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tc::tmem_alloc(tslot, TN_);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *tslot;
    tc::wait_previous();
    const int q = warp & 3;
    bool ok = true;

    if (warp == 0) {
        {
            int issued = 0;
            for (int kt = kb; kt < ke; ++kt, ++issued) {
                const int s = issued % NS;
                if (issued >= NS && !tc::bar_wait_warp(&empty[s], ((issued / NS) - 1) & 1)) {
                    atomicOr(g.flag, 1);
                    break;
                }
                unsigned char* st = sm + s * S::stage;
                if (tc::elect()) {
                    tc::bar_expect_tx(&full[s], S::stage);
                    tc::tma_3d(st, &G.ta, m0, 2 * kt, &full[s]);
                    tc::tma_3d(st + 2 * A_BYTES, &G.tb, n0, 2 * kt, &full[s]);
                }
                __syncwarp();
            }
            // the copies still in flight complete before the block leaves
            for (int s = 0; s < NS && s < issued; ++s) {
                const int last = issued - 1 - ((issued - 1 - s) % NS);
                tc::bar_wait(&full[s], (last / NS) & 1);
            }
        }
    } else if (warp == 1) {
        {
            const uint32_t idesc = tc::bf16_f32_idesc(TM, TN_);
            const uint64_t d0 = tc::sw128_kmajor_desc(tc::smem_u32(sm));
            for (int u = 0; u < ke - kb; ++u) {
                const int s = u % NS;
                if (!tc::bar_wait_warp(&full[s], (u / NS) & 1)) {
                    atomicOr(g.flag, 1);
                    break;
                }
                const uint64_t da = d0 + (uint64_t)(s * (S::stage / 16)), db = da + 2 * A_BYTES / 16;
                if (tc::elect()) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int ks = 0; ks < TK / 16; ++ks)
                            tc::umma_bf16(tmem, da + h * (A_BYTES / 16) + 2 * ks, db + h * (S::b_bytes / 16) + 2 * ks,
                                          idesc, (u | h | ks) != 0);
                    tc::umma_commit(&empty[s]);
                }
                __syncwarp();
            }
            if (tc::elect()) tc::umma_commit(done);  // accumulator complete (or the issued part of it)
        }
    } else {
        ok = __all_sync(0xffffffffu, tc::bar_wait(done, 0));
        if (!ok && lane == 0) atomicOr(g.flag, 1);
        tc::fence_after();
        const int row = 32 * q + lane;
        if (ok) {
#pragma unroll 1
            for (int c = 0; c < TN_ / 32; ++c) {
                float v[32];
                tc::tmem_ld32(tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(32 * c), v);
                if (split > 1) {
                    // every MMA that read the ring has completed
                    float4* p = reinterpret_cast<float4*>(sm) + (row * S::part_ld + 32 * c) / 4;
#pragma unroll
                    for (int j = 0; j < 8; ++j) p[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                } else if (NG > 1 || G.epi == EPI_F32) {
                    epilogue32<EPI_F32>(g, v, m0 + row, n0 + 32 * c);
                } else if (G.epi == EPI_RELU) {
                    epilogue32<EPI_RELU>(g, v, m0 + row, n0 + 32 * c);
                } else {
                    epilogue32<EPI_MASK>(g, v, m0 + row, n0 + 32 * c);
                }
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (split > 1) {
        tc::cluster_sync();  // all shares written
        if (warp >= 2) {
            const int w = TN_ / split, row = 32 * q + lane, c0 = part * w;
            const uint32_t mine = tc::smem_u32(sm) + (uint32_t)(row * S::part_ld + c0) * 4;
            float* dst = g.c32 + (size_t)(m0 + row) * g.ldc + n0 + c0;
#pragma unroll 1
            for (int j = 0; j < w; j += 4) {
                float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                for (int z = 0; z < split; ++z) {
                    const float4 b = tc::ld_cluster(tc::mapa(mine + (uint32_t)j * 4, (uint32_t)z));
                    if (z == 0) a = b;
                    else a = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
                }
                *reinterpret_cast<float4*>(dst + j) = a;
            }
        }
        __syncthreads();
        tc::cluster_sync();  // no CTA leaves while its share is read
    }
    if (warp == 1) {
        __syncwarp();
        tc::fence_after();
        tc::tmem_dealloc(tmem, TN_);
    }
}

// ---- small kernels ---------------------------------------------------------
// Tiles of 64 x 64 BF16 values on their way into a matrix and its transpose,
// whose rows of 64 values leave as 128-byte runs. 256 threads.
constexpr int SQ = 64;
struct alignas(16) SquareTile {
    bf16 v[SQ][SQ + 2];
    // the transpose: row c0 + c of t[.][ld] from r0 on; after a barrier
    __device__ __forceinline__ void store_transposed(bf16* t, size_t ld, int c0, int r0) const {
        for (int k = threadIdx.x; k < SQ * SQ / 2; k += 256) {
            const int c = k / (SQ / 2), r = k % (SQ / 2) * 2;
            *reinterpret_cast<__nv_bfloat162*>(t + (size_t)(c0 + c) * ld + r0 + r) =
                __nv_bfloat162(v[r][c], v[r + 1][c]);
        }
    }
};

// Fourier features: f[r][j] = sin(2 pi <x_r, B_j>) (j < n_freq) and the
// cosine at j + n_freq; rows r >= n are zero. Block: 16 rows, 32 frequencies
// (columns 0..31 of the tile the sines, 32..63 the cosines); with 64 rows a
// block 64 blocks of 1024 rows took 9.5 us.
constexpr int kFourierRows = 16;
__global__ void __launch_bounds__(256) k_fourier(const float* x, int n, int n_in, const float* Bf, int n_freq,
                                                 int rows, bf16* f, bf16* ft) {
    __shared__ alignas(16) bf16 t[kFourierRows][SQ + 2];
    const int r0 = blockIdx.x * kFourierRows, j0 = blockIdx.y * 32, F = 2 * n_freq;
    const int jj = threadIdx.x & 31;
    tc::launch_dependents();
    for (int rr = threadIdx.x >> 5; rr < kFourierRows; rr += 8) {
        const int r = r0 + rr, j = j0 + jj;
        float s = 0.0f, c = 0.0f;
        if (r < n) {
            float a = 0.0f;
            for (int i = 0; i < n_in; ++i) a += x[(size_t)r * n_in + i] * Bf[(size_t)i * n_freq + j];
            const float ph = 6.283185307179586f * a;
            s = sinf(ph);
            c = cosf(ph);
        }
        t[rr][jj] = __float2bfloat16_rn(s);
        t[rr][32 + jj] = __float2bfloat16_rn(c);
        f[(size_t)r * F + j] = t[rr][jj];
        f[(size_t)r * F + j + n_freq] = t[rr][32 + jj];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < SQ * kFourierRows / 2; k += 256) {
        const int c = k / (kFourierRows / 2), r = k % (kFourierRows / 2) * 2;
        const int row = c < 32 ? j0 + c : n_freq + j0 + c - 32;
        *reinterpret_cast<__nv_bfloat162*>(ft + (size_t)row * rows + r0 + r) = __nv_bfloat162(t[r][c], t[r + 1][c]);
    }
}

// Loss gradient of the mean squared error over n valid rows:
// d = 2 (pred - y) / (n * n_out); rows >= n get zero. Loss partial sums per
// block (FP32; the loss value is for reporting). Block: 64 x 64 values.
__global__ void __launch_bounds__(256) k_mse_grad(const float* pred, const float* y, int n, int n_out, int rows,
                                                  float scale, bf16* d, bf16* dt, float* loss_acc) {
    __shared__ SquareTile t;
    __shared__ float part[8];
    const int c0 = blockIdx.x * SQ, r0 = blockIdx.y * SQ;
    const int c = threadIdx.x % 16 * 4;
    tc::launch_dependents();
    tc::wait_previous();
    float sq = 0.0f;
#pragma unroll
    for (int rr = threadIdx.x / 16; rr < SQ; rr += 16) {
        const int r = r0 + rr;
        const size_t at = (size_t)r * n_out + c0 + c;
        float e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (r < n) {
            const float4 p = *reinterpret_cast<const float4*>(pred + at), q = *reinterpret_cast<const float4*>(y + at);
            e[0] = p.x - q.x;
            e[1] = p.y - q.y;
            e[2] = p.z - q.z;
            e[3] = p.w - q.w;
        }
        bf16 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = __float2bfloat16_rn(scale * e[k]);
            t.v[rr][c + k] = v[k];
            sq += e[k] * e[k];
        }
        __nv_bfloat162* out = reinterpret_cast<__nv_bfloat162*>(d + at);
        out[0] = __nv_bfloat162(v[0], v[1]);
        out[1] = __nv_bfloat162(v[2], v[3]);
    }
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sq;
    __syncthreads();
    t.store_transposed(dt, (size_t)rows, c0, r0);
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) sq += part[k];
        if (sq != 0.0f) atomicAdd(loss_acc, sq);
    }
}

// What the bias gradients and the Adam update use of the layers.
constexpr int kMaxLayers = 16;
struct LayerDev {
    int in, out, first;      // first: block of k_adam or warp of k_bias_grad
    const bf16* gt;          // [out][rows]: gradient at the layer's output, transposed
    float *w, *gw, *mw, *vw, *b, *gb, *mb, *vb;
    bf16 *w16, *w16t;
};
struct Layers {
    LayerDev l[kMaxLayers];
    int n, rows, total;
};

// Bias gradients of all layers: db[o] = sum_r d[r][o], from the transposed
// copy (rows contiguous), summed in order by one warp per output.
__global__ void k_bias_grad(const __grid_constant__ Layers a) {
    const int w = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    tc::launch_dependents();
    if (w >= a.total) return;
    tc::wait_previous();
    int k = 0, o = w;
    while (o >= a.l[k].out) o -= a.l[k++].out;
    const bf16* dt = a.l[k].gt + (size_t)o * a.rows;
    float s = 0.0f;
#pragma unroll 8
    for (int r = lane; r < a.rows; r += 32) s += __bfloat162float(dt[r]);
    for (int i = 16; i > 0; i >>= 1) s += __shfl_down_sync(0xffffffffu, s, i);
    if (lane == 0) a.l[k].gb[o] = s;
}

// Adam on FP32 master weights; refreshes the BF16 copies w16 ([out][in])
// and w16t ([in][out]). All layers in one launch: a block takes a 64 x 64 tile
// of a weight matrix, the blocks after a layer's tiles 256 biases each.
struct AdamStep {
    float lr, b1, b2, eps, c1, c2;
    __device__ __forceinline__ float operator()(float w, float g, float* m, float* v) const {
        const float mm = b1 * *m + (1.0f - b1) * g;
        const float vv = b2 * *v + (1.0f - b2) * g * g;
        *m = mm;
        *v = vv;
        return w - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    }
};
__global__ void __launch_bounds__(256) k_adam(const __grid_constant__ Layers a, AdamStep step) {
    __shared__ SquareTile t;
    int k = 0;
    while (k + 1 < a.n && (int)blockIdx.x >= a.l[k + 1].first) ++k;
    const LayerDev& L = a.l[k];
    const int tile = (int)blockIdx.x - L.first, tx = L.in / SQ, tiles = tx * (L.out / SQ);
    tc::wait_previous();
    if (tile >= tiles) {
        const int i = (tile - tiles) * 256 + (int)threadIdx.x;
        if (i < L.out) L.b[i] = step(L.b[i], L.gb[i], L.mb + i, L.vb + i);
        return;
    }
    const int r0 = tile / tx * SQ, c0 = tile % tx * SQ, c = (int)threadIdx.x % 16 * 4;
#pragma unroll
    for (int rr = threadIdx.x / 16; rr < SQ; rr += 16) {
        const size_t at = (size_t)(r0 + rr) * L.in + c0 + c;
        float4 w = *reinterpret_cast<float4*>(L.w + at), m = *reinterpret_cast<float4*>(L.mw + at),
               v = *reinterpret_cast<float4*>(L.vw + at);
        const float4 g = *reinterpret_cast<const float4*>(L.gw + at);
        w.x = step(w.x, g.x, &m.x, &v.x);
        w.y = step(w.y, g.y, &m.y, &v.y);
        w.z = step(w.z, g.z, &m.z, &v.z);
        w.w = step(w.w, g.w, &m.w, &v.w);
        *reinterpret_cast<float4*>(L.w + at) = w;
        *reinterpret_cast<float4*>(L.mw + at) = m;
        *reinterpret_cast<float4*>(L.vw + at) = v;
        const __nv_bfloat162 lo = __floats2bfloat162_rn(w.x, w.y), hi = __floats2bfloat162_rn(w.z, w.w);
        __nv_bfloat162* out = reinterpret_cast<__nv_bfloat162*>(L.w16 + at);
        out[0] = lo;
        out[1] = hi;
        *reinterpret_cast<__nv_bfloat162*>(&t.v[rr][c]) = lo;
        *reinterpret_cast<__nv_bfloat162*>(&t.v[rr][c + 2]) = hi;
    }
    __syncthreads();
    t.store_transposed(L.w16t, (size_t)L.out, c0, r0);
}

__global__ void k_f32_to_bf16_both(const float* w, int outs, int in, bf16* w16, bf16* w16t) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)outs * in) return;
    const bf16 b = __float2bfloat16_rn(w[i]);
    w16[i] = b;
    w16t[(size_t)(i % in) * outs + i / in] = b;
}

// ---- host ------------------------------------------------------------------
template <typename T>
struct Dev {
    T* p = nullptr;
    size_t n = 0;
    Dev() = default;
    Dev(const Dev&) = delete;
    Dev& operator=(const Dev&) = delete;
    ~Dev() {
        if (p) cudaFree(p);
    }
    void alloc(size_t count) {
        if (p) cudaFree(p);
        p = nullptr;
        n = count;
        if (count) {
            MCK(cudaMalloc(&p, count * sizeof(T)));
            // the zeroing runs on the legacy stream, which the surrogate's
            // non-blocking stream does not wait for: finished before return
            MCK(cudaMemset(p, 0, count * sizeof(T)));
            MCK(cudaStreamSynchronize(cudaStreamLegacy));
        }
    }
};

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeFn encoder() {
    static EncodeFn fn = nullptr;
    if (!fn) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        MCK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q));
        if (!f || q != cudaDriverEntryPointSuccess) throw Err(AFD_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        fn = (EncodeFn)f;
    }
    return fn;
}

// K-major BF16 operand [rows][K] (row stride K) as 64-element column blocks:
// boxes of box_rows rows of `blocks` neighbouring blocks, 128-byte swizzle;
// blocks past the last one read as zeros.
static CUtensorMap operand_map(const bf16* base, int rows, int K, int box_rows, int blocks) {
    if (rows % 128 || K % 64 || ((uintptr_t)base & 15)) throw Err(AFD_ERR_ARG, "GEMM operand not tile-aligned");
    CUtensorMap m;
    const cuuint64_t dims[3] = {TK, (cuuint64_t)rows, (cuuint64_t)(K / TK)};
    const cuuint64_t strides[2] = {(cuuint64_t)K * 2, TK * 2};
    const cuuint32_t box[3] = {TK, (cuuint32_t)box_rows, (cuuint32_t)blocks}, estr[3] = {1, 1, 1};
    CUresult r = encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)base, dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Err(AFD_ERR_CUDA, "tensor map encoding failed");
    return m;
}

struct Gemm {
    CUtensorMap ta, tb;
    GemmOut o;
    int epi;
    GemmPlan plan;
};

// Shared-memory limits of the GEMM kernels and the SM count, per device
// (function attributes belong to the current device).
struct DeviceGemm {
    bool ready = false;
    int sms = 0;
};

static std::mutex g_gemm_mu;  // guards the per-device tables below

static int set_smem_attr() {
    static DeviceGemm devs[64];
    std::lock_guard<std::mutex> lock(g_gemm_mu);
    int dev = 0;
    MCK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) throw Err(AFD_ERR_ARG, "device ordinal out of range");
    DeviceGemm& d = devs[dev];
    if (d.ready) return d.sms;
    const int s2 = (int)PGEMM_SMEM, s3 = (int)QGEMM_SMEM;
    auto tile_attr = [](auto kernel, size_t smem) {
        MCK(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    };
    tile_attr(k_gemm<EPI_F32>, GEMM_SMEM);
    tile_attr(k_gemm<EPI_RELU>, GEMM_SMEM);
    tile_attr(k_gemm<EPI_MASK>, GEMM_SMEM);
    tile_attr(k_gemm_tile<128, 1>, Tile<128>::smem);
    tile_attr(k_gemm_tile<64, 1>, Tile<64>::smem);
    tile_attr(k_gemm_tile<32, 1>, Tile<32>::smem);
    tile_attr(k_gemm_tile<128, kMaxLayers>, Tile<128>::smem);
    tile_attr(k_gemm_tile<64, kMaxLayers>, Tile<64>::smem);
    tile_attr(k_gemm_tile<32, kMaxLayers>, Tile<32>::smem);
    MCK(cudaFuncSetAttribute((const void*)k_gemm_p<EPI_F32>, cudaFuncAttributeMaxDynamicSharedMemorySize, s2));
    MCK(cudaFuncSetAttribute((const void*)k_gemm_p<EPI_RELU>, cudaFuncAttributeMaxDynamicSharedMemorySize, s2));
    MCK(cudaFuncSetAttribute((const void*)k_gemm_p<EPI_MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize, s2));
    MCK(cudaFuncSetAttribute((const void*)k_gemm_pair<EPI_F32>, cudaFuncAttributeMaxDynamicSharedMemorySize, s3));
    MCK(cudaFuncSetAttribute((const void*)k_gemm_pair<EPI_RELU>, cudaFuncAttributeMaxDynamicSharedMemorySize, s3));
    MCK(cudaFuncSetAttribute((const void*)k_gemm_pair<EPI_MASK>, cudaFuncAttributeMaxDynamicSharedMemorySize, s3));
    MCK(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev));
    d.ready = true;
    return d.sms;
}

// A launch that may start before the stream's previous kernel has ended, for
// the network's kernels, which wait for it themselves (wait_previous): a
// training step is a chain of kernels of 5 to 14 us (135 -> 100 us a step at
// 1024 rows, 512 wide). split > 1: clusters of that
// many CTAs along y. Calls of a single GEMM start after what the stream holds.
template <typename... P, typename... A>
static void launch_after(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, int split,
                         bool early, const A&... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute at[2]{};
    if (early) {
        at[c.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[c.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (split > 1) {
        at[c.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[c.numAttrs].val.clusterDim.x = 1;
        at[c.numAttrs].val.clusterDim.y = (unsigned)split;
        at[c.numAttrs++].val.clusterDim.z = 1;
    }
    c.attrs = at;
    MCK(cudaLaunchKernelEx(&c, kernel, args...));
}
template <int TN_, int NG>
static void launch_tiles(const GemmGroup<NG>& gg, int tiles, int split, bool early, cudaStream_t st) {
    launch_after(k_gemm_tile<TN_, NG>, dim3((unsigned)tiles, (unsigned)split), GEMM_THREADS, Tile<TN_>::smem, st, split,
                 early, gg);
}

// The GEMMs of `v` (n <= NG, all planned with the same tile columns) in one launch.
template <int NG>
static void launch_group(const Gemm* v, int n, cudaStream_t st, bool early) {
    GemmGroup<NG> gg;
    gg.n = n;
    const int tn = v[0].plan.form;
    int tiles = 0;
    for (int i = 0; i < n; ++i) {
        gg.g[i].ta = v[i].ta;
        gg.g[i].tb = v[i].tb;
        gg.g[i].o = v[i].o;
        gg.g[i].epi = v[i].epi;
        gg.g[i].first = tiles;
        tiles += (v[i].o.M / TM) * (v[i].o.N / tn);
    }
    const int split = NG == 1 ? v[0].plan.split : 1;
    if (tn == 128) launch_tiles<128, NG>(gg, tiles, split, early, st);
    else if (tn == 64) launch_tiles<64, NG>(gg, tiles, split, early, st);
    else launch_tiles<32, NG>(gg, tiles, split, early, st);
}

static void launch(const Gemm& G, cudaStream_t st, bool early = false) {
    const int sms = set_smem_attr();
    if (G.plan.form == kPair) {
        const int tiles = (G.o.M / (2 * TM)) * (G.o.N / PTN);
        const unsigned grid = 2u * (unsigned)std::max(1, std::min(tiles, sms / 2));
        switch (G.epi) {
            case EPI_F32: k_gemm_pair<EPI_F32><<<grid, GEMM_THREADS, QGEMM_SMEM, st>>>(G.ta, G.tb, G.o); break;
            case EPI_RELU: k_gemm_pair<EPI_RELU><<<grid, GEMM_THREADS, QGEMM_SMEM, st>>>(G.ta, G.tb, G.o); break;
            default: k_gemm_pair<EPI_MASK><<<grid, GEMM_THREADS, QGEMM_SMEM, st>>>(G.ta, G.tb, G.o); break;
        }
    } else if (G.plan.form == kPersist) {
        const int tiles = (G.o.M / TM) * (G.o.N / PTN);
        const unsigned grid = (unsigned)std::max(1, std::min(tiles, sms));
        switch (G.epi) {
            case EPI_F32: k_gemm_p<EPI_F32><<<grid, GEMM_THREADS, PGEMM_SMEM, st>>>(G.ta, G.tb, G.o); break;
            case EPI_RELU: k_gemm_p<EPI_RELU><<<grid, GEMM_THREADS, PGEMM_SMEM, st>>>(G.ta, G.tb, G.o); break;
            default: k_gemm_p<EPI_MASK><<<grid, GEMM_THREADS, PGEMM_SMEM, st>>>(G.ta, G.tb, G.o); break;
        }
    } else if (G.plan.form == kDual) {
        const dim3 grid((unsigned)(G.o.N / TN), (unsigned)(G.o.M / TM));
        switch (G.epi) {
            case EPI_F32: k_gemm<EPI_F32><<<grid, GEMM_THREADS, GEMM_SMEM, st>>>(G.ta, G.tb, G.o); break;
            case EPI_RELU: k_gemm<EPI_RELU><<<grid, GEMM_THREADS, GEMM_SMEM, st>>>(G.ta, G.tb, G.o); break;
            default: k_gemm<EPI_MASK><<<grid, GEMM_THREADS, GEMM_SMEM, st>>>(G.ta, G.tb, G.o); break;
        }
    } else {
        launch_group<1>(&G, 1, st, early);
    }
    MCK(cudaGetLastError());
}

static Gemm make_gemm(int epi, const bf16* A, const bf16* B, int M, int N, int K, int* flag, bool may_split = false,
                      int tile = -1) {
    if (M % TM || N % TN || K % TK || K <= 0) throw Err(AFD_ERR_ARG, "GEMM sizes must be multiples of 128 x 128 x 64");
    Gemm G;
    G.plan = tile < 0 ? plan_gemm(M, N, K, may_split, set_smem_attr()) : GemmPlan{tile, 1};
    const int form = G.plan.form, blocks = form >= 32 ? 2 : 1;
    G.ta = operand_map(A, M, K, TM, blocks);
    G.tb = operand_map(B, N, K, form >= 32 ? form : form == kPersist ? PTN : TN, blocks);
    std::memset(&G.o, 0, sizeof(G.o));
    G.o.M = M;
    G.o.N = N;
    G.o.K = K;
    G.o.flag = flag;
    G.epi = epi;
    return G;
}

struct Layer {
    int in = 0, out = 0;
    Dev<float> w, b, gw, gb, mw, vw, mb, vb;
    Dev<bf16> w16, w16t;
};

}  // namespace mlp
}  // namespace afd

using namespace afd::mlp;

struct afd_mlp {
    afd_mlp_params prm{};
    std::string err;
    int device = 0;
    cudaStream_t own = nullptr, stream = nullptr;
    int rows = 0, F = 0;
    std::vector<Layer*> L;
    Dev<float> fourier;             // [n_in][n_freq]
    Dev<float> xin, yin;            // staging copies of inputs / targets
    Dev<bf16> feat, featT;          // [rows][F], [F][rows]
    std::vector<Dev<bf16>*> H, HT;  // hidden activations per hidden layer: [rows][hidden], [hidden][rows]
    std::vector<Dev<bf16>*> G, GT;  // gradients w.r.t. each layer's output (pre-activation)
    Dev<float> pred;                // [rows][n_out]
    Dev<float> loss;                // 1
    Dev<int> flag;
    int64_t step = 0;
    std::vector<Gemm> fwd, bwd_w, bwd_x;
    bool group_w = false;           // the weight gradients in one launch
    Layers bias_dev{}, adam_dev{};

    ~afd_mlp() {
        if (stream) cudaStreamSynchronize(stream);
        for (auto* l : L) delete l;
        for (auto* p : H) delete p;
        for (auto* p : HT) delete p;
        for (auto* p : G) delete p;
        for (auto* p : GT) delete p;
        if (own) cudaStreamDestroy(own);
    }

    const bf16* layer_input(int l) const { return l == 0 ? feat.p : H[l - 1]->p; }
    const bf16* layer_input_t(int l) const { return l == 0 ? featT.p : HT[l - 1]->p; }

    void build() {
        const afd_mlp_params& p = prm;
        if (p.n_in < 1 || p.n_freq < 32 || (2 * p.n_freq) % 128 || p.hidden % 128 || p.n_out % 128 ||
            p.n_layers < 2 || p.n_layers > 16 || p.batch < 128 || p.batch % 128)
            throw Err(AFD_ERR_ARG, "surrogate sizes: 2*n_freq, hidden, n_out and batch must be multiples of 128");
        int ndev = 0;
        if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) throw Err(AFD_ERR_CUDA, "no CUDA device available");
        device = p.device;
        MCK(cudaSetDevice(device));
        MCK(cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking));
        stream = own;
        set_smem_attr();
        rows = p.batch;
        F = 2 * p.n_freq;
        std::mt19937_64 rng(p.seed);
        std::normal_distribution<double> nd(0.0, 1.0);
        std::vector<float> fb((size_t)p.n_in * p.n_freq);
        for (auto& v : fb) v = (float)(nd(rng) * p.fourier_sigma);
        fourier.alloc(fb.size());
        MCK(cudaMemcpyAsync(fourier.p, fb.data(), fb.size() * 4, cudaMemcpyHostToDevice, stream));
        MCK(cudaStreamSynchronize(stream));
        for (int l = 0; l < p.n_layers; ++l) {
            Layer* ly = new Layer;
            L.push_back(ly);
            ly->in = l == 0 ? F : p.hidden;
            ly->out = l == p.n_layers - 1 ? p.n_out : p.hidden;
            const size_t nw = (size_t)ly->in * ly->out;
            // He-uniform initialisation from the seed
            std::vector<float> w(nw);
            const double a = std::sqrt(6.0 / ly->in);
            std::uniform_real_distribution<double> ud(-a, a);
            for (auto& v : w) v = (float)ud(rng);
            ly->w.alloc(nw);
            MCK(cudaMemcpyAsync(ly->w.p, w.data(), nw * 4, cudaMemcpyHostToDevice, stream));
            MCK(cudaStreamSynchronize(stream));
            ly->b.alloc(ly->out);
            ly->gw.alloc(nw);
            ly->gb.alloc(ly->out);
            ly->mw.alloc(nw);
            ly->vw.alloc(nw);
            ly->mb.alloc(ly->out);
            ly->vb.alloc(ly->out);
            ly->w16.alloc(nw);
            ly->w16t.alloc(nw);
            refresh_bf16(l);
        }
        xin.alloc((size_t)rows * p.n_in);
        yin.alloc((size_t)rows * p.n_out);
        feat.alloc((size_t)rows * F);
        featT.alloc((size_t)rows * F);
        for (int l = 0; l + 1 < p.n_layers; ++l) {
            H.push_back(new Dev<bf16>);
            H.back()->alloc((size_t)rows * p.hidden);
            HT.push_back(new Dev<bf16>);
            HT.back()->alloc((size_t)rows * p.hidden);
        }
        for (int l = 0; l < p.n_layers; ++l) {
            const int o = L[(size_t)l]->out;
            G.push_back(new Dev<bf16>);
            G.back()->alloc((size_t)rows * o);
            GT.push_back(new Dev<bf16>);
            GT.back()->alloc((size_t)rows * o);
        }
        pred.alloc((size_t)rows * p.n_out);
        loss.alloc(1);
        flag.alloc(1);
        // one launch for the weight gradients where they would not fill the chip one by one
        std::vector<std::pair<int, int>> sizes;
        for (auto* ly : L) sizes.emplace_back(ly->out, ly->in);
        const int form_w = plan_group(sizes, rows, set_smem_attr());
        group_w = form_w >= 0;
        // the GEMMs of one training step, with their tensor maps
        for (int l = 0; l < p.n_layers; ++l) {
            Layer& ly = *L[(size_t)l];
            const bool last = l == p.n_layers - 1;
            Gemm f = make_gemm(last ? EPI_F32 : EPI_RELU, layer_input(l), ly.w16.p, rows, ly.out, ly.in, flag.p);
            f.o.bias = ly.b.p;
            if (last) {
                f.o.c32 = pred.p;
                f.o.ldc = ly.out;
            } else {
                f.o.c16 = H[(size_t)l]->p;
                f.o.c16t = HT[(size_t)l]->p;
                f.o.ld16 = ly.out;
                f.o.ld16t = rows;
            }
            fwd.push_back(f);
            // dW = G^T (out x rows) * X^T (in x rows)^T
            Gemm w = make_gemm(EPI_F32, GT[(size_t)l]->p, layer_input_t(l), ly.out, ly.in, rows, flag.p, false, form_w);
            w.o.c32 = ly.gw.p;
            w.o.ldc = ly.in;
            bwd_w.push_back(w);
            if (l > 0) {
                // dX = G (rows x out) * W^T-as-[in][out] -> masked by the ReLU of layer l-1
                Gemm x = make_gemm(EPI_MASK, G[(size_t)l]->p, ly.w16t.p, rows, ly.in, ly.out, flag.p);
                x.o.c16 = G[(size_t)l - 1]->p;
                x.o.c16t = GT[(size_t)l - 1]->p;
                x.o.ld16 = ly.in;
                x.o.ld16t = rows;
                x.o.mask = H[(size_t)l - 1]->p;
                x.o.ldmask = ly.in;
                bwd_x.push_back(x);
            }
        }
        Layers& t = bias_dev;
        t.n = p.n_layers;
        t.rows = rows;
        for (int l = 0; l < p.n_layers; ++l) {
            Layer& ly = *L[(size_t)l];
            t.l[l] = LayerDev{ly.in, ly.out, 0, GT[(size_t)l]->p, ly.w.p, ly.gw.p, ly.mw.p, ly.vw.p, ly.b.p, ly.gb.p,
                              ly.mb.p, ly.vb.p, ly.w16.p, ly.w16t.p};
            t.total += ly.out;
        }
        adam_dev = t;
        adam_dev.total = 0;
        for (int l = 0; l < p.n_layers; ++l) {
            LayerDev& d = adam_dev.l[l];
            d.first = adam_dev.total;
            adam_dev.total += (d.in / SQ) * (d.out / SQ) + (d.out + 255) / 256;
        }
    }

    void refresh_bf16(int l) {
        Layer& ly = *L[(size_t)l];
        const int64_t n = (int64_t)ly.in * ly.out;
        k_f32_to_bf16_both<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(ly.w.p, ly.out, ly.in, ly.w16.p, ly.w16t.p);
        MCK(cudaGetLastError());
    }

    void check_flag() {
        int f = 0;
        MCK(cudaMemcpyAsync(&f, flag.p, 4, cudaMemcpyDeviceToHost, stream));
        MCK(cudaStreamSynchronize(stream));
        if (f) throw Err(AFD_ERR_CUDA, "surrogate GEMM pipeline wait timed out");
    }

    void features(const float* x_dev, int n) {
        if (n < 1 || n > rows) throw Err(AFD_ERR_ARG, "row count outside 1..batch");
        MCK(cudaMemcpyAsync(xin.p, x_dev, (size_t)n * prm.n_in * 4, cudaMemcpyDefault, stream));
        const dim3 grd((unsigned)(rows / kFourierRows), (unsigned)(prm.n_freq / 32));
        k_fourier<<<grd, 256, 0, stream>>>(xin.p, n, prm.n_in, fourier.p, prm.n_freq, rows, feat.p, featT.p);
        MCK(cudaGetLastError());
    }

    void forward() {
        for (auto& g : fwd) launch(g, stream, true);
    }

    void backward(const float* y_dev, int n) {
        MCK(cudaMemcpyAsync(yin.p, y_dev, (size_t)n * prm.n_out * 4, cudaMemcpyDefault, stream));
        MCK(cudaMemsetAsync(loss.p, 0, 4, stream));
        const int nl = prm.n_layers;
        const float scale = 2.0f / ((float)n * (float)prm.n_out);
        const dim3 grd((unsigned)(prm.n_out / SQ), (unsigned)(rows / SQ));
        launch_after(k_mse_grad, grd, 256, 0, stream, 1, true, (const float*)pred.p, (const float*)yin.p, n, (int)prm.n_out,
                     rows, scale, G[(size_t)nl - 1]->p, GT[(size_t)nl - 1]->p, loss.p);
        for (int l = nl - 1; l >= 0; --l) {
            if (!group_w) launch(bwd_w[(size_t)l], stream, true);
            if (l > 0) launch(bwd_x[(size_t)l - 1], stream, true);
        }
        if (group_w) launch_group<kMaxLayers>(bwd_w.data(), nl, stream, true);
        launch_after(k_bias_grad, dim3((unsigned)((bias_dev.total + 7) / 8)), 256, 0, stream, 1, true, bias_dev);
    }

    void adam() {
        ++step;
        const float b1 = prm.beta1, b2 = prm.beta2;
        const float c1 = 1.0f - (float)std::pow((double)b1, (double)step);
        const float c2 = 1.0f - (float)std::pow((double)b2, (double)step);
        launch_after(k_adam, dim3((unsigned)adam_dev.total), 256, 0, stream, 1, true, adam_dev,
                     AdamStep{prm.lr, b1, b2, prm.eps, c1, c2});
    }
};

namespace {

template <typename F>
int mguard(afd_mlp* m, F&& f) {
    try {
        f();
        return AFD_OK;
    } catch (const Err& e) {
        if (m) m->err = e.what();
        return e.code;
    } catch (const std::exception& e) {
        if (m) m->err = e.what();
        return AFD_ERR_STATE;
    }
}

thread_local std::string g_create_err;

// The wait-expired words of the synchronous GEMM calls: host memory that a
// kernel writes only when a wait expires, so that a call needs neither a
// clearing launch nor a copy back. Never destroyed: a thread may outlive main.
int* mapped_word() {
    int* w = nullptr;
    MCK(cudaHostAlloc((void**)&w, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
    return w;
}
afd::WaitFlags& gemm_flags() {
    static afd::WaitFlags* flags = new afd::WaitFlags(mapped_word);
    return *flags;
}

}  // namespace

extern "C" {

void afd_mlp_default_params(afd_mlp_params* p) {
    std::memset(p, 0, sizeof(*p));
    p->n_in = 10;
    p->n_freq = 128;
    p->hidden = 512;
    p->n_layers = 5;
    p->n_out = 2048;
    p->batch = 1024;
    p->device = 0;
    p->fourier_sigma = 1.0f;
    p->seed = 1;
    p->lr = 1e-3f;
    p->beta1 = 0.9f;
    p->beta2 = 0.999f;
    p->eps = 1e-8f;
}

int afd_mlp_create(afd_mlp** out, const afd_mlp_params* p) {
    if (!out || !p) return AFD_ERR_ARG;
    *out = nullptr;
    afd_mlp* m = new afd_mlp;
    m->prm = *p;
    const int st = mguard(m, [&] { m->build(); });
    if (st != AFD_OK) {
        g_create_err = m->err;
        delete m;
        return st;
    }
    *out = m;
    return AFD_OK;
}

void afd_mlp_destroy(afd_mlp* m) { delete m; }

const char* afd_mlp_last_error(const afd_mlp* m) { return m ? m->err.c_str() : g_create_err.c_str(); }

int afd_mlp_set_stream(afd_mlp* m, void* stream) {
    if (!m) return AFD_ERR_ARG;
    return mguard(m, [&] {
        MCK(cudaStreamSynchronize(m->stream));
        m->stream = stream ? (cudaStream_t)stream : m->own;
    });
}

int afd_mlp_train_step(afd_mlp* m, const float* x, const float* y, int32_t n, float* loss) {
    if (!m || !x || !y) return AFD_ERR_ARG;
    return mguard(m, [&] {
        MCK(cudaSetDevice(m->device));
        m->features(x, n);
        m->forward();
        m->backward(y, n);
        m->adam();
        if (loss) {
            float s = 0.0f;
            MCK(cudaMemcpyAsync(&s, m->loss.p, 4, cudaMemcpyDeviceToHost, m->stream));
            m->check_flag();
            *loss = s / ((float)n * (float)m->prm.n_out);
        }
    });
}

int afd_mlp_gradients(afd_mlp* m, const float* x, const float* y, int32_t n, float* loss) {
    if (!m || !x || !y) return AFD_ERR_ARG;
    return mguard(m, [&] {
        MCK(cudaSetDevice(m->device));
        m->features(x, n);
        m->forward();
        m->backward(y, n);
        float s = 0.0f;
        MCK(cudaMemcpyAsync(&s, m->loss.p, 4, cudaMemcpyDeviceToHost, m->stream));
        m->check_flag();
        if (loss) *loss = s / ((float)n * (float)m->prm.n_out);
    });
}

int afd_mlp_predict(afd_mlp* m, const float* x, int32_t n, float* out) {
    if (!m || !x || !out) return AFD_ERR_ARG;
    return mguard(m, [&] {
        MCK(cudaSetDevice(m->device));
        m->features(x, n);
        m->forward();
        MCK(cudaMemcpyAsync(out, m->pred.p, (size_t)n * m->prm.n_out * 4, cudaMemcpyDefault, m->stream));
        m->check_flag();
    });
}

int afd_mlp_sync(afd_mlp* m) {
    if (!m) return AFD_ERR_ARG;
    return mguard(m, [&] { m->check_flag(); });
}

int afd_mlp_get(afd_mlp* m, int32_t what, int32_t layer, float* out, int64_t cap) {
    if (!m || !out) return AFD_ERR_ARG;
    return mguard(m, [&] {
        MCK(cudaSetDevice(m->device));
        MCK(cudaStreamSynchronize(m->stream));
        if (what == AFD_MLP_FOURIER) {
            if (cap < (int64_t)m->fourier.n) throw Err(AFD_ERR_ARG, "output buffer too small");
            MCK(cudaMemcpy(out, m->fourier.p, m->fourier.n * 4, cudaMemcpyDeviceToHost));
            return;
        }
        if (what == AFD_MLP_FEATURES) {
            const size_t n = (size_t)m->rows * m->F;
            if (cap < (int64_t)n) throw Err(AFD_ERR_ARG, "output buffer too small");
            std::vector<bf16> h(n);
            MCK(cudaMemcpy(h.data(), m->feat.p, n * 2, cudaMemcpyDeviceToHost));
            for (size_t i = 0; i < n; ++i) out[i] = __bfloat162float(h[i]);
            return;
        }
        if (layer < 0 || layer >= (int)m->L.size()) throw Err(AFD_ERR_ARG, "layer index out of range");
        Layer& ly = *m->L[(size_t)layer];
        const Dev<float>* src = what == AFD_MLP_WEIGHT ? &ly.w : what == AFD_MLP_BIAS ? &ly.b
                                : what == AFD_MLP_GRAD_WEIGHT ? &ly.gw : what == AFD_MLP_GRAD_BIAS ? &ly.gb : nullptr;
        if (!src) throw Err(AFD_ERR_ARG, "unknown tensor");
        if (cap < (int64_t)src->n) throw Err(AFD_ERR_ARG, "output buffer too small");
        MCK(cudaMemcpy(out, src->p, src->n * 4, cudaMemcpyDeviceToHost));
    });
}

int afd_mlp_set_weights(afd_mlp* m, int32_t layer, const float* w, const float* b) {
    if (!m || !w || !b) return AFD_ERR_ARG;
    return mguard(m, [&] {
        MCK(cudaSetDevice(m->device));
        if (layer < 0 || layer >= (int)m->L.size()) throw Err(AFD_ERR_ARG, "layer index out of range");
        Layer& ly = *m->L[(size_t)layer];
        MCK(cudaMemcpyAsync(ly.w.p, w, ly.w.n * 4, cudaMemcpyHostToDevice, m->stream));
        MCK(cudaMemcpyAsync(ly.b.p, b, ly.b.n * 4, cudaMemcpyHostToDevice, m->stream));
        m->refresh_bf16(layer);
        MCK(cudaStreamSynchronize(m->stream));
    });
}

int afd_gemm_bf16_async(const void* a, const void* b, float* c, int32_t M, int32_t N, int32_t K, void* stream,
                        int32_t* status) {
    try {
        if (!a || !b || !c || !status) throw Err(AFD_ERR_ARG, "null pointer");
        Gemm g = make_gemm(EPI_F32, (const bf16*)a, (const bf16*)b, M, N, K, status, true);
        g.o.c32 = c;
        g.o.ldc = N;
        launch(g, (cudaStream_t)stream);
        return AFD_OK;
    } catch (const Err& e) {
        g_create_err = e.what();
        return e.code;
    } catch (const std::exception& e) {
        g_create_err = e.what();
        return AFD_ERR_STATE;
    }
}

int afd_gemm_bf16(const void* a, const void* b, float* c, int32_t M, int32_t N, int32_t K, void* stream) {
    try {
        if (!a || !b || !c) throw Err(AFD_ERR_ARG, "null pointer");
        int dev = 0;
        MCK(cudaGetDevice(&dev));
        if (dev < 0 || dev >= 64) throw Err(AFD_ERR_ARG, "device ordinal out of range");
        afd::WaitFlags::Lease flag(gemm_flags());
        int* mapped = nullptr;
        MCK(cudaHostGetDevicePointer((void**)&mapped, flag.word(), 0));
        Gemm g = make_gemm(EPI_F32, (const bf16*)a, (const bf16*)b, M, N, K, mapped, true);
        g.o.c32 = c;
        g.o.ldc = N;
        cudaStream_t st = (cudaStream_t)stream;
        launch(g, st);
        MCK(cudaStreamSynchronize(st));
        if (flag.raised()) throw Err(AFD_ERR_CUDA, "GEMM pipeline wait timed out");
        return AFD_OK;
    } catch (const Err& e) {
        g_create_err = e.what();
        return e.code;
    } catch (const std::exception& e) {
        g_create_err = e.what();
        return AFD_ERR_STATE;
    }
}

}  // extern "C"
