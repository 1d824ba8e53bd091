// LMS impulse-response estimation on the GPU: the estimator of
// anc_field_py/ancutil.py:24-37 (EstimateIr), which the reference runs as a
// Python loop over samples ("takes hours" for the 10 s, 64000-tap case).
//
// The reference's recursion, per pass over the samples (delay line u
// cleared at the start of each pass, weights w kept):
//     u <- [x_k, u_0 .. u_{N-2}],  e_k = d_k - w.u,  w <- w + (2 mu e_k) u.
// Over a block of B samples k0 .. k0+B-1 the weights seen by sample k are
// the block-start weights plus the updates of the block's earlier samples,
// so  e_k = d_k - (y0_k + 2 mu sum_{m<k} e_m R(m, k))  with
//   y0_k = sum_j w_j x_{k-j}                 (block-start weights)
//   R(m, k) = sum_{j<N} x_{m-j} x_{k-j}       (sliding-window correlation)
// and R(m, m+l) = r_l(m) follows from r_l(m-1) by adding x_m x_{m+l} and
// removing x_{m-N} x_{m+l-N}. In matrix form (I + 2 mu L) e = d - y0 with the
// strictly lower triangular L_km = R(m, k). The matrix follows from x alone:
// it is the same in every pass, and the blocks' matrices do not depend on one
// another. So all inverses are formed first, in parallel,
//   k_lms_lags<0>  sums of the r_l increments per block
//   k_lms_scan     their running sums: r_l at the block starts
//   k_lms_lags<1>  the matrices, column by column
//   k_lms_diag     inverses of the 32 x 32 diagonal blocks
//   k_lms_inverse  the inverses, 32 columns a CTA, by block substitution
// and what stays sequential is one cooperative kernel over the blocks, k_lms_pass:
// weight update by the last block's errors, y0, and e = M (d - y0). Where an
// inverse has an entry above kMaxEntry, the call runs by substitution instead
// (lms_subst.cuh). All arithmetic is FP64, as in the reference.
#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/afd_lms.h"
#include "sync.cuh"

namespace afd {
namespace lms {

constexpr int B = 512;          // samples per block
constexpr int NB = B / 32;      // 32-sample blocks of it
constexpr int kTri = 1024 * NB * (NB + 1) / 2;  // packed inverse: row block i keeps (i + 1) 32 columns
constexpr int P_THREADS = 512;  // k_lms_pass
constexpr int P_WARPS = P_THREADS / 32;
constexpr int kRowSets = B / 4;  // sets of 4 samples and 4 inverse rows dealt to the CTAs
// Bits of the flag word (grid_barrier raises 2): an entry of an inverse is larger
// than kMaxEntry or not a number. Entries tell how far an error of one sample grows
// within the block; sums over 512 samples that grow and fall again lose that much,
// where those over 128 of the substitution lose less and the recursion itself
// forgets. Against extended precision (relative; 3000 samples of white noise, mu x
// taps x power 0.5 to 1.2, in turn the block inverses and substitution): entries up to
// 3: 1e-16 to 1e-14, both alike; up to 100: alike within a factor of 2; 700 with 32
// taps 7e-13 and 1e-13; 2400 with 4 taps 2e-11 and 7e-13; 6e4 with 2 taps, converged,
// 4e-8 and 5e-13. Few taps near the stable limit come here (4 taps from 0.7 on),
// 100 taps not below 1.2.
constexpr int kFlagInverse = 4;
constexpr double kMaxEntry = 64.0;

// r_l over the samples of block n0 + blockIdx.x, thread l (0 < l < B).
// WRITE = 0: the sum of the increments into r[n][l]. WRITE = 1: from r[n][l]
// at the block's start, the matrix I + 2 mu L below the diagonal, column m
// at tri[blockIdx.x][m B + k] (consecutive threads store consecutive rows).
template <int WRITE>
__global__ void __launch_bounds__(B) k_lms_lags(const double* __restrict__ xs, int64_t o, int N, int64_t n0,
                                                double mu2, double* r, double* tri) {
    __shared__ double xa[2 * B], xb[2 * B];
    const int64_t n = n0 + blockIdx.x, k0 = n * B;
    const int l = threadIdx.x;
    for (int q = l; q < 2 * B; q += B) {
        xa[q] = xs[o + k0 + q];
        xb[q] = xs[o + k0 - N + q];
    }
    __syncthreads();
    double s = WRITE ? r[n * B + l] : 0.0;
    double* t = WRITE ? tri + (size_t)blockIdx.x * B * B + l : nullptr;
#pragma unroll 8
    for (int i = 0; i < B; ++i) {
        s = fma(xa[i], xa[i + l], s);
        s = fma(-xb[i], xb[i + l], s);
        if (WRITE && l > 0 && i + l < B) t[(size_t)i * B + i] = mu2 * s;
    }
    if (!WRITE) r[n * B + l] = s;
}

// Block sums -> values at the block starts, per lag.
__global__ void k_lms_scan(double* r, int64_t nblocks) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    double s = 0.0;
    int64_t n = 0;
    for (; n + 8 <= nblocks; n += 8) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = r[(n + u) * B + l];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            r[(n + u) * B + l] = s;
            s += v[u];
        }
    }
    for (; n < nblocks; ++n) {
        const double v = r[n * B + l];
        r[n * B + l] = s;
        s += v;
    }
}

// Inverse of the unit lower triangular diagonal block i = blockIdx.x of block
// blockIdx.y, lane c one column, stored column by column.
__global__ void __launch_bounds__(32) k_lms_diag(const double* __restrict__ tri, double* diag) {
    __shared__ double t[32][32];  // [column][row]
    const int i = blockIdx.x, c = threadIdx.x;
    const double* p = tri + (size_t)blockIdx.y * B * B + (size_t)(32 * i) * B + 32 * i;
    for (int q = 0; q < 32; ++q) t[q][c] = c > q ? p[(size_t)q * B + c] : 0.0;
    __syncwarp();
    double x[32];
#pragma unroll
    for (int r = 0; r < 32; ++r) {
        double s = r == c ? 1.0 : 0.0;
#pragma unroll
        for (int q = 0; q < r; ++q) s = fma(-t[q][r], x[q], s);
        x[r] = s;
    }
    double* out = diag + ((size_t)blockIdx.y * NB + i) * 1024 + c * 32;
#pragma unroll
    for (int r = 0; r < 32; ++r) out[r] = x[r];
}

// 32 columns of the inverse, panel j of block g: X_i = D_i (E_i - sum_{j<=k<i}
// T_ik X_k) for i = j .. NB-1, X in shared memory, the T and D tiles
// streamed through two buffers. The longest panels (j = 0) come first. Entries
// above kMaxEntry raise kFlagInverse.
constexpr int I_THREADS = 256;
constexpr size_t I_SMEM = (size_t)(B * 32 + 2 * 1024) * sizeof(double);
__global__ void __launch_bounds__(I_THREADS) k_lms_inverse(const double* __restrict__ tri,
                                                           const double* __restrict__ diag, int blocks, double* inv,
                                                           int* flag) {
    extern __shared__ double i_smem[];
    double* X = i_smem;         // [32 (i - j) + row][column]
    double* A = X + B * 32;     // [2][column][row]
    const int j = blockIdx.x / blocks, g = blockIdx.x % blocks, tid = threadIdx.x;
    const int r = tid >> 4 << 1, c = (tid & 15) << 1;  // the thread's 2 x 2 of a tile
    tri += (size_t)g * B * B;
    diag += (size_t)g * NB * 1024;
    inv += (size_t)g * kTri;
    double p[4];
    auto fetch = [&](int i, int k) {  // tile T_ik, or D_i for k = i
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int at = tid + u * I_THREADS;
            p[u] = k == i ? diag[(size_t)i * 1024 + at]
                          : tri[(size_t)(32 * k + (at >> 5)) * B + 32 * i + (at & 31)];
        }
    };
    fetch(j, j);
    int buf = 0;
    bool small = true;
    for (int i = j; i < NB; ++i) {
        double s[2][2];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < 2; ++v) s[u][v] = i == j && r + u == c + v ? 1.0 : 0.0;
        double* Xi = X + (size_t)(i - j) * 1024;
        for (int k = j; k <= i; ++k, buf ^= 1) {
            double* a = A + buf * 1024;
#pragma unroll
            for (int u = 0; u < 4; ++u) a[tid + u * I_THREADS] = p[u];
            if (k < i) fetch(i, k + 1);
            else if (i + 1 < NB) fetch(i + 1, j);
            const double* Xk = X + (size_t)(k - j) * 1024;
            if (k == i)
#pragma unroll
                for (int u = 0; u < 2; ++u) *reinterpret_cast<double2*>(Xi + (r + u) * 32 + c) = make_double2(s[u][0], s[u][1]);
            __syncthreads();
            double d[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 8
            for (int m = 0; m < 32; ++m) {
                const double2 t = *reinterpret_cast<const double2*>(a + m * 32 + r);
                const double2 x = *reinterpret_cast<const double2*>(Xk + m * 32 + c);
                d[0][0] = fma(t.x, x.x, d[0][0]);
                d[0][1] = fma(t.x, x.y, d[0][1]);
                d[1][0] = fma(t.y, x.x, d[1][0]);
                d[1][1] = fma(t.y, x.y, d[1][1]);
            }
            if (k < i) {
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int v = 0; v < 2; ++v) s[u][v] -= d[u][v];
            } else {
                __syncthreads();  // all have read S
                double* out = inv + 512 * i * (i + 1) + (size_t)r * 32 * (i + 1) + 32 * j + c;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const double2 v = make_double2(d[u][0], d[u][1]);
                    *reinterpret_cast<double2*>(Xi + (r + u) * 32 + c) = v;
                    *reinterpret_cast<double2*>(out + u * 32 * (i + 1)) = v;
                    small &= fabs(v.x) <= kMaxEntry && fabs(v.y) <= kMaxEntry;
                }
            }
        }
    }
    if (__any_sync(0xffffffffu, !small) && (tid & 31) == 0) atomicOr(flag, kFlagInverse);
}

struct PassArgs {
    const double* xs;   // xs[o + t] = x_t for 0 <= t < steps, zero elsewhere
    const double* d;    // zero from steps on
    const double* inv;  // packed inverses of blocks b0, b0 + 1, ...
    double* w;          // tiles of 32 T taps, zero from N on
    double* partial;    // [CTA][B]
    double* f;          // [B]: d - y0
    double* e;          // [B]
    unsigned int* bar;
    int* flag;
    int64_t o, steps, nblocks;
    int64_t a, b;       // steps of the recursion: block n mod nblocks for n = a .. b-1
    int64_t b0;
    double mu2;
    int N, tiles, last; // last: one more weight update at the end
};

__device__ __forceinline__ void copy8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// The sequential part: per block of B samples, each CTA over its tiles of
// 32 T taps adds the last block's updates to the weights and forms its share
// of y0 from them; after a grid barrier four samples a CTA are summed over the
// CTAs, after a second one four rows a CTA of the inverse give the errors, and
// a third ends the block.
//
// Both tap loops are Toeplitz products with one operand in registers: lane =
// tap (sample) mod 32, a warp takes residues `warp` and `warp + 16` of the
// other index, so x_{k-j} runs over 16 + T - 1 consecutive 32-strides, each
// loaded once for up to T products (conflict-free, lanes consecutive), and
// the warps' sums meet in shared memory.
//
// A block of 512 samples with 64000 taps takes 14.8 us: 65.5 M products at the
// FP64 rate are 3.6, the three barriers and the small sums between them 8 (9.1
// with 500 taps, where hardly a product is left). Larger blocks would save
// barriers and pay more for the inverses: 6.4 us a block at 512, growing with
// the square. One launch per stage over 128-sample blocks with a serial
// substitution measured 35.5 us per 128 samples; 64000 taps, 128000 samples, 4
// passes: 141 -> 17.3 ms a call.
template <int T>
constexpr size_t pass_smem() {
    return (size_t)(4 * (B + 32 * T) + P_WARPS * (B > 32 * T ? B : 32 * T) + 32 * T + B) * sizeof(double);
}
template <int T>
__global__ void __launch_bounds__(P_THREADS, 1) k_lms_pass(const __grid_constant__ PassArgs a) {
    constexpr int TJ = 32 * T, W = B + TJ;  // taps of a tile, window length
    constexpr int RED = B > TJ ? B : TJ;
    extern __shared__ double p_smem[];
    double* win = p_smem;             // [2][2][W]: windows of the update and of y0
    double* red = win + 4 * W;        // [P_WARPS][RED]
    double* ws = red + P_WARPS * RED; // [TJ]
    double* cs = ws + TJ;             // [B]: 2 mu e
    __shared__ double quad[P_WARPS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cta = blockIdx.x, G = gridDim.x, np = min(G, a.tiles);
    const int64_t end = a.b + a.last;
    // nothing to do with inverses that are not used (set by the launches before
    // this one, so alike for all CTAs)
    if (__ldcg(a.flag) & kFlagInverse) return;
    unsigned int raised = 0;
    auto prefetch = [&](int64_t n, int tile, int buf) {
        const int64_t bu = (n + a.nblocks - 1) % a.nblocks, by = n % a.nblocks;
        const double* u = a.xs + a.o + bu * B - (int64_t)(tile + 1) * TJ + 1;
        const double* y = a.xs + a.o + by * B - (int64_t)(tile + 1) * TJ + 1;
        double* dst = win + buf * 2 * W;
        for (int q = tid; q < W - 1; q += P_THREADS) {
            copy8(dst + q, u + q);
            copy8(dst + W + q, y + q);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto barrier = [&]() {
        raised += G;
        if (grid_barrier(a.bar, raised, a.flag)) return true;
        copies_landed();  // the next block's windows are on their way
        return false;
    };
    if (cta < a.tiles) prefetch(a.a, cta, 0);
    int buf = 0;
    for (int64_t n = a.a; n < end; ++n) {
        const bool update = n > 0, output = n < a.b;
        const int64_t blk = n % a.nblocks, k0 = blk * B;
        if (update) {
            const int64_t kp = (n - 1) % a.nblocks * B;
            cs[tid] = kp + tid < a.steps ? a.mu2 * __ldcg(a.e + tid) : 0.0;
        }
        double y[NB];
#pragma unroll
        for (int s = 0; s < NB; ++s) y[s] = 0.0;
        for (int tile = cta; tile < a.tiles; tile += G, buf ^= 1) {
            const int j = tile * TJ + tid;
            const double wv = tid < TJ ? a.w[j] : 0.0;
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            if (tile + G < a.tiles) prefetch(n, tile + G, buf ^ 1);
            else if (n + 1 < end) prefetch(n + 1, cta, buf ^ 1);
            if (update) {
                double u[T];
#pragma unroll
                for (int s = 0; s < T; ++s) u[s] = 0.0;
#pragma unroll 1
                for (int m0 = warp; m0 < 32; m0 += P_WARPS) {
                    const double* x = win + buf * 2 * W + m0 - lane + TJ - 1;
                    double v[NB + T - 1];
#pragma unroll
                    for (int s = 0; s < T - 1; ++s) v[s] = x[32 * (s - (T - 1))];
#pragma unroll
                    for (int t = 0; t < NB; ++t) {
                        v[t + T - 1] = x[32 * t];
                        const double c = cs[m0 + 32 * t];
#pragma unroll
                        for (int s = 0; s < T; ++s) u[s] = fma(c, v[t - s + T - 1], u[s]);
                    }
                }
#pragma unroll
                for (int s = 0; s < T; ++s) red[warp * RED + 32 * s + lane] = u[s];
                __syncthreads();
                if (tid < TJ) {
                    double v = 0.0;
#pragma unroll
                    for (int q = 0; q < P_WARPS; ++q) v += red[q * RED + tid];
                    v = j < a.N ? wv + v : 0.0;
                    ws[tid] = v;
                    a.w[j] = v;
                }
            } else if (tid < TJ) {
                ws[tid] = wv;
            }
            __syncthreads();
            if (output) {
#pragma unroll 1
                for (int i0 = warp; i0 < 32; i0 += P_WARPS) {
                    const double* x = win + (buf * 2 + 1) * W + lane - i0 + TJ - 1;
                    double v[NB + T - 1];
#pragma unroll
                    for (int s = 0; s < T - 1; ++s) v[s] = x[32 * (s - (T - 1))];
#pragma unroll
                    for (int s = 0; s < NB; ++s) {
                        v[s + T - 1] = x[32 * s];
#pragma unroll
                        for (int t = 0; t < T; ++t) y[s] = fma(ws[i0 + 32 * t], v[s - t + T - 1], y[s]);
                    }
                }
            }
        }
        if (!output) break;
        // the CTA's share of y0
        if (cta < np) {
            __syncthreads();
#pragma unroll
            for (int s = 0; s < NB; ++s) red[warp * RED + 32 * s + lane] = y[s];
            __syncthreads();
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < P_WARPS; ++q) v += red[q * RED + tid];
            a.partial[(size_t)cta * B + tid] = v;
        }
        // rows of the inverse: rows h, 255 - h, 256 + h, 511 - h of set h, four
        // warps a row; the first set is loaded ahead of the barriers
        const double* M = a.inv + (size_t)(blk - a.b0) * kTri;
        const int q = warp >> 2, col = (warp & 3) * 32 + lane;
        auto row_of = [&](int h) { return (q & 1) ? 256 * (q >> 1) + 255 - h : 256 * (q >> 1) + h; };
        double m[4];
        auto rows = [&](int h) {
            const int row = row_of(h), i = row >> 5;
            const double* p = M + 512 * i * (i + 1) + (size_t)(row & 31) * 32 * (i + 1);
#pragma unroll
            for (int u = 0; u < 4; ++u) m[u] = col + 128 * u < 32 * (i + 1) ? __ldg(p + col + 128 * u) : 0.0;
        };
        if (cta < kRowSets) rows(cta);
        if (!barrier()) return;
        for (int h = cta; h < kRowSets; h += G) {
            double v = 0.0;
            for (int c = tid >> 2; c < np; c += P_THREADS / 4) v += __ldcg(a.partial + (size_t)c * B + 4 * h + (tid & 3));
            for (int s = 16; s >= 4; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
            if (lane < 4) red[warp * 4 + lane] = v;
            __syncthreads();
            if (tid < 4) {
                v = 0.0;
#pragma unroll
                for (int p = 0; p < P_WARPS; ++p) v += red[p * 4 + tid];
                a.f[4 * h + tid] = __ldg(a.d + k0 + 4 * h + tid) - v;
            }
            __syncthreads();
        }
        if (!barrier()) return;
        for (int h = cta; h < kRowSets; h += G) {
            if (h != cta) rows(h);
            const int row = row_of(h);
            double v = 0.0;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                // a later sample takes no part, not even where its f is not finite
                const double f = __ldcg(a.f + col + 128 * u);
                v = fma(m[u], col + 128 * u <= row ? f : 0.0, v);
            }
            for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
            if (lane == 0) quad[warp] = v;
            __syncthreads();
            if (lane == 0 && (warp & 3) == 0)
                a.e[row] = (quad[warp] + quad[warp + 1]) + (quad[warp + 2] + quad[warp + 3]);
            __syncthreads();
        }
        if (!barrier()) return;
    }
}

struct Err : std::runtime_error {
    int code;
    Err(int cd, const std::string& m) : std::runtime_error(m), code(cd) {}
};

#define LCK(call)                                                                                   \
    do {                                                                                            \
        cudaError_t e__ = (call);                                                                   \
        if (e__ != cudaSuccess) throw Err(AFD_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e__)); \
    } while (0)

// Device memory of a call: one block of the device's pool, in stream order.
// The pool keeps what calls gave back, kPoolKeep at most (an estimate needs
// tens to hundreds of MB, and mapping and unmapping them took 5 to 60 ms a call
// beside 16 ms of kernels); the rest returns to the device at the next
// synchronization, and all that no call holds when another allocation of the
// process needs it or the caller says so (release).
constexpr uint64_t kPoolKeep = (uint64_t)1 << 30;
cudaMemPool_t device_pool(int device, bool make = true) {
    static std::mutex mu;
    static std::map<int, cudaMemPool_t> pools;
    std::lock_guard<std::mutex> hold(mu);
    auto it = pools.find(device);
    if (it != pools.end()) return it->second;
    if (!make) return nullptr;
    cudaMemPoolProps p{};
    p.allocType = cudaMemAllocationTypePinned;
    p.location.type = cudaMemLocationTypeDevice;
    p.location.id = device;
    cudaMemPool_t pool = nullptr;
    LCK(cudaMemPoolCreate(&pool, &p));
    uint64_t keep = kPoolKeep;
    LCK(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    return pools[device] = pool;
}
struct Block {
    char* p = nullptr;
    cudaStream_t st = nullptr;
    ~Block() {
        if (p) cudaFreeAsync(p, st);
    }
    bool alloc(size_t bytes, cudaMemPool_t pool, cudaStream_t stream) {
        st = stream;
        if (cudaMallocFromPoolAsync((void**)&p, bytes, pool, st) == cudaSuccess) return true;
        cudaGetLastError();
        p = nullptr;
        return false;
    }
};

// The call's own stream; everything on it has ended once it is gone.
struct Stream {
    cudaStream_t st = nullptr;
    Stream() { LCK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)); }
    ~Stream() {
        cudaStreamSynchronize(st);
        cudaStreamDestroy(st);
    }
};

thread_local std::string g_err;

#include "lms_subst.cuh"

// The whole recursion by substitution: w, zero on entry, from device inputs.
void substitute(const double* xs, int64_t o, const double* d, int64_t steps, int N, double mu, int epochs, double* w,
                int device, cudaStream_t st) {
    using namespace subst;
    const int nchunk = (N + J - 1) / J;
    Block mem;
    if (!mem.alloc(((size_t)nchunk + 2) * subst::B * sizeof(double), device_pool(device), st))
        throw Err(AFD_ERR_CUDA, "out of device memory");
    double* const partial = reinterpret_cast<double*>(mem.p);
    double* const r = partial + (size_t)nchunk * subst::B;
    double* const e = r + subst::B;
    LCK(cudaFuncSetAttribute((const void*)k_lms_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SOLVE_SMEM));
    LCK(cudaFuncSetAttribute((const void*)k_lms_y0, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Y0_SMEM));
    auto pass = [&]() {
        LCK(cudaMemsetAsync(r, 0, subst::B * sizeof(double), st));
        for (int64_t k0 = 0; k0 < steps; k0 += subst::B) {
            const int nb = (int)std::min<int64_t>(subst::B, steps - k0);
            k_lms_y0<<<dim3((unsigned)nchunk, (unsigned)((nb + SPC - 1) / SPC)), Y0_THREADS, Y0_SMEM, st>>>(
                w, xs, o, N, k0, nb, partial);
            k_lms_solve<<<1, subst::B, SOLVE_SMEM, st>>>(xs, o, N, k0, nb, partial, nchunk, d, mu, r, e);
            k_lms_update<<<(N + UPD_THREADS - 1) / UPD_THREADS, UPD_THREADS, 0, st>>>(w, xs, o, N, k0, nb, e, mu);
        }
        LCK(cudaGetLastError());
    };
    if (epochs < 2) {
        pass();
        return;
    }
    // every pass launches the same kernels with the same arguments: captured
    // once and replayed (16 passes of 20000 samples, 4 taps: 72 ms launched one by
    // one, 60 replayed)
    struct Graph {
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        ~Graph() {
            if (exec) cudaGraphExecDestroy(exec);
            if (graph) cudaGraphDestroy(graph);
        }
    } g;
    LCK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    try {
        pass();
    } catch (...) {
        cudaStreamEndCapture(st, &g.graph);  // leave the stream out of capture mode
        throw;
    }
    LCK(cudaStreamEndCapture(st, &g.graph));
    LCK(cudaGraphInstantiate(&g.exec, g.graph, 0));
    for (int ep = 0; ep < epochs; ++ep) LCK(cudaGraphLaunch(g.exec, st));
    LCK(cudaStreamSynchronize(st));
}

void estimate(const double* x, int64_t nx, const double* d, int64_t nd, int32_t taps, double mu, int32_t epochs,
              int32_t device, double* w_out) {
    if (!x || !d || !w_out) throw Err(AFD_ERR_ARG, "null pointer");
    if (taps < 1 || taps > (1 << 26)) throw Err(AFD_ERR_ARG, "taps must be in 1 .. 2^26");
    if (nx < 0 || nd < 0 || epochs < 0) throw Err(AFD_ERR_ARG, "negative length or epoch count");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) throw Err(AFD_ERR_CUDA, "no CUDA device available");
    if (device < 0 || device >= ndev) throw Err(AFD_ERR_ARG, "device ordinal out of range");
    LCK(cudaSetDevice(device));
    const int N = taps;
    const int64_t steps = std::min(nx, nd);
    if (steps == 0 || epochs == 0) {
        std::memset(w_out, 0, (size_t)N * sizeof(double));
        return;
    }
    int sms = 0;
    LCK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    // taps per tile: what the CTA with the most tiles walks, a tile costing its
    // taps and about a third of the largest tile's time for windows and sums
    int T = 1;
    double best = 0.0;
    for (int t : {1, 2, 4, 7, 14}) {
        const int64_t tiles = (N + 32 * t - 1) / (32 * t);
        const double cost = (double)((tiles + sms - 1) / sms) * (t + 4.0);
        if (best == 0.0 || cost < best) {
            best = cost;
            T = t;
        }
    }
    const int tiles = (N + 32 * T - 1) / (32 * T), Np = tiles * 32 * T;
    const int64_t nblocks = (steps + B - 1) / B;
    const int64_t o = (int64_t)Np + B;  // zeros in front of x_0
    const size_t nxs = (size_t)(o + (nblocks + 1) * B);
    std::vector<double> hx(nxs, 0.0);
    std::memcpy(hx.data() + o, x, (size_t)steps * sizeof(double));
    const int grid = std::min(sms, std::max(tiles, kRowSets));
    // Inverses of `seg` blocks at a time (1.1 MB each), formed `group` at a
    // time from their matrices (2.2 MB each): a GB in all; less where the
    // device has less to give. More blocks than one segment holds form their
    // inverses again in every pass.
    int64_t seg = std::min<int64_t>(nblocks, 768), group = std::min<int64_t>(seg, 64);
    const size_t tri_n = (size_t)B * B + NB * 1024;
    Stream stream;
    Block mem;
    cudaStream_t st = stream.st;
    const size_t fixed = (size_t)grid * B + 2 * B + (size_t)nblocks * B * 2 + nxs + (size_t)Np;
    for (;;) {
        if (mem.alloc((fixed + (size_t)seg * kTri + (size_t)group * tri_n + 1) * sizeof(double), device_pool(device),
                      st))
            break;
        if (seg == 1) throw Err(AFD_ERR_CUDA, "out of device memory");
        seg = (seg + 1) / 2;
        group = std::min(group, seg);
    }
    double* at = reinterpret_cast<double*>(mem.p);
    auto take = [&](size_t n) {
        double* p = at;
        at += n;
        return p;
    };
    double* const inv = take((size_t)seg * kTri);  // first: 16-byte aligned like all after it of even size
    double* const tri = take((size_t)group * tri_n);
    double* const diag = tri + (size_t)group * B * B;
    double* const xs = take(nxs);
    double* const dd = take((size_t)nblocks * B);
    double* const r = take((size_t)nblocks * B);
    double* const partial = take((size_t)grid * B);
    double* const fe = take(2 * B);
    double* const w = take((size_t)Np);
    int* const sync = reinterpret_cast<int*>(take(1));
    LCK(cudaMemsetAsync(w, 0, ((size_t)Np + 1) * sizeof(double), st));  // and `sync`
    LCK(cudaMemcpyAsync(xs, hx.data(), nxs * sizeof(double), cudaMemcpyHostToDevice, st));
    LCK(cudaMemcpyAsync(dd, d, (size_t)steps * sizeof(double), cudaMemcpyHostToDevice, st));
    LCK(cudaMemsetAsync(dd + steps, 0, (size_t)(nblocks * B - steps) * sizeof(double), st));
    LCK(cudaFuncSetAttribute((const void*)k_lms_inverse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)I_SMEM));
    k_lms_lags<0><<<(unsigned)nblocks, B, 0, st>>>(xs, o, N, 0, 2 * mu, r, nullptr);
    k_lms_scan<<<B / 32, 32, 0, st>>>(r, nblocks);
    // inverses of blocks b0 .. b0 + n - 1
    auto invert = [&](int64_t b0, int64_t n) {
        for (int64_t g = 0; g < n; g += group) {
            const int m = (int)std::min(group, n - g);
            k_lms_lags<1><<<m, B, 0, st>>>(xs, o, N, b0 + g, 2 * mu, r, tri);
            k_lms_diag<<<dim3(NB, m), 32, 0, st>>>(tri, diag);
            k_lms_inverse<<<m * NB, I_THREADS, I_SMEM, st>>>(tri, diag, m, inv + (size_t)g * kTri, sync + 1);
        }
        LCK(cudaGetLastError());
    };
    PassArgs a{};
    a.xs = xs;
    a.d = dd;
    a.inv = inv;
    a.w = w;
    a.partial = partial;
    a.f = fe;
    a.e = fe + B;
    a.bar = reinterpret_cast<unsigned int*>(sync);
    a.flag = sync + 1;
    a.o = o;
    a.steps = steps;
    a.nblocks = nblocks;
    a.mu2 = 2 * mu;
    a.N = N;
    a.tiles = tiles;
    auto run = [&](auto t) {
        constexpr int TT = decltype(t)::value;
        LCK(cudaFuncSetAttribute((const void*)k_lms_pass<TT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)pass_smem<TT>()));
        LCK(cudaMemsetAsync(a.bar, 0, sizeof(unsigned int), st));
        void* args[] = {&a};
        LCK(cudaLaunchCooperativeKernel((const void*)k_lms_pass<TT>, dim3(grid), dim3(P_THREADS), args,
                                        pass_smem<TT>(), st));
    };
    // blocks per launch: a launch stays below some seconds for any tap count
    const int64_t most = std::max<int64_t>(1, std::min<int64_t>(8192, ((int64_t)1 << 38) / ((int64_t)Np * 2 * B)));
    const int64_t total = nblocks * epochs;
    for (int64_t n = 0, have = -1; n < total;) {
        const int64_t s = n % nblocks / seg;
        if (s != have) invert(s * seg, std::min(seg, nblocks - s * seg));
        have = s;
        // up to the segment's end, or through the passes when there is one segment
        const int64_t stop = seg == nblocks ? total : std::min(n / nblocks * nblocks + (s + 1) * seg,
                                                               (n / nblocks + 1) * nblocks);
        a.a = n;
        a.b = std::min(stop, n + most);
        a.b0 = s * seg;
        a.last = a.b == total;
        switch (T) {
            case 1: run(std::integral_constant<int, 1>{}); break;
            case 2: run(std::integral_constant<int, 2>{}); break;
            case 4: run(std::integral_constant<int, 4>{}); break;
            case 7: run(std::integral_constant<int, 7>{}); break;
            default: run(std::integral_constant<int, 14>{}); break;
        }
        n = a.b;
    }
    LCK(cudaGetLastError());
    int flag = 0;
    LCK(cudaMemcpyAsync(&flag, a.flag, sizeof(int), cudaMemcpyDeviceToHost, st));
    LCK(cudaMemcpyAsync(w_out, w, (size_t)N * sizeof(double), cudaMemcpyDeviceToHost, st));
    LCK(cudaStreamSynchronize(st));
    if (flag & ~kFlagInverse) throw Err(AFD_ERR_CUDA, "a wait of the recursion kernel ran out");
    if (!flag) return;
    LCK(cudaMemsetAsync(w, 0, (size_t)Np * sizeof(double), st));
    substitute(xs, o, dd, steps, N, mu, epochs, w, device, st);
    LCK(cudaMemcpyAsync(w_out, w, (size_t)N * sizeof(double), cudaMemcpyDeviceToHost, st));
    LCK(cudaStreamSynchronize(st));
}

// Gives back what the device's pool keeps beyond the calls in progress.
void release(int32_t device) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) throw Err(AFD_ERR_CUDA, "no CUDA device available");
    if (device < 0 || device >= ndev) throw Err(AFD_ERR_ARG, "device ordinal out of range");
    if (cudaMemPool_t pool = device_pool(device, false)) LCK(cudaMemPoolTrimTo(pool, 0));
}

template <typename F>
int guard(F&& f) {
    try {
        f();
        return AFD_OK;
    } catch (const Err& e) {
        g_err = e.what();
        return e.code;
    } catch (const std::exception& e) {
        g_err = e.what();
        return AFD_ERR_STATE;
    }
}

}  // namespace lms
}  // namespace afd

extern "C" {

int afd_lms_estimate(const double* x, int64_t nx, const double* d, int64_t nd, int32_t taps, double mu,
                     int32_t epochs, int32_t device, double* w) {
    return afd::lms::guard([&] { afd::lms::estimate(x, nx, d, nd, taps, mu, epochs, device, w); });
}

int afd_lms_release(int32_t device) {
    return afd::lms::guard([&] { afd::lms::release(device); });
}

const char* afd_lms_last_error(void) { return afd::lms::g_err.c_str(); }

}  // extern "C"
