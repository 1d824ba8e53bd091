// The estimator's recursion by forward substitution, block by block: the path of
// the calls whose explicit inverses have large entries (kMaxEntry), or leave the
// range of FP64 where the recursion itself stays in it because its errors are zero
// or small. Included by lms.cu inside namespace afd::lms. Per block of 128 samples
//   k_lms_y0     y0 for the block, taps and samples split over CTAs
//                (partial sums per tap chunk)
//   k_lms_solve  one CTA: y0 from the partials, R by lag, the errors
//   k_lms_update w_j <- w_j + (2 mu e_m) x_{m-j} in sample order, per tap
// 35 us per 128 samples at 64000 taps, of which the substitution on one CTA 21;
// with the inverses 3.7.
#pragma once

namespace subst {

constexpr int B = 128;       // samples per block
constexpr int J = 4096;      // taps per CTA of k_lms_y0
constexpr int SPC = 16;      // samples per CTA of k_lms_y0 (16 x 8 = 128 CTAs at 64000 taps)
constexpr int Y0_THREADS = 256;
constexpr size_t Y0_SMEM = (size_t)(2 * J + SPC) * sizeof(double);

// CTA (c, g): taps j0 = c J .. j0 + J - 1 of samples k0 + g SPC .. +SPC-1.
// xs[o + t] = x_t for 0 <= t < steps, zero elsewhere; what would lie in front of xs is zero too.
__global__ void __launch_bounds__(Y0_THREADS) k_lms_y0(const double* __restrict__ w, const double* __restrict__ xs,
                                                       int64_t o, int N, int64_t k0, int nb, double* partial) {
    extern __shared__ double y0_smem[];
    double* ws = y0_smem;      // [J]
    double* xw = ws + J;       // [J + SPC - 1]
    const int j0 = blockIdx.x * J, s0 = blockIdx.y * SPC;
    if (s0 >= nb) return;  // whole CTA
    const int nj = min(J, N - j0);
    for (int t = threadIdx.x; t < nj; t += blockDim.x) ws[t] = w[j0 + t];
    // x_{k-j} for k in [k0+s0, k0+s0+SPC), j in [j0, j0+J): xw[q] = x_{k0+s0-j0-(J-1)+q}
    const int64_t base = o + k0 + s0 - j0 - (J - 1);
    for (int t = threadIdx.x; t < J + SPC - 1; t += blockDim.x) xw[t] = base + t >= 0 ? xs[base + t] : 0.0;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = warp; i < SPC && s0 + i < nb; i += Y0_THREADS / 32) {
        double acc = 0.0;
        // x_{k0+s0+i-j0-jj} = xw[(J - 1) + i - jj]
        for (int jj = lane; jj < nj; jj += 32) acc += ws[jj] * xw[(J - 1) + i - jj];
        for (int s = 16; s > 0; s >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, s);
        if (lane == 0) partial[(size_t)blockIdx.x * B + s0 + i] = acc;
    }
}

// One CTA of B threads. r_state[l]: r_l at the last sample of the previous
// block (zero at the start of a pass). The two windows of x the lag sums
// read (x_{k0 ..}, x_{k0-N ..}, 2 B - 1 values each) are staged in shared
// memory first, so the sequential sums wait on shared, not global, loads.
constexpr int XW = 2 * B;  // window length (2 B - 1 used)
constexpr size_t SOLVE_SMEM = (size_t)(B * B + 3 * B + 2 * XW) * sizeof(double);
__global__ void __launch_bounds__(B) k_lms_solve(const double* __restrict__ xs, int64_t o, int N, int64_t k0,
                                                 int nb, const double* __restrict__ partial, int nchunk,
                                                 const double* __restrict__ d, double mu, double* r_state,
                                                 double* e_out) {
    extern __shared__ double smem[];
    double* R = smem;          // R[i * B + l] = r_l(k0 + i)
    double* y0 = R + B * B;    // [B]
    double* e = y0 + B;        // [B]
    double* xa = e + B;        // [XW]: x_{k0 + q}
    double* xb = xa + XW;      // [XW]: x_{k0 - N + q}
    double* dd = xb + XW;      // [B]: d_{k0 + i}
    const int t = threadIdx.x;
    for (int q = t; q < nb + B - 1; q += B) {
        xa[q] = xs[o + k0 + q];
        xb[q] = xs[o + k0 - N + q];
    }
    if (t < nb) {
        dd[t] = d[k0 + t];
        // the partials in chunk order; unrolled so that the loads overlap
        double s = 0.0;
        int c = 0;
        for (; c + 8 <= nchunk; c += 8) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = partial[(size_t)(c + u) * B + t];
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
        }
        for (; c < nchunk; ++c) s += partial[(size_t)c * B + t];
        y0[t] = s;
    }
    __syncthreads();
    if (t >= 1) {
        double r = r_state[t];
        for (int i = 0; i < nb; ++i) {
            r += xa[i] * xa[i + t] - xb[i] * xb[i + t];
            R[i * B + t] = r;
        }
        r_state[t] = r;
    }
    __syncthreads();
    // e_i = d_i - (y0_i + 2 mu sum_{m<i} e_m R(m, i)), forward substitution
    // by one warp over sub-blocks of 32 samples: lane j of a sub-block first
    // takes the earlier sub-blocks' errors, then each error of its own
    // sub-block as the owning lane finalises it (one shuffle per sample);
    // every sum runs in sample order.
    if (t < 32) {
        const double c2 = 2 * mu;
        for (int b0 = 0; b0 < nb; b0 += 32) {
            const int j = b0 + t;
            double acc = 0.0;
            if (j < nb)
                for (int m = 0; m < b0; ++m) acc += e[m] * R[m * B + (j - m)];
            const int b1 = min(b0 + 32, nb);
            for (int i = b0; i < b1; ++i) {
                double ei = 0.0;
                if (j == i) {
                    ei = dd[i] - (y0[i] + c2 * acc);
                    e[i] = ei;
                }
                ei = __shfl_sync(0xffffffffu, ei, i - b0);
                if (j > i && j < nb) acc += ei * R[i * B + (j - i)];
            }
            __syncwarp();
        }
    }
    __syncthreads();
    if (t < nb) e_out[t] = e[t];
}

// w_j <- w_j + (2 mu e_m) x_{m-j} for the block's samples in order. The
// CTA's taps j0 .. j0+255 read x_{k0-j0-255} .. x_{k0-j0+nb-1}, staged in
// shared memory first.
constexpr int UPD_THREADS = 256;
__global__ void __launch_bounds__(UPD_THREADS) k_lms_update(double* w, const double* __restrict__ xs, int64_t o,
                                                            int N, int64_t k0, int nb,
                                                            const double* __restrict__ e_in, double mu) {
    __shared__ double c[B];
    __shared__ double win[UPD_THREADS + B];
    const int tid = threadIdx.x;
    const int j0 = blockIdx.x * UPD_THREADS;
    if (tid < nb) c[tid] = 2 * mu * e_in[tid];
    const int64_t base = o + k0 - j0 - (UPD_THREADS - 1);
    for (int q = tid; q < UPD_THREADS - 1 + nb; q += UPD_THREADS) win[q] = xs[base + q];
    __syncthreads();
    const int j = j0 + tid;
    if (j >= N) return;
    double v = w[j];
    const double* xp = win + (UPD_THREADS - 1 - tid);  // xp[i] = x_{k0 + i - j}
    for (int i = 0; i < nb; ++i) v = v + c[i] * xp[i];
    w[j] = v;
}

}  // namespace subst
