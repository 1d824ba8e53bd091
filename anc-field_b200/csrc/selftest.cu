// Self-tests of the bounded device waits. afd_wait_selftest: one block
// waits on a shared-memory mbarrier with the streaming kernel's wait
// (fused.cuh, which = 0) or the GEMM kernels' wait (tc.cuh, which = 1).
// With `complete` = 0 nothing ever arrives on the barrier, so the wait gives
// up at its time limit; the kernel records that and the time it waited and
// returns normally, so the host reads a status and the context stays usable.
// afd_barrier_selftest: the same with the grid barrier (sync.cuh), which waits
// for one more block than there is, beside copies to shared memory in flight as
// the LMS kernel has them.
#include <cuda_runtime.h>

#include "afd.h"
#include "fused.cuh"
#include "sync.cuh"
#include "tc.cuh"

namespace afd {
namespace {

__global__ void k_wait_selftest(int which, int complete, unsigned long long* out) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (complete) mbar_arrive(&bar);
    const unsigned long long t0 = global_ns();
    const bool ok = which == 0 ? mbar_wait(&bar, 0) : tc::bar_wait(&bar, 0);
    out[0] = ok ? 0ull : 1ull;
    out[1] = global_ns() - t0;
}

// out: time waited, threads told that the barrier gave up, copied words that
// arrived
constexpr int kBarThreads = 64;
__global__ void __launch_bounds__(kBarThreads) k_barrier_selftest(unsigned int target, unsigned int* bar, int* flag,
                                                                  const int* words, unsigned long long* out) {
    __shared__ __align__(16) int copy[kBarThreads];
    copy[threadIdx.x] = 0;
    __syncthreads();
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(copy + threadIdx.x)),
                 "l"(words + threadIdx.x)
                 : "memory");
    const unsigned long long t0 = global_ns();
    const bool ok = grid_barrier(bar, target, flag);
    if (threadIdx.x == 0) out[0] = global_ns() - t0;
    copies_landed();
    if (!ok) atomicAdd(out + 1, 1ull);
    if (copy[threadIdx.x] == (int)threadIdx.x + 1) atomicAdd(out + 2, 1ull);
}

}  // namespace
}  // namespace afd

extern "C" int afd_wait_selftest(int32_t device, int32_t which, int32_t complete, int32_t* timed_out,
                                 int64_t* waited_ns) {
    if ((which != 0 && which != 1) || !timed_out || !waited_ns) return AFD_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return AFD_ERR_CUDA;
    if (device < 0 || device >= ndev) return AFD_ERR_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return AFD_ERR_CUDA;
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, 2 * sizeof(unsigned long long)) != cudaSuccess) return AFD_ERR_CUDA;
    afd::k_wait_selftest<<<1, 32>>>(which, complete != 0, d);
    unsigned long long h[2] = {0ull, 0ull};
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return AFD_ERR_CUDA;
    *timed_out = (int32_t)h[0];
    *waited_ns = (int64_t)h[1];
    return AFD_OK;
}

extern "C" int afd_barrier_selftest(int32_t device, int32_t complete, int32_t* timed_out, int64_t* waited_ns) {
    if (!timed_out || !waited_ns) return AFD_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return AFD_ERR_CUDA;
    if (device < 0 || device >= ndev) return AFD_ERR_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return AFD_ERR_CUDA;
    struct Work {
        unsigned long long out[3];
        unsigned int bar;
        int flag;
        int words[afd::kBarThreads];
    } h{};
    for (int k = 0; k < afd::kBarThreads; ++k) h.words[k] = k + 1;
    Work* d = nullptr;
    if (cudaMalloc(&d, sizeof(Work)) != cudaSuccess) return AFD_ERR_CUDA;
    cudaError_t e = cudaMemcpy(d, &h, sizeof(h), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        afd::k_barrier_selftest<<<1, afd::kBarThreads>>>(complete ? 1u : 2u, &d->bar, &d->flag, d->words, d->out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return AFD_ERR_CUDA;
    // told to every thread or to none, with the flag that the host reads
    const bool gave_up = h.out[1] != 0;
    if ((gave_up && h.out[1] != (unsigned long long)afd::kBarThreads) || gave_up != ((h.flag & 2) != 0) ||
        h.out[2] != (unsigned long long)afd::kBarThreads)
        return AFD_ERR_STATE;
    *timed_out = gave_up ? 1 : 0;
    *waited_ns = (int64_t)h.out[0];
    return AFD_OK;
}
