// Self-tests of the failure path of the bounded waits: a wait that runs out reports a status the host reads, and
// the context stays usable afterwards. No counterpart in the reference. The kernels wait through the same
// routines as the others: on an mbarrier that nothing arrives on (arrive = 0) or that the kernel has completed
// itself (arrive = 1), and, a warp of the chained plume kernel's kind, on progress that nobody publishes (0) or
// that one of its lanes does (1).
#include "chain_wait.cuh"
#include "common.cuh"
#include "tma.cuh"

namespace bd {

__global__ void k_selftest_wait(unsigned polls, int arrive, int* __restrict__ status) {
    __shared__ __align__(8) unsigned long long bar;
    if (threadIdx.x != 0) return;
    mbar_init(&bar, 1);
    mbar_init_fence();
    if (arrive) mbar_arrive(&bar);
    *status = mbar_wait_limit(&bar, 0, polls) ? 0 : 1;
}

// Lane l waits for plane l of its own progress word; the warp's vote and the error flag make the status.
__global__ void k_selftest_chain_wait(unsigned polls, int arrive, int* __restrict__ status, int* progress, int* err) {
    const int lane = threadIdx.x & 31;
    if (arrive && lane == 0)
        for (int l = 0; l < 32; ++l) st_release(progress + l, l + 1);
    __syncwarp();
    int seen = 0;
    bool ok = chain_wait(progress + lane, lane, seen, err, polls);
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) *status = ok && ld_acquire(err) == 0 ? 0 : !ok && ld_acquire(err) != 0 ? 1 : 2;
}

// The status word of a self-test as the call's result.
static int wait_result(const char* what, int host, int max_polls) {
    if (host == 1) return fail(BD_ERR_TIMEOUT, "%s: the bounded wait gave up after %d polls", what, max_polls);
    if (host != 0) return fail(BD_ERR_STATE, "%s: the kernel did not report", what);
    return BD_OK;
}

}  // namespace bd

using namespace bd;

extern "C" int bd_selftest_wait_timeout(int max_polls, int arrive, void* stream) {
    BD_REQUIRE(max_polls >= 1 && max_polls <= (1 << 20), "bd_selftest_wait_timeout: max_polls must be 1..2^20");
    cudaStream_t st = as_stream(stream);
    int* status = nullptr;
    BD_CUDA(cudaMallocAsync((void**)&status, sizeof(int), st));
    int host = -1;
    cudaError_t e = cudaMemsetAsync(status, 0xff, sizeof(int), st);
    if (e == cudaSuccess) {
        k_selftest_wait<<<1, 32, 0, st>>>((unsigned)max_polls, arrive ? 1 : 0, status);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&host, status, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaError_t e2 = cudaFreeAsync(status, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_status(e, "bd_selftest_wait_timeout");
    if (e2 != cudaSuccess) return cuda_status(e2, "bd_selftest_wait_timeout: cudaFreeAsync");
    return wait_result("bd_selftest_wait_timeout", host, max_polls);
}

extern "C" int bd_selftest_chain_wait_timeout(int max_polls, int arrive, void* stream) {
    BD_REQUIRE(max_polls >= 1 && max_polls <= (1 << 20), "bd_selftest_chain_wait_timeout: max_polls must be 1..2^20");
    cudaStream_t st = as_stream(stream);
    int* words = nullptr;   // the status, the error flag, 32 progress words
    BD_CUDA(cudaMallocAsync((void**)&words, 34 * sizeof(int), st));
    int host = -1;
    cudaError_t e = cudaMemsetAsync(words, 0, 34 * sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(words, 0xff, sizeof(int), st);
    if (e == cudaSuccess) {
        k_selftest_chain_wait<<<1, 32, 0, st>>>((unsigned)max_polls, arrive ? 1 : 0, words, words + 2, words + 1);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&host, words, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaError_t e2 = cudaFreeAsync(words, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return cuda_status(e, "bd_selftest_chain_wait_timeout");
    if (e2 != cudaSuccess) return cuda_status(e2, "bd_selftest_chain_wait_timeout: cudaFreeAsync");
    return wait_result("bd_selftest_chain_wait_timeout", host, max_polls);
}
