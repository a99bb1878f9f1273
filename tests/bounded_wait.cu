// What the waits of the tensor-core kernels do when nothing arrives: one barrier and one thread per case, for test_gpu_bounded_wait.py.
#include <cstdio>

#include "dense_gemm.cuh"
using namespace lmrs;
using namespace lmrs::dense;

// case 0: nothing arrives | 1: the barrier's phase has ended | 2: nothing arrives, but another role has given up
static __global__ void wait_kernel(int which, int* out, unsigned long long* ns) {
    __shared__ __align__(8) uint64_t bar;
    __shared__ volatile int abort_flag;
    mbar_init(&bar, 1);
    fence_barrier_init();
    abort_flag = which == 2 ? TG_PAIR + TG_SUMS : 0;
    if (which == 1) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bar)) : "memory");
    unsigned long long a, b;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(a));
    out[0] = mbar_wait_bounded(&bar, 0, &abort_flag, TG_ATTENTION + TG_SCORES);
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(b));
    out[1] = abort_flag;
    *ns = b - a;
}

int main() {
    int *out, res[2];
    unsigned long long *ns, took;
    if (cudaMalloc(&out, 8) != cudaSuccess || cudaMalloc(&ns, 8) != cudaSuccess) return 1;
    for (int which = 0; which < 3; which++) {
        wait_kernel<<<1, 1>>>(which, out, ns);
        if (cudaMemcpy(res, out, 8, cudaMemcpyDeviceToHost) != cudaSuccess || cudaMemcpy(&took, ns, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
        printf("%d|%llu|%s\n", res[0], took / 1000000, res[1] ? tg_gave_up(res[1]).c_str() : "");
    }
    return 0;
}
