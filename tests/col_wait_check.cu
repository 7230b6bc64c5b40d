// The wait of a group of k_col_solve (colsolve.cuh) when it runs out: for some of the group's warps
// only, for all of them, for none.  Every thread must come to the same verdict and the kernel end.
#include <cstdio>

#include "../cfd_b200/csrc/colsolve.cuh"

using namespace cfd;

// scenario 0: the transfer has arrived, one warp has no tries left; 1: nothing arrives; 2: it has
// arrived and every warp sees it
__global__ void k_waits(int scenario, int* verdict) {
    __shared__ __align__(16) unsigned long long b[1];
    __shared__ int word[4];
    volatile int* gave = word;
    const unsigned bar = smem_u32(b);
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        for (int k = 0; k < 4; ++k) gave[k] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && scenario != 1) mbar_expect(bar, 0);
    __syncthreads();
    group_wait(bar, 0, scenario == 1 ? 16 : (scenario == 0 && threadIdx.x / 32 == 2 ? 0 : 1024), gave);
    __syncthreads();
    verdict[threadIdx.x] = gave[0];
}

int main() {
    int *d, h[128], bad = 0;
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return 2;
    for (int s = 0; s < 3; ++s) {
        k_waits<<<1, 128>>>(s, d);
        if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
        for (int t = 0; t < 128; ++t) bad += h[t] != (s < 2);
    }
    std::printf(bad ? "FAILED %d\n" : "OK\n", bad);
    return bad != 0;
}
