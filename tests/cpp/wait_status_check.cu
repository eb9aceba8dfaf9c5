// A bounded wait that runs out in one warp after the others have gone through their roles: the CTA still reports it.
// Prints the status word.
#include <cstdio>

#include "lev_internal.h"
#include "lev_umma.cuh"

__global__ void k_one_waits(int* status, int wait) {
    __shared__ __align__(8) unsigned long long bar;
    __shared__ int abort_s;
    if (threadIdx.x == 0) {
        abort_s = 0;
        mbar_init(smem_u32(&bar), 1);
    }
    __syncthreads();
    volatile int* abort_flag = &abort_s;
    if (wait && threadIdx.x >= 32) pk_wait(smem_u32(&bar), 0u, abort_flag);   // nothing arrives: about a second
    pk_finish(abort_flag, status, LEV_DEV_TIMEOUT);
}

int main() {
    int *d, h[2] = {-1, -1};
    if (cudaMalloc(&d, 2 * sizeof(int)) != cudaSuccess || cudaMemset(d, 0, 2 * sizeof(int)) != cudaSuccess) return 1;
    k_one_waits<<<1, 64>>>(d, 0);
    k_one_waits<<<1, 64>>>(d + 1, 1);
    if (cudaMemcpy(h, d, 2 * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    printf("%d %d\n", h[0], h[1]);
    return 0;
}
