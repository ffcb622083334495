// A launch that the runtime refuses (blocks of 2000 threads): launch_early returns the error and leaves none behind
// for the next launch's check.
#include <stdio.h>

#include "qcb_ops.h"

__global__ void k_nothing() {}

int main() {
    const cudaError_t e = qcb::launch_early(k_nothing, 1u, 2000u, (cudaStream_t)0);
    const cudaError_t left = cudaPeekAtLastError();
    printf("%s %s\n", cudaGetErrorName(e), cudaGetErrorName(left));
    return e != cudaSuccess && left == cudaSuccess ? 0 : 1;
}
