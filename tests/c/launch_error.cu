// launch_error.cu -- a launch that the runtime refuses.
//
// launch_dep (spike_common.cuh) returns an error for it and must leave CUDA's
// last error clean, since the next launch reads it in its own check.  The
// runtime's launch and error state are stand-ins here (linked with --wrap), so
// no GPU is needed.  Built by tests/test_launch_error.py; test code only.
#include <stdio.h>

#include "spike_common.cuh"

static cudaError_t last = cudaSuccess;
extern "C" cudaError_t __wrap_cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **)
{
    return last = cudaErrorInvalidConfiguration;
}
extern "C" cudaError_t __wrap_cudaGetLastError()
{
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}

__global__ void k_nothing() {}

int main()
{
    const int rc = launch_dep(k_nothing, dim3(1), 4096, 0, 1, true, 0);
    printf("rc %d, left %d\n", rc, (int)last);
    return rc == SPK_ECUDA && last == cudaSuccess ? 0 : 1;
}
