// emu_leave.cu -- the way out of the 64-row FP64 chains when a wait runs out.
//
// Three buffers as in k_emu_fwd (EmuBar, spike_emu64.cuh): the wait of the
// first runs out (its barrier counts a thread that never arrives), the copy of
// the second is in flight, the third is idle.  After emu_leave the error bit is
// set and the second copy has landed: its barrier's phase is over without
// another wait.  Built by tests/test_gpu_emu_leave.py; test code only.
#include "spike_emu64.cuh"

__global__ void __launch_bounds__(256) k_leave(const double *g, double *o, unsigned *err, int *out)
{
    constexpr int KB = 64, LD = KB + 2;
    extern __shared__ __align__(16) char sm[];
    uint64_t *bars = (uint64_t *)sm;
    double *s = (double *)(sm + 64);
    if (threadIdx.x == 0) {
        mbar_init(bars, 2); // one arrival short for ever
        mbar_init(bars + 1, 1);
        mbar_init(bars + 2, 1);
        mbar_init_fence();
    }
    __syncthreads();
    EmuBar<KB> a{bars, 0u, false}, b{bars + 1, 0u, false}, c{bars + 2, 0u, false};
    a.inflight = true;
    b.issue(s, LD, g);
    if (a.wait()) return;
    if (threadIdx.x == 0) out[0] = a.inflight && b.inflight && !c.inflight;
    emu_leave(err, a, b, c);
    if (threadIdx.x == 0) out[1] = mbar_try_wait(bars + 1, 0u);
    __syncthreads();
    for (int q = threadIdx.x; q < KB * KB; q += 256) o[q] = s[q / KB * LD + q % KB];
}

// returns 0 or the CUDA error code; h: 64 x 64 values there and back
extern "C" int leave_check(double *h, unsigned *herr, int *hout)
{
    constexpr int BYTES = 64 * 64 * 8, SM = 64 + 64 * 66 * 8;
    double *g = nullptr, *o = nullptr;
    unsigned *err = nullptr;
    int *out = nullptr;
    cudaError_t e = cudaMalloc(&g, BYTES);
    if (e == cudaSuccess) e = cudaMalloc(&o, BYTES);
    if (e == cudaSuccess) e = cudaMalloc(&err, 16);
    if (e == cudaSuccess) e = cudaMalloc(&out, 16);
    if (e == cudaSuccess) e = cudaMemcpy(g, h, BYTES, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(err, 0, 16);
    if (e == cudaSuccess) e = cudaMemset(out, 0, 16);
    if (e == cudaSuccess) {
        k_leave<<<1, 256, SM>>>(g, o, err, out);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(h, o, BYTES, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(herr, err, 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(hout, out, 8, cudaMemcpyDeviceToHost);
    cudaFree(g);
    cudaFree(o);
    cudaFree(err);
    cudaFree(out);
    return (int)e;
}
