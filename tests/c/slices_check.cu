// slices_check.cu -- sums of digit products (spike_slices.cuh) of one 16 x K by
// K x 8 product, with the largest terms' scale exponents, for comparison with
// exact sums.  Built by tests/test_gpu_slices.py; test code only.
#include "spike_slices.cuh"

// K <= 512 in steps of 16; one warp
__global__ void k_slices(const double *a, const double *b, int K, double *out, float *mag)
{
    extern __shared__ unsigned short px[]; // [digit][column][ldx]
    __shared__ int ec[8], er[16];
    const int lane = threadIdx.x, g = lane >> 2, t = lane & 3, ldx = K + 8;
    if (lane < 8) {
        int e = 0;
        for (int k = 0; k < K; k++) e = max(e, sl_exp(b[k * 8 + lane]));
        ec[lane] = e;
    }
    if (lane < 16) {
        int e = 0;
        for (int k = 0; k < K; k++) e = max(e, sl_exp(a[lane * K + k]));
        er[lane] = e;
    }
    __syncwarp();
    for (int q = lane; q < 8 * K / 2; q += 32) {
        const int c = q / (K / 2), k = q % (K / 2) * 2;
        SlPair(b[k * 8 + c], b[(k + 1) * 8 + c], ec[c]).store((unsigned *)(px + c * ldx + k), 8 * ldx / 2);
    }
    __syncwarp();
    long long hi[4] = {0, 0, 0, 0}, lo[4] = {0, 0, 0, 0};
    float mg[4] = {0.f, 0.f, 0.f, 0.f};
    for (int s0 = 0; s0 < K / 16; s0 += SL_FLUSH) {
        SlAcc acc;
        acc.zero();
        for (int s = s0; s < min(K / 16, s0 + SL_FLUSH); s++) {
            double w[2][4];
            for (int p = 0; p < 2; p++)
                for (int q = 0; q < 4; q++) w[p][q] = a[(g + 8 * p) * K + s * 16 + 2 * t + (q & 1) + (q >> 1) * 8];
            SlFragA A;
            A.split(w, er[g], er[g + 8]);
            const unsigned *xb = (const unsigned *)(px + g * ldx + s * 16 + 2 * t);
            acc.step(A, [&](int i, int q) { return xb[i * (8 * ldx / 2) + 4 * q]; });
        }
        for (int e = 0; e < 4; e++) {
            long long h, l;
            acc.total(e, h, l);
            hi[e] += h;
            lo[e] += l;
            mg[e] += acc.g[e];
        }
    }
    for (int e = 0; e < 4; e++) {
        const int r = g + 8 * (e >> 1), c = 2 * t + (e & 1);
        out[r * 8 + c] = sl_round(hi[e], lo[e], 56 + er[r] + ec[c] - 2 * (1023 + 61));
        mag[r * 8 + c] = mg[e];
    }
}

extern "C" int slices_check(const double *a, const double *b, int K, double *out, float *mag)
{
    double *da = nullptr, *db = nullptr, *dout = nullptr;
    float *dm = nullptr;
    cudaError_t e = cudaMalloc(&da, sizeof(double) * 16 * K);
    if (e == cudaSuccess) e = cudaMalloc(&db, sizeof(double) * 8 * K);
    if (e == cudaSuccess) e = cudaMalloc(&dout, sizeof(double) * 128);
    if (e == cudaSuccess) e = cudaMalloc(&dm, sizeof(float) * 128);
    if (e == cudaSuccess) e = cudaMemcpy(da, a, sizeof(double) * 16 * K, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(db, b, sizeof(double) * 8 * K, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        const int sm = (SL_D + 1) * 8 * (K + 8) * 2;
        e = cudaFuncSetAttribute(k_slices, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        if (e == cudaSuccess) {
            k_slices<<<1, 32, sm>>>(da, db, K, dout, dm);
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof(double) * 128, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(mag, dm, sizeof(float) * 128, cudaMemcpyDeviceToHost);
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    cudaFree(dm);
    return (int)e;
}
