// spike_emu64.cuh -- FP64 tile products and inverses of one CTA on the tensor
// cores, by exact digit products (spike_slices.cuh).
//
// A 64 x 64 x 64 FP64 product is 262,144 multiply-adds: 131,000 clocks of an
// SM's FP64 pipe, 9,700 of its tensor cores as digit products.  Operands are FP64
// tiles in shared or global memory; the right one is split once per product into
// digit planes in shared memory (scaled by column), the left one into registers by
// the warps that use its rows (scaled by row).  A result rounds once, and what
// the scales leave out of it is below 2^-57 of its row's and column's scales.  It
// is taken where that is below 2^-51 of the terms that some result of its row or of
// its column sums, as in a chain of FP64 multiply-adds over
// data of one magnitude; where a row's and a column's large values never meet
// (columns of A scaled up and the rows of B down, say), or a row or column is
// outside FP64's comfortable exponents or not finite, one warp forms the result
// as that chain.
//
// A product takes 27,000 clocks of one CTA: 15,000 in the k loop, where the eight
// warps (two per scheduler, all that the 144 accumulator registers leave room
// for) do not quite hide the splitting behind the products, 5,000 to round, the
// rest for scales and stores.  The inverse takes 125,000 clocks where FP64
// Gauss-Jordan by halves takes 205,000 and on whole rows 290,000.
#pragma once
#include "spike_slices.cuh"

template <int KB> struct Emu {
    static constexpr int WARPS = KB / 8, NT = 32 * WARPS; // the Tile kernels' own thread count (NTOf)
    static constexpr int LD = KB + 8;                     // row stride of FP64 tiles: conflict-free row fragments
    static constexpr int LDC = KB + 2;                    // column stride of tiles kept column-major
    static constexpr int LDP = KB + 8;                    // halves per column of a digit plane
    static constexpr int TILE = KB * LD;
    static constexpr size_t PLANES = (size_t)(SL_D + 1) * KB * LDP * 2;
    static constexpr int GUARD = 6; // binary orders

    unsigned short *px; // digit planes of the right operand: [digit][column][k]
    int *ec;            // its columns' scale exponents, [KB]; then [2][2 KB]: the products' row and column maxima
    static constexpr int EC_INTS = 7 * KB; // and an inverse's row and column scales

    // exponent class of a row or column from the largest |high word| met:
    // 0 when every value is zero, else at least 1
    static __device__ __forceinline__ unsigned mag_of(double v)
    {
        const unsigned h = (unsigned)__double2hiint(v) & 0x7fffffffu;
        return max(h, __double2loint(v) != 0 ? 1u : 0u);
    }
    static __device__ __forceinline__ int exp_of(unsigned m) { return m == 0u ? 0 : max((int)(m >> 20), 1); }
    static __device__ __forceinline__ bool usable(int e) { return e >= 64 && e < 0x7ff; }

    // planes of the K x N right operand, B(k, c) = B[k bk + c bc]; a warp splits
    // eight columns.  All threads call; a barrier must follow.  (build and mul are
    // calls, not inlined: a kernel of a dozen inlined products does not fit the
    // instruction cache.)
    template <int K> __device__ __noinline__ void build(const double *B, int bk, int bc, int N) const
    {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        for (int q = threadIdx.x; q < 4 * KB; q += NT) ec[KB + q] = 0;
        if (warp >= N / 8) return;
        const int c = warp * 8 + (lane & 7), k4 = lane >> 3;
        double v[K / 8][2];
        unsigned m = 0;
#pragma unroll
        for (int i = 0; i < K / 8; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                v[i][j] = B[(2 * (k4 + 4 * i) + j) * bk + c * bc];
                m = max(m, mag_of(v[i][j]));
            }
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
        const int E = exp_of(m);
        if (k4 == 0) ec[c] = E;
        const bool live = usable(E);
        unsigned *o = (unsigned *)px + (c * LDP) / 2 + k4;
        constexpr int ST = KB * LDP / 2;
#pragma unroll
        for (int i = 0; i < K / 8; i++) {
            SlPair(live ? v[i][0] : 0.0, live ? v[i][1] : 0.0, live ? E : 64).store(o + 4 * i, ST);
        }
    }

    // D = C + A B or C - A B (C may be NULL, or D itself), D2 = the same where
    // given; every operand by element strides.  tri: 1 / 2 = A upper / lower
    // triangular, 3 = B lower triangular: k steps of zeros are skipped.
    struct Op {
        const double *A;
        int ar, ak;
        const double *B;
        int bk, bc;
        const double *C;
        int cr, cc;
        double *D;
        int dr, dc;
        double *D2;
        int d2r, d2c;
        int tri;
        bool neg;
    };
    // element e of K <= 64 products at scale exponent p (of the units of 256^7)
    // as FP64, with integer instructions.  The eight sums hold 74 bits; the last 11
    // go (2^-56 of the scales' product), so that the rest is one 64-bit integer.
    // Sums 0-3 are at most 2^22 and 6, 7 need no last bit: FP32 additions of 1.5
    // times 2^23 and 2^24 convert them.
    static __device__ __forceinline__ double result(const SlAcc &a, int e, int p)
    {
        constexpr unsigned M = 0x4b400000u, M2 = 0x4bc00000u;
        const unsigned b0 = __float_as_uint(a.c[0][e] + 12582912.f), b1 = __float_as_uint(a.c[1][e] + 12582912.f);
        const unsigned b2 = __float_as_uint(a.c[2][e] + 12582912.f), b3 = __float_as_uint(a.c[3][e] + 12582912.f);
        const unsigned b6 = __float_as_uint(a.c[6][e] + 25165824.f), b7 = __float_as_uint(a.c[7][e] + 25165824.f);
        const int h01 = (int)(b0 * 256u + b1 - 257u * M), h23 = (int)(b2 * 256u + b3 - 257u * M);
        const int h45 = __float2int_rn(a.c[4][e]) * 256 + __float2int_rn(a.c[5][e]);
        const int h67 = (int)(b6 * 512u + b7 * 2u - 514u * M2);
        const long long T = (((long long)h01 * 65536 + h23) << 21) + ((long long)h45 * 32 + (h67 >> 11));
        const unsigned sg = (unsigned)((int)(T >> 32) >> 31);
        const unsigned long long sg2 = ((unsigned long long)sg << 32) | sg, m = ((unsigned long long)T ^ sg2) - sg2;
        const int z = __clzll((long long)m) & 63;
        const unsigned long long n = m << z, r = (n >> 11) + ((unsigned)n >> 10 & 1u); // 53 bits
        const unsigned long long bits = ((unsigned long long)(unsigned)(p + 11 + 63 - z + 1022) << 52) + r;
        return m == 0 ? 0.0 : __longlong_as_double((long long)(bits | ((unsigned long long)(sg & 0x80000000u) << 32)));
    }

    // M x N over K (B's planes built), NTL column tiles of 8 per warp.  All
    // threads call; a barrier inside ends the reads of A, so D may be A or C.
    // use: 0 for the first product with these planes, 1 for the second.  ND <
    // SL_D: a small correction, of which only the leading sums are formed, and
    // whose results need no more than the scales' own precision.
    template <int NTL, int ND = SL_D>
    __device__ __noinline__ void mul(const Op &P, int M, int N, int K, int use) const
    {
        const int MT = M / 16, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
        if (warp >= MT * (N / 8) / NTL) {
            __syncthreads();
            return;
        }
        int *mx = ec + KB + use * 2 * KB; // largest sums of magnitudes: rows, columns
        const int r0 = (warp % MT) * 16, c0 = (warp / MT) * NTL * 8;
        const double *A0 = P.A + (size_t)(r0 + g) * P.ar;
        const int ar = P.ar, ak = P.ak;
        int E[2];
#pragma unroll
        for (int p = 0; p < 2; p++) {
            unsigned m = 0;
#pragma unroll 2
            for (int k = 0; k < K; k += 8)
#pragma unroll
                for (int j = 0; j < 2; j++) m = max(m, mag_of(A0[8 * p * ar + (k + 2 * t + j) * ak]));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
            E[p] = exp_of(m);
        }
        SlAcc acc[NTL];
#pragma unroll
        for (int j = 0; j < NTL; j++) acc[j].zero();
        const int s0 = P.tri == 1 ? r0 / 16 : P.tri == 3 ? c0 / 16 : 0, s1 = P.tri == 2 ? r0 / 16 + 1 : K / 16;
        double w[2][4];
        auto fetch = [&](int s) {
#pragma unroll
            for (int p = 0; p < 2; p++)
#pragma unroll
                for (int q = 0; q < 4; q++)
                    w[p][q] = usable(E[p]) ? A0[8 * p * ar + (s * 16 + 2 * t + (q & 1) + (q >> 1) * 8) * ak] : 0.0;
        };
        fetch(s0);
#pragma unroll 1
        for (int s = s0; s < s1; s++) {
            const int k0 = s * 16 + 2 * t;
            SlFragA F;
            F.split(w, usable(E[0]) ? E[0] : 64, usable(E[1]) ? E[1] : 64);
            if (s + 1 < s1) fetch(s + 1);
#pragma unroll
            for (int j = 0; j < NTL; j++) {
                const unsigned *xb = (const unsigned *)px + ((c0 + 8 * j + g) * LDP + k0) / 2;
                acc[j].template step<ND>(F, [&](int i, int q) { return xb[i * (KB * LDP / 2) + 4 * q]; });
            }
        }
        // the largest sums of magnitudes (binary exponents) of the product's rows,
        // in units of the row's scale, and columns, in units of the column's
        int rm[2] = {0, 0};
        if (ND == SL_D) {
#pragma unroll
            for (int jq = 0; jq < 2 * NTL; jq++) {
                const int j = jq / 2, q = jq % 2, c = c0 + 8 * j + 2 * t + q;
                int m = 0;
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const int l = __float_as_int(acc[j].g[2 * p + q]) >> 23; // 0: nothing summed
                    m = max(m, l > 0 ? l + E[p] : 0);
                    rm[p] = max(rm[p], l > 0 ? l + ec[c] : 0);
                }
#pragma unroll
                for (int o = 4; o < 32; o *= 2) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
                if (g == 0) atomicMax(mx + KB + c, m);
            }
#pragma unroll
            for (int p = 0; p < 2; p++) {
                rm[p] = max(rm[p], __shfl_xor_sync(0xffffffffu, rm[p], 1));
                rm[p] = max(rm[p], __shfl_xor_sync(0xffffffffu, rm[p], 2));
                if (t == 0) atomicMax(mx + r0 + g + 8 * p, rm[p]);
            }
        }
        __syncthreads();
        if (ND == SL_D) {
            rm[0] = mx[r0 + g];
            rm[1] = mx[r0 + g + 8];
        }
        double v[NTL][4];
        unsigned redo = 0; // bit 4 j + e: the result is outside the scales' reach
        bool ur[2], zr[2]; // rows: usable; zero
#pragma unroll
        for (int p = 0; p < 2; p++) ur[p] = usable(E[p]), zr[p] = E[p] == 0;
#pragma unroll
        for (int j = 0; j < NTL; j++) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int c = c0 + 8 * j + 2 * t + (e & 1), p = e >> 1;
                const int Ec = ec[c], sc = 56 + E[p] + Ec - 2 * (1023 + 61);
                const bool met = ND < SL_D || max(rm[p] - Ec, mx[KB + c] - E[p]) >= 127 - GUARD;
                const bool fine = ur[p] && usable(Ec) && met && (unsigned)(sc + 900) < 1750u;
                const bool zero = (zr[p] && Ec < 0x7ff) || (Ec == 0 && E[p] < 0x7ff);
                v[j][e] = result(acc[j], e, sc); // (meaningless unless fine)
                if (!fine) {
                    v[j][e] = 0.0;
                    redo |= zero || ND < SL_D ? 0u : 1u << (4 * j + e);
                }
            }
        }
        if (__any_sync(0xffffffffu, redo != 0u)) {
#pragma unroll
            for (int j = 0; j < NTL; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int r = r0 + g + 8 * (e >> 1), c = c0 + 8 * j + 2 * t + (e & 1);
                    for (unsigned todo = __ballot_sync(0xffffffffu, redo >> (4 * j + e) & 1u); todo; todo &= todo - 1) {
                        const int src = __ffs(todo) - 1;
                        const int rr = __shfl_sync(0xffffffffu, r, src), cc = __shfl_sync(0xffffffffu, c, src);
                        double sum = 0.0;
                        for (int k = lane; k < K; k += 32)
                            sum = fma(P.A[rr * P.ar + k * P.ak], P.B[k * P.bk + cc * P.bc], sum);
                        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                        if (lane == src) v[j][e] = sum;
                    }
                }
        }
        const double *C = P.C;
        double *D = P.D, *D2 = P.D2;
        const int dr = P.dr, dc = P.dc;
        if (P.neg)
#pragma unroll
            for (int j = 0; j < NTL; j++)
#pragma unroll
                for (int e = 0; e < 4; e++) v[j][e] = -v[j][e];
        if (C) {
            const int cr = P.cr, cc = P.cc;
#pragma unroll
            for (int j = 0; j < NTL; j++)
#pragma unroll
                for (int e = 0; e < 4; e++)
                    v[j][e] = C[(r0 + g + 8 * (e >> 1)) * cr + (c0 + 8 * j + 2 * t + (e & 1)) * cc] + v[j][e];
        }
#pragma unroll
        for (int j = 0; j < NTL; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) D[(r0 + g + 8 * (e >> 1)) * dr + (c0 + 8 * j + 2 * t + (e & 1)) * dc] = v[j][e];
        if (D2) {
            const int d2r = P.d2r, d2c = P.d2c;
#pragma unroll
            for (int j = 0; j < NTL; j++)
#pragma unroll
                for (int e = 0; e < 4; e++)
                    D2[(r0 + g + 8 * (e >> 1)) * d2r + (c0 + 8 * j + 2 * t + (e & 1)) * d2c] = v[j][e];
        }
    }
    // whole tiles: KB x KB x KB
    template <int ND = SL_D> __device__ __forceinline__ void product(const Op &P) const
    {
        mul<KB / 16, ND>(P, KB, KB, KB, 0);
    }

    // FP64 to FP32 and back, and x 2^k, with integer instructions (the FP64 pipe
    // converts and multiplies at two results a clock)
    static __device__ __forceinline__ float to_f32(double v, int k = 0)
    {
        const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
        const int e = (int)(h >> 20 & 0x7ffu) + k - 896;
        const unsigned m = ((h & 0xfffffu) << 3 | l >> 29) + (l >> 28 & 1u);
        return __uint_as_float((h & 0x80000000u) | (e <= 0 ? 0u : e >= 255 ? 0x7f800000u : ((unsigned)e << 23) + m));
    }
    static __device__ __forceinline__ double to_f64(float f)
    {
        const unsigned u = __float_as_uint(f), a = u & 0x7fffffffu;
        return a < 0x800000u ? 0.0 : __hiloint2double((int)((u & 0x80000000u) | ((a >> 3) + (896u << 20))), (int)(a << 29));
    }
    static __device__ __forceinline__ double scaled(double v, int k)
    {
        const int h = __double2hiint(v), e = (h >> 20 & 0x7ff), n = e + k;
        if (e > 0 && n > 0 && e < 0x7ff && n < 0x7ff) return __hiloint2double(h + (k << 20), __double2loint(v));
        return e == 0 && (h & 0xfffff) == 0 && __double2loint(v) == 0 ? v : scalbn(v, k);
    }

    // In-place inverse without pivoting of the KB x KB tile S (row stride LD):
    // rows and columns scaled by powers of two, an FP32 inverse X0, and with
    // R = I - S X0 (a full product) the result (X0 + X0 R)(I + R R), whose error
    // beyond R's own rounding is X0 R^4.  Where ||R|| > 2^-13 (an FP32 pivot of
    // zero, an ill-conditioned tile) the inverse by halves takes over.  X and R:
    // scratch tiles (row stride LD).  All threads call; barriers inside and after.
    __device__ __noinline__ bool inverse_tile(double *S, double *X, double *R) const
    {
        constexpr int LF = KB + 4, CH = KB * KB / NT;
        float *F = (float *)px; // the FP32 tile, where planes go later
        int *re = ec + 5 * KB, *ce = re + KB;
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        {
            const int r = warp * 8 + (lane >> 2); // four lanes a row
            unsigned m = 0;
#pragma unroll 4
            for (int c = lane & 3; c < KB; c += 4) m = max(m, mag_of(S[r * LD + c]));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
            const int e = exp_of(m);
            if ((lane & 3) == 0) re[r] = usable(e) ? 1023 - e : 0;
        }
        __syncthreads();
        {
            const int c = warp * 8 + (lane & 7); // four lanes a column
            unsigned m = 0;
#pragma unroll 4
            for (int r = lane >> 3; r < KB; r += 4) m = max(m, mag_of(S[r * LD + c] = scaled(S[r * LD + c], re[r])));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 8));
            m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
            const int e = exp_of(m), k = usable(e) ? 1023 - e : 0;
            if (lane < 8) ce[c] = k;
#pragma unroll 4
            for (int r = lane >> 3; r < KB; r += 4) {
                const double v = scaled(S[r * LD + c], k);
                S[r * LD + c] = v;
                F[r * LF + c] = to_f32(v);
            }
        }
        __syncthreads();
        bool good = BlkInv<NT, LF>::template run<KB>(F);
#pragma unroll 4
        for (int i = 0; i < CH; i++) {
            const int q = tid + i * NT;
            X[q / KB * LD + q % KB] = to_f64(F[q / KB * LF + q % KB]);
        }
        __syncthreads();
        build<KB>(X, LD, 1, KB);
        __syncthreads();
        product({S, LD, 1, X, LD, 1, nullptr, 0, 0, R, LD, 1, nullptr, 0, 0, 0, true});
        __syncthreads();
        float n2 = 0.f; // this thread's part of ||R||^2, in units of 2^-40
#pragma unroll 4
        for (int i = 0; i < CH; i++) {
            const int q = tid + i * NT, r = q / KB, c = q % KB;
            double v = R[r * LD + c];
            if (r == c) R[r * LD + c] = v = v + 1.0;
            const float x = to_f32(v, 20);
            n2 = fmaf(x, x, n2);
        }
        good = good && n2 <= 16384.f / NT; // (false for NaN) ||R||^2 <= 2^-26 in all
        bool ok = true;
        if (__syncthreads_and(good)) {
            build<KB>(R, LD, 1, KB);
            __syncthreads();
            // the corrections are below 2^-13 and 2^-26 of X0: six and four leading digit sums
            product<6>({X, LD, 1, R, LD, 1, X, LD, 1, S, LD, 1, nullptr, 0, 0, 0, false});
            product<4>({R, LD, 1, R, LD, 1, nullptr, 0, 0, X, LD, 1, nullptr, 0, 0, 0, false});
            __syncthreads();
            build<KB>(X, LD, 1, KB);
            __syncthreads();
            product<4>({S, LD, 1, X, LD, 1, S, LD, 1, S, LD, 1, nullptr, 0, 0, 0, false});
            __syncthreads();
        } else {
            ok = inverse<KB>(S, X);
        }
#pragma unroll 4
        for (int i = 0; i < CH; i++) {
            const int q = tid + i * NT, r = q / KB, c = q % KB;
            S[r * LD + c] = scaled(S[r * LD + c], ce[r] + re[c]);
        }
        __syncthreads();
        return ok;
    }

    // In-place inverse without pivoting of the N x N block S (row stride LD) in
    // shared memory, by halves as BlkInv; 16-row leaves are one warp's FP64
    // Gauss-Jordan.  X: scratch of N rows.  All threads call; barriers inside and
    // after.  false (in the leaf's warp) on a zero or non-finite pivot.
    template <int N> __device__ bool inverse(double *S, double *X) const
    {
        if constexpr (N == 16) {
            bool ok = true;
            if (threadIdx.x < 32) ok = leaf(S);
            __syncthreads();
            return ok;
        } else {
            constexpr int h = N / 2;
            double *A12 = S + h, *A21 = S + h * LD, *A22 = A21 + h, *X2 = X + h;
            auto prod = [&](const double *A, const double *B, const double *C, double *D, bool neg, int use = 0) {
                const Op P{A, LD, 1, B, LD, 1, C, LD, 1, D, LD, 1, nullptr, 0, 0, 0, neg};
                mul<1>(P, h, h, h, use);
            };
            auto copy = [&](double *D, const double *A) {
                for (int q = threadIdx.x; q < h * h; q += NT) D[q / h * LD + q % h] = A[q / h * LD + q % h];
            };
            bool ok = inverse<h>(S, X); // H11
            build<h>(S, LD, 1, h);
            __syncthreads();
            prod(A21, S, nullptr, X, false); // U = A21 H11
            __syncthreads();
            copy(A21, X);
            build<h>(A12, LD, 1, h);
            __syncthreads();
            prod(A21, A12, A22, A22, true);    // A22 - U A12
            prod(S, A12, nullptr, X2, false, 1); // T = H11 A12
            __syncthreads();
            copy(A12, X2);
            ok = inverse<h>(A22, X) && ok; // H22 (barriers inside)
            build<h>(A22, LD, 1, h);
            __syncthreads();
            prod(A12, A22, nullptr, X, true); // G12 = -T H22
            __syncthreads();
            copy(A12, X);
            build<h>(A21, LD, 1, h);
            __syncthreads();
            prod(A12, A21, S, S, true);        // G11 = H11 - G12 U
            prod(A22, A21, nullptr, X2, true, 1); // G21 = -H22 U
            __syncthreads();
            copy(A21, X2);
            __syncthreads();
            return ok;
        }
    }

    // one warp: 16 x 16 Gauss-Jordan, lane (a, b) holding rows 2a, 2a + 1 and columns 4b .. 4b + 3
    static __device__ __forceinline__ bool leaf(double *S)
    {
        constexpr unsigned FULL = 0xffffffffu;
        const int lane = threadIdx.x & 31, a = lane >> 2, b = lane & 3;
        double s[2][4];
        bool ok = true;
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) s[i][j] = S[(2 * a + i) * LD + 4 * b + j];
        for (int kb = 0; kb < 4; kb++) {
#pragma unroll
            for (int kk = 0; kk < 4; kk++) { // pivot k = 4 kb + kk: lane (ra, kb), register [kk % 2][kk]
                const int ra = 2 * kb + kk / 2;
                const double piv = __shfl_sync(FULL, s[kk % 2][kk], (ra << 2) | kb);
                double row[4], col[2];
#pragma unroll
                for (int j = 0; j < 4; j++) row[j] = __shfl_sync(FULL, s[kk % 2][j], (ra << 2) | b);
#pragma unroll
                for (int i = 0; i < 2; i++) col[i] = __shfl_sync(FULL, s[i][kk], (a << 2) | kb);
                const unsigned ph = (unsigned)__double2hiint(piv) & 0x7fffffffu;
                if (ph >= 0x7ff00000u || (ph == 0u && __double2loint(piv) == 0)) ok = false;
                const double pr = __drcp_rn(piv);
                const bool myrow = a == ra, mycol = b == kb;
#pragma unroll
                for (int j = 0; j < 4; j++) row[j] = row[j] * pr;
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const bool pivrow = myrow && i == kk % 2;
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const double x = pivrow ? row[j] : fma(-col[i], row[j], s[i][j]);
                        s[i][j] = x;
                    }
                    const double y = pivrow ? pr : -(col[i] * pr); // the pivot's column
                    s[i][kk] = mycol ? y : s[i][kk];
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) S[(2 * a + i) * LD + 4 * b + j] = s[i][j];
        return ok;
    }
};

// KB rows of KB doubles, `ld` apart in shared memory, by bulk copies on bar; warp 0 calls
template <int KB> __device__ __forceinline__ void bulk_rows(double *s, int ld, const double *g, uint64_t *bar)
{
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        fence_proxy_async();
        mbar_arrive_expect_tx(bar, KB * KB * 8);
    }
    __syncwarp();
    for (int r = lane; r < KB; r += 32) bulk_g2s(s + (size_t)r * ld, g + (size_t)r * KB, KB * 8, bar);
}

// one shared buffer that bulk copies fill: all threads call issue() after a
// barrier that ends its last use, and wait()
template <int KB> struct EmuBar {
    uint64_t *bar;
    unsigned phase;
    bool inflight;
    __device__ __forceinline__ void issue(double *s, int ld, const double *g)
    {
        if (threadIdx.x < 32) bulk_rows<KB>(s, ld, g, bar);
        inflight = true;
    }
    // false in every thread when the copy has not landed in time (a barrier
    // inside): it still counts as in flight
    __device__ __forceinline__ bool wait()
    {
        if (__syncthreads_or(!mbar_wait(bar, phase))) return false;
        phase ^= 1u;
        inflight = false;
        return true;
    }
    __device__ __forceinline__ void drain()
    {
        if (inflight) mbar_wait(bar, phase);
    }
};

// a wait has run out: say so, and give every copy still in flight the time of
// one more wait, since the block's shared memory is another's once it leaves
template <class... Bar> __device__ __forceinline__ void emu_leave(unsigned *err, Bar &...b)
{
    if (threadIdx.x == 0) atomicOr(err, SPK_DEV_ERR_TIMEOUT);
    (b.drain(), ...);
}
