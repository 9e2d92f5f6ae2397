// spike_emu64.cuh -- FP64 tile products and inverses of one CTA on the tensor
// cores where their results allow it, by digit products (spike_slices.cuh).
//
// A 64 x 64 x 64 FP64 product is 262,144 multiply-adds: 131,000 clocks of an
// SM's FP64 pipe, 9,700 of its tensor cores as digit products.  Operands are FP64
// tiles in shared or global memory; the right one is split once per product into
// digit planes in shared memory (scaled by column), the left one into registers by
// the warps that use its rows (scaled by row).  What the digits leave out of a
// result is measured by its row's and its column's scale, so a result is taken
// from them only where the terms it sums come near those scales (SL_GUARD); the
// others -- entries that a column's decay, a triangle's corner or a strong diagonal
// leaves small -- are formed as FP64 multiply-adds, one by one where they are
// few.  So every entry is as good as a chain of FP64 multiply-adds makes it,
// however far its row and column reach
// (n = 1,500, unit right-hand sides: half of the solution's entries within 1e-15 at
// dominances of 1.5 to 1e4 and bands of 40 and 64, like FP64 tiles throughout; results
// taken by row and column scales alone lost up to 1e-8 of them).
//
// A product takes 19,900 clocks of one CTA and its planes 2,700; at dominance 1.5
// a few percent of the chains' results are formed in FP64 after all, at 1e4 most
// (135,000 clocks a product, the FP64 pipe's own time).  The inverse, by halves to 16-row leaves, takes
// 134,000 clocks, where Gauss-Jordan on whole FP64 rows took 290,000.
#pragma once
#include "spike_slices.cuh"

template <int KB> struct Emu {
    static constexpr int WARPS = KB / 8, NT = 32 * WARPS; // the Tile kernels' own thread count (NTOf)
    static constexpr int LD = KB + 8;                     // row stride of FP64 tiles: conflict-free row fragments
    static constexpr int LDC = KB + 2;                    // column stride of tiles kept column-major
    static constexpr int LDP = KB + 8;                    // halves per column of a digit plane
    static constexpr int TILE = KB * LD;
    static constexpr size_t PLANES = (size_t)(SL_D + 1) * KB * LDP * 2;
    static constexpr int REDO = 96; // a warp's list of results to form one by one
    static constexpr size_t AUX = sizeof(int) * KB + sizeof(unsigned short) * REDO * WARPS;

    unsigned short *px; // digit planes of the right operand: [digit][column][k]
    int *ec;            // its columns' scale exponents, [KB]; then the warps' lists of results to form in FP64

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

    // D = C + A B or C - A B (C may be NULL, or D itself; D is neither A nor B,
    // which results formed in FP64 read to the end), D2 = the same where given; every operand by element strides.  tri: 1 / 2 = A upper / lower
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
        // element (r, c) of the result, from its sum
        __device__ __forceinline__ void put(int r, int c, double v) const
        {
            v = neg ? -v : v;
            if (C) v = C[r * cr + c * cc] + v;
            D[r * dr + c * dc] = v;
            if (D2) D2[r * d2r + c * d2c] = v;
        }
    };
    // element e of K <= 64 products at scale exponent p (of the units of 256^7)
    // as FP64, with integer instructions.  The eight sums hold 74 bits; the last 11
    // are rounded off (2^-56 of the scales' product), so that the rest is one 64-bit integer.
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
        const int h67 = (int)(b6 * 512u + b7 * 2u - 514u * M2 + 1024u);
        const long long T = (((long long)h01 * 65536 + h23) << 21) + ((long long)h45 * 32 + (h67 >> 11));
        const unsigned sg = (unsigned)((int)(T >> 32) >> 31);
        const unsigned long long sg2 = ((unsigned long long)sg << 32) | sg, m = ((unsigned long long)T ^ sg2) - sg2;
        const int z = __clzll((long long)m) & 63;
        const unsigned long long n = m << z, r = (n >> 11) + ((unsigned)n >> 10 & 1u); // 53 bits
        const unsigned long long bits = ((unsigned long long)(unsigned)(p + 11 + 63 - z + 1022) << 52) + r;
        return m == 0 ? 0.0 : __longlong_as_double((long long)(bits | ((unsigned long long)(sg & 0x80000000u) << 32)));
    }

    // M x N over K (B's planes built), NTL column tiles of 8 per warp; no
    // barrier inside
    template <int NTL> __device__ __noinline__ void mul(const Op &P, int M, int N, int K) const
    {
        const int MT = M / 16, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
        if (warp >= MT * (N / 8) / NTL) return;
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
                acc[j].step(F, [&](int i, int q) { return xb[i * (KB * LDP / 2) + 4 * q]; });
            }
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
                const bool fine = ur[p] && usable(Ec) && acc[j].g[e] >= SL_GUARD && (unsigned)(sc + 900) < 1750u;
                const bool zero = (zr[p] && Ec < 0x7ff) || (Ec == 0 && E[p] < 0x7ff);
                v[j][e] = result(acc[j], e, sc); // (meaningless unless fine)
                if (!fine) {
                    v[j][e] = 0.0;
                    redo |= zero ? 0u : 1u << (4 * j + e);
                }
            }
        }
        const int todo = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(redo));
        if (todo > 0) {
            const int ka = 16 * s0, kb = 16 * s1;
            if (todo <= 64 * NTL) // of 128 NTL: 61 against 33 clocks each, but of all of them
                few(P, redo, r0, c0, ka, kb, 4 * NTL);
            else
                all<NTL>(P, redo, r0 + g, c0 + 2 * t, ka, kb);
        }
        place<NTL>(P, ~redo, r0 + g, c0 + 2 * t, v);
    }
    // a lane's results, rows r and r + 8, columns c + 8 j and the next, into place where `mask` has their bits
    template <int NTL>
    static __device__ __forceinline__ void place(const Op &P, unsigned mask, int r, int c, double (&v)[NTL][4])
    {
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
                    if (mask >> (4 * j + e) & 1u) v[j][e] = C[(r + 8 * (e >> 1)) * cr + (c + 8 * j + (e & 1)) * cc] + v[j][e];
        }
#pragma unroll
        for (int j = 0; j < NTL; j++)
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (mask >> (4 * j + e) & 1u) D[(r + 8 * (e >> 1)) * dr + (c + 8 * j + (e & 1)) * dc] = v[j][e];
        if (D2) {
            const int d2r = P.d2r, d2c = P.d2c;
#pragma unroll
            for (int j = 0; j < NTL; j++)
#pragma unroll
                for (int e = 0; e < 4; e++)
                    if (mask >> (4 * j + e) & 1u) D2[(r + 8 * (e >> 1)) * d2r + (c + 8 * j + (e & 1)) * d2c] = v[j][e];
        }
    }
    // the results marked in `redo` over k = ka .. kb - 1, four at a time on eight
    // lanes each, into place: 61 clocks per result of the CTA
    __device__ __noinline__ void few(const Op &P, unsigned redo, int r0, int c0, int ka, int kb, int slots) const
    {
        const int lane = threadIdx.x & 31;
        unsigned short *l = (unsigned short *)(ec + KB) + (threadIdx.x >> 5) * REDO;
        const int ar = P.ar, ak = P.ak, bk = P.bk, bc = P.bc;
        int cnt = 0;
        for (int s = 0; s < slots; s++) {
            const unsigned m = __ballot_sync(0xffffffffu, redo >> s & 1u);
            if (redo >> s & 1u) l[cnt + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(s * 32 + lane);
            cnt += __popc(m);
            if (cnt <= REDO - 32 && s + 1 < slots) continue; // room for another slot
            __syncwarp();
            for (int i = 0; i < cnt; i += 4) {
                const int q = i + (lane >> 3), x = l[q < cnt ? q : i], b = x >> 5, o = x & 31;
                const int r = r0 + (o >> 2) + 8 * (b >> 1 & 1), c = c0 + 8 * (b >> 2) + 2 * (o & 3) + (b & 1);
                double sum = 0.0;
#pragma unroll 4
                for (int k = ka + (lane & 7); k < kb; k += 8) sum = fma(P.A[r * ar + k * ak], P.B[k * bk + c * bc], sum);
#pragma unroll
                for (int h = 4; h > 0; h >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, h);
                if (q < cnt && (lane & 7) == 0) P.put(r, c, sum);
            }
            __syncwarp(); // the list is written again
            cnt = 0;
        }
    }
    // the same with every result formed, each by its own lane, and those marked
    // put into place: 33 clocks per result
    template <int NTL> static __device__ __noinline__ void all(const Op &P, unsigned redo, int r, int c, int ka, int kb)
    {
        double w[NTL][4];
#pragma unroll
        for (int j = 0; j < NTL; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) w[j][e] = 0.0;
        const double *A = P.A + r * P.ar, *B = P.B + c * P.bc;
        const int ar8 = 8 * P.ar, ak = P.ak, bk = P.bk, bc = P.bc;
#pragma unroll 2
        for (int k = ka; k < kb; k++) {
            const double a0 = A[k * ak], a1 = A[ar8 + k * ak];
#pragma unroll
            for (int j = 0; j < NTL; j++)
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const double b = B[k * bk + (8 * j + q) * bc];
                    w[j][q] = fma(a0, b, w[j][q]);
                    w[j][2 + q] = fma(a1, b, w[j][2 + q]);
                }
        }
        place<NTL>(P, redo, r, c, w);
    }
    // whole tiles: KB x KB x KB
    __device__ __forceinline__ void product(const Op &P) const { mul<KB / 16>(P, KB, KB, KB); }

    // In-place inverse without pivoting of the KB x KB block S (row stride LD) in
    // shared memory, by halves as BlkInv.  X: scratch of KB / 2 rows.  All threads
    // call, S complete; barriers inside and after.  false (in the leaves' warps) on a
    // zero or non-finite pivot.
    __device__ __noinline__ bool inverse(double *S, double *X) const
    {
        constexpr int h = KB / 2;
        double *A12 = S + h, *A21 = S + h * LD, *A22 = A21 + h, *X2 = X + h;
        auto prod = [&](const double *A, const double *B, const double *C, double *D, bool neg) {
            const Op P{A, LD, 1, B, LD, 1, C, LD, 1, D, LD, 1, nullptr, 0, 0, 0, neg};
            mul<1>(P, h, h, h);
        };
        auto copy = [&](double *D, const double *A) {
            for (int q = threadIdx.x; q < h * h; q += NT) D[q / h * LD + q % h] = A[q / h * LD + q % h];
        };
        bool ok = half(S); // H11
        build<h>(S, LD, 1, h);
        __syncthreads();
        prod(A21, S, nullptr, X, false); // U = A21 H11
        __syncthreads();
        copy(A21, X);
        build<h>(A12, LD, 1, h);
        __syncthreads();
        prod(A21, A12, A22, A22, true);   // A22 - U A12
        prod(S, A12, nullptr, X2, false); // T = H11 A12
        __syncthreads();
        copy(A12, X2);
        ok = half(A22) && ok; // H22 (barriers inside)
        build<h>(A22, LD, 1, h);
        __syncthreads();
        prod(A12, A22, nullptr, X, true); // G12 = -T H22
        __syncthreads();
        copy(A12, X);
        build<h>(A21, LD, 1, h);
        __syncthreads();
        prod(A12, A21, S, S, true);        // G11 = H11 - G12 U
        prod(A22, A21, nullptr, X2, true); // G21 = -H22 U
        __syncthreads();
        copy(A21, X2);
        __syncthreads();
        return ok;
    }
    // the same of a 32 x 32 block on the FP64 pipe, a thread per entry of a
    // 16 x 16 product; the leaves are Gauss-Jordan
    __device__ __noinline__ bool half(double *S) const
    {
        constexpr int h = 16;
        static_assert(KB == 4 * h && NT == h * h, "a thread per entry of a quarter's half");
        double *A12 = S + h, *A21 = S + h * LD, *A22 = A21 + h;
        const int r = threadIdx.x / h, c = threadIdx.x % h, o = r * LD + c;
        auto dot = [&](double s, const double *A, const double *B, bool neg) {
#pragma unroll
            for (int k = 0; k < h; k++) s = fma(neg ? -A[r * LD + k] : A[r * LD + k], B[k * LD + c], s);
            return s;
        };
        bool ok = true;
        double *w = (double *)px; // (no planes are in use here)
        if (threadIdx.x < 128) ok = leaf(S, w); // H11
        __syncthreads();
        const double u = dot(0.0, A21, S, false), t = dot(0.0, S, A12, false);
        __syncthreads();
        A21[o] = u; // U = A21 H11
        __syncthreads();
        A22[o] = dot(A22[o], A21, A12, true); // A22 - U A12
        __syncthreads();
        A12[o] = t; // T = H11 A12 (read after the next barrier)
        if (threadIdx.x < 128) ok = leaf(A22, w) && ok; // H22
        __syncthreads();
        const double g12 = dot(0.0, A12, A22, true), g21 = dot(0.0, A22, A21, true); // -T H22, -H22 U
        __syncthreads();
        A12[o] = g12;
        __syncthreads();
        S[o] = dot(S[o], A12, A21, true); // H11 - G12 U
        __syncthreads();
        A21[o] = g21;
        __syncthreads();
        return ok;
    }

    // 16 x 16 Gauss-Jordan on four warps, one per scheduler (a scheduler retires
    // half an FP64 multiply-add per clock): a thread holds two entries of a row, the
    // pivot's row and column pass through w (64 values).  Threads 0 .. 127 call.
    static __device__ __forceinline__ bool leaf(double *S, double *w)
    {
        const int r = threadIdx.x >> 3, c = (threadIdx.x & 7) * 2;
        double s[2] = {S[r * LD + c], S[r * LD + c + 1]};
        bool ok = true;
#pragma unroll 2
        for (int k = 0; k < 16; k++) {
            double *row = w + (k & 1) * 32, *col = row + 16;
            if (r == k) row[c] = s[0], row[c + 1] = s[1];
            if (c == (k & 14)) col[r] = s[k & 1];
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const double piv = col[k];
            const unsigned ph = (unsigned)__double2hiint(piv) & 0x7fffffffu;
            if (ph >= 0x7ff00000u || (ph == 0u && __double2loint(piv) == 0)) ok = false;
            const double pr = __drcp_rn(piv), a = col[r];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const double b = row[c + j] * pr;
                s[j] = r == k ? b : fma(-a, b, s[j]);
            }
            if (c == (k & 14)) s[k & 1] = r == k ? pr : -(a * pr); // the pivot's column
        }
        S[r * LD + c] = s[0];
        S[r * LD + c + 1] = s[1];
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
