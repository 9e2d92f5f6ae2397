// spike_reduced.cu -- factorization of the reduced system of the SPIKE solve on
// sm_103a (its solution: spike_redsolve.cu).
//
// The reference assembles R as a CSR matrix (matrix_CreateEmptyReducedSystem
// and matrix_AddTipToReducedMatrix, OpenMP/spike_matrix.c:657-740,1414-1495)
// and solves it with MKL PARDISO on the host (directSolver_Host_Solve,
// OpenMP/spike_algebra.c:263-420).  Here R stays on the device in its natural
// block form.  With one 2KB-vector of unknowns per interface i,
// u_i = (b_i, t_{i+1}), R is block tridiagonal:
//
//     D_i = [[I, P_i], [Q_i, I]]     P_i = V_i bottom tip, Q_i = W_{i+1} top tip
//     A_i = [[X_i, 0], [0, 0]]       X_i = W_i bottom tip       (couples u_{i-1})
//     C_i = [[0, 0], [0, Y_i]]       Y_i = V_{i+1} top tip      (couples u_{i+1})
//
// Block cyclic reduction keeps that quadrant structure at every level (the
// products A M C, C M A, A M A, C M C each fill a single KB x KB quadrant), so
// a level costs ~13 KB^3 multiply-adds per eliminated pair instead of the
// dense (2KB)^3 form.  The factorization runs in the factor precision
// (FP32/complex64 in mixed mode, FP64 in plain mode); the solve wraps it in
// FP64 refinement on R itself, u += CR^{-1}(g - R u), so the reduced solution
// is FP64-accurate in both modes.
#include "spike_common.cuh"

#include <type_traits>

namespace {

template <class T, int KB> struct RedSmem {
    using TL = Tile<T, KB, NTOf<KB>::value>;
    static constexpr size_t bytes = 3 * sizeof(T) * TL::ELEMS + sizeof(T) * TL::INV_BUF + 64;
};

template <class T, int KB> __device__ void ld(T *s, const T *g)
{
    copy_tile_g2s<T, KB, NTOf<KB>::value>(s, g);
}
template <class T, int KB, class Reg> __device__ void set_identity(const Tile<T, KB, NTOf<KB>::value> &t, Reg &a)
{
#pragma unroll
    for (int i = 0; i < t.TR; i++)
#pragma unroll
        for (int j = 0; j < t.TC; j++) a[i][j] = (t.row(i) == t.col(j)) ? sc_one<T>() : sc_zero<T>();
}

// level-0 blocks: FP64 -> factor precision
template <class T>
__global__ void k_red_cvt(const typename HighOf<T>::type *__restrict__ src, T *dst, long long count)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < count; q += (long long)gridDim.x * blockDim.x)
        dst[q] = cvt_fast<T, typename HighOf<T>::type>(src[q]);
}

// Odd blocks j of a level (or the single top block): M = D_j^{-1} by quadrants
//   S = I - Q P, M11 = S^{-1}, M10 = -M11 Q, M01 = -P M11, M00 = I - P M10.
// Three shared tiles: P, Q (overwritten by M10 once M10 exists) and M11.
template <class T, int KB>
__global__ void __launch_bounds__(NTOf<KB>::value)
    k_cr_odd(const T *__restrict__ Pl, const T *__restrict__ Ql, int first, int stride, T *M, unsigned *err)
{
    constexpr int NT = NTOf<KB>::value;
    using TL = Tile<T, KB, NT>;
    constexpr size_t TS = (size_t)KB * KB;
    const int j = first + blockIdx.x * stride;
    T *Mj = M + (size_t)blockIdx.x * 4 * TS;
    extern __shared__ char smraw[];
    T *sP = (T *)smem_align(smraw), *sQ = sP + TL::ELEMS, *sH = sQ + TL::ELEMS;
    T *buf = sH + TL::ELEMS;
    TL t(threadIdx.x);
    typename TL::Reg a;
    ld<T, KB>(sP, Pl + (size_t)j * TS);
    ld<T, KB>(sQ, Ql + (size_t)j * TS);
    __syncthreads();
    set_identity<T, KB>(t, a);
    t.mms(a, sQ, sP);
    const bool ok = t.inverse(a, buf);
    if (!ok && threadIdx.x == 0) atomicOr(err, SPK_DEV_ERR_PIVOT);
    t.rstore(sH, a);
    t.gstore(Mj + 3 * TS, a);
    __syncthreads();
    t.rzero(a);
    t.mms(a, sH, sQ); // M10
    t.gstore(Mj + 2 * TS, a);
    __syncthreads(); // every read of Q is done
    t.rstore(sQ, a);
    t.rzero(a);
    t.mms(a, sP, sH); // M01
    t.gstore(Mj + 1 * TS, a);
    __syncthreads();
    set_identity<T, KB>(t, a);
    t.mms(a, sP, sQ); // M00 = I - P M10
    t.gstore(Mj, a);
}

// acc += sign * L (M R); L, M, R global tiles; uses sA, sB, sC
template <class T, int KB>
__device__ __forceinline__ void chain3(const Tile<T, KB, NTOf<KB>::value> &t, typename Tile<T, KB, NTOf<KB>::value>::Reg &acc,
                       const T *L, const T *Mg, const T *R, T *sA, T *sB, T *sC, bool negate)
{
    typename Tile<T, KB, NTOf<KB>::value>::Reg tmp;
    __syncthreads();
    ld<T, KB>(sA, Mg);
    ld<T, KB>(sB, R);
    __syncthreads();
    t.rzero(tmp);
    t.mma(tmp, sA, sB);
    t.rstore(sC, tmp);
    __syncthreads();
    ld<T, KB>(sA, L);
    __syncthreads();
    if (negate)
        t.mms(acc, sA, sC);
    else
        t.mma(acc, sA, sC);
}

// Even blocks i of level l produce block i/2 of level l+1:
//   P' = P_i - X_i M01_{i-1} Y_{i-1}    Q' = Q_i - Y_i M10_{i+1} X_{i+1}
//   X' = -X_i M00_{i-1} X_{i-1}         Y' = -Y_i M11_{i+1} Y_{i+1}
template <class T, int KB>
__global__ void __launch_bounds__(NTOf<KB>::value)
    k_cr_even(const T *__restrict__ Pl, const T *__restrict__ Ql, const T *__restrict__ Xl, const T *__restrict__ Yl,
              const T *__restrict__ Ml, int cnt, T *Pn, T *Qn, T *Xn, T *Yn)
{
    constexpr int NT = NTOf<KB>::value;
    using TL = Tile<T, KB, NT>;
    constexpr size_t TS = (size_t)KB * KB;
    const int i = 2 * blockIdx.x, a_out = blockIdx.x;
    extern __shared__ char smraw[];
    T *sA = (T *)smem_align(smraw), *sB = sA + TL::ELEMS, *sC = sB + TL::ELEMS;
    TL t(threadIdx.x);
    typename TL::Reg acc;
    const bool left = i - 1 >= 0, right = i + 1 < cnt;
    const T *Ml_left = left ? Ml + (size_t)((i - 2) / 2) * 4 * TS : nullptr;  // odd block i-1
    const T *Ml_right = right ? Ml + (size_t)(i / 2) * 4 * TS : nullptr;      // odd block i+1
    // the four results are independent: one CTA each (blockIdx.y), so a level
    // of few blocks still spreads over the SMs
    switch (blockIdx.y) {
    case 0: // P'
        ld<T, KB>(sA, Pl + (size_t)i * TS);
        __syncthreads();
        t.rload(acc, sA);
        if (left)
            chain3<T, KB>(t, acc, Xl + (size_t)i * TS, Ml_left + 1 * TS, Yl + (size_t)(i - 1) * TS, sA, sB, sC, true);
        t.gstore(Pn + (size_t)a_out * TS, acc);
        break;
    case 1: // Q'
        ld<T, KB>(sA, Ql + (size_t)i * TS);
        __syncthreads();
        t.rload(acc, sA);
        if (right)
            chain3<T, KB>(t, acc, Yl + (size_t)i * TS, Ml_right + 2 * TS, Xl + (size_t)(i + 1) * TS, sA, sB, sC, true);
        t.gstore(Qn + (size_t)a_out * TS, acc);
        break;
    case 2: // X'
        t.rzero(acc);
        if (left)
            chain3<T, KB>(t, acc, Xl + (size_t)i * TS, Ml_left + 0 * TS, Xl + (size_t)(i - 1) * TS, sA, sB, sC, true);
        t.gstore(Xn + (size_t)a_out * TS, acc);
        break;
    default: // Y'
        t.rzero(acc);
        if (right)
            chain3<T, KB>(t, acc, Yl + (size_t)i * TS, Ml_right + 3 * TS, Yl + (size_t)(i + 1) * TS, sA, sB, sC, true);
        t.gstore(Yn + (size_t)a_out * TS, acc);
    }
}

// ---------------------------------------------------------------- FP32, KB >= 32: products by column slices
// A level has few blocks (63, 32, 16, ... of 127 interfaces), so its time is that
// of one block.  Columns of a product's right operand are independent through
// all of k_cr_odd's and k_cr_even's formulas but the inverse, so every block's
// products are split into slices of CW columns: a CTA streams the left operands
// through a ring of 32-column pieces while its slice of the right one stays in
// shared memory (FP32 multiply-adds: 128 a clock and SM, where three TF32
// products come to 85).  Level by level: S and its inverse (one CTA; from 128 rows
// on S has a launch of its own), the other quadrants, the even blocks, each launched
// while the one before runs out.  A block to a CTA, with TF32 products: 1,090 us
// for 127 interfaces of 128 rows (99 for an odd block, 35 for an even one), 607
// so; 299 for 155 of 64 rows, 230; 195 for 303 of 32 rows, 136.
template <int KB, int CW> struct ColMul {
    static constexpr int NT = 256, NS = KB / CW, KC = 32, ST = 4;
    static constexpr int TX = CW / 4, RS = NT / TX, RPT = KB / RS; // a thread's rows, RS apart, of 4 columns
    static constexpr int LDA = KC + 4, LDB = CW + 4, NC = KB / KC; // conflict-free 16-byte reads
    static constexpr int RING = ST * KB * LDA, SLICE = KB * LDB;
    static constexpr size_t SMEM = sizeof(float) * (RING + 2 * SLICE);
    using Acc = float[RPT][4];
    float *ring, *b0, *b1; // pieces of the left operands; two slices
    const float *A[2];     // the left operands of the first NC pieces and of the others
    int total;
    __device__ __forceinline__ ColMul(char *sm, int passes) : ring((float *)sm), b0(ring + RING), b1(b0 + SLICE), total(passes * NC) {}
    static __device__ __forceinline__ int row(int i) { return threadIdx.x / TX + RS * i; }
    static __device__ __forceinline__ int col() { return threadIdx.x % TX * 4; }
    __device__ __forceinline__ void issue(int c) const
    {
        if (c < total) {
            const float *src = A[c / NC] + c % NC * KC;
            float *dst = ring + c % ST * KB * LDA;
#pragma unroll
            for (int q = threadIdx.x; q < KB * KC / 4; q += NT)
                cp_async16(dst + q / (KC / 4) * LDA + q % (KC / 4) * 4, src + (size_t)(q / (KC / 4)) * KB + q % (KC / 4) * 4);
        }
        cp_async_commit(); // (empty past the end: the waits count groups)
    }
    // columns [c0, c0 + CW) of a global tile, with the first piece's group
    static __device__ __forceinline__ void slice(float *s, const float *g, int c0)
    {
#pragma unroll
        for (int q = threadIdx.x; q < KB * CW / 4; q += NT)
            cp_async16(s + q / (CW / 4) * LDB + q % (CW / 4) * 4, g + (size_t)(q / (CW / 4)) * KB + c0 + q % (CW / 4) * 4);
    }
    __device__ __forceinline__ void start() const
    {
        for (int c = 0; c < ST - 1; c++) issue(c);
    }
    // acc = A[p] b (and acc2 = A[p] b2): pieces p NC .. p NC + NC - 1
    template <bool TWO> __device__ __forceinline__ void pass(int p, Acc &acc, const float *b, Acc &acc2, const float *b2) const
    {
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = acc2[i][j] = 0.f;
        const int cc = col(), r0 = row(0);
        for (int c = p * NC; c < (p + 1) * NC; c++) {
            cp_async_wait_n<ST - 2>();
            __syncthreads(); // the piece is everyone's, and the one before it has been used
            issue(c + ST - 1);
            const float *a0 = ring + c % ST * KB * LDA + r0 * LDA, *bb = b + c % NC * KC * LDB + cc, *bb2 = b2 + c % NC * KC * LDB + cc;
#pragma unroll 2
            for (int k = 0; k < KC; k += 4) {
                float a[RPT][4];
#pragma unroll
                for (int i = 0; i < RPT; i++) vld<float, 4>(a[i], a0 + RS * i * LDA + k);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    float x[4];
                    vld<float, 4>(x, bb + (k + q) * LDB);
#pragma unroll
                    for (int i = 0; i < RPT; i++)
#pragma unroll
                        for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i][q], x[j], acc[i][j]);
                    if constexpr (TWO) {
                        vld<float, 4>(x, bb2 + (k + q) * LDB);
#pragma unroll
                        for (int i = 0; i < RPT; i++)
#pragma unroll
                            for (int j = 0; j < 4; j++) acc2[i][j] = fmaf(a[i][q], x[j], acc2[i][j]);
                    }
                }
            }
        }
    }
    // f(row, first of four columns of the slice, i) per row of this thread
    template <class F> static __device__ __forceinline__ void each(F f)
    {
#pragma unroll
        for (int i = 0; i < RPT; i++) f(row(i), col(), i);
    }
};

// columns [c0, c0 + CW) of S = I - Q P of odd block j, where M11 goes
template <int KB, int CW>
__global__ void __launch_bounds__(256)
    k_cr_schur(const float *__restrict__ Pl, const float *__restrict__ Ql, int first, int stride, float *M)
{
    using C = ColMul<KB, CW>;
    constexpr size_t TS = (size_t)KB * KB;
    const int c0 = blockIdx.y * CW;
    const size_t o = (size_t)(first + blockIdx.x * stride) * TS;
    float *S = M + (size_t)blockIdx.x * 4 * TS + 3 * TS;
    extern __shared__ __align__(16) char sm[];
    C m(sm, 1);
    m.A[0] = Ql + o;
    dep_launch();
    dep_wait();
    C::slice(m.b0, Pl + o, c0);
    m.start();
    typename C::Acc a, u;
    m.template pass<false>(0, a, m.b0, u, m.b0);
    C::each([&](int r, int c, int i) {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = (r == c0 + c + j ? 1.f : 0.f) - a[i][j];
        vst<float, 4>(S + (size_t)r * KB + c0 + c, v);
    });
}
// M11 = S^{-1} in place
template <int KB>
__global__ void __launch_bounds__(256) k_cr_inv(float *M, unsigned *err)
{
    constexpr int LD = KB + 4;
    float *S = M + ((size_t)blockIdx.x * 4 + 3) * KB * KB;
    extern __shared__ __align__(16) char sm[];
    float *s = (float *)sm;
    dep_launch();
    dep_wait();
    for (int q = threadIdx.x; q < KB * KB / 4; q += 256) {
        float v[4];
        vld<float, 4>(v, S + q * 4);
        vst<float, 4>(s + q / (KB / 4) * LD + q % (KB / 4) * 4, v);
    }
    __syncthreads();
    const bool ok = BlkInv<256, LD>::template run<KB>(s);
    if (!ok) atomicOr(err, SPK_DEV_ERR_PIVOT);
    for (int q = threadIdx.x; q < KB * KB / 4; q += 256) {
        float v[4];
        vld<float, 4>(v, s + q / (KB / 4) * LD + q % (KB / 4) * 4);
        vst<float, 4>(S + q * 4, v);
    }
}
// both at once for tiles whose S one CTA forms soon enough
template <int KB>
__global__ void __launch_bounds__(256)
    k_cr_schur_inv(const float *__restrict__ Pl, const float *__restrict__ Ql, int first, int stride, float *M,
                   unsigned *err)
{
    constexpr int LD = KB + 4;
    using B = BlkMul<KB, 256, LD>;
    const size_t o = (size_t)(first + blockIdx.x * stride) * KB * KB;
    float *S = M + ((size_t)blockIdx.x * 4 + 3) * KB * KB;
    extern __shared__ __align__(16) char sm[];
    float *p = (float *)sm, *q = p + KB * LD;
    dep_launch();
    dep_wait();
    for (int i = threadIdx.x; i < KB * KB / 4; i += 256) {
        cp_async16(p + i / (KB / 4) * LD + i % (KB / 4) * 4, Pl + o + i * 4);
        cp_async16(q + i / (KB / 4) * LD + i % (KB / 4) * 4, Ql + o + i * 4);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    typename B::Acc a;
    B::mul(threadIdx.x, a, q, p);
    __syncthreads();
    B::template put<false, true>(threadIdx.x, p, a);
    __syncthreads();
    if (threadIdx.x < KB) p[threadIdx.x * LD + threadIdx.x] += 1.f;
    __syncthreads();
    const bool ok = BlkInv<256, LD>::template run<KB>(p);
    if (!ok) atomicOr(err, SPK_DEV_ERR_PIVOT);
    for (int i = threadIdx.x; i < KB * KB / 4; i += 256) {
        float v[4];
        vld<float, 4>(v, p + i / (KB / 4) * LD + i % (KB / 4) * 4);
        vst<float, 4>(S + i * 4, v);
    }
}
// columns [c0, c0 + CW) of M10 = -M11 Q, M01 = -P M11, M00 = I - P M10
template <int KB, int CW>
__global__ void __launch_bounds__(256)
    k_cr_quads(const float *__restrict__ Pl, const float *__restrict__ Ql, int first, int stride, float *M)
{
    using C = ColMul<KB, CW>;
    constexpr size_t TS = (size_t)KB * KB;
    const int c0 = blockIdx.y * CW;
    const size_t o = (size_t)(first + blockIdx.x * stride) * TS;
    float *Mj = M + (size_t)blockIdx.x * 4 * TS;
    extern __shared__ __align__(16) char sm[];
    C m(sm, 2);
    m.A[0] = Mj + 3 * TS;
    m.A[1] = Pl + o;
    dep_launch();
    dep_wait();
    C::slice(m.b0, Ql + o, c0);
    C::slice(m.b1, Mj + 3 * TS, c0);
    m.start();
    typename C::Acc a, u;
    m.template pass<false>(0, a, m.b0, u, m.b0);
    __syncthreads(); // Q's slice has been used
    C::each([&](int r, int c, int i) {
        float v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = -a[i][j];
        vst<float, 4>(m.b0 + r * C::LDB + c, v);
        vst<float, 4>(Mj + 2 * TS + (size_t)r * KB + c0 + c, v);
    });
    m.template pass<true>(1, a, m.b1, u, m.b0); // (a barrier before its first read)
    C::each([&](int r, int c, int i) {
        float v[4], w[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[j] = -a[i][j];
            w[j] = (r == c0 + c + j ? 1.f : 0.f) - u[i][j];
        }
        vst<float, 4>(Mj + TS + (size_t)r * KB + c0 + c, v);
        vst<float, 4>(Mj + (size_t)r * KB + c0 + c, w);
    });
}
// columns [c0, c0 + CW) of an even block's result blockIdx.y % 4 (k_cr_even)
//   0: P' = P_i - X_i (M01 Y)_{i-1}   1: Q' = Q_i - Y_i (M10 X)_{i+1}
//   2: X' = -X_i (M00 X)_{i-1}        3: Y' = -Y_i (M11 Y)_{i+1}
template <int KB, int CW>
__global__ void __launch_bounds__(256)
    k_cr_even_cols(const float *__restrict__ Pl, const float *__restrict__ Ql, const float *__restrict__ Xl,
                   const float *__restrict__ Yl, const float *__restrict__ Ml, int cnt, float *Pn, float *Qn, float *Xn,
                   float *Yn)
{
    using C = ColMul<KB, CW>;
    constexpr size_t TS = (size_t)KB * KB;
    const int i = 2 * blockIdx.x, w = blockIdx.y % 4, c0 = blockIdx.y / 4 * CW;
    const bool lft = w == 0 || w == 2, has = lft ? i > 0 : i + 1 < cnt;
    const int j = lft ? i - 1 : i + 1;
    const float *base = w == 0 ? Pl + (size_t)i * TS : w == 1 ? Ql + (size_t)i * TS : nullptr;
    float *out = (w == 0 ? Pn : w == 1 ? Qn : w == 2 ? Xn : Yn) + (size_t)blockIdx.x * TS;
    extern __shared__ __align__(16) char sm[];
    C m(sm, 2);
    dep_launch();
    dep_wait();
    typename C::Acc a, u;
    if (has) {
        m.A[0] = Ml + ((size_t)(j / 2) * 4 + (w == 0 ? 1 : w == 1 ? 2 : w == 2 ? 0 : 3)) * TS;
        m.A[1] = (lft ? Xl : Yl) + (size_t)i * TS;
        C::slice(m.b0, (w == 0 || w == 3 ? Yl : Xl) + (size_t)j * TS, c0);
        m.start();
        m.template pass<false>(0, a, m.b0, u, m.b0);
        C::each([&](int r, int c, int q) { vst<float, 4>(m.b1 + r * C::LDB + c, a[q]); });
        m.template pass<false>(1, a, m.b1, u, m.b1); // (a barrier before its first read)
    } else { // no neighbour on this side: P' = P_i, Q' = Q_i, X' = Y' = 0
#pragma unroll
        for (int q = 0; q < C::RPT; q++)
#pragma unroll
            for (int k = 0; k < 4; k++) a[q][k] = 0.f;
    }
    C::each([&](int r, int c, int q) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (base) vld<float, 4>(v, base + (size_t)r * KB + c0 + c);
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] -= a[q][k];
        vst<float, 4>(out + (size_t)r * KB + c0 + c, v);
    });
}

// ------------------------------------------------------------ KB <= 16 (8 in FP64): segments of several levels
// The factorization's counterpart of the solve's segments (spike_redsolve.cu):
// of an even block's four results P' and X' depend on its left odd neighbour
// only, Q' and Y' on its right one, so a CTA takes a segment between two
// survivors through several levels on its own -- a group of GL lanes per tile
// product, everything in shared memory.  One launch per level and parity took
// 127 us for 2,431 interfaces of 8-row tiles (11 levels of two launches of
// 3.5 to 6 us each and four conversions); 42 us.
template <class T, int KB> struct RfCfg {
    static constexpr int TS = KB * KB;
    static constexpr int GL = TS < 32 ? TS : 32; // lanes per tile
    static constexpr int EPL = TS / GL;          // elements per lane
    static constexpr int SCR = TS + 4 * KB;      // scratch elements per group: a tile, the pivot rows and columns
};

template <class T, int KB, int NT>
__global__ void __launch_bounds__(NT)
    k_rf_seg(T *gP, T *gQ, T *gX, T *gY, T *gM, const __grid_constant__ RsLevels lv, int l0, int l1, int top,
             unsigned *err)
{
    using C = RfCfg<T, KB>;
    constexpr int TS = C::TS, GL = C::GL, EPL = C::EPL, NG = NT / GL;
    const int s = l1 - l0, full = 1 << s;
    int b = top ? 0 : (int)blockIdx.x << s;
    const int left = lv.cnt[l0] - b, n0 = top || left <= full ? left : full + 1;
    int end = top || left <= full ? 1 << 30 : full; // the right survivor: only its P' and X' are ours
    const bool first = b == 0;
    extern __shared__ __align__(16) char smraw[];
    T *cur = (T *)smraw;                        // P, Q, X, Y of the level's blocks
    T *nxt = cur + (size_t)4 * n0 * TS;         // of the next level's
    T *sM = nxt + (size_t)4 * ((n0 + 1) / 2) * TS; // four tiles per odd block
    T *scr = sM + (size_t)4 * (n0 / 2 > 0 ? n0 / 2 : 1) * TS;
    const int grp = threadIdx.x / GL, e0 = threadIdx.x % GL;
    const unsigned gm = GL == 32 ? 0xffffffffu : ((1u << GL) - 1u) << ((threadIdx.x & 31) / GL * GL);
    T *tmp = scr + (size_t)grp * C::SCR, *piv = tmp + TS;
    bool ok = true;

    auto er = [&](int q) { return (e0 + q * GL) / KB; };
    auto ec = [&](int q) { return (e0 + q * GL) % KB; };
    // acc -= A B (dense shared tiles)
    auto msub_t = [&](T (&acc)[EPL], const T *A, const T *B) {
#pragma unroll
        for (int q = 0; q < EPL; q++)
#pragma unroll
            for (int k = 0; k < KB; k++) acc[q] = msub(acc[q], A[er(q) * KB + k], B[k * KB + ec(q)]);
    };
    auto madd_t = [&](T (&acc)[EPL], const T *A, const T *B) {
#pragma unroll
        for (int q = 0; q < EPL; q++)
#pragma unroll
            for (int k = 0; k < KB; k++) acc[q] = madd(acc[q], A[er(q) * KB + k], B[k * KB + ec(q)]);
    };
    auto put = [&](T *d, const T (&v)[EPL]) {
#pragma unroll
        for (int q = 0; q < EPL; q++) d[e0 + q * GL] = v[q];
    };
    // M = D^{-1} of the block with tiles P, Q, by quadrants: S = I - Q P, M11 =
    // S^{-1}, M10 = -M11 Q, M01 = -P M11, M00 = I - P M10
    auto odd = [&](const T *P, const T *Q, T *M, T *out) {
        T a[EPL];
#pragma unroll
        for (int q = 0; q < EPL; q++) a[q] = er(q) == ec(q) ? sc_one<T>() : sc_zero<T>();
        msub_t(a, Q, P);
        // Gauss-Jordan without pivoting, row and column of the pivot through shared memory
        for (int j = 0; j < KB; j++) {
            T *row = piv + (j & 1) * 2 * KB, *col = row + KB;
#pragma unroll
            for (int q = 0; q < EPL; q++) {
                if (er(q) == j) row[ec(q)] = a[q];
                if (ec(q) == j) col[er(q)] = a[q];
            }
            __syncwarp(gm);
            const T p = col[j];
            if (!sc_finite_nonzero(p)) ok = false;
            const T pr = sc_frcp(p);
#pragma unroll
            for (int q = 0; q < EPL; q++) {
                const T bv = row[ec(q)] * pr, av = col[er(q)];
                a[q] = ec(q) == j ? (er(q) == j ? pr : -(av * pr)) : er(q) == j ? bv : msub(a[q], av, bv);
            }
        }
        put(M + 3 * TS, a);
        put(out + 3 * TS, a);
        __syncwarp(gm);
        T z[EPL];
#pragma unroll
        for (int q = 0; q < EPL; q++) a[q] = z[q] = sc_zero<T>();
        msub_t(a, M + 3 * TS, Q);
        msub_t(z, P, M + 3 * TS);
        put(M + 2 * TS, a);
        put(out + 2 * TS, a);
        put(M + TS, z);
        put(out + TS, z);
        __syncwarp(gm);
#pragma unroll
        for (int q = 0; q < EPL; q++) a[q] = er(q) == ec(q) ? sc_one<T>() : sc_zero<T>();
        msub_t(a, P, M + 2 * TS);
        put(M, a);
        put(out, a);
    };

    dep_launch();
    dep_wait();
    {
        const size_t o = (size_t)(lv.off[l0] + b) * TS;
        for (int q = threadIdx.x; q < n0 * TS; q += NT) {
            cur[q] = gP[o + q];
            cur[(size_t)n0 * TS + q] = gQ[o + q];
            cur[(size_t)2 * n0 * TS + q] = gX[o + q];
            cur[(size_t)3 * n0 * TS + q] = gY[o + q];
        }
    }
    __syncthreads();
    int nl = n0;
    for (int l = l0; l < l1; l++) {
        const int nodd = nl >> 1, nn = (nl + 1) >> 1;
        const T *P = cur, *Q = P + (size_t)nl * TS, *X = Q + (size_t)nl * TS, *Y = X + (size_t)nl * TS;
        for (int j = grp; j < nodd; j += NG)
            odd(P + (size_t)(2 * j + 1) * TS, Q + (size_t)(2 * j + 1) * TS, sM + (size_t)j * 4 * TS,
                gM + (size_t)(lv.moff[l] + b / 2 + j) * 4 * TS);
        __syncthreads();
        // P' = P_i - X_i (M01 Y)_{i-1}, Q' = Q_i - Y_i (M10 X)_{i+1}, X' = -X_i (M00 X)_{i-1}, Y' = -Y_i (M11 Y)_{i+1}
        for (int it = grp; it < 4 * nn; it += NG) {
            const int a = it >> 2, w = it & 3, i = 2 * a;
            const bool lft = w == 0 || w == 2;
            const int j = lft ? i - 1 : i + 1;
            T v[EPL];
#pragma unroll
            for (int q = 0; q < EPL; q++)
                v[q] = w == 0 ? P[(size_t)i * TS + e0 + q * GL] : w == 1 ? Q[(size_t)i * TS + e0 + q * GL] : sc_zero<T>();
            if (lft ? j >= 0 : j < nl) {
                const T *M = sM + (size_t)(j >> 1) * 4 * TS;
                T m[EPL];
#pragma unroll
                for (int q = 0; q < EPL; q++) m[q] = sc_zero<T>();
                madd_t(m, M + (w == 0 ? 1 : w == 1 ? 2 : w == 2 ? 0 : 3) * TS,
                       (w == 0 || w == 3 ? Y : X) + (size_t)j * TS);
                put(tmp, m);
                __syncwarp(gm);
                msub_t(v, (lft ? X : Y) + (size_t)i * TS, tmp);
                __syncwarp(gm); // tmp is free again
            }
            put(nxt + (size_t)(w * nn + a) * TS, v);
            if (lft ? (i > 0 || first) : i < end)
                put((w == 0 ? gP : w == 1 ? gQ : w == 2 ? gX : gY) + (size_t)(lv.off[l + 1] + b / 2 + a) * TS, v);
        }
        __syncthreads();
        T *sw = cur;
        cur = nxt;
        nxt = sw;
        nl = nn;
        b >>= 1;
        end >>= 1;
    }
    if (top && grp == 0) odd(cur, cur + TS, sM, gM + (size_t)lv.moff[lv.L] * 4 * TS); // the last single block
    if (!ok && e0 == 0) atomicOr(err, SPK_DEV_ERR_PIVOT);
}

template <class T, int KB> int run_red_factor_s(spk_plan *P, cudaStream_t st)
{
    using C = RfCfg<T, KB>;
    constexpr int NT = 256, NTT = 512;
    constexpr size_t SMEM = 220 * 1024;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_rf_seg<T, KB, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_rf_seg<T, KB, NTT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) !=
                cudaSuccess)
            return SPK_ECUDA;
        attr = true;
    }
    RsLevels lv;
    if (!rs_levels(P, lv)) return SPK_EARG;
    auto bytes = [](int n, int, bool top) {
        const size_t tiles = 4 * (size_t)n + 4 * ((n + 1) / 2) + 4 * (size_t)(n / 2 > 0 ? n / 2 : 1);
        return (tiles * C::TS + (size_t)(top ? NTT : NT) / C::GL * C::SCR) * sizeof(T) + 16;
    };
    int tier[RS_MAXL + 1], nt;
    const int lt = rs_schedule(lv, SMEM, bytes, tier, nt);
    bool dep = false;
    auto run = [&](auto kern, int grid, int nthr, size_t smem, int l0, int l1, int top) {
        const int rc = launch_dep(kern, dim3(grid), nthr, smem, 1, dep, st, (T *)P->d_crP, (T *)P->d_crQ,
                                  (T *)P->d_crX, (T *)P->d_crY, (T *)P->d_crM, lv, l0, l1, top, P->d_err);
        dep = chained(P);
        P->launches++;
        return rc;
    };
    for (int q = 0; q < nt; q++) {
        const int l0 = tier[q], l1 = tier[q + 1], s = l1 - l0;
        if (run(k_rf_seg<T, KB, NT>, (lv.cnt[l0] + (1 << s) - 1) >> s, NT, bytes((1 << s) + 1, s, false), l0, l1, 0) !=
            SPK_OK)
            return SPK_ECUDA;
    }
    return run(k_rf_seg<T, KB, NTT>, 1, NTT, bytes(lv.cnt[lt], lv.L - lt, true), lt, lv.L, 1);
}

template <int KB> int run_red_factor_c(spk_plan *P, cudaStream_t st)
{
    using C = ColMul<KB, 32>;
    constexpr int FINE = KB == 32 ? 32 : 16;
    using C2 = ColMul<KB, FINE>;
    constexpr size_t TS = (size_t)KB * KB, INV = sizeof(float) * KB * (KB + 4);
    static bool attr = false;
    if (!attr) {
        const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
        if (cudaFuncSetAttribute(k_cr_quads<KB, 32>, a, (int)C::SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(k_cr_even_cols<KB, 32>, a, (int)C::SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(k_cr_quads<KB, FINE>, a, (int)C2::SMEM) != cudaSuccess ||
            cudaFuncSetAttribute(k_cr_even_cols<KB, FINE>, a, (int)C2::SMEM) != cudaSuccess)
            return SPK_ECUDA;
        if constexpr (KB <= 64) {
            if (cudaFuncSetAttribute(k_cr_schur_inv<KB>, a, (int)(2 * INV)) != cudaSuccess) return SPK_ECUDA;
        } else {
            if (cudaFuncSetAttribute(k_cr_schur<KB, 32>, a, (int)C::SMEM) != cudaSuccess ||
                cudaFuncSetAttribute(k_cr_schur<KB, FINE>, a, (int)C2::SMEM) != cudaSuccess ||
                cudaFuncSetAttribute(k_cr_inv<KB>, a, (int)INV) != cudaSuccess)
                return SPK_ECUDA;
        }
        attr = true;
    }
    float *cP = (float *)P->d_crP, *cQ = (float *)P->d_crQ, *cX = (float *)P->d_crX, *cY = (float *)P->d_crY,
          *cM = (float *)P->d_crM;
    bool dep = false; // (what ran before these kernels does not let them start early)
    int rc = SPK_OK;
    auto run = [&](auto kern, dim3 grid, size_t smem, auto... args) {
        if (rc == SPK_OK) rc = launch_dep(kern, grid, C::NT, smem, 1, dep, st, args...);
        dep = chained(P);
        P->launches++;
    };
    auto odd = [&](const float *p, const float *q, int first, int stride, int count, float *M) {
        // slices of 16 columns while they leave an SM to each
        const bool fine = count * C2::NS <= 152;
        if constexpr (KB <= 64) {
            run(k_cr_schur_inv<KB>, dim3(count), 2 * INV, p, q, first, stride, M, P->d_err);
        } else {
            if (fine)
                run(k_cr_schur<KB, FINE>, dim3(count, C2::NS), C2::SMEM, p, q, first, stride, M);
            else
                run(k_cr_schur<KB, 32>, dim3(count, C::NS), C::SMEM, p, q, first, stride, M);
            run(k_cr_inv<KB>, dim3(count), INV, M, P->d_err);
        }
        if (fine)
            run(k_cr_quads<KB, FINE>, dim3(count, C2::NS), C2::SMEM, p, q, first, stride, M);
        else
            run(k_cr_quads<KB, 32>, dim3(count, C::NS), C::SMEM, p, q, first, stride, M);
    };
    for (int l = 0; l < P->cr_levels; l++) {
        const int cnt = P->cr_count[l];
        const size_t o = (size_t)P->cr_off[l] * TS, on = (size_t)P->cr_off[l + 1] * TS;
        float *Ml = cM + (size_t)P->cr_moff[l] * 4 * TS;
        if (cnt / 2 > 0) odd(cP + o, cQ + o, 1, 2, cnt / 2, Ml);
        auto even = [&](auto kern, int ns, size_t smem) {
            run(kern, dim3((cnt + 1) / 2, 4 * ns), smem, (const float *)cP + o, (const float *)cQ + o,
                (const float *)cX + o, (const float *)cY + o, (const float *)Ml, cnt, cP + on, cQ + on, cX + on, cY + on);
        };
        if ((cnt + 1) / 2 * 4 * C2::NS <= 152)
            even(k_cr_even_cols<KB, FINE>, C2::NS, C2::SMEM);
        else
            even(k_cr_even_cols<KB, 32>, C::NS, C::SMEM);
    }
    const size_t o = (size_t)P->cr_off[P->cr_levels] * TS; // the top block
    odd(cP + o, cQ + o, 0, 1, 1, cM + (size_t)P->cr_moff[P->cr_levels] * 4 * TS);
    return rc;
}

template <class T, int KB> int run_red_factor(spk_plan *P, cudaStream_t st)
{
    using S = RedSmem<T, KB>;
    constexpr int NT = NTOf<KB>::value;
    constexpr size_t TS = (size_t)KB * KB;
    using H = typename HighOf<T>::type;
    if (!P->red_direct) { // the blocks come in FP64 (a sharded solve's records)
        const long long c0 = (long long)P->n_iface * TS;
        k_red_cvt<T><<<256, 256, 0, st>>>((const H *)P->d_RP, (T *)P->d_crP, c0);
        k_red_cvt<T><<<256, 256, 0, st>>>((const H *)P->d_RQ, (T *)P->d_crQ, c0);
        k_red_cvt<T><<<256, 256, 0, st>>>((const H *)P->d_RX, (T *)P->d_crX, c0);
        k_red_cvt<T><<<256, 256, 0, st>>>((const H *)P->d_RY, (T *)P->d_crY, c0);
        SPK_CHECK_LAUNCH();
        P->launches += 4;
    }
    // (a group of 32 lanes takes a 16-row tile's FP64 products and pivots too long:
    // n = 50,000, k = 16 1,118 us a solve in segments, 1,003 with a CTA per block and
    // level; complex128 3,985 and 2,784)
    constexpr bool LOW = std::is_same<T, float>::value || std::is_same<T, cfloat>::value;
    if constexpr (KB <= 8 || (KB == 16 && LOW)) {
        return run_red_factor_s<T, KB>(P, st);
    } else if constexpr (std::is_same<T, float>::value) {
        return run_red_factor_c<KB>(P, st);
    } else {
    // FP64 with 64-row tiles: the products on the tensor cores, by exact digits (spike_emu64.cu)
    constexpr bool EMU = std::is_same<T, double>::value && KB == 64;
    static bool attr = false;
    if (!attr) {
        if constexpr (!EMU) {
            if (cudaFuncSetAttribute(k_cr_odd<T, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes) !=
                    cudaSuccess ||
                cudaFuncSetAttribute(k_cr_even<T, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes) !=
                    cudaSuccess)
                return SPK_ECUDA;
        }
        attr = true;
    }
    auto odd = [&](const T *Pp, const T *Qp, int first, int stride, int count, T *Mo) -> int {
        if constexpr (EMU)
            return spk_emu_cr_odd(Pp, Qp, first, stride, count, Mo, P->d_err, st);
        else {
            k_cr_odd<T, KB><<<count, NT, S::bytes, st>>>(Pp, Qp, first, stride, Mo, P->d_err);
            SPK_CHECK_LAUNCH();
            return SPK_OK;
        }
    };
    T *cP = (T *)P->d_crP, *cQ = (T *)P->d_crQ, *cX = (T *)P->d_crX, *cY = (T *)P->d_crY, *cM = (T *)P->d_crM;
    auto even = [&](size_t o, size_t on, const T *Ml, int cnt) -> int {
        if constexpr (EMU)
            return spk_emu_cr_even(cP + o, cQ + o, cX + o, cY + o, Ml, cnt, cP + on, cQ + on, cX + on, cY + on, st);
        else {
            k_cr_even<T, KB><<<dim3((cnt + 1) / 2, 4), NT, S::bytes, st>>>(cP + o, cQ + o, cX + o, cY + o, Ml, cnt, cP + on,
                                                                          cQ + on, cX + on, cY + on);
            SPK_CHECK_LAUNCH();
            return SPK_OK;
        }
    };
    for (int l = 0; l < P->cr_levels; l++) {
        const int cnt = P->cr_count[l];
        const size_t o = (size_t)P->cr_off[l] * TS, on = (size_t)P->cr_off[l + 1] * TS;
        T *Ml = cM + (size_t)P->cr_moff[l] * 4 * TS;
        int rc = cnt / 2 > 0 ? odd(cP + o, cQ + o, 1, 2, cnt / 2, Ml) : SPK_OK;
        if (rc == SPK_OK) rc = even(o, on, Ml, cnt);
        if (rc != SPK_OK) return rc;
        P->launches += 2;
    }
    // top: a single block
    const size_t o = (size_t)P->cr_off[P->cr_levels] * TS;
    const int rc = odd(cP + o, cQ + o, 0, 1, 1, cM + (size_t)P->cr_moff[P->cr_levels] * 4 * TS);
    P->launches++;
    return rc;
    }
}

#define SPK_KB_SWITCH(FN, T, ...)                                                                               \
    switch (P->KB) {                                                                                            \
    case 2: return FN<T, 2>(__VA_ARGS__);                                                                       \
    case 4: return FN<T, 4>(__VA_ARGS__);                                                                       \
    case 8: return FN<T, 8>(__VA_ARGS__);                                                                       \
    case 16: return FN<T, 16>(__VA_ARGS__);                                                                     \
    case 32: return FN<T, 32>(__VA_ARGS__);                                                                     \
    case 64:                                                                                                    \
        if constexpr (sizeof(T) <= 8) return FN<T, 64>(__VA_ARGS__);                                            \
        else return SPK_EBAND;                                                                                  \
    case 128:                                                                                                   \
        if constexpr (std::is_same<T, float>::value) return FN<T, 128>(__VA_ARGS__);                            \
        else return SPK_EBAND;                                                                                  \
    default: return SPK_EBAND;                                                                                  \
    }

template <class T> int disp_rf(spk_plan *P, cudaStream_t st) { SPK_KB_SWITCH(run_red_factor, T, P, st) }

} // namespace

extern "C" int spk_reduced_factor(spk_plan *P, void *stream)
{
    if (P->n_iface <= 0) return SPK_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const bool low = P->mode == SPK_MIXED && !P->red_fp64; // factor-precision cyclic reduction
    if (P->is_complex) return low ? disp_rf<cfloat>(P, st) : disp_rf<cdouble>(P, st);
    return low ? disp_rf<float>(P, st) : disp_rf<double>(P, st);
}
