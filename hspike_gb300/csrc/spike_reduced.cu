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

// ---------------------------------------------------------------- tensor-core products
// The reduced system's 2KB x 2KB block products for KB >= 64 (FP32 factors)
// run on the tensor cores: warp-level mma.sync m16n8k8 with TF32 operands,
// each FP32 operand split into a TF32 high part and a TF32 remainder, and
// the three significant partial products (lo*hi, hi*lo, hi*hi) accumulated
// in FP32, which keeps FP32 accuracy.  Warp w of the CTA (KB*KB/512 warps:
// the Tile kernels' own thread count) owns the 32 x 16 output block at rows
// 32 (w / (KB/16)), columns 16 (w % (KB/16)); operands are shared tiles in
// the Tile layout (row-major, row stride KB + 4).
__device__ __forceinline__ void tf32_split(float x, uint32_t &hi, uint32_t &lo)
{
    uint32_t h, l;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(x - __uint_as_float(h)));
    hi = h;
    lo = l;
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2])
{
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
using TcAcc = float[2][2][4];
__device__ __forceinline__ void tc_zero(TcAcc &acc)
{
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[i][j][e] = 0.f;
}
// acc += A B (A, B: KB x KB shared tiles, row-major, row stride KB + 4)
template <int KB> __device__ __forceinline__ void tc_mm(TcAcc &acc, const float *A, const float *B)
{
    constexpr int LD = TileLD<float, KB>::value;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = (warp / (KB / 16)) * 32, c0 = (warp % (KB / 16)) * 16;
#pragma unroll 2
    for (int k0 = 0; k0 < KB; k0 += 8) {
        uint32_t ah[2][4], al[2][4], bh[2][2], bl[2][2];
#pragma unroll
        for (int i = 0; i < 2; i++) { // A fragment: (g, t), (g + 8, t), (g, t + 4), (g + 8, t + 4)
            const float *Ar = A + (r0 + i * 16 + g) * LD + k0 + t;
            tf32_split(Ar[0], ah[i][0], al[i][0]);
            tf32_split(Ar[8 * LD], ah[i][1], al[i][1]);
            tf32_split(Ar[4], ah[i][2], al[i][2]);
            tf32_split(Ar[8 * LD + 4], ah[i][3], al[i][3]);
        }
#pragma unroll
        for (int j = 0; j < 2; j++) { // B fragment: (t, g), (t + 4, g)
            const float *Bc = B + (k0 + t) * LD + c0 + j * 8 + g;
            tf32_split(Bc[0], bh[j][0], bl[j][0]);
            tf32_split(Bc[4 * LD], bh[j][1], bl[j][1]);
        }
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                mma_tf32(acc[i][j], al[i], bh[j]);
                mma_tf32(acc[i][j], ah[i], bl[j]);
                mma_tf32(acc[i][j], ah[i], bh[j]);
            }
    }
}
// f(row, col, value) for every accumulator element this thread holds:
// (g, 2t), (g, 2t + 1), (g + 8, 2t), (g + 8, 2t + 1) of each 16 x 8 block
template <int KB, class F> __device__ __forceinline__ void tc_each(const TcAcc &acc, F f)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int r0 = (warp / (KB / 16)) * 32, c0 = (warp % (KB / 16)) * 16;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) f(r0 + i * 16 + g + (e >> 1) * 8, c0 + j * 8 + 2 * t + (e & 1), acc[i][j][e]);
}

// k_cr_odd with tensor-core products: S = I - Q P, M11 = S^{-1} (the Tile
// inverse), M10 = -M11 Q, M01 = -P M11, M00 = I - P M10.
template <int KB>
__global__ void __launch_bounds__(NTOf<KB>::value)
    k_cr_odd_tc(const float *__restrict__ Pl, const float *__restrict__ Ql, int first, int stride, float *M,
                unsigned *err)
{
    constexpr int NT = NTOf<KB>::value, LD = TileLD<float, KB>::value;
    using TL = Tile<float, KB, NT>;
    constexpr size_t TS = (size_t)KB * KB;
    static_assert(NT == KB * KB / 16, "one warp per 32 x 16 output block");
    const int j = first + blockIdx.x * stride;
    float *Mj = M + (size_t)blockIdx.x * 4 * TS;
    extern __shared__ char smraw[];
    float *sP = (float *)smem_align(smraw), *sQ = sP + TL::ELEMS, *sH = sQ + TL::ELEMS;
    float *buf = sH + TL::ELEMS;
    TL t(threadIdx.x);
    typename TL::Reg a;
    TcAcc acc;
    ld<float, KB>(sP, Pl + (size_t)j * TS);
    ld<float, KB>(sQ, Ql + (size_t)j * TS);
    __syncthreads();
    tc_zero(acc);
    tc_mm<KB>(acc, sQ, sP);
    tc_each<KB>(acc, [&](int r, int c, float v) { sH[r * LD + c] = (r == c ? 1.f : 0.f) - v; }); // S
    __syncthreads();
    t.rload(a, sH);
    __syncthreads();
    bool ok;
    if constexpr (KB == 64)
        ok = t.inverse_blk(a, sH);
    else
        ok = t.inverse(a, buf);
    if (!ok && threadIdx.x == 0) atomicOr(err, SPK_DEV_ERR_PIVOT);
    __syncthreads();
    t.rstore(sH, a); // M11
    t.gstore(Mj + 3 * TS, a);
    __syncthreads();
    tc_zero(acc);
    tc_mm<KB>(acc, sH, sQ);
    tc_each<KB>(acc, [&](int r, int c, float v) { Mj[2 * TS + r * KB + c] = -v; }); // M10
    __syncthreads(); // every read of Q is done
    tc_each<KB>(acc, [&](int r, int c, float v) { sQ[r * LD + c] = -v; });
    tc_zero(acc);
    tc_mm<KB>(acc, sP, sH);
    tc_each<KB>(acc, [&](int r, int c, float v) { Mj[TS + r * KB + c] = -v; }); // M01
    __syncthreads();
    tc_zero(acc);
    tc_mm<KB>(acc, sP, sQ);
    tc_each<KB>(acc, [&](int r, int c, float v) { Mj[r * KB + c] = (r == c ? 1.f : 0.f) - v; }); // M00
}

// k_cr_even with tensor-core products: blockIdx.y picks the result
//   0: P' = P_i - X_i (M01 Y)_{i-1}   1: Q' = Q_i - Y_i (M10 X)_{i+1}
//   2: X' = -X_i (M00 X)_{i-1}        3: Y' = -Y_i (M11 Y)_{i+1}
template <int KB>
__global__ void __launch_bounds__(NTOf<KB>::value)
    k_cr_even_tc(const float *__restrict__ Pl, const float *__restrict__ Ql, const float *__restrict__ Xl,
                 const float *__restrict__ Yl, const float *__restrict__ Ml, int cnt, float *Pn, float *Qn,
                 float *Xn, float *Yn)
{
    constexpr int NT = NTOf<KB>::value, LD = TileLD<float, KB>::value;
    using TL = Tile<float, KB, NT>;
    constexpr size_t TS = (size_t)KB * KB;
    const int i = 2 * blockIdx.x, a_out = blockIdx.x, which = blockIdx.y;
    const bool left = i - 1 >= 0, right = i + 1 < cnt;
    const bool has = (which == 0 || which == 2) ? left : right;
    const float *base = which == 0 ? Pl + (size_t)i * TS : which == 1 ? Ql + (size_t)i * TS : nullptr;
    float *out = (which == 0 ? Pn : which == 1 ? Qn : which == 2 ? Xn : Yn) + (size_t)a_out * TS;
    if (!has) { // no neighbour on this side: P' = P_i, Q' = Q_i, X' = Y' = 0
        for (int q = threadIdx.x; q < KB * KB; q += NT) out[q] = base ? base[q] : 0.f;
        return;
    }
    const float *Mnb = Ml + (size_t)(left && (which == 0 || which == 2) ? (i - 2) / 2 : i / 2) * 4 * TS;
    const float *Lt = (which == 0 || which == 2 ? Xl : Yl) + (size_t)i * TS;
    const float *Mq = Mnb + (size_t)(which == 0 ? 1 : which == 1 ? 2 : which == 2 ? 0 : 3) * TS;
    const float *Rt = (which == 0 || which == 3 ? Yl : Xl) + (size_t)(which == 0 || which == 2 ? i - 1 : i + 1) * TS;
    extern __shared__ char smraw[];
    float *sA = (float *)smem_align(smraw), *sB = sA + TL::ELEMS, *sC = sB + TL::ELEMS;
    ld<float, KB>(sA, Mq);
    ld<float, KB>(sB, Rt);
    __syncthreads();
    TcAcc acc;
    tc_zero(acc);
    tc_mm<KB>(acc, sA, sB);
    tc_each<KB>(acc, [&](int r, int c, float v) { sC[r * LD + c] = v; });
    __syncthreads();
    ld<float, KB>(sA, Lt);
    __syncthreads();
    tc_zero(acc);
    tc_mm<KB>(acc, sA, sC);
    tc_each<KB>(acc, [&](int r, int c, float v) { out[r * KB + c] = (base ? base[r * KB + c] : 0.f) - v; });
}

// ------------------------------------------------------------ KB <= 16: segments of several levels
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
        dep = true;
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
    if constexpr (KB <= 16) {
        return run_red_factor_s<T, KB>(P, st);
    } else {
    // FP32 factors with 64- or 128-row tiles: the block products on the tensor cores
    constexpr bool TC = std::is_same<T, float>::value && (KB == 64 || KB == 128);
    // FP64 with 64-row tiles: likewise, by exact digit products (spike_emu64.cu)
    constexpr bool EMU = std::is_same<T, double>::value && KB == 64;
    static bool attr = false;
    if (!attr) {
        if constexpr (!TC && !EMU) {
            if (cudaFuncSetAttribute(k_cr_odd<T, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes) !=
                    cudaSuccess ||
                cudaFuncSetAttribute(k_cr_even<T, KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes) !=
                    cudaSuccess)
                return SPK_ECUDA;
        }
        if constexpr (TC) {
            if (cudaFuncSetAttribute(k_cr_odd_tc<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes) !=
                    cudaSuccess ||
                cudaFuncSetAttribute(k_cr_even_tc<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes) !=
                    cudaSuccess)
                return SPK_ECUDA;
        }
        attr = true;
    }
    auto odd = [&](const T *Pp, const T *Qp, int first, int stride, int count, T *Mo) {
        if constexpr (EMU)
            spk_emu_cr_odd(Pp, Qp, first, stride, count, Mo, P->d_err, st);
        else if constexpr (TC)
            k_cr_odd_tc<KB><<<count, NT, S::bytes, st>>>(Pp, Qp, first, stride, Mo, P->d_err);
        else
            k_cr_odd<T, KB><<<count, NT, S::bytes, st>>>(Pp, Qp, first, stride, Mo, P->d_err);
    };
    T *cP = (T *)P->d_crP, *cQ = (T *)P->d_crQ, *cX = (T *)P->d_crX, *cY = (T *)P->d_crY, *cM = (T *)P->d_crM;
    for (int l = 0; l < P->cr_levels; l++) {
        const int cnt = P->cr_count[l];
        const size_t o = (size_t)P->cr_off[l] * TS, on = (size_t)P->cr_off[l + 1] * TS;
        T *Ml = cM + (size_t)P->cr_moff[l] * 4 * TS;
        const int nodd = cnt / 2, neven = (cnt + 1) / 2;
        if (nodd > 0) {
            odd(cP + o, cQ + o, 1, 2, nodd, Ml);
            SPK_CHECK_LAUNCH();
        }
        if constexpr (EMU)
            spk_emu_cr_even(cP + o, cQ + o, cX + o, cY + o, Ml, cnt, cP + on, cQ + on, cX + on, cY + on, st);
        else if constexpr (TC)
            k_cr_even_tc<KB><<<dim3(neven, 4), NT, S::bytes, st>>>(cP + o, cQ + o, cX + o, cY + o, Ml, cnt, cP + on,
                                                                   cQ + on, cX + on, cY + on);
        else
            k_cr_even<T, KB><<<dim3(neven, 4), NT, S::bytes, st>>>(cP + o, cQ + o, cX + o, cY + o, Ml, cnt, cP + on,
                                                                   cQ + on, cX + on, cY + on);
        SPK_CHECK_LAUNCH();
        P->launches += 2;
    }
    // top: a single block
    {
        const int L = P->cr_levels;
        const size_t o = (size_t)P->cr_off[L] * TS;
        odd(cP + o, cQ + o, 0, 1, 1, cM + (size_t)P->cr_moff[L] * 4 * TS);
        SPK_CHECK_LAUNCH();
        P->launches++;
    }
    return SPK_OK;
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
