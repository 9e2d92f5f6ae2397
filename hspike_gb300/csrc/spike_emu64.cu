// spike_emu64.cu -- plain-FP64 factorization chains of 64-row tiles (real data)
// with their products on the tensor cores (spike_emu64.cuh).
//
// The recurrences and global layouts are those of k_factor_fwd / k_factor_bwd
// (spike_factor.cu) and k_cr_odd / k_cr_even (spike_reduced.cu), which the FP64
// pipe bounds: 73 + 55 + 5 ms of the 139 ms of n = 2,000,000, k = 64 in plain
// FP64, for 3 KB^3 multiply-adds per block and direction.  With digit products
// the three take 35 + 16 + 3 ms: a step's three products 23,000 clocks each, its
// inverse 134,000.  One CTA of 256 threads fills an SM: the right operand's digit
// planes take 83 KB, three working tiles 111 KB, and the next block's coupling
// tiles arrive by bulk copies in what is free.
#include "spike_emu64.cuh"

#include <type_traits>

namespace {

template <int KB> struct EmuSmem {
    using E = Emu<KB>;
    static constexpr size_t tile = sizeof(double) * E::TILE;
    static constexpr size_t ctile = sizeof(double) * KB * E::LDC;
    static constexpr size_t head = 64 + E::AUX; // mbarriers, scales, lists
    static constexpr size_t fwd = head + E::PLANES + 3 * tile + ctile;
    static constexpr size_t bwd = head + E::PLANES + 2 * tile + 2 * ctile;
    static constexpr size_t red = head + E::PLANES + 4 * tile;
};

// L_J = F G, S_J = D - L E, G_J = S^{-1}, z_J = -L z_{J-1} (z_0 = C^)
template <int KB>
__global__ void __launch_bounds__(Emu<KB>::NT, 1)
    k_emu_fwd(const double *__restrict__ gT, const int *__restrict__ blk_off, double *gL, double *gG, double *gZ,
              unsigned *err)
{
    using E = Emu<KB>;
    using S = EmuSmem<KB>;
    constexpr int LD = E::LD, LDC = E::LDC;
    constexpr size_t TS = (size_t)KB * KB;
    const int part = blockIdx.x, N = blk_off[part + 1] - blk_off[part];
    const size_t tb = (size_t)blk_off[part] * TS;
    const double *gTp = gT + (size_t)blk_off[part] * 3 * TS; // per block: D, A(J,J-1) column-major, A(J,J+1)
    const bool doW = part > 0;
    extern __shared__ __align__(16) char sm[];
    uint64_t *bars = (uint64_t *)sm;
    E em{(unsigned short *)(sm + S::head), (int *)(sm + 64)};
    double *sS = (double *)(sm + S::head + E::PLANES), *sL = sS + E::TILE, *sF = sL + E::TILE, *sE = sF + KB * LDC;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 3; i++) mbar_init(bars + i, 1);
        mbar_init_fence();
    }
    __syncthreads();
    EmuBar<KB> bD{bars, 0u, false}, bF{bars + 1, 0u, false}, bE{bars + 2, 0u, false};
    bD.issue(sS, LD, gTp);
    if (N > 1) bF.issue(sF, LDC, gTp + 3 * TS + TS);
    bool ok = true;
    for (int J = 0; J < N; J++) {
        double *gLj = gL + tb + (size_t)J * TS, *gGj = gG + tb + (size_t)J * TS;
        if (J > 0) {
            const double *gGp = gGj - TS;
            if (!bF.wait()) return emu_leave(err, bD, bF, bE); // (and every thread built G's planes)
            // L_J; A(J, J-1) is upper triangular (KB >= kl)
            em.product({sF, 1, LDC, gGp, 1, KB, nullptr, 0, 0, sL, LD, 1, gLj, 1, KB, 1, false});
            if (!bE.wait()) return emu_leave(err, bD, bF, bE); // E_{J-1}; L_J is complete
            if (J + 1 < N) bF.issue(sF, LDC, gTp + (size_t)(J + 1) * 3 * TS + TS);
            em.template build<KB>(sE, LD, 1, KB);
            if (!bD.wait()) return emu_leave(err, bD, bF, bE);
            // S_J = D_J - L_J E_{J-1}; A(J-1, J) is lower triangular
            em.product({sL, LD, 1, sE, LD, 1, sS, LD, 1, sS, LD, 1, nullptr, 0, 0, 3, true});
            __syncthreads();
            if (doW) {
                const double *zp = gZ + tb + (size_t)(J - 1) * TS;
                double *zj = gZ + tb + (size_t)J * TS;
                em.template build<KB>(zp, KB, 1, KB);
                __syncthreads();
                em.product({sL, LD, 1, zp, KB, 1, nullptr, 0, 0, zj, KB, 1, nullptr, 0, 0, 0, true});
                __syncthreads();
            }
        } else if (!bD.wait()) {
            return emu_leave(err, bD, bF, bE);
        }
        ok = em.inverse(sS, sL) && ok; // (L_J has been used)
        if (J + 1 < N) bE.issue(sE, LD, gTp + (size_t)J * 3 * TS + 2 * TS);
        for (int q = threadIdx.x; q < KB * KB; q += E::NT) { // column-major, 8 x 4 pieces per warp
            const int w = q >> 5, r = (w % (KB / 8)) * 8 + (q & 7), c = w / (KB / 8) * 4 + ((q >> 3) & 3);
            gGj[(size_t)c * KB + r] = sS[r * LD + c];
        }
        if (J + 1 < N) {
            em.template build<KB>(sS, LD, 1, KB);
            __syncthreads(); // every read of G_J is done
            bD.issue(sS, LD, gTp + (size_t)(J + 1) * 3 * TS);
        }
    }
    bD.drain();
    bE.drain();
    bF.drain();
    if (!ok) atomicOr(err, SPK_DEV_ERR_PIVOT);
}

// X_J = G_J (Z_J - E_J X_{J+1}); blockIdx.y = 0: V of partition blockIdx.x, 1: its W
template <int KB>
__global__ void __launch_bounds__(Emu<KB>::NT, 1)
    k_emu_bwd(const int *__restrict__ part_start, const int *__restrict__ blk_off, int p, const double *__restrict__ gL,
              const double *__restrict__ gG, const double *__restrict__ gE, const double *__restrict__ gBhat,
              double *gV, double *gW, unsigned *err)
{
    using E = Emu<KB>;
    using S = EmuSmem<KB>;
    constexpr int LD = E::LD, LDC = E::LDC;
    constexpr size_t TS = (size_t)KB * KB;
    const bool isV = blockIdx.y == 0;
    const int part = blockIdx.x;
    if (isV ? part >= p - 1 : part == 0) return; // the whole CTA: no spike to compute
    const int m = part_start[part + 1] - part_start[part], N = blk_off[part + 1] - blk_off[part];
    const size_t tb = (size_t)blk_off[part] * TS;
    extern __shared__ __align__(16) char sm[];
    uint64_t *bars = (uint64_t *)sm;
    E em{(unsigned short *)(sm + S::head), (int *)(sm + 64)};
    double *sT = (double *)(sm + S::head + E::PLANES), *sX = sT + E::TILE, *sG = sX + E::TILE, *sE = sG + KB * LDC;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; i++) mbar_init(bars + i, 1);
        mbar_init_fence();
    }
    __syncthreads();
    EmuBar<KB> bG{bars, 0u, false}, bE{bars + 1, 0u, false};
    bG.issue(sG, LDC, gG + tb + (size_t)(N - 1) * TS);
    double *gX = isV ? gV : gW;
    // V's right-hand side [0; B^] is nonzero only in the last KB real rows:
    // blocks J0 (rows o..KB-1) and J0+1 (rows 0..o-1, when o > 0), where the forward
    // sweep has z_{J0+1} = [B^'s last rows; 0] - L_{J0+1} z_{J0}.  (o < 0: a
    // partition shorter than a tile takes B^'s last m rows.)
    const int J0 = (m - KB) / KB, o = (m - KB) - J0 * KB;
    const double *bh = gBhat + (size_t)part * TS;
    if (isV) {
        for (int q = threadIdx.x; q < KB * KB; q += E::NT) {
            const int r = q / KB, c = q - r * KB;
            const double v = r >= o && r - o < KB ? bh[(r - o) * KB + c] : 0.0;
            sT[r * LD + c] = v;
            gV[tb + (size_t)J0 * TS + q] = v;
        }
        __syncthreads();
        if (o > 0) {
            const double *l = gL + tb + (size_t)(J0 + 1) * TS;
            double *z = gV + tb + (size_t)(J0 + 1) * TS;
            for (int q = threadIdx.x; q < KB * KB; q += E::NT) z[q] = q / KB < o ? bh[(KB - o) * KB + q] : 0.0;
            em.template build<KB>(sT, LD, 1, KB);
            __syncthreads();
            em.product({l, 1, KB, sT, LD, 1, z, KB, 1, z, KB, 1, nullptr, 0, 0, 0, true});
        }
        __syncthreads();
    }
    for (int J = N - 1; J >= 0; J--) {
        const double *zj = gX + tb + (size_t)J * TS; // Z_J, row-major, where the spike has one
        double *xj = gX + tb + (size_t)J * TS;
        const bool hasZ = !isV || J == J0 || (o > 0 && J == J0 + 1);
        if (J < N - 1) {
            if (!bE.wait()) return emu_leave(err, bG, bE); // (and X_{J+1}'s planes are built)
            // T = Z_J - E_J X_{J+1}; A(J, J+1) is lower triangular
            em.product({sE, 1, LDC, sX, LD, 1, hasZ ? zj : nullptr, KB, 1, sT, LD, 1, nullptr, 0, 0, 2, true});
            __syncthreads();
        } else {
            for (int q = threadIdx.x; q < KB * KB; q += E::NT) sT[q / KB * LD + q % KB] = hasZ ? zj[q] : 0.0;
            __syncthreads();
        }
        if (J > 0) bE.issue(sE, LDC, gE + tb + (size_t)(J - 1) * TS);
        em.template build<KB>(sT, LD, 1, KB);
        if (!bG.wait()) return emu_leave(err, bG, bE);
        em.product({sG, 1, LDC, sT, LD, 1, nullptr, 0, 0, sX, LD, 1, xj, 1, KB, 0, false});
        __syncthreads();
        if (J > 0) {
            bG.issue(sG, LDC, gG + tb + (size_t)(J - 1) * TS);
            em.template build<KB>(sX, LD, 1, KB);
        }
    }
    bG.drain();
    bE.drain();
}

// odd blocks of a cyclic-reduction level (k_cr_odd): S = I - Q P, M11 = S^{-1},
// M10 = -M11 Q, M01 = -P M11, M00 = I - P M10
template <int KB>
__global__ void __launch_bounds__(Emu<KB>::NT, 1)
    k_emu_cr_odd(const double *__restrict__ Pl, const double *__restrict__ Ql, int first, int stride, double *M,
                 unsigned *err)
{
    using E = Emu<KB>;
    using S = EmuSmem<KB>;
    constexpr int LD = E::LD;
    constexpr size_t TS = (size_t)KB * KB;
    const double *P = Pl + (size_t)(first + blockIdx.x * stride) * TS, *Q = Ql + (size_t)(first + blockIdx.x * stride) * TS;
    double *Mj = M + (size_t)blockIdx.x * 4 * TS;
    extern __shared__ __align__(16) char sm[];
    E em{(unsigned short *)(sm + S::head), (int *)(sm + 64)};
    double *sP = (double *)(sm + S::head + E::PLANES), *sQ = sP + E::TILE, *sH = sQ + E::TILE;
    double *sX = sH + E::TILE; // the inverse's scratch, then M10
    for (int q = threadIdx.x; q < KB * KB; q += E::NT) {
        const int r = q / KB, c = q % KB;
        sP[r * LD + c] = P[q];
        sQ[r * LD + c] = Q[q];
        sH[r * LD + c] = Mj[q] = r == c ? 1.0 : 0.0; // (Mj: where M00 = I - P M10 starts)
    }
    __syncthreads();
    em.template build<KB>(sP, LD, 1, KB);
    __syncthreads();
    em.product({sQ, LD, 1, sP, LD, 1, sH, LD, 1, sH, LD, 1, nullptr, 0, 0, 0, true}); // S
    __syncthreads();
    const bool ok = em.inverse(sH, sX);
    if (!ok) atomicOr(err, SPK_DEV_ERR_PIVOT);
    for (int q = threadIdx.x; q < KB * KB; q += E::NT) Mj[3 * TS + q] = sH[q / KB * LD + q % KB];
    em.template build<KB>(sH, LD, 1, KB);
    __syncthreads();
    em.product({sP, LD, 1, sH, LD, 1, nullptr, 0, 0, Mj + TS, KB, 1, nullptr, 0, 0, 0, true}); // M01
    __syncthreads();
    em.template build<KB>(sQ, LD, 1, KB);
    __syncthreads();
    em.product({sH, LD, 1, sQ, LD, 1, nullptr, 0, 0, Mj + 2 * TS, KB, 1, sX, LD, 1, 0, true}); // M10
    __syncthreads();
    em.template build<KB>(sX, LD, 1, KB);
    __syncthreads();
    em.product({sP, LD, 1, sX, LD, 1, Mj, KB, 1, Mj, KB, 1, nullptr, 0, 0, 0, true}); // M00
}

// even blocks (k_cr_even), blockIdx.y the result:
//   0: P' = P_i - X_i (M01 Y)_{i-1}   1: Q' = Q_i - Y_i (M10 X)_{i+1}
//   2: X' = -X_i (M00 X)_{i-1}        3: Y' = -Y_i (M11 Y)_{i+1}
template <int KB>
__global__ void __launch_bounds__(Emu<KB>::NT, 1)
    k_emu_cr_even(const double *__restrict__ Pl, const double *__restrict__ Ql, const double *__restrict__ Xl,
                  const double *__restrict__ Yl, const double *__restrict__ Ml, int cnt, double *Pn, double *Qn,
                  double *Xn, double *Yn)
{
    using E = Emu<KB>;
    using S = EmuSmem<KB>;
    constexpr int LD = E::LD;
    constexpr size_t TS = (size_t)KB * KB;
    const int i = 2 * blockIdx.x, w = blockIdx.y;
    const bool lft = w == 0 || w == 2;
    const int j = lft ? i - 1 : i + 1;
    const double *base = w == 0 ? Pl + (size_t)i * TS : w == 1 ? Ql + (size_t)i * TS : nullptr;
    double *out = (w == 0 ? Pn : w == 1 ? Qn : w == 2 ? Xn : Yn) + (size_t)blockIdx.x * TS;
    if (lft ? j < 0 : j >= cnt) {
        for (int q = threadIdx.x; q < KB * KB; q += E::NT) out[q] = base ? base[q] : 0.0;
        return;
    }
    const double *Mq = Ml + (size_t)(j / 2) * 4 * TS + (size_t)(w == 0 ? 1 : w == 1 ? 2 : w == 2 ? 0 : 3) * TS;
    const double *Rt = (w == 0 || w == 3 ? Yl : Xl) + (size_t)j * TS, *Lt = (lft ? Xl : Yl) + (size_t)i * TS;
    extern __shared__ __align__(16) char sm[];
    E em{(unsigned short *)(sm + S::head), (int *)(sm + 64)};
    double *sA = (double *)(sm + S::head + E::PLANES), *sT = sA + E::TILE;
    for (int q = threadIdx.x; q < KB * KB; q += E::NT) sA[q / KB * LD + q % KB] = Mq[q];
    em.template build<KB>(Rt, KB, 1, KB);
    __syncthreads();
    em.product({sA, LD, 1, Rt, KB, 1, nullptr, 0, 0, sT, LD, 1, nullptr, 0, 0, 0, false});
    __syncthreads();
    for (int q = threadIdx.x; q < KB * KB; q += E::NT) sA[q / KB * LD + q % KB] = Lt[q];
    em.template build<KB>(sT, LD, 1, KB);
    __syncthreads();
    em.product({sA, LD, 1, sT, LD, 1, base, KB, 1, out, KB, 1, nullptr, 0, 0, 0, true});
}

template <int KB> int attrs()
{
    using S = EmuSmem<KB>;
    static_assert(S::fwd <= 227 * 1024 && S::bwd <= 227 * 1024 && S::red <= 227 * 1024, "shared memory");
    static bool done = false;
    if (done) return SPK_OK;
    if (cudaFuncSetAttribute(k_emu_fwd<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::fwd) != cudaSuccess ||
        cudaFuncSetAttribute(k_emu_bwd<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bwd) != cudaSuccess ||
        cudaFuncSetAttribute(k_emu_cr_odd<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::red) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_emu_cr_even<KB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::red) !=
            cudaSuccess)
        return SPK_ECUDA;
    done = true;
    return SPK_OK;
}

} // namespace

// one-sided chains of 64-row FP64 tiles (forward: block LU and W's sweep; else the spikes)
extern "C" int spk_emu_factor(spk_plan *P, int forward, void *stream)
{
    constexpr int KB = 64;
    using S = EmuSmem<KB>;
    if (attrs<KB>() != SPK_OK) return SPK_ECUDA;
    cudaStream_t st = (cudaStream_t)stream;
    if (forward)
        k_emu_fwd<KB><<<P->p, Emu<KB>::NT, S::fwd, st>>>((const double *)P->d_T, P->d_blk_off, (double *)P->d_L,
                                                         (double *)P->d_G, (double *)P->d_W, P->d_err);
    else
        k_emu_bwd<KB><<<dim3(P->p, 2), Emu<KB>::NT, S::bwd, st>>>(
            P->d_part_start, P->d_blk_off, P->p, (const double *)P->d_L, (const double *)P->d_G,
            (const double *)P->d_E, (const double *)P->d_Bhat, (double *)P->d_V, (double *)P->d_W, P->d_err);
    SPK_CHECK_LAUNCH();
    return SPK_OK;
}
extern "C" int spk_emu_cr_odd(const double *P, const double *Q, int first, int stride, int count, double *M,
                              unsigned *err, void *stream)
{
    if (attrs<64>() != SPK_OK) return SPK_ECUDA;
    k_emu_cr_odd<64><<<count, Emu<64>::NT, EmuSmem<64>::red, (cudaStream_t)stream>>>(P, Q, first, stride, M, err);
    SPK_CHECK_LAUNCH();
    return SPK_OK;
}
extern "C" int spk_emu_cr_even(const double *P, const double *Q, const double *X, const double *Y, const double *M,
                               int cnt, double *Pn, double *Qn, double *Xn, double *Yn, void *stream)
{
    if (attrs<64>() != SPK_OK) return SPK_ECUDA;
    k_emu_cr_even<64><<<dim3((cnt + 1) / 2, 4), Emu<64>::NT, EmuSmem<64>::red, (cudaStream_t)stream>>>(P, Q, X, Y, M, cnt,
                                                                                                 Pn, Qn, Xn, Yn);
    SPK_CHECK_LAUNCH();
    return SPK_OK;
}
