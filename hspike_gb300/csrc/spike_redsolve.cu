// spike_redsolve.cu -- solution of the reduced system on sm_103a.
//
// spike_reduced.cu factors the reduced system R by block cyclic reduction; here
// u = R^{-1} g for the interface unknowns u_i = (b_i, t_{i+1}), wrapped in FP64
// refinement on R itself, u += CR^{-1}(g - R u) (the reference solves R with
// MKL PARDISO on the host, directSolver_Host_Solve,
// OpenMP/spike_algebra.c:263-420).
//
// A level of cyclic reduction is a handful of small matrix-vector products,
// so the time is the number of dependent steps, not the work.  Two forms:
//
//   KB <= 16  k_rs_*: a CTA takes a whole segment of the system through several
//             levels.  By the quadrant structure an even block's two halves are
//             updated from one side each -- g^0 by its left odd neighbour, g^1 by
//             its right one -- so a segment between two surviving blocks
//             (every 2^s-th) needs nothing from the next segment until only
//             those survivors are left: s levels cost a few barriers of one
//             CTA instead of 2 s launches.  Whole solves against one launch per
//             level and direction: n = 1,000, k = 2 (249 interfaces, one CTA)
//             655 -> 247 us; n = 300,007, k = 8 (2,431 interfaces, three tiers)
//             888 -> 586 us.
//   KB >= 32  k_crq_*: one launch per level and direction, a cluster of CTAs per
//             block: four rows of the products per warp, every operand of both
//             products requested before the first is used, the vector between
//             them exchanged through the cluster's shared memory.
#include "spike_slices.cuh"

#include <cooperative_groups.h>
#include <type_traits>

namespace cg = cooperative_groups;

namespace {

// ------------------------------------------------------------ KB <= 16: segments
template <class T> struct RsArgs {
    using H = typename HighOf<T>::type;
    const T *X, *Y, *M;
    const H *RP, *RQ, *RX, *RY; // level-0 blocks of R
    const H *g;                 // right-hand side, ld NR
    H *u;                       // solution, ld NR
    T *cg, *cu;                 // per-level work, ld stride
    unsigned *err;
    long long stride, NR;
    int nif, nrhs;
};

// A segment: levels [l0, l1), local block 0 is block b0 of level l0 and n0
// blocks are held (the right survivor included).  `end` = local index of the
// right survivor at level l0 when another segment owns its right half, else a
// number no block reaches; `first`: local block 0's left half is owned too
// (nothing to the left).  The segment's tiles of every level -- contiguous
// runs of M, X and Y -- come into shared memory by bulk copies at the start, so
// a level costs two barriers and no memory round trip.
template <class T, int KB, int NRC, int NT> struct RsSeg {
    using H = typename HighOf<T>::type;
    static constexpr int R = 2 * KB;
    static constexpr size_t TS = (size_t)KB * KB;

    const RsArgs<T> &A;
    const RsLevels &lv;
    int l0, l1, b0, n0, end, h0, nr;
    bool first, with_top;
    T *st; // tiles, level by level: M of the odd blocks, X, Y of every block (and the last level's M)
    T *sg; // g, level by level: [block][row][NRC]
    T *sv; // products of the level's odd blocks
    T *su; // u at level-l0 block positions

    // offsets within st (in tiles) and sg (in blocks) of level l, and its blocks
    __device__ __forceinline__ void level(int l, int &to, int &go, int &nl) const
    {
        to = go = 0;
        nl = n0;
        for (int q = l0; q < l; q++) {
            to += 4 * (nl >> 1) + 2 * nl;
            go += nl;
            nl = (nl + 1) >> 1;
        }
    }
    __device__ __forceinline__ void carve(char *raw)
    {
        int to, go, nl;
        level(l1, to, go, nl);
        st = (T *)smem_align(raw + 16);
        sg = st + (size_t)(to + (with_top ? 4 : 0)) * TS;
        sv = sg + (size_t)(go + nl) * R * NRC;
        su = sv + (size_t)(n0 / 2 + 1) * R * NRC;
    }
    // one thread: all bulk copies on `bar`
    __device__ __forceinline__ void issue(uint64_t *bar) const
    {
        int to, go, nl;
        level(l1, to, go, nl);
        mbar_arrive_expect_tx(bar, (unsigned)((size_t)(to + (with_top ? 4 : 0)) * TS * sizeof(T)));
        T *d = st;
        nl = n0;
        int b = b0;
        for (int l = l0; l < l1; l++) {
            const int nodd = nl >> 1;
            const unsigned mb = (unsigned)(nodd * 4 * TS * sizeof(T)), xb = (unsigned)(nl * TS * sizeof(T));
            if (nodd) bulk_g2s(d, A.M + (size_t)(lv.moff[l] + b / 2) * 4 * TS, mb, bar);
            d += nodd * 4 * TS;
            bulk_g2s(d, A.X + (size_t)(lv.off[l] + b) * TS, xb, bar);
            d += nl * TS;
            bulk_g2s(d, A.Y + (size_t)(lv.off[l] + b) * TS, xb, bar);
            d += nl * TS;
            nl = (nl + 1) >> 1;
            b >>= 1;
        }
        if (with_top) bulk_g2s(d, A.M + (size_t)lv.moff[lv.L] * 4 * TS, (unsigned)(4 * TS * sizeof(T)), bar);
    }
    // start the copies, then (after the predecessor's vectors exist) wait for
    // them; false in every thread when a copy never landed
    __device__ __forceinline__ void start(uint64_t *bar)
    {
        if (threadIdx.x == 0) {
            mbar_init(bar, 1);
            mbar_init_fence();
            issue(bar);
        }
        dep_launch();
        __syncthreads();
        dep_wait();
    }
    __device__ __forceinline__ bool ready(uint64_t *bar) const
    {
        const bool ok = mbar_wait(bar, 0);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) atomicOr(A.err, SPK_DEV_ERR_TIMEOUT);
            mbar_wait(bar, 0); // once more: the shared memory is another block's after this one
            return false;
        }
        return true;
    }
    // acc (+|-)= m[0..KB) v[0..KB)[h], m one row of a tile
    template <bool SUB> __device__ __forceinline__ T dot(T acc, const T *m, const T *v) const
    {
        T r[KB];
        vld<T, KB>(r, m);
#pragma unroll
        for (int k = 0; k < KB; k++) acc = SUB ? msub(acc, r[k], v[k * NRC]) : madd(acc, r[k], v[k * NRC]);
        return acc;
    }

    // forward reduction through levels l0 .. l1 - 1; the new g also go to global
    __device__ __forceinline__ void forward(bool store) const
    {
        T *g = sg;
        const T *tile = st;
        int nl = n0, b = b0, e = end;
        for (int l = l0; l < l1; l++) {
            const int nodd = nl >> 1, nn = (nl + 1) >> 1;
            const T *Ml = tile, *Xl = Ml + nodd * 4 * TS, *Yl = Xl + nl * TS;
            // v_j = M_j g_j of the odd blocks
            for (int t = threadIdx.x; t < nodd * R * NRC; t += NT) {
                const int h = t % NRC, q = (t / NRC) % R, jj = t / (NRC * R);
                const T *m = Ml + (size_t)jj * 4 * TS + (q / KB) * 2 * TS + (q % KB) * KB;
                const T *v = g + (size_t)(2 * jj + 1) * R * NRC + h;
                sv[t] = dot<false>(dot<false>(sc_zero<T>(), m, v), m + TS, v + KB * NRC);
            }
            __syncthreads();
            // g'^0_i = g^0_i - X_i v^0_{i-1},  g'^1_i = g^1_i - Y_i v^1_{i+1}
            T *gn = g + (size_t)nl * R * NRC;
            T *out = A.cg + (size_t)(lv.off[l + 1] + b / 2) * R;
            for (int t = threadIdx.x; t < nn * R * NRC; t += NT) {
                const int h = t % NRC, q = (t / NRC) % R, a = t / (NRC * R);
                const int half = q / KB, i = 2 * a, j = half ? i + 1 : i - 1;
                T v = g[(size_t)(i * R + q) * NRC + h];
                if (half ? j < nl : j >= 0)
                    v = dot<true>(v, (half ? Yl : Xl) + (size_t)i * TS + (q - half * KB) * KB,
                                  sv + (size_t)((j >> 1) * R + half * KB) * NRC + h);
                gn[t] = v; // (a half another segment owns: its value here is not used)
                if (store && h < nr && (half ? i < e : (i > 0 || first)))
                    out[(h0 + h) * A.stride + (size_t)a * R + q] = v;
            }
            __syncthreads();
            tile = Yl + nl * TS;
            g = gn;
            nl = nn;
            b >>= 1;
            e >>= 1;
        }
    }
    // back substitution from the survivors' u (in su) down to level l0
    __device__ __forceinline__ void backward() const
    {
        for (int l = l1 - 1; l >= l0; l--) {
            const int sh = l - l0;
            int to, go, nl;
            level(l, to, go, nl);
            const int nodd = nl >> 1;
            const T *g = sg + (size_t)go * R * NRC;
            const T *Ml = st + (size_t)to * TS, *Xl = Ml + nodd * 4 * TS, *Yl = Xl + nl * TS;
            // t_j = g_j - [X_j u^0_{j-1} ; Y_j u^1_{j+1}]
            for (int t = threadIdx.x; t < nodd * R * NRC; t += NT) {
                const int h = t % NRC, q = (t / NRC) % R, jj = t / (NRC * R), j = 2 * jj + 1;
                const int half = q / KB, nb = half ? j + 1 : j - 1;
                T v = g[(size_t)(j * R + q) * NRC + h];
                if (nb < nl)
                    v = dot<true>(v, (half ? Yl : Xl) + (size_t)j * TS + (q - half * KB) * KB,
                                  su + (size_t)((nb << sh) * R + half * KB) * NRC + h);
                sv[t] = v;
            }
            __syncthreads();
            // u_j = M_j t_j
            for (int t = threadIdx.x; t < nodd * R * NRC; t += NT) {
                const int h = t % NRC, q = (t / NRC) % R, jj = t / (NRC * R);
                const T *m = Ml + (size_t)jj * 4 * TS + (q / KB) * 2 * TS + (q % KB) * KB;
                const T *v = sv + (size_t)jj * R * NRC + h;
                su[(size_t)(((2 * jj + 1) << sh) * R + q) * NRC + h] =
                    dot<false>(dot<false>(sc_zero<T>(), m, v), m + TS, v + KB * NRC);
            }
            __syncthreads();
        }
    }
    // the single block of level L: u = M g
    __device__ __forceinline__ void top() const
    {
        int to, go, nl;
        level(l1, to, go, nl);
        const T *g = sg + (size_t)go * R * NRC, *Mt = st + (size_t)to * TS;
        for (int t = threadIdx.x; t < R * NRC; t += NT) {
            const int h = t % NRC, q = t / NRC;
            const T *m = Mt + (q / KB) * 2 * TS + (q % KB) * KB;
            su[q * NRC + h] = dot<false>(dot<false>(sc_zero<T>(), m, g + h), m + TS, g + KB * NRC + h);
        }
        __syncthreads();
    }
    // level-0 right-hand side: g, or the FP64 residual g - R u (narrowed after
    // the subtraction), into sg and, for the back substitution's kernel, to global
    __device__ __forceinline__ void load0(bool resid, bool store) const
    {
        for (int t = threadIdx.x; t < n0 * R * NRC; t += NT) {
            const int h = t % NRC, q = (t / NRC) % R, a = t / (NRC * R), i = b0 + a;
            const int half = q / KB, rr = q - half * KB;
            if (h >= nr || !(half ? a < end : (a > 0 || first))) {
                sg[t] = sc_zero<T>();
                continue;
            }
            H acc = A.g[(h0 + h) * A.NR + (long long)i * R + q];
            if (resid) {
                const H *uh = A.u + (h0 + h) * A.NR + (long long)i * R;
                acc = acc - uh[q];
                const H *p = (half ? A.RQ : A.RP) + (size_t)i * TS + rr * KB;
                const H *x = uh + (half ? 0 : KB);
#pragma unroll
                for (int c = 0; c < KB; c++) acc = msub(acc, p[c], x[c]);
                if (half ? i + 1 < A.nif : i > 0) { // t-equation: Y_i t_{i+2}; b-equation: X_i b_{i-1}
                    p = (half ? A.RY : A.RX) + (size_t)i * TS + rr * KB;
                    x = uh + (half ? R + KB : -R);
#pragma unroll
                    for (int c = 0; c < KB; c++) acc = msub(acc, p[c], x[c]);
                }
            }
            const T v = cvt_fast<T, H>(acc);
            sg[t] = v;
            if (store) A.cg[(h0 + h) * A.stride + (size_t)i * R + q] = v;
        }
    }
    // U = u or U += u at level 0, for the first n of the local blocks
    __device__ __forceinline__ void accumulate(int n, bool set) const
    {
        for (int t = threadIdx.x; t < n * R * NRC; t += NT) {
            const int h = t / (n * R), q = t - h * n * R; // rows fastest: coalesced
            if (h < nr) {
                H *o = A.u + (h0 + h) * A.NR + (long long)b0 * R + q;
                const H d = cvt_fast<H, T>(su[(size_t)q * NRC + h]);
                *o = set ? d : *o + d;
            }
        }
    }
    // n blocks of one level between shared memory ([block][row][NRC]) and global work vectors
    __device__ __forceinline__ void get(T *s, const T *g, int n) const
    {
        for (int t = threadIdx.x; t < n * R * NRC; t += NT) {
            const int h = t / (n * R), q = t - h * n * R;
            s[(size_t)q * NRC + h] = h < nr ? g[(h0 + h) * A.stride + q] : sc_zero<T>();
        }
    }
    __device__ __forceinline__ void put(T *g, const T *s, int n) const
    {
        for (int t = threadIdx.x; t < n * R * NRC; t += NT) {
            const int h = t / (n * R), q = t - h * n * R;
            if (h < nr) g[(h0 + h) * A.stride + q] = s[(size_t)q * NRC + h];
        }
    }
};

// shared bytes of a segment holding n blocks of its first level, `levels` levels
template <class T> static size_t rs_bytes(int n, int levels, int KB, int NRC, bool top)
{
    size_t tiles = top ? 4 : 0, blocks = n + n / 2 + 1; // (su, sv)
    int c = n;
    for (int l = 0; l <= levels; l++) {
        if (l < levels) tiles += 4 * (c / 2) + 2 * c;
        blocks += c;
        c = (c + 1) / 2;
    }
    return (tiles * KB * KB + blocks * 2 * KB * NRC) * sizeof(T) + 64;
}

template <class T, int KB, int NRC, int NT>
__device__ __forceinline__ RsSeg<T, KB, NRC, NT> rs_segment(const RsArgs<T> &A, const RsLevels &lv, int l0, int l1)
{
    const int k = blockIdx.x, s = l1 - l0, h0 = blockIdx.y * NRC;
    const int b0 = k << s, left = lv.cnt[l0] - b0, full = 1 << s;
    RsSeg<T, KB, NRC, NT> S{A, lv, l0, l1, b0, left > full ? full + 1 : left, left > full ? full : 1 << 30, h0,
                            min(NRC, A.nrhs - h0), k == 0, false, nullptr, nullptr, nullptr, nullptr};
    return S;
}

constexpr int RS_NT = 256, RS_TOP_NT = 512;

// forward through levels [l0, l1), one segment (and NRC columns) per CTA
template <class T, int KB, int NRC>
__global__ void __launch_bounds__(RS_NT)
    k_rs_fwd(const __grid_constant__ RsArgs<T> A, const __grid_constant__ RsLevels lv, int l0, int l1, int resid)
{
    extern __shared__ __align__(16) char smraw[];
    uint64_t *bar = (uint64_t *)smraw;
    auto S = rs_segment<T, KB, NRC, RS_NT>(A, lv, l0, l1);
    S.carve(smraw);
    S.start(bar);
    if (l0 == 0)
        S.load0(resid != 0, true);
    else
        S.get(S.sg, A.cg + (size_t)(lv.off[l0] + S.b0) * S.R, S.n0);
    if (!S.ready(bar)) return;
    S.forward(true);
}

// back through levels [l0, l1): the survivors' u of level l1 comes from cu
template <class T, int KB, int NRC>
__global__ void __launch_bounds__(RS_NT)
    k_rs_bwd(const __grid_constant__ RsArgs<T> A, const __grid_constant__ RsLevels lv, int l0, int l1, int set)
{
    extern __shared__ __align__(16) char smraw[];
    uint64_t *bar = (uint64_t *)smraw;
    auto S = rs_segment<T, KB, NRC, RS_NT>(A, lv, l0, l1);
    S.carve(smraw);
    S.start(bar);
    constexpr int R = 2 * KB;
    int nl = S.n0;
    size_t o = 0;
    for (int l = l0; l < l1; l++) { // g of every level
        S.get(S.sg + o * NRC, A.cg + (size_t)(lv.off[l] + (S.b0 >> (l - l0))) * R, nl);
        o += (size_t)nl * R;
        nl = (nl + 1) >> 1;
    }
    const int sh = l1 - l0;
    const T *cu = A.cu + (size_t)(lv.off[l1] + (S.b0 >> sh)) * R;
    for (int t = threadIdx.x; t < nl * R * NRC; t += RS_NT) { // the survivors
        const int h = t / (nl * R), q = t - h * nl * R, a = q / R, r = q % R;
        S.su[(size_t)((a << sh) * R + r) * NRC + h] = h < S.nr ? cu[(S.h0 + h) * A.stride + q] : sc_zero<T>();
    }
    if (!S.ready(bar)) return;
    S.backward();
    const int n = min(S.n0, 1 << sh); // the right survivor is the next segment's
    if (l0 == 0)
        S.accumulate(n, set != 0);
    else
        S.put(A.cu + (size_t)(lv.off[l0] + S.b0) * R, S.su, n);
}

// levels [l0, L] and back in one CTA per NRC columns; at l0 = 0 the whole
// solve, every refinement sweep included
template <class T, int KB, int NRC>
__global__ void __launch_bounds__(RS_TOP_NT)
    k_rs_top(const __grid_constant__ RsArgs<T> A, const __grid_constant__ RsLevels lv, int l0, int iters)
{
    extern __shared__ __align__(16) char smraw[];
    uint64_t *bar = (uint64_t *)smraw;
    const int h0 = blockIdx.y * NRC;
    RsSeg<T, KB, NRC, RS_TOP_NT> S{A, lv, l0, lv.L, 0, lv.cnt[l0], 1 << 30, h0, min(NRC, A.nrhs - h0), true, true,
                                   nullptr, nullptr, nullptr, nullptr};
    S.carve(smraw);
    S.start(bar);
    if (l0 > 0) iters = 1;
    for (int it = 0; it < iters; it++) {
        if (l0 == 0)
            S.load0(it > 0, false);
        else
            S.get(S.sg, A.cg + (size_t)lv.off[l0] * S.R, S.n0);
        if (it == 0) {
            if (!S.ready(bar)) return;
        } else {
            __syncthreads();
        }
        S.forward(false);
        S.top();
        S.backward();
        if (l0 == 0)
            S.accumulate(S.n0, it == 0);
        else
            S.put(A.cu + (size_t)lv.off[l0] * S.R, S.su, S.n0);
        __syncthreads();
    }
}

template <class T, int KB, int NRC> int run_red_solve_s(spk_plan *P, int nrhs, int iters, cudaStream_t st)
{
    using H = typename HighOf<T>::type;
    constexpr int R = 2 * KB;
    constexpr size_t SMEM = 220 * 1024;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_rs_fwd<T, KB, NRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_rs_bwd<T, KB, NRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_rs_top<T, KB, NRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) !=
                cudaSuccess)
            return SPK_ECUDA;
        attr = true;
    }
    const int L = P->cr_levels;
    RsLevels lv;
    if (!rs_levels(P, lv)) return SPK_EARG;
    RsArgs<T> A;
    A.X = (const T *)P->d_crX;
    A.Y = (const T *)P->d_crY;
    A.M = (const T *)P->d_crM;
    A.RP = (const H *)P->d_RP;
    A.RQ = (const H *)P->d_RQ;
    A.RX = (const H *)P->d_RX;
    A.RY = (const H *)P->d_RY;
    A.g = (const H *)P->d_g;
    A.u = (H *)P->d_u;
    A.cg = (T *)P->d_crg;
    A.cu = A.cg + P->crg_stride * P->nrhs_max;
    A.err = P->d_err;
    A.stride = P->crg_stride;
    A.NR = (long long)P->n_iface * R;
    A.nif = P->n_iface;
    A.nrhs = nrhs;
    const int hy = (nrhs + NRC - 1) / NRC;
    auto bytes = [&](int n, int levels, bool top) { return rs_bytes<T>(n, levels, KB, NRC, top); };
    int tier[RS_MAXL + 1], nt;
    const int lt = rs_schedule(lv, SMEM, bytes, tier, nt);
    const bool chain = chained(P);
    bool dep = false; // the first kernel of the solve starts after everything before it
    for (int it = 0; it < (lt == 0 ? 1 : iters); it++) {
        int rc = SPK_OK;
        for (int q = 0; q < nt && rc == SPK_OK; q++) {
            const int l0 = tier[q], l1 = tier[q + 1], s = l1 - l0;
            const int segs = (lv.cnt[l0] + (1 << s) - 1) >> s;
            rc = launch_dep(k_rs_fwd<T, KB, NRC>, dim3(segs, hy), RS_NT, bytes((1 << s) + 1, s, false), 1, dep, st, A,
                            lv, l0, l1, (int)(it > 0));
            dep = chain;
        }
        if (rc == SPK_OK)
            rc = launch_dep(k_rs_top<T, KB, NRC>, dim3(1, hy), RS_TOP_NT, bytes(lv.cnt[lt], L - lt, true), 1, dep, st,
                            A, lv, lt, iters);
        dep = chain;
        for (int q = nt - 1; q >= 0 && rc == SPK_OK; q--) {
            const int l0 = tier[q], l1 = tier[q + 1], s = l1 - l0;
            const int segs = (lv.cnt[l0] + (1 << s) - 1) >> s;
            rc = launch_dep(k_rs_bwd<T, KB, NRC>, dim3(segs, hy), RS_NT, bytes((1 << s) + 1, s, false), 1, dep, st, A,
                            lv, l0, l1, (int)(it == 0));
        }
        if (rc != SPK_OK) return rc;
        P->launches += 2 * nt + 1;
    }
    return SPK_OK;
}

// ------------------------------------------------------------ KB >= 32: one cluster per block
// A CTA has eight warps of four rows each, CS = KB / 16 CTAs make up the 2 KB
// rows of a block.  A block's products are bound by latency at every level but
// the first: one CTA walking a 128-row block's 384 KB of tiles took 32 us a
// level (eight columns), a cluster of eight takes about a memory round trip.
constexpr int QNT = 256, QWARPS = QNT / 32, QRPW = 4, QROWS = QWARPS * QRPW;

template <class T, int KB, int NRC> struct QSolve {
    static constexpr size_t TS = (size_t)KB * KB;
    static constexpr int R = 2 * KB;
    static constexpr int CS = R / QROWS; // CTAs per block
    static constexpr int VW = KB / 32;   // elements of a tile row per lane
    static constexpr int V = QRPW * NRC; // values per warp sum
    static constexpr int SH = V == 4 ? 3 : V == 16 ? 1 : 0;
    static_assert(KB % 32 == 0 && KB % QROWS == 0 && CS <= 8 && (V == 4 || V == 16 || V == 32), "QSolve shape");
};

// element (row q, column h) of level block a: input g (FP64 at level 0)
template <class T, class H>
__device__ __forceinline__ T q_in(const void *g, bool l0, long long ld, long long a, int q, int h, int KB)
{
    const long long o = h * ld + a * 2 * KB + q;
    return l0 ? cvt_fast<T, H>(((const H *)g)[o]) : ((const T *)g)[o];
}

// this warp's four rows of (NT1 tiles side by side) times x[h][ldx], lanes
// along k; the lane holding a (row, column) result calls emit(row, column, sum)
template <class T, int KB, int NRC, int NTL, class Emit>
__device__ __forceinline__ void q_dots(const T (&m)[QRPW][NTL][KB / 32], const T *x, int ldx, int nr, Emit emit)
{
    using Q = QSolve<T, KB, NRC>;
    const int lane = threadIdx.x & 31;
    T v[Q::V];
#pragma unroll
    for (int h = 0; h < NRC; h++) {
        T xv[NTL][Q::VW];
#pragma unroll
        for (int e = 0; e < NTL; e++) vld<T, Q::VW>(xv[e], x + h * ldx + e * KB + lane * Q::VW);
#pragma unroll
        for (int g = 0; g < QRPW; g++) {
            T acc = sc_zero<T>();
#pragma unroll
            for (int e = 0; e < NTL; e++)
#pragma unroll
                for (int w = 0; w < Q::VW; w++) acc = madd(acc, m[g][e][w], xv[e][w]);
            v[g * NRC + h] = acc;
        }
    }
    const T sum = warp_tsum(v, lane);
    if ((lane & ((1 << Q::SH) - 1)) == 0) {
        const int idx = lane >> Q::SH, g = idx / NRC, h = idx - g * NRC;
        if (h < nr) emit(g, h, sum);
    }
}

// Forward reduction, one cluster per even block i of level l:
//   g'_i = g_i - [X_i (M00 x0 + M01 x1)_{i-1} ; Y_i (M10 x0 + M11 x1)_{i+1}]
// g at level 0 is FP64 (gld = n_iface * 2KB); level l+1 goes to gn.
template <class T, int KB, int NRC>
__global__ void __launch_bounds__(QNT)
    k_crq_fwd(const T *__restrict__ Xl, const T *__restrict__ Yl, const T *__restrict__ Ml, int cnt, const void *gin,
              int l0, long long gld, long long off_l, T *gn, long long stride, long long off_n, int nrhs)
{
    using H = typename HighOf<T>::type;
    using Q = QSolve<T, KB, NRC>;
    constexpr size_t TS = Q::TS;
    __shared__ __align__(16) T sx[NRC * 2 * KB];  // the neighbour's block, [h][2KB]; then w, [h][KB]
    __shared__ __align__(16) T sw[NRC * QROWS];   // this CTA's rows of w, [h][row]
    const int rank = blockIdx.x % Q::CS, a = blockIdx.x / Q::CS, i = 2 * a;
    const int h0 = blockIdx.y * NRC, nr = min(NRC, nrhs - h0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lr0 = warp * QRPW, r0 = rank * QROWS + lr0, half = rank * QROWS / KB, q0 = r0 - half * KB;
    const bool has = half ? i + 1 < cnt : i - 1 >= 0;
    T m[QRPW][2][Q::VW], c[QRPW][1][Q::VW];
    if (has) { // every tile row of both products in flight at once
        const T *Mh = Ml + (size_t)(half ? i / 2 : (i - 2) / 2) * 4 * TS + half * 2 * TS;
        const T *Ch = (half ? Yl : Xl) + (size_t)i * TS;
#pragma unroll
        for (int g = 0; g < QRPW; g++) {
            vld<T, Q::VW>(m[g][0], Mh + (size_t)(q0 + g) * KB + lane * Q::VW);
            vld<T, Q::VW>(m[g][1], Mh + TS + (size_t)(q0 + g) * KB + lane * Q::VW);
            vld<T, Q::VW>(c[g][0], Ch + (size_t)(q0 + g) * KB + lane * Q::VW);
        }
    }
    dep_launch();
    dep_wait();
    if (has) {
        for (int q = threadIdx.x; q < NRC * 2 * KB; q += QNT) {
            const int h = q / (2 * KB), k = q - h * 2 * KB;
            sx[q] = h < nr ? q_in<T, H>(gin, l0, gld, off_l + i + (half ? 1 : -1), k, h0 + h, KB) : sc_zero<T>();
        }
    }
    __syncthreads();
    if (has) q_dots<T, KB, NRC, 2>(m, sx, 2 * KB, nr, [&](int g, int h, T v) { sw[h * QROWS + lr0 + g] = v; });
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    if (has) { // the half's w from the CTAs that hold its rows
        for (int q = threadIdx.x; q < NRC * KB; q += QNT) {
            const int h = q / KB, k = q - h * KB, row = half * KB + k;
            const T *src = cl.map_shared_rank(sw, row / QROWS);
            sx[h * KB + k] = h < nr ? src[h * QROWS + row % QROWS] : sc_zero<T>();
        }
    }
    cl.sync(); // sx is complete, and no CTA leaves while its rows are read
    T *gout = gn + (off_n + a) * 2 * KB;
    if (has) {
        q_dots<T, KB, NRC, 1>(c, sx, KB, nr, [&](int g, int h, T v) {
            gout[(h0 + h) * stride + r0 + g] = q_in<T, H>(gin, l0, gld, off_l + i, r0 + g, h0 + h, KB) - v;
        });
    } else {
        for (int q = threadIdx.x; q < QROWS * nr; q += QNT) {
            const int h = q / QROWS, r = rank * QROWS + q - h * QROWS;
            gout[(h0 + h) * stride + r] = q_in<T, H>(gin, l0, gld, off_l + i, r, h0 + h, KB);
        }
    }
}

// Back substitution at level l, one cluster per odd block (top: the single
// block of the last level): u_j = M_j (g_j - [X_j u0_{j-1} ; Y_j u1_{j+1}]).
// u is kept at the blocks' level-0 positions (block j of level l at j << l),
// so an even block's value is in place already; every block also goes into
// the FP64 solution U (ld uld) as it is found: U = d on the first refinement
// pass, U += d after.
template <class T, int KB, int NRC>
__global__ void __launch_bounds__(QNT)
    k_crq_bwd(const T *__restrict__ Xl, const T *__restrict__ Yl, const T *__restrict__ Ml, int cnt, const void *gin,
              int l0, long long gld, long long off_l, T *u, long long stride, int lsh,
              typename HighOf<T>::type *U, long long uld, int first, int nrhs, int top)
{
    using H = typename HighOf<T>::type;
    using Q = QSolve<T, KB, NRC>;
    constexpr size_t TS = Q::TS;
    __shared__ __align__(16) T sx[NRC * 2 * KB]; // neighbour values of this CTA's half, [h][KB]; then all of t, [h][2KB]
    __shared__ __align__(16) T st[NRC * QROWS];  // this CTA's rows of t
    const int rank = blockIdx.x % Q::CS, jj = blockIdx.x / Q::CS, j = top ? 0 : 2 * jj + 1;
    const int h0 = blockIdx.y * NRC, nr = min(NRC, nrhs - h0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lr0 = warp * QRPW, r0 = rank * QROWS + lr0, half = rank * QROWS / KB, q0 = r0 - half * KB;
    const bool has = !top && (half ? j + 1 < cnt : true);
    T m[QRPW][2][Q::VW], c[QRPW][1][Q::VW];
    const T *Mh = Ml + (size_t)jj * 4 * TS + half * 2 * TS;
#pragma unroll
    for (int g = 0; g < QRPW; g++) {
        vld<T, Q::VW>(m[g][0], Mh + (size_t)(q0 + g) * KB + lane * Q::VW);
        vld<T, Q::VW>(m[g][1], Mh + TS + (size_t)(q0 + g) * KB + lane * Q::VW);
    }
    if (has) {
        const T *Ch = (half ? Yl : Xl) + (size_t)j * TS;
#pragma unroll
        for (int g = 0; g < QRPW; g++) vld<T, Q::VW>(c[g][0], Ch + (size_t)(q0 + g) * KB + lane * Q::VW);
    }
    dep_launch();
    dep_wait();
    if (has) {
        const long long nb = (long long)(half ? j + 1 : j - 1) << lsh;
        for (int q = threadIdx.x; q < NRC * KB; q += QNT) {
            const int h = q / KB, k = q - h * KB;
            sx[q] = h < nr ? u[(h0 + h) * stride + nb * 2 * KB + half * KB + k] : sc_zero<T>();
        }
    }
    for (int q = threadIdx.x; q < NRC * QROWS; q += QNT) {
        const int h = q / QROWS, r = q - h * QROWS;
        st[q] = h < nr ? q_in<T, H>(gin, l0, gld, off_l + j, rank * QROWS + r, h0 + h, KB) : sc_zero<T>();
    }
    __syncthreads();
    if (has)
        q_dots<T, KB, NRC, 1>(c, sx, KB, nr, [&](int g, int h, T v) {
            st[h * QROWS + lr0 + g] = st[h * QROWS + lr0 + g] - v;
        });
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    for (int q = threadIdx.x; q < NRC * 2 * KB; q += QNT) {
        const int h = q / (2 * KB), row = q - h * 2 * KB;
        const T *src = cl.map_shared_rank(st, row / QROWS);
        sx[q] = src[h * QROWS + row % QROWS];
    }
    cl.sync(); // sx is complete, and no CTA leaves while its rows are read
    const long long pos = ((long long)j << lsh) * 2 * KB;
    q_dots<T, KB, NRC, 2>(m, sx, 2 * KB, nr, [&](int g, int h, T v) {
        u[(h0 + h) * stride + pos + r0 + g] = v;
        H *o = U + (h0 + h) * uld + pos + r0 + g;
        const H d = cvt_fast<H, T>(v);
        *o = first ? d : *o + d;
    });
}

// a factor-precision value in FP64, exactly, with integer instructions (subnormals too)
__device__ __forceinline__ double widen(double v) { return v; }
__device__ __forceinline__ cdouble widen(cdouble v) { return v; }
__device__ __forceinline__ double widen(float v)
{
    const unsigned u = __float_as_uint(v);
    if ((u & 0x7f800000u) == 0x7f800000u) return (double)v;
    const bool sub = (u & 0x7f800000u) == 0u;
    const unsigned w = sub ? __float_as_uint(v * 0x1p64f) : u; // a normal number, or zero
    const unsigned e = (w >> 23) & 0xffu;
    const unsigned hi = (u & 0x80000000u) |
                        (e == 0u ? 0u : (((e + (1023u - 127u) - (sub ? 64u : 0u)) << 20) | ((w & 0x7fffffu) >> 3)));
    return __hiloint2double((int)hi, (int)(w << 29));
}
__device__ __forceinline__ cdouble widen(cfloat v) { return {widen(v.re), widen(v.im)}; }

// res = g - R u in FP64 with the level-0 quadrant blocks (spikes' tips: values
// of the factor precision), 32 rows per CTA, a
// warp per four rows with its lanes along k: every tile is read once,
// coalesced (one thread per row walking its KB columns took 281 us at 155
// interfaces of 64 rows, 16 columns)
template <class T, int KB, int NRC>
__global__ void __launch_bounds__(QNT)
    k_red_resid(const T *__restrict__ RP, const T *__restrict__ RQ, const T *__restrict__ RX, const T *__restrict__ RY,
                const typename HighOf<T>::type *__restrict__ g, const typename HighOf<T>::type *__restrict__ u,
                typename HighOf<T>::type *res, int nif, int nrhs)
{
    using H = typename HighOf<T>::type;
    using Q = QSolve<H, KB, NRC>;
    constexpr size_t TS = Q::TS;
    __shared__ __align__(16) H sx[NRC * 2 * KB]; // [h]: the two KB-vectors this half's rows meet
    const int rank = blockIdx.x % Q::CS, i = blockIdx.x / Q::CS;
    const int h0 = blockIdx.y * NRC, nr = min(NRC, nrhs - h0);
    const long long NR = (long long)nif * 2 * KB, b = (long long)i * 2 * KB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = rank * QROWS + warp * QRPW, half = rank * QROWS / KB, q0 = r0 - half * KB;
    const bool far = half ? i + 1 < nif : i > 0; // the neighbouring interface exists
    H m[QRPW][2][Q::VW];
    const T *A0 = (half ? RQ : RP) + (size_t)i * TS, *A1 = (half ? RY : RX) + (size_t)i * TS;
    T mt[QRPW][2][Q::VW];
#pragma unroll
    for (int gq = 0; gq < QRPW; gq++) {
        vld<T, Q::VW>(mt[gq][0], A0 + (size_t)(q0 + gq) * KB + lane * Q::VW);
        vld<T, Q::VW>(mt[gq][1], A1 + (size_t)(q0 + gq) * KB + lane * Q::VW);
    }
#pragma unroll
    for (int gq = 0; gq < QRPW; gq++)
#pragma unroll
        for (int w = 0; w < Q::VW; w++) {
            m[gq][0][w] = widen(mt[gq][0][w]);
            m[gq][1][w] = far ? widen(mt[gq][1][w]) : sc_zero<H>();
        }
    dep_launch();
    dep_wait();
    for (int q = threadIdx.x; q < NRC * 2 * KB; q += QNT) {
        const int h = q / (2 * KB), k = q - h * 2 * KB, kk = k % KB;
        // b-equation: P_i t_{i+1} + X_i b_{i-1}; t-equation: Q_i b_i + Y_i t_{i+2}
        const long long o = k < KB ? b + (half ? 0 : KB) + kk : half ? b + 2 * KB + KB + kk : b - 2 * KB + kk;
        sx[q] = h < nr && (k < KB || far) ? u[(h0 + h) * NR + o] : sc_zero<H>();
    }
    __syncthreads();
    q_dots<H, KB, NRC, 2>(m, sx, 2 * KB, nr, [&](int gq, int h, H v) {
        const long long o = (h0 + h) * NR + b + r0 + gq;
        res[o] = g[o] - u[o] - v;
    });
}

// The same on the tensor cores by exact digit products (spike_slices.cuh), eight
// columns per CTA: 8 KB^2 FP64 multiply-adds per interface and column are what
// bounds k_red_resid (102 us at 155 interfaces of 64 rows and 16 columns, 143 at
// 127 of 128 rows and 8), here 32 and 53.  A CTA forms 64 rows of one equation: its
// warps take 16 rows and two KB / 32-th parts of the 2 KB columns each, split
// the tiles' values from registers and the vectors' through shared planes, and
// add their integer sums there.
template <int KB> struct RedSl {
    static constexpr int ROWS = KB < 64 ? KB : 64, KS = KB / 32, WARPS = ROWS / 16 * KS, NT = 32 * WARPS;
    static constexpr int NC = 8, K = 2 * KB, STEPS = K / 16 / KS, LDX = K + 8; // LDX = 8 mod 64: conflict-free fragments
    static constexpr int UPW = NC * K / 64 / WARPS;                            // units of 64 values of u per warp
    static constexpr size_t PL = (size_t)(SL_D + 1) * NC * LDX * 2, PART = (size_t)KS * ROWS * NC * 20;
    static constexpr size_t SM = ((PL > PART ? PL : PART) + 15) / 16 * 16;
    static constexpr int CPI = K / ROWS; // CTAs per interface
};
template <int KB>
__global__ void __launch_bounds__(RedSl<KB>::NT)
    k_red_resid_sl(const float *__restrict__ RP, const float *__restrict__ RQ, const float *__restrict__ RX,
                   const float *__restrict__ RY, const double *__restrict__ g, const double *__restrict__ u, double *res,
                   int nif, int nrhs)
{
    using Q = RedSl<KB>;
    constexpr size_t TS = (size_t)KB * KB;
    __shared__ __align__(16) char pl[Q::SM];
    __shared__ int er[Q::ROWS], ec[Q::NC];
    unsigned short *px = (unsigned short *)pl;          // [digit][column][LDX]; plane SL_D: magnitudes
    long long *xh = (long long *)pl, *xl = xh + Q::KS * Q::ROWS * Q::NC; // partial sums, [ks][column][row]
    float *xg = (float *)(xl + Q::KS * Q::ROWS * Q::NC);
    const int i = blockIdx.x / Q::CPI, part = blockIdx.x % Q::CPI, r0 = part * Q::ROWS, half = r0 / KB, q0 = r0 - half * KB;
    const int h0 = blockIdx.y * Q::NC, nr = min(Q::NC, nrhs - h0);
    const long long NR = (long long)nif * 2 * KB, b = (long long)i * 2 * KB;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gr = lane >> 2, t = lane & 3;
    const int wr = warp % (Q::ROWS / 16) * 16, k0 = warp / (Q::ROWS / 16) * Q::STEPS * 16; // this warp's rows and columns
    const bool far = half ? i + 1 < nif : i > 0; // the neighbouring interface exists
    const float *A0 = (half ? RQ : RP) + (size_t)i * TS, *A1 = (half ? RY : RX) + (size_t)i * TS;
    // b-equation: P_i t_{i+1} + X_i b_{i-1}; t-equation: Q_i b_i + Y_i t_{i+2}
    auto where = [&](int k) {
        const int kk = k % KB;
        return k < KB ? b + (half ? 0 : KB) + kk : half ? b + 2 * KB + KB + kk : b - 2 * KB + kk;
    };
    float2 av[Q::STEPS][2][2]; // [step][row g, g + 8][columns 2 t, 2 t + 8]
#pragma unroll
    for (int s = 0; s < Q::STEPS; s++)
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int k = k0 + s * 16 + 2 * t + 8 * c;
                const float *A = (k < KB ? A0 : A1) + (size_t)(q0 + wr + gr + 8 * p) * KB + k % KB;
                av[s][p][c] = k < KB || far ? *reinterpret_cast<const float2 *>(A) : make_float2(0.f, 0.f);
            }
    if (tid < Q::ROWS) er[tid] = 0;
    if (tid < Q::NC) ec[tid] = 0;
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 2; p++) {
        unsigned m = 0;
#pragma unroll
        for (int s = 0; s < Q::STEPS; s++)
#pragma unroll
            for (int c = 0; c < 2; c++)
                m = max(m, max(__float_as_uint(av[s][p][c].x) & 0x7fffffffu, __float_as_uint(av[s][p][c].y) & 0x7fffffffu));
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
        // the FP64 exponent; subnormals at most the smallest normal's, inf and NaN no scale
        if (t == 0 && m) atomicMax(&er[wr + gr + 8 * p], m >= 0x7f800000u ? 0x7ff : (int)max(m >> 23, 1u) + 1023 - 127);
    }
    dep_launch();
    dep_wait();
    double v[Q::UPW][2]; // unit x = warp + w WARPS: column x / (K / 64), rows 64 (x % (K / 64)) + 2 lane
#pragma unroll
    for (int w = 0; w < Q::UPW; w++) {
        const int x = warp + w * Q::WARPS, h = x / (Q::K / 64), k = x % (Q::K / 64) * 64 + 2 * lane;
        const bool live = h < nr && (k < KB || far);
        v[w][0] = live ? u[(h0 + h) * NR + where(k)] : 0.0;
        v[w][1] = live ? u[(h0 + h) * NR + where(k + 1)] : 0.0;
        const unsigned a0 = (unsigned)__double2hiint(v[w][0]) & 0x7fffffffu, l0 = (unsigned)__double2loint(v[w][0]);
        const unsigned a1 = (unsigned)__double2hiint(v[w][1]) & 0x7fffffffu, l1 = (unsigned)__double2loint(v[w][1]);
        const unsigned e = __reduce_max_sync(0xffffffffu, max(max(a0, a1) >> 20, (a0 | l0 | a1 | l1) != 0u ? 1u : 0u));
        if (lane == 0 && e) atomicMax(&ec[h], (int)e);
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < Q::UPW; w++) {
        const int x = warp + w * Q::WARPS, h = x / (Q::K / 64), k = x % (Q::K / 64) * 64 + 2 * lane;
        const int E = ec[h];
        const bool live = E >= 64 && E < 0x7ff;
        SlPair(live ? v[w][0] : 0.0, live ? v[w][1] : 0.0, live ? E : 64)
            .store((unsigned *)(px + h * Q::LDX + k), Q::NC * Q::LDX / 2);
    }
    __syncthreads();
    SlAcc acc;
    acc.zero();
    int E[2];
    bool on[2];
#pragma unroll
    for (int p = 0; p < 2; p++) {
        E[p] = er[wr + gr + 8 * p];
        on[p] = E[p] >= 64 && E[p] < 0x7ff;
        if (!on[p]) E[p] = 64;
    }
#pragma unroll
    for (int s = 0; s < Q::STEPS; s++) {
        double w[2][4];
#pragma unroll
        for (int p = 0; p < 2; p++)
#pragma unroll
            for (int c = 0; c < 2; c++) {
                w[p][2 * c] = on[p] ? widen(av[s][p][c].x) : 0.0;
                w[p][2 * c + 1] = on[p] ? widen(av[s][p][c].y) : 0.0;
            }
        SlFragA F;
        F.split(w, E[0], E[1]);
        const unsigned *xb = (const unsigned *)(px + gr * Q::LDX + k0 + s * 16 + 2 * t);
        acc.step(F, [&](int d, int q) { return xb[d * (Q::NC * Q::LDX / 2) + 4 * q]; });
    }
    __syncthreads(); // the planes have been read
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int o = (warp / (Q::ROWS / 16) * Q::NC + 2 * t + (e & 1)) * Q::ROWS + wr + gr + 8 * (e >> 1);
        long long hi, lo;
        acc.total(e, hi, lo);
        xh[o] = hi;
        xl[o] = lo;
        xg[o] = acc.g[e];
    }
    __syncthreads();
    for (int o = tid; o < Q::ROWS * Q::NC; o += Q::NT) { // (whole warps: one column each)
        const int h = o / Q::ROWS, rw = o % Q::ROWS;
        if (h >= nr) break;
        long long hi = 0, lo = 0;
        float mg = 0.f;
#pragma unroll
        for (int s = 0; s < Q::KS; s++) {
            hi += xh[s * Q::ROWS * Q::NC + o];
            lo += xl[s * Q::ROWS * Q::NC + o];
            mg += xg[s * Q::ROWS * Q::NC + o];
        }
        const int Er = er[rw], Ec = ec[h], sc = 56 + Er + Ec - 2 * (1023 + 61);
        const bool zero = (Er == 0 && Ec < 0x7ff) || (Ec == 0 && Er < 0x7ff);
        const bool fine = Er >= 64 && Er < 0x7ff && Ec >= 64 && Ec < 0x7ff && mg >= SL_GUARD && sc > -900 && sc < 850;
        double ax = fine ? sl_round(hi, lo, sc) : 0.0;
        // the few results outside the scales' reach, one by one in FP64
        for (unsigned todo = __ballot_sync(0xffffffffu, !fine && !zero); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1, rr = __shfl_sync(0xffffffffu, rw, src);
            double sum = 0.0;
            for (int k = lane; k < (far ? 2 * KB : KB); k += 32)
                sum = fma(widen((k < KB ? A0 : A1)[(size_t)(q0 + rr) * KB + k % KB]), u[(h0 + h) * NR + where(k)], sum);
            for (int q = 16; q > 0; q >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, q);
            if (lane == src) ax = sum;
        }
        const long long x = (h0 + h) * NR + b + r0 + rw;
        res[x] = g[x] - u[x] - ax;
    }
}

template <class T, int KB, int NRC> int run_red_solve_q(spk_plan *P, int nrhs, int iters, cudaStream_t st)
{
    using H = typename HighOf<T>::type;
    using Q = QSolve<T, KB, NRC>;
    constexpr size_t TS = Q::TS;
    const long long NR = (long long)P->n_iface * 2 * KB;
    const long long stride = P->crg_stride;
    T *cgv = (T *)P->d_crg;
    T *cu = cgv + stride * P->nrhs_max;
    const T *cX = (const T *)P->d_crX, *cY = (const T *)P->d_crY, *cM = (const T *)P->d_crM;
    const int L = P->cr_levels;
    const unsigned hy = (nrhs + NRC - 1) / NRC;
    const bool chain = chained(P); // (every kernel but the first)
    for (int it = 0; it < iters; it++) {
        const H *res = it == 0 ? (const H *)P->d_g : (const H *)P->d_rr;
        auto in = [&](int l) { return l == 0 ? (const void *)res : (const void *)cgv; };
        auto ld = [&](int l) { return l == 0 ? NR : stride; };
        for (int l = 0; l < L; l++) {
            const int cnt = P->cr_count[l];
            if (launch_dep(k_crq_fwd<T, KB, NRC>, dim3((cnt + 1) / 2 * Q::CS, hy), QNT, 0, Q::CS, chain && it + l > 0, st,
                               cX + (size_t)P->cr_off[l] * TS, cY + (size_t)P->cr_off[l] * TS,
                               cM + (size_t)P->cr_moff[l] * 4 * TS, cnt, in(l), (int)(l == 0), ld(l),
                               (long long)P->cr_off[l], cgv, stride, (long long)P->cr_off[l + 1], nrhs) != SPK_OK)
                return SPK_ECUDA;
        }
        for (int l = L; l >= 0; l--) { // level L: the top block
            const int cnt = P->cr_count[l], nodd = l == L ? 1 : cnt / 2;
            if (launch_dep(k_crq_bwd<T, KB, NRC>, dim3(nodd * Q::CS, hy), QNT, 0, Q::CS, chain && it + L > 0, st,
                               cX + (size_t)P->cr_off[l] * TS, cY + (size_t)P->cr_off[l] * TS,
                               cM + (size_t)P->cr_moff[l] * 4 * TS, cnt, in(l), (int)(l == 0), ld(l),
                               (long long)P->cr_off[l], cu, stride, l, (H *)P->d_u, NR, (int)(it == 0), nrhs,
                               (int)(l == L)) != SPK_OK)
                return SPK_ECUDA;
        }
        P->launches += 2 * L + 1;
        if (it + 1 < iters) {
            constexpr int RC = NRC > 4 ? 4 : NRC;
            int rc = SPK_OK;
            // (one column: the FP64 pipe is done sooner, 18 against 32 us at 255 interfaces of 64
            // rows; two columns 30 against 25 us at 127 of 128 rows)
            if constexpr (std::is_same<T, float>::value && NRC > 1) {
                using S = RedSl<KB>;
                rc = launch_dep(k_red_resid_sl<KB>, dim3(P->n_iface * S::CPI, (nrhs + S::NC - 1) / S::NC), S::NT, 0, 1,
                                chain, st, (const T *)P->d_crP, (const T *)P->d_crQ, cX, cY, (const H *)P->d_g,
                                (const H *)P->d_u, (H *)P->d_rr, P->n_iface, nrhs);
            } else if (launch_dep(k_red_resid<T, KB, RC>, dim3(P->n_iface * Q::CS, (nrhs + RC - 1) / RC), QNT, 0, 1, chain, st,
                           (const T *)P->d_crP, (const T *)P->d_crQ, cX, cY, (const H *)P->d_g, (const H *)P->d_u, (H *)P->d_rr, P->n_iface, nrhs) != SPK_OK)
                rc = SPK_ECUDA;
            if (rc != SPK_OK) return rc;
            P->launches++;
        }
    }
    return SPK_OK;
}

template <class T, int KB> int run_red_solve(spk_plan *P, int nrhs, int iters, cudaStream_t st)
{
    if constexpr (KB >= 32) {
        if (nrhs == 1) return run_red_solve_q<T, KB, 1>(P, nrhs, iters, st);
        if constexpr (sizeof(T) == 4)
            if (nrhs > 4) return run_red_solve_q<T, KB, 8>(P, nrhs, iters, st);
        return run_red_solve_q<T, KB, 4>(P, nrhs, iters, st);
    } else {
        if (nrhs == 1) return run_red_solve_s<T, KB, 1>(P, nrhs, iters, st);
        return run_red_solve_s<T, KB, 4>(P, nrhs, iters, st);
    }
}

template <class T> int disp_rs(spk_plan *P, int nrhs, int it, cudaStream_t st)
{
    switch (P->KB) {
    case 2: return run_red_solve<T, 2>(P, nrhs, it, st);
    case 4: return run_red_solve<T, 4>(P, nrhs, it, st);
    case 8: return run_red_solve<T, 8>(P, nrhs, it, st);
    case 16: return run_red_solve<T, 16>(P, nrhs, it, st);
    case 32: return run_red_solve<T, 32>(P, nrhs, it, st);
    case 64:
        if constexpr (sizeof(T) <= 8) return run_red_solve<T, 64>(P, nrhs, it, st);
        else return SPK_EBAND;
    case 128:
        if constexpr (std::is_same<T, float>::value) return run_red_solve<T, 128>(P, nrhs, it, st);
        else return SPK_EBAND;
    default: return SPK_EBAND;
    }
}

} // namespace

extern "C" int spk_reduced_solve(spk_plan *P, int nrhs, int refine_iters, void *stream)
{
    if (P->n_iface <= 0) return SPK_OK;
    if (refine_iters < 1) refine_iters = 1;
    cudaStream_t st = (cudaStream_t)stream;
    const bool low = P->mode == SPK_MIXED && !P->red_fp64;
    if (P->is_complex)
        return low ? disp_rs<cfloat>(P, nrhs, refine_iters, st) : disp_rs<cdouble>(P, nrhs, refine_iters, st);
    return low ? disp_rs<float>(P, nrhs, refine_iters, st) : disp_rs<double>(P, nrhs, refine_iters, st);
}
