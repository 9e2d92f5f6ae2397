// spike_residual.cu -- the FP64 residual of full bands with several columns, on
// the tensor cores (spike_slices.cuh); the other residuals: spike_util.cu.
//
// r = b - A x over C columns costs 2 C flops per entry, and GB300's FP64 pipe
// (2 multiply-adds per clock and SM) is what bounds it from two columns on:
// n = 2,000,000, k = 64, 16 columns took 8.93 ms a pass, 75 % of that pipe's
// rate, where reading the 2.1 GB of values takes 0.31 ms.  Here a warp forms 16
// rows x 8 columns at a time by exact FP16 digit products: 2.35 ms.
//
// A full band -- its entry count says so, since the columns of a row are
// distinct and within the band -- has row r's entries in columns
// max(0, r - kl) .. min(n - 1, r + ku) in order, so neither the column indices
// nor the row pointers are read.  A CTA walks over tiles of 32 or 64 rows: a
// tile's values, one contiguous run of the CSR, come into shared memory by a
// bulk copy issued as soon as the tile before has used its own; the window of x
// they meet is split into digit planes of 8 columns; then every warp takes
// 16 rows and a share of the k steps, splits its values into registers step by
// step, and the warps' integer sums are added, scaled and rounded once per
// result.  The integer instructions of the splitting bound it (ALU pipe 56 %,
// tensor 22 %, FP64 7 % at k = 64), so the FP64 pipe sees two or three operations
// per result and two CTAs share an SM, each one's loads and barriers behind the
// other's work.
#include "spike_slices.cuh"

namespace {

constexpr int RT_NC = 8; // columns per pass (two column tiles per split measured the same)

// geometry of a tile of 16 NW rows, shared by host and device
struct RtGeom {
    int rows, nc, ks, kl16, steps, w, ldx, cap;
    __host__ __device__ RtGeom(int nw, int ks_, int ku, int kl)
    {
        rows = 16 * nw;
        nc = RT_NC;
        ks = ks_;
        kl16 = (kl + 15) & ~15;
        const int ku16 = (ku + 15) & ~15;
        steps = (kl16 + ku16) / 16 + 1;   // k steps of a warp's 16 rows
        w = kl16 + ku16 + rows;           // window of x
        ldx = w + ((72 - (w & 63)) & 63); // = 8 mod 64 halves: conflict-free fragments
        cap = (rows * (kl + ku + 1) + 3) & ~1; // staged values (and the alignment element)
    }
    // digit planes of x; afterwards the warps' partial sums
    __host__ __device__ size_t planes() const
    {
        const size_t p = (size_t)(SL_D + 1) * nc * ldx * sizeof(__half), e = (size_t)ks * rows * nc * 20;
        return ((p > e ? p : e) + 15) & ~(size_t)15;
    }
    __host__ __device__ size_t bytes() const { return 16 + (2 + 8) * 16 * 8 + 64 + 256 + planes() + (size_t)cap * 8; }
};

// entries of a full band before row r (modulo 2^32: the true value fits an int)
__device__ __forceinline__ int band_off(int r, int n, int ku, int kl)
{
    const unsigned m = (unsigned)min(r, kl), q = (unsigned)max(0, r - (n - ku));
    return (int)((unsigned)r * (unsigned)(ku + kl + 1) - (m * (unsigned)kl - m * (m - 1u) / 2u) - q * (q + 1u) / 2u);
}

// The results of a tile of rows from R0 on without digits, from the values
// sv[band_off(row) ..]: four rows per warp at a time and all of a row's columns
// together, eight lanes to a row, so that a value of A is read once and a result
// costs 68 clocks of the FP64 pipe at k = 64 (86 in k_residual, 160 one by one).
// Squared norms go into sw, a warp's own sixteen values.  (A call: the digits' loop
// needs its registers.)
template <int ROWS, int WARPS>
__device__ __noinline__ void in_fp64(int R0, const double *sv, int n, int ku, int kl,
                                     const double *__restrict__ x, const double *__restrict__ b, double *r, int nc,
                                     int want_b, double *sw)
{
    constexpr int NC = RT_NC;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = lane & 7;
    double qr = 0.0, qb = 0.0; // squared norms of column h
    for (int rg = warp * 4; rg < ROWS && R0 + rg < n; rg += WARPS * 4) {
        const int row = R0 + rg + (lane >> 3), rl = min(row, n - 1), first = max(0, rl - kl);
        const int len = row < n ? min(n - 1, row + ku) - first + 1 : 0;
        const double *av = sv + band_off(rl, n, ku, kl), *xc = x + first;
        const bool mine = row < n && h < nc;
        const double bv = mine ? b[(size_t)h * n + row] : 0.0;
        double f[NC];
#pragma unroll
        for (int c = 0; c < NC; c++) f[c] = 0.0;
        for (int q = h; q < ku + kl + 1; q += 8) {
            const bool on = q < len;
            const double v = on ? av[q] : 0.0;
#pragma unroll
            for (int c = 0; c < NC; c++)
                if (c < nc) f[c] = fma(v, on ? xc[(size_t)c * n + q] : 0.0, f[c]);
        }
        __syncwarp();
        // column c's sum ends at lane c of the eight
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            const bool up = (h & o) != 0;
#pragma unroll
            for (int e = 0; e < o; e++) {
                const double send = up ? f[e] : f[e + o];
                f[e] = (up ? f[e + o] : f[e]) + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        if (mine) {
            const double rv = bv - f[0];
            r[(size_t)h * n + row] = rv;
            qr = fma(rv, rv, qr);
            if (want_b) qb = fma(bv, bv, qb);
        }
    }
#pragma unroll
    for (int o = 8; o < 32; o *= 2) {
        qr += __shfl_xor_sync(0xffffffffu, qr, o);
        qb += __shfl_xor_sync(0xffffffffu, qb, o);
    }
    if (lane < 8) {
        sw[warp * 16 + h] += qr;
        sw[warp * 16 + 8 + h] += qb;
    }
}

// NW groups of 16 rows, KS warps per group (each every KS-th k step, at most
// SL_FLUSH of them), at most UPW units (32 pairs of rows of one column) of the
// window per warp
template <int NW, int KS, int UPW>
__global__ void __launch_bounds__(32 * NW * KS, 2)
    k_residual_sl(int n, int ku, int kl, const double *__restrict__ a, const double *__restrict__ x,
                  const double *__restrict__ b, double *r, int nc, int want_b, double *norms, double *bnorms,
                  unsigned *err)
{
    constexpr int WARPS = NW * KS, NTH = 32 * WARPS, ROWS = 16 * NW, NC = RT_NC;
    constexpr int OPT = (ROWS * NC + NTH - 1) / NTH; // results per thread and tile
    const RtGeom G(NW, KS, ku, kl);
    extern __shared__ __align__(16) char sm[];
    uint64_t *bar = (uint64_t *)sm;
    double *sr = (double *)(sm + 16), *sb = sr + 16;  // squared norms of r and b per column
    double *sw = sb + 16;                             // and, by warp, those of tiles without digits
    int *ec = (int *)(sw + 8 * 16), *er = ec + 16; // scale exponents of the columns and rows
    char *pl = (char *)(er + 64);
    unsigned short *px = (unsigned short *)pl;        // [digit][column][ldx]; plane SL_D: magnitudes
    long long *xh = (long long *)pl, *xl = xh + KS * ROWS * NC; // partial sums, [ks][column][row]
    float *xg = (float *)(xl + KS * ROWS * NC);
    double *sa0 = (double *)(pl + G.planes());

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int wr = warp % NW, wk = warp / NW; // this warp's rows and k steps
    for (int q = tid; q < 10 * 16; q += NTH) sr[q] = 0.0; // sr, sb, sw
    if (tid == 0) {
        mbar_init(bar, 1);
        mbar_init_fence();
    }
    __syncthreads();
    const int tiles = (n + ROWS - 1) / ROWS;
    // The values of tile i: whole 16-byte pieces by a bulk copy (one thread), the
    // odd ones at the ends by plain stores; element e of the CSR sits at index
    // e - e0 + mis.
    auto fetch = [&](int i) {
        if (i >= tiles) return;
        const int e0 = band_off(i * ROWS, n, ku, kl), cnt = band_off(min(n, (i + 1) * ROWS), n, ku, kl) - e0;
        const double *src = a + e0;
        const int mis = (int)(((uintptr_t)src >> 3) & 1), head = mis && cnt ? 1 : 0, body = (cnt - head) & ~1;
        if (head) sa0[mis] = src[0];
        if (cnt > head + body) sa0[mis + head + body] = src[head + body];
        fence_proxy_async();
        mbar_arrive_expect_tx(bar, (unsigned)body * 8);
        if (body) bulk_g2s(sa0 + mis + head, src + head, (unsigned)body * 8, bar);
    };
    // the window of x of tile i, held in registers until its scale is known
    double v[UPW][2];
    int uhk[UPW]; // the units' (column << 16 | first row of the lane's pair); column NC: none
    {
        const int cpu = (G.w + 63) / 64; // units per column
#pragma unroll
        for (int u = 0; u < UPW; u++) {
            const int un = warp + u * WARPS, h = un / cpu, k = (un - h * cpu) * 64 + 2 * lane;
            uhk[u] = (h < NC && k < G.w ? h : NC) << 16 | k;
        }
    }
    auto window = [&](int i) {
#pragma unroll
        for (int u = 0; u < UPW; u++) {
            const int h = uhk[u] >> 16, c = i * ROWS - G.kl16 + (uhk[u] & 0xffff);
            v[u][0] = v[u][1] = 0.0;
            if (h < nc && i < tiles) {
                const double *xc = x + (size_t)h * n;
                if (c >= 0 && c < n) v[u][0] = xc[c];
                if (c + 1 >= 0 && c + 1 < n) v[u][1] = xc[c + 1];
            }
        }
    };
    unsigned phase = 0u;
    double nr[OPT], nb[OPT];
#pragma unroll
    for (int i = 0; i < OPT; i++) nr[i] = nb[i] = 0.0;
    int skip = 0; // tiles yet to be formed without trying the digits
    if (tid == 0) fetch(blockIdx.x);
    window(blockIdx.x);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int R0 = tile * ROWS, xw0 = R0 - G.kl16, e0 = band_off(R0, n, ku, kl);
        const double *sa = sa0 + (int)(((uintptr_t)(a + e0) >> 3) & 1);
        // ---- scales of the columns and the rows
        if (tid < NC) ec[tid] = 0;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < UPW; u++) {
            // (integer tests: a comparison would go through the FP64 pipe)
            const unsigned h0 = (unsigned)__double2hiint(v[u][0]) & 0x7fffffffu, l0 = (unsigned)__double2loint(v[u][0]);
            const unsigned h1 = (unsigned)__double2hiint(v[u][1]) & 0x7fffffffu, l1 = (unsigned)__double2loint(v[u][1]);
            // 0: zero; a subnormal counts as the smallest exponent
            const unsigned e = __reduce_max_sync(0xffffffffu, max(max(h0, h1) >> 20, (h0 | l0 | h1 | l1) != 0u ? 1u : 0u));
            // the unit's column is its lane 0's: lanes past the window hold zeros
            if (lane == 0 && e) atomicMax(&ec[uhk[u] >> 16], (int)e);
        }
        const bool landed = mbar_wait(bar, phase);
        if (__syncthreads_or(!landed)) { // no norm: the solve must not take this for converged
            if (tid == 0) {
                atomicOr(err, SPK_DEV_ERR_TIMEOUT);
                norms[0] = __longlong_as_double(0x7ff8000000000000ll);
            }
            mbar_wait(bar, phase); // once more: the shared memory is another block's after this one
            return;
        }
        phase ^= 1u;
        if (skip > 0) {
            skip--;
            in_fp64<ROWS, WARPS>(R0, sa - e0, n, ku, kl, x, b, r, nc, want_b, sw);
            __syncthreads(); // every value has been used
            if (tid == 0) fetch(tile + gridDim.x);
            window(tile + gridDim.x);
            continue;
        }
        const bool inner = R0 >= kl && R0 + ROWS <= n - ku; // rows of ku + kl + 1 entries each
        const int wid = ku + kl + 1;
        for (int i = warp; i < ROWS; i += WARPS) {
            unsigned m = 0;
            if (R0 + i < n) {
                const int t0 = inner ? i * wid : band_off(R0 + i, n, ku, kl) - e0;
                const int t1 = inner ? t0 + wid : band_off(R0 + i + 1, n, ku, kl) - e0;
                for (int q = t0 + lane; q < t1; q += 32) m = max(m, (unsigned)__double2hiint(sa[q]) & 0x7fffffffu);
            }
            m = __reduce_max_sync(0xffffffffu, m) >> 20;
            if (lane == 0) er[i] = (int)m;
        }
        // ---- digit planes
#pragma unroll
        for (int u = 0; u < UPW; u++) {
            const int h = uhk[u] >> 16, k = uhk[u] & 0xffff;
            if (h < NC) {
                const int E = ec[h];
                const bool live = E >= 64 && E < 0x7ff;
                SlPair(live ? v[u][0] : 0.0, live ? v[u][1] : 0.0, live ? E : 64)
                    .store((unsigned *)(px + (size_t)h * G.ldx + k), NC * G.ldx / 2);
            }
        }
        __syncthreads();
        // ---- 16 rows x NC columns, every KS-th k step
        SlAcc acc;
        acc.zero();
        {
            int lo[2], hi[2], E[2];
            const double *row[2];
#pragma unroll
            for (int p = 0; p < 2; p++) {
                const int rw = wr * 16 + g + 8 * p, rr = R0 + rw;
                lo[p] = 1 << 20;
                hi[p] = 0;
                row[p] = sa;
                E[p] = er[rw];
                if (rr < n && E[p] >= 64 && E[p] < 0x7ff) {
                    lo[p] = max(0, rr - kl) - xw0;
                    hi[p] = min(n - 1, rr + ku) - xw0;
                    row[p] = sa + (inner ? rw * wid : band_off(rr, n, ku, kl) - e0) - lo[p];
                } else {
                    E[p] = 64;
                }
            }
            // steps whose 16 columns every row of the warp holds need no test
            const int lo_all = __reduce_max_sync(0xffffffffu, max(lo[0], lo[1]));
            const int hi_all = __reduce_min_sync(0xffffffffu, min(hi[0], hi[1]));
            for (int s = wk; s < G.steps; s += KS) {
                const int kb = wr * 16 + s * 16, k0 = kb + 2 * t;
                double w[2][4];
                if (kb >= lo_all && kb + 15 <= hi_all) {
#pragma unroll
                    for (int p = 0; p < 2; p++)
#pragma unroll
                        for (int q = 0; q < 4; q++) w[p][q] = row[p][k0 + (q & 1) + (q >> 1) * 8];
                } else {
#pragma unroll
                    for (int p = 0; p < 2; p++)
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const int k = k0 + (q & 1) + (q >> 1) * 8;
                            w[p][q] = k >= lo[p] && k <= hi[p] ? row[p][k] : 0.0;
                        }
                }
                SlFragA A;
                A.split(w, E[0], E[1]);
                const unsigned *xb = (const unsigned *)(px + g * G.ldx + k0);
                const int st = NC * G.ldx / 2;
                acc.step(A, [&](int i, int q) { return xb[i * st + 4 * q]; });
            }
        }
        __syncthreads(); // every value and plane has been read
        if (tid == 0) fetch(tile + gridDim.x);
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int o = (wk * NC + 2 * t + (e & 1)) * ROWS + wr * 16 + g + 8 * (e >> 1);
            long long hi, lo;
            acc.total(e, hi, lo);
            xh[o] = hi;
            xl[o] = lo;
            xg[o] = acc.g[e];
        }
        window(tile + gridDim.x); // lands while the results are formed
        __syncthreads();
        // ---- r = b - A x, a row of one column per thread
        bool many = false;
#pragma unroll
        for (int i = 0; i < OPT; i++) { // (whole warps: one column each, the same in every tile)
            const int o = tid + i * NTH, h = o / ROWS, rw = o - h * ROWS, row = R0 + rw;
            if (h >= nc) break;
            const bool live = row < n;
            const double bv = live ? b[(size_t)h * n + row] : 0.0;
            long long hi = 0, lo = 0;
            float mg = 0.f;
#pragma unroll
            for (int s = 0; s < KS; s++) {
                hi += xh[s * ROWS * NC + o];
                lo += xl[s * ROWS * NC + o];
                mg += xg[s * ROWS * NC + o];
            }
            const int E = er[rw], Ec = ec[h], sc = 56 + E + Ec - 2 * (1023 + 61);
            const bool redo = live && !(E < 0x7ff && (Ec == 0 || (E >= 64 && Ec >= 64 && Ec < 0x7ff && mg >= SL_GUARD &&
                                                                 sc > -900 && sc < 850)));
            double ax = redo || Ec == 0 ? 0.0 : sl_round(hi, lo, sc);
            // the results outside the scales' reach, one by one in FP64
            many = many || redo;
            for (unsigned todo = __ballot_sync(0xffffffffu, redo); todo; todo &= todo - 1) {
                const int src = __ffs(todo) - 1, rr = __shfl_sync(0xffffffffu, row, src);
                const int t0 = band_off(rr, n, ku, kl), len = band_off(rr + 1, n, ku, kl) - t0;
                const double *xc = x + (size_t)h * n + max(0, rr - kl);
                double sum = 0.0;
                for (int q = lane; q < len; q += 32) sum = fma(a[t0 + q], xc[q], sum);
                for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
                if (lane == src) ax = sum;
            }
            if (live) {
                const double rv = bv - ax;
                r[(size_t)h * n + row] = rv;
                nr[i] = fma(rv, rv, nr[i]);
                if (want_b) nb[i] = fma(bv, bv, nb[i]);
            }
        }
        // (The partial sums may be overwritten by the next planes.)  Where many results
        // were formed in FP64 -- a solution that falls off between its sources -- what
        // follows looks alike, and fifteen tiles go without trying the digits.  n = 400,000,
        // two residuals, a source every 4 k rows: k = 64, 16 columns 8.47 -> 3.98 ms
        // (k_residual 3.80), k = 24, 4 columns 1.46 -> 0.65 (0.45); n = 200,000, k = 100, 8
        // columns 1.97 -> 1.46 (1.55).  U[-1,1] solutions pay 1.5 % for the count.
        if (__syncthreads_count(many) > NTH / 4) skip = 15;
    }
#pragma unroll
    for (int i = 0; i < OPT; i++) {
        const int h = (tid + i * NTH) / ROWS;
        if (h >= nc) break;
        for (int s = 16; s > 0; s >>= 1) {
            nr[i] += __shfl_xor_sync(0xffffffffu, nr[i], s);
            nb[i] += __shfl_xor_sync(0xffffffffu, nb[i], s);
        }
        if (lane == 0) {
            atomicAdd(&sr[h], nr[i]);
            atomicAdd(&sb[h], nb[i]);
        }
    }
    __syncthreads();
    if (tid < nc) {
        double qr = sr[tid], qb = sb[tid];
        for (int w = 0; w < WARPS; w++) {
            qr += sw[w * 16 + tid];
            qb += sw[w * 16 + 8 + tid];
        }
        atomicAdd(&norms[tid], qr);
        if (want_b) atomicAdd(&bnorms[tid], qb);
    }
}

template <int NW, int KS, int UPW>
int run(const spk_plan *P, const double *a, const double *x, const double *b, double *r, int h0, int nc, int nrhs,
        int want_b, double *norms, cudaStream_t st)
{
    const RtGeom G(NW, KS, P->ku, P->kl);
    const size_t smem = G.bytes();
    if (G.nc * ((G.w + 63) / 64) > UPW * NW * KS || (G.steps + KS - 1) / KS > SL_FLUSH) return SPK_EARG;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_residual_sl<NW, KS, UPW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 227 * 1024) != cudaSuccess)
            return SPK_ECUDA;
        attr = true;
    }
    const int tiles = (P->n + G.rows - 1) / G.rows, ctas = 152 * (smem <= 112 * 1024 ? 2 : 1);
    const size_t o = (size_t)h0 * P->n;
    k_residual_sl<NW, KS, UPW><<<tiles < ctas ? tiles : ctas, 32 * NW * KS, smem, st>>>(
        P->n, P->ku, P->kl, a, x + o, b + o, r + o, nc, want_b, norms + h0, norms + nrhs + h0, P->d_err);
    if (cudaGetLastError() != cudaSuccess) return SPK_ECUDA;
    ((spk_plan *)P)->launches++;
    return SPK_OK;
}

} // namespace

// a full band (the caller checked the entry count), up to 128 each side
extern "C" int spk_residual_slices(const spk_plan *P, const double *d_aij, const double *d_x, const double *d_b,
                                   double *d_r, int nrhs, int want_bnorm, double *d_norms, void *stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    // 64 rows per tile while two CTAs with their values fit an SM, 32 beyond
    const bool wide = P->ku > 64 || P->kl > 64;
    for (int h0 = 0; h0 < nrhs; h0 += 8) {
        const int nc = nrhs - h0 < 8 ? nrhs - h0 : 8;
        const int rc = wide ? run<2, 4, 5>(P, d_aij, d_x, d_b, d_r, h0, nc, nrhs, want_bnorm, d_norms, st)
                            : run<4, 2, 3>(P, d_aij, d_x, d_b, d_r, h0, nc, nrhs, want_bnorm, d_norms, st);
        if (rc != SPK_OK) return rc;
    }
    return SPK_OK;
}
