// spike_slices.cuh -- FP64 dot products on the tensor cores, by exact products of digits.
//
// GB300 retires 2 FP64 multiply-adds per clock and SM, its tensor cores about
// a thousand FP16 ones.  An FP64 value that shares a power-of-two scale with
// the other values of its row (left operand) or column (right operand) is a
// 62-bit integer, X = v 2^(61 - E) with |v| < 2^(E+1), and that integer is eight
// signed byte digits, X = sum_i d_i 256^(7-i), -128 <= d_i <= 127.  Digits are
// exact in FP16 and their products exact in FP32, so
//
//     sum_k X_k Y_k = sum_s 256^(14-s) sum_{i+j=s} sum_k d_i(X_k) d_j(Y_k)
//
// takes one m16n8k16 product per digit pair with the FP32 accumulator of each
// s exact as long as it holds at most SL_FLUSH k steps: 8 pairs x 2^14 x 128
// <= 2^24 at s = 7 (the splitting is Ozaki, Ogita, Oishi, Rump's, Numer.
// Algorithms 59, 2012, with the digits taken by bytes).  The pairs with s >= 8 are
// left out: per term at most 7.03 x 2^14 x 256^6, 2^-57.2 of the two scales'
// product, and the bits of values far below their scale that shift out of the
// digits, at most 2^-59.  A sum of K terms can miss K times that, 2^-51 of the
// scales' product at K = 64 and 2^-49 at 257, where every digit is near its
// extreme and of one sign; unrelated digits miss sqrt(K) 2^-60, 2^-57 and 2^-56.
//
// That is measured by the scales, an FP64 sum's error by the terms it adds.  So
// the scales' reach is watched by one more product, of |x| and |y| as powers of
// two rounded down: where sum |x||y| is below SL_GUARD of the scales' product the
// caller forms that result in FP64 as before.  Above it a result misses at most
// 2^6 times the above of its terms' magnitudes, 2^-50 for unrelated digits (an FP64
// chain of K terms: up to K 2^-53), and where the terms come near the scales, as in
// the rows of a dominant band, less than the chain's roundings (K = 129, terms of
// one magnitude: rms 2.6e-16 against 2.2e-14).
#pragma once
#include <cuda_fp16.h>

#include "spike_common.cuh"

constexpr int SL_D = 8;              // digits
constexpr int SL_FLUSH = 8;          // k steps (of 16) an FP32 accumulator holds exactly
constexpr float SL_GUARD = 0.015625f; // 2^-6

// biased exponent of |v| (0 for zero and subnormals, 0x7ff for inf and NaN)
__device__ __forceinline__ int sl_exp(double v) { return (int)(((unsigned)__double2hiint(v) >> 20) & 0x7ffu); }

// the 64-bit word whose bytes are the digits of |v| (+128 each) at scale exponent
// E (biased; every value of the row has exponent <= E, 64 <= E < 0x7ff; a zero
// or subnormal v shifts out whole), and |v| 2^-E rounded down to a power of two, in FP16
__device__ __forceinline__ void sl_split(double v, int E, unsigned &hi, unsigned &lo, unsigned &mag)
{
    const unsigned vh = (unsigned)__double2hiint(v), vl = (unsigned)__double2loint(v);
    const unsigned sh = (unsigned)(E - (int)((vh >> 20) & 0x7ffu));
    // 53 bits at the top of 62: v 2^(61 - E) where v has exponent E
    const unsigned mh = __funnelshift_l(vl, (vh & 0xfffffu) | 0x100000u, 9), ml = vl << 9;
    unsigned long long m = ((unsigned long long)mh << 32) | ml, q;
    asm("shr.u64 %0, %1, %2;" : "=l"(q) : "l"(m), "r"(sh)); // shifts of 64 and more give 0
    m = q + 0x8080808080808080ull;
    hi = (unsigned)(m >> 32);
    lo = (unsigned)m;
    mag = (unsigned)max(15 - (int)sh, 0) << 10;
}

// Two values of one row (or column), their digits packed as FP16 pairs on
// demand.  A digit's bytes under the exponent of 1024 are 1024 + 128 + d, exact,
// and one fused multiply-add takes the bias off and puts the sign on: d is a
// digit of |v|, which spares negating the 64-bit words.
struct SlPair {
    unsigned q[4];      // bytes of digits 2 i (v0, v1), 2 i + 1 (v0, v1)
    unsigned sg, nb;    // +-1 and -+1152 of both signs
    unsigned mg;        // the magnitudes
    __device__ __forceinline__ SlPair(double v0, double v1, int E)
    {
        unsigned h0, l0, m0, h1, l1, m1;
        sl_split(v0, E, h0, l0, m0);
        sl_split(v1, E, h1, l1, m1);
        q[0] = __byte_perm(h0, h1, 0x6273);
        q[1] = __byte_perm(h0, h1, 0x4051);
        q[2] = __byte_perm(l0, l1, 0x6273);
        q[3] = __byte_perm(l0, l1, 0x4051);
        const unsigned s = __byte_perm((unsigned)__double2hiint(v0), (unsigned)__double2hiint(v1), 0x7030) & 0x80008000u;
        sg = s | 0x3c003c00u;
        nb = s ^ 0xe480e480u;
        mg = m0 | (m1 << 16);
    }
    // digit I (0 = leading): low half of v0, high half of v1
    template <int I> __device__ __forceinline__ unsigned digit() const
    {
        const unsigned p = __byte_perm(q[I / 2], 0x64646464u, I & 1 ? 0x4342 : 0x4140);
        const __half2 d = __hfma2(*reinterpret_cast<const __half2 *>(&p), *reinterpret_cast<const __half2 *>(&sg),
                                  *reinterpret_cast<const __half2 *>(&nb));
        return *reinterpret_cast<const unsigned *>(&d);
    }
    // all digits and the magnitudes, st words apart
    __device__ __forceinline__ void store(unsigned *o, int st) const
    {
        o[0] = digit<0>();
        o[st] = digit<1>();
        o[2 * st] = digit<2>();
        o[3 * st] = digit<3>();
        o[4 * st] = digit<4>();
        o[5 * st] = digit<5>();
        o[6 * st] = digit<6>();
        o[7 * st] = digit<7>();
        o[8 * st] = mg;
    }
};

__device__ __forceinline__ void sl_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// A digits of one k step: a[i] = the m16n8k16 left fragment of digit i, mg = of the magnitudes
struct SlFragA {
    unsigned a[SL_D][4], mg[4];
    // v[r][q]: rows (lane / 4) and (lane / 4) + 8 (r), columns 2 (lane % 4) + {0, 1, 8, 9} (q)
    __device__ __forceinline__ void split(const double (&v)[2][4], int E0, int E1)
    {
#pragma unroll
        for (int r = 0; r < 2; r++)
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const SlPair d(v[r][2 * q], v[r][2 * q + 1], r ? E1 : E0);
                const int f = r + 2 * q; // fragment registers: (g, lo), (g + 8, lo), (g, hi), (g + 8, hi)
                a[0][f] = d.digit<0>();
                a[1][f] = d.digit<1>();
                a[2][f] = d.digit<2>();
                a[3][f] = d.digit<3>();
                a[4][f] = d.digit<4>();
                a[5][f] = d.digit<5>();
                a[6][f] = d.digit<6>();
                a[7][f] = d.digit<7>();
                mg[f] = d.mg;
            }
    }
};

// one warp's 16 x 8 sums of digit products.  Element e of a lane: row
// (lane / 4) + 8 (e / 2), column 2 (lane % 4) + e % 2.
struct SlAcc {
    float c[SL_D][4], g[4];
    __device__ __forceinline__ void zero()
    {
#pragma unroll
        for (int e = 0; e < 4; e++) {
#pragma unroll
            for (int s = 0; s < SL_D; s++) c[s][e] = 0.f;
            g[e] = 0.f;
        }
    }
    // += the step's products; bfrag(i, r): register r of digit i's right
    // fragment (i = SL_D: the magnitudes').  ND < SL_D: the leading ND sums only.
    template <int ND = SL_D, class B> __device__ __forceinline__ void step(const SlFragA &A, B bfrag)
    {
        sl_mma(g, A.mg, bfrag(SL_D, 0), bfrag(SL_D, 1));
#pragma unroll
        for (int j = 0; j < ND; j++) {
            const unsigned b0 = bfrag(j, 0), b1 = bfrag(j, 1);
#pragma unroll
            for (int i = 0; i + j < ND; i++) sl_mma(c[i + j], A.a[i], b0, b1);
        }
    }
    // element e as integers, hi 2^32 + lo in units of 256^7
    __device__ __forceinline__ void total(int e, long long &hi, long long &lo) const
    {
        hi = __float2int_rn(c[3][e]);
        lo = __float2int_rn(c[7][e]);
#pragma unroll
        for (int s = 0; s < 3; s++) { // one wide multiply-add each
            hi += (long long)__float2int_rn(c[s][e]) * (1 << (24 - 8 * s));
            lo += (long long)__float2int_rn(c[4 + s][e]) * (1 << (24 - 8 * s));
        }
    }
};

// (hi 2^32 + lo) 2^p to FP64, rounded to nearest, with integer instructions
// (the FP64 pipe is the scarce one); |hi| < 2^60, |lo| < 2^60, and p such that
// a nonzero result is normal
__device__ __forceinline__ double sl_round(long long hi, long long lo, int p)
{
    hi += lo >> 32;
    unsigned w0 = (unsigned)lo; // value = hi 2^32 + w0
    const unsigned neg = (unsigned)((int)(hi >> 32) >> 31);
    // (no branches: several results are in flight at once)
    w0 = (w0 ^ neg) - neg;
    unsigned long long h = ((unsigned long long)hi ^ (((unsigned long long)neg << 32) | neg)) + (neg && w0 == 0u ? 1u : 0u);
    const bool small = h == 0;
    h = small ? (unsigned long long)w0 << 31 : h;
    p = small ? p - 63 : p;
    const unsigned wl = small ? 0u : w0;
    const bool none = h == 0;
    const int z = __clzll((long long)h) & 63; // h < 2^62 unless small (bit 63 free)
    unsigned long long m = (h << z) | (((unsigned long long)wl << 31) >> (63 - z)); // top bit at 63
    p += 32 - z;
    const unsigned rest = (unsigned)m & 0x7ffu;
    m >>= 11;
    m += rest > 0x400u || (rest == 0x400u && ((unsigned)m & 1u)) ? 1u : 0u; // 53 bits, to nearest
    // m 2^(p + 11): a carry to 2^53 bumps the exponent through the addition
    const unsigned long long bits = ((unsigned long long)(unsigned)(p + 11 + 52 + 1022) << 52) + m;
    return none ? 0.0 : __longlong_as_double((long long)(bits | ((unsigned long long)(neg & 0x80000000u) << 32)));
}
