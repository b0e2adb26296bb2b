// kernels_int.cuh -- the FP64 correlator in exact integer arithmetic.
//
// GB300 executes 1.7 FP64 operations per clock and SM (measured) against 58
// 32x32 -> 64-bit integer multiply-adds and 110 integer additions, so FP64
// data are correlated without the FP64 pipe:
//
//   * A block of N = 4096 samples becomes integers X of up to 54 bits: each
//     sample's significand shifted to a common exponent (62 bits, exact for
//     samples within 2^9 of the largest), the block's mean level taken off
//     (the numerator does not depend on it, templates are zero-mean), the
//     result rounded once.  The unit is the finest at which every window's
//     2-norm stays below 2^54.6 (about 2^-52 of the largest deviation for a
//     seismogram).  Template coefficients (demeaned, unit norm) become
//     integers B = round(b 2^53).
//   * The numerators sum X[k + j] B[j] are then computed exactly: cyclic
//     correlation by number-theoretic transforms of N points modulo four
//     primes p = 1 mod 8192 just below 2^31 / 14, and the Chinese remainder
//     theorem.  |numerator| <= 2^54.6 2^53 stays below half the primes' product
//     (2^107.7) by Cauchy-Schwarz.
//   * Window variances come from prefix sums of X (50 bits, sums 64) and X^2
//     (sums 128 bits) of a tile: V = L S2 - S1^2 is exact.  1 / sqrt(V) starts from the
//     FP32 reciprocal square root and takes one third-order step in 60-bit
//     fixed point.
//
// The remaining errors are the two roundings of the inputs and three roundings
// to FP64 at the end: below those of an FP64 transform, whose rounding grows
// with the block's energy and log N (relative errors of the coefficients of
// band-passed templates of 200 .. 2,000 samples against two-pass sums in
// quadruple precision: 5.9e-16 .. 7.6e-16, FP64 transforms 7.8e-16 ..
// 1.75e-15).
//
// Arithmetic modulo p: signed Montgomery products with R = 2^32 (three
// instructions: wide multiply, low multiply, wide multiply-add), whose result
// is at most |a b| / 2^32 + p / 2 in magnitude.  With constants |b| <= p / 2
// and |a| < 2^31 that is at most 0.75 p, so a 16-point transform of such
// values, additions only between the products, stays within 12 p < 2^31:
// no reduction is needed inside a pass.
#pragma once
#include "kernels_mf.cuh"
#include "int_params.h"

namespace mfgpu {

struct IntParams
{
    XcorrParams<double> x;  // as the FFT correlator's (spectra and twiddles unused)
    const int *B;           // [template][prime][kIntN]
    const int *tw;          // [prime][kIntTw]
    int Lmax;               // longest template
    long n;                 // samples per row
    IntConsts c;
};

// a b R^-1 mod p (nq = -p^-1 mod 2^32)
__device__ __forceinline__ int mont(int a, int b, int p, int nq)
{
    long long t, r;
    int m;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(t) : "r"(a), "r"(b));
    m = (int) t * nq;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(m), "r"(p), "l"(t));
    return (int) (r >> 32);
}

// the constants of one prime, in registers
struct IntField
{
    int p, nq, one, w1, w2, w3, w4, w6, w9;
    __device__ __forceinline__ explicit IntField(const IntPrime &c)
        : p(c.p), nq(c.nq), one(c.one), w1(c.w1), w2(c.w2), w3(c.w3), w4(c.w4), w6(c.w6), w9(c.w9)
    {
    }
    __device__ __forceinline__ int mul(int a, int b) const { return mont(a, b, p, nq); }
};

__device__ __forceinline__ void int_dft4(const IntField &f, int &a0, int &a1, int &a2, int &a3)
{
    const int s0 = a0 + a2, d0 = a0 - a2, s1 = a1 + a3, d1 = f.mul(a1 - a3, f.w4);
    a0 = s0 + s1;
    a2 = s0 - s1;
    a1 = d0 + d1;
    a3 = d0 - d1;
}

// 16-point transform with the 16th root w1; input at most 0.75 p, output at
// most 12 p in magnitude (the same index scheme as dft16)
__device__ __forceinline__ void int_dft16(const IntField &f, int (&a)[16])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) int_dft4(f, a[j], a[j + 4], a[j + 8], a[j + 12]);
    a[5] = f.mul(a[5], f.w1);
    a[9] = f.mul(a[9], f.w2);
    a[13] = f.mul(a[13], f.w3);
    a[6] = f.mul(a[6], f.w2);
    a[10] = f.mul(a[10], f.w4);
    a[14] = f.mul(a[14], f.w6);
    a[7] = f.mul(a[7], f.w3);
    a[11] = f.mul(a[11], f.w6);
    a[15] = f.mul(a[15], f.w9);
#pragma unroll
    for (int m = 0; m < 4; ++m) int_dft4(f, a[4 * m], a[4 * m + 1], a[4 * m + 2], a[4 * m + 3]);
    int t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) t[i] = a[i];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int q = 0; q < 4; ++q) a[m + 4 * q] = t[4 * m + q];
}

// Shared-memory position of element i between the passes: bank bits 0-3 mix
// in index bits 5-8, bank bit 4 mixes in bit 8, so the strided stores of the
// first two passes (lanes 16 apart; two runs of 16 lanes 256 apart) and the
// contiguous loads all hit 32 different banks.
__device__ __forceinline__ int int_swz(int i) { return i ^ ((i >> 5) & 15) ^ ((i >> 4) & 16); }

// The three radix-16 passes of one transform by a team of 256 threads
// (natural order in and out): a holds the elements q + 256 r on entry and on
// return.  s: 4096 words of exchange buffer, free on entry; the team's loads
// of it are done on return.  tw: rows r = 1 .. 15 of the twiddles of the
// second (16 columns) and third pass (256 columns).
template <bool LD_ALIAS>
__device__ __forceinline__ void int_ntt(const IntField &f, int (&a)[16], int *s, const int *tw, int q, int bar_id)
{
    int_dft16(f, a);
    if constexpr (LD_ALIAS) __syncthreads();  // the first pass's inputs lie in the exchange buffers
    {
        // element 16 q + r
        const int hi = 16 * q ^ ((q >> 4 & 1) << 4), x = (q >> 1) & 15;
#pragma unroll
        for (int r = 0; r < 16; ++r) s[hi + (r ^ x)] = a[r];
    }
    team_sync<-1, 256>(bar_id);
    const int qe = int_swz(q), qo = int_swz(q + 256) - 256;
#pragma unroll
    for (int r = 0; r < 16; ++r) a[r] = s[256 * r + ((r & 1) ? qo : qe)];
    team_sync<-1, 256>(bar_id);
    {
        const int k = q & 15;
        a[0] = f.mul(a[0], f.one);
#pragma unroll
        for (int r = 1; r < 16; ++r) a[r] = f.mul(a[r], tw[(r - 1) * 16 + k]);
        int_dft16(f, a);
        // element 256 (q >> 4) + 16 r + k
        const int b = (q >> 4) & 1, lo = k ^ (b << 3), hi = 256 * (q >> 4);
#pragma unroll
        for (int r = 0; r < 16; ++r) s[hi + ((16 * r) ^ (b << 4)) + (lo ^ (r >> 1))] = a[r];
    }
    team_sync<-1, 256>(bar_id);
#pragma unroll
    for (int r = 0; r < 16; ++r) a[r] = s[256 * r + ((r & 1) ? qo : qe)];
    team_sync<-1, 256>(bar_id);
    a[0] = f.mul(a[0], f.one);
#pragma unroll
    for (int r = 1; r < 16; ++r) a[r] = f.mul(a[r], tw[240 + (r - 1) * 256 + q]);
    int_dft16(f, a);
}

// v mod p for |v| <= 2^54: v = vh 2^25 + vl (at most 0.79 p)
__device__ __forceinline__ int int_mod(const IntField &f, int c25, long long v)
{
    return f.mul((int) (v >> 25), c25) + (int) (v & ((1 << 25) - 1));
}

// ---- fixed point ------------------------------------------------------------
// biased exponent of a sample (subnormals: 1), 2047 for an infinity or NaN
__device__ __forceinline__ int int_expo(long long bits)
{
    const int e = (int) (bits >> 52) & 2047;
    return e > 0 ? e : 1;
}
// the sample in units of 2^(emax - 1084): exact within 2^9 of the largest
// exponent emax, rounded below; |result| < 2^62
__device__ __forceinline__ long long int_fixed(long long bits, int emax)
{
    const int e = (int) (bits >> 52) & 2047;
    unsigned long long m = (unsigned long long) bits & ((1ull << 52) - 1);
    if (e > 0) m |= 1ull << 52;
    const int d = emax - (e > 0 ? e : 1) - 9;
    m = d <= 0 ? m << -d : (d < 60 ? (m + (1ull << (d - 1))) >> d : 0ull);
    return bits < 0 ? -(long long) m : (long long) m;
}

// Block-wide reductions of NTH threads (NTH / 32 warps); red: 32 words.
template <int NTH> __device__ __forceinline__ int int_block_max(int v, int *red)
{
    v = __reduce_max_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const int l = threadIdx.x & 31;
    return __reduce_max_sync(0xffffffffu, l < NTH / 32 ? red[l] : -(1 << 30));
}
template <int NTH> __device__ __forceinline__ long long int_block_sum(long long v, long long *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const int l = threadIdx.x & 31;
    v = l < NTH / 32 ? red[l] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int NTH> __device__ __forceinline__ float int_block_fsum(float v, float *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    const int l = threadIdx.x & 31;
    v = l < NTH / 32 ? red[l] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Quantises the PER samples (bit patterns) each of NTH threads holds, N = NTH
// PER in all: v[] receives the integers, the return value is the exponent of
// their unit (x - level = v 2^ex up to half a unit).  An infinity or NaN
// counts as 0 and sets *bad.  NORM false: at most kIntXBits bits.  NORM true:
// the finest unit at which the 2-norm of every window of at most L samples
// stays below 2^kIntNormBits (bounded by sqrt(L) times the largest deviation
// and by the norm of all samples), at most 54 bits.
template <int NTH, int PER, bool NORM>
__device__ __forceinline__ int int_quantise(long long (&v)[PER], int *ired, long long *lred, float L, bool *bad)
{
    constexpr int LOG2N = NTH * PER == 4096 ? 12 : 13;
    static_assert(NTH * PER == 1 << LOG2N, "the level is a sum shifted by log2 N");
    int em = 1;
    bool nf = false;
#pragma unroll
    for (int i = 0; i < PER; ++i)
    {
        const int e = int_expo(v[i]);
        if (e == 2047)
        {
            nf = true;
            v[i] = 0;
        }
        else
            em = max(em, e);
    }
    const int emx = int_block_max<NTH>(em | (nf ? 1 << 12 : 0), ired);
    // (with a non-finite sample the largest exponent of the others is found
    // again: rare)
    *bad = (emx >> 12) != 0;
    const int emax = *bad ? int_block_max<NTH>(em, ired) : emx;
    long long s = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i)
    {
        v[i] = int_fixed(v[i], emax);
        s += v[i] >> LOG2N;
    }
    const long long lev = int_block_sum<NTH>(s, lred);  // about the mean
    int nb = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i)
    {
        v[i] -= lev;
        nb = max(nb, 64 - __clzll(v[i] < 0 ? -v[i] : v[i]));
    }
    nb = int_block_max<NTH>(nb, ired);
    int sh;
    if constexpr (NORM)
    {
        const int d = max(0, nb - 31);
        float q = 0.f;
#pragma unroll
        for (int i = 0; i < PER; ++i)
        {
            const float y = (float) (int) (v[i] >> d);
            q = fmaf(y, y, q);
        }
        q = int_block_fsum<NTH>(q, reinterpret_cast<float *>(ired));
        const float n2 = fminf(1.02f * q, L * exp2f((float) (2 * (nb - d))));
        sh = max(max(0, nb - 54), (int) ceilf(0.5f * log2f(n2) + ((float) d + 0.02f - kIntNormBits)));
    }
    else
        sh = max(0, nb - kIntXBits);
    const long long half = sh > 0 ? 1ll << (sh - 1) : 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) v[i] = (v[i] + half) >> sh;
    return emax - 1084 + sh;
}

// ---- template table -----------------------------------------------------------
// One CTA per (template, prime): B[t][prime][k] = transform of round(b 2^53),
// b the demeaned unit-norm template (FP64, as template_spectra_kernel), times
// R / N modulo p, centred.
__global__ void __launch_bounds__(256) int_bank_kernel(IntBankParams p)
{
    __shared__ double red[8];
    __shared__ int buf[kIntN];
    const int t = blockIdx.x / kIntPrimes, pi = blockIdx.x % kIntPrimes, tid = threadIdx.x;
    const IntField f(p.c.prime[pi]);
    const int L = p.tlen[t];
    int *out = p.B + ((long) t * kIntPrimes + pi) * kIntN;
    if (L > kIntN) return;  // correlated directly: in no plan
    const double *b = p.tmpl + p.toff[t];
    double s = 0;
    for (int i = tid; i < L; i += 256) s += b[i];
    const double mean = block_sum<double>(s, red) / (double) L;
    double q = 0;
    for (int i = tid; i < L; i += 256)
    {
        const double d = b[i] - mean;
        q += d * d;
    }
    const double nrm2 = block_sum<double>(q, red);
    const double inv = nrm2 > 0 ? 1.0 / sqrt(nrm2) : 0.0, scale = ldexp(1.0, kIntBBits);
    int a[16];
#pragma unroll
    for (int r = 0; r < 16; ++r)
    {
        const int j = tid + 256 * r;
        a[r] = j < L ? int_mod(f, p.c.prime[pi].c25, llrint((b[j] - mean) * inv * scale)) : 0;
    }
    int_ntt<false>(f, a, buf, p.tw + pi * kIntTw, tid, 1);
#pragma unroll
    for (int r = 0; r < 16; ++r)
    {
        int v = f.mul(a[r], p.c.prime[pi].rrn);
        v = v > f.p / 2 ? v - f.p : (v < -(f.p / 2) ? v + f.p : v);
        out[tid + 256 * r] = v;
    }
}

// ---- normalisation -----------------------------------------------------------
// sqrt(L) / sqrt(V 2^(2 ex)) for V > 0 (0 for V = 0, a constant window; sqrt(L)
// / tol where the deviation is at most tol), as DenOps<double>::out
__device__ __forceinline__ double int_inv_den(unsigned __int128 V, int ex, double sqrtL, double tol, long long tol2_bits)
{
    if (V == 0) return 0.0;
    const unsigned long long vh = (unsigned long long) (V >> 64);
    const int lz = vh ? __clzll((long long) vh) : 64 + __clzll((long long) (unsigned long long) V);
    const unsigned long long m = (unsigned long long) ((V << lz) >> 64);  // V = m 2^(64 - lz), m >= 2^63
    int E = 128 - lz + 2 * ex;  // V 2^(2 ex) = (m / 2^64) 2^E
    // its FP64 bit pattern, for the comparison with tol^2 (exponents below
    // FP64's range are below tol^2, above it above)
    const long long vb = E < -1000 ? 0 : (E > 1000 ? 0x7fe0000000000000ll : ((long long) (E + 1021) << 52) + (long long) (m >> 11));
    if (vb <= tol2_bits) return sqrtL / tol;
    // fm in [1/4, 1) with an even exponent
    unsigned long long fm = m;
    if (E & 1)
    {
        fm >>= 1;
        E += 1;
    }
    const float f0 = (float) (unsigned) (fm >> 32) * 0x1p-32f;
    // y in (1, 2]: 30 fractional bits of the FP32 value
    const unsigned y = (unsigned) (rsqrtf(f0) * 0x1p30f);
    const unsigned long long y2 = (unsigned long long) y * y;                   // 60 fractional bits
    const long long e = (1ll << 60) - (long long) __umul64hi(fm, y2);            // 1 - fm y^2, about 2^-21
    const long long es = e >> 16;                                                // 44 bits
    const long long corr = (e >> 1) + ((3 * (es * es)) >> 31);                   // e / 2 + 3 e^2 / 8, 60 bits
    const long long lo = (long long) (unsigned) corr * y, hi = (corr >> 32) * (long long) y;  // corr y, 90 bits
    const unsigned long long y60 = ((unsigned long long) y << 30) + (unsigned long long) ((hi << 2) + (long long) ((unsigned long long) lo >> 30));
    // y60 in [2^60, 2^61]: 1 / sqrt(V) = y60 2^-60 2^(-E / 2)
    const long long yb = ((long long) (1022 - (E >> 1)) << 52) + (long long) ((y60 + 128) >> 8);
    return sqrtL * __longlong_as_double(yb);
}

// One CTA per (tile of kIntTile samples, group).  MULTI false (one template
// length): the channel's row den[c][k].  MULTI true: for every template of
// the group, its own rows, written where the coefficients go (the correlator
// reads each value before it stores the coefficient in its place).
//
// The tile's prefix sums (24 bytes per sample, 196 KB of shared memory) give
// any window of any length in two loads each of S1 and S2: about 60 integer
// instructions and one FP64 product per lag, against some 27 FP64 operations
// (16 clocks per SM) of the running FP64 form.
__device__ __forceinline__ int int_pswz(int i) { return i ^ ((i >> 3) & 15); }

template <bool MULTI> __global__ void __launch_bounds__(kIntThreads, 1) int_den_kernel(IntDenParams p)
{
    extern __shared__ __align__(16) unsigned char smem_id[];
    __shared__ long long lred[32], wlo[33], whi[33], w1[33];
    __shared__ int ired[32];
    constexpr int PER = kIntTile / kIntThreads;  // consecutive samples per thread
    constexpr int NP = kIntTile + 16;            // prefixes 0 .. kIntTile, swizzled in groups of 16
    long long *P1 = reinterpret_cast<long long *>(smem_id);
    unsigned long long *PL = reinterpret_cast<unsigned long long *>(P1 + NP), *PH = PL + NP;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = blockIdx.y;
    const int c = MULTI ? p.grp_chan[g] : g;
    if (p.dead[c]) return;
    const long k0 = (long) blockIdx.x * p.lags;
    const long long *x = reinterpret_cast<const long long *>(p.x + (long) c * p.ldx);
    long long v[PER];
    const long long first = x[k0];
#pragma unroll
    for (int i = 0; i < PER; i += 2)
    {
        // rows are 16-byte aligned and hold an even count of at least n; past
        // the data the tile's first sample (as in the correlator)
        const long k = k0 + PER * tid + i;
        longlong2 d = make_longlong2(first, first);
        if (k < p.n) d = *reinterpret_cast<const longlong2 *>(x + k);
        v[i] = d.x;
        v[i + 1] = k + 1 < p.n ? d.y : first;
    }
    bool bad;
    const int ex = int_quantise<kIntThreads, PER, false>(v, ired, lred, 0.f, &bad);
    // ---- prefix sums: thread, warp, block
    long long s1 = 0;
    unsigned __int128 s2 = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i)
    {
        s1 += v[i];
        s2 += (unsigned __int128) ((__int128) v[i] * v[i]);
    }
    long long i1 = s1;
    unsigned __int128 i2 = s2;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const long long u1 = __shfl_up_sync(0xffffffffu, i1, o);
        const unsigned long long ul = __shfl_up_sync(0xffffffffu, (unsigned long long) i2, o);
        const unsigned long long uh = __shfl_up_sync(0xffffffffu, (unsigned long long) (i2 >> 64), o);
        if (lane >= o)
        {
            i1 += u1;
            i2 += ((unsigned __int128) uh << 64) | ul;
        }
    }
    if (lane == 31)
    {
        w1[w] = i1;
        wlo[w] = (long long) (unsigned long long) i2;
        whi[w] = (long long) (unsigned long long) (i2 >> 64);
    }
    __syncthreads();
    long long e1 = i1 - s1;
    unsigned __int128 e2 = i2 - s2;
    for (int u = 0; u < w; ++u)
    {
        e1 += w1[u];
        e2 += ((unsigned __int128) (unsigned long long) whi[u] << 64) | (unsigned long long) wlo[u];
    }
#pragma unroll
    for (int i = 0; i < PER; ++i)
    {
        const int k = int_pswz(PER * tid + i);
        P1[k] = e1;
        PL[k] = (unsigned long long) e2;
        PH[k] = (unsigned long long) (e2 >> 64);
        e1 += v[i];
        e2 += (unsigned __int128) ((__int128) v[i] * v[i]);
    }
    if (tid == kIntThreads - 1)
    {
        const int k = int_pswz(kIntTile);
        P1[k] = e1;
        PL[k] = (unsigned long long) e2;
        PH[k] = (unsigned long long) (e2 >> 64);
    }
    __syncthreads();
    const long long tol2 = __double_as_longlong(p.tol * p.tol);
    auto lags_of = [&](int L, long nv, double *out) {
        const double sqrtL = sqrt((double) L);
        const int n = (int) (nv - k0 < (long) p.lags ? nv - k0 : (long) p.lags);
        for (int k = tid; k < n; k += kIntThreads)
        {
            const int a = int_pswz(k), b = int_pswz(k + L);
            const long long S1 = P1[b] - P1[a];
            const unsigned __int128 S2 = (((unsigned __int128) PH[b] << 64) | PL[b]) - (((unsigned __int128) PH[a] << 64) | PL[a]);
            const unsigned __int128 V = S2 * (unsigned) L - (unsigned __int128) ((__int128) S1 * S1);
            out[k0 + k] = int_inv_den(V, ex, sqrtL, p.tol, tol2);
        }
    };
    if constexpr (MULTI)
    {
        for (int j = p.grp_tb[g]; j < p.grp_te[g]; ++j)
        {
            const int t = p.tids[j];
            lags_of(p.tlen[t], p.nvalid[t], p.rho + (long) t * p.ldr);
        }
    }
    else
        lags_of(p.L, p.nv, p.den + (long) c * p.ldd);
}

// ---- correlator --------------------------------------------------------------
// One CTA of 1024 threads per (block of S lags, template group), four teams of
// 256, one prime each: the team's transforms need no other team, and a thread
// holds 16 elements of one prime (61 registers, 32 warps per SM).  Per
// template the teams leave their residues in their exchange buffers, and all
// threads combine them, four lags each.  Shared memory: the block's four
// spectra (64 KB), four exchange buffers (64 KB), the twiddles (65 KB).
//
// Bound by the integer pipes.  160 templates of 200 .. 2,000 samples against 8
// channels x 360,000: 8.35 ms (FP64 transforms with in-block normalisation)
// -> 2.14 ms + 0.54 ms normalisation; 64 channels x 360,000 with one template
// of 500 each: 2.69 + 1.15 (den_kernel) -> 0.98 + 0.38 ms.
struct IntLayout
{
    static constexpr size_t off_red = 64;                    // after the barrier: reductions
    static constexpr size_t off_mask = off_red + 512;        // two masks of 64 chunk bits
    static constexpr size_t off_xh = 1024;
    static constexpr size_t off_buf = off_xh + sizeof(int) * kIntPrimes * kIntN;
    static constexpr size_t off_tw = off_buf + sizeof(int) * kIntPrimes * kIntN;
    static constexpr size_t bytes = off_tw + sizeof(int) * kIntPrimes * kIntTw;
};

// FP64 value of the numerator in (v0, v1, v2, v3) mixed radix times 2^e2
__device__ __forceinline__ double int_value(const IntConsts &c, int v0, int v1, int v2, int v3, int e2)
{
    const long long A = (long long) c.prime[2].p * v3 + v2;
    const unsigned long long B = (unsigned long long) ((long long) c.prime[0].p * v1 + v0);
    const __int128 V = (__int128) A * (long long) c.p01 + (__int128) B;
    const bool neg = V < 0;
    const unsigned __int128 u = neg ? (unsigned __int128) -V : (unsigned __int128) V;
    const unsigned long long uh = (unsigned long long) (u >> 64), ul = (unsigned long long) u;
    if ((uh | ul) == 0) return 0.0;
    const int lz = uh ? __clzll((long long) uh) : 64 + __clzll((long long) ul);
    const unsigned long long m = (unsigned long long) ((u << lz) >> 64);  // u = m 2^(64 - lz)
    const int E = 1150 - lz + e2;  // value = (m / 2^11) 2^(75 - lz + e2)
    unsigned long long bits = ((unsigned long long) (unsigned) (E - 1) << 52) + ((m >> 11) + ((m >> 10) & 1));
    if (E < 2) bits = 0;
    else if (E > 2045) bits = 0x7ff0000000000000ull;
    return __longlong_as_double((long long) (bits | (neg ? 1ull << 63 : 0ull)));
}

template <bool SHARED_DEN> __global__ void __launch_bounds__(kIntThreads, 1) int_xcorr_kernel(IntParams p)
{
    extern __shared__ __align__(128) unsigned char smem_ix[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem_ix);
    long long *lred = reinterpret_cast<long long *>(smem_ix + IntLayout::off_red);
    int *ired = reinterpret_cast<int *>(lred + 32);
    unsigned *Mk = reinterpret_cast<unsigned *>(smem_ix + IntLayout::off_mask);
    int *xh = reinterpret_cast<int *>(smem_ix + IntLayout::off_xh);
    int *buf = reinterpret_cast<int *>(smem_ix + IntLayout::off_buf);
    int *tws = reinterpret_cast<int *>(smem_ix + IntLayout::off_tw);
    const int tid = threadIdx.x, bx = blockIdx.x, g = blockIdx.y;
    const XcorrParams<double> &x = p.x;
    const int c = x.grp_chan[g], S = x.S;
    const long k0 = (long) bx * S;
    const int t_begin = x.grp_tb[g], t_end = x.grp_te[g];
    if (t_end <= t_begin) return;
    if (x.dead[c])
    {
        // dead trace (|min| == |max|, src/matchedFilter.cpp:886-894): rho = 0
        for (int ti = t_begin; ti < t_end; ++ti)
        {
            const int t = x.tids[ti];
            const long nv = x.nvalid[t];
            double *dst = x.rho + (long) t * x.ldr;
            for (int k = tid; k < S; k += kIntThreads)
                if (k0 + k < nv) dst[k0 + k] = 0.0;
        }
        return;
    }
    // ---- samples and twiddles
    constexpr uint32_t kSeg = sizeof(double) * kIntN, kTwBytes = sizeof(int) * kIntPrimes * kIntTw;
    if (tid < 4) Mk[tid] = 0u;
    if (tid == 0)
    {
        mbar_init(bar, 1);
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(bar, kSeg + kTwBytes);
        if (!x.test_skip_copy)
        {
            tma_load_1d(buf, x.x + (long) c * x.ldx + k0, kSeg, bar);
            tma_load_1d(tws, p.tw, kTwBytes, bar);
        }
    }
    __syncthreads();
    if (!xcorr_wait(bar, 0, x.err, x.test_skip_copy ? (1u << 12) : (1u << 24))) return;
    bool bad;
    int ex;
    {
        // samples in the first half of the exchange buffers, integers to the
        // second half, reversed: X[(N - j) mod N] at j, so that transforms of
        // one direction give the correlation
        const long long *seg = reinterpret_cast<const long long *>(buf);
        long long *xq = reinterpret_cast<long long *>(buf) + kIntN;
        constexpr int PER = kIntN / kIntThreads;
        long long v[PER];
#pragma unroll
        for (int i = 0; i < PER; ++i)
        {
            // past the data: the block's first sample instead of the zero
            // tail, which would set the scale of a signal with an offset
            const int j = tid + kIntThreads * i;
            v[i] = seg[k0 + j < p.n ? j : 0];
        }
        ex = int_quantise<kIntThreads, PER, true>(v, ired, lred, (float) p.Lmax, &bad);
#pragma unroll
        for (int i = 0; i < PER; ++i) xq[(kIntN - (tid + kIntThreads * i)) & (kIntN - 1)] = v[i];
        __syncthreads();
    }
    if (bad)
    {
        // an infinity or NaN reaches every lag of an FP64 transform's block
        for (int ti = t_begin; ti < t_end; ++ti)
        {
            const int t = x.tids[ti];
            const long nv = x.nvalid[t];
            double *dst = x.rho + (long) t * x.ldr;
            for (int k = tid; k < S; k += kIntThreads)
                if (k0 + k < nv) dst[k0 + k] = __longlong_as_double(0x7ff8000000000000ll);
        }
        return;
    }
    const int team = tid >> 8, q = tid & 255, bar_id = 1 + team;
    const IntField f(p.c.prime[team]);
    const int *tw = tws + team * kIntTw;
    int *s = buf + team * kIntN, *xt = xh + team * kIntN;
    int a[16];
    {
        const long long *xq = reinterpret_cast<const long long *>(buf) + kIntN;
        const int c25 = p.c.prime[team].c25;
#pragma unroll
        for (int r = 0; r < 16; ++r) a[r] = int_mod(f, c25, xq[q + 256 * r]);
        int_ntt<true>(f, a, s, tw, q, bar_id);
#pragma unroll
        for (int r = 0; r < 16; ++r) xt[q + 256 * r] = a[r];  // read by this thread only
    }
    const bool pk = x.pk_on != 0;
    const int e2 = ex - kIntBBits;
    int t_prev = -1;
    for (int ti = t_begin; ti < t_end; ++ti)
    {
        const int t = x.tids[ti], it = ti - t_begin;
        const int *Bt = p.B + ((long) t * kIntPrimes + team) * kIntN;
#pragma unroll
        for (int r = 0; r < 16; ++r) a[r] = f.mul(xt[q + 256 * r], __ldg(Bt + q + 256 * r));
        if (it > 0)
        {
            __syncthreads();  // residues of the previous template read, its coefficients stored
            if (pk)
            {
                pk_scan<double, kIntThreads, 2>(x, Mk + ((it - 1) & 1) * 2, t_prev, tid, bx, k0);
                if (tid < 2) Mk[(it & 1) * 2 + tid] = 0u;
            }
        }
        int_ntt<false>(f, a, s, tw, q, bar_id);
#pragma unroll
        for (int r = 0; r < 16; ++r) s[q + 256 * r] = a[r];
        __syncthreads();
        const long nv = x.nvalid[t];
        const int kmax = (int) (nv - k0 < (long) S ? nv - k0 : (long) S);
        double *dst = x.rho + (long) t * x.ldr + k0;
        const double *den = SHARED_DEN ? x.den + (long) c * x.ldd + k0 : dst;
        unsigned *mk = Mk + (it & 1) * 2;
#pragma unroll 2
        for (int k = tid; k < kmax; k += kIntThreads)
        {
            const double inv = den[k];
            // mixed-radix digits of the numerator, the last one centred
            const IntConsts &cc = p.c;
            const int p0 = cc.prime[0].p, p1 = cc.prime[1].p, p2 = cc.prime[2].p, p3 = cc.prime[3].p;
            const int n1 = cc.prime[1].nq, n2 = cc.prime[2].nq, n3 = cc.prime[3].nq;
            int v0 = mont(buf[k], cc.prime[0].one, p0, cc.prime[0].nq);
            v0 += (v0 >> 31) & p0;
            int v1 = mont(buf[kIntN + k] - v0, cc.i01, p1, n1);
            v1 += (v1 >> 31) & p1;
            int v2 = mont(mont(buf[2 * kIntN + k] - v0, cc.i02, p2, n2) - v1, cc.i12, p2, n2);
            v2 += (v2 >> 31) & p2;
            int v3 = mont(mont(mont(buf[3 * kIntN + k] - v0, cc.i03, p3, n3) - v1, cc.i13, p3, n3) - v2, cc.i23, p3, n3);
            v3 = v3 > p3 / 2 ? v3 - p3 : (v3 < -(p3 / 2) ? v3 + p3 : v3);
            const double r = clamp_rho(int_value(cc, v0, v1, v2, v3, e2) * inv);
            dst[k] = r;
            if (pk && r > x.pk_thr) atomicOr(mk + (k >> 11), 1u << ((k >> 6) & 31));
        }
        t_prev = t;
    }
    if (pk)
    {
        __syncthreads();
        pk_scan<double, kIntThreads, 2>(x, Mk + ((t_end - 1 - t_begin) & 1) * 2, t_prev, tid, bx, k0);
    }
}

}  // namespace mfgpu
