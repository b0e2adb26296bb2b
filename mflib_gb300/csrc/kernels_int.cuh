// kernels_int.cuh -- the FP64 correlator in exact integer arithmetic.
//
// GB300 executes 1.7 FP64 operations per clock and SM (measured) against 58
// 32x32 -> 64-bit integer multiply-adds and 110 integer additions, so FP64
// data are correlated without the FP64 pipe:
//
//   * A block of N = 4096 samples becomes integers X of up to 55 bits: each
//     sample's significand shifted to a common exponent (62 bits, exact for
//     samples within 2^9 of the largest), the block's mean level taken off
//     (the numerator does not depend on it, templates are zero-mean), the
//     result rounded once.  The unit is the finest at which every window's
//     2-norm stays below 2^55.1 (about 2^-53 of the largest deviation for a
//     seismogram).  Template coefficients (demeaned, unit norm) become
//     integers B = round(b 2^53).
//   * The numerators sum X[k + j] B[j] are then computed exactly: cyclic
//     correlation by number-theoretic transforms of N points modulo four
//     primes p = 1 mod 8192 just below 2^32 / 26, and the Chinese remainder
//     theorem.  |numerator| <= 2^55.1 2^53 stays below half the primes' product
//     (2^108.19) by Cauchy-Schwarz.
//   * Window variances come from prefix sums of the same X (64 bits) and X^2 (128
//     bits) of the block: V = L S2 - S1^2 is exact.  1 / sqrt(V) starts from the
//     FP32 reciprocal square root and takes one third-order step in 60-bit
//     fixed point.
//   * The Chinese remainder theorem as a sum of fractions, numerator / M = sum
//     y_i / p_i modulo 1 (M the product of the primes), in 96-bit fixed point:
//     the numerator to 2^-64 of M.
//
// The remaining errors are the two roundings of the inputs and three roundings
// to FP64 at the end.  A sample's is at most half a unit of its block, so a
// coefficient whose window has the 2-norm W about its mean, in a block whose
// loudest window has the norm A, errs by less than 2^-53 sqrt(L) A / W besides
// the roundings at the end (about 2^-56 A / W as a rule); no sample outside the
// block counts.  An FP64 transform's rounding is 2^-53 of the block's norm spread
// over its lags, and its in-block sums of squares lose (A / W)^2 2^-53 of a
// window after a loud part.  Errors against sums in 64 bits (whose own rounding
// is in them) in the workloads of perf/cases.py: 1.2e-15 (three templates of
// 1,001), 4.0e-16 (64 of 500) and 1.1e-15 (160 of 200 .. 2,000), by FP64
// transforms 1.3e-15, 6.7e-16 and 1.2e-15.
//
// Arithmetic modulo p: Montgomery products with R = 2^32 on unsigned words
// (wide multiply, low multiply, wide multiply-add; the signed forms cost two
// more instructions each), whose result is below p (1 + a / 2^32) < 2 p for any
// 32-bit a and a constant b < p.  A 16-point transform of values below 2 p,
// with multiples of p added to keep differences positive, stays below 26 p <
// 2^32 with one reduction of one value inside.
#pragma once
#include "kernels_mf.cuh"
#include "int_params.h"

namespace mfgpu {

struct IntParams
{
    XcorrParams<double> x;  // as the FFT correlator's (spectra and twiddles unused)
    const unsigned *B;      // [template][prime][kIntN]
    const unsigned *tw;     // [prime][kIntTw]
    const IntUnit *unit;    // [channel][block], by the normalisation
    long n;                 // samples per row
    IntConsts c;
};

// a b R^-1 mod p, below p (1 + a / 2^32) for b < p (nq = -p^-1 mod 2^32)
__device__ __forceinline__ unsigned mont(unsigned a, unsigned b, unsigned p, unsigned nq)
{
    const unsigned long long t = (unsigned long long) a * b;
    const unsigned m = (unsigned) t * nq;
    return (unsigned) ((t + (unsigned long long) m * p) >> 32);
}

// a w mod p for a constant w with ws = floor(w 2^32 / p): below 2 p for any
// 32-bit a.  One wide and two low multiplies where mont takes two wide and one
// low (a wide one occupies the integer multiplier twice as long).
__device__ __forceinline__ unsigned shoup(unsigned a, unsigned w, unsigned ws, unsigned p)
{
    return a * w - __umulhi(a, ws) * p;
}

// The constants of one prime.  `c` is the same for all threads of a warp: the
// fields are read from the kernel parameters where they are used.
struct IntField
{
    const IntPrime &c;
    __device__ __forceinline__ explicit IntField(const IntPrime &cc) : c(cc) {}
    __device__ __forceinline__ unsigned mul(unsigned a, unsigned b) const { return mont(a, b, c.p, c.nq); }
    template <int K> __device__ __forceinline__ unsigned root(unsigned a) const { return shoup(a, c.w[K], c.ws[K], c.p); }
    // a mod p, below 2 p
    __device__ __forceinline__ unsigned reduce(unsigned a) const { return a - __umulhi(a, c.inv) * c.p; }
};

// 4-point transform.  MB = 2: a0 below 8 p, the others below 2 p, outputs below
// 14 p (8 p if a0 is below 2 p); MB = 8: a0 below 2 p, the others below 8 p,
// outputs below 26 p.  The multiples of p are parameters of their own, so that
// the offsets are additions.
template <int MB>
__device__ __forceinline__ void int_dft4(const IntField &f, unsigned &a0, unsigned &a1, unsigned &a2, unsigned &a3)
{
    const unsigned m1 = MB == 8 ? f.c.p8 : f.c.p2, m2 = MB == 8 ? f.c.p16 : f.c.p4;
    const unsigned s0 = a0 + a2, d0 = a0 - a2 + m1, s1 = a1 + a3, d1 = f.root<4>(a1 - a3 + m1);
    a0 = s0 + s1;
    a2 = s0 - s1 + m2;
    a1 = d0 + d1;
    a3 = d0 - d1 + f.c.p2;
}

// 16-point transform with the 16th root w1; input below 2 p, output below 26 p
// (the same index scheme as dft16).  After the first four transforms every
// value is below 8 p; the products bring theirs below 2 p again, so only row
// m = 0 meets values of up to 8 p: one of its four is reduced.
__device__ __forceinline__ void int_dft16(const IntField &f, unsigned (&a)[16])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) int_dft4<2>(f, a[j], a[j + 4], a[j + 8], a[j + 12]);
    a[5] = f.root<1>(a[5]);
    a[9] = f.root<2>(a[9]);
    a[13] = f.root<3>(a[13]);
    a[6] = f.root<2>(a[6]);
    a[10] = f.root<4>(a[10]);
    a[14] = f.root<6>(a[14]);
    a[7] = f.root<3>(a[7]);
    a[11] = f.root<6>(a[11]);
    a[15] = f.root<9>(a[15]);
    a[0] = f.reduce(a[0]);
    int_dft4<8>(f, a[0], a[1], a[2], a[3]);
#pragma unroll
    for (int m = 1; m < 4; ++m) int_dft4<2>(f, a[4 * m], a[4 * m + 1], a[4 * m + 2], a[4 * m + 3]);
    unsigned t[16];
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
__device__ __forceinline__ void int_ntt(const IntField &f, unsigned (&a)[16], unsigned *s, const unsigned *tw, int q,
                                        int bar_id)
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
        a[0] = f.reduce(a[0]);
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
    a[0] = f.reduce(a[0]);
#pragma unroll
    for (int r = 1; r < 16; ++r) a[r] = f.mul(a[r], tw[240 + (r - 1) * 256 + q]);
    int_dft16(f, a);
}

// v mod p for |v| <= 2^55: v = vh 2^25 + vl, vh made positive by 8 p (below 1.8 p)
__device__ __forceinline__ unsigned int_mod(const IntField &f, unsigned c25, long long v)
{
    return f.mul((unsigned) (int) (v >> 25) + f.c.p8, c25) + ((unsigned) v & ((1u << 25) - 1));
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
    const int d = min(emax - max(e, 1), 63);
    m = ((m << 9) + ((1ull << d) >> 1)) >> d;  // (up to d = 9 the half is shifted out again)
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

// log2 of a bound on sum v^2 over any L consecutive samples, |v| <= 2^nb, sample
// 8 tid + i in v[i]: the largest sum of the runs of 32 samples that a window can
// touch, each sample's square taken above its value (12 bits).  red: 128 words.
__device__ __forceinline__ float int_window_norm(const long long (&v)[8], int nb, int L, unsigned *red)
{
    static_assert(8 * kIntDenThreads == 4096, "128 runs, four per lane");
    const int lane = threadIdx.x & 31, d = max(0, nb - 12);
    unsigned own = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
    {
        const unsigned y = (unsigned) ((v[i] < 0 ? -v[i] : v[i]) >> d) + 1u;
        own += y * y;
    }
    own += __shfl_xor_sync(0xffffffffu, own, 1);
    own += __shfl_xor_sync(0xffffffffu, own, 2);  // a run of 32: below 2^30
    __syncthreads();
    if ((lane & 3) == 0) red[threadIdx.x >> 2] = (own >> 5) + 1u;
    __syncthreads();
    uint4 r = reinterpret_cast<const uint4 *>(red)[lane];
    r.y += r.x;
    r.z += r.y;
    r.w += r.z;
    unsigned inc = r.w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const unsigned u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    const unsigned ex = inc - r.w, total = __shfl_sync(0xffffffffu, inc, 31);
    const unsigned P[5] = {ex, ex + r.x, ex + r.y, ex + r.z, inc};  // sums of the runs before 4 lane .. 4 lane + 4
    const int nc = (L + 62) / 32;                                   // runs touched
    unsigned best = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        const int to = k + nc, j = to & 3;
        const unsigned src = j == 0 ? P[0] : j == 1 ? P[1] : j == 2 ? P[2] : P[3];
        const unsigned e = __shfl_sync(0xffffffffu, src, (lane + (to >> 2)) & 31);
        best = max(best, (4 * lane + to < 128 ? e : total) - P[k]);
    }
    best = __reduce_max_sync(0xffffffffu, best);
    return fminf(log2f((float) best) + 5.f, log2f((float) L) + (float) (2 * (nb - d))) + (float) (2 * d);
}

// A block's integers, from the samples as bit patterns: what the normalisation
// finds (int_quantise) and the correlator applies again.
__device__ __forceinline__ long long int_sample(const IntUnit &u, long long fixed)
{
    const long long half = u.sh > 0 ? 1ll << (u.sh - 1) : 0;
    return (fixed - u.level + half) >> u.sh;
}
// exponent of their unit: x - level = v 2^ex up to half a unit
__device__ __forceinline__ int int_unit_exponent(const IntUnit &u) { return u.emax - 1084 + u.sh; }

// Quantises a block's samples, sample 8 tid + i in v[i]: the finest unit at which
// the 2-norm of every window of at most L samples stays below 2^kIntNormBits, at
// most 55 bits.  Infinities and NaN count as 0; nf: their bits.  lred: 64 words.
__device__ __forceinline__ IntUnit int_quantise(long long (&v)[8], int *ired, long long *lred, int L, unsigned &nf)
{
    constexpr int LOG2N = 12, NTH = kIntDenThreads;
    static_assert(kIntN == 1 << LOG2N, "the level is a sum shifted by log2 N");
    int em = 1;
    nf = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
    {
        const int e = int_expo(v[i]);
        if (e == 2047)
        {
            nf |= 1u << i;
            v[i] = 0;
        }
        else
            em = max(em, e);
    }
    const int emx = int_block_max<NTH>(em | (nf ? 1 << 12 : 0), ired);
    // (with a non-finite sample the largest exponent of the others is found
    // again: rare)
    IntUnit u;
    u.bad = emx >> 12;
    u.emax = u.bad ? int_block_max<NTH>(em, ired) : emx;
    long long s = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
    {
        v[i] = int_fixed(v[i], u.emax);
        s += v[i] >> LOG2N;
    }
    u.level = int_block_sum<NTH>(s, lred);  // about the mean
    unsigned long long any = 0;
    long long d[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
    {
        d[i] = v[i] - u.level;
        any |= (unsigned long long) (d[i] ^ (d[i] >> 63));
    }
    const int nb = int_block_max<NTH>(64 - __clzll((long long) any), ired);  // |d| <= 2^nb
    const float n2 = int_window_norm(d, nb, L, reinterpret_cast<unsigned *>(lred));
    u.sh = max(max(0, nb - 55), (int) ceilf(0.5f * n2 - kIntNormBits));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = int_sample(u, v[i]);
    return u;
}

// ---- template table -----------------------------------------------------------
// One CTA per (template, prime): B[t][prime][k] = transform of round(b 2^53),
// b the demeaned unit-norm template (FP64, as template_spectra_kernel), times
// R / N (M / p)^-1 modulo p, in [0, p).
__global__ void __launch_bounds__(256) int_bank_kernel(IntBankParams p)
{
    __shared__ double red[8];
    __shared__ unsigned buf[kIntN];
    const int t = blockIdx.x / kIntPrimes, pi = blockIdx.x % kIntPrimes, tid = threadIdx.x;
    const IntField f(p.c.prime[pi]);
    const int L = p.tlen[t];
    unsigned *out = p.B + ((long) t * kIntPrimes + pi) * kIntN;
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
    unsigned a[16];
#pragma unroll
    for (int r = 0; r < 16; ++r)
    {
        const int j = tid + 256 * r;
        a[r] = j < L ? int_mod(f, p.c.prime[pi].c25, llrint((b[j] - mean) * inv * scale)) : 0u;
    }
    int_ntt<false>(f, a, buf, p.tw + pi * kIntTw, tid, 1);
#pragma unroll
    for (int r = 0; r < 16; ++r)
    {
        const unsigned v = f.mul(a[r], p.c.prime[pi].rrn);
        out[tid + 256 * r] = min(v, v - f.c.p);
    }
}

// ---- normalisation -----------------------------------------------------------
// The smallest integer V whose V 2^(2 ex), rounded down to FP64, is above
// tol2 >= 0 (all ones: none)
__device__ __forceinline__ unsigned __int128 int_tol(double tol2, int ex)
{
    const long long b = __double_as_longlong(tol2) + 1;
    const int e = (int) (b >> 52) & 2047;
    unsigned long long m = (unsigned long long) b & ((1ull << 52) - 1);
    if (e > 0) m |= 1ull << 52;
    const int sh = max(e, 1) - 1075 - 2 * ex;  // V >= m 2^sh
    if (sh >= 75) return ~(unsigned __int128) 0;
    if (sh >= 0) return (unsigned __int128) m << sh;
    return sh <= -64 ? 1 : (unsigned __int128) ((m - 1) >> -sh) + 1;
}

// scale / sqrt(V 2^(2 ex)) for V > 0
__device__ __forceinline__ double int_inv_den(unsigned __int128 V, int ex, double scale)
{
    // V = fm 2^E, fm in [1/4, 1), E even
    unsigned w3 = (unsigned) (V >> 96), w2 = (unsigned) (V >> 64), w1 = (unsigned) (V >> 32), w0 = (unsigned) V;
    int E2 = 64 + ex;  // E / 2 + ex
    while (w3 == 0)
    {
        w3 = w2;
        w2 = w1;
        w1 = w0;
        w0 = 0;
        E2 -= 16;
    }
    const int sh = __clz((int) w3) & ~1;
    E2 -= sh >> 1;
    const unsigned fh = __funnelshift_l(w2, w3, sh), fl = __funnelshift_l(w1, w2, sh);
    const unsigned long long fm = ((unsigned long long) fh << 32) | fl;
    // y in [1, 2): FP32 reciprocal square root, 23 fractional bits (formed in
    // and taken from the bit patterns: conversions go through the slow pipe)
    const float f0 = __uint_as_float(0x3f800000u | (fh >> 9)) - 1.0f;
    const unsigned y = (__float_as_uint(fminf(rsqrtf(f0), 0x1.fffffep0f)) & 0x7fffffu) | 0x800000u;
    const unsigned long long y2 = (unsigned long long) (y << 7) * (y << 7);    // 60 fractional bits
    const long long e = (1ll << 60) - (long long) __umul64hi(fm, y2);          // 1 - fm y^2, below 2^-19
    const int es = (int) (e >> 16);                                            // 44 bits
    const long long corr = (e >> 1) + ((3 * ((long long) es * es)) >> 31);     // e / 2 + 3 e^2 / 8, 60 bits
    const unsigned long long y60 = ((unsigned long long) y << 37) + (unsigned long long) ((corr * (long long) y) >> 23);
    // y60 in [2^60, 2^61]: 1 / sqrt(V 2^(2 ex)) = y60 2^-60 2^-E2
    // (0 where that is below FP64's normal range)
    const long long yb = E2 > 1021 ? 0 : ((long long) (1022 - E2) << 52) + (long long) ((y60 + 128) >> 8);
    return scale * __longlong_as_double(yb);
}

// One CTA per (block, group), on the correlator's blocks and integers.  MULTI
// false (one template length): the channel's row den[c][k].  MULTI true: for
// every template of the group, its own rows, written where the coefficients go
// (the correlator reads each value before it stores the coefficient in its
// place).
//
// The block's prefix sums (24 bytes per sample, 98 KB: two CTAs of 512 threads
// per SM, whose loads, scans and lags overlap) give any window of any length in
// two loads each of S1 and S2: about 90 integer instructions and one FP64
// product per lag, against some 27 FP64 operations (16 clocks per SM) of the
// running FP64 form.  64 x 360,000, L = 500: 335 us; 8 x 360,000, 160 templates of
// 200 .. 2,000: 450 us; bound by the ALU pipe (65 % busy, issue 63 %) and, with
// several lengths, by the FP64 product per lag (its pipe 63 %).  The block's unit
// is found here and read by the correlator, whose own reductions for it took 80 and 60 us
// of the same cases.  Tiles and integers of its own (50 bits; tiles of 8,192
// samples above L = 1,024) took 308 and 424 us, but a loud sample outside a
// block then took digits from that block's coefficients (a sample 1e6 times the
// signal, L = 200: 3e-11, now below 1e-15).  Where a block leaves few lags they
// were cheaper, too: one template of 4,065 on each of 8 channels x 120,000, 32
// lags per block: 3.10 -> 3.57 ms (of 3,500: 242 -> 249 us; of 2,500: 131 -> 119).
__device__ __forceinline__ int int_pswz(int i) { return i ^ ((i >> 3) & 15); }
__host__ __device__ constexpr size_t int_den_bytes() { return 3 * sizeof(long long) * (size_t) (kIntN + 16); }

// sums of x and of x^2 as al^2 + 2^28 ah al + 2^54 ah^2, |x| = 2^27 ah + al <=
// 2^55, over at most 256 samples: three multiplies and no carries (al^2 sums to
// 2^62, ah al to 2^63; ah^2 to 2^63.2, as windows of two samples or more stay
// below 2^55.1); x itself modulo 2^64
struct IntSums
{
    unsigned long long s, a, b, c;
    __device__ __forceinline__ void add(long long v)
    {
        s += (unsigned long long) v;
        const unsigned long long m = v < 0 ? -v : v;
        const unsigned l = (unsigned) m & ((1u << 27) - 1), h = (unsigned) (m >> 27);
        a += (unsigned long long) l * l;
        b += (unsigned long long) h * l;
        c += (unsigned long long) h * h;
    }
    __device__ __forceinline__ void add(const IntSums &o)
    {
        s += o.s;
        a += o.a;
        b += o.b;
        c += o.c;
    }
    __device__ __forceinline__ IntSums shfl_up(int d) const
    {
        return IntSums{__shfl_up_sync(0xffffffffu, s, d), __shfl_up_sync(0xffffffffu, a, d),
                       __shfl_up_sync(0xffffffffu, b, d), __shfl_up_sync(0xffffffffu, c, d)};
    }
    __device__ __forceinline__ unsigned __int128 squares() const
    {
        return ((unsigned __int128) c << 54) + ((unsigned __int128) b << 28) + a;
    }
};

template <bool MULTI> __global__ void __launch_bounds__(kIntDenThreads, 2) int_den_kernel(IntDenParams p)
{
    extern __shared__ __align__(16) unsigned char smem_id[];
    constexpr int NTH = kIntDenThreads, PER = 8, NW = NTH / 32;  // PER consecutive samples per thread, 256 per warp
    constexpr int NP = kIntN + 16;  // prefixes 0 .. N, swizzled in groups of 16
    __shared__ __align__(16) long long lred[64];
    __shared__ unsigned long long ws[NW], wl[NW], wh[NW];  // sums up to and with each warp: x, x^2 (low, high)
    __shared__ int ired[32];
    __shared__ __align__(4) unsigned char bad_bytes[NTH];  // a bit per sample that is an infinity or NaN
    unsigned long long *P1 = reinterpret_cast<unsigned long long *>(smem_id), *PL = P1 + NP, *PH = PL + NP;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = blockIdx.y;
    const int c = MULTI ? p.grp_chan[g] : g;
    if (p.dead[c]) return;
    const long k0 = (long) blockIdx.x * p.S;
    const long long *x = reinterpret_cast<const long long *>(p.x + (long) c * p.ldx);
    long long v[PER];
    const long long first = x[k0];
#pragma unroll
    for (int i = 0; i < PER; i += 2)
    {
        // rows are 16-byte aligned and hold an even count of at least n; past
        // the data the block's first sample (as in the correlator)
        const long k = k0 + PER * tid + i;
        longlong2 d = make_longlong2(first, first);
        if (k < p.n) d = *reinterpret_cast<const longlong2 *>(x + k);
        v[i] = d.x;
        v[i + 1] = k + 1 < p.n ? d.y : first;
    }
    unsigned nf;
    const IntUnit unit = int_quantise(v, ired, lred, p.Lmax, nf);
    const int ex = int_unit_exponent(unit);
    if (unit.bad) bad_bytes[tid] = (unsigned char) nf;
    // (the groups of a channel write the same)
    if (tid == 0) p.unit[(long) c * gridDim.x + blockIdx.x] = unit;
    // ---- prefix sums: thread, warp, block
    IntSums inc{0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < PER; ++i) inc.add(v[i]);
    // (the products are formed again below: 24 of them would not stay in registers)
#pragma unroll
    for (int i = 0; i < PER; ++i) asm volatile("" : "+l"(v[i]));
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const IntSums u = inc.shfl_up(o);
        if (lane >= o) inc.add(u);
    }
    if (lane == 31)
    {
        const unsigned __int128 q = inc.squares();
        ws[w] = inc.s;
        wl[w] = (unsigned long long) q;
        wh[w] = (unsigned long long) (q >> 64);
    }
    __syncthreads();
    if (w == 0)
    {
        unsigned long long s1 = lane < NW ? ws[lane] : 0;
        unsigned __int128 s2 = lane < NW ? ((unsigned __int128) wh[lane] << 64) | wl[lane] : 0;
#pragma unroll
        for (int o = 1; o < NW; o <<= 1)
        {
            const unsigned long long u1 = __shfl_up_sync(0xffffffffu, s1, o);
            const unsigned long long ul = __shfl_up_sync(0xffffffffu, (unsigned long long) s2, o);
            const unsigned long long uh = __shfl_up_sync(0xffffffffu, (unsigned long long) (s2 >> 64), o);
            if (lane >= o)
            {
                s1 += u1;
                s2 += ((unsigned __int128) uh << 64) | ul;
            }
        }
        if (lane < NW)
        {
            ws[lane] = s1;
            wl[lane] = (unsigned long long) s2;
            wh[lane] = (unsigned long long) (s2 >> 64);
        }
    }
    __syncthreads();
    IntSums ex_ = inc.shfl_up(1);
    if (lane == 0) ex_ = IntSums{0, 0, 0, 0};
    const unsigned long long s0 = w > 0 ? ws[w - 1] : 0;
    const unsigned __int128 q0 = w > 0 ? ((unsigned __int128) wh[w - 1] << 64) | wl[w - 1] : 0;
    auto put = [&](int at) {
        const unsigned __int128 q = q0 + ex_.squares();
        const int k = int_pswz(at);
        P1[k] = s0 + ex_.s;
        PL[k] = (unsigned long long) q;
        PH[k] = (unsigned long long) (q >> 64);
    };
#pragma unroll
    for (int i = 0; i < PER; ++i)
    {
        put(PER * tid + i);
        ex_.add(v[i]);
    }
    if (tid == NTH - 1) put(kIntN);
    __syncthreads();
    const unsigned __int128 vtol = int_tol(p.tol * p.tol, ex);
    // sqrtL: sqrt(L) times the factor of the correlator's numerators
    auto lags_of = [&](int L, long nv, double *out, double sqrtL) {
        const int n = (int) (nv - k0 < (long) p.S ? nv - k0 : (long) p.S);
        for (int k = tid; k < n; k += NTH)
        {
            const int a = int_pswz(k), b = int_pswz(k + L);
            const long long S1 = (long long) (P1[b] - P1[a]);  // below 2^61.1 by the window's norm
            const unsigned long long u = S1 < 0 ? 0ull - (unsigned long long) S1 : (unsigned long long) S1;
            const unsigned __int128 S2 = (((unsigned __int128) PH[b] << 64) | PL[b]) - (((unsigned __int128) PH[a] << 64) | PL[a]);
            const unsigned __int128 V = S2 * (unsigned) L - (unsigned __int128) u * u;
            // 0 for a constant window, sqrt(L) / tol where the deviation is
            // at most tol, as DenOps<double>::out
            out[k0 + k] = V < vtol ? (V == 0 ? 0.0 : sqrtL / p.tol) : int_inv_den(V, ex, sqrtL);
        }
        if (unit.bad)
        {
            // a window that holds an infinity or NaN has no coefficient (rare:
            // each lag scans its window's words)
            const unsigned *bits = reinterpret_cast<const unsigned *>(bad_bytes);
            for (int k = tid; k < n; k += NTH)
            {
                const int a = k >> 5, b = (k + L - 1) >> 5;
                unsigned any = 0;
                for (int j = a; j <= b; ++j)
                    any |= bits[j] & (j == a ? ~0u << (k & 31) : ~0u) & (j == b ? ~0u >> (31 - ((k + L - 1) & 31)) : ~0u);
                if (any) out[k0 + k] = __longlong_as_double(0x7ff8000000000000ll);
            }
        }
    };
    if constexpr (MULTI)
    {
        // square roots of up to 64 templates at a time: by every thread they
        // would cost more (FP64 pipe) than a template's lags
        __shared__ double rootL[64];
        for (int j0 = p.grp_tb[g], je = p.grp_te[g]; j0 < je; j0 += 64)
        {
            const int m = min(64, je - j0);
            __syncthreads();
            if (tid < m) rootL[tid] = sqrt((double) p.tlen[p.tids[j0 + tid]]) * p.scale;
            __syncthreads();
            for (int j = 0; j < m; ++j)
            {
                const int t = p.tids[j0 + j];
                lags_of(p.tlen[t], p.nvalid[t], p.rho + (long) t * p.ldr, rootL[j]);
            }
        }
    }
    else
        lags_of(p.L, p.nv, p.den + (long) c * p.ldd, p.scale);
}

// ---- correlator --------------------------------------------------------------
// One CTA of 1024 threads per (block of S lags, template group), four teams of
// 256, one prime each: the team's transforms need no other team, and a thread
// holds 16 elements of one prime (61 registers, 32 warps per SM).  Per
// template the teams leave their residues in their exchange buffers, and all
// threads combine them, four lags each.  Shared memory: the block's four
// spectra (64 KB), four exchange buffers (64 KB), the twiddles (65 KB).
//
// Bound by the multiplier (the largest stall is its throttle), then barriers and
// spectra from L2; issue 2.0 of 4 per clock.  160
// templates of 200 .. 2,000 samples against 8 channels x 360,000: 8.35 ms (FP64
// transforms with in-block normalisation) -> 1.65 ms + 0.45 ms normalisation;
// 64 channels x 360,000 with one template of 500 each: 2.69 + 1.15 (den_kernel)
// -> 0.76 + 0.33 ms.  Signed words with centred residues took 2.14 and 0.98 ms.
struct IntLayout
{
    static constexpr size_t off_mask = 64;                   // after the barrier: two masks of 64 chunk bits
    static constexpr size_t off_xh = 128;
    static constexpr size_t off_buf = off_xh + sizeof(int) * kIntPrimes * kIntN;
    static constexpr size_t off_tw = off_buf + sizeof(int) * kIntPrimes * kIntN;
    static constexpr size_t bytes = off_tw + sizeof(int) * kIntPrimes * kIntTw;
};

// numerator / M as a signed 64-bit fraction: sum of y_i / p_i modulo 1 with
// 1 / p_i to 96 bits, from r_i = y_i mod p_i (any 32 bits), y_i the numerator
// times (M / p_i)^-1, a factor that the template table carries
__device__ __forceinline__ long long int_fraction(const IntConsts &c, const unsigned (&r)[kIntPrimes])
{
    unsigned long long t0 = 1ull << 31, t1 = 0;  // rounds to nearest: a numerator of 0 stays 0
    unsigned t2 = 0;
#pragma unroll
    for (int i = 0; i < kIntPrimes; ++i)
    {
        const unsigned y = r[i] - __umulhi(r[i], c.prime[i].inv) * c.prime[i].p;  // below 2 p
        t0 += (unsigned long long) y * c.prime[i].f0;
        t1 += (unsigned long long) y * c.prime[i].f1;
        t2 += y * c.prime[i].f2;
    }
    t1 += t0 >> 32;
    t2 += (unsigned) (t1 >> 32);
    return (long long) (((unsigned long long) t2 << 32) | (unsigned) t1);
}

// v 2^e as FP64, rounded to nearest (0 below, infinity above its range)
__device__ __forceinline__ double int_to_double(long long v, int e)
{
    if (v == 0) return 0.0;
    const unsigned long long u = v < 0 ? 0ull - (unsigned long long) v : (unsigned long long) v;
    const int lz = __clzll((long long) u);
    const unsigned long long m = u << lz;
    const int E = 1086 - lz + e;  // value = (m / 2^11) 2^(11 - lz + e)
    unsigned long long bits = ((unsigned long long) (unsigned) (E - 1) << 52) + ((m >> 11) + ((m >> 10) & 1));
    if (E < 2) bits = 0;
    else if (E > 2045) bits = 0x7ff0000000000000ull;
    return __longlong_as_double((long long) (bits | ((unsigned long long) v & (1ull << 63))));
}

// clamp_rho and v > thr >= 0 on the bit patterns (a comparison in FP64 costs
// 19 clocks per warp and SM, as much as the product before it)
__device__ __forceinline__ long long int_clamp(long long v)
{
    constexpr long long inf = 0x7ff0000000000000ll, lim = 0x3ff199999999999all;  // 1.1
    const long long m = v & 0x7fffffffffffffffll;
    return m > lim && m <= inf ? 0 : v;  // a NaN stays
}
__device__ __forceinline__ bool int_above(long long v, long long thr) { return v > thr && v <= 0x7ff0000000000000ll; }

template <bool SHARED_DEN> __global__ void __launch_bounds__(kIntThreads, 1) int_xcorr_kernel(IntParams p)
{
    extern __shared__ __align__(128) unsigned char smem_ix[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem_ix);
    unsigned *Mk = reinterpret_cast<unsigned *>(smem_ix + IntLayout::off_mask);
    unsigned *xh = reinterpret_cast<unsigned *>(smem_ix + IntLayout::off_xh);
    unsigned *buf = reinterpret_cast<unsigned *>(smem_ix + IntLayout::off_buf);
    unsigned *tws = reinterpret_cast<unsigned *>(smem_ix + IntLayout::off_tw);
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
    const IntUnit unit = p.unit[(long) c * gridDim.x + bx];
    if (!xcorr_wait(bar, 0, x.err, x.test_skip_copy ? (1u << 12) : (1u << 24))) return;
    const int ex = int_unit_exponent(unit);
    {
        // samples in the first half of the exchange buffers, integers to the
        // second half, reversed: X[(N - j) mod N] at j, so that transforms of
        // one direction give the correlation
        const long long *seg = reinterpret_cast<const long long *>(buf);
        long long *xq = reinterpret_cast<long long *>(buf) + kIntN;
#pragma unroll
        for (int i = 0; i < kIntN / kIntThreads; ++i)
        {
            // past the data: the block's first sample instead of the zero
            // tail, which would set the scale of a signal with an offset
            const int j = tid + kIntThreads * i;
            long long b = seg[k0 + j < p.n ? j : 0];
            if (unit.bad && int_expo(b) == 2047) b = 0;
            xq[(kIntN - j) & (kIntN - 1)] = int_sample(unit, int_fixed(b, unit.emax));
        }
        __syncthreads();
    }
    // (the same for the warp, and known to be: the constants stay uniform)
    const int team = __shfl_sync(0xffffffffu, tid >> 8, 0), q = tid & 255, bar_id = 1 + team;
    const IntField f(p.c.prime[team]);
    const unsigned *tw = tws + team * kIntTw;
    unsigned *s = buf + team * kIntN, *xt = xh + team * kIntN;
    unsigned a[16];
    {
        const long long *xq = reinterpret_cast<const long long *>(buf) + kIntN;
        const unsigned c25 = p.c.prime[team].c25;
#pragma unroll
        for (int r = 0; r < 16; ++r) a[r] = int_mod(f, c25, xq[q + 256 * r]);
        int_ntt<true>(f, a, s, tw, q, bar_id);
#pragma unroll
        for (int r = 0; r < 16; ++r) xt[q + 256 * r] = a[r];  // read by this thread only
    }
    const bool pk = x.pk_on != 0;
    const long long thr = __double_as_longlong(x.pk_thr + 0.0);  // (not -0)
    int t_prev = -1;
    for (int ti = t_begin; ti < t_end; ++ti)
    {
        const int t = x.tids[ti], it = ti - t_begin;
        const unsigned *Bt = p.B + ((long) t * kIntPrimes + team) * kIntN;
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
        const long nv = x.nvalid[t];
        const int kmax = (int) (nv - k0 < (long) S ? nv - k0 : (long) S);
        double *dst = x.rho + (long) t * x.ldr + k0;
        const double *den = SHARED_DEN ? x.den + (long) c * x.ldd + k0 : dst;
        unsigned *mk = Mk + (it & 1) * 2;
        __syncthreads();
#pragma unroll 2
        for (int k = tid; k < kmax; k += kIntThreads)
        {
            const double inv = den[k];
            const unsigned rs[kIntPrimes] = {buf[k], buf[kIntN + k], buf[2 * kIntN + k], buf[3 * kIntN + k]};
            // (the factor M / 2^64 2^-53 is in the normalisation)
            const long long r = int_clamp(__double_as_longlong(int_to_double(int_fraction(p.c, rs), ex) * inv));
            dst[k] = __longlong_as_double(r);
            if (pk && int_above(r, thr)) atomicOr(mk + (k >> 11), 1u << ((k >> 6) & 31));
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
