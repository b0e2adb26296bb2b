// int_params.h -- constants and parameters of the integer FP64 correlator
// (kernels_int.cuh), shared by the host code that fills them.
#pragma once

namespace mfgpu {

constexpr int kIntN = 4096;       // transform length: the samples of a block
constexpr int kIntPrimes = 4;
constexpr int kIntThreads = 1024;
constexpr int kIntTw = 240 + 3840;  // twiddles per prime: rows r = 1 .. 15 of the second and third pass
constexpr int kIntDenThreads = 512;
constexpr int kIntBBits = 53;     // fraction bits of a template coefficient
constexpr float kIntNormBits = 55.1f;  // a block's windows: 2-norm below 2^55.1, so that a numerator stays below
                                       // 2^108.1 and half the primes' product (2^108.19)
// the window length that bounds a block's unit: of the longest template, at
// least 2 (the sums of squares of 256 samples, IntSums)
constexpr int int_norm_length(int Lmax) { return Lmax < 2 ? 2 : Lmax; }

// One prime: c25 and rrn are times R = 2^32 modulo p; all in [0, p).
struct IntPrime
{
    unsigned p, nq;                 // nq = -p^-1 mod 2^32
    unsigned p2, p4, p8, p16;       // multiples of p
    unsigned inv;                   // floor(2^32 / p)
    unsigned w[10], ws[10];         // powers of the 16th root, floor(w 2^32 / p)
    unsigned c25;                   // 2^25
    unsigned rrn;                   // R / N (M / p)^-1, M the product of the primes (a product with it gives a
                                    // value times that)
    unsigned f0, f1, f2;            // floor(2^96 / p), low word first
};
struct IntConsts
{
    IntPrime prime[kIntPrimes];
};

struct IntBankParams
{
    const double *tmpl;
    const long *toff;
    const int *tlen;
    unsigned *B;                    // [template][prime][kIntN]
    const unsigned *tw;             // [prime][kIntTw]
    IntConsts c;
};

// A block's integers: v = (f - level) 2^-sh, f the sample in units of 2^(emax -
// 1084).  bad: the block holds an infinity or NaN, which count as f = 0 (the
// windows that hold one are marked in the normalisation)
struct IntUnit
{
    long long level;
    int emax, sh;
    int bad;
};

struct IntDenParams
{
    const double *x;
    long ldx;
    long n;                         // samples per row
    const unsigned char *dead;
    double tol;
    double scale;                   // factor of the correlator's numerators (int_numerator_scale);
                                    // one length: times sqrt(L)
    int S;                          // lags per block, as the correlator's
    int Lmax;                       // int_norm_length of the longest template
    IntUnit *unit;                  // [channel][block]
    // one length: L, valid lags, rows den
    int L;
    long nv;
    double *den;
    long ldd;
    // several lengths: the groups' templates, rows rho
    const int *grp_chan, *grp_tb, *grp_te, *tids, *tlen, *nvalid;
    double *rho;
    long ldr;
};

}  // namespace mfgpu
