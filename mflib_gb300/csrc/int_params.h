// int_params.h -- constants and parameters of the integer FP64 correlator
// (kernels_int.cuh), shared by the host code that fills them.
#pragma once

namespace mfgpu {

constexpr int kIntN = 4096;       // transform length: the samples of a block
constexpr int kIntPrimes = 4;
constexpr int kIntThreads = 1024;
constexpr int kIntTw = 240 + 3840;  // twiddles per prime: rows r = 1 .. 15 of the second and third pass
// samples of a normalisation tile for templates of up to L samples
constexpr int int_tile(int L) { return L <= 1024 ? 4096 : 8192; }
constexpr int kIntXBits = 50;     // bits of a quantised sample of a normalisation tile
constexpr int kIntBBits = 53;     // fraction bits of a template coefficient
constexpr float kIntNormBits = 55.1f;  // a block's windows: 2-norm below 2^55.1, so that a numerator stays below
                                       // 2^108.1 and half the primes' product (2^108.19)

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

struct IntDenParams
{
    const double *x;
    long ldx;
    long n;                         // samples per row
    const unsigned char *dead;
    double tol;
    double scale;                   // factor of the correlator's numerators (int_numerator_scale);
                                    // one length: times sqrt(L)
    int lags;                       // lags per tile
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
