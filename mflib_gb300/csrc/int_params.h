// int_params.h -- constants and parameters of the integer FP64 correlator
// (kernels_int.cuh), shared by the host code that fills them.
#pragma once

namespace mfgpu {

constexpr int kIntN = 4096;       // transform length: the samples of a block
constexpr int kIntPrimes = 4;
constexpr int kIntThreads = 1024;
constexpr int kIntTw = 240 + 3840;  // twiddles per prime: rows r = 1 .. 15 of the second and third pass
constexpr int kIntTile = 8192;    // samples of a normalisation tile
constexpr int kIntXBits = 50;     // bits of a quantised sample of a normalisation tile
constexpr int kIntBBits = 53;     // fraction bits of a template coefficient
constexpr float kIntNormBits = 54.6f;  // a block's windows: 2-norm below 2^54.6, so that a numerator stays below
                                       // 2^107.6 and half the primes' product (2^107.7)

// One prime: everything but p and nq is times R = 2^32 modulo p, centred.
struct IntPrime
{
    int p, nq;                      // nq = -p^-1 mod 2^32
    int one;                        // 1
    int w1, w2, w3, w4, w6, w9;     // powers of the 16th root
    int c25;                        // 2^25
    int rrn;                        // R / N (so that a product with it gives a value times R / N)
};
struct IntConsts
{
    IntPrime prime[kIntPrimes];
    int i01, i02, i12, i03, i13, i23;  // inverse of prime a modulo prime b, times R
    unsigned long long p01;            // product of the first two primes
};

struct IntBankParams
{
    const double *tmpl;
    const long *toff;
    const int *tlen;
    int *B;                         // [template][prime][kIntN]
    const int *tw;                  // [prime][kIntTw]
    IntConsts c;
};

struct IntDenParams
{
    const double *x;
    long ldx;
    long n;                         // samples per row
    const unsigned char *dead;
    double tol;
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
