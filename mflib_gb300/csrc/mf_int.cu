// mf_int.cu -- tables and launchers of the integer FP64 correlator
// (kernels_int.cuh).
#include <cmath>
#include "launch.h"
#include "kernels_int.cuh"

namespace mfgpu {

namespace {

uint64_t pow_mod(uint64_t b, uint64_t e, uint64_t p)
{
    uint64_t r = 1;
    for (b %= p; e; e >>= 1, b = b * b % p)
        if (e & 1) r = r * b % p;
    return r;
}

bool is_prime(uint32_t n)
{
    for (uint32_t d = 2; (uint64_t) d * d <= n; ++d)
        if (n % d == 0) return false;
    return true;
}

// v times 2^32 modulo p
unsigned mont_of(uint64_t v, uint32_t p) { return (unsigned) ((v % p) * ((1ull << 32) % p) % p); }

struct Tables
{
    IntConsts c;
    std::vector<unsigned> tw;
    double scale;
    Tables() : tw((size_t) kIntPrimes * kIntTw)
    {
        // the largest primes = 1 mod 8192 below 2^32 / 26 (int_dft16)
        uint32_t cand = (uint32_t) ((1ull << 32) / 26) / 8192 * 8192 + 1;
        if (cand > (1ull << 32) / 26) cand -= 8192;
        uint64_t pr[kIntPrimes];
        double M = 1.0;
        for (int i = 0; i < kIntPrimes; ++i, cand -= 8192)
        {
            while (!is_prime(cand)) cand -= 8192;
            const uint32_t p = cand;
            pr[i] = p;
            M *= p;
            // a root of order N: g^((p-1)/N) with its N/2-th power = -1
            uint64_t w = 0;
            for (uint64_t g = 2; !w; ++g)
            {
                const uint64_t r = pow_mod(g, (p - 1) / kIntN, p);
                if (pow_mod(r, kIntN / 2, p) == p - 1) w = r;
            }
            IntPrime &q = c.prime[i];
            q.p = p;
            uint32_t inv = 1;  // p^-1 modulo 2^32 by Newton's iteration
            for (int k = 0; k < 6; ++k) inv *= 2u - p * inv;
            q.nq = 0u - inv;
            q.p2 = 2 * p;
            q.p4 = 4 * p;
            q.p8 = 8 * p;
            q.p16 = 16 * p;
            q.inv = (unsigned) ((1ull << 32) / p);
            const uint64_t w16 = pow_mod(w, kIntN / 16, p);
            for (int k = 0; k < 10; ++k)
            {
                const uint64_t v = pow_mod(w16, k, p);
                q.w[k] = (unsigned) v;
                q.ws[k] = (unsigned) ((v << 32) / p);
            }
            q.c25 = mont_of(1ull << 25, p);
            const uint64_t R = (1ull << 32) % p;
            q.rrn = mont_of(R * pow_mod(kIntN, p - 2, p) % p, p);
            unsigned __int128 f = ((unsigned __int128) 1 << 96) / p;
            q.f0 = (unsigned) f;
            q.f1 = (unsigned) (f >> 32);
            q.f2 = (unsigned) (f >> 64);
            unsigned *t = &tw[(size_t) i * kIntTw];
            const uint64_t w256 = pow_mod(w, kIntN / 256, p);
            for (int r = 1; r < 16; ++r)
            {
                for (int k = 0; k < 16; ++k) t[(r - 1) * 16 + k] = mont_of(pow_mod(w256, (uint64_t) r * k, p), p);
                uint64_t v = 1;
                const uint64_t wr = pow_mod(w, r, p);
                for (int k = 0; k < 256; ++k, v = v * wr % p) t[240 + (r - 1) * 256 + k] = mont_of(v, p);
            }
        }
        for (int i = 0; i < kIntPrimes; ++i)
        {
            uint64_t m = 1;
            for (int k = 0; k < kIntPrimes; ++k)
                if (k != i) m = m * (pr[k] % pr[i]) % pr[i];
            c.prime[i].rrn = (unsigned) (c.prime[i].rrn * pow_mod(m, pr[i] - 2, pr[i]) % pr[i]);
        }
        scale = std::ldexp(M, -64 - kIntBBits);
    }
};

const Tables &tables()
{
    static const Tables t;
    return t;
}

}  // namespace

const std::vector<unsigned> &int_twiddles() { return tables().tw; }
double int_numerator_scale() { return tables().scale; }

cudaError_t launch_int_bank(const double *tmpl, const long *toff, const int *tlen, int nt, const unsigned *tw, unsigned *B,
                            cudaStream_t s)
{
    IntBankParams p{tmpl, toff, tlen, B, tw, tables().c};
    int_bank_kernel<<<nt * kIntPrimes, 256, 0, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_int_den(const IntDenParams &p, bool multi, int nblocks, int ngroups, cudaStream_t s)
{
    static SmemCap caps, capm;
    cudaError_t e = multi ? raise_smem_cap(int_den_kernel<true>, int_den_bytes(), capm)
                          : raise_smem_cap(int_den_kernel<false>, int_den_bytes(), caps);
    if (e != cudaSuccess) return e;
    if (multi) int_den_kernel<true><<<dim3(nblocks, ngroups), kIntDenThreads, int_den_bytes(), s>>>(p);
    else int_den_kernel<false><<<dim3(nblocks, ngroups), kIntDenThreads, int_den_bytes(), s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_int_xcorr(const XcorrParams<double> &x, bool shared_den, const unsigned *B, const unsigned *tw,
                             const IntUnit *unit, long n, int nblocks, int ngroups, cudaStream_t s)
{
    IntParams p{x, B, tw, unit, n, tables().c};
    static SmemCap caps, capm;
    cudaError_t e = shared_den ? raise_smem_cap(int_xcorr_kernel<true>, IntLayout::bytes, caps)
                               : raise_smem_cap(int_xcorr_kernel<false>, IntLayout::bytes, capm);
    if (e != cudaSuccess) return e;
    if (shared_den) int_xcorr_kernel<true><<<dim3(nblocks, ngroups), kIntThreads, IntLayout::bytes, s>>>(p);
    else int_xcorr_kernel<false><<<dim3(nblocks, ngroups), kIntThreads, IntLayout::bytes, s>>>(p);
    return cudaGetLastError();
}

}  // namespace mfgpu
