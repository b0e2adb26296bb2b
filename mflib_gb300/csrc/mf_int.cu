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

// v times 2^32 modulo p, in (-p/2, p/2)
int mont_of(uint64_t v, uint32_t p)
{
    const uint64_t r = (v % p) * ((1ull << 32) % p) % p;
    return r > p / 2 ? (int) ((long long) r - (long long) p) : (int) r;
}

struct Tables
{
    IntConsts c;
    std::vector<int> tw;
    Tables() : tw((size_t) kIntPrimes * kIntTw)
    {
        // the largest primes = 1 mod 8192 below 2^31 / 14
        uint32_t cand = ((uint32_t) ((1ull << 31) / 14) - 1) / 8192 * 8192 + 1;
        uint64_t pr[kIntPrimes];
        for (int i = 0; i < kIntPrimes; ++i, cand -= 8192)
        {
            while (!is_prime(cand)) cand -= 8192;
            const uint32_t p = cand;
            pr[i] = p;
            // a root of order N: g^((p-1)/N) with its N/2-th power = -1
            uint64_t w = 0;
            for (uint64_t g = 2; !w; ++g)
            {
                const uint64_t r = pow_mod(g, (p - 1) / kIntN, p);
                if (pow_mod(r, kIntN / 2, p) == p - 1) w = r;
            }
            IntPrime &q = c.prime[i];
            q.p = (int) p;
            uint32_t inv = 1;  // p^-1 modulo 2^32 by Newton's iteration
            for (int k = 0; k < 6; ++k) inv *= 2u - p * inv;
            q.nq = (int) (0u - inv);
            q.one = mont_of(1, p);
            const uint64_t w16 = pow_mod(w, kIntN / 16, p);
            q.w1 = mont_of(w16, p);
            q.w2 = mont_of(pow_mod(w16, 2, p), p);
            q.w3 = mont_of(pow_mod(w16, 3, p), p);
            q.w4 = mont_of(pow_mod(w16, 4, p), p);
            q.w6 = mont_of(pow_mod(w16, 6, p), p);
            q.w9 = mont_of(pow_mod(w16, 9, p), p);
            q.c25 = mont_of(1ull << 25, p);
            const uint64_t R = (1ull << 32) % p;
            q.rrn = mont_of(R * pow_mod(kIntN, p - 2, p) % p, p);
            int *t = &tw[(size_t) i * kIntTw];
            const uint64_t w256 = pow_mod(w, kIntN / 256, p);
            for (int r = 1; r < 16; ++r)
            {
                for (int k = 0; k < 16; ++k) t[(r - 1) * 16 + k] = mont_of(pow_mod(w256, (uint64_t) r * k, p), p);
                uint64_t v = 1;
                const uint64_t wr = pow_mod(w, r, p);
                for (int k = 0; k < 256; ++k, v = v * wr % p) t[240 + (r - 1) * 256 + k] = mont_of(v, p);
            }
        }
        auto inv_of = [&](int a, int b) { return mont_of(pow_mod(pr[a], pr[b] - 2, pr[b]), (uint32_t) pr[b]); };
        c.i01 = inv_of(0, 1);
        c.i02 = inv_of(0, 2);
        c.i12 = inv_of(1, 2);
        c.i03 = inv_of(0, 3);
        c.i13 = inv_of(1, 3);
        c.i23 = inv_of(2, 3);
        c.p01 = pr[0] * pr[1];
    }
};

const Tables &tables()
{
    static const Tables t;
    return t;
}

}  // namespace

const std::vector<int> &int_twiddles() { return tables().tw; }

cudaError_t launch_int_bank(const double *tmpl, const long *toff, const int *tlen, int nt, const int *tw, int *B,
                            cudaStream_t s)
{
    IntBankParams p{tmpl, toff, tlen, B, tw, tables().c};
    int_bank_kernel<<<nt * kIntPrimes, 256, 0, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_int_den(const IntDenParams &p, bool multi, int ntiles, int ngroups, cudaStream_t s)
{
    const size_t bytes = 3 * sizeof(long long) * (kIntTile + 16);
    static SmemCap cap1, capm;
    cudaError_t e = multi ? raise_smem_cap(int_den_kernel<true>, bytes, capm) : raise_smem_cap(int_den_kernel<false>, bytes, cap1);
    if (e != cudaSuccess) return e;
    if (multi) int_den_kernel<true><<<dim3(ntiles, ngroups), kIntThreads, bytes, s>>>(p);
    else int_den_kernel<false><<<dim3(ntiles, ngroups), kIntThreads, bytes, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_int_xcorr(const XcorrParams<double> &x, bool shared_den, const int *B, const int *tw, int Lmax, long n,
                             int nblocks, int ngroups, cudaStream_t s)
{
    IntParams p{x, B, tw, Lmax, n, tables().c};
    static SmemCap caps, capm;
    cudaError_t e = shared_den ? raise_smem_cap(int_xcorr_kernel<true>, IntLayout::bytes, caps)
                               : raise_smem_cap(int_xcorr_kernel<false>, IntLayout::bytes, capm);
    if (e != cudaSuccess) return e;
    if (shared_den) int_xcorr_kernel<true><<<dim3(nblocks, ngroups), kIntThreads, IntLayout::bytes, s>>>(p);
    else int_xcorr_kernel<false><<<dim3(nblocks, ngroups), kIntThreads, IntLayout::bytes, s>>>(p);
    return cudaGetLastError();
}

}  // namespace mfgpu
