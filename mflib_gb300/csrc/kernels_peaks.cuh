// kernels_peaks.cuh -- peak finder (PeakFinder<T>::apply, src/peakFinder.cpp:329-446)
// over many traces at once.
//
// Candidates follow the reference's sign-of-difference rules
// (:345-381): i = 0 if sign(x[1]-x[0]) < 0; 0 < i < n-1 if
// sign(x[i]-x[i-1]) >= 0 and sign(x[i+1]-x[i]) < 0 (right end of a
// plateau); i = n-1 if sign(x[n-1]-x[n-2]) > 0; always x[i] > threshold.
//
// Minimum-separation pruning (:396-433) is a greedy pass in value order.
// Here it runs as rounds over all traces in parallel: an undecided
// candidate is accepted when no undecided candidate within min_distance
// has a higher priority (value descending, then index ascending), and the
// undecided candidates within min_distance of an accepted one are
// rejected.  By induction on priority this accepts exactly the candidates
// the sequential greedy pass accepts under the same total order.
//
// The packed candidate arrays have a host-chosen capacity `cap`; kernels
// read the true count from device memory and never index past `cap`.  A
// count above `cap` raises the overflow flag and the host reruns with a
// larger capacity, so the common path needs a single synchronisation.
#pragma once
#include <cstdint>
#include "kernels_util.cuh"

namespace mfgpu {

constexpr int kPkThreads = 256;
constexpr int kPkPer = 16;                          // lags per thread
constexpr int kPkChunk = kPkThreads * kPkPer;       // lags per CTA

template <class T> struct PeakTraces
{
    const T *x;       // trace i starts at x + row[i] * ldx
    long ldx;
    const int *row;   // row of each trace
    int len;          // lags per trace
    T thr;
    // optional: bit c of row r (word r * fwords + c / 32) set when a lag in
    // [64c, 64c + 64) of that row exceeds thr; a warp whose 512 lags have no
    // bit set finds no candidate and skips its reads
    const unsigned *flags = nullptr;
    int fwords = 0;
};

template <class T> __device__ __forceinline__ bool is_candidate(const T *x, int i, int n, T thr)
{
    if (i >= n) return false;
    T xi = x[i];
    if (!(xi > thr)) return false;
    if (n == 1) return xi > (T) 0;  // reference reads x[1] out of bounds; 0 assumed
    if (i == 0) return sgn<T>(x[1] - x[0]) < 0;
    if (i == n - 1) return sgn<T>(x[n - 1] - x[n - 2]) > 0;
    return sgn<T>(xi - x[i - 1]) >= 0 && sgn<T>(x[i + 1] - xi) < 0;
}

template <class T> struct vec16;
template <> struct vec16<float>
{
    static __device__ __forceinline__ void load(const float *p, float *v)
    {
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            float4 a = reinterpret_cast<const float4 *>(p)[i];
            v[4 * i] = a.x; v[4 * i + 1] = a.y; v[4 * i + 2] = a.z; v[4 * i + 3] = a.w;
        }
    }
};
template <> struct vec16<double>
{
    static __device__ __forceinline__ void load(const double *p, double *v)
    {
#pragma unroll
        for (int i = 0; i < 8; ++i)
        {
            double2 a = reinterpret_cast<const double2 *>(p)[i];
            v[2 * i] = a.x; v[2 * i + 1] = a.y;
        }
    }
};

// Candidate mask of the 16 lags [i0, i0+16) of a trace of n lags (bit q set
// when lag i0+q is a candidate).  The 16 samples are read with 16-byte
// loads: the trace storage must be readable up to round_up(n, 16) and
// 16-byte aligned at every multiple of 16.
// Called by all 32 lanes of a warp with consecutive i0 (step 16): the
// neighbours x[i0-1] and x[i0+16] come from the adjacent lanes' vectors; only
// the first and last lane of the warp read them from memory.
template <class T> __device__ __forceinline__ unsigned cand_mask16(const T *x, int i0, int n, T thr)
{
    T v[16];
    const bool any = i0 < n;
    if (any) vec16<T>::load(x + i0, v);
    else
    {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = (T) 0;
    }
    const int lane = threadIdx.x & 31;
    T left = __shfl_up_sync(0xffffffffu, v[15], 1);
    T right = __shfl_down_sync(0xffffffffu, v[0], 1);
    if (lane == 0) left = (any && i0 > 0) ? x[i0 - 1] : (T) 0;
    if (lane == 31) right = (i0 + 16 < n) ? x[i0 + 16] : (T) 0;
    if (!any) return 0u;
    unsigned mask = 0;
#pragma unroll
    for (int q = 0; q < 16; ++q)
    {
        const int i = i0 + q;
        if (i >= n) break;
        const T xi = v[q];
        if (!(xi > thr)) continue;
        const T xl = q > 0 ? v[q - 1] : left;
        const T xr = q < 15 ? v[q + 1] : right;
        bool cand;
        if (n == 1) cand = xi > (T) 0;  // reference reads x[1] out of bounds; 0 assumed
        else if (i == 0) cand = sgn<T>(xr - xi) < 0;
        else if (i == n - 1) cand = sgn<T>(xi - xl) > 0;
        else cand = sgn<T>(xi - xl) >= 0 && sgn<T>(xr - xi) < 0;
        if (cand) mask |= 1u << q;
    }
    return mask;
}

// Phase 1: find candidates of one chunk; write up to kPkCap of them into the
// chunk's slot, and the exact count.
template <class T>
static __global__ void __launch_bounds__(kPkThreads) peak_cand_kernel(PeakTraces<T> tr, int nchunks, int *counts,
                                                                      int *slot_idx, T *slot_val)
{
    __shared__ long long sh[32];
    const int trace = blockIdx.y, chunk = blockIdx.x;
    const T *x = tr.x + (long) tr.row[trace] * tr.ldx;
    const int n = tr.len;
    const int i0 = chunk * kPkChunk + threadIdx.x * kPkPer;
    bool scan = true;
    if (tr.flags)
    {
        // the warp's 512 lags are chunks c64 .. c64 + 7 (c64 a multiple of 8)
        const int c64 = (chunk * kPkChunk + (threadIdx.x >> 5) * 32 * kPkPer) / 64;
        scan = c64 / 32 < tr.fwords &&
               ((tr.flags[(long) tr.row[trace] * tr.fwords + c64 / 32] >> (c64 % 32)) & 0xFFu) != 0u;
    }
    unsigned mask = scan ? cand_mask16<T>(x, i0, n, tr.thr) : 0u;  // warp-uniform choice
    long long tot;
    long long r = block_excl_scan((long long) __popc(mask), sh, &tot);
    const long slot = (long) trace * nchunks + chunk;
    while (mask)
    {
        int q = __ffs(mask) - 1;
        mask &= mask - 1;
        if (r < kPkCap)
        {
            slot_idx[slot * kPkCap + r] = i0 + q;
            slot_val[slot * kPkCap + r] = x[i0 + q];
        }
        ++r;
    }
    if (threadIdx.x == 0) counts[slot] = (int) tot;
}

// Phase 3: gather the slots (or re-scan overflowed chunks) into the packed,
// index-ordered candidate arrays (entries at or beyond cap are dropped and
// flagged).
template <class T>
static __global__ void __launch_bounds__(kPkThreads) peak_gather_kernel(PeakTraces<T> tr, int nchunks, const int *counts,
                                                                        const long long *offs, const int *slot_idx,
                                                                        const T *slot_val, int *cidx, T *cval, int *ctr,
                                                                        long long cap, int *overflow)
{
    __shared__ long long sh[32];
    const int trace = blockIdx.y, chunk = blockIdx.x;
    const long slot = (long) trace * nchunks + chunk;
    const int cnt = counts[slot];
    const long long off = offs[slot];
    if (cnt == 0) return;
    if (threadIdx.x == 0 && off + cnt > cap) *overflow = 1;
    if (cnt <= kPkCap)
    {
        for (int r = threadIdx.x; r < cnt; r += kPkThreads)
        {
            if (off + r >= cap) break;
            cidx[off + r] = slot_idx[slot * kPkCap + r];
            cval[off + r] = slot_val[slot * kPkCap + r];
            ctr[off + r] = trace;
        }
        return;
    }
    const T *x = tr.x + (long) tr.row[trace] * tr.ldx;
    const int n = tr.len;
    const int i0 = chunk * kPkChunk + threadIdx.x * kPkPer;
    bool scan = true;
    if (tr.flags)
    {
        // the warp's 512 lags are chunks c64 .. c64 + 7 (c64 a multiple of 8)
        const int c64 = (chunk * kPkChunk + (threadIdx.x >> 5) * 32 * kPkPer) / 64;
        scan = c64 / 32 < tr.fwords &&
               ((tr.flags[(long) tr.row[trace] * tr.fwords + c64 / 32] >> (c64 % 32)) & 0xFFu) != 0u;
    }
    unsigned mask = scan ? cand_mask16<T>(x, i0, n, tr.thr) : 0u;  // warp-uniform choice
    long long tot;
    long long r = block_excl_scan((long long) __popc(mask), sh, &tot);
    while (mask)
    {
        int q = __ffs(mask) - 1;
        mask &= mask - 1;
        if (off + r < cap)
        {
            cidx[off + r] = i0 + q;
            cval[off + r] = x[i0 + q];
            ctr[off + r] = trace;
        }
        ++r;
    }
}

// candidate states
enum : unsigned char { PK_UNDECIDED = 0, PK_ACCEPTED = 1, PK_NEW = 2, PK_REJECTED = 3 };

template <class T> __device__ __forceinline__ bool higher(T vj, int ij, T vg, int ig)
{
    return vj > vg || (vj == vg && ij < ig);
}

__device__ __forceinline__ long long pk_count(const long long *ncand, long long cap)
{
    long long n = *ncand;
    return n < cap ? n : cap;
}

// Round step 1: accept undecided candidates that have no undecided
// higher-priority neighbour within dist.  PK_NEW counts as undecided for
// the neighbours' tests, so the outcome does not depend on timing.
template <class T>
static __global__ void __launch_bounds__(kPkThreads) peak_decide_kernel(const long long *ncand_p, long long cap,
                                                                        const int *cidx, const T *cval, const int *ctr,
                                                                        const long long *trace_beg,
                                                                        unsigned char *state, int dist,
                                                                        int *n_undecided)
{
    const long long ncand = pk_count(ncand_p, cap);
    long long g = (long long) blockIdx.x * kPkThreads + threadIdx.x;
    if (g >= ncand) return;
    if (state[g] != PK_UNDECIDED) return;
    const int t = ctr[g];
    const long long tb = trace_beg[t], te = trace_beg[t + 1];
    const int ig = cidx[g];
    const T vg = cval[g];
    bool best = true;
    for (long long j = g - 1; j >= tb && ig - cidx[j] <= dist; --j)
    {
        unsigned char s = state[j];
        if ((s == PK_UNDECIDED || s == PK_NEW) && higher<T>(cval[j], cidx[j], vg, ig)) { best = false; break; }
    }
    if (best)
        for (long long j = g + 1; j < te && cidx[j] - ig <= dist; ++j)
        {
            unsigned char s = state[j];
            if ((s == PK_UNDECIDED || s == PK_NEW) && higher<T>(cval[j], cidx[j], vg, ig)) { best = false; break; }
        }
    if (best) state[g] = PK_NEW;
    else atomicAdd(n_undecided, 1);
}

// Round step 2: newly accepted candidates reject their undecided neighbours.
static __global__ void __launch_bounds__(kPkThreads) peak_suppress_kernel(const long long *ncand_p, long long cap,
                                                                          const int *cidx, const int *ctr,
                                                                          const long long *trace_beg,
                                                                          unsigned char *state, int dist)
{
    const long long ncand = pk_count(ncand_p, cap);
    long long g = (long long) blockIdx.x * kPkThreads + threadIdx.x;
    if (g >= ncand) return;
    if (state[g] != PK_NEW) return;
    const int t = ctr[g];
    const long long tb = trace_beg[t], te = trace_beg[t + 1];
    const int ig = cidx[g];
    for (long long j = g - 1; j >= tb && ig - cidx[j] <= dist; --j)
        if (state[j] == PK_UNDECIDED) state[j] = PK_REJECTED;
    for (long long j = g + 1; j < te && cidx[j] - ig <= dist; ++j)
        if (state[j] == PK_UNDECIDED) state[j] = PK_REJECTED;
    state[g] = PK_ACCEPTED;
}

// accepted flag (as int) for the final compaction; zero past the count
static __global__ void peak_flags_kernel(const long long *ncand_p, long long cap, const unsigned char *state, int all,
                                         int *flags)
{
    const long long ncand = pk_count(ncand_p, cap);
    long long g = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= cap) return;
    flags[g] = (g < ncand && (all || state[g] == PK_ACCEPTED)) ? 1 : 0;
}

static __global__ void peak_compact_kernel(const long long *ncand_p, long long cap, const int *flags,
                                           const long long *pos, const int *cidx, int *peaks)
{
    const long long ncand = pk_count(ncand_p, cap);
    long long g = (long long) blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= ncand) return;
    if (flags[g]) peaks[pos[g]] = cidx[g];
}

// per-trace peak offsets: peak_off[t] = pos[trace_beg[t]]
// The traces' peak offsets; res[ntr + 1 ..]: candidates, whether the search is
// dense, the object's device status word, candidates left undecided, overflow
// (read back in one copy).
static __global__ void peak_trace_offsets_kernel(int ntr, const long long *trace_beg, const long long *pos,
                                                 const long long *ncand, const int *flags, const int *err,
                                                 const int *counter, long long *res)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0)
    {
        res[ntr + 1] = *ncand;
        res[ntr + 2] = flags[0];
        res[ntr + 3] = err ? *err : 0;
        res[ntr + 4] = counter[0];
        res[ntr + 5] = counter[1];
    }
    if (t > ntr) return;
    res[t] = pos[trace_beg[t]];
}

// trace_beg[t] = min(offs[t * nchunks], cap): candidate offsets of each trace
static __global__ void peak_trace_beg_kernel(int ntr, int nchunks, const long long *offs, long long cap,
                                             long long *trace_beg)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t > ntr) return;
    long long v = offs[(long) t * nchunks];
    trace_beg[t] = v < cap ? v : cap;
}

// ----------------------------------------------------------------------------
// Candidates gathered by the correlator.  Chunk b of a trace is correlator
// block b, lags [b*S, b*S + S): the correlator decided the body lags
// [b*S+1, b*S+S-2] from the values it stored (count body_cnt, up to kPkCap
// unordered slot entries, indexed by row * nblk + b); peak_totals_kernel
// decides the first and last lag of each block from the stored trace (bits 0
// and 1 of ht) and forms the chunk's total count.

// Packs chunk b of a trace in index order: first lag, body (slot entries
// ranked by index, or a re-scan of the stored trace when more than kPkCap
// body lags passed), last lag.  One warp per 32 consecutive chunks of a
// trace: the lanes read the 32 counts, and the warp packs the non-empty
// chunks one after another (most chunks are empty).
static_assert(kPkCap == 32, "peak_gather_fused_kernel ranks one slot entry per lane");
constexpr int kPkGatherSpan = 32;  // chunks per warp

template <class T>
static __global__ void __launch_bounds__(kPkThreads)
    peak_gather_fused_kernel(PeakTraces<T> tr, FusedSlots<T> fs, const int *counts, const unsigned char *ht,
                             const long long *offs, int *cidx, T *cval, int *ctr, long long cap, int *overflow)
{
    const int lane = threadIdx.x & 31;
    const int trace = blockIdx.y;
    const int b0 = (blockIdx.x * (kPkThreads / 32) + (threadIdx.x >> 5)) * kPkGatherSpan;
    if (b0 >= fs.nblk) return;
    const int row = tr.row[trace];
    const T *x = tr.x + (long) row * tr.ldx;
    const long n = tr.len;
    auto put = [&](long long o, long i, T v) {
        if (o < cap)
        {
            cidx[o] = (int) i;
            cval[o] = v;
            ctr[o] = trace;
        }
    };
    const int bl = b0 + lane;
    const int cnt_l = bl < fs.nblk ? counts[(long) trace * fs.nblk + bl] : 0;
    unsigned todo = __ballot_sync(0xffffffffu, cnt_l != 0);
    while (todo)
    {
        const int q = __ffs(todo) - 1;  // warp-uniform
        todo &= todo - 1;
        const int b = b0 + q;
        const int cnt = __shfl_sync(0xffffffffu, cnt_l, q);
        const long slot = (long) trace * fs.nblk + b;
        const long long off = offs[slot];
        if (lane == 0 && off + cnt > cap) *overflow = 1;
        const int hv = ht[slot];
        const long S = fs.row_S ? fs.row_S[row] : fs.S;
        const long i0 = (long) b * S;
        if (lane == 0)
        {
            if (hv & 1) put(off, i0, x[i0]);
            if (hv & 2) put(off + cnt - 1, i0 + S - 1, x[i0 + S - 1]);
        }
        const long long boff = off + (hv & 1);
        const long bs = (long) row * fs.nblk + b;
        const int bc = fs.cnt[bs];
        if (bc <= kPkCap)
        {
            // kPkCap == 32: one entry per lane, ranked by index
            const int *si = fs.idx + bs * kPkCap;
            if (lane < bc)
            {
                const int ir = si[lane];
                int rank = 0;
                for (int r = 0; r < bc; ++r) rank += si[r] < ir ? 1 : 0;
                put(boff + rank, ir, fs.val[bs * kPkCap + lane]);
            }
            continue;
        }
        const long lo = i0 + 1, hi = (i0 + S - 1 < n) ? i0 + S - 1 : n;
        long long base = boff;
        for (long c0 = lo; c0 < hi; c0 += 32 * kPkPer)
        {
            const long a = c0 + (long) lane * kPkPer;
            unsigned mask = 0;
#pragma unroll 4
            for (int r = 0; r < kPkPer; ++r)
                if (a + r < hi && cand_rule<T>(x[a + r - 1], x[a + r], a + r + 1 < n ? x[a + r + 1] : (T) 0, a + r, n,
                                               tr.thr))
                    mask |= 1u << r;
            const int c = __popc(mask);
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            long long r = base + incl - c;
            while (mask)
            {
                const int qq = __ffs(mask) - 1;
                mask &= mask - 1;
                put(r, a + qq, x[a + qq]);
                ++r;
            }
            base += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
}

// ----------------------------------------------------------------------------
// Pruning per trace.  Traces are independent, so one CTA takes a trace's
// candidates into shared memory, runs the rounds above until none is
// undecided and compacts the accepted ones: three launches (totals, prune,
// emit) instead of two launches and a clear per round over a grid sized for
// the candidate capacity, three scans and a compaction (25 launches, about
// 130 us of mostly empty grids for the banks measured; now 15 us for 100 traces,
// 31 for 2,000).  A trace
// with more than kPkTraceCap candidates, or a chunk with more than its slot
// holds, makes the search dense: the totals raise flags[0], and the host takes
// the launches above, which have no such limit.  More candidates in all than
// the packed arrays hold leave the counts only; the host enlarges the arrays.
constexpr int kPkTraceCap = 4096;
constexpr int kPkTotThreads = 128;
template <class T> constexpr size_t pk_prune_bytes() { return (sizeof(int) + sizeof(T) + 1) * (size_t) kPkTraceCap; }

// Exclusive prefix of n ints by one CTA: out[0..n]; sh holds 32 values.
static __device__ __forceinline__ void cta_prefix(const int *in, int n, long long *out, long long *sh)
{
    long long base = 0;
    for (int i0 = 0; i0 < n; i0 += blockDim.x)
    {
        const int i = i0 + threadIdx.x;
        long long tot;
        const long long e = block_excl_scan((long long) (i < n ? __ldcg(in + i) : 0), sh, &tot);
        if (i < n) out[i] = base + e;
        base += tot;
    }
    if (threadIdx.x == 0) out[n] = base;
}

// True in every thread of the last CTA of the grid to get here (whose other
// CTAs' global stores before the call are then visible); the ticket is left
// at 0 for the next launch.
static __device__ __forceinline__ bool last_cta(int *ticket, int *sh)
{
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
    {
        *sh = atomicAdd(ticket, 1) == (int) gridDim.x - 1;
        if (*sh) *ticket = 0;
    }
    __syncthreads();
    const bool last = *sh != 0;
    if (last) __threadfence();
    return last;
}

// Candidates per trace (FUSED: with the block-edge lags decided here), and by the last CTA the traces' offsets and flags[0] (1: a
// dense search; flags[1] collects it and is left at 0).
template <class T, bool FUSED>
static __global__ void __launch_bounds__(kPkTotThreads)
    peak_totals_kernel(PeakTraces<T> tr, FusedSlots<T> fs, int nchunks, int *counts, unsigned char *ht, int *totals,
                       long long *trace_beg, int *ticket, int *flags)
{
    __shared__ long long sh[32];
    __shared__ int lsh;
    const int trace = blockIdx.x, row = tr.row[trace];
    const long n = tr.len;
    const T *x = tr.x + (long) row * tr.ldx;
    const int nb = FUSED && fs.row_nblk ? fs.row_nblk[row] : nchunks;
    const long S = FUSED && fs.row_S ? fs.row_S[row] : fs.S;
    long long mine = 0;
    bool over = false;
    for (int b = threadIdx.x; b < nchunks; b += kPkTotThreads)
    {
        const long g = (long) trace * nchunks + b;
        int cnt;
        if constexpr (FUSED)
        {
            const long i0 = (long) b * S, i1 = i0 + S - 1;
            int h = 0, tl = 0;
            cnt = 0;
            if (b < nb)
            {
                h = (i0 < n && is_candidate<T>(x, (int) i0, (int) n, tr.thr)) ? 1 : 0;
                tl = (i1 < n && is_candidate<T>(x, (int) i1, (int) n, tr.thr)) ? 1 : 0;
                cnt = fs.cnt[(long) row * fs.nblk + b];
                over |= cnt > kPkCap;
                cnt += h + tl;
            }
            counts[g] = cnt;
            ht[g] = (unsigned char) (h | (tl << 1));
        }
        else
        {
            cnt = counts[g];
            over |= cnt > kPkCap;
        }
        mine += cnt;
    }
    long long tot;
    block_excl_scan(mine, sh, &tot);
    over = __syncthreads_or(over);
    if (threadIdx.x == 0)
    {
        totals[trace] = (int) tot;
        if (over || tot > kPkTraceCap) atomicOr(flags + 1, 1);
    }
    if (last_cta(ticket, &lsh))
    {
        cta_prefix(totals, gridDim.x, trace_beg, sh);
        if (threadIdx.x == 0) flags[0] = atomicExch(flags + 1, 0);
    }
}

// One CTA per trace: gather, prune, compact into raw[trace_beg[t]...], the
// accepted count in nacc; the last CTA forms the traces' peak offsets.
template <class T, bool FUSED>
static __global__ void __launch_bounds__(kPkThreads)
    peak_prune_kernel(PeakTraces<T> tr, FusedSlots<T> fs, int nchunks, const int *counts, const unsigned char *ht,
                      const int *slot_idx, const T *slot_val, int dist, const long long *trace_beg, long long cap,
                      int *raw, int *nacc, long long *peak_off, int *ticket, const int *flags)
{
    extern __shared__ __align__(16) unsigned char smem_pk[];
    __shared__ long long sh[32];
    __shared__ int lsh;
    T *val = reinterpret_cast<T *>(smem_pk);
    int *idx = reinterpret_cast<int *>(val + kPkTraceCap);
    unsigned char *state = reinterpret_cast<unsigned char *>(idx + kPkTraceCap);
    const int tid = threadIdx.x, trace = blockIdx.x, row = tr.row[trace];
    const long long tb = trace_beg[trace];
    const long long total = trace_beg[trace + 1] - tb;
    const T *x = tr.x + (long) row * tr.ldx;
    int accepted = 0;
    if (flags[0] == 0 && trace_beg[gridDim.x] <= cap && total > 0)
    {
        const int nc = (int) total;
        // ---- candidates in index order; a thread packs one chunk
        long long base = 0;
        for (int b0 = 0; b0 < nchunks; b0 += kPkThreads)
        {
            const int b = b0 + tid;
            const long g = (long) trace * nchunks + b;
            const int cnt = b < nchunks ? counts[g] : 0;
            long long tot;
            int o = (int) (base + block_excl_scan((long long) cnt, sh, &tot));
            base += tot;
            if (cnt == 0) continue;
            if constexpr (FUSED)
            {
                const int hv = ht[g];
                const long S = fs.row_S ? fs.row_S[row] : fs.S;
                const long i0 = (long) b * S, bs = (long) row * fs.nblk + b;
                const int bc = cnt - (hv & 1) - (hv >> 1);
                if (hv & 1)
                {
                    idx[o] = (int) i0;
                    val[o++] = x[i0];
                }
                for (int q = 0; q < bc; ++q)
                {
                    // insertion by index: the slot's entries are unordered
                    const int ir = fs.idx[bs * kPkCap + q];
                    const T vr = fs.val[bs * kPkCap + q];
                    int k = o + q;
                    for (; k > o && idx[k - 1] > ir; --k)
                    {
                        idx[k] = idx[k - 1];
                        val[k] = val[k - 1];
                    }
                    idx[k] = ir;
                    val[k] = vr;
                }
                o += bc;
                if (hv & 2)
                {
                    idx[o] = (int) (i0 + S - 1);
                    val[o] = x[i0 + S - 1];
                }
            }
            else
            {
                for (int q = 0; q < cnt; ++q)
                {
                    idx[o + q] = slot_idx[g * kPkCap + q];
                    val[o + q] = slot_val[g * kPkCap + q];
                }
            }
        }
        __syncthreads();
        for (int i = tid; i < nc; i += kPkThreads) state[i] = dist > 0 ? PK_UNDECIDED : PK_ACCEPTED;
        __syncthreads();
        // ---- rounds: each accepts at least the best undecided candidate
        bool left = dist > 0;
        while (left)
        {
            bool mine = false;
            for (int g = tid; g < nc; g += kPkThreads)
            {
                if (state[g] != PK_UNDECIDED) continue;
                const int ig = idx[g];
                const T vg = val[g];
                bool best = true;
                for (int k = g - 1; k >= 0 && ig - idx[k] <= dist; --k)
                    if (state[k] <= PK_NEW && state[k] != PK_ACCEPTED && higher<T>(val[k], idx[k], vg, ig))
                    {
                        best = false;
                        break;
                    }
                if (best)
                    for (int k = g + 1; k < nc && idx[k] - ig <= dist; ++k)
                        if (state[k] <= PK_NEW && state[k] != PK_ACCEPTED && higher<T>(val[k], idx[k], vg, ig))
                        {
                            best = false;
                            break;
                        }
                if (best) state[g] = PK_NEW;
                else mine = true;
            }
            left = __syncthreads_or(mine);
            for (int g = tid; g < nc; g += kPkThreads)
            {
                if (state[g] != PK_NEW) continue;
                const int ig = idx[g];
                for (int k = g - 1; k >= 0 && ig - idx[k] <= dist; --k)
                    if (state[k] == PK_UNDECIDED) state[k] = PK_REJECTED;
                for (int k = g + 1; k < nc && idx[k] - ig <= dist; ++k)
                    if (state[k] == PK_UNDECIDED) state[k] = PK_REJECTED;
                state[g] = PK_ACCEPTED;
            }
            __syncthreads();
        }
        // ---- accepted lags, ascending
        for (int g0 = 0; g0 < nc; g0 += kPkThreads)
        {
            const int g = g0 + tid;
            const bool a = g < nc && state[g] == PK_ACCEPTED;
            long long tot;
            const long long o = block_excl_scan((long long) (a ? 1 : 0), sh, &tot);
            if (a) raw[tb + accepted + o] = idx[g];
            accepted += (int) tot;
        }
    }
    if (tid == 0) nacc[trace] = accepted;
    if (last_cta(ticket, &lsh)) cta_prefix(nacc, gridDim.x, peak_off, sh);
}

// The traces' accepted lags side by side (none in a dense search, or one with
// more candidates than cap); res[ntr + 1 ..]: candidates, whether the search is
// dense, the object's device status word.
static __global__ void __launch_bounds__(64) peak_emit_kernel(int ntr, const int *raw, const long long *trace_beg,
                                                              const int *flags, const int *err, long long *res,
                                                              int *peaks)
{
    const int t = blockIdx.x;
    if (t == 0 && threadIdx.x == 0)
    {
        res[ntr + 1] = trace_beg[ntr];
        res[ntr + 2] = flags[0];
        res[ntr + 3] = err ? *err : 0;
    }
    const long long o = res[t], b = trace_beg[t];
    const int n = (int) (res[t + 1] - o);
    for (int i = threadIdx.x; i < n; i += 64) peaks[o + i] = raw[b + i];
}

}  // namespace mfgpu
