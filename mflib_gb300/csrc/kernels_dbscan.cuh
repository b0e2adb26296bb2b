// kernels_dbscan.cuh -- DBSCAN (MFLib::DBSCAN::cluster, src/dbscan.cpp:187-214,
// which calls Intel DAAL dbscan::Batch<double>) on the device, for one or
// many independent segments.
//
// Semantics (DAAL's published algorithm):
//   N(i) = { j in segment(i) : ||x_i - x_j||_2 <= eps } including i;
//   core(i) iff sum_{j in N(i)} w_j >= minObservations (w = 1 unweighted);
//   clusters are the connected components of core points under the
//   eps-neighbour relation; DAAL visits observations in index order and
//   opens a new cluster at the first unassigned core point, so cluster ids
//   are ordered by each component's lowest core index;
//   a non-core point with a core neighbour takes the smallest id among its
//   neighbours' clusters (the first cluster to reach it); others are -1.
//
// Device formulation: one warp per point scans its segment; weighted
// neighbour sums; union-find with atomic CAS that always hooks the larger
// root under the smaller (so every component's root is its lowest core
// index); exclusive scan of root flags for the ids; then labels.
// One feature: |x_i - x_j| <= eps, which equals sqrt((x_i - x_j)^2) <= eps
// exactly in IEEE arithmetic and avoids the FP64 square root.
#pragma once
#include <cstdint>
#include "kernels_util.cuh"

namespace mfgpu {

constexpr int kDbThreads = 256;
constexpr int kDbWarps = kDbThreads / 32;

struct DbParams
{
    const double *X;        // [n x nf] row-major
    int nf;
    const double *w;        // weights or null
    double eps;
    double min_obs;
    const int *seg_of;      // segment of each point
    const int *seg_off;     // [nseg + 1]
    int n;
};

__device__ __forceinline__ bool db_near(const DbParams &p, int i, int j)
{
    if (p.nf == 1) return fabs(p.X[i] - p.X[j]) <= p.eps;
    const double *a = p.X + (long) i * p.nf, *b = p.X + (long) j * p.nf;
    double s = 0;
    for (int f = 0; f < p.nf; ++f)
    {
        double d = a[f] - b[f];
        s = fma(d, d, s);
    }
    return sqrt(s) <= p.eps;
}

// core flags: weighted neighbourhood size >= minObservations
static __global__ void __launch_bounds__(kDbThreads) db_core_kernel(DbParams p, unsigned char *core, int *parent)
{
    const int i = blockIdx.x * kDbWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= p.n) return;
    const int s = p.seg_of[i];
    const int jb = p.seg_off[s], je = p.seg_off[s + 1];
    double acc = 0;
    for (int j = jb + lane; j < je; j += 32)
        if (db_near(p, i, j)) acc += p.w ? p.w[j] : 1.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0)
    {
        core[i] = acc >= p.min_obs ? 1 : 0;
        parent[i] = i;
    }
}

// Root of x with path halving: each visited node is re-pointed at its
// grandparent.  Safe under concurrent unions: parents only ever move to an
// ancestor (unions hook a root under a smaller root), so the write never
// detaches a node from its component, and roots are never written here.
// Without it the predecessor unions of the 1-D case build chains as long as
// a component, and every find walks them.
__device__ __forceinline__ int db_find(volatile int *parent, int x)
{
    int p = parent[x];
    while (p != x)
    {
        const int g = parent[p];
        if (g != p) parent[x] = g;
        x = g;
        p = parent[x];
    }
    return x;
}

__device__ __forceinline__ void db_unite(int *parent, int a, int b)
{
    volatile int *vp = parent;
    for (int guard = 0; guard < (1 << 30); ++guard)
    {
        a = db_find(vp, a);
        b = db_find(vp, b);
        if (a == b) return;
        if (a > b) { int t = a; a = b; b = t; }
        int old = atomicCAS(parent + b, b, a);  // hook the larger root under the smaller
        if (old == b) return;
        b = old;
    }
}

// Components of the core points.  Several features: every core pair within
// eps is united.  One feature: ordered by (x, index), the components are the
// runs of consecutive core points whose gaps are at most eps (any core pair
// within eps spans only such gaps), so each core point is united with its
// predecessor in that order alone -- O(n) unions instead of O(n k) on the
// same few roots.
static __global__ void __launch_bounds__(kDbThreads) db_union_kernel(DbParams p, const unsigned char *core, int *parent)
{
    const int i = blockIdx.x * kDbWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= p.n || !core[i]) return;
    const int s = p.seg_of[i];
    const int jb = p.seg_off[s], je = p.seg_off[s + 1];
    if (p.nf != 1)
    {
        for (int j = i + 1 + lane; j < je; j += 32)
            if (core[j] && db_near(p, i, j)) db_unite(parent, i, j);
        return;
    }
    const double xi = p.X[i];
    double bx = 0.0;
    int bj = -1;  // predecessor: the largest (x_j, j) below (x_i, i)
    for (int j = jb + lane; j < je; j += 32)
    {
        if (j == i || !core[j]) continue;
        const double xj = p.X[j];
        const bool below = xj < xi || (xj == xi && j < i);
        if (below && (bj < 0 || xj > bx || (xj == bx && j > bj)))
        {
            bx = xj;
            bj = j;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        const double ox = __shfl_xor_sync(0xffffffffu, bx, o);
        const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
        if (oj >= 0 && (bj < 0 || ox > bx || (ox == bx && oj > bj)))
        {
            bx = ox;
            bj = oj;
        }
    }
    if (lane == 0 && bj >= 0 && fabs(xi - bx) <= p.eps) db_unite(parent, i, bj);
}

// Root without writes: in the roots pass a halving write from one thread
// could land after another thread stored its node's final root and replace
// it with an intermediate ancestor.
__device__ __forceinline__ int db_find_ro(const volatile int *parent, int x)
{
    int p = parent[x];
    while (p != x)
    {
        x = p;
        p = parent[x];
    }
    return x;
}

static __global__ void db_roots_kernel(int n, const unsigned char *core, int *parent, int *is_root)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (!core[i]) { is_root[i] = 0; return; }
    int r = db_find_ro(parent, i);
    parent[i] = r;
    is_root[i] = r == i ? 1 : 0;
}

// labels: core -> id of its root; border -> smallest id among core neighbours
static __global__ void __launch_bounds__(kDbThreads) db_label_kernel(DbParams p, const unsigned char *core, const int *root,
                                                                     const long long *root_pos, int *labels)
{
    const int i = blockIdx.x * kDbWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= p.n) return;
    const int s = p.seg_of[i];
    const int jb = p.seg_off[s], je = p.seg_off[s + 1];
    const long long base = root_pos[jb];
    if (core[i])
    {
        if (lane == 0) labels[i] = (int) (root_pos[root[i]] - base);
        return;
    }
    long long best = 0x7fffffffffffffffLL;
    for (int j = jb + lane; j < je; j += 32)
    {
        if (!core[j] || !db_near(p, i, j)) continue;
        long long id = root_pos[root[j]] - base;
        best = id < best ? id : best;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        long long v = __shfl_xor_sync(0xffffffffu, best, o);
        best = v < best ? v : best;
    }
    if (lane == 0) labels[i] = best == 0x7fffffffffffffffLL ? -1 : (int) best;
}

// ----------------------------------------------------------------------------
// One feature with the points of every segment sorted by (x, index) on the
// host: xs[r] is the r-th smallest value of its segment (positions keep the
// segment offsets), perm[r] its point, rank[i] the position of point i.  The
// eps-neighbourhood of a point is then the contiguous range of positions
// [lo, hi) found by binary search with the same predicate |x_i - x_j| <= eps
// (a rounded difference is monotone in x_j), so every pass visits the
// neighbours only: O(n log n + sum of neighbourhood sizes) instead of a scan
// of the whole segment per point.
struct Db1Sorted
{
    const double *xs;
    const int *perm;
    const int *rank;
    // per segment, the end of its non-NaN values (NaN sorted last, no
    // neighbour of anything); null when no value is NaN
    const int *fend;
};

__device__ __forceinline__ int db1_end(const DbParams &p, const Db1Sorted &q, int s)
{
    return q.fend ? q.fend[s] : p.seg_off[s + 1];
}

// [lo, hi): positions of the segment [jb, je) within eps of the value xi
__device__ __forceinline__ void db1_range(const double *xs, int jb, int je, double xi, double eps, int &lo, int &hi)
{
    int a = jb, b = je;  // first position with xi - xs <= eps
    while (a < b)
    {
        const int m = (a + b) >> 1;
        if (xi - xs[m] <= eps) b = m;
        else a = m + 1;
    }
    lo = a;
    b = je;              // first position with xs - xi > eps
    while (a < b)
    {
        const int m = (a + b) >> 1;
        if (xs[m] - xi <= eps) a = m + 1;
        else b = m;
    }
    hi = a;
}

static __global__ void __launch_bounds__(kDbThreads) db1_core_kernel(DbParams p, Db1Sorted q, unsigned char *core,
                                                                     int *parent)
{
    const int i = blockIdx.x * kDbWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= p.n) return;
    const int s = p.seg_of[i];
    int lo = 0, hi = 0;
    if (lane == 0) db1_range(q.xs, p.seg_off[s], db1_end(p, q, s), p.X[i], p.eps, lo, hi);
    lo = __shfl_sync(0xffffffffu, lo, 0);
    hi = __shfl_sync(0xffffffffu, hi, 0);
    double acc = 0;
    for (int r = lo + lane; r < hi; r += 32) acc += p.w ? p.w[q.perm[r]] : 1.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0)
    {
        core[i] = acc >= p.min_obs ? 1 : 0;
        parent[i] = i;
    }
}

// each core point united with the nearest core point before it in the sorted
// order when that one lies within eps (the runs of consecutive core points
// with gaps <= eps are the components, as in db_union_kernel's 1-D case)
static __global__ void __launch_bounds__(kDbThreads) db1_union_kernel(DbParams p, Db1Sorted q, const unsigned char *core,
                                                                      int *parent)
{
    const int i = blockIdx.x * kDbWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= p.n || !core[i]) return;
    const int s = p.seg_of[i];
    const int jb = p.seg_off[s];
    const double xi = p.X[i];
    for (int r0 = q.rank[i] - 1; r0 >= jb; r0 -= 32)
    {
        const int r = r0 - lane;
        const bool in = r >= jb && xi - q.xs[r] <= p.eps;
        const bool hit = in && core[q.perm[r]];
        const unsigned hm = __ballot_sync(0xffffffffu, hit), im = __ballot_sync(0xffffffffu, in);
        if (hm)
        {
            const int l = __ffs(hm) - 1;  // the nearest position (lowest lane)
            if (lane == l) db_unite(parent, i, q.perm[r]);
            return;
        }
        if (im != 0xffffffffu) return;  // left the neighbourhood before finding a core point
    }
}

// border points: the smallest cluster id among their core neighbours
static __global__ void __launch_bounds__(kDbThreads) db1_label_kernel(DbParams p, Db1Sorted q, const unsigned char *core,
                                                                      const int *root, const long long *root_pos,
                                                                      int *labels)
{
    const int i = blockIdx.x * kDbWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (i >= p.n) return;
    const int s = p.seg_of[i];
    const int jb = p.seg_off[s], je = db1_end(p, q, s);
    const long long base = root_pos[jb];
    if (core[i])
    {
        if (lane == 0) labels[i] = (int) (root_pos[root[i]] - base);
        return;
    }
    int lo = 0, hi = 0;
    if (lane == 0) db1_range(q.xs, jb, je, p.X[i], p.eps, lo, hi);
    lo = __shfl_sync(0xffffffffu, lo, 0);
    hi = __shfl_sync(0xffffffffu, hi, 0);
    long long best = 0x7fffffffffffffffLL;
    for (int r = lo + lane; r < hi; r += 32)
    {
        const int j = q.perm[r];
        if (!core[j]) continue;
        const long long id = root_pos[root[j]] - base;
        best = id < best ? id : best;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        const long long v = __shfl_xor_sync(0xffffffffu, best, o);
        best = v < best ? v : best;
    }
    if (lane == 0) labels[i] = best == 0x7fffffffffffffffLL ? -1 : (int) best;
}

// Device-side preparation of Db1Sorted, for callers whose data are already
// on the device: perm (n2 = a power of two >= n entries, padding indices
// n .. n2-1 sorting last) sorted by (segment, value, index) with NaN after
// every number in its segment, by a bitonic network (one launch per step),
// then the sorted values, each point's position and every segment's end of
// non-NaN values.
__device__ __forceinline__ bool db1_less(const DbParams &p, int a, int b)
{
    if (a >= p.n) return b >= p.n && a < b;
    if (b >= p.n) return true;
    const int sa = p.seg_of[a], sb = p.seg_of[b];
    if (sa != sb) return sa < sb;
    const double xa = p.X[a], xb = p.X[b];
    const bool na = isnan(xa), nb = isnan(xb);
    if (na != nb) return nb;
    if (!na && xa != xb) return xa < xb;
    return a < b;
}

static __global__ void db1_iota_kernel(int *perm, int n2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n2) perm[i] = i;
}

// one compare-exchange step (distance j, merge size k) of the bitonic network
static __global__ void db1_bitonic_kernel(DbParams p, int *perm, int n2, int j, int k)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n2) return;
    const int l = i ^ j;
    if (l <= i) return;
    const int a = perm[i], b = perm[l];
    const bool up = (i & k) == 0;
    if (up ? db1_less(p, b, a) : db1_less(p, a, b))
    {
        perm[i] = b;
        perm[l] = a;
    }
}

static __global__ void db1_gather_kernel(DbParams p, const int *perm, double *xs, int *rank)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= p.n) return;
    const int i = perm[r];
    xs[r] = p.X[i];
    rank[i] = r;
}

// fend[s]: the first position of segment s holding NaN (its end if none)
static __global__ void db1_fend_kernel(int nseg, const int *seg_off, const double *xs, int *fend)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    int a = seg_off[s], b = seg_off[s + 1];
    while (a < b)
    {
        const int m = (a + b) >> 1;
        if (isnan(xs[m])) b = m;
        else a = m + 1;
    }
    fend[s] = a;
}

static __global__ void db_count_kernel(int nseg, const int *seg_off, const long long *root_pos, int *n_clusters)
{
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nseg) return;
    n_clusters[s] = (int) (root_pos[seg_off[s + 1]] - root_pos[seg_off[s]]);
}

// ----------------------------------------------------------------------------
// One feature, segments of at most kDb1Cap points: one CTA does a segment in
// shared memory, from its unsorted points to its labels.  Sorted by (value,
// index) with NaN last, a point's neighbourhood is a range of positions; the
// clusters are the runs of consecutive core points with gaps of at most eps,
// numbered by their lowest point index.  One launch between one upload and
// one read-back, where the sort on the host, nine uploads, nine launches and
// the scans took 465 of the 535 us of an association (9,500 points in 8
// segments; now 106 us in all).  A segment's size is limited by the sort in
// shared memory (20 bytes for each of a power of two of points: 164 KB); up to
// there this form was the faster one wherever it was measured (one segment,
// spread or in one neighbourhood, with and without weights: 1,024 points 64 .. 87
// us against 106 .. 137, 8,192 points 0.31 .. 0.46 ms against 0.53 .. 0.75).
// Larger segments keep the launches above.
//
// A CTA of NT threads takes segments of up to 8 NT points: 1,024 threads, and
// where there are more segments than the chip holds CTAs of that size (two per
// SM), 32 or 128 if the largest segment allows.  (100,000 segments of two points:
// in CTAs of 1,024 threads 3.9 .. 5.0 ms, of one warp 0.37, the launches above 1.9;
// 5,000 of 100: 0.55 .. 0.69, 0.33 and 14.7 ms.)
constexpr int kDb1Per = 8, kDb1Cap = 8192;
constexpr int kDb1Resident = 2 * 152;
__host__ __device__ constexpr size_t db1_bytes(int n2) { return (sizeof(double) + 3 * sizeof(int)) * (size_t) n2; }

// exclusive scan over the CTA of one value per thread (sum or maximum);
// sh: 33 ints; the total goes to *total
template <bool MAX, int NT> __device__ __forceinline__ int db1_scan(int v, int *sh, int *total)
{
    constexpr int none = MAX ? -1 : 0;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = MAX ? max(x, y) : x + y;
    }
    __syncthreads();
    if (lane == 31) sh[w] = x;
    __syncthreads();
    int before = none, all = none;
    for (int i = 0; i < NT / 32; ++i)
    {
        const int t = sh[i];
        if (i < w) before = MAX ? max(before, t) : before + t;
        all = MAX ? max(all, t) : all + t;
    }
    *total = all;
    int e = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) e = none;
    return MAX ? max(before, e) : before + e;
}

// exclusive scan over the CTA of one weight sum per thread; total and the total
// of the magnitudes in every thread
template <int NT>
__device__ __forceinline__ void db1_scan_weights(double own, double mag, double &before, double &total, double &mags)
{
    constexpr int NW = NT / 32;
    __shared__ double sw[NW], sm[NW], all[2];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const double y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mag += __shfl_xor_sync(0xffffffffu, mag, o);
    if (lane == 31)
    {
        sw[w] = x;
        sm[w] = mag;
    }
    __syncthreads();
    // the warps' sums by one warp: 32 warps adding 32 sums each would keep the
    // FP64 pipe busy for 30 us
    if (w == 0)
    {
        const double y = lane < NW ? sw[lane] : 0.0;
        double t = y, m = lane < NW ? sm[lane] : 0.0;
#pragma unroll
        for (int o = 1; o < NW; o <<= 1)
        {
            const double u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += u;
            m += __shfl_xor_sync(0xffffffffu, m, o);
        }
        const double e = __shfl_up_sync(0xffffffffu, t, 1);
        if (lane < NW) sw[lane] = lane > 0 ? e : 0.0;
        if (lane == NW - 1) all[0] = t;
        if (lane == 0) all[1] = m;
    }
    __syncthreads();
    total = all[0];
    mags = all[1];
    const double e = __shfl_up_sync(0xffffffffu, x, 1);
    before = sw[w] + (lane > 0 ? e : 0.0);
}

template <int NT>
static __global__ void __launch_bounds__(NT) db1_segment_kernel(const double *X, const double *wt, const int *seg_off,
                                                               int n2max, double eps, double min_obs, int *labels,
                                                               int *n_clusters)
{
    extern __shared__ __align__(16) unsigned char smem_db[];
    __shared__ int sh[33];
    unsigned long long *key = reinterpret_cast<unsigned long long *>(smem_db);
    double *xs = reinterpret_cast<double *>(smem_db);  // the sorted values, over the keys
    // run of each position; not core: -2 - the core position before (-1: none)
    int *run = reinterpret_cast<int *>(key + n2max);
    int *aux = run + n2max;                            // per run, then per point
    int *idx = aux + n2max;                            // point of each position
    double *ps = reinterpret_cast<double *>(run);      // prefix sums of the weights, over run and aux
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, s = blockIdx.x;
    const int b = seg_off[s], n = seg_off[s + 1] - b;
    if (n <= 0)
    {
        if (tid == 0) n_clusters[s] = 0;
        return;
    }
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    // ---- sort: order-preserving integer keys (-0 as +0), NaN and padding last
    for (int i = tid; i < n2; i += NT)
    {
        unsigned long long k = ~0ull;
        if (i < n)
        {
            const double v = X[b + i] + 0.0;
            const long long u = __double_as_longlong(v);
            if (!isnan(v)) k = u < 0 ? ~(unsigned long long) u : (unsigned long long) u | (1ull << 63);
        }
        key[i] = k;
        idx[i] = i;
    }
    __syncthreads();
    for (int k = 2; k <= n2; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1)
        {
            for (int i = tid; i < n2 / 2; i += NT)
            {
                const int p = 2 * i - (i & (j - 1)), q = p + j;
                const unsigned long long ka = key[p], kb = key[q];
                const int ia = idx[p], ib = idx[q];
                const bool gt = ka > kb || (ka == kb && ia > ib);
                if (gt == ((p & k) == 0))
                {
                    key[p] = kb;
                    key[q] = ka;
                    idx[p] = ib;
                    idx[q] = ia;
                }
            }
            __syncthreads();
        }
    // ---- values in place; nv: points that are no NaN
    int mine = 0;
    for (int i = tid; i < n; i += NT)
    {
        const unsigned long long k = key[i];
        if (k != ~0ull)
        {
            ++mine;
            xs[i] = __longlong_as_double((long long) (k >> 63 ? k & ~(1ull << 63) : ~k));
        }
    }
    int nv;
    db1_scan<false, NT>(mine, sh, &nv);
    __syncthreads();
    if (wt && nv < n)
    {
        if (tid == 0) n_clusters[s] = -1;  // weights beside a NaN: left to the full scans
        return;
    }
    // ---- core points
    if (!wt)
    {
        for (int r = tid; r < nv; r += NT)
        {
            int lo, hi;
            db1_range(xs, 0, nv, xs[r], eps, lo, hi);
            run[r] = (double) (hi > lo ? hi - lo : 0) >= min_obs ? 0 : -1;
        }
    }
    else
    {
        // A neighbourhood's weight from prefix sums, where it is further from
        // min_obs than both this sum and db1_core_kernel's can be off (less
        // than 360 roundings of the weights' magnitudes together); the others
        // (and weights that are no numbers) are summed as that kernel does, so
        // that the decision is its own.  (8,192 points in one neighbourhood:
        // 0.36 ms, without weights 0.31; a warp summing each neighbourhood took
        // 24 ms on the one SM, the general launches take 0.74.)
        const int per = (nv + NT - 1) / NT, r0 = min(nv, tid * per), r1 = min(nv, r0 + per);
        double own = 0, mag = 0;
        for (int r = r0; r < r1; ++r)
        {
            const double v = wt[b + idx[r]];
            own += v;
            mag += fabs(v);
        }
        double before, total, mags;
        db1_scan_weights<NT>(own, mag, before, total, mags);
        for (int r = r0; r < r1; ++r)
        {
            ps[r] = before;
            before += wt[b + idx[r]];
        }
        __syncthreads();
        const double margin = mags * 0x1p-42;
        int core[kDb1Per];
#pragma unroll
        for (int u = 0; u < kDb1Per; ++u)
        {
            const int r = tid + u * NT;
            core[u] = -1;
            if (r < nv)
            {
                int lo, hi;
                db1_range(xs, 0, nv, xs[r], eps, lo, hi);
                const double d = (hi > lo ? (hi < nv ? ps[hi] : total) - ps[lo] : 0.0) - min_obs;
                core[u] = d > margin ? 0 : d < -margin ? -1 : -2;
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kDb1Per; ++u)
            if (tid + u * NT < nv) run[tid + u * NT] = core[u];
        __syncthreads();
        for (int r = w; r < nv; r += NT / 32)
        {
            if (run[r] != -2) continue;  // uniform across the warp
            int lo = 0, hi = 0;
            if (lane == 0) db1_range(xs, 0, nv, xs[r], eps, lo, hi);
            lo = __shfl_sync(0xffffffffu, lo, 0);
            hi = __shfl_sync(0xffffffffu, hi, 0);
            double acc = 0;
            for (int i = lo + lane; i < hi; i += 32) acc += wt[b + idx[i]];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0) run[r] = acc >= min_obs ? 0 : -1;
        }
    }
    __syncthreads();
    // ---- runs: each thread a piece of consecutive positions
    const int per = (nv + NT - 1) / NT, r0 = min(nv, tid * per), r1 = min(nv, r0 + per);
    int last = -1, tot;
    for (int r = r0; r < r1; ++r)
        if (run[r] == 0) last = r;
    int prev = db1_scan<true, NT>(last, sh, &tot);  // nearest core position before the piece
    const int prev0 = prev;
    int starts = 0;
    for (int r = r0; r < r1; ++r)
        if (run[r] == 0)
        {
            if (prev < 0 || !(xs[r] - xs[prev] <= eps)) ++starts;
            prev = r;
        }
    int nrun;
    int id = db1_scan<false, NT>(starts, sh, &nrun) - 1;  // the run the piece begins in
    prev = prev0;
    for (int r = r0; r < r1; ++r)
    {
        if (run[r] == 0)
        {
            if (prev < 0 || !(xs[r] - xs[prev] <= eps)) ++id;
            prev = r;
            run[r] = id;
        }
        else
            run[r] = -2 - prev;
    }
    for (int i = tid; i < nrun; i += NT) aux[i] = n;
    __syncthreads();
    for (int r = tid; r < nv; r += NT)
        if (run[r] >= 0) atomicMin(aux + run[r], idx[r]);
    __syncthreads();
    // ---- cluster number of a run: how many runs have a lower first point.
    // The first points in index order, by a scan over marks
    int root[kDb1Per];
#pragma unroll
    for (int u = 0; u < kDb1Per; ++u)
    {
        const int i = tid + u * NT;
        root[u] = i < nrun ? aux[i] : -1;
    }
    __syncthreads();
    for (int i = tid; i < n; i += NT) aux[i] = 0;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kDb1Per; ++u)
        if (root[u] >= 0) aux[root[u]] = 1;
    __syncthreads();
    const int pern = (n + NT - 1) / NT, i0 = min(n, tid * pern), i1 = min(n, i0 + pern);
    int marks = 0;
    for (int i = i0; i < i1; ++i) marks += aux[i];
    int base = db1_scan<false, NT>(marks, sh, &tot);
    for (int i = i0; i < i1; ++i)
    {
        const int m = aux[i];
        aux[i] = base;
        base += m;
    }
    __syncthreads();
    int num[kDb1Per];
#pragma unroll
    for (int u = 0; u < kDb1Per; ++u) num[u] = root[u] >= 0 ? aux[root[u]] : 0;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kDb1Per; ++u)
        if (root[u] >= 0) aux[tid + u * NT] = num[u];
    __syncthreads();
    // ---- labels: a core point's run; else the lowest cluster among the core
    // neighbours.  Those before it lie within eps of each other, so they are of
    // the nearest one's run, and so are those after it
    for (int r = tid; r < n; r += NT)
    {
        int lab = -1;
        if (r < nv)
        {
            if (run[r] >= 0) lab = aux[run[r]];
            else if (nrun > 0)
            {
                int lo, hi;
                db1_range(xs, 0, nv, xs[r], eps, lo, hi);
                const int p = -2 - run[r];
                int best = p >= lo ? aux[run[p]] : n;
                int q = r + 1;  // the first core position after r
                for (int e = hi; q < e;)
                {
                    const int m = (q + e) >> 1, v = run[m];
                    if ((v >= 0 ? m : -2 - v) > p) e = m;
                    else q = m + 1;
                }
                if (q < hi) best = min(best, aux[run[q]]);
                if (best < n) lab = best;
            }
        }
        labels[b + idx[r]] = lab;
    }
    if (tid == 0) n_clusters[s] = nrun;
}

}  // namespace mfgpu
