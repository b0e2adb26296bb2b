// work_groups.h -- division of a correlator launch into work groups (host code
// only).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

namespace mfgpu {

// group g: templates tids[gtb[g]] .. tids[gte[g] - 1] of channel gch[g]
struct WorkGroups
{
    std::vector<int> gch, gtb, gte, tids;
};

// Work groups of one plan: each channel's templates of the bucket in one or
// more groups of about equal size, one CTA per (block, group).  The CTAs run
// on `slots` places in order, a CTA of m templates for setup + m units of
// time (a block's load and transform cost about as much as three templates
// of the FFT forms, two of the integer one; two teams take templates in
// pairs).  Few large groups leave the last wave of CTAs nearly empty, many
// small ones repeat the setup; so most channels are split alike and the last
// few into smaller groups, which run last and fill that wave: the division
// with the earliest end by this estimate.  (Groups halved until the grid had
// 1,216 CTAs, as before, against this: 64 channels x 12 blocks of 31 or 32
// templates of several lengths, 152 places, 692 -> 605 us; one channel x
// 603 blocks of 96 templates of one length, 304 places, 450 -> 395 us; 8
// channels x 173 blocks of 20 in FP64 1.73 -> 1.70 ms.)
// mine: the plan's templates of each channel.  A plan without templates or
// without blocks (every template in no transform, or longer than the signal) is
// never launched and has no groups.  False: more groups than a grid holds.
inline bool divide_work(const std::vector<std::vector<int>> &mine, int nblocks, long slots, int setup, bool pairs,
                        WorkGroups &gr)
{
    std::vector<int> used;
    int mx = 1;
    for (size_t c = 0; c < mine.size(); ++c)
    {
        if (mine[c].empty()) continue;
        used.push_back((int) c);
        mx = std::max(mx, (int) mine[c].size());
    }
    if (used.empty() || nblocks <= 0) return true;
    auto cost = [&](int m) { return setup + (!pairs ? m : m == 1 ? 1.5 : (m + 1) / 2 * 2.0); };
    // groups of at most G templates and their templates, channels [u0, u1)
    auto count = [&](int G, size_t u0, size_t u1, long &templates) {
        long ng = 0;
        templates = 0;
        for (size_t u = u0; u < u1; ++u)
        {
            const long m = (long) mine[used[u]].size();
            ng += (m + G - 1) / G;
            templates += m;
        }
        return ng;
    };
    auto mean_cost = [&](long ng, long templates) { return ng > 0 ? cost((int) ((2 * templates + ng) / (2 * ng))) : 0.0; };
    // end of n1 CTAs of cost c1 followed by n2 of cost c2
    auto finish = [&](double n1, double c1, double n2, double c2) {
        const double q = std::floor(n1 / slots), r = n1 - q * slots;
        double lo = r > 0 ? (q + 1) * c1 : q * c1;
        auto room = [&](double T) {
            return (slots - r) * std::floor(std::max(0.0, T - q * c1) / c2 + 1e-9) +
                   r * std::floor(std::max(0.0, T - (q + 1) * c1) / c2 + 1e-9);
        };
        if (n2 <= 0 || room(lo) >= n2) return lo;
        double hi = lo + c2 * (std::ceil(n2 / slots) + 1);
        for (int i = 0; i < 16; ++i)
        {
            const double m = 0.5 * (lo + hi);
            (room(m) >= n2 ? hi : lo) = m;
        }
        return hi;
    };
    double best = 1e300;
    int G1 = 0, G2 = 0, ntail = 0;
    const size_t nu = used.size();
    for (int k = 1, last = 0; k <= mx; ++k)
    {
        const int G = (mx + k - 1) / k;
        if (G == last) continue;
        last = G;
        long m1, m2;
        const long all = count(G, 0, nu, m1);
        // splits that leave every place many CTAs are only worse
        if (all > 65535 || (k > 1 && (double) nblocks * all > 64.0 * slots)) break;
        const size_t tmax = std::min<size_t>(nu, (size_t) (2 * slots / ((long) nblocks * k)) + 1);
        for (size_t tail = 0; tail <= tmax; tail = tail < 8 ? tail + 1 : tail + tail / 4)
            for (int h = 2; h <= 8; h *= 2)
            {
                const int Gt = (G + h - 1) / h;
                const long g1 = count(G, 0, nu - tail, m1), g2 = count(Gt, nu - tail, nu, m2);
                if (g1 + g2 > 65535) break;
                const double c1 = mean_cost(g1, m1), c2 = mean_cost(g2, m2);
                const double n1 = (double) nblocks * g1, n2 = (double) nblocks * g2;
                if (n1 * c1 + n2 * c2 >= best * slots) continue;
                const double T = finish(n1, c1, n2, c2);
                if (T < best * (1 - 1e-6))
                {
                    best = T;
                    G1 = G;
                    G2 = Gt;
                    ntail = (int) tail;
                }
                if (tail == 0) break;
            }
    }
    if (G1 == 0) return false;
    for (size_t u = 0; u < nu; ++u)
    {
        const std::vector<int> &m = mine[used[u]];
        const int G = u + ntail >= nu ? G2 : G1, ng = ((int) m.size() + G - 1) / G;
        // about equal parts (pairs stay together)
        const int unit = pairs && G > 1 ? 2 : 1, units = ((int) m.size() + unit - 1) / unit;
        for (int i = 0; i < ng; ++i)
        {
            const size_t j0 = (size_t) unit * ((long) units * i / ng);
            const size_t j1 = std::min(m.size(), (size_t) unit * ((long) units * (i + 1) / ng));
            if (j0 >= j1) continue;
            gr.gch.push_back(used[u]);
            gr.gtb.push_back((int) gr.tids.size());
            gr.tids.insert(gr.tids.end(), m.begin() + (long) j0, m.begin() + (long) j1);
            gr.gte.push_back((int) gr.tids.size());
        }
    }
    return true;
}

}  // namespace mfgpu
