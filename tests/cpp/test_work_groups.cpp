// The division of a correlator launch into work groups: plans without blocks
// or templates, single templates, and random banks, in which every template is
// in exactly one group of its channel.
#include <cstdio>
#include <random>
#include "work_groups.h"

using mfgpu::WorkGroups;

static int failures = 0;

static void check(const std::vector<int> &per_channel, int nblocks, long slots, int setup, bool pairs)
{
    std::vector<std::vector<int>> mine(per_channel.size());
    int nt = 0;
    for (size_t c = 0; c < mine.size(); ++c)
        for (int i = 0; i < per_channel[c]; ++i) mine[c].push_back(nt++);
    WorkGroups g;
    bool ok = mfgpu::divide_work(mine, nblocks, slots, setup, pairs, g);
    if (nblocks <= 0 || nt == 0)
        ok = ok && g.gch.empty() && g.gtb.empty() && g.gte.empty() && g.tids.empty();
    else
    {
        std::vector<int> seen(nt, 0);
        ok = ok && g.gch.size() <= 65535 && g.gtb.size() == g.gch.size() && g.gte.size() == g.gch.size();
        for (size_t i = 0; ok && i < g.gch.size(); ++i)
        {
            ok = g.gtb[i] < g.gte[i] && g.gte[i] <= (int) g.tids.size();
            for (int j = g.gtb[i]; ok && j < g.gte[i]; ++j)
            {
                bool mine_has = false;
                for (int t : mine[g.gch[i]]) mine_has |= t == g.tids[j];
                ok = mine_has && ++seen[g.tids[j]] == 1;
            }
        }
        for (int t = 0; ok && t < nt; ++t) ok = seen[t] == 1;
    }
    if (!ok)
    {
        std::printf("failed: %zu channels, %d templates, %d blocks, %ld slots, pairs %d\n", per_channel.size(), nt, nblocks,
                    slots, (int) pairs);
        ++failures;
    }
}

int main()
{
    for (bool pairs : {false, true})
    {
        // templates too long for any transform, a signal shorter than its templates
        for (int nblocks : {0, -3}) for (const auto &pc : {std::vector<int>{}, {0}, {0, 0}, {1}, {3, 0, 40}}) check(pc, nblocks, 152, 2, pairs);
        for (int nblocks : {1, 5000}) for (const auto &pc : {std::vector<int>{}, {0}, {1}, {0, 1, 0}, {7000}}) check(pc, nblocks, 304, 3, pairs);
    }
    std::mt19937 rng(7);
    auto below = [&](int n) { return (int) (rng() % (unsigned) n); };
    for (int i = 0; i < 400; ++i)
    {
        std::vector<int> pc(1 + below(i % 3 ? 20 : 300));
        for (int &m : pc) m = below(4) ? below(1 + below(60)) : 0;
        check(pc, 1 + below(i % 2 ? 8 : 3000), below(2) ? 152 : 304, 2 + below(2), below(2) != 0);
    }
    std::printf("%d failures\n", failures);
    return failures != 0;
}
