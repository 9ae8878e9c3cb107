// work_items_fast_selftest.cc -- the material phase's work items for the integer
// EOS (lg::build_material_items with fast_eos): every element's repetitions once, one
// writer each, inside the device arrays' capacity, split by the stated rule.
#include <cstdio>
#include <map>
#include <vector>

#include "lg_problem.h"

int main()
{
    const long long resident = 152LL * 1024;
    const int cases[][4] = {{1, 1, 1, 1},   {4, 4, 1, 30},  {20, 11, 1, 1}, {33, 11, 1, 0},
                            {45, 11, 1, 1}, {64, 11, 1, 1}, {64, 16, 2, 4}, {80, 11, 2, 1}};
    int bad = 0;
    for (const auto &c : cases) {
        const lg::Problem p = lg::build_sedov_scalars(c[0], c[1], c[2], c[3], 3.0, 1.0);
        std::vector<int> elem, rep, left(p.numElem, 0), writers(p.numElem, 0);
        const bool split = lg::build_material_items(p, resident, elem, rep, true);
        long long total = 0, most = 0;
        for (int r = 0; r < p.numReg; ++r)
            for (int e : p.regElemlist[r]) {
                const int n = lg::region_rep(r, p.numReg, p.cost);
                left[e] = n;
                total += n;
                if (n > most) most = n;
            }
        if (split != (most >= 2 && 5 * most * resident > 12 * total)) ++bad;
        if (elem.size() != rep.size() || (long long)elem.size() > p.numElem + 4 * resident) ++bad;
        for (size_t i = 0; i < elem.size(); ++i) {
            if (elem[i] < 0 || elem[i] >= p.numElem || rep[i] == 0) { ++bad; continue; }
            left[elem[i]] -= rep[i] > 0 ? rep[i] : -rep[i];
            writers[elem[i]] += rep[i] > 0;
        }
        for (int e = 0; e < p.numElem; ++e)
            if (left[e] != 0 || writers[e] != 1) ++bad;
        std::printf("s=%d r=%d b=%d c=%d: %zu items, %s, bad %d\n", c[0], c[1], c[2], c[3],
                    elem.size(), split ? "split" : "one per element", bad);
    }
    return bad != 0;
}
