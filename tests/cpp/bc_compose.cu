// Host check of the one-pass boundary fill (bc_composable, bc_compose_value,
// BcShell): over random condition tables, every field kind and grids from
// three cells up, filling the ghost shell in place, its points in a random
// order, gives the bits of the edge by edge fill.
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <random>
#include <vector>

#include "lare_bc.cuh"

using namespace sams;

int main()
{
    std::mt19937_64 rng(5);
    int bad = 0, composed = 0;
    const int grids[][3] = {{3, 3, 3}, {4, 3, 6}, {3, 7, 5}, {9, 4, 3}, {2, 5, 4}};
    const int fields[] = {SAMS_F_RHO, SAMS_F_VX, SAMS_F_BX, SAMS_F_BY, SAMS_F_BZ};
    for (const auto &n : grids)
        for (int f : fields)
            for (int rep = 0; rep < 400; ++rep) {
                Geom g{};
                g.nx = n[0];
                g.ny = n[1];
                g.nz = n[2];
                g.zoff = 2;
                g.sy = n[2] + 5;
                g.sx = g.sy * (n[1] + 5);
                g.nelem = (long long)g.sx * (n[0] + 5);
                BcTable t{};
                for (int d = 0; d < 3; ++d) {
                    const int both = (int)(rng() % 6);  // periodic on both edges in a third of the dimensions
                    for (int e = 0; e < 2; ++e) {
                        const int kinds[5] = {SAMS_BC_NONE, SAMS_BC_PERIODIC, SAMS_BC_ZERO_GRADIENT, SAMS_BC_MIRROR, SAMS_BC_CLAMP};
                        t.kind[f][d][e] = (signed char)(both < 2 ? SAMS_BC_PERIODIC : kinds[rng() % 5]);
                        t.value[f][d][e] = 0.25 * (double)(rng() % 7);
                    }
                }
                if (!bc_composable(t, f, n)) continue;
                ++composed;
                std::vector<double> a((size_t)g.nelem), b;
                for (double &v : a) v = (double)(int64_t)(rng() >> 20) * 1e-9;
                b = a;
                for (int d = 0; d < 3; ++d)
                    for (int e = 0; e < 2; ++e) {
                        if (t.kind[f][d][e] == SAMS_BC_NONE) continue;
                        const BcEdge s = bc_edge_slab(g, f, d, e);
                        int q[3];
                        for (int i = s.lo[0]; i <= s.hi[0]; ++i)
                            for (int j = s.lo[1]; j <= s.hi[1]; ++j)
                                for (int k = s.lo[2]; k <= s.hi[2]; ++k) {
                                    q[0] = i;
                                    q[1] = j;
                                    q[2] = k;
                                    bc_edge_apply(a.data(), g, s, t, f, d, e, q);
                                }
                    }
                const BcShell sh(g, f);
                std::vector<int> order;
                int i, j, k, count = 0;
                while (sh.point(count, i, j, k)) order.push_back(count++);
                std::shuffle(order.begin(), order.end(), rng);
                for (int q : order) {
                    sh.point(q, i, j, k);
                    b[(size_t)box_off(g, i, j, k)] = bc_compose_value<2>(b.data(), g, t, f, i, j, k);
                }
                if (std::memcmp(a.data(), b.data(), a.size() * sizeof(double))) ++bad;
            }
    std::printf("{\"bad\": %d, \"composed\": %d}\n", bad, composed);
    return bad || composed < 200 ? 1 : 0;
}
