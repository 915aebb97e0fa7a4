// Host check of the fused kernels' tilings (lare_march.cuh): over a range of
// grids, every own point of each phase falls to exactly one thread, and every
// ring cell or window point stays inside the block's store.
#include <cstdio>
#include <vector>

#include "lare_march.cuh"

using namespace sams;

static int bad = 0;
static void fail(const char *what, int nx, int ny, int nz)
{
    if (bad++ < 20) std::printf("%s %dx%dx%d\n", what, nx, ny, nz);
}

static void check_march(int nx, int ny, int nz, int grow, int sm_blocks)
{
    const int ni = nx + grow, nj = ny + grow, nk = nz + grow;
    const march::MarchTile m = march::march_tile(nk, nj, ni, sm_blocks);
    if (m.W * m.R > march::kMThreads || m.W < 2 || m.R < 2 || m.MI < 1) fail("march shape", nx, ny, nz);
    std::vector<int> hits((size_t)ni * nj * nk, 0);
    for (int b = 0; b < m.blocks; ++b)
        for (int t = 0; t < march::kMThreads; ++t) {
            const march::MarchAt a = march::march_at(m, b, t);
            if (a.own && !a.cell) fail("own point without a ring cell", nx, ny, nz);
            const int j = a.j0 + a.pj, k = a.k0 + a.pk;
            if (!a.own || j >= nj || k >= nk) continue;
            // the cells it reads at +1 in y and z are other threads' ring cells
            if (t + m.W + 1 >= m.W * m.R) fail("ring", nx, ny, nz);
            for (int i = a.i0; i < a.i0 + m.MI && i < ni; ++i) ++hits[((size_t)i * nj + j) * nk + k];
        }
    for (int h : hits)
        if (h != 1) { fail("march cover", nx, ny, nz); return; }
}

// nd + 1 points along the sweep, (na + 1) x nk transverse points
static void check_win(int nd, int na, int nk, int sm_blocks)
{
    const march::WinTile w = march::win_tile(nd + 1, (long long)(na + 1) * nk, 3, sm_blocks);
    if (w.S < 1 || w.S > ops::kWinS) fail("window length", nd, na, nk);
    std::vector<int> hits((size_t)(nd + 1) * (na + 1) * nk, 0);
    for (int b = 0; b < w.blocks; ++b)
        for (int t = 0; t < ops::kWinThreads; ++t) {
            const march::WinAt p = march::win_at(w, b, t, nd, nk);
            if (p.a > na) continue;
            for (int s = p.s0 + p.sl; s <= p.s1; s += ops::kWinThreads / ops::kWinK)
                ++hits[((size_t)s * (na + 1) + p.a) * nk + p.k];
        }
    for (int h : hits)
        if (h != 1) { fail("window cover", nd, na, nk); return; }
}

static void check_z(int nx, int ny, int nz)
{
    const march::ZTile z = march::z_tile(nz, (long long)(nx + 2) * (ny + 2));
    if (z.S < 1 || z.L < 1 || z.L * (z.S + 3) > march::kZCtThreads) fail("z shape", nx, ny, nz);
    Geom g{};
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    std::vector<int> hits((size_t)(nx + 2) * (ny + 2) * (nz + 1), 0);
    for (int b = 0; b < z.blocks; ++b)
        for (int t = 0; t < march::kZCtThreads; ++t) {
            const march::ZAt p = march::z_at(z, b, t, g);
            if (!p.own) continue;
            if (p.k < 0 || p.k > nz || t < 1 || t + 2 >= march::kZCtThreads) fail("z range", nx, ny, nz);
            else ++hits[((size_t)p.i * (ny + 2) + p.j) * (nz + 1) + p.k];
        }
    for (int h : hits)
        if (h != 1) { fail("z cover", nx, ny, nz); return; }
}

int main()
{
    const int sizes[] = {1, 2, 3, 4, 7, 8, 21, 31, 32, 47, 64, 97};
    const int long_z[] = {200, 256, 284, 285, 700};
    auto all = [](int nx, int ny, int nz) {
        for (int sm_blocks : {1, 444, 740}) {
            for (int grow : {1, 2, 3, 5}) check_march(nx, ny, nz, grow, sm_blocks);
            check_win(nx, ny, nz + 1, sm_blocks);
            check_win(nx, ny + 1, nz + 2, sm_blocks);
        }
        check_z(nx, ny, nz);
    };
    for (int nx : {1, 5, 33})
        for (int ny : sizes)
            for (int nz : sizes) all(nx, ny, nz);
    for (int nz : long_z) all(9, 6, nz);
    all(300, 5, 4);
    std::printf("{\"bad\": %d}\n", bad);
    return bad ? 1 : 0;
}
