// Checks the resident path's plan (fwi_gb300/csrc/resident_plan.h) over a sweep of windows, grid
// heights, layer widths and batches: every launch within the SMs, threads, registers and shared
// memory; rows covered once; every index the kernels form inside its array; every halo row a CTA
// reads published by an owner at most kResReach CTAs away, and no copy of an exchanged row overwritten
// before its readers are done (the most steps such CTAs can be apart).
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../fwi_gb300/csrc/resident_plan.h"

using namespace fwi;

#define CHECK(c)                                                                                             \
    do {                                                                                                     \
        if (!(c)) {                                                                                          \
            std::printf("FAILED %s: nx %d nz %d cpml %d adjoint %d (line %d)\n", #c, nx, nz, cpml, adjoint, __LINE__); \
            return false;                                                                                    \
        }                                                                                                    \
    } while (0)

static long plans = 0, launches = 0, bands = 0;

static bool check_cta(const ResidentSet &set, int c, int nx, int nz, int cpml, int adjoint, int pitch)
{
    const int pt = set.pitch;
    const ResidentGrid &g = set.grid;
    const int nzi = nz - 8, nrow = g.nrow[c], row0 = g.row0[c], nq = res_pairs(nx, cpml).nq;
    const bool bottom = res_bottom(row0 + nrow, nz, cpml);
    const int hr = res_halo(row0, row0 + nrow, nz, cpml), lanes = g.lanes[c], R = (nrow + lanes - 1) / std::max(lanes, 1);
    const ResShape shape = res_shape(pt);
    const ResPairs P = res_pairs(nx, cpml);
    CHECK(lanes >= 1 && P.threads(lanes) <= set.threads && set.threads <= shape.threads && set.threads % 32 == 0);
    CHECK(R >= 1 && R <= (adjoint ? shape.adj_rows : shape.fwd_rows));
    // every pair once: the side pairs are those within reach of a side layer, in order
    std::vector<int> cols;
    for (int t = 0; t < P.nside; t++) cols.push_back(4 + 2 * (t < P.nleft ? t : P.nq - P.nside + t));
    for (int x : cols) CHECK(x < cpml + 4 || x + 1 > nx - cpml - 5);
    for (int t = 0; t < P.nq - P.nside; t++) {
        cols.push_back(4 + 2 * (P.nleft + t));
        CHECK(cpml <= 4 || !(cols.back() < cpml + 4 || cols.back() + 1 > nx - cpml - 5));
    }
    std::sort(cols.begin(), cols.end());
    for (int q = 0; q < (int)cols.size(); q++) CHECK(cols[q] == 4 + 2 * q);
    const ResGeom G = res_geom(nx, cpml);
    CHECK(res_floats(pt, nrow, hr > kRad, bottom, adjoint) * sizeof(float) <= set.smem);
    CHECK(pt % 4 == 0 && kResSide % 4 == 0 && pt >= nx);
    // rows with a z memory variable or within its reach lie in bottom bands
    for (int r = row0; r < row0 + nrow; r++) CHECK(!(cpml > 4 && 4 + r >= nz - cpml - 4) || bottom);
    // column pairs: windows inside a row, side windows inside the band storage
    for (int q = 0; q < nq; q++) {
        const int ix = 4 + 2 * q;
        CHECK(ix <= nx - 5 && ix + 5 < pt && ix + 1 < pitch);
        if (cpml > 4 && (ix < cpml + 4 || ix + 1 > nx - cpml - 5)) {
            const int a = G.col(ix);
            CHECK(a - 4 >= 0 && a + 5 < kResSide && a % 2 == 0);
            for (int k = -4; k < 6; k++) CHECK(G.col(ix + k) == a + k);
        }
    }
    CHECK(4 + 2 * nq >= nx - 4);
    const int nbx = cpml > 4 ? std::min(2 * (cpml - 4), nx - 8) : 0;
    for (int k = 0; k < nbx; k++) {  // the side-layer columns, each once, inside both storages
        const int col = k < nbx / 2 ? 4 + k : nx - 4 - nbx + k;
        CHECK((col < cpml || col > nx - cpml - 1) && col >= 4 && col < nx - 4);
        CHECK(G.col(col) >= 0 && G.col(col) < kResSide && col + 4 < pt);
    }
    // halo rows: published by their owner, at most kResReach CTAs away, and the window rows inside
    for (int h = 0; h < 2 * hr; h++) {
        const int r = h < hr ? h - hr : nrow + h - hr, gi = row0 + r;
        if (gi < 0 || gi >= nzi) continue;
        int owner = -1;
        for (int k = g.first[c]; k < g.first[c] + g.count[c]; k++)
            if (gi >= g.row0[k] && gi < g.row0[k] + g.nrow[k]) owner = k;
        CHECK(owner >= 0 && owner != c && std::abs(owner - c) <= kResReach);
        int lo = 0, hi = 0;
        for (int k = std::max((int)g.first[c], owner - kResReach); k < std::min(g.first[c] + g.count[c], owner + kResReach + 1); k++) {
            if (k == owner) continue;
            const int a = g.row0[k], e = a + g.nrow[k], hk = res_halo(a, e, nz, cpml);
            if (k < owner) lo = std::max(lo, e + hk - g.row0[owner]);
            else hi = std::max(hi, g.row0[owner] + g.nrow[owner] - (a - hk));
        }
        const int ro = gi - g.row0[owner];
        CHECK(ro < lo || ro >= g.nrow[owner] - hi);
        // a CTA writing step t + 1 is followed by CTAs d apart that have read step t - d
        CHECK(std::abs(owner - c) + 1 <= kResSlots);
    }
    // the threads' windows: rows r0 - 4 .. of every segment that owns rows
    for (int r0 = 0; r0 < nrow; r0 += R) CHECK(r0 - 4 >= -hr && r0 + 3 < nrow + hr && std::min(r0 + R, nrow) + 3 < nrow + hr);
    // z memory variables recomputed 4 rows either side: their taps inside the halo
    const int zb = nz - cpml, iz0 = 4 + row0;
    const int b0 = std::max(std::max(4, zb), iz0 - kRad) - iz0, b1 = std::min(nz - 4, iz0 + nrow + kRad) - iz0;
    if (bottom)
        for (int r = b0; r < b1; r++) CHECK(r >= -kRad && r < nrow + kRad && r - 4 >= -hr && r + 4 < nrow + hr);
    bands++;
    return true;
}

static bool check(const std::vector<int> &w, int nz, int cpml, int adjoint, size_t lim, int n_sm, bool expect)
{
    const int nx = w[0];
    std::vector<ResidentSet> sets;
    const bool ok = resident_plan(w, nz, cpml, lim, n_sm, adjoint, sets);
    CHECK(!expect || ok);
    if (!ok) return true;
    plans++;
    int pitch = 0;
    for (int x : w) pitch = std::max(pitch, (x + 31) / 32 * 32);
    std::vector<int> rows(w.size(), 0), seen(w.size(), 0);
    for (const ResidentSet &set : sets) {
        const ResidentGrid &g = set.grid;
        launches++;
        CHECK(g.n >= 1 && g.n <= n_sm && g.n <= kResMaxCtas && set.smem <= lim);
        for (int c = 0; c < g.n; c++) {
            const int s = g.shot[c];
            CHECK(s < (int)w.size() && g.xs[c] < set.nshots);
            CHECK(c >= g.first[c] && c < g.first[c] + g.count[c] && g.first[c] + g.count[c] <= g.n);
            CHECK(g.shot[g.first[c]] == s && g.nrow[c] >= (g.count[c] > 1 ? res_min_rows((int)w.size()) : 1));
            CHECK(g.row0[c] == rows[s]);
            rows[s] += g.nrow[c];
            if (c == g.first[c]) seen[s]++;
            if (!check_cta(set, c, w[s], nz, cpml, adjoint, pitch)) return false;
        }
    }
    for (size_t s = 0; s < w.size(); s++) CHECK(rows[s] == nz - 8 && seen[s] == 1);
    return true;
}

int main()
{
    const size_t lim = 227 * 1024 - 1024;
    std::mt19937 rng(7);
    bool ok = true;
    auto pick = [&](int a, int b) { return a + (int)(rng() % (unsigned)(b - a + 1)); };
    for (int adj : {0, 4, 2}) {  // the forward, the adjoint with 4- and 2-byte images
        // the benchmark's and the tests' grids, which have to fit
        for (int nb : {1, 2, 5, 8, 32}) {
            ok = ok && check(std::vector<int>(nb, 209), 209, 20, adj, lim, 152, true);
            ok = ok && check(std::vector<int>(nb, 609), 309, 20, adj, lim, 152, adj != 0);
            ok = ok && check(std::vector<int>(nb, 72), 56, 12, adj, lim, 152, true);
        }
        for (int nx = 33; nx < 130 && ok; nx++)
            for (int cpml : {4, 5, 8, 12})
                for (int nz : {cpml + 9, 24, 37, 60})
                    if (nx >= 2 * cpml + 9 && nz >= cpml + 9) ok = ok && check({nx}, nz, cpml, adj, lim, 152, false);
        for (int k = 0; k < 1500 && ok; k++) {  // batches of one or several widths, other device sizes
            const int cpml = pick(0, 32), nz = cpml + 9 + pick(0, 900), nb = pick(1, 40), n_sm = pick(0, 3) ? 152 : pick(8, 160);
            const int nx0 = 2 * cpml + 9 + pick(0, 1300);
            std::vector<int> w;
            const bool mixed = pick(0, 1);
            for (int s = 0; s < nb; s++) w.push_back(mixed ? 2 * cpml + 9 + pick(0, nx0 - 2 * cpml - 9) : nx0);
            ok = ok && check(w, nz, cpml, adj, lim, n_sm, false);
        }
    }
    std::printf("%s: %ld plans, %ld launches, %ld bands\n", ok ? "OK" : "FAILED", plans, launches, bands);
    return ok ? 0 : 1;
}
