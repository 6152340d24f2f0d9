// Checks the rows that the resident path exchanges (fwi_gb300/csrc/resident_plan.h): over drawn batches,
// ResidentSet::slots is one more than the farthest exchange; in random orders of the CTAs' steps no copy of
// a row is overwritten before its readers have read it; and no launch takes more words than a context of
// that many shots, that window and those rows sets aside (res_exchange_words), 40 bytes a point of the
// shots in flight, 72 of a shot alone, at the kernels' row pitch.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../fwi_gb300/csrc/resident_plan.h"

using namespace fwi;

static std::mt19937 rng(11);
static int pick(int a, int b) { return a + (int)(rng() % (unsigned)(b - a + 1)); }

// Steps of the CTAs of shot [k0, k1) in random order: a CTA at step t (t > 0) needs the copies of step t of
// the rows in its halo; then it writes its rows' copies of step t + 1.  False: a reader found another step.
static bool ordered(const ResidentSet &set, int k0, int k1, int nz, int cpml)
{
    const ResidentGrid &g = set.grid;
    const int nzi = nz - 8, S = set.slots, steps = 40;
    std::vector<int> word((size_t)S * nzi, -1), owner(nzi), at(k1 - k0, 0);
    for (int c = k0; c < k1; c++)
        for (int r = g.row0[c]; r < g.row0[c] + g.nrow[c]; r++) owner[r] = c;
    // a step goes in two parts, as the kernels': halo in, rows out (other CTAs' between them)
    std::vector<char> read(k1 - k0, 0);
    const int lead = pick(k0, k1 - 1);  // runs ahead as far as it can
    for (long it = 0;; it++) {
        bool all = true, moved = false;
        for (int n = 0; n < k1 - k0; n++) {
            const int c = n == 0 && it % 3 ? lead : pick(k0, k1 - 1), i = c - k0;
            if (at[i] == steps) continue;
            const int t = at[i], row0 = g.row0[c], e = row0 + g.nrow[c], hr = res_halo(row0, e, nz, cpml);
            if (!read[i]) {
                bool come = true;
                for (int r = std::max(0, row0 - hr); r < std::min(nzi, e + hr); r++) {
                    if (owner[r] == c || t == 0) continue;
                    const int v = word[(size_t)(t % S) * nzi + r];
                    if (v > t) return false;  // overwritten unread
                    come = come && v == t;
                }
                read[i] = come;
                moved = moved || come;
            } else {
                for (int r = row0; r < e; r++) word[(size_t)((t + 1) % S) * nzi + r] = t + 1;
                at[i]++;
                read[i] = 0;
                moved = true;
            }
        }
        for (int a : at) all = all && a == steps;
        if (all) return true;
        if (it > 1000000) return false;
        (void)moved;
    }
}

int main()
{
    const size_t lim = 227 * 1024 - 1024;
    int plans = 0, sims = 0, reaches[kResReach + 1] = {};
    for (int it = 0; it < 4000; it++) {
        const int img = pick(0, 2) * 2, cpml = pick(0, 32), nz = cpml + 9 + pick(0, it % 3 ? 150 : 1100), nb = pick(0, 2) ? pick(1, 40) : 1;
        const int nx0 = 2 * cpml + 9 + pick(0, 640 - 2 * cpml - 9), n_sm = pick(0, 3) ? 152 : pick(8, 160);
        std::vector<int> w;
        const bool mixed = pick(0, 1);
        for (int s = 0; s < nb; s++) w.push_back(mixed ? 2 * cpml + 9 + pick(0, nx0 - 2 * cpml - 9) : nx0);
        std::vector<ResidentSet> sets;
        if (!resident_plan(w, nz, cpml, lim, n_sm, img, sets)) continue;
        plans++;
        for (const ResidentSet &set : sets) {
            const ResidentGrid &g = set.grid;
            int reach = 0;
            for (int a = 0; a < g.n; a++)
                for (int c = g.first[a]; c < g.first[a] + g.count[a]; c++) {
                    const int lo = g.row0[c], hi = lo + g.nrow[c], hr = res_halo(lo, hi, nz, cpml);
                    if (a != c && g.row0[a] < hi + hr && g.row0[a] + g.nrow[a] > lo - hr) reach = std::max(reach, std::abs(a - c));
                }
            reaches[reach]++;
            const int window = nx0 + (pick(0, 1) ? pick(0, 1500) : 0), shots = nb + pick(0, 3);
            if (set.slots != reach + 1 || set.slots > res_most_slots(nb) ||
                set.words(nz) + (size_t)kResSlots * kResMaxCtas > res_exchange_words(shots, window, nz)) {
                std::printf("FAILED slots %d reach %d: nz %d cpml %d nb %d nx %d\n", set.slots, reach, nz, cpml, nb, nx0);
                return 1;
            }
            for (int a = 0; a < g.n && sims < 3000; a += g.count[a]) {
                sims++;
                if (!ordered(set, a, a + g.count[a], nz, cpml)) {
                    std::printf("FAILED order: slots %d nz %d cpml %d nb %d nx %d\n", set.slots, nz, cpml, nb, nx0);
                    return 1;
                }
            }
        }
    }
    std::printf("OK: %d plans, %d orders; farthest exchange", plans, sims);
    for (int r : reaches) std::printf(" %d", r);
    std::printf("\n");
    return 0;
}
