// The resident path's plan (prop_resident.cuh): which shots of a batch share the GPU, which rows
// of each shot a CTA holds, and the shared memory each CTA needs.  Host code (with the CUDA
// headers' qualifiers), so that the plan can be checked on the CPU.
//
// A launch holds one CTA per SM.  A CTA owns a band of interior rows of one shot's window, every
// column; a shot's CTAs exchange the few edge rows their z-stencils need.  The shots of a batch
// that do not fit on the SMs at once run in several sets, one launch after another.
#pragma once

#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdint>
#include <map>
#include <vector>

#include "common.cuh"

namespace fwi {

constexpr int kResMaxCtas = 160;  // CTAs of a launch (one per SM)
// Rows of a CTA at least: 1 for a shot that has the GPU to itself, 2 beside others, which leave it
// fewer CTAs, better spent on shorter upper bands.  Microseconds a forward / adjoint step with 3, 2, 1:
// one C1 shot 3.03 / 3.47, 2.84 / 3.27, 2.75 / 3.20, one 400 x 200 5.2 / 4.9, 5.0 / 4.4, 4.8 / 3.9, the adjoint
// of one 609 x 309 8.5, 6.7, 6.6; 4 shots of 300 x 200 4.6 / 4.0, 4.5 / 4.0, 5.0 / 4.7.
constexpr int kResMinRows = 1;
inline int res_min_rows(int nshots) { return nshots == 1 ? kResMinRows : 2; }
constexpr int kResReach = (2 * kRad + kResMinRows - 1) / kResMinRows;  // a halo comes from so many CTAs either side at most
constexpr int kResSlots = 16;     // copies of the exchanged maxima (step modulo kResSlots)
static_assert(kResSlots > kResReach && (kResSlots & (kResSlots - 1)) == 0, "copies of the exchanged maxima");
// Copies of the exchanged rows a launch needs at most (ResidentSet::slots: its farthest exchange and one).
inline int res_most_slots(int nshots) { return (2 * kRad + res_min_rows(nshots) - 1) / res_min_rows(nshots) + 1; }
constexpr int kResSide = 96;      // floats of a side array's row
constexpr int kResMaxCpml = 32;   // the widest layer whose side columns fit one
constexpr int kResFwdOwn = 5, kResAdjOwn = 8;    // own-row arrays
constexpr int kResFwdSide = 3, kResAdjSide = 5;  // side arrays
// Shared row pitches the kernels are compiled for, and at each the threads of a CTA at most (the
// fewer, the more registers each) and the rows a thread holds at most (the more, the fewer launches a
// batch takes; past these they spill).  Microseconds a forward / adjoint step, to 320 columns with 512
// threads x 4 rows -> 448 x 5 / 4: one 209 x 209 3.15 / 3.50 -> 3.05 / 3.48, 8 of them 4.9 / 4.6 -> 4.8 / 4.6,
// 16 of 300 x 300 18.0 / 36.0 -> 14.1 / 33.3 (448 x 6: 11.5 / 30.2, but one 209 x 209 3.22); beyond with
// 640 x 6 forward -> 640 x 4: 8 of 400 x 200 8.7 -> 7.4.
constexpr int kResPitches[] = {96, 160, 224, 320, 400, 512, 640};
constexpr int kResFwdPitch = 400;  // the widest forward kernel's
struct ResShape {
    int threads, fwd_rows, adj_rows;
};
__host__ __device__ constexpr ResShape res_shape(int pitch)
{
    return pitch <= 320 ? ResShape{448, 5, 4} : ResShape{640, 4, 4};
}

// The pitch for windows nx wide (rows end at a multiple of 4), 0: none.
inline int res_pitch(int nx, bool forward)
{
    for (int p : kResPitches)
        if ((nx + 3) / 4 * 4 <= p) return forward && p > kResFwdPitch ? 0 : p;
    return 0;
}

// CTA c of a launch: rows row0 .. row0 + nrow of the interior of shot `shot`, which is the xs-th
// of the launch and whose CTAs are first .. first + count; lanes: the segments its rows are split in.
struct ResidentGrid {
    int n;
    unsigned short shot[kResMaxCtas], xs[kResMaxCtas], first[kResMaxCtas], count[kResMaxCtas], row0[kResMaxCtas],
        nrow[kResMaxCtas], lanes[kResMaxCtas];
};

// One launch: its grid, shared row pitch (the widest window's), threads and dynamic shared memory.
struct ResidentSet {
    ResidentGrid grid;
    int pitch, threads, nshots;
    int slots;  // copies of the exchanged rows (step modulo slots)
    size_t smem;
    // words of the exchanged rows: [shot][slots][nz][pitch]
    size_t words(int nz) const { return (size_t)nshots * slots * nz * pitch; }
};

// Words a context's batches exchange at most: shots in flight, window and rows of the grid.  (0: more
// rows than the CTAs hold at the narrowest pitch in 227 KB each, forward rows of own and haloed arrays.)
inline size_t res_exchange_words(int max_shots, int window, int nz)
{
    if (nz - 8 > kResMaxCtas * (int)(232448 / ((kResFwdOwn + 2) * sizeof(float) * kResPitches[0]))) return 0;
    int pt = 0;
    for (int p : kResPitches)
        if (!pt && ((window + 3) / 4 * 4 <= p || p == 640)) pt = p;
    const size_t row = (size_t)nz * pt, one = res_most_slots(1) * row, all = (size_t)max_shots * res_most_slots(2) * row;
    return (max_shots > 1 && all > one ? all : one) + (size_t)kResSlots * kResMaxCtas;
}

// Whose roundings of the CPML terms a forward launch follows: the cluster path's, those of the layer tiles
// that advance psi themselves, those of the layer tiles after the strip pass.
enum ResOrder { kResAsCluster, kResAsInline, kResAsStrip };

// Arguments of one forward launch: global steps [g0, g1) of a batch whose clock runs to ntb.
struct ResFwdArgs {
    int ntb, g0, g1;
    int img_first;   // images are kept from this step on (>= g1: none), in slot
    int period;      // g - seg period + (seg & 1) period of step g, seg = g / period (nt_max: slot g)
    int load_ck;     // checkpoint to start from, or -1: zero state
    int save_ck;     // checkpoints 0 .. save_ck - 1 are written (step k period)
    int order;       // ResOrder: the path this batch would otherwise take
    int plain_images;  // images of the plain stencils (reference mode)
    float *ck;       // [checkpoint][8][ck_stride]
    long ck_stride;
    uint64_t *x;     // exchanged rows: [xs][slots][nz][shared row pitch] words
    int slots;
    uint64_t *w;     // exchanged maxima: [kResSlots][kResMaxCtas] words
    unsigned tag0;   // a word of step g carries tag0 + g
};

// One adjoint launch: iterations [j0, j1); images at slot (global step - img_base).
struct ResAdjArgs {
    int ntb, j0, j1, img_base;
    uint64_t *x;
    int slots;
    unsigned tag0;
};

// The side layers' CPML arrays keep only the columns near the layers: column ix at ix (left,
// ix < wl) or wl + ix - xr0 (right); windows too narrow for two separate sides keep whole rows.
struct ResGeom {
    int wl, xr0;
    __host__ __device__ int col(int ix) const { return ix < wl ? ix : wl + ix - xr0; }
};

__host__ __device__ inline ResGeom res_geom(int nx, int cpml)
{
    ResGeom g;
    g.wl = (cpml + 3) / 4 * 4 + 12;      // pairs with a column < cpml + 4, their 10-wide windows
    g.xr0 = (nx - cpml - 5) / 2 * 2 - 4;  // the same from the right
    if (g.xr0 < g.wl) {
        g.wl = kResSide;
        g.xr0 = 0;
    }
    return g;
}

// Whether a band ending before interior row `end` holds a row whose update reads the bottom
// layer's z memory variables (from 4 rows above the layer on).
__host__ __device__ inline bool res_bottom(int end, int nz, int cpml) { return cpml > 4 && 4 + end > nz - cpml - 4; }

// Halo rows of the z-stencil field of the band [row0, end): 4, or 8 where it recomputes z memory
// variables of its neighbours from it (bottom bands but one that holds the whole bottom zone).
__host__ __device__ inline int res_halo(int row0, int end, int nz, int cpml)
{
    return res_bottom(end, nz, cpml) && (4 + row0 > nz - cpml - 4 || end < nz - 8) ? 2 * kRad : kRad;
}

// Floats of a CTA's shared arrays at row pitch pt.  Forward: F (haloed) and P, two levels of each;
// the three models; psi_x, zeta_x and what they add to Dxx P (side columns); bottom bands also psi_z
// (4 rows either side), zeta_z and what they add to Dzz F.  Adjoint: u_z (haloed) and u_x, two
// levels of each; the three models and three gradients; Y_x, Z_x, a Y_x, u_x at layer points,
// -Dx(a Y_x); bottom bands Y_z, Z_z, -Dz(a Y_z); the 16-bit images of a step.  And the CPML tables.
// img_bytes: bytes of an image value (0: the forward).
__host__ __device__ inline size_t res_floats(int pt, int nrow, bool wide_halo, bool bottom, int img_bytes)
{
    size_t rows = (size_t)(img_bytes ? kResAdjOwn : kResFwdOwn) * nrow + 2 * (nrow + (wide_halo ? 4 : 2) * kRad);
    if (bottom) rows += (size_t)3 * nrow + 2 * kRad;
    size_t n = rows * pt + (size_t)((img_bytes ? kResAdjSide : kResFwdSide) * nrow + 2) * kResSide +
               (size_t)2 * (nrow + 2 * kRad);
    if (img_bytes == 2) n = (n + 3) / 4 * 4 + (size_t)nrow * pt;
    return n;
}

// Column pairs of a window: nq in all, nside of them (nleft left) within reach of a side layer.  A
// CTA's threads: whole warps for the side pairs of every row segment, then the others'.
struct ResPairs {
    int nq, nleft, nside;
    __host__ __device__ int side_threads(int lanes) const { return (nside * lanes + 31) / 32 * 32; }
    __host__ __device__ int threads(int lanes) const
    {
        return side_threads(lanes) + ((nq - nside) * lanes + 31) / 32 * 32;
    }
};
__host__ __device__ inline ResPairs res_pairs(int nx, int cpml)
{
    ResPairs p;
    p.nq = (nx - 8 + 1) / 2;
    p.nleft = p.nside = 0;
    if (cpml > 4) {
        p.nleft = (cpml + 1) / 2 < p.nq ? (cpml + 1) / 2 : p.nq;  // pairs at 4 + 2 k < cpml + 4
        int right = (nx - cpml - 8) / 2;                         // first pair with 4 + 2 k + 1 > nx - cpml - 5
        if (right < p.nleft) right = p.nleft;
        p.nside = p.nleft + (right < p.nq ? p.nq - right : 0);
    }
    return p;
}

// Row segments a CTA's threads can take.
inline int res_lanes(int nx, int pt, int cpml)
{
    const ResPairs p = res_pairs(nx, cpml);
    int n = 0;
    while (p.nq > 0 && n < 64 && p.threads(n + 1) <= res_shape(pt).threads) n++;
    return n;
}

// The most rows a CTA of this window can hold (threads, registers, shared memory).
inline int res_row_cap(int nx, int pt, int cpml, bool wide_halo, bool bottom, int img_bytes, size_t smem_limit)
{
    const ResShape sh = res_shape(pt);
    const int most = res_lanes(nx, pt, cpml) * (img_bytes ? sh.adj_rows : sh.fwd_rows);
    if (!pt || cpml > kResMaxCpml) return 0;
    int n = 0;
    while (n < most && res_floats(pt, n + 1, wide_halo, bottom, img_bytes) * sizeof(float) <= smem_limit) n++;
    return n;
}

// Rows of a window's n CTAs: `upper` bands over the rows above the bottom zone, then `lower`
// bands over the zone (and `extra` rows above it).  cost: the largest band's, in rows; a row of a
// bottom band counts more (the recomputed z memory variables and their two block barriers).
struct ResPartition {
    int upper = 0, lower = 0, extra = 0;
    double cost = -1.0;  // < 0: no partition
};

// What a window's CTAs can take: row segments, and rows of an upper band, of the only bottom band, of
// one of several.
struct ResCaps {
    int lanes, upper, only, lower;
};
inline ResCaps res_caps(int nx, int pt, int cpml, int img_bytes, size_t smem_limit)
{
    return {std::max(1, res_lanes(nx, pt, cpml)), res_row_cap(nx, pt, cpml, false, false, img_bytes, smem_limit),
            res_row_cap(nx, pt, cpml, false, true, img_bytes, smem_limit),
            res_row_cap(nx, pt, cpml, true, true, img_bytes, smem_limit)};
}

// The cheapest partition into at most n CTAs, for every n to `most`.  A cost depends on the tallest upper
// and the tallest lower band only, so that for each of these heights the fewest CTAs are tried (a few
// hundred partitions; all counts and splits, a thousand times as many, took 0.3 ms a width).
inline std::vector<ResPartition> res_partitions(const ResCaps &cap, int nz, int cpml, int most, int min_rows)
{
    const int nzi = nz - 8, zone = cpml > 4 ? std::min(nzi, cpml) : 0;
    std::vector<ResPartition> best(std::max(1, most + 1));
    // rows a thread takes in turn
    auto turns = [&](int rows) { return (double)((rows + cap.lanes - 1) / cap.lanes); };
    auto tallest = [](int rows, int n) { return (rows + n - 1) / n; };
    for (int extra = 0; extra <= (zone ? std::min(nzi - zone, 12) : 0); extra++) {
        const int low = zone + (zone ? extra : 0), rest = nzi - low;
        for (int lower = zone ? 1 : 0, next; lower <= (zone ? std::min(most, low / min_rows) : 0); lower = next) {
            const int lmax = lower ? tallest(low, lower) : 0;
            // the next count with a lower tallest band (one bottom band costs otherwise than several)
            next = lower <= 1 ? lower + 1 : lmax > 1 ? tallest(low, lmax - 1) : most + 1;
            if (lmax > (lower == 1 ? cap.only : cap.lower)) continue;
            const double cl = lower ? turns(lmax) * 1.5 + turns(lower == 1 ? lmax : lmax + 8) * 0.7 + 1.5 : 0.0;
            auto offer = [&](int upper, int umax) {
                if (upper + lower < 1 || upper + lower > most) return;
                const double cu = turns(umax), c = std::max(cu, cl) + 1e-2 * (cu + cl) + 1e-3 * (umax + lmax);
                ResPartition &p = best[upper + lower];
                if (p.cost >= 0 && c >= p.cost - 1e-9) return;
                p.upper = upper;
                p.lower = lower;
                p.extra = extra;
                p.cost = c;
            };
            if (rest == 0) {
                offer(0, 0);
                continue;
            }
            for (int umax = std::min(cap.upper, rest); umax >= 1;) {
                const int upper = tallest(rest, umax);
                if (rest / upper < min_rows || upper + lower > most) break;
                offer(upper, tallest(rest, upper));
                umax = tallest(rest, upper) - 1;
            }
        }
    }
    for (int n = 1; n <= most; n++)
        if (best[n - 1].cost >= 0 && (best[n].cost < 0 || best[n].cost > best[n - 1].cost)) best[n] = best[n - 1];
    return best;
}

// Row counts of a partition, top band first.
inline std::vector<int> res_bands(const ResPartition &p, int nz, int cpml)
{
    const int nzi = nz - 8, zone = (cpml > 4 ? std::min(nzi, cpml) : 0) + p.extra, rest = nzi - zone;
    std::vector<int> r;
    for (int k = 0; k < p.upper; k++) r.push_back(rest / p.upper + (k < rest % p.upper ? 1 : 0));
    for (int k = 0; k < p.lower; k++) r.push_back(zone / p.lower + (k < zone % p.lower ? 1 : 0));
    return r;
}

// The partitions of a window's width, and those of the widths seen so far, which a context keeps for its
// grid (about kResWidths at most; 10 to 25 microseconds a width to make).
struct ResWidth {
    int least = 0;                   // the fewest CTAs that hold the window (0: none do)
    std::vector<ResPartition> part;  // by CTA count
    std::vector<int> more;           // the next count that lowers the cost (past the last: none)
};
using ResWidths = std::map<long, ResWidth>;
constexpr size_t kResWidths = 512;

// The launches of a batch whose shots have windows nx[0], nx[1], ...: consecutive shots share a
// launch while their fewest CTAs fit on n_sm SMs (windows of one width: the same number in each),
// then the SMs left go one by one to the shot with the costliest band.  False if some window does
// not fit at all.  `kept`: the widths of earlier plans for the same grid, layer, limit and SMs.
inline bool resident_plan(const std::vector<int> &nx, int nz, int cpml, size_t smem_limit, int n_sm, int img_bytes,
                          std::vector<ResidentSet> &out, ResWidths *kept = nullptr)
{
    out.clear();
    int wmax = 0;
    for (int w : nx) wmax = std::max(wmax, w);
    const int pt = res_pitch(wmax, img_bytes == 0);
    const int nb = (int)nx.size(), nzi = nz - 8, sms = std::min(n_sm, kResMaxCtas), min_rows = res_min_rows(nb), most = std::min(sms, nzi / min_rows);
    if (nzi < 1) return false;
    ResWidths own, &widths = kept ? *kept : own;
    if (widths.size() > kResWidths) widths.clear();
    std::vector<const ResWidth *> of(nb);  // each shot's
    bool uniform = true;
    for (int k = 0; k < nb; k++) {
        ResWidth &x = widths[(long)nx[k] << 32 | pt << 8 | img_bytes << 4 | min_rows];
        if (x.part.empty()) {
            x.part = res_partitions(res_caps(nx[k], pt, cpml, img_bytes, smem_limit), nz, cpml, most, min_rows);
            for (int n = 1; n <= most && !x.least; n++)
                if (x.part[n].cost >= 0) x.least = n;
            x.more.assign(most + 2, most + 1);
            for (int n = most - 1; n >= 1; n--) x.more[n] = x.part[n + 1].cost < x.part[n].cost ? n + 1 : x.more[n + 1];
        }
        if (!x.least) return false;
        of[k] = &x;
        uniform = uniform && nx[k] == nx[0];
    }
    int per = nb;
    if (uniform) {
        const int fit = sms / of[0]->least, sets = (nb + fit - 1) / fit;
        per = (nb + sets - 1) / sets;
    }
    for (int s0 = 0; s0 < nb;) {
        int s1 = s0, used = 0;
        std::vector<int> n;
        while (s1 < nb && s1 - s0 < per && used + of[s1]->least <= sms) {
            n.push_back(of[s1]->least);
            used += n.back();
            s1++;
        }
        for (;;) {  // the SMs left
            int pick = -1;
            double worst = 0.0;
            for (int k = 0; k < (int)n.size(); k++) {
                const ResWidth &w = *of[s0 + k];
                const int m = w.more[n[k]];
                if (m > most || used + m - n[k] > sms || (pick >= 0 && w.part[n[k]].cost <= worst)) continue;
                pick = k;
                worst = w.part[n[k]].cost;
            }
            if (pick < 0) break;
            const int m = of[s0 + pick]->more[n[pick]];
            used += m - n[pick];
            n[pick] = m;
        }
        ResidentSet set{};
        set.nshots = s1 - s0;
        ResidentGrid &g = set.grid;
        set.pitch = pt;
        int c = 0;
        for (int k = 0; k < set.nshots; k++) {
            const int w = nx[s0 + k], first = c;
            const std::vector<int> bands = res_bands(of[s0 + k]->part[n[k]], nz, cpml);
            int row = 0;
            for (int r : bands) {
                g.shot[c] = (unsigned short)(s0 + k);
                g.xs[c] = (unsigned short)k;
                g.first[c] = (unsigned short)first;
                g.count[c] = (unsigned short)bands.size();
                g.row0[c] = (unsigned short)row;
                g.nrow[c] = (unsigned short)r;
                row += r;
                const size_t f = res_floats(pt, r, res_halo(row - r, row, nz, cpml) > kRad, res_bottom(row, nz, cpml), img_bytes) *
                                 sizeof(float);
                set.smem = std::max(set.smem, f);
                // as many segments as it has rows, if the threads allow (as many as they allow in a bottom
                // band: its z memory variables span more rows than its own)
                const int lanes = res_lanes(w, pt, cpml);
                g.lanes[c] = (unsigned short)(res_bottom(row, nz, cpml) ? std::min(lanes, r + 8) : std::min(lanes, r));
                set.threads = std::max(set.threads, res_pairs(w, cpml).threads(g.lanes[c]));
                c++;
            }
        }
        g.n = c;
        // the farthest CTAs that exchange rows
        for (int a = 0; a < c; a++)
            for (int d = 1; d <= kResReach && a + d < g.first[a] + g.count[a]; d++) {
                const int e = g.row0[a] + g.nrow[a], low = g.row0[a + d];
                if (e + res_halo(g.row0[a], e, nz, cpml) > low || low - res_halo(low, low + g.nrow[a + d], nz, cpml) < e)
                    set.slots = std::max(set.slots, d);
            }
        set.slots++;
        if (set.smem > smem_limit) {  // a grid lower than the bottom layer: not a window the library takes
            out.clear();
            return false;
        }
        out.push_back(set);
        s0 = s1;
    }
    return true;
}

}  // namespace fwi
