// Shots resident on chip over the whole GPU (FP32, exact adjoint, images kept or recomputed from
// checkpoints), sm_103a.
//
// The tile passes (prop_tma.cuh, prop_layer.cuh) move the state of every shot through memory each
// step and pay two launches and a join for it.  Here one cooperative launch, one CTA per SM, takes
// the shots of a set (resident_plan.h) through all the steps of a phase (or of a checkpoint
// segment).  A CTA holds a band of rows of one shot in shared memory and registers for all of
// them.  P is only differenced along x and F only along z, so that bands of whole rows exchange
// nothing but 4 edge rows of one field (8 next to the bottom layer, whose z memory variables each
// CTA recomputes for the 4 rows either side of its own: the same inputs and operations, so
// bit-identical to the owner's).
//
// The exchange goes through L2, value by value: an edge value is stored as 8 bytes, the float and
// the step it belongs to, and the reader polls the very values it needs.  Neither a fence nor a
// flag is needed, and the latency is one store and one load.  The per-shot maximum that scales
// 16-bit images travels the same way (one 8-byte word per CTA).  Rows of step t go to copy t mod
// slots, one more than the CTAs between the farthest that exchange rows.  No copy is overwritten
// unread: a CTA that writes step t + 1 has its neighbours' rows of step t, so they have read theirs of
// step t - 1, the next ones theirs of step t - 2, and CTAs d apart theirs of step t - d.
// Every wait is bounded; one that gives up sets the status word, and its CTA waits no more.
//
// A thread owns 2 columns x R consecutive rows; the z-window of its rows slides through registers.
// Forward: the increments VP, VF in registers; two levels of F (with halo) and of P, and the
// models, in shared memory.  Step: the warps that hold the side layers' columns advance psi_x, then
// what these layers add to Dxx P (no halo needed: this runs while the neighbours' rows are on their
// way); halo rows in; bottom bands: psi_z, then what the bottom layer adds to Dzz F; increments,
// next level, edge rows out, images, receivers.  Adjoint: lambda and its increments in registers;
// two levels of u_x and of u_z (halo), the models and the gradient accumulators in shared memory.
// Step: Y_x and Dx(a Y) of the side layers; halo rows in; bottom bands: Y_z, Dz(a Y); increments,
// residual, next u and Z, edge rows out, imaging.  A block barrier ends each part.  Arithmetic on
// pairs of columns (FADD2, FFMA2) halves the instructions of the stencils.
//
// What bounds it: latency.  A C1 step (209 x 209; 2.75 us forward, 3.2 us adjoint) is about 1.8 us (2.2 us
// of adjoint) of arithmetic between block barriers, about 4.5 cycles an instruction of the longest
// thread, and 1.0 us for the exchange (a bare exchange of one row measures 0.9 - 1.1 us a step, of
// 4 rows of 100 pairs 1.3 us, whatever the number of CTAs; flags with fences 1.7 - 2.0 us).  So: the
// fewest barriers (two levels, one barrier a part), values published from the registers that hold
// them, registers over shared memory up to the point where they spill (spills miss the small L1
// that this much shared memory leaves), 2 columns a thread (4: C1 3.75 us an adjoint step against
// 3.3, fewer threads a band).  A 2000-step C1 gradient with FP32 images took 16.8 ms on one 16-CTA
// cluster, takes 11.7; 8 shots with FP16 images 36.2 -> 18.6 (two waves of clusters before); the
// adjoint of one 609 x 309 shot 34 -> 20 ms for 3000 steps.
#pragma once

#include "prop_layer.cuh"
#include "resident_plan.h"

namespace fwi {

// ------------------------------------------------------------------ exchanged words

// Two values of a row and the step they belong to, 16 bytes.
struct ResPair {
    uint64_t a, b;
    __device__ __forceinline__ void load(const uint64_t *p)
    {
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    }
    __device__ __forceinline__ bool is(unsigned tag) const
    {
        return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag;
    }
    __device__ __forceinline__ float2 value() const
    {
        return make_float2(__uint_as_float((unsigned)a), __uint_as_float((unsigned)b));
    }
    __device__ __forceinline__ static void put(uint64_t *p, const float2 &v, unsigned tag)
    {
        const uint64_t t = (uint64_t)tag << 32;
        asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | __float_as_uint(v.x)),
                     "l"(t | __float_as_uint(v.y))
                     : "memory");
    }
};

__device__ __forceinline__ void res_st1(uint64_t *p, uint64_t a)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(a) : "memory");
}
__device__ __forceinline__ uint64_t res_ld1(const uint64_t *p)
{
    uint64_t a;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    return a;
}

// A wait that gave up: the status word and the CTA's flag (its later waits end at once).
__device__ __forceinline__ bool res_give_up(int polls, volatile int *dead, unsigned *status, long limit = kWaitLimit)
{
    if (*dead) return true;
    if (polls < limit) return false;
    *dead = 1;
    atomicOr(status, kStatusTimeout);
    return true;
}

// ------------------------------------------------------------------ arithmetic on column pairs

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 ld2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ void put2(float *p, const float2 &v) { *reinterpret_cast<float2 *>(p) = v; }
__device__ __forceinline__ float2 add(const float2 &x, const float2 &y) { return __fadd2_rn(x, y); }
__device__ __forceinline__ float2 mul(const float2 &x, const float2 &y) { return __fmul2_rn(x, y); }
__device__ __forceinline__ float2 fma(const float2 &x, const float2 &y, const float2 &z) { return __ffma2_rn(x, y, z); }
__device__ __forceinline__ float2 scaled(const float2 &x, float v) { return __fmul2_rn(x, both(v)); }
// A product that goes into a sum rounded, as the sum is.  A packed product with one use is merged into the
// packed sum that takes it (one rounding, whatever the intrinsics' names say: measured on every such
// form); of scalars it is not.
__device__ __forceinline__ float2 rounded(const float2 &x, float v) { return make_float2(__fmul_rn(x.x, v), __fmul_rn(x.y, v)); }
// the columns below nval, zero from there on (nval >= 1)
__device__ __forceinline__ float2 keep(const float2 &v, int nval) { return make_float2(v.x, nval > 1 ? v.y : 0.f); }

// 8th-order second derivative (unnormalised, difference form) from the four pair sums of
// differences, and first derivative from the four differences: the multiply-adds as the tile
// passes' d2_row, d1_row evaluate them, written out so that every use rounds alike.
__device__ __forceinline__ float2 res_d2(const float2 &s1, const float2 &s2, const float2 &s3, const float2 &s4)
{
    using C = Coef<float>;
    return __ffma2_rn(both(-C::d2_4), s4,
                      __ffma2_rn(both(C::d2_3), s3, __ffma2_rn(both(C::d2_1), s1, __fmul2_rn(both(-C::d2_2), s2))));
}
__device__ __forceinline__ float2 res_d1(const float2 &e1, const float2 &e2, const float2 &e3, const float2 &e4)
{
    using C = Coef<float>;
    return __ffma2_rn(both(-C::d1_4), e4,
                      __ffma2_rn(both(C::d1_3), e3, __ffma2_rn(both(C::d1_1), e1, __fmul2_rn(both(-C::d1_2), e2))));
}
__device__ __forceinline__ float2 res_pair(const float2 &p, const float2 &m, const float2 &no)
{
    return __fadd2_rn(__fadd2_rn(p, no), __fadd2_rn(m, no));
}
__device__ __forceinline__ float2 res_diff(const float2 &p, const float2 &m)
{
    return __fadd2_rn(p, make_float2(-m.x, -m.y));
}

// The memory variables' updates, psi' = b psi + a D and zeta' = b zeta + a (d2 + D), D = d1 inv_dh,
// and the layer's term D + zeta'.  nvcc contracts these sums in one way in the cluster kernels, in another
// in the layer tiles, and psi_x in a third in the strip pass; a batch rounds as the path that would
// otherwise take it (ResOrder), so that its traces and images are that path's bit for bit: a last-bit
// difference turns into one of 2^-8 where a BF16 image falls on the other side of a rounding boundary.
__device__ __forceinline__ float2 res_psi(bool strip, const float2 &b, const float2 &psi, const float2 &a, const float2 &D)
{
    return strip ? fma(a, D, mul(b, psi)) : fma(b, psi, mul(a, D));
}
__device__ __forceinline__ float2 res_zeta(bool tile, const float2 &b, const float2 &zeta, const float2 &a,
                                           const float2 &d2, const float2 &d1, float inv_dh)
{
    return fma(b, zeta, mul(a, tile ? fma(d1, both(inv_dh), d2) : add(d2, rounded(d1, inv_dh))));
}
__device__ __forceinline__ float2 res_term(bool tile, const float2 &d1, float inv_dh, const float2 &zeta)
{
    return tile ? fma(d1, both(inv_dh), zeta) : add(rounded(d1, inv_dh), zeta);
}

// Derivatives of 2 columns, along z from 9 rows, along x from the 10 values at p - 4 .. p + 5.
__device__ __forceinline__ float2 res_d2z(const float2 *w)
{
    const float2 no = make_float2(-w[4].x, -w[4].y);
    return res_d2(res_pair(w[5], w[3], no), res_pair(w[6], w[2], no), res_pair(w[7], w[1], no), res_pair(w[8], w[0], no));
}
__device__ __forceinline__ float2 res_d1z(const float2 *w)
{
    return res_d1(res_diff(w[5], w[3]), res_diff(w[6], w[2]), res_diff(w[7], w[1]), res_diff(w[8], w[0]));
}
struct ResWindow {
    float2 a, b, m, c, d;
    __device__ __forceinline__ explicit ResWindow(const float *p)
        : a(ld2(p - 4)), b(ld2(p - 2)), m(ld2(p)), c(ld2(p + 2)), d(ld2(p + 4))
    {
    }
    // odd distances cross the pairs' register alignment: their sums are made one by one
    __device__ __forceinline__ float2 d2() const
    {
        auto odd = [](float p, float q, float o) { return (p - o) + (q - o); };
        const float2 no = make_float2(-m.x, -m.y);
        return res_d2(make_float2(odd(m.y, b.y, m.x), odd(c.x, m.x, m.y)), res_pair(c, b, no),
                      make_float2(odd(c.y, a.y, m.x), odd(d.x, b.x, m.y)), res_pair(d, a, no));
    }
    __device__ __forceinline__ float2 d1() const
    {
        return res_d1(make_float2(m.y - b.y, c.x - m.x), res_diff(c, b), make_float2(c.y - a.y, d.x - b.x),
                      res_diff(d, a));
    }
};

// ------------------------------------------------------------------ images of 2 columns

// Copies that complete asynchronously (cp.async; waited with cp.async.wait_group).
template <int BYTES> __device__ __forceinline__ void res_copy(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src), "n"(BYTES) : "memory");
}

// Two image values: encoded with the step's scale, decoded with its inverse.
template <typename Cd> struct ResImage;
template <> struct ResImage<Codec<float, kStoreHalf>> {
    __device__ __forceinline__ static float2 value(const __half *p, float inv_sc)
    {
        return scaled(__half22float2(*reinterpret_cast<const __half2 *>(p)), inv_sc);
    }
    // `sat` as Codec::enc_flag: a value beyond FP16 (or NaN); the common case costs an integer add
    // and a test for both values (a half at or above the largest finite one)
    __device__ __forceinline__ static void store(__half *p, const float2 &v, float sc, bool &sat)
    {
        const float2 x = scaled(v, sc);
        __half2 h = __floats2half2_rn(x.x, x.y);
        if (((*reinterpret_cast<const uint32_t *>(&h) & 0x7fff7fffu) + 0x04010401u) & 0x80008000u) {
            using Cd = Codec<float, kStoreHalf>;
            h = __halves2half2(Cd::enc_flag(v.x, sc, sat), Cd::enc_flag(v.y, sc, sat));
        }
        *reinterpret_cast<__half2 *>(p) = h;
    }
};
template <> struct ResImage<Codec<float, kStoreBf16>> {
    __device__ __forceinline__ static float2 value(const __nv_bfloat16 *p, float inv_sc)
    {
        return scaled(__bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(p)), inv_sc);
    }
    __device__ __forceinline__ static void store(__nv_bfloat16 *p, const float2 &v, float sc, bool &)
    {
        const float2 x = scaled(v, sc);
        *reinterpret_cast<__nv_bfloat162 *>(p) = __floats2bfloat162_rn(x.x, x.y);
    }
};
template <> struct ResImage<Codec<float, kStoreNative>> {
    __device__ __forceinline__ static float2 value(const float *p, float) { return ld2(p); }
    __device__ __forceinline__ static void store(float *p, const float2 &v, float, bool &) { put2(p, v); }
};

// ------------------------------------------------------------------ one CTA's band

struct ResBand {
    int s, xs, k0, k1, self;      // shot; the shot's CTAs [k0, k1) of the launch, this one
    int nx, nz, cpml;             // window
    int row0, nrow, iz0, nzi, hr; // own rows (interior index), first global row, interior rows, halo rows
    int zb;                       // first row of the bottom layer
    int pub_lo, pub_hi;           // own rows < pub_lo or >= pub_hi are read by other CTAs
    int nlane, seg, ix;           // row segments of the CTA; the thread's segment and first column
    int rows;                     // rows of a segment
    int nside_threads;            // threads (whole warps) of the column pairs within reach of a side layer
    bool bottom, side, use;       // bottom band; the thread's pair is within reach of a side layer; it has one
    ResGeom g;

    __device__ __forceinline__ ResBand(const Batch<float> &b, const ResidentGrid &grid, const DevShot &sh)
    {
        self = blockIdx.x;
        s = grid.shot[self];
        xs = grid.xs[self];
        k0 = grid.first[self];
        k1 = k0 + grid.count[self];
        nx = sh.nx;
        nz = b.nz;
        cpml = b.cpml;
        row0 = grid.row0[self];
        nrow = grid.nrow[self];
        nlane = grid.lanes[self];
        iz0 = 4 + row0;
        nzi = nz - 8;
        bottom = res_bottom(row0 + nrow, nz, cpml);
        hr = res_halo(row0, row0 + nrow, nz, cpml);
        zb = nz - cpml;
        rows = (nrow + nlane - 1) / nlane;
        g = res_geom(nx, cpml);
        // the side pairs in warps of their own, then the pairs between them
        const ResPairs p = res_pairs(nx, cpml);
        nside_threads = p.side_threads(nlane);
        const int t = (int)threadIdx.x - nside_threads;
        side = t < 0;
        const int w = max(side ? p.nside : p.nq - p.nside, 1), q = side ? (int)threadIdx.x : t;
        seg = q / w;
        const int k = q - seg * w;
        ix = 4 + 2 * (side ? (k < p.nleft ? k : p.nq - p.nside + k) : p.nleft + k);
        use = seg < nlane && (side ? p.nside > 0 : p.nq > p.nside);
        // rows the CTAs above (below) read as their lower (upper) halo
        int lo = 0, hi = 0;
        for (int c = max(k0, self - kResReach); c <= min(k1 - 1, self + kResReach); c++) {
            if (c == self) continue;
            const int a = grid.row0[c], e = a + grid.nrow[c], h = res_halo(a, e, nz, cpml);
            if (c < self) lo = max(lo, e + h - row0);
            else hi = max(hi, row0 + nrow - (a - h));
        }
        pub_lo = min(lo, nrow);
        pub_hi = nrow - min(hi, nrow);
    }
    __device__ __forceinline__ bool published(int r) const { return r < pub_lo || r >= pub_hi; }
    __device__ __forceinline__ bool layer_col(int c) const { return c < cpml || c > nx - cpml - 1; }
};

// A barrier of the side warps.
__device__ __forceinline__ void res_side_sync(const ResBand &B)
{
    asm volatile("bar.sync 1, %0;" ::"r"(B.nside_threads) : "memory");
}

// Exchanged words of interior row gi, columns col, col + 1, in copy `copy` of `slots`.
template <int PT>
__device__ __forceinline__ uint64_t *res_words(const ResBand &B, uint64_t *x, int slots, int copy, int gi, int col)
{
    return x + ((long)(B.xs * slots + copy) * B.nz + 4 + gi) * PT + (col - 4);
}
__device__ __forceinline__ int res_next(int copy, int slots) { return copy + 1 == slots ? 0 : copy + 1; }

// The halo rows of step `tag` (`base`: the words of the band's first row at the thread's columns) into f
// (row r of the band at f + r PT): a thread its column pair's rows seg, seg + nlane, ....  Up to U rows
// are asked for together and those that have not come again, by every thread for itself (one lane
// polling for its warp measured slower: C1 3.5 us a forward step against 2.9).
template <int PT>
__device__ __forceinline__ void res_halo_in(const ResBand &B, float *f, const uint64_t *base, unsigned tag, volatile int *dead,
                                            unsigned *status)
{
    constexpr int U = 6;
    if (!B.use) return;
    for (int h0 = B.seg; h0 < 2 * B.hr; h0 += U * B.nlane) {
        ResPair q[U];
        unsigned late = 0;
        auto row = [&](int u) {
            const int h = h0 + u * B.nlane;
            return h < B.hr ? h - B.hr : B.nrow + h - B.hr;
        };
#pragma unroll
        for (int u = 0; u < U; u++)
            if (h0 + u * B.nlane < 2 * B.hr && (unsigned)(B.row0 + row(u)) < (unsigned)B.nzi) late |= 1u << u;
        const unsigned all = late;
        for (int k = 0; late; k++) {
#pragma unroll
            for (int u = 0; u < U; u++)
                if (late >> u & 1) q[u].load(base + row(u) * PT);
#pragma unroll
            for (int u = 0; u < U; u++)
                if ((late >> u & 1) && q[u].is(tag)) late &= ~(1u << u);
            if (late && res_give_up(k, dead, status)) break;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (all >> u & 1) put2(f + row(u) * PT + B.ix, q[u].value());
    }
}

// f(row, its 9 z-neighbours of 2 columns) for rows [ra, rb) of a field (row r at field + r PT), a
// thread a run of consecutive rows of its column pair (the window slides).
template <int PT, typename Fn>
__device__ __forceinline__ void res_rows(const ResBand &B, int ra, int rb, const float *field, Fn f)
{
    constexpr int M = 3;
    if (!B.use) return;
    const int n = (rb - ra + B.nlane - 1) / B.nlane;  // rows of a thread
    const int r0 = ra + B.seg * n, r1 = min(r0 + n, rb);
    for (int r = r0; r < r1; r += M) {
        float2 w[M + 8];
        const float *const p = field + (r - 4) * PT + B.ix;
#pragma unroll
        for (int k = 0; k < 8; k++) w[k] = ld2(p + k * PT);
#pragma unroll
        for (int m = 0; m < M; m++) {
            if (r + m >= r1) break;
            w[m + 8] = ld2(p + (m + 8) * PT);
            f(r + m, w + m);
        }
    }
}

// CPML tables: by side column (band storage) and by row from 4 above the band.
__device__ __forceinline__ void res_tables(const Batch<float> &b, const ResBand &B, float *ax, float *bx, float *az,
                                           float *bz)
{
    const int cp = B.cpml;
    for (int c = threadIdx.x; c < kResSide; c += blockDim.x) {
        const int ix = c < B.g.wl ? c : B.g.xr0 + c - B.g.wl;
        const int d = ix >= B.nx ? 0 : ix < cp ? cp - ix : ix > B.nx - cp - 1 ? ix - B.nx + cp + 1 : 0;
        ax[c] = d ? b.cpa[d] : 0.f;
        bx[c] = d ? b.cpb[d] : 0.f;
    }
    for (int r = threadIdx.x; r < B.nrow + 2 * kRad; r += blockDim.x) {
        const int iz = B.iz0 - kRad + r;
        const int d = (iz > B.nz - cp - 1 && iz < B.nz) ? iz - B.nz + cp + 1 : 0;
        az[r] = d ? b.cpa[d] : 0.f;
        bz[r] = d ? b.cpb[d] : 0.f;
    }
}

// Shared arrays (resident_plan.h: res_floats).  Row pitches are compile-time constants (PT for
// whole rows, kResSide for side columns) and a row's own arrays lie side by side, so that a thread
// reaches all of them from one address register with immediate offsets; with run-time pitches the
// addresses alone took more registers than the state, and spilled.
template <int PT, int OWN, int SIDE> struct ResShared {
    float *halo[2];  // the two levels of the z-stencil field, row r at halo + r PT, r from -hr
    float *own;      // OWN arrays of row r at own + (r OWN + k) PT
    float *side;     // SIDE arrays of row r at side + (r SIDE + k) kResSide
    float *ax, *bx, *az, *bz;  // CPML tables; rows from -4
    float *zh;       // bottom bands: the z memory variable, row r at zh + r PT, r from -4
    float *zo;       // bottom bands: two arrays of row r at zo + (2 r + k) PT
    float *img;      // adjoint: the staged images, G and H of row r at (2 r + k) PT elements
    __device__ __forceinline__ ResShared(float *csm, const ResBand &B)
    {
        halo[0] = csm + B.hr * PT;
        halo[1] = halo[0] + (B.nrow + 2 * B.hr) * PT;
        own = csm + 2 * (B.nrow + 2 * B.hr) * PT;
        side = own + B.nrow * OWN * PT;
        ax = side + B.nrow * SIDE * kResSide;
        bx = ax + kResSide;
        zh = bx + kResSide + kRad * PT;
        zo = zh + (B.nrow + kRad) * PT;
        az = (B.bottom ? zo + B.nrow * 2 * PT : bx + kResSide) + kRad;
        bz = az + B.nrow + 2 * kRad;
        img = bz + B.nrow + kRad;
        img += (4 - ((img - csm) & 3)) & 3;
    }
};

// ------------------------------------------------------------------ forward

template <int ST, int PT>
__global__ void __launch_bounds__(res_shape(PT).threads, 1)
k_resident_fwd(const __grid_constant__ Batch<float> b, const __grid_constant__ ResidentGrid grid,
               const __grid_constant__ ResFwdArgs a)
{
    using Cd = Codec<float, ST>;
    using SI = typename Cd::S;
    using Img = ResImage<Cd>;
    constexpr int R = res_shape(PT).fwd_rows;
    constexpr int OWN = kResFwdOwn;                   // own arrays: P (two levels), v_hor, v_po, v_nmo
    constexpr int WB = kResSide, SD = kResFwdSide;    // side arrays: psi_x, zeta_x, what they add to Dxx P
    extern __shared__ __align__(16) float csm[];
    __shared__ int dead;
    __shared__ unsigned s_max[2];  // the band's max |P|, |F| after a step (bits; alternate steps)
    __shared__ float s_sc;         // the image scale of the step
    const DevShot sh = b.shots[grid.shot[blockIdx.x]];
    if (a.ntb - sh.nt >= a.g1) return;  // the shot starts later
    const ResBand B(b, grid, sh);
    const ResShared<PT, OWN, SD> S(csm, B);
    const int tid = threadIdx.x, nrow = B.nrow, ix = B.ix;
    const int start = a.ntb - sh.nt;  // the shot's first global step
    const int nfl = (int)res_floats(PT, nrow, B.hr > kRad, B.bottom, 0);
    for (int i = tid; i < nfl; i += blockDim.x) csm[i] = 0.f;
    if (tid == 0) dead = 0;
    if (tid < 2) s_max[tid] = 0;
    __syncthreads();
    res_tables(b, B, S.ax, S.bx, S.az - kRad, S.bz - kRad);
    const float inv_dh = b.inv_dh, inv_dh2 = b.inv_dh2;
    const bool tile = a.order != kResAsCluster, strip = a.order == kResAsStrip, plain = a.plain_images;
    const long so = (long)B.s * b.slot;
    const int r0 = B.seg * B.rows, nr = B.use ? min(B.rows, nrow - r0) : 0;  // the thread's rows [r0, r0 + nr)
    const int nval = min(2, B.nx - 4 - ix);                                   // its interior columns
    const bool lay0 = B.layer_col(ix), lay1 = nval > 1 && B.layer_col(ix + 1);  // ... in a side layer
    const int cx = B.side ? B.g.col(ix) : 0;
    float *const pO = S.own + r0 * OWN * PT + ix, *const pS = S.side + r0 * SD * WB + cx;
    // state at the first step: a checkpoint, or zero before the shot's first step
    const int gs = max(a.g0, start);
    const bool load = a.load_ck >= 0 && a.g0 > start;
    const float *const ck0 = a.ck + (long)(load ? a.load_ck : 0) * 8 * a.ck_stride + so;
    const long i0 = (long)(B.iz0 + r0) * b.pitch + ix;  // the thread's first point in a slot
    float2 VP[R], VF[R];
#pragma unroll
    for (int rr = 0; rr < R; rr++) {
        VP[rr] = VF[rr] = both(0.f);
        if (rr >= nr) continue;
        const long i = i0 + (long)rr * b.pitch, mi = (long)(B.iz0 + r0 + rr) * b.mpitch + sh.x0 + ix;
        float *const o = pO + rr * OWN * PT;
        for (int j = 0; j < nval; j++) {
            o[2 * PT + j] = b.mh[mi + j];
            o[3 * PT + j] = b.mp[mi + j];
            o[4 * PT + j] = b.mn[mi + j];
        }
        if (load) {
            put2(o, ld2(ck0 + i));
            VP[rr] = ld2(ck0 + 2 * a.ck_stride + i);
            VF[rr] = ld2(ck0 + 3 * a.ck_stride + i);
            if (lay0 || lay1) {
                put2(pS + rr * SD * WB, ld2(ck0 + 4 * a.ck_stride + i));
                put2(pS + (rr * SD + 1) * WB, ld2(ck0 + 6 * a.ck_stride + i));
            }
            if (B.bottom && B.iz0 + r0 + rr >= B.zb) put2(S.zo + (r0 + rr) * 2 * PT + ix, ld2(ck0 + 7 * a.ck_stride + i));
        }
    }
    if (load && B.use)  // F with its halo, psi_z of a bottom band with 4 rows either side
        for (int r = B.seg - B.hr; r < nrow + B.hr; r += B.nlane) {
            const int gi = B.row0 + r;
            if (gi < 0 || gi >= B.nzi) continue;
            const long i = (long)(4 + gi) * b.pitch + ix;
            put2(S.halo[0] + r * PT + ix, ld2(ck0 + a.ck_stride + i));
            if (B.bottom && r >= -kRad && r < nrow + kRad && 4 + gi >= B.zb)
                put2(S.zh + r * PT + ix, ld2(ck0 + 5 * a.ck_stride + i));
        }
    // the rows of psi_z this CTA advances: those of the bottom layer within 4 of its own
    const int bz0 = max(max(4, B.zb), B.iz0 - kRad) - B.iz0, bz1 = min(b.nz - 4, B.iz0 + nrow + kRad) - B.iz0;
    const int src_rr = sh.sx >= ix && sh.sx < ix + 2 ? sh.sz - B.iz0 - r0 : -1;  // the source among the thread's rows
    const int rec_rr = sh.rz - B.iz0 - r0;                                      // the receivers' row
    float *const amax = b.amax + (long)B.s * (b.nt_max + 1);
    int seg = gs / a.period, gseg = gs - seg * a.period;  // segment of the step, step in it
    int cur = 0;                                          // the current level
    int copy = (int)((a.tag0 + gs) % a.slots);            // ... and the copy of the exchanged rows
    __syncthreads();
    for (int g = gs; g < a.g1; g++) {
        const unsigned tag = a.tag0 + g;
        const bool img = g >= a.img_first;
        const bool ck_now = gseg == 0 && seg < a.save_ck, ck_next = gseg + 1 == a.period && seg + 1 < a.save_ck;
        float *const F = S.halo[cur], *const pc = pO + cur * PT, *const pn = pO + (1 - cur) * PT;
        if (ck_now) {  // checkpoint of the state before the step
            float *const ck = a.ck + (long)seg * 8 * a.ck_stride + so;
#pragma unroll
            for (int rr = 0; rr < R; rr++) {
                if (rr >= nr) break;
                const long i = i0 + (long)rr * b.pitch;
                put2(ck + i, ld2(pc + rr * OWN * PT));
                put2(ck + a.ck_stride + i, ld2(F + (r0 + rr) * PT + ix));
                put2(ck + 2 * a.ck_stride + i, VP[rr]);
                put2(ck + 3 * a.ck_stride + i, VF[rr]);
                if (lay0 || lay1) {
                    put2(ck + 4 * a.ck_stride + i, ld2(pS + rr * SD * WB));
                    put2(ck + 6 * a.ck_stride + i, ld2(pS + (rr * SD + 1) * WB));
                }
                if (B.bottom) {
                    put2(ck + 5 * a.ck_stride + i, ld2(S.zh + (r0 + rr) * PT + ix));
                    put2(ck + 7 * a.ck_stride + i, ld2(S.zo + (r0 + rr) * 2 * PT + ix));
                }
            }
        }
        if (B.side) {
            // psi_x of the side layers (src/parallelcalls.cu:48-63; the coefficients are zero off them)
            const float2 ax = ld2(S.ax + cx), bx = ld2(S.bx + cx);
            for (int rr = 0; rr < nr; rr++) {
                float *const ps = pS + rr * SD * WB;
                put2(ps, keep(res_psi(strip, bx, ld2(ps), ax, scaled(ResWindow(pc + rr * OWN * PT).d1(), inv_dh)), nval));
            }
            res_side_sync(B);
            // what they add to Dxx P: zeta_x and Dx psi_x (in the bottom layer also where only psi_x reaches)
            for (int rr = 0; rr < nr; rr++) {
                float *const ps = pS + rr * SD * WB;
                const float2 gp = rounded(ResWindow(pc + rr * OWN * PT).d2(), inv_dh2);
                const float2 dx = ResWindow(ps).d1();
                const float2 z = keep(res_zeta(tile, bx, ld2(ps + WB), ax, gp, dx, inv_dh), nval);
                const float2 d = res_term(tile, dx, inv_dh, z);
                const bool zl = B.iz0 + r0 + rr >= B.zb;
                put2(ps + WB, z);
                put2(ps + 2 * WB, make_float2(lay0 || zl ? d.x : 0.f, lay1 || (zl && nval > 1) ? d.y : 0.f));
            }
        }
        // the image scale of the step from every band's max (the last warp), the halo rows (all)
        if (Cd::scaled && img && (tid >> 5) == (int)(blockDim.x >> 5) - 1) {
            float m = 0.f;
            if (g == gs) {
                m = load ? amax[g] : 0.f;
            } else {
                for (int k = B.k0 + (tid & 31); k < B.k1; k += 32) {
                    const uint64_t *p = a.w + (tag & (kResSlots - 1)) * kResMaxCtas + k;
                    uint64_t v = res_ld1(p);
                    for (int n = 0; (unsigned)(v >> 32) != tag && !res_give_up(n, &dead, b.status); n++) v = res_ld1(p);
                    m = fmaxf(m, __uint_as_float((unsigned)v));
                }
                m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
            }
            if ((tid & 31) == 0) {
                const float sc = image_scale(m, inv_dh2);
                s_sc = sc;
                if (B.self == B.k0) b.scale[(long)B.s * b.nt_max + g] = sc;
            }
        }
        if (g > gs) res_halo_in<PT>(B, F, res_words<PT>(B, a.x, a.slots, copy, B.row0, ix), tag, &dead, b.status);
        copy = res_next(copy, a.slots);
        __syncthreads();
        if (B.bottom) {
            // psi_z of the bottom layer's points of the own rows and 4 either side
            res_rows<PT>(B, bz0, bz1, F, [&](int r, const float2 *fz) {
                float *const ps = S.zh + r * PT + ix;
                const float2 d = scaled(res_d1z(fz), inv_dh), az = both(S.az[r]), bz = both(S.bz[r]);
                put2(ps, keep(fma(bz, ld2(ps), mul(az, d)), nval));
                if (r >= 0 && r < nrow) put2(S.zo + (r * 2 + 1) * PT + ix, scaled(res_d2z(fz), inv_dh2));  // for the next pass
            });
            __syncthreads();
            // what the bottom layer adds to Dzz F: zeta_z and Dz psi_z (above the layer the side
            // layers' points only)
            res_rows<PT>(B, max(B.zb - 4 - B.iz0, 0), nrow, S.zh, [&](int r, const float2 *pz) {
                float *const z = S.zo + r * 2 * PT + ix;
                const float2 dz = res_d1z(pz);
                float2 t;
                if (B.iz0 + r >= B.zb) {
                    const float2 n = keep(res_zeta(tile, both(S.bz[r]), ld2(z), both(S.az[r]), ld2(z + PT), dz, inv_dh), nval);
                    put2(z, n);
                    t = res_term(tile, dz, inv_dh, n);
                } else {
                    t = scaled(dz, inv_dh);
                    t = make_float2(lay0 ? t.x : 0.f, lay1 ? t.y : 0.f);
                }
                put2(z + PT, t);
            });
            __syncthreads();
        }
        // the state's max: scales the next step's images, and those of a recompute from its checkpoint
        const bool mx_img = g + 1 >= a.img_first && g + 1 < a.g1, mx = Cd::scaled && (mx_img || ck_next);
        float lmax = 0.f;
        if (nr > 0) {
            const float sc = Cd::scaled && img ? s_sc : 1.f;
            SI *const image = (SI *)b.store + ((long)B.s * b.n_img + (img ? gseg + (seg & 1) * a.period : 0)) * 2 * b.slot + i0;
            uint64_t *const out = res_words<PT>(B, a.x, a.slots, copy, B.row0 + r0, ix);
            const float *const fc = F + r0 * PT + ix;
            float *const fn = S.halo[1 - cur] + r0 * PT + ix;
            bool sat = false;
            float2 win[R + 8];
#pragma unroll
            for (int k = 0; k < 8; k++) win[k] = ld2(fc + (k - 4) * PT);
#pragma unroll
            for (int rr = 0; rr < R; rr++) {
                if (rr >= nr) break;
                win[rr + 8] = ld2(fc + (rr + 4) * PT);
                const float *const o = pO + rr * OWN * PT;
                const ResWindow w(pc + rr * OWN * PT);
                const float2 G0 = rounded(w.d2(), inv_dh2), H0 = rounded(res_d2z(win + rr), inv_dh2);
                float2 G = G0, H = H0;
                if (B.side) G = add(G, ld2(pS + (rr * SD + 2) * WB));
                if (B.bottom) H = add(H, ld2(S.zo + ((r0 + rr) * 2 + 1) * PT + ix));
                const float2 mp = ld2(o + 3 * PT);
                VP[rr] = add(VP[rr], fma(mp, H, mul(ld2(o + 2 * PT), G)));
                VF[rr] = add(VF[rr], fma(mp, H, mul(ld2(o + 4 * PT), G)));
                if (rr == src_rr) {
                    const float v = b.wavelet[g - start];
                    const float2 e = make_float2(sh.sx == ix ? v : 0.f, sh.sx == ix ? 0.f : v);
                    VP[rr] = add(VP[rr], e);
                    VF[rr] = add(VF[rr], e);
                }
                if (nval < 2) {
                    VP[rr].y = VF[rr].y = 0.f;
                    G.y = H.y = 0.f;
                }
                const float2 p = add(w.m, VP[rr]), f = add(win[rr + 4], VF[rr]);
                if (B.published(r0 + rr)) ResPair::put(out + rr * PT, f, tag + 1);
                put2(pn + rr * OWN * PT, p);
                put2(fn + rr * PT, f);
                if (img) {
                    Img::store(image + (long)rr * b.pitch, plain ? keep(G0, nval) : G, sc, sat);
                    Img::store(image + b.slot + (long)rr * b.pitch, plain ? keep(H0, nval) : H, sc, sat);
                }
                if (mx) lmax = fmaxf(lmax, fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fmaxf(fabsf(f.x), fabsf(f.y))));
                if (rr == rec_rr) {
                    float *const rec = b.rec + sh.rec_off + (long)(g - start) * (sh.rx1 - sh.rx0) - sh.rx0 + ix;
                    const float2 v = add(p, f);
                    if (ix >= sh.rx0 && ix < sh.rx1) rec[0] = v.x;
                    if (ix + 1 >= sh.rx0 && ix + 1 < sh.rx1) rec[1] = v.y;
                }
            }
            if (sat) atomicOr(b.status, kStatusSaturated);
        }
        if (mx) {
            const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(lmax));
            if ((tid & 31) == 0) atomicMax(&s_max[g & 1], m);
        }
        __syncthreads();  // the new level; the current one read
        if (mx && tid == 0) {
            const unsigned m = s_max[g & 1];
            s_max[g & 1] = 0;
            if (mx_img) res_st1(a.w + ((tag + 1) & (kResSlots - 1)) * kResMaxCtas + B.self, (uint64_t)(tag + 1) << 32 | m);
            if (ck_next && m) atomicMax((unsigned *)amax + g + 1, m);
        }
        cur ^= 1;
        if (++gseg == a.period) {
            gseg = 0;
            seg++;
        }
    }
}

// ------------------------------------------------------------------ adjoint

// REF: the reference's adjoint, whose CPML is the forward's, applied to the model-weighted fields
// (src/parallelcalls.cu:179-243).  Its four psi and four zeta are linear in them and pairs share their
// coefficients and enter the update as sums, so that the sums are advanced: psi_x' = b psi_x + a Dx u_x
// with u_x = v_hor lambda_P + v_nmo lambda_F (and z, u_z = v_po (lambda_P + lambda_F)): the forward's two psi
// and two zeta.  Iteration j images step nt - 2 - j (the exact adjoint: nt - 1 - j).

template <int ST, int PT, bool REF>
__global__ void __launch_bounds__(res_shape(PT).threads, 1)
k_resident_adj(const __grid_constant__ Batch<float> b, const __grid_constant__ ResidentGrid grid,
               const __grid_constant__ ResAdjArgs a)
{
    using Cd = Codec<float, ST>;
    using SI = typename Cd::S;
    using Img = ResImage<Cd>;
    constexpr int R = res_shape(PT).adj_rows;
    constexpr int OWN = kResAdjOwn;                 // own arrays: u_x (two levels), v_hor, v_po, v_nmo, three gradients
    constexpr int WB = kResSide, SD = kResAdjSide;  // side arrays: Y_x, Z_x, a Y_x, u_x at layer points,
                                                  // -Dx(a Y_x); REF: psi_x, zeta_x, what they add to Dxx u_x
    extern __shared__ __align__(16) float csm[];
    __shared__ int dead;
    const DevShot sh = b.shots[grid.shot[blockIdx.x]];
    if (a.j0 >= sh.nt) return;  // the shot is done
    const ResBand B(b, grid, sh);
    const ResShared<PT, OWN, SD> S(csm, B);
    const int tid = threadIdx.x, nrow = B.nrow, ix = B.ix;
    const int nfl = (int)res_floats(PT, nrow, B.hr > kRad, B.bottom, (int)sizeof(SI));
    for (int i = tid; i < nfl; i += blockDim.x) csm[i] = 0.f;
    if (tid == 0) dead = 0;
    __syncthreads();
    res_tables(b, B, S.ax, S.bx, S.az - kRad, S.bz - kRad);
    __syncthreads();
    const float inv_dh = b.inv_dh, inv_dh2 = b.inv_dh2;
    const long so = (long)B.s * b.slot;
    const int r0 = B.seg * B.rows, nr = B.use ? min(B.rows, nrow - r0) : 0;  // the thread's rows [r0, r0 + nr)
    const int nval = min(2, B.nx - 4 - ix);
    const bool lay0 = B.layer_col(ix), lay1 = nval > 1 && B.layer_col(ix + 1);
    const int cx = B.side ? B.g.col(ix) : 0;
    float *const pO = S.own + r0 * OWN * PT + ix, *const pS = S.side + r0 * SD * WB + cx;
    const int j1 = min(a.j1, sh.nt);
    const bool load = a.j0 > 0;
    const long i0 = (long)(B.iz0 + r0) * b.pitch + ix;
    // the next step's u from lambda at row rr, into level `to`, its edge rows to the neighbours: u = g
    // (+ a Z at layer points, Z advanced first, Z' = g + b Z, or not)
    auto make_u = [&](int rr, int to, const float2 &lp, const float2 &lf, bool advance, unsigned tag, int copy) {
        float *const o = pO + rr * OWN * PT;
        float2 ux = fma(ld2(o + 2 * PT), lp, mul(ld2(o + 4 * PT), lf)), uz = mul(ld2(o + 3 * PT), add(lp, lf));
        const int r = r0 + rr;
        const bool zl = !REF && B.bottom && B.iz0 + r >= B.zb;
        if (zl) {
            float *const z_ = S.zo + r * 2 * PT + ix;
            float2 z = ld2(z_);
            if (advance) {
                z = fma(both(S.bz[r]), z, uz);
                put2(z_, z);
            }
            uz = fma(both(S.az[r]), z, uz);
        }
        if (!REF && B.side) {
            float *const ps = pS + rr * SD * WB;
            if (lay0 || lay1) {
                float2 z = ld2(ps + WB);
                if (advance) {
                    z = fma(ld2(S.bx + cx), z, ux);
                    z = make_float2(lay0 ? z.x : 0.f, lay1 ? z.y : 0.f);
                    put2(ps + WB, z);
                }
                ux = fma(ld2(S.ax + cx), z, ux);
            }
            if (nval < 2) ux.y = 0.f;
            put2(ps + 3 * WB, make_float2(lay0 || zl ? ux.x : 0.f, lay1 || zl ? ux.y : 0.f));
        }
        if (nval < 2) ux.y = uz.y = 0.f;
        if (B.published(r)) ResPair::put(res_words<PT>(B, a.x, a.slots, copy, B.row0 + r, ix), uz, tag);
        put2(o + to * PT, ux);
        put2(S.halo[to] + r * PT + ix, uz);
    };
    int copy = (int)((a.tag0 + a.j0) % a.slots);  // of the exchanged rows
    float2 LP[R], LF[R], WP[R], WF[R];
    // u of the first step from the loaded lambda and Z (zero at the first iteration); its edge rows out
#pragma unroll
    for (int rr = 0; rr < R; rr++) {
        LP[rr] = LF[rr] = WP[rr] = WF[rr] = both(0.f);
        if (rr >= nr) continue;
        const long i = so + i0 + (long)rr * b.pitch, mi = (long)(B.iz0 + r0 + rr) * b.mpitch + sh.x0 + ix;
        float *const o = pO + rr * OWN * PT;
        for (int j = 0; j < nval; j++) {
            o[2 * PT + j] = b.mh[mi + j];
            o[3 * PT + j] = b.mp[mi + j];
            o[4 * PT + j] = b.mn[mi + j];
        }
        if (load) {
            LP[rr] = ld2(b.lvl[0] + i);
            LF[rr] = ld2(b.lvl[2] + i);
            WP[rr] = ld2(b.lvl[4] + i);
            WF[rr] = ld2(b.lvl[5] + i);
            if (lay0 || lay1) {
                put2(pS + rr * SD * WB, ld2(b.cp[0] + i));
                put2(pS + (rr * SD + 1) * WB, ld2(b.cp[2] + i));
            }
            if (B.bottom && B.iz0 + r0 + rr >= B.zb) put2(S.zo + (r0 + rr) * 2 * PT + ix, ld2(b.cp[4] + i));
            make_u(rr, 0, LP[rr], LF[rr], false, a.tag0 + a.j0, copy);
        }
    }
    if (load && B.bottom && B.use)  // Y_z with 4 rows either side
        for (int r = B.seg - kRad; r < nrow + kRad; r += B.nlane) {
            const int gi = B.row0 + r;
            if (gi >= 0 && gi < B.nzi && 4 + gi >= B.zb)
                put2(S.zh + r * PT + ix, ld2(b.cp[1] + so + (long)(4 + gi) * b.pitch + ix));
        }
    const int bz0 = max(max(4, B.zb), B.iz0 - kRad) - B.iz0, bz1 = min(b.nz - 4, B.iz0 + nrow + kRad) - B.iz0;
    const SI *const images = (const SI *)b.store + (long)B.s * b.n_img * 2 * b.slot + i0;
    const int rec_rr = sh.rz - B.iz0 - r0;  // the receivers' row among the thread's
    // the images of global step g at the thread's own points, asked for as soon as the last ones are
    // used, a step before they are needed: 16-bit ones into its own part of the stage, FP32 ones (a
    // stage of theirs would cost two rows a row) into L2
    constexpr bool STAGE = sizeof(SI) == 2;
    SI *const pI = reinterpret_cast<SI *>(S.img) + r0 * 2 * PT + ix;
    auto stage_images = [&](int g) {
        const SI *const image = images + (long)(g - a.img_base) * 2 * b.slot;
        for (int rr = 0; rr < nr; rr++)
            for (int k = 0; k < 2; k++) {
                const SI *const src = image + k * b.slot + (long)rr * b.pitch;
                if constexpr (STAGE) res_copy<2 * sizeof(SI)>(pI + (rr * 2 + k) * PT, src);
                else asm volatile("prefetch.global.L2 [%0];" ::"l"(src));
            }
        if constexpr (STAGE) asm volatile("cp.async.commit_group;" ::: "memory");
    };
    constexpr int LAG = REF ? 1 : 0;
    if (a.j0 < j1 && sh.nt - 1 - LAG - a.j0 >= 0) stage_images(a.ntb - 1 - LAG - a.j0);
    int cur = 0;
    __syncthreads();
    for (int j = a.j0; j < j1; j++) {
        const unsigned tag = a.tag0 + j;
        const int g_img = a.ntb - 1 - LAG - j;
        const bool img = !REF || sh.nt - 2 - j >= 0;
        float *const UZ = S.halo[cur], *const pc = pO + cur * PT;
        // this step's residuals and scale: in flight until the increments are done
        float2 d = both(0.f);
        const float scale = Cd::scaled && img ? b.scale[(long)B.s * b.nt_max + g_img] : 1.f;
        if (rec_rr >= 0 && rec_rr < nr) {
            const float *const res = b.rec + sh.rec_off + (long)(sh.nt - j - 1) * (sh.rx1 - sh.rx0) - sh.rx0 + ix;
            if (ix >= sh.rx0 && ix < sh.rx1) d.x = res[0];
            if (ix + 1 >= sh.rx0 && ix + 1 < sh.rx1) d.y = res[1];
        }
        if (REF && B.side) {
            // as the forward: psi_x, then zeta_x and what the side layers add to Dxx u_x
            const float2 ax = ld2(S.ax + cx), bx = ld2(S.bx + cx);
            for (int rr = 0; rr < nr; rr++) {
                float *const ps = pS + rr * SD * WB;
                put2(ps, keep(fma(bx, ld2(ps), mul(ax, scaled(ResWindow(pc + rr * OWN * PT).d1(), inv_dh))), nval));
            }
            res_side_sync(B);
            for (int rr = 0; rr < nr; rr++) {
                float *const ps = pS + rr * SD * WB;
                const float2 gp = scaled(ResWindow(pc + rr * OWN * PT).d2(), inv_dh2), dx = ResWindow(ps).d1();
                const float2 z = keep(res_zeta(true, bx, ld2(ps + WB), ax, gp, dx, inv_dh), nval);
                const float2 t = res_term(true, dx, inv_dh, z);
                const bool zl = B.iz0 + r0 + rr >= B.zb;
                put2(ps + WB, z);
                put2(ps + 2 * WB, make_float2(lay0 || zl ? t.x : 0.f, lay1 || (zl && nval > 1) ? t.y : 0.f));
            }
        }
        if (!REF && B.side) {
            // Y_x of the side layers: Y' = -D(w) + b Y, w = u at layer points, 0 elsewhere; and a Y'
            const float2 ax = ld2(S.ax + cx), bx = ld2(S.bx + cx);
            for (int rr = 0; rr < nr; rr++) {
                float *const ps = pS + rr * SD * WB;
                const float2 y = fma(bx, ld2(ps), scaled(ResWindow(ps + 3 * WB).d1(), -inv_dh));
                put2(ps, make_float2(lay0 ? y.x : 0.f, lay1 ? y.y : 0.f));
                put2(ps + 2 * WB, make_float2(lay0 ? ax.x * y.x : 0.f, lay1 ? ax.y * y.y : 0.f));
            }
            res_side_sync(B);
            for (int rr = 0; rr < nr; rr++)  // -Dx(a Y) within their reach
                put2(pS + (rr * SD + 4) * WB, scaled(ResWindow(pS + (rr * SD + 2) * WB).d1(), -inv_dh));
        }
        if (j > a.j0 || load) res_halo_in<PT>(B, UZ, res_words<PT>(B, a.x, a.slots, copy, B.row0, ix), tag, &dead, b.status);
        copy = res_next(copy, a.slots);
        __syncthreads();
        if (REF && B.bottom) {
            // psi_z, then zeta_z and what the bottom layer adds to Dzz u_z, as the forward
            res_rows<PT>(B, bz0, bz1, UZ, [&](int r, const float2 *uz) {
                float *const ps = S.zh + r * PT + ix;
                put2(ps, keep(fma(both(S.bz[r]), ld2(ps), mul(both(S.az[r]), scaled(res_d1z(uz), inv_dh))), nval));
                if (r >= 0 && r < nrow) put2(S.zo + (r * 2 + 1) * PT + ix, scaled(res_d2z(uz), inv_dh2));
            });
            __syncthreads();
            res_rows<PT>(B, max(B.zb - 4 - B.iz0, 0), nrow, S.zh, [&](int r, const float2 *pz) {
                float *const z = S.zo + r * 2 * PT + ix;
                const float2 dz = res_d1z(pz);
                float2 t;
                if (B.iz0 + r >= B.zb) {
                    const float2 n = keep(res_zeta(true, both(S.bz[r]), ld2(z), both(S.az[r]), ld2(z + PT), dz, inv_dh), nval);
                    put2(z, n);
                    t = res_term(true, dz, inv_dh, n);
                } else {
                    t = scaled(dz, inv_dh);
                    t = make_float2(lay0 ? t.x : 0.f, lay1 ? t.y : 0.f);
                }
                put2(z + PT, t);
            });
            __syncthreads();
        }
        if (!REF && B.bottom) {
            // Y_z of the bottom layer's points of the own rows and 4 either side
            res_rows<PT>(B, bz0, bz1, UZ, [&](int r, const float2 *uz) {
                const int iz = B.iz0 + r;
                float *const y = S.zh + r * PT + ix;
                float2 w[9];
#pragma unroll
                for (int k = 0; k < 9; k++)  // rows above the bottom layer count only in the side layers
                    w[k] = k < 4 && iz - 4 + k < B.zb ? make_float2(lay0 ? uz[k].x : 0.f, lay1 ? uz[k].y : 0.f) : uz[k];
                put2(y, keep(fma(both(S.bz[r]), ld2(y), scaled(res_d1z(w), -inv_dh)), nval));
            });
            __syncthreads();
            // -Dz(a Y) within reach of the bottom layer
            res_rows<PT>(B, max(B.zb - 4 - B.iz0, 0), nrow, S.zh, [&](int r, const float2 *y) {
                float2 w[9];
#pragma unroll
                for (int k = 0; k < 9; k++) w[k] = mul(both(S.az[r - 4 + k]), y[k]);
                put2(S.zo + (r * 2 + 1) * PT + ix, scaled(res_d1z(w), -inv_dh));
            });
            __syncthreads();
        }
        // lambda^m: increments += Dxx(u) - Dx(a Y) (and z), residual at the receivers; imaging; the
        // next step's u
        if constexpr (STAGE) asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (nr > 0) {
            const float inv_sc = Cd::scaled ? 1.f / scale : 1.f;
            const float2 kk = both(b.img_scale);
            const float *const uc = UZ + r0 * PT + ix;
            float2 win[R + 8];
#pragma unroll
            for (int k = 0; k < 8; k++) win[k] = ld2(uc + (k - 4) * PT);
#pragma unroll
            for (int rr = 0; rr < R; rr++) {
                if (rr >= nr) break;
                win[rr + 8] = ld2(uc + (rr + 4) * PT);
                float *const o = pO + rr * OWN * PT;
                float2 ex = scaled(ResWindow(pc + rr * OWN * PT).d2(), inv_dh2), ez = scaled(res_d2z(win + rr), inv_dh2);
                if (B.side) ex = add(ex, ld2(pS + (rr * SD + (REF ? 2 : 4)) * WB));
                if (B.bottom) ez = add(ez, ld2(S.zo + ((r0 + rr) * 2 + 1) * PT + ix));
                WP[rr] = add(WP[rr], ex);
                WF[rr] = add(WF[rr], ez);
                if (rr == rec_rr) {
                    WP[rr] = add(WP[rr], d);
                    WF[rr] = add(WF[rr], d);
                }
                if (nval < 2) WP[rr].y = WF[rr].y = 0.f;
                LP[rr] = add(LP[rr], WP[rr]);
                LF[rr] = add(LF[rr], WF[rr]);
                make_u(rr, 1 - cur, LP[rr], LF[rr], true, tag + 1, copy);
                if (!img) continue;
                const SI *const image = images + (long)(g_img - a.img_base) * 2 * b.slot + (long)rr * b.pitch;
                const float2 gi = keep(mul(kk, Img::value(STAGE ? pI + rr * 2 * PT : image, inv_sc)), nval),
                             hi = keep(mul(kk, Img::value(STAGE ? pI + (rr * 2 + 1) * PT : image + b.slot, inv_sc)), nval);
                put2(o + 5 * PT, fma(gi, LP[rr], ld2(o + 5 * PT)));
                put2(o + 6 * PT, fma(hi, add(LP[rr], LF[rr]), ld2(o + 6 * PT)));
                put2(o + 7 * PT, fma(gi, LF[rr], ld2(o + 7 * PT)));
            }
        }
        if (j + 1 < j1 && (!REF || sh.nt - 3 - j >= 0)) stage_images(g_img - 1);
        __syncthreads();  // the next u; this one and Y read
        cur ^= 1;
    }
    // the shot's gradient, and the state for the next launch
    const bool save = a.j1 < sh.nt;
#pragma unroll
    for (int rr = 0; rr < R; rr++) {
        if (rr >= nr) break;
        const long i = so + i0 + (long)rr * b.pitch;
        const float *const o = pO + rr * OWN * PT;
        put2(b.g[0] + i, add(ld2(b.g[0] + i), ld2(o + 5 * PT)));
        put2(b.g[1] + i, add(ld2(b.g[1] + i), ld2(o + 6 * PT)));
        put2(b.g[2] + i, add(ld2(b.g[2] + i), ld2(o + 7 * PT)));
        if (!save) continue;
        put2(b.lvl[0] + i, LP[rr]);
        put2(b.lvl[2] + i, LF[rr]);
        put2(b.lvl[4] + i, WP[rr]);
        put2(b.lvl[5] + i, WF[rr]);
        if (lay0 || lay1) {
            put2(b.cp[0] + i, ld2(pS + rr * SD * WB));
            put2(b.cp[2] + i, ld2(pS + (rr * SD + 1) * WB));
        }
        if (B.bottom) {
            put2(b.cp[1] + i, ld2(S.zh + (r0 + rr) * PT + ix));
            put2(b.cp[4] + i, ld2(S.zo + (r0 + rr) * 2 * PT + ix));
        }
    }
}

// ------------------------------------------------------------------ launches

template <typename Args> using ResKernel = void (*)(Batch<float>, ResidentGrid, Args);

template <int ST, bool REF> ResKernel<ResAdjArgs> res_adj_kernel(int pitch)
{
    switch (pitch) {
    case 96: return k_resident_adj<ST, 96, REF>;
    case 160: return k_resident_adj<ST, 160, REF>;
    case 224: return k_resident_adj<ST, 224, REF>;
    case 320: return k_resident_adj<ST, 320, REF>;
    case 400: return k_resident_adj<ST, 400, REF>;
    case 512: return k_resident_adj<ST, 512, REF>;
    case 640: return k_resident_adj<ST, 640, REF>;
    default: return nullptr;
    }
}
template <bool REF> ResKernel<ResAdjArgs> res_adj_kernel(int store_type, int pitch)
{
    return store_type == kStoreHalf ? res_adj_kernel<kStoreHalf, REF>(pitch)
           : store_type == kStoreBf16 ? res_adj_kernel<kStoreBf16, REF>(pitch) : res_adj_kernel<kStoreNative, REF>(pitch);
}

// Cooperative: every CTA of the launch is resident before any of them waits on another.
template <typename Args>
cudaError_t res_launch(ResKernel<Args> k, const Batch<float> &b, const ResidentSet &set, const Args &a, cudaStream_t st)
{
    if (!k) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(set.grid.n);
    cfg.blockDim = dim3(set.threads);
    cfg.dynamicSmemBytes = set.smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, b, set.grid, a);
}

// Every kernel of a table may take `smem` bytes of dynamic shared memory.
template <typename Kernel> bool res_allow(Kernel kernel, int smem)
{
    bool ok = true;
    for (int st : {(int)kStoreNative, (int)kStoreHalf, (int)kStoreBf16})
        for (int p : kResPitches)
            if (const void *k = (const void *)kernel(st, p))
                ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
    return ok;
}

}  // namespace fwi
