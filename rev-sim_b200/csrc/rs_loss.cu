// rs_loss.cu -- smoothed-RDF loss and its gradient on the device.
//
// rdf_differentiable (water.jl:631-691): every (set1, set2) atom pair at minimum-image
// distance d != 0 is smeared over the grid x_k = x_min + step*k with
// g_k(d) = exp(-(x_k - d)^2 / width), restricted to the window |x_k - d| <= cutoff and
// normalised by den(d) = sum of g_k over the index window [ceil((d-c)/step) - off,
// floor((d+c)/step) - off] (water.jl:660-667); h_k = V / (4 pi n1 n2 step) * sum / x_k^2.
// The loss (loss_rdf_part, water.jl:693-697) compares a strided slice of h with a
// target; the gradient is the analytic derivative of the same windowed sums (the
// quantity Enzyme differentiates in the reference's pullback, water.jl:715-736).
// The loss and its gradient read h at the slice points only, so the loss kernels (k_rdf_loss)
// smear only the pairs those points can see onto those points; the whole histogram
// (revsim_rdf) is k_rdf's.  FP64 throughout; the window's Gaussians by a two-multiplication
// recurrence re-anchored on exp every 16 points.
#include <cmath>
#include <mutex>

#include "revsim.h"
#include "rs_internal.h"

namespace rs {

namespace {

__device__ __forceinline__ int rdf_atom(int sel, int atom0, int i) {
    return sel == 0 ? atom0 + 3 * i : atom0 + 3 * (i >> 1) + 1 + (i & 1);
}

__device__ __forceinline__ double grid_x(const RdfArgs &a, int k) {
    return __dadd_rn(a.x_min, __dmul_rn(a.step, (double)k));
}

// Normaliser window, 0-based inclusive.
__device__ __forceinline__ void den_window(const RdfArgs &a, double d, int &lo, int &hi) {
    long long s = (long long)ceil(__ddiv_rn(__dsub_rn(d, a.cutoff), a.step)) - a.off;
    long long e = (long long)floor(__ddiv_rn(__dadd_rn(d, a.cutoff), a.step)) - a.off;
    if (s < 1) s = 1;
    if (e > a.n_grid) e = a.n_grid;
    lo = (int)(s - 1);
    hi = (int)(e - 1);
}

// Histogram window: grid points with x - c <= d <= x + c.
__device__ __forceinline__ void hist_window(const RdfArgs &a, double d, int &lo, int &hi) {
    long long s = (long long)floor(__ddiv_rn(__dsub_rn(__dsub_rn(d, a.cutoff), a.x_min), a.step)) - 1;
    long long e = (long long)ceil(__ddiv_rn(__dsub_rn(__dadd_rn(d, a.cutoff), a.x_min), a.step)) + 1;
    if (s < 0) s = 0;
    if (e > a.n_grid - 1) e = a.n_grid - 1;
    int l = (int)s, h = (int)e;
    while (l <= h && !(d <= __dadd_rn(grid_x(a, l), a.cutoff))) l++;
    while (h >= l && !(d >= __dsub_rn(grid_x(a, h), a.cutoff))) h--;
    lo = l;
    hi = h;
}

// The Gaussians g_k = exp(-(x_k - d)^2 / width) of consecutive grid points by the recurrence
// g_{k+1} = g_k r_k, r_{k+1} = r_k q with r_k = exp(-(2 e_k step + step^2) / width) and
// q = exp(-2 step^2 / width): two multiplications per point instead of an exp.  The
// recurrence restarts from exp every kGaussAnchor points, which bounds the accumulated
// rounding at about kGaussAnchor^2 / 2 ulp (~1e-14 relative).
constexpr int kGaussAnchor = 16;

struct Gauss {
    double g, r;
};

// S: the spacing of the points the recurrence visits (a grid step, or a slice stride).
__device__ __forceinline__ void gauss_anchor(const RdfArgs &a, double d, int k, double S, double inv_w,
                                             Gauss &G) {
    const double e = __dsub_rn(grid_x(a, k), d);
    G.g = exp(-__dmul_rn(__dmul_rn(e, e), inv_w));
    G.r = exp(-__dmul_rn(__fma_rn(__dmul_rn(2.0, e), S, __dmul_rn(S, S)), inv_w));
}

__device__ __forceinline__ void gauss_next(Gauss &G, double q) {
    G.g = __dmul_rn(G.g, G.r);
    G.r = __dmul_rn(G.r, q);
}

__device__ __forceinline__ void den_sums(const RdfArgs &a, double d, double inv_w, double q,
                                         double &den, double &dden) {
    int lo, hi;
    den_window(a, d, lo, hi);
    double s = 0.0, ds = 0.0;
    Gauss G{0.0, 0.0};
    for (int k = lo; k <= hi; k++) {
        if (((k - lo) % kGaussAnchor) == 0) gauss_anchor(a, d, k, a.step, inv_w, G);
        const double e = __dsub_rn(grid_x(a, k), d);
        s = __dadd_rn(s, G.g);
        ds = __fma_rn(__dmul_rn(__dmul_rn(G.g, 2.0), e), inv_w, ds);
        gauss_next(G, q);
    }
    den = s;
    dden = ds;
}

// The same sums from the polynomial of the pair's window (RdfDen); false where the window is
// clipped by the grid, is not one of the four of an unclipped pair, or there is no polynomial.
// The window's ends are those of den_window: a product with 1 / step decides them unless it falls
// within 1e-6 of an integer (its rounding is below 1e-9 on any grid of less than 10^6 points),
// where the division does.  The cell only has to hold d to rounding.
__device__ __forceinline__ bool den_poly(const RdfArgs &a, const RdfDen &dn, double inv_step, double d, double &den,
                                         double &dden) {
    if (dn.M == 0) return false;
    const double da = __dsub_rn(d, a.cutoff), db = __dadd_rn(d, a.cutoff);
    double qa = __dmul_rn(da, inv_step), qb = __dmul_rn(db, inv_step);
    if (fabs(__dsub_rn(qa, rint(qa))) < 1e-6 || fabs(__dsub_rn(qb, rint(qb))) < 1e-6 || qb > 1e6) {
        qa = __ddiv_rn(da, a.step);
        qb = __ddiv_rn(db, a.step);
    }
    const long long s = (long long)ceil(qa), e = (long long)floor(qb);
    if (s - a.off < 1 || e - a.off > a.n_grid) return false;
    const double j = floor(__dmul_rn(d, inv_step));
    const int ca = (int)(s - (long long)j) + dn.n, cb = (int)(e - (long long)j) - dn.n;
    if (ca < 0 || ca > 1 || cb < 0 || cb > 1) return false;
    const double u = __dsub_rn(d, __dmul_rn(__dadd_rn(j, 0.5), a.step));
    const double *c = dn.c[2 * ca + cb];
    double v = c[dn.M - 1], dv = 0.0;
    for (int m = dn.M - 2; m >= 0; m--) {
        dv = __fma_rn(dv, u, v);
        v = __fma_rn(v, u, c[m]);
    }
    den = v;
    dden = dv;
    return true;
}

// The whole histogram: one thread per ordered atom pair, shared-memory histogram.
__global__ void k_rdf(RdfArgs a) {
    extern __shared__ double s_hist[];
    const int r = blockIdx.y;
    const int nm = a.rep_nmol[r];
    const int atom0 = a.rep_atom0[r];
    const long long n1 = a.sel1 == 0 ? nm : 2LL * nm;
    const long long n2 = a.sel2 == 0 ? nm : 2LL * nm;
    const double L = a.rep_box[r];
    const bool use_smem = a.n_grid <= 6144;
    double *hist = a.hist + (size_t)r * a.n_grid;
    if (use_smem) {
        for (int k = threadIdx.x; k < a.n_grid; k += blockDim.x) s_hist[k] = 0.0;
        __syncthreads();
    }
    const double inv_w = __drcp_rn(a.width);
    const double q = exp(-__dmul_rn(__dmul_rn(2.0, __dmul_rn(a.step, a.step)), inv_w));
    const double dmin = __dsub_rn(__dsub_rn(a.x_min, a.cutoff), a.step);
    const double dmax = __dadd_rn(__dadd_rn(grid_x(a, a.n_grid - 1), a.cutoff), a.step);
    const long long total = n1 * n2;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < total;
         p += (long long)gridDim.x * blockDim.x) {
        const int i1 = (int)(p / n2), i2 = (int)(p % n2);
        const int ia = rdf_atom(a.sel1, atom0, i1), ib = rdf_atom(a.sel2, atom0, i2);
        const double *xa = a.x + 3 * (size_t)ia, *xb = a.x + 3 * (size_t)ib;
        double dr[3];
#pragma unroll
        for (int u = 0; u < 3; u++) dr[u] = vec1d(xa[u], xb[u], L);
        const double d = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dr[0], dr[0]), __dmul_rn(dr[1], dr[1])),
                                              __dmul_rn(dr[2], dr[2])));
        if (d == 0.0 || d < dmin || d > dmax) continue;
        int lo, hi;
        hist_window(a, d, lo, hi);
        if (lo > hi) continue;
        double den, dden;
        den_sums(a, d, inv_w, q, den, dden);
        const double inv_den = __drcp_rn(den);
        Gauss G{0.0, 0.0};
        for (int k = lo; k <= hi; k++) {
            if (((k - lo) % kGaussAnchor) == 0) gauss_anchor(a, d, k, a.step, inv_w, G);
            const double g = __dmul_rn(G.g, inv_den);
            if (use_smem)
                atomicAdd(s_hist + k, g);
            else
                atomicAdd(hist + k, g);
            gauss_next(G, q);
        }
    }
    if (use_smem) {
        __syncthreads();
        for (int k = threadIdx.x; k < a.n_grid; k += blockDim.x)
            if (s_hist[k] != 0.0) atomicAdd(hist + k, s_hist[k]);
    }
}

// The slice points' sums (GRAD false) and the loss gradient from their weights (true).
//
// A warp owns one atom i of the first set; the CTA's eight stage the second set in tiles of
// 256 FP32 positions, and each lane tests one tile atom against the distances the slice can
// see (an FP32 test with a margin far above its rounding).  The atoms that pass are queued
// per warp and evaluated 32 at a time in FP64, so the window loops run with full warps
// whatever the fraction in range (5 % in the 4.5 nm box).  Equal sets take each unordered
// pair once (half ring: i with the next n/2 atoms, modulo n) and count it twice.  The gradient
// sums atom i's share in registers.
//
// The value kernel deposits with PTS = 16 or 32 lanes a pair, a lane per slice point, into
// copies of the slice sums that no other group of lanes touches: plain additions.  PTS = 0 (the
// window has more points, the sums are too many for the copies, or the factors too far apart)
// deposits with a lane per pair, shared-memory FP64 atomics on a copy per lane where they fit.
//
// Window ends and normaliser cells come from products with 1 / S and 1 / step: divisions only
// where those lie within 1e-6 of an integer.  The window's ends take two steps without branches:
// loops that few lanes repeat left a warp's lanes apart for the whole pair (66 us instead of 38 a
// gradient on the 895-water box).
//
// Bound by FP64 latency at 16 to 24 warps an SM (three CTAs an SM at 80 registers suit PTS = 16, 60 ->
// 54 us, and PTS = 0, 3,000 waters, O-H, 400 points a window 7.8 -> 4.7 ms; the others slow by 3-5 us).  Us per value / gradient, mean over the O-O and O-H
// terms of the experimental grid (4,801 points, of which the loss reads 248 and 281; 27 a window)
// on the 895-water box, and the 200-bin O-O term (16 a window) on the 3,000-water box: every
// ordered pair over the whole grid, as k_rdf does, 567 / 535 and 215 / 298; a lane per pair with
// atomics on eight copies and divisions 63 / 44 and 67 / 76; now 41 / 28 and 54 / 44 (the gradient by
// sums 52 where a window has 16 points, per point 38 where it has 27).
constexpr int kRlWarps = 8, kRlTile = 256;
constexpr size_t kRlSmem = 65536;   // dynamic shared memory of a value CTA at most

template <bool GRAD, int PTS>
__global__ void __launch_bounds__(32 * kRlWarps, !GRAD && PTS != 32 ? 3 : 0) k_rdf_loss(RdfArgs a, RdfSlice sl, RdfDen dn, int split,
                                                            int ncopy) {
    constexpr bool COOP = !GRAD && PTS > 0;
    constexpr int W = PTS ? PTS : 32;   // lanes a pair
    constexpr int NC = COOP ? 64 / W : 0;   // pairs deposited at a time, copies of the sums a warp
    // GRAD false: [nt][ncopy] partial sums (ncopy 0: none; COOP: [warps][NC][nt])
    extern __shared__ double s_sum[];
    __shared__ double2 s_g[COOP ? kRlWarps : 1][COOP ? 32 : 1];   // a pair's first point and ratio
    __shared__ int2 s_t[COOP ? kRlWarps : 1][COOP ? 32 : 1];      // its first point's index and their number
    __shared__ float s_x[3][kRlTile];
    __shared__ int s_q[kRlWarps][64];
    const int r = blockIdx.y, nm = a.rep_nmol[r], atom0 = a.rep_atom0[r];
    const bool same = a.sel1 == a.sel2;
    const int n1 = a.sel1 == 0 ? nm : 2 * nm, n2 = a.sel2 == 0 ? nm : 2 * nm;
    const int i0 = (int)(blockIdx.x / split) * kRlWarps, part = (int)(blockIdx.x % split);
    if (i0 >= n1) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = i0 + warp;
    // tile positions p of the CTA: atom (i0 + 1 + p) mod n for equal sets, atom p otherwise
    const int half = n1 / 2;
    const int np = same ? half + kRlWarps - 1 : n2;
    const int nunit = (np + 31) / 32;   // the CTA's share of the positions, in units of a warp's test
    const int p0 = 32 * (int)((long long)nunit * part / split),
              p1 = min(np, 32 * (int)((long long)nunit * (part + 1) / split));
    if (p0 >= p1) return;
    const double L = a.rep_box[r];
    const float Lf = (float)L, hLf = 0.5f * Lf;
    const double inv_w = __drcp_rn(a.width);
    const double S = __dmul_rn(a.step, (double)sl.sd);   // slice spacing
    const double inv_step = __drcp_rn(a.step), inv_S = __drcp_rn(S), x0 = grid_x(a, sl.s0);
    const double q1 = exp(-__dmul_rn(__dmul_rn(2.0, __dmul_rn(a.step, a.step)), inv_w));
    const double qS = exp(-__dmul_rn(__dmul_rn(2.0, __dmul_rn(S, S)), inv_w));
    const double dmin = __dsub_rn(__dsub_rn(grid_x(a, sl.s0), a.cutoff), a.step);
    const double dmax = __dadd_rn(__dadd_rn(grid_x(a, sl.s0 + (sl.nt - 1) * sl.sd), a.cutoff), a.step);
    // FP32 coordinates of atoms within 16 boxes of the origin (NaN beyond, which decides nothing):
    // their distances err by < 4e-6 L, a margin that no pair in range can miss
    const double xmax = 16.0 * L;
    auto test_x = [xmax](double x) { return fabs(x) <= xmax ? (float)x : __int_as_float(0x7FC00000); };
    const float marg = 1e-3f + 1e-5f * Lf;
    const float far = (float)dmax + marg, near = fmaxf(0.f, (float)dmin - marg);
    const float far2 = far * far, near2 = near * near;
    const double pair_w = same ? 2.0 : 1.0;
    if (COOP) {
        for (int k = threadIdx.x; k < sl.nt * NC * kRlWarps; k += blockDim.x) s_sum[k] = 0.0;
    } else if (!GRAD && ncopy > 0) {
        for (int k = threadIdx.x; k < sl.nt * ncopy; k += blockDim.x) s_sum[k] = 0.0;
    }
    double xi[3] = {0.0, 0.0, 0.0};
    float xf[3] = {0.f, 0.f, 0.f};
    const bool live = i < n1;
    const int ia = rdf_atom(a.sel1, atom0, live ? i : 0);
    if (live) {
#pragma unroll
        for (int u = 0; u < 3; u++) {
            xi[u] = a.x[3 * (size_t)ia + u];
            xf[u] = test_x(xi[u]);
        }
    }
    // equal sets: atom i takes the pairs (i, i + k mod n), k = 1 .. n/2, the last of them (n
    // even) only for i < n/2, so that each unordered pair comes once
    const int kmax = !live ? -1 : (n1 % 2 == 0 && i >= half ? half - 1 : half);
    double gi[3] = {0.0, 0.0, 0.0};
    double *sums = sl.sum + (size_t)r * sl.nt;
    const double *wt = sl.wt + (size_t)r * sl.nt;

    // COOP: lane m of PTS deposits point m of a pair, exp(-(e0 + m S)^2 / w) = exp(-e0^2 / w) r^m A_m
    // with r = exp(-2 e0 S / w)
    const int m = COOP ? lane % W : 0, group = COOP ? lane / W : 0;
    const double Am = COOP ? exp(-__dmul_rn(__dmul_rn((double)m * S, (double)m * S), inv_w)) : 0.0;
    double *mine = s_sum + (COOP ? ((size_t)warp * NC + group) * sl.nt : 0);

    // The pair of atom i with atom j: the slice points ta .. tb it reaches, its distance,
    // displacement and normaliser; false if there are none.
    auto pair_of = [&](int j, double dr[3], double &d, int &ta, int &tb, double &inv_den, double &dden) {
        const double *xb = a.x + 3 * (size_t)rdf_atom(a.sel2, atom0, j);
#pragma unroll
        for (int u = 0; u < 3; u++) dr[u] = vec1d(xi[u], xb[u], L);
        d = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dr[0], dr[0]), __dmul_rn(dr[1], dr[1])),
                                              __dmul_rn(dr[2], dr[2])));
        if (d == 0.0 || !(d >= dmin && d <= dmax)) return false;
        // The slice points of the window, x - c <= d <= x + c.  The product with 1 / S, rounded
        // outwards, is the first (last) of them, the point before it or, within its rounding of a
        // point, the one before that: two steps inwards without branches.
        ta = (int)floor(__dmul_rn(__dsub_rn(__dsub_rn(d, a.cutoff), x0), inv_S));
        tb = (int)ceil(__dmul_rn(__dsub_rn(__dadd_rn(d, a.cutoff), x0), inv_S));
#pragma unroll
        for (int q = 0; q < 2; q++) {
            ta += d <= __dadd_rn(grid_x(a, sl.s0 + ta * sl.sd), a.cutoff) ? 0 : 1;
            tb -= d >= __dsub_rn(grid_x(a, sl.s0 + tb * sl.sd), a.cutoff) ? 0 : 1;
        }
        ta = max(ta, 0);
        tb = min(tb, sl.nt - 1);
        if (ta > tb) return false;
        double den;
        if (!den_poly(a, dn, inv_step, d, den, dden)) den_sums(a, d, inv_w, q1, den, dden);
        inv_den = __drcp_rn(den);
        return true;
    };
    auto eval = [&](int j, bool on) {
        double dr[3], d = 0.0, inv_den = 0.0, dden = 0.0;
        int ta = 0, tb = -1;
        on = on && pair_of(j, dr, d, ta, tb, inv_den, dden);
        if constexpr (COOP) {
            double2 g = make_double2(0.0, 1.0);
            if (on) {
                const double e0 = __dsub_rn(grid_x(a, sl.s0 + ta * sl.sd), d), c = __dmul_rn(pair_w, inv_den);
                g.x = __dmul_rn(c, exp(-__dmul_rn(__dmul_rn(e0, e0), inv_w)));
                g.y = exp(-__dmul_rn(__dmul_rn(__dmul_rn(2.0, e0), S), inv_w));
                // a window of one point more than the lanes: both its ends on slice points
                for (int t = ta + PTS; t <= tb; t++) {
                    const double e = __dsub_rn(grid_x(a, sl.s0 + t * sl.sd), d);
                    atomicAdd(sums + t, __dmul_rn(c, exp(-__dmul_rn(__dmul_rn(e, e), inv_w))));
                }
            }
            s_g[warp][lane] = g;
            s_t[warp][lane] = make_int2(ta, tb - ta + 1);
            __syncwarp();
            for (int p = 0; p < 32; p += NC) {
                // NC pairs at a time, two a group of lanes, each into its own copy of the sums
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int q = p + h * (32 / PTS) + group;
                    const double2 gp = s_g[warp][q];
                    const int2 tp = s_t[warp][q];
                    double r = gp.y, v = __dmul_rn(gp.x, Am);
#pragma unroll
                    for (int b = 1; b < PTS; b <<= 1) {
                        v = __dmul_rn(v, m & b ? r : 1.0);
                        r = __dmul_rn(r, r);
                    }
                    if (m < tp.y) {
                        double *at = mine + (size_t)h * (32 / PTS) * sl.nt + tp.x + m;
                        *at = __dadd_rn(*at, v);
                    }
                }
                __syncwarp();
            }
            return;
        }
        if (!on) return;
        const int ib = rdf_atom(a.sel2, atom0, j);
        Gauss G{0.0, 0.0};
        if (!GRAD) {
            const double c = __dmul_rn(pair_w, inv_den);
            for (int t = ta; t <= tb; t++) {
                if (!sl.recur || ((t - ta) % kGaussAnchor) == 0) gauss_anchor(a, d, sl.s0 + t * sl.sd, S, inv_w, G);
                const double g = __dmul_rn(G.g, c);
                if (ncopy > 0)
                    atomicAdd(s_sum + (size_t)t * ncopy + (lane & (ncopy - 1)), g);
                else
                    atomicAdd(sums + t, g);
                gauss_next(G, qS);
            }
        } else {
            // dL/dd = sum_t wt (g' / den - g den' / den^2)
            double dLdd = 0.0;
            if constexpr (PTS == 16) {
                const double dd2 = __dmul_rn(dden, __dmul_rn(inv_den, inv_den));
                for (int t = ta; t <= tb; t++) {
                    if (!sl.recur || ((t - ta) % kGaussAnchor) == 0) gauss_anchor(a, d, sl.s0 + t * sl.sd, S, inv_w, G);
                    const double e = __dsub_rn(grid_x(a, sl.s0 + t * sl.sd), d);
                    const double gp = __dmul_rn(__dmul_rn(__dmul_rn(G.g, 2.0), e), inv_w);
                    dLdd = __fma_rn(wt[t], __dsub_rn(__dmul_rn(gp, inv_den), __dmul_rn(G.g, dd2)), dLdd);
                    gauss_next(G, qS);
                }
            } else {
                // the same from the sums of wt g and wt g e, g' = 2 e g / w: half the instructions a point, at
                // 113 registers (two CTAs an SM; the other form's 80 hold three)
                double s0 = 0.0, s1 = 0.0;
                const double e0 = __dsub_rn(grid_x(a, sl.s0 + ta * sl.sd), d);
                const int run = sl.recur ? kGaussAnchor : 1;
                for (int t = ta; t <= tb; t += run) {
                    gauss_anchor(a, d, sl.s0 + t * sl.sd, S, inv_w, G);
                    const int t1 = min(t + run - 1, tb);
                    for (int q = t; q <= t1; q++) {
                        const double p = __dmul_rn(wt[q], G.g);
                        s0 = __dadd_rn(s0, p);
                        s1 = __fma_rn(p, __fma_rn((double)(q - ta), S, e0), s1);
                        gauss_next(G, qS);
                    }
                }
                dLdd = __dsub_rn(__dmul_rn(__dmul_rn(__dmul_rn(2.0, inv_w), s1), inv_den),
                                 __dmul_rn(__dmul_rn(s0, dden), __dmul_rn(inv_den, inv_den)));
            }
            if (dLdd != 0.0) {
                const double s = __ddiv_rn(__dmul_rn(pair_w, dLdd), d);
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    const double gu = __dmul_rn(s, dr[u]);
                    atomicAdd(a.dLdx + 3 * (size_t)ib + u, gu);
                    gi[u] = __dsub_rn(gi[u], gu);
                }
            }
        }
    };

    int nq = 0;
    for (int pt = p0; pt < p1; pt += kRlTile) {
        __syncthreads();
        {
            const int p = pt + threadIdx.x;
            if (p < p1) {
                const int j = same ? (i0 + 1 + p) % n1 : p;
                const double *xj = a.x + 3 * (size_t)rdf_atom(a.sel2, atom0, j);
#pragma unroll
                for (int u = 0; u < 3; u++) s_x[u][threadIdx.x] = test_x(xj[u]);
            }
        }
        __syncthreads();
        for (int b = 0; b < kRlTile && pt + b < p1; b += 32) {
            const int p = pt + b + lane;
            // equal sets: k = j - i before the ring's wrap
            const int k = i0 + 1 + p - i;
            bool ok = p < p1 && (same ? k >= 1 && k <= kmax : live);
            if (ok) {
                float r2 = 0.f;
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    float d = s_x[u][b + lane] - xf[u];
                    d = d > hLf ? d - Lf : (d < -hLf ? d + Lf : d);
                    r2 = fmaf(d, d, r2);
                }
                ok = !(r2 > far2) && !(r2 < near2);
            }
            const unsigned m = __ballot_sync(0xffffffffu, ok);
            if (ok) {
                const int j = !same ? p : (i + k < n1 ? i + k : i + k - n1);
                s_q[warp][nq + __popc(m & ((1u << lane) - 1u))] = j;
            }
            nq += __popc(m);
            __syncwarp();
            if (nq >= 32) {
                nq -= 32;
                eval(s_q[warp][nq + lane], true);
                __syncwarp();
            }
        }
    }
    if (nq > 0) eval(s_q[warp][min(lane, nq - 1)], lane < nq);
    if (GRAD) {
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 3; u++) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) gi[u] += __shfl_xor_sync(0xffffffffu, gi[u], o);
            if (lane == 0 && live && gi[u] != 0.0) atomicAdd(a.dLdx + 3 * (size_t)ia + u, gi[u]);
        }
    } else if (COOP) {
        __syncthreads();
        for (int t = threadIdx.x; t < sl.nt; t += blockDim.x) {
            double v = 0.0;
            for (int c = 0; c < NC * kRlWarps; c++) v += s_sum[(size_t)c * sl.nt + t];
            if (v != 0.0) atomicAdd(sums + t, v);
        }
    } else if (ncopy > 0) {
        __syncthreads();
        for (int t = threadIdx.x; t < sl.nt; t += blockDim.x) {
            double v = 0.0;
            // (rotated: the threads of a warp read different banks)
            for (int c = 0; c < ncopy; c++) v += s_sum[(size_t)t * ncopy + ((c + t) & (ncopy - 1))];
            if (v != 0.0) atomicAdd(sums + t, v);
        }
    }
}

// h = pre sum / x^2 at the slice points, loss += weight sum |h - target|^norm, and the
// gradient's weights dL/dh pre / x^2.  One CTA per replica.
__global__ void __launch_bounds__(256) k_rdf_loss_finalize(RdfArgs a, RdfSlice sl, const double *pre,
                                                           const double *target, int norm, double weight,
                                                           double *loss) {
    __shared__ double s_l[256];
    const int r = blockIdx.x;
    const double *sum = sl.sum + (size_t)r * sl.nt;
    double *wt = sl.wt + (size_t)r * sl.nt;
    double l = 0.0;
    for (int t = threadIdx.x; t < sl.nt; t += blockDim.x) {
        const double xk = grid_x(a, sl.s0 + t * sl.sd), x2 = __dmul_rn(xk, xk);
        const double e = __dsub_rn(__ddiv_rn(__dmul_rn(pre[r], sum[t]), x2), target[(size_t)r * sl.nt + t]);
        double g;
        if (norm == 1) {
            l = __dadd_rn(l, fabs(e));
            g = weight * (e > 0.0 ? 1.0 : (e < 0.0 ? -1.0 : 0.0));
        } else {
            l = __dadd_rn(l, __dmul_rn(e, e));
            g = __dmul_rn(weight, __dmul_rn(2.0, e));
        }
        wt[t] = g == 0.0 ? 0.0 : __ddiv_rn(__dmul_rn(g, pre[r]), x2);   // (x = 0 with no weight)
    }
    s_l[threadIdx.x] = l;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) s_l[threadIdx.x] = __dadd_rn(s_l[threadIdx.x], s_l[threadIdx.x + o]);
        __syncthreads();
    }
    if (threadIdx.x == 0) loss[r] = __dadd_rn(loss[r], __dmul_rn(weight, s_l[0]));
}

// h_k = pre * sum_k / x_k^2.  One CTA per replica.
__global__ void k_rdf_scale(RdfArgs a, const double *pre) {
    const int r = blockIdx.x;
    double *h = a.hist + (size_t)r * a.n_grid;
    for (int k = threadIdx.x; k < a.n_grid; k += blockDim.x) {
        const double xk = grid_x(a, k);
        h[k] = __ddiv_rn(__dmul_rn(pre[r], h[k]), __dmul_rn(xk, xk));
    }
}

}  // namespace

cudaError_t launch_rdf(const RdfArgs &a, int R, int max_n1, int max_n2, const double *pre, cudaStream_t st) {
    const long long pairs = (long long)max_n1 * max_n2;
    long long blocks = (pairs + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    if (blocks < 1) blocks = 1;
    const size_t smem = a.n_grid <= 6144 ? sizeof(double) * a.n_grid : 0;
    k_rdf<<<dim3((unsigned)blocks, R), 256, smem, st>>>(a);
    k_rdf_scale<<<R, 256, 0, st>>>(a, pre);
    return cudaGetLastError();
}

// den(d) of an unclipped pair depends only on where d lies in its grid cell: with j the cell,
// u = d - (j + 1/2) step, the window is [j - n + a, j + n + b], a, b in {0, 1}, and
// exp(-(e - u)^2 / w) = sum_m A_m(e) u^m with A_0 = exp(-e^2 / w), A_1 = (2 e / w) A_0,
// A_{m+1} = ((2 e / w) A_m - (2 / w) A_{m-1}) / (m + 1) (Hermite's recurrence).  The series is
// cut where its terms at |u| = step / 2 fall below 1e-18 of the sum; a grid too coarse for
// that within kMaxTerms keeps the direct sum (M = 0).
RdfDen rdf_den_poly(double step, double width, double cutoff) {
    constexpr int T = RdfDen::kMaxTerms;
    RdfDen dn;
    dn.M = 0;
    const double cells = std::floor(cutoff / step);
    if (!(cells < 4096.0)) return dn;
    dn.n = (int)cells;
    double inner[T + 2] = {}, edge[2][T + 2] = {}, mag[T + 2] = {};   // edge: k = -n and n + 1
    for (int k = -dn.n; k <= dn.n + 1; k++) {
        const double e = (k - 0.5) * step, w2 = 2.0 / width;
        double *c = k == -dn.n ? edge[0] : (k == dn.n + 1 ? edge[1] : inner);
        double p0 = 0.0, p1 = std::exp(-e * e / width), h = 1.0;
        for (int m = 0; m < T + 2; m++) {
            c[m] += p1;
            mag[m] += std::fabs(p1) * h;
            const double p2 = (w2 * e * p1 - w2 * p0) / (m + 1);
            p0 = p1;
            p1 = p2;
            h *= 0.5 * step;
        }
    }
    for (int m = 1; m <= T; m++)
        if (mag[m] < 1e-18 * mag[0] && mag[m + 1] < 1e-18 * mag[0]) {
            dn.M = m;
            break;
        }
    for (int ca = 0; ca < 2; ca++)
        for (int cb = 0; cb < 2; cb++)
            for (int m = 0; m < T; m++)
                dn.c[2 * ca + cb][m] = inner[m] + (ca ? 0.0 : edge[0][m]) + (cb ? edge[1][m] : 0.0);
    return dn;
}

// split: CTAs per eight first atoms.  Two an SM, of whole tiles while every SM has one at least, else of
// less (150 waters, O-H, 700 points of which 41 a window, value alone: 51 us a call, 121 with two tiles
// a group, 53 as k_rdf does it).  A lane per pair evaluates long windows, three CTAs an SM, and their
// CTAs' times differ: nine an SM (895 waters, O-H, value alone, 200 points a window 572 us a call,
// 694 with three an SM, 1,009 with two, 724 as k_rdf; 160 points a window of 4,000 785 and 805).  ncopy: as many
// shared-memory copies of the slice sums (a power of two, at most 32) as kRlSmem holds.
cudaError_t launch_rdf_loss(const RdfArgs &a, const RdfSlice &sl, const RdfDen &dn, int R, int max_n1, int max_n2,
                            const double *pre, const double *target, int norm, double weight, bool grad,
                            double *loss, cudaStream_t st) {
    if (sl.nt < 1) return cudaSuccess;
    const int groups = (max_n1 + kRlWarps - 1) / kRlWarps;
    const int np = a.sel1 == a.sel2 ? max_n1 / 2 + kRlWarps : max_n2;
    const int tiles = (np + kRlTile - 1) / kRlTile, units = (np + 31) / 32;
    // a lane per slice point of a pair's window where 16 or 32 cover it and the factors stay finite
    const double points = 2.0 * a.cutoff / (sl.sd * a.step) * (1.0 - 1e-9);
    const bool finite = 4.0 * a.cutoff * a.cutoff <= 300.0 * a.width;
    const auto coop_smem = [&](int pts) { return sizeof(double) * (64 / pts) * kRlWarps * (size_t)sl.nt; };
    const int pts = !finite ? 0 : points <= 16.0 && coop_smem(16) <= kRlSmem ? 16 : points <= 32.0 && coop_smem(32) <= kRlSmem ? 32 : 0;
    const auto ctas = [&](int s) { return (long long)groups * R * s; };
    const int want = (pts ? 2 : 9) * kSMs;
    int split = 1;
    while (split < tiles && ctas(split) < want) split++;
    if (ctas(split) < (pts ? kSMs : want))
        while (split < units && ctas(split) < want) split++;
    int ncopy = 32;
    while (ncopy > 0 && sizeof(double) * ncopy * (size_t)sl.nt > kRlSmem) ncopy >>= 1;
    const auto value = pts == 16 ? k_rdf_loss<false, 16> : pts == 32 ? k_rdf_loss<false, 32> : k_rdf_loss<false, 0>;
    const size_t smem = pts ? coop_smem(pts) : sizeof(double) * ncopy * (size_t)sl.nt;
    const dim3 grid(groups * split, R);
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(value, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRlSmem))) return e;
    if ((e = cudaMemsetAsync(sl.sum, 0, sizeof(double) * (size_t)R * sl.nt, st))) return e;
    value<<<grid, 32 * kRlWarps, smem, st>>>(a, sl, dn, split, ncopy);
    k_rdf_loss_finalize<<<R, 256, 0, st>>>(a, sl, pre, target, norm, weight, loss);
    if (grad) {
        if (pts == 16)
            k_rdf_loss<true, 16><<<grid, 32 * kRlWarps, 0, st>>>(a, sl, dn, split, 0);
        else
            k_rdf_loss<true, 32><<<grid, 32 * kRlWarps, 0, st>>>(a, sl, dn, split, 0);
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Allocation-free RDF loss and gradient for one water box.
//
// Some callers cannot let this library call cudaMalloc: a host that owns every byte
// of device memory through its own pool allocator (a Julia or Python framework that
// hands out device pointers), a loop that must not hit the device-wide
// synchronisation cudaMalloc/cudaFree imply, or a service whose memory is budgeted
// in full before it starts.  For them this entry point takes the caller's device
// buffers and keeps its scratch (the slice sums, the gradient weights, the normalisation constant
// and a one-box table, at most kNoallocMaxGrid grid points) in the file-scope
// array g_rdf_scratch, which every GPU that loads the library holds until the
// process exits.  Host code cannot use the array's name as a device address: the
// address is looked up once per device with cudaGetSymbolAddress, with that device
// current, on the first call that device sees (make that first call before any
// stream capture).  The looked-up address belongs to the device's current context: a
// cudaDeviceReset of that device invalidates it, so the entry point must not be called
// again in a process after it has reset the device.  All calls share the one array and
// leave the last call's values in it; each call clears what must start at zero, and calls
// that overlap on the GPU (concurrent streams, or several host threads on one device) race
// on it.  On an error return the outputs may be partly written.
namespace {

constexpr int kNoallocMaxGrid = 8192;
// layout (doubles): slice sums [kNoallocMaxGrid + 1] (the normaliser V / (4 pi n1 n2 step)
// sits after n_grid entries) | gradient weights [kNoallocMaxGrid] | box [1] |
// {atom0, n_mol} as two ints [1]
constexpr int kNoallocDLdh = kNoallocMaxGrid + 1;
constexpr int kNoallocBox = 2 * kNoallocMaxGrid + 1;
constexpr int kNoallocInts = 2 * kNoallocMaxGrid + 2;
constexpr int kNoallocDoubles = 2 * kNoallocMaxGrid + 3;
static __device__ __align__(256) double g_rdf_scratch[kNoallocDoubles];

__global__ void k_noalloc_tables(double *s, int n_grid, double pre, double box, int n_mol) {
    s[n_grid] = pre;
    s[kNoallocBox] = box;
    int *t = reinterpret_cast<int *>(s + kNoallocInts);
    t[0] = 0;
    t[1] = n_mol;
}

std::mutex g_noalloc_mu;
double *g_noalloc_addr[256] = {};

}  // namespace

}  // namespace rs

extern "C" int32_t revsim_rdf_loss_grad_noalloc(const double *d_x, int32_t n_mol, double box,
                                                const revsim_rdf_term *t, const double *d_target,
                                                double *d_loss, double *d_dLdx, void *stream) {
    using namespace rs;
    if (!d_x || !t || !d_target || !d_loss || !d_dLdx || n_mol < 1 || !(box > 0)) return REVSIM_ERR_BADARG;
    if (t->n_grid < 1 || t->n_grid > kNoallocMaxGrid) return REVSIM_ERR_BADARG;   // beyond the scratch size
    if (!(t->step > 0) || !(t->width > 0) || !(t->exp_cutoff >= 0) || t->n_target < 1 || t->slice_start < 0 ||
        t->slice_stride < 1 || t->slice_start + (long long)(t->n_target - 1) * t->slice_stride >= t->n_grid ||
        (t->norm != 1 && t->norm != 2) || (t->sel1 != 0 && t->sel1 != 1) || (t->sel2 != 0 && t->sel2 != 1))
        return REVSIM_ERR_BADARG;
    const double q = t->x_min / t->step;
    if (std::fabs(q - std::llround(q)) > 1e-6) return REVSIM_ERR_BADARG;
    if (!rdf_term_recurrence_ok(t->step, t->width, t->exp_cutoff)) return REVSIM_ERR_BADARG;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return REVSIM_ERR_CUDA;
    double *s = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_noalloc_mu);
        if (!g_noalloc_addr[dev]) {
            void *p = nullptr;
            if (cudaGetSymbolAddress(&p, g_rdf_scratch) != cudaSuccess || !p) return REVSIM_ERR_CUDA;
            g_noalloc_addr[dev] = static_cast<double *>(p);
        }
        s = g_noalloc_addr[dev];
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const double n1 = t->sel1 == 0 ? n_mol : 2.0 * n_mol;
    const double n2 = t->sel2 == 0 ? n_mol : 2.0 * n_mol;
    const double pre = box * box * box / (4 * 3.14159265358979323846 * n1 * n2 * t->step);
    k_noalloc_tables<<<1, 1, 0, st>>>(s, t->n_grid, pre, box, n_mol);
    if (cudaGetLastError() != cudaSuccess) return REVSIM_ERR_CUDA;
    if (cudaMemsetAsync(d_loss, 0, sizeof(double), st) != cudaSuccess ||
        cudaMemsetAsync(d_dLdx, 0, sizeof(double) * 9 * (size_t)n_mol, st) != cudaSuccess)
        return REVSIM_ERR_CUDA;
    RdfArgs a;
    a.x = d_x;
    a.rep_atom0 = reinterpret_cast<const int *>(s + kNoallocInts);
    a.rep_nmol = a.rep_atom0 + 1;
    a.rep_box = s + kNoallocBox;
    a.sel1 = t->sel1;
    a.sel2 = t->sel2;
    a.x_min = t->x_min;
    a.step = t->step;
    a.width = t->width;
    a.cutoff = t->exp_cutoff;
    a.n_grid = t->n_grid;
    a.off = (int)std::llround(q) - 1;
    a.hist = nullptr;
    a.dLdx = d_dLdx;
    RdfSlice sl = rdf_slice(t->slice_start, t->slice_stride, t->n_target, t->step, t->width, t->exp_cutoff);
    sl.sum = s;
    sl.wt = s + kNoallocDLdh;
    if (launch_rdf_loss(a, sl, rdf_den_poly(t->step, t->width, t->exp_cutoff), 1, (int)n1, (int)n2, s + t->n_grid,
                        d_target, t->norm, t->weight, true, d_loss, st) != cudaSuccess)
        return REVSIM_ERR_CUDA;
    return cudaGetLastError() == cudaSuccess ? REVSIM_OK : REVSIM_ERR_CUDA;
}

