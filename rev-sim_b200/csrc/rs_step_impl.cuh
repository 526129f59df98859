// rs_step_impl.cuh -- fused forward and reverse step kernels for flexible 3-site water
// (included by the per-precision, per-pair-form instantiation files rs_step_*.cu).
//
// Forward step (water.jl:1030-1037): calc_F! (non-bonded water.jl:892-913, bonds
// 915-934, angles 936-968) followed by the B-A-O-A update and the wrap.
// Reverse step (water.jl:1505-1521 and, fused, 1496-1502 of the next step):
// calc_F_and_grads! (water.jl:1212-1433) with the force VJP against
// dl_dfi_prev = accum_C, the contraction of dF/dtheta with A dt^2 / (2m)
// (water.jl:1517-1519, never materialised as a 3N x P matrix), the velocity
// un-kick, the B/A adjoint updates and the un-integration of the next step.
//
// Work decomposition: a group of G lanes owns one molecule; the lanes stride over
// the molecule's neighbour row (entries of 3 atoms each), accumulate the forces of
// the 3 own atoms in registers, and reduce them in the order of a fixed xor butterfly.
// Further warps of the CTA, one lane per atom, form the bonded terms meanwhile and then run
// the FP64 integrator.  Every atom's force is computed by exactly one group in a fixed order,
// so there are no atomics and the forward and reverse kernels produce bit-identical forces.
#pragma once

#include <type_traits>

#include "rs_internal.h"
#include "rs_pack.cuh"

namespace rs {

namespace {

template <typename R>
__device__ __forceinline__ DualN<R, 1> d1(R v, R t) {
    DualN<R, 1> r;
    r.v = v;
    r.d[0] = t;
    return r;
}
template <typename R>
__device__ __forceinline__ DualN<R, 1> d1_sqrt(const DualN<R, 1> &a) {
    const R s = xsqrt(a.v);
    return d1(s, xdiv(a.d[0], xadd(s, s)));
}
__device__ __forceinline__ float r_acos(float c) { return acosf(c); }
__device__ __forceinline__ double r_acos(double c) { return acos(c); }
template <typename R>
__device__ __forceinline__ DualN<R, 1> d1_acos(const DualN<R, 1> &a) {
    return d1(r_acos(a.v), -xdiv(a.d[0], xsqrt(xsub(R(1), xmul(a.v, a.v)))));
}

// Harmonic angle H1-O-H2 (O central) of water.jl:936-968 / 1316-1356 on dual numbers:
// value = the reference's force construction (p1 = a x (a x b) / |.|, p3 = -b x (a x b) / |.|,
// F = k_a (theta0 - theta)), tangent along (w_H1 - w_O, w_H2 - w_O) = J w, which equals
// the reference's J^T w because the Hessian is symmetric.  Returns false when a x b = 0.
template <typename R>
__device__ __forceinline__ bool angle_term(const R a_[3], const R b_[3], const R ta[3],
                                           const R tb[3], R ka, R th0, DualN<R, 1> Fi[3],
                                           DualN<R, 1> Fk[3], R p1d[3], R p3d[3], R &disp) {
    using D = DualN<R, 1>;
    D a[3], b[3];
#pragma unroll
    for (int u = 0; u < 3; u++) {
        a[u] = d1(a_[u], ta[u]);
        b[u] = d1(b_[u], tb[u]);
    }
    const D ra = d1_sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]);
    const D rb = d1_sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
    D cr[3], p1[3], p3[3];
    cr[0] = a[1] * b[2] - a[2] * b[1];
    cr[1] = a[2] * b[0] - a[0] * b[2];
    cr[2] = a[0] * b[1] - a[1] * b[0];
    if (cr[0].v == R(0) && cr[1].v == R(0) && cr[2].v == R(0)) return false;
    p1[0] = a[1] * cr[2] - a[2] * cr[1];
    p1[1] = a[2] * cr[0] - a[0] * cr[2];
    p1[2] = a[0] * cr[1] - a[1] * cr[0];
    const D zero = d1(R(0), R(0));
    p3[0] = zero - (b[1] * cr[2] - b[2] * cr[1]);
    p3[1] = zero - (b[2] * cr[0] - b[0] * cr[2]);
    p3[2] = zero - (b[0] * cr[1] - b[1] * cr[0]);
    const D n1 = d1_sqrt(p1[0] * p1[0] + p1[1] * p1[1] + p1[2] * p1[2]);
    const D n3 = d1_sqrt(p3[0] * p3[0] + p3[1] * p3[1] + p3[2] * p3[2]);
    const D cth = (a[0] * b[0] + a[1] * b[1] + a[2] * b[2]) / (ra * rb);
    const D th = d1_acos(cth);
    const D F = d1(ka, R(0)) * (d1(th0, R(0)) - th);
    const D s1 = n1 * ra, s3 = n3 * rb;
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const D q1 = p1[u] / s1;
        const D q3 = p3[u] / s3;
        Fi[u] = F * q1;
        Fk[u] = F * q3;
        p1d[u] = q1.v;
        p3d[u] = q3.v;
    }
    disp = xsub(th0, th.v);
    return true;
}

// Bonded terms of one molecule in pair precision R: forces Fb on (O, H1, H2); in
// reverse also the VJP Gb against w = C/m and the bonded dtheta contraction with
// acoef.  Intramolecular vectors and bond lengths come from the FP64 state (the
// displacement r - r0 is formed in FP64, so FP32 mode does not lose it to cancellation).
template <typename R, bool REV>
__device__ __forceinline__ void bonded(const double xm[9], double L, const BondConsts &bc,
                                       const R w[9], const R ac[9], R Fb[9], R Gb[9], R tb[4]) {
#pragma unroll
    for (int u = 0; u < 9; u++) {
        Fb[u] = R(0);
        Gb[u] = R(0);
    }
    tb[0] = tb[1] = tb[2] = tb[3] = R(0);
    const R kb = (R)bc.kb;
    R av[2][3];
    // Bonds (O, H1), (O, H2): radial pair with F(r) = -k_b (r - r0), F' = -k_b.
#pragma unroll
    for (int h = 1; h <= 2; h++) {
        double dd[3];
#pragma unroll
        for (int u = 0; u < 3; u++) dd[u] = vec1d(xm[u], xm[3 * h + u], L);
        const double r2d = __dadd_rn(__dadd_rn(__dmul_rn(dd[0], dd[0]), __dmul_rn(dd[1], dd[1])),
                                     __dmul_rn(dd[2], dd[2]));
        const double rd = __dsqrt_rn(r2d);
        const R disp = (R)__dsub_rn(rd, bc.r0);
        R dr[3];
#pragma unroll
        for (int u = 0; u < 3; u++) {
            dr[u] = (R)dd[u];
            av[h - 1][u] = dr[u];
        }
        const R rinv = xrsqrt((R)r2d);
        const R F = -xmul(kb, disp);
        const R Fr = xmul(F, rinv);
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const R f = xmul(Fr, dr[u]);
            Fb[u] = xsub(Fb[u], f);
            Fb[3 * h + u] = xadd(Fb[3 * h + u], f);
        }
        if (REV) {
            // M delta with delta = w_H - w_O: -(F' - F/r) s n - (F/r) delta, s = n . delta
            R dl[3];
#pragma unroll
            for (int u = 0; u < 3; u++) dl[u] = xsub(w[3 * h + u], w[u]);
            const R s = xmul(rinv, xfma(dr[2], dl[2], xfma(dr[1], dl[1], xmul(dr[0], dl[0]))));
            const R k1 = xmul(xmul(xsub(-kb, Fr), s), rinv);
            R t = R(0);
#pragma unroll
            for (int u = 0; u < 3; u++) {
                const R m = -xfma(k1, dr[u], xmul(Fr, dl[u]));
                Gb[u] = xadd(Gb[u], m);
                Gb[3 * h + u] = xsub(Gb[3 * h + u], m);
                t = xfma(xsub(ac[u], ac[3 * h + u]), dr[u], t);
            }
            t = xmul(t, rinv);
            // dF_O/dk_b = disp n, dF_O/dr0 = -k_b n (water.jl:1298-1301)
            tb[0] = xfma(disp, t, tb[0]);
            tb[1] = xfma(-kb, t, tb[1]);
        }
    }
    // Angle H1-O-H2.
    R ta[3], tb3[3];
#pragma unroll
    for (int u = 0; u < 3; u++) {
        ta[u] = REV ? xsub(w[3 + u], w[u]) : R(0);
        tb3[u] = REV ? xsub(w[6 + u], w[u]) : R(0);
    }
    DualN<R, 1> Fi[3], Fk[3];
    R p1d[3], p3d[3], disp;
    if (angle_term<R>(av[0], av[1], ta, tb3, (R)bc.ka, (R)bc.th0, Fi, Fk, p1d, p3d, disp)) {
        R t = R(0);
#pragma unroll
        for (int u = 0; u < 3; u++) {
            Fb[3 + u] = xadd(Fb[3 + u], Fi[u].v);
            Fb[6 + u] = xadd(Fb[6 + u], Fk[u].v);
            Fb[u] = xsub(Fb[u], xadd(Fi[u].v, Fk[u].v));
            if (REV) {
                Gb[3 + u] = xadd(Gb[3 + u], Fi[u].d[0]);
                Gb[6 + u] = xadd(Gb[6 + u], Fk[u].d[0]);
                Gb[u] = xsub(Gb[u], xadd(Fi[u].d[0], Fk[u].d[0]));
                t = xadd(t, xsub(xfma(ac[3 + u], p1d[u], xmul(ac[6 + u], p3d[u])),
                                 xmul(ac[u], xadd(p1d[u], p3d[u]))));
            }
        }
        if (REV) {
            tb[2] = xmul(disp, t);           // dF/dk_a
            tb[3] = xmul((R)bc.ka, t);       // dF/dtheta0
        }
    }
}

template <int G>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
template <int G>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

template <typename T>
__device__ __forceinline__ T pick3(int k, T a, T b, T c) {
    return k == 0 ? a : (k == 1 ? b : c);
}

__device__ __forceinline__ float r_rint(float v) { return rintf(v); }
__device__ __forceinline__ double r_rint(double v) { return rint(v); }

// Minimum-image component for the step kernels: d - L rint(d / L).  For every pair
// within the cutoff (|d| < L/2 - margin) it returns the same bits as Molly's rule
// (vec1d), one rounding of (c2 - c1) -/+ L; it differs only for pairs near L/2,
// which are far outside the cutoff.  Branch-free, unlike vec1d.
template <typename R>
__device__ __forceinline__ R vec_mi(R c1, R c2, R L, R invL) {
    const R d = xsub(c2, c1);
    return xfma(-r_rint(xmul(d, invL)), L, d);
}

// The learned pair correction's cubic segment at distance r of type QI (O-O, O-H, H-H):
// interval gi, offset sm in it, F contribution -d1 = -u'(r) = -(c1 + 2 c2 s + 3 c3 s^2) / h and
// dF/dr contribution -d2 = -(2 c2 + 6 c3 s) / h^2.
template <typename R, bool REV>
__device__ __forceinline__ void mlp_segment(const NbConsts<R> &nb, int QI, R r, int &gi, R &sm, R &d1,
                                            R &d2) {
    using V4m = typename V4T<R>::T;
    const R q = xmul(r, nb.mlp_hinv);
    gi = max(min((int)q, MLP_NG - 1), 0);   // (a double NaN, of overlapping atoms, converts to INT_MIN)
    sm = xsub(q, (R)gi);
    const V4m cf = reinterpret_cast<const V4m *>(nb.mlp_tab)[QI * MLP_NG + gi];
    d1 = xmul(xfma(sm, xfma(xmul(R(3), sm), cf.w, xmul(R(2), cf.z)), cf.y), nb.mlp_hinv);
    d2 = R(0);
    if (REV) d2 = xmul(xmul(xfma(xmul(R(6), sm), cf.w, xmul(R(2), cf.z)), nb.mlp_hinv), nb.mlp_hinv);
}

// -(dF/dc_k) (n . acoef_a) for the interval's coefficients c1, c2, c3 (one in-cutoff pair).
template <typename R>
__device__ __forceinline__ void mlp_adjoint(double *madj, int QI, int gi, R na, R sm, R hinv) {
    const double v = (double)na * (double)hinv, s1 = (double)sm;
    double *adj = madj + ((size_t)QI * MLP_NG + gi) * 4;
    atomicAdd(adj + 1, v);
    atomicAdd(adj + 2, 2.0 * s1 * v);
    atomicAdd(adj + 3, 3.0 * s1 * s1 * v);
}

// The reverse kernels' charge contraction sum_slots (2 / q_O) (-A_c) (d . a) equals, per own
// atom, (2 / q_O) a . (F - F_form): the Coulomb share of the atom's pair force, known once the
// row is done.  So the slots only accumulate the O-O form's share F_form (one slot in nine), and
// the contraction is formed after the row -- except with the learned term, whose share is on
// every slot and which needs n . a per slot anyway.
__host__ __device__ constexpr bool charge_from_forces(int form) { return form != F_LJ_MLP; }

// One (own atom KA, neighbour atom KB) slot with displacement (dx, dy, dz), evaluated
// unconditionally: pairs outside the neighbour mask or the cutoff contribute exact zeros, so
// the nine slots of an entry run as straight-line code with no divergence between the lanes of
// a warp (each lane holds a different neighbour).
//
// The slot works with A = F/r and B = (dF/dr - F/r) / r^2 of the radial force F(r): the force
// on the own atom is -A d, the force Jacobian is M = -(B d d^T + A I), so the VJP adds
// -(B (d . e) d + A e), e = w_b - w_a, and the contraction of dF/dtheta with the adjoint a is
// -(dF/dtheta / r) (d . a).  For the reaction-field Coulomb term F = qq (1/r^2 - 2 k_rf r),
// A = qq (1/r^3 - 2 k_rf) and B = -3 qq / r^5 in closed form; the O-O form and the learned
// term add their own A and B.  The accumulators receive -A and -B times the vectors ("mA",
// "mB").  A dead slot is a zero charge product and a zero weight z on the other terms (its own
// r is finite: a molecule is never its own neighbour).
//
// One entry per lane in both precisions.  FP32 took two entries per lane in packed arithmetic
// before: that halves the instructions but not the FMA pipe's time, and the second entry's
// operands held the reverse kernel at 168 registers, 12 warps an SM and 35 % issue (16 x 895
// waters at 16 lanes, event-timed: 108 us a reverse and 66 us a forward step); one entry runs at 96
// registers, 20 warps and 65 % issue (90 and 52 us).
template <typename R, int FORM, bool REV, int KA, int KB>
__device__ __forceinline__ void pair_term(bool bit, R dx, R dy, R dz, const typename V4T<R>::T &wa,
                                          const typename V4T<R>::T &wb, const R ca[3],
                                          const NbConsts<R> &nb, R f[3], R g[3], R *th,
                                          R fnc[3], double *madj) {
    constexpr int NF = FormInfo<FORM>::NP;
    constexpr int PF = FORM == F_LJ_MLP ? F_LJ : FORM;   // the O-O pair form
    constexpr int QI = (KA > 0) + (KB > 0);
    constexpr bool OO = KA == 0 && KB == 0;
    constexpr bool CHG_F = charge_from_forces(FORM);
    const R r2 = xfma(dz, dz, xfma(dy, dy, xmul(dx, dx)));
    const bool on = bit && r2 <= nb.rc2;
    const R qz = on ? nb.qq[QI] : R(0);
    R rinv = R(0), invr2, rinv3;
    if (OO || FORM == F_LJ_MLP) {
        rinv = xrsqrt(r2);
        invr2 = xmul(rinv, rinv);
        rinv3 = xmul(invr2, rinv);
    } else {
        inv_r23(r2, invr2, rinv3);
    }
    const R mAc = xmul(qz, xsub(nb.krf2, rinv3));   // -A of the Coulomb term
    R mA = mAc;
    R mB = R(0);
    if (REV) mB = xmul(xmul(qz, R(3)), xmul(rinv3, invr2));   // 3 qq / r^5 = -B
    R dca = R(0);
    if (REV && (OO || !CHG_F)) dca = xfma(dz, ca[2], xfma(dy, ca[1], xmul(dx, ca[0])));
    if (OO || FORM == F_LJ_MLP) {
        const R z = on ? R(1) : R(0);
        const R r = xmul(r2, rinv);
        R Ff = R(0), dFf = R(0), gf[4];
        bool have = false;
        if (OO && nb.fc.on) {
            have = true;
            pair_form<R, PF, REV>(nb.fc, r, rinv, invr2, Ff, dFf, gf);
        }
        int gi = 0;
        R sm = R(0);
        if constexpr (FORM == F_LJ_MLP) {
            // the learned correction: F -= u'(r), dF/dr -= u''(r)
            R d1, d2;
            mlp_segment<R, REV>(nb, QI, r, gi, sm, d1, d2);
            Ff = xsub(Ff, d1);
            if (REV) dFf = xsub(dFf, d2);
            have = true;
        }
        if (have) {
            Ff = xmul(Ff, z);
            const R Af = xmul(Ff, rinv);
            mA = xsub(mA, Af);
            if (REV) mB = xfma(xsub(Af, xmul(dFf, z)), invr2, mB);
            if (REV && CHG_F) {
                // the O-O form's share of the own-atom force, so that the Coulomb share is
                // known after the row
                fnc[0] = xfma(Af, dx, fnc[0]);
                fnc[1] = xfma(Af, dy, fnc[1]);
                fnc[2] = xfma(Af, dz, fnc[2]);
            }
        }
        if (REV) {
            const R na = xmul(xmul(rinv, dca), z);   // n . a
            if (OO && nb.fc.on) {
#pragma unroll
                for (int p = 0; p < NF; p++) th[p] = xfma(-gf[p], na, th[p]);
            }
            if constexpr (FORM == F_LJ_MLP) {
                if (on) mlp_adjoint<R>(madj, QI, gi, na, sm, nb.mlp_hinv);
            }
        }
    }
    // force on the own atom: -A d
    f[0] = xfma(mA, dx, f[0]);
    f[1] = xfma(mA, dy, f[1]);
    f[2] = xfma(mA, dz, f[2]);
    if (REV) {
        // VJP: -(B (d . e) d + A e), e = w_b - w_a
        const R ex = xsub(wb.x, wa.x), ey = xsub(wb.y, wa.y), ez = xsub(wb.z, wa.z);
        const R mt = xmul(mB, xfma(dz, ez, xfma(dy, ey, xmul(dx, ex))));
        g[0] = xfma(mt, dx, xfma(mA, ex, g[0]));
        g[1] = xfma(mt, dy, xfma(mA, ey, g[1]));
        g[2] = xfma(mt, dz, xfma(mA, ez, g[2]));
        // charge, per slot when the learned term is on: acoef . dF/dq_O = (2 / q_O) (-A_c) (d . a)
        if (!CHG_F) th[NF] = xfma(xmul(mAc, nb.twoinvq), dca, th[NF]);
    }
}

// Nearest integer of a small FP32 value by the rounding of a sum with 1.5 x 2^23 (two FMA-pipe
// instructions; rint is a slow conversion).  It differs from rint only on ties.
__device__ __forceinline__ float near_int(float a, float b) {
    return xsub(xfma(a, b, 12582912.f), 12582912.f);
}

// FP64, 1.5 x 2^52.
__device__ __forceinline__ double near_int(double a, double b) {
    return xsub(xfma(a, b, 6755399441055744.0), 6755399441055744.0);
}

// Displacement of one slot.  SHIFT: one periodic image per molecule pair, chosen from the O-O
// vector and the minimum one for every pair within the cutoff whenever L > 2 (cutoff + 2 * max
// O-H distance).  Otherwise the image is chosen per slot.  FP64: d + s rounds exactly as Molly's
// (c2 - c1) -/+ L; vec_mi per slot.  FP32: the gather coordinates are offsets from per-molecule
// cell origins (gather_f32) and s carries the origins' difference (an exact multiple of 0.5 nm)
// and, with SHIFT, the image; s stays exact, so d + s is the one rounding of a vector within the
// cutoff.
template <typename R, bool SHIFT>
__device__ __forceinline__ R slot_d(R ca_, R cb_, R s, R L, R invL) {
    const R d = xsub(cb_, ca_);
    if (SHIFT) return xadd(d, s);
    if constexpr (sizeof(R) == 4) return xadd(d, xfma(-near_int(xadd(d, s), invL), L, s));
    return vec_mi(ca_, cb_, L, invL);
}

// The image shift of the O-O vector d, added to the origins' difference o (FP64: no origins).
__device__ __forceinline__ float image_of(float d, float o, float L, float invL) {
    return xfma(-near_int(d, invL), L, o);
}
__device__ __forceinline__ double image_of(double d, double, double L, double) {
    return d > 0.5 * L ? -L : (d < -0.5 * L ? L : 0.0);
}

template <typename R, int FORM, bool REV, bool SHIFT, int KA>
__device__ __forceinline__ void pair_row(uint32_t mask, const typename V4T<R>::T &pa,
                                         const typename V4T<R>::T pb[3],
                                         const typename V4T<R>::T &wa,
                                         const typename V4T<R>::T wb[3], const R ca[3],
                                         const R sh[3], R L, R invL, const NbConsts<R> &nb,
                                         R f[3], R g[3], R *th, R fnc[3], double *madj) {
#define RS_SLOT(KB)                                                                             \
    pair_term<R, FORM, REV, KA, KB>((mask >> (3 * KA + KB)) & 1u,                               \
                                    slot_d<R, SHIFT>(pa.x, pb[KB].x, sh[0], L, invL),           \
                                    slot_d<R, SHIFT>(pa.y, pb[KB].y, sh[1], L, invL),           \
                                    slot_d<R, SHIFT>(pa.z, pb[KB].z, sh[2], L, invL), wa, wb[KB], \
                                    ca, nb, f, g, th, fnc, madj)
    RS_SLOT(0);
    RS_SLOT(1);
    RS_SLOT(2);
#undef RS_SLOT
}

// What an atom's update reads besides its force: the FP64 state and the step's noise.  Loaded
// before the force is known (atom_load), so that the loads and the noise draw are off the
// step's critical path, and every load precedes the atom's stores (the state arrays are
// distinct, but the compiler cannot know that and would otherwise serialise the components).
struct AtomState {
    double x[3], v[3], B[3], A[3], D[3], C[3], xi[3];
};

template <bool REV>
__device__ __forceinline__ void atom_load(const StepArgs &a, int I, int k, int rep, AtomState &s) {
    const size_t ia = 3 * (size_t)I + k;
#pragma unroll
    for (int u = 0; u < 3; u++) {
        s.x[u] = a.x[3 * ia + u];
        s.xi[u] = 0.0;
    }
    if (a.mode & MODE_FORCES_ONLY) return;
    const bool fuse = !REV || (a.mode & MODE_FUSE_NEXT) != 0;
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const size_t e = 3 * ia + u;
        s.v[u] = a.v[e];
        if (REV) {
            if (!(a.mode & MODE_DEFER_BA)) {
                s.B[u] = a.B[e];
                s.A[u] = a.A[e];
            }
            if (fuse) {
                s.D[u] = a.D[e];
                s.C[u] = a.C[e];
            }
        }
    }
    // noise of this step (forward) or of the next reverse step (fused part 1)
    if (fuse && a.s != 0.0) {
        const double *given = REV ? a.noise_next : a.noise_cur;
        if (given) {
#pragma unroll
            for (int u = 0; u < 3; u++) s.xi[u] = given[3 * ia + u];
        } else {
            const uint32_t la = (uint32_t)(ia - a.rep_atom0[rep]);
            atom_noise(REV ? a.seed_next[rep] : a.seed_cur[rep], la, k == 0 ? a.rep_sdO[rep] : a.rep_sdH[rep], s.xi);
        }
    }
}

// wrap1d without its division for a coordinate already inside the box (floor(c / L) is 0
// there: c / L < 1 rounds below 1), which all but a few atoms of a step are.
__device__ __forceinline__ double wrap_near(double c, double L) {
    return c >= 0.0 && c < L ? c : wrap1d(c, L);
}
__device__ __forceinline__ double wrap_exact_near(double c, double L) {
    return c >= 0.0 && c < L ? c : wrap_exact(c, L);
}

// The per-atom update of a step after the pair, bonded and reduction phases: forces F and
// VJP Gv of atom k of molecule I (FP64 sums), then forces-only output, the forward B-A-O-A
// update or the reverse un-kick with the adjoint updates and the next step's part 1.
// n2 receives |Gv|^2, xn the new FP64 position when wpos.
template <typename R, bool REV>
__device__ __forceinline__ void atom_finish(const StepArgs &a, int I, int k, double Ld, const AtomState &s,
                                            const double F[3], const double Gv[3], double &n2,
                                            double xn[3], bool &wpos) {
    using V4 = typename V4T<R>::T;
    const size_t ia = 3 * (size_t)I + k;
    const double m = k == 0 ? a.mO : a.mH;
    // The exact integrator multiplies by dt / m and 1 / m (its increments are rounded to the
    // grid, and forward and reverse use the same expression); the reference's arithmetic
    // divides as water.jl does.
    const double dtm = k == 0 ? a.dtm_O : a.dtm_H, invm = k == 0 ? a.invm_O : a.invm_H;
    if (!isfinite(F[0]) || !isfinite(F[1]) || !isfinite(F[2])) atomicOr(a.status, ST_NAN);
    if (a.mode & MODE_FORCES_ONLY) {
#pragma unroll
        for (int u = 0; u < 3; u++) {
            a.F_out[3 * ia + u] = F[u];
            if (REV) a.G[3 * ia + u] = Gv[u];
        }
    } else if (!REV) {
        // B-A-O-A (water.jl:1032-1037)
        const bool ex = a.exact != 0;
#pragma unroll
        for (int u = 0; u < 3; u++) {
            double v = s.v[u], x = s.x[u];
            const double kick = ex ? __dmul_rn(F[u], dtm) : __ddiv_rn(__dmul_rn(F[u], a.dt), m);
            v = __dadd_rn(v, ex ? qgrid(kick) : kick);
            const double h1 = __dmul_rn(__dmul_rn(v, a.dt), 0.5);
            x = __dadd_rn(x, ex ? qgrid(h1) : h1);
            v = __dadd_rn(__dmul_rn(v, a.c), __dmul_rn(s.xi[u], a.s));
            if (ex) v = qgrid(v);
            const double h2 = __dmul_rn(__dmul_rn(v, a.dt), 0.5);
            x = __dadd_rn(x, ex ? qgrid(h2) : h2);
            x = ex ? wrap_exact_near(x, Ld) : wrap_near(x, Ld);
            a.v[3 * ia + u] = v;
            a.x[3 * ia + u] = x;
            xn[u] = x;
        }
        wpos = true;
    } else {
        const double dt2 = __dmul_rn(a.dt, a.dt);
        const bool fuse = (a.mode & MODE_FUSE_NEXT) != 0;
        const bool defer = (a.mode & MODE_DEFER_BA) != 0;
        double Cm[3];
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const size_t e = 3 * ia + u;
            a.G[e] = Gv[u];
            n2 = __dadd_rn(n2, __dmul_rn(Gv[u], Gv[u]));
            // v_{n-1} = v' - F dt / m (water.jl:1516)
            const double kick = a.exact ? __dmul_rn(F[u], dtm) : __ddiv_rn(__dmul_rn(F[u], a.dt), m);
            double v = __dsub_rn(s.v[u], a.exact ? qgrid(kick) : kick);
            if (!defer) {
                // water.jl:1520-1521
                const double B = __dadd_rn(__dmul_rn(a.c, s.B[u]), __dmul_rn(dt2, Gv[u]));
                a.B[e] = B;
                a.A[e] = __dadd_rn(s.A[u], B);
            }
            if (fuse) {
                // part 1 of the next reverse step (water.jl:1496-1502)
                double x = s.x[u];
                const double h2 = __dmul_rn(__dmul_rn(v, a.dt), 0.5);
                x = __dsub_rn(x, a.exact ? qgrid(h2) : h2);
                v = __dsub_rn(v, __dmul_rn(s.xi[u], a.s));
                if (a.c != 1.0) v = __ddiv_rn(v, a.c);   // v / 1 is v: the same bits at gamma = 0
                if (a.exact) v = qgrid(v);
                const double h1 = __dmul_rn(__dmul_rn(v, a.dt), 0.5);
                x = __dsub_rn(x, a.exact ? qgrid(h1) : h1);
                x = a.exact ? wrap_exact_near(x, Ld) : wrap_near(x, Ld);
                // (dt^2 G (1 + c)) / 2, the halving as the (exact) product with 0.5
                const double D = __dadd_rn(__dmul_rn(a.c, s.D[u]),
                                           __dmul_rn(__dmul_rn(__dmul_rn(dt2, Gv[u]), __dadd_rn(1.0, a.c)), 0.5));
                const double C = __dadd_rn(s.C[u], D);
                a.D[e] = D;
                a.C[e] = C;
                a.x[e] = x;
                xn[u] = x;
                Cm[u] = a.exact ? __dmul_rn(C, invm) : __ddiv_rn(C, m);
            }
            a.v[e] = v;
        }
        if (fuse) {
            V4 wo;
            wo.x = (R)Cm[0];
            wo.y = (R)Cm[1];
            wo.z = (R)Cm[2];
            wo.w = R(0);
            ((V4 *)a.wgt_out)[ia] = wo;
            wpos = true;
        }
    }
}

// Sum N values over the G lanes of a group, each total left in one lane: at every level a lane
// gives away half of its values and adds the other half of its partner's, so N values cost
// about N + log2 G shuffles instead of N log2 G.  The pairs added at each level are those of
// group_sum's butterfly, so the totals are the same bits.  On return v[0 .. M) (M = N halved
// log2 G times, rounded up) hold the totals of values base .. min(base + M, end).
template <int G, int N, typename R>
struct GroupScatter {
    static constexpr int HALF = (N + 1) / 2;
    static constexpr int M = GroupScatter<G / 2, HALF, R>::M;
    static __device__ __forceinline__ void run(R *v, int lane, int &base, int &end) {
        const bool up = (lane & (G / 2)) != 0;
#pragma unroll
        for (int i = 0; i < HALF; i++) {
            const R hi = i + HALF < N ? v[i + HALF] : R(0);
            const R send = up ? v[i] : hi;
            v[i] = xadd(up ? hi : v[i], __shfl_xor_sync(0xffffffffu, send, G / 2));
        }
        if (up) base += HALF;
        else end = min(end, base + HALF);
        GroupScatter<G / 2, HALF, R>::run(v, lane, base, end);
    }
};
template <int N, typename R>
struct GroupScatter<1, N, R> {
    static constexpr int M = N;
    static __device__ __forceinline__ void run(R *, int, int &, int &) {}
};

// Register budget per thread: step_nreg (rs_internal.h).
template <typename R, bool REV, int U>
constexpr int step_maxnreg() {
    return step_nreg(sizeof(R) == 4, REV, U);
}

// U = 1: one neighbour entry per lane per iteration; 2: two, all loads
// issued first; 3: one, with the next one's indices and coordinates loaded while the
// current one is computed (software pipelining; launched with at most 256 pair threads).  Every
// form sums a lane's entries in the same order, so at one lane count they give the same bits.
//
// Pair warps and update warps.  The first n_pair threads of a CTA are the pair lanes (G per
// molecule): they walk the rows, reduce the molecule's sums and leave them in shared memory.
// The warps behind them own the molecules' remaining work, ten molecules a warp, one lane per
// atom: while the pair warps walk the rows they load the FP64 state, draw the noise and (first
// lane of each molecule) form the bonded terms; after the CTA's barrier they run the
// integrator.  With all of that on lanes 0-2 of every pair group, a molecule cost ~2,300 warp
// instructions outside its row at 32 lanes (5,080 in all, reverse, ncu on 16 x 895 waters),
// nearly all with 1-3 lanes active, and its latency came before and after the row's.
//
// Bound by instruction issue (65 % at 16 x 895 waters, FMA pipe 47 %) where molecules are many
// and by the latency of one row where they are few.  us per forward | reverse step at the
// default shapes (a pass's time per step, launches chained), with the former kernels and now: mixed 895
// waters 13.7 | 17.2 -> 10.0 | 11.9, 3,000 27.0 | 45.8 -> 17.3 | 23.5, 16 x 895 92 | 196 -> 53 | 86; FP64
// 895 22.7 | 38.5 -> 12.5 | 17.1, 3,000 46.5 | 95.5 -> 25.6 | 47.0, 16 x 895 166 | 337 -> 90 | 182.
template <typename R, int FORM, int G, bool REV, int U>
__global__ void __maxnreg__((step_maxnreg<R, REV, U>())) k_water_step(StepArgs a, NbConsts<R> nb,
                                                                      BondConsts bc) {
    using V4 = typename V4T<R>::T;
    constexpr int NF = FormInfo<FORM>::NP;
    constexpr int NTH = NF + 1;
    constexpr int NS = REV ? 18 + NTH : 9;   // sums per molecule: forces, VJP, dtheta
    // dynamic shared memory: [molecules][NS] sums, then [molecules][22] bonded results:
    // forces (9), VJP (9), dtheta (4)
    extern __shared__ double s_dyn[];
    R *s_sum = (R *)s_dyn, *s_bonded = s_sum + NS * (a.n_pair / G);
    chain_wait();
    if (a.chain_early) chain_next();

    const int blk = blockIdx.x;
    const int rep = a.blk_rep[blk];
    const int mol0 = a.blk_mol0[blk], nmol = a.blk_nmol[blk];
    const double Ld = a.rep_box[rep];
    const V4 *__restrict__ wgt = (const V4 *)a.wgt_in;

    if ((int)threadIdx.x >= a.n_pair) {
        // ---------------------------------------------------------------- update warps
        const int l = threadIdx.x & 31;
        const int mol = ((int)threadIdx.x - a.n_pair) / 32 * kMolsPerUpdateWarp + l / 3, k = l % 3;
        const bool live = l < 3 * kMolsPerUpdateWarp && mol < nmol;
        const int I = mol0 + (live ? mol : 0);
        R *sb = s_bonded + 22 * mol;
        AtomState st;
        constexpr int NPT = NF + 5;   // classical parameters, NPL of them per lane
        constexpr int NPL = (NPT + 2) / 3;
        double pold[NPL];
        if (live) {
            if (k == 0) {
                double xm[9];
#pragma unroll
                for (int u = 0; u < 9; u++) xm[u] = a.x[9 * (size_t)I + u];
                R w[9], ac[9];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    V4 wq;
                    wq.x = wq.y = wq.z = R(0);
                    if (REV) wq = wgt[3 * I + q];
                    w[3 * q] = wq.x;
                    w[3 * q + 1] = wq.y;
                    w[3 * q + 2] = wq.z;
                    const double sc = q == 0 ? a.acoefO : a.acoefH;
#pragma unroll
                    for (int u = 0; u < 3; u++)
                        ac[3 * q + u] = REV ? (R)__dmul_rn(a.A[9 * (size_t)I + 3 * q + u], sc) : R(0);
                }
                R Fb[9], Gb[9], tb[4];
                bonded<R, REV>(xm, Ld, bc, w, ac, Fb, Gb, tb);
#pragma unroll
                for (int u = 0; u < 9; u++) {
                    sb[u] = Fb[u];
                    if (REV) sb[9 + u] = Gb[u];
                }
                if (REV) {
#pragma unroll
                    for (int q = 0; q < 4; q++) sb[18 + q] = tb[q];
                }
            }
            atom_load<REV>(a, I, k, rep, st);
            if (REV) {
#pragma unroll
                for (int q = 0; q < NPL; q++) {
                    const int p = k + 3 * q;
                    pold[q] = p < NPT ? a.part[(size_t)I * NPT + p] : 0.0;
                }
            }
        }
        __syncthreads();   // the pair warps' sums; every read of the old state and adjoints
        if (!a.chain_early) chain_next();

        double n2 = 0.0;
        double xn[3] = {0.0, 0.0, 0.0};   // new FP64 position of the lane's atom
        bool wpos = false;
        const R *ss = s_sum + NS * mol;
        if (live) {
            double F[3], Gv[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int u = 0; u < 3; u++) {
                F[u] = __dadd_rn((double)ss[3 * k + u], (double)sb[3 * k + u]);
                if (REV) Gv[u] = __dadd_rn((double)ss[9 + 3 * k + u], (double)sb[9 + 3 * k + u]);
            }
            atom_finish<R, REV>(a, I, k, Ld, st, F, Gv, n2, xn, wpos);
        }
        // Gather buffer of the next step: H atoms are written next to their O (the molecule's
        // first lane), so that molecules are contiguous (gather_coord).
        const int src = l - k;
        const double o0 = __shfl_sync(0xffffffffu, xn[0], src);
        const double o1 = __shfl_sync(0xffffffffu, xn[1], src);
        const double o2 = __shfl_sync(0xffffffffu, xn[2], src);
        if (wpos) {
            V4 po;
            if constexpr (sizeof(R) == 4) {
                const double xo[3] = {o0, o1, o2};
                po = gather_f32(xo, xn, k, Ld);   // offsets from the molecule's cell origin
            } else {
                po.x = (R)gather_coord(o0, xn[0], k != 0, Ld);
                po.y = (R)gather_coord(o1, xn[1], k != 0, Ld);
                po.z = (R)gather_coord(o2, xn[2], k != 0, Ld);
                po.w = R(0);
            }
            ((V4 *)a.pos_out)[3 * (size_t)I + k] = po;
        }
        if (REV) {
            // This molecule's dtheta contributions and |dl_dfi|^2, into its own slots: one
            // group per molecule and step, so every slot sums its steps in step order.
            const double n2a = __shfl_sync(0xffffffffu, n2, src + 1 < 32 ? src + 1 : 31);
            const double n2b = __shfl_sync(0xffffffffu, n2, src + 2 < 32 ? src + 2 : 31);
            if (live) {
#pragma unroll
                for (int q = 0; q < NPL; q++) {
                    const int p = k + 3 * q;
                    if (p < NPT)
                        a.part[(size_t)I * NPT + p] =
                            __dadd_rn(pold[q], (double)(p < NTH ? ss[18 + p] : sb[18 + p - NTH]));
                }
                if (k == 0 && a.norm2) a.norm2[I] = __dadd_rn(__dadd_rn(n2, n2a), n2b);
            }
        }
        return;
    }

    // -------------------------------------------------------------------- pair warps
    const int grp = threadIdx.x / G;
    const int lane = threadIdx.x % G;
    const int I = mol0 + grp;
    const bool active = grp < nmol;
    const R L = (R)Ld;
    const R invL = (R)(1.0 / Ld);
    const V4 *__restrict__ pos = (const V4 *)a.pos_in;
    // this replica's accumulator of the learned term's interval-coefficient adjoints
    double *madj = FORM == F_LJ_MLP && REV
                       ? nb.mlp_adj + ((size_t)rep * MLP_NCOPY + (blk % MLP_NCOPY)) * MLP_NT * MLP_NG * 4
                       : nullptr;

    R f[3][3], g[3][3], th[NTH], fnc[3];
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int u = 0; u < 3; u++) {
            f[k][u] = R(0);
            g[k][u] = R(0);
        }
#pragma unroll
    for (int p = 0; p < NTH; p++) th[p] = R(0);
#pragma unroll
    for (int u = 0; u < 3; u++) fnc[u] = R(0);

    if (active) {
        const uint32_t *__restrict__ row = a.nbr + (size_t)I * a.cap;
        const int cnt = min(a.nbr_cnt[I], a.cap);
        // padding entries (past the row end): the row's first neighbour with an empty mask
        const uint32_t pad = cnt > 0 ? __ldg(row) & 0x7FFFFFu : 0u;
        auto ent_at = [&](int e) { return e < cnt ? __ldg(row + e) : pad; };
        // the lane's first row entries (lane + q G, q < 4 covers every loop form)
        uint32_t first[4];
#pragma unroll
        for (int q = 0; q < 4; q++) first[q] = ent_at(lane + q * G);
        V4 pa[3], wa[3];
        // the contraction weights A dt^2 / (2 m): the row needs the O's (the pair form's slot;
        // all three with the learned term), the rest are read after it
        R ca[3][3];
        auto load_ca = [&](int k) {
            const double sc = k == 0 ? a.acoefO : a.acoefH;
#pragma unroll
            for (int u = 0; u < 3; u++) ca[k][u] = (R)__dmul_rn(a.A[9 * (size_t)I + 3 * k + u], sc);
        };
#pragma unroll
        for (int k = 0; k < 3; k++) {
            pa[k] = pos[3 * I + k];
            if (REV) {
                wa[k] = wgt[3 * I + k];
                if (k == 0 || !charge_from_forces(FORM)) load_ca(k);
            }
        }
        auto fetch = [&](uint32_t ent, V4 pbq[3], V4 wbq[3]) {
            const int J = (int)(ent & 0x7FFFFFu);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                pbq[k] = pos[3 * J + k];
                if (REV) wbq[k] = wgt[3 * J + k];
            }
        };
        // One periodic image per molecule pair where the replica's box allows it (a.shift_box)
        auto walk = [&](auto shift) {
        constexpr bool SHIFT = decltype(shift)::value;
        {
            // one neighbour entry: displacement image and the nine slots
            auto entry = [&](uint32_t ent, const V4 pbq[3], const V4 wbq[3]) {
                const uint32_t mask = ent >> 23;
                R sh[3] = {R(0), R(0), R(0)};
                if constexpr (sizeof(R) == 4) {
#pragma unroll
                    for (int u = 0; u < 3; u++) sh[u] = xsub(pbq[u].w, pa[u].w);
                }
                if (SHIFT) {
                    const R dO[3] = {xsub(pbq[0].x, pa[0].x), xsub(pbq[0].y, pa[0].y), xsub(pbq[0].z, pa[0].z)};
#pragma unroll
                    for (int u = 0; u < 3; u++)
                        sh[u] = image_of(sizeof(R) == 4 ? xadd(dO[u], sh[u]) : dO[u], sh[u], L, invL);
                }
                pair_row<R, FORM, REV, SHIFT, 0>(mask, pa[0], pbq, wa[0], wbq, ca[0], sh, L, invL, nb, f[0],
                                                  g[0], th, fnc, madj);
                pair_row<R, FORM, REV, SHIFT, 1>(mask, pa[1], pbq, wa[1], wbq, ca[1], sh, L, invL, nb, f[1],
                                                  g[1], th, fnc, madj);
                pair_row<R, FORM, REV, SHIFT, 2>(mask, pa[2], pbq, wa[2], wbq, ca[2], sh, L, invL, nb, f[2],
                                                  g[2], th, fnc, madj);
            };
            if (U == 3) {
                uint32_t ent_n = first[0];
                V4 pbn[3], wbn[3];
                fetch(ent_n, pbn, wbn);
                for (int e = lane; e < cnt; e += G) {
                    const uint32_t ent = ent_n;
                    V4 pbq[3], wbq[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        pbq[k] = pbn[k];
                        if (REV) wbq[k] = wbn[k];
                    }
                    ent_n = ent_at(e + G);
                    if (e + G < cnt) fetch(ent_n, pbn, wbn);
                    entry(ent, pbq, wbq);
                }
            } else {
                // U entries per lane per iteration: all their loads are issued first, and the
                // next iteration's row entries are loaded one iteration ahead
                constexpr int UE = step_entries(sizeof(R) == 4, REV, U);
                uint32_t nxt[UE];
#pragma unroll
                for (int q = 0; q < UE; q++) nxt[q] = first[q];
                for (int e0 = lane; e0 < cnt; e0 += UE * G) {
                    uint32_t ent[UE];
#pragma unroll
                    for (int q = 0; q < UE; q++) {
                        ent[q] = nxt[q];
                        nxt[q] = ent_at(e0 + UE * G + q * G);
                    }
                    V4 pb[UE][3], wb[UE][3];
#pragma unroll
                    for (int q = 0; q < UE; q++) fetch(ent[q], pb[q], wb[q]);
#pragma unroll
                    for (int q = 0; q < UE; q++) entry(ent[q], pb[q], wb[q]);
                }
            }
        }
        };
        if (Ld > a.shift_box) walk(std::true_type{});
        else walk(std::false_type{});

    // The charge contraction from the forces (charge_from_forces), per lane on its partial
    // sums: (2 / q_O) sum_k a_k . (F_k - F_form,k), F_form only on the O atom.
    if constexpr (REV && charge_from_forces(FORM)) {
        {
            load_ca(1);
            load_ca(2);
            R q = R(0);
#pragma unroll
            for (int k = 0; k < 3; k++)
#pragma unroll
                for (int u = 0; u < 3; u++)
                    q = xfma(ca[k][u], k == 0 ? xadd(f[0][u], fnc[u]) : f[k][u], q);
            th[NF] = xfma(nb.twoinvq, q, th[NF]);
        }
    }
    }   // active

    // The group's totals, each in one lane, to shared memory.
    R v[NS];
#pragma unroll
    for (int q = 0; q < 9; q++) {
        v[q] = f[q / 3][q % 3];
        if (REV) v[9 + q] = g[q / 3][q % 3];
    }
    if (REV) {
#pragma unroll
        for (int p = 0; p < NTH; p++) v[18 + p] = th[p];
    }
    int base = 0, end = NS;
    using Sc = GroupScatter<G, NS, R>;
    Sc::run(v, lane, base, end);
    if (active) {
#pragma unroll
        for (int q = 0; q < Sc::M; q++)
            if (base + q < end) s_sum[NS * grp + base + q] = v[q];
    }
    __syncthreads();
    if (!a.chain_early) chain_next();
}

// Launch of one (precision, pair form): dispatch on lanes per molecule and entries per
// iteration; mols = molecules per CTA (a.n_pair = G mols pair threads, then the update warps).
template <typename R, int FORM, int G, int U>
cudaError_t launch_one(bool rev, int n_blk, int mols, const StepArgs &a, const NbConsts<R> &nb,
                       const BondConsts &bc, cudaStream_t st) {
    const int threads = a.n_pair + 32 * update_warps(mols);
    const size_t smem = sizeof(R) * (size_t)mols * (22 + (rev ? 19 + FormInfo<FORM>::NP : 9));
    if (rev)
        return launch_chained(k_water_step<R, FORM, G, true, U>, dim3(n_blk), dim3(threads), smem, st, a, nb, bc);
    return launch_chained(k_water_step<R, FORM, G, false, U>, dim3(n_blk), dim3(threads), smem, st, a, nb, bc);
}

template <typename R, int FORM, int G>
cudaError_t launch_u(bool rev, int unroll, int n_blk, int mols, const StepArgs &a, const NbConsts<R> &nb,
                     const BondConsts &bc, cudaStream_t st) {
    switch (unroll) {
        case 1: return launch_one<R, FORM, G, 1>(rev, n_blk, mols, a, nb, bc, st);
        case 2: return launch_one<R, FORM, G, 2>(rev, n_blk, mols, a, nb, bc, st);
        case 3:
            if (a.n_pair > 256) return cudaErrorInvalidValue;
            return launch_one<R, FORM, G, 3>(rev, n_blk, mols, a, nb, bc, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

template <typename R, int FORM>
cudaError_t launch_form(bool rev, int G, int unroll, int n_blk, int mols, const StepArgs &a,
                        const NbConsts<R> &nb, const BondConsts &bc, cudaStream_t st) {
    switch (G) {
        case 8: return launch_u<R, FORM, 8>(rev, unroll, n_blk, mols, a, nb, bc, st);
        case 16: return launch_u<R, FORM, 16>(rev, unroll, n_blk, mols, a, nb, bc, st);
        case 32: return launch_u<R, FORM, 32>(rev, unroll, n_blk, mols, a, nb, bc, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace rs
