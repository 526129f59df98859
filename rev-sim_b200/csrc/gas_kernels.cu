// gas_kernels.cu -- kernels of the gas-in-water engine (diffusion/diffusion.jl): neighbour
// rows, the fused forward and reverse step kernels, the energy and the small helpers.
//
// Work decomposition: one warp per atom walks the atom's neighbour row (every other atom within
// the list cutoff, both directions, grouped by site kind), queues the entries inside the cutoff
// and evaluates them 32 at a time (see k_gas_step); a further warp of the CTA, one lane per
// atom, forms the bonded terms meanwhile and then runs the integrator.  Each atom's sums are
// computed by one warp in a fixed order: no atomics, deterministic results.  Positions for the
// pair terms come from gather copies (pos_in, posf_in) that the step writes into the other
// buffers (pos_out, posf_out), so no warp reads a position another warp has already moved.
#include "gas_internal.h"

#include <algorithm>

#include "rs_form_energy.cuh"
#include "rs_step_impl.cuh"

namespace gs {

using namespace rs;

namespace {

__device__ __forceinline__ double kind_mass(int k, double mO, double mH) { return k == 1 ? mH : mO; }

__device__ __forceinline__ double4 ld3(const double *x, int i) {
    const size_t b = 3 * (size_t)i;
    return make_double4(x[b], x[b + 1], x[b + 2], 0.0);
}

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Radial bond own atom -> partner (displacement d, own to partner): force on the own atom
// -(F/r) d with F = -k (r - r0), and in reverse the VJP M (w_p - w_o).
template <bool REV>
__device__ __forceinline__ void o2_bond(const double d[3], double kb, double r0, const double wo[3],
                                        const double wp[3], double f[3], double g[3]) {
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])),
                                __dmul_rn(d[2], d[2]));
    const double r = __dsqrt_rn(r2);
    const double rinv = __drcp_rn(r);
    const double F = -__dmul_rn(kb, __dsub_rn(r, r0));
    const double Fr = __dmul_rn(F, rinv);
#pragma unroll
    for (int u = 0; u < 3; u++) f[u] = __fma_rn(-Fr, d[u], f[u]);
    if (REV) {
        double e[3];
#pragma unroll
        for (int u = 0; u < 3; u++) e[u] = __dsub_rn(wp[u], wo[u]);
        const double s = __dmul_rn(rinv, __fma_rn(d[2], e[2], __fma_rn(d[1], e[1], __dmul_rn(d[0], e[0]))));
        const double k1 = __dmul_rn(__dmul_rn(__dsub_rn(-kb, Fr), s), rinv);
#pragma unroll
        for (int u = 0; u < 3; u++) g[u] = __dsub_rn(g[u], __fma_rn(k1, d[u], __dmul_rn(Fr, e[u])));
    }
}

// FP32 coordinates for distance tests: those of an atom inside the box (a step's wrap leaves all
// of them there; a little slack for its rounding), NaN otherwise.  Two atoms' FP32 distance is
// then within 5.2e-7 L of the exact one -- 6e-8 L per rounded coordinate, difference and image,
// over three components -- and test_slack covers it, while a NaN decides nothing.
__device__ __forceinline__ float test_coord(double x, double L) {
    return x >= -0.001 * L && x <= 1.001 * L ? (float)x : __int_as_float(0x7FC00000);
}
// ... of an atom of molecule mol, the molecule's number in w.
__device__ __forceinline__ float4 test_pos(const double x[3], int mol, double L) {
    return make_float4(test_coord(x[0], L), test_coord(x[1], L), test_coord(x[2], L), __int_as_float(mol));
}
__device__ __forceinline__ float test_slack(double L) { return 2e-6f * (float)L; }

__device__ __forceinline__ float test_r2(const float4 &p, const float4 &q, float L, float invL) {
    const float d0 = xsub(q.x, p.x), d1 = xsub(q.y, p.y), d2 = xsub(q.z, p.z);
    const float e0 = xfma(-near_int(d0, invL), L, d0), e1 = xfma(-near_int(d1, invL), L, d1),
                e2 = xfma(-near_int(d2, invL), L, d2);
    return xfma(e2, e2, xfma(e1, e1, xmul(e0, e0)));
}

// ------------------------------------------------------------------ gather order
// The gather buffers and the rows number the atoms by site kind: the water O, then the water H (a
// molecule's two adjacent), then the gas.  Consecutive entries of a row, which are of one kind and
// ascending, then lie close together: a quarter of a 3 nm box is within the list cutoff, so 32
// entries touch 15 lines of FP32 test positions where they touched 32 in atom order.
__device__ __forceinline__ int gather_index(int i, int nw3) {
    const int m = i / 3, k = i - 3 * m;
    return i >= nw3 ? i : (k == 0 ? m : nw3 / 3 + 2 * m + k - 1);
}
__device__ __forceinline__ int gather_atom(int c, int nw3) {   // its inverse
    const int nw = nw3 / 3, q = c - nw;
    return c >= nw3 ? c : (c < nw ? 3 * c : 3 * (q >> 1) + 1 + (q & 1));
}
__device__ __forceinline__ int gather_kind(int c, int nw, int nw3) { return c < nw ? 0 : (c < nw3 ? 1 : 2); }
__device__ __forceinline__ int atom_mol(int i, int nw3) {
    return i < nw3 ? i / 3 : nw3 / 3 + (i - nw3) / 2;
}

// ------------------------------------------------------------------ neighbour rows
// Row of atom i: the gather index of every atom of another molecule with min-image d^2 <= rc_nl^2
// (Molly's per-dimension rule), except water H - gas pairs, which carry no term (no charge on the
// gas, no pair form on H), in ascending order (ballot compaction).
//
// One warp per atom; the FP32 distance decides all but the pairs within test_slack of the cutoff,
// which take the exact FP64 test.  Bound by the tests' issue.  2,675 atoms: 17 us a build; 51
// us with the FP64 test and strided FP64 loads on every candidate.
constexpr int kRowU = 4;
__global__ void __launch_bounds__(kThreads) k_gas_rows(GasRowArgs a) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
    if (i >= a.N) return;
    const int nw = a.nw3 / 3;
    const float L = (float)a.L, invL = (float)(1.0 / a.L);
    const float rcf = (float)sqrt(a.rc_nl2), slack = test_slack(a.L);
    const float hi = (rcf + slack) * (rcf + slack) * 1.000001f;
    const float lo = slack < rcf ? (rcf - slack) * (rcf - slack) * 0.999999f : 0.f;
    const float4 paf = a.posf[gather_index(i, a.nw3)];
    const int ka = site_kind(i, a.nw3), mi = atom_mol(i, a.nw3);
    int n = 0;
    int *row = a.rows + (size_t)i * a.cap;
    // the candidates an atom takes: an H no gas, a gas atom no H
    for (int part = 0; part < (ka == 2 ? 2 : 1); part++) {
        const int c0 = part == 0 ? 0 : a.nw3, c1 = ka == 2 && part == 0 ? nw : (ka == 1 ? a.nw3 : a.N);
        for (int base = c0; base < c1; base += 32 * kRowU) {
            float4 q[kRowU];
            bool ok[kRowU];
#pragma unroll
            for (int u = 0; u < kRowU; u++) q[u] = a.posf[min(base + 32 * u + lane, a.N - 1)];
#pragma unroll
            for (int u = 0; u < kRowU; u++) {
                const int c = base + 32 * u + lane;
                const float r2f = test_r2(paf, q[u], L, invL);
                ok[u] = c < c1 && !(r2f > hi) && __float_as_int(q[u].w) != mi;
                if (ok[u] && !(r2f <= lo)) {
                    const double4 pa = ld3(a.x, i), pb = ld3(a.x, gather_atom(c, a.nw3));
                    const double d0 = vec1d(pa.x, pb.x, a.L), d1 = vec1d(pa.y, pb.y, a.L),
                                 d2 = vec1d(pa.z, pb.z, a.L);
                    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)),
                                                __dmul_rn(d2, d2));
                    ok[u] = r2 <= a.rc_nl2;
                }
            }
#pragma unroll
            for (int u = 0; u < kRowU; u++) {
                const unsigned m = __ballot_sync(0xffffffffu, ok[u]);
                if (ok[u]) {
                    const int k = n + __popc(m & ((1u << lane) - 1u));
                    if (k < a.cap) row[k] = base + 32 * u + lane;
                }
                n += __popc(m);
            }
        }
    }
    if (lane == 0) {
        a.cnt[i] = min(n, a.cap);
        if (n > a.cap) atomicOr(a.status, ST_NLIST_OVERFLOW);
    }
}

// ------------------------------------------------------------------ step kernels
// Register budget per thread.  An SM's scheduler holds 512 / budget warps: FP64 LJ at 96 five of
// them, 20 an SM, so that the 2,675 atoms of the diffusion box run in one wave (19 pair warps and
// an update warp a CTA, 141 CTAs); the other forms' reverse kernels (dual numbers, more live
// values) want 128.
__host__ __device__ constexpr int gas_nreg(bool fp32, bool lj, bool rev) {
    return fp32 ? (rev ? 80 : 64) : (lj || !rev ? 96 : 128);
}

// Sums per atom: force, and in reverse VJP, charge and the two pair classes an atom meets.
template <int FORM, bool REV>
__host__ __device__ constexpr int gas_sums() { return REV ? 7 + 2 * FormInfo<FORM>::NP : 3; }

// Atoms per CTA (pair warps; one update warp more).  While one wave holds all atoms the busiest SM
// sets the time: the count with the fewest atoms on it, of those the largest (fewer update
// warps).  Otherwise half an SM's warps a CTA.
int gas_cta_atoms(int nreg, int N) {
    const int cap = std::min(64, 4 * (512 / nreg));   // warps an SM holds
    int best = 0, load = 0;
    for (int m = 1; m <= 31; m++) {
        const int ctas = ((N + m - 1) / m + kSMs - 1) / kSMs;
        if (ctas * (m + 1) > cap || (best && ctas * m > load)) continue;
        best = m;
        load = ctas * m;
    }
    return best ? best : cap / 2 - 1;
}

constexpr int kGasU = 4, kQueue = 32 * kGasU + 32;   // row entries a lane tests at a time; a warp's queue

// Gather buffers hold a vector's components apart, [3][N]: a warp's gather of 32 neighbours takes
// three loads of a few lines each, where 32-byte entries take a line each for either half.
template <typename T>
__device__ __forceinline__ void gather3(const T *buf, int N, int c, T v[3]) {
#pragma unroll
    for (int u = 0; u < 3; u++) v[u] = buf[(size_t)u * N + c];
}
template <typename T>
__device__ __forceinline__ void scatter3(T *buf, int N, int c, const double v[3]) {
#pragma unroll
    for (int u = 0; u < 3; u++) buf[(size_t)u * N + c] = (T)v[u];
}
// The position of atom i into the gather buffers.
template <typename R>
__device__ __forceinline__ void store_pos(int N, int nw3, double L, int i, const double x[3], void *pos, double *pos64,
                                          float4 *posf) {
    const int c = gather_index(i, nw3);
    scatter3(static_cast<R *>(pos), N, c, x);
    if (sizeof(R) == 4) scatter3(pos64, N, c, x);   // FP64: the same buffer
    posf[c] = test_pos(x, atom_mol(i, nw3), L);
}

// R: pair arithmetic (float in mixed precision, double in FP64).  The pair loop gathers R
// positions and weights, [3][N] components; the per-lane sums are R and are combined in FP64; the
// bonded terms and the integrator run in FP64 on the FP64 gather copy pos64.
//
// The first a.apc warps are the pair warps.  Each walks its atom's row in two phases.  Phase 1:
// each lane loads kGasU row entries (all loads issued before any is used, so that kGasU neighbour
// gathers per lane are in flight; the next entries' indices are loaded ahead of phase 2), tests
// their FP32 distances and pushes the ones that may be inside the cutoff (about 58 % at the list
// cutoff 1.2 nm) onto a per-warp queue in shared memory.  Phase 2: while 32 or more are queued, all
// lanes evaluate one each, with the exact test on the pair's own displacement, so the pair
// arithmetic runs with full warps.  The queue is processed last-in first-out in a fixed order
// (deterministic sums).  The warp behind them owns the atoms' remaining work, one lane per atom:
// while the rows are walked it forms the bonded terms, loads the FP64 state and draws the noise;
// after the CTA's barrier it runs the integrator.
//
// Bound by the latency of a row's gathers and FP64 chains at five warps a scheduler (ncu, forward:
// 2,670 warp instructions an atom, FP64 pipe 15 %, L1 34 %; loads and fixed latencies are the
// stalls).  Evaluating two or three queued entries a lane at a time, or testing six or eight entries
// a lane, changed nothing (13.1-13.8 | 19.7-21.7 us).  2,675 atoms, FP64, LJ: 13.7 us a forward and
// 19.4 us a reverse step; 19.3 and 32.8 us with the FP64 test on every entry, the displacements in the
// queue, and the bonded terms and integrator on lane 0 of every pair warp.
template <typename R, int FORM, bool REV>
__global__ void __maxnreg__((gas_nreg(sizeof(R) == 4, FORM == F_LJ, REV)))
    k_gas_step(const GasConstsT<R> k, const GasArgs a) {
    constexpr int NP = FormInfo<FORM>::NP, NS = gas_sums<FORM, REV>();
    // [apc][NS] sums, then [apc][kQueue] queues
    extern __shared__ double s_dyn[];
    chain_wait();
    if (a.chain_early) chain_next();
    const R *pos_in = static_cast<const R *>(a.pos_in), *wgt_in = static_cast<const R *>(a.wgt_in);
    const int nw = a.nw3 / 3;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i0 = blockIdx.x * a.apc, n_at = min(a.apc, a.N - i0);

    if (w == a.apc) {
        // ---------------------------------------------------------------- update warp
        const bool live = lane < n_at;
        const int i = i0 + (live ? lane : 0);
        const int ka = site_kind(i, a.nw3);
        const double ma = kind_mass(ka, a.mO, a.mH);
        const size_t b = 3 * (size_t)i;
        const bool upd = !(a.mode & MODE_FORCES_ONLY), fuse = (a.mode & MODE_FUSE_NEXT) != 0;
        double fb[3] = {0.0, 0.0, 0.0}, gb[3] = {0.0, 0.0, 0.0};
        double xk[3] = {0.0, 0.0, 0.0}, vk[3] = {0.0, 0.0, 0.0}, xi[3] = {0.0, 0.0, 0.0};
        double Bk[3] = {0.0, 0.0, 0.0}, Ak[3] = {0.0, 0.0, 0.0}, Dk[3] = {0.0, 0.0, 0.0}, Ck[3] = {0.0, 0.0, 0.0};
        if (live) {
            // bonded terms of the atom's molecule (diffusion.jl:997-1050, 1367-1498)
            if (ka != 2) {
                const int kk = i % 3, m0 = i - kk;
                double xm[9], w9[9], ac9[9], Fb[9], Gb[9], tb[4];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const int c = gather_index(m0 + q, a.nw3);
                    gather3(a.pos64_in, a.N, c, xm + 3 * q);
                    R wq[3] = {R(0), R(0), R(0)};
                    if (REV) gather3(wgt_in, a.N, c, wq);
#pragma unroll
                    for (int u = 0; u < 3; u++) w9[3 * q + u] = wq[u];
                    ac9[3 * q] = ac9[3 * q + 1] = ac9[3 * q + 2] = 0.0;
                }
                bonded<double, REV>(xm, a.L, a.bw, w9, ac9, Fb, Gb, tb);
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    fb[u] = pick3(kk, Fb[u], Fb[3 + u], Fb[6 + u]);
                    if (REV) gb[u] = pick3(kk, Gb[u], Gb[3 + u], Gb[6 + u]);
                }
            } else {
                const int p = ((i - a.nw3) ^ 1) + a.nw3;
                double po[3], pp[3], d[3], wo[3] = {0.0, 0.0, 0.0}, wp[3] = {0.0, 0.0, 0.0};
                gather3(a.pos64_in, a.N, i, po);
                gather3(a.pos64_in, a.N, p, pp);
                R w0[3], w1[3];
                if (REV) {
                    gather3(wgt_in, a.N, i, w0);
                    gather3(wgt_in, a.N, p, w1);
                }
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    d[u] = vec1d(po[u], pp[u], a.L);
                    if (REV) {
                        wo[u] = w0[u];
                        wp[u] = w1[u];
                    }
                }
                o2_bond<REV>(d, a.kb_g, a.r0_g, wo, wp, fb, gb);
            }
            if (upd) {
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    vk[u] = a.v[b + u];
                    if (!REV || fuse) xk[u] = a.x[b + u];
                    if (REV) {
                        Bk[u] = a.B[b + u];
                        Ak[u] = a.A[b + u];
                        if (fuse) {
                            Dk[u] = a.D[b + u];
                            Ck[u] = a.C[b + u];
                        }
                    }
                }
                // noise of this step (forward) or of the next reverse step (fused part 1)
                if ((!REV || fuse) && a.s != 0.0)
                    atom_noise(REV ? a.seed_next : a.seed_cur, (uint32_t)i, ka == 1 ? a.sdH : a.sdO, xi);
            }
        }
        __syncthreads();   // the pair warps' sums; every read of the atoms' A
        if (!a.chain_early) chain_next();
        if (!live) return;
        const double *ss = s_dyn + NS * lane;
        double f[3], g[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int u = 0; u < 3; u++) {
            f[u] = __dadd_rn(ss[u], fb[u]);
            if (REV) g[u] = __dadd_rn(ss[3 + u], gb[u]);
        }
        if (!isfinite(f[0]) || !isfinite(f[1]) || !isfinite(f[2])) atomicOr(a.status, ST_NAN);

        if (REV) {
            // dtheta of the atom: each parameter's contributions in (q, class) order, then the
            // charge term, with compile-time parameter indices so that the sums stay in
            // registers; the partials' loads all issued before their stores
            double *pt = a.part + (size_t)i * k.P;
            double old[kMaxP];
#pragma unroll
            for (int p = 0; p < kMaxP; p++) old[p] = p < k.P ? pt[p] : 0.0;
#pragma unroll
            for (int p = 0; p < kMaxP; p++) {
                double t = 0.0;
#pragma unroll
                for (int q = 0; q < NP; q++)
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        // class c = (own gas) + (neighbour gas): sums 7 .. of a water, 7 + NP .. of
                        // a gas neighbour
                        const int other = c - (ka == 2);
                        const double acc = other == 0 ? ss[7 + q] : (other == 1 ? ss[7 + NP + q] : 0.0);
                        if (k.iw[q] == p) t = __fma_rn(k.fw[c][q], acc, t);
                        if (k.ig[q] == p) t = __fma_rn(k.fg[c][q], acc, t);
                    }
                if (k.iq == p) t = __dadd_rn(t, ss[6]);
                if (p < k.P) pt[p] = __dadd_rn(old[p], t);
            }
        }
        if (!upd) {
#pragma unroll
            for (int u = 0; u < 3; u++) {
                a.F_out[b + u] = f[u];
                if (REV) a.G[b + u] = g[u];
            }
            return;
        }
        double xn[3];
        if (!REV) {
            // B-A-O-A (diffusion.jl:1228-1233)
#pragma unroll
            for (int u = 0; u < 3; u++) {
                double v = vk[u], x = xk[u];
                v = __dadd_rn(v, __ddiv_rn(__dmul_rn(f[u], a.dt), ma));
                x = __dadd_rn(x, __dmul_rn(__dmul_rn(v, a.dt), 0.5));
                v = __dadd_rn(__dmul_rn(v, a.c), __dmul_rn(xi[u], a.s));
                x = __dadd_rn(x, __dmul_rn(__dmul_rn(v, a.dt), 0.5));
                x = wrap_near(x, a.L);
                a.v[b + u] = v;
                a.x[b + u] = x;
                xn[u] = x;
            }
            store_pos<R>(a.N, a.nw3, a.L, i, xn, a.pos_out, a.pos64_out, a.posf_out);
            return;
        }
        // reverse part 2 (diffusion.jl:1580-1586) and, fused, part 1 of the next step (1566-1572)
        const double dt2 = __dmul_rn(a.dt, a.dt);
        double Cm[3];
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const size_t e = b + u;
            a.G[e] = g[u];
            double v = __dsub_rn(vk[u], __ddiv_rn(__dmul_rn(f[u], a.dt), ma));
            const double B = __dadd_rn(__dmul_rn(a.c, Bk[u]), __dmul_rn(dt2, g[u]));
            a.B[e] = B;
            a.A[e] = __dadd_rn(Ak[u], B);
            if (fuse) {
                double x = xk[u];
                x = __dsub_rn(x, __dmul_rn(__dmul_rn(v, a.dt), 0.5));
                v = __ddiv_rn(__dsub_rn(v, __dmul_rn(xi[u], a.s)), a.c);
                x = __dsub_rn(x, __dmul_rn(__dmul_rn(v, a.dt), 0.5));
                x = wrap_near(x, a.L);
                const double D = __dadd_rn(__dmul_rn(a.c, Dk[u]),
                                           __ddiv_rn(__dmul_rn(__dmul_rn(dt2, g[u]), __dadd_rn(1.0, a.c)), 2.0));
                const double C = __dadd_rn(Ck[u], D);
                a.D[e] = D;
                a.C[e] = C;
                a.x[e] = x;
                xn[u] = x;
                Cm[u] = __ddiv_rn(C, ma);
            }
            a.v[e] = v;
        }
        if (fuse) {
            store_pos<R>(a.N, a.nw3, a.L, i, xn, a.pos_out, a.pos64_out, a.posf_out);
            scatter3(static_cast<R *>(a.wgt_out), a.N, gather_index(i, a.nw3), Cm);
        }
        return;
    }

    // -------------------------------------------------------------------- pair warps
    if (w < n_at) {
        const int i = i0 + w;
        const R L = (R)a.L, invL = (R)a.invL;
        const float Lf = (float)a.L, invLf = (float)a.invL;
        const int ka = site_kind(i, a.nw3);
        const int ci = gather_index(i, a.nw3);
        const float4 paf = a.posf_in[ci];
        R pa[3], wa[3] = {R(0), R(0), R(0)}, ca[3] = {R(0), R(0), R(0)};
        gather3(pos_in, a.N, ci, pa);
        if (REV) {
            gather3(wgt_in, a.N, ci, wa);
#pragma unroll
            for (int u = 0; u < 3; u++)
                ca[u] = (R)(a.acoef_in ? a.acoef_in[3 * (size_t)i + u]
                                       : __dmul_rn(a.A[3 * (size_t)i + u], ka == 1 ? a.cfH : a.cfO));
        }
        R fr[3] = {R(0), R(0), R(0)}, gr[3] = {R(0), R(0), R(0)}, thq = R(0);
        R acc[2][NP];   // of water and of gas neighbours
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
            for (int q = 0; q < NP; q++) acc[c][q] = R(0);
        // Pair terms of the queued neighbour j (gather index).
        auto pair = [&](const int j) {
            R pb[3], wb[3];
            gather3(pos_in, a.N, j, pb);
            if (REV) gather3(wgt_in, a.N, j, wb);
            const int kb = gather_kind(j, nw, a.nw3);
            R d[3];
#pragma unroll
            for (int u = 0; u < 3; u++) {
                const R c = xsub(pb[u], pa[u]);
                d[u] = xfma(-near_int(c, invL), L, c);
            }
            const R dx = d[0], dy = d[1], dz = d[2];
            const R r2 = xfma(dz, dz, xfma(dy, dy, xmul(dx, dx)));
            if (!(r2 <= k.rc2)) return;
            const R rinv = xrsqrt(r2);
            const R r = xmul(r2, rinv);
            const R invr2 = xmul(rinv, rinv);
            R F = R(0), dF = R(0), Fc = R(0);
            const bool coul = ka != 2 && kb != 2;
            if (coul) {
                const int qi = (ka == 1) + (kb == 1);
                const R qq = qi == 0 ? k.qq[0] : qi == 1 ? k.qq[1] : k.qq[2];
                Fc = xmul(qq, xsub(invr2, xmul(k.krf2, r)));
                F = Fc;
                if (REV) dF = -xmul(xadd(qq, qq), xadd(xmul(invr2, rinv), k.krf));
            }
            R gf[4] = {R(0), R(0), R(0), R(0)};
            bool form = false;
            if (ka != 1 && kb != 1) {
                const int cls = (ka == 2) + (kb == 2);
                form = cls == 0 ? k.on[0] : cls == 1 ? k.on[1] : k.on[2];
                if (form) {
                    // constant class indices keep the constants in the parameter bank
                    R Ff = R(0), dFf = R(0);
                    if (cls == 0)
                        pair_form<R, FORM, REV>(k.fc[0], r, rinv, invr2, Ff, dFf, gf);
                    else if (cls == 1)
                        pair_form<R, FORM, REV>(k.fc[1], r, rinv, invr2, Ff, dFf, gf);
                    else
                        pair_form<R, FORM, REV>(k.fc[2], r, rinv, invr2, Ff, dFf, gf);
                    F = xadd(F, Ff);
                    if (REV) dF = xadd(dF, dFf);
                }
            }
            const R Fr = xmul(F, rinv);
            fr[0] = xfma(-Fr, dx, fr[0]);
            fr[1] = xfma(-Fr, dy, fr[1]);
            fr[2] = xfma(-Fr, dz, fr[2]);
            if (REV) {
                const R ex = xsub(wb[0], wa[0]), ey = xsub(wb[1], wa[1]), ez = xsub(wb[2], wa[2]);
                const R s = xmul(rinv, xfma(dz, ez, xfma(dy, ey, xmul(dx, ex))));
                const R k1 = xmul(xmul(xsub(dF, Fr), s), rinv);
                gr[0] = xsub(gr[0], xfma(k1, dx, xmul(Fr, ex)));
                gr[1] = xsub(gr[1], xfma(k1, dy, xmul(Fr, ey)));
                gr[2] = xsub(gr[2], xfma(k1, dz, xmul(Fr, ez)));
                const R na = xmul(rinv, xfma(dz, ca[2], xfma(dy, ca[1], xmul(dx, ca[0]))));
                if (coul) thq = xfma(-xmul(Fc, k.twoinvq), na, thq);
                if (form) {
#pragma unroll
                    for (int c = 0; c < 2; c++)
                        if (c == (kb == 2))
#pragma unroll
                            for (int q = 0; q < NP; q++) acc[c][q] = xfma(-gf[q], na, acc[c][q]);
                }
            }
        };
        int *queue = (int *)(s_dyn + NS * a.apc) + kQueue * w;
        const int n = a.cnt[i];
        const int *row = a.rows + (size_t)i * a.cap;
        const unsigned lt = (1u << lane) - 1u;
        int qn = 0, next[kGasU];
#pragma unroll
        for (int u = 0; u < kGasU; u++) next[u] = 32 * u + lane < n ? __ldg(row + 32 * u + lane) : -1;
        for (int base = 0; base < n; base += 32 * kGasU) {
            int jj[kGasU];
            float4 pb[kGasU];
#pragma unroll
            for (int u = 0; u < kGasU; u++) {
                jj[u] = next[u];
                pb[u] = a.posf_in[max(jj[u], 0)];
            }
#pragma unroll
            for (int u = 0; u < kGasU; u++) {
                const int e = base + 32 * (kGasU + u) + lane;
                next[u] = e < n ? __ldg(row + e) : -1;
            }
#pragma unroll
            for (int u = 0; u < kGasU; u++) {
                const bool ok = jj[u] >= 0 && !(test_r2(paf, pb[u], Lf, invLf) > a.rc2_test);
                const unsigned m = __ballot_sync(0xffffffffu, ok);
                if (ok) queue[qn + __popc(m & lt)] = jj[u];
                qn += __popc(m);
            }
            __syncwarp();
            while (qn >= 32) {
                pair(queue[qn - 32 + lane]);
                qn -= 32;
            }
            __syncwarp();
        }
        if (lane < qn) pair(queue[lane]);
        __syncwarp();
        // the sums over the lanes, in FP64
        double v[NS];
#pragma unroll
        for (int u = 0; u < 3; u++) {
            v[u] = (double)fr[u];
            if (REV) v[3 + u] = (double)gr[u];
        }
        if (REV) {
            v[6] = (double)thq;
#pragma unroll
            for (int c = 0; c < 2; c++)
#pragma unroll
                for (int q = 0; q < NP; q++) v[7 + c * NP + q] = (double)acc[c][q];
        }
        int at = 0, end = NS;
        GroupScatter<32, NS, double>::run(v, lane, at, end);
#pragma unroll
        for (int q = 0; q < GroupScatter<32, NS, double>::M; q++)
            if (at + q < end) s_dyn[NS * w + at + q] = v[q];
    }
    __syncthreads();
}

template <typename R>
__global__ void k_gas_part1(const GasArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.N) return;
    const int ka = site_kind(i, a.nw3);
    const double ma = kind_mass(ka, a.mO, a.mH);
    const double dt2 = __dmul_rn(a.dt, a.dt);
    double xi[3] = {0.0, 0.0, 0.0};
    if (a.s != 0.0) atom_noise(a.seed_next, (uint32_t)i, ka == 1 ? a.sdH : a.sdO, xi);
    double xn[3], Cm[3];
    const size_t b = 3 * (size_t)i;
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const size_t e = b + u;
        double v = a.v[e], x = a.x[e];
        x = __dsub_rn(x, __dmul_rn(__dmul_rn(v, a.dt), 0.5));
        v = __ddiv_rn(__dsub_rn(v, __dmul_rn(xi[u], a.s)), a.c);
        x = __dsub_rn(x, __dmul_rn(__dmul_rn(v, a.dt), 0.5));
        x = wrap1d(x, a.L);
        const double D = __dadd_rn(__dmul_rn(a.c, a.D[e]),
                                   __ddiv_rn(__dmul_rn(__dmul_rn(dt2, a.G[e]), __dadd_rn(1.0, a.c)), 2.0));
        const double C = __dadd_rn(a.C[e], D);
        a.D[e] = D;
        a.C[e] = C;
        a.x[e] = x;
        a.v[e] = v;
        xn[u] = x;
        Cm[u] = __ddiv_rn(C, ma);
    }
    store_pos<R>(a.N, a.nw3, a.L, i, xn, a.pos_out, a.pos64_out, a.posf_out);
    scatter3(static_cast<R *>(a.wgt_out), a.N, gather_index(i, a.nw3), Cm);
}

template <typename R>
__global__ void k_gas_pack(int N, int nw3, double L, const double *x, void *pos, double *pos64, float4 *posf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const double4 p = ld3(x, i);
    const double xi[3] = {p.x, p.y, p.z};
    store_pos<R>(N, nw3, L, i, xi, pos, pos64, posf);
}

template <typename R>
__global__ void k_gas_pack_w(int N, int nw3, const double *w, double mO, double mH, R *wgt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const double m = site_kind(i, nw3) == 1 ? mH : mO;
    const size_t b = 3 * (size_t)i;
    const double v[3] = {__ddiv_rn(w[b], m), __ddiv_rn(w[b + 1], m), __ddiv_rn(w[b + 2], m)};
    scatter3(wgt, N, gather_index(i, nw3), v);
}

__global__ void k_gas_reset(int n3, const double *g, double f1, double f2, double f3, double *A,
                            double *B, double *C, double *D, double *G) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n3) return;
    const double ge = g[e];
    const double a = __dmul_rn(ge, f1);
    A[e] = a;
    B[e] = a;
    C[e] = 0.0;
    D[e] = __ddiv_rn(__dmul_rn(ge, f2), f3);
    G[e] = 0.0;
}

__global__ void k_gas_axpy(int n, double k, const double *x, double *y) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) y[e] = __fma_rn(k, x[e], y[e]);
}

// ------------------------------------------------------------------ energy
template <int FORM>
__global__ void __launch_bounds__(kThreads) k_gas_energy(const GasConsts k, const GasArgs a,
                                                         double *epart) {
    constexpr int NP = FormInfo<FORM>::NP;
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
    if (i >= a.N) return;
    const int ka = site_kind(i, a.nw3);
    const double4 pa = ld3(a.x, i);
    double E = 0.0, eq = 0.0;
    double acc[3][NP];
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int q = 0; q < NP; q++) acc[c][q] = 0.0;
    const int n = a.cnt[i];
    const int *row = a.rows + (size_t)i * a.cap;
    for (int e = lane; e < n; e += 32) {
        const int j = gather_atom(row[e], a.nw3);
        if (j <= i) continue;
        const double4 pb = ld3(a.x, j);
        const double d0 = vec1d(pa.x, pb.x, a.L), d1 = vec1d(pa.y, pb.y, a.L), d2 = vec1d(pa.z, pb.z, a.L);
        const double r2 = d0 * d0 + d1 * d1 + d2 * d2;
        if (!(r2 <= k.rc2)) continue;
        const double r = sqrt(r2);
        const int kb = site_kind(j, a.nw3);
        if (ka != 2 && kb != 2) {
            // Molly CoulombReactionField energy; dE/dq_O = 2 E_c / q_O
            const double Ec = k.qq[(ka == 1) + (kb == 1)] * (1.0 / r + k.krf * r2 - k.crf_shift);
            E += Ec;
            eq += Ec * k.twoinvq;
        }
        if (ka != 1 && kb != 1) {
            const int cls = (ka == 2) + (kb == 2);
            if (k.on[cls]) {
                const DualN<double, 4> Ef = form_energy<FORM>(cls == 0 ? k.fc[0].p : cls == 1 ? k.fc[1].p : k.fc[2].p, r);
                E += Ef.v;
#pragma unroll
                for (int c = 0; c < 3; c++)
                    if (c == cls)
#pragma unroll
                        for (int q = 0; q < NP; q++) acc[c][q] += Ef.d[q];
            }
        }
    }
    E = wsum(E);
    eq = wsum(eq);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int q = 0; q < NP; q++) acc[c][q] = wsum(acc[c][q]);
    if (lane != 0) return;
    // bonded terms on the molecule's first atom
    if (ka == 0) {
        double x[9];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const double4 p = ld3(a.x, i + q);
            x[3 * q] = p.x;
            x[3 * q + 1] = p.y;
            x[3 * q + 2] = p.z;
        }
        double dd[2][3];
        for (int h = 1; h <= 2; h++) {
            for (int u = 0; u < 3; u++) dd[h - 1][u] = vec1d(x[u], x[3 * h + u], a.L);
            const double bl = sqrt(dd[h - 1][0] * dd[h - 1][0] + dd[h - 1][1] * dd[h - 1][1] +
                                   dd[h - 1][2] * dd[h - 1][2]) - a.bw.r0;
            E += 0.5 * a.bw.kb * bl * bl;
        }
        const double *u1 = dd[0], *u2 = dd[1];
        const double cth = (u1[0] * u2[0] + u1[1] * u2[1] + u1[2] * u2[2]) /
                           (sqrt(u1[0] * u1[0] + u1[1] * u1[1] + u1[2] * u1[2]) *
                            sqrt(u2[0] * u2[0] + u2[1] * u2[1] + u2[2] * u2[2]));
        const double th = acos(cth) - a.bw.th0;
        E += 0.5 * a.bw.ka * th * th;
    } else if (ka == 2 && ((i - a.nw3) & 1) == 0) {
        const double4 pp = ld3(a.x, i + 1);
        const double d0 = vec1d(pa.x, pp.x, a.L), d1 = vec1d(pa.y, pp.y, a.L), d2 = vec1d(pa.z, pp.z, a.L);
        const double bl = sqrt(d0 * d0 + d1 * d1 + d2 * d2) - a.r0_g;
        E += 0.5 * a.kb_g * bl * bl;
    }
    double th[kMaxP];
#pragma unroll
    for (int p = 0; p < kMaxP; p++) th[p] = 0.0;
#pragma unroll
    for (int q = 0; q < NP; q++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
            th[k.iw[q]] += k.fw[c][q] * acc[c][q];
            if (k.ig[q] >= 0) th[k.ig[q]] += k.fg[c][q] * acc[c][q];
        }
    th[k.iq] += eq;
    double *out = epart + (size_t)i * (k.P + 1);
    out[0] = E;
    for (int p = 0; p < k.P; p++) out[1 + p] = th[p];
}

// Single CTA: out[q] = scale * sum over atoms (strided per thread, then a fixed tree).
__global__ void __launch_bounds__(256) k_gas_esum(int N, int P, const double *epart, double e_scale,
                                                  double g_scale, int accumulate, double *out) {
    __shared__ double sh[256];
    for (int q = 0; q <= P; q++) {
        double s = 0.0;
        for (int a = threadIdx.x; a < N; a += 256) s += epart[(size_t)a * (P + 1) + q];
        sh[threadIdx.x] = s;
        __syncthreads();
        for (int w = 128; w > 0; w >>= 1) {
            if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            const double v = sh[0] * (q == 0 ? e_scale : g_scale);
            out[q] = accumulate ? out[q] + v : v;
        }
        __syncthreads();
    }
}

template <typename R, bool REV, int FORM>
void step_launch(const GasConstsT<R> &k, GasArgs a, cudaStream_t st) {
    constexpr int NS = gas_sums<FORM, REV>(), nreg = gas_nreg(sizeof(R) == 4, FORM == F_LJ, REV);
    a.cfO = a.dt * a.dt / (2.0 * a.mO);
    a.cfH = a.dt * a.dt / (2.0 * a.mH);
    a.apc = gas_cta_atoms(nreg, a.N);
    const int grid = (a.N + a.apc - 1) / a.apc;
    a.chain_early = grid <= kSMs;
    launch_chained(k_gas_step<R, FORM, REV>, dim3(grid), dim3(32 * (a.apc + 1)),
                   (size_t)a.apc * (NS * sizeof(double) + kQueue * sizeof(int)), st, k, a);
}
template <typename R, bool REV>
void step_form(int form, const GasConstsT<R> &k, const GasArgs &a, cudaStream_t st) {
    switch (form) {
        case F_LJ: step_launch<R, REV, F_LJ>(k, a, st); break;
        case F_DEXP: step_launch<R, REV, F_DEXP>(k, a, st); break;
        case F_BUCK: step_launch<R, REV, F_BUCK>(k, a, st); break;
        case F_LJSC: step_launch<R, REV, F_LJSC>(k, a, st); break;
        case F_BUFF: step_launch<R, REV, F_BUFF>(k, a, st); break;
    }
}

}  // namespace

void launch_gas_rows(const GasRowArgs &a, cudaStream_t st) {
    k_gas_rows<<<(a.N + kWarpsPerCta - 1) / kWarpsPerCta, kThreads, 0, st>>>(a);
}

void launch_gas_step(bool mixed, int form, bool rev, const GasConstsT<float> &kf,
                     const GasConstsT<double> &kd, const GasArgs &a, cudaStream_t st) {
    if (mixed) {
        if (rev)
            step_form<float, true>(form, kf, a, st);
        else
            step_form<float, false>(form, kf, a, st);
    } else {
        if (rev)
            step_form<double, true>(form, kd, a, st);
        else
            step_form<double, false>(form, kd, a, st);
    }
}

void launch_gas_part1(bool mixed, const GasArgs &a, cudaStream_t st) {
    if (mixed)
        k_gas_part1<float><<<(a.N + 127) / 128, 128, 0, st>>>(a);
    else
        k_gas_part1<double><<<(a.N + 127) / 128, 128, 0, st>>>(a);
}

void launch_gas_pack(bool mixed, int N, int nw3, double L, const double *x, void *pos, double *pos64, float4 *posf,
                     cudaStream_t st) {
    if (mixed)
        k_gas_pack<float><<<(N + 127) / 128, 128, 0, st>>>(N, nw3, L, x, pos, pos64, posf);
    else
        k_gas_pack<double><<<(N + 127) / 128, 128, 0, st>>>(N, nw3, L, x, pos, pos64, posf);
}

void launch_gas_pack_w(bool mixed, int N, int nw3, const double *w, double mO, double mH, void *wgt,
                       cudaStream_t st) {
    if (mixed)
        k_gas_pack_w<float><<<(N + 127) / 128, 128, 0, st>>>(N, nw3, w, mO, mH, static_cast<float *>(wgt));
    else
        k_gas_pack_w<double><<<(N + 127) / 128, 128, 0, st>>>(N, nw3, w, mO, mH, static_cast<double *>(wgt));
}

void launch_gas_reset(int n3, const double *g, double f1, double f2, double f3, double *A,
                      double *B, double *C, double *D, double *G, cudaStream_t st) {
    k_gas_reset<<<(n3 + 255) / 256, 256, 0, st>>>(n3, g, f1, f2, f3, A, B, C, D, G);
}

void launch_gas_axpy(int n, double k, const double *x, double *y, cudaStream_t st) {
    k_gas_axpy<<<(n + 255) / 256, 256, 0, st>>>(n, k, x, y);
}

void launch_gas_energy(int form, const GasConsts &k, const GasArgs &a, double *epart,
                       cudaStream_t st) {
    const dim3 grid((a.N + kWarpsPerCta - 1) / kWarpsPerCta);
    switch (form) {
        case F_LJ: k_gas_energy<F_LJ><<<grid, kThreads, 0, st>>>(k, a, epart); break;
        case F_DEXP: k_gas_energy<F_DEXP><<<grid, kThreads, 0, st>>>(k, a, epart); break;
        case F_BUCK: k_gas_energy<F_BUCK><<<grid, kThreads, 0, st>>>(k, a, epart); break;
        case F_LJSC: k_gas_energy<F_LJSC><<<grid, kThreads, 0, st>>>(k, a, epart); break;
        case F_BUFF: k_gas_energy<F_BUFF><<<grid, kThreads, 0, st>>>(k, a, epart); break;
    }
}

void launch_gas_esum(int N, int P, const double *epart, double e_scale, double g_scale,
                     bool accumulate, double *out, cudaStream_t st) {
    k_gas_esum<<<1, 256, 0, st>>>(N, P, epart, e_scale, g_scale, accumulate ? 1 : 0, out);
}

}  // namespace gs
