// sw_kernels.cu -- Stillinger-Weber diamond kernels (sm_100a): candidate-list build,
// per-centre terms with forward-mode tangents, deterministic gather + integrators,
// stress reductions.  Follows diamond/diamond.jl: SW terms 348-381 and 444-532, the
// Enzyme VJP and parameter pullback of sw_force_and_grads! 1658-1697, the stress
// tensor and loss 753-786, the forward step 1462-1467 and the reverse step 1801-1846.
// The decomposition into per-centre slot gradients is described in sw_internal.h.
#include "sw_internal.h"

namespace rs {
namespace sw {

namespace {

__device__ __forceinline__ float xrcp(float a) { return __frcp_rn(a); }
__device__ __forceinline__ double xrcp(double a) { return __drcp_rn(a); }

__device__ __forceinline__ double dist2(const double *xa, const double *xb, double L, double d[3]) {
    // (vec1d's first value, c2 - c1, is its result for all that lies well within half a box)
    bool near = true;
#pragma unroll
    for (int u = 0; u < 3; u++) {
        d[u] = __dsub_rn(xb[u], xa[u]);
        near = near && fabs(d[u]) < 0.49 * L;
    }
    if (!near) {
#pragma unroll
        for (int u = 0; u < 3; u++) d[u] = vec1d(xa[u], xb[u], L);
    }
    return __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])), __dmul_rn(d[2], d[2]));
}

// Sum NV per-thread doubles over the CTA in a fixed order; thread k < NV then adds (or
// writes) the total to out[k].
template <int NV>
__device__ __forceinline__ void cta_sum(double (*s_red)[9], const double *val, double *out,
                                        bool accumulate) {
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        v[k] = val[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] = __dadd_rn(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
    }
    const int warp = threadIdx.x / 32, nw = blockDim.x / 32;
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) s_red[warp][k] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double t = 0.0;
        for (int w = 0; w < nw; w++) t = __dadd_rn(t, s_red[w][threadIdx.x]);
        out[threadIdx.x] = accumulate ? __dadd_rn(out[threadIdx.x], t) : t;
    }
    __syncthreads();
}

// ------------------------------------------------------------ candidate list
__global__ void k_cell_count(SwNlArgs a) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.N) return;
    const int r = a.atom_rep[e];
    const int nc = a.rep_nc[r];
    const double L = a.rep_box[r];
    int ci[3];
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const double xu = a.x[3 * (size_t)e + u];
        a.x_nl[3 * (size_t)e + u] = xu;
        int cc = (int)floor(xu / L * nc);
        ci[u] = cc < 0 ? 0 : (cc >= nc ? nc - 1 : cc);
    }
    const int cell = a.rep_cell_off[r] + (ci[2] * nc + ci[1]) * nc + ci[0];
    a.cell_of[e] = cell;
    atomicAdd(a.cell_cnt + cell, 1);
}

// Exclusive scan of the cell counts, one CTA per replica (its cells hold its atoms, so its scan
// starts at its first atom): every pass takes two consecutive cells a thread, a shuffle scan a warp
// and one scan of the warps' sums.  16 replicas of 1,331 cells: under 4 us; 40 us in one CTA with
// one cell a thread and a barrier per doubling.
__global__ void __launch_bounds__(1024) k_cell_scan(SwNlArgs a) {
    constexpr int PER = 2;
    const int r = blockIdx.x, nc = a.rep_nc[r], first = a.rep_cell_off[r], end = first + nc * nc * nc;
    __shared__ int s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = a.rep_atom0[r];
    for (int base = first; base < end; base += 1024 * PER) {
        const int c0 = base + threadIdx.x * PER;
        int v[PER], sum = 0;
#pragma unroll
        for (int k = 0; k < PER; k++) {
            v[k] = c0 + k < end ? a.cell_cnt[c0 + k] : 0;
            sum += v[k];
        }
        int inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int q = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += q;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        const int wsum = s_warp[lane];
        int winc = wsum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int q = __shfl_up_sync(0xffffffffu, winc, o);
            if (lane >= o) winc += q;
        }
        int run = carry + inc - sum + __shfl_sync(0xffffffffu, winc - wsum, warp);
        carry += __shfl_sync(0xffffffffu, winc, 31);
#pragma unroll
        for (int k = 0; k < PER; k++)
            if (c0 + k < end) {
                a.cell_start[c0 + k] = run;
                a.cell_fill[c0 + k] = 0;
                run += v[k];
            }
        __syncthreads();
    }
}

// Cell-ordered FP32 copy of the positions with the atom index in .w: the candidate test
// streams one 16-byte load per atom.
__global__ void k_cell_fill(SwNlArgs a) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.N) return;
    const int c = a.cell_of[e];
    const double *x = a.x + 3 * (size_t)e;
    a.cell_pos[a.cell_start[c] + atomicAdd(a.cell_fill + c, 1)] =
        make_float4((float)x[0], (float)x[1], (float)x[2], __int_as_float(e));
}

// Candidate row of atom e: every other atom of its replica within a sigma + skin, ascending
// index.  The rows only need to hold every active pair (the terms kernel decides activity
// exactly, in FP64), so the test is FP32 with a 1e-4 nm margin.  Cells are at least that
// wide and number at least 3 per side, so the 27 cells around e are distinct and hold
// every candidate.  One warp per atom: lane l < 27 scans cell l, hits are collected in
// shared memory in any order, then each hit is written at its rank (distinct atoms).
constexpr int ROWS_WARPS = 8;
__global__ void __launch_bounds__(32 * ROWS_WARPS) k_rows(SwNlArgs a) {
    __shared__ int s_list[ROWS_WARPS][CAND];
    __shared__ int s_cnt[ROWS_WARPS];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int e = blockIdx.x * ROWS_WARPS + warp;
    if (e >= a.N) return;
    const int r = a.atom_rep[e];
    const int nc = a.rep_nc[r], off = a.rep_cell_off[r];
    const double L = a.rep_box[r];
    const int loc = a.cell_of[e] - off;
    const int cx = loc % nc, cy = (loc / nc) % nc, cz = loc / (nc * nc);
    const float xe0 = (float)a.x[3 * (size_t)e], xe1 = (float)a.x[3 * (size_t)e + 1],
                xe2 = (float)a.x[3 * (size_t)e + 2];
    const float Lf = (float)L, iLf = (float)(1.0 / L), rl2 = a.rl2f;
    if (lane == 0) s_cnt[warp] = 0;
    __syncwarp();
    if (lane < 27) {
        const int z = (cz + lane / 9 - 1 + nc) % nc;
        const int y = (cy + (lane / 3) % 3 - 1 + nc) % nc;
        const int xx = (cx + lane % 3 - 1 + nc) % nc;
        const int cell = off + (z * nc + y) * nc + xx;
        const int s0 = a.cell_start[cell], s1 = s0 + a.cell_cnt[cell];
        for (int q = s0; q < s1; q++) {
            const float4 pj = a.cell_pos[q];
            const int j = __float_as_int(pj.w);
            float dx = pj.x - xe0, dy = pj.y - xe1, dz = pj.z - xe2;
            dx -= Lf * rintf(dx * iLf);
            dy -= Lf * rintf(dy * iLf);
            dz -= Lf * rintf(dz * iLf);
            if (j != e && dx * dx + dy * dy + dz * dz < rl2) {
                const int k = atomicAdd(&s_cnt[warp], 1);
                if (k < CAND) s_list[warp][k] = j;
            }
        }
    }
    __syncwarp();
    const int cnt = s_cnt[warp];
    const int m = cnt < CAND ? cnt : CAND;
    int *out = a.cand + (size_t)e * CAND;
    for (int it = lane; it < m; it += 32) {
        const int v = s_list[warp][it];
        int rank = 0;
        for (int k = 0; k < m; k++) rank += s_list[warp][k] < v ? 1 : 0;
        out[rank] = v;
    }
    if (lane == 0) {
        if (cnt > CAND) atomicOr(a.status, ST_NLIST_OVERFLOW);
        a.cand_n[e] = m;
        atomicMax(a.max_cnt, cnt);
    }
}

// ------------------------------------------------------------------ terms
// One group of G lanes per centre c.  Phase 1: the candidates are tested in FP64
// (r / sigma < a, as diamond.jl:351) and the active ones compacted into slots in
// ascending index order.  Phase 2: lane q prepares slot q (unit vector, 3-body radial
// factor h = exp(gamma / (s - a)), its derivative factors, the 2-body radial
// derivative).  Phase 3: lane q sums over the other slots q' the 3-body gradient with
// respect to d_q; with u = d / r, cos = u_q . u_q', c3 = cos + 1/3,
//   dE3/dd_q = eps lambda h_q' c3 [ (c3 alpha_q - cos beta_q) u_q + beta_q u_q' ],
//   alpha_q = dh_q/ds / sigma,  beta_q = 2 h_q / r_q,
// so T_q = u_q (eps A g2_q / 2 + eps lambda S1) + eps lambda beta_q V with
// S1 = sum h_q' c3 (c3 alpha_q - cos beta_q), V = sum h_q' c3 u_q'.
//
// Bound by instruction issue (65 %; half of a group's lanes hold a slot).  16 x 8,000 atoms, FP32
// terms, learned pair term, 16 lanes a centre: 144 us with tangents and contraction, 67 us values
// only (event-timed).  205 and 75 us with four tangents carried through dual numbers (94 registers, 20 warps an
// SM) and vec1d's comparisons on every candidate; at 64 registers, some spilled, 32 warps fit (154 ->
// 149 us).
template <typename R, int G, int MODE>
__global__ void __launch_bounds__(TERM_THREADS, sizeof(R) == 4 && MODE != TM_VALUE ? 8 : 0) k_terms(SwTermArgs t, SwConsts<R> p) {
    constexpr bool TAN = MODE != TM_VALUE;
    constexpr int GPB = TERM_THREADS / G;
    __shared__ double s_d[GPB][G][3];
    __shared__ R s_dd[GPB][G][3];
    __shared__ int s_j[GPB][G];
    // slot data read by the other lanes, in 4-vectors: (u, h), (u', h'_pos), (h'_a, h'_gamma,
    // h'_sigma, -) -- the unit vector, its position tangent (u does not depend on theta)
    // and the 3-body radial factor h with its tangents
    using V4 = typename V4T<R>::T;
    __shared__ V4 s_uh[GPB][G];
    __shared__ V4 s_ut[GPB][TAN ? G : 1];
    chain_enter();
    __shared__ V4 s_ht[GPB][TAN ? G : 1];
    __shared__ double s_red[TERM_THREADS / 32][9];

    const int lane = threadIdx.x % G, grp = threadIdx.x / G;
    const int gshift = (threadIdx.x % 32) / G * G;
    const unsigned gbits = G == 32 ? 0xffffffffu : ((1u << G) - 1u);
    const unsigned gmask = gbits << gshift;
    const int b = blockIdx.x;
    const int rep = t.blk_rep[b];
    const bool live = grp < t.blk_n[b];
    const int c = t.blk_atom0[b] + grp;
    const double L = t.rep_box[rep];

    double xc[3] = {0.0, 0.0, 0.0}, wc[3] = {0.0, 0.0, 0.0}, ac[3] = {0.0, 0.0, 0.0};
    int nc = 0;
    if (live) {
#pragma unroll
        for (int u = 0; u < 3; u++) xc[u] = t.x[3 * (size_t)c + u];
        nc = t.cand_n[c];
        if (lane == 0) {
            double d[3];
            if (dist2(t.x_nl + 3 * (size_t)c, xc, L, d) > t.half_skin2) atomicOr(t.status, ST_SKIN);
        }
        if (MODE == TM_REV) {
#pragma unroll
            for (int u = 0; u < 3; u++) {
                wc[u] = __dmul_rn(t.C[3 * (size_t)c + u], t.inv_m);
                ac[u] = __dmul_rn(t.A[3 * (size_t)c + u], t.acoef_scale);
            }
        }
    }
    const double *S = MODE == TM_LOSS ? t.S + 9 * rep : nullptr;
    const double invV = MODE == TM_LOSS ? 1.0 / t.rep_vol[rep] : 0.0;

    // Phase 1: active slots.
    int n = 0;
    for (int k0 = 0; k0 < nc; k0 += G) {
        const int k = k0 + lane;
        bool act = false;
        double d[3] = {0.0, 0.0, 0.0};
        int j = -1;
        if (k < nc) {
            j = t.cand[(size_t)c * CAND + k];
            const double r2 = dist2(xc, t.x + 3 * (size_t)j, L, d);
            // r / sigma < a decided in FP64 as the reference rounds it; r^2 outside a
            // 1e-9 relative band around (a sigma)^2 decides it without the root.
            act = r2 < p.lo2 || (r2 <= p.hi2 && __ddiv_rn(__dsqrt_rn(r2), p.sig64) < p.a64);
        }
        const unsigned bal = (__ballot_sync(gmask, act) >> gshift) & gbits;
        if (act) {
            const int q = n + __popc(bal & ((1u << lane) - 1u));
            if (q < G) {
                s_j[grp][q] = j;
#pragma unroll
                for (int u = 0; u < 3; u++) s_d[grp][q][u] = d[u];
                if (MODE == TM_REV) {
#pragma unroll
                    for (int u = 0; u < 3; u++)
                        s_dd[grp][q][u] = (R)__dsub_rn(__dmul_rn(t.C[3 * (size_t)j + u], t.inv_m), wc[u]);
                } else if (MODE == TM_LOSS) {
#pragma unroll
                    for (int u = 0; u < 3; u++)
                        s_dd[grp][q][u] = (R)__dadd_rn(__dadd_rn(__dmul_rn(S[3 * u], d[0]),
                                                                  __dmul_rn(S[3 * u + 1], d[1])),
                                                       __dmul_rn(S[3 * u + 2], d[2]));
                }
            }
        }
        n += __popc(bal);
    }
    if (n > G) {
        if (lane == 0) atomicOr(t.status, ST_NLIST_OVERFLOW);
        n = G;
    }
    if (live && lane == 0) {
        t.act_n[c] = n;
        atomicMax(t.max_act, n);
    }
    __syncwarp(gmask);

    // Phase 2: per-slot quantities (u = d / r, h = exp(gamma / t), alpha = dh/ds / sigma,
    // beta = 2 h / r with s = r / sigma, t = s - a; t from an FP64 difference to keep its
    // digits near the cutoff).  Divisions are reciprocals.  Tangents 0 (the position direction), 1
    // (a), 2 (gamma) and 3 (sigma) follow from those of s (0: r' / sigma, 3: -s / sigma) and t
    // (those, and 1: -1), in closed form: most of a dual number's tangents would be zeros here.
    const bool own = lane < n;
    R u[3] = {R(0), R(0), R(0)}, alpha = R(0), beta = R(0), g2 = R(0), gB = R(0);
    R gm = R(0);              // learned term: u'(r) / 2, the slot's half of the pair
    int mg = -1;              // its interval (-1: off) and position in it
    R msv = R(0);
    R u0[3] = {R(0), R(0), R(0)}, al[4], be[4], g2t[4], gm0 = R(0);   // tangents
    R z[3] = {R(0), R(0), R(0)};   // the contraction's weights of this slot
    if (TAN) {
#pragma unroll
        for (int k = 0; k < 4; k++) al[k] = be[k] = g2t[k] = R(0);
    }
    if (own) {
        double d64[3];
#pragma unroll
        for (int k = 0; k < 3; k++) d64[k] = s_d[grp][lane][k];
        const int j = s_j[grp][lane];
        t.act_idx[(size_t)c * G + lane] = j;
        if (MODE == TM_REV && t.part) {
#pragma unroll
            for (int k = 0; k < 3; k++)
                z[k] = (R)__dsub_rn(__dmul_rn(t.A[3 * (size_t)j + k], t.acoef_scale), ac[k]);
        } else if (MODE == TM_LOSS && t.part) {
#pragma unroll
            for (int k = 0; k < 3; k++)
                z[k] = (R)__dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(S[3 * k], d64[0]), __dmul_rn(S[3 * k + 1], d64[1])),
                                              __dmul_rn(S[3 * k + 2], d64[2])),
                                    invV);
        }
        const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(d64[0], d64[0]), __dmul_rn(d64[1], d64[1])),
                                    __dmul_rn(d64[2], d64[2]));
        const R r = xsqrt((R)r2), ir = xrcp(r);
#pragma unroll
        for (int k = 0; k < 3; k++) u[k] = xmul((R)d64[k], ir);
        const R sv = xmul(r, p.isig);
        // t = s - a = (r^2 - (a sigma)^2) / (sigma (r + a sigma)), the difference in FP64
        const R tv = xmul((R)__dsub_rn(r2, p.lim2), xrcp(xmul(p.sig, xadd(r, p.asig))));
        const R it = xrcp(tv), it2 = xmul(it, it);
        const R h = xexp(xmul(p.gam, it));
        alpha = -xmul(xmul(xmul(p.gam, h), it2), p.isig);
        beta = xmul(R(2), xmul(h, ir));
        // 2-body: dE2/dr / (eps A) = e^{1/t} (-4 B s^-5 - (B s^-4 - 1) / t^2) / sigma
        // (diamond.jl:453), and its B derivative.
        const R e1 = xexp(it);
        const R is = xrcp(sv);
        const R is2 = xmul(is, is), is4 = xmul(is2, is2), is5 = xmul(is4, is);
        const R B4 = xsub(xmul(p.B, is4), R(1));   // B s^-4 - 1
        const R gv = xadd(xmul(xmul(R(4), p.B), is5), xmul(B4, it2));
        g2 = xmul(xmul(e1, -gv), p.isig);
        gB = xmul(xmul(e1, -xadd(xmul(R(4), is5), xmul(is4, it2))), p.isig);
        R rdot = R(0), h0 = R(0), hp[3] = {R(0), R(0), R(0)};
        if constexpr (TAN) {
            // r' = u . d'; u' = (d' - u r') / r
            R dd[3];
#pragma unroll
            for (int k = 0; k < 3; k++) dd[k] = s_dd[grp][lane][k];
            rdot = xfma(u[0], dd[0], xfma(u[1], dd[1], xmul(u[2], dd[2])));
#pragma unroll
            for (int k = 0; k < 3; k++) u0[k] = xmul(xsub(dd[k], xmul(u[k], rdot)), ir);
            // 1/t' = -s' / t^2.  1/t has no bound (5e15 an ulp of r^2 inside the cutoff) and only
            // e^{1/t} and h make its powers vanish: FP32 holds its square, so every product takes one
            // of the two factors (through q, h / t, gamma h) before a second 1 / t^2.
            const R s0 = xmul(rdot, p.isig), s3 = -xmul(sv, p.isig);
            const R gh = xmul(p.gam, h);
            hp[0] = xmul(gh, it2);
            hp[1] = xmul(h, it);
            hp[2] = -xmul(hp[0], s3);
            h0 = -xmul(hp[0], s0);
            const R A0 = xmul(xmul(p.gam, it2), p.isig), c1 = xmul(xmul(R(2), gh), xmul(p.isig, it));
            al[1] = -xfma(hp[0], A0, xmul(c1, it2));
            al[0] = -xmul(al[1], s0);
            al[2] = -xfma(hp[1], A0, xmul(xmul(h, it2), p.isig));
            al[3] = -xfma(al[1], s3, xmul(alpha, p.isig));
            const R b2 = xadd(ir, ir);
            be[0] = xmul(b2, xfma(-xmul(h, rdot), ir, h0));
            be[1] = xmul(b2, hp[0]);
            be[2] = xmul(b2, hp[1]);
            be[3] = xmul(b2, hp[2]);
            // d(gv) = gs ds + 2 (B s^-4 - 1) (1/t) d(1/t), d(e^{1/t}) = e^{1/t} d(1/t); along s both
            // s and t move (g2s), along a only t
            const R is3 = xmul(is2, is);
            const R gs = -xmul(xmul(R(4), p.B), xmul(is2, xfma(R(5), is4, xmul(is3, it2))));
            const R H = xfma(xmul(R(2), B4), it, gv), E = -xmul(e1, p.isig), q = xmul(E, it2);
            const R g2s = xfma(-q, H, xmul(E, gs));
            g2t[0] = xmul(g2s, s0);
            g2t[1] = xmul(q, H);
            g2t[3] = xsub(xmul(g2s, s3), xmul(g2, p.isig));
        }
        if (t.mlp_tab && r2 < p.mlp_rc2) {
            // u'/2 = (c1 + s (2 c2 + 3 s c3)) NG / (2 rc) on the cubic segment of interval
            // g, s = r NG / rc - g; its position tangent u''/2 r' = (c2 + 3 s c3) (NG/rc)^2 r'
            const R q = xmul(r, p.mlp_hinv);
            mg = min((int)q, MLP_NG - 1);
            msv = xsub(q, (R)mg);
            const V4 cc = reinterpret_cast<const V4 *>(t.mlp_tab)[mg];
            const R s3 = xmul(R(3), msv);
            gm = xmul(xfma(msv, xfma(s3, cc.w, xmul(R(2), cc.z)), cc.y), p.mlp_hhalf);
            if (TAN) gm0 = xmul(xmul(xfma(s3, cc.w, cc.z), p.mlp_hinv2), rdot);
        }
        V4 uh;
        uh.x = u[0];
        uh.y = u[1];
        uh.z = u[2];
        uh.w = h;
        s_uh[grp][lane] = uh;
        if constexpr (TAN) {
            V4 ut, ht;
            ut.x = u0[0];
            ut.y = u0[1];
            ut.z = u0[2];
            ut.w = h0;
            ht.x = hp[0];
            ht.y = hp[1];
            ht.z = hp[2];
            ht.w = R(0);
            s_ut[grp][lane] = ut;
            s_ht[grp][lane] = ht;
        }
    }
    __syncwarp(gmask);

    // Phase 3: 3-body sums over the other slots.  The value arithmetic is the same
    // sequence of rounded operations in every mode.  With w = h' c3 and X = c3 alpha - cos beta
    // the tangents of S1 = sum w X and V = sum w u' need, besides the position direction's,
    // only sums that the parameters share: P = sum w c3 and Q = sum w cos multiply the slot's
    // own alpha', beta'; the neighbours' h' enter the contraction z . T' through
    // Y_m = sum h'_m c3 (zu X + beta z . u'), zu = z . u.
    R S1 = R(0), V[3] = {R(0), R(0), R(0)};
    R S10 = R(0), V0[3] = {R(0), R(0), R(0)}, P = R(0), Q = R(0), Y[3] = {R(0), R(0), R(0)};
    const R zu = TAN ? xfma(z[2], u[2], xfma(z[1], u[1], xmul(z[0], u[0]))) : R(0);
    if (own) {
        const R third = R(1) / R(3);
        R Rc = R(0);   // sum w cos'
        for (int q2 = 0; q2 < n; q2++) {
            // the slot itself enters with weight 0 (its terms are finite), which keeps the
            // lanes of a group on one path
            const R one = q2 == lane ? R(0) : R(1);
            const V4 uh2 = s_uh[grp][q2];
            const R u2[3] = {uh2.x, uh2.y, uh2.z};
            const R h2 = xmul(uh2.w, one);
            const R cs = xadd(xadd(xmul(u[0], u2[0]), xmul(u[1], u2[1])), xmul(u[2], u2[2]));
            const R c3 = xadd(cs, third);
            const R w = xmul(h2, c3);
            const R X = xsub(xmul(c3, alpha), xmul(cs, beta));
            S1 = xadd(S1, xmul(w, X));
#pragma unroll
            for (int k = 0; k < 3; k++) V[k] = xadd(V[k], xmul(w, u2[k]));
            if constexpr (TAN) {
                const V4 ut2 = s_ut[grp][q2], ht2 = s_ht[grp][q2];
                const R u20[3] = {ut2.x, ut2.y, ut2.z};
                const R cs0 = xfma(u0[0], u2[0], xfma(u[0], u20[0], xfma(u0[1], u2[1], xfma(u[1], u20[1],
                                   xfma(u0[2], u2[2], xmul(u[2], u20[2]))))));
                const R c31 = xmul(c3, one);
                const R w0 = xfma(ut2.w, c31, xmul(h2, cs0));
                S10 = xfma(w0, X, S10);
                Rc = xfma(w, cs0, Rc);
                P = xfma(w, c3, P);
                Q = xfma(w, cs, Q);
#pragma unroll
                for (int k = 0; k < 3; k++) V0[k] = xfma(w0, u2[k], xfma(w, u20[k], V0[k]));
                const R zu2 = xfma(z[2], u2[2], xfma(z[1], u2[1], xmul(z[0], u2[0])));
                const R y = xmul(c31, xfma(zu, X, xmul(beta, zu2)));
                Y[0] = xfma(ht2.x, y, Y[0]);
                Y[1] = xfma(ht2.y, y, Y[1]);
                Y[2] = xfma(ht2.z, y, Y[2]);
            }
        }
        if (TAN) S10 = xadd(xfma(xsub(alpha, beta), Rc, S10), xfma(al[0], P, -xmul(be[0], Q)));
    }
    double d64[3] = {0.0, 0.0, 0.0};
    if (own) {
#pragma unroll
        for (int k = 0; k < 3; k++) d64[k] = s_d[grp][lane][k];
    }
    R T[3];
    const R coef = xadd(xadd(xmul(p.half_eA, g2), xmul(p.el, S1)), gm);
    const R elb = xmul(p.el, beta);
#pragma unroll
    for (int k = 0; k < 3; k++) T[k] = xadd(xmul(u[k], coef), xmul(elb, V[k]));
    if (own) {
        V4 tv;
        tv.x = T[0];
        tv.y = T[1];
        tv.z = T[2];
        tv.w = R(0);
        reinterpret_cast<V4 *>(t.Tv)[(size_t)c * G + lane] = tv;
        if constexpr (TAN) {
            const R coef0 = xadd(xfma(p.half_eA, g2t[0], xmul(p.el, S10)), gm0), elb0 = xmul(p.el, be[0]);
            R T0[3];
#pragma unroll
            for (int k = 0; k < 3; k++)
                T0[k] = xfma(u0[k], coef, xfma(u[k], coef0, xfma(elb0, V[k], xmul(elb, V0[k]))));
            V4 tt;
            tt.x = T0[0];
            tt.y = T0[1];
            tt.z = T0[2];
            tt.w = R(0);
            reinterpret_cast<V4 *>(t.Tt)[(size_t)c * G + lane] = tt;
        }
    }

    // Parameter contraction sum_q z_q . dT_q/dtheta (theta order A, B, a, lambda, gamma,
    // sigma, eps); the linear parameters from the value parts.
    if constexpr (TAN) {
      if (t.part) {
        double con[NP] = {0, 0, 0, 0, 0, 0, 0};
        if (own) {
            const R zV = xfma(z[2], V[2], xfma(z[1], V[1], xmul(z[0], V[0])));
            const R zT3 = xfma(zu, S1, xmul(beta, zV));
            R zd[3];
#pragma unroll
            for (int m = 0; m < 3; m++) {
                const R s1 = xsub(xmul(al[1 + m], P), xmul(be[1 + m], Q));
                zd[m] = xfma(xmul(p.half_eA, g2t[1 + m]), zu, xmul(p.el, xadd(Y[m], xfma(zu, s1, xmul(be[1 + m], zV)))));
            }
            const double sgn = MODE == TM_REV ? -1.0 : 1.0;
            const double half_g2zu = 0.5 * (double)g2 * (double)zu;
            con[0] = sgn * (double)p.eps * half_g2zu;
            con[1] = sgn * (double)p.half_eA * (double)gB * (double)zu;
            con[2] = sgn * (double)zd[0];
            con[3] = sgn * (double)p.eps * (double)zT3;
            con[4] = sgn * (double)zd[1];
            con[5] = sgn * (double)zd[2];
            con[6] = sgn * ((double)p.A * half_g2zu + (double)p.lam * (double)zT3);
            if (t.mlp_adj && mg >= 0) {
                // z . dT/dc_k = zu k s^(k-1) NG / (2 rc), k = 1..3, into the replica's copy
                const double w = sgn * (double)zu * (double)p.mlp_hhalf, sv = (double)msv;
                double *ad = t.mlp_adj + (((size_t)rep * MLP_NCOPY + (size_t)(c % MLP_NCOPY)) * MLP_NG + mg) * 4;
                atomicAdd(ad + 1, w);
                atomicAdd(ad + 2, 2.0 * w * sv);
                atomicAdd(ad + 3, 3.0 * w * sv * sv);
            }
        }
        cta_sum<NP>(s_red, con, t.part + (size_t)b * NP, true);
      }
    }
    // Virial sum_q T_q (x) d_q (diamond.jl:757-769, as the strain derivative of the energy).
    if (t.wpart) {
        double w9[9];
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int bb = 0; bb < 3; bb++) w9[3 * a + bb] = own ? __dmul_rn((double)T[a], d64[bb]) : 0.0;
        cta_sum<9>(s_red, w9, t.wpart + (size_t)b * 9, false);
    }
}

// ------------------------------------------------------------------ gather
__device__ __forceinline__ void part1(const SwGatherArgs &g, int e, int rep, const uint64_t *seeds) {
    // Un-integration of diamond.jl:1806-1812: x -= v dt/2; v = (v - xi s) / c; x -= v dt/2;
    // wrap; D = c D + dt^2 dl_dfi (1 + c) / 2; C += D.
    const double L = g.rep_box[rep];
    double xi[3] = {0.0, 0.0, 0.0};
    if (seeds) atom_noise(seeds[rep], (uint32_t)(e - g.rep_atom0[rep]), g.rep_sd[rep], xi);
#pragma unroll
    for (int u = 0; u < 3; u++) {
        const size_t i = 3 * (size_t)e + u;
        double x = g.x[i], v = g.v[i];
        x = __dsub_rn(x, __ddiv_rn(__dmul_rn(v, g.dt), 2.0));
        v = __ddiv_rn(__dsub_rn(v, __dmul_rn(xi[u], g.s)), g.c);
        x = __dsub_rn(x, __ddiv_rn(__dmul_rn(v, g.dt), 2.0));
        g.x[i] = wrap1d(x, L);
        g.v[i] = v;
        const double Dn = __dadd_rn(__dmul_rn(g.c, g.D[i]),
                                    __ddiv_rn(__dmul_rn(__dmul_rn(g.dt2, g.G[i]), __dadd_rn(1.0, g.c)), 2.0));
        g.D[i] = Dn;
        g.C[i] = __dadd_rn(g.C[i], Dn);
    }
}

template <typename R, int G, bool TAN>
__global__ void __launch_bounds__(256) k_gather(SwGatherArgs g) {
    // G lanes per atom e: lane q reads slot q (T_{e,q}) and the matching slot of its
    // neighbour (T_{j_q, slot of e}); a butterfly sum over the lanes (every lane ends
    // with the same bits: each level adds two equal-order pairs) gives f = dE/dx_e and
    // tg, its derivative along the tangent (H w or H u).  Lane 0 writes F = -f and
    // G = -tg; k_finish integrates.
    chain_enter();
    const int lane = threadIdx.x % G;
    const int e = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G);
    const int gshift = (threadIdx.x % 32) / G * G;
    const unsigned gmask = (G == 32 ? 0xffffffffu : ((1u << G) - 1u)) << gshift;
    using V4 = typename V4T<R>::T;
    const V4 *Tv = reinterpret_cast<const V4 *>(g.Tv);
    const V4 *Tt = reinterpret_cast<const V4 *>(g.Tt);
    const bool live = e < g.N;
    double f[3] = {0.0, 0.0, 0.0}, tg[3] = {0.0, 0.0, 0.0};
    if (live) {
        const int n = g.act_n[e];
        if (lane < n) {
            const int j = g.act_idx[(size_t)e * G + lane];
            const int nj = g.act_n[j];
            // the neighbour's whole slot row in G/4 16-byte loads, then compare
            const int4 *rj = reinterpret_cast<const int4 *>(g.act_idx + (size_t)j * G);
            int4 row[G / 4];
#pragma unroll
            for (int k = 0; k < G / 4; k++) row[k] = rj[k];
            int pos = -1;
#pragma unroll
            for (int k = 0; k < G / 4; k++) {
                if (4 * k + 0 < nj && row[k].x == e) pos = 4 * k + 0;
                if (4 * k + 1 < nj && row[k].y == e) pos = 4 * k + 1;
                if (4 * k + 2 < nj && row[k].z == e) pos = 4 * k + 2;
                if (4 * k + 3 < nj && row[k].w == e) pos = 4 * k + 3;
            }
            if (pos < 0) {
                atomicOr(g.status, ST_NLIST_OVERFLOW);
            } else {
                const size_t ie = (size_t)e * G + lane, ij = (size_t)j * G + pos;
                const V4 a = Tv[ij], b = Tv[ie];
                f[0] = __dsub_rn((double)a.x, (double)b.x);
                f[1] = __dsub_rn((double)a.y, (double)b.y);
                f[2] = __dsub_rn((double)a.z, (double)b.z);
                if (TAN) {
                    const V4 at = Tt[ij], bt = Tt[ie];
                    tg[0] = __dsub_rn((double)at.x, (double)bt.x);
                    tg[1] = __dsub_rn((double)at.y, (double)bt.y);
                    tg[2] = __dsub_rn((double)at.z, (double)bt.z);
                }
            }
        }
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
#pragma unroll
        for (int u = 0; u < 3; u++) {
            f[u] = __dadd_rn(f[u], __shfl_xor_sync(gmask, f[u], o));
            if (TAN) tg[u] = __dadd_rn(tg[u], __shfl_xor_sync(gmask, tg[u], o));
        }
    }
    if (!live || lane != 0) return;
#pragma unroll
    for (int u = 0; u < 3; u++) {
        g.F[3 * (size_t)e + u] = -f[u];
        if (TAN) g.G[3 * (size_t)e + u] = -tg[u];
    }
    if (!(isfinite(f[0]) && isfinite(f[1]) && isfinite(f[2]) && isfinite(tg[0]) && isfinite(tg[1]) &&
          isfinite(tg[2])))
        atomicOr(g.status, ST_NAN);
}

// One thread per atom: the step (or loss) arithmetic after the gather.
template <int MODE>
__global__ void __launch_bounds__(256) k_finish(SwGatherArgs g) {
    chain_enter();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= g.N) return;
    double f[3], tg[3];
#pragma unroll
    for (int u = 0; u < 3; u++) {
        f[u] = -g.F[3 * (size_t)e + u];
        tg[u] = MODE == GM_FWD ? 0.0 : -g.G[3 * (size_t)e + u];
    }
    const int rep = g.atom_rep[e];
    // f = dE/dx_e, tg = its derivative along the tangent (H w or H u).
    if (MODE == GM_FWD) {
        // diamond.jl:1462-1467
        const double L = g.rep_box[rep];
        double xi[3] = {0.0, 0.0, 0.0};
        if (g.seed_cur) atom_noise(g.seed_cur[rep], (uint32_t)(e - g.rep_atom0[rep]), g.rep_sd[rep], xi);
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const size_t i = 3 * (size_t)e + u;
            const double F = -f[u];
            double v = __dadd_rn(g.v[i], __ddiv_rn(__dmul_rn(F, g.dt), g.m));
            double x = __dadd_rn(g.x[i], __ddiv_rn(__dmul_rn(v, g.dt), 2.0));
            v = __dadd_rn(__dmul_rn(v, g.c), __dmul_rn(xi[u], g.s));
            x = __dadd_rn(x, __ddiv_rn(__dmul_rn(v, g.dt), 2.0));
            g.x[i] = wrap1d(x, L);
            g.v[i] = v;
        }
        return;
    }
    if (MODE == GM_REV) {
        // diamond.jl:1838-1846: v -= F dt / m; B = c B + dt^2 dl_dfi; A += B
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const size_t i = 3 * (size_t)e + u;
            const double F = -f[u], Gn = -tg[u];
            g.v[i] = __dsub_rn(g.v[i], __ddiv_rn(__dmul_rn(F, g.dt), g.m));
            const double Bn = __dadd_rn(__dmul_rn(g.c, g.B[i]), __dmul_rn(g.dt2, Gn));
            g.B[i] = Bn;
            g.A[i] = __dadd_rn(g.A[i], Bn);
        }
        if (g.fuse_next) part1(g, e, rep, g.seed_next);
        return;
    }
    if (MODE == GM_LOSS) {
        // dL/dx = (H u + S^T dE/dx) / V,  dL/dv = -(m / V) (S + S^T)(v - vbar)
        const double *S = g.S + 9 * rep;
        const double V = g.rep_vol[rep];
        double gx[3], gv[3];
#pragma unroll
        for (int gm = 0; gm < 3; gm++) {
            double st = 0.0;
#pragma unroll
            for (int al = 0; al < 3; al++) st = __dadd_rn(st, __dmul_rn(S[3 * al + gm], f[al]));
            gx[gm] = __ddiv_rn(__dadd_rn(tg[gm], st), V);
            double tv = 0.0;
            if (g.vel_term) {
#pragma unroll
                for (int bb = 0; bb < 3; bb++)
                    tv = __dadd_rn(tv, __dmul_rn(__dadd_rn(S[3 * gm + bb], S[3 * bb + gm]),
                                                 __dsub_rn(g.v[3 * (size_t)e + bb], g.vbar[3 * rep + bb])));
            }
            gv[gm] = g.vel_term ? __ddiv_rn(__dmul_rn(-g.m, tv), V) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 3; u++) {
            const size_t i = 3 * (size_t)e + u;
            if (g.dLdx) g.dLdx[i] = gx[u];
            if (g.dLdv) g.dLdv[i] = gv[u];
            if (g.init_adjoint) {
                // diamond.jl:1789-1793
                const double c = g.c, dt = g.dt;
                g.A[i] = __dadd_rn(__dmul_rn(gx[u], __dadd_rn(1.0, c)), __ddiv_rn(__dmul_rn(__dmul_rn(gv[u], c), 2.0), dt));
                g.B[i] = __dadd_rn(__dmul_rn(gx[u], __dadd_rn(1.0, c)),
                                   __ddiv_rn(__dmul_rn(__dmul_rn(gv[u], __dsub_rn(c, 1.0)), 2.0), dt));
                g.C[i] = __ddiv_rn(__dmul_rn(gv[u], __dadd_rn(1.0, c)), dt);
                g.D[i] = __dadd_rn(__ddiv_rn(__dmul_rn(gx[u], __dadd_rn(__dadd_rn(1.0, __dmul_rn(2.0, c)), __dmul_rn(c, c))),
                                             __dmul_rn(2.0, c)),
                                   __ddiv_rn(__dmul_rn(gv[u], __dsub_rn(c, __ddiv_rn(1.0, c))), dt));
                g.G[i] = 0.0;
            }
        }
    }
}

__global__ void k_part1(SwGatherArgs g) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= g.N) return;
    part1(g, e, g.atom_rep[e], g.seed_cur);
}

__global__ void k_noise(int N, const int *atom_rep, const int *rep_atom0, const double *rep_sd,
                        const uint64_t *seeds, double *xi) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= N) return;
    const int r = atom_rep[e];
    atom_noise(seeds[r], (uint32_t)(e - rep_atom0[r]), rep_sd[r], xi + 3 * (size_t)e);
}

// ------------------------------------------------------------- reductions
template <int NV>
__device__ __forceinline__ void block_sum256(double (*s)[256], double *v, double *out) {
#pragma unroll
    for (int k = 0; k < NV; k++) s[k][threadIdx.x] = v[k];
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
#pragma unroll
            for (int k = 0; k < NV; k++) s[k][threadIdx.x] = __dadd_rn(s[k][threadIdx.x], s[k][threadIdx.x + o]);
        }
        __syncthreads();
    }
    if (threadIdx.x < NV) out[threadIdx.x] = s[threadIdx.x][0];
}

__global__ void __launch_bounds__(256) k_vsum(SwRedArgs a) {
    __shared__ double s[3][256];
    const int b = blockIdx.x;
    const int i = threadIdx.x;
    double v[3] = {0.0, 0.0, 0.0};
    if (i < a.ablk_n[b]) {
        const size_t e = (size_t)a.ablk_atom0[b] + i;
#pragma unroll
        for (int u = 0; u < 3; u++) v[u] = a.v[3 * e + u];
    }
    block_sum256<3>(s, v, a.vpart + 3 * (size_t)b);
}

// Per-replica sums of block partials: thread t adds blocks b0 + t, b0 + t + 256, ... in
// order, then a fixed tree over the threads.
template <int NV>
__device__ __forceinline__ void range_sum256(double (*s)[256], const double *part, int b0, int b1,
                                             double *out) {
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = 0.0;
    for (int b = b0 + threadIdx.x; b < b1; b += 256) {
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = __dadd_rn(v[k], part[(size_t)b * NV + k]);
    }
    block_sum256<NV>(s, v, out);
    __syncthreads();
}

__global__ void __launch_bounds__(256) k_vbar(SwRedArgs a) {
    __shared__ double s[3][256];
    __shared__ double tot[3];
    const int r = blockIdx.x;
    range_sum256<3>(s, a.vpart, a.rep_ablk0[r], a.rep_ablk0[r + 1], tot);
    if (threadIdx.x < 3) a.vbar[3 * r + threadIdx.x] = __ddiv_rn(tot[threadIdx.x], (double)a.rep_n[r]);
}

__global__ void __launch_bounds__(256) k_kin(SwRedArgs a) {
    __shared__ double s[9][256];
    const int b = blockIdx.x;
    const int i = threadIdx.x;
    double k9[9];
#pragma unroll
    for (int k = 0; k < 9; k++) k9[k] = 0.0;
    if (i < a.ablk_n[b]) {
        const size_t e = (size_t)a.ablk_atom0[b] + i;
        const int r = a.ablk_rep[b];
        double dv[3];
#pragma unroll
        for (int u = 0; u < 3; u++) dv[u] = __dsub_rn(a.v[3 * e + u], a.vbar[3 * r + u]);
#pragma unroll
        for (int al = 0; al < 3; al++)
#pragma unroll
            for (int be = 0; be < 3; be++) k9[3 * al + be] = __dmul_rn(dv[al], dv[be]);
    }
    block_sum256<9>(s, k9, a.kpart + 9 * (size_t)b);
}

// sigma = (K + W) / V (diamond.jl:753-770); loss = weight sum (sigma - target)^2 / 9
// (diamond.jl:772-775); S = dL/dsigma.
__global__ void __launch_bounds__(256) k_loss_final(SwRedArgs a) {
    __shared__ double s[9][256];
    __shared__ double W[9], Kt[9];
    const int r = blockIdx.x;
    range_sum256<9>(s, a.wpart, a.rep_blk0[r], a.rep_blk0[r + 1], W);
    if (a.vel_term) range_sum256<9>(s, a.kpart, a.rep_ablk0[r], a.rep_ablk0[r + 1], Kt);
    if (threadIdx.x != 0) return;
    const double V = a.rep_vol[r];
    double l = 0.0;
    for (int k = 0; k < 9; k++) {
        const double K = a.vel_term ? __dmul_rn(-a.m, Kt[k]) : 0.0;
        const double sg = __ddiv_rn(__dadd_rn(K, W[k]), V);
        if (a.sigma) a.sigma[9 * r + k] = sg;
        const double e = __dsub_rn(sg, a.target[9 * r + k]);
        l = __dadd_rn(l, __dmul_rn(e, e));
        if (a.S) a.S[9 * r + k] = __ddiv_rn(__dmul_rn(__dmul_rn(2.0, a.weight), e), 9.0);
    }
    l = __dmul_rn(l, __ddiv_rn(a.weight, 9.0));
    if (a.loss) a.loss[r] = l;
    if (a.loss_acc) a.loss_acc[r] = __dadd_rn(a.loss_acc[r], l);
}

__global__ void k_active_pairs(int N, int G, const int *act_idx, const int *act_n, int32_t *pairs,
                               unsigned long long *count, long long max_pairs) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= N) return;
    for (int q = 0; q < act_n[e]; q++) {
        const int j = act_idx[(size_t)e * G + q];
        if (j <= e) continue;
        const unsigned long long k = atomicAdd(count, 1ull);
        if ((long long)k < max_pairs) {
            pairs[2 * k] = e;
            pairs[2 * k + 1] = j;
        }
    }
}

inline int nblk(int n, int t) { return (n + t - 1) / t; }

}  // namespace

// ------------------------------------------------------------------ launchers
cudaError_t launch_sw_nlist(const SwNlArgs &a, cudaStream_t st) {
    cudaError_t e;
    if ((e = cudaMemsetAsync(a.cell_cnt, 0, sizeof(int) * a.n_cells, st))) return e;
    k_cell_count<<<nblk(a.N, 256), 256, 0, st>>>(a);
    k_cell_scan<<<a.R, 1024, 0, st>>>(a);
    k_cell_fill<<<nblk(a.N, 256), 256, 0, st>>>(a);
    k_rows<<<nblk(a.N, ROWS_WARPS), 32 * ROWS_WARPS, 0, st>>>(a);
    return cudaGetLastError();
}

template <typename R>
cudaError_t launch_sw_terms(int mode, int G, int n_blk, const SwTermArgs &a, const SwConsts<R> &p,
                            cudaStream_t st) {
#define RS_TERMS(GG, MM) launch_chained(k_terms<R, GG, MM>, dim3(n_blk), dim3(TERM_THREADS), 0, st, a, p)
    if (G == 16) {
        if (mode == TM_VALUE) RS_TERMS(16, TM_VALUE);
        else if (mode == TM_REV) RS_TERMS(16, TM_REV);
        else RS_TERMS(16, TM_LOSS);
    } else if (G == 32) {
        if (mode == TM_VALUE) RS_TERMS(32, TM_VALUE);
        else if (mode == TM_REV) RS_TERMS(32, TM_REV);
        else RS_TERMS(32, TM_LOSS);
    } else {
        return cudaErrorInvalidValue;
    }
#undef RS_TERMS
    return cudaGetLastError();
}

template <typename R>
cudaError_t launch_sw_gather(int mode, int G, bool tangent, const SwGatherArgs &a, cudaStream_t st) {
    const int nb = (int)(((size_t)a.N * G + 255) / 256);
    const bool tan = tangent || mode == GM_REV || mode == GM_LOSS;
    if (G == 16) {
        if (tan) launch_chained(k_gather<R, 16, true>, dim3(nb), dim3(256), 0, st, a);
        else launch_chained(k_gather<R, 16, false>, dim3(nb), dim3(256), 0, st, a);
    } else if (G == 32) {
        if (tan) launch_chained(k_gather<R, 32, true>, dim3(nb), dim3(256), 0, st, a);
        else launch_chained(k_gather<R, 32, false>, dim3(nb), dim3(256), 0, st, a);
    } else {
        return cudaErrorInvalidValue;
    }
    const int na = nblk(a.N, 256);
    if (mode == GM_FWD) launch_chained(k_finish<GM_FWD>, dim3(na), dim3(256), 0, st, a);
    else if (mode == GM_REV) launch_chained(k_finish<GM_REV>, dim3(na), dim3(256), 0, st, a);
    else if (mode == GM_LOSS) launch_chained(k_finish<GM_LOSS>, dim3(na), dim3(256), 0, st, a);
    return cudaGetLastError();
}

cudaError_t launch_sw_stress(const SwRedArgs &a, cudaStream_t st) {
    k_vsum<<<a.n_ablk, 256, 0, st>>>(a);
    k_vbar<<<a.R, 256, 0, st>>>(a);
    k_kin<<<a.n_ablk, 256, 0, st>>>(a);
    k_loss_final<<<a.R, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sw_part1(int N, const SwGatherArgs &a, cudaStream_t st) {
    k_part1<<<nblk(N, 256), 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_sw_noise(int N, const int *atom_rep, const int *rep_atom0, const double *rep_sd,
                            const uint64_t *seeds, double *xi, cudaStream_t st) {
    k_noise<<<nblk(N, 256), 256, 0, st>>>(N, atom_rep, rep_atom0, rep_sd, seeds, xi);
    return cudaGetLastError();
}

cudaError_t launch_sw_active_pairs(int N, int G, const int *act_idx, const int *act_n,
                                   int32_t *pairs, unsigned long long *count, long long max_pairs,
                                   cudaStream_t st) {
    k_active_pairs<<<nblk(N, 256), 256, 0, st>>>(N, G, act_idx, act_n, pairs, count, max_pairs);
    return cudaGetLastError();
}

template cudaError_t launch_sw_terms<float>(int, int, int, const SwTermArgs &, const SwConsts<float> &,
                                            cudaStream_t);
template cudaError_t launch_sw_terms<double>(int, int, int, const SwTermArgs &,
                                             const SwConsts<double> &, cudaStream_t);
template cudaError_t launch_sw_gather<float>(int, int, bool, const SwGatherArgs &, cudaStream_t);
template cudaError_t launch_sw_gather<double>(int, int, bool, const SwGatherArgs &, cudaStream_t);

}  // namespace sw
}  // namespace rs
