// rs_energy.cu -- potential energy and its parameter gradient at the current state: the
// per-snapshot dE/dtheta of the reweighting estimator (reweighting_sim, water.jl:1107-1210;
// the Zygote gradient of potential_energy at water.jl:1176-1183).  FP64, once per loss point.
//
// One warp per molecule I sums the molecule pairs (I, J > I) of its neighbour row (each
// unordered pair once; the row's 9-bit mask gives the listed atom pairs), the pair-form
// energy on dual numbers whose tangents are the form's parameters, the reaction-field
// Coulomb energy (dE/dq_O = 2 E_c / q_O), its own two bonds and angle, and -- with the
// learned term -- the interval-coefficient adjoints (1, s, s^2, s^3) of each pair's Hermite
// segment, which the MLP backpropagation turns into dE/dtheta_mlp.  Per-molecule partials
// [E, dE/dtheta...] are summed per replica by one CTA each (k_rep_sums), or -- for the
// enthalpy-of-vaporisation loss term (loss_enth_vap, water.jl:738-755) -- by
// k_enth_finalize, which also turns U into the loss and its coefficient 2 e / n.
#include "rs_form_energy.cuh"
#include "rs_internal.h"

namespace rs {

namespace {

constexpr int EG_WARPS = 4, EG_THREADS = 32 * EG_WARPS;

// Nearest integer by the rounding of a sum with 1.5 x 2^52.
__device__ __forceinline__ double near_int64(double a, double b) {
    return __dadd_rn(__fma_rn(a, b, 6755399441055744.0), -6755399441055744.0);
}

// A warp per molecule.  The row's entries J > I (about half, in runs) are queued in shared
// memory and evaluated 32 at a time, the nine atom pairs of an entry as straight-line code with
// the pairs outside the mask or the cutoff at weight zero.  FP64-pipe bound.  With 16 lanes a
// molecule, each walking its entries pair by pair past the skipped ones: 124 us on the 895-water
// box, 133 us on 3,000 waters; this form: 18 and 19 us.
template <int FORM, typename V4>
__global__ void __launch_bounds__(EG_THREADS) k_energy_grads(EnergyArgs a) {
    __shared__ uint32_t s_q[EG_WARPS][64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int I = blockIdx.x * EG_WARPS + warp;
    if (I >= a.M) return;   // whole warps
    constexpr int NFm = FormInfo<FORM>::NP;
    const int rep = a.mol_rep[I];
    const double L = a.rep_box[rep], invL = 1.0 / L;
    const double *x = a.x;
    const int P = a.P;   // classical parameters
    const bool gate = a.form_p[FORM == F_BUCK ? 0 : 1] != 0.0;
    const double aw = a.adj_scale ? a.adj_mul * a.adj_scale[rep] : 1.0;
    const double qq[3] = {a.ke * (a.qO * a.qO), a.ke * (a.qO * (-0.5 * a.qO)), a.ke * (0.25 * a.qO * a.qO)};
    double *madj = a.mlp_adj ? a.mlp_adj + ((size_t)rep * MLP_NCOPY + (I % MLP_NCOPY)) * MLP_NT * MLP_NG * 4
                             : nullptr;
    const uint32_t *row = a.nbr + (size_t)I * a.cap;
    const int cnt = min(a.nbr_cnt[I], a.cap);
    double xi[9];
#pragma unroll
    for (int u = 0; u < 9; u++) xi[u] = x[9 * (size_t)I + u];
    double ec = 0.0, ef = 0.0, df[NFm];   // Coulomb and other energies, form parameters' derivatives
#pragma unroll
    for (int k = 0; k < NFm; k++) df[k] = 0.0;

    auto eval = [&](uint32_t ent) {
        const int J = (int)(ent & 0x7FFFFFu);
        const uint32_t mask = ent >> 23;
        double xj[9];
#pragma unroll
        for (int u = 0; u < 9; u++) xj[u] = x[9 * (size_t)J + u];
#pragma unroll
        for (int ka = 0; ka < 3; ka++)
#pragma unroll
            for (int kb = 0; kb < 3; kb++) {
                double d[3];
#pragma unroll
                for (int u = 0; u < 3; u++) {
                    d[u] = __dsub_rn(xj[3 * kb + u], xi[3 * ka + u]);
                    d[u] = __fma_rn(-near_int64(d[u], invL), L, d[u]);
                }
                const double r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
                const bool on = ((mask >> (3 * ka + kb)) & 1u) && r2 <= a.rc2;
                const double rinv = rsqrt(on ? r2 : 1.0);
                const double r = r2 > 0.0 ? r2 * rinv : 0.0;   // overlapping atoms: infinite terms, not 0 x inf
                const int QI = (ka > 0) + (kb > 0);
                ec += (on ? qq[QI] : 0.0) * (rinv + a.krf * r2 - a.crf_shift);
                if (ka == 0 && kb == 0 && gate && on) {
                    const DN<4> Ef = form_energy<FORM>(a.form_p, r);
                    ef += Ef.v;
                    if (a.grads) {
#pragma unroll
                        for (int k = 0; k < NFm; k++) df[k] += Ef.d[k];
                    }
                }
                if (FORM == F_LJ_MLP && on) {
                    const double q = r * a.mlp_hinv;
                    const int g = min((int)q, MLP_NG - 1);
                    const double s = q - g;
                    const V4 c = reinterpret_cast<const V4 *>(a.mlp_tab)[QI * MLP_NG + g];
                    ef += (double)c.x + s * ((double)c.y + s * ((double)c.z + s * (double)c.w));
                    if (madj) {
                        double *ad = madj + ((size_t)QI * MLP_NG + g) * 4;
                        atomicAdd(ad, aw);
                        atomicAdd(ad + 1, aw * s);
                        atomicAdd(ad + 2, aw * s * s);
                        atomicAdd(ad + 3, aw * s * s * s);
                    }
                }
            }
    };
    int nq = 0;
    for (int base = 0; base < cnt; base += 32) {
        const uint32_t ent = base + lane < cnt ? row[base + lane] : 0u;
        const bool own = (int)(ent & 0x7FFFFFu) > I;
        const unsigned m = __ballot_sync(0xffffffffu, own);
        if (own) s_q[warp][nq + __popc(m & ((1u << lane) - 1u))] = ent;
        nq += __popc(m);
        __syncwarp();
        if (nq >= 32) {
            nq -= 32;
            eval(s_q[warp][nq + lane]);
            __syncwarp();
        }
    }
    if (lane < nq) eval(s_q[warp][lane]);
    __syncwarp();
    // fixed butterflies over the lanes
    auto wsum = [](double v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    };
    double acc[1 + NFm + 5];
#pragma unroll
    for (int k = 0; k < 1 + NFm + 5; k++) acc[k] = 0.0;
    ec = wsum(ec);
    acc[0] = __dadd_rn(wsum(ef), ec);
    if (a.grads) {
#pragma unroll
        for (int k = 0; k < NFm; k++) acc[1 + k] = wsum(df[k]);
        acc[1 + NFm] = 2.0 * ec / a.qO;
    }
    if (lane != 0) return;
    // bonds (O, H1), (O, H2) and the angle H1-O-H2 (water.jl:915-968 energies)
    const double *xo = x + 9 * (size_t)I;
    double b[2][3];
    for (int h = 0; h < 2; h++) {
        for (int u = 0; u < 3; u++) b[h][u] = vec1d(xo[u], xo[3 * (h + 1) + u], L);
        const double d = sqrt(b[h][0] * b[h][0] + b[h][1] * b[h][1] + b[h][2] * b[h][2]) - a.r0;
        acc[0] += 0.5 * a.kb * d * d;
        acc[1 + NFm + 1] += 0.5 * d * d;
        acc[1 + NFm + 2] += -a.kb * d;
    }
    const double c = (b[0][0] * b[1][0] + b[0][1] * b[1][1] + b[0][2] * b[1][2]) /
                     (sqrt(b[0][0] * b[0][0] + b[0][1] * b[0][1] + b[0][2] * b[0][2]) *
                      sqrt(b[1][0] * b[1][0] + b[1][1] * b[1][1] + b[1][2] * b[1][2]));
    const double th = acos(fmin(1.0, fmax(-1.0, c))) - a.th0;
    acc[0] += 0.5 * a.ka * th * th;
    acc[1 + NFm + 3] += 0.5 * th * th;
    acc[1 + NFm + 4] += -a.ka * th;
#pragma unroll
    for (int k = 0; k < 1 + NFm + 5; k++)
        if (k == 0 || a.grads) a.part[(size_t)I * (P + 1) + k] = acc[k];
}

constexpr int kSumThreads = 512, kSumCols = 10;   // columns: energy and up to nine parameters

// Sums of the first ncol columns of rows r0 .. r0 + n of part (row length stride) over the CTA,
// in a fixed order, into s_tot.  Columns are summed together: one pass over the rows.
__device__ __forceinline__ void col_sums(const double *part, int r0, int n, int stride, int ncol, double *s_tot) {
    __shared__ double s_w[kSumThreads / 32][kSumCols];
    double v[kSumCols];
#pragma unroll
    for (int c = 0; c < kSumCols; c++) v[c] = 0.0;
    for (int i = threadIdx.x; i < n; i += kSumThreads) {
        const double *p = part + (size_t)(r0 + i) * stride;
#pragma unroll
        for (int c = 0; c < kSumCols; c++)
            if (c < ncol) v[c] += p[c];
    }
#pragma unroll
    for (int c = 0; c < kSumCols; c++)
        if (c < ncol) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
            if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5][c] = v[c];
        }
    __syncthreads();
    if ((int)threadIdx.x < ncol) {
        double t = 0.0;
        for (int w = 0; w < kSumThreads / 32; w++) t += s_w[w][threadIdx.x];
        s_tot[threadIdx.x] = t;
    }
    __syncthreads();
}

// Per replica: the sums of the first ncol columns of its molecules' rows.
__global__ void __launch_bounds__(kSumThreads) k_rep_sums(const int *rep_atom0, const int *rep_nmol,
                                                          const double *part, int stride, int ncol, double *out) {
    __shared__ double s_tot[kSumCols];
    const int r = blockIdx.x;
    col_sums(part, rep_atom0[r] / 3, rep_nmol[r], stride, ncol, s_tot);
    if ((int)threadIdx.x < ncol) out[(size_t)r * ncol + threadIdx.x] = s_tot[threadIdx.x];
}

__global__ void __launch_bounds__(kSumThreads) k_enth_finalize(EnthArgs a) {
    __shared__ double s_tot[kSumCols];
    const int r = blockIdx.x, t = threadIdx.x, n = a.rep_nmol[r];
    col_sums(a.part, a.rep_atom0[r] / 3, n, a.P + 1, a.grads ? a.P + 1 : 1, s_tot);
    // enthalpy_vaporization and loss_enth_vap, water.jl:738-755
    const double e = a.u_gas - s_tot[0] / n + a.rt - a.target, kr = 2.0 * e / n;
    if (t == 0) {
        a.acc[r] += e * e;
        if (a.ev_acc) a.ev_acc[r] += e * e;
        a.k[r] = kr;
    }
    if (a.grads && t < a.P) a.dgrad[(size_t)r * a.P + t] += -kr * s_tot[1 + t];
}

__global__ void k_enth_dldx(int n3, const int *atom_rep, const double *k, const double *F, double *dLdx) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n3) dLdx[i] += k[atom_rep[i / 3]] * F[i];
}

template <int FORM>
cudaError_t launch_f(int prec, const EnergyArgs &a, cudaStream_t st) {
    const int b = (a.M + EG_WARPS - 1) / EG_WARPS;
    if (prec == 1)
        k_energy_grads<FORM, float4><<<b, EG_THREADS, 0, st>>>(a);
    else
        k_energy_grads<FORM, double4><<<b, EG_THREADS, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_enth_finalize(const EnthArgs &a, cudaStream_t st) {
    static_assert(kSumCols >= 1 + 4 + 5, "energy, form parameters, charge and bonded parameters");
    if (a.R > 0) k_enth_finalize<<<a.R, kSumThreads, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_rep_sums(int R, const int *rep_atom0, const int *rep_nmol, const double *part, int stride,
                            int ncol, double *out, cudaStream_t st) {
    if (ncol > kSumCols) return cudaErrorInvalidValue;
    if (R > 0) k_rep_sums<<<R, kSumThreads, 0, st>>>(rep_atom0, rep_nmol, part, stride, ncol, out);
    return cudaGetLastError();
}

cudaError_t launch_enth_dldx(int N, const int *atom_rep, const double *k, const double *F, double *dLdx,
                             cudaStream_t st) {
    const int n3 = 3 * N, t = 256;
    if (n3 > 0) k_enth_dldx<<<(n3 + t - 1) / t, t, 0, st>>>(n3, atom_rep, k, F, dLdx);
    return cudaGetLastError();
}

cudaError_t launch_energy_grads(int form, int prec, const EnergyArgs &a, cudaStream_t st) {
    switch (form) {
        case F_LJ: return launch_f<F_LJ>(prec, a, st);
        case F_DEXP: return launch_f<F_DEXP>(prec, a, st);
        case F_BUCK: return launch_f<F_BUCK>(prec, a, st);
        case F_LJSC: return launch_f<F_LJSC>(prec, a, st);
        case F_BUFF: return launch_f<F_BUFF>(prec, a, st);
        case F_LJ_MLP: return launch_f<F_LJ_MLP>(prec, a, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace rs
