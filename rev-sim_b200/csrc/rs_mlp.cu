// rs_mlp.cu -- the learned pair correction of the water model (no reference counterpart;
// it stands in for the reference's PyTorch / JAX learned terms, water_maceoff.jl:147-163).
//
// Per element pair tau in {O-O, O-H, H-H}: u_tau(r) = MLP_tau(phi(r)) fc(r), 16 Gaussian
// radial basis functions (centres k rc / 15, width 0.05 nm), 64 -> 64 SiLU, scalar output,
// fc(r) = (cos(pi r / rc) + 1) / 2.  The MLP depends on r alone, so it is evaluated once per
// parameter update at NG + 1 nodes of [0, rc] (value and r-derivative, FP64) and the step
// kernels interpolate each pair with the cubic Hermite segment of its interval (one
// 16- or 32-byte table load per pair).  The reverse pass accumulates the adjoints of the
// interval coefficients; k_mlp_* below carry them back to the weights once per pass.
// The same code serves the Stillinger-Weber path's learned radial term (one type, its own
// cutoff and width): the type count nt and width w are arguments.
#include <algorithm>

#include "rs_internal.h"

namespace rs {

namespace {

constexpr int NR = MLP_NRBF, H = MLP_H, NG = MLP_NG;
constexpr int NA = 4 * H + 4;   // per-node activations: z1, dz1, z2, dz2, y, dy, fc, dfc

struct View {
    const double *W1, *b1, *W2, *b2, *w3, *b3;
};

__device__ __forceinline__ View view(const double *theta, int t) {
    View v;
    v.W1 = theta + (size_t)t * MLP_PER_TYPE;
    v.b1 = v.W1 + H * NR;
    v.W2 = v.b1 + H;
    v.b2 = v.W2 + H * H;
    v.w3 = v.b2 + H;
    v.b3 = v.w3 + H;
    return v;
}

__device__ __forceinline__ double sigm(double z) { return 1.0 / (1.0 + exp(-z)); }
__device__ __forceinline__ double silu0(double z) { return z * sigm(z); }
__device__ __forceinline__ double silu1(double z) {
    const double s = sigm(z);
    return s * (1.0 + z * (1.0 - s));
}
__device__ __forceinline__ double silu2(double z) {
    const double s = sigm(z);
    return s * (1.0 - s) * (2.0 + z * (1.0 - 2.0 * s));
}

__device__ __forceinline__ void rbf(double r, double rc, double w, int k, double &phi, double &dphi) {
    const double mu = k * rc / (NR - 1), e = r - mu;
    phi = exp(-e * e / (2.0 * w * w));
    dphi = -e / (w * w) * phi;
}

// The node batch: kNodes nodes per CTA, thread (i, q) = hidden unit i of nodes q and q + 4, so
// that W2 is read once per eight nodes, from shared memory (rows padded to 65: lanes of one
// warp read one column of 32 rows without bank conflicts).  FP64-pipe work of ~3 us for the
// three types; one 64-thread CTA per node, which read W2 from L2 with a 512-byte lane stride,
// took 66 us for the water model's 3 x 1,025 nodes.
constexpr int kNodes = 8, kMlpThreads = 256, kQ = kMlpThreads / H, kPer = kNodes / kQ;
constexpr int kW2Ld = H + 1;

__device__ __forceinline__ void load_w2(const View &m, double *s_w2) {
    for (int k = threadIdx.x; k < H * H; k += kMlpThreads) s_w2[(k / H) * kW2Ld + k % H] = m.W2[k];
}

__global__ void __launch_bounds__(kMlpThreads) k_mlp_nodes(const double *theta, double rc, double w, double *act,
                                                           double *u, double *du) {
    extern __shared__ double s_w2[];   // [H][kW2Ld]
    __shared__ double s_phi[kNodes][NR], s_dphi[kNodes][NR], s_h[kNodes][H], s_dh[kNodes][H];
    __shared__ double s_red[kNodes][2][2];
    const int t = blockIdx.y, g0 = blockIdx.x * kNodes, i = threadIdx.x % H, q = threadIdx.x / H;
    const View m = view(theta, t);
    load_w2(m, s_w2);
    if (threadIdx.x < kNodes * NR) {
        const int n = threadIdx.x / NR, k = threadIdx.x % NR;
        rbf((g0 + n) * (rc / NG), rc, w, k, s_phi[n][k], s_dphi[n][k]);
    }
    __syncthreads();
    double z1[kPer], dz1[kPer], z2[kPer], dz2[kPer];
#pragma unroll
    for (int p = 0; p < kPer; p++) {
        z1[p] = m.b1[i];
        dz1[p] = 0.0;
    }
    for (int k = 0; k < NR; k++) {
        const double wk = m.W1[i * NR + k];
#pragma unroll
        for (int p = 0; p < kPer; p++) {
            z1[p] += wk * s_phi[q + kQ * p][k];
            dz1[p] += wk * s_dphi[q + kQ * p][k];
        }
    }
#pragma unroll
    for (int p = 0; p < kPer; p++) {
        s_h[q + kQ * p][i] = silu0(z1[p]);
        s_dh[q + kQ * p][i] = silu1(z1[p]) * dz1[p];
        z2[p] = m.b2[i];
        dz2[p] = 0.0;
    }
    __syncthreads();
#pragma unroll 8
    for (int j = 0; j < H; j++) {
        const double wj = s_w2[i * kW2Ld + j];
#pragma unroll
        for (int p = 0; p < kPer; p++) {
            z2[p] += wj * s_h[q + kQ * p][j];
            dz2[p] += wj * s_dh[q + kQ * p][j];
        }
    }
    const double w3 = m.w3[i];
#pragma unroll
    for (int p = 0; p < kPer; p++) {
        // y and y' over the 64 units: the unit's two warps, then their sum
        double y = w3 * silu0(z2[p]), dy = w3 * silu1(z2[p]) * dz2[p];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            y += __shfl_xor_sync(0xffffffffu, y, o);
            dy += __shfl_xor_sync(0xffffffffu, dy, o);
        }
        if ((threadIdx.x & 31) == 0) {
            s_red[q + kQ * p][i / 32][0] = y;
            s_red[q + kQ * p][i / 32][1] = dy;
        }
        const int g = g0 + q + kQ * p;
        if (g <= NG) {
            double *a = act + ((size_t)t * (NG + 1) + g) * NA;
            a[i] = z1[p];
            a[H + i] = dz1[p];
            a[2 * H + i] = z2[p];
            a[3 * H + i] = dz2[p];
        }
    }
    __syncthreads();
    const int n = threadIdx.x, g = g0 + n;
    if (n < kNodes && g <= NG) {
        const double y = m.b3[0] + (s_red[n][0][0] + s_red[n][1][0]), dy = s_red[n][0][1] + s_red[n][1][1];
        const double r = g * (rc / NG), x = 3.14159265358979323846 * r / rc;
        const double fc = 0.5 * (cos(x) + 1.0), dfc = -0.5 * 3.14159265358979323846 / rc * sin(x);
        double *a = act + ((size_t)t * (NG + 1) + g) * NA;
        a[4 * H] = y;
        a[4 * H + 1] = dy;
        a[4 * H + 2] = fc;
        a[4 * H + 3] = dfc;
        u[t * (NG + 1) + g] = y * fc;
        du[t * (NG + 1) + g] = dy * fc + y * dfc;
    }
}

// Hermite coefficients of every interval: p(s) = c0 + c1 s + c2 s^2 + c3 s^3, s in [0, 1].
template <typename V4>
__global__ void k_mlp_coef(const double *u, const double *du, double rc, int nt, V4 *tab) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nt * NG) return;
    const int t = k / NG, g = k % NG;
    const double h = rc / NG;
    const double y0 = u[t * (NG + 1) + g], y1 = u[t * (NG + 1) + g + 1];
    const double d0 = du[t * (NG + 1) + g], d1 = du[t * (NG + 1) + g + 1];
    V4 c;
    c.x = y0;
    c.y = h * d0;
    c.z = 3.0 * (y1 - y0) - h * (2.0 * d0 + d1);
    c.w = 2.0 * (y0 - y1) + h * (d0 + d1);
    tab[k] = c;
}

// Coefficient adjoints (summed over the ncopy accumulators in order) -> node value /
// derivative adjoints (the transpose of k_mlp_coef).
__device__ __forceinline__ void sum_copies(const double *cadj, int ncopy, int nt, size_t off, double c[4]) {
    c[0] = c[1] = c[2] = c[3] = 0.0;
    for (int q = 0; q < ncopy; q++) {
        const double *p = cadj + (size_t)q * nt * NG * 4 + off;
        c[0] += p[0];
        c[1] += p[1];
        c[2] += p[2];
        c[3] += p[3];
    }
}

__global__ void k_mlp_adj_nodes(const double *cadj, int ncopy, int nt, double rc, double *au, double *ad) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nt * (NG + 1)) return;
    cadj += (size_t)blockIdx.y * ncopy * nt * NG * 4;   // one replica per grid row
    au += (size_t)blockIdx.y * nt * (NG + 1);
    ad += (size_t)blockIdx.y * nt * (NG + 1);
    const int t = k / (NG + 1), g = k % (NG + 1);
    const double h = rc / NG;
    double a = 0.0, d = 0.0, c[4];
    if (g < NG) {
        sum_copies(cadj, ncopy, nt, ((size_t)t * NG + g) * 4, c);
        a += c[0] - 3.0 * c[2] + 2.0 * c[3];
        d += h * (c[1] - 2.0 * c[2] + c[3]);
    }
    if (g > 0) {
        sum_copies(cadj, ncopy, nt, ((size_t)t * NG + g - 1) * 4, c);
        a += 3.0 * c[2] - 2.0 * c[3];
        d += h * (c[3] - c[2]);
    }
    au[k] = a;
    ad[k] = d;
}

// Backward pass and weight gradients: CTA (chunk c, type t, replica r) takes the nodes of its
// chunk eight at a time -- the node adjoints of z2, z2', z1, z1' (reverse mode through both
// streams; W2 from shared memory), then the outer products, W2's as a 4 x 4 tile and W1's as
// four entries per thread, kept in registers over the chunk -- and writes its partial
// gradient; k_mlp_wgrad_sum adds the chunks in order.  All replicas run in one launch.
// FP64-pipe bound.  One thread per parameter and replica, summing over the nodes with the
// activations formed again for each of the 4,096 W2 entries, took 712 us for the water
// model's three types and 484 us per replica for the diamond's one.
__global__ void __launch_bounds__(kMlpThreads) k_mlp_wgrad(const double *theta, double rc, double w, int nt,
                                                           const double *act, const double *au,
                                                           const double *ad, double *part) {
    extern __shared__ double s_dyn[];   // W2 [H][kW2Ld], then six [kNodes][H] arrays
    double *s_w2 = s_dyn;
    using Row = double[H];
    Row *s_h = (Row *)(s_dyn + H * kW2Ld), *s_dh = s_h + kNodes, *s_z2 = s_dh + kNodes, *s_dz2 = s_z2 + kNodes,
        *s_z1 = s_dz2 + kNodes, *s_dz1 = s_z1 + kNodes;
    __shared__ double s_phi[kNodes][NR], s_dphi[kNodes][NR], s_y[kNodes][2];
    const int C = gridDim.x, c = blockIdx.x, t = blockIdx.y, r = blockIdx.z;
    const int g_lo = (int)((long long)(NG + 1) * c / C), g_hi = (int)((long long)(NG + 1) * (c + 1) / C);
    const int i = threadIdx.x % H, q = threadIdx.x / H;
    const View m = view(theta, t);
    load_w2(m, s_w2);
    const double w3 = m.w3[i];
    const double *aur = au + ((size_t)r * nt + t) * (NG + 1), *adr = ad + ((size_t)r * nt + t) * (NG + 1);
    const int ti = 4 * (threadIdx.x / 16), tj = 4 * (threadIdx.x % 16);   // W2 tile
    const int vi = threadIdx.x / 4, vk = 4 * (threadIdx.x % 4);           // W1 entries
    double aw2[4][4] = {}, aw1[4] = {}, ab1 = 0.0, ab2 = 0.0, aw3 = 0.0, ab3 = 0.0;
    for (int g0 = g_lo; g0 < g_hi; g0 += kNodes) {
        __syncthreads();
        if (threadIdx.x < kNodes * NR) {
            const int n = threadIdx.x / NR, k = threadIdx.x % NR;
            rbf((g0 + n) * (rc / NG), rc, w, k, s_phi[n][k], s_dphi[n][k]);
        }
        double s1[kPer], s2[kPer];   // silu'(z1), silu''(z1) z1'
#pragma unroll
        for (int p = 0; p < kPer; p++) {
            const int n = q + kQ * p, g = g0 + n;
            // nodes past the chunk: zero adjoints, finite activations
            const bool in = g < g_hi;
            const double *a = act + ((size_t)t * (NG + 1) + (in ? g : g_lo)) * NA;
            const double fc = a[4 * H + 2], dfc = a[4 * H + 3];
            const double un = in ? aur[g] : 0.0, dn = in ? adr[g] : 0.0;
            // u = y fc, u' = y' fc + y fc'
            const double yb = un * fc + dn * dfc, dyb = dn * fc;
            const double z1 = a[i], dz1 = a[H + i], z2 = a[2 * H + i], dz2 = a[3 * H + i];
            const double f2 = silu1(z2);
            s1[p] = silu1(z1);
            s2[p] = silu2(z1) * dz1;
            s_h[n][i] = silu0(z1);
            s_dh[n][i] = s1[p] * dz1;
            const double h2b = yb * w3, dh2b = dyb * w3;
            const double z2b = h2b * f2 + dh2b * silu2(z2) * dz2;
            s_z2[n][i] = z2b;
            s_dz2[n][i] = dh2b * f2;
            ab2 += z2b;
            aw3 += yb * silu0(z2) + dyb * f2 * dz2;
            if (i == 0) ab3 += yb;
        }
        __syncthreads();
        double h1b[kPer], dh1b[kPer];
#pragma unroll
        for (int p = 0; p < kPer; p++) h1b[p] = dh1b[p] = 0.0;
#pragma unroll 8
        for (int k = 0; k < H; k++) {
            const double wk = s_w2[k * kW2Ld + i];
#pragma unroll
            for (int p = 0; p < kPer; p++) {
                h1b[p] += wk * s_z2[q + kQ * p][k];
                dh1b[p] += wk * s_dz2[q + kQ * p][k];
            }
        }
#pragma unroll
        for (int p = 0; p < kPer; p++) {
            const double z1b = h1b[p] * s1[p] + dh1b[p] * s2[p];
            s_z1[q + kQ * p][i] = z1b;
            s_dz1[q + kQ * p][i] = dh1b[p] * s1[p];
            ab1 += z1b;
        }
        __syncthreads();
        for (int n = 0; n < kNodes; n++) {
            double zb[4], db[4], hv[4], dv[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                zb[k] = s_z2[n][ti + k];
                db[k] = s_dz2[n][ti + k];
                hv[k] = s_h[n][tj + k];
                dv[k] = s_dh[n][tj + k];
            }
#pragma unroll
            for (int x = 0; x < 4; x++)
#pragma unroll
                for (int y = 0; y < 4; y++) aw2[x][y] += zb[x] * hv[y] + db[x] * dv[y];
            const double z1b = s_z1[n][vi], dz1b = s_dz1[n][vi];
#pragma unroll
            for (int k = 0; k < 4; k++) aw1[k] += z1b * s_phi[n][vk + k] + dz1b * s_dphi[n][vk + k];
        }
    }
    double *out = part + (((size_t)r * nt + t) * C + c) * MLP_PER_TYPE;
#pragma unroll
    for (int k = 0; k < 4; k++) out[vi * NR + vk + k] = aw1[k];
    double *o2 = out + H * NR + H;
#pragma unroll
    for (int x = 0; x < 4; x++)
#pragma unroll
        for (int y = 0; y < 4; y++) o2[(ti + x) * H + tj + y] = aw2[x][y];
    // the four threads of a unit, in order
    __syncthreads();
    s_h[q][i] = ab1;
    s_dh[q][i] = ab2;
    s_z2[q][i] = aw3;
    if (i == 0) s_y[q][0] = ab3;
    __syncthreads();
    if (threadIdx.x < H) {
        double b1 = 0.0, b2 = 0.0, v3 = 0.0;
        for (int k = 0; k < kQ; k++) {
            b1 += s_h[k][i];
            b2 += s_dh[k][i];
            v3 += s_z2[k][i];
        }
        out[H * NR + i] = b1;
        o2[H * H + i] = b2;
        o2[H * H + H + i] = v3;
        if (i == 0) o2[H * H + 2 * H] = s_y[0][0] + s_y[1][0] + s_y[2][0] + s_y[3][0];
    }
}

// dtheta of (replica, type) = blockIdx.y: the chunks' partials in order.
__global__ void k_mlp_wgrad_sum(int C, const double *part, double *dtheta) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= MLP_PER_TYPE) return;
    const double *p = part + (size_t)blockIdx.y * C * MLP_PER_TYPE + k;
    double s = 0.0;
    for (int c = 0; c < C; c++) s += p[(size_t)c * MLP_PER_TYPE];
    dtheta[(size_t)blockIdx.y * MLP_PER_TYPE + k] = s;
}

// Scratch of the FP64 network: activations, the weight-gradient partials of one launch (two
// CTAs per SM), the node arrays u, du, au, ad and the node adjoints of a batch of replicas.
constexpr int kWgradCtas = 2 * kSMs, kWgradReps = 16;
constexpr size_t kActLen = (size_t)MLP_NT * (NG + 1) * NA, kPartLen = (size_t)kWgradCtas * MLP_PER_TYPE,
                 kNodeLen = (size_t)MLP_NT * (NG + 1);
constexpr size_t kNodesSmem = sizeof(double) * H * kW2Ld,
                 kWgradSmem = sizeof(double) * (H * kW2Ld + 6 * kNodes * H);

}  // namespace

// scratch layout: act | partials | u, du, au, ad [NT][NG+1] | au, ad of kWgradReps replicas
size_t mlp_scratch_doubles() { return kActLen + kPartLen + 4 * kNodeLen + 2 * kWgradReps * kNodeLen; }

double *mlp_scratch_nodes(double *scratch, int which) {
    return scratch + kActLen + kPartLen + (size_t)which * kNodeLen;   // 0: u, 1: du, 2: au, 3: ad
}

cudaError_t launch_mlp_table(int prec, const double *theta, double rc, double *scratch, void *tab,
                             cudaStream_t st, int nt, double w) {
    if (nt < 1 || nt > MLP_NT) return cudaErrorInvalidValue;
    k_mlp_nodes<<<dim3((NG + kNodes) / kNodes, nt), kMlpThreads, kNodesSmem, st>>>(
        theta, rc, w, scratch, mlp_scratch_nodes(scratch, 0), mlp_scratch_nodes(scratch, 1));
    return launch_mlp_table_from_nodes(prec, scratch, rc, tab, st, nt);
}

// The tensor-core path (rs_mlp_tc.cu) shares the node arrays of this scratch: the interval
// table from node values computed elsewhere, and the node adjoints alone.
cudaError_t launch_mlp_table_from_nodes(int prec, double *scratch, double rc, void *tab, cudaStream_t st,
                                        int nt) {
    if (nt < 1 || nt > MLP_NT) return cudaErrorInvalidValue;
    const double *u = mlp_scratch_nodes(scratch, 0), *du = mlp_scratch_nodes(scratch, 1);
    const int n = nt * NG;
    if (prec == 1)
        k_mlp_coef<float4><<<(n + 255) / 256, 256, 0, st>>>(u, du, rc, nt, (float4 *)tab);
    else
        k_mlp_coef<double4><<<(n + 255) / 256, 256, 0, st>>>(u, du, rc, nt, (double4 *)tab);
    return cudaGetLastError();
}

cudaError_t launch_mlp_node_adjoints(const double *cadj, int ncopy, double rc, double *scratch, cudaStream_t st,
                                     int nt) {
    if (nt < 1 || nt > MLP_NT) return cudaErrorInvalidValue;
    const int nn = nt * (NG + 1);
    k_mlp_adj_nodes<<<(nn + 255) / 256, 256, 0, st>>>(cadj, ncopy, nt, rc, mlp_scratch_nodes(scratch, 2),
                                                        mlp_scratch_nodes(scratch, 3));
    return cudaGetLastError();
}

// Chunks per (replica, type): as many as give every SM two CTAs, at most one per node batch.
cudaError_t launch_mlp_backprop(const double *theta, double rc, const double *cadj, int R, int ncopy,
                                double *scratch, double *dtheta, cudaStream_t st, int *n_kernels, int nt, double w) {
    if (nt < 1 || nt > MLP_NT) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_mlp_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWgradSmem);
    if (e != cudaSuccess) return e;
    double *part = scratch + kActLen, *au = mlp_scratch_nodes(scratch, 4);
    const int nn = nt * (NG + 1);
    *n_kernels = 0;
    for (int r0 = 0; r0 < R; r0 += kWgradReps) {
        const int rb = std::min(kWgradReps, R - r0);
        const int C = std::min((NG + kNodes) / kNodes, kWgradCtas / (rb * nt));
        double *ad = au + (size_t)rb * nn;
        k_mlp_adj_nodes<<<dim3((nn + 255) / 256, rb), 256, 0, st>>>(cadj + (size_t)r0 * ncopy * nt * NG * 4, ncopy, nt,
                                                                    rc, au, ad);
        k_mlp_wgrad<<<dim3(C, nt, rb), kMlpThreads, kWgradSmem, st>>>(theta, rc, w, nt, scratch, au, ad, part);
        k_mlp_wgrad_sum<<<dim3((MLP_PER_TYPE + 255) / 256, rb * nt), 256, 0, st>>>(
            C, part, dtheta + (size_t)r0 * nt * MLP_PER_TYPE);
        *n_kernels += 3;
    }
    return cudaGetLastError();
}

}  // namespace rs
