// fem_sensitivity.cu -- shape sensitivities of the strain energy through the
// level-set coefficients (adjoint method).
//
//   dQ/dp = sum_v G[v] dt_v/dp,   G[v] = d/dt_v ( Q(u, t) - lambda^T R(u, t) ),
//   K^T lambda = dQ/du,
//
// where t_v is the edge coordinate of intersection vertex v
// (x_v = x_p0 + t_v (x_p1 - x_p0)).  The reference assembles dR/dp by finite
// differences of the IG vertex coordinates (IWG::select_dRdp_FD_geometry_bulk,
// FEM/INT/src/IWG/cl_FEM_IWG.cpp:2997-3154, plus the cluster-measure terms
// :3827-3924) and contracts with the adjoint in Interpolation_Element::
// compute_dQIdp_explicit_implicit (FEM/INT/src/ELEM/cl_FEM_Interpolation_
// Element.cpp:820-948).  Here the derivative is exact and taken in reverse:
// per integration cell (TET4) and interface facet (TRI3) the integrand and its
// spatial gradient at every point, from which the derivative by each vertex is
// a sum over the points; the contraction with u and lambda happens inside the
// kernel:
//
//   tet     F = sum_q w detJ (1/2 sigma(u):eps(u) - sigma(u):eps(lambda))
//   facet   -lambda^T R_interface = -( w_L A + w_F B + gamma C ),
//           A = sum_q w* (-[lambda].t_L(u) + beta t_L(lambda).[u]),  B likewise
//           with t_F, C = sum_q w* [lambda].[u]  (IWG_Isotropic_Struc_Linear_
//           Interface residual contracted with lambda), and the SP_Nitsche_
//           Interface weights / gamma differentiated through the cluster
//           volumes (the cut clusters' tets) and the interface measure.
// Rectangular IP cells: xi = -1 + 2 (x - X0) / (X6 - X0).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "fem_internal.hpp"

namespace fem {
namespace {

// A trilinear field of a rectangular HEX8 cell (nodal values f_a, shape
// functions N_a = (1 + s_x xi)(1 + s_y eta)(1 + s_z zeta) / 8) written as a
// polynomial in the physical offsets (x, y, z) from the cell centre:
//   f = k0 + k1 x + k2 y + k3 z + k4 xy + k5 yz + k6 xz + k7 xyz,
// k_m = (1/8) sum_a f_a prod_{d in m} s_d(a) / prod_{d in m} jd_d  (jd the half
// edge lengths).  Its gradient needs only the pair products:
//   df/dx = k1 + k4 y + k6 z + k7 yz,  df/dy = k2 + k4 x + k5 z + k7 xz,
//   df/dz = k3 + k6 x + k5 y + k7 xy.
// Monomial m -> the set of coordinates it contains (bit d for coordinate d).
__device__ __forceinline__ int monomial_mask(int m) {
    return m < 4 ? (m == 0 ? 0 : 1 << (m - 1)) : (m == 4 ? 3 : m == 5 ? 6 : m == 6 ? 5 : 7);
}
// coefficient r = comp * 8 + m of the field with nodal values f[comp * 8 + a]
// on the cell X[8][3] (node 0 and node 6 opposite corners)
__device__ double monomial_coefficient(const double* f, const double* X, int r) {
    const int fl = r >> 3, mask = monomial_mask(r & 7);
    double c = 0.0;
    for (int a = 0; a < 8; ++a) {
        const int sx = ((a & 3) == 1 || (a & 3) == 2) ? 1 : -1;
        const int sy = ((a & 3) >= 2) ? 1 : -1;
        const int sz = a >= 4 ? 1 : -1;
        const int sg = ((mask & 1) ? sx : 1) * ((mask & 2) ? sy : 1) * ((mask & 4) ? sz : 1);
        c += sg > 0 ? f[fl * 8 + a] : -f[fl * 8 + a];
    }
    double den = 8.0;
    for (int d = 0; d < 3; ++d)
        if (mask & (1 << d)) den *= 0.5 * (X[18 + d] - X[d]);
    return c / den;
}

// One component of such a field at the offsets x (pr = xy, yz, xz): gradient
// g[d] and mixed second derivatives h = (xy, yz, xz); the pure ones vanish.
__device__ __forceinline__ void mono_grad(const double* __restrict__ c, const double x[3], const double pr[3],
                                          double g[3], double h[3]) {
    const double c1 = c[1], c2 = c[2], c3 = c[3], c4 = c[4], c5 = c[5], c6 = c[6], c7 = c[7];
    g[0] = fma(c7, pr[1], fma(c6, x[2], fma(c4, x[1], c1)));
    g[1] = fma(c7, pr[2], fma(c5, x[2], fma(c4, x[0], c2)));
    g[2] = fma(c7, pr[0], fma(c5, x[1], fma(c6, x[0], c3)));
    h[0] = fma(c7, x[2], c4);
    h[1] = fma(c7, x[0], c5);
    h[2] = fma(c7, x[1], c6);
}
// its value, given g[0]: k0 + k2 y + k3 z + k5 yz + x df/dx
__device__ __forceinline__ double mono_value(const double* __restrict__ c, const double x[3], const double pr[3],
                                             double g0) {
    return fma(x[0], g0, fma(c[5], pr[1], fma(c[3], x[2], fma(c[2], x[1], c[0]))));
}

// sigma = lam tr(G) I + mu (G + G^T) of a displacement gradient G[f][i] = du_f/dx_i,
// as xx, yy, zz, xy, yz, xz
__device__ __forceinline__ void stress(const double G[3][3], double lam, double mu, double S[6]) {
    const double tr = lam * (G[0][0] + G[1][1] + G[2][2]), m2 = 2.0 * mu;
    for (int i = 0; i < 3; ++i) S[i] = fma(m2, G[i][i], tr);
    S[3] = mu * (G[0][1] + G[1][0]);
    S[4] = mu * (G[1][2] + G[2][1]);
    S[5] = mu * (G[0][2] + G[2][0]);
}
__device__ constexpr int sym(int i, int j) { return i == j ? i : i + j == 1 ? 3 : i + j == 3 ? 4 : 5; }

// o[d] += sum_fj W_fj dG_fj/dx_d with a symmetric W and dG_fj/dx_d = h_f(j, d) (0 for j = d)
__device__ __forceinline__ void push_gradient(const double W[6], const double H[3][3], double o[3]) {
    for (int f = 0; f < 3; ++f) {
        const double w0 = W[sym(f, 0)], w1 = W[sym(f, 1)], w2 = W[sym(f, 2)];
        o[0] = fma(w1, H[f][0], fma(w2, H[f][2], o[0]));
        o[1] = fma(w0, H[f][0], fma(w2, H[f][1], o[1]));
        o[2] = fma(w0, H[f][2], fma(w1, H[f][1], o[2]));
    }
}
__device__ __forceinline__ void cross(const double a[3], const double b[3], double c[3]) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}
__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
    return fma(a[2], b[2], fma(a[1], b[1], a[0] * b[0]));
}

struct AdjArgs {
    // vertex table
    const int32_t* vkind;
    const int32_t* vpar;  // [nv][8]
    const double* vx;     // [nv][3]
    double* G;            // [nv]
    // adof vectors
    const double* u;
    const double* lam;
    int64_t nu;
};

struct CutSetDev {
    int64_t neq;
    const double* xe;      // [neq][8][3]
    const double* E;
    const int32_t* nb;
    const int32_t* bases;  // [neq][W]
    const double* T;       // [neq][8][W]
    int W;
    double lam_c, mu_c;
    const int64_t* ig_off;
    const int32_t* vid;    // [ig][4]
    const double* gp;      // TET rule points [ngp][3]
    const double* gw;
    int ngp;
};

__device__ void pdof_values(const double* T, const int32_t* bases, int nb, int W, const double* ua, int64_t nu,
                            double* out /*[24]*/, int tid, int nt) {
    for (int r = tid; r < 24; r += nt) {
        const int f = r / 8, a = r % 8;
        double v = 0.0;
        if (ua)
            for (int j = 0; j < nb; ++j) {
                const double t = T[a * W + j];
                if (t != 0.0) v = fma(t, ua[f * nu + bases[j]], v);
            }
        out[r] = v;
    }
}

// position of a vertex, and (moving vertices: intersections) dx/dt; returns whether it moves
__device__ __forceinline__ bool vertex(const AdjArgs& A, int32_t v, double x[3], double dx[3]) {
    const bool moving = A.vkind[v] == 3;
    const int32_t p0 = moving ? A.vpar[(int64_t)v * 8] : v, p1 = moving ? A.vpar[(int64_t)v * 8 + 1] : v;
    for (int d = 0; d < 3; ++d) {
        x[d] = A.vx[(int64_t)v * 3 + d];
        dx[d] = A.vx[(int64_t)p1 * 3 + d] - A.vx[(int64_t)p0 * 3 + d];
    }
    return moving;
}

// signed volume of a TET4 (vertices X, edges from vertex 2) and its gradient by every vertex
__device__ __forceinline__ double tet_volume(const double X[4][3], double dV[4][3]) {
    double a[3], b[3], c[3];
    for (int d = 0; d < 3; ++d) {
        a[d] = X[0][d] - X[2][d];
        b[d] = X[1][d] - X[2][d];
        c[d] = X[3][d] - X[2][d];
    }
    cross(b, c, dV[0]);
    cross(c, a, dV[1]);
    cross(a, b, dV[3]);
    const double v = dot3(a, dV[0]);
    for (int d = 0; d < 3; ++d) {
        for (int k : {0, 1, 3}) dV[k][d] *= 1.0 / 6.0;
        dV[2][d] = -(dV[0][d] + dV[1][d] + dV[3][d]);
    }
    return v * (1.0 / 6.0);
}

// Cut clusters: F = detJ Phi, Phi = sum_q w phi(x_q), phi = 1/2 sigma(u):eps(u) -
// sigma(u):eps(lambda), over every integration cell.  Then
//   dF/dX_k = Phi ddetJ/dX_k + detJ sum_q w N_k(q) grad phi(x_q),
// added along dx/dt to G of the moving vertices.  The gradient of phi costs 60
// FMAs on top of the 110 of phi, whatever the number of moving vertices, where
// dual numbers multiplied the whole integrand by 1 + that number.  One thread
// per integration cell with a moving vertex (listed in `cells`): the cells of a
// cluster (1 to about 100) rarely fill whole warps, and on this GPU an FP64 warp
// instruction costs the pipe the same however few of its lanes are active.  (A
// lane per point, summed by shuffles, was slower: the FP64 pipe binds, not the
// number of warps.)  The cluster's field polynomials are formed once per cluster
// first (adjoint_cluster_values), which also writes every cell's cluster index.
// Measured, 156 k moving cells (44^3): 700 -> 260 us with six CTAs per SM (168
// registers; at 246 registers and four CTAs 274 us).
__global__ void adjoint_cluster_values(AdjArgs A, CutSetDev S, double* UL /*[neq][48]*/, int32_t* cell_cluster) {
    const int64_t e = blockIdx.x;
    if (e >= S.neq) return;
    __shared__ double nod[48];
    for (int64_t g = S.ig_off[e] + threadIdx.x; g < S.ig_off[e + 1]; g += blockDim.x) cell_cluster[g] = (int32_t)e;
    const int nb = S.nb[e];
    pdof_values(S.T + e * 8 * S.W, S.bases + e * S.W, nb, S.W, A.u, A.nu, nod, threadIdx.x, blockDim.x);
    pdof_values(S.T + e * 8 * S.W, S.bases + e * S.W, nb, S.W, A.lam, A.nu, nod + 24, threadIdx.x, blockDim.x);
    __syncthreads();
    for (int r = threadIdx.x; r < 48; r += blockDim.x)
        UL[e * 48 + r] = monomial_coefficient(nod + (r / 24) * 24, S.xe + e * 24, r % 24);
}

__global__ void __launch_bounds__(64, 6) adjoint_tets(AdjArgs A, CutSetDev S, const double* __restrict__ UL,
                                                   const int32_t* __restrict__ cell_cluster,
                                                   const int32_t* __restrict__ cells, int64_t ncells) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ncells) return;
    const int64_t g = cells[i], e = cell_cluster[g];
    const double* X = S.xe + e * 24;
    const double* U = UL + e * 48;
    const double lam = S.E[e] * S.lam_c, mu = S.E[e] * S.mu_c;
    double Xv[4][3], R[4][3] = {};  // vertex offsets from the cell centre
    for (int d = 0; d < 3; ++d) {
        const double xc = 0.5 * (X[18 + d] + X[d]);
        for (int k = 0; k < 4; ++k) Xv[k][d] = A.vx[(int64_t)S.vid[g * 4 + k] * 3 + d] - xc;
    }
    double Phi = 0.0;
#pragma unroll 1
    for (int q = 0; q < S.ngp; ++q) {
        asm volatile("" : "+l"(U));  // keeps the 48 coefficients out of registers
        const double* L = U + 24;
        const double z0 = S.gp[q * 3], z1 = S.gp[q * 3 + 1], z2 = S.gp[q * 3 + 2], w = S.gw[q];
        const double N[4] = {z0, z1, 1.0 - z0 - z1 - z2, z2};
        double x[3];
        for (int d = 0; d < 3; ++d)
            x[d] = fma(N[3], Xv[3][d], fma(N[2], Xv[2][d], fma(N[1], Xv[1][d], N[0] * Xv[0][d])));
        const double pr[3] = {x[0] * x[1], x[1] * x[2], x[0] * x[2]};
        double Gu[3][3], Hu[3][3], Gl[3][3], Hl[3][3], Su[6], Sl[6];
        for (int f = 0; f < 3; ++f) {
            mono_grad(U + f * 8, x, pr, Gu[f], Hu[f]);
            mono_grad(L + f * 8, x, pr, Gl[f], Hl[f]);
        }
        stress(Gu, lam, mu, Su);
        stress(Gl, lam, mu, Sl);
        double phi = 0.0, gr[3] = {0.0, 0.0, 0.0};
        for (int f = 0; f < 3; ++f)
            for (int j = 0; j < 3; ++j) phi = fma(Su[sym(f, j)], fma(0.5, Gu[f][j], -Gl[f][j]), phi);
        Phi = fma(w, phi, Phi);
        // dphi = (sigma(u) - sigma(lambda)) : dGu - sigma(u) : dGl
        for (int m = 0; m < 6; ++m) {
            Sl[m] = w * (Su[m] - Sl[m]);
            Su[m] *= -w;
        }
        push_gradient(Sl, Hu, gr);
        push_gradient(Su, Hl, gr);
        for (int k = 0; k < 4; ++k)
            for (int d = 0; d < 3; ++d) R[k][d] = fma(N[k], gr[d], R[k][d]);
    }
    double dx[4][3], dV[4][3];
    bool mv[4];
    for (int k = 0; k < 4; ++k) mv[k] = vertex(A, S.vid[g * 4 + k], Xv[k], dx[k]);
    const double detJ = tet_volume(Xv, dV);
    // skipped points (detJ < -1e-6) contribute nothing (cl_FEM_Element_Bulk.cpp:164)
    if (detJ < -1.0e-6) return;
    for (int k = 0; k < 4; ++k)
        if (mv[k]) atomicAdd(A.G + S.vid[g * 4 + k], fma(Phi, dot3(dV[k], dx[k]), detJ * dot3(R[k], dx[k])));
}

struct IfSetDev {
    int64_t neq;
    int beta_sym;
    double alpha, lam_c, mu_c;
    const double* xe;      // [neq][2][8][3]
    const double* E;
    const double* EF;
    const int32_t* nb;     // [neq][2]
    const int32_t* bases;  // [neq][2][W]
    const double* T;       // [neq][2][8][W]
    int W;
    const int64_t* fc_off;
    const int32_t* vid;    // [facet][3]
    const double* gp;      // TRI rule [ngp][2]
    const double* gw;
    int ngp;
    const double* vol;     // [neq][2]
    const int32_t* link;   // [neq][4]: leader (set, eq), follower (set, eq) among the cut sets
};

// The interface sum, flattened like the cut cells (a cluster has a few facets).
// With the facet's vector area cr / 2 = (x0 - x2) x (x1 - x2) / 2, the mean
// stress s(.) = w_L sigma_L + w_F sigma_F and the jumps [.], the facet's share of
// w_L A + w_F B + gamma C is
//   1/2 sum_q w ( cr . (beta s(lambda) [u] - s(u) [lambda]) + gamma |cr| [lambda].[u] ),
// with no unit normal in it.  The weights depend on the cluster volumes only and
// gamma on the volumes and the cluster's area, so with the area summed first the
// derivative is one reverse sweep.  Jumps and stresses are linear in the fields,
// so each cluster combines the sides' polynomials beforehand, about the leader's
// centre: the jump u_L - u_F, the mean w_L E_L u_L + w_F E_F u_F (its unit-modulus
// stress is s) and the difference E_L u_L - E_F u_F (for A - B), of u and lambda.
//   iface_cluster_values   per cluster: the six polynomials, area, weights and
//                          gamma, each facet's cluster index;
//   iface_facets           one thread per facet: A - B and C into the cluster
//                          sums, per vertex the derivative at fixed gamma and
//                          that of the area;
//   iface_apply            one thread per facet: dF/dt with the cluster's C;
//   iface_volumes          one thread per (cluster, side, cell of the linked
//                          cut cluster): dF/dV through w_L, w_F and gamma.
// Measured for 43 k facets of 7 points (44^3): iface_facets 1,167 -> 300 us.
// The whole call with the chain to the coefficients takes 774 us (2,620 before).
constexpr int kIfParts = 6;     // per vertex: derivative at fixed gamma, of the area
constexpr int kIfFields = 144;  // [jump, mean, difference][u, lambda][3][8]
constexpr int kIfSums = 8;      // A - B, C, |G|, gamma, w_L, w_F, 1 / (V_L/E_L + V_F/E_F)

// k about another origin: p(x + d)
__device__ void shift_polynomial(double* k, const double d[3]) {
    const double xy = d[0] * d[1], yz = d[1] * d[2], xz = d[0] * d[2], k7 = k[7];
    k[0] += k[1] * d[0] + k[2] * d[1] + k[3] * d[2] + k[4] * xy + k[5] * yz + k[6] * xz + k7 * xy * d[2];
    k[1] += k[4] * d[1] + k[6] * d[2] + k7 * yz;
    k[2] += k[4] * d[0] + k[5] * d[2] + k7 * xz;
    k[3] += k[6] * d[0] + k[5] * d[1] + k7 * xy;
    k[4] += k7 * d[2];
    k[5] += k7 * d[0];
    k[6] += k7 * d[1];
}

__global__ void iface_cluster_values(AdjArgs A, IfSetDev S, double* fields /*[neq][kIfFields]*/,
                                     int32_t* facet_cluster, double* sums /*[neq][kIfSums]*/) {
    const int64_t e = blockIdx.x;
    if (e >= S.neq) return;
    __shared__ double nod[96], pol[96], part[2], wt[2];
    double wsum = 0.0, area = 0.0;
    for (int q = 0; q < S.ngp; ++q) wsum += S.gw[q];
    for (int64_t f = S.fc_off[e] + threadIdx.x; f < S.fc_off[e + 1]; f += blockDim.x) {
        facet_cluster[f] = (int32_t)e;
        double a[3], b[3], c[3];
        for (int d = 0; d < 3; ++d) {
            const double o = A.vx[(int64_t)S.vid[f * 3 + 2] * 3 + d];
            a[d] = A.vx[(int64_t)S.vid[f * 3] * 3 + d] - o;
            b[d] = A.vx[(int64_t)S.vid[f * 3 + 1] * 3 + d] - o;
        }
        cross(a, b, c);
        area = fma(0.5 * wsum, sqrt(dot3(c, c)), area);
    }
    for (int o = 16; o > 0; o >>= 1) area += __shfl_xor_sync(0xffffffffu, area, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = area;
    for (int s = 0; s < 2; ++s) {
        const int nb = S.nb[2 * e + s];
        pdof_values(S.T + (e * 2 + s) * 8 * S.W, S.bases + (e * 2 + s) * S.W, nb, S.W, A.u, A.nu, nod + 24 * s,
                    threadIdx.x, blockDim.x);
        pdof_values(S.T + (e * 2 + s) * 8 * S.W, S.bases + (e * 2 + s) * S.W, nb, S.W, A.lam, A.nu,
                    nod + 48 + 24 * s, threadIdx.x, blockDim.x);
    }
    __syncthreads();
    const double* X = S.xe + e * 48;
    // [u side 0, u side 1, lambda side 0, lambda side 1], each on its side's cell
    for (int r = threadIdx.x; r < 96; r += blockDim.x)
        pol[r] = monomial_coefficient(nod + (r / 24) * 24, X + 24 * ((r / 24) & 1), r % 24);
    if (threadIdx.x == 0) {
        const double vl = S.vol[2 * e] / S.E[e], vf = S.vol[2 * e + 1] / S.EF[e], inv = 1.0 / (vl + vf);
        double* q = sums + e * kIfSums;
        q[0] = q[1] = 0.0;
        q[2] = part[0] + part[1];
        q[3] = 2.0 * S.alpha * q[2] * inv;
        q[4] = vl * inv;
        q[5] = vf * inv;
        q[6] = inv;
        wt[0] = q[4] * S.E[e];
        wt[1] = q[5] * S.EF[e];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        // the follower's polynomials about the leader's centre
        const int fl = threadIdx.x / 3;
        double d[3];
        for (int i = 0; i < 3; ++i) d[i] = 0.5 * (X[18 + i] + X[i]) - 0.5 * (X[42 + i] + X[24 + i]);
        if (d[0] != 0.0 || d[1] != 0.0 || d[2] != 0.0) shift_polynomial(pol + fl * 48 + 24 + threadIdx.x % 3 * 8, d);
    }
    __syncthreads();
    for (int r = threadIdx.x; r < kIfFields; r += blockDim.x) {
        const int kind = r / 48, at = (r / 24 & 1) * 48 + r % 24;
        const double p0 = pol[at], p1 = pol[at + 24];
        fields[e * kIfFields + r] = kind == 0   ? p0 - p1
                                    : kind == 1 ? fma(wt[0], p0, wt[1] * p1)
                                                : S.E[e] * p0 - S.EF[e] * p1;
    }
}

__global__ void __launch_bounds__(64, 6) iface_facets(AdjArgs A, IfSetDev S, const double* __restrict__ fields,
                                                   const int32_t* __restrict__ facet_cluster, int64_t nfacets,
                                                   double* sums, double* parts /*[nf][kIfParts]*/) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nfacets) return;
    const int64_t e = facet_cluster[f];
    const double* X = S.xe + e * 48;
    const double* P = fields + e * kIfFields;
    const double beta = S.beta_sym ? -1.0 : 1.0, gamma = sums[e * kIfSums + 3];
    double Xv[3][3], a[3], b[3], cr[3];
    for (int k = 0; k < 3; ++k)
        for (int d = 0; d < 3; ++d) Xv[k][d] = A.vx[(int64_t)S.vid[f * 3 + k] * 3 + d] - 0.5 * (X[18 + d] + X[d]);
    for (int d = 0; d < 3; ++d) {
        a[d] = Xv[0][d] - Xv[2][d];
        b[d] = Xv[1][d] - Xv[2][d];
    }
    cross(a, b, cr);
    const double nn = sqrt(dot3(cr, cr));
    double* out = parts + f * kIfParts;
    if (!(nn > 0.0)) {
        for (int k = 0; k < kIfParts; ++k) out[k] = 0.0;
        return;
    }
    const double gn = gamma * nn;
    double V[3] = {0.0, 0.0, 0.0}, cs = 0.0, ab = 0.0, wsum = 0.0;  // sums of v, [lambda].[u], A - B, w
    double R[3][3] = {};
#pragma unroll 1
    for (int q = 0; q < S.ngp; ++q) {
        // the coefficients stay in L1: hoisted out of the loop, all 144 spill
        asm volatile("" : "+l"(P));
        const double z0 = S.gp[q * 2], z1 = S.gp[q * 2 + 1], w = S.gw[q];
        const double N[3] = {z0, z1, 1.0 - z0 - z1};
        double x[3], gr[3] = {0.0, 0.0, 0.0}, jv[2][3], dj[2][3][3], t[2][3], v[3] = {0.0, 0.0, 0.0};
        for (int d = 0; d < 3; ++d) x[d] = fma(N[2], Xv[2][d], fma(N[1], Xv[1][d], N[0] * Xv[0][d]));
        const double pr[3] = {x[0] * x[1], x[1] * x[2], x[0] * x[2]};
#pragma unroll
        for (int fl = 0; fl < 2; ++fl)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                double h[3];
                mono_grad(P + fl * 24 + i * 8, x, pr, dj[fl][i], h);
                jv[fl][i] = mono_value(P + fl * 24 + i * 8, x, pr, dj[fl][i][0]);
            }
        // v = beta s(lambda) [u] - s(u) [lambda], t = s(.) cr, and the gradient of
        // cr . v through the stresses: (sigma(G) cr) . j = G : W with
        // W = lam (cr . j) I + mu (cr j^T + j cr^T)
        double da = 0.0;
#pragma unroll
        for (int fl = 0; fl < 2; ++fl) {
            const double sg = fl ? beta : -1.0;
            const double* j = jv[1 - fl];
            double G[3][3], H[3][3], Sg[6], W[6];
            for (int i = 0; i < 3; ++i) mono_grad(P + 48 + fl * 24 + i * 8, x, pr, G[i], H[i]);
            stress(G, S.lam_c, S.mu_c, Sg);
            const double tr = S.lam_c * sg * dot3(cr, j), m = S.mu_c * sg;
            const double mj[3] = {m * j[0], m * j[1], m * j[2]};
            for (int k = 0; k < 3; ++k) {
                W[k] = fma(2.0 * cr[k], mj[k], tr);
                const double row[3] = {Sg[sym(k, 0)], Sg[sym(k, 1)], Sg[sym(k, 2)]};
                t[fl][k] = dot3(row, cr);
                v[k] = fma(sg, dot3(row, j), v[k]);
            }
            W[3] = fma(cr[0], mj[1], cr[1] * mj[0]);
            W[4] = fma(cr[1], mj[2], cr[2] * mj[1]);
            W[5] = fma(cr[0], mj[2], cr[2] * mj[0]);
            push_gradient(W, H, gr);
            // the share of A - B: the same product with the difference field
            for (int i = 0; i < 3; ++i) {
                mono_grad(P + 96 + fl * 24 + i * 8, x, pr, G[i], H[i]);
                for (int k = 0; k < 3; ++k) da = fma(W[sym(i, k)], G[i][k], da);
            }
        }
        ab = fma(w, da, ab);
        cs = fma(w, dot3(jv[0], jv[1]), cs);
        wsum += w;
        for (int i = 0; i < 3; ++i) {
            V[i] = fma(w, v[i], V[i]);
            // the gradient through [u] and [lambda]
            const double au = fma(gn, jv[1][i], beta * t[1][i]), al = fma(gn, jv[0][i], -t[0][i]);
            for (int d = 0; d < 3; ++d) gr[d] = fma(au, dj[0][i][d], fma(al, dj[1][i][d], gr[d]));
        }
        for (int k = 0; k < 3; ++k) {
            const double wn = 0.5 * w * N[k];
            for (int d = 0; d < 3; ++d) R[k][d] = fma(wn, gr[d], R[k][d]);
        }
    }
    atomicAdd(sums + e * kIfSums, 0.5 * ab);
    atomicAdd(sums + e * kIfSums + 1, 0.5 * nn * cs);
    // by the vector area: Y = (V + gamma cs cr / |cr|) / 2, the area's own cr / (2 |cr|)
    double Y[3], Z[3], d0[3], d1[3], dx[3][3];
    bool mv[3];
    for (int k = 0; k < 3; ++k) mv[k] = vertex(A, S.vid[f * 3 + k], d0, dx[k]);
    const double in = 1.0 / nn;
    for (int i = 0; i < 3; ++i) {
        Z[i] = 0.5 * wsum * cr[i] * in;
        Y[i] = 0.5 * fma(gamma * cs, cr[i] * in, V[i]);
    }
    for (int pass = 0; pass < 2; ++pass) {
        const double* y = pass ? Z : Y;
        cross(b, y, d0);
        cross(y, a, d1);
        for (int k = 0; k < 3; ++k) {
            double s = 0.0;
            for (int d = 0; d < 3; ++d) {
                const double g = k == 0 ? d0[d] : k == 1 ? d1[d] : -(d0[d] + d1[d]);
                s = fma(pass ? g : g + R[k][d], dx[k][d], s);
            }
            // a vertex that does not move has no derivative
            out[pass * 3 + k] = mv[k] ? s : 0.0;
        }
    }
}

__global__ void iface_apply(AdjArgs A, IfSetDev S, const int32_t* __restrict__ facet_cluster, int64_t nfacets,
                            const double* __restrict__ sums, const double* __restrict__ parts) {
    const int64_t f = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nfacets) return;
    // F = -(wL A + wF B + gamma C), gamma = 2 alpha |G| / S
    const double* q = sums + facet_cluster[f] * (int64_t)kIfSums;
    const double cg = q[1] * 2.0 * S.alpha * q[6];
    const double* P = parts + f * kIfParts;
    for (int k = 0; k < 3; ++k)
        if (P[k] != 0.0 || P[3 + k] != 0.0) atomicAdd(A.G + S.vid[f * 3 + k], -fma(cg, P[3 + k], P[k]));
}

// items: (interface cluster e, side) per cell of the linked cut cluster
__global__ void iface_volumes(AdjArgs A, IfSetDev S, const CutSetDev* cuts, int64_t nitems,
                              const int64_t* __restrict__ item_e, const int64_t* __restrict__ item_cell,
                              const double* __restrict__ sums) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nitems) return;
    const int64_t es = item_e[t], e = es >> 1;
    const int side = (int)(es & 1);
    const CutSetDev& C = cuts[S.link[e * 4 + side * 2]];
    const int64_t g = item_cell[t];
    double Xv[4][3], dx[4][3], dV[4][3];
    bool mv[4], any = false;
    int32_t vids[4];
    for (int k = 0; k < 4; ++k) {
        vids[k] = C.vid[g * 4 + k];
        mv[k] = vertex(A, vids[k], Xv[k], dx[k]);
        any |= mv[k];
    }
    if (!any) return;
    // dw_L/dV_L = w_F / S, dw_L/dV_F = -w_L / S, dgamma/dV = -gamma / S (per V / E)
    const double* q = sums + e * kIfSums;
    const double coef = -(q[0] * (side == 0 ? q[5] : -q[4]) - q[1] * q[3]) * q[6] / (side == 0 ? S.E[e] : S.EF[e]);
    tet_volume(Xv, dV);
    for (int k = 0; k < 4; ++k)
        if (mv[k]) atomicAdd(A.G + vids[k], coef * dot3(dV[k], dx[k]));
}

// dQ/dp = sum_v G[v] dt_v/dp through the parents' level set, in two steps: the
// weight of every background node (a vertex touches up to 16), then the nodes'
// coefficients, one warp per node with a weight.  A vertex writing its
// coefficients itself repeats the width (64 for cubic splines) for every node.
__global__ void dqdp_nodes(int64_t nv, const int32_t* vkind, const int32_t* vpar, const double* vphi, const double* G,
                           double* node_weight) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv || vkind[v] != 3 || G[v] == 0.0) return;
    const int32_t p[2] = {vpar[v * 8], vpar[v * 8 + 1]};
    const double f0 = vphi[p[0]], f1 = vphi[p[1]];
    const double den = (f0 - f1) * (f0 - f1);
    // t = f0 / (f0 - f1): dt/df0 = -f1 / (f0-f1)^2, dt/df1 = f0 / (f0-f1)^2
    const double dt[2] = {-f1 / den, f0 / den};
    for (int k = 0; k < 2; ++k) {
        const int32_t q = p[k];
        const int kind = vkind[q];
        const int cnt = kind == 0 ? 1 : kind == 1 ? 4 : 8;
        const double w = G[v] * dt[k] / (double)cnt;
        for (int m = 0; m < cnt; ++m) atomicAdd(node_weight + vpar[(int64_t)q * 8 + m], w);
    }
}
__global__ void dqdp_coefficients(int64_t nbn, int width, const int32_t* __restrict__ cols,
                                  const double* __restrict__ tmat, const double* __restrict__ node_weight,
                                  double* dqdp) {
    const int64_t n = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (n >= nbn) return;
    const double w = node_weight[n];
    if (w == 0.0) return;
    for (int j = threadIdx.x & 31; j < width; j += 32) {
        const double tv = tmat[n * width + j];
        if (tv != 0.0) atomicAdd(dqdp + cols[n * width + j], w * tv);
    }
}

__global__ void dot_kernel(int64_t n, const double* a, const double* b, double* out) {
    double s = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s = fma(a[i], b[i], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __shared__ double ws[32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        s = threadIdx.x < (blockDim.x >> 5) ? ws[threadIdx.x] : 0.0;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) atomicAdd(out, s);
    }
}

void dfree(DeviceBuf& b) {
    if (b.p) cudaFree(b.p);
    b.p = nullptr;
    b.bytes = 0;
}

template <class T>
cudaError_t upload(DeviceBuf& b, const std::vector<T>& v, cudaStream_t st) {
    dfree(b);
    b.bytes = std::max<size_t>(v.size() * sizeof(T), 16);
    cudaError_t e = cudaMalloc(&b.p, b.bytes);
    if (e != cudaSuccess) return e;
    if (!v.empty()) e = cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st);
    return e;
}

// in-place refresh (same size: kernel arguments and captured graphs keep their pointers)
template <class T>
cudaError_t refresh(DeviceBuf& b, const std::vector<T>& v, cudaStream_t st) {
    if (!b.p || b.bytes < v.size() * sizeof(T)) return upload(b, v, st);
    if (v.empty()) return cudaSuccess;
    return cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st);
}

fem_gpu_status sfail(fem_gpu_ctx* c, cudaError_t e, const char* what) {
    return fail(c, e == cudaErrorMemoryAllocation ? FEM_GPU_OUT_OF_MEMORY : FEM_GPU_CUDA_ERROR,
                std::string(what) + ": " + cudaGetErrorString(e));
}

double lam_of(int model, double nu) {
    return model == FEM_GPU_MODEL_PLANE_STRESS ? nu / (1.0 - nu * nu) : nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
}

bool is_cut(const SetData& s) { return s.kind == 0 && !s.ig_off.empty(); }
bool is_interface(const SetData& s) {
    return s.kind == 2 && !is_ghost_iwg(s.dside.iwg_type);
}

}  // namespace

void sensitivity_release(fem_gpu_ctx* c) {
    dfree(c->d_vkind);
    dfree(c->d_vpar);
    dfree(c->d_vx);
    dfree(c->d_adjcuts);
    dfree(c->d_vval);
    dfree(c->d_lscols);
    dfree(c->d_lst);
    dfree(c->d_lsw);
    c->ls_nbn = 0;
    c->ls_phi = false;
    for (auto& s : c->sets) {
        dfree(s.d_vid);
        dfree(s.d_link);
        dfree(s.d_adjul);
        dfree(s.d_items);
        dfree(s.d_moving);
        s.nitems = s.nmoving = 0;
    }
    c->adj_topo = c->adj_coords = false;
}

}  // namespace fem

using namespace fem;

extern "C" {

fem_gpu_status fem_gpu_set_ig_vertices(fem_gpu_ctx* c, int64_t nv, const int32_t* kind, const int32_t* parents,
                                       const double* coords, const double* value) {
    if (!c || nv <= 0 || !kind || !parents || !coords || !value) return FEM_GPU_BAD_ARG;
    c->vkind.assign(kind, kind + nv);
    c->vpar.assign(parents, parents + nv * 8);
    c->vx.assign(coords, coords + nv * 3);
    c->vval.assign(value, value + nv);
    c->adj_topo = c->adj_coords = c->ls_phi = false;
    c->ls_checked_nbn = -1;
    for (int64_t v = 0; v < nv; ++v) {
        const int k = c->vkind[v];
        if (k < 0 || k > 3) return fail(c, FEM_GPU_BAD_ARG, "IG vertex kind");
        const int cnt = k == 0 ? 1 : k == 1 ? 4 : k == 2 ? 8 : 2;
        for (int m = 0; m < cnt; ++m) {
            const int32_t p = c->vpar[v * 8 + m];
            const int64_t lim = k == 3 ? nv : c->num_nodes;
            if (p < 0 || p >= lim) return fail(c, FEM_GPU_OOB_INDEX, "IG vertex parent");
            if (k == 3 && c->vkind[p] == 3) return fail(c, FEM_GPU_BAD_ARG, "intersection of intersections");
        }
    }
    for (auto& s : c->sets) {
        if (!(is_cut(s) || is_interface(s)) || s.neq == 0) continue;
        if (s.vid.empty()) return fail(c, FEM_GPU_BAD_ARG, "cut / interface set without IG vertex ids");
        for (int32_t v : s.vid)
            if (v < 0 || v >= nv) return fail(c, FEM_GPU_OOB_INDEX, "IG vertex id");
    }
    return FEM_GPU_OK;
}

fem_gpu_status fem_gpu_update_ig_vertices(fem_gpu_ctx* c, const double* t) {
    if (!c || !t) return FEM_GPU_BAD_ARG;
    if (!c->dev_final) return FEM_GPU_NOT_FINALIZED;
    if (c->vkind.empty()) return fail(c, FEM_GPU_BAD_ARG, "no IG vertex table");
    if (c->shape != FEM_GPU_SHAPE_RECTANGULAR) return fail(c, FEM_GPU_UNSUPPORTED, "geometry update needs rectangular cells");
    const int64_t nv = (int64_t)c->vkind.size();
    for (int64_t v = 0; v < nv; ++v) {
        if (c->vkind[v] != 3) continue;
        if (!std::isfinite(t[v])) return fail(c, FEM_GPU_NONFINITE, "edge coordinate");
        const int32_t p0 = c->vpar[v * 8], p1 = c->vpar[v * 8 + 1];
        for (int d = 0; d < 3; ++d) c->vx[v * 3 + d] = c->vx[p0 * 3 + d] + t[v] * (c->vx[p1 * 3 + d] - c->vx[p0 * 3 + d]);
        c->vval[v] = t[v];
    }
    c->adj_coords = false;
    const int npe = c->npe;
    auto param = [&](int64_t cell, const double* x, double* xi) {
        const double* X0 = &c->coords[(int64_t)c->cells[cell * npe + 0] * 3];
        const double* X6 = &c->coords[(int64_t)c->cells[cell * npe + 6] * 3];
        for (int d = 0; d < 3; ++d) xi[d] = -1.0 + 2.0 * (x[d] - X0[d]) / (X6[d] - X0[d]);
    };
    cudaStream_t st = (cudaStream_t)c->stream;
    cudaError_t e = cudaSuccess;
    for (auto& s : c->sets) {
        if (s.neq == 0) continue;
        if (is_cut(s)) {
            for (int64_t i = 0; i < s.neq; ++i)
                for (int64_t g = s.ig_off[i]; g < s.ig_off[i + 1]; ++g)
                    for (int k = 0; k < 4; ++k) {
                        const int32_t v = s.vid[g * 4 + k];
                        if (c->vkind[v] != 3) continue;
                        for (int d = 0; d < 3; ++d) s.ig_coords[(g * 4 + k) * 3 + d] = c->vx[v * 3 + d];
                        param(s.ip_cell[i], &c->vx[v * 3], &s.ig_param[(g * 4 + k) * 3]);
                    }
            if (e == cudaSuccess) e = refresh(s.d_igx, s.ig_coords, st);
            if (e == cudaSuccess) e = refresh(s.d_igxi, s.ig_param, st);
        } else if (is_interface(s)) {
            for (int64_t i = 0; i < s.neq; ++i)
                for (int64_t f = s.fc_off[i]; f < s.fc_off[i + 1]; ++f)
                    for (int k = 0; k < s.nfv; ++k) {
                        const int32_t v = s.vid[f * s.nfv + k];
                        if (c->vkind[v] != 3) continue;
                        for (int d = 0; d < 3; ++d) s.fc_x[(f * s.nfv + k) * 3 + d] = c->vx[v * 3 + d];
                        param(s.ip_cell[i], &c->vx[v * 3], &s.fc_xl[(f * s.nfv + k) * 3]);
                        param(s.fcell[i], &c->vx[v * 3], &s.fc_xf[(f * s.nfv + k) * 3]);
                    }
            if (e == cudaSuccess) e = refresh(s.d_fcx, s.fc_x, st);
            if (e == cudaSuccess) e = refresh(s.d_fcxl, s.fc_xl, st);
            if (e == cudaSuccess) e = refresh(s.d_fcxf, s.fc_xf, st);
        }
    }
    fem_gpu_status r = interface_volumes(c);
    if (r != FEM_GPU_OK) return r;
    for (auto& s : c->sets)
        if (is_interface(s) && s.neq > 0 && e == cudaSuccess) e = refresh(s.d_vol, s.vol, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return sfail(c, e, "geometry update");
    return FEM_GPU_OK;
}

fem_gpu_status fem_gpu_strain_energy(fem_gpu_ctx* c, const double* u, double* dqdu, double* q) {
    if (!c || !u || !dqdu) return FEM_GPU_BAD_ARG;
    if (!c->dev_final) return FEM_GPU_NOT_FINALIZED;
    // residual-only assembly of the bulk sets: dQ/du = K_bulk u (linear CM, no body load)
    cudaStream_t st = (cudaStream_t)c->stream;
    const int64_t nad = c->num_used * c->dim;
    cudaError_t e = cudaMemsetAsync(dqdu, 0, nad * sizeof(double), st);
    if (e != cudaSuccess) return sfail(c, e, "strain energy zero");
    fem_gpu_status r = FEM_GPU_OK;
    for (int k = 0; k < (int)c->sets.size() && r == FEM_GPU_OK; ++k) {
        if (c->sets[k].kind != 0) continue;
        r = assemble_set(c, k, u, nullptr, dqdu);
    }
    if (r != FEM_GPU_OK) return r;
    if (q) {
        double* d = nullptr;
        e = cudaMallocAsync(&d, sizeof(double), st);
        if (e == cudaSuccess) e = cudaMemsetAsync(d, 0, sizeof(double), st);
        if (e == cudaSuccess) {
            dot_kernel<<<(unsigned)sm_count() * 4, 256, 0, st>>>(nad, u, dqdu, d);
            e = cudaMemcpyAsync(q, d, sizeof(double), cudaMemcpyDeviceToHost, st);
        }
        if (d) cudaFreeAsync(d, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return sfail(c, e, "strain energy");
        *q *= 0.5;
    }
    return fem_gpu_check_status(c);
}

fem_gpu_status fem_gpu_drdp_adjoint(fem_gpu_ctx* c, const double* u, const double* lambda, double* G) {
    if (!c || !u || !lambda || !G) return FEM_GPU_BAD_ARG;
    if (!c->dev_final) return FEM_GPU_NOT_FINALIZED;
    if (c->vkind.empty()) return fail(c, FEM_GPU_BAD_ARG, "no IG vertex table");
    if (c->shape != FEM_GPU_SHAPE_RECTANGULAR || c->dim != 3)
        return fail(c, FEM_GPU_UNSUPPORTED, "shape sensitivities need 3D rectangular cells");
    cudaStream_t st = (cudaStream_t)c->stream;
    const int64_t nv = (int64_t)c->vkind.size();
    // the vertex table, vertex ids, interface links and volume items depend on
    // the topology only and go to the device once per vertex table; the
    // coordinates once per geometry update
    const bool topo = !c->adj_topo;
    c->adj_topo = false;
    cudaError_t e = cudaSuccess;
    if (topo) {
        e = refresh(c->d_vkind, c->vkind, st);
        if (e == cudaSuccess) e = refresh(c->d_vpar, c->vpar, st);
    }
    if (e == cudaSuccess && !c->adj_coords) e = refresh(c->d_vx, c->vx, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(G, 0, nv * sizeof(double), st);
    if (e != cudaSuccess) return sfail(c, e, "adjoint vertex table");
    c->adj_coords = true;
    AdjArgs A{};
    A.vkind = (const int32_t*)c->d_vkind.p;
    A.vpar = (const int32_t*)c->d_vpar.p;
    A.vx = (const double*)c->d_vx.p;
    A.G = G;
    A.u = u;
    A.lam = lambda;
    A.nu = c->num_used;
    // cut sets
    std::vector<CutSetDev> cuts;
    std::vector<int> cut_index(c->sets.size(), -1), cut_set;  // set -> cut index, cut index -> set
    std::vector<std::pair<int32_t, int64_t>> cell_cluster(topo ? c->num_cells : 0, {-1, -1});
    for (size_t k = 0; k < c->sets.size(); ++k) {
        SetData& s = c->sets[k];
        if (!is_cut(s) || s.neq == 0) continue;
        if (s.vid.empty()) return fail(c, FEM_GPU_BAD_ARG, "cut set without IG vertex ids");
        if (s.bulk.integration_rule != FEM_GPU_RULE_TET_4 && s.bulk.integration_rule != FEM_GPU_RULE_TET_11)
            return fail(c, FEM_GPU_UNSUPPORTED, "sensitivities of cut clusters need TET4 cells");
        if (topo && (e = refresh(s.d_vid, s.vid, st)) != cudaSuccess) return sfail(c, e, "vertex ids");
        CutSetDev d{};
        d.neq = s.neq;
        d.xe = (const double*)s.d_xe.p;
        d.E = (const double*)s.d_E.p;
        d.nb = (const int32_t*)s.d_nb.p;
        d.bases = (const int32_t*)s.d_bases.p;
        d.T = (const double*)s.d_T.p;
        d.W = s.nbsel;
        d.lam_c = lam_of(s.bulk.model_type, s.bulk.poisson_ratio);
        d.mu_c = 1.0 / (2.0 * (1.0 + s.bulk.poisson_ratio));
        d.ig_off = (const int64_t*)s.d_igoff.p;
        d.vid = (const int32_t*)s.d_vid.p;
        d.gp = (const double*)s.d_gp.p;
        d.gw = (const double*)s.d_gw.p;
        d.ngp = s.ngp;
        cut_index[k] = (int)cuts.size();
        cut_set.push_back((int)k);
        if (topo)
            for (int64_t i = 0; i < s.neq; ++i) cell_cluster[s.ip_cell[i]] = {(int32_t)cuts.size(), i};
        cuts.push_back(d);
    }
    for (size_t k = 0, ci = 0; k < c->sets.size(); ++k) {
        if (cut_index[k] < 0) continue;
        SetData& s = c->sets[k];
        const CutSetDev& d = cuts[ci++];
        const int64_t ncells = s.ig_off.empty() ? 0 : s.ig_off.back();
        // per-cluster pdof values of u and lambda, then one thread per cell
        // [neq][48] doubles, then [ncells] cluster indices
        const size_t need =
            (size_t)d.neq * 48 * sizeof(double) + (size_t)std::max<int64_t>(ncells, 1) * sizeof(int32_t);
        if (!s.d_adjul.p || s.d_adjul.bytes < need) {
            dfree(s.d_adjul);
            if ((e = cudaMalloc(&s.d_adjul.p, need)) != cudaSuccess) return sfail(c, e, "adjoint cluster values");
            s.d_adjul.bytes = need;
        }
        double* UL = (double*)s.d_adjul.p;
        int32_t* cc = reinterpret_cast<int32_t*>(UL + (size_t)d.neq * 48);
        if (topo) {
            // integration cells with a moving (intersection) vertex
            std::vector<int32_t> moving;
            for (int64_t g = 0; g < ncells; ++g)
                for (int k = 0; k < 4; ++k)
                    if (c->vkind[s.vid[g * 4 + k]] == 3) {
                        moving.push_back((int32_t)g);
                        break;
                    }
            s.nmoving = (int64_t)moving.size();
            if ((e = upload(s.d_moving, moving, st)) != cudaSuccess) return sfail(c, e, "moving cells");
        }
        adjoint_cluster_values<<<(unsigned)std::max<int64_t>(d.neq, 1), 64, 0, st>>>(A, d, UL, cc);
        c->launches++;
        if (s.nmoving > 0) {
            adjoint_tets<<<(unsigned)((s.nmoving + 63) / 64), 64, 0, st>>>(A, d, UL, cc, (const int32_t*)s.d_moving.p,
                                                                           s.nmoving);
            c->launches++;
        }
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return sfail(c, e, "adjoint tets");
    if ((e = refresh(c->d_adjcuts, cuts, st)) != cudaSuccess) return sfail(c, e, "cut table");
    fem_gpu_status r = FEM_GPU_OK;
    for (auto& s : c->sets) {
        if (!is_interface(s) || s.neq == 0) continue;
        if (s.vid.empty() || s.nfv != 3) {
            r = fail(c, FEM_GPU_UNSUPPORTED, "interface sensitivities need TRI3 facets with vertex ids");
            break;
        }
        if (topo) {
            s.link.assign(s.neq * 4, 0);
            for (int64_t i = 0; i < s.neq; ++i) {
                const auto L = cell_cluster[s.ip_cell[i]], F = cell_cluster[s.fcell[i]];
                if (L.first < 0 || F.first < 0) {
                    r = fail(c, FEM_GPU_BAD_ARG, "interface cluster without cut clusters on its cells");
                    break;
                }
                s.link[i * 4 + 0] = L.first;
                s.link[i * 4 + 1] = (int32_t)L.second;
                s.link[i * 4 + 2] = F.first;
                s.link[i * 4 + 3] = (int32_t)F.second;
            }
            if (r != FEM_GPU_OK) break;
            // volume items: (e * 2 + side) in the first half, the integration cell in the second
            std::vector<int64_t> items;
            for (int pass = 0; pass < 2; ++pass)
                for (int64_t i = 0; i < s.neq; ++i)
                    for (int side = 0; side < 2; ++side) {
                        const int cs = s.link[i * 4 + side * 2];
                        const int64_t ce = s.link[i * 4 + side * 2 + 1];
                        const std::vector<int64_t>& io = c->sets[cut_set[cs]].ig_off;
                        for (int64_t g = io[ce]; g < io[ce + 1]; ++g) items.push_back(pass == 0 ? i * 2 + side : g);
                    }
            s.nitems = (int64_t)items.size() / 2;
            if ((e = refresh(s.d_link, s.link, st)) != cudaSuccess || (e = refresh(s.d_vid, s.vid, st)) != cudaSuccess ||
                (e = upload(s.d_items, items, st)) != cudaSuccess) {
                r = sfail(c, e, "interface links");
                break;
            }
        }
        IfSetDev d{};
        d.neq = s.neq;
        d.beta_sym = s.dside.iwg_type == FEM_GPU_IWG_STRUC_LINEAR_INTERFACE_SYMMETRIC_NITSCHE;
        d.alpha = s.dside.alpha;
        d.lam_c = lam_of(s.dside.model_type, s.dside.poisson_ratio);
        d.mu_c = 1.0 / (2.0 * (1.0 + s.dside.poisson_ratio));
        d.xe = (const double*)s.d_xe.p;
        d.E = (const double*)s.d_E.p;
        d.EF = (const double*)s.d_EF.p;
        d.nb = (const int32_t*)s.d_nb.p;
        d.bases = (const int32_t*)s.d_bases.p;
        d.T = (const double*)s.d_T.p;
        d.W = s.nbsel;
        d.fc_off = (const int64_t*)s.d_fcoff.p;
        d.vid = (const int32_t*)s.d_vid.p;
        d.gp = (const double*)s.d_gp.p;
        d.gw = (const double*)s.d_gw.p;
        d.ngp = s.ngp;
        d.vol = (const double*)s.d_vol.p;
        d.link = (const int32_t*)s.d_link.p;
        // scratch: per cluster the field polynomials and sums; per facet the cluster
        // index and the derivative parts; the volume items
        const int64_t nf = s.fc_off.empty() ? 0 : s.fc_off.back();
        const int64_t ni = s.nitems;
        const int64_t* item_e = (const int64_t*)s.d_items.p;
        const size_t need = (size_t)s.neq * (kIfFields + kIfSums) * sizeof(double) +
                            (size_t)std::max<int64_t>(nf, 1) * (kIfParts * sizeof(double) + sizeof(int32_t));
        if (!s.d_adjul.p || s.d_adjul.bytes < need) {
            dfree(s.d_adjul);
            if ((e = cudaMalloc(&s.d_adjul.p, need)) != cudaSuccess) {
                r = sfail(c, e, "interface scratch");
                break;
            }
            s.d_adjul.bytes = need;
        }
        double* UL = (double*)s.d_adjul.p;
        double* sums = UL + (size_t)s.neq * kIfFields;
        double* parts = sums + (size_t)s.neq * kIfSums;
        int32_t* fcl = reinterpret_cast<int32_t*>(parts + (size_t)std::max<int64_t>(nf, 1) * kIfParts);
        const auto grid_of = [](int64_t n) { return (unsigned)std::max<int64_t>(1, (n + 63) / 64); };
        iface_cluster_values<<<(unsigned)std::max<int64_t>(s.neq, 1), 64, 0, st>>>(A, d, UL, fcl, sums);
        iface_facets<<<grid_of(nf), 64, 0, st>>>(A, d, UL, fcl, nf, sums, parts);
        iface_apply<<<grid_of(nf), 64, 0, st>>>(A, d, fcl, nf, sums, parts);
        iface_volumes<<<grid_of(ni), 64, 0, st>>>(A, d, (const CutSetDev*)c->d_adjcuts.p, ni, item_e, item_e + ni,
                                                  sums);
        c->launches += 4;
        if ((e = cudaGetLastError()) != cudaSuccess) {
            r = sfail(c, e, "adjoint interface");
            break;
        }
    }
    if (r != FEM_GPU_OK) return r;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return sfail(c, e, "adjoint");
    c->adj_topo = true;
    return FEM_GPU_OK;
}

fem_gpu_status fem_gpu_set_level_set_field(fem_gpu_ctx* c, int64_t nbn, int32_t width, const int32_t* cols,
                                           const double* tmat, int64_t ncoef) {
    if (!c || !cols || !tmat || width <= 0 || nbn <= 0 || ncoef <= 0) return FEM_GPU_BAD_ARG;
    const int64_t n = nbn * width;
    for (int64_t k = 0; k < n; ++k)
        if (cols[k] < 0 || cols[k] >= ncoef) return fail(c, FEM_GPU_OOB_INDEX, "level-set coefficient id");
    c->ls_nbn = 0;
    cudaStream_t st = (cudaStream_t)c->stream;
    cudaError_t e = cudaSuccess;
    if (!c->d_lscols.p || c->d_lscols.bytes < (size_t)n * sizeof(int32_t)) {
        dfree(c->d_lscols);
        if ((e = cudaMalloc(&c->d_lscols.p, (size_t)n * sizeof(int32_t))) == cudaSuccess)
            c->d_lscols.bytes = (size_t)n * sizeof(int32_t);
    }
    if (e == cudaSuccess && (!c->d_lst.p || c->d_lst.bytes < (size_t)n * sizeof(double))) {
        dfree(c->d_lst);
        if ((e = cudaMalloc(&c->d_lst.p, (size_t)n * sizeof(double))) == cudaSuccess)
            c->d_lst.bytes = (size_t)n * sizeof(double);
    }
    if (e == cudaSuccess && (!c->d_lsw.p || c->d_lsw.bytes < (size_t)nbn * sizeof(double))) {
        dfree(c->d_lsw);
        if ((e = cudaMalloc(&c->d_lsw.p, (size_t)nbn * sizeof(double))) == cudaSuccess)
            c->d_lsw.bytes = (size_t)nbn * sizeof(double);
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(c->d_lscols.p, cols, (size_t)n * sizeof(int32_t), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(c->d_lst.p, tmat, (size_t)n * sizeof(double), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return sfail(c, e, "level-set field");
    c->ls_nbn = nbn;
    c->ls_width = width;
    c->ls_ncoef = ncoef;
    return FEM_GPU_OK;
}

fem_gpu_status fem_gen_dqdp(fem_gpu_ctx* c, const double* G, int64_t nbn, int32_t width, const int32_t* cols,
                            const double* tmat, int64_t ncoef, double* dqdp) {
    if (!c || !G || !dqdp || width <= 0 || nbn <= 0 || ncoef <= 0 || (!cols) != (!tmat)) return FEM_GPU_BAD_ARG;
    if (c->vkind.empty()) return fail(c, FEM_GPU_BAD_ARG, "no IG vertex table");
    if (cols) {
        const fem_gpu_status r = fem_gpu_set_level_set_field(c, nbn, width, cols, tmat, ncoef);
        if (r != FEM_GPU_OK) return r;
    } else if (c->ls_nbn != nbn || c->ls_width != width || c->ls_ncoef != ncoef) {
        return fail(c, FEM_GPU_BAD_ARG, "no level-set field of these sizes (fem_gpu_set_level_set_field)");
    }
    const int64_t nv = (int64_t)c->vkind.size();
    // background parents of the vertex table against this field (once per table and field size)
    if (c->ls_checked_nbn != nbn) {
        for (int64_t v = 0; v < nv; ++v)
            if (c->vkind[v] != 3)
                for (int m = 0; m < 8; ++m)
                    if (c->vpar[v * 8 + m] >= nbn) return fail(c, FEM_GPU_OOB_INDEX, "background node of an IG vertex");
        c->ls_checked_nbn = nbn;
    }
    cudaStream_t st = (cudaStream_t)c->stream;
    // level set at the parents: vval holds phi for kinds 0-2 (set with the
    // vertex table; geometry updates change the kind-3 entries only)
    cudaError_t e = cudaSuccess;
    if (!c->ls_phi) e = refresh(c->d_vval, c->vval, st);
    if (e == cudaSuccess && !c->adj_topo) e = refresh(c->d_vkind, c->vkind, st);
    if (e == cudaSuccess && !c->adj_topo) e = refresh(c->d_vpar, c->vpar, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(dqdp, 0, ncoef * sizeof(double), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(c->d_lsw.p, 0, nbn * sizeof(double), st);
    if (e == cudaSuccess) {
        c->ls_phi = true;
        double* nw = (double*)c->d_lsw.p;
        dqdp_nodes<<<(unsigned)((nv + 127) / 128), 128, 0, st>>>(nv, (const int32_t*)c->d_vkind.p,
                                                                 (const int32_t*)c->d_vpar.p,
                                                                 (const double*)c->d_vval.p, G, nw);
        dqdp_coefficients<<<(unsigned)((nbn + 7) / 8), 256, 0, st>>>(nbn, width, (const int32_t*)c->d_lscols.p,
                                                                     (const double*)c->d_lst.p, nw, dqdp);
        c->launches += 2;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return sfail(c, e, "dq/dp chain");
    return FEM_GPU_OK;
}

}  // extern "C"
