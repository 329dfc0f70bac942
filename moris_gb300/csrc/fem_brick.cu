// fem_brick.cu -- XFEM clusters on axis-aligned brick cells: uncut cells, cut
// clusters, Nitsche interfaces inside one cell, ghost faces and (linear splines)
// boundary facets.
//
// The general cluster kernel (fem_cluster.cu) forms every element matrix from
// per-point operators and projects it through column lists.  On bricks with
// the extraction of level-0 HMR meshes far less is left to do:
//
//   * dN_a/dx_i = (1/J_i) s_i (1 + s_j xi_j)(1 + s_k xi_k) / 8 with constant J, so
//     every integral of two shape functions or gradients is a signed sum of the
//     27 monomial moments sum_q w* xi^p eta^q zeta^r, p, q, r <= 2.  A bulk
//     cluster needs its moments and the 63 distinct values of its 300 Gram
//     entries; an interface the moments weighted with the facet normals; an
//     uncut cell and a whole-face ghost only tables and cell sizes;
//   * linear splines: every node carries one basis with weight 1, the element
//     matrix is the nodal one.  A warp takes one equation object, each lane
//     some node pairs: it forms the pair's 3 x 3 block in registers, adds it to
//     the CSR and to its share of the residual.  No element matrix is stored and
//     there is no CTA barrier;
//   * quadratic splines: T = P/8 with P the tensor-product pattern of the cell
//     (fem_bulk_cta.cuh), both sides of K T and T^T (K T) are axis-wise sums of
//     additions.  One CTA per object: the first warp forms K / 64, all four
//     project and scatter.
//
// brick_classify decides per equation object, exactly (coordinates, extraction
// weights, facet corners); the rest stays with the general kernel.
//
// Measured on GB300, batched assembly with residual, general kernel -> here:
// 64^3 cells cut by 40 spheres, linear splines 32.5 -> 4.36 ms (ghost 27, cut
// 24, uncut 22, interface 19 % of it); 22^3, 12 spheres, quadratic splines 7.93
// -> 0.869 ms.  The general kernel spent 27 k FP64 products on a ghost face (now
// 4 k) and 180 k on an interface cluster (now 19 k).  Bound: the L2's FP64
// atomics (576 per cell, 1,408 per ghost face, 2,304 per interface) and the FP64
// pipe about equally.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <thread>

#include "fem_bits.cuh"
#include "fem_brick.cuh"

namespace fem {
namespace {

enum { KIND_UNCUT = 0, KIND_CUT = 1, KIND_GHOST = 2, KIND_INTERFACE = 3, KIND_SIDE = 4 };
__host__ __device__ constexpr int sides_of(int kind) { return kind == KIND_GHOST || kind == KIND_INTERFACE ? 2 : 1; }

struct BrickArgs {
    int64_t n;             // equation objects
    const int32_t* list;   // their indices in the set
    const uint8_t* code;   // SetData::fast
    const uint8_t* map;    // [neq][sides][W]: linear: column of node a; quadratic: column of basis code
    const double* xe;      // [neq][sides][8][3]
    const double* E;
    const double* EF;
    const int32_t* bases;  // [neq][sides][W]
    const uint16_t* sidx;  // [neq][sides W][sides W]
    const double* gp;      // integration cell / facet points
    const double* gw;
    int ngp, normal_field, neumann;
    double lam_c, mu_c, alpha, beta;
    double value[3], thickness;  // boundary facets
    const double* tab;     // uncut: 63 reference sums; ghost: kGhostTab per face
    const double* geo;     // reciprocals and roots of the cells (kGeoUncut, kGeoGhost per object)
    const int64_t* off;    // integration cells / facets of an object
    const double* x;       // their vertex coordinates
    const double* xi;      // their parametric coordinates
    const double* vol;     // interface: cluster volumes
    const int32_t* rowptr;
    const int32_t* ulen;
    int64_t nu;
    const double* u;
    double* vals;
    double* rhs;
    int* status;
};

// HEX8 node: its side (0 lower, 1 upper) along axis d
__host__ __device__ constexpr int corner(int a, int d) {
    return d == 0 ? ((a & 3) == 1 || (a & 3) == 2) : d == 1 ? (a & 3) >= 2 : a >= 4;
}
__host__ __device__ constexpr int node_at(int x, int y, int z) { return 4 * z + (y ? (x ? 2 : 3) : (x ? 1 : 0)); }

// The 63 sums of a bulk object: per axis either both functions are
// differentiated (one sum, of 1), neither (three sums, of (1+x)^2, (1-x)^2 and
// 1-x^2) or one of them (two sums, of 1+x and 1-x); products over the axes for
// the component pairs xx, yy, zz, xy, xz, yz, z fastest.
constexpr int kSums = 63;
// pair (i, j) of differentiated components, i <= j -> offset of its sums
__host__ __device__ constexpr int pair_off(int i, int j) {
    return i == j ? 9 * i : i + j == 1 ? 27 : i + j == 2 ? 39 : 51;
}
// number of sums along axis d for the pair (i, j)
__host__ __device__ constexpr int axis_sums(int i, int j, int d) {
    return d == i && d == j ? 1 : d == i || d == j ? 2 : 3;
}
// sum index and sign of A(i, j)(a, b) = integral dN_a/dx_i dN_b/dx_j
__host__ __device__ constexpr int gram_index(int i, int j, int a, int b, bool& neg) {
    int at = 0;
    neg = false;
    for (int d = 0; d < 3; ++d) {
        const int sa = corner(a, d), sb = corner(b, d);
        int v = 0;
        if (d == i && d == j) {
            neg ^= sa != sb;
        } else if (d == i) {  // N'_a N_b: the sign of a, the factor 1 +- x of b
            neg ^= sa == 0;
            v = sb ? 0 : 1;
        } else if (d == j) {
            neg ^= sb == 0;
            v = sa ? 0 : 1;
        } else {
            v = sa != sb ? 2 : sa ? 0 : 1;
        }
        at = at * axis_sums(i, j, d) + v;
    }
    return pair_off(i < j ? i : j, i < j ? j : i) + at;
}
// coefficients of 1, x, x^2 of sum v (of n) along an axis
__host__ __device__ constexpr int sum_coef(int n, int v, int p) {
    return p == 0   ? 1
           : p == 1 ? (n == 3 ? (v == 0 ? 2 : v == 1 ? -2 : 0) : n == 2 ? (v == 0 ? 1 : -1) : 0)
                    : (n == 3 ? (v == 2 ? -1 : 1) : 0);
}

__device__ __forceinline__ double signed_word(double v, unsigned neg) {
    // sign flip on the integer side (an FP64 negation would take the FP64 pipe)
    return __hiloint2double(__double2hiint(v) ^ (int)(neg << 31), __double2loint(v));
}
__device__ __forceinline__ double shfl(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }

// Where a node pair's block goes.  Linear splines: rows and columns are nodes.
struct Scatter {
    double* vals;
    int32_t row[3], ul;
    bool bad = false;
    __device__ __forceinline__ void add(const double K[9], int slot) {
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                const double v = K[f * 3 + g];
                bad |= !fem_finite(v);
                // structural zeros of ghost blocks are not added
                if (fem_nonzero(v)) atomicAdd(vals + row[f] + g * ul + slot, v);
            }
    }
};

// ---------------------------------------------------------------------------
// the 63 sums of a bulk object, times mu, into q (warp-wide); index tables in tab
// Per object, computed once when the set is classified, because a division or a root
// takes a warp 12 to 20 instructions of the FP64 pipe, a sixth of an uncut cell (64^3
// cells, 40 spheres 4.60 -> 4.34 ms for the batch): the
// reciprocal half lengths of an uncut cell; of both cells of a ghost face, then
// sqrt(16 J_t1 J_t2 / pi) and J_t1 J_t2.
constexpr int kGeoUncut = 3, kGeoGhost = 8;
__device__ void uncut_sums(const BrickArgs& p, int64_t e, double* q, int lane) {
    const double* X = p.xe + e * 24;
    // lane d = 0..2: half length along axis d and its reciprocal
    const int d = lane % 3;
    const double j = 0.5 * (__ldg(X + 18 + d) - __ldg(X + d)), r = __ldg(p.geo + e * kGeoUncut + d);
    const double j0 = shfl(j, 0), j1 = shfl(j, 1), j2 = shfl(j, 2);
    // scale of the component pair t = 0..5 (xx, yy, zz, xy, xz, yz) on lane t:
    // E mu detJ / (J_i J_j)
    const int t = lane % 6;
    const double em = p.E[e] * p.mu_c;
    const double rd = shfl(r, t < 3 ? t : 0);
    const double s1 = t == 0 ? j1 : j0, s2 = t == 2 ? j1 : j2;
    const double one = t == 3 ? j2 : t == 4 ? j1 : j0;
    const double s = em * (t < 3 ? s1 * s2 * rd : one);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int k = lane + 32 * m;
        const int ty = k < 27 ? k / 9 : k < 39 ? 3 : k < 51 ? 4 : 5;
        const double sc = shfl(s, ty);
        if (k < kSums) q[k] = sc * __ldg(p.tab + k);
    }
}

// cut cluster: the moments of its points, then the sums.  A lane forms one
// point (w*, xi), lane l < 27 owns moment l = (p, q, r) and adds the 32 points of
// the round from shared memory, one FMA each, in eight sums: one sum over the 96 to 240
// points of a cluster carried a rounding error of 7e-16, eight 1e-16.
constexpr int kPt = 13;  // doubles per staged point: x^p y^q (9), w z^r (3), padding
__device__ void cut_sums(const BrickArgs& p, int64_t e, double* st, double* q, int lane) {
    const int64_t c0 = p.off[e];
    const int np = (int)(p.off[e + 1] - c0) * p.ngp;
    const int l = lane < 27 ? lane : 0;
    double acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.0;
    for (int q0 = 0; q0 < np; q0 += 32) {
        const int t = q0 + lane;
        if (t < np) {
            const int k = t / p.ngp, g = t - k * p.ngp;
            const double* xh = p.xi + (c0 + k) * 12;
            const double* xx = p.x + (c0 + k) * 12;
            // TET4: barycentric coordinates xi_0, xi_1, 1 - sum, xi_2
            const double z0 = __ldg(p.gp + g * 3), z1 = __ldg(p.gp + g * 3 + 1), z2 = __ldg(p.gp + g * 3 + 2);
            const double N[4] = {z0, z1, 1.0 - z0 - z1 - z2, z2};
            double xi[3], a[3][3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                xi[d] = N[0] * __ldg(xh + d);
#pragma unroll
                for (int v = 1; v < 4; ++v) xi[d] = fma(N[v], __ldg(xh + v * 3 + d), xi[d]);
                const double o = __ldg(xx + 6 + d);
                a[0][d] = __ldg(xx + d) - o;
                a[1][d] = __ldg(xx + 3 + d) - o;
                a[2][d] = __ldg(xx + 9 + d) - o;
            }
            const double det = (a[0][0] * (a[1][1] * a[2][2] - a[2][1] * a[1][2]) -
                                a[0][1] * (a[1][0] * a[2][2] - a[1][2] * a[2][0]) +
                                a[0][2] * (a[1][0] * a[2][1] - a[1][1] * a[2][0])) *
                               (1.0 / 6.0);
            // points with detJ below -1e-6 are skipped (cl_FEM_Element_Bulk.cpp:164)
            const double w = det < -1.0e-6 ? 0.0 : __ldg(p.gw + g) * det;
            const double x2 = xi[0] * xi[0], y = xi[1], y2 = y * y;
            double* o = st + lane * kPt;
            o[0] = 1.0;
            o[1] = xi[0];
            o[2] = x2;
            o[3] = y;
            o[4] = xi[0] * y;
            o[5] = x2 * y;
            o[6] = y2;
            o[7] = xi[0] * y2;
            o[8] = x2 * y2;
            const double wz = w * xi[2];
            o[9] = w;
            o[10] = wz;
            o[11] = wz * xi[2];
        }
        __syncwarp();
        const int n = min(32, np - q0);
        const double* o = st + l % 9;
        const double* z = st + 9 + l / 9;
        int k = 0;
        for (; k + 8 <= n; k += 8)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] = fma(o[(k + j) * kPt], z[(k + j) * kPt], acc[j]);
        for (; k < n; ++k) acc[0] = fma(o[k * kPt], z[k * kPt], acc[0]);
        __syncwarp();
    }
    double* M = st;  // the moments
    if (lane < 27) M[lane] = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
    __syncwarp();
    const double* X = p.xe + e * 24;
    const int d = lane % 3;
    const double r = 2.0 / (__ldg(X + 18 + d) - __ldg(X + d));
    const double em = p.E[e] * p.mu_c * (1.0 / 64.0);
    double out[2];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const int k = lane + 32 * m;
        const int i = k < 27 ? k / 9 : k < 51 ? 0 : 1, j = k < 27 ? i : k < 39 ? 1 : 2;
        const double s = em * shfl(r, i) * shfl(r, j);
        const int n0 = axis_sums(i, j, 0), n1 = axis_sums(i, j, 1), n2 = axis_sums(i, j, 2);
        const int at = k < kSums ? k - pair_off(i, j) : 0;
        const int v2 = at % n2, v1 = at / n2 % n1, v0 = at / (n2 * n1);
        double a2 = 0.0;
        for (int c = 0; c < n2; ++c) {
            double a1 = 0.0;
            for (int b = 0; b < n1; ++b) {
                double a0 = 0.0;
                for (int a = 0; a < n0; ++a) a0 = fma((double)sum_coef(n0, v0, a), M[c * 9 + b * 3 + a], a0);
                a1 = fma((double)sum_coef(n1, v1, b), a0, a1);
            }
            a2 = fma((double)sum_coef(n2, v2, c), a1, a2);
        }
        out[m] = s * a2;
    }
    __syncwarp();
    q[lane] = out[0];
    if (lane + 32 < kSums) q[lane + 32] = out[1];
}

// the block of node pair (a, b) from the sums: K_fg = lam A_fg + mu A_gf (+ mu tr A)
__device__ __forceinline__ void bulk_block(const double* q, const uint8_t* gt, int a, int b, double ld, double lo,
                                           double K[9]) {
    double A[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) {
        const unsigned t = gt[m * 64 + a * 8 + b];
        A[m] = signed_word(q[t & 63], t >> 7);
    }
    const double tr = A[0] + A[4] + A[8];
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int g = 0; g < 3; ++g)
            K[f * 3 + g] = f == g ? fma(ld, A[f * 4], tr) : fma(lo, A[f * 3 + g], A[g * 3 + f]);
}

// sum index | sign << 7 of A(i, j)(a, b), [i * 3 + j][a][b]
__device__ void build_gram_table(uint8_t* gt) {
    for (int t = threadIdx.x; t < 576; t += blockDim.x) {
        bool neg;
        const int m = t >> 6, at = gram_index(m / 3, m % 3, t >> 3 & 7, t & 7, neg);
        gt[t] = (uint8_t)(at | (neg ? 128 : 0));
    }
}

// ---------------------------------------------------------------------------
// ghost: coefficients of the side pair (s, s2) of a lane.  With the normal along
// axis k and the tangents t1 < t2, A = J_t1 J_t2 and g the physical gradients,
//   K[k][k] = (lam + 2 mu) I_kk + mu (I_11 + I_22),   K[t][t] = mu I_kk,
//   K[k][t] = lam I_kt + mu I_tk,                     K[t][k] = mu I_kt,
// I_ij(a, b) = integral g_ia g_jb over the face, zero for the other tangent
// pairs; moduli of the column's side, sign - across the face, times alpha h with
// h = sqrt(4 area / pi) (SP_Ghost_Virtual_Work); the normal-field ghost is
// +-alpha h E_L I_kk on the diagonal (SP_Ghost_Displacement).
struct GhostCoef {
    double kk, kk_t, c11, c22, lam1, lam2, mu1, mu2, tk1, tk2;
    int k, t1, t2;
};
__device__ GhostCoef ghost_coef(const BrickArgs& p, int64_t e, int face, int s, int s2, double scale) {
    GhostCoef c;
    c.k = face >> 1;
    c.t1 = c.k == 0 ? 1 : 0;
    c.t2 = c.k == 2 ? 1 : 2;
    // reciprocal half lengths: lane 3 side + axis
    const int lane = threadIdx.x & 31, q = lane % 6;
    const double* geo = p.geo + e * kGeoGhost;
    const double rr = __ldg(geo + q);
    const double rk = shfl(rr, s * 3 + c.k), r1 = shfl(rr, s * 3 + c.t1), r2 = shfl(rr, s * 3 + c.t2);
    const double ok = shfl(rr, s2 * 3 + c.k), o1 = shfl(rr, s2 * 3 + c.t1), o2 = shfl(rr, s2 * 3 + c.t2);
    const double gam = p.alpha * __ldg(geo + 6) * __ldg(geo + 7) * (s == s2 ? scale : -scale);
    if (p.normal_field) {
        c.kk = c.kk_t = gam * p.E[e] * rk * ok;
        c.c11 = c.c22 = c.lam1 = c.lam2 = c.mu1 = c.mu2 = c.tk1 = c.tk2 = 0.0;
        return c;
    }
    const double Eo = s2 ? p.EF[e] : p.E[e];
    const double lam = gam * Eo * p.lam_c, mu = gam * Eo * p.mu_c;
    c.kk_t = mu * rk * ok;
    c.kk = (lam + 2.0 * mu) * rk * ok;
    c.c11 = mu * r1 * o1;
    c.c22 = mu * r2 * o2;
    c.lam1 = lam * rk * o1;
    c.lam2 = lam * rk * o2;
    c.mu1 = mu * rk * o1;
    c.mu2 = mu * rk * o2;
    c.tk1 = mu * r1 * ok;
    c.tk2 = mu * r2 * ok;
    return c;
}
// block of the lane's node and node b of the other side; tables [mat][b][lane]:
// I_kk, I_11, I_22, I_k1, I_k2, I_1k, I_2k in reference gradients
__device__ __forceinline__ void ghost_block(const GhostCoef& c, const double* tab, int b, int lane, bool normal_field,
                                            double K[9]) {
    const double* t = tab + b * 32 + lane;
    const double ikk = __ldg(t);
    double kk, tt = c.kk_t * ikk, k1 = 0.0, k2 = 0.0, q1 = 0.0, q2 = 0.0;
    if (normal_field) {
        kk = tt;
    } else {
        const double i1 = __ldg(t + 3 * 256), i2 = __ldg(t + 4 * 256);
        kk = fma(c.c22, __ldg(t + 2 * 256), fma(c.c11, __ldg(t + 256), c.kk * ikk));
        k1 = fma(c.tk1, __ldg(t + 5 * 256), c.lam1 * i1);
        k2 = fma(c.tk2, __ldg(t + 6 * 256), c.lam2 * i2);
        q1 = c.mu1 * i1;
        q2 = c.mu2 * i2;
    }
    // rows and columns in component order: selects only
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const bool fk = f == c.k, gk = g == c.k;
            K[f * 3 + g] = fk && gk  ? kk
                           : f == g  ? tt
                           : fk      ? (g == c.t1 ? k1 : k2)
                           : gk      ? (f == c.t1 ? q1 : q2)
                                     : 0.0;
        }
}

// ---------------------------------------------------------------------------
// interface inside one cell.  M[i][k](a, b) = sum w* n_i N_a dN_b/dx_k and
// Q(a, b) = sum w* N_a N_b come from the 27 moments weighted with n_0, n_1, n_2 and
// 1; then X[(f,a),(g,b)] = lam M[f][g] + mu M[g][f] + delta_fg mu tr M (a, b),
// lam, mu per unit modulus, and with w, E, sg per side
//   K = -sg_r w_c E_c X + beta w_r E_r sg_c X^T +- gamma Q
// (IWG_Isotropic_Struc_Linear_Interface, SP_Nitsche_Interface).  X at
// ((f*3+g)*8 + b)*9 + a, Q behind it.
constexpr int kIfX = 648, kIfQ = 72, kIfStage = 28 * kPt + 32 * 4;
constexpr int kIfMom = 108, kIfM = 720;
constexpr int kIfSmem = kIfX + kIfQ + (kIfStage > kIfMom + kIfM ? kIfStage : kIfMom + kIfM);
__device__ void interface_matrices(const BrickArgs& p, int64_t e, double* sm, double& area, int lane) {
    double* X = sm;
    double* st = sm + kIfX + kIfQ;
    double* nrm = st + 28 * kPt;  // per facet of a block of 32: normal, measure
    const int64_t f0 = p.off[e];
    const int nf = (int)(p.off[e + 1] - f0), ngp = p.ngp;
    const int per = 28 / ngp;  // facets per round (4 of 7 points)
    const int l = lane < 27 ? lane : 0;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    double meas = 0.0, wsum = 0.0;
    // from the last point to the first, whose weight is the largest: the other way round
    // the seven weights' sum is an ulp low in every facet and with it the penalty
    for (int k = ngp - 1; k >= 0; --k) wsum += __ldg(p.gw + k);
    for (int b0 = 0; b0 < nf; b0 += 32) {
        // facet normals and measures: detJ = |t1 x t2| / 2 of a TRI3
        if (b0 + lane < nf) {
            const double* x = p.x + (f0 + b0 + lane) * 9;
            double a[3], b[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                a[d] = x[d] - x[6 + d];
                b[d] = x[3 + d] - x[6 + d];
            }
            const double c0 = a[1] * b[2] - a[2] * b[1], c1 = a[2] * b[0] - a[0] * b[2], c2 = a[0] * b[1] - a[1] * b[0];
            const double nn = sqrt(c0 * c0 + c1 * c1 + c2 * c2), inv = nn > 0.0 ? 1.0 / nn : 0.0;
            nrm[lane * 4] = c0 * inv;
            nrm[lane * 4 + 1] = c1 * inv;
            nrm[lane * 4 + 2] = c2 * inv;
            nrm[lane * 4 + 3] = 0.5 * nn;
            meas = fma(0.5 * nn, wsum, meas);
        }
        __syncwarp();
        const int nb = min(32, nf - b0);
        for (int r0 = 0; r0 < nb; r0 += per) {
            const int fl = lane / ngp, g = lane - fl * ngp, fa = r0 + fl;
            if (fl < per && fa < nb) {
                const double* xh = p.xi + (f0 + b0 + fa) * 9;
                const double z0 = __ldg(p.gp + g * 2), z1 = __ldg(p.gp + g * 2 + 1), z2 = 1.0 - z0 - z1;
                double xi[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) xi[d] = fma(z2, xh[6 + d], fma(z1, xh[3 + d], z0 * xh[d]));
                const double w = __ldg(p.gw + g) * nrm[fa * 4 + 3];
                const double x2 = xi[0] * xi[0], y = xi[1], y2 = y * y;
                double* o = st + lane * kPt;
                o[0] = 1.0;
                o[1] = xi[0];
                o[2] = x2;
                o[3] = y;
                o[4] = xi[0] * y;
                o[5] = x2 * y;
                o[6] = y2;
                o[7] = xi[0] * y2;
                o[8] = x2 * y2;
                const double wz = w * xi[2];
                o[9] = w;
                o[10] = wz;
                o[11] = wz * xi[2];
            }
            __syncwarp();
            const int m = min(per, nb - r0);
            for (int k = 0; k < m; ++k) {
                const double* o = st + k * ngp * kPt + l % 9;
                const double* z = st + k * ngp * kPt + 9 + l / 9;
                int g2 = ngp - 1;
                double s = o[g2 * kPt] * z[g2 * kPt];
                while (--g2 >= 0) s = fma(o[g2 * kPt], z[g2 * kPt], s);
                const double* n = nrm + (r0 + k) * 4;
                acc[0] = fma(n[0], s, acc[0]);
                acc[1] = fma(n[1], s, acc[1]);
                acc[2] = fma(n[2], s, acc[2]);
                acc[3] += s;
            }
            __syncwarp();
        }
    }
    for (int o = 16; o > 0; o >>= 1) meas += __shfl_xor_sync(0xffffffffu, meas, o);
    area = meas;
    double* mom = st;            // [weight][27]
    double* M = st + kIfMom;     // [i*3+k | Q][b*9 + a]
    if (lane < 27)
        for (int c = 0; c < 4; ++c) mom[c * 27 + lane] = acc[c];
    const double* Xc = p.xe + e * 48;
    const double rj = 2.0 / (Xc[18 + lane % 3] - Xc[lane % 3]);
    __syncwarp();
    // task (matrix, x and y sides of a and b): three z moments, then the four z sides
    for (int t = lane; t < 160; t += 32) {
        const int ik = t >> 4, k = ik < 9 ? ik % 3 : 3;
        const double rk = shfl(rj, k < 3 ? k : 0);  // every lane takes part
        const double scale = k < 3 ? rk * (1.0 / 64.0) : 1.0 / 64.0;
        const double* mo = mom + (ik < 9 ? ik / 3 : 3) * 27;
        const int ax = t & 1, bx = t >> 1 & 1, ay = t >> 2 & 1, by = t >> 3 & 1;
        // coefficients of 1, x, x^2: N_a N_b, or N_a N'_b along axis k
        const double sa = ax ? 1.0 : -1.0, sb = bx ? 1.0 : -1.0, ta = ay ? 1.0 : -1.0, tb = by ? 1.0 : -1.0;
        const double x0 = k == 0 ? sb : 1.0, x1 = k == 0 ? (ax == bx ? 1.0 : -1.0) : ax == bx ? 2.0 * sa : 0.0,
                     x2 = k == 0 ? 0.0 : ax == bx ? 1.0 : -1.0;
        const double y0 = k == 1 ? tb : 1.0, y1 = k == 1 ? (ay == by ? 1.0 : -1.0) : ay == by ? 2.0 * ta : 0.0,
                     y2 = k == 1 ? 0.0 : ay == by ? 1.0 : -1.0;
        double v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double* q = mo + c * 9;
            const double a0 = fma(x2, q[2], fma(x1, q[1], x0 * q[0])), a1 = fma(x2, q[5], fma(x1, q[4], x0 * q[3])),
                         a2 = fma(x2, q[8], fma(x1, q[7], x0 * q[6]));
            v[c] = scale * fma(y2, a2, fma(y1, a1, y0 * a0));
        }
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            const int az = z & 1, bz = z >> 1;
            const double sz = az ? 1.0 : -1.0, uz = bz ? 1.0 : -1.0;
            const double val = k == 2 ? fma(sz * uz, v[1], uz * v[0])
                                      : fma(sz * uz, v[2], fma(sz + uz, v[1], v[0]));
            M[ik * 72 + node_at(bx, by, bz) * 9 + node_at(ax, ay, az)] = val;
        }
    }
    __syncwarp();
    for (int t = lane; t < 576; t += 32) {
        const int fg = t >> 6, f = fg / 3, g = fg - 3 * f, b = t >> 3 & 7, a = t & 7, at = b * 9 + a;
        double v = fma(p.lam_c, M[fg * 72 + at], p.mu_c * M[(g * 3 + f) * 72 + at]);
        if (f == g) v = fma(p.mu_c, M[at] + M[4 * 72 + at] + M[8 * 72 + at], v);
        X[fg * 72 + at] = v;
    }
    for (int t = lane; t < 64; t += 32) X[kIfX + (t >> 3) * 9 + (t & 7)] = M[9 * 72 + (t >> 3) * 9 + (t & 7)];
    __syncwarp();
}
struct InterfaceCoef {
    double c1, c2, cg;
};
__device__ InterfaceCoef interface_coef(const BrickArgs& p, int64_t e, double area, int s, int s2, double scale) {
    // w = (V/E) / (V_L/E_L + V_F/E_F) over a common denominator
    const double EL = p.E[e], EF = p.EF[e], vl = p.vol[2 * e] * EF, vf = p.vol[2 * e + 1] * EL;
    const double inv = 1.0 / (vl + vf), wl = vl * inv, wf = vf * inv;
    const double gamma = 2.0 * p.alpha * area * (EL * EF * inv);
    InterfaceCoef c;
    c.c1 = (s ? scale : -scale) * (s2 ? wf * EF : wl * EL);
    c.c2 = p.beta * (s2 ? -scale : scale) * (s ? wf * EF : wl * EL);
    c.cg = s == s2 ? scale * gamma : -scale * gamma;
    return c;
}
__device__ __forceinline__ void interface_block(const InterfaceCoef& c, const double* X, int a, int b, double K[9]) {
    const double q = c.cg * X[kIfX + b * 9 + a];
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const double x1 = X[((f * 3 + g) * 8 + b) * 9 + a], x2 = X[((g * 3 + f) * 8 + a) * 9 + b];
            K[f * 3 + g] = fma(c.c2, x2, f == g ? fma(c.c1, x1, q) : c.c1 * x1);
        }
}

// ---------------------------------------------------------------------------
// boundary facet: the Nitsche terms of IWG_Isotropic_Struc_Linear_Dirichlet with
// M = I (..._Dirichlet.cpp:52-240).  On a brick face n = +-e_k, and with
// I_i(a, b) = integral N_a dN_b/dx_i, NN(a, b) = integral N_a N_b (w* includes the
// thickness) the traction of column b has the entries
//   T(k, k) = (lam + 2 mu) n I_k,  T(t, t) = mu n I_k,  T(k, t) = lam n I_t,
//   T(t, k) = mu n I_t,
// K = -T(a, b) + beta T(b, a)^T + gamma NN, gamma = alpha E / h, h = sqrt(4 A / pi).  A
// constant displacement has no traction, so the residual is K (u - g); the
// Neumann residual is -t integral N_a.
// Bound by the atomics of the 24 x 24 blocks, a warp per facet: with the general
// side kernel (a CTA per facet, operators per point) the two faces of 9,216 facets
// of a 96^3 density model cost 231 us more: 3563 -> 3332 us for its assembly.
struct SideCoef {
    int k;
    double kk, tt, lam[3], mu[3], nn;  // scales of I_k, I_k, I_t, I_t, NN
};
__device__ SideCoef side_coef(const BrickArgs& p, int64_t e, int ord, int lane) {
    SideCoef c;
    c.k = ord == 1 || ord == 3 ? 0 : ord == 0 || ord == 2 ? 1 : 2;
    const bool up = ord == 1 || ord == 2 || ord == 5;
    const double* X = p.xe + e * 24;
    const double j = 0.5 * (X[18 + lane % 3] - X[lane % 3]), r = 1.0 / j;
    const double area = shfl(j, c.k == 0 ? 1 : 0) * shfl(j, c.k == 2 ? 1 : 2);  // detJ of the face
    const double E = p.E[e], w = area * p.thickness;
    const double s = up ? w * E : -w * E;
    const double rk = shfl(r, c.k);
    c.kk = (p.lam_c + 2.0 * p.mu_c) * s * rk;
    c.tt = p.mu_c * s * rk;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const double ri = s * shfl(r, i);
        c.lam[i] = p.lam_c * ri;
        c.mu[i] = p.mu_c * ri;
    }
    c.nn = p.neumann ? w : p.alpha * E * w / sqrt(16.0 * area / 3.14159265358979323846);
    return c;
}
__device__ __forceinline__ void side_block(const SideCoef& c, const double* tab, double beta, int a, int b,
                                           double K[9]) {
    double ab[3], ba[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        ab[i] = __ldg(tab + i * 64 + b * 8 + a);
        ba[i] = beta * __ldg(tab + i * 64 + a * 8 + b);
    }
    const double ik = c.k == 0 ? ab[0] : c.k == 1 ? ab[1] : ab[2], jk = c.k == 0 ? ba[0] : c.k == 1 ? ba[1] : ba[2];
    const double nn = c.nn * __ldg(tab + 192 + b * 8 + a);
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            double v = 0.0;
            if (f == g) v = fma(f == c.k ? c.kk : c.tt, jk - ik, nn);
            else if (f == c.k) v = fma(c.mu[g], ba[g], -c.lam[g] * ab[g]);
            else if (g == c.k) v = fma(c.lam[f], ba[f], -c.mu[f] * ab[f]);
            K[f * 3 + g] = v;
        }
}

template <int KIND>
__host__ __device__ constexpr int warp_doubles() {
    return KIND == KIND_UNCUT       ? 64
           : KIND == KIND_CUT       ? 32 * kPt + 64
           : KIND == KIND_INTERFACE ? kIfSmem
                                    : 2;
}

// ---------------------------------------------------------------------------
// Linear splines: one warp per equation object.
template <int KIND>
__host__ __device__ constexpr int warps_of() {
    return KIND == KIND_INTERFACE ? 2 : 4;  // 12 KB of shared memory per interface warp
}

template <int KIND>
__global__ void __launch_bounds__(32 * warps_of<KIND>()) brick_linear(BrickArgs p) {
    constexpr int WD = warp_doubles<KIND>(), kWarps = warps_of<KIND>();
    __shared__ double sm[kWarps * WD];
    __shared__ uint8_t gt[576];
    const int lane = threadIdx.x & 31;
    double* ws = sm + (threadIdx.x >> 5) * WD;
    if (KIND <= KIND_CUT) {
        build_gram_table(gt);
        __syncthreads();
    }
    const int64_t w = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
    if (w >= p.n) return;
    const int64_t e = p.list[w];
    constexpr int SIDES = sides_of(KIND);
    // lane -> row node and the columns it takes: bulk (a, pair of b), double
    // (side, a, other side) with all eight b
    const int s = SIDES == 1 ? 0 : lane >> 4, s2 = SIDES == 1 ? 0 : lane & 1;
    const int a = SIDES == 1 ? lane >> 2 : lane >> 1 & 7;
    const int b0 = SIDES == 1 ? (lane & 3) * 2 : 0, nb = SIDES == 1 ? 2 : 8;
    const int64_t ro = (e * SIDES + s) * 8;
    const int col = p.map[ro + a], basis = p.bases[ro + col];
    Scatter sc;
    sc.vals = p.vals;
    sc.ul = __ldg(p.ulen + basis);
    double ua[3] = {0.0, 0.0, 0.0}, r[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        sc.row[f] = __ldg(p.rowptr + f * p.nu + basis);
        if (p.u) ua[f] = __ldg(p.u + f * p.nu + basis);
    }
    const uint16_t* si = p.sidx + ((e * SIDES + s) * 8 + col) * (8 * SIDES) + s2 * 8;
    double area = 0.0;
    if (KIND == KIND_UNCUT) uncut_sums(p, e, ws, lane);
    if (KIND == KIND_CUT) cut_sums(p, e, ws, ws + 32 * kPt, lane);
    if (KIND == KIND_INTERFACE) interface_matrices(p, e, ws, area, lane);
    __syncwarp();
    GhostCoef gc;
    InterfaceCoef ic;
    const double* gtab = nullptr;
    if (KIND == KIND_GHOST) {
        const int face = p.code[e] - kFastGhost;
        gc = ghost_coef(p, e, face, s, s2, 1.0);
        gtab = p.tab + face * kGhostTab;
    }
    if (KIND == KIND_INTERFACE) ic = interface_coef(p, e, area, s, s2, 1.0);
    SideCoef sd;
    if (KIND == KIND_SIDE) {
        const int ord = p.code[e] - kFastSide;
        sd = side_coef(p, e, ord, lane);
        gtab = p.tab + ord * kSideTab;
        for (int f = 0; f < 3; ++f) ua[f] -= p.value[f];
    }
    const double ld = (p.lam_c + p.mu_c) / p.mu_c, lo = p.lam_c / p.mu_c;
#pragma unroll 2
    for (int t = 0; t < nb; ++t) {
        const int b = b0 + t;
        double K[9];
        if (KIND == KIND_UNCUT) bulk_block(ws, gt, a, b, ld, lo, K);
        if (KIND == KIND_CUT) bulk_block(ws + 32 * kPt, gt, a, b, ld, lo, K);
        if (KIND == KIND_GHOST) ghost_block(gc, gtab, b, lane, p.normal_field, K);
        if (KIND == KIND_INTERFACE) interface_block(ic, ws, a, b, K);
        if (KIND == KIND_SIDE) {
            if (p.neumann) {
                const double nn = sd.nn * __ldg(gtab + 192 + b * 8 + a);
                for (int f = 0; f < 3; ++f) r[f] = fma(-nn, p.value[f], r[f]);
                continue;
            }
            side_block(sd, gtab, p.beta, a, b, K);
        }
        // the lane that holds column node b (of side s2)
        const int src = SIDES == 1 ? b * 4 : s2 * 16 + b * 2;
        const int cb = __shfl_sync(0xffffffffu, col, src);
        if (p.rhs) {
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                const double ug = shfl(ua[g], src);
#pragma unroll
                for (int f = 0; f < 3; ++f) r[f] = fma(K[f * 3 + g], ug, r[f]);
            }
        }
        if (p.vals) sc.add(K, si[cb]);
    }
    if (p.rhs) {
        // over the lanes of one row node
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            r[f] += __shfl_xor_sync(0xffffffffu, r[f], 1);
            if (SIDES == 1) r[f] += __shfl_xor_sync(0xffffffffu, r[f], 2);
        }
        const int q = SIDES == 1 ? lane & 3 : lane & 1;
        if (SIDES == 1 && q < 3) atomicAdd(p.rhs + q * p.nu + basis, q == 0 ? r[0] : q == 1 ? r[1] : r[2]);
        if (SIDES == 2) {
            atomicAdd(p.rhs + q * p.nu + basis, q ? r[1] : r[0]);
            if (q == 0) atomicAdd(p.rhs + 2 * p.nu + basis, r[2]);
        }
    }
    if (sc.bad) atomicOr(p.status, 1);
}

// ---------------------------------------------------------------------------
// Quadratic splines: one CTA per equation object.  K / 64 (pdof, 24 or 48 rows)
// by the first warp; then K P axis by axis (8 node values -> 27 bases, 19
// additions) and P^T (K P) the same way along the rows, scattered as it is formed.
template <int KIND>
struct QuadLayout {
    static constexpr int SIDES = sides_of(KIND), NP = 24 * SIDES, NA = 81 * SIDES;
    static constexpr int K = 0, KT = K + NP * NP, R = KT + NP * NA, WS = R + NP, END = WS + warp_doubles<KIND>();
    static constexpr size_t bytes = (size_t)END * 8 + 576 + SIDES * (27 + 27 * 4 * 4) + 64 +
                                    (size_t)(27 * SIDES) * (27 * SIDES) * 2;
};

template <int KIND>
__global__ void __launch_bounds__(128) brick_quadratic(BrickArgs p) {
    using L = QuadLayout<KIND>;
    constexpr int SIDES = L::SIDES, NP = L::NP, NA = L::NA, NB = 27 * SIDES, NT = 128;
    extern __shared__ double sm[];
    double* K = sm + L::K;
    double* KT = sm + L::KT;
    double* R = sm + L::R;
    double* ws = sm + L::WS;
    int32_t* row = reinterpret_cast<int32_t*>(sm + L::END);  // [basis][3] CSR row starts, basis in code order
    int32_t* ul = row + 3 * NB;
    uint16_t* S = reinterpret_cast<uint16_t*>(ul + NB);       // [row code][column code]
    uint8_t* nat = reinterpret_cast<uint8_t*>(S + NB * NB);   // column of a code
    uint8_t* gt = nat + NB;
    const int tid = threadIdx.x, lane = tid & 31;
    const int64_t e = p.list[blockIdx.x];
    if (KIND <= KIND_CUT) build_gram_table(gt);
    for (int j = tid; j < NB; j += NT) {
        const int s = j / 27, c = p.map[e * NB + j];
        nat[j] = (uint8_t)c;
        const int basis = p.bases[e * NB + s * 27 + c];
        ul[j] = __ldg(p.ulen + basis);
        for (int f = 0; f < 3; ++f) row[j * 3 + f] = __ldg(p.rowptr + f * p.nu + basis);
    }
    __syncthreads();
    if (p.vals)
        for (int k = tid; k < NB * NB; k += NT) {
            const int i = k / NB, j = k - i * NB;
            S[k] = p.sidx[e * NB * NB + ((i / 27) * 27 + nat[i]) * NB + (j / 27) * 27 + nat[j]];
        }
    if (tid < 32) {
        const int s = SIDES == 1 ? 0 : lane >> 4, s2 = SIDES == 1 ? 0 : lane & 1;
        const int a = SIDES == 1 ? lane >> 2 : lane >> 1 & 7;
        const int b0 = SIDES == 1 ? (lane & 3) * 2 : 0, nb = SIDES == 1 ? 2 : 8;
        // nodal displacements: 1/8 of the sum over the node's eight bases
        double ua[3] = {0.0, 0.0, 0.0}, r[3] = {0.0, 0.0, 0.0};
        if (p.u)
            for (int q = 0; q < 8; ++q) {
                const int code =
                    corner(a, 0) + (q & 1) + 3 * (corner(a, 1) + (q >> 1 & 1)) + 9 * (corner(a, 2) + (q >> 2));
                const int basis = p.bases[e * NB + s * 27 + nat[s * 27 + code]];
                for (int f = 0; f < 3; ++f) ua[f] += __ldg(p.u + f * p.nu + basis);
            }
        for (int f = 0; f < 3; ++f) ua[f] *= 0.125;
        double area = 0.0;
        if (KIND == KIND_UNCUT) uncut_sums(p, e, ws, lane);
        if (KIND == KIND_CUT) cut_sums(p, e, ws, ws + 32 * kPt, lane);
        if (KIND == KIND_INTERFACE) interface_matrices(p, e, ws, area, lane);
        __syncwarp();
        GhostCoef gc;
        InterfaceCoef ic;
        const double* gtab = nullptr;
        if (KIND == KIND_GHOST) {
            const int face = p.code[e] - kFastGhost;
            gc = ghost_coef(p, e, face, s, s2, 1.0 / 64.0);
            gtab = p.tab + face * kGhostTab;
        }
        if (KIND == KIND_INTERFACE) ic = interface_coef(p, e, area, s, s2, 1.0 / 64.0);
        const double ld = (p.lam_c + p.mu_c) / p.mu_c, lo = p.lam_c / p.mu_c;
        for (int t = 0; t < nb; ++t) {
            const int b = b0 + t;
            double B[9];
            if (KIND <= KIND_CUT) {
                bulk_block(KIND == KIND_UNCUT ? ws : ws + 32 * kPt, gt, a, b, ld, lo, B);
                for (int k = 0; k < 9; ++k) B[k] *= 1.0 / 64.0;
            }
            if (KIND == KIND_GHOST) ghost_block(gc, gtab, b, lane, p.normal_field, B);
            if (KIND == KIND_INTERFACE) interface_block(ic, ws, a, b, B);
            const int src = SIDES == 1 ? b * 4 : s2 * 16 + b * 2;
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                const double ug = shfl(ua[g], src);
#pragma unroll
                for (int f = 0; f < 3; ++f) {
                    r[f] = fma(B[f * 3 + g], ug, r[f]);
                    // stored transposed: the lanes of the projection take rows
                    K[(s2 * 24 + g * 8 + b) * NP + s * 24 + f * 8 + a] = B[f * 3 + g];
                }
            }
        }
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            r[f] += __shfl_xor_sync(0xffffffffu, r[f], 1);
            if (SIDES == 1) r[f] += __shfl_xor_sync(0xffffffffu, r[f], 2);
            R[s * 24 + f * 8 + a] = r[f];
        }
    }
    __syncthreads();
    if (p.rhs)
        for (int t = tid; t < NA; t += NT) {
            // basis (side, code), component f: 8 = 64 / 8 times the nodes of its pattern
            const int f = t / NB, j = t - f * NB, s = j / 27, c = j - s * 27, c0 = c % 3, c1 = c / 3 % 3, c2 = c / 9;
            double v = 0.0;
            for (int q = 0; q < 8; ++q) {
                const int x = q & 1, y = q >> 1 & 1, z = q >> 2;
                if ((c0 == 1 || c0 == 2 * x) && (c1 == 1 || c1 == 2 * y) && (c2 == 1 || c2 == 2 * z))
                    v += R[s * 24 + f * 8 + node_at(x, y, z)];
            }
            atomicAdd(p.rhs + f * p.nu + p.bases[e * NB + s * 27 + nat[j]], 8.0 * v);
        }
    if (!p.vals) return;
    // K P: thread (row r, column block (s, g), y code): y stage, then x and z
    for (int t = tid; t < NP * 9 * SIDES; t += NT) {
        const int r = t % NP, k = t / NP, sg = k / 3, jy = k - 3 * sg;
        double w[2][2];
#pragma unroll
        for (int bz = 0; bz < 2; ++bz)
#pragma unroll
            for (int bx = 0; bx < 2; ++bx) {
                const double v0 = K[(sg * 8 + node_at(bx, 0, bz)) * NP + r];
                const double v1 = K[(sg * 8 + node_at(bx, 1, bz)) * NP + r];
                w[bx][bz] = jy == 0 ? v0 : jy == 2 ? v1 : v0 + v1;
            }
#pragma unroll
        for (int jx = 0; jx < 3; ++jx) {
            const double u0 = jx == 0 ? w[0][0] : jx == 2 ? w[1][0] : w[0][0] + w[1][0];
            const double u1 = jx == 0 ? w[0][1] : jx == 2 ? w[1][1] : w[0][1] + w[1][1];
            double* o = KT + r * NA + sg * 27 + jx + 3 * jy;
            o[0] = u0;
            o[9] = u0 + u1;
            o[18] = u1;
        }
    }
    __syncthreads();
    // P^T (K P): thread (column c, row block (s, f), y code), scattered at once;
    // zero blocks of the ghost penalty (two tangent components) are skipped
    bool bad = false;
    for (int t = tid; t < NA * 9 * SIDES; t += NT) {
        const int c = t % NA, k = t / NA, sf = k / 3, iy = k - 3 * sf, s = sf / 3, f = sf - 3 * s;
        const int sg = c / 27, j = (sg / 3) * 27 + c - sg * 27, g = sg % 3;
        if (KIND == KIND_GHOST && f != g) {
            const int ax = (p.code[e] - kFastGhost) >> 1;
            if (p.normal_field || (f != ax && g != ax)) continue;
        }
        double w[2][2];
#pragma unroll
        for (int bz = 0; bz < 2; ++bz)
#pragma unroll
            for (int bx = 0; bx < 2; ++bx) {
                const double v0 = KT[(sf * 8 + node_at(bx, 0, bz)) * NA + c];
                const double v1 = KT[(sf * 8 + node_at(bx, 1, bz)) * NA + c];
                w[bx][bz] = iy == 0 ? v0 : iy == 2 ? v1 : v0 + v1;
            }
#pragma unroll
        for (int ix = 0; ix < 3; ++ix) {
            const double u0 = ix == 0 ? w[0][0] : ix == 2 ? w[1][0] : w[0][0] + w[1][0];
            const double u1 = ix == 0 ? w[0][1] : ix == 2 ? w[1][1] : w[0][1] + w[1][1];
            const double v[3] = {u0, u0 + u1, u1};
#pragma unroll
            for (int iz = 0; iz < 3; ++iz) {
                const int i = s * 27 + ix + 3 * iy + 9 * iz;
                bad |= !fem_finite(v[iz]);
                atomicAdd(p.vals + row[i * 3 + f] + g * ul[i] + S[i * NB + j], v[iz]);
            }
        }
    }
    if (bad) atomicOr(p.status, 1);
}

// ---------------------------------------------------------------------------
// host side
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
    if (e == cudaSuccess && !v.empty())
        e = cudaMemcpyAsync(b.p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st);
    return e;
}

// column map of one side's extraction T [8][width] (nb columns): linear: column
// of every node (one basis of weight 1 each); quadratic: column of every code
// (x + 3 y + 9 z, 0 left node only, 1 both, 2 right only), weights 1/8
bool extraction_map(const double* T, int width, int nb, uint8_t* map) {
    if (nb == 8) {
        bool used[8] = {};
        for (int a = 0; a < 8; ++a) {
            int col = -1;
            for (int j = 0; j < 8; ++j) {
                const double t = T[a * width + j];
                if (t == 0.0) continue;
                if (t != 1.0 || col >= 0) return false;
                col = j;
            }
            if (col < 0 || used[col]) return false;
            used[col] = true;
            map[a] = (uint8_t)col;
        }
        return true;
    }
    if (nb != 27) return false;
    bool have[27] = {};
    for (int j = 0; j < 27; ++j) {
        unsigned mask = 0;
        for (int a = 0; a < 8; ++a) {
            const double t = T[a * width + j];
            if (t == 0.0) continue;
            if (t != 0.125) return false;
            mask |= 1u << a;
        }
        int code = 0, mul = 1;
        unsigned expect = 0xff;
        for (int d = 0; d < 3; ++d, mul *= 3) {
            unsigned lo = 0;
            for (int a = 0; a < 8; ++a)
                if (!corner(a, d)) lo |= 1u << a;
            const unsigned up = ~lo & 0xff;
            const int c = (mask & lo) ? ((mask & up) ? 1 : 0) : 2;
            expect &= c == 0 ? lo : c == 2 ? up : 0xff;
            code += c * mul;
        }
        if (!mask || mask != expect || have[code]) return false;
        have[code] = true;
        map[code] = (uint8_t)j;
    }
    return true;
}

bool brick(const double* xe) {
    for (int d = 0; d < 3; ++d)
        if (!(xe[18 + d] > xe[d])) return false;
    for (int a = 0; a < 8; ++a)
        for (int d = 0; d < 3; ++d)
            if (xe[a * 3 + d] != (corner(a, d) ? xe[18 + d] : xe[d])) return false;
    return true;
}

// whole-face ghost: 2 axis + (leader side up), or -1
int ghost_face(const SetData& s, int64_t i) {
    if (s.nfv != 4 || s.fc_off[i + 1] - s.fc_off[i] != 1) return -1;
    const double* l = &s.fc_xl[s.fc_off[i] * 12];
    const double* f = &s.fc_xf[s.fc_off[i] * 12];
    const double* x = &s.fc_x[s.fc_off[i] * 12];
    const double* X = &s.xe[i * 48];
    for (int k = 0; k < 3; ++k) {
        if (std::abs(l[k]) != 1.0 || l[3 + k] != l[k] || l[6 + k] != l[k] || l[9 + k] != l[k]) continue;
        bool ok = true;
        int corners = 0, last = -1;
        for (int v = 0; v < 4 && ok; ++v) {
            int bit = 0, m = 1;
            for (int d = 0; d < 3; ++d) {
                const double xl = l[v * 3 + d], xf = f[v * 3 + d];
                ok &= std::abs(xl) == 1.0 && xf == (d == k ? -xl : xl);
                // the vertex is the corner of both cells
                ok &= x[v * 3 + d] == X[(xl > 0.0 ? 18 : 0) + d] && x[v * 3 + d] == X[24 + (xf > 0.0 ? 18 : 0) + d];
                if (d != k) {
                    bit += xl > 0.0 ? m : 0;
                    m *= 2;
                }
            }
            corners |= 1 << bit;
            // neighbours around the facet differ in one coordinate (a bow-tie has zero measure)
            if (last >= 0) ok &= (bit ^ last) == 1 || (bit ^ last) == 2;
            last = bit;
        }
        if (ok && corners == 15) return 2 * k + (l[k] > 0.0);
    }
    return -1;
}

}  // namespace

void brick_classify(const fem_gpu_ctx* c, SetData& s) {
    s.fast.clear();
    s.fmap.clear();
    s.fgeo.clear();
    const int sides = s.kind == 2 ? 2 : 1;
    if (c->dim != 3 || c->shape != FEM_GPU_SHAPE_RECTANGULAR || s.neq == 0) return;
    if (!s.node_rho.empty()) return;
    const int W = s.maxnb;
    if (s.kind == 1) {
        // boundary facets: linear splines, the whole projection
        if (W != 8 || s.side.integration_rule != FEM_GPU_RULE_QUAD_2x2) return;
        for (int k = 0; k < 9; ++k)
            if (s.side_select[k] != (k % 4 ? 0.0 : 1.0)) return;
    }
    if ((W != 8 && W != 27) || (s.kind == 0 && s.bulk.model_type != FEM_GPU_MODEL_3D)) return;
    if (s.kind == 0 && !s.ig_off.empty() && s.bulk.ig_cell_type != FEM_GPU_CELL_TET4) return;
    const bool iface = s.kind == 2 && !is_ghost_iwg(s.dside.iwg_type);
    if (iface && (s.nfv != 3 || gauss_rule(s.dside.integration_rule).n > 7)) return;
    s.fast.assign(s.neq, 0);
    s.fmap.assign((size_t)s.neq * sides * W, 0);
    const int geo = s.kind == 0 && s.ig_off.empty() ? kGeoUncut : s.kind == 2 && !iface ? kGeoGhost : 0;
    s.fgeo.assign((size_t)s.neq * geo, 0.0);
    const auto classify = [&](int64_t i) {
        bool ok = true;
        for (int k = 0; k < sides && ok; ++k) {
            const int64_t r = i * sides + k;
            ok = s.nb[r] == W && brick(&s.xe[r * 24]) && extraction_map(&s.T[r * 8 * W], W, W, &s.fmap[r * W]);
        }
        if (!ok) return;
        if (s.kind == 1) {
            s.fast[i] = (uint8_t)(kFastSide + s.ordinal[i]);
        } else if (s.kind == 0) {
            s.fast[i] = kFastBulk;
            for (int d = 0; !s.fgeo.empty() && d < 3; ++d)
                s.fgeo[i * kGeoUncut + d] = 1.0 / (0.5 * (s.xe[i * 24 + 18 + d] - s.xe[i * 24 + d]));
        } else if (iface) {
            const int64_t a = s.fc_off[i] * 9, b = s.fc_off[i + 1] * 9;
            if (std::equal(&s.xe[i * 48], &s.xe[i * 48] + 24, &s.xe[i * 48] + 24) &&
                std::equal(s.fc_xl.begin() + a, s.fc_xl.begin() + b, s.fc_xf.begin() + a))
                s.fast[i] = kFastInterface;
        } else {
            const int face = ghost_face(s, i);
            if (face < 0) return;
            s.fast[i] = (uint8_t)(kFastGhost + face);
            const double* X = &s.xe[i * 48];
            double* g = &s.fgeo[i * kGeoGhost];
            for (int q = 0; q < 6; ++q) g[q] = 2.0 / (X[(q / 3) * 24 + 18 + q % 3] - X[(q / 3) * 24 + q % 3]);
            const int k = face >> 1, t1 = k == 0 ? 1 : 0, t2 = k == 2 ? 1 : 2;
            g[7] = 0.25 * (X[18 + t1] - X[t1]) * (X[18 + t2] - X[t2]);
            g[6] = std::sqrt(16.0 * g[7] / 3.14159265358979323846);
        }
    };
    const int nt = (int)std::min<int64_t>(std::max(1u, std::thread::hardware_concurrency()), 1 + s.neq / 4096);
    std::vector<std::thread> th;
    for (int t = 0; t < nt; ++t)
        th.emplace_back([&, t] {
            for (int64_t i = s.neq * t / nt; i < s.neq * (t + 1) / nt; ++i) classify(i);
        });
    for (auto& t : th) t.join();
    if (std::none_of(s.fast.begin(), s.fast.end(), [](uint8_t f) { return f != 0; })) {
        s.fast.clear();
        s.fmap.clear();
        s.fgeo.clear();
    }
}

fem_gpu_status brick_upload(fem_gpu_ctx* c, SetData& s) {
    if (s.fast.empty()) return FEM_GPU_OK;
    cudaStream_t st = (cudaStream_t)c->stream;
    s.flist.clear();
    for (int64_t i = 0; i < s.neq; ++i)
        if (s.fast[i]) s.flist.push_back((int32_t)i);
    std::vector<double> tab;
    if (s.kind == 0 && s.ig_off.empty()) {
        // reference sums of the rule
        const Rule r = gauss_rule(s.bulk.integration_rule);
        for (int i = 0; i < 3; ++i)
            for (int j = i; j < 3; ++j) {
                const int n[3] = {axis_sums(i, j, 0), axis_sums(i, j, 1), axis_sums(i, j, 2)};
                tab.resize(kSums);
                for (int t = 0; t < n[0] * n[1] * n[2]; ++t) {
                    const int v[3] = {t / (n[1] * n[2]), t / n[2] % n[1], t % n[2]};
                    double sum = 0.0;
                    for (int q = 0; q < r.n; ++q) {
                        double f = r.w[q] / 64.0;
                        for (int d = 0; d < 3; ++d) {
                            const double x = r.pts[q * 3 + d];
                            f *= n[d] == 1   ? 1.0
                                 : n[d] == 2 ? (v[d] ? 1.0 - x : 1.0 + x)
                                 : v[d] == 0 ? (1.0 + x) * (1.0 + x)
                                 : v[d] == 1 ? (1.0 - x) * (1.0 - x)
                                             : (1.0 + x) * (1.0 - x);
                        }
                        sum += f;
                    }
                    tab[pair_off(i, j) + t] = sum;
                }
            }
    } else if (s.kind == 1) {
        const Rule r = gauss_rule(s.side.integration_rule);
        tab.assign((size_t)6 * kSideTab, 0.0);
        for (int o = 0; o < 6; ++o) {
            const int k = o == 1 || o == 3 ? 0 : o == 0 || o == 2 ? 1 : 2, t1 = k == 0 ? 1 : 0, t2 = k == 2 ? 1 : 2;
            for (int q = 0; q < r.n; ++q) {
                double xi[3], N[8], dN[24];
                xi[k] = o == 1 || o == 2 || o == 5 ? 1.0 : -1.0;
                xi[t1] = r.pts[q * 2];
                xi[t2] = r.pts[q * 2 + 1];
                lagrange(FEM_GPU_CELL_HEX8, xi, N, dN);
                for (int b = 0; b < 8; ++b)
                    for (int a = 0; a < 8; ++a) {
                        double* t = &tab[(size_t)o * kSideTab + b * 8 + a];
                        for (int i = 0; i < 3; ++i) t[i * 64] += r.w[q] * N[a] * dN[i * 8 + b];
                        t[192] += r.w[q] * N[a] * N[b];
                    }
            }
        }
    } else if (s.kind == 2 && is_ghost_iwg(s.dside.iwg_type)) {
        const Rule r = gauss_rule(s.dside.integration_rule);
        tab.assign((size_t)6 * kGhostTab, 0.0);
        for (int face = 0; face < 6; ++face) {
            const int k = face >> 1, t1 = k == 0 ? 1 : 0, t2 = k == 2 ? 1 : 2;
            const int ij[kGhostMats][2] = {{k, k}, {t1, t1}, {t2, t2}, {k, t1}, {k, t2}, {t1, k}, {t2, k}};
            for (int q = 0; q < r.n; ++q) {
                double N[2][8], dN[2][24];
                for (int sd = 0; sd < 2; ++sd) {
                    double xi[3];
                    xi[k] = (face & 1) == (sd == 0) ? 1.0 : -1.0;
                    xi[t1] = r.pts[q * 2];
                    xi[t2] = r.pts[q * 2 + 1];
                    lagrange(FEM_GPU_CELL_HEX8, xi, N[sd], dN[sd]);
                }
                for (int m = 0; m < kGhostMats; ++m)
                    for (int b = 0; b < 8; ++b)
                        for (int lane = 0; lane < 32; ++lane)
                            tab[(size_t)face * kGhostTab + m * 256 + b * 32 + lane] +=
                                r.w[q] * dN[lane >> 4][ij[m][0] * 8 + (lane >> 1 & 7)] * dN[lane & 1][ij[m][1] * 8 + b];
            }
        }
    }
    // tables, reciprocals, list, kinds and maps in one buffer
    s.ftab_count = tab.size();
    tab.insert(tab.end(), s.fgeo.begin(), s.fgeo.end());
    s.fgeo.clear();
    s.fgeo.shrink_to_fit();
    const size_t nt = tab.size() * sizeof(double), nl = s.flist.size() * sizeof(int32_t);
    std::vector<uint8_t> all(nt + nl + s.fast.size() + s.fmap.size());
    if (nt) std::memcpy(all.data(), tab.data(), nt);
    std::memcpy(all.data() + nt, s.flist.data(), nl);
    std::memcpy(all.data() + nt + nl, s.fast.data(), s.fast.size());
    std::memcpy(all.data() + nt + nl + s.fast.size(), s.fmap.data(), s.fmap.size());
    s.ftab_bytes = nt;
    cudaError_t e = upload(s.d_fast, all, st);
    if (e == cudaErrorMemoryAllocation) {  // the general kernels need none of it
        cudaGetLastError();
        s.fast.clear();
        s.fmap.clear();
        s.flist.clear();
        return FEM_GPU_OK;
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? FEM_GPU_OK
                            : fail(c, FEM_GPU_CUDA_ERROR, std::string("brick data: ") + cudaGetErrorString(e));
}

void brick_release(SetData& s) {
    dfree(s.d_fast);
}

int64_t brick_count(const SetData& s, int64_t first, int64_t count) {
    if (s.fast.empty()) return 0;
    const auto lo = std::lower_bound(s.flist.begin(), s.flist.end(), first);
    return std::lower_bound(lo, s.flist.end(), first + count) - lo;
}

fem_gpu_status brick_launch(fem_gpu_ctx* c, const SetData& s, int64_t first, int64_t count, const double* u,
                            double* vals, double* rhs, void* stream) {
    const int64_t n = brick_count(s, first, count);
    if (n == 0) return FEM_GPU_OK;
    cudaStream_t st = (cudaStream_t)stream;
    BrickArgs a{};
    a.n = n;
    const uint8_t* data = (const uint8_t*)s.d_fast.p;
    a.list = (const int32_t*)(data + s.ftab_bytes) +
             (std::lower_bound(s.flist.begin(), s.flist.end(), first) - s.flist.begin());
    a.code = data + s.ftab_bytes + s.flist.size() * sizeof(int32_t);
    a.map = a.code + s.fast.size();
    a.xe = (const double*)s.d_xe.p;
    a.E = (const double*)s.d_E.p;
    a.bases = (const int32_t*)s.d_bases.p;
    a.sidx = (const uint16_t*)s.d_sidx.p;
    a.gp = (const double*)s.d_gp.p;
    a.gw = (const double*)s.d_gw.p;
    a.ngp = s.ngp;
    a.tab = (const double*)data;
    a.geo = a.tab + s.ftab_count;
    a.rowptr = (const int32_t*)c->d_rowptr.p;
    a.ulen = (const int32_t*)c->d_ulen.p;
    a.nu = c->num_used;
    a.u = u;
    a.vals = vals;
    a.rhs = rhs;
    a.status = (int*)c->d_status.p;
    const double nu = s.kind == 0   ? s.bulk.poisson_ratio
                      : s.kind == 1 ? s.side.poisson_ratio
                                    : s.dside.poisson_ratio;
    a.lam_c = nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
    a.mu_c = 1.0 / (2.0 * (1.0 + nu));
    int kind = KIND_UNCUT;
    if (s.kind == 0) {
        if (!s.ig_off.empty()) kind = KIND_CUT;
        a.off = (const int64_t*)s.d_igoff.p;
        a.x = (const double*)s.d_igx.p;
        a.xi = (const double*)s.d_igxi.p;
    } else if (s.kind == 1) {
        kind = KIND_SIDE;
        a.neumann = s.side.iwg_type == FEM_GPU_IWG_STRUC_LINEAR_NEUMANN;
        a.beta = s.side.iwg_type == FEM_GPU_IWG_STRUC_LINEAR_DIRICHLET_SYMMETRIC_NITSCHE ? -1.0 : 1.0;
        a.alpha = s.side.nitsche_alpha;
        a.thickness = s.side_thickness;
        for (int d = 0; d < 3; ++d) a.value[d] = s.side.value[d];
        if (a.neumann) a.vals = nullptr;  // K = 0
    } else {
        kind = is_ghost_iwg(s.dside.iwg_type) ? KIND_GHOST : KIND_INTERFACE;
        a.normal_field = s.dside.iwg_type == FEM_GPU_IWG_GHOST_NORMAL_FIELD;
        a.alpha = s.dside.alpha;
        a.beta = s.dside.iwg_type == FEM_GPU_IWG_STRUC_LINEAR_INTERFACE_SYMMETRIC_NITSCHE ? -1.0 : 1.0;
        a.EF = (const double*)s.d_EF.p;
        a.off = (const int64_t*)s.d_fcoff.p;
        a.x = (const double*)s.d_fcx.p;
        a.xi = (const double*)s.d_fcxl.p;
        a.vol = (const double*)s.d_vol.p;
    }
    using Fn = void (*)(BrickArgs);
    cudaError_t e = cudaSuccess;
    if (s.maxnb == 8) {
        static const Fn fn[5] = {brick_linear<0>, brick_linear<1>, brick_linear<2>, brick_linear<3>, brick_linear<4>};
        const int w = kind == KIND_INTERFACE ? warps_of<KIND_INTERFACE>() : warps_of<KIND_UNCUT>();
        fn[kind]<<<(unsigned)((n + w - 1) / w), 32 * w, 0, st>>>(a);
    } else {
        static const Fn fn[4] = {brick_quadratic<0>, brick_quadratic<1>, brick_quadratic<2>, brick_quadratic<3>};
        static const size_t bytes[4] = {QuadLayout<0>::bytes, QuadLayout<1>::bytes, QuadLayout<2>::bytes,
                                        QuadLayout<3>::bytes};
        e = cudaFuncSetAttribute((const void*)fn[kind], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes[kind]);
        if (e == cudaSuccess) fn[kind]<<<(unsigned)n, 128, bytes[kind], st>>>(a);
    }
    c->launches++;
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? FEM_GPU_OK
                            : fail(c, FEM_GPU_CUDA_ERROR, std::string("brick launch: ") + cudaGetErrorString(e));
}

}  // namespace fem
