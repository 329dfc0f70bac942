// fem_hex.cuh -- hexahedra of any shape on a tensor lattice of nodes: element
// matrices, added to the 27-point block stencil of the nodes or to the CSR, and the
// element residual without a matrix.
//
// A warp takes one cell, with no barrier but its own.  Both kernels are bound by the
// FP64 pipe, where a warp instruction takes 16 cycles of the SM whatever its active
// lanes, so the work is laid out for few instructions:
//   * J at the N^3 tensor points: dX/dxi_i depends on the other two coordinates only,
//     9 N^2 values of a bilinear interpolation of edge vectors;
//   * the inverse and the gradients: a lane per point (27 points) or four (8 points);
//   * the Gram matrix A(a, b) = sum_q w* g_a g_b^T: a lane per pair a < b (28 of 32),
//     9 FMAs per point.  The diagonal blocks follow from the rows of K, which sum to
//     zero because the gradients of a point do, and so the residual is the sum of
//     K(a, b) (u_b - u_a);
//   * without a matrix: gradient of u, stress and nodal forces by the same
//     interpolation and its transpose.
// 27 points: 470 instructions per cell for the matrix, 190 for the residual alone.
// The element loop (fem_bulk_cta.cuh) spends a CTA with a barrier after every stage
// on a cell and projects every matrix to the splines; here the projection is done
// once per node.  12,558 cells with 27 points: 371 us; with all 64 pairs (lane =
// row node and two column nodes) and four lanes per point it was 654 us.
#pragma once

#include <cstdint>

#include "fem_bits.cuh"

namespace fem {

struct HexArgs {
    int ne[3], nn[3];
    int64_t pitch;         // x pitch of the stencil array
    const double* E;       // modulus per cell
    const double* xe;      // [cells][8][3]
    double xq[3], wq[27];  // 1-D points, weights (x fastest) times mu and a scale
    double ld, lo;         // (lam + mu) / mu, lam / mu
    const double* u;       // nodal displacements [3][nodes] (nullable: zero)
    double* r;             // nodal residual [3][nodes], added to (nullable)
    double* S;             // [27][9][nn2][nn1][pitch], added to
    double* vals;          // CSR values (linear splines: node = basis), added to
    const int32_t* rowptr;
    int* status;
};

enum { HEX_STENCIL = 0, HEX_CSR = 1 };
constexpr int kHexWarps = 4;

// HEX8 node: its side (0 lower, 1 upper) along axis d
__device__ __forceinline__ int hex_corner(int a, int d) {
    return d == 0 ? (a ^ a >> 1) & 1 : d == 1 ? a >> 1 & 1 : a >> 2;
}
__device__ __forceinline__ int hex_node(int x, int y, int z) { return 4 * z + (y ? 3 - x : x); }

struct HexCell {
    int64_t cell, nodes;
    int c0[3];
    __device__ __forceinline__ bool init(const HexArgs& p, int64_t n) {
        cell = n;
        nodes = (int64_t)p.nn[0] * p.nn[1] * p.nn[2];
        if (cell >= (int64_t)p.ne[0] * p.ne[1] * p.ne[2]) return false;
        const unsigned yz = (unsigned)cell / (unsigned)p.ne[0];
        c0[0] = (int)((unsigned)cell - yz * p.ne[0]);
        c0[1] = (int)(yz % p.ne[1]);
        c0[2] = (int)(yz / p.ne[1]);
        return true;
    }
    __device__ __forceinline__ int64_t node(const HexArgs& p, int a) const {
        return ((int64_t)(c0[2] + hex_corner(a, 2)) * p.nn[1] + c0[1] + hex_corner(a, 1)) * p.nn[0] + c0[0] +
               hex_corner(a, 0);
    }
};

// G[(i N^2 + jk) 3 + c]: dV_c / dxi_i at the points (j, k) of the two axes after i, of
// the nodal field V[a][c]; one warp
template <int N>
__device__ __forceinline__ void hex_gradients(const HexArgs& p, const double* V, double* G, int lane) {
    for (int v = lane; v < 9 * N * N; v += 32) {
        const int c = v % 3, jk = v / 3 % (N * N), i = v / (3 * N * N), j = jk / N, k = jk % N;
        double e[2][2];  // half the edge vectors along i, [side of axis i + 1][side of i + 2]
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int s1 = m >> 1, s2 = m & 1;
            const int lo = i == 0 ? hex_node(0, s1, s2) : i == 1 ? hex_node(s2, 0, s1) : hex_node(s1, s2, 0);
            const int hi = i == 0 ? hex_node(1, s1, s2) : i == 1 ? hex_node(s2, 1, s1) : hex_node(s1, s2, 1);
            e[s1][s2] = V[hi * 3 + c] - V[lo * 3 + c];
        }
        const double tj = 0.5 + 0.5 * p.xq[j], tk = 0.5 + 0.5 * p.xq[k];
        const double a = fma(tj, e[1][0] - e[0][0], e[0][0]), b = fma(tj, e[1][1] - e[0][1], e[0][1]);
        G[v] = 0.5 * fma(tk, b - a, a);
    }
}

// cofactors of J at point (q0, q1, q2) (the inverse transposed times det) and det
template <int N>
__device__ __forceinline__ double hex_cofactors(const double* G, const int q[3], double C[3][3]) {
    double J[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) J[i][c] = G[(i * N * N + q[(i + 1) % 3] * N + q[(i + 2) % 3]) * 3 + c];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            C[i][j] = J[(i + 1) % 3][(j + 1) % 3] * J[(i + 2) % 3][(j + 2) % 3] -
                      J[(i + 1) % 3][(j + 2) % 3] * J[(i + 2) % 3][(j + 1) % 3];
    return J[0][0] * C[0][0] + J[0][1] * C[0][1] + J[0][2] * C[0][2];
}

// w* of a point: points with detJ below -1e-6 are skipped
__device__ __forceinline__ double hex_weight(double E, double w, double det) {
    return E * (det < -1.0e-6 ? 0.0 : w * det);
}

template <int N, int OUT>
__global__ void __launch_bounds__(32 * kHexWarps) hex_cells(HexArgs p) {
    constexpr int NQ = N * N * N, QS = 25;  // an odd stride: the lanes write one point each
    constexpr int LPP = N == 2 ? 4 : 1, NPL = 8 / LPP;  // lanes per point, nodes per lane
    constexpr int kX = 24, kG = 9 * N * N, kGrad = 2 * NQ * QS, kPairs = 28 * 9 + 28 * 6;
    constexpr int kWarp = kX + kG + (kGrad > kPairs ? kGrad : kPairs);
    __shared__ double sm[kHexWarps][kWarp];
    const int lane = threadIdx.x & 31;
    double* X = sm[threadIdx.x >> 5];
    double* G = X + kX;
    double* gg = G + kG;          // g and w* g: [point][axis][node]
    double* wg = gg + NQ * QS;
    double* kb = gg;              // later: K of the pairs, then their shares of the residual
    double* rb = gg + 28 * 9;
    HexCell cl;
    if (!cl.init(p, (int64_t)blockIdx.x * kHexWarps + (threadIdx.x >> 5))) return;
    if (lane < 24) X[lane] = __ldg(p.xe + cl.cell * 24 + lane);
    const double E = __ldg(p.E + cl.cell);
    // the lane's pair a < b of nodes
    int a = 0, b = lane < 28 ? lane : 0;
    while (b >= 7 - a) b -= 7 - a++;
    b += a + 1;
    const int64_t na = cl.node(p, a), nb = cl.node(p, b);
    __syncwarp();
    hex_gradients<N>(p, X, G, lane);
    __syncwarp();
    {
        const int q = lane / LPP, n0 = lane % LPP * NPL;
        if (q < NQ) {
            const int qi[3] = {q % N, q / N % N, q / (N * N)};
            double C[3][3];
            const double det = hex_cofactors<N>(G, qi, C), id = 1.0 / det;
            const double ws = hex_weight(E, p.wq[q], det);
            double t[3][2];  // 1-D shape functions of the two sides
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                t[d][1] = 0.5 + 0.5 * p.xq[qi[d]];
                t[d][0] = 0.5 - 0.5 * p.xq[qi[d]];
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) C[i][j] *= 0.5 * id;
#pragma unroll
            for (int h = 0; h < NPL; ++h) {
                const int n = n0 + h, s0 = hex_corner(n, 0), s1 = hex_corner(n, 1), s2 = hex_corner(n, 2);
                const double l0 = s0 ? t[0][1] : t[0][0], l1 = s1 ? t[1][1] : t[1][0], l2 = s2 ? t[2][1] : t[2][0];
                // dN/dxi_i: the sign of the node's side times the other two functions
                const double d0 = s0 ? l1 * l2 : -(l1 * l2), d1 = s1 ? l0 * l2 : -(l0 * l2),
                             d2 = s2 ? l0 * l1 : -(l0 * l1);
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const double g = fma(C[2][j], d2, fma(C[1][j], d1, C[0][j] * d0));
                    gg[q * QS + j * 8 + n] = g;
                    wg[q * QS + j * 8 + n] = ws * g;
                }
            }
        }
    }
    __syncwarp();
    double A[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) A[k] = 0.0;
#pragma unroll 3
    for (int q = 0; q < NQ; ++q) {
        double w[3], g[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            w[i] = wg[q * QS + i * 8 + a];
            g[i] = gg[q * QS + i * 8 + b];
        }
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) A[i * 3 + j] = fma(w[i], g[j], A[i * 3 + j]);
    }
    double K[9];  // rows of node a, columns of node b
    {
        const double tr = A[0] + A[4] + A[8];
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int g = 0; g < 3; ++g)
                K[f * 3 + g] = f == g ? fma(p.ld, A[f * 4], tr) : fma(p.lo, A[f * 3 + g], A[g * 3 + f]);
    }
    // from here on with what an overlapped kernel writes: u, and the sums
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    double du[3] = {0.0, 0.0, 0.0};
    if (p.u)
#pragma unroll
        for (int f = 0; f < 3; ++f) du[f] = p.u[f * cl.nodes + nb] - p.u[f * cl.nodes + na];
    __syncwarp();  // the gradients are read
    if (lane < 28) {
#pragma unroll
        for (int k = 0; k < 9; ++k) kb[lane * 9 + k] = K[k];
        if (p.u && p.r)
#pragma unroll
            for (int f = 0; f < 3; ++f) {
                rb[lane * 6 + f] = fma(K[f * 3 + 2], du[2], fma(K[f * 3 + 1], du[1], K[f * 3] * du[0]));
                rb[lane * 6 + 3 + f] = fma(K[6 + f], du[2], fma(K[3 + f], du[1], K[f] * du[0]));
            }
    }
    __syncwarp();
    const auto pair = [](int m, int n) { return m * 7 - m * (m - 1) / 2 + n - m - 1; };
    if (p.u && p.r && lane < 24) {
        const int n = lane / 3, f = lane % 3;
        double v = 0.0;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if (m == n) continue;
            // K(b, a) (u_a - u_b) = -K(a, b)^T (u_b - u_a)
            if (n < m) v += rb[pair(n, m) * 6 + f];
            else v -= rb[pair(m, n) * 6 + 3 + f];
        }
        atomicAdd(p.r + f * cl.nodes + cl.node(p, n), v);
    }
    // where the blocks go
    const int64_t plane = (int64_t)p.nn[2] * p.nn[1] * p.pitch;
    const auto add = [&](int m, int n, int64_t node, int f, int g, double v) {  // row node m, column node n
        const int x = cl.c0[0] + hex_corner(m, 0), y = cl.c0[1] + hex_corner(m, 1), z = cl.c0[2] + hex_corner(m, 2);
        const int dx = hex_corner(n, 0) - hex_corner(m, 0), dy = hex_corner(n, 1) - hex_corner(m, 1),
                  dz = hex_corner(n, 2) - hex_corner(m, 2);
        if (OUT == HEX_STENCIL) {
            const int k = (dx + 1) + 3 * (dy + 1) + 9 * (dz + 1);
            atomicAdd(p.S + (k * 9 + f * 3 + g) * plane + ((int64_t)z * p.nn[1] + y) * p.pitch + x, v);
        } else {
            const int lx = x > 0 ? -1 : 0, ly = y > 0 ? -1 : 0, lz = z > 0 ? -1 : 0;
            const int cx = (x + 1 < p.nn[0] ? 2 : 1) - lx, cy = (y + 1 < p.nn[1] ? 2 : 1) - ly,
                      cz = (z + 1 < p.nn[2] ? 2 : 1) - lz;
            atomicAdd(p.vals + __ldg(p.rowptr + f * cl.nodes + node) + g * (cx * cy * cz) +
                          ((dz - lz) * cy + (dy - ly)) * cx + (dx - lx),
                      v);
        }
    };
    bool bad = false;
    if (lane < 28) {
#pragma unroll
        for (int f = 0; f < 3; ++f)
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                add(a, b, na, f, g, K[f * 3 + g]);
                add(b, a, nb, g, f, K[f * 3 + g]);
                bad |= !fem_finite(K[f * 3 + g]);
            }
    }
    for (int t = lane; t < 72; t += 32) {
        const int n = t / 9, f = t % 9 / 3, g = t % 3;
        double v = 0.0;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if (m == n) continue;
            v -= n < m ? kb[pair(n, m) * 9 + f * 3 + g] : kb[pair(m, n) * 9 + g * 3 + f];
        }
        add(n, n, cl.node(p, n), f, g, v);
        bad |= !fem_finite(v);
    }
    if (bad) atomicOr(p.status, 1);
}

// nodal residual of u, no matrix: a lane per point
template <int N>
__global__ void __launch_bounds__(32 * kHexWarps) hex_residual(HexArgs p) {
    constexpr int NQ = N * N * N, kG = 9 * N * N, kWarp = 48 + 2 * kG + 9 * NQ;
    __shared__ double sm[kHexWarps][kWarp];
    const int lane = threadIdx.x & 31;
    double* X = sm[threadIdx.x >> 5];
    double* U = X + 24;
    double* GX = U + 24;
    double* GU = GX + kG;
    double* F = GU + kG;  // [axis i][component][point]
    double* D = GX;       // later: sums along i [i][component][jk], then of edges [i][component][4]
    double* T = GU;
    HexCell cl;
    if (!cl.init(p, (int64_t)blockIdx.x * kHexWarps + (threadIdx.x >> 5))) return;
    if (lane < 24) X[lane] = __ldg(p.xe + cl.cell * 24 + lane);
    const double E = __ldg(p.E + cl.cell);
    __syncwarp();
    hex_gradients<N>(p, X, GX, lane);
    cudaGridDependencySynchronize();  // u
    cudaTriggerProgrammaticLaunchCompletion();
    if (lane < 24) U[lane] = p.u[lane % 3 * cl.nodes + cl.node(p, lane / 3)];
    __syncwarp();
    hex_gradients<N>(p, U, GU, lane);
    __syncwarp();
    if (lane < NQ) {
        const int q[3] = {lane % N, lane / N % N, lane / (N * N)};
        double C[3][3], H[3][3];
        const double det = hex_cofactors<N>(GX, q, C), id = 1.0 / det;
        const double ws = hex_weight(E, p.wq[lane], det);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) C[i][j] *= id;
#pragma unroll
        for (int j = 0; j < 3; ++j)  // du_c / dx_j
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                double v = 0.0;
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const double g = GU[(i * N * N + q[(i + 1) % 3] * N + q[(i + 2) % 3]) * 3 + c];
                    v = i ? fma(C[i][j], g, v) : C[i][j] * g;
                }
                H[j][c] = v;
            }
        const double tr = p.lo * (H[0][0] + H[1][1] + H[2][2]);
        double s[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int c = j; c < 3; ++c) s[j][c] = s[c][j] = ws * (j == c ? fma(2.0, H[j][j], tr) : H[j][c] + H[c][j]);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                F[(i * 3 + c) * NQ + lane] = fma(C[i][2], s[2][c], fma(C[i][1], s[1][c], C[i][0] * s[0][c]));
    }
    __syncwarp();
    // along axis i (the derivative of N_a is constant there), then the two other axes
    for (int v = lane; v < kG; v += 32) {
        const int jk = v % (N * N), ic = v / (N * N), i = ic / 3;
        constexpr int st[3] = {1, N, N * N};
        const double* f = F + ic * NQ + jk / N * (i == 0 ? st[1] : i == 1 ? st[2] : st[0]) +
                          jk % N * (i == 0 ? st[2] : i == 1 ? st[0] : st[1]);
        const int step = i == 0 ? st[0] : i == 1 ? st[1] : st[2];
        double t = f[0];
#pragma unroll
        for (int k = 1; k < N; ++k) t += f[k * step];
        D[v] = t;
    }
    __syncwarp();
    for (int v = lane; v < 36; v += 32) {
        const int s2 = v & 1, s1 = v >> 1 & 1, ic = v >> 2;
        double t = 0.0;
#pragma unroll
        for (int j = 0; j < N; ++j) {
            double r = 0.0;
#pragma unroll
            for (int k = 0; k < N; ++k)
                r = fma(0.5 + (s2 ? 0.5 : -0.5) * p.xq[k], D[ic * N * N + j * N + k], r);
            t = fma(0.5 + (s1 ? 0.5 : -0.5) * p.xq[j], r, t);
        }
        T[v] = t;
    }
    __syncwarp();
    if (lane < 24) {
        const int n = lane / 3, c = lane % 3;
        double v = 0.0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double t =
                T[(i * 3 + c) * 4 + hex_corner(n, (i + 1) % 3) * 2 + hex_corner(n, (i + 2) % 3)];
            v = hex_corner(n, i) ? v + t : v - t;
        }
        atomicAdd(p.r + c * cl.nodes + cl.node(p, n), 0.5 * v);
    }
}

}  // namespace fem
