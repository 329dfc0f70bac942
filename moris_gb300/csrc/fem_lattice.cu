// fem_lattice.cu -- assembly on uniform tensor lattices of brick cells.
//
// A level-0 HMR mesh is a tensor lattice: nodes, cells and B-splines numbered
// i-fastest, the extraction row of a node the same for every node (one basis
// for linear splines, the eight bases around it with weight 1/8 for quadratic
// ones).  Then sum_e T_e^T K_e T_e = T^T (sum_e K_e) T with T the node-to-basis
// matrix of the whole mesh, and both factors are stencils:
//
//   lattice_const / lattice_density   the 27-point block stencil of sum_e K_e,
//       one thread per node: every 3 x 3 block is a sum over the elements that
//       share the node pair, gathered in a fixed order (no atomics on values, no
//       zero fill, one store per value), and the nodal residual K u on the way;
//   lattice_project   T^T S T for quadratic splines, axis by axis: 3 -> 5 taps
//       per axis with 5 additions (the weights are powers of two, folded into
//       the modulus), written row by row into the CSR;
//   lattice_rows      the stencil as CSR rows for linear splines;
//   lattice_product   the residual alone, without a stencil.
//
// The element loop (fem_bulk_cta.cuh) spends 6,561 atomic updates on each
// quadratic element and is bound by shared-memory latency and the L2's atomic
// rate; here a CSR value costs about 2.5 FP64 additions and one store.  The
// FP64 pipe (2 lanes per SM and clock on GB300) binds, 68-77 % busy: 2,340 additions
// per basis for the projection, 750 operations per node for the stencil.
//
// Measured on GB300 against the element loop (whole calls, residual included):
// 64^3 quadratic 7.75 -> 2.21 ms, 15 x 13 x 11 quadratic 120 -> 78 us, 96^3 density set
// with linear splines 13.4 -> 2.50 ms, matrix-free product of 48 x 47 x 45 quadratic
// cells 969 -> 76 us.  Small models keep the element loop (lattice_pays).
//
// Cells of any shape on the same lattice of nodes (FEM_GPU_SHAPE_GENERAL): the cells
// add their matrices to the block stencil (fem_hex.cuh), or to the CSR for linear
// splines, and the projection is the same.  26 x 23 x 21 quadratic 699 -> 531 us (hex
// 371, projection 128); 26^3 linear 467 -> 294 us, matrix-free products 401 -> 206
// (linear) and 622 -> 264 us.
//
// A model takes this path when lattice_finalize finds all of the above to hold
// exactly (coordinates, numbering, weights, and a CSR whose rows are the full
// boxes of neighbours); any other model keeps the element loop.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "fem_bits.cuh"
#include "fem_hex.cuh"
#include "fem_internal.hpp"
#include "fem_launch.cuh"

namespace fem {
namespace {

// a stencil CTA: 32 consecutive nodes, one warp per z offset
constexpr int kStencilNodes = 32, kStencilThreads = 3 * kStencilNodes, kDensityThreads = 2 * kStencilNodes;
// bases of a projection tile
constexpr int kPX = 5, kPY = 3;

enum { OUT_NONE = 0, OUT_STENCIL = 1, OUT_CSR = 2 };

struct LatArgs {
    int ne[3], nn[3];
    int64_t pitch;         // x pitch of the stencil array
    const double* E;       // modulus per cell
    const double* jac;     // half edge lengths [ne0], [ne1], [ne2], then their reciprocals
    const double* rho;     // nodal densities (density sets)
    double* Q;             // density sets: element sums [kQN][ne2 + 2][ne1 + 2][ne0 + 2], zero around the lattice
    const double* u;       // nodal displacements [3][nodes] (nullable: zero)
    double* r;             // nodal residual [3][nodes] (nullable)
    double* S;             // [27][9][nn2][nn1][pitch]
    double* vals;          // CSR values (linear splines: node = basis)
    const int32_t* rowptr;
    int acc_v, acc_r;      // add to vals / r instead of storing
    int* status;
    double coef[27][9];    // constant E: see lattice_const
    double xq[3], wq[27];  // density: 1-D points, weights (x fastest) times mu
    double beta, ld, lo;   // density exponent, (lam + mu) / mu, lam / mu
    double wmu;            // lattice_product: mu times a scale over 8
};

// One warp's share of a node's row: the blocks of neighbour offsets
// (dx, dy, DZ), consumed as they are formed.
template <int OUT, int DZ>
struct NodeOut {
    const LatArgs& p;
    int x, y, z;
    int64_t node, nodes;
    double r[3] = {0.0, 0.0, 0.0};
    int32_t row[3];
    int cx, cy, cz, lx, ly, lz;  // CSR box of the node's row
    bool live, bad = false;

    __device__ NodeOut(const LatArgs& a, int64_t n) : p(a), node(n) {
        nodes = (int64_t)p.nn[0] * p.nn[1] * p.nn[2];
        live = node < nodes;
        const unsigned i = live ? (unsigned)node : 0u, yz = i / (unsigned)p.nn[0];
        x = (int)(i - yz * (unsigned)p.nn[0]);
        z = (int)(yz / (unsigned)p.nn[1]);
        y = (int)(yz - (unsigned)z * (unsigned)p.nn[1]);
        if constexpr (OUT == OUT_CSR) {
            lx = x > 0 ? -1 : 0;
            ly = y > 0 ? -1 : 0;
            lz = z > 0 ? -1 : 0;
            cx = (x + 1 < p.nn[0] ? 2 : 1) - lx;
            cy = (y + 1 < p.nn[1] ? 2 : 1) - ly;
            cz = (z + 1 < p.nn[2] ? 2 : 1) - lz;
            for (int f = 0; f < 3; ++f) row[f] = live ? __ldg(p.rowptr + f * nodes + node) : 0;
        }
    }
    __device__ __forceinline__ bool inside(int dx, int dy) const {
        return live && x + dx >= 0 && x + dx < p.nn[0] && y + dy >= 0 && y + dy < p.nn[1] && z + DZ >= 0 &&
               z + DZ < p.nn[2];
    }
    // displacements of the row of neighbours dy, ahead of its blocks: plain loads (an
    // earlier kernel that this one overlaps wrote them), which do not pass the stores
    // of a block
    __device__ __forceinline__ void neighbours(int dy, double un[3][3]) const {
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const int64_t j = node + dx + (int64_t)p.nn[0] * (dy + (int64_t)p.nn[1] * DZ);
#pragma unroll
            for (int g = 0; g < 3; ++g) un[dx + 1][g] = p.u && inside(dx, dy) ? p.u[g * nodes + j] : 0.0;
        }
    }
    __device__ __forceinline__ void block(int dx, int dy, const double un[3][3], const double K[9]) {
        const bool in = inside(dx, dy);
        if (p.u && in) {
#pragma unroll
            for (int g = 0; g < 3; ++g)
#pragma unroll
                for (int f = 0; f < 3; ++f) r[f] = fma(K[f * 3 + g], un[dx + 1][g], r[f]);
        }
        if constexpr (OUT != OUT_NONE) {
#pragma unroll
            for (int k = 0; k < 9; ++k) bad |= !fem_finite(K[k]);
        }
        if constexpr (OUT == OUT_STENCIL) {
            // blocks that leave the lattice are sums over no element: zeros the projection reads
            const int k = (dx + 1) + 3 * (dy + 1) + 9 * (DZ + 1);
            const int64_t plane = (int64_t)p.nn[2] * p.nn[1] * p.pitch;
            double* s = p.S + (int64_t)k * 9 * plane + ((int64_t)z * p.nn[1] + y) * p.pitch + x;
            if (live) {
#pragma unroll
                for (int c = 0; c < 9; ++c) s[c * plane] = K[c];
            }
        } else if (OUT == OUT_CSR && in) {
            const int at = ((DZ - lz) * cy + (dy - ly)) * cx + (dx - lx), ul = cx * cy * cz;
#pragma unroll
            for (int f = 0; f < 3; ++f)
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    double* v = p.vals + row[f] + g * ul + at;
                    *v = p.acc_v ? *v + K[f * 3 + g] : K[f * 3 + g];
                }
        }
    }
    // the block K of neighbour (dx, dy, DZ) at the neighbour's row: K^T, and its share of
    // the neighbour's residual; ui: displacements of the node
    __device__ __forceinline__ void transposed(int dx, int dy, const double ui[3], const double K[9]) {
        const int k = 26 - ((dx + 1) + 3 * (dy + 1) + 9 * (DZ + 1));
        const int64_t plane = (int64_t)p.nn[2] * p.nn[1] * p.pitch;
        double* s = p.S + (int64_t)k * 9 * plane + ((int64_t)z * p.nn[1] + y) * p.pitch + x;
        if constexpr (OUT == OUT_STENCIL) {
            // no node writes the blocks that leave the lattice on the other side
            const bool out = x - dx < 0 || x - dx >= p.nn[0] || y - dy < 0 || y - dy >= p.nn[1] || z - DZ < 0;
            if (live && out) {
#pragma unroll
                for (int c = 0; c < 9; ++c) s[c * plane] = 0.0;
            }
        }
        if (!inside(dx, dy)) return;
        const int64_t j = node + dx + (int64_t)p.nn[0] * (dy + (int64_t)p.nn[1] * DZ);
        if constexpr (OUT == OUT_STENCIL) {
            s += ((int64_t)DZ * p.nn[1] + dy) * p.pitch + dx;
#pragma unroll
            for (int f = 0; f < 3; ++f)
#pragma unroll
                for (int g = 0; g < 3; ++g) s[(g * 3 + f) * plane] = K[f * 3 + g];
        }
        if (p.u) {
#pragma unroll
            for (int g = 0; g < 3; ++g)
                atomicAdd(p.r + g * nodes + j, fma(K[6 + g], ui[2], fma(K[3 + g], ui[1], K[g] * ui[0])));
        }
    }
    __device__ void finish_atomic() {
        if (bad && live) atomicOr(p.status, 1);
        if (p.u && live)
            for (int f = 0; f < 3; ++f) atomicAdd(p.r + f * nodes + node, r[f]);
    }
    __device__ void finish(double red[kStencilNodes][3]) {
        if (bad && live) atomicOr(p.status, 1);
        for (int f = 0; f < 3; ++f) red[threadIdx.x % kStencilNodes][f] = r[f];
    }
};

// the three warps' shares of the nodal residual, in the order of the z offsets
__device__ __forceinline__ void store_residual(const LatArgs& p, int64_t node, const double red[3][kStencilNodes][3]) {
    const int64_t nodes = (int64_t)p.nn[0] * p.nn[1] * p.nn[2];
    if (!p.r || node >= nodes || threadIdx.x >= kStencilNodes) return;
    for (int f = 0; f < 3; ++f) {
        const double v = (red[0][threadIdx.x][f] + red[1][threadIdx.x][f]) + red[2][threadIdx.x][f];
        double* q = p.r + f * nodes + node;
        *q = p.acc_r ? *q + v : v;
    }
}

// Constant modulus per element.  With detJ = J0 J1 J2 an element's block is
//   K[(f,a),(f,b)] = sum_k w_k c_fk(a,b),  w_k = E detJ / J_k^2
//   K[(f,a),(g,b)] = v_h H_fg(a,b),        v_h = E J_h (h the third axis)
// and c, H factor into 1-D mass, stiffness and gradient matrices whose entries
// depend on the node offset only, up to a sign along gradient axes: for offset
// 0 the lower element counts + and the upper one -.  So a block needs the box
// sums of six element weights (summed along mass and stiffness axes,
// differenced along the two gradient axes) times the coefficients p.coef[k] =
// {c_00..c_02 as G_kk, H_fg}: 500 FP64 operations per node against 960 for the
// product of every shared element.
// A thread forms the nine blocks of one z offset, so that 96 threads work on
// 32 nodes: a small lattice still fills the SMs, and consecutive lanes are
// consecutive nodes whatever the edge lengths (no partial tiles).
// (A warp per (dy, dz) as well: 2 us less up to 13^3 cells, a quarter more from 16^3 on.)
template <int OUT, int DZ>
__device__ __forceinline__ void const_blocks(const LatArgs& p, int64_t node, double red[kStencilNodes][3]) {
    NodeOut<OUT, DZ> out(p, node);
    // columns after the z axis: weights 0-2 and the xy pair (v_2) sum, the xz
    // (v_1) and yz (v_0) pairs difference
    double c[6][2][2];
    const double* ij = p.jac + p.ne[0] + p.ne[1] + p.ne[2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            double w[2][6];
            const int ex = out.x - 1 + i, ey = out.y - 1 + j;
            const int qx = min(max(ex, 0), p.ne[0] - 1), qy = p.ne[0] + min(max(ey, 0), p.ne[1] - 1);
            const double j0 = __ldg(p.jac + qx), i0 = __ldg(ij + qx), j1 = __ldg(p.jac + qy), i1 = __ldg(ij + qy);
#pragma unroll
            for (int k = DZ > 0 ? 1 : 0; k <= (DZ < 0 ? 0 : 1); ++k) {
                const int ez = out.z - 1 + k, qz = p.ne[0] + p.ne[1] + min(max(ez, 0), p.ne[2] - 1);
                const double j2 = __ldg(p.jac + qz), i2 = __ldg(ij + qz);
                const bool in =
                    out.live && ex >= 0 && ex < p.ne[0] && ey >= 0 && ey < p.ne[1] && ez >= 0 && ez < p.ne[2];
                const double E = in ? __ldg(p.E + ((int64_t)ez * p.ne[1] + ey) * p.ne[0] + ex) : 0.0;
                w[k][3] = E * j0;
                w[k][4] = E * j1;
                w[k][5] = E * j2;
                w[k][0] = w[k][4] * j2 * i0;
                w[k][1] = w[k][3] * j2 * i1;
                w[k][2] = w[k][3] * j1 * i2;
            }
#pragma unroll
            for (int m = 0; m < 6; ++m)
                c[m][j][i] = DZ < 0             ? w[0][m]
                             : DZ > 0           ? w[1][m]
                             : m == 3 || m == 4 ? w[0][m] - w[1][m]
                                                : w[0][m] + w[1][m];
        }
    cudaGridDependencySynchronize();  // the nodal displacements
    cudaTriggerProgrammaticLaunchCompletion();
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
        double un[3][3], d[6][2];
        out.neighbours(dy, un);
#pragma unroll
        for (int m = 0; m < 6; ++m)
#pragma unroll
            for (int i = 0; i < 2; ++i)
                d[m][i] = dy < 0             ? c[m][0][i]
                          : dy > 0           ? c[m][1][i]
                          : m == 3 || m == 5 ? c[m][0][i] - c[m][1][i]
                                             : c[m][0][i] + c[m][1][i];
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            double s[6];
#pragma unroll
            for (int m = 0; m < 6; ++m)
                s[m] = dx < 0 ? d[m][0] : dx > 0 ? d[m][1] : m == 4 || m == 5 ? d[m][0] - d[m][1] : d[m][0] + d[m][1];
            const double* q = p.coef[(dx + 1) + 3 * (dy + 1) + 9 * (DZ + 1)];
            const double a0 = s[0] * q[0], a1 = s[1] * q[1], a2 = s[2] * q[2], tr = a0 + a1 + a2;
            const double K[9] = {fma(p.ld, a0, tr), s[5] * q[3],       s[4] * q[4],
                                 s[5] * q[5],       fma(p.ld, a1, tr), s[3] * q[6],
                                 s[4] * q[7],       s[3] * q[8],       fma(p.ld, a2, tr)};
            out.block(dx, dy, un, K);
        }
    }
    out.finish(red);
}

template <int OUT>
__global__ void __launch_bounds__(kStencilThreads) lattice_const(LatArgs p) {
    __shared__ double red[3][kStencilNodes][3];
    const int64_t node = (int64_t)blockIdx.x * kStencilNodes + threadIdx.x % kStencilNodes;
    const int w = threadIdx.x / kStencilNodes;
    if (w == 0) const_blocks<OUT, -1>(p, node, red[0]);
    else if (w == 1) const_blocks<OUT, 0>(p, node, red[1]);
    else const_blocks<OUT, 1>(p, node, red[2]);
    __syncthreads();
    store_residual(p, node, red);
}

// Residual alone, constant modulus per element: r += sum_e K_e u without a block.  On a
// brick a trilinear field is a sum of the monomials x^m, m in {0, 1}^3, whose
// gradients are orthogonal: with h_m = sum over the corners of s^m u (s = -+1) the
// strains are single coefficients, the integral over the cell is V / 3^|n| for every
// monomial x^n, and the corner forces come back by the transposed sums.  258 FP64
// operations per cell and 24 coalesced atomics, where the stencil took 750 operations
// per node: product of 48 x 47 x 45 quadratic cells 210 -> 76 us
// (kernel 58, FP64 pipe 69 %).
__global__ void __launch_bounds__(128) lattice_product(LatArgs p) {
    const unsigned cells = (unsigned)p.ne[0] * p.ne[1] * p.ne[2], e = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = e < cells;
    const unsigned ec = live ? e : 0, yz = ec / p.ne[0];
    const int ex = (int)(ec - yz * p.ne[0]), ey = (int)(yz % p.ne[1]), ez = (int)(yz / p.ne[1]);
    const int64_t nodes = (int64_t)p.nn[0] * p.nn[1] * p.nn[2];
    const double J[3] = {__ldg(p.jac + ex), __ldg(p.jac + p.ne[0] + ey), __ldg(p.jac + p.ne[0] + p.ne[1] + ez)};
    const double* ij = p.jac + p.ne[0] + p.ne[1] + p.ne[2];
    const double k[3] = {__ldg(ij + ex), __ldg(ij + p.ne[0] + ey), __ldg(ij + p.ne[0] + p.ne[1] + ez)};
    // V / 64 = detJ / 8 (the 1/8 of the field's and of the test function's monomials)
    const double w = __ldg(p.E + ec) * p.wmu * (J[0] * J[1] * J[2]);
    cudaGridDependencySynchronize();  // u, and the sums
    cudaTriggerProgrammaticLaunchCompletion();
    const int64_t n0 = ((int64_t)ez * p.nn[1] + ey) * p.nn[0] + ex;
    const int64_t sy = p.nn[0], sz = (int64_t)p.nn[0] * p.nn[1];
    double h[3][8];  // component, monomial (bit d: x_d)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double* u = p.u + c * nodes + n0;
#pragma unroll
        for (int m = 0; m < 8; ++m) h[c][m] = u[(m & 1) + (m >> 1 & 1) * sy + (m >> 2) * sz];
#pragma unroll
        for (int b = 1; b < 8; b <<= 1)
#pragma unroll
            for (int m = 0; m < 8; ++m)
                if (!(m & b)) {
                    const double lo = h[c][m], up = h[c][m | b];
                    h[c][m] = lo + up;
                    h[c][m | b] = up - lo;
                }
    }
    // T[i][c][n]: stress i c over mu at the monomials n of the other two axes than i
    // (index without bit i); gradients g(i, c, n) = k_i h[c][n + e_i]
    double T[3][3][8];
    {
        double g[3][3][8];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int n = 0; n < 8; ++n)
                    if (!(n & 1 << i)) g[i][c][n] = k[i] * h[c][n | 1 << i];
        const double t0 = p.lo * (g[0][0][0] + g[1][1][0] + g[2][2][0]);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int a = (i + 1) % 3, b = (i + 2) % 3, xi = 1 << i, xa = 1 << a, xb = 1 << b;
            T[i][i][0] = fma(2.0, g[i][i][0], t0);
            T[i][i][xa | xb] = (2.0 + p.lo) * g[i][i][xa | xb];
            // monomial x_i: the strains along the other two axes
            const double t = p.lo * (g[a][a][xi] + g[b][b][xi]);
            T[a][a][xi] = fma(2.0, g[a][a][xi], t);
            T[b][b][xi] = fma(2.0, g[b][b][xi], t);
            // shear of the axes a and b
            T[a][b][0] = T[b][a][0] = g[a][b][0] + g[b][a][0];
            T[a][b][xi] = T[b][a][xi] = g[a][b][xi] + g[b][a][xi];
            T[a][b][xb] = g[a][b][xb];
            T[b][a][xa] = g[b][a][xa];
            T[a][b][xb | xi] = g[a][b][xb | xi];
            T[b][a][xa | xi] = g[b][a][xa | xi];
        }
    }
    const double w3 = w * (1.0 / 3.0), w9 = w * (1.0 / 9.0);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double r[8];
        r[0] = 0.0;
#pragma unroll
        for (int m = 1; m < 8; ++m) {
            double v = 0.0;
#pragma unroll
            for (int i = 2; i >= 0; --i)
                if (m & 1 << i) v = fma(k[i], T[i][c][m & ~(1 << i)], v);
            const int bits = (m & 1) + (m >> 1 & 1) + (m >> 2);
            r[m] = (bits == 1 ? w : bits == 2 ? w3 : w9) * v;
        }
        // r(s) = sum_m s^m r_m
#pragma unroll
        for (int b = 1; b < 8; b <<= 1)
#pragma unroll
            for (int m = 0; m < 8; ++m)
                if (!(m & b)) {
                    const double a = r[m], d = r[m | b];
                    r[m] = a - d;
                    r[m | b] = a + d;
                }
        if (live) {
            double* q = p.r + c * nodes + n0;
#pragma unroll
            for (int m = 0; m < 8; ++m) atomicAdd(q + (m & 1) + (m >> 1 & 1) * sy + (m >> 2) * sz, r[m]);
        }
    }
}

// 1-D factors of the density path.  Along an axis a pair of nodes (offset d)
// meets the lower element (side 0, d <= 0) and the upper one (side 1, d >= 0);
// type 0: N' N' (one quadrature sum), 1: N N (three sums, of (1+x)^2, (1-x)^2
// and 1-x^2), 2: N' N (row differentiated) and 3: N N' (two sums, of 1+x and
// 1-x); each element contributes one of the sums with a sign.
__device__ constexpr int ax_n(int d) { return d == 0 ? 2 : 1; }
__device__ constexpr int ax_side(int d, int i) { return d == 0 ? i : d < 0 ? 0 : 1; }
__device__ constexpr int ax_var(int type, int d, int i) {
    return type == 0   ? 0
           : type == 1 ? (d == 0 ? i : 2)
           : type == 2 ? (d == 0 ? i : d < 0 ? 1 : 0)
                       : (d == 0 ? i : d < 0 ? 0 : 1);
}
__device__ constexpr bool ax_neg(int type, int d, int i) {
    return type == 0   ? d != 0
           : type == 1 ? false
           : type == 2 ? (d == 0 ? i == 1 : d > 0)
                       : (d == 0 ? i == 1 : d < 0);
}
__device__ constexpr int ax_vars(int type) { return type == 0 ? 1 : type == 1 ? 3 : 2; }

// sums of an element: {xx, yy, zz, xy, xz, yz} at these offsets, the variants
// of the axes in x, y, z order (z fastest)
constexpr int kXX = 0, kYY = 9, kZZ = 18, kXY = 27, kXZ = 39, kYZ = 51, kQN = 63;

// block entry of a node from the sums of its elements; q: the sums of the
// lower element along every axis, qs / ey / ez: strides of a sum, an element
// row and an element layer
template <int TX, int TY, int TZ, int DZ>
__device__ __forceinline__ double gather(const double* __restrict__ q, int64_t qs, int64_t ey, int64_t ez, int off,
                                         int dx, int dy) {
    double s = 0.0;
    bool first = true;
#pragma unroll
    for (int k = 0; k < ax_n(DZ); ++k)
#pragma unroll
        for (int j = 0; j < ax_n(dy); ++j)
#pragma unroll
            for (int i = 0; i < ax_n(dx); ++i) {
                const int at = off + (ax_var(TX, dx, i) * ax_vars(TY) + ax_var(TY, dy, j)) * ax_vars(TZ) +
                               ax_var(TZ, DZ, k);
                const double v = __ldg(q + at * qs + ax_side(DZ, k) * ez + ax_side(dy, j) * ey + ax_side(dx, i));
                const bool neg = ax_neg(TX, dx, i) ^ ax_neg(TY, dy, j) ^ ax_neg(TZ, DZ, k);
                s = first ? (neg ? -v : v) : neg ? s - v : s + v;
                first = false;
            }
    return s;
}

// Density sets: E(x_q) = E rho(x_q)^beta at N^3 tensor Gauss points.  A brick's
// gradients factor per axis, so its 300 Gram entries are signed copies of 63
// sums over the points (1-D factors above), formed axis by axis: 300 FMAs
// instead of 300 N^3.  One thread per element writes them (504 bytes, read back
// from L2 and L1 by the eight nodes around it); staging them per node tile in
// shared memory instead recomputed 1.76 elements per node and left a quarter of
// the lanes on partial tiles.
template <int N>
__global__ void __launch_bounds__(128) lattice_moments(LatArgs p) {
    const unsigned cells = (unsigned)p.ne[0] * p.ne[1] * p.ne[2];
    const int64_t qy = p.ne[0] + 2, qz = qy * (p.ne[1] + 2), qs = qz * (p.ne[2] + 2);
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < cells; t += gridDim.x * blockDim.x) {
        const int ex = (int)(t % p.ne[0]), yz = (int)(t / p.ne[0]), ey = yz % p.ne[1], ez = yz / p.ne[1];
        double* q = p.Q + (ez + 1) * qz + (ey + 1) * qy + ex + 1;
        const double E = p.E[((int64_t)ez * p.ne[1] + ey) * p.ne[0] + ex];
        double W[N][N][N];  // [z][y][x]
        {
            // densities at the points, interpolated axis by axis
            const int64_t n0 = ((int64_t)ez * p.nn[1] + ey) * p.nn[0] + ex;
            double c[2][2][N];
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const double* r = p.rho + n0 + (int64_t)p.nn[0] * (j + (int64_t)p.nn[1] * k);
                    const double m = 0.5 * (r[0] + r[1]), d = 0.5 * (r[1] - r[0]);
#pragma unroll
                    for (int i = 0; i < N; ++i) c[k][j][i] = fma(p.xq[i], d, m);
                }
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = 0; j < N; ++j) {
                    double l[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        l[k] = fma(p.xq[j], 0.5 * (c[k][1][i] - c[k][0][i]), 0.5 * (c[k][0][i] + c[k][1][i]));
                    const double m = 0.5 * (l[0] + l[1]), d = 0.5 * (l[1] - l[0]);
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        const double r = fma(p.xq[k], d, m);
                        W[k][j][i] = p.wq[(k * N + j) * N + i] * E * (p.beta == 3.0 ? r * r * r : pow(r, p.beta));
                    }
                }
        }
        // 1-D coefficients: [axis][variant][point], with the axis' Jacobian factor
        // (1/J for N' N', J for N N, 1 for N' N)
        const double J[3] = {__ldg(p.jac + ex), __ldg(p.jac + p.ne[0] + ey), __ldg(p.jac + p.ne[0] + p.ne[1] + ez)};
        double iJ[3], M[3][3][N], G[2][N];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            iJ[a] = 1.0 / J[a];
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const double x = p.xq[i];
                M[a][0][i] = J[a] * ((1.0 + x) * (1.0 + x));
                M[a][1][i] = J[a] * ((1.0 - x) * (1.0 - x));
                M[a][2][i] = J[a] * ((1.0 + x) * (1.0 - x));
                G[0][i] = 1.0 + x;
                G[1][i] = 1.0 - x;
            }
        }
        auto dot = [](const double* v, const double* w) {
            double s = v[0] * w[0];
#pragma unroll
            for (int i = 1; i < N; ++i) s = fma(v[i], w[i], s);
            return s;
        };
        auto sum = [](const double* v, double f) {
            double s = v[0];
#pragma unroll
            for (int i = 1; i < N; ++i) s += v[i];
            return s * f;
        };
        // x variants: 0 = N' N', 1-3 = N N, 4-5 = N' N
#pragma unroll
        for (int vx = 0; vx < 6; ++vx) {
            double X[N][N];  // [z][y]
#pragma unroll
            for (int k = 0; k < N; ++k)
#pragma unroll
                for (int j = 0; j < N; ++j)
                    X[k][j] = vx == 0  ? sum(W[k][j], iJ[0])
                              : vx < 4 ? dot(W[k][j], M[0][vx - 1])
                                       : dot(W[k][j], G[vx - 4]);
            double Y[N];
            if (vx > 0 && vx < 4) {  // yy: y differentiated
#pragma unroll
                for (int k = 0; k < N; ++k) Y[k] = sum(X[k], iJ[1]);
#pragma unroll
                for (int vz = 0; vz < 3; ++vz) q[(kYY + (vx - 1) * 3 + vz) * qs] = dot(Y, M[2][vz]);
            }
#pragma unroll
            for (int vy = 0; vy < 3; ++vy) {
#pragma unroll
                for (int k = 0; k < N; ++k) Y[k] = dot(X[k], M[1][vy]);
                if (vx == 0) {
#pragma unroll
                    for (int vz = 0; vz < 3; ++vz) q[(kXX + vy * 3 + vz) * qs] = dot(Y, M[2][vz]);
                } else if (vx < 4) {
                    q[(kZZ + (vx - 1) * 3 + vy) * qs] = sum(Y, iJ[2]);
                } else {
#pragma unroll
                    for (int vz = 0; vz < 2; ++vz) q[(kXZ + ((vx - 4) * 3 + vy) * 2 + vz) * qs] = dot(Y, G[vz]);
                }
            }
            if (vx > 0) {
#pragma unroll
                for (int vy = 0; vy < 2; ++vy) {
#pragma unroll
                    for (int k = 0; k < N; ++k) Y[k] = dot(X[k], G[vy]);
                    if (vx < 4) {
#pragma unroll
                        for (int vz = 0; vz < 2; ++vz) q[(kYZ + ((vx - 1) * 2 + vy) * 2 + vz) * qs] = dot(Y, G[vz]);
                    } else {
#pragma unroll
                        for (int vz = 0; vz < 3; ++vz) q[(kXY + ((vx - 4) * 2 + vy) * 3 + vz) * qs] = dot(Y, M[2][vz]);
                    }
                }
            }
        }
    }
}

// The operator is symmetric: a node forms the blocks of itself and of the 13
// neighbours after it, and writes each to its own row and, transposed, to the
// neighbour's.  The share of the residual that belongs to the neighbour is added with
// coalesced atomics.  Two warps per 32 nodes, the plane of the node (5 blocks) and the
// next one (9): 595 FP64 operations and 324 loads per node, where all 27 blocks took
// 873 and 576.
template <int OUT, int DZ>
__device__ __forceinline__ void density_blocks(const LatArgs& p, int64_t node) {
    NodeOut<OUT, DZ> out(p, node);
    const int64_t ey = p.ne[0] + 2, ez = ey * (p.ne[1] + 2), qs = ez * (p.ne[2] + 2);
    const double* q = p.Q + out.z * ez + out.y * ey + out.x;
    double ui[3] = {0.0, 0.0, 0.0};
    if (p.u && out.live)
#pragma unroll
        for (int g = 0; g < 3; ++g) ui[g] = p.u[g * out.nodes + node];
#pragma unroll
    for (int dy = DZ ? -1 : 0; dy <= 1; ++dy) {
        double un[3][3];
        out.neighbours(dy, un);
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            if (DZ == 0 && dy == 0 && dx < 0) continue;
            const double a0 = gather<0, 1, 1, DZ>(q, qs, ey, ez, kXX, dx, dy),
                         a1 = gather<1, 0, 1, DZ>(q, qs, ey, ez, kYY, dx, dy),
                         a2 = gather<1, 1, 0, DZ>(q, qs, ey, ez, kZZ, dx, dy), tr = a0 + a1 + a2;
            const double xy = gather<2, 3, 1, DZ>(q, qs, ey, ez, kXY, dx, dy),
                         yx = gather<3, 2, 1, DZ>(q, qs, ey, ez, kXY, dx, dy),
                         xz = gather<2, 1, 3, DZ>(q, qs, ey, ez, kXZ, dx, dy),
                         zx = gather<3, 1, 2, DZ>(q, qs, ey, ez, kXZ, dx, dy),
                         yz = gather<1, 2, 3, DZ>(q, qs, ey, ez, kYZ, dx, dy),
                         zy = gather<1, 3, 2, DZ>(q, qs, ey, ez, kYZ, dx, dy);
            // K_fg = lam A_fg + mu A_gf (+ mu tr A), mu inside the weights
            const double K[9] = {fma(p.ld, a0, tr), fma(p.lo, xy, yx), fma(p.lo, xz, zx),
                                 fma(p.lo, yx, xy), fma(p.ld, a1, tr), fma(p.lo, yz, zy),
                                 fma(p.lo, zx, xz), fma(p.lo, zy, yz), fma(p.ld, a2, tr)};
            out.block(dx, dy, un, K);
            if (DZ || dy || dx) out.transposed(dx, dy, ui, K);
        }
    }
    out.finish_atomic();
}

template <int OUT>
__global__ void __launch_bounds__(kDensityThreads, 6) lattice_density(LatArgs p) {
    cudaTriggerProgrammaticLaunchCompletion();
    const int64_t node = (int64_t)blockIdx.x * kStencilNodes + threadIdx.x % kStencilNodes;
    if (threadIdx.x < kStencilNodes) density_blocks<OUT, 0>(p, node);
    else density_blocks<OUT, 1>(p, node);
}

// Linear splines: the stencil as CSR values, a CTA per 32 consecutive nodes and row
// component, whose rows are one range of the CSR.  Bound by HBM (the stencil in, the
// values out).  Written by the stencil kernels themselves, a lane per row, every value
// is a sector of its own: a 96^3 density set took 3.39 ms so, and 2.50 with this kernel
// (5.5 TB/s).
// The constant-modulus kernel has less to hide the second pass behind and gains from
// kRowsNodes on: 20^3 cells 52 us direct, 64 with rows, 32^3 114 and 128, 48^3 372 and
// 337.
constexpr int64_t kRowsNodes = 65536;
__global__ void __launch_bounds__(256) lattice_rows(int n0, int n1, int n2, int64_t pitch, const double* S,
                                                    const int32_t* __restrict__ rowptr, double* vals, int acc) {
    __shared__ double rows[kStencilNodes * 81];
    const int lane = threadIdx.x & 31, f = blockIdx.y;
    const int nodes = n0 * n1 * n2, node0 = blockIdx.x * kStencilNodes, node = node0 + lane;
    const bool live = node < nodes;
    const int i = live ? node : 0, yz = i / n0, x = i - yz * n0, z = yz / n1, y = yz - z * n1;
    const int lx = x > 0 ? -1 : 0, ly = y > 0 ? -1 : 0, lz = z > 0 ? -1 : 0;
    const int cx = (x + 1 < n0 ? 2 : 1) - lx, cy = (y + 1 < n1 ? 2 : 1) - ly, ul = cx * cy * ((z + 1 < n2 ? 2 : 1) - lz);
    const int64_t first = __ldg(rowptr + (int64_t)f * nodes + node0);
    const int64_t last = __ldg(rowptr + (int64_t)f * nodes + min(node0 + kStencilNodes, nodes));
    double* row = rows + (__ldg(rowptr + (int64_t)f * nodes + i) - first);
    const int64_t plane = (int64_t)n2 * n1 * pitch;
    const double* s = S + (int64_t)f * 3 * plane + (int64_t)yz * pitch + x;
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const int w = threadIdx.x >> 5, at0 = -(lz * cy + ly) * cx - lx;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int k = t * 8 + w, dx = k % 3 - 1, dy = k / 3 % 3 - 1, dz = k / 9 - 1;
        if (k < 27 && live && (unsigned)(x + dx) < (unsigned)n0 && (unsigned)(y + dy) < (unsigned)n1 &&
            (unsigned)(z + dz) < (unsigned)n2) {
            const double* v = s + k * 9 * plane;
            double* q = row + (dz * cy + dy) * cx + dx + at0;
#pragma unroll
            for (int g = 0; g < 3; ++g) q[g * ul] = v[g * plane];
        }
    }
    __syncthreads();
    double* v = vals + first;
    const int n = (int)(last - first);
    for (int t = threadIdx.x; t < n; t += 256) v[t] = acc ? v[t] + rows[t] : rows[t];
}

// A = T^T S T for quadratic splines (basis b covers the nodes b-1 and b along
// every axis; the weights are inside S).  Along one axis, with the row sums
// r(-2) = s_-(-1), r(-1) = s_-(0) + s(-1), r(0) = s_-(1) + s(0), r(1) = s(1) of
// the stencils s_- and s of nodes b-1 and b, the basis stencil is A(D) =
// r(D-1) + r(D): 5 additions for 5 taps, 2,340 per basis with the tile's halo.
// A CTA takes 5 x 3 bases and one row component and marches along z, one node
// plane per step: x stage from global memory (every stencil value is read once
// per tile), y stage, then the z stage on registers: thread (g, Dy, Dx) keeps
// the three z taps of the previous plane for five of the columns and writes the
// five z offsets of every row straight into the CSR, 25 consecutive values per
// (row, g, Dz).  48 KB and 80 registers, three CTAs per SM (two with 118
// registers and no spill: 2 % slower at 64^3), 225 of 256 threads in the y and z
// stages.  A first version that looped over Dz with all nine components and
// staged the values for the copy took 3.3 ms at 64^3 (FP64 pipe 49 % busy, 47
// instructions per FP64 one, most of them index arithmetic).
struct ProjArgs {
    int nn[3], nb[3];
    int tx, ty, chunks;
    int64_t pitch;
    const double* S;
    double* vals;
    const int32_t* rowptr;
    int acc;
    int* status;
};
constexpr int kProjThreads = 256, kProjCtas = 3;
constexpr int kXLen = (kPY + 1) * kPX * 135, kXYLen = kPY * kPX * 225;
constexpr size_t kProjSmem = (size_t)(kXLen + kXYLen) * sizeof(double);

__global__ void __launch_bounds__(kProjThreads, kProjCtas) lattice_project(ProjArgs p) {
    extern __shared__ double sm[];
    double* X = sm;            // [iy][ix][Dx][ky][kz][g]
    double* XY = sm + kXLen;   // [iy][ix][kz][g][Dy][Dx]
    const int tid = threadIdx.x;
    const int f = blockIdx.x % 3, tile = blockIdx.x / 3, bx = tile % p.tx, by = tile / p.tx;
    // tiles and z ranges of nearly equal size
    const int x0 = (int)((int64_t)p.nb[0] * bx / p.tx), wx = (int)((int64_t)p.nb[0] * (bx + 1) / p.tx) - x0;
    const int y0 = (int)((int64_t)p.nb[1] * by / p.ty), wy = (int)((int64_t)p.nb[1] * (by + 1) / p.ty) - y0;
    const int z0 = (int)((int64_t)p.nb[2] * blockIdx.y / p.chunks);
    const int z1 = (int)((int64_t)p.nb[2] * (blockIdx.y + 1) / p.chunks);
    const int64_t plane = (int64_t)p.nn[2] * p.nn[1] * p.pitch, layer = (int64_t)p.nn[1] * p.pitch;
    const int64_t nb01 = (int64_t)p.nb[0] * p.nb[1], nu = nb01 * p.nb[2];
    // x stage: line (ky, kz, g) of node row iy
    const int xl = tid % 27, xiy = tid / 27, xg = xl % 3, xkz = xl / 3 % 3, xky = xl / 9, xrow = y0 - 1 + xiy;
    const bool xlive = xiy <= wy && xrow >= 0 && xrow < p.nn[1];
    const double* xs = p.S + (int64_t)((xkz * 3 + xky) * 27 + f * 3 + xg) * plane +
                       (int64_t)(xlive ? xrow : 0) * p.pitch + x0 - 1;
    unsigned xin = 0;  // nodes x0 - 1 + i of the row that exist
    for (int i = 0; i <= wx; ++i)
        if (xlive && x0 - 1 + i >= 0 && x0 - 1 + i < p.nn[0]) xin |= 1u << i;
    // y stage: line (Dx, kz, g) of base column ix
    const int yix = tid / 45, yl = tid % 45, yd = yl / 9, yk = yl % 9;
    // z stage: (g, Dy, Dx), columns zc, zc + 3, ...
    const int zl = tid % 75, zc = tid / 75, zg = zl / 25, zdy = zl % 25 / 5 - 2, zdx = zl % 5 - 2;
    double m[5][3];
#pragma unroll
    for (int k = 0; k < 5; ++k) m[k][0] = m[k][1] = m[k][2] = 0.0;
    // per column its index and the in-plane box of its row: lengths cx, cy and
    // the column's own place ox, oy (cx = 0: no such column).  In shared memory:
    // as registers they and their products, hoisted out of the z loop, spill
    __shared__ int cidx[kPX * kPY], cbox[kPX * kPY];
    if (tid < kPX * kPY) {
        const int ix = tid % kPX, iy = tid / kPX, gx = x0 + ix, gy = y0 + iy;
        const int ox = min(gx, 2), oy = min(gy, 2);
        const int cx = ix < wx && iy < wy ? min(gx + 2, p.nb[0] - 1) - (gx - ox) + 1 : 0;
        const int cy = min(gy + 2, p.nb[1] - 1) - (gy - oy) + 1;
        cidx[tid] = gy * p.nb[0] + gx;
        cbox[tid] = cx | cy << 8 | ox << 16 | oy << 24;
    }
    __syncthreads();
    bool bad = false;
    cudaGridDependencySynchronize();  // the stencil
    cudaTriggerProgrammaticLaunchCompletion();
    for (int z = z0 - 1; z < z1; ++z) {  // node plane z; basis layer z from z0 on
        const bool have = z >= 0 && z < p.nn[2];
        if (have) {
            if (xiy <= wy) {
                // (plain loads: the kernel that writes the stencil may still run when this
                // one starts, see fem_launch.cuh)
                double v[kPX + 1][3];
                const double* s0 = xs + z * layer;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
#pragma unroll
                    for (int i = 0; i <= kPX; ++i) v[i][k] = xin >> i & 1 ? s0[i] : 0.0;
                    s0 += 9 * plane;
                }
                double* o = X + xiy * kPX * 135 + xl;
#pragma unroll
                for (int i = 0; i < kPX; ++i)
                    if (i < wx) {
                        const double ra = v[i][1] + v[i + 1][0], rb = v[i][2] + v[i + 1][1];
                        o[i * 135] = v[i][0];
                        o[i * 135 + 27] = v[i][0] + ra;
                        o[i * 135 + 54] = ra + rb;
                        o[i * 135 + 81] = rb + v[i + 1][2];
                        o[i * 135 + 108] = v[i + 1][2];
                    }
            }
            __syncthreads();
            if (yix < wx) {
                const double* q = X + yix * 135 + yd * 27 + yk;
                double m0 = q[0], m1 = q[9], m2 = q[18];
                double* o = XY + yix * 225 + yk * 25 + yd;
                for (int i = 0; i < wy; ++i) {
                    q += kPX * 135;
                    const double s0 = q[0], s1 = q[9], s2 = q[18];
                    const double ra = m1 + s0, rb = m2 + s1;
                    o[0] = m0;
                    o[5] = m0 + ra;
                    o[10] = ra + rb;
                    o[15] = rb + s2;
                    o[20] = s2;
                    o += kPX * 225;
                    m0 = s0;
                    m1 = s1;
                    m2 = s2;
                }
            }
            __syncthreads();
        }
        if (zc < 3) {
            const int lz = max(z - 2, 0), cz = min(z + 2, p.nb[2] - 1) - lz + 1;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const int c = zc + 3 * k, box = cbox[c];
                const double* q = XY + c * 225 + zl;
                const double s[3] = {have ? q[0] : 0.0, have ? q[75] : 0.0, have ? q[150] : 0.0};
                const int cx = box & 255, cy = box >> 8 & 255, ax = (box >> 16 & 255) + zdx, ay = (box >> 24) + zdy;
                if (z >= z0 && ax >= 0 && ax < cx && ay >= 0 && ay < cy) {
                    const double ra = m[k][1] + s[0], rb = m[k][2] + s[1];
                    const double v[5] = {m[k][0], m[k][0] + ra, ra + rb, rb + s[2], s[2]};
                    const int cxy = cx * cy;
                    double* w = p.vals + __ldg(p.rowptr + f * nu + z * nb01 + cidx[c]) + ay * cx + ax +
                                (zg * cz - lz + z - 2) * cxy;
#pragma unroll
                    for (int D = -2; D <= 2; ++D) {
                        if (z + D >= 0 && z + D < p.nb[2]) {
                            bad |= !fem_finite(v[D + 2]);
                            *w = p.acc ? *w + v[D + 2] : v[D + 2];
                        }
                        w += cxy;
                    }
                }
#pragma unroll
                for (int i = 0; i < 3; ++i) m[k][i] = s[i];
            }
        }
    }
    if (bad) atomicOr(p.status, 1);
}

// nodal values of a quadratic spline field: un[g][node] = 1/8 of the sum of its eight bases
__global__ void lattice_nodal(int n0, int n1, int n2, const double* __restrict__ u, double* un) {
    cudaTriggerProgrammaticLaunchCompletion();
    const unsigned nodes = (unsigned)n0 * n1 * n2, nu = (unsigned)(n0 + 1) * (n1 + 1) * (n2 + 1);
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < 3 * nodes; t += gridDim.x * blockDim.x) {
        const unsigned g = (t >= nodes) + (t >= 2 * nodes), i = t - g * nodes, yz = i / n0, z = yz / n1;
        const unsigned x = i - yz * n0, y = yz - z * n1, sy = n0 + 1, sz = sy * (n1 + 1);
        const double* b = u + g * nu + (z * (n1 + 1) + y) * sy + x;
        const double lo = (b[0] + b[1]) + (b[sy] + b[sy + 1]);
        const double up = (b[sz] + b[sz + 1]) + (b[sz + sy] + b[sz + sy + 1]);
        un[t] = 0.125 * (lo + up);
    }
}

// r[f][basis] (+)= scale * the sum of rn over the basis' eight nodes
__global__ void lattice_restrict(int n0, int n1, int n2, const double* rn, double scale, int acc, double* r) {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const unsigned b0 = n0 + 1, b1 = n1 + 1, nodes = (unsigned)n0 * n1 * n2, nu = b0 * b1 * (n2 + 1);
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < 3 * nu; t += gridDim.x * blockDim.x) {
        const unsigned f = (t >= nu) + (t >= 2 * nu), i = t - f * nu, yz = i / b0;
        const int z = (int)(yz / b1), x = (int)(i - yz * b0), y = (int)(yz - z * b1);
        const double* v = rn + (int64_t)f * nodes + ((int64_t)z * n1 + y) * n0 + x;
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {  // nodes z - 1, z; y - 1, y; x - 1, x
            const int dz = (k >> 2) - 1, dy = (k >> 1 & 1) - 1, dx = (k & 1) - 1;
            const bool in = (unsigned)(z + dz) < (unsigned)n2 && (unsigned)(y + dy) < (unsigned)n1 &&
                            (unsigned)(x + dx) < (unsigned)n0;
            s += in ? v[((int64_t)dz * n1 + dy) * n0 + dx] : 0.0;
        }
        r[t] = acc ? fma(scale, s, r[t]) : scale * s;
    }
}

// ---------------------------------------------------------------------------
// Plane lattices (QUAD4, splines of order 1 to 3, constant modulus per element).
// With the extraction of one axis a (p + 1) x 2 matrix, the element matrices
// between splines are products of 1-D ones (mass M, stiffness D, gradient G), so
//   A_xx(i, j) = sum_e E J_y / J_x D(i_x, j_x) M(i_y, j_y), ...
// over the at most (p + 1)^2 elements that splines i and j share: summed along x,
// then along y, four products per element and offset, no element matrix.  Lane =
// basis, warp = y offset: p + 1 of the warps form the sums along x, which all share
// (without that 864 instead of 560 FP64 instructions per basis, p = 2); a thread forms
// the 2 p + 1 blocks of its offsets and their share of the residual.  The element loop spent a CTA on 8 x 8 to 32 x 32
// matrices; measured (assembly with two side sets): 257 x 130, p = 2, 237 -> 68.5 us
// (kernel 44, FP64 pipe 68 %), 256 x 256, p = 3, 544 -> 201 us, 24 x 17, p = 1, 61 ->
// 29 us.
struct PlaneArgs {
    int ne[2], nb[2];
    const double* E;
    const double* jac;  // half edge lengths [ne0], [ne1], then their reciprocals
    const double* u;
    double* vals;
    double* rhs;
    const int32_t* rowptr;
    int acc_v, acc_r;
    int* status;
    double mu, ld, lo;                      // mu per unit modulus, (lam + mu) / mu, lam / mu
    double M[4][4], D[4][4], G[4][4];       // 1-D matrices on the reference element
};

template <int P>
__global__ void __launch_bounds__(32 * (2 * P + 1)) lattice_plane(PlaneArgs p) {
    cudaTriggerProgrammaticLaunchCompletion();
    constexpr int ND = 2 * P + 1;
    __shared__ double red[ND][32][2];
    const int lane = threadIdx.x & 31, Dy = (int)(threadIdx.x >> 5) - P;
    const int nu = p.nb[0] * p.nb[1], b = blockIdx.x * 32 + lane;
    const bool live = b < nu;
    const int bx = live ? b % p.nb[0] : 0, by = live ? b / p.nb[0] : 0;
    const bool row = live && by + Dy >= 0 && by + Dy < p.nb[1];
    const int nj = p.ne[0] + p.ne[1];
    // sums along x over the elements of row by - iy, one warp per iy
    __shared__ double xs[P + 1][ND][4][32];
    if (Dy <= 0) {
        const int iy = -Dy, ey = by - iy;
        const bool have = live && ey >= 0 && ey < p.ne[1];
        const double Jy = have ? __ldg(p.jac + p.ne[0] + ey) : 0.0, Iy = have ? __ldg(p.jac + nj + p.ne[0] + ey) : 0.0;
        double E[P + 1], wx[P + 1], wy[P + 1];
#pragma unroll
        for (int i = 0; i <= P; ++i) {
            const int ex = bx - i;
            const bool in = have && ex >= 0 && ex < p.ne[0];
            E[i] = in ? __ldg(p.E + (int64_t)ey * p.ne[0] + ex) * p.mu : 0.0;
            wx[i] = E[i] * Jy * (in ? __ldg(p.jac + nj + ex) : 0.0);
            wy[i] = E[i] * Iy * (in ? __ldg(p.jac + ex) : 0.0);
        }
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
#pragma unroll
            for (int i = 0; i <= P; ++i) {
                const int j = i + d - P;
                if (j < 0 || j > P) continue;
                a0 = fma(wx[i], p.D[i][j], a0);
                a1 = fma(wy[i], p.M[i][j], a1);
                a2 = fma(E[i], p.G[i][j], a2);
                a3 = fma(E[i], p.G[j][i], a3);
            }
            xs[iy][d][0][lane] = a0;
            xs[iy][d][1][lane] = a1;
            xs[iy][d][2][lane] = a2;
            xs[iy][d][3][lane] = a3;
        }
    }
    __syncthreads();
    double S[ND][4];  // xx, yy, xy, yx of offset Dx
#pragma unroll
    for (int d = 0; d < ND; ++d) S[d][0] = S[d][1] = S[d][2] = S[d][3] = 0.0;
    for (int iy = max(0, -Dy); iy <= min(P, P - Dy); ++iy) {
        const int jy = iy + Dy;
        const double My = p.M[iy][jy], Dyy = p.D[iy][jy], Gy = p.G[iy][jy], Hy = p.G[jy][iy];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            S[d][0] = fma(xs[iy][d][0][lane], My, S[d][0]);
            S[d][1] = fma(xs[iy][d][1][lane], Dyy, S[d][1]);
            S[d][2] = fma(xs[iy][d][2][lane], Hy, S[d][2]);
            S[d][3] = fma(xs[iy][d][3][lane], Gy, S[d][3]);
        }
    }
    double r[2] = {0.0, 0.0};
    bool bad = false;
    if (row) {
        const int lx = max(bx - P, 0), cx = min(bx + P, p.nb[0] - 1) - lx + 1;
        const int ly = max(by - P, 0), cy = min(by + P, p.nb[1] - 1) - ly + 1;
        const int32_t r0 = p.vals ? __ldg(p.rowptr + b) : 0, r1 = p.vals ? __ldg(p.rowptr + nu + b) : 0;
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const int x = bx + d - P;
            if (x < 0 || x >= p.nb[0]) continue;
            const double tr = S[d][0] + S[d][1];
            const double K[4] = {fma(p.ld, S[d][0], tr), fma(p.lo, S[d][2], S[d][3]), fma(p.lo, S[d][3], S[d][2]),
                                 fma(p.ld, S[d][1], tr)};
            if (p.u) {
                const int j = (by + Dy) * p.nb[0] + x;
                const double u0 = __ldg(p.u + j), u1 = __ldg(p.u + nu + j);
                r[0] = fma(K[0], u0, fma(K[1], u1, r[0]));
                r[1] = fma(K[2], u0, fma(K[3], u1, r[1]));
            }
            if (p.vals) {
                const int at = (by + Dy - ly) * cx + x - lx, ul = cx * cy;
                double* v[4] = {p.vals + r0 + at, p.vals + r0 + ul + at, p.vals + r1 + at, p.vals + r1 + ul + at};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    bad |= !fem_finite(K[k]);
                    *v[k] = p.acc_v ? *v[k] + K[k] : K[k];
                }
            }
        }
    }
    if (bad) atomicOr(p.status, 1);
    if (!p.rhs) return;
    red[Dy + P][lane][0] = r[0];
    red[Dy + P][lane][1] = r[1];
    __syncthreads();
    if (threadIdx.x < 64 && blockIdx.x * 32 + (threadIdx.x & 31) < nu) {
        const int f = threadIdx.x >> 5;
        double v = 0.0;
        for (int k = 0; k < ND; ++k) v += red[k][lane][f];
        double* q = p.rhs + f * nu + b;
        *q = p.acc_r ? *q + v : v;
    }
}

// ---------------------------------------------------------------------------
// Boundary facets of plane lattices: as the boundary facets of bricks (fem_brick.cu),
// with tables of the products between splines, because the extraction is the same for
// every cell:  I_i(a, b) = integral N_a dN_b / dxi_i, NN(a, b) = integral N_a N_b per
// facet ordinal.  K(a, b) = -T(a, b) + beta T(b, a)^T + gamma NN with T(k, k) = (lam +
// 2 mu) n I_k, T(t, t) = mu n I_k, T(k, t) = lam n I_t, T(t, k) = mu n I_t for the normal
// axis k; a constant displacement has no traction, so the residual is K (u - g).  A
// warp per facet, a lane per pair (or three, or eight) of splines; the pairs' shares of
// the residual meet in shared memory.  One short phase, where the general kernel
// (side_cta_kernel) is a chain of twelve: calls with clamp and load, 24 x 17 linear 32.5
// -> 28.8 us, 24 x 24 cubic 53 -> 42 us.
struct PlaneSide {
    int64_t n;
    const int32_t* facet;  // cell * 4 + ordinal
    const double* E;
    const double* tab;     // [ordinal][I_0, I_1, NN][b][a]
    int neumann;
    double lam, mu, alpha, beta, thickness, wsum, value[2];
};
constexpr int kPlaneSides = 4, kPlaneSideWarps = 4;
struct PlaneSides {
    PlaneSide set[kPlaneSides];
    int ne[2], nb[2];
    const double* jac;
    const double* u;
    double* vals;
    double* rhs;
    const int32_t* rowptr;
    int* status;
};

template <int P>
__global__ void __launch_bounds__(32 * kPlaneSideWarps) lattice_plane_sides(const __grid_constant__ PlaneSides p) {
    constexpr int NB = (P + 1) * (P + 1), PAIRS = NB * NB, PER = (PAIRS + 31) / 32;
    __shared__ double sm[kPlaneSideWarps][PAIRS][2];
    const PlaneSide& s = p.set[blockIdx.y];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t e = (int64_t)blockIdx.x * kPlaneSideWarps + warp;
    if (e >= s.n) return;
    const int fc = __ldg(s.facet + e), ord = fc & 3, cell = fc >> 2, ci = cell % p.ne[0], cj = cell / p.ne[0];
    const int nu = p.nb[0] * p.nb[1];
    const bool x = ord & 1;  // the normal is along x
    const double n = ord == 1 || ord == 2 ? 1.0 : -1.0;
    const double J0 = __ldg(p.jac + ci), J1 = __ldg(p.jac + p.ne[0] + cj), E = __ldg(s.E + e);
    const double Jk = x ? J0 : J1, Jt = x ? J1 : J0;
    const double w = Jt * s.thickness, sc = n * w * E;
    const double ck = sc / Jk, ct = sc / Jt;
    const double kk = (s.lam + 2.0 * s.mu) * ck, tt = s.mu * ck, lt = s.lam * ct, mt = s.mu * ct;
    const double nn = s.neumann ? w : s.alpha * E * w / (Jt * s.wsum);
    const double* tab = s.tab + ord * 3 * PAIRS;
    double K[PER][4];  // row component, column component
    bool bad = false;
#pragma unroll
    for (int m = 0; m < PER; ++m) {
        const int t = lane + 32 * m, b = t / NB, a = t - b * NB;
        if (t >= PAIRS) continue;
        const double N = nn * __ldg(tab + 2 * PAIRS + t);
        double r0, r1;
        if (s.neumann) {
            r0 = -N * s.value[0];
            r1 = -N * s.value[1];
        } else {
            const int o = a * NB + b;
            const double ik = __ldg(tab + (x ? 0 : PAIRS) + t), jk = s.beta * __ldg(tab + (x ? 0 : PAIRS) + o);
            const double it = __ldg(tab + (x ? PAIRS : 0) + t), jt = s.beta * __ldg(tab + (x ? PAIRS : 0) + o);
            const double k0 = fma(kk, jk - ik, N), k1 = fma(tt, jk - ik, N);
            const double kt = fma(mt, jt, -lt * it), tk = fma(lt, jt, -mt * it);
            K[m][0] = x ? k0 : k1;
            K[m][1] = x ? kt : tk;
            K[m][2] = x ? tk : kt;
            K[m][3] = x ? k1 : k0;
            const int j = (cj + b / (P + 1)) * p.nb[0] + ci + b % (P + 1);
            const double u0 = (p.u ? __ldg(p.u + j) : 0.0) - s.value[0], u1 = (p.u ? __ldg(p.u + nu + j) : 0.0) - s.value[1];
            r0 = fma(K[m][0], u0, K[m][1] * u1);
            r1 = fma(K[m][2], u0, K[m][3] * u1);
#pragma unroll
            for (int k = 0; k < 4; ++k) bad |= !fem_finite(K[m][k]);
        }
        sm[warp][t][0] = r0;
        sm[warp][t][1] = r1;
    }
    __syncwarp();
    double r = 0.0;
    const int ra = lane % NB, rf = lane / NB;
    if (rf < 2)
#pragma unroll
        for (int b = 0; b < NB; ++b) r += sm[warp][b * NB + ra][rf];
    cudaGridDependencySynchronize();  // the sums of the kernel before
    if (rf < 2 && p.rhs)
        atomicAdd(p.rhs + rf * nu + (cj + ra / (P + 1)) * p.nb[0] + ci + ra % (P + 1), r);
    if (p.vals && !s.neumann) {
#pragma unroll
        for (int m = 0; m < PER; ++m) {
            const int t = lane + 32 * m, b = t / NB, a = t - b * NB;
            if (t >= PAIRS) continue;
            const int rx = ci + a % (P + 1), ry = cj + a / (P + 1), row = ry * p.nb[0] + rx;
            const int lx = max(rx - P, 0), cx = min(rx + P, p.nb[0] - 1) - lx + 1;
            const int ly = max(ry - P, 0), cy = min(ry + P, p.nb[1] - 1) - ly + 1;
            const int at = (cj + b / (P + 1) - ly) * cx + ci + b % (P + 1) - lx, ul = cx * cy;
            double* v0 = p.vals + __ldg(p.rowptr + row) + at;
            double* v1 = p.vals + __ldg(p.rowptr + nu + row) + at;
            atomicAdd(v0, K[m][0]);
            atomicAdd(v0 + ul, K[m][1]);
            atomicAdd(v1, K[m][2]);
            atomicAdd(v1 + ul, K[m][3]);
        }
        if (bad) atomicOr(p.status, 1);
    }
}

struct Lattice {
    int dim = 3, p = 0;
    bool brick = true;  // axis-aligned cells (FEM_GPU_SHAPE_RECTANGULAR)
    int ne[3], nn[3], nb[3];
    int64_t pitch = 0;
    DeviceBuf mem;     // all of the following
    DeviceBuf jac;     // half edge lengths and their reciprocals
    DeviceBuf S, vec;  // block stencil; quadratic splines: nodal vectors
    DeviceBuf Q;       // density sets: element sums
    cudaEvent_t done = nullptr;  // the last use of S, vec and Q
};

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

// weights of the splines at a node along one axis (splines i .. i + p - 1 of node i)
const double* axis_weights(int p) {
    static const double w[3][3] = {{1.0}, {0.5, 0.5}, {1.0 / 6.0, 4.0 / 6.0, 1.0 / 6.0}};
    return w[p - 1];
}

// the lattice of a mesh, or nothing where any of its properties does not hold
// exactly (the extraction weights of order 3, which are not dyadic, up to 1e-15)
bool find_lattice(const fem_gpu_ctx* c, Lattice& L, std::vector<double>& jac) {
    const int D = c->dim;
    L.brick = c->shape == FEM_GPU_SHAPE_RECTANGULAR;
    if ((D == 2 && !L.brick) || c->num_used != c->num_bases || c->num_cells < 1) return false;
    const double* X = c->coords.data();
    const int64_t N = c->num_nodes;
    // edges from the first cell's nodes: (0, 1) is nn0, (0, 0, 1) is nn0 nn1
    int64_t nn[3] = {c->cells[3], 1, 1}, step[3] = {1, nn[0], 1};
    if (nn[0] < 2) return false;
    if (D == 3) {
        step[2] = c->cells[4];
        if (step[2] < nn[0] || step[2] % nn[0]) return false;
        nn[1] = step[2] / nn[0];
    }
    if (N % step[D - 1]) return false;
    nn[D - 1] = N / step[D - 1];
    const int64_t width = c->t_off[1];
    L.dim = D;
    L.p = 0;
    for (int p = 1; p <= 4 - D + 1; ++p)
        if (width == (D == 2 ? p * p : p * p * p)) L.p = p;
    if (!L.p) return false;
    int64_t cells = 1, bases = 1;
    for (int d = 0; d < 3; ++d) {
        L.nn[d] = (int)nn[d];
        L.ne[d] = d < D ? (int)nn[d] - 1 : 1;
        L.nb[d] = d < D ? L.ne[d] + L.p : 1;
        if (d >= D) continue;
        if (nn[d] < 2 || nn[d] > 1 << 20) return false;
        cells *= L.ne[d];
        bases *= L.nb[d];
        for (int e = 0; L.brick && e < L.ne[d]; ++e) {
            jac.push_back(0.5 * (X[(e + 1) * step[d] * D + d] - X[e * step[d] * D + d]));
            if (!(jac.back() > 0.0)) return false;
        }
    }
    if (c->num_cells != cells || c->num_bases != bases) return false;
    // layers of nodes, cells and bases (rows of them in a plane), shared among threads
    const double* w1 = axis_weights(L.p);
    const double tol = L.p == 3 ? 1e-15 : 0.0;
    const int last = D - 1, npe = D == 2 ? 4 : 8;
    static const int corner[8][3] = {{0, 0, 0}, {1, 0, 0}, {1, 1, 0}, {0, 1, 0},
                                     {0, 0, 1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1}};
    const auto layer = [&](int l) {
        int64_t lo[3] = {0, 0, 0}, n[3] = {nn[0], nn[1], nn[2]};
        lo[last] = l;
        n[last] = l + 1;
        // nodes: coordinates and extraction rows
        for (int64_t z = lo[2]; z < n[2] && l < nn[last]; ++z)
            for (int64_t y = lo[1]; y < n[1]; ++y)
                for (int64_t x = 0; x < nn[0]; ++x) {
                    const int64_t at = (z * nn[1] + y) * nn[0] + x;
                    if (L.brick && (X[at * D] != X[x * D] || X[at * D + 1] != X[y * step[1] * D + 1] ||
                                    (D == 3 && X[at * D + 2] != X[z * step[2] * D + 2])))
                        return false;
                    int64_t k = c->t_off[at];
                    if (k != at * width || c->t_off[at + 1] != k + width) return false;
                    for (int c2 = 0; c2 < (D == 3 ? L.p : 1); ++c2)
                        for (int b = 0; b < L.p; ++b)
                            for (int a = 0; a < L.p; ++a, ++k) {
                                const int64_t basis = ((z + c2) * L.nb[1] + y + b) * L.nb[0] + x + a;
                                const double w = w1[a] * w1[b] * (D == 3 ? w1[c2] : 1.0);
                                if (c->t_bases[k] != basis || !(std::abs(c->t_w[k] - w) <= tol)) return false;
                            }
                }
        // cells: node numbering
        for (int d = 0; d < 3; ++d) n[d] = L.ne[d];
        n[last] = l + 1;
        for (int64_t z = lo[2]; z < n[2] && l < L.ne[last]; ++z)
            for (int64_t y = lo[1]; y < n[1]; ++y)
                for (int64_t x = 0; x < L.ne[0]; ++x) {
                    const int64_t e = (z * L.ne[1] + y) * L.ne[0] + x;
                    for (int a = 0; a < npe; ++a)
                        if (c->cells[e * npe + a] !=
                            ((z + corner[a][2]) * nn[1] + y + corner[a][1]) * nn[0] + x + corner[a][0])
                            return false;
                }
        // CSR rows: the full box of bases within p along every axis (the bulk set
        // puts the box into every row, so equal lengths are equal rows)
        for (int d = 0; d < 3; ++d) n[d] = L.nb[d];
        n[last] = l + 1;
        const auto box = [&](int d, int64_t i) {
            return std::min<int64_t>(i + L.p, L.nb[d] - 1) - std::max<int64_t>(i - L.p, 0) + 1;
        };
        for (int64_t z = lo[2]; z < n[2] && l < L.nb[last]; ++z)
            for (int64_t y = lo[1]; y < n[1]; ++y) {
                const int64_t yz = box(1, y) * (D == 3 ? box(2, z) : 1);
                for (int64_t x = 0; x < L.nb[0]; ++x)
                    if (c->ulen[(z * L.nb[1] + y) * L.nb[0] + x] != yz * box(0, x)) return false;
            }
        return true;
    };
    const int layers = L.nb[last];
    const int nt = (int)std::min<int64_t>({16, std::max(1u, std::thread::hardware_concurrency()), 1 + N / 16384});
    std::atomic<bool> ok{true};
    std::vector<std::thread> th;
    for (int t = 0; t < nt; ++t)
        th.emplace_back([&, t] {
            for (int l = t; l < layers && ok.load(std::memory_order_relaxed); l += nt)
                if (!layer(l)) ok.store(false, std::memory_order_relaxed);
        });
    for (auto& t : th) t.join();
    if (!ok) return false;
    L.pitch = (L.nn[0] + 3) / 4 * 4;
    for (size_t k = 0, n = jac.size(); k < n; ++k) jac.push_back(1.0 / jac[k]);
    return true;
}

}  // namespace

void lattice_release(fem_gpu_ctx* c);

// tables and facets of a side set of a plane lattice (identity projection)
static cudaError_t plane_side_upload(const fem_gpu_ctx* c, const Lattice& L, SetData& s, cudaStream_t st) {
    for (int i = 0; i < 2; ++i)
        for (int j = 0; j < 2; ++j)
            if (s.side_select[i * 3 + j] != (i == j ? 1.0 : 0.0)) return cudaSuccess;
    if (c->num_cells >= (int64_t)1 << 29) return cudaSuccess;
    const Rule r = gauss_rule(s.side.integration_rule);
    const int p1 = L.p + 1, NB = p1 * p1, PAIRS = NB * NB;
    std::vector<double> tab((size_t)4 * 3 * PAIRS, 0.0);
    static const int corner[4][2] = {{0, 0}, {1, 0}, {1, 1}, {0, 1}};
    for (int o = 0; o < 4; ++o)
        for (int q = 0; q < r.n; ++q) {
            const int k = o & 1 ? 0 : 1;
            double xi[2], N[4], dN[8], B[16] = {}, dB[2][16] = {};
            xi[k] = o == 1 || o == 2 ? 1.0 : -1.0;
            xi[1 - k] = r.pts[q * r.dim];
            lagrange(FEM_GPU_CELL_QUAD4, xi, N, dN);
            for (int n = 0; n < 4; ++n)
                for (int b = 0; b < L.p; ++b)
                    for (int a = 0; a < L.p; ++a) {
                        const double w = axis_weights(L.p)[a] * axis_weights(L.p)[b];
                        const int f = (corner[n][1] + b) * p1 + corner[n][0] + a;
                        B[f] += w * N[n];
                        for (int i = 0; i < 2; ++i) dB[i][f] += w * dN[i * 4 + n];
                    }
            for (int b = 0; b < NB; ++b)
                for (int a = 0; a < NB; ++a) {
                    double* t = &tab[(size_t)o * 3 * PAIRS + b * NB + a];
                    for (int i = 0; i < 2; ++i) t[i * PAIRS] += r.w[q] * B[a] * dB[i][b];
                    t[2 * PAIRS] += r.w[q] * B[a] * B[b];
                }
        }
    std::vector<int32_t> facet(s.neq);
    for (int64_t i = 0; i < s.neq; ++i) facet[i] = s.ip_cell[i] * 4 + s.ordinal[i];
    s.side_wsum = 0.0;
    for (double w : r.w) s.side_wsum += w;
    cudaError_t e = upload(s.d_ptab, tab, st);
    if (e == cudaSuccess) e = upload(s.d_pfacet, facet, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e;
}

// Finds out whether the model is a lattice and which of its bulk sets cover
// every cell exactly once; those are assembled here (SetData::lattice).
fem_gpu_status lattice_finalize(fem_gpu_ctx* c) {
    Lattice L;
    std::vector<double> jac;
    cudaStream_t st = (cudaStream_t)c->stream;
    bool any = false;
    // bricks that neither assembly nor product would take this way (lattice_pays)
    if (c->dim == 3 && c->shape == FEM_GPU_SHAPE_RECTANGULAR && c->num_cells < kLatticeCells) return FEM_GPU_OK;
    for (const SetData& s : c->sets) any |= s.kind == 0 && s.ig_off.empty() && s.neq == c->num_cells;
    if (!any || !find_lattice(c, L, jac)) return FEM_GPU_OK;
    cudaError_t e = cudaSuccess;
    any = false;
    for (SetData& s : c->sets) {
        if (s.kind != 0 || !s.ig_off.empty() || s.neq != c->num_cells) continue;
        const int rule = s.bulk.integration_rule;
        if (c->dim == 3 ? rule != FEM_GPU_RULE_HEX_2x2x2 && rule != FEM_GPU_RULE_HEX_3x3x3
                        : rule != FEM_GPU_RULE_QUAD_2x2 || !s.node_rho.empty())
            continue;
        std::vector<char> seen(c->num_cells, 0);
        bool once = true, ordered = true;
        for (int64_t i = 0; i < s.neq; ++i) {
            once &= !seen[s.ip_cell[i]];
            seen[s.ip_cell[i]] = 1;
            ordered &= s.ip_cell[i] == i;
        }
        // cells of any shape: the modulus and the coordinates in the set's order
        if (!once || (!L.brick && (!ordered || !s.node_rho.empty()))) continue;
        if (!ordered && e == cudaSuccess) {
            std::vector<double> E(s.neq);
            for (int64_t i = 0; i < s.neq; ++i) E[s.ip_cell[i]] = s.E[i];
            e = upload(s.d_latE, E, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        }
        if (!s.node_rho.empty() && e == cudaSuccess) e = upload(s.d_latrho, s.node_rho, st);
        s.lattice = any = true;
    }
    if (!any) return FEM_GPU_OK;
    if (c->dim == 2)
        for (SetData& s : c->sets)
            if (s.kind == 1 && s.neq > 0 && e == cudaSuccess) e = plane_side_upload(c, L, s, st);
    auto* K = new Lattice(L);
    c->lattice = K;
    // workspaces (243 doubles per node, 0.22 of the CSR values for quadratic and as
    // much as them for linear splines; quadratic: six nodal values per node; density
    // sets: 63 doubles per cell), one allocation; a device that cannot hold them keeps
    // the element loop
    bool rho = false;
    for (const SetData& s : c->sets) rho |= s.lattice && !s.node_rho.empty();
    const bool quad = c->dim == 3 && K->p == 2;
    const bool stencil = quad || (c->dim == 3 && L.brick && (rho || c->num_nodes >= kRowsNodes));
    const size_t want[4] = {jac.size(), stencil ? (size_t)243 * L.nn[2] * L.nn[1] * L.pitch : 0,
                            quad ? (size_t)6 * c->num_nodes : 0,
                            rho ? (size_t)kQN * (L.ne[0] + 2) * (L.ne[1] + 2) * (L.ne[2] + 2) : 0};
    DeviceBuf* const buf[4] = {&K->jac, &K->S, &K->vec, &K->Q};
    size_t at[4], bytes = 0;
    for (int k = 0; k < 4; ++k) {
        at[k] = bytes;
        buf[k]->bytes = want[k] * sizeof(double);
        bytes += (buf[k]->bytes + 255) / 256 * 256;
    }
    if (e == cudaSuccess) e = cudaMalloc(&K->mem.p, std::max<size_t>(bytes, 256));
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        cudaStreamSynchronize(st);
        lattice_release(c);
        return FEM_GPU_OK;
    }
    for (int k = 0; k < 4; ++k) buf[k]->p = want[k] ? (char*)K->mem.p + at[k] : nullptr;
    if (e == cudaSuccess && !jac.empty())
        e = cudaMemcpyAsync(K->jac.p, jac.data(), K->jac.bytes, cudaMemcpyHostToDevice, st);
    if (rho && e == cudaSuccess) e = cudaMemsetAsync(K->Q.p, 0, K->Q.bytes, st);
    if (K->S.p && e == cudaSuccess) e = cudaEventCreateWithFlags(&K->done, cudaEventDisableTiming);
    if (K->done && e == cudaSuccess) e = cudaEventRecord(K->done, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? FEM_GPU_OK
                            : fail(c, FEM_GPU_CUDA_ERROR, std::string("lattice data: ") + cudaGetErrorString(e));
}

void lattice_release(fem_gpu_ctx* c) {
    for (SetData& s : c->sets) {
        dfree(s.d_latE);
        dfree(s.d_latrho);
        dfree(s.d_ptab);
        dfree(s.d_pfacet);
        s.lattice = false;
    }
    Lattice* L = (Lattice*)c->lattice;
    if (!L) return;
    dfree(L->mem);
    if (L->done) cudaEventDestroy(L->done);
    delete L;
    c->lattice = nullptr;
}

namespace {

fem_gpu_status plane_assemble(fem_gpu_ctx* c, const Lattice& L, const SetData& s, const double* u, double* vals,
                              double* rhs, bool acc_v, bool acc_r) {
    PlaneArgs a{};
    for (int d = 0; d < 2; ++d) {
        a.ne[d] = L.ne[d];
        a.nb[d] = L.nb[d];
    }
    a.E = (const double*)(s.d_latE.p ? s.d_latE.p : s.d_E.p);
    a.jac = (const double*)L.jac.p;
    a.u = rhs ? u : nullptr;
    a.vals = vals;
    a.rhs = rhs;
    a.rowptr = (const int32_t*)c->d_rowptr.p;
    a.acc_v = acc_v;
    a.acc_r = acc_r;
    a.status = (int*)c->d_status.p;
    const double nu = s.bulk.poisson_ratio;
    const double lam = s.bulk.model_type == FEM_GPU_MODEL_PLANE_STRESS ? nu / (1.0 - nu * nu)
                                                                       : nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
    a.mu = 1.0 / (2.0 * (1.0 + nu));
    a.ld = (lam + a.mu) / a.mu;
    a.lo = lam / a.mu;
    // 1-D matrices from the rule's points along one axis (unit weights of the 2 x 2 rule)
    const Rule r = gauss_rule(s.bulk.integration_rule);
    double T[2][4] = {};  // extraction of the element's two nodes
    for (int k = 0; k < L.p; ++k) T[0][k] = T[1][k + 1] = axis_weights(L.p)[k];
    const double x = std::abs(r.pts[0]);
    for (int i = 0; i <= L.p; ++i)
        for (int j = 0; j <= L.p; ++j)
            for (int n = 0; n < 2; ++n)
                for (int m = 0; m < 2; ++m)
                    for (const double q : {-x, x}) {
                        const double sn = n ? 0.5 : -0.5, sm = m ? 0.5 : -0.5, w = T[n][i] * T[m][j];
                        a.M[i][j] += w * (0.5 + sn * q) * (0.5 + sm * q);
                        a.D[i][j] += w * sn * sm;
                        a.G[i][j] += w * sn * (0.5 + sm * q);
                    }
    const unsigned g = (unsigned)((c->num_used + 31) / 32);
    cudaStream_t st = (cudaStream_t)c->stream;
    if (L.p == 1) lattice_plane<1><<<g, 96, 0, st>>>(a);
    else if (L.p == 2) lattice_plane<2><<<g, 160, 0, st>>>(a);
    else lattice_plane<3><<<g, 224, 0, st>>>(a);
    c->launches++;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FEM_GPU_OK
                            : fail(c, FEM_GPU_CUDA_ERROR, std::string("lattice launch: ") + cudaGetErrorString(e));
}

// The workspaces of one call.  A matrix-free product returns before it has run, so a call
// waits for the one before it, whatever its stream: a handle does not name a stream (that
// of a destroyed stream is given out again), and on the stream of the call before the wait
// is empty.  Memory of its own, instead, has a captured call, which may be replayed beside
// any other (nodes of the graph), and a product on the per-thread default stream, one handle
// for a stream of every thread that goes with its thread: ordered by events, products of two
// threads that ended while they were pending left cudaDeviceSynchronize waiting.  (An
// assembly has run when it returns.)
struct LatticeWork {
    Lattice& L;
    cudaStream_t st;
    bool shared = true;
    void *S, *vec, *Q;
    cudaError_t e = cudaSuccess;
    LatticeWork(Lattice& l, cudaStream_t stream, bool stencil)
        : L(l), st(stream), S(l.S.p), vec(l.vec.p), Q(l.Q.p) {
        if (!L.done) return;
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) cudaGetLastError();
        if (cs == cudaStreamCaptureStatusActive || (st == cudaStreamPerThread && !stencil)) {
            shared = false;
            S = vec = Q = nullptr;
            if (L.S.p && stencil) e = cudaMallocAsync(&S, L.S.bytes, st);
            if (L.vec.p && e == cudaSuccess) e = cudaMallocAsync(&vec, L.vec.bytes, st);
            if (L.Q.p && e == cudaSuccess) e = cudaMallocAsync(&Q, L.Q.bytes, st);
            if (Q && e == cudaSuccess) e = cudaMemsetAsync(Q, 0, L.Q.bytes, st);
        } else {
            e = cudaStreamWaitEvent(st, L.done, 0);
        }
    }
    ~LatticeWork() {
        if (!shared) {
            for (void* p : {S, vec, Q})
                if (p) cudaFreeAsync(p, st);
        } else if (L.done) {
            cudaEventRecord(L.done, st);
        }
    }
};

}  // namespace

// One lattice set: CSR values (nullable) and residual (nullable) of the adof
// vector u (nullable), stored, or added with acc_v / acc_r.
fem_gpu_status lattice_assemble(fem_gpu_ctx* c, int set, const double* u, double* vals, double* rhs, bool acc_v,
                                bool acc_r) {
    Lattice& L = *(Lattice*)c->lattice;
    const SetData& s = c->sets[set];
    if (L.dim == 2) return plane_assemble(c, L, s, u, vals, rhs, acc_v, acc_r);
    cudaStream_t st = (cudaStream_t)c->stream;
    const int64_t nodes = (int64_t)L.nn[0] * L.nn[1] * L.nn[2];
    const bool quad = L.p == 2;
    LatticeWork work(L, st, vals != nullptr);
    cudaError_t e = work.e;
    if (e != cudaSuccess)
        return fail(c, FEM_GPU_CUDA_ERROR, std::string("lattice workspace: ") + cudaGetErrorString(e));
    LatArgs a{};
    for (int d = 0; d < 3; ++d) {
        a.ne[d] = L.ne[d];
        a.nn[d] = L.nn[d];
    }
    a.pitch = L.pitch;
    a.E = (const double*)(s.d_latE.p ? s.d_latE.p : s.d_E.p);
    a.jac = (const double*)L.jac.p;
    const int32_t* rowptr = (const int32_t*)c->d_rowptr.p;
    a.rho = s.node_rho.empty() ? nullptr : (const double*)s.d_latrho.p;
    a.status = (int*)c->d_status.p;
    a.vals = vals;
    a.rowptr = rowptr;
    a.acc_v = acc_v;
    a.S = (double*)work.S;
    a.Q = (double*)work.Q;
    double* un = (double*)work.vec;
    double* rn = un + 3 * nodes;
    const bool want_u = u && rhs;
    a.u = want_u ? (quad ? un : u) : nullptr;
    a.r = rhs ? (quad ? rn : rhs) : nullptr;
    a.acc_r = quad ? 0 : acc_r;
    // material and rule: T^T S T with T = P / 8 is P^T (S / 64) P (exact powers of two)
    const double nu = s.bulk.poisson_ratio, scale = quad ? 1.0 / 64.0 : 1.0;
    const double lam = nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), mu = 1.0 / (2.0 * (1.0 + nu));
    a.ld = (lam + mu) / mu;
    a.lo = lam / mu;
    a.beta = s.bulk.density_exponent;
    const Rule r = gauss_rule(s.bulk.integration_rule);
    const int N = r.n == 8 ? 2 : 3;
    for (int i = 0; i < N; ++i) a.xq[i] = N == 2 ? (i ? -r.pts[0] : r.pts[0]) : (i - 1) * -r.pts[0];
    // the rule's points to tensor order, weights with the material factor and the 1/64 of the shape functions
    for (int q = 0; q < r.n; ++q) {
        int at = 0, mul = 1;
        for (int d = 0; d < 3; ++d, mul *= N) {
            const double x = r.pts[q * 3 + d];
            at += mul * (N == 2 ? x > 0.0 : x < 0.0 ? 0 : x > 0.0 ? 2 : 1);
        }
        a.wq[at] = r.w[q] * mu * scale / 64.0;
    }
    if (L.brick && !a.rho) {
        // coefficients of every offset: the reference sums for the element and
        // nodes that lattice_const counts with a plus sign
        for (int k = 0; k < 27; ++k) {
            const int d[3] = {k % 3 - 1, k / 3 % 3 - 1, k / 9 - 1};
            double sa[3], sb[3];  // corner signs of the row node and its neighbour in that element
            for (int i = 0; i < 3; ++i) {
                sa[i] = d[i] > 0 ? -1.0 : 1.0;
                sb[i] = d[i] < 0 ? -1.0 : 1.0;
            }
            double G[3][3] = {};
            for (int q = 0; q < N * N * N; ++q) {
                const double x[3] = {a.xq[q % N], a.xq[q / N % N], a.xq[q / (N * N)]};
                double ga[3], gb[3];
                for (int i = 0; i < 3; ++i) {
                    ga[i] = sa[i];
                    gb[i] = sb[i];
                    for (int o = 0; o < 3; ++o)
                        if (o != i) {
                            ga[i] *= 1.0 + sa[o] * x[o];
                            gb[i] *= 1.0 + sb[o] * x[o];
                        }
                }
                for (int i = 0; i < 3; ++i)
                    for (int j = 0; j < 3; ++j) G[i][j] += a.wq[q] * ga[i] * gb[j];
            }
            double* o = a.coef[k];
            for (int i = 0; i < 3; ++i) o[i] = G[i][i];
            int m = 3;
            static const int fg[6][2] = {{0, 1}, {0, 2}, {1, 0}, {1, 2}, {2, 0}, {2, 1}};
            for (const auto& q : fg) o[m++] = a.lo * G[q[0]][q[1]] + G[q[1]][q[0]];
        }
    }
    const unsigned grid3 = (unsigned)sm_count() * 16;
    // the kernels of a call overlap their beginnings with the end of the one before
    // (4 to 6 launches of 4 to 40 us on small lattices)
    bool overlap = false;
    // a product of bricks with constant moduli, and cells of any shape, add to what they
    // find
    const bool product = L.brick && !a.rho && !vals;
    if ((product || (a.rho && a.r)) && !a.acc_r) e = cudaMemsetAsync(a.r, 0, 3 * nodes * sizeof(double), st);
    if (!L.brick) {
        if (quad && vals) e = cudaMemsetAsync(a.S, 0, L.S.bytes, st);
        if (!quad && vals && !acc_v) e = cudaMemsetAsync(vals, 0, c->nnz * sizeof(double), st);
        if (e == cudaSuccess && rhs && !a.acc_r) e = cudaMemsetAsync(a.r, 0, 3 * nodes * sizeof(double), st);
    }
    if (quad && want_u) {
        lattice_nodal<<<(unsigned)std::min<int64_t>((3 * nodes + 255) / 256, grid3), 256, 0, st>>>(
            L.nn[0], L.nn[1], L.nn[2], u, un);
        c->launches++;
        overlap = true;
    }
    if (!L.brick) {
        HexArgs h{};
        for (int d = 0; d < 3; ++d) {
            h.ne[d] = L.ne[d];
            h.nn[d] = L.nn[d];
        }
        h.pitch = L.pitch;
        h.E = a.E;
        h.xe = (const double*)s.d_xe.p;
        for (int i = 0; i < N; ++i) h.xq[i] = a.xq[i];
        for (int i = 0; i < r.n; ++i) h.wq[i] = 64.0 * a.wq[i];
        h.ld = a.ld;
        h.lo = a.lo;
        h.u = a.u;
        h.r = a.r;
        h.S = a.S;
        h.vals = vals;
        h.rowptr = rowptr;
        h.status = a.status;
        const unsigned g = (unsigned)((c->num_cells + kHexWarps - 1) / kHexWarps);
        using Fn = void (*)(HexArgs);
        static const Fn cells[2][2] = {{hex_cells<2, HEX_STENCIL>, hex_cells<2, HEX_CSR>},
                                       {hex_cells<3, HEX_STENCIL>, hex_cells<3, HEX_CSR>}};
        const Fn hex = vals ? cells[N == 3][quad ? HEX_STENCIL : HEX_CSR] : N == 2 ? hex_residual<2> : hex_residual<3>;
        if (e == cudaSuccess && (vals || want_u)) {
            e = launch_kernel(hex, g, 32 * kHexWarps, 0, st, overlap, h);
            c->launches++;
            overlap = true;
        }
    }
    const unsigned ctas = (unsigned)((nodes + kStencilNodes - 1) / kStencilNodes);
    const int out = vals ? OUT_STENCIL : OUT_NONE;
    const bool direct = !quad && !a.rho && nodes < kRowsNodes;
    using Fn = void (*)(LatArgs);
    static const Fn density[2] = {lattice_density<OUT_NONE>, lattice_density<OUT_STENCIL>};
    if (a.rho) {
        const unsigned g = (unsigned)std::min<int64_t>((c->num_cells + 127) / 128, (int64_t)sm_count() * 64);
        if (N == 2) lattice_moments<2><<<g, 128, 0, st>>>(a);
        else lattice_moments<3><<<g, 128, 0, st>>>(a);
        density[out]<<<ctas, kDensityThreads, 0, st>>>(a);
        c->launches += 2;
        overlap = true;
    } else if (product && e == cudaSuccess) {
        a.wmu = mu * scale / 8.0;
        const unsigned g = (unsigned)((c->num_cells + 127) / 128);
        if (want_u) e = launch_kernel(lattice_product, g, 128, 0, st, overlap, a);
        c->launches += want_u;
        overlap |= want_u;
    } else if (L.brick && e == cudaSuccess) {
        e = launch_kernel(direct ? lattice_const<OUT_CSR> : lattice_const<OUT_STENCIL>, ctas, kStencilThreads, 0, st, overlap, a);
        c->launches++;
        overlap = true;
    }
    if (quad && rhs && e == cudaSuccess) {
        e = launch_kernel(lattice_restrict, (unsigned)std::min<int64_t>((3 * (c->num_used) + 255) / 256, grid3), 256, 0,
                          st, overlap, L.nn[0], L.nn[1], L.nn[2], rn, 8.0, acc_r, rhs);
        c->launches++;
    }
    if (!quad && L.brick && vals && !direct && e == cudaSuccess) {
        e = launch_kernel(lattice_rows, dim3(ctas, 3), 256, 0, st, overlap, L.nn[0], L.nn[1], L.nn[2], L.pitch,
                          (const double*)a.S, rowptr, vals, (int)acc_v);
        c->launches++;
    }
    if (quad && vals && e == cudaSuccess) {
        ProjArgs q{};
        for (int d = 0; d < 3; ++d) {
            q.nn[d] = L.nn[d];
            q.nb[d] = L.nb[d];
        }
        q.tx = (L.nb[0] + kPX - 1) / kPX;
        q.ty = (L.nb[1] + kPY - 1) / kPY;
        q.pitch = L.pitch;
        q.S = a.S;
        q.vals = vals;
        q.rowptr = rowptr;
        q.acc = acc_v;
        q.status = a.status;
        // z ranges: every range repeats one node plane, and the CTAs should fill
        // whole waves; the count with the fewest plane steps in sequence
        const int64_t tiles = (int64_t)q.tx * q.ty * 3, slots = (int64_t)sm_count() * kProjCtas;
        int64_t best = INT64_MAX;
        for (int n = 1; n <= q.nb[2]; ++n) {
            const int64_t steps = (tiles * n + slots - 1) / slots * ((q.nb[2] + n - 1) / n + 1);
            if (steps < best) {
                best = steps;
                q.chunks = n;
            }
        }
        e = cudaFuncSetAttribute(lattice_project, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kProjSmem);
        if (e == cudaSuccess)
            e = launch_kernel(lattice_project, dim3((unsigned)tiles, (unsigned)q.chunks), kProjThreads, kProjSmem, st,
                              overlap, q);
        c->launches++;
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? FEM_GPU_OK
                            : fail(c, FEM_GPU_CUDA_ERROR, std::string("lattice launch: ") + cudaGetErrorString(e));
}

// The side sets among `sets` (at most kPlaneSides of a launch) of a plane lattice,
// added to vals and rhs; see fem_launch.cuh for overlap (u is read ahead of the wait).
fem_gpu_status lattice_sides(fem_gpu_ctx* c, const std::vector<int>& sets, const double* u, double* vals, double* rhs,
                             bool overlap) {
    const Lattice& L = *(const Lattice*)c->lattice;
    PlaneSides a{};
    for (int d = 0; d < 2; ++d) {
        a.ne[d] = L.ne[d];
        a.nb[d] = L.nb[d];
    }
    a.jac = (const double*)L.jac.p;
    a.u = u;
    a.vals = vals;
    a.rhs = rhs;
    a.rowptr = (const int32_t*)c->d_rowptr.p;
    a.status = (int*)c->d_status.p;
    cudaError_t e = cudaSuccess;
    for (size_t k = 0; k < sets.size() && e == cudaSuccess; k += kPlaneSides) {
        int64_t most = 0;
        const int n = (int)std::min<size_t>(kPlaneSides, sets.size() - k);
        for (int m = 0; m < n; ++m) {
            const SetData& s = c->sets[sets[k + m]];
            PlaneSide& q = a.set[m];
            q.n = s.neq;
            q.facet = (const int32_t*)s.d_pfacet.p;
            q.E = (const double*)s.d_E.p;
            q.tab = (const double*)s.d_ptab.p;
            q.neumann = s.side.iwg_type == FEM_GPU_IWG_STRUC_LINEAR_NEUMANN;
            const double nu = s.side.poisson_ratio;
            q.lam = s.side.model_type == FEM_GPU_MODEL_PLANE_STRESS ? nu / (1.0 - nu * nu)
                                                                    : nu / ((1.0 + nu) * (1.0 - 2.0 * nu));
            q.mu = 1.0 / (2.0 * (1.0 + nu));
            q.alpha = s.side.nitsche_alpha;
            q.beta = s.side.iwg_type == FEM_GPU_IWG_STRUC_LINEAR_DIRICHLET_SYMMETRIC_NITSCHE ? -1.0 : 1.0;
            q.thickness = s.side_thickness;
            q.wsum = s.side_wsum;
            for (int d = 0; d < 2; ++d) q.value[d] = s.side.value[d];
            most = std::max(most, q.n);
        }
        const dim3 grid((unsigned)((most + kPlaneSideWarps - 1) / kPlaneSideWarps), (unsigned)n);
        void (*const fn)(PlaneSides) = L.p == 1   ? lattice_plane_sides<1>
                                       : L.p == 2 ? lattice_plane_sides<2>
                                                  : lattice_plane_sides<3>;
        e = launch_kernel(fn, grid, 32 * kPlaneSideWarps, 0, (cudaStream_t)c->stream, overlap, a);
        c->launches++;
        overlap = true;
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? FEM_GPU_OK
                            : fail(c, FEM_GPU_CUDA_ERROR, std::string("side launch: ") + cudaGetErrorString(e));
}

}  // namespace fem
