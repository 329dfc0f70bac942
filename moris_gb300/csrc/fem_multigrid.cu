// fem_multigrid.cu -- geometric multigrid V-cycle for the assembled operator of
// a uniform linear-B-spline hex mesh (the config-5 SIMP solves).
//
// The reference offers a PETSc PCMG preconditioner (Preconditioner_PETSc::
// build_multigrid_preconditioner, SOL/DLA/src/cl_DLA_Preconditioner_PETSc.cpp:
// 77-345): a multiplicative V-cycle with Galerkin coarse operators
// A_(l+1) = P^T A_l P (PC_MG_GALERKIN_BOTH), prolongations from the B-spline
// two-scale relation (Geometric_Multigrid, SOL/DLA/src/cl_DLA_Geometric_
// Multigrid.cpp:47-121, HMR get_fine_basis_weights_of_basis), SOR smoothing
// and an LU coarse solve.  The same preconditioner, laid out for the GPU:
//
//   * levels l = 0..L of node grids n_l^3, n_(l+1) = (n_l - 1) / 2 + 1.  The
//     linear B-spline two-scale relation is trilinear interpolation: coarse
//     node I weighs fine node i by prod_d (1 - |i_d - 2 I_d| / 2);
//   * every operator is a 27-point block stencil S[k][f][g][node]
//     (tap k = (dx+1) + 3 (dy+1) + 9 (dz+1); f, g displacement components)
//     with the node index fastest, so a warp reads 32 consecutive nodes of one
//     coefficient; level 0 is scattered from the CSR, level l+1 = P^T S_l P is
//     formed on the device one axis at a time (P is a Kronecker product of
//     1D two-scale relations), each pass a thread per node and component pair;
//   * smoothing is Chebyshev-accelerated point Jacobi of degree `degree` on
//     [lo, hi] * lambda_max(D^-1 A) (lambda_max by power iteration): SOR is
//     sequential, a polynomial in D^-1 A is one stencil sweep per degree.  Pre-
//     and post-smoothing use the same polynomial, so the V-cycle is a
//     symmetric positive definite operator;
//   * the coarsest level (n_L <= coarse_max) is solved with its dense inverse,
//     formed by Gauss-Jordan elimination on the device (the operator is SPD,
//     so no pivoting), 16 pivots per launch;
//   * the finest fp32_levels levels smooth, restrict and prolong in FP32 (an
//     FP32 copy of the stencil, FP32 vectors): the FP64 stencil sweep is bound
//     by the FP64 pipe (243 FMAs per node), the FP32 one by HBM.  The V-cycle
//     is a preconditioner inside an FP64 Krylov method, whose true residual
//     decides convergence.
// Vectors are type-major like the adof vector: v[g n_l^3 + node].  All work
// is issued on the legacy default stream, like fem_gpu_fcg.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>
#include <chrono>
#include <cmath>
#include <cstring>
#include <vector>

#include "fem_internal.hpp"
#include "fem_launch.cuh"
#include "fem_reduce.cuh"

using fem::fail;
using fem::launch_kernel;

namespace {

__host__ __device__ __forceinline__ int64_t sidx(int k, int f, int g, int64_t N, int64_t i) {
    return (int64_t)((k * 3 + f) * 3 + g) * N + i;
}

constexpr int kTpb = 256;  // threads per block of every kernel that sums

// level-0 stencil from the CSR of the assembled operator (one thread per row);
// err |= 1 for a column outside the 27-node neighbourhood
// One CTA per block of kCsRows consecutive rows: their nonzeros are one contiguous
// range of the CSR, loaded coalesced into shared memory; then kCsPart threads
// per row take its entries with stride kCsPart, the lanes of a warp on 32
// consecutive rows with the same part.  Consecutive rows are consecutive
// nodes, and interior rows have the same column pattern, so a warp's lanes
// write entry p of 32 neighbouring nodes: consecutive words of one tap.  A block whose range exceeds the
// staging space (rows longer than 27 x 3 entries, which are an error anyway)
// reads from global memory.
constexpr int kCsRows = 64, kCsPart = 8, kCsCap = kCsRows * 81;
constexpr size_t kCsSmem = (size_t)kCsCap * (sizeof(double) + sizeof(int32_t));
__global__ void __launch_bounds__(kCsPart * kCsRows) mg_csr_to_stencil(int n, const int32_t* __restrict__ rp,
                                                               const int32_t* __restrict__ ci,
                                                               const double* __restrict__ v,
                                                               double* __restrict__ S, int* err) {
    extern __shared__ __align__(16) unsigned char cs_smem[];
    double* sv = reinterpret_cast<double*>(cs_smem);
    int32_t* sc = reinterpret_cast<int32_t*>(sv + kCsCap);
    // 32-bit throughout (3 N rows and their nonzeros are int32 in the CSR): the kernel is
    // bound by its index operations: 438 -> 286 us at 65^3 nodes
    const int N = n * n * n, rows = 3 * N, n2 = n * n;
    for (int r0 = blockIdx.x * kCsRows; r0 < rows; r0 += gridDim.x * kCsRows) {
        const int r1 = r0 + kCsRows < rows ? r0 + kCsRows : rows;
        const int e0 = rp[r0], e1 = rp[r1];
        const bool staged = e1 - e0 <= kCsCap;
        if (staged)
            for (int e = threadIdx.x; e < e1 - e0; e += kCsPart * kCsRows) {
                sv[e] = v[e0 + e];
                sc[e] = ci[e0 + e];
            }
        __syncthreads();
        const int row = r0 + threadIdx.x % kCsRows;
        if (row < r1) {
            const int f = (row >= N) + (row >= 2 * N), i = row - f * N;
            const int ix = i % n, iy = i / n % n, iz = i / n2;
            const int b = rp[row + 1];
            double* Si = S + (int64_t)(f * 3) * N + i;
            for (int e = rp[row] + threadIdx.x / kCsRows; e < b; e += kCsPart) {
                const int col = staged ? sc[e - e0] : ci[e];
                // component and node offset d = j - i without divisions: d =
                // dx + n dy + n^2 dz with |dx|, |dy|, |dz| <= 1 is split by
                // sign tests (n >= 3); any other column leaves |dx| > 1 or a
                // neighbour outside the grid and is flagged
                const int g = (col >= N) + (col >= 2 * N);
                int d = col - g * N - i;
                const int dz = (d > n2 / 2) - (d < -(n2 / 2));
                d -= dz * n2;
                const int dy = (d > n / 2) - (d < -(n / 2));
                d -= dy * n;
                if ((unsigned)col >= (unsigned)rows || (unsigned)(d + 1) > 2u || (unsigned)(ix + d) >= (unsigned)n ||
                    (unsigned)(iy + dy) >= (unsigned)n || (unsigned)(iz + dz) >= (unsigned)n) {
                    atomicOr(err, 1);
                    continue;
                }
                Si[(int64_t)((d + 1 + 3 * (dy + 1) + 9 * (dz + 1)) * 9 + g) * N] = staged ? sv[e - e0] : v[e];
            }
        }
        __syncthreads();
    }
}

__global__ void mg_diag_inv(int64_t N, const double* __restrict__ S, double* __restrict__ dinv) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < 3 * N; t += (int64_t)gridDim.x * blockDim.x) {
        const int f = (int)(t / N);
        const double d = S[sidx(13, f, f, N, t - f * N)];
        dinv[t] = d != 0.0 ? 1.0 / d : 0.0;
    }
}

// out(t, pre(t), (A x)_t) for every row t = f N + i of a stencil; pre loads what out
// needs, ahead of the sum.  A warp takes 32 consecutive nodes and one of the nine
// (dz, dy) rows of neighbours (FP32; one dz plane in FP64, whose pipe also pays for
// the sums over the warps): its 27 coefficients and 9 values per lane are loads that
// do not wait for one another, where a thread per node walked the nine rows one after
// the other.  The rows meet in shared memory; warp f ends component f.
// Measured, FP32 Chebyshev step, thread per node -> here: 9^3 nodes 23 -> 4.0 us,
// 17^3 22.5 -> 4.3, 33^3 24 -> 9.4, 65^3 59 -> 46.7 (5.9 TB/s; with the coefficients
// in 243 planes instead of tiles 57).  FP64 product at 65^3: 121 -> 124 us, 107 of
// them FP64 instructions.
template <typename TV>
struct Sweep {
    static constexpr int G = sizeof(TV) == 4 ? 9 : 3, threads = 32 * G, per_sm = sizeof(TV) == 4 ? 4 : 10;
};
template <typename TS, typename TV, typename L, typename F>
__device__ __forceinline__ void stencil_sweep(int n, const TS* __restrict__ S, const TV* x, L&& pre, F&& out) {
    constexpr int G = Sweep<TV>::G;
    __shared__ TV red[G][3][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int N = n * n * n;  // 243 N doubles are on the device: N < 2^28
    bool first = true;
    for (int i0 = blockIdx.x * 32; i0 < N; i0 += gridDim.x * 32) {
        const int i = i0 + lane, ic = min(i, N - 1);
        const int ix = ic % n, iy = ic / n % n, iz = ic / (n * n);
        // FP32: 243 x 32 coefficients of the tile in sequence (mg_stencil32)
        const int64_t tap = sizeof(TS) == 4 ? 32 : N;
        const TS* Si = S + (sizeof(TS) == 4 ? (int64_t)(i0 / 32) * (243 * 32) + lane : ic);
        const int64_t t = (int64_t)(w < 3 ? w : 0) * N + ic;
        decltype(pre(t)) own{};
        TV s[3] = {TV(0), TV(0), TV(0)};
#pragma unroll
        for (int r = 0; r < 9 / G; ++r) {
            const int row = w * (9 / G) + r, dz = row / 3 - 1, dy = row % 3 - 1;
            const bool in = (unsigned)(iz + dz) < (unsigned)n && (unsigned)(iy + dy) < (unsigned)n;
            const TS* Sr = Si + 27 * row * tap;
            const TV* xr = x + ic + n * (dy + n * dz);
            TS c[27];  // FP32: loaded here (27 FP64 values would not fit the registers)
            if constexpr (sizeof(TS) == 4) {
#pragma unroll
                for (int k = 0; k < 27; ++k) c[k] = __ldg(Sr + k * tap);
            }
            if (first) {
                // the coefficients do not change during a solve: their first loads run
                // beside the end of the kernel before
                cudaGridDependencySynchronize();
                cudaTriggerProgrammaticLaunchCompletion();
                first = false;
            }
            if (r == 0 && w < 3) own = pre(t);
            TV xg[3][3];
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                const bool inx = in && (unsigned)(ix + dx) < (unsigned)n;
#pragma unroll
                for (int g = 0; g < 3; ++g) xg[dx + 1][g] = inx ? xr[(int64_t)g * N + dx] : TV(0);
            }
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int g = 0; g < 3; ++g)
#pragma unroll
                    for (int f = 0; f < 3; ++f) {
                        const int k = (d * 3 + f) * 3 + g;
                        s[f] = fma((TV)(sizeof(TS) == 4 ? c[k] : __ldg(Sr + k * tap)), xg[d][g], s[f]);
                    }
        }
#pragma unroll
        for (int f = 0; f < 3; ++f) red[w][f][lane] = s[f];
        __syncthreads();
        if (w < 3) {
            TV v = red[0][w][lane];
#pragma unroll
            for (int k = 1; k < G; ++k) v += red[k][w][lane];
            if (i < N) out(t, own, v);
        }
        __syncthreads();
    }
}
unsigned sweep_blocks(int64_t N) { return (unsigned)((N + 31) / 32); }
// of a sweep that ends in a block sum: two rounds of resident blocks (an atomic each)
template <typename TV>
unsigned sum_sweep_blocks(int64_t N) {
    return std::min<unsigned>(sweep_blocks(N), (unsigned)fem::sm_count() * Sweep<TV>::per_sm * 2);
}

// power iteration step: y = D^-1 A (a x), a = 1 / sqrt(*xx) (1 without xx: x
// is the previous step's y, normalised here instead of in a pass of its own);
// dots += y.y (in the level's precision; xx and dots in parts)
template <typename TS, typename TV>
__global__ void __launch_bounds__(Sweep<TV>::threads, Sweep<TV>::per_sm) mg_power(int n, const TS* __restrict__ S, const TV* dinv, const TV* x,
                         const double* __restrict__ xx, TV* y, double* dots) {
    // the scale by one warp: FP64 roots and divisions in every warp took the pipe longer
    // than the sums of the sweep (65^3 nodes 56 -> 48 us with it and the sums in parts, 33^3
    // 17 -> 11); read behind the first barrier of the sweep
    __shared__ TV scale;
    if (threadIdx.x < 32) {
        const double d = xx ? fem::parts_total(xx) : 1.0;
        if (threadIdx.x == 0) scale = (TV)(d > 0.0 ? 1.0 / sqrt(d) : 0.0);
    }
    double acc = 0.0;
    stencil_sweep<TS, TV>(n, S, x, [&](int64_t t) { return dinv[t]; }, [&](int64_t t, TV d, TV s) {
        const TV v = d * s * scale;
        y[t] = v;
        acc += (double)v * (double)v;
    });
    const double sum[1] = {acc};
    fem::block_sum_add<Sweep<TV>::threads, 1, 1>(sum, {fem::part_of(dots)});
}

template <typename TV>
__global__ void mg_sumsq(int64_t m, const TV* __restrict__ x, double* dots) {
    double acc = 0.0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x)
        acc += (double)x[t] * (double)x[t];
    const double sum[1] = {acc};
    fem::block_sum_add<kTpb, 1, 1>(sum, {fem::part_of(dots)});
}

template <typename TV>
__global__ void mg_scale(int64_t m, double a, const TV* __restrict__ y, TV* __restrict__ x) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x)
        x[t] = (TV)(a * (double)y[t]);
}
// splitmix64 uniform in [-0.5, 0.5): element t of the stream of `seed`
__global__ void mg_random(int64_t m, uint64_t seed, double* __restrict__ x) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
        uint64_t z = seed + (uint64_t)(t + 1) * 0x9E3779B97F4A7C15ULL;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        z ^= z >> 31;
        x[t] = (double)(z >> 11) * (1.0 / 9007199254740992.0) - 0.5;
    }
}

template <typename TA, typename TB>
__global__ void mg_convert(int64_t m, const TA* a, TB* b) {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x)
        b[t] = (TB)a[t];
}

// FP32 copy of a stencil in tiles of 32 nodes, S32[tile][tap][32]: a block of a sweep
// reads 31 KB in sequence, where 243 planes of the node grid were as many DRAM streams
// of one (for odd N misaligned) line each
__global__ void mg_stencil32(int64_t N, const double* __restrict__ S, float* __restrict__ S32) {
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * 32 + lane;
    float* b = S32 + (int64_t)blockIdx.x * (243 * 32) + lane;
#pragma unroll 8
    for (int k = threadIdx.x >> 5; k < 243; k += kTpb / 32) b[k * 32] = i < N ? (float)S[k * N + i] : 0.0f;
}

// q = A p on an FP64 stencil and dot += p.q (the outer Krylov product)
__global__ void __launch_bounds__(Sweep<double>::threads, Sweep<double>::per_sm)
    mg_apply_dot(int n, const double* __restrict__ S, const double* p, double* q,
                 double* dot) {
    double acc = 0.0;
    stencil_sweep<double, double>(n, S, p, [&](int64_t t) { return p[t]; }, [&](int64_t t, double pt, double s) {
        q[t] = s;
        acc = fma(pt, s, acc);
    });
    const double sum[1] = {acc};
    fem::block_sum_add<Sweep<double>::threads, 1, 1>(sum, {fem::part_of(dot)});
}

// Chebyshev start with x = 0: r = b, d = D^-1 b / theta, x = d
template <typename TB, typename TV>
__global__ void mg_cheb_init(int64_t m, const TB* b, const TV* __restrict__ dinv, TV inv_theta, TV* r, TV* d, TV* x) {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < m; t += (int64_t)gridDim.x * blockDim.x) {
        const TV bt = (TV)b[t];
        const TV dt = dinv[t] * bt * inv_theta;
        r[t] = bt;
        d[t] = dt;
        x[t] = dt;
    }
}

template <typename TV>
struct Row {
    TV r, d, dinv, x;
};

// Chebyshev step: r -= A din; dout = c1 din + c2 D^-1 r; x += dout
template <typename TS, typename TV>
__global__ void __launch_bounds__(Sweep<TV>::threads, Sweep<TV>::per_sm)
    mg_cheb_step(int n, const TS* __restrict__ S, const TV* din, TV* r,
                 const TV* dinv, TV c1, TV c2, TV* dout, TV* x) {
    stencil_sweep<TS, TV>(
        n, S, din, [&](int64_t t) { return Row<TV>{r[t], din[t], dinv[t], x[t]}; },
        [&](int64_t t, const Row<TV>& o, TV s) {
            const TV rt = o.r - s;
            const TV dt = fma(c1, o.d, c2 * o.dinv * rt);
            r[t] = rt;
            dout[t] = dt;
            x[t] = o.x + dt;
        });
}

// r -= A d
template <typename TS, typename TV>
__global__ void __launch_bounds__(Sweep<TV>::threads, Sweep<TV>::per_sm)
    mg_residual_update(int n, const TS* __restrict__ S, const TV* d, TV* r) {
    stencil_sweep<TS, TV>(n, S, d, [&](int64_t t) { return r[t]; },
                          [&](int64_t t, TV rt, TV s) { r[t] = rt - s; });
}

// first post-smoothing step after the coarse correction e:
// r -= A e; d = D^-1 r / theta; x += e + d
template <typename TS, typename TV>
__global__ void __launch_bounds__(Sweep<TV>::threads, Sweep<TV>::per_sm)
    mg_post_first(int n, const TS* __restrict__ S, const TV* e, TV* r,
                  const TV* dinv, TV inv_theta, TV* d, TV* x) {
    stencil_sweep<TS, TV>(
        n, S, e, [&](int64_t t) { return Row<TV>{r[t], e[t], dinv[t], x[t]}; },
        [&](int64_t t, const Row<TV>& o, TV s) {
            const TV rt = o.r - s;
            const TV dt = o.dinv * rt * inv_theta;
            r[t] = rt;
            d[t] = dt;
            x[t] = o.x + (o.d + dt);
        });
}

// full-weighting restriction bc = P^T r (fine grid nf = 2 (nc - 1) + 1), a thread per
// coarse row, the 27 loads independent
template <typename TF, typename TC>
__global__ void mg_restrict(int nf, int nc, const TF* r, TC* bc) {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const int Nc = nc * nc * nc, Nf = nf * nf * nf;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 3 * Nc; t += gridDim.x * blockDim.x) {
        const int g = t / Nc, I = t - g * Nc;
        const int X = I % nc, Y = I / nc % nc, Z = I / (nc * nc);
        const TF* rg = r + (int64_t)g * Nf + 2 * (X + nf * (Y + nf * Z));
        TF s = TF(0);
#pragma unroll
        for (int az = -1; az <= 1; ++az)
#pragma unroll
            for (int ay = -1; ay <= 1; ++ay)
#pragma unroll
                for (int ax = -1; ax <= 1; ++ax) {
                    const bool in = (unsigned)(2 * X + ax) < (unsigned)nf && (unsigned)(2 * Y + ay) < (unsigned)nf &&
                                    (unsigned)(2 * Z + az) < (unsigned)nf;
                    const TF w = TF((ax ? 0.5 : 1.0) * (ay ? 0.5 : 1.0) * (az ? 0.5 : 1.0));
                    s = fma(w, in ? rg[ax + nf * (ay + nf * az)] : TF(0), s);
                }
        bc[t] = (TC)s;
    }
}

// trilinear prolongation e = P xc
template <typename TC, typename TF>
__global__ void mg_prolong(int nf, int nc, const TC* xc, TF* e) {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const int Nc = nc * nc * nc, Nf = nf * nf * nf;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 3 * Nf; t += gridDim.x * blockDim.x) {
        const int g = t / Nf, i = t - g * Nf;
        const int x = i % nf, y = i / nf % nf, z = i / (nf * nf);
        const TC wx = (x & 1) ? TC(0.5) : TC(1), wy = (y & 1) ? TC(0.5) : TC(1), wz = (z & 1) ? TC(0.5) : TC(1);
        const TC* c = xc + (int64_t)g * Nc + (x >> 1) + nc * ((y >> 1) + nc * (z >> 1));
        TC v[2][2][2];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int a = k & 1, b = k >> 1 & 1, d = k >> 2;
            const bool in = (!a || (x & 1)) && (!b || (y & 1)) && (!d || (z & 1));
            v[d][b][a] = in ? c[a + nc * (b + nc * d)] : TC(0);
        }
        const TC s = ((v[0][0][0] + v[0][0][1]) + (v[0][1][0] + v[0][1][1])) +
                     ((v[1][0][0] + v[1][0][1]) + (v[1][1][0] + v[1][1][1]));
        e[t] = (TF)(s * wx * wy * wz);
    }
}

// 1D two-scale targets: fine offset sum s (a + b) reaches the coarse tap s / 2
// (weight 1) when even, the two taps (s -+ 1) / 2 (weight 1/2 each) when odd
__device__ __forceinline__ int ntarget(int s) { return (s & 1) ? 2 : 1; }
__device__ __forceinline__ int target(int s, int t) { return (s & 1) ? ((s - 1) >> 1) + t : (s >> 1); }

// err |= 2 where the level-0 operator is not symmetric (A_ij vs A_ji beyond
// the rounding of the assembly's atomic sums, relative to the entries and to
// the diagonals of rows i and j)
__global__ void mg_check_symmetric(int n, const double* __restrict__ S, int* err) {
    // one thread per node I: every tap k <= 13 and component pair (f, g) of row
    // I against the mirrored entry (26 - k, g, f) of the neighbour J; threads of
    // a warp are consecutive nodes, so both operands load coalesced.  An
    // element adds the same value to both entries in one scatter, so they are
    // usually equal to the bit: an integer comparison (finite values only)
    // settles a pair, and the tolerance test on the FP64 pipe runs only when a
    // lane of the warp needs it.  The loop bound is uniform per warp, so every
    // vote sees all 32 lanes (blockDim a multiple of 32).
    const int64_t N = (int64_t)n * n * n;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    bool bad = false;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < N; base += stride) {
        const int64_t I = base + (threadIdx.x & 31);
        const bool live = I < N;
        const int X = live ? (int)(I % n) : 0, Y = live ? (int)((I / n) % n) : 0,
                  Z = live ? (int)(I / ((int64_t)n * n)) : 0;
        for (int k = 0; k <= 13; ++k) {
            const int dx = k % 3 - 1, dy = (k / 3) % 3 - 1, dz = k / 9 - 1;
            const bool inside = live && X + dx >= 0 && X + dx < n && Y + dy >= 0 && Y + dy < n && Z + dz >= 0 &&
                                Z + dz < n;
            const int64_t J = I + dx + (int64_t)n * (dy + (int64_t)n * dz);
#pragma unroll
            for (int f = 0; f < 3; ++f)
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    double a = 0.0, b = 0.0;
                    if (inside) {
                        a = S[sidx(k, f, g, N, I)];
                        b = S[sidx(26 - k, g, f, N, J)];
                    }
                    const long long ab = __double_as_longlong(a);
                    const bool same = ab == __double_as_longlong(b) && ((ab >> 52) & 0x7ff) != 0x7ff;
                    if (__all_sync(0xffffffffu, same)) continue;
                    if (!same) {
                        // entries that cancel to near zero carry the rounding of
                        // their terms, which scales with the diagonals: measure the
                        // asymmetry against them too (in FP32: a square root on the
                        // FP64 pipe costs far more)
                        const float di = fabsf((float)S[sidx(13, f, f, N, I)]);
                        const float dj = fabsf((float)S[sidx(13, g, g, N, J)]);
                        const float tol = 1e-10f * (float)(fabs(a) + fabs(b)) + 1e-12f * sqrtf(di * dj);
                        bad |= !((float)fabs(a - b) <= tol);
                    }
                }
        }
    }
    if (bad) atomicOr(err, 2);
}

// One-axis Galerkin coarsening of a 27-point block stencil: P = P_z (x) P_y (x)
// P_x is separable, so P^T S P is three passes, each coarsening one axis of an
// (nx, ny, nz) node box with the 1D two-scale relation while the taps along
// the other two axes pass through.  One thread per output node and component
// pair; the 3 x 3 (a, b) pairs along the axis times the 9 taps across it are
// unrolled (117 FMAs for the 27 output taps).
__host__ __device__ __forceinline__ int tap_of(int AX, int along, int o1, int o2) {
    int d[3];
    d[AX] = along;
    d[(AX + 1) % 3] = o1;
    d[(AX + 2) % 3] = o2;
    return (d[0] + 1) + 3 * (d[1] + 1) + 9 * (d[2] + 1);
}

template <int AX>
__global__ void __launch_bounds__(128) mg_rap_axis(int3 din, int3 dout, const double* __restrict__ Sin,
                                                   double* __restrict__ Sout) {
    const int64_t Nin = (int64_t)din.x * din.y * din.z, Nout = (int64_t)dout.x * dout.y * dout.z;
    const int nin_ax = AX == 0 ? din.x : AX == 1 ? din.y : din.z;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < 9 * Nout;
         t += (int64_t)gridDim.x * blockDim.x) {
        const int fg = (int)(t / Nout);
        const int64_t I = t - fg * Nout;
        const int f = fg / 3, g = fg % 3;
        int c[3] = {(int)(I % dout.x), (int)((I / dout.x) % dout.y), (int)(I / ((int64_t)dout.x * dout.y))};
        const int C = c[AX];
        double acc[27];
#pragma unroll
        for (int k = 0; k < 27; ++k) acc[k] = 0.0;
#pragma unroll
        for (int a = -1; a <= 1; ++a) {
            const int fc = 2 * C + a;
            if (fc < 0 || fc >= nin_ax) continue;
            int ci[3] = {c[0], c[1], c[2]};
            ci[AX] = fc;
            const int64_t i = ci[0] + (int64_t)din.x * (ci[1] + (int64_t)din.y * ci[2]);
            const double wa = a ? 0.5 : 1.0;
#pragma unroll
            for (int b = -1; b <= 1; ++b) {
                const int sm = a + b;
                const double pw = (sm & 1) ? 0.5 : 1.0;
#pragma unroll
                for (int o2 = -1; o2 <= 1; ++o2)
#pragma unroll
                    for (int o1 = -1; o1 <= 1; ++o1) {
                        const double v = wa * pw * __ldg(Sin + sidx(tap_of(AX, b, o1, o2), f, g, Nin, i));
#pragma unroll
                        for (int tt = 0; tt < 2; ++tt) {
                            if (tt >= ntarget(sm)) continue;
                            acc[tap_of(AX, target(sm, tt), o1, o2)] += v;
                        }
                    }
            }
        }
#pragma unroll
        for (int k = 0; k < 27; ++k) Sout[sidx(k, f, g, Nout, I)] = acc[k];
    }
}

// dense operator of the coarsest level, row-major m x m (m = 3 N)
__global__ void mg_dense(int n, const double* __restrict__ S, double* __restrict__ A) {
    const int64_t N = (int64_t)n * n * n, m = 3 * N;
    for (int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; row < m; row += (int64_t)gridDim.x * blockDim.x) {
        const int f = (int)(row / N);
        const int64_t i = row - f * N;
        const int ix = (int)(i % n), iy = (int)((i / n) % n), iz = (int)(i / ((int64_t)n * n));
        for (int k = 0; k < 27; ++k) {
            const int dx = k % 3 - 1, dy = (k / 3) % 3 - 1, dz = k / 9 - 1;
            if (ix + dx < 0 || ix + dx >= n || iy + dy < 0 || iy + dy >= n || iz + dz < 0 || iz + dz >= n) continue;
            const int64_t j = i + dx + (int64_t)n * (dy + (int64_t)n * dz);
            for (int g = 0; g < 3; ++g) A[row * m + g * N + j] = S[sidx(k, f, g, N, i)];
        }
    }
}

// Gauss-Jordan inversion, kGj pivots at a time, from A to B (two buffers, so the
// pivot rows and columns are read from the previous step without a copy): with K
// the pivot rows, P = A_KK^-1 and Y = P A_K. (columns of K: P itself),
//   B_K. = Y,   B_i. = A_i. - A_iK Y  (A_iK read as 0 in the first term).
// One CTA per 32 x 32 tile; every CTA inverts the 16 x 16 pivot block itself (a
// thread per entry, one barrier per pivot; > 0 pivots of an SPD operator, so no
// pivoting).  One launch per pivot was latency-bound: 375 unknowns (the 5^3
// coarsest grid) took 1.97 ms, here 24 launches take 0.42 ms.
constexpr int kGj = 16, kGjTile = 32;
__global__ void __launch_bounds__(kGj * kGj) mg_gj_block(int m, const double* __restrict__ A, double* __restrict__ B,
                                                         int k0) {
    __shared__ double P[2][kGj][kGj + 1], Y[kGj][kGjTile + 1], C[kGjTile][kGj + 1], inv[kGj];
    const int tid = threadIdx.x, i = tid / kGj, j = tid % kGj;
    const int nk = min(kGj, m - k0), i0 = blockIdx.y * kGjTile, j0 = blockIdx.x * kGjTile;
    // a short last block is completed with the identity
    const double d = i < nk && j < nk ? A[(int64_t)(k0 + i) * m + k0 + j] : (i == j ? 1.0 : 0.0);
    P[0][i][j] = d;
    if (tid == 0) inv[0] = 1.0 / d;
    for (int t = tid; t < kGjTile * kGj; t += kGj * kGj) {
        const int r = t / kGj, k = t % kGj;
        C[r][k] = i0 + r < m && k < nk ? A[(int64_t)(i0 + r) * m + k0 + k] : 0.0;
        const int kk = t / kGjTile, c = t % kGjTile;
        Y[kk][c] = kk < nk && j0 + c < m ? A[(int64_t)(k0 + kk) * m + j0 + c] : 0.0;
    }
    __syncthreads();
    for (int k = 0; k < kGj; ++k) {
        const double(*a)[kGj + 1] = P[k & 1];
        const double rk = (j == k ? 1.0 : a[k][j]) * inv[k];
        const double v = i == k ? rk : (j == k ? 0.0 : a[i][j]) - a[i][k] * rk;
        P[(k + 1) & 1][i][j] = v;
        if (i == k + 1 && j == k + 1) inv[k + 1] = 1.0 / v;
        __syncthreads();
    }
    static_assert(kGj % 2 == 0, "the inverse ends in the first buffer");
    // Y = P A_K. (in place through registers)
    double y[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int c = j + h * kGj, col = j0 + c - k0;
        double s = 0.0;
        for (int k = 0; k < kGj; ++k) s = fma(P[0][i][k], Y[k][c], s);
        y[h] = col >= 0 && col < nk ? P[0][i][col] : s;
    }
    __syncthreads();
    Y[i][j] = y[0];
    Y[i][j + kGj] = y[1];
    __syncthreads();
    for (int t = tid; t < kGjTile * kGjTile; t += kGj * kGj) {
        const int r = t / kGjTile, c = t % kGjTile, row = i0 + r, col = j0 + c;
        if (row >= m || col >= m) continue;
        double v;
        if (row >= k0 && row < k0 + nk) {
            v = Y[row - k0][c];
        } else {
            v = col >= k0 && col < k0 + nk ? 0.0 : A[(int64_t)row * m + col];
            for (int k = 0; k < kGj; ++k) v = fma(-C[r][k], Y[k][c], v);
        }
        B[(int64_t)row * m + col] = v;
    }
}

// x = Ainv b, one warp per row
__global__ void mg_gemv(int64_t m, const double* __restrict__ A, const double* b, double* x) {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < m; row += warps) {
        double s = 0.0;
        for (int64_t j = lane; j < m; j += 32) s = fma(A[row * m + j], b[j], s);
        s = fem::warp_total(s);
        if (lane == 0) x[row] = s;
    }
}

unsigned blocks_for(int64_t work, int tpb) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((work + tpb - 1) / tpb, (int64_t)fem::sm_count() * 32));
}
// of a sum over short rows of work: fewer blocks, each ends with a block sum
unsigned sum_blocks(int64_t work, int tpb) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((work + tpb - 1) / tpb, (int64_t)fem::sm_count() * 4));
}

}  // namespace

struct fem_mg {
    struct Level {
        int n = 0;
        int64_t N = 0;
        bool fp32 = false;        // smoothing and vectors in FP32
        double* S = nullptr;      // FP64 stencil (Galerkin products, power iteration, FP64 smoothing)
        float* S32 = nullptr;     // FP32 copy of an FP32 level
        double* dinv = nullptr;
        float* dinv32 = nullptr;
        double lmax = 0.0;
        // vectors in the level's precision; level 0 of an FP64 hierarchy uses the caller's b and x
        void *x = nullptr, *b = nullptr, *r = nullptr, *d0 = nullptr, *d1 = nullptr;
    };
    std::vector<Level> lv;
    double* ainv = nullptr;  // dense inverse of the coarsest operator
    int64_t m = 0;
    fem_mg_opts o{};
    double setup_seconds = 0.0;
    double* pdots = nullptr;  // power-iteration norms (power_iters + 1)
    int* err = nullptr;
    // all arrays in one allocation (45 of their own cost a millisecond to make and
    // another to free): reserved one by one, then placed by commit()
    struct Arena {
        char* base = nullptr;
        size_t bytes = 0;
        std::vector<std::pair<void**, size_t>> at;
        template <typename T>
        void reserve(T** p, size_t count) {
            at.push_back({(void**)p, bytes});
            bytes += (count * sizeof(T) + 255) / 256 * 256;
        }
        bool commit() {
            if (cudaMalloc((void**)&base, bytes) != cudaSuccess) {
                base = nullptr;
                return false;
            }
            for (auto& [p, o] : at) *p = base + o;
            return true;
        }
        ~Arena() {
            if (base) cudaFree(base);
        }
    } arena;
    ~fem_mg() { cudaDeviceSynchronize(); }
};

namespace {

template <typename TV>
struct Cheb {
    TV inv_theta, delta, sigma;
    explicit Cheb(const fem_mg::Level& L, const fem_mg_opts& o) {
        const double lo = o.lo_frac * L.lmax, hi = o.hi_frac * L.lmax;
        const double theta = 0.5 * (hi + lo), dl = 0.5 * (hi - lo);
        inv_theta = (TV)(1.0 / theta);
        delta = (TV)dl;
        sigma = (TV)(theta / dl);
    }
};

// Chebyshev pre-smoothing from x = 0; on return r = b - A x
template <typename TS, typename TB, typename TV>
void smooth_pre(const fem_mg::Level& L, const TS* S, const TV* dinv, const fem_mg_opts& o, const TB* b, TV* x,
                bool overlap) {
    const Cheb<double> c(L, o);
    const unsigned vb = blocks_for(3 * L.N, kTpb), nb = sweep_blocks(L.N);
    TV *r = (TV*)L.r, *din = (TV*)L.d0, *dout = (TV*)L.d1;
    launch_kernel(mg_cheb_init<TB, TV>, vb, kTpb, 0, 0, overlap, 3 * L.N, b, dinv, (TV)c.inv_theta, r, din, x);
    double rho = 1.0 / c.sigma;
    for (int k = 1; k < o.degree; ++k) {
        const double rn = 1.0 / (2.0 * c.sigma - rho);
        launch_kernel(mg_cheb_step<TS, TV>, nb, Sweep<TV>::threads, 0, 0, true, L.n, S, din, r, dinv, (TV)(rn * rho),
                      (TV)(2.0 * rn / c.delta), dout, x);
        rho = rn;
        std::swap(din, dout);
    }
    launch_kernel(mg_residual_update<TS, TV>, nb, Sweep<TV>::threads, 0, 0, true, L.n, S, din, r);
}

// Chebyshev post-smoothing after the coarse correction e, which lives in d1:
// the first step reads it and writes d0, after which d1 is free for the ping-pong
template <typename TS, typename TV>
void smooth_post(const fem_mg::Level& L, const TS* S, const TV* dinv, const fem_mg_opts& o, const TV* e, TV* x) {
    const Cheb<double> c(L, o);
    const unsigned nb = sweep_blocks(L.N);
    TV *r = (TV*)L.r, *din = (TV*)L.d0, *dout = (TV*)L.d1;
    launch_kernel(mg_post_first<TS, TV>, nb, Sweep<TV>::threads, 0, 0, true, L.n, S, e, r, dinv, (TV)c.inv_theta, din,
                  x);
    double rho = 1.0 / c.sigma;
    for (int k = 1; k < o.degree; ++k) {
        const double rn = 1.0 / (2.0 * c.sigma - rho);
        launch_kernel(mg_cheb_step<TS, TV>, nb, Sweep<TV>::threads, 0, 0, true, L.n, S, din, r, dinv, (TV)(rn * rho),
                      (TV)(2.0 * rn / c.delta), dout, x);
        rho = rn;
        std::swap(din, dout);
    }
}

void vcycle(fem_mg* g, size_t l, const void* b, void* x);

// smoothing, restriction, the coarser cycle, prolongation on a level of vector type
// TV; b in the type of the caller.  Every kernel but the first of a cycle overlaps the
// one before it: on the coarse levels (4 us a kernel) the launch and the loads of the
// coefficients were half the time.  13 FCG iterations at 65^3 nodes 7.4 -> 6.5 ms, 11 at
// 17^3 1.27 -> 0.86.
template <typename TV, typename TB>
void level_cycle(fem_mg* g, size_t l, const TB* b, TV* x) {
    fem_mg::Level& L = g->lv[l];
    fem_mg::Level& C = g->lv[l + 1];
    constexpr bool f32 = std::is_same<TV, float>::value;
    if constexpr (f32) smooth_pre(L, L.S32, L.dinv32, g->o, b, x, l > 0);
    else smooth_pre(L, L.S, L.dinv, g->o, b, x, l > 0);
    const unsigned cb = blocks_for(3 * C.N, kTpb), fb = blocks_for(3 * L.N, kTpb);
    if (C.fp32) launch_kernel(mg_restrict<TV, float>, cb, kTpb, 0, 0, true, L.n, C.n, (const TV*)L.r, (float*)C.b);
    else launch_kernel(mg_restrict<TV, double>, cb, kTpb, 0, 0, true, L.n, C.n, (const TV*)L.r, (double*)C.b);
    vcycle(g, l + 1, C.b, C.x);
    TV* e = (TV*)L.d1;
    if (C.fp32) launch_kernel(mg_prolong<float, TV>, fb, kTpb, 0, 0, true, L.n, C.n, (const float*)C.x, e);
    else launch_kernel(mg_prolong<double, TV>, fb, kTpb, 0, 0, true, L.n, C.n, (const double*)C.x, e);
    if constexpr (f32) smooth_post(L, L.S32, L.dinv32, g->o, e, x);
    else smooth_post(L, L.S, L.dinv, g->o, e, x);
}

// x_l = V_l(b_l) in the level's precision
void vcycle(fem_mg* g, size_t l, const void* b, void* x) {
    if (l + 1 == g->lv.size()) {  // coarsest level: FP64 dense inverse
        launch_kernel(mg_gemv, blocks_for(g->m * 32, kTpb), kTpb, 0, 0, true, g->m, g->ainv, (const double*)b,
                      (double*)x);
        return;
    }
    if (g->lv[l].fp32) level_cycle<float>(g, l, (const float*)b, (float*)x);
    else level_cycle<double>(g, l, (const double*)b, (double*)x);
}

// power iteration for lambda_max(D^-1 A) of a level from the seeded vector in px
// (FP64; converted for an FP32 level); px / py are finest-size scratch.  Squared
// norms on the device: pd[0] = |x0|^2, pd[it + 1] = |y_it|^2 with y_it = D^-1 A x_it
// and x_(it+1) = y_it / |y_it|, the normalisation done by the next step as it reads
// y_it.
template <typename TS, typename TV>
void power_iterate(const fem_mg::Level& L, const TS* S, const TV* dinv, double* px, double* py, int iters, double* pd) {
    const unsigned vb = blocks_for(3 * L.N, kTpb), sb = sum_blocks(3 * L.N, kTpb);
    TV *x = (TV*)px, *y = (TV*)py;
    if (!std::is_same<TV, double>::value) {
        mg_convert<double, TV><<<vb, kTpb>>>(3 * L.N, px, y);
        mg_scale<TV><<<vb, kTpb>>>(3 * L.N, 1.0, y, x);
    }
    mg_sumsq<TV><<<sb, kTpb>>>(3 * L.N, x, pd);
    for (int it = 0; it < iters; ++it) {
        mg_power<TS, TV><<<sum_sweep_blocks<TV>(L.N), Sweep<TV>::threads>>>(
            L.n, S, dinv, x, it ? pd + it * fem::kSumParts : nullptr, y,
            pd + (it + 1) * fem::kSumParts);
        std::swap(x, y);
    }
}
double power_lambda(const double* parts, int iters) {
    const auto norm = [&](int k) {
        double v = 0.0;
        for (int m = 0; m < fem::kSumParts; ++m) v += parts[k * fem::kSumParts + m];
        return std::sqrt(v);
    };
    double xn = norm(0), lam = 0.0;
    for (int it = 0; it < iters; ++it) {
        const double yn = norm(it + 1);
        lam = yn / xn;
        if (!(yn > 0.0)) break;
        xn = 1.0;
    }
    return lam;
}

}  // namespace

bool mg_operator(fem_mg* g, const double* p, double* q, double* dot) {
    if (!g) return false;
    const fem_mg::Level& L = g->lv[0];
    mg_apply_dot<<<sum_sweep_blocks<double>(L.N), Sweep<double>::threads>>>(L.n, L.S, p, q, dot);
    return cudaGetLastError() == cudaSuccess;
}

bool mg_vcycle(fem_mg* g, const double* r, double* z) {
    if (!g) return false;
    fem_mg::Level& L = g->lv[0];
    if (L.fp32) {
        level_cycle<float>(g, 0, r, (float*)L.x);
        launch_kernel(mg_convert<float, double>, blocks_for(3 * L.N, kTpb), kTpb, 0, 0, true, 3 * L.N,
                      (const float*)L.x, z);
    } else {
        vcycle(g, 0, r, z);
    }
    return cudaGetLastError() == cudaSuccess;
}

extern "C" {

fem_gpu_status fem_mg_default_opts(fem_mg_opts* o) {
    if (!o) return FEM_GPU_BAD_ARG;
    o->coarse_max = 5;
    o->degree = 2;
    o->lo_frac = 0.1;
    o->hi_frac = 1.1;
    o->power_iters = 12;
    o->fp32_levels = 8;
    return FEM_GPU_OK;
}

fem_gpu_status fem_mg_create(fem_gpu_ctx* c, const int32_t* rowptr, const int32_t* colidx, const double* vals,
                             const fem_mg_opts* opts, fem_mg** out) {
    if (!c || !rowptr || !colidx || !vals || !out) return FEM_GPU_BAD_ARG;
    *out = nullptr;
    if (!c->host_final) return FEM_GPU_NOT_FINALIZED;
    fem_mg_opts o;
    fem_mg_default_opts(&o);
    if (opts) o = *opts;
    if (o.degree < 1 || o.degree > 8 || !(o.lo_frac > 0.0) || !(o.hi_frac > o.lo_frac) || o.power_iters < 1 ||
        o.coarse_max < 3 || o.coarse_max > 9 || o.fp32_levels < 0)
        return fail(c, FEM_GPU_BAD_ARG, "multigrid: options out of range");
    const int64_t nu = c->num_used;
    const int nf = (int)std::llround(std::cbrt((double)nu));
    if (c->dim != 3 || (int64_t)nf * nf * nf != nu)
        return fail(c, FEM_GPU_BAD_ARG, "multigrid: needs a 3D model on a cubic node grid");
    std::vector<int> ns{nf};
    while (ns.back() > o.coarse_max) {
        const int n = ns.back();
        if ((n - 1) % 2) return fail(c, FEM_GPU_BAD_ARG, "multigrid: node grid edge - 1 must halve down to coarse_max");
        ns.push_back((n - 1) / 2 + 1);
    }
    if (ns.size() < 2) return fail(c, FEM_GPU_BAD_ARG, "multigrid: grid already at or below coarse_max");
    const auto t0 = std::chrono::steady_clock::now();
    fem_mg* g = new fem_mg();
    g->o = o;
    g->lv.resize(ns.size());
    const size_t iters = (size_t)o.power_iters + 1;
    fem_mg::Arena& ar = g->arena;
    ar.reserve(&g->pdots, iters * ns.size() * fem::kSumParts);
    ar.reserve(&g->err, 1);
    for (size_t l = 0; l < ns.size(); ++l) {
        fem_mg::Level& L = g->lv[l];
        L.n = ns[l];
        L.N = (int64_t)L.n * L.n * L.n;
        L.fp32 = (int)l < o.fp32_levels && l + 1 < ns.size();
        const size_t w = L.fp32 ? sizeof(float) : sizeof(double);
        ar.reserve(&L.S, 243 * L.N);
        ar.reserve(&L.dinv, 3 * L.N);
        for (void** v : {&L.r, &L.d0, &L.d1}) ar.reserve((char**)v, 3 * L.N * w);
        if (l > 0 || L.fp32)
            for (void** v : {&L.x, &L.b}) ar.reserve((char**)v, 3 * L.N * w);
        if (L.fp32) {
            ar.reserve(&L.S32, 243 * 32 * (size_t)sweep_blocks(L.N));
            ar.reserve(&L.dinv32, 3 * L.N);
        }
    }
    g->m = 3 * g->lv.back().N;
    ar.reserve(&g->ainv, g->m * g->m);
    // scratch of the setup: the boxes of the Galerkin products, the vectors of the
    // power iterations, the second buffer of the inversion
    fem_mg::Arena scratch;
    double *t1 = nullptr, *t2 = nullptr, *px = nullptr, *py = nullptr, *ainv2 = nullptr;
    {
        const int64_t n0 = ns[0], n1 = ns[1];
        scratch.reserve(&t1, 243 * n0 * n0 * n1);
        scratch.reserve(&t2, 243 * n0 * n1 * n1);
        scratch.reserve(&px, 3 * n0 * n0 * n0);
        scratch.reserve(&py, 3 * n0 * n0 * n0);
        scratch.reserve(&ainv2, g->m * g->m);
    }
    if (!ar.commit() || !scratch.commit()) {
        cudaGetLastError();
        delete g;
        return fail(c, FEM_GPU_OUT_OF_MEMORY, "multigrid hierarchy");
    }
    // level 0 from the CSR, then the Galerkin products
    fem_mg::Level& L0 = g->lv[0];
    cudaMemset(L0.S, 0, 243 * L0.N * sizeof(double));
    cudaMemset(g->err, 0, sizeof(int));
    cudaFuncSetAttribute(mg_csr_to_stencil, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCsSmem);
    mg_csr_to_stencil<<<blocks_for(3 * L0.N, kCsRows), kCsPart * kCsRows, kCsSmem>>>(L0.n, rowptr, colidx, vals,
                                                                                    L0.S, g->err);
    mg_check_symmetric<<<blocks_for(L0.N, kTpb), kTpb>>>(L0.n, L0.S, g->err);
    // Galerkin products axis by axis through two scratch boxes
    for (size_t l = 0; l + 1 < g->lv.size(); ++l) {
        const int nf = g->lv[l].n, ncs = g->lv[l + 1].n;
        const int3 a{nf, nf, nf}, b{nf, nf, ncs}, cc{nf, ncs, ncs}, d{ncs, ncs, ncs};
        mg_rap_axis<2><<<blocks_for(9 * (int64_t)b.x * b.y * b.z, 128), 128>>>(a, b, g->lv[l].S, t1);
        mg_rap_axis<1><<<blocks_for(9 * (int64_t)cc.x * cc.y * cc.z, 128), 128>>>(b, cc, t1, t2);
        mg_rap_axis<0><<<blocks_for(9 * (int64_t)d.x * d.y * d.z, 128), 128>>>(cc, d, t2, g->lv[l + 1].S);
    }
    int herr = 0;
    cudaMemcpy(&herr, g->err, sizeof(int), cudaMemcpyDeviceToHost);
    if (herr) {
        delete g;
        return fail(c, FEM_GPU_BAD_ARG, (herr & 1) ? "multigrid: operator is not a 27-point nodal stencil on the node grid"
                                                   : "multigrid: operator is not symmetric");
    }
    // smoother data: diagonal, FP32 copies, lambda_max(D^-1 A) by power iteration
    // (norms on the device, read once for all levels)
    cudaMemset(g->pdots, 0, iters * ns.size() * fem::kSumParts * sizeof(double));
    for (size_t l = 0; l + 1 < g->lv.size(); ++l) {
        fem_mg::Level& L = g->lv[l];
        const unsigned vb = blocks_for(3 * L.N, kTpb);
        mg_diag_inv<<<blocks_for(3 * L.N, kTpb), kTpb>>>(L.N, L.S, L.dinv);
        if (L.fp32) {
            mg_stencil32<<<sweep_blocks(L.N), kTpb>>>(L.N, L.S, L.S32);
            mg_convert<double, float><<<vb, kTpb>>>(3 * L.N, L.dinv, L.dinv32);
        }
        mg_random<<<vb, kTpb>>>(3 * L.N, 0x5EEDULL + l, px);
        // FP64 levels iterate on the FP64 stencil; FP32 levels on their FP32 copy
        // (the smoothing interval needs lambda_max to a few digits only)
        if (L.fp32) power_iterate<float, float>(L, L.S32, L.dinv32, px, py, o.power_iters, g->pdots + l * iters * fem::kSumParts);
        else power_iterate<double, double>(L, L.S, L.dinv, px, py, o.power_iters, g->pdots + l * iters * fem::kSumParts);
    }
    // coarsest level: dense inverse
    fem_mg::Level& LC = g->lv.back();
    cudaMemset(g->ainv, 0, g->m * g->m * sizeof(double));
    mg_dense<<<blocks_for(g->m, kTpb), kTpb>>>(LC.n, LC.S, g->ainv);
    const unsigned tiles = (unsigned)((g->m + kGjTile - 1) / kGjTile);
    double *from = g->ainv, *to = ainv2;
    for (int64_t k = 0; k < g->m; k += kGj) {
        mg_gj_block<<<dim3(tiles, tiles), kGj * kGj>>>((int)g->m, from, to, (int)k);
        std::swap(from, to);
    }
    if (from != g->ainv) cudaMemcpyAsync(g->ainv, from, g->m * g->m * sizeof(double), cudaMemcpyDeviceToDevice, 0);
    std::vector<double> norms(iters * ns.size() * fem::kSumParts, 0.0);
    if (cudaMemcpy(norms.data(), g->pdots, norms.size() * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaDeviceSynchronize() != cudaSuccess || cudaGetLastError() != cudaSuccess) {
        delete g;
        return fail(c, FEM_GPU_CUDA_ERROR, "multigrid setup");
    }
    for (size_t l = 0; l + 1 < g->lv.size(); ++l) {
        const double lam = power_lambda(norms.data() + l * iters * fem::kSumParts, o.power_iters);
        g->lv[l].lmax = lam;
        if (!(lam > 0.0) || !std::isfinite(lam)) {
            delete g;
            return fail(c, FEM_GPU_NONFINITE, "multigrid: power iteration gave no positive lambda_max");
        }
    }
    g->setup_seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    *out = g;
    return FEM_GPU_OK;
}

fem_gpu_status fem_mg_destroy(fem_mg* g) {
    delete g;
    return FEM_GPU_OK;
}

int32_t fem_mg_num_levels(const fem_mg* g) { return g ? (int32_t)g->lv.size() : 0; }

double fem_mg_setup_seconds(const fem_mg* g) { return g ? g->setup_seconds : 0.0; }

fem_gpu_status fem_mg_level_info(const fem_mg* g, int32_t level, int32_t* n, double* lambda_max) {
    if (!g || level < 0 || level >= (int32_t)g->lv.size()) return FEM_GPU_BAD_ARG;
    if (n) *n = g->lv[level].n;
    if (lambda_max) *lambda_max = g->lv[level].lmax;
    return FEM_GPU_OK;
}

fem_gpu_status fem_mg_get_stencil(const fem_mg* g, int32_t level, double* host_out) {
    if (!g || !host_out || level < 0 || level >= (int32_t)g->lv.size()) return FEM_GPU_BAD_ARG;
    const fem_mg::Level& L = g->lv[level];
    return cudaMemcpy(host_out, L.S, 243 * L.N * sizeof(double), cudaMemcpyDeviceToHost) == cudaSuccess
               ? FEM_GPU_OK
               : FEM_GPU_CUDA_ERROR;
}

fem_gpu_status fem_mg_apply(fem_mg* g, const double* r, double* z) {
    if (!g || !r || !z) return FEM_GPU_BAD_ARG;
    return mg_vcycle(g, r, z) ? FEM_GPU_OK : FEM_GPU_CUDA_ERROR;
}

}  // extern "C"
