// fem_solver.cu -- preconditioned conjugate gradients on the assembled CSR
// operator (the reference delegates this to Trilinos AztecOO AZ_cg with
// AZ_Jacobi, SOL/DLA/src/cl_DLA_Linear_Solver_Aztec.cpp:260-355).
//
// One iteration is four launches on the context stream:
//   k1  q = A p and the partial sums of p.q            (4 lanes per CSR row)
//   k2  alpha = rz/pq; x += alpha p; r -= alpha q; z = M^-1 r; sums of r.z, r.r
//   k3  convergence test; beta = rz'/rz; p = z + beta p
//   k4  (one thread) advance the iteration counter
// Scalars live in a device ring indexed by the iteration counter, so the
// launches carry no host-side values and a chunk of iterations is captured
// once into a CUDA graph and replayed.  The host reads the done flag once per
// chunk; iterations after convergence return immediately on the device.  Small
// systems, whose iteration is shorter than its launches, are solved by one cluster
// of CTAs (k_cluster_cg) or take two launches per iteration (k_pair_*).
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <mutex>
#include <string>
#include <vector>

#include "fem_internal.hpp"
#include "fem_launch.cuh"
#include "fem_reduce.cuh"
#include "fem_spmv.cuh"

namespace {

constexpr int kParts = 8;
struct CgState {
    int it;          // current iteration
    int done;        // 1 converged, 2 breakdown
    int converged_at;
    int stopped_at;  // k_pair_*: iteration whose test ended the solve
    int wide;        // a row longer than the limit given to k_diag_inv
    double thresh2;  // (rtol * ||b||)^2
    double bn2;
    // ring of per-iteration scalars: [slot][0]=pq, [1]=rz, [2]=rr
    double ring[4][4];
    // the sums p.Ap, r.z and r.r of four iterations, each in parts: an FP64 atomic of
    // every block to one address takes 10 ns, 24 us for the blocks of a large product.
    // Per iteration, one address -> parts: plane systems of 132,098 rows 27.0 -> 23.0 us,
    // 526,338 rows 67 -> 59; solids of 107,811 rows 40.1 -> 37.4, 823,875 rows 210 -> 197.
    double part[4][3][kParts];
};

// threads per block of every kernel that sums
constexpr int kThreads = 256;

__device__ __forceinline__ double* part_of(CgState* st, int slot, int kind) {
    return &st->part[slot][kind][blockIdx.x % kParts];
}
// Totals of up to four sums by one warp, eight lanes each.  It also divides, for the
// block: in every warp the division alone was 2,000 cycles of the FP64 pipe.
__device__ __forceinline__ double sum_parts(const double* part) {
    double t = *part;
#pragma unroll
    for (int o = kParts / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}
// to all threads of the block: num / den of two sums (slot, kind), by its first warp
__device__ __forceinline__ double block_quotient(const CgState* st, int ns, int nk, int ds, int dk) {
    __shared__ double ratio;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        const double t = sum_parts(lane < kParts ? &st->part[ns][nk][lane] : &st->part[ds][dk][lane % kParts]);
        const double den = __shfl_sync(0xffffffffu, t, kParts);
        if (lane == 0) ratio = t / den;
    }
    __syncthreads();
    return ratio;
}

__global__ void k_diag_inv(int64_t n, const int32_t* rp, const int32_t* ci, const double* v, double* dinv,
                           int jacobi, int limit, CgState* st) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (rp[i + 1] - rp[i] > limit) st->wide = 1;
    double d = 1.0;
    if (jacobi) {
        int lo = rp[i], hi = rp[i + 1] - 1;
        while (lo <= hi) {  // columns ascending
            const int mid = (lo + hi) >> 1;
            if (ci[mid] == i) {
                d = v[mid];
                break;
            }
            if (ci[mid] < i) lo = mid + 1;
            else hi = mid - 1;
        }
        d = (d != 0.0) ? 1.0 / d : 1.0;
    }
    dinv[i] = d;
}

// r = b - A x ; z = M^-1 r ; p = z ; accumulate r.z, r.r into slot 0, b.b into slot 3
__global__ void k_init(int64_t n, const int32_t* rp, const int32_t* ci, const double* v, const double* b,
                       const double* x, double* r, double* z, double* p, const double* dinv, CgState* st) {
    const int sub = threadIdx.x % fem::kLanesPerRow;
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / fem::kLanesPerRow;
    double sum[3] = {0.0, 0.0, 0.0};
    const double s = fem::csr_row_dot(n, rp, ci, v, x, row, sub);
    if (row < n && sub == 0) {
        const double ri = b[row] - s, zi = dinv[row] * ri;
        r[row] = ri;
        z[row] = zi;
        p[row] = zi;
        sum[0] = ri * zi;
        sum[1] = ri * ri;
        sum[2] = b[row] * b[row];
    }
    fem::block_sum_add<kThreads, fem::kLanesPerRow, 3>(sum, {part_of(st, 0, 1), part_of(st, 0, 2), part_of(st, 3, 2)});
}

// q = A p (warp per row, grid-stride over rows so that each block adds its
// share of p.q with one atomic) and p.q into the ring
__global__ void k_spmv_pq(int64_t n, const int32_t* rp, const int32_t* ci, const double* v, const double* p,
                          double* q, CgState* st) {
    if (st->done) return;
    const int slot = st->it & 3;
    const int sub = threadIdx.x % fem::kLanesPerRow;
    const int64_t groups = ((int64_t)gridDim.x * blockDim.x) / fem::kLanesPerRow;
    // the warp's first row; the trip count is uniform over the warp (the row
    // reduction shuffles need all 32 lanes)
    const int64_t first = ((int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / fem::kLanesPerRow;
    double pq = 0.0;
    for (int64_t base = first; base < n; base += groups) {
        const int64_t row = base + (threadIdx.x & 31) / fem::kLanesPerRow;
        const double s = fem::csr_row_dot(n, rp, ci, v, p, row, sub);
        if (sub == 0 && row < n) {
            q[row] = s;
            pq = fma(s, p[row], pq);
        }
    }
    const double sum[1] = {pq};
    fem::block_sum_add<kThreads, fem::kLanesPerRow, 1>(sum, {part_of(st, slot, 0)});
}

__global__ void k_update_xr(int64_t n, double* x, double* r, double* z, const double* p, const double* q,
                            const double* dinv, CgState* st) {
    if (st->done) return;
    const int slot = st->it & 3, nxt = (st->it + 1) & 3;
    const double alpha = block_quotient(st, slot, 1, slot, 0);
    double rz = 0.0, rr = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        x[i] = fma(alpha, p[i], x[i]);
        const double ri = fma(-alpha, q[i], r[i]);
        r[i] = ri;
        const double zi = dinv[i] * ri;
        z[i] = zi;
        rz = fma(ri, zi, rz);
        rr = fma(ri, ri, rr);
    }
    const double sum[2] = {rz, rr};
    fem::block_sum_add<kThreads, 1, 2>(sum, {part_of(st, nxt, 1), part_of(st, nxt, 2)});
}

__global__ void k_update_p(int64_t n, double* p, const double* z, CgState* st) {
    if (st->done) return;
    const int slot = st->it & 3, nxt = (st->it + 1) & 3;
    const double beta = block_quotient(st, nxt, 1, slot, 1);  // (of no use once k4 records convergence)
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = fma(beta, p[i], z[i]);
}

// (one warp)
__global__ void k_advance(CgState* st, int max_iter) {
    if (st->done) return;
    const int it = st->it, slot = it & 3, nxt = (it + 1) & 3, nn = (it + 2) & 3, lane = threadIdx.x;
    const int what = lane / kParts;  // r.z, r.r of the next iteration, p.Ap
    const double t = sum_parts(&st->part[what == 2 ? slot : nxt][what == 0 ? 1 : what == 1 ? 2 : 0][lane % kParts]);
    const double rz = __shfl_sync(0xffffffffu, t, 0), rr = __shfl_sync(0xffffffffu, t, kParts),
                 pq = __shfl_sync(0xffffffffu, t, 2 * kParts);
    if (lane < 3 * kParts) (&st->part[nn][0][0])[lane] = 0.0;
    if (lane == 0) {
        st->it = it + 1;
        st->ring[nxt][1] = rz;
        st->ring[nxt][2] = rr;
        if (rr <= st->thresh2) {
            st->done = 1;
            st->converged_at = it + 1;
        } else if (!(rz == rz) || pq == 0.0) {
            st->done = 2;  // breakdown (NaN or p.Ap == 0)
        } else if (it + 1 >= max_iter) {
            st->done = 3;
        }
    }
}

// Two launches per iteration.  The direction p = z + beta p is formed where the
// product gathers it (one FMA and one more load per nonzero, no pass of its
// own), written for the next iteration to the other of two arrays; convergence
// and breakdown of an iteration are tested by the next product, every block from
// the same ring values.  k is the iteration within the chunk; chunks are multiples
// of four, so k & 3 is the ring slot and no load waits for the iteration counter,
// which is advanced at the chunk's end (k_pair_end).  An iteration of a small
// system is a chain of L2 latencies: the launches overlap (programmatic
// dependent launch), and the first entries of the thread's row, which no kernel
// writes, are loaded before the previous one is waited for.
constexpr int kPairCached = 5;  // entries per lane of a row loaded ahead

// of the iteration before k: 0 go on, 1 converged, 2 breakdown (NaN or p.Ap == 0), 3 limit
__device__ __forceinline__ int pair_test(const CgState* st, double rz, double rr, double pq, int it, int max_iter) {
    if (it == 0) return 0;  // k_set_thresh has tested the start
    if (rr <= st->thresh2) return 1;
    if (!(rz == rz) || pq == 0.0) return 2;
    return it >= max_iter ? 3 : 0;
}
// by one thread; st->it stays until the chunk's end, other blocks still read it
__device__ __forceinline__ void pair_record(CgState* st, int it, int state, double rr) {
    if (state == 1) st->converged_at = it;
    st->ring[it & 3][2] = rr;
    st->stopped_at = it;
    st->done = state;
}
__global__ void __launch_bounds__(kThreads) k_pair_product(int n, const int32_t* __restrict__ rp,
                                                           const int32_t* __restrict__ ci,
                                                           const double* __restrict__ v, const double* z, double* pa,
                                                           double* pb, double* q, CgState* st, int k,
                                                           int max_iter) {
    constexpr int L = fem::kLanesPerRow;
    __shared__ double sbeta;
    __shared__ int stop;
    const int sub = threadIdx.x % L, row = (blockIdx.x * kThreads + threadIdx.x) / L, lane = threadIdx.x & 31;
    int j = 0, e = 0;
    if (row < n) {
        j = rp[row] + sub;
        e = rp[row + 1];
    }
    int32_t cc[kPairCached];
    double cv[kPairCached], zc[kPairCached], pc[kPairCached];
#pragma unroll
    for (int m = 0; m < kPairCached; ++m) {
        const bool in = j + m * L < e;
        cc[m] = in ? ci[j + m * L] : -1;
        cv[m] = in ? v[j + m * L] : 0.0;
    }
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const double* po = k & 1 ? pb : pa;
    double* pn = k & 1 ? pa : pb;
#pragma unroll
    for (int m = 0; m < kPairCached; ++m) {
        zc[m] = cc[m] >= 0 ? z[cc[m]] : 0.0;
        pc[m] = cc[m] >= 0 ? po[cc[m]] : 0.0;
    }
    const bool own = sub == 0 && row < n;
    const double zr = own ? z[row] : 0.0, pr = own ? po[row] : 0.0;
    if (threadIdx.x < 32) {
        // r.z, r.r, and p.Ap, r.z of the iteration before
        const int what = lane / kParts, slot = what < 2 ? k & 3 : (k + 3) & 3;
        const double t = sum_parts(&st->part[slot][what == 1 ? 2 : what == 2 ? 0 : 1][lane % kParts]);
        const double rz = __shfl_sync(0xffffffffu, t, 0), rr = __shfl_sync(0xffffffffu, t, kParts),
                     pq = __shfl_sync(0xffffffffu, t, 2 * kParts), old = __shfl_sync(0xffffffffu, t, 3 * kParts);
        if (lane == 0) {
            const int it = st->it + k, done = st->done;
            const int state = done ? done : pair_test(st, rz, rr, pq, it, max_iter);
            if (blockIdx.x == 0 && !done && state) pair_record(st, it, state, rr);
            stop = state;
            sbeta = it ? rz / old : 0.0;
        }
    }
    __syncthreads();
    if (stop) return;
    const double beta = sbeta;
    double dot = 0.0, pq = 0.0;
#pragma unroll
    for (int m = 0; m < kPairCached; ++m) dot = fma(cv[m], fma(beta, pc[m], zc[m]), dot);
#pragma unroll 4
    for (j += kPairCached * L; j < e; j += L) {
        const int c = ci[j];
        dot = fma(v[j], fma(beta, po[c], z[c]), dot);
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    if (own) {
        const double p = fma(beta, pr, zr);
        pn[row] = p;
        q[row] = dot;
        pq = dot * p;
    }
    const double sum[1] = {pq};
    fem::block_sum_add<kThreads, L, 1>(sum, {part_of(st, k & 3, 0)});
    if (blockIdx.x == 0 && threadIdx.x < 3 * kParts) (&st->part[(k + 2) & 3][0][0])[threadIdx.x] = 0.0;
}

constexpr int kPairThreads = 128;  // of the update: a small system spreads over more SMs
__global__ void __launch_bounds__(kPairThreads) k_pair_update(int n, double* x, double* r, double* z,
                                                              const double* pa, const double* pb, const double* q,
                                                              const double* dinv, CgState* st, int k) {
    __shared__ double salpha;
    __shared__ int stop;
    const int i = blockIdx.x * kPairThreads + threadIdx.x, lane = threadIdx.x & 31, at = i < n ? i : 0;
    const double di = dinv[at];
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const double* p = k & 1 ? pa : pb;
    const double xi = x[at], pi = p[at], qi = q[at];
    double ri = r[at];
    if (threadIdx.x < 32) {
        const double t = sum_parts(&st->part[k & 3][lane < kParts ? 1 : 0][lane % kParts]);
        const double rz = __shfl_sync(0xffffffffu, t, 0), pq = __shfl_sync(0xffffffffu, t, kParts);
        if (lane == 0) {
            stop = st->done;
            salpha = rz / pq;
        }
    }
    __syncthreads();
    if (stop) return;
    const double alpha = salpha;
    double sum[2] = {0.0, 0.0};
    if (i < n) {
        x[i] = fma(alpha, pi, xi);
        ri = fma(-alpha, qi, ri);
        r[i] = ri;
        const double zi = di * ri;
        z[i] = zi;
        sum[0] = ri * zi;
        sum[1] = ri * ri;
    }
    const int nxt = (k + 1) & 3;
    fem::block_sum_add<kPairThreads, 1, 2>(sum, {part_of(st, nxt, 1), part_of(st, nxt, 2)});
}

// end of a chunk: its last iteration's test, and the next chunk's base
__global__ void k_pair_end(CgState* st, int chunk, int max_iter) {
    if (!st->done) {
        double rz = 0.0, rr = 0.0, pq = 0.0;
        for (int m = 0; m < kParts; ++m) {
            rz += st->part[chunk & 3][1][m];
            rr += st->part[chunk & 3][2][m];
            pq += st->part[(chunk + 3) & 3][0][m];
        }
        const int it = st->it + chunk, state = pair_test(st, rz, rr, pq, it, max_iter);
        st->it = it;
        if (state) pair_record(st, it, state, rr);
    } else {
        st->it = st->stopped_at;
    }
}

// One cluster of 16 CTAs runs the iterations by itself: a thread per row with its
// entries of x, r, p in registers, the rows of the matrix in shared memory (entry k of
// all rows together, columns as 16 bits), sums over the cluster in the order of the
// ranks.  z is exchanged through distributed shared memory with the second sum, and
// every CTA forms p = z + beta p itself in the blocks of 32 entries that its columns
// name.  An iteration is two cluster barriers, five of the CTA and W FMAs per row on 16
// SMs: no launch and no trip to the L2.  Every CTA takes the same decisions from the
// same sums, so all leave the loop together.
// Microseconds per iteration, two launches -> here: plane systems of 578 rows 10.7 ->
// 6.2, 2,178 rows 8.8 -> 6.0, 5,000 rows 7.6 -> 7.0, 8,450 rows 8.1 -> 9.3 to 9.9 (not
// used); solids of 1,029 rows 13.7 -> 10.0, 3,000 rows 12.0 -> 10.3.
constexpr int kClusterCtas = 16, kClusterRows = 320;  // rows per CTA at most
constexpr int kClusterChunk = 2048;                   // iterations per launch
struct ClusterShape {
    int rows = 0, width = 0;  // rows per CTA (a multiple of 32), entries per row
    size_t smem = 0;
};
ClusterShape cluster_shape(int64_t n, int width) {
    ClusterShape c;
    const int64_t rows = (n + kClusterCtas * 32 - 1) / (kClusterCtas * 32) * 32, blocks = (n + 31) / 32;
    if (rows > kClusterRows) return c;
    c.rows = (int)rows;
    c.width = width;
    c.smem = (blocks * 32 + 3 * rows + 3 * kClusterCtas + 4 + width * rows) * sizeof(double) +
             width * rows * sizeof(uint16_t) + ((blocks + 31) / 32 + 1) * sizeof(unsigned) + blocks * sizeof(uint16_t);
    return c;
}

__global__ void __launch_bounds__(kClusterRows) k_cluster_cg(int n, int W, const int32_t* __restrict__ rp,
                                                     const int32_t* __restrict__ ci, const double* __restrict__ v,
                                                     double* x, double* r, double* p, const double* dinv, CgState* st,
                                                     int max_iter) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char raw[];
    const cg::cluster_group cluster = cg::this_cluster();
    const int R = blockDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = R >> 5;
    const int rank = (int)cluster.block_rank(), row = rank * R + tid, NB = (n + 31) / 32;
    const bool live = row < n;
    double* P = (double*)raw;             // p, where this CTA reads it
    double* zown = P + NB * 32;           // z of this CTA's rows
    double* red = zown + R;               // [2][R]
    double* slots = red + 2 * R;          // [3][rank]
    double* bc = slots + 3 * kClusterCtas;
    double* av = bc + 4;                  // [W][R]
    uint16_t* ac = (uint16_t*)(av + (size_t)W * R);
    unsigned* bits = (unsigned*)(ac + (size_t)W * R);
    unsigned* count = bits + (NB + 31) / 32;
    uint16_t* list = (uint16_t*)(count + 1);
    if (st->done || st->wide) return;  // the same for all
    for (int k = tid; k <= (NB + 31) / 32; k += R) bits[k] = 0;
    __syncthreads();
    const int j0 = live ? rp[row] : 0, len = live ? rp[row + 1] - j0 : 0;
    for (int k = 0; k < W; ++k) {
        const int c = k < len ? ci[j0 + k] : live ? row : 0;
        av[k * R + tid] = k < len ? v[j0 + k] : 0.0;
        ac[k * R + tid] = (uint16_t)c;
        if (k < len && c / R != rank) atomicOr(bits + (c >> 10), 1u << (c >> 5 & 31));
    }
    __syncthreads();
    for (int k = tid; k < NB; k += R)
        if (bits[k >> 5] >> (k & 31) & 1) list[atomicAdd(count, 1u)] = (uint16_t)k;
    __syncthreads();
    const int blocks = (int)*count;
    for (int b = warp; b < blocks; b += warps) {
        const int at = list[b] * 32 + lane;
        P[at] = at < n ? p[at] : 0.0;
    }
    double xi = 0.0, ri = 0.0, pi = 0.0, di = 0.0, zi = 0.0;
    if (live) {
        xi = x[row];
        ri = r[row];
        pi = p[row];
        di = dinv[row];
        P[row] = pi;
    }
    int it = st->it, state = 0;
    double rz = st->ring[it & 3][1], rr = 0.0;
    const double thresh2 = st->thresh2;
    // sum of a[0..R) by one warp, to slot set k of every CTA
    const auto share = [&](const double* a, int k) {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        int m = lane;
        for (; m + 96 < R; m += 128) {
            s[0] += a[m];
            s[1] += a[m + 32];
            s[2] += a[m + 64];
            s[3] += a[m + 96];
        }
        for (; m < R; m += 32) s[0] += a[m];
        const double t = fem::warp_total((s[0] + s[1]) + (s[2] + s[3]));
        if (lane < kClusterCtas) cluster.map_shared_rank(slots, lane)[k * kClusterCtas + rank] = t;
    };
    // all of p is read, and all CTAs run, before anything is written
    cluster.sync();
    for (int k = 0; k < kClusterChunk && !state; ++k) {
        double q = 0.0;
#pragma unroll 6
        for (int m = 0; m < W; ++m) q = fma(av[m * R + tid], P[ac[m * R + tid]], q);
        red[tid] = live ? q * pi : 0.0;
        __syncthreads();
        if (warp == 0) share(red, 0);
        cluster.sync();
        if (warp == 0) {
            double t = slots[lane & 15];
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) {
                bc[0] = t;
                bc[1] = rz / t;
            }
        }
        __syncthreads();
        const double pq = bc[0], alpha = bc[1];
        xi = fma(alpha, pi, xi);
        ri = fma(-alpha, q, ri);
        zi = di * ri;
        zown[tid] = zi;
        red[tid] = live ? ri * zi : 0.0;
        red[R + tid] = live ? ri * ri : 0.0;
        __syncthreads();
        if (warp == 0) share(red, 1);
        if (warp == warps - 1) share(red + R, 2);
        cluster.sync();
        if (warp == 0) {
            double t = slots[kClusterCtas + lane];  // lanes 0 to 15 r.z, 16 to 31 r.r
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) {
                bc[0] = t;
                bc[1] = t / rz;
            }
            if (lane == 16) bc[2] = t;
        }
        __syncthreads();
        rz = bc[0];
        rr = bc[2];
        ++it;
        state = rr <= thresh2 ? 1 : !(rz == rz) || pq == 0.0 ? 2 : it >= max_iter ? 3 : 0;
        const double beta = bc[1];
        pi = fma(beta, pi, zi);
        if (live) P[row] = pi;
        for (int b = warp; b < blocks; b += warps) {
            const int at = list[b] * 32, owner = at / R;
            P[at + lane] = fma(beta, P[at + lane], cluster.map_shared_rank(zown, owner)[at - owner * R + lane]);
        }
        __syncthreads();
    }
    if (live) {
        x[row] = xi;
        r[row] = ri;
        p[row] = pi;
    }
    cluster.sync();  // no CTA leaves while its memory is read, or the state before it is
    if (rank == 0 && tid == 0) {
        st->ring[it & 3][1] = rz;
        st->ring[it & 3][2] = rr;
        st->it = it;
        if (state == 1) st->converged_at = it;
        st->done = state;
    }
}

// Two launches where every lane group has one row and every SM at most one block
// of the product (9,728 rows on GB300).  Microseconds per iteration, four launches ->
// two: plane systems of 5,618 rows 14.7 -> 7.6, 8,450 rows 14.7 -> 8.1; solids of 6,591
// rows 17.5 -> 11.7.  Past the line the second gather costs more than the launches:
// without the line 18,818 rows 15.0 -> 15.1, 132,098 rows 33 -> 39, solid of 14,739
// rows 18.5 -> 49.
bool pair_system(int64_t n) { return n * fem::kLanesPerRow <= (int64_t)fem::sm_count() * kThreads; }

__global__ void k_set_thresh(CgState* st, double rtol) {
    double rz = 0.0, rr = 0.0, bb = 0.0;
    for (int k = 0; k < kParts; ++k) {
        rz += st->part[0][1][k];
        rr += st->part[0][2][k];
        bb += st->part[3][2][k];  // b.b of k_init; iteration 1 clears the slot
    }
    const double bn2 = bb > 0.0 ? bb : 1.0;
    st->bn2 = bn2;
    st->thresh2 = rtol * rtol * bn2;
    st->ring[0][1] = rz;
    st->ring[0][2] = rr;
    if (rr <= st->thresh2) {
        st->done = 1;
        st->converged_at = 0;
    }
}

// launch of k_cluster_cg for n rows of at most width entries
struct ClusterLaunch {
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg{};
    bool init(int64_t n, int width, cudaStream_t st) {
        const ClusterShape s = cluster_shape(n, width);
        int dev = 0, limit = 0, clusters = 0;
        if (!s.rows || width < 1 || cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            s.smem > (size_t)limit)
            return false;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kClusterCtas;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3(kClusterCtas);
        cfg.blockDim = dim3((unsigned)s.rows);
        cfg.dynamicSmemBytes = s.smem;
        cfg.stream = st;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        // the attributes belong to the function: the same values whatever the system, because
        // other threads launch theirs between these lines and this one's launch
        const bool ok =
            cudaFuncSetAttribute(k_cluster_cg, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaFuncSetAttribute(k_cluster_cg, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, k_cluster_cg, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) cudaGetLastError();
        return ok;
    }
};

}  // namespace

using namespace fem;

extern "C" fem_gpu_status fem_gpu_pcg(fem_gpu_ctx* c, const int32_t* rowptr, const int32_t* colidx,
                                      const double* vals, const double* b, double* x, const fem_gpu_pcg_opts* opts,
                                      fem_gpu_pcg_report* rep, uint32_t flags) {
    if (!c || !rowptr || !colidx || !vals || !b || !x || !opts) return FEM_GPU_BAD_ARG;
    if (flags & FEM_GPU_HOST_BUFFERS) return fail(c, FEM_GPU_UNSUPPORTED, "pcg takes device buffers");
    if (!c->host_final) return FEM_GPU_NOT_FINALIZED;
    if (!(opts->rel_tol > 0.0) || opts->max_iter < 1) return FEM_GPU_BAD_ARG;
    if (!c->stream && !c->stream_set) {
        cudaStream_t s;
        if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess)
            return fail(c, FEM_GPU_CUDA_ERROR, "stream create");
        c->stream = s;
        c->own_stream = true;
    }
    // stream capture needs a non-default stream: on the legacy default stream
    // the solve runs on a private stream after the default stream's work
    cudaStream_t sm = (cudaStream_t)c->stream;
    cudaStream_t own = nullptr;
    if (!sm) {
        if (cudaStreamCreateWithFlags(&own, cudaStreamNonBlocking) != cudaSuccess)
            return fail(c, FEM_GPU_CUDA_ERROR, "stream create");
        cudaStreamSynchronize(nullptr);
        sm = own;
    }
    const int64_t n = c->num_used * c->dim;
    const auto t0 = std::chrono::steady_clock::now();
    double *r = nullptr, *z = nullptr, *p = nullptr, *q = nullptr, *dinv = nullptr;
    CgState* st = nullptr;
    cudaError_t e = cudaMallocAsync(&r, 6 * n * sizeof(double), sm);
    if (e == cudaSuccess) e = cudaMallocAsync(&st, sizeof(CgState), sm);
    if (e != cudaSuccess) return fail(c, FEM_GPU_OUT_OF_MEMORY, "pcg workspace");
    z = r + n;
    p = z + n;
    q = p + n;
    dinv = q + n;  // then the second direction array of the two-launch iteration
    const bool pair = pair_system(n);
    const unsigned upd_blocks = (unsigned)((n + kPairThreads - 1) / kPairThreads);
    cudaMemsetAsync(st, 0, sizeof(CgState), sm);
    const int tpb = kThreads;
    const unsigned row_blocks = (unsigned)((n * fem::kLanesPerRow + tpb - 1) / tpb);
    const unsigned spmv_blocks = (unsigned)std::min<int64_t>(row_blocks, (int64_t)sm_count() * 16);
    const unsigned vec_blocks = (unsigned)std::min<int64_t>((n + tpb - 1) / tpb, (int64_t)sm_count() * 8);
    // one cluster where its shared memory holds the rows of the model's graph (their
    // longest is sought only where the rows are few enough)
    int width = 0;
    if (n <= kClusterCtas * kClusterRows && !c->ulen.empty())
        width = c->dim * *std::max_element(c->ulen.begin(), c->ulen.end());
    ClusterLaunch cluster;
    const bool clustered = cluster.init(n, width, sm);
    k_diag_inv<<<(unsigned)((n + tpb - 1) / tpb), tpb, 0, sm>>>(n, rowptr, colidx, vals, dinv, opts->preconditioner == 1,
                                                                clustered ? width : INT_MAX, st);
    k_init<<<row_blocks, tpb, 0, sm>>>(n, rowptr, colidx, vals, b, x, r, z, p, dinv, st);
    k_set_thresh<<<1, 1, 0, sm>>>(st, opts->rel_tol);
    c->launches += 3;
    CgState hs{};
    const auto read_state = [&] {
        e = cudaMemcpyAsync(&hs, st, sizeof(CgState), cudaMemcpyDeviceToHost, sm);
        if (e == cudaSuccess) e = cudaStreamSynchronize(sm);
        return e == cudaSuccess && !hs.done;
    };
    if (clustered)
        do {
            e = cudaLaunchKernelEx(&cluster.cfg, k_cluster_cg, (int)n, width, rowptr, colidx, vals, x, r, p,
                                   (const double*)dinv, st, (int)opts->max_iter);
            c->launches++;
        } while (e == cudaSuccess && read_state() && !hs.wide);
    // a matrix with longer rows than the model's graph takes the launches
    const bool launches = !clustered || (hs.wide && !hs.done);
    // capture a chunk of iterations into a graph
    const int chunk = 32;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    if (e == cudaSuccess && launches) e = cudaStreamBeginCapture(sm, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess && launches) {
        for (int k = 0; k < chunk && pair; ++k) {
            e = launch_kernel(k_pair_product, row_blocks, tpb, 0, sm, true, n, rowptr, colidx, vals, z, p, dinv + n, q,
                              st, k, opts->max_iter);
            if (e == cudaSuccess)
                e = launch_kernel(k_pair_update, upd_blocks, kPairThreads, 0, sm, true, n, x, r, z, p, dinv + n, q,
                                  dinv, st, k);
            if (e != cudaSuccess) break;
        }
        if (pair) k_pair_end<<<1, 1, 0, sm>>>(st, chunk, opts->max_iter);
        for (int k = 0; k < chunk && !pair; ++k) {
            k_spmv_pq<<<spmv_blocks, tpb, 0, sm>>>(n, rowptr, colidx, vals, p, q, st);
            k_update_xr<<<vec_blocks, tpb, 0, sm>>>(n, x, r, z, p, q, dinv, st);
            k_update_p<<<vec_blocks, tpb, 0, sm>>>(n, p, z, st);
            k_advance<<<1, 32, 0, sm>>>(st, opts->max_iter);
        }
        const cudaError_t ended = cudaStreamEndCapture(sm, &graph);
        if (e == cudaSuccess) e = ended;
    }
    if (e == cudaSuccess && launches) e = cudaGraphInstantiate(&exec, graph, 0);
    fem_gpu_status result = FEM_GPU_OK;
    if (e == cudaSuccess && launches) {
        for (int launched = 0; launched < opts->max_iter + chunk; launched += chunk) {
            e = cudaGraphLaunch(exec, sm);
            if (e != cudaSuccess) break;
            c->launches += pair ? 2 * chunk + 1 : 4 * chunk;
            if (!read_state()) break;
        }
    }
    if (e != cudaSuccess) result = fail(c, FEM_GPU_CUDA_ERROR, std::string("pcg: ") + cudaGetErrorString(e));
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    cudaFreeAsync(r, sm);
    cudaFreeAsync(st, sm);
    cudaStreamSynchronize(sm);
    if (own) cudaStreamDestroy(own);
    const double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (rep) {
        rep->iterations = hs.done == 1 ? hs.converged_at : hs.it;
        rep->converged = hs.done == 1;
        const int slot = hs.it & 3;
        rep->rel_residual = std::sqrt(hs.ring[slot][2] / (hs.bn2 > 0 ? hs.bn2 : 1.0));
        rep->seconds = secs;
    }
    if (result != FEM_GPU_OK) return result;
    if (hs.done == 2) return fail(c, FEM_GPU_NONFINITE, "pcg breakdown");
    if (hs.done != 1) return fail(c, FEM_GPU_NOT_CONVERGED, "pcg hit max_iter");
    return FEM_GPU_OK;
}

// ---------------------------------------------------------------------------
// PCG without device allocation.
//
// Some callers cannot allocate device memory while they solve: code that runs
// inside a host callback, a signal-safe or real-time section, or a framework
// that owns a fixed device memory budget and forbids cudaMalloc/cudaFree (and
// any allocating library call) after start-up.  For them the Jacobi-PCG work
// vectors live in one file-scope device array of fixed size instead of
// stream-ordered allocations, and the iterations are launched directly (no
// graph instantiation).  The array holds the solver state (first 1,024 bytes)
// and the five work vectors r, z, p, q and 1/diag(A), so systems up to
// kNoAllocMaxRows rows are accepted; larger ones are rejected with
// FEM_GPU_BAD_ARG.  Every GPU that loads the library keeps this array
// (about 5.2 MB) until the process exits.  The array comes with this file's
// module, which CUDA loads lazily: fem_gpu_finalize resolves the array's
// address on the current device (noalloc_prepare), so the module is loaded
// there; after fem_gpu_finalize_host alone the first fem_gpu_pcg_noalloc call
// on a device does it.
namespace {

constexpr int64_t kNoAllocMaxRows = 131072;
constexpr int64_t kNoAllocStateDoubles = 128;  // 1,024 bytes for CgState
static_assert(sizeof(CgState) <= kNoAllocStateDoubles * sizeof(double), "CgState fits the state slot");

static __device__ __align__(256) double g_pcg_noalloc_scratch[kNoAllocStateDoubles + 5 * kNoAllocMaxRows];

// device address of the scratch array, resolved once per device with that
// device current (the host-side symbol is only a stand-in, never a device
// address)
constexpr int kMaxDevices = 64;
double* g_scratch_addr[kMaxDevices] = {nullptr};
std::mutex g_scratch_mutex;

fem_gpu_status noalloc_scratch(fem_gpu_ctx* c, double** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
        return fail(c, FEM_GPU_NO_DEVICE, "pcg_noalloc: no current CUDA device");
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_pcg_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return fail(c, FEM_GPU_CUDA_ERROR, std::string("pcg_noalloc: scratch address: ") + cudaGetErrorString(e));
        g_scratch_addr[dev] = static_cast<double*>(p);
    }
    *out = g_scratch_addr[dev];
    return FEM_GPU_OK;
}

}  // namespace

namespace fem {
fem_gpu_status noalloc_prepare(fem_gpu_ctx* c) {
    double* p = nullptr;
    fem_gpu_status st = noalloc_scratch(c, &p);
    if (st != FEM_GPU_OK) return st;
    // with lazy loading a kernel's code is loaded at its first launch; reading
    // the attributes of the solver's kernels loads them now
    const void* kernels[] = {(const void*)k_diag_inv, (const void*)k_init,     (const void*)k_set_thresh,
                             (const void*)k_spmv_pq,  (const void*)k_update_xr, (const void*)k_update_p,
                             (const void*)k_advance};
    for (const void* k : kernels) {
        cudaFuncAttributes a;
        const cudaError_t e = cudaFuncGetAttributes(&a, k);
        if (e != cudaSuccess)
            return fail(c, FEM_GPU_CUDA_ERROR, std::string("pcg_noalloc: kernel load: ") + cudaGetErrorString(e));
    }
    return FEM_GPU_OK;
}
}  // namespace fem

extern "C" fem_gpu_status fem_gpu_pcg_noalloc(fem_gpu_ctx* c, const int32_t* rowptr, const int32_t* colidx,
                                              const double* vals, const double* b, double* x,
                                              const fem_gpu_pcg_opts* opts, fem_gpu_pcg_report* rep,
                                              uint32_t flags) {
    if (!c || !rowptr || !colidx || !vals || !b || !x || !opts) return FEM_GPU_BAD_ARG;
    if (flags & FEM_GPU_HOST_BUFFERS) return fail(c, FEM_GPU_UNSUPPORTED, "pcg_noalloc takes device buffers");
    if (!c->host_final) return FEM_GPU_NOT_FINALIZED;
    if (!(opts->rel_tol > 0.0) || opts->max_iter < 1) return FEM_GPU_BAD_ARG;
    const int64_t n = c->num_used * c->dim;
    if (n > kNoAllocMaxRows)
        return fail(c, FEM_GPU_BAD_ARG,
                    "pcg_noalloc: " + std::to_string(n) + " rows exceed the fixed scratch limit of " +
                        std::to_string(kNoAllocMaxRows) + " rows; use fem_gpu_pcg");
    double* base = nullptr;
    fem_gpu_status st = noalloc_scratch(c, &base);
    if (st != FEM_GPU_OK) return st;
    // the caller's stream, or the legacy default stream when none was set
    cudaStream_t sm = (cudaStream_t)c->stream;
    const auto t0 = std::chrono::steady_clock::now();
    CgState* cs = reinterpret_cast<CgState*>(base);
    double* r = base + kNoAllocStateDoubles;
    double* z = r + n;
    double* p = z + n;
    double* q = p + n;
    double* dinv = q + n;
    // the array keeps the previous call's contents: the state must start at zero
    cudaError_t e = cudaMemsetAsync(cs, 0, sizeof(CgState), sm);
    if (e != cudaSuccess) return fail(c, FEM_GPU_CUDA_ERROR, std::string("pcg_noalloc: ") + cudaGetErrorString(e));
    const int tpb = kThreads;
    const unsigned row_blocks = (unsigned)((n * fem::kLanesPerRow + tpb - 1) / tpb);
    const unsigned vec_blocks = (unsigned)std::min<int64_t>((n + tpb - 1) / tpb, (int64_t)sm_count() * 8);
    k_diag_inv<<<(unsigned)((n + tpb - 1) / tpb), tpb, 0, sm>>>(n, rowptr, colidx, vals, dinv,
                                                                opts->preconditioner == 1, INT_MAX, cs);
    k_init<<<row_blocks, tpb, 0, sm>>>(n, rowptr, colidx, vals, b, x, r, z, p, dinv, cs);
    k_set_thresh<<<1, 1, 0, sm>>>(cs, opts->rel_tol);
    c->launches += 3;
    CgState hs{};
    const int chunk = 32;
    for (int launched = 0; launched < opts->max_iter + chunk; launched += chunk) {
        for (int k = 0; k < chunk; ++k) {
            k_spmv_pq<<<row_blocks, tpb, 0, sm>>>(n, rowptr, colidx, vals, p, q, cs);
            k_update_xr<<<vec_blocks, tpb, 0, sm>>>(n, x, r, z, p, q, dinv, cs);
            k_update_p<<<vec_blocks, tpb, 0, sm>>>(n, p, z, cs);
            k_advance<<<1, 32, 0, sm>>>(cs, opts->max_iter);
        }
        c->launches += 4 * chunk;
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(&hs, cs, sizeof(CgState), cudaMemcpyDeviceToHost, sm);
        if (e == cudaSuccess) e = cudaStreamSynchronize(sm);
        if (e != cudaSuccess) return fail(c, FEM_GPU_CUDA_ERROR, std::string("pcg_noalloc: ") + cudaGetErrorString(e));
        if (hs.done) break;
    }
    const double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (rep) {
        rep->iterations = hs.done == 1 ? hs.converged_at : hs.it;
        rep->converged = hs.done == 1;
        rep->rel_residual = std::sqrt(hs.ring[hs.it & 3][2] / (hs.bn2 > 0 ? hs.bn2 : 1.0));
        rep->seconds = secs;
    }
    if (hs.done == 2) return fail(c, FEM_GPU_NONFINITE, "pcg_noalloc breakdown");
    if (hs.done != 1) return fail(c, FEM_GPU_NOT_CONVERGED, "pcg_noalloc hit max_iter");
    return FEM_GPU_OK;
}

// ---------------------------------------------------------------------------
// Jacobi-PCG that also records its iterates: x after every `every`
// iterations is copied into snaps[j * n ...] (device, max_snaps slots).  The
// residual/error pairs of the learned preconditioner's training set come from
// these iterates of the solver itself.
extern "C" fem_gpu_status fem_gpu_pcg_snapshots(fem_gpu_ctx* c, const int32_t* rowptr, const int32_t* colidx,
                                                const double* vals, const double* b, double* x,
                                                const fem_gpu_pcg_opts* opts, fem_gpu_pcg_report* rep, int32_t every,
                                                double* snaps, int32_t max_snaps, int32_t* n_snaps) {
    if (!c || !rowptr || !colidx || !vals || !b || !x || !opts || every < 1 || !snaps || max_snaps < 1 || !n_snaps)
        return FEM_GPU_BAD_ARG;
    if (!c->host_final) return FEM_GPU_NOT_FINALIZED;
    if (!(opts->rel_tol > 0.0) || opts->max_iter < 1) return FEM_GPU_BAD_ARG;
    const int64_t n = c->num_used * c->dim;
    cudaStream_t sm = nullptr;
    if (cudaStreamCreateWithFlags(&sm, cudaStreamNonBlocking) != cudaSuccess)
        return fail(c, FEM_GPU_CUDA_ERROR, "stream create");
    cudaDeviceSynchronize();
    const auto t0 = std::chrono::steady_clock::now();
    double* r = nullptr;
    CgState* st = nullptr;
    cudaError_t e = cudaMallocAsync(&r, 5 * n * sizeof(double), sm);
    if (e == cudaSuccess) e = cudaMallocAsync(&st, sizeof(CgState), sm);
    if (e != cudaSuccess) {
        cudaStreamDestroy(sm);
        return fail(c, FEM_GPU_OUT_OF_MEMORY, "pcg workspace");
    }
    double *z = r + n, *p = z + n, *q = p + n, *dinv = q + n;
    cudaMemsetAsync(st, 0, sizeof(CgState), sm);
    const int tpb = kThreads;
    const unsigned row_blocks = (unsigned)((n * fem::kLanesPerRow + tpb - 1) / tpb);
    const unsigned spmv_blocks = (unsigned)std::min<int64_t>(row_blocks, (int64_t)sm_count() * 16);
    const unsigned vec_blocks = (unsigned)std::min<int64_t>((n + tpb - 1) / tpb, (int64_t)sm_count() * 8);
    k_diag_inv<<<(unsigned)((n + tpb - 1) / tpb), tpb, 0, sm>>>(n, rowptr, colidx, vals, dinv, opts->preconditioner == 1,
                                                                INT_MAX, st);
    k_init<<<row_blocks, tpb, 0, sm>>>(n, rowptr, colidx, vals, b, x, r, z, p, dinv, st);
    k_set_thresh<<<1, 1, 0, sm>>>(st, opts->rel_tol);
    CgState hs{};
    int taken = 0;
    for (int done_it = 0; done_it < opts->max_iter; done_it += every) {
        for (int k = 0; k < every; ++k) {
            k_spmv_pq<<<spmv_blocks, tpb, 0, sm>>>(n, rowptr, colidx, vals, p, q, st);
            k_update_xr<<<vec_blocks, tpb, 0, sm>>>(n, x, r, z, p, q, dinv, st);
            k_update_p<<<vec_blocks, tpb, 0, sm>>>(n, p, z, st);
            k_advance<<<1, 32, 0, sm>>>(st, opts->max_iter);
        }
        c->launches += 4 * every;
        e = cudaMemcpyAsync(&hs, st, sizeof(CgState), cudaMemcpyDeviceToHost, sm);
        if (e == cudaSuccess) e = cudaStreamSynchronize(sm);
        if (e != cudaSuccess) break;
        if (hs.done) break;
        if (taken < max_snaps) {
            e = cudaMemcpyAsync(snaps + (int64_t)taken * n, x, n * sizeof(double), cudaMemcpyDeviceToDevice, sm);
            if (e != cudaSuccess) break;
            ++taken;
        }
    }
    cudaFreeAsync(r, sm);
    cudaFreeAsync(st, sm);
    cudaStreamSynchronize(sm);
    cudaStreamDestroy(sm);
    *n_snaps = taken;
    if (rep) {
        rep->iterations = hs.done == 1 ? hs.converged_at : hs.it;
        rep->converged = hs.done == 1;
        rep->rel_residual = std::sqrt(hs.ring[hs.it & 3][2] / (hs.bn2 > 0 ? hs.bn2 : 1.0));
        rep->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    }
    if (e != cudaSuccess) return fail(c, FEM_GPU_CUDA_ERROR, std::string("pcg snapshots: ") + cudaGetErrorString(e));
    if (hs.done == 2) return fail(c, FEM_GPU_NONFINITE, "pcg breakdown");
    if (hs.done != 1) return fail(c, FEM_GPU_NOT_CONVERGED, "pcg hit max_iter");
    return FEM_GPU_OK;
}
