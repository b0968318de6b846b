// Variable-coefficient leaf patches (FiniteVolumeSolverType::FivePointStencil).
//
// The reference assembles, for every patch, the dense n^2 x n^2 operator of
//     alpha div(beta grad u) + lambda u = f
// with cW = alpha_ij beta_{i-1/2,j} / dx^2, ..., cC = -alpha_ij ((beta_E + beta_W)/dx^2 +
// (beta_N + beta_S)/dy^2) + lambda_ij, subtracts c_side from the diagonal of boundary rows and adds
// -2 c_side g to their right-hand side (FiniteVolumeSolver.cpp:27-223), and LU-factors it with
// PETSc for every solve.  Here the same matrix is factored once per leaf at build time: with cell
// index j + i*n it is banded (bandwidth n); the factorisation runs in a shared-memory window of n+1
// band rows (n^4 work instead of n^6) and its band is kept in HBM for every later solve.
//
// No pivoting.  The matrix is A = D S with D = diag(alpha) and S symmetric (the face couplings
// beta/d^2 are shared by both cells of a face; S_ii = -sum beta/d^2 + lambda/alpha).  Gaussian
// elimination of D S without pivoting produces the pivots alpha_r u_rr(S), and u_rr(S) < 0 for every
// r exactly when S is negative definite -- then elimination without pivoting is backward stable (the
// Cholesky-type bound), whatever lambda's sign.  Every pivot is checked: a pivot with
// pivot * alpha_r >= 0 means S is not negative definite (lambda above the smallest eigenvalue of the
// diffusion part, alpha beta changing sign, alpha = 0), where elimination without pivoting is not
// safe; the factorisation flags it (info = -(r + 1)) and the build refuses the tree instead of
// returning results that could depart from the reference's pivoted LU.  An exact zero pivot is
// flagged as singular (info = r + 1).
//
// Coefficients arrive sampled per cell exactly as the reference samples them (cpp:66-79):
// alpha(x_i, y_j), beta at the four faces (x_i -/+ dx/2, y_j), (x_i, y_j -/+ dy/2), lambda(x_i, y_j).
#include <algorithm>

#include "ef_kernels.cuh"

namespace efgb {

namespace {

// band row r holds columns r-n .. r+n at positions 0 .. 2n
//
// The five stencil entries of every row in place in the band (k_fp_stencil, one thread per cell), then the
// factorisation over them.
__global__ void __launch_bounds__(256) k_fp_stencil(const FpLeaf* __restrict__ leaves) {
    const FpLeaf& lf = leaves[blockIdx.y];
    const int n = lf.n, N = n * n, w = 2 * n + 1, r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= N) return;
    const double dx2 = lf.dx * lf.dx, dy2 = lf.dy * lf.dy;
    const int i = r / n, j = r - (r / n) * n;
    const double a = lf.alpha[r];
    const double bW = lf.beta[r], bE = lf.beta[N + r], bS = lf.beta[2 * N + r], bN = lf.beta[3 * N + r];
    const double cW = a * bW / dx2, cE = a * bE / dx2, cS = a * bS / dy2, cN = a * bN / dy2;
    const double cC = -a * ((bE + bW) / dx2 + (bN + bS) / dy2) + lf.lambda[r];
    double* row = lf.band + (long long)r * w + n;
    double d = cC;
    if (i == 0) d -= cW;
    if (i == n - 1) d -= cE;
    if (j == 0) d -= cS;
    if (j == n - 1) d -= cN;
    row[-n] = i > 0 ? cW : 0.0;
    row[n] = i < n - 1 ? cE : 0.0;
    row[-1] = j > 0 ? cS : 0.0;
    row[1] = j < n - 1 ? cN : 0.0;
    row[0] = d;
    // boundary coupling coefficients for the right-hand side f_b = -2 c_side g
    if (i == 0) lf.bcoef[0 * n + j] = cW;
    if (i == n - 1) lf.bcoef[1 * n + j] = cE;
    if (j == 0) lf.bcoef[2 * n + i] = cS;
    if (j == n - 1) lf.bcoef[3 * n + i] = cN;
}

// A window of n + 2 rows lives in shared memory: the n + 1 rows that step k works on and the one that step
// k + 1 adds.  The last warp keeps the step's chain short: while the others update, it brings in the next row
// (its entries loaded a step earlier), stores the finished one, updates the next pivot and takes its
// reciprocal, so that a multiplier is a product with one correction instead of a division.  FP64 pipe bound
// with several leaves per SM (n^2 multiply-adds per step, two per clock and SM: 1.8 ms for 1024 leaves of
// 32 x 32 cells); two barriers and the reciprocal per step with few.
__global__ void __launch_bounds__(256) k_fp_factor(const FpLeaf* __restrict__ leaves) {
    const FpLeaf lf = leaves[blockIdx.x];
    const int n = lf.n, N = n * n, w = 2 * n + 1, nslot = n + 2;
    extern __shared__ double win[];  // nslot rows x w
    double* lm = win + nslot * w;     // n multipliers
    __shared__ double s_rcp;
    const int lane = threadIdx.x & 31, workers = blockDim.x - 32;
    const bool keeper = threadIdx.x >= workers;
    // entry `lane` of the five of band row r (c - r + n = 0, n-1, n, n+1, 2n)
    const int at = lane == 0 ? 0 : lane == 4 ? 2 * n : n - 2 + lane;
    auto fetch = [&](int r) { return lane < 5 ? lf.band[(long long)r * w + at] : 0.0; };
    auto place = [&](int r, double v) {
        double* row = win + (r % nslot) * w;
        for (int c = lane; c < w; c += 32) row[c] = 0.0;
        __syncwarp();
        if (lane < 5) row[at] = v;
        __syncwarp();
    };
    for (int r = threadIdx.x >> 5; r <= n && r < N; r += blockDim.x >> 5) place(r, fetch(r));
    double next = 0.0;
    if (keeper && n + 1 < N) next = fetch(n + 1);
    __syncthreads();
    if (threadIdx.x == 0) s_rcp = 1.0 / win[n];
    __syncthreads();
    int k0 = 0;  // slot of row k
    for (int k = 0; k < N; ++k) {
        const double* pr = win + k0 * w;  // pivot row k
        const double piv = pr[n];
        const int rows = min(n, N - 1 - k);
        auto slot = [&](int d) { return win + (k0 + d >= nslot ? k0 + d - nslot : k0 + d) * w; };
        // multipliers l_i = A[k+d][k] / piv for d = 1..rows; A[k+d][k] sits at position n - d
        if (threadIdx.x < rows) {
            const int d = threadIdx.x + 1;
            double* ri = slot(d);
            const double x = ri[n - d], rcp = s_rcp, q = x * rcp, l = fma(fma(-q, piv, x), rcp, q);
            lm[threadIdx.x] = l;
            ri[n - d] = l;
        }
        __syncthreads();
        // A[k+d][k+e] -= l_d * A[k][k+e], e = 1..n  (positions: row k+d at n-d+e, row k at n+e)
        if (!keeper) {
            for (int t = threadIdx.x; t < rows * n; t += workers) {
                const int d = t / n + 1, e = t - (t / n) * n + 1;
                if (t > 0) slot(d)[n - d + e] -= lm[d - 1] * pr[n + e];
            }
        } else {
            if (rows > 0) {
                double* r1 = slot(1);
                const double p1 = r1[n] - lm[0] * pr[n + 1];
                if (lane == 0) {
                    r1[n] = p1;
                    s_rcp = 1.0 / p1;
                }
            }
            // row k is final: store it; row k+n+1 into the slot that neither this step nor its rows use
            for (int c = lane; c < w; c += 32) lf.band[(long long)k * w + c] = pr[c];
            if (lane == 0 && *lf.info == 0) {
                if (piv == 0.0) *lf.info = k + 1;
                else if (!(piv * lf.alpha[k] < 0.0)) *lf.info = -(k + 1);  // not (scaled) negative definite
            }
            if (k + n + 1 < N) {
                place(k + n + 1, next);
                if (k + n + 2 < N) next = fetch(k + n + 2);
            }
        }
        if (++k0 == nslot) k0 = 0;
        __syncthreads();
    }
}

__device__ __forceinline__ void copy8_async(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(unsigned(__cvta_generic_to_shared(dst))), "l"(src)
                 : "memory");
}

// All columns of a leaf's DtN map: one column of 4n per thread, the leaf's band row blocks (the n rows of one
// grid column) through shared memory.  In block I the forward substitution takes rows a of
//   y_I = L_II^-1 (b_I - L_{I,I-1} y_{I-1}),  L_{I,I-1} upper, L_II unit lower triangular,
// with y_{I-1} and y_I in registers (the loops are unrolled to NP >= n rows), every band entry read once per
// warp as a broadcast; the backward substitution the same with U_II, U_{I,I+1}.  y goes through `scratch` (4n
// consecutive values per row, one n^2 x 4n slot per block) between the two.  Sums run from the far, small factors to the
// near, large ones and add y last (from the near ones on, with y first, the solutions of trees of 20 x 20 to 32 x 32
// leaves erred 2 to 5% more; now 0 to 2% less than with a column per warp).  FP64 pipe bound: 2 n^3 multiply-adds
// per column, two per clock and SM (1024 leaves of 32 x 32 cells: 174 ms with a column per warp, 16.1 ms).  Warps whose
// columns start in a later block (data on E) skip the blocks before it.
// The staged rows are spread to NP (zeros where a block row has no entry), so the loops need no bounds.
template <int NP>
__global__ void __launch_bounds__(128) k_fp_columns(const FpLeaf* __restrict__ leaves, const LeafItem* __restrict__ items,
                                                    int nleaves, double* __restrict__ scratch) {
    constexpr int W = 2 * NP + 1;
    __shared__ double rinv[NP];  // reciprocals of U's diagonal
    extern __shared__ double fc_smem[];  // two stages of NP x W
    const int n = leaves[0].n, w = 2 * n + 1, m = 4 * n, col = threadIdx.x;
    for (int e = threadIdx.x; e < 2 * NP * W; e += blockDim.x) fc_smem[e] = 0.0;
    if (threadIdx.x < NP) rinv[threadIdx.x] = 0.0;
    __syncthreads();
    const bool live = col < m;
    const int side = min(col, m - 1) / n, pos = min(col, m - 1) - side * n;
    const int eI = side == 0 ? 0 : side == 1 ? n - 1 : pos, ea = side < 2 ? pos : side == 2 ? 0 : n - 1;
    const int first = int(__reduce_min_sync(0xffffffffu, unsigned(eI)));
    for (int leaf = blockIdx.x; leaf < nleaves; leaf += gridDim.x) {
        const FpLeaf& lf = leaves[leaf];
        const double* band = lf.band;
        double* out = items[leaf * m].out + col;
        double* Y = scratch + (long long)blockIdx.x * n * n * m + col;
        const double be = -2.0 * lf.bcoef[min(col, m - 1)];
        // entry c of band row a belongs to block I-1 (c < n - a), I, or I+1 (c >= 2n - a)
        auto load = [&](int I) {
            const double* src = band + (long long)I * n * w;
            double* dst = fc_smem + (I & 1) * NP * W;
            for (int e = threadIdx.x; e < n * w; e += blockDim.x) {
                const int a = e / w, c = e - a * w;
                copy8_async(dst + a * W + c + (c < n - a ? 0 : c < 2 * n - a ? NP - n : 2 * (NP - n)), src + e);
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        auto arrived = [&](bool more) {
            if (more) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();
        };
        double yp[NP], y[NP];
#pragma unroll
        for (int a = 0; a < NP; ++a) yp[a] = 0.0;
        load(0);
        for (int I = 0; I < n; ++I) {
            if (I + 1 < n) load(I + 1);
            arrived(I + 1 < n);
            if (I >= first) {
                const double* blk = fc_smem + (I & 1) * NP * W;
#pragma unroll
                for (int a = 0; a < NP; ++a) {
                    double s0 = I == eI && a == ea ? be : 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
                    for (int b = NP - 1; b >= a; b -= 2) s0 = fma(-blk[a * W + b - a], yp[b], s0);
#pragma unroll
                    for (int b = NP - 2; b >= a; b -= 2) s1 = fma(-blk[a * W + b - a], yp[b], s1);
#pragma unroll
                    for (int b = 0; b < a; b += 2) s2 = fma(-blk[a * W + NP + b - a], y[b], s2);
#pragma unroll
                    for (int b = 1; b < a; b += 2) s3 = fma(-blk[a * W + NP + b - a], y[b], s3);
                    y[a] = (s0 + s1) + (s2 + s3);
                }
            } else {
#pragma unroll
                for (int a = 0; a < NP; ++a) y[a] = 0.0;
            }
#pragma unroll
            for (int a = 0; a < NP; ++a) {
                if (a < n && live) Y[(long long)(I * n + a) * m] = y[a];
                yp[a] = y[a];
            }
            __syncthreads();
        }
        const double dtn_x = 2.0 / lf.dx, dtn_y = 2.0 / lf.dy;
#pragma unroll
        for (int a = 0; a < NP; ++a) yp[a] = 0.0;  // x_{I+1}
        load(n - 1);
        for (int I = n - 1; I >= 0; --I) {
            if (I > 0) load(I - 1);
#pragma unroll
            for (int a = 0; a < NP; ++a) y[a] = a < n && live ? Y[(long long)(I * n + a) * m] : 0.0;
            arrived(I > 0);
            const double* blk = fc_smem + (I & 1) * NP * W;
            if (threadIdx.x < n) rinv[threadIdx.x] = 1.0 / blk[threadIdx.x * W + NP];
            __syncthreads();
#pragma unroll
            for (int a = NP - 1; a >= 0; --a) {
                double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
                for (int b = 0; b <= a; b += 2) s0 = fma(-blk[a * W + 2 * NP + b - a], yp[b], s0);
#pragma unroll
                for (int b = 1; b <= a; b += 2) s1 = fma(-blk[a * W + 2 * NP + b - a], yp[b], s1);
#pragma unroll
                for (int b = NP - 1; b > a; b -= 2) s2 = fma(-blk[a * W + NP + b - a], y[b], s2);
#pragma unroll
                for (int b = NP - 2; b > a; b -= 2) s3 = fma(-blk[a * W + NP + b - a], y[b], s3);
                // quotient by the diagonal: the product with its reciprocal and one correction
                const double x = y[a] + ((s0 + s1) + (s2 + s3)), r = rinv[a], q = x * r;
                y[a] = fma(fma(-q, blk[a * W + NP], x), r, q);
            }
            if (live) {
#pragma unroll
                for (int a = 0; a < NP; ++a) {
                    if (a < n) {
                        if (I == 0) out[(long long)a * m] = dtn_x * (y[a] - (col == a ? 1.0 : 0.0));
                        if (I == n - 1) out[(long long)(n + a) * m] = (-dtn_x) * (y[a] - (col == n + a ? 1.0 : 0.0));
                        if (a == 0) out[(long long)(2 * n + I) * m] = dtn_y * (y[a] - (col == 2 * n + I ? 1.0 : 0.0));
                        if (a == n - 1) out[(long long)(3 * n + I) * m] = (-dtn_y) * (y[a] - (col == 3 * n + I ? 1.0 : 0.0));
                    }
                }
            }
#pragma unroll
            for (int a = 0; a < NP; ++a) yp[a] = y[a];
            __syncthreads();
        }
    }
}

int columns_blocks(int nleaves) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::min(nleaves, 2 * std::max(1, sms));
}

// One warp per (leaf, right-hand side): y = L^{-1} b, x = U^{-1} y on the stored band.
// MODE LEAF_DTN_COLUMN: g = e_unit, f = 0, write column `unit` of T; LEAF_NEUMANN: g = 0;
// LEAF_SOLVE: write u; LEAF_MAPD2N: write h.
template <int MODE>
__global__ void __launch_bounds__(256) k_fp_solve(const FpLeaf* __restrict__ leaves,
                                                  const LeafItem* __restrict__ items, int nitems) {
    const int warp = int((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (warp >= nitems) return;  // whole warp exits together
    const LeafItem it = items[warp];
    const FpLeaf lf = leaves[it.type];
    const int n = lf.n, N = n * n, w = 2 * n + 1;
    extern __shared__ double ybuf[];
    double* y = ybuf + (threadIdx.x >> 5) * N;
    const double* band = lf.band;

    auto gval = [&](int side, int pos) -> double {
        if (MODE == LEAF_DTN_COLUMN) return (it.unit == side * n + pos) ? 1.0 : 0.0;
        if (MODE == LEAF_NEUMANN) return 0.0;
        return it.g[side * n + pos];
    };
    // right-hand side f + f_boundary (FiniteVolumeSolver.cpp:96-184)
    for (int r = lane; r < N; r += 32) {
        const int i = r / n, j = r - (r / n) * n;
        double v = (MODE != LEAF_DTN_COLUMN && it.f != nullptr) ? it.f[r] : 0.0;
        if (i == 0 || i == n - 1 || j == 0 || j == n - 1) {
            double acc = 0.0;
            bool any = false;
            if (i == 0) { acc = lf.bcoef[j] * gval(0, j); any = true; }
            else if (i == n - 1) { acc = lf.bcoef[n + j] * gval(1, j); any = true; }
            if (j == 0) { const double t = lf.bcoef[2 * n + i] * gval(2, i); acc = any ? acc + t : t; }
            else if (j == n - 1) { const double t = lf.bcoef[3 * n + i] * gval(3, i); acc = any ? acc + t : t; }
            v += -2.0 * acc;
        }
        y[r] = v;
    }
    __syncwarp();
    // forward: y_k -= sum_{d=1..n} L[k][k-d] y_{k-d}
    for (int k = 1; k < N; ++k) {
        double s = 0.0;
        for (int d = lane + 1; d <= n; d += 32)
            if (k - d >= 0) s = fma(band[(long long)k * w + n - d], y[k - d], s);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) y[k] -= s;
        __syncwarp();
    }
    // backward: x_k = (y_k - sum_{e=1..n} U[k][k+e] x_{k+e}) / U[k][k]
    for (int k = N - 1; k >= 0; --k) {
        double s = 0.0;
        for (int e = lane + 1; e <= n; e += 32)
            if (k + e < N) s = fma(band[(long long)k * w + n + e], y[k + e], s);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        if (lane == 0) y[k] = (y[k] - s) / band[(long long)k * w + n];
        __syncwarp();
    }
    if (MODE == LEAF_SOLVE) {
        for (int r = lane; r < N; r += 32) it.out[r] = y[r];
    } else {
        // Neumann data of FiniteVolumeSolver.cpp:296-353
        const double dtn_x = 2.0 / lf.dx, dtn_y = 2.0 / lf.dy;
        const int m = 4 * n;
        for (int r = lane; r < m; r += 32) {
            const int side = r / n, pos = r - (r / n) * n;
            int cell;
            if (side == 0) cell = pos;
            else if (side == 1) cell = (n - 1) * n + pos;
            else if (side == 2) cell = pos * n;
            else cell = pos * n + n - 1;
            const double gv = gval(side, pos);
            double h;
            if (side == 0) h = dtn_x * (y[cell] - gv);
            else if (side == 1) h = (-dtn_x) * (y[cell] - gv);
            else if (side == 2) h = dtn_y * (y[cell] - gv);
            else h = (-dtn_y) * (y[cell] - gv);
            if (MODE == LEAF_DTN_COLUMN) it.out[(long long)r * m + it.unit] = h;
            else it.out[r] = h;
        }
    }
}

// sum of coef(b) x[b] over b < n in four partial sums
template <class F>
__device__ __forceinline__ double rows_sum(int n, F&& coef, const double* x) {
    double p0 = 0.0, p1 = 0.0, p2 = 0.0, p3 = 0.0;
    int b = 0;
    for (; b + 3 < n; b += 4) {
        p0 = fma(coef(b), x[b], p0);
        p1 = fma(coef(b + 1), x[b + 1], p1);
        p2 = fma(coef(b + 2), x[b + 2], p2);
        p3 = fma(coef(b + 3), x[b + 3], p3);
    }
    for (; b < n; ++b) p0 = fma(coef(b), x[b], p0);
    return (p0 + p1) + (p2 + p3);
}

// The same for leaves of at most 32 x 32 cells, one right-hand side each: a warp takes the band block row by
// block row (the n rows of one grid column, one row per lane) through shared memory, two blocks in flight.
// In a block the n products with the previous block's values run in all lanes at once; the triangle then takes
// one shuffle and one multiply-add per row (and the quotient by U's diagonal on the way back, from reciprocals
// taken for the block together).  Latency bound: 2 n^2 steps of ~100 to 300 clocks, several leaves per SM, where
// a row at a time took two reductions over the warp from global memory per row.  Solve and Neumann step of 1024 leaves
// of 32 x 32 cells: 0.8 ms each.
template <int MODE>
__global__ void __launch_bounds__(32) k_fp_solve_blocks(const FpLeaf* __restrict__ leaves,
                                                        const LeafItem* __restrict__ items) {
    const LeafItem it = items[blockIdx.x];
    const FpLeaf& lf = leaves[it.type];
    const int n = lf.n, N = n * n, w = 2 * n + 1, lane = threadIdx.x;
    const int W = n + 2 - (n & 1);  // row stride: lanes read along diagonals, W - 1 odd spreads them over the banks
    extern __shared__ double fb_smem[];
    double* y = fb_smem + 2 * n * W;  // N values
    const double* band = lf.band;
    const bool row_lane = lane < n;
    auto gval = [&](int side, int pos) -> double {
        if (MODE == LEAF_NEUMANN) return 0.0;
        return it.g[side * n + pos];
    };
    // half of a block's band entries: `half` 0: c - r + n in [0, n) (L), 1: [n, 2n] (U)
    auto load = [&](int I, int half) {
        const double* src = band + (long long)I * n * w + half * n;
        double* dst = fb_smem + (I & 1) * n * W;
        const int len = n + half;
        for (int a = 0; a < n; ++a)
            for (int c = lane; c < len; c += 32) copy8_async(dst + a * W + c, src + a * w + c);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto arrived = [&](bool more) {
        if (more) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncwarp();
    };
    load(0, 0);
    for (int I = 0; I < n; ++I) {
        if (I + 1 < n) load(I + 1, 0);
        // right-hand side f + f_boundary (FiniteVolumeSolver.cpp:96-184)
        double s = 0.0;
        if (row_lane) {
            const int r = I * n + lane, j = lane;
            s = it.f != nullptr ? it.f[r] : 0.0;
            if (I == 0 || I == n - 1 || j == 0 || j == n - 1) {
                double acc = 0.0;
                bool any = false;
                if (I == 0) { acc = lf.bcoef[j] * gval(0, j); any = true; }
                else if (I == n - 1) { acc = lf.bcoef[n + j] * gval(1, j); any = true; }
                if (j == 0) { const double t = lf.bcoef[2 * n + I] * gval(2, I); acc = any ? acc + t : t; }
                else if (j == n - 1) { const double t = lf.bcoef[3 * n + I] * gval(3, I); acc = any ? acc + t : t; }
                s += -2.0 * acc;
            }
        }
        arrived(I + 1 < n);
        const double* row = fb_smem + (I & 1) * n * W + (row_lane ? lane * (W - 1) : 0);  // row[b]: entry b - lane
        if (I > 0) {
            const double* yp = y + (I - 1) * n;
            s += rows_sum(n, [&](int b) { return row_lane && b >= lane ? -row[b] : 0.0; }, yp);
        }
        for (int b = 0; b < n - 1; ++b) {
            const double yb = __shfl_sync(0xffffffffu, s, b);
            if (row_lane && lane > b) s = fma(-row[n + b], yb, s);
        }
        if (row_lane) y[I * n + lane] = s;
        __syncwarp();
    }
    load(n - 1, 1);
    for (int I = n - 1; I >= 0; --I) {
        if (I > 0) load(I - 1, 1);
        arrived(I > 0);
        double s = row_lane ? y[I * n + lane] : 0.0;
        const double* row = fb_smem + (I & 1) * n * W + (row_lane ? lane * (W - 1) : 0);
        const double d = row_lane ? row[lane] : 1.0, r = 1.0 / d;
        if (I < n - 1) {
            const double* xn = y + (I + 1) * n;
            s += rows_sum(n, [&](int b) { return row_lane && b <= lane ? -row[n + b] : 0.0; }, xn);
        }
        for (int b = n - 1; b >= 0; --b) {
            const double q = s * r, x = fma(fma(-q, d, s), r, q);  // s / d: the product and one correction
            const double xb = __shfl_sync(0xffffffffu, x, b);
            if (lane == b) s = x;
            else if (lane < b) s = fma(-row[b], xb, s);
        }
        if (row_lane) y[I * n + lane] = s;
        __syncwarp();
    }
    if (MODE == LEAF_SOLVE) {
        for (int r = lane; r < N; r += 32) it.out[r] = y[r];
    } else {
        // Neumann data of FiniteVolumeSolver.cpp:296-353
        const double dtn_x = 2.0 / lf.dx, dtn_y = 2.0 / lf.dy;
        for (int r = lane; r < 4 * n; r += 32) {
            const int side = r / n, pos = r - side * n;
            const int cell = side == 0 ? pos : side == 1 ? (n - 1) * n + pos : side == 2 ? pos * n : pos * n + n - 1;
            const double scale = side == 0 ? dtn_x : side == 1 ? -dtn_x : side == 2 ? dtn_y : -dtn_y;
            it.out[r] = scale * (y[cell] - gval(side, pos));
        }
    }
}

template <int MODE>
void launch_fp_solve(cudaStream_t st, const FpLeaf* leaves, const LeafItem* items, int nitems, int nmax) {
    if (MODE != LEAF_DTN_COLUMN && nmax <= 32) {
        const size_t smem = (2 * size_t(nmax) * (nmax + 2) + size_t(nmax) * nmax) * sizeof(double);
        cudaFuncSetAttribute(k_fp_solve_blocks<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        k_fp_solve_blocks<MODE><<<unsigned(nitems), 32, smem, st>>>(leaves, items);
        ++g_kernel_launches;
        return;
    }
    // one n*n work vector per warp in shared memory (at most 192 KB per CTA)
    const size_t per_warp = size_t(nmax) * nmax * sizeof(double);
    int warps_per_cta = int((192 * 1024) / per_warp);
    if (warps_per_cta > 8) warps_per_cta = 8;
    if (warps_per_cta < 1) warps_per_cta = 1;
    const size_t smem = size_t(warps_per_cta) * per_warp;
    // set on every launch: the attribute is per device and per context, and the call is cheap
    cudaFuncSetAttribute(k_fp_solve<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    const unsigned blocks = unsigned((nitems + warps_per_cta - 1) / warps_per_cta);
    k_fp_solve<MODE><<<blocks, 32 * warps_per_cta, smem, st>>>(leaves, items, nitems);
    ++g_kernel_launches;
}

}  // namespace

void fp_factor(cudaStream_t st, const FpLeaf* leaves, int nleaves, int nmax) {
    if (nleaves <= 0) return;
    const size_t smem = size_t((nmax + 2) * (2 * nmax + 1) + nmax) * sizeof(double);
    cudaFuncSetAttribute(k_fp_factor, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    for (int k = 0; k < nleaves; k += 65535) {
        const int c = std::min(65535, nleaves - k);
        k_fp_stencil<<<dim3(unsigned((nmax * nmax + 255) / 256), unsigned(c)), 256, 0, st>>>(leaves + k);
        ++g_kernel_launches;
    }
    k_fp_factor<<<nleaves, 256, smem, st>>>(leaves);
    ++g_kernel_launches;
}

size_t fp_columns_scratch(int nleaves, int n) {
    return n <= 32 && nleaves > 0 ? size_t(columns_blocks(nleaves)) * n * n * 4 * n * sizeof(double) : 0;
}

void fp_columns(cudaStream_t st, const FpLeaf* leaves, const LeafItem* items, int nleaves, int n, double* scratch) {
    const int threads = (4 * n + 31) / 32 * 32, blocks = columns_blocks(nleaves);
    auto launch = [&](auto kernel, int np) {
        const size_t smem = 2 * size_t(np) * (2 * np + 1) * sizeof(double);
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        kernel<<<blocks, threads, smem, st>>>(leaves, items, nleaves, scratch);
        ++g_kernel_launches;
    };
    if (n <= 8) launch(k_fp_columns<8>, 8);
    else if (n <= 16) launch(k_fp_columns<16>, 16);
    else if (n <= 24) launch(k_fp_columns<24>, 24);
    else launch(k_fp_columns<32>, 32);
}

void fp_solve(cudaStream_t st, int mode, const FpLeaf* leaves, const LeafItem* items, int nitems, int nmax) {
    if (nitems <= 0) return;
    if (mode == LEAF_DTN_COLUMN) launch_fp_solve<LEAF_DTN_COLUMN>(st, leaves, items, nitems, nmax);
    else if (mode == LEAF_NEUMANN) launch_fp_solve<LEAF_NEUMANN>(st, leaves, items, nitems, nmax);
    else if (mode == LEAF_SOLVE) launch_fp_solve<LEAF_SOLVE>(st, leaves, items, nitems, nmax);
    else launch_fp_solve<LEAF_MAPD2N>(st, leaves, items, nitems, nmax);
}

}  // namespace efgb
