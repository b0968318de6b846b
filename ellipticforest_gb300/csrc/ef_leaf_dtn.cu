// Leaf Dirichlet-to-Neumann maps of the constant-coefficient (FISHPACK90) leaf types
// (FiniteVolumeSolver::buildD2N, FiniteVolumeSolver.cpp:355-455).
//
// Column j of T is mapD2N(e_j, f = 0): the solve of A u = -2 c_side e_j at the edge cell of boundary
// point j, then h = +-(2/d)(u_edge - g) (cpp:296-353).  Every leaf of a type takes the same T, so its
// rounding errors add up coherently over the tree, and T applied to smooth data cancels to O(1) from
// entries of O(1/d): T is wanted as close to the rounded exact map as can be had.
//
// Negative definite operators (k_dtn_modes): separation of variables.  With sine modes along the data's
// side the problem across is one-dimensional with constant coefficients, and each entry of T is a sum over
// the n modes.  In FP64 that sum spreads its rounding over every mode (trees built on it drifted by ~N^2
// eps at the leaf solutions, 1.2e-11 at 1024^2 cells); here sines, one-dimensional solutions and sums are
// double-double (unevaluated sums of two doubles; Dekker, "A floating-point technique for extending the
// available precision", Numer. Math. 18, 1971), so an entry is the exact one rounded once or twice.
// For 16 x 16 cells it takes 0.15 ms (the chain of double-double divisions of a mode, then 16 terms per entry)
// where the pivoted LU of the 256 x 256 operator, a chain of pivots, took 2.9 ms.
//
// Others (lambda at or above half the smallest eigenvalue): the pivoted dense LU of the 5-point operator,
// batched over the types (ef_linalg.cu), which also finds singular operators.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "ef_kernels.cuh"

namespace efgb {

namespace {

// A (nn x nn, row-major, cell index j + i n) of u_xx + u_yy + lambda u with the Dirichlet ghost
// 2g - u at the patch faces, as the oracle's five_point_matrix builds it (cpp:66-200 with
// alpha = beta = 1): cW = cE = 1/dx^2, cS = cN = 1/dy^2, cC = -(2/dx^2 + 2/dy^2) + lambda, and the
// ghost moves -c_side onto the diagonal at the faces.
__global__ void k_dtn_assemble(int n, const double* __restrict__ dxs, const double* __restrict__ dys,
                               double lambda, double* const* A) {
    const long long nn = (long long)n * n, tot = nn * nn;
    const int t = blockIdx.y;
    const double dx = dxs[t], dy = dys[t];
    const double cx = 1.0 * 1.0 / (dx * dx), cy = 1.0 * 1.0 / (dy * dy);
    const double cC = -1.0 * ((1.0 + 1.0) / (dx * dx) + (1.0 + 1.0) / (dy * dy)) + lambda;
    double* __restrict__ a = A[t];
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot;
         e += (long long)gridDim.x * blockDim.x) {
        const int r = int(e / nn), c = int(e - (e / nn) * nn);
        const int i = r / n, j = r - (r / n) * n;
        double v = 0.0;
        if (c == r) {
            double d = cC;
            if (i == 0) d -= cx;
            if (i == n - 1) d -= cx;
            if (j == 0) d -= cy;
            if (j == n - 1) d -= cy;
            v = d;
        } else if (c == r - n && i > 0) {
            v = cx;
        } else if (c == r + n && i < n - 1) {
            v = cx;
        } else if (c == r - 1 && j > 0) {
            v = cy;
        } else if (c == r + 1 && j < n - 1) {
            v = cy;
        }
        a[e] = v;
    }
}

// edge cell (j + i n) next to boundary point p in WESN order
__device__ __forceinline__ int edge_cell(int p, int n) {
    const int side = p / n, k = p - (p / n) * n;
    if (side == 0) return k;                  // W: i = 0, j = k
    if (side == 1) return (n - 1) * n + k;    // E: i = n-1
    if (side == 2) return k * n;              // S: j = 0, i = k
    return k * n + n - 1;                     // N: j = n-1
}

// right-hand sides of the 4n unit Dirichlet data, rows already permuted by the LU's row order:
// B[r][p] = f_boundary(e_p)[perm[r]] = -2 c_side(p) at the edge cell of p (cpp:96-184)
__global__ void k_dtn_rhs(int n, const double* __restrict__ dxs, const double* __restrict__ dys,
                          const int* const* perm, double* const* B) {
    const int nn = n * n, m = 4 * n;
    const int t = blockIdx.y;
    const double cx = 1.0 * 1.0 / (dxs[t] * dxs[t]), cy = 1.0 * 1.0 / (dys[t] * dys[t]);
    const int* __restrict__ pm = perm[t];
    double* __restrict__ b = B[t];
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nn * m; e += gridDim.x * blockDim.x) {
        const int r = e / m, p = e - (e / m) * m;
        const int src = pm[r];
        b[e] = (src == edge_cell(p, n)) ? -2.0 * (p < 2 * n ? cx : cy) : 0.0;
    }
}

// T[q][p] = s_q (2/d_q)(u_p[edge_cell(q)] - delta_qp): W +2/dx, E -2/dx, S +2/dy, N -2/dy
__global__ void k_dtn_extract(int n, const double* __restrict__ dxs, const double* __restrict__ dys,
                              const double* const* U, double* const* T) {
    const int m = 4 * n;
    const int t = blockIdx.y;
    const double dtn_x = 2.0 / dxs[t], dtn_y = 2.0 / dys[t];
    const double* __restrict__ u = U[t];
    double* __restrict__ out = T[t];
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m * m; e += gridDim.x * blockDim.x) {
        const int q = e / m, p = e - (e / m) * m;
        const int side = q / n;
        const double diff = u[(long long)edge_cell(q, n) * m + p] - (q == p ? 1.0 : 0.0);
        const double scale = side == 0 ? dtn_x : side == 1 ? -dtn_x : side == 2 ? dtn_y : -dtn_y;
        out[e] = scale * diff;
    }
}

// ---- double-double ----
struct dd {
    double h, l;
};
// A compiler may fuse a product with a sum that it feeds, which these steps cannot stand: on the device they are
// written with the operations that are never fused, on the host the products are fused multiply-adds already.
__host__ __device__ inline double add_rn(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dadd_rn(a, b);
#else
    return a + b;
#endif
}
__host__ __device__ inline double fma_rn(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
__host__ __device__ inline double mul_rn(double a, double b) {
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return std::fma(a, b, 0.0);
#endif
}
__host__ __device__ inline dd quick_sum(double a, double b) {  // |a| >= |b|
    const double s = add_rn(a, b);
    return {s, add_rn(b, -add_rn(s, -a))};
}
__host__ __device__ inline dd two_sum(double a, double b) {
    const double s = add_rn(a, b), t = add_rn(s, -a);
    return {s, add_rn(add_rn(a, -add_rn(s, -t)), add_rn(b, -t))};
}
__host__ __device__ inline dd operator+(dd a, dd b) {
    const dd s = two_sum(a.h, b.h), t = two_sum(a.l, b.l);
    const dd u = quick_sum(s.h, add_rn(s.l, t.h));
    return quick_sum(u.h, add_rn(u.l, t.l));
}
__host__ __device__ inline dd operator-(dd a) { return {-a.h, -a.l}; }
__host__ __device__ inline dd operator-(dd a, dd b) { return a + (-b); }
__host__ __device__ inline dd operator*(dd a, dd b) {
    const double p = mul_rn(a.h, b.h);
    return quick_sum(p, add_rn(fma_rn(a.h, b.h, -p), fma_rn(a.h, b.l, mul_rn(a.l, b.h))));
}
__host__ __device__ inline dd operator/(dd a, dd b) {
    const double q1 = a.h / b.h;
    dd r = a - b * dd{q1, 0.0};
    const double q2 = r.h / b.h;
    r = r - b * dd{q2, 0.0};
    const dd q = quick_sum(q1, q2);
    return q + dd{r.h / b.h, 0.0};
}

constexpr int kMaxSide = 64;
struct SineTable {
    dd s[kMaxSide + 1];  // sin(pi k / (2n)), k = 0 .. n
};
// Taylor series in double-double; the angle is at most pi / 2, so 30 terms reach 1e-33
SineTable sine_table(int n) {
    const dd pi{3.141592653589793116, 1.224646799147353207e-16};
    SineTable t{};
    for (int k = 0; k <= n; ++k) {
        const dd x = pi * dd{double(k), 0.0} / dd{2.0 * n, 0.0}, x2 = x * x;
        dd term = x, sum = x;
        for (int j = 1; j < 30; ++j) {
            term = -(term * x2 / dd{2.0 * j * (2.0 * j + 1.0), 0.0});
            sum = sum + term;
        }
        t.s[k] = sum;
    }
    return t;
}

// One-dimensional problem across the patch for mode l of data on its near side (cell spacing d, along the
// side e): with kappa = (d/e)^2 4 sin^2(pi (l+1) / 2n) - lambda d^2 the solution m cells from the far side
// grows like q_0 = 1, q_1 = 3 + kappa, q_{m+1} = (2 + kappa) q_m - q_{m-1} (ghost -q_0 beyond the far side,
// 2g - u beyond the near one), u_m = 2 q_m / (q_{n-1} + q_n) g.  Carried as the ratios r_m = q_{m-1} / q_m
// = 1 / (2 + kappa - r_{m-1}), which neither overflow nor cancel.
// Entry (q, p) of T: the modes' sum of sine at q x sine at p x one-dimensional solution, times 2 / spacing.
__global__ void __launch_bounds__(256) k_dtn_modes(const __grid_constant__ SineTable S, int n,
                                                   const LeafType* __restrict__ types, double lambda, double* T) {
    extern __shared__ dd sm_dd[];
    dd* V = sm_dd;          // V[l][j] = sin(pi (l+1)(2j+1) / 2n)
    dd* R = V + n * n;      // [2][l][m]: weight of mode l times u_m; across x (data on W, E), across y
    dd* D = R + 2 * n * n;  // [2][l]: weight times (u at the near cell - g)
    const double dx = types[blockIdx.y].dx, dy = types[blockIdx.y].dy;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int l = e / n, j = e - l * n;
        int k = ((l + 1) * (2 * j + 1)) % (4 * n);
        const bool neg = k > 2 * n;
        if (neg) k -= 2 * n;
        const dd v = S.s[k > n ? 2 * n - k : k];
        V[e] = neg ? -v : v;
    }
    for (int e = threadIdx.x; e < 2 * n; e += blockDim.x) {
        const int dir = e / n, l = e - dir * n;
        const double d = dir == 0 ? dx : dy, g = dir == 0 ? dy : dx;
        const dd d2 = dd{d, 0.0} * dd{d, 0.0}, g2 = dd{g, 0.0} * dd{g, 0.0}, s = S.s[l + 1];
        const dd kappa = dd{4.0, 0.0} * s * s * (d2 / g2) - d2 * dd{lambda, 0.0};
        const dd two = dd{2.0, 0.0} + kappa, one{1.0, 0.0};
        const dd weight = dd{l == n - 1 ? 1.0 : 2.0, 0.0} / dd{double(n), 0.0};
        dd* r = R + (dir * n + l) * n;
        dd q = one / (one + two);  // r_1
        for (int m = 1; m < n; ++m) {
            r[m - 1] = q;
            q = one / (two - q);
        }
        D[e] = weight * ((q - one) / (q + one));
        dd u = weight * (dd{2.0, 0.0} * q / (q + one));  // near cell (m = n - 1), then inwards
        for (int m = n - 1; m > 0; --m) {
            const dd next = u * r[m - 1];
            r[m] = u;
            u = next;
        }
        r[0] = u;
    }
    __syncthreads();
    const int m4 = 4 * n;
    double* out = T + (long long)blockIdx.y * m4 * m4;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < m4 * m4; e += gridDim.x * blockDim.x) {
        const int q = e / m4, p = e - q * m4, a = q / n, o = q - a * n, b = p / n, c = p - b * n;
        const int dir = b < 2 ? 0 : 1;           // the data's sides lie across this direction
        const bool low = (b & 1) == 0;           // W or S
        const dd* r = R + dir * n * n;
        dd sum{0.0, 0.0};
        if (a == b) {
            for (int l = 0; l < n; ++l) sum = sum + V[l * n + o] * V[l * n + c] * D[dir * n + l];
        } else if ((a < 2) == (b < 2)) {         // the opposite side: the far cell
            for (int l = 0; l < n; ++l) sum = sum + V[l * n + o] * V[l * n + c] * r[l * n];
        } else {                                 // a neighbouring side: its o-th cell, n-1-o or o cells from the far side
            const int m = low ? n - 1 - o : o, end = (a & 1) ? n - 1 : 0;
            for (int l = 0; l < n; ++l) sum = sum + V[l * n + end] * V[l * n + c] * r[l * n + m];
        }
        const double scale = (a & 1 ? -2.0 : 2.0) / (a < 2 ? dx : dy);
        const dd t = sum * dd{scale, 0.0};
        out[e] = t.h + t.l;
    }
}

void ck(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string("CUDA error in ") + what + ": " + cudaGetErrorString(e));
}

}  // namespace

bool leaf_dtn_definite(int n, double lambda, double dx, double dy) {
    const double q = std::sin(M_PI / (2.0 * n));
    const double smallest = 4.0 * q * q * (1.0 / (dx * dx) + 1.0 / (dy * dy));  // of the negative Laplacian
    return n <= kMaxSide && lambda < 0.5 * smallest;
}

void leaf_dtn_modes(cudaStream_t st, int n, double lambda, const LeafType* types_dev, int nt, double* T) {
    if (nt <= 0) return;
    const SineTable S = sine_table(n);
    const size_t smem = (3 * size_t(n) * n + 2 * n) * sizeof(dd);
    ck(cudaFuncSetAttribute(k_dtn_modes, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)), "leaf DtN attribute");
    // a block per 128 entries, every block with its own tables, up to about a block per SM over all types
    const int slices = std::max(1, std::min(16 * n * n / 128, 152 / nt));
    k_dtn_modes<<<dim3(slices, nt), 256, smem, st>>>(S, n, types_dev, lambda, T);
    ++g_kernel_launches;
    ck(cudaGetLastError(), "leaf DtN launch");
}

int leaf_dtn_lu(cudaStream_t st, int n, double lambda, const std::vector<double>& dx, const std::vector<double>& dy,
                const std::vector<double*>& T) {
    const int nt = int(dx.size());
    if (nt == 0) return 0;
    if (int(dy.size()) != nt || int(T.size()) != nt) throw std::invalid_argument("leaf_dtn_lu: table sizes differ");
    const size_t nn = size_t(n) * n, m = 4 * size_t(n);
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t oA = 0, oB = oA + up(nt * nn * nn * 8), oP = oB + up(nt * nn * m * 8),
                 oQ = oP + up(nt * nn * 4), oI = oQ + up(nt * nn * 4), oDx = oI + up(nt * 4),
                 oDy = oDx + up(nt * 8), oArr = oDy + up(nt * 8), total = oArr + up(6 * nt * sizeof(void*));
    char* buf = nullptr;
    const cudaError_t got = cudaMalloc(&buf, total);
    if (got == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();
        throw std::bad_alloc();
    }
    ck(got, "cudaMalloc(leaf DtN LU)");
    std::vector<void*> arr(6 * nt);
    for (int t = 0; t < nt; ++t) {
        arr[0 * nt + t] = buf + oA + t * nn * nn * 8;  // A (LU in place)
        arr[1 * nt + t] = buf + oB + t * nn * m * 8;   // B -> U
        arr[2 * nt + t] = buf + oP + t * nn * 4;       // piv
        arr[3 * nt + t] = buf + oQ + t * nn * 4;       // perm
        arr[4 * nt + t] = T[t];                        // T out
        arr[5 * nt + t] = nullptr;
    }
    int bad = 0;
    try {
        ck(cudaMemcpyAsync(buf + oDx, dx.data(), nt * 8, cudaMemcpyHostToDevice, st), "dx");
        ck(cudaMemcpyAsync(buf + oDy, dy.data(), nt * 8, cudaMemcpyHostToDevice, st), "dy");
        ck(cudaMemcpyAsync(buf + oArr, arr.data(), arr.size() * sizeof(void*), cudaMemcpyHostToDevice, st), "arrays");
        ck(cudaMemsetAsync(buf + oI, 0, nt * 4, st), "info");
        auto** dA = reinterpret_cast<double**>(buf + oArr);
        auto** dB = dA + nt;
        auto** dP = reinterpret_cast<int**>(dA + 2 * nt);
        auto** dQ = reinterpret_cast<int**>(dA + 3 * nt);
        auto** dT = dA + 4 * nt;
        const double* ddx = reinterpret_cast<const double*>(buf + oDx);
        const double* ddy = reinterpret_cast<const double*>(buf + oDy);
        int* dinfo = reinterpret_cast<int*>(buf + oI);
        const int ga = int(std::min<size_t>((nn * nn + 255) / 256, 4096));
        k_dtn_assemble<<<dim3(ga, nt), 256, 0, st>>>(n, ddx, ddy, lambda, dA);
        ++g_kernel_launches;
        dgetrf_batched(st, int(nn), dA, int(nn), dP, dinfo, nt);
        piv_to_perm(st, int(nn), dP, dQ, nt);
        const int gb = int(std::min<size_t>((nn * m + 255) / 256, 4096));
        k_dtn_rhs<<<dim3(gb, nt), 256, 0, st>>>(n, ddx, ddy, dQ, dB);
        ++g_kernel_launches;
        dlu_solve_permuted(st, int(nn), int(m), (const double* const*)dA, int(nn), dB, int(m), nt);
        const int gt = int(std::min<size_t>((m * m + 255) / 256, 4096));
        k_dtn_extract<<<dim3(gt, nt), 256, 0, st>>>(n, ddx, ddy, (const double* const*)dB, dT);
        ++g_kernel_launches;
        ck(cudaGetLastError(), "leaf DtN launch");
        std::vector<int> info(nt);
        ck(cudaMemcpyAsync(info.data(), dinfo, nt * 4, cudaMemcpyDeviceToHost, st), "info");
        ck(cudaStreamSynchronize(st), "leaf DtN sync");
        for (int v : info) bad += (v != 0);
    } catch (...) {
        cudaStreamSynchronize(st);
        cudaFree(buf);
        throw;
    }
    cudaFree(buf);
    return bad;
}

}  // namespace efgb
