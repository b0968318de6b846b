// Mixed-precision passes for variable-coefficient leaves (FiniteVolumeSolverType::FivePointStencil).
//
// The FP64 band LU of every leaf's 5-point operator (factored once at build time, see ef_leaf_fp.cu)
// has bandwidth n, so with the cells split into n blocks of n rows the triangular solves are
//     forward   y_j = L_jj^{-1} q_j - (L_jj^{-1} L_{j,j-1}) y_{j-1}
//     backward  x_j = U_jj^{-1} y_j - (U_jj^{-1} U_{j,j+1}) x_{j+1}
// At set-up the four n x n matrices of every block row are formed in FP64 and stored in FP32; a block of
// requests is then solved per leaf in 2n steps of two products over the requests, only one of which
// waits for the step before.  The FP64 stencil coefficients cW, cE, cS, cN,
// cC of FiniteVolumeSolver.cpp:66-100 are tabulated per cell for the residual, which uses the same
// ghost treatment as the reference's boundary rows (cpp:100-184): a missing neighbour is 2g - u_C.
#include <algorithm>

#include "ef_kernels.cuh"
#include "ef_mixed_common.cuh"

namespace efgb {

namespace {

// one CTA per leaf: FP32 boundary coefficients, FP64 stencil table
__global__ void __launch_bounds__(256) k_mx_fp_convert(const FpLeaf* __restrict__ src, const MixFp* __restrict__ dst) {
    const FpLeaf lf = src[blockIdx.x];
    const MixFp mf = dst[blockIdx.x];
    const int n = lf.n, N = n * n;
    const double dx2 = lf.dx * lf.dx, dy2 = lf.dy * lf.dy;
    for (int e = threadIdx.x; e < 4 * n; e += blockDim.x) mf.bcoef[e] = float(lf.bcoef[e]);
    for (int r = threadIdx.x; r < N; r += blockDim.x) {
        const double a = lf.alpha[r];
        const double bW = lf.beta[r], bE = lf.beta[N + r], bS = lf.beta[2 * N + r], bN = lf.beta[3 * N + r];
        mf.coef[r] = a * bW / dx2;
        mf.coef[N + r] = a * bE / dx2;
        mf.coef[2 * N + r] = a * bS / dy2;
        mf.coef[3 * N + r] = a * bN / dy2;
        mf.coef[4 * N + r] = -a * ((bE + bW) / dx2 + (bN + bS) / dy2) + lf.lambda[r];
    }
}

// Block rows of the band LU, CTA = (block j, leaf): each thread takes one column of one of the four matrices
// { L_jj^{-1}, L_jj^{-1} L_{j,j-1}, U_jj^{-1}, U_jj^{-1} U_{j,j+1} } by substitution in FP64, stored FP32 as
// blocks[j][4][n][n] with the columns contiguous (entry (a, k) at k n + a).  Band row r holds columns
// r-n .. r+n at positions 0 .. 2n (L multipliers | U); the block's rows and the columns under way lie in
// shared memory.
__global__ void k_mx_fp_blocks(const FpLeaf* __restrict__ src, const MixFp* __restrict__ dst) {
    const FpLeaf& lf = src[blockIdx.y];
    const int n = lf.n, w = 2 * n + 1, j = blockIdx.x, nt = blockDim.x;
    extern __shared__ double fbk_smem[];
    double* band = fbk_smem;      // n x w
    double* X = band + n * w;     // n x nt: a column per thread
    for (int e = threadIdx.x; e < n * w; e += nt) band[e] = lf.band[(long long)j * n * w + e];
    __syncthreads();
    float* out = dst[blockIdx.y].blocks + (long long)j * 4 * n * n;
    const int kind = threadIdx.x / n, k = threadIdx.x - kind * n;
    double* x = X + threadIdx.x;
    if (kind < 2) {
        // x_a = v_a - sum_{b<a} L[a][b] x_b, L[a][b] at n - (a - b); L_{j,j-1}[a][b] (b >= a) at b - a
        for (int a = 0; a < n; ++a) {
            double v = kind == 0 ? (a == k ? 1.0 : 0.0) : (j > 0 && k >= a ? band[a * w + k - a] : 0.0);
            for (int b = kind == 0 ? k : 0; b < a; ++b) v = fma(-band[a * w + n - (a - b)], x[b * nt], v);
            x[a * nt] = a < k && kind == 0 ? 0.0 : v;
        }
    } else if (kind < 4) {
        // x_a = (v_a - sum_{b>a} U[a][b] x_b) / U[a][a], U[a][b] at n + (b - a); U_{j,j+1}[a][b] (b <= a) at 2n + b - a
        for (int a = n - 1; a >= 0; --a) {
            double v = kind == 2 ? (a == k ? 1.0 : 0.0) : (j < n - 1 && k <= a ? band[a * w + 2 * n + k - a] : 0.0);
            for (int b = a + 1; b <= (kind == 2 ? k : n - 1); ++b) v = fma(-band[a * w + n + (b - a)], x[b * nt], v);
            x[a * nt] = a > k && kind == 2 ? 0.0 : v / band[a * w + n];
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 4 * n * n; e += nt) {
        const int col = e / n, a = e - col * n;  // column of all four matrices: kind * n + k
        out[e] = float(X[a * nt + col]);
    }
}

constexpr int kFpReq = 8;     // requests per warp
constexpr int kFpWarps = 2;
constexpr int kFpGroup = kFpReq * kFpWarps;
constexpr int kFpStages = 3;  // block rows in flight

// Block solve of one leaf for a group of 16 requests (blockIdx.y).  A warp takes eight requests, a lane one
// row of the block; the two matrices of a step stream through a ring of three stages that both warps
// read.  Per k a lane reads its two matrix entries and, as broadcasts, the eight right-hand sides and the
// eight previous values of row k: six shared-memory wavefronts for 512 multiply-adds, which bounds the kernel
// (the matrices' 512 MB of a 1024-leaf, 32 x 32 tree would take 75 us).  A warp exchanges rows inside itself, so
// the only block barrier of a step is the ring's.  y goes through `scratch` between the sweeps.  A block of 16
// requests on that tree, four leaf solves and the rest: 5.4 ms with a group's vectors in shared memory and 2n dependent
// products, 1.7 ms.
// NEUMANN: g = 0, load q, write h32 = DtN(0, q).  SOLVE: load q + boundary terms of g32, add (or store,
// accumulate == 0) the solution to u64.
// FEW: the loop over k unrolled by eight, both products side by side; else by four, one after the other (the same sums).
template <int MODE, bool FEW>
__global__ void __launch_bounds__(32 * kFpWarps) k_mx_fp_leaf32(const MixFp* __restrict__ fps, const MixLeaf* __restrict__ leaves,
                                                              int L, int B, int n, const float* __restrict__ q,
                                                              double* __restrict__ u64, float* __restrict__ scratch,
                                                              int accumulate) {
    extern __shared__ __align__(16) float fsm[];
    const int N = n * n, n2 = n * n;
    const int leaf = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b0 = (blockIdx.y * kFpWarps + warp) * kFpReq, nb = max(0, min(kFpReq, B - b0));
    const bool row = lane < n;
    const int a = row ? lane : 0;
    float* ring = fsm;                                                       // [stage][2][n][n]
    float* sq = fsm + kFpStages * 2 * n2 + warp * 2 * 32 * kFpReq;           // [32][8] right-hand sides of the block
    float* sy = sq + 32 * kFpReq;                                            // [32][8] values of the block before
    const MixFp mf = fps[leaf];
    const MixLeaf lf = leaves[leaf];
    float* Y = scratch + (((long long)blockIdx.y * L + leaf) * kFpWarps + warp) * N * kFpReq;
    const float* qb = q + ((long long)b0 * L + leaf) * N;
    const long long qs = (long long)L * N;
    auto stage = [&](int j, int half, int slot) {
        const float* g = mf.blocks + ((long long)j * 4 + 2 * half) * n2;
        for (int e = 4 * tid; e < 2 * n2; e += 4 * 32 * kFpWarps) cp_async16(ring + slot * 2 * n2 + e, g + e, 16);
    };
    // boundary terms of a cell on a W/E face (side 0, 1) and on an S/N face (side 2, 3)
    auto face = [&](int side, int pos, int r) {
        return -2.0f * mf.bcoef[side * n + pos] * lf.g32[(long long)(side * n + pos) * B + b0 + r];
    };
    auto fetch_q = [&](int j, float (&v)[kFpReq]) {
#pragma unroll
        for (int r = 0; r < kFpReq; ++r) v[r] = row && r < nb ? qb[r * qs + j * n + a] : 0.f;
        if (MODE == LEAF_SOLVE && row) {
            const bool x = j == 0 || j == n - 1, y = a == 0 || a == n - 1;
            if (x || y) {
#pragma unroll
                for (int r = 0; r < kFpReq; ++r)
                    if (r < nb) {
                        float t = x ? face(j == 0 ? 0 : 1, a, r) : 0.f;
                        if (y) t += face(a == 0 ? 2 : 3, j, r);
                        v[r] += t;
                    }
            }
        }
    };
    // one row of both products: acc = M1 rhs - M2 prev.  Each has a sum of its own: the two are large against their
    // difference, and in one chain every addition rounded at the size of what has been added so far (the error of a block after
    // one sweep 1.1 to 1.9 times that of products formed one after the other, now 0.7 to 0.9).
    auto products = [&](int slot, float (&acc)[kFpReq]) {
        const float* m1 = ring + slot * 2 * n2 + a;
        const float* m2 = m1 + n2;
        float sub[kFpReq];
#pragma unroll
        for (int r = 0; r < kFpReq; ++r) acc[r] = sub[r] = 0.f;
        auto add = [](float (&c)[kFpReq], float x, const float4& p0, const float4& p1) {
            c[0] = fmaf(x, p0.x, c[0]); c[1] = fmaf(x, p0.y, c[1]); c[2] = fmaf(x, p0.z, c[2]); c[3] = fmaf(x, p0.w, c[3]);
            c[4] = fmaf(x, p1.x, c[4]); c[5] = fmaf(x, p1.y, c[5]); c[6] = fmaf(x, p1.z, c[6]); c[7] = fmaf(x, p1.w, c[7]);
        };
        auto row4 = [](const float* p, int k, int h) { return *reinterpret_cast<const float4*>(p + k * kFpReq + 4 * h); };
        if (FEW) {
#pragma unroll 8
            for (int k = 0; k < n; ++k) {
                const float x = m1[k * n], y = m2[k * n];
                const float4 p0 = row4(sq, k, 0), p1 = row4(sq, k, 1), t0 = row4(sy, k, 0), t1 = row4(sy, k, 1);
                add(acc, x, p0, p1);
                add(sub, y, t0, t1);
            }
        } else {
            for (int k = 0; k < n; k += 4) {  // n is a multiple of four
#pragma unroll
                for (int o = 0; o < 4; ++o) add(acc, m1[(k + o) * n], row4(sq, k + o, 0), row4(sq, k + o, 1));
#pragma unroll
                for (int o = 0; o < 4; ++o) add(sub, m2[(k + o) * n], row4(sy, k + o, 0), row4(sy, k + o, 1));
            }
        }
#pragma unroll
        for (int r = 0; r < kFpReq; ++r) acc[r] -= sub[r];
    };
    auto put = [&](float* dst, const float (&v)[kFpReq]) {
        if (row) {
            *reinterpret_cast<float4*>(dst + a * kFpReq) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(dst + a * kFpReq + 4) = make_float4(v[4], v[5], v[6], v[7]);
        }
    };
    float v[kFpReq], acc[kFpReq];
#pragma unroll
    for (int r = 0; r < kFpReq; ++r) v[r] = 0.f;
    put(sy, v);
    // forward sweep
    for (int i = 0; i < kFpStages - 1; ++i) {
        if (i < n) stage(i, 0, i);
        cp_async_commit();
    }
    fetch_q(0, v);
    int slot = 0;
    for (int j = 0; j < n; ++j) {
        cp_async_wait<kFpStages - 2>();
        __syncthreads();  // the stage has arrived for everyone, and the one before is free
        if (j + kFpStages - 1 < n) stage(j + kFpStages - 1, 0, slot == 0 ? kFpStages - 1 : slot - 1);
        cp_async_commit();
        put(sq, v);
        __syncwarp();
        if (j + 1 < n) fetch_q(j + 1, v);
        products(slot, acc);
        __syncwarp();
        put(sy, acc);
        if (row) {
            *reinterpret_cast<float4*>(Y + (long long)(j * n + a) * kFpReq) = make_float4(acc[0], acc[1], acc[2], acc[3]);
            *reinterpret_cast<float4*>(Y + (long long)(j * n + a) * kFpReq + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
        }
        if (++slot == kFpStages) slot = 0;
    }
    cp_async_wait<0>();
    __syncthreads();
    // backward sweep
    for (int i = 0; i < kFpStages - 1; ++i) {
        if (n - 1 - i >= 0) stage(n - 1 - i, 1, i);
        cp_async_commit();
    }
    auto fetch_y = [&](int j, float (&t)[kFpReq]) {
        const float4 t0 = row ? *reinterpret_cast<const float4*>(Y + (long long)(j * n + a) * kFpReq) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 t1 = row ? *reinterpret_cast<const float4*>(Y + (long long)(j * n + a) * kFpReq + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        t[0] = t0.x; t[1] = t0.y; t[2] = t0.z; t[3] = t0.w;
        t[4] = t1.x; t[5] = t1.y; t[6] = t1.z; t[7] = t1.w;
    };
    double* ub = MODE == LEAF_SOLVE ? u64 + ((long long)b0 * L + leaf) * N : nullptr;
    fetch_y(n - 1, v);
#pragma unroll
    for (int r = 0; r < kFpReq; ++r) acc[r] = 0.f;
    put(sy, acc);
    slot = 0;
    for (int j = n - 1; j >= 0; --j) {
        cp_async_wait<kFpStages - 2>();
        __syncthreads();
        if (j - (kFpStages - 1) >= 0) stage(j - (kFpStages - 1), 1, slot == 0 ? kFpStages - 1 : slot - 1);
        cp_async_commit();
        put(sq, v);
        double old[kFpReq];
        if (MODE == LEAF_SOLVE) {
#pragma unroll
            for (int r = 0; r < kFpReq; ++r) old[r] = accumulate && row && r < nb ? ub[r * qs + j * n + a] : 0.0;
        }
        __syncwarp();
        if (j > 0) fetch_y(j - 1, v);
        products(slot, acc);
        __syncwarp();
        put(sy, acc);
        if (MODE == LEAF_SOLVE) {
#pragma unroll
            for (int r = 0; r < kFpReq; ++r)
                if (row && r < nb) {
                    const double t = f2d_bits(acc[r]);
                    ub[r * qs + j * n + a] = accumulate ? old[r] + t : t;
                }
        } else if (row) {
            // Neumann data of FiniteVolumeSolver.cpp:296-353 with g = 0
            auto flux = [&](int side, int pos, float scale) {
#pragma unroll
                for (int r = 0; r < kFpReq; ++r)
                    if (r < nb) lf.h32[(long long)(side * n + pos) * B + b0 + r] = scale * acc[r];
            };
            if (j == 0) flux(0, a, float(mf.dtn_x));
            if (j == n - 1) flux(1, a, -float(mf.dtn_x));
            if (a == 0) flux(2, j, float(mf.dtn_y));
            if (a == n - 1) flux(3, j, -float(mf.dtn_y));
        }
        if (++slot == kFpStages) slot = 0;
    }
    cp_async_wait<0>();
}

// FP64 residual with the tabulated stencil (see the constant-coefficient kernel in ef_mixed.cu for
// the layout and the two phases): r = f - (cW x_W + cE x_E + cS x_S + cN x_N + cC u_C).
__global__ void __launch_bounds__(256) k_mx_fp_residual(const MixFp* __restrict__ fps, const MixLeaf* __restrict__ leaves,
                                                        int L, int B, int n, int ipc, int zero_state,
                                                        const double* __restrict__ f, const double* __restrict__ u64,
                                                        float* __restrict__ q, float* __restrict__ rleaf) {
    __shared__ unsigned smax[256];
    const int nn = n * n, tpi = nn / 4;
    const int tpe = tpi < 256 ? tpi : 256;
    const int slot = threadIdx.x / tpe, lt = threadIdx.x - slot * tpe;
    const int item = blockIdx.x * ipc + slot;
    const bool act = slot < ipc && (long long)item < (long long)L * B;
    if (threadIdx.x < ipc) smax[threadIdx.x] = 0u;
    __syncthreads();
    const int leaf = act ? item / B : 0;
    const int b = act ? item - leaf * B : 0;
    const MixLeaf lf = leaves[leaf];
    const MixFp mf = fps[leaf];
    const double* cW = mf.coef;
    const double* cE = mf.coef + nn;
    const double* cS = mf.coef + 2 * nn;
    const double* cN = mf.coef + 3 * nn;
    const double* cC = mf.coef + 4 * nn;
    const long long base = ((long long)b * L + leaf) * nn;
    const double* uu = u64 + base;
    const double* ff = f + base;
    float mx = 0.f;
    if (act) {
        for (int e4 = lt; e4 < tpi; e4 += tpe) {
            const int e = 4 * e4, i = e / n, j0 = e - (e / n) * n;
            float rr[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int c = e + t, j = j0 + t;
                double r = ff[c];
                if (!zero_state) {
                    const double uc = uu[c];
                    r = fma(-cC[c], uc, r);
                    if (i > 0) r = fma(-cW[c], uu[c - n], r);
                    if (i < n - 1) r = fma(-cE[c], uu[c + n], r);
                    if (j > 0) r = fma(-cS[c], uu[c - 1], r);
                    if (j < n - 1) r = fma(-cN[c], uu[c + 1], r);
                }
                rr[t] = d2f_rn_bits(r);
            }
            const bool edge_row = i == 0 || i == n - 1;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int j = j0 + t;
                const bool interior = !edge_row && j > 0 && j < n - 1;
                mx = fmaxf(mx, interior ? fabsf(rr[t]) : 0.f);
            }
            *reinterpret_cast<float4*>(q + base + e) = make_float4(rr[0], rr[1], rr[2], rr[3]);
        }
    }
    __syncthreads();  // the boundary phase rewrites cells stored by other threads of the block
    if (act) {
        // Dirichlet data row k of the leaf
        auto gr = [&](int k) { return mx_row<const double>(lf.arena, lf.gsrc[k], B); };
        for (int k = lt; k < 4 * n - 4; k += tpe) {
            int i, j;
            if (k < n) { i = 0; j = k; }
            else if (k < 2 * n) { i = n - 1; j = k - n; }
            else { const int m = k - 2 * n; i = 1 + (m >> 1); j = (m & 1) ? n - 1 : 0; }
            const int c = i * n + j;
            const double uc = zero_state ? 0.0 : uu[c];
            const double xm = i > 0 ? (zero_state ? 0.0 : uu[c - n]) : fma(2.0, gr(j)[b], -uc);
            const double xp = i < n - 1 ? (zero_state ? 0.0 : uu[c + n]) : fma(2.0, gr(n + j)[b], -uc);
            const double ym = j > 0 ? (zero_state ? 0.0 : uu[c - 1]) : fma(2.0, gr(2 * n + i)[b], -uc);
            const double yp = j < n - 1 ? (zero_state ? 0.0 : uu[c + 1]) : fma(2.0, gr(3 * n + i)[b], -uc);
            const double r = fma(-cN[c], yp, fma(-cS[c], ym, fma(-cE[c], xp, fma(-cW[c], xm, fma(-cC[c], uc, ff[c])))));
            const float rf = d2f_rn_bits(r);
            q[base + c] = rf;
            mx = fmaxf(mx, fabsf(rf));
        }
        atomicMax(&smax[slot], __float_as_uint(mx));
        for (int r = lt; r < 4 * n; r += tpe) {
            const int side = r / n, pos = r - (r / n) * n;
            int cell;
            if (side == 0) cell = pos;
            else if (side == 1) cell = (n - 1) * n + pos;
            else if (side == 2) cell = pos * n;
            else cell = pos * n + n - 1;
            const double gv = gr(r)[b];
            const double dtn = (side == 0 || side == 2) ? (side < 2 ? mf.dtn_x : mf.dtn_y)
                                                        : -(side < 2 ? mf.dtn_x : mf.dtn_y);
            lf.h64[(long long)r * B + b] = zero_state ? -dtn * gv : dtn * (uu[cell] - gv);
        }
    }
    __syncthreads();
    if (rleaf && act && lt == 0) rleaf[(long long)b * L + leaf] = __uint_as_float(smax[slot]);
}

}  // namespace

void mx_fp_blocks(cudaStream_t st, const FpLeaf* src, const MixFp* dst, int L, int n) {
    if (L <= 0) return;
    const int threads = (4 * n + 31) / 32 * 32;
    const size_t smem = (size_t(n) * (2 * n + 1) + size_t(n) * threads) * sizeof(double);
    cudaFuncSetAttribute(k_mx_fp_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    for (int k = 0; k < L; k += 65535) {
        k_mx_fp_blocks<<<dim3(unsigned(n), unsigned(std::min(65535, L - k))), threads, smem, st>>>(src + k, dst + k);
        ++g_kernel_launches;
    }
}

void mx_fp_convert(cudaStream_t st, const FpLeaf* src, const MixFp* dst, int L, int n) {
    if (L <= 0) return;
    k_mx_fp_convert<<<L, 256, 0, st>>>(src, dst);
    ++g_kernel_launches;
    mx_fp_blocks(st, src, dst, L, n);
}

size_t mx_fp_leaf_scratch(int L, int B, int n) {
    return size_t(L) * ((B + kFpGroup - 1) / kFpGroup) * kFpGroup * n * n;
}

void mx_fp_leaf32(cudaStream_t st, int mode, const MixFp* fps, const MixLeaf* leaves, int L, int B, int n,
                  const float* q, double* u64, float* scratch, int accumulate) {
    const size_t smem = (size_t(kFpStages) * 2 * n * n + size_t(kFpWarps) * 2 * 32 * kFpReq) * sizeof(float);
    dim3 grid(unsigned(L), unsigned((B + kFpGroup - 1) / kFpGroup));
    // up to five blocks per SM, all at once at the unrolled form's registers, a step's latency counts (64 leaves of 32 x 32
    // cells, 23 requests: 638 us by fours, 597 unrolled); beyond, the blocks per SM (1024 leaves, 16 requests: 1712 and 1935)
    const bool few = (long long)grid.x * grid.y <= 5 * 152;
    auto kernel = mode == LEAF_NEUMANN ? (few ? k_mx_fp_leaf32<LEAF_NEUMANN, true> : k_mx_fp_leaf32<LEAF_NEUMANN, false>)
                                       : (few ? k_mx_fp_leaf32<LEAF_SOLVE, true> : k_mx_fp_leaf32<LEAF_SOLVE, false>);
    kernel<<<grid, 32 * kFpWarps, smem, st>>>(fps, leaves, L, B, n, q, u64, scratch, mode == LEAF_NEUMANN ? 0 : accumulate);
    ++g_kernel_launches;
}

void mx_fp_residual(cudaStream_t st, const MixFp* fps, const MixLeaf* leaves, int L, int B, int n, int zero_state,
                    const double* f, const double* u64, float* q, float* rleaf, double* rmax) {
    const int tpi = n * n / 4, tpe = tpi < 256 ? tpi : 256, ipc = 256 / tpe;
    const long long items = (long long)L * B;
    const unsigned grid = unsigned((items + ipc - 1) / ipc);
    k_mx_fp_residual<<<grid, unsigned(ipc * tpe), 0, st>>>(fps, leaves, L, B, n, ipc, zero_state, f, u64, q,
                                                           rmax ? rleaf : nullptr);
    ++g_kernel_launches;
    if (rmax) mx_rmax(st, rleaf, L, B, rmax);
}

}  // namespace efgb
