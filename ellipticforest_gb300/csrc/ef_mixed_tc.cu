// Tensor-core (tcgen05) form of the mixed solver's node GEMMs Y[rows][B] = A[rows][K] X[K][B]
// (the FP32 passes' mergeW / mergeH / applyS products, HPSAlgorithm.hpp:1059-1117, :1194-1230).
//
// Precision.  The operators are FP32; each entry a is split once, at set-up, into three bf16 parts
// a = a1 + a2 + a3 (round to nearest at every step: a1 = bf16(a), a2 = bf16(a - a1),
// a3 = bf16(a - a1 - a2); the three 8-bit significands cover FP32's 24 bits, so the sum is exact),
// and the request block X the same way as it is staged.  Every product is formed from the six
// partial products that reach 2^-24 of |a x|:
//     D_hi   += a1 x1                   (TMEM accumulator 1)
//     D_lo_a += a1 x2 + a2 x1 + a3 x1    (TMEM accumulator 2)
//     D_lo_b += a1 x3 + a2 x2            (TMEM accumulator 3)
// with tcgen05.mma kind::f16 (bf16 inputs, exact products, FP32 accumulation); y = D_hi + D_lo_a +
// D_lo_b.  The three X planes lie in shared memory as consecutive rows of one K-major operand
// [x1 | x2 | x3], and the three accumulators as consecutive TMEM columns, so one k-step is three
// MMAs: a1 [x1 x2 x3] (N = 96), a2 [x1 x2] (N = 64, into the two low accumulators) and a3 x1
// (N = 32), each A plane read from shared memory once per k-step (six MMAs of N = 32 read a1 three
// times and a2 twice).  Keeping the small terms in their own accumulators stops them from being
// rounded against the large running sum.  The dropped terms a2 x3, a3 x2, a3 x3 are below
// 2^-24 |a x|.  The tensor core's own FP32 accumulation is not round-to-nearest (a first version
// that accumulated all of K in TMEM made an FP32 pass 2.1x less accurate than CUDA-core FMA
// chains), so every 64-wide K chunk goes to a fresh set of TMEM accumulators and the epilogue warps
// add the chunk's sums to FP32 registers with round-to-nearest: the pass is then at least as
// accurate as the FMA chains, which the one FP64 refinement sweep is sized for (a 3-pass split-TF32
// would round each product to ~2^-21).  The CTA holds all 512 TMEM columns (its shared memory keeps
// it alone on the SM): five sets of 96 columns for one request block per tile, two of 192 for two,
// so the MMAs run that many chunks ahead of the epilogue warps while they store a tile's rows.
//
// Layout.  The three planes of a group's operators (the rows of one kind's operators back to back,
// H with each child's two runs of s rows made adjacent) are stored tiled: each 128-row x 64-column
// block (one 128-byte swizzle row of bf16 per row) is 16 KB of sequential memory already in the
// canonical K-major SWIZZLE_128B order of the MMA operand, so a stage loads each plane with one
// bulk copy (cp.async.bulk) of sequential bytes rather than a tensor-map box of 128 rows K apart.  X is read as FP32 from the pass buffers ([K][B], requests fastest), split, and written
// to shared memory in the same swizzled K-major form by the producer warps.  A tile is 128 rows; a
// tile whose rows use several right-hand-side blocks (nodes of 4s < 128 rows, or the compact H's
// four children) puts the blocks side by side in N (32 requests each) and keeps each row's own
// block in the epilogue.
//
// Roles (288 threads, nine warps, so up to 224 registers a thread):
// warps 0-3 add each chunk's accumulators to registers and run the epilogue (warp w reads TMEM lanes
// 32w..32w+31; the operands a row's epilogue reads are prefetched when its tile starts; the
// exterior rows of DOWN's children are copied by their own launch, k_mx_ext32), warps 4-6
// stage X (the next chunk's loads in flight while the current one is split and written), warp 7
// allocates TMEM and issues the MMAs, warp 8 the bulk copies of the A planes.  Stages
// are handed over through mbarriers; the MMA issuer frees a stage with tcgen05.commit.  Every wait
// gives up after about one second: the kernel then sets the error word, lets its copies and MMAs in
// flight finish (bounded waits), frees its TMEM and returns.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>
#include <map>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

#include "ef_kernels.cuh"
#include "ef_mixed_common.cuh"
#include "ef_tcgen05.cuh"

namespace cg = cooperative_groups;

namespace efgb {

namespace {

constexpr int kTM = 128;                  // rows per tile (MMA M)
constexpr int kTK = 64;                   // K per stage: 64 bf16 = one 128-byte swizzle row
constexpr int kTB = 32;                   // requests per right-hand-side block (MMA N per block)
constexpr int kPlaneA = kTM * kTK * 2;    // bytes of one A plane per stage (16 KB)
constexpr int kPlaneX = kTB * kTK * 2;    // bytes of one X plane per block per stage (4 KB)
constexpr int kTcThreads = 288;
constexpr int kStageThreads = 96;  // warps 4-6
constexpr int kMaxSeg = 2;
constexpr int kXRing = 3;  // FP32 request-block chunks in the staging ring

struct TcShape {
    int rows_item, K, seg_rows, nseg;
};

__host__ __device__ inline TcShape tc_shape(int kind, int s) {
    TcShape t;
    if (kind == MX_W) { t.rows_item = 4 * s; t.K = 4 * s; t.seg_rows = 4 * s; }
    else if (kind == MX_H) { t.rows_item = 8 * s; t.K = 2 * s; t.seg_rows = 2 * s; }
    else { t.rows_item = 4 * s; t.K = 8 * s; t.seg_rows = 4 * s; }
    t.nseg = t.seg_rows >= kTM ? 1 : kTM / t.seg_rows;
    return t;
}

__host__ __device__ constexpr int tc_stages(int nseg) { return nseg <= 1 ? 3 : 2; }
__host__ __device__ constexpr int tc_stage_bytes(int nseg) { return 3 * kPlaneA + 3 * nseg * kPlaneX; }
// stages, barriers (256 bytes), then the FP32 staging ring of the request blocks
__host__ __device__ constexpr size_t tc_smem_bytes(int nseg) {
    return 1024 + size_t(tc_stages(nseg)) * tc_stage_bytes(nseg) + 256 + size_t(kXRing) * nseg * kTK * kTB * 4;
}
// accumulator sets of a chunk: D_hi, D_lo_a, D_lo_b of 32 nseg columns each, as many as fit in 512
__host__ __device__ constexpr int tc_acc_sets(int nseg) { return 512 / (3 * kTB * nseg); }
__host__ __device__ constexpr int tc_tmem_cols(int) { return 512; }
// all of TMEM per CTA needs one CTA per SM: the shared memory of two would exceed the SM's 228 KB
static_assert(2 * tc_smem_bytes(1) > 228 * 1024 && 2 * tc_smem_bytes(2) > 228 * 1024, "one CTA per SM");
// the barrier block (256 bytes): 3 per stage, 2 per accumulator set, drain, never, TMEM slot, abort
static_assert((3 * tc_stages(1) + 2 * tc_acc_sets(1) + 2) * 8 + 8 <= 256, "barrier block");
static_assert((3 * tc_stages(2) + 2 * tc_acc_sets(2) + 2) * 8 + 8 <= 256, "barrier block");

// compact H row order of the planes: child c's rows [2s c, 2s c + 2s) are its W/E run and then its
// S/N run; returns the row p of the WESN compact H (the exterior index) of permuted row pr
__host__ __device__ inline int tc_h_unpermute(int pr, int s) {
    const int c = pr / (2 * s), k = pr - c * 2 * s;
    const int run = k >= s ? 1 : 0, o = k - run * s;
    // alpha: W[0,s) S[4s,5s); beta: E[2s,3s) S[5s,6s); gamma: W[s,2s) N[6s,7s); omega: E[3s,4s) N[7s,8s)
    const int base0[4] = {0, 2, 1, 3}, base1[4] = {4, 5, 6, 7};
    return (run ? base1[c] : base0[c]) * s + o;
}

// bf16 parts of x (round to nearest at each step): x = p0 + p1 + p2 for every finite FP32 x
__device__ __forceinline__ void split3(float x, __nv_bfloat16& p0, __nv_bfloat16& p1, __nv_bfloat16& p2) {
    p0 = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(p0);
    p1 = __float2bfloat16_rn(r1);
    const float r2 = r1 - __bfloat162float(p1);
    p2 = __float2bfloat16_rn(r2);
}
// the same for a pair (a, b) with packed conversions: planes p0, p1, p2 as (a, b) bf16x2 words
__device__ __forceinline__ void split3x2(float a, float b, unsigned& p0, unsigned& p1, unsigned& p2) {
    const __nv_bfloat162 q0 = __floats2bfloat162_rn(a, b);
    const float ra = a - __low2float(q0), rb = b - __high2float(q0);
    const __nv_bfloat162 q1 = __floats2bfloat162_rn(ra, rb);
    const __nv_bfloat162 q2 = __floats2bfloat162_rn(ra - __low2float(q1), rb - __high2float(q1));
    p0 = *reinterpret_cast<const unsigned*>(&q0);
    p1 = *reinterpret_cast<const unsigned*>(&q1);
    p2 = *reinterpret_cast<const unsigned*>(&q2);
}

// right-hand-side block of segment `gseg` of a group (W, DOWN: one per node; H: one per child)
struct TcSeg {
    const float* X1;  // rows k < kb
    const float* X2;  // rows k >= kb (indexed with the same k)
    int kb;
};
template <int KIND>
__device__ __forceinline__ TcSeg tc_seg(const MixItem* __restrict__ items, int s, int B, int gseg) {
    TcSeg t;
    if (KIND == MX_W) { t.X1 = items[gseg].hd; t.X2 = t.X1; t.kb = 4 * s; }
    else if (KIND == MX_DOWN) { t.X1 = items[gseg].gf; t.X2 = t.X1; t.kb = 8 * s; }
    else {
        const MixItem& it = items[gseg >> 2];
        int Ia, Ib;
        mx_child_ifaces(gseg & 3, Ia, Ib);
        t.X1 = it.w + (long long)Ia * s * B;
        t.X2 = it.w + (long long)(Ib - 1) * s * B;  // row k >= s of [w_Ia; w_Ib] is w_Ib[k - s]
        t.kb = s;
    }
    return t;
}

// ---- epilogue of 32 tile rows by one warp ----------------------------------------------------------
// A lane holds a row's sums for the 32 requests of a block.  Rows are 128 bytes (B = 32) in memory, so with 16-byte
// accesses by rows every instruction touched 32 of them.  With B a multiple of 4 the warp therefore exchanges
// its 4-request pieces first: lane (piece c = lane / 4, a = lane mod 4) gets piece c of the rows 4 i + a, i = 0 .. 7, and
// an instruction covers four whole rows (L7 block 4.00 -> 3.94 ms).  Launches with single units per block keep their
// rows (see tc_access), and where B is no multiple of 4 the lane takes its row one request at a time.

// where a tile row reads and writes: its addresses, null for a row past the group's end
struct TcRow {
    const float* src;  // added to the sums: H the child's particular flux hc, DOWN w
    float *d0, *d1;    // W: w; H: h; DOWN: both children's interface rows
    double* state;     // DOWN: the FP64 interface state (null: one launch adds the whole pass's values at its end)
};
template <int KIND>
__device__ __forceinline__ TcRow tc_row(const MixItem* __restrict__ items, int s, int B, int rows_item, int grow, bool in) {
    TcRow t{nullptr, nullptr, nullptr, nullptr};
    if (!in) return t;
    const int item = grow / rows_item, r = grow - item * rows_item;
    const MixItem& it = items[item];
    if (KIND == MX_W) {
        t.d0 = it.w + (long long)r * B;
    } else if (KIND == MX_H) {
        const int p = tc_h_unpermute(r, s);
        int c, q2;
        mx_ext_map(p, s, c, q2);
        t.src = it.hc[c] + (long long)q2 * B;
        t.d0 = it.h + (long long)p * B;
    } else {
        const int I = r / s, o = r - I * s;
        t.src = it.w + (long long)r * B;
        t.d0 = it.gc[mx_lower_child(I)] + (long long)mx_q_lower(I, o, s) * B;
        t.d1 = it.gc[mx_upper_child(I)] + (long long)mx_q_upper(I, o, s) * B;
        if (it.uG) t.state = it.uG + (long long)r * B;
    }
    return t;
}
template <class T>
__device__ __forceinline__ T* row_of_lane(T* p, int lane) {
    return reinterpret_cast<T*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(p), lane));
}

// How the epilogue accesses memory: one request at a time, in 16-byte pieces of a lane's own row, or in pieces exchanged
// first.  The exchange and its addresses are some 110 shuffles, which a block with one unit has nothing to hide behind:
// blocks of 12 requests on trees of 16 x 16 leaves, 1 / 2 / 3 / 5 levels, us: 82 / 121 / 168 / 375 with the exchange
// throughout, 76 / 117 / 162 / 366 without it for single units; 7 levels, 32 requests: 3928 and 3932 (3960 without it).
enum TcAccess : int { TC_SINGLE = 0, TC_ROWS = 1, TC_EXCHANGED = 2 };

// the operand that the epilogue adds, in the layout of the accesses (issued early, so that its latency is hidden)
template <int KIND, TcAccess ACC>
__device__ __forceinline__ void tc_prefetch(const TcRow& row, int B, int b0, float (&pre)[32]) {
    if (KIND == MX_W) return;
    const int lane = threadIdx.x & 31, nb = min(32, B - b0);
    if (KIND == MX_DOWN && row.state) {  // its 256 bytes to L2: read once more per sweep only
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(row.state + b0));
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(row.state + b0 + nb - 1));
    }
    if constexpr (ACC == TC_ROWS) {
#pragma unroll
        for (int q = 0; q < 32; q += 4) {
            const float4 x = row.src && q < nb ? *reinterpret_cast<const float4*>(row.src + b0 + q) : make_float4(0.f, 0.f, 0.f, 0.f);
            pre[q] = x.x; pre[q + 1] = x.y; pre[q + 2] = x.z; pre[q + 3] = x.w;
        }
    } else if constexpr (ACC == TC_EXCHANGED) {
        const int c = lane >> 2, a = lane & 3;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float* p = row_of_lane(row.src, 4 * i + a);
            const float4 x = p && 4 * c < nb ? *reinterpret_cast<const float4*>(p + b0 + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
            pre[4 * i] = x.x; pre[4 * i + 1] = x.y; pre[4 * i + 2] = x.z; pre[4 * i + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int q = 0; q < 32; ++q) pre[q] = row.src && q < nb ? row.src[b0 + q] : 0.f;
    }
}

// v[q] = (A X)[row][b0 + q] of this lane's row (v is used up)
template <int KIND, TcAccess ACC>
__device__ __forceinline__ void tc_store(const TcRow& row, int B, int b0, float (&v)[32], const float (&pre)[32]) {
    const int lane = threadIdx.x & 31, nb = min(32, B - b0);
    if constexpr (ACC == TC_ROWS) {
        if (!row.d0) return;
        if (KIND != MX_W) {
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] += pre[q];
        }
#pragma unroll
        for (int q = 0; q < 32; q += 4) {
            if (q >= nb) continue;
            const float4 o = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
            *reinterpret_cast<float4*>(row.d0 + b0 + q) = o;
            if (KIND == MX_DOWN) *reinterpret_cast<float4*>(row.d1 + b0 + q) = o;
        }
        if (KIND == MX_DOWN && row.state) {
#pragma unroll
            for (int h = 0; h < 32; h += 8) {
                double2 u[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    u[i] = h + 2 * i < nb ? *reinterpret_cast<const double2*>(row.state + b0 + h + 2 * i) : make_double2(0.0, 0.0);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (h + 2 * i < nb)
                        *reinterpret_cast<double2*>(row.state + b0 + h + 2 * i) =
                            make_double2(u[i].x + f2d_bits(v[h + 2 * i]), u[i].y + f2d_bits(v[h + 2 * i + 1]));
            }
        }
        return;
    }
    if constexpr (ACC == TC_EXCHANGED) {
        const int c = lane >> 2, a = lane & 3;
        // piece bits and lane bits change places
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int bit = 1 << k;
            const bool up = (lane >> 2) & bit;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (i & bit) continue;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float &x = v[4 * i + e], &y = v[4 * (i | bit) + e];
                    const float got = __shfl_xor_sync(0xffffffffu, up ? x : y, 4 * bit);
                    if (up) x = got;
                    else y = got;
                }
            }
        }
        if (KIND != MX_W) {
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] += pre[q];
        }
        const bool in = 4 * c < nb;
        const int at = b0 + 4 * c;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float* d0 = row_of_lane(row.d0, 4 * i + a);
            float* d1 = KIND == MX_DOWN ? row_of_lane(row.d1, 4 * i + a) : nullptr;
            if (d0 && in) {
                const float4 o = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                *reinterpret_cast<float4*>(d0 + at) = o;
                if (KIND == MX_DOWN) *reinterpret_cast<float4*>(d1 + at) = o;
            }
        }
        if (KIND == MX_DOWN && __any_sync(0xffffffffu, row.state != nullptr)) {
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                double* st[2];
                double2 u[2][2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    st[k] = row_of_lane(row.state, 4 * (i + k) + a);
                    st[k] = st[k] && in ? st[k] + at : nullptr;
                    if (st[k]) {
                        u[k][0] = *reinterpret_cast<const double2*>(st[k]);
                        u[k][1] = *reinterpret_cast<const double2*>(st[k] + 2);
                    }
                }
#pragma unroll
                for (int k = 0; k < 2; ++k)
                    if (st[k]) {
                        const float* w = v + 4 * (i + k);
                        *reinterpret_cast<double2*>(st[k]) = make_double2(u[k][0].x + f2d_bits(w[0]), u[k][0].y + f2d_bits(w[1]));
                        *reinterpret_cast<double2*>(st[k] + 2) = make_double2(u[k][1].x + f2d_bits(w[2]), u[k][1].y + f2d_bits(w[3]));
                    }
            }
        }
    } else if (row.d0) {
#pragma unroll
        for (int h = 0; h < 32; h += 4) {
            double u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) u[i] = KIND == MX_DOWN && row.state && h + i < nb ? row.state[b0 + h + i] : 0.0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int q = h + i;
                if (q >= nb) continue;
                const float x = KIND == MX_W ? v[q] : v[q] + pre[q];
                row.d0[b0 + q] = x;
                if (KIND == MX_DOWN) {
                    row.d1[b0 + q] = x;
                    if (row.state) row.state[b0 + q] = u[i] + f2d_bits(x);
                }
            }
        }
    }
}

// K split: a thread's 32 partial sums in shared memory, four to a vector and vector i of all n threads together (with
// a thread's own next to each other the 32 lanes of a warp met in one bank, 13 us of a launch), and the sum of
// another rank's added to its own
__device__ __forceinline__ void put_partial(unsigned char* red, const float (&v)[32], int t, int n) {
    float4* r = reinterpret_cast<float4*>(red) + t;
#pragma unroll
    for (int q = 0; q < 32; q += 4) r[q / 4 * n] = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
}
__device__ __forceinline__ void add_partial(const unsigned char* red, float (&v)[32], int t, int n) {
    const float4* r = reinterpret_cast<const float4*>(red) + t;
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = r[i * n];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[4 * i] += x[i].x; v[4 * i + 1] += x[i].y; v[4 * i + 2] += x[i].z; v[4 * i + 3] += x[i].w;
    }
}

template <int KIND, int NSEG, TcAccess ACC>
__global__ void __launch_bounds__(kTcThreads, 1)
    k_mx_umma(const __nv_bfloat16* __restrict__ A3, const MixItem* __restrict__ items, int s, int B, int cnt,
              int ksplit, int ntiles, const int* __restrict__ tmap, int nplanes, int* __restrict__ err) {
    const TcShape sh = tc_shape(KIND, s);  // sh.nseg == NSEG (checked by the launcher)
    const int K = sh.K, R = cnt * sh.rows_item;
    const int nsegs_total = KIND == MX_H ? 4 * cnt : cnt;
    constexpr int NS = tc_stages(NSEG), SB = tc_stage_bytes(NSEG);
    constexpr int ncol = kTB * NSEG, tcols = tc_tmem_cols(NSEG);
    constexpr int NP = tc_acc_sets(NSEG);
    constexpr unsigned idesc1 = tc_idesc(kTM, ncol), idesc2 = tc_idesc(kTM, 2 * ncol), idesc3 = tc_idesc(kTM, 3 * ncol);
    extern __shared__ unsigned char tc_smem[];
    unsigned char* base = tc_smem + ((1024u - (smem_u32(tc_smem) & 1023u)) & 1023u);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(base + size_t(NS) * SB);
    unsigned long long* a_full = bars;             // [NS] bulk-copy transaction barriers
    unsigned long long* x_full = bars + NS;        // [NS] kStageThreads staging arrivals
    unsigned long long* empty = bars + 2 * NS;     // [NS] MMA commit
    unsigned long long* acc_full = bars + 3 * NS;   // [NP] MMA commit at the end of a chunk
    unsigned long long* acc_empty = acc_full + NP;  // [NP] 128 epilogue arrivals
    unsigned long long* drain = acc_full + 2 * NP;  // MMA commit before TMEM is freed
    unsigned long long* never = drain + 1;          // nothing arrives on it (failure-path test)
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(drain + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nkc = (K + kTK - 1) / kTK;
    int first_tile, tile_step, nunits, cpu, cbase;
    if (ksplit > 1) {
        const int kp = blockIdx.x % ksplit, cpp = (nkc + ksplit - 1) / ksplit;
        first_tile = blockIdx.x / ksplit;
        tile_step = 0;
        nunits = 1;
        cbase = min(nkc, kp * cpp);
        cpu = min(nkc, cbase + cpp) - cbase;
    } else {
        first_tile = blockIdx.x;
        tile_step = gridDim.x;
        nunits = first_tile < ntiles ? (ntiles - 1 - first_tile) / tile_step + 1 : 0;
        cbase = 0;
        cpu = nkc;
    }
    if (cpu <= 0) nunits = 0;
    const int total = nunits * cpu;
    const int b0 = blockIdx.y * kTB;

    if (tid == 0) {
        for (int i = 0; i < NS; ++i) {
            mbar_init(&a_full[i], 1);
            mbar_init(&x_full[i], kStageThreads);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < NP; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 128);
        }
        mbar_init(drain, 1);
        mbar_init(never, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 7) {
        tmem_alloc(tmem_slot, unsigned(tcols));
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;

    // per unit: the tile's rows [128 t, 128 t + 128) of the group and its first segment
    auto tile_of = [&](int u) { return first_tile + u * tile_step; };
    auto seg0_of = [&](int tl) { return sh.seg_rows >= kTM ? (tl * kTM) / sh.seg_rows : tl * NSEG; };

    // epilogue state that the K-split reduction below still needs: the row's running sums (v holds
    // the row's result at a unit's end) and its prefetched epilogue operand (w for DOWN, hc for H)
    float v[32];
    float pre[32];
    TcRow row{};
    bool ep_ok = true;

    if (warp == 7) {
        // ---- the warp stays converged and elects a lane for the MMAs: a branch on the lane number has the compiler
        //      move every operand into uniform registers through a loop over the active lanes (~100 clocks
        //      per MMA, 12 of them per chunk).  The bulk copies of the A planes have a warp of their own ----
        bool ok = true;
        if (g_mx_inject_timeout && nunits > 0) ok = __all_sync(0xffffffffu, tc_wait(never, 0u, abort_flag, 1000000LL));
        const uint64_t d0 = tc_desc(smem_u32(base));
        // the stages are unrolled, so that an operand's descriptor is the shared base plus a constant: computed per
        // stage, the descriptors alone took as long as the MMAs
        int c = 0, bf = 0, bf_turn = 0;
        for (int g0 = 0, turn = 0; g0 < total && ok; g0 += NS, ++turn) {
#pragma unroll
            for (int st = 0; st < NS; ++st) {
                const int gch = g0 + st;
                if (gch >= total || !ok) break;
                // the chunk's accumulator set was drained NP chunks ago
                if (bf_turn > 0) ok = tc_wait(&acc_empty[bf], unsigned(bf_turn - 1) & 1u, abort_flag);
                if (ok) ok = tc_wait(&a_full[st], unsigned(turn) & 1u, abort_flag) && tc_wait(&x_full[st], unsigned(turn) & 1u, abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                tc_fence_after();
                const uint64_t da = d0 + uint64_t(unsigned(st) * (unsigned(SB) >> 4));
                const uint64_t dx = da + uint64_t(3 * kPlaneA >> 4);
                const unsigned dhi = tmem + unsigned(bf * 3 * ncol), dlo = dhi + unsigned(ncol);
                const int kleft = K - (cbase + c) * kTK;
                const int nk = kleft >= kTK ? kTK / 16 : (kleft + 15) / 16;
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kTK / 16; ++kk) {
                        if (kk < nk) {
                            const uint64_t ko = uint64_t(2 * kk), x123 = dx + ko;
                            // the three X planes are consecutive rows of one K-major operand: [x1 | x2 | x3]
                            tc_mma(dhi, da + ko, x123, idesc3, kk > 0 ? 1u : 0u);  // D_hi = a1 x1, D_lo_a = a1 x2, D_lo_b = a1 x3
                            tc_mma(dlo, da + uint64_t(kPlaneA >> 4) + ko, x123, idesc2, 1u);      // D_lo_a += a2 x1, D_lo_b += a2 x2
                            tc_mma(dlo, da + uint64_t(2 * kPlaneA >> 4) + ko, x123, idesc1, 1u);  // D_lo_a += a3 x1
                        }
                    }
                    tc_commit(&empty[st]);
                    tc_commit(&acc_full[bf]);
                }
                __syncwarp();
                if (++c == cpu) c = 0;
                if (++bf == NP) { bf = 0; ++bf_turn; }
            }
        }
        // every MMA issued has completed before TMEM is freed
        if (elect_one()) tc_commit(drain);
        __syncwarp();
        volatile int never_set = 0;
        if (!tc_wait(drain, 0u, &never_set)) ok = false;
        if (!ok && lane == 0) atomicExch(err, 1);
    } else if (warp == 8) {
        const long long pstride = (long long)nplanes * nkc * (kTM * kTK);  // elements per plane
        // planes that several tiles read stay in L2; the others are read once per pass and go first
        const unsigned long long pol = tmap ? l2_evict_normal() : l2_evict_first();
        bool ok = true;
        int issued = 0, sl = 0;
        unsigned ph = 1;
        for (int u = 0; u < nunits && ok; ++u) {
            const int tl = tile_of(u);
            const __nv_bfloat16* src = A3 + ((long long)(tmap ? __ldg(tmap + tl) : tl) * nkc + cbase) * (kTM * kTK);
            for (int c = 0; c < cpu; ++c, src += kTM * kTK) {
                if (issued >= NS) ok = tc_wait(&empty[sl], ph, abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                if (elect_one()) {
                    unsigned char* sa = base + size_t(sl) * SB;
                    mbar_expect_tx(&a_full[sl], 3u * kPlaneA);
                    for (int p = 0; p < 3; ++p) bulk_load(sa + p * kPlaneA, src + p * pstride, kPlaneA, &a_full[sl], pol);
                }
                __syncwarp();
                ++issued;
                if (++sl == NS) { sl = 0; ph ^= 1u; }
            }
        }
        // the loads still in flight land before the shared memory goes away
        volatile int never_set = 0;
        for (int q = issued > NS ? issued - NS : 0; q < issued; ++q)
            if (!tc_wait(&a_full[q % NS], unsigned(q / NS) & 1u, &never_set)) ok = false;
        if (!ok && lane == 0) atomicExch(err, 1);
    } else if (warp >= 4) {
        // ---- warps 4-6: stage X.  FP32 request rows travel by cp.async into a ring of kXRing
        //      chunks (kXRing - 1 chunks ahead of the one being split, so no global-load latency sits
        //      on a chunk's path), then are split into bf16 planes in the swizzled K-major layout ----
        const int t = tid - 128;  // 0 .. kStageThreads-1
        float* ring = reinterpret_cast<float*>(base + size_t(NS) * SB + 256);
        constexpr int RC = NSEG * kTK * kTB;  // floats of one ring chunk: [seg][k][request]
        int st = 0;
        unsigned ph = 0;
        int staged = 0;
        bool ok = true;
        TcSeg seg[NSEG];
        bool sval[NSEG];
        int seg_unit = -1;
        auto issue = [&](int g) {
            if (g < total) {
                const int u = g / cpu, c = g - u * cpu;
                if (u != seg_unit) {
                    seg_unit = u;
                    const int gs0 = seg0_of(tile_of(u));
#pragma unroll
                    for (int j = 0; j < NSEG; ++j) {
                        sval[j] = gs0 + j < nsegs_total;
                        seg[j] = sval[j] ? tc_seg<KIND>(items, s, B, gs0 + j) : TcSeg{nullptr, nullptr, 0};
                    }
                }
                const int k0 = (cbase + c) * kTK;
                float* dst = ring + (g % kXRing) * RC;
                if constexpr (ACC != TC_SINGLE) {
                    // 16-byte pieces: 8 per row of 32 requests (B % 4 == 0: a piece is all in or all out)
#pragma unroll
                    for (int j = 0; j < NSEG; ++j)
                        for (int e = t; e < kTK * 8; e += kStageThreads) {
                            const int k = k0 + (e >> 3), p4 = (e & 7) * 4;
                            const bool in = sval[j] && k < K && b0 + p4 < B;
                            const float* src = in ? (k < seg[j].kb ? seg[j].X1 : seg[j].X2) + (long long)k * B + b0 + p4
                                                  : reinterpret_cast<const float*>(items);
                            cp_async16(dst + (j * kTK + (e >> 3)) * kTB + p4, src, in ? 16 : 0);
                        }
                } else {
#pragma unroll
                    for (int j = 0; j < NSEG; ++j)
                        for (int e = t; e < kTK * kTB; e += kStageThreads) {
                            const int k = k0 + (e >> 5), q = e & 31;
                            const bool in = sval[j] && k < K && b0 + q < B;
                            const float* src = in ? (k < seg[j].kb ? seg[j].X1 : seg[j].X2) + (long long)k * B + b0 + q
                                                  : reinterpret_cast<const float*>(items);
                            cp_async4(dst + (j * kTK + (e >> 5)) * kTB + q, src, in ? 4 : 0);
                        }
                }
            }
            cp_async_commit();  // one group per chunk (empty past the end) keeps the counting simple
        };
        for (int g = 0; g < kXRing - 1; ++g) issue(g);
        for (int g = 0; g < total && ok; ++g) {
            cp_async_wait<kXRing - 2>();                               // this thread's copies of chunk g
            asm volatile("bar.sync 1, %0;\n" ::"n"(kStageThreads) : "memory");  // everyone's
            issue(g + kXRing - 1);  // into the slot of chunk g - 1, which every thread has split
            // the stage must be free; the staging threads leave together if any of them gives up (a
            // thread left alone at the named barrier would wait forever)
            const bool free_stage = staged < NS || tc_wait(&empty[st], ph ^ 1u, abort_flag);
            if (!(ok = bar_and(2, kStageThreads, free_stage))) break;
            const float* src = ring + (g % kXRing) * RC;
            unsigned char* sx = base + size_t(st) * SB + 3 * kPlaneA;
            constexpr unsigned xp = unsigned(NSEG) * kPlaneX;
            // one 16-byte swizzle chunk (8 consecutive k) of one request per item and plane:
            // NSEG x 8 chunks x 32 requests, the ring read by consecutive requests
            for (int e = t; e < NSEG * 8 * kTB; e += kStageThreads) {
                const int n = e & 31, kg = (e >> 5) & 7, j = e >> 8;
                const float* x = src + (j * kTK + 8 * kg) * kTB + n;
                uint4 c0, c1, c2;
                split3x2(x[0], x[kTB], c0.x, c1.x, c2.x);
                split3x2(x[2 * kTB], x[3 * kTB], c0.y, c1.y, c2.y);
                split3x2(x[4 * kTB], x[5 * kTB], c0.z, c1.z, c2.z);
                split3x2(x[6 * kTB], x[7 * kTB], c0.w, c1.w, c2.w);
                const unsigned off = unsigned(j) * kPlaneX + unsigned(n) * 128u + ((unsigned(kg) ^ unsigned(n & 7)) << 4);
                *reinterpret_cast<uint4*>(sx + off) = c0;
                *reinterpret_cast<uint4*>(sx + xp + off) = c1;
                *reinterpret_cast<uint4*>(sx + 2 * xp + off) = c2;
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            mbar_arrive(&x_full[st]);
            ++staged;
            if (++st == NS) { st = 0; ph ^= 1u; }
        }
        cp_async_wait<0>();  // nothing of this thread's may land after the shared memory is gone
        if (!ok) atomicExch(err, 1);
    } else {
        // ---- warps 0-3: add every chunk's accumulators to FP32 running sums (round to nearest),
        //      run the epilogue of each unit with its operands prefetched at the unit's start ----
        const int t = tid;  // 0..127 = TMEM lane of this thread's tile row
        float rlo[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) { v[q] = 0.f; rlo[q] = 0.f; pre[q] = 0.f; }
        const int jrow = sh.seg_rows >= kTM ? 0 : t / sh.seg_rows;
        const unsigned lane_off = unsigned(warp * 32) << 16;
        for (int gch = 0; gch < total; ++gch) {
            const int u = gch / cpu;
            if (gch - u * cpu == 0) {
                const int grow = tile_of(u) * kTM + t;
                row = tc_row<KIND>(items, s, B, sh.rows_item, grow, grow < R);
                tc_prefetch<KIND, ACC>(row, B, b0, pre);
            }
            const int bf = gch % NP;
            if (!(ep_ok = tc_wait(&acc_full[bf], unsigned(gch / NP) & 1u, abort_flag))) break;
            tc_fence_after();
            const unsigned col = unsigned(bf * 3 * ncol + jrow * kTB);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float hi[16], la[16], lb[16];
                tmem_ld16(tmem + lane_off + col + unsigned(16 * hf), hi);
                tmem_ld16(tmem + lane_off + col + unsigned(ncol + 16 * hf), la);
                tmem_ld16(tmem + lane_off + col + unsigned(2 * ncol + 16 * hf), lb);
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    v[16 * hf + q] += hi[q];
                    rlo[16 * hf + q] += la[q];
                    rlo[16 * hf + q] += lb[q];
                }
            }
            tc_fence_before();
            mbar_arrive(&acc_empty[bf]);
            if ((gch + 1) % cpu != 0) continue;
            // ---- epilogue of the unit ----
#pragma unroll
            for (int q = 0; q < 32; ++q) {
                v[q] += rlo[q];
                rlo[q] = 0.f;
            }
            if (ksplit > 1) {
                // partial tiles -> rank 0 of the cluster through distributed shared memory, in rank
                // order (deterministic); the stage memory is free once every MMA has completed
                put_partial(base, v, t, 128);
                break;  // the cluster reduction and the epilogue follow below
            }
            tc_store<KIND, ACC>(row, B, b0, v, pre);
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] = 0.f;
        }
        if (!ep_ok) atomicExch(err, 1);
    }

    // ---- K split: rank 0 of the cluster adds the partial tiles and runs the epilogue ----
    if (ksplit > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        if (nunits == 0 && tid < 128) {
            // a rank without K chunks adds zeros
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] = 0.f;
            put_partial(base, v, tid, 128);
        }
        cluster.sync();
        if (cluster.block_rank() == 0 && tid < 128 && nunits > 0 && __all_sync(0xffffffffu, !*abort_flag)) {
            const int t = tid;
            for (int rk = 1; rk < ksplit; ++rk) add_partial(cluster.map_shared_rank(base, rk), v, t, 128);
            tc_store<KIND, ACC>(row, B, b0, v, pre);
        }
        cluster.sync();
    }

    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 7) tmem_dealloc(tmem, unsigned(tcols));
}

// ---- two nodes with equal operators per tile --------------------------------------------------------------
// The same sums as k_mx_umma (term for term: bit-identical results) for the two nodes of a pair of row tiles that
// share a stored tile: an A chunk (48 KB) is loaded once for both, and one MMA takes the 64 requests of both.  The
// bound is shared memory: 96 KB read by the MMAs of a chunk and 72 KB written for them, 1,340 clocks at 128 bytes
// per clock, against 1,180 for one node in k_mx_umma (measured: about 1,800 and 1,950).  Per stage 48 KB of A
// and 24 KB of X; the rows of X come straight into registers one chunk ahead (an FP32 copy in shared memory would
// cost the third stage and its bandwidth).  All node GEMMs of a block of 32 requests on a 7-level tree with
// 16 x 16 leaves, two passes: 1.65 ms by single tiles, 1.39 ms (1.32 since the epilogue exchanges pieces).
// Roles: warps 0-7 collect and write (four per node), warps 8-15 stage X, warp 16 issues the MMAs, warp 17 copies A.
constexpr int kPairThreads = 576, kPairStage = 256, kPairStages = 3, kPairSets = 2;
constexpr int kPairCols = 2 * kTB;  // right-hand side columns per plane
constexpr int kPairStageBytes = 3 * kPlaneA + 3 * 2 * kPlaneX;
constexpr size_t kPairSmem = 1024 + size_t(kPairStages) * kPairStageBytes + 256;
static_assert(kPairSmem <= 227 * 1024, "shared memory of one CTA");
static_assert(2 * kPairSmem > 228 * 1024, "one CTA per SM: each takes all of TMEM");
static_assert(kPairSets * 3 * kPairCols <= 512, "accumulator sets");

// Rows of both nodes are whole tiles (128 rows or more per segment), K is a multiple of 64.
bool pair_supported(int kind, int s) {
    const TcShape sh = tc_shape(kind, s);
    return sh.nseg == 1 && sh.K % kTK == 0;
}

// *p where `get`, else zero; a load in any case, never a branch
__device__ __forceinline__ float load_if(const float* p, bool get) {
    float x;
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n mov.f32 %0, 0f00000000;\n @p ld.global.cg.f32 %0, [%1];\n}\n"
                 : "=f"(x)
                 : "l"(p), "r"(unsigned(get))
                 : "memory");
    return x;
}

template <int KIND, TcAccess ACC>
__global__ void __launch_bounds__(kPairThreads, 1)
    k_mx_umma_pair(const __nv_bfloat16* __restrict__ A3, const MixItem* __restrict__ items, int s, int B, int cnt,
                   int ksplit, const int2* __restrict__ pairs, int npairs, const int* __restrict__ tmap, int nplanes,
                   int* __restrict__ err) {
    const TcShape sh = tc_shape(KIND, s);
    const int K = sh.K, R = cnt * sh.rows_item, nkc = K / kTK;
    constexpr int NS = kPairStages, SB = kPairStageBytes, NP = kPairSets, ncol = kPairCols;
    constexpr unsigned idesc1 = tc_idesc(kTM, ncol), idesc2 = tc_idesc(kTM, 2 * ncol), idesc3 = tc_idesc(kTM, 3 * ncol);
    extern __shared__ unsigned char tc_smem[];
    unsigned char* base = tc_smem + ((1024u - (smem_u32(tc_smem) & 1023u)) & 1023u);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(base + size_t(NS) * SB);
    unsigned long long *a_full = bars, *x_full = a_full + NS, *empty = x_full + NS, *acc_full = empty + NS,
                       *acc_empty = acc_full + NP, *drain = acc_empty + NP, *never = drain + 1;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(never + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    int first, step, nunits, cpu, cbase;
    if (ksplit > 1) {
        const int kp = blockIdx.x % ksplit, cpp = (nkc + ksplit - 1) / ksplit;
        first = blockIdx.x / ksplit;
        step = 0;
        nunits = 1;
        cbase = min(nkc, kp * cpp);
        cpu = min(nkc, cbase + cpp) - cbase;
    } else {
        first = blockIdx.x;
        step = gridDim.x;
        nunits = first < npairs ? (npairs - 1 - first) / step + 1 : 0;
        cbase = 0;
        cpu = nkc;
    }
    if (cpu <= 0) nunits = 0;
    const int total = nunits * cpu, b0 = blockIdx.y * kTB;
    if (tid == 0) {
        for (int i = 0; i < NS; ++i) {
            mbar_init(a_full + i, 1);
            mbar_init(x_full + i, kPairStage);
            mbar_init(empty + i, 1);
        }
        for (int i = 0; i < NP; ++i) {
            mbar_init(acc_full + i, 1);
            mbar_init(acc_empty + i, 256);
        }
        mbar_init(drain, 1);
        mbar_init(never, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 16) {
        tmem_alloc(tmem_slot, 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;

    float v[32];  // collecting threads: the row's sums
    bool ep_ok = true;
    if (warp == 16) {
        // converged, one elected lane issuing; stages and accumulator sets unrolled (constant descriptors).  The copies
        // have a warp of their own: issuing them here took 400 of 2,200 clocks per chunk from the MMAs.
        bool ok = true;
        if (g_mx_inject_timeout && nunits > 0) ok = __all_sync(0xffffffffu, tc_wait(never, 0u, abort_flag, 1000000LL));
        const uint64_t d0 = tc_desc(smem_u32(base));
        constexpr int UN = 6;  // a multiple of NS and NP
        static_assert(UN % NS == 0 && UN % NP == 0 && (UN / NS) % 2 == 0, "phases of the unrolled chunks");
        for (int g0 = 0, turn = 0; g0 < total && ok; g0 += UN, ++turn) {
#pragma unroll
            for (int o = 0; o < UN; ++o) {
                const int g = g0 + o;
                if (g >= total || !ok) break;
                constexpr int perset = UN / NP;  // uses of a set per turn
                const int st = o % NS, bf = o % NP;
                const unsigned ph = unsigned(o / NS) & 1u;
                if (g >= NP) ok = tc_wait(acc_empty + bf, unsigned(turn * perset + o / NP + 1) & 1u, abort_flag);
                if (ok) ok = tc_wait(a_full + st, ph, abort_flag) && tc_wait(x_full + st, ph, abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                tc_fence_after();
                const uint64_t da = d0 + uint64_t(unsigned(st) * (unsigned(SB) >> 4)), dx = da + uint64_t(3 * kPlaneA >> 4);
                const unsigned dhi = tmem + unsigned(bf * 3 * ncol), dlo = dhi + unsigned(ncol);
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kTK / 16; ++kk) {
                        const uint64_t ko = uint64_t(2 * kk), x123 = dx + ko;
                        tc_mma(dhi, da + ko, x123, idesc3, kk > 0 ? 1u : 0u);
                        tc_mma(dlo, da + uint64_t(kPlaneA >> 4) + ko, x123, idesc2, 1u);
                        tc_mma(dlo, da + uint64_t(2 * kPlaneA >> 4) + ko, x123, idesc1, 1u);
                    }
                    tc_commit(empty + st);
                    tc_commit(acc_full + bf);
                }
                __syncwarp();
            }
        }
        volatile int never_set = 0;
        if (elect_one()) tc_commit(drain);
        __syncwarp();
        if (!tc_wait(drain, 0u, &never_set)) ok = false;
        if (!ok && lane == 0) atomicExch(err, 1);
    } else if (warp == 17) {
        const long long pstride = (long long)nplanes * nkc * (kTM * kTK);
        const unsigned long long pol = l2_evict_normal();
        bool ok = true;
        int issued = 0, sl = 0;
        unsigned ph = 1;
        for (int u = 0; u < nunits && ok; ++u) {
            const __nv_bfloat16* src = A3 + ((long long)__ldg(tmap + pairs[first + u * step].x) * nkc + cbase) * (kTM * kTK);
            for (int c = 0; c < cpu; ++c, src += kTM * kTK) {
                if (issued >= NS) ok = tc_wait(empty + sl, ph, abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                if (elect_one()) {
                    unsigned char* sa = base + size_t(sl) * SB;
                    mbar_expect_tx(a_full + sl, 3u * kPlaneA);
                    for (int p = 0; p < 3; ++p) bulk_load(sa + p * kPlaneA, src + p * pstride, kPlaneA, a_full + sl, pol);
                }
                __syncwarp();
                ++issued;
                if (++sl == NS) { sl = 0; ph ^= 1u; }
            }
        }
        // the loads still in flight land before the shared memory goes away
        volatile int never_set = 0;
        for (int q = issued > NS ? issued - NS : 0; q < issued; ++q)
            if (!tc_wait(a_full + q % NS, unsigned(q / NS) & 1u, &never_set)) ok = false;
        if (!ok && lane == 0) atomicExch(err, 1);
    } else if (warp >= 8) {
        // ---- X: thread = (8 consecutive k, request) of both nodes; the next chunk's rows are loaded before this
        //      chunk's are split
        const int t = tid - 256, n = t & 31, kg = t >> 5;
        const bool in = b0 + n < B;
        float xa[2][8], xb[2][8];
        const float *p1[2], *p2[2];  // this thread's rows of the next chunk, for k < kb and from there on
        bool have[2];
        int kb = 0, lu = 0, lc = 0;  // the next chunk to load: lc of unit lu
        const long long row = (long long)B;
        auto load = [&](float (&x)[2][8]) {
            if (lc == 0 && lu < nunits) {
                const int2 pr = pairs[first + lu * step];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int tile = j ? pr.y : pr.x;
                    have[j] = tile >= 0 && in;
                    const TcSeg sg = tc_seg<KIND>(items, s, B, max(tile, 0) * kTM / sh.seg_rows);
                    const long long off = (long long)(cbase * kTK + 8 * kg) * B + b0 + (in ? n : 0);
                    p1[j] = sg.X1 + off;
                    p2[j] = sg.X2 + off;
                    kb = sg.kb;
                }
            }
            const bool one = (cbase + lc) * kTK + 8 * kg < kb;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float* p = one ? p1[j] : p2[j];
                const bool get = have[j] && lu < nunits;
#pragma unroll
                for (int i = 0; i < 8; ++i) x[j][i] = load_if(p + i * row, get);
                p1[j] += kTK * row;
                p2[j] += kTK * row;
            }
            if (++lc == cpu) { lc = 0; ++lu; }
        };
        bool ok = true;
        int st = 0;
        unsigned ph = 0;
        auto stage = [&](int g, const float (&x)[2][8]) {
            if (g >= NS && !tc_wait(empty + st, ph ^ 1u, abort_flag)) return false;
            unsigned char* sx = base + size_t(st) * SB + 3 * kPlaneA;
            constexpr unsigned xp = 2u * kPlaneX;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                uint4 c0, c1, c2;
                split3x2(x[j][0], x[j][1], c0.x, c1.x, c2.x);
                split3x2(x[j][2], x[j][3], c0.y, c1.y, c2.y);
                split3x2(x[j][4], x[j][5], c0.z, c1.z, c2.z);
                split3x2(x[j][6], x[j][7], c0.w, c1.w, c2.w);
                const unsigned off = unsigned(j) * kPlaneX + unsigned(n) * 128u + ((unsigned(kg) ^ unsigned(n & 7)) << 4);
                *reinterpret_cast<uint4*>(sx + off) = c0;
                *reinterpret_cast<uint4*>(sx + xp + off) = c1;
                *reinterpret_cast<uint4*>(sx + 2 * xp + off) = c2;
            }
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            mbar_arrive(x_full + st);
            if (++st == NS) { st = 0; ph ^= 1u; }
            return true;
        };
        if (total > 0) load(xa);
        for (int g = 0; g < total; g += 2) {
            load(xb);  // (nothing past the last chunk)
            if (!(ok = stage(g, xa)) || g + 1 >= total) break;
            load(xa);
            if (!(ok = stage(g + 1, xb))) break;
        }
        if (!ok) atomicExch(err, 1);
    } else {
        // ---- collect: warps 0-3 the first node's columns, 4-7 the second's; warp w holds rows 32 (w mod 4) ..
        const int t = tid & 127, j = tid >> 7;
        float rlo[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) { v[q] = 0.f; rlo[q] = 0.f; }
        const unsigned acc = tmem + (unsigned((warp & 3) * 32) << 16) + unsigned(j * kTB);
        int c = 0, u = 0;
        for (int g = 0; g < total; ++g) {
            const int bf = g % NP;
            if (!(ep_ok = tc_wait(acc_full + bf, unsigned(g / NP) & 1u, abort_flag))) break;
            tc_fence_after();
            const unsigned col = acc + unsigned(bf * 3 * ncol);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float x[16];
                tmem_ld16(col + unsigned(16 * hf), x);
#pragma unroll
                for (int q = 0; q < 16; ++q) v[16 * hf + q] += x[q];
                tmem_ld16(col + unsigned(ncol + 16 * hf), x);
#pragma unroll
                for (int q = 0; q < 16; ++q) rlo[16 * hf + q] += x[q];
                tmem_ld16(col + unsigned(2 * ncol + 16 * hf), x);
#pragma unroll
                for (int q = 0; q < 16; ++q) rlo[16 * hf + q] += x[q];
            }
            tc_fence_before();
            mbar_arrive(acc_empty + bf);
            if (++c < cpu) continue;
            c = 0;
#pragma unroll
            for (int q = 0; q < 32; ++q) {
                v[q] += rlo[q];
                rlo[q] = 0.f;
            }
            if (ksplit > 1) break;  // the cluster's reduction and the epilogue follow below
            const int2 pr = pairs[first + u * step];
            const int tile = j ? pr.y : pr.x, grow = tile * kTM + t;
            {
                float pre[32];
                const TcRow row = tc_row<KIND>(items, s, B, sh.rows_item, grow, tile >= 0 && grow < R);
                tc_prefetch<KIND, ACC>(row, B, b0, pre);
                tc_store<KIND, ACC>(row, B, b0, v, pre);
            }
            ++u;
#pragma unroll
            for (int q = 0; q < 32; ++q) v[q] = 0.f;
        }
        if (!ep_ok) atomicExch(err, 1);
    }

    // ---- K split: rank 0 of the cluster adds the partial tiles in rank order and runs the epilogue ----
    if (ksplit > 1) {
        cg::cluster_group cluster = cg::this_cluster();
        __syncthreads();  // every MMA has completed (drain): the stages are free
        if (tid < 256) {
            if (nunits == 0) {
#pragma unroll
                for (int q = 0; q < 32; ++q) v[q] = 0.f;
            }
            put_partial(base, v, tid, 256);
        }
        cluster.sync();
        if (cluster.block_rank() == 0 && tid < 256 && nunits > 0 && __all_sync(0xffffffffu, !*abort_flag)) {
            for (int rk = 1; rk < ksplit; ++rk) add_partial(cluster.map_shared_rank(base, rk), v, tid, 256);
            const int2 pr = pairs[first];
            const int tile = tid >> 7 ? pr.y : pr.x, grow = tile * kTM + (tid & 127);
            {
                float pre[32];
                const TcRow row = tc_row<KIND>(items, s, B, sh.rows_item, grow, tile >= 0 && grow < R);
                tc_prefetch<KIND, ACC>(row, B, b0, pre);
                tc_store<KIND, ACC>(row, B, b0, v, pre);
            }
        }
        cluster.sync();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 16) tmem_dealloc(tmem, 512u);
}

// A planes of one group: three bf16 planes with src[R][K] = plane 0 + plane 1 + plane 2, each stored
// tiled: the block of row tile t (128 rows) and K chunk c (64 columns) is 16 KB of sequential memory
// at element ((p * ntiles + t) * nkc + c) * 8192 of the group's planes, in the order of its shared-
// memory image (row r at 64 r, its 8-element groups g at 8 (g ^ (r & 7)): the 128-byte swizzle that
// the MMA's shared-memory descriptors read), so that a pipeline stage loads each plane's tile with
// one bulk copy of sequential bytes instead of 128 row pieces K columns apart.  Rows past R and
// columns past K of the last tile and chunk stay as the caller zeroed them.  H rows in the
// child-major order of tc_h_unpermute.
// `rep`: the source tile of each stored tile (null: all of them in order).
__global__ void k_tc_split(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, long long R, int K,
                           int s, int permute_h, const int* __restrict__ rep, int ntiles) {
    const long long tot = (long long)ntiles * kTM * K;
    const int nkc = (K + kTK - 1) / kTK;
    const long long pstride = (long long)ntiles * nkc * (kTM * kTK);
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot;
         e += (long long)gridDim.x * blockDim.x) {
        const long long out_row = e / K;
        const int k = int(e - out_row * K);
        const long long tile = out_row / kTM;
        const int r = int(out_row - tile * kTM), c = k / kTK, kk = k - c * kTK;
        const long long row = (rep ? rep[tile] : tile) * kTM + r;
        if (row >= R) continue;
        long long srow = row;
        if (permute_h) {
            const long long node = row / (8 * s);
            const int pr = int(row - node * 8 * s);
            srow = node * 8 * s + tc_h_unpermute(pr, s);
        }
        const long long off = (tile * nkc + c) * (kTM * kTK) + r * kTK + (((kk >> 3) ^ (r & 7)) << 3) + (kk & 7);
        __nv_bfloat16 p0, p1, p2;
        split3(src[srow * K + k], p0, p1, p2);
        dst[off] = p0;
        dst[pstride + off] = p1;
        dst[2 * pstride + off] = p2;
    }
}

// The form of the epilogue's accesses.  The exchange and its addresses are some 110 shuffles, which a launch without a
// second unit per block has nothing to hide behind; and a kernel for each form fetches less code (and spills less) than one
// with all three.  Blocks of 12 requests on trees of 16 x 16 leaves, 1 / 3 / 5 levels, us: 80 / 168 / 371 with the exchange
// throughout, 80 / 164 / 364 with rows for single units in the same kernel, 74 / 158 / 359 now; of 5 requests on 7 levels
// 1616 and 1555, of 32 3932 and 3917 (3960 without the exchange).  Pairs of nodes exchange always: without it for single
// units blocks of 64 requests on 5 levels take 736 us against 721.
TcAccess tc_access(int B, int ksplit, long long units, long long blocks) {
    return (B & 3) != 0 ? TC_SINGLE : ksplit > 1 || units <= blocks ? TC_ROWS : TC_EXCHANGED;
}

template <int KIND, int NSEG>
void launch_umma_n(cudaStream_t st, const TcPlanes& A, const MixItem* items, int cnt, int s, int B, int* err,
                   int ksplit) {
    const TcShape sh = tc_shape(KIND, s);
    const long long R = (long long)cnt * sh.rows_item;
    const int ntiles = int((R + kTM - 1) / kTM);
    const int chunks = (B + kTB - 1) / kTB;
    const size_t smem = tc_smem_bytes(NSEG);
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    unsigned gx;
    if (ksplit > 1) gx = unsigned(ntiles * ksplit);
    else gx = unsigned(std::max(1, std::min(ntiles, std::max(1, sms / chunks))));
    const TcAccess access = tc_access(B, ksplit, ntiles, gx);
    const auto kernel = access == TC_SINGLE ? k_mx_umma<KIND, NSEG, TC_SINGLE>
                        : access == TC_ROWS ? k_mx_umma<KIND, NSEG, TC_ROWS> : k_mx_umma<KIND, NSEG, TC_EXCHANGED>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(gx, unsigned(chunks));
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(ksplit);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ksplit > 1 ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, reinterpret_cast<const __nv_bfloat16*>(A.planes),
                                             items, s, B, cnt, ksplit, ntiles, A.tile, A.tile ? A.count : ntiles, err);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        throw std::runtime_error(std::string("tensor-core node GEMM launch (K split ") + std::to_string(ksplit) +
                                 "): " + cudaGetErrorString(e));
    }
    ++g_kernel_launches;
}

template <int KIND>
void launch_pair(cudaStream_t st, const TcPlanes& A, const MixItem* items, int cnt, int s, int B, int* err, int ksplit) {
    const int chunks = (B + kTB - 1) / kTB;
    const auto kernel = (B & 3) != 0 ? k_mx_umma_pair<KIND, TC_SINGLE> : k_mx_umma_pair<KIND, TC_EXCHANGED>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kPairSmem));
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(ksplit > 1 ? A.npairs * ksplit : std::max(1, std::min(A.npairs, std::max(1, sms / chunks)))),
                       unsigned(chunks));
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = kPairSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(ksplit);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ksplit > 1 ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, reinterpret_cast<const __nv_bfloat16*>(A.planes), items, s,
                                             B, cnt, ksplit, reinterpret_cast<const int2*>(A.pair), A.npairs, A.tile, A.count, err);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        throw std::runtime_error(std::string("tensor-core node GEMM launch (pairs, K split ") + std::to_string(ksplit) +
                                 "): " + cudaGetErrorString(e));
    }
    ++g_kernel_launches;
}

template <int KIND>
void launch_umma(cudaStream_t st, const TcPlanes& A, const MixItem* items, int cnt, int s, int B, int* err,
                 int ksplit) {
    const int nseg = tc_shape(KIND, s).nseg;
    if (A.pair) launch_pair<KIND>(st, A, items, cnt, s, B, err, ksplit);
    else if (nseg == 1) launch_umma_n<KIND, 1>(st, A, items, cnt, s, B, err, ksplit);
    else launch_umma_n<KIND, 2>(st, A, items, cnt, s, B, err, ksplit);
}

}  // namespace

bool mx_tc_supported(int kind, int s) {
    // s a power of two >= 16: K a multiple of 16, each right-hand-side block a power-of-two number
    // of rows of at least 64, at most two blocks per tile (the compact H of s = 16 stays on the
    // CUDA-core kernel)
    if (s < 16 || (s & (s - 1)) != 0) return false;
    const TcShape sh = tc_shape(kind, s);
    return sh.nseg <= kMaxSeg && sh.K % 16 == 0;
}

int mx_tc_max_split(int kind, int s) {
    const TcShape sh = tc_shape(kind, s);
    const int nkc = (sh.K + kTK - 1) / kTK;
    int k = 1;
    while (k < 8 && nkc / (2 * k) >= 2) k *= 2;
    return k;
}

long long mx_tc_plane_elems(int ntiles, int K) {
    return 3LL * ntiles * ((K + kTK - 1) / kTK) * (kTM * kTK);
}

void mx_tc_tiles(int kind, int s, const std::vector<int>& cls, std::vector<int>& tile, std::vector<int>& rep) {
    const int rows = tc_shape(kind, s).rows_item, cnt = int(cls.size());
    const int ntiles = int(((long long)cnt * rows + kTM - 1) / kTM);
    const int per = rows >= kTM ? 1 : kTM / rows;  // nodes of a tile (rows: a power of two)
    std::map<std::pair<int, std::vector<int>>, int> first;
    tile.clear();
    rep.clear();
    for (int t = 0; t < ntiles; ++t) {
        const int node = int((long long)t * kTM / rows), part = rows >= kTM ? t % (rows / kTM) : 0;
        std::vector<int> key;
        for (int i = 0; i < per; ++i) key.push_back(node + i < cnt ? cls[node + i] : -1);
        const auto it = first.emplace(std::make_pair(part, key), int(rep.size()));
        if (it.second) rep.push_back(t);
        tile.push_back(it.first->second);
    }
}

std::vector<int> mx_tc_pairs(int kind, int s, const std::vector<int>& tile, int stored) {
    std::vector<int> pairs;
    if (!pair_supported(kind, s)) return pairs;
    std::vector<std::vector<int>> users(stored);
    for (size_t t = 0; t < tile.size(); ++t) users[tile[t]].push_back(int(t));
    for (const auto& u : users)
        for (size_t i = 0; i < u.size(); i += 2) {
            pairs.push_back(u[i]);
            pairs.push_back(i + 1 < u.size() ? u[i + 1] : -1);
        }
    // a pair costs about what one tile does, a tile alone in its pair a little more
    if (pairs.size() / 2 * 4 > tile.size() * 3) pairs.clear();
    return pairs;
}

void mx_tc_split(cudaStream_t st, int kind, const float* src, const TcPlanes& dst, const int* rep, long long R, int K, int s) {
    const int ntiles = dst.tile ? dst.count : int((R + kTM - 1) / kTM);
    const long long tot = (long long)ntiles * kTM * K;
    const int grid = int(std::min<long long>((tot + 255) / 256, 8192));
    k_tc_split<<<grid, 256, 0, st>>>(src, reinterpret_cast<__nv_bfloat16*>(dst.planes), R, K, s, kind == MX_H ? 1 : 0,
                                     dst.tile ? rep : nullptr, ntiles);
    ++g_kernel_launches;
}

void mx_tc_set_inject_timeout(int on) {
    if (cudaMemcpyToSymbol(g_mx_inject_timeout, &on, sizeof(int)) != cudaSuccess)
        throw std::runtime_error("tensor-core GEMM: setting the failure-path test switch failed");
}

void mx_gemm_tc(cudaStream_t st, int kind, const TcPlanes& planes, const MixItem* items, int nitems, int s, int B,
                int* err, int ksplit) {
    if (!mx_tc_supported(kind, s)) throw std::invalid_argument("tensor-core node GEMM: unsupported interface size");
    if (ksplit < 1) ksplit = 1;
    if (kind == MX_W) launch_umma<MX_W>(st, planes, items, nitems, s, B, err, ksplit);
    else if (kind == MX_H) launch_umma<MX_H>(st, planes, items, nitems, s, B, err, ksplit);
    else launch_umma<MX_DOWN>(st, planes, items, nitems, s, B, err, ksplit);
}

}  // namespace efgb
