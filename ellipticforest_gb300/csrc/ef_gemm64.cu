// FP64-accurate GEMMs on the tensor cores, and the merges of the build on top of them.
//
// GB300 multiplies doubles at ~1.2 TFLOP/s (two FMA per clock and SM); its tensor cores multiply bf16 at
// ~1900.  A row of A and a column of B are therefore written as 64-bit fixed-point numbers on one scale per
// row and column, cut into eight signed base-256 digits, and the digits multiplied as bf16 integers (the
// error-free splitting of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix
// multiplication by using fast routines of matrix multiplication", Numer. Algorithms 59, 2012):
//   * digits lie in [-128, 127], so a digit is exact in bf16 and a product is an integer below 2^14;
//   * the products of digit i of A and digit j of B carry the weight 256^-(i+j).  All pairs of one weight
//     w = i + j add up in one FP32 accumulator: at most 8 pairs x 128 values of k x 2^14 = 2^24, so every
//     partial sum is an integer that FP32 holds exactly, whatever the order;
//   * pairs with w > 7 are left out: they are below 2^-62 of (row maximum) x (column maximum);
//   * after every 128 values of k the eight sums per entry go to two 64-bit integers (exact), and the entry
//     is rounded to a double once, at the end.
// An entry's error is K 2^-62 of its row maximum times its column maximum plus one rounding; a chain of
// FP64 FMAs errs by up to K 2^-53 of the sum of its |products|.
#include <cuda_bf16.h>

#include <algorithm>
#include <climits>
#include <stdexcept>
#include <string>
#include <vector>

#include "ef_gemm64.hpp"
#include "ef_kernels.cuh"
#include "ef_tcgen05.cuh"

namespace efgb {

namespace {

constexpr int kDigits = 8;
constexpr int kMT = 128, kNT = 32, kKB = 64;             // tile rows, tile columns, k per block
constexpr int kPlane = kMT * kKB * 2;                    // one digit of an A block: 16 KB
constexpr int kBBlock = kDigits * kNT * kKB * 2;         // all digits of a B block: 32 KB
constexpr int kASlots = 9, kBSlots = 2, kSets = 2;       // rings: A digits, B blocks, accumulator sets
constexpr int kFlush = 2;                                // k blocks per accumulator set (128 values of k)
constexpr int kNotFinite = 1 << 20;                      // exponent of a row that holds an infinity or NaN
constexpr int kMaxOps = 8, kMaxGemms = 4;
constexpr size_t kSmem = 1024 + size_t(kASlots) * kPlane + size_t(kBSlots) * kBBlock + 512;
static_assert(2 * kSmem > 228 * 1024, "one CTA per SM: each takes all of TMEM");

__device__ __forceinline__ double* table_ptr(const PtrTable& t, int b) {
    return *reinterpret_cast<double* const*>(static_cast<const char*>(t.p) + b * t.stride);
}

struct SplitOp {
    MatView v;
    int rows, K, role;  // role 0: rows of A; 1: columns of B (element (r, k) at k * ld + r)
    int neg0, neg1;     // sign of the part k < ks and of the rest
    unsigned char* planes;
    long long pstride;
    int* ex;
    int estride, blk0;
};
struct SplitList {
    int n;
    SplitOp op[kMaxOps];
};

// Digits of one operand: a block takes 32 rows (or columns), finds their largest magnitudes and writes the
// digits of every 64 values of k as the GEMM's shared-memory image (128-byte rows, 16-byte groups swizzled),
// zeros past the operand's ends.  Memory bound: 8 B in (twice, the second time from L2), 16 B out.
__global__ void __launch_bounds__(256) k_split64(const __grid_constant__ SplitList L) {
    int o = 0;
    while (o + 1 < L.n && int(blockIdx.x) >= L.op[o + 1].blk0) ++o;
    const SplitOp& P = L.op[o];
    const int b = blockIdx.y, r0 = (int(blockIdx.x) - P.blk0) * 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int K = P.K, nkb = (K + kKB - 1) / kKB;
    const bool cols = P.role != 0;
    const double* base = table_ptr(P.v.base, b) + P.v.off;
    const long long sr = cols ? 1 : P.v.ld, sk = cols ? P.v.ld : 1;
    __shared__ unsigned s_max[8][32];
    __shared__ uint4 stage[kDigits * 256];
    auto row_ptr = [&](int r) { return base + r * sr + (r >= P.v.rs ? P.v.dr : 0); };
    auto high_word = [&](const double* p, int k) {
        return unsigned(__double2hiint(p[k * sk + (k >= P.v.ks ? P.v.dk : 0)])) & 0x7fffffffu;
    };
    if (cols) {
        const int r = r0 + lane;
        unsigned m = 0;
        if (r < P.rows) {
            const double* p = row_ptr(r);
            int k = warp;
            for (; k + 56 < K; k += 64) {
#pragma unroll
                for (int u = 0; u < 8; ++u) m = max(m, high_word(p, k + 8 * u));
            }
            for (; k < K; k += 8) m = max(m, high_word(p, k));
        }
        s_max[warp][lane] = m;
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int w = 1; w < 8; ++w) m = max(m, s_max[w][lane]);
            s_max[0][lane] = m;
        }
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = r0 + 4 * warp + q;
            unsigned m = 0;
            if (r < P.rows) {
                const double* p = row_ptr(r);
                int k = lane;
                for (; k + 224 < K; k += 256) {
#pragma unroll
                    for (int u = 0; u < 8; ++u) m = max(m, high_word(p, k + 32 * u));
                }
                for (; k < K; k += 32) m = max(m, high_word(p, k));
            }
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) s_max[0][4 * warp + q] = m;
        }
    }
    __syncthreads();
    // rows of this thread in the second pass: columns of B by lanes (coalesced reads), rows of A by
    // groups of eight threads that each take eight consecutive k
    const int rl = cols ? lane : tid >> 3, oct = cols ? warp : tid & 7;
    const int r = r0 + rl;
    const unsigned mx = s_max[0][rl];
    const bool finite = mx < 0x7ff00000u;
    const int E = max(int(mx >> 20), 1);  // |x| < 2^(E - 1022)
    if (tid < 32 && r0 + tid < P.rows) {
        const unsigned m2 = s_max[0][tid];
        P.ex[(long long)b * P.estride + r0 + tid] = m2 < 0x7ff00000u ? max(int(m2 >> 20), 1) - 1022 : kNotFinite;
    }
    const bool live = r < P.rows && finite;
    const double* p = row_ptr(min(r, P.rows - 1));
    unsigned char* out = P.planes + (long long)b * P.pstride;
    for (int kb = 0; kb < nkb; ++kb) {
        const int k0 = kb * kKB + 8 * oct;
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = k0 + u;
            x[u] = live && k < K ? p[k * sk + (k >= P.v.ks ? P.v.dk : 0)] : 0.0;
        }
        unsigned uh[8], ul[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int hi = __double2hiint(x[u]);
            const unsigned lo = unsigned(__double2loint(x[u]));
            const int ex = (hi >> 20) & 0x7ff;
            long long m = (long long)(((unsigned long long)((hi & 0xfffff) | (ex ? 0x100000 : 0)) << 32) | lo);
            const int sh = 9 - (E - max(ex, 1));  // x 2^(62 - exponent of the row)
            if (sh >= 0) m <<= sh;
            else m = sh < -54 ? 0 : (m + (1LL << (-sh - 1))) >> -sh;
            const bool neg = (hi < 0) != ((k0 + u < P.v.ks ? P.neg0 : P.neg1) != 0);
            if (neg) m = -m;
            // balanced digits: adding 128 to every byte below the top one turns byte - 128 into the digit;
            // the top byte is signed already, and its flipped sign bit brings it to the same form
            const unsigned long long v = (unsigned long long)(m + 0x0080808080808080LL) ^ 0x8000000000000000ULL;
            uh[u] = unsigned(v >> 32);
            ul[u] = unsigned(v);
        }
        // digit as bf16: the byte in the last bits of 2^23, minus 2^23 + 128, has its digits in the high half
        auto word = [&](const unsigned (&w)[8], int u, int byte) {
            const unsigned sel = 0x7440u | unsigned(byte);
            const float f0 = __uint_as_float(__byte_perm(w[u], 0x4B000000u, sel)) - 8388736.0f;
            const float f1 = __uint_as_float(__byte_perm(w[u + 1], 0x4B000000u, sel)) - 8388736.0f;
            return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
        };
        const unsigned at = unsigned(rl) * 128u + ((unsigned(oct) ^ unsigned(rl & 7)) << 4);
#pragma unroll
        for (int i = 0; i < kDigits; ++i) {
            const unsigned (&w)[8] = i < 4 ? uh : ul;
            const int byte = 3 - (i & 3);
            const uint4 d = make_uint4(word(w, 0, byte), word(w, 2, byte), word(w, 4, byte), word(w, 6, byte));
            if (cols) {
                stage[i * 256 + (at >> 4)] = d;
            } else {
                const long long blk = ((long long)(r0 / kMT) * nkb + kb) * kDigits + i;
                *reinterpret_cast<uint4*>(out + blk * kPlane + (r0 % kMT) * 128 + at) = d;
            }
        }
        if (cols) {
            // lanes hold columns, so their 16-byte groups lie 128 bytes apart: through shared memory
            __syncthreads();
            uint4* dst = reinterpret_cast<uint4*>(out + ((long long)(r0 / kNT) * nkb + kb) * kBBlock);
#pragma unroll
            for (int i = 0; i < kDigits; ++i) dst[i * 256 + tid] = stage[i * 256 + tid];
            __syncthreads();
        }
    }
}

struct GemmOp {
    const unsigned char *A, *B;
    long long astride, bstride;
    const int *ea, *eb;
    int eastride, ebstride;
    int M, N, K;
    MatView c;  // C; rows >= c.rs shifted by c.dr, columns >= c.ks by c.dk
    int neg, add;  // C = (add ? C : 0) + (neg ? -1 : 1) A B
    int mt, nt, tile0;
};
struct GemmList {
    int n, tiles;
    GemmOp op[kMaxGemms];
};

struct TileAt {
    int o, b, m, n;
};
// tile t: operands one after another, their batch items, and inside one product bands of eight tile rows
// walked column by column, so that the tiles in flight share their A and B blocks in L2
__device__ __forceinline__ TileAt tile_at(const GemmList& L, int t) {
    TileAt r;
    r.o = 0;
    while (r.o + 1 < L.n && t >= L.op[r.o + 1].tile0) ++r.o;
    const GemmOp& g = L.op[r.o];
    int i = t - g.tile0;
    const int per = g.mt * g.nt;
    r.b = i / per;
    i -= r.b * per;
    const int band = i / (8 * g.nt), rows = min(8, g.mt - 8 * band);
    i -= band * 8 * g.nt;
    r.n = i / rows;
    r.m = 8 * band + i - r.n * rows;
    return r;
}

// C tile of 128 x 32 per step, one CTA per SM walking over the tiles.  Warp 4 copies digit blocks (one bulk
// copy each, the layout is the shared-memory image), warp 5 issues the MMAs, warps 0-3 collect.  For every
// 16 values of k one MMA per digit i of A multiplies it with digits 0 .. 7 - i of B, which are consecutive
// rows of one K-major operand, into the consecutive accumulators of weights i .. 7: N = 32 (8 - i), so a
// digit of A is read from shared memory once.  Two accumulator sets of 256 TMEM columns alternate, so the
// collecting of 128 values of k (8 sums per entry: convert, multiply-add into 64 bits) hides behind the
// MMAs of the next.  Bound: the 160 KB of digits per 64 values of k (2304 MMA clocks) from L2.
__global__ void __launch_bounds__(192, 1) k_gemm64(const __grid_constant__ GemmList L, int* __restrict__ err) {
    extern __shared__ unsigned char g_smem[];
    unsigned char* base = g_smem + ((1024u - (smem_u32(g_smem) & 1023u)) & 1023u);
    unsigned char* bbase = base + size_t(kASlots) * kPlane;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(bbase + size_t(kBSlots) * kBBlock);
    unsigned long long *a_full = bars, *a_empty = a_full + kASlots, *b_full = a_empty + kASlots,
                       *b_empty = b_full + kBSlots, *acc_full = b_empty + kBSlots, *acc_empty = acc_full + kSets,
                       *drain = acc_empty + kSets;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < kASlots; ++i) { mbar_init(a_full + i, 1); mbar_init(a_empty + i, 1); }
        for (int i = 0; i < kBSlots; ++i) { mbar_init(b_full + i, 1); mbar_init(b_empty + i, 1); }
        for (int i = 0; i < kSets; ++i) { mbar_init(acc_full + i, 1); mbar_init(acc_empty + i, 128); }
        mbar_init(drain, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 5) {
        tmem_alloc(tmem_slot, 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;

    if (warp == 4) {
        if (lane == 0) {
            unsigned na = 0, nb = 0;  // copies issued into either ring
            bool ok = true;
            for (int t = blockIdx.x; t < L.tiles && ok; t += gridDim.x) {
                const TileAt at = tile_at(L, t);
                const GemmOp& g = L.op[at.o];
                const int nkb = (g.K + kKB - 1) / kKB;
                const unsigned char* A = g.A + at.b * g.astride + (long long)at.m * nkb * (kDigits * kPlane);
                const unsigned char* B = g.B + at.b * g.bstride + (long long)at.n * nkb * kBBlock;
                for (int kb = 0; kb < nkb && ok; ++kb) {
                    const unsigned sb = nb % kBSlots;
                    if (nb >= kBSlots) ok = tc_wait(b_empty + sb, (nb / kBSlots - 1) & 1u, abort_flag);
                    if (!ok) break;
                    mbar_expect_tx(b_full + sb, kBBlock);
                    bulk_copy(bbase + size_t(sb) * kBBlock, B + (long long)kb * kBBlock, kBBlock, b_full + sb);
                    ++nb;
                    for (int i = 0; i < kDigits; ++i) {
                        const unsigned sa = na % kASlots;
                        if (na >= kASlots) ok = tc_wait(a_empty + sa, (na / kASlots - 1) & 1u, abort_flag);
                        if (!ok) break;
                        mbar_expect_tx(a_full + sa, kPlane);
                        bulk_copy(base + size_t(sa) * kPlane, A + ((long long)kb * kDigits + i) * kPlane, kPlane, a_full + sa);
                        ++na;
                    }
                }
            }
            if (!ok) {
                // let the copies still in flight land before the shared memory goes away
                volatile int never_set = 0;
                for (unsigned q = na > kASlots ? na - kASlots : 0; q < na; ++q)
                    (void)tc_wait(a_full + q % kASlots, (q / kASlots) & 1u, &never_set);
                for (unsigned q = nb > kBSlots ? nb - kBSlots : 0; q < nb; ++q)
                    (void)tc_wait(b_full + q % kBSlots, (q / kBSlots) & 1u, &never_set);
                atomicExch(err, 1);
            }
        }
    } else if (warp == 5) {
        if (lane == 0) {
            unsigned na = 0, nb = 0, ns = 0;
            bool ok = true;
            const uint32_t a0 = smem_u32(base), b0 = smem_u32(bbase);
            for (int t = blockIdx.x; t < L.tiles && ok; t += gridDim.x) {
                const GemmOp& g = L.op[tile_at(L, t).o];
                const int nkb = (g.K + kKB - 1) / kKB;
                for (int kb = 0; kb < nkb && ok; ++kb) {
                    const unsigned set = ns % kSets;
                    if (kb % kFlush == 0 && ns >= kSets) ok = tc_wait(acc_empty + set, (ns / kSets - 1) & 1u, abort_flag);
                    const unsigned sb = nb % kBSlots;
                    if (ok) ok = tc_wait(b_full + sb, (nb / kBSlots) & 1u, abort_flag);
                    const int steps = min(4, (g.K - kb * kKB + 15) / 16);
                    for (int i = 0; i < kDigits && ok; ++i) {
                        const unsigned sa = na % kASlots;
                        ok = tc_wait(a_full + sa, (na / kASlots) & 1u, abort_flag);
                        if (!ok) break;
                        tc_fence_after();
                        const unsigned d = tmem + set * 256u + unsigned(i * kNT);
                        const unsigned idesc = tc_idesc(kMT, kNT * (kDigits - i));
                        for (int kk = 0; kk < steps; ++kk)
                            tc_mma(d, tc_desc(a0 + sa * kPlane + kk * 32u), tc_desc(b0 + sb * kBBlock + kk * 32u), idesc,
                                   kb % kFlush == 0 && i == 0 && kk == 0 ? 0u : 1u);
                        tc_commit(a_empty + sa);
                        ++na;
                    }
                    if (!ok) break;
                    tc_commit(b_empty + sb);
                    ++nb;
                    if (kb % kFlush == kFlush - 1 || kb == nkb - 1) {
                        tc_commit(acc_full + set);
                        ++ns;
                    }
                }
            }
            // every MMA issued has completed before TMEM is freed
            tc_commit(drain);
            volatile int never_set = 0;
            if (!tc_wait(drain, 0u, &never_set)) ok = false;
            if (!ok) atomicExch(err, 1);
        }
    } else {
        const unsigned lane_off = unsigned(warp * 32) << 16;
        unsigned ns = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < L.tiles && ok; t += gridDim.x) {
            const TileAt at = tile_at(L, t);
            const GemmOp& g = L.op[at.o];
            const int nkb = (g.K + kKB - 1) / kKB, flushes = (nkb + kFlush - 1) / kFlush;
            long long hi[kNT], lo[kNT];
#pragma unroll
            for (int c = 0; c < kNT; ++c) { hi[c] = 0; lo[c] = 0; }
            for (int f = 0; f < flushes; ++f, ++ns) {
                const unsigned set = ns % kSets;
                if (!(ok = tc_wait(acc_full + set, (ns / kSets) & 1u, abort_flag))) break;
                tc_fence_after();
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int w = 0; w < kDigits; ++w) {
                        float v[16];
                        tmem_ld16(tmem + lane_off + set * 256u + unsigned(w * kNT + 16 * half), v);
#pragma unroll
                        for (int c = 0; c < 16; ++c) {
                            const long long q = (long long)__float2int_rn(v[c]) * (1LL << (8 * (3 - (w & 3))));
                            if (w < 4) hi[16 * half + c] += q;
                            else lo[16 * half + c] += q;
                        }
                    }
                tc_fence_before();
                mbar_arrive(acc_empty + set);
            }
            if (!ok) break;
            const int row = at.m * kMT + tid, n0 = at.n * kNT;
            if (row >= g.M) continue;
            double* C = table_ptr(g.c.base, at.b) + g.c.off + (long long)row * g.c.ld + (row >= g.c.rs ? g.c.dr : 0);
            const int ea = g.ea[(long long)at.b * g.eastride + row];
            const int* eb = g.eb + (long long)at.b * g.ebstride + n0;
#pragma unroll
            for (int c = 0; c < kNT; ++c) {
                if (n0 + c >= g.N) break;
                // (hi + lo 2^-32) 2^(ea + eb - 36): the carry of lo first, then both parts as doubles by their
                // bits (1.5 2^52 + integer, 2^20 + fraction), one rounding in the last addition
                const long long h = hi[c] + (lo[c] >> 32);
                const double d1 = __longlong_as_double(0x4338000000000000LL + h);
                const double d2 = __hiloint2double(0x41300000, int(unsigned(lo[c])));
                double v = (d1 - (6755399441055744.0 + 1048576.0)) + d2;
                const int e1 = eb[c], k = ea + e1 - 36;
                const int hw = __double2hiint(v), e = (hw >> 20) & 0x7ff;
                if (e != 0) {
                    if (e + k >= 1 && e + k <= 2046) v = __hiloint2double(hw + (k << 20), __double2loint(v));
                    else v = scalbn(v, k);
                }
                if (ea >= kNotFinite || e1 >= kNotFinite) v = __longlong_as_double(0x7ff8000000000000LL);
                if (g.neg) v = -v;
                double* dst = C + n0 + c + (n0 + c >= g.c.ks ? g.c.dk : 0);
                *dst = g.add ? *dst + v : v;
            }
        }
        if (!ok) atomicExch(err, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 5) tmem_dealloc(tmem, 512u);
}

// In-place inverse of one matrix of at most 64 rows per block by Gauss-Jordan steps (row k of the result
// from the pivot row of step k): 256 threads hold 4 x 4 entries each.  The pivot of column k is the largest
// entry of the rows not used yet, compared by its leading 26 bits (the row's number in the last six, so one
// warp reduction finds both); rows are not moved but put in order when they are written.  Bound by the SM's
// two FP64 multiply-adds per clock (n^3 of them: ~65 us for 64 rows).  A pivot that is zero or not finite
// sets info.
struct InvList {
    int nv;
    MatView v[2];
};
__global__ void __launch_bounds__(256) k_inv64(const __grid_constant__ InvList L, int n, int* __restrict__ info) {
    const MatView& V = L.v[blockIdx.x];
    double* A = table_ptr(V.base, blockIdx.y) + V.off;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, lane = tid & 31;
    __shared__ double s_col[2][64], s_row[2][64];
    __shared__ int s_p[64], s_k[64];
    double a[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = 4 * ty + i, c = 4 * tx + j;
            a[i][j] = r < n && c < n ? A[(long long)r * V.ld + c] : (r == c ? 1.0 : 0.0);
        }
    unsigned used0 = 0, used1 = 0;
    bool bad = false;
    for (int k = 0; k < n; ++k) {
        const int bf = k & 1;
        if (tx == (k >> 2)) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j == (k & 3)) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) s_col[bf][4 * ty + i] = a[i][j];
                }
        }
        __syncthreads();
        const unsigned h0 = unsigned(__double2hiint(s_col[bf][lane])) & 0x7fffffffu;
        const unsigned h1 = unsigned(__double2hiint(s_col[bf][lane + 32])) & 0x7fffffffu;
        const unsigned k0 = (used0 >> lane) & 1u || lane >= n ? 0u : ((h0 << 1) & ~63u) | unsigned(63 - lane);
        const unsigned k1 = (used1 >> lane) & 1u || lane + 32 >= n ? 0u : ((h1 << 1) & ~63u) | unsigned(31 - lane);
        const unsigned best = __reduce_max_sync(0xffffffffu, max(k0, k1));
        const int p = 63 - int(best & 63u);
        const double piv = s_col[bf][p];
        if (!(fabs(piv) > 0.0) || best >= 0xffe00000u) bad = true;
        if (p < 32) used0 |= 1u << p;
        else used1 |= 1u << (p - 32);
        if (ty == (p >> 2)) {
            const double inv = 1.0 / piv;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i == (p & 3)) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) s_row[bf][4 * tx + j] = 4 * tx + j == k ? inv : a[i][j] * inv;
                }
        }
        if (tid == 0) { s_p[k] = p; s_k[p] = k; }
        __syncthreads();
        double rj[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) rj[j] = s_row[bf][4 * tx + j];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 4 * ty + i;
            const double c = s_col[bf][r];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool kc = 4 * tx + j == k;
                a[i][j] = r == p ? rj[j] : fma(-c, rj[j], kc ? 0.0 : a[i][j]);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = 4 * ty + i, c = 4 * tx + j;
            if (r < n && c < n) A[(long long)s_k[r] * V.ld + s_p[c]] = a[i][j];
        }
    if (tid == 0 && bad) info[blockIdx.y] = 1;
}

// X^{-1} from the X buffer to its place behind S in the RHS buffer (columns [8s, 12s))
__global__ void k_place_inverse(const MergeItem* __restrict__ items, int s) {
    const MergeItem& it = items[blockIdx.y];
    const int m = 4 * s, half = m / 2;
    const long long tot = (long long)m * half;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < tot; e += (long long)gridDim.x * blockDim.x) {
        const int r = int(e / half), c = int(e - (long long)r * half);
        reinterpret_cast<double2*>(it.RHS + (long long)r * 3 * m + 2 * m)[c] = reinterpret_cast<const double2*>(it.X)[e];
    }
}

__device__ __forceinline__ double check_entry(int i) { return (unsigned(i) * 2654435761u) >> 31 ? 1.0 : -1.0; }

// y = X^{-1} v for a vector v of +-1, into w (free during a build); one warp per row
__global__ void __launch_bounds__(256) k_check_y(const MergeItem* __restrict__ items, int s) {
    const MergeItem& it = items[blockIdx.y];
    const int m = 4 * s, r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= m) return;
    double acc = 0.0;
    for (int k = lane; k < m; k += 32) acc = fma(it.X[(long long)r * m + k], check_entry(k), acc);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) it.w[r] = acc;
}
// |v - X y| <= 1e-12 (|v| + |X| |y|) for every row, X read from the children's T as it was gathered:
// block elimination without row exchanges between blocks is accepted only where its residual is that of
// an elimination with them (~1e-15); info is set otherwise
__global__ void __launch_bounds__(256) k_check_r(const MergeItem* __restrict__ items, int s, int* __restrict__ info) {
    const MergeItem& it = items[blockIdx.y];
    const int m = 4 * s, r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= m) return;
    const int I = r / s, o = r - I * s;
    const int lower[4] = {0, 1, 0, 2}, upper[4] = {2, 3, 1, 3};
    double acc = 0.0, mag = 0.0;
#pragma unroll
    for (int up = 0; up < 2; ++up) {
        const int c = up ? upper[I] : lower[I];
        const double* row = it.Tc[c] + (long long)((up ? (I < 2 ? 2 * s : 0) : (I < 2 ? 3 * s : s)) + o) * m;
        const int Js[2] = {c & 1, c < 2 ? 2 : 3};  // alpha: I0, I2; beta: I1, I2; gamma: I0, I3; omega: I1, I3
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int J = Js[j];
            const bool low = lower[J] == c;
            const double* t = row + (low ? (J < 2 ? 3 * s : s) : (J < 2 ? 2 * s : 0));
            const double* y = it.w + J * s;
            for (int k = lane; k < s; k += 32) {
                const double p = t[k] * y[k];
                acc += up ? -p : p;
                mag += fabs(p);
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        acc += __shfl_xor_sync(0xffffffffu, acc, off);
        mag += __shfl_xor_sync(0xffffffffu, mag, off);
    }
    if (lane == 0 && !(fabs(check_entry(r) - acc) <= 1e-12 * (1.0 + mag))) info[blockIdx.y] = 1;
}

int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(1, sms);
}

// The operands and products of one merge step, launched together: digits first, then the products.  With
// `dry` nothing runs and only the workspace is added up.
class Runner {
public:
    Runner(cudaStream_t st, char* ws, int* err, int cnt, bool dry) : st_(st), ws_(ws), err_(err), cnt_(cnt), dry_(dry) {}
    size_t mark() const { return off_; }
    void release(size_t m) { off_ = m; }
    size_t peak() const { return peak_; }
    bool dry() const { return dry_; }
    int count() const { return cnt_; }
    cudaStream_t stream() const { return st_; }

    struct Digits {
        unsigned char* planes;
        long long pstride;
        int* ex;
        int estride, len, K;
    };
    // role 0: rows of A (len = M); 1: columns of B (len = N)
    Digits split(const MatView& v, int len, int K, int role, int neg0 = 0, int neg1 = 0) {
        const int nkb = (K + kKB - 1) / kKB;
        Digits d;
        d.pstride = role ? (long long)((len + kNT - 1) / kNT) * nkb * kBBlock
                         : (long long)((len + kMT - 1) / kMT) * nkb * kDigits * kPlane;
        d.estride = len;
        d.len = len;
        d.K = K;
        d.planes = reinterpret_cast<unsigned char*>(take(size_t(d.pstride) * cnt_));
        d.ex = reinterpret_cast<int*>(take(size_t(len) * 4 * cnt_));
        if (sl_.n == kMaxOps) flush_split();
        SplitOp& op = sl_.op[sl_.n];
        op = SplitOp{v, len, K, role, neg0, neg1, d.planes, d.pstride, d.ex, d.estride, blocks_};
        // whole tiles: the rows past the end are written as zeros
        blocks_ += role ? (len + kNT - 1) / kNT : (len + kMT - 1) / kMT * (kMT / 32);
        ++sl_.n;
        return d;
    }
    void gemm(const Digits& a, const Digits& b, const MatView& c, bool neg, bool add) {
        if (gl_.n == kMaxGemms) flush();
        GemmOp& g = gl_.op[gl_.n];
        const int mt = (a.len + kMT - 1) / kMT, nt = (b.len + kNT - 1) / kNT;
        g = GemmOp{a.planes, b.planes, a.pstride, b.pstride, a.ex, b.ex, a.estride, b.estride, a.len, b.len, a.K,
                   c, neg, add, mt, nt, gl_.tiles};
        gl_.tiles += mt * nt * cnt_;
        ++gl_.n;
    }
    void flush_split() {
        if (sl_.n && !dry_) {
            k_split64<<<dim3(unsigned(blocks_), unsigned(cnt_)), 256, 0, st_>>>(sl_);
            ++g_kernel_launches;
        }
        sl_.n = 0;
        blocks_ = 0;
    }
    void flush() {
        flush_split();
        if (gl_.n && !dry_) {
            cudaFuncSetAttribute(k_gemm64, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem));
            k_gemm64<<<unsigned(std::min(gl_.tiles, sm_count())), 192, kSmem, st_>>>(gl_, err_);
            ++g_kernel_launches;
        }
        gl_.n = 0;
        gl_.tiles = 0;
    }

private:
    char* take(size_t bytes) {
        char* p = ws_ + off_;
        off_ += (bytes + 1023) / 1024 * 1024;
        peak_ = std::max(peak_, off_);
        return p;
    }
    cudaStream_t st_;
    char* ws_;
    int* err_;
    int cnt_;
    bool dry_;
    size_t off_ = 0, peak_ = 0;
    int blocks_ = 0;
    SplitList sl_{};
    GemmList gl_{};
};

MatView at(const MatView& v, long long r, long long c) {
    MatView o = v;
    o.off += r * v.ld + c;
    return o;
}

// Inverses of one or two h x h matrices per item, in place, by 2 x 2 block elimination:
//   [A B; C D]: G = A^-1 B, F = C A^-1, D <- (D - C G)^-1, B <- -G D, C <- -D F, A <- A^-1 - B F.
// Every product is an accurate GEMM, so the only FP64 roundings are those of the stored blocks.  tmp: room
// for G and F of all views and of the blocks below, h^2 doubles per view.
void invert(Runner& R, const std::vector<MatView>& v, int h, const MatView& tmp, int* info) {
    if (h <= 64) {
        if (!R.dry()) {
            InvList L{};
            L.nv = int(v.size());
            for (size_t i = 0; i < v.size(); ++i) L.v[i] = v[i];
            k_inv64<<<dim3(unsigned(v.size()), unsigned(R.count())), 256, 0, R.stream()>>>(L, h, info);
            ++g_kernel_launches;
        }
        return;
    }
    const int h1 = (h / 2 + 31) / 32 * 32, h2 = h - h1;
    const size_t n = v.size(), m0 = R.mark();
    std::vector<MatView> A, B, C, D, G, F;
    MatView below = tmp;
    for (const auto& x : v) {
        A.push_back(x);
        B.push_back(at(x, 0, h1));
        C.push_back(at(x, h1, 0));
        D.push_back(at(x, h1, h1));
        MatView g = below, f = below;
        g.ld = h2;
        f.off += (long long)h1 * h2;
        f.ld = h1;
        G.push_back(g);
        F.push_back(f);
        below.off += 2LL * h1 * h2;
    }
    invert(R, A, h1, below, info);
    std::vector<Runner::Digits> c0;
    for (size_t i = 0; i < n; ++i) {
        const auto aA = R.split(A[i], h1, h1, 0), aB = R.split(A[i], h1, h1, 1), bB = R.split(B[i], h2, h1, 1);
        c0.push_back(R.split(C[i], h2, h1, 0));
        R.gemm(aA, bB, G[i], false, false);
        R.gemm(c0[i], aB, F[i], false, false);
    }
    R.flush();
    for (size_t i = 0; i < n; ++i) R.gemm(c0[i], R.split(G[i], h2, h1, 1), D[i], true, true);
    R.flush();
    R.release(m0);
    invert(R, D, h2, below, info);
    std::vector<Runner::Digits> f0;
    for (size_t i = 0; i < n; ++i) {
        const auto dA = R.split(D[i], h2, h2, 0), dB = R.split(D[i], h2, h2, 1), gA = R.split(G[i], h1, h2, 0);
        f0.push_back(R.split(F[i], h1, h2, 1));
        R.gemm(gA, dB, B[i], true, false);
        R.gemm(dA, f0[i], C[i], true, false);
    }
    R.flush();
    for (size_t i = 0; i < n; ++i) R.gemm(R.split(B[i], h1, h2, 0), f0[i], A[i], true, true);
    R.flush();
    R.release(m0);
}

PtrTable field(const MergeItem* items, const void* member_of_first) {
    return PtrTable{reinterpret_cast<const char*>(items) + (static_cast<const char*>(member_of_first) -
                                                            reinterpret_cast<const char*>(items)),
                    (long long)sizeof(MergeItem)};
}

// Merge of `R.count()` nodes from `items` on, X, H and T_LHS gathered: X <- X^{-1}, S, T (the steps of
// HPSAlgorithm.hpp:752-993).  X couples the interfaces I0, I1 only through I2, I3 (and the other way round),
// so its leading 2s x 2s block is block diagonal and the first elimination step runs on two s x s blocks at
// once.  kids: children whose products of S and T are launched together.
void merge_steps(Runner& R, const MergeItem* items, int s, int kids, int* info) {
    const int m = 4 * s;
    const MergeItem* z = items;
    const MatView X{field(z, &z->X), 0, m}, S{field(z, &z->RHS), 0, 3 * m}, H{field(z, &z->H), 0, 2 * s},
        T{field(z, &z->T), 0, 2 * m};
    // ---- X^{-1}
    const MatView A0 = X, A1 = at(X, s, s), B0 = at(X, 0, 2 * s), B1 = at(X, s, 2 * s), C0 = at(X, 2 * s, 0),
                  C1 = at(X, 2 * s, s), D = at(X, 2 * s, 2 * s);
    MatView G = S, F = S, below = S;  // the RHS buffer is free until S is written
    G.ld = 2 * s;
    F.ld = 2 * s;
    F.off = 4LL * s * s;
    below.off = 8LL * s * s;
    invert(R, {A0, A1}, s, below, info);
    {
        const auto a0 = R.split(A0, s, s, 0), a0b = R.split(A0, s, s, 1), a1 = R.split(A1, s, s, 0),
                   a1b = R.split(A1, s, s, 1), b0 = R.split(B0, 2 * s, s, 1), b1 = R.split(B1, 2 * s, s, 1),
                   c0 = R.split(C0, 2 * s, s, 0), c1 = R.split(C1, 2 * s, s, 0);
        R.gemm(a0, b0, G, false, false);
        R.gemm(a1, b1, at(G, s, 0), false, false);
        R.gemm(c0, a0b, F, false, false);
        R.gemm(c1, a1b, at(F, 0, s), false, false);
        R.flush();
        R.release(0);
        const auto c = R.split(C0, 2 * s, 2 * s, 0), g = R.split(G, 2 * s, 2 * s, 1);
        R.gemm(c, g, D, true, true);
        R.flush();
        R.release(0);
    }
    invert(R, {D}, 2 * s, below, info);
    {
        const auto dA = R.split(D, 2 * s, 2 * s, 0), dB = R.split(D, 2 * s, 2 * s, 1), g = R.split(G, 2 * s, 2 * s, 0),
                   f = R.split(F, 2 * s, 2 * s, 1);
        R.gemm(g, dB, B0, true, false);
        R.gemm(dA, f, C0, true, false);
        R.flush();
        R.gemm(R.split(B0, 2 * s, 2 * s, 0), f, A0, true, true);
        R.flush();
        R.release(0);
    }
    if (!R.dry()) {
        const dim3 rows(unsigned((m + 7) / 8), unsigned(R.count()));
        k_check_y<<<rows, 256, 0, R.stream()>>>(items, s);
        k_check_r<<<rows, 256, 0, R.stream()>>>(items, s, info);
        g_kernel_launches += 2;
    }
    // ---- S = X^{-1} S_RHS: the columns of child c's exterior sides have entries on c's two interfaces only
    // child: interfaces Ia, Ib (c's sides qa, qb), sign of S_RHS there, c's exterior sides and their runs of s
    // columns in the parent's WESN order
    struct Kid {
        int Ia, Ib, qa, qb, nega, negb, e0, e1, p0, p1;
    };
    static const Kid kid[4] = {
        {0, 2, 3, 1, 1, 1, 0, 2, 0, 4},  // alpha: lower on I0 (its N side) and I2 (E); exterior W, S
        {1, 2, 3, 0, 1, 0, 1, 2, 2, 5},  // beta: lower on I1 (N), upper on I2 (W); exterior E, S
        {0, 3, 2, 1, 0, 1, 0, 3, 1, 6},  // gamma: upper on I0 (S), lower on I3 (E); exterior W, N
        {1, 3, 2, 0, 0, 0, 1, 3, 3, 7},  // omega: upper on I1 (S) and I3 (W); exterior E, N
    };
    for (int c0 = 0; c0 < 4; c0 += kids) {
        for (int c = c0; c < c0 + kids; ++c) {
            const Kid& q = kid[c];
            MatView x = at(X, 0, (long long)q.Ia * s);
            x.ks = s;
            x.dk = (long long)(q.Ib - q.Ia - 1) * s;
            MatView t{field(z, &z->Tc[c]), (long long)q.qa * s * m + (long long)q.e0 * s, m};
            t.ks = s;
            t.dk = (long long)(q.qb - q.qa - 1) * s * m;
            t.rs = s;
            t.dr = (long long)(q.e1 - q.e0 - 1) * s;
            MatView o = at(S, 0, (long long)q.p0 * s);
            o.ks = s;
            o.dk = (long long)(q.p1 - q.p0 - 1) * s;
            const auto xa = R.split(x, m, 2 * s, 0), tb = R.split(t, 2 * s, 2 * s, 1, q.nega, q.negb);
            R.gemm(xa, tb, o, false, false);
        }
        R.flush();
        R.release(0);
    }
    if (!R.dry()) {
        const long long tot = 8LL * s * s;
        k_place_inverse<<<dim3(unsigned(std::min(2048LL, (tot + 255) / 256)), unsigned(R.count())), 256, 0, R.stream()>>>(items, s);
        ++g_kernel_launches;
    }
    // ---- T += H S: the exterior rows of child c take the S rows of its two interfaces
    for (int c0 = 0; c0 < 4; c0 += kids) {
        for (int c = c0; c < c0 + kids; ++c) {
            const Kid& q = kid[c];
            MatView h = at(H, (long long)q.p0 * s, 0);
            h.rs = s;
            h.dr = (long long)(q.p1 - q.p0 - 1) * s * 2 * s;
            MatView b = at(S, (long long)q.Ia * s, 0);
            b.ks = s;
            b.dk = (long long)(q.Ib - q.Ia - 1) * s * 3 * m;
            MatView o = at(T, (long long)q.p0 * s, 0);
            o.rs = s;
            o.dr = (long long)(q.p1 - q.p0 - 1) * s * 2 * m;
            R.gemm(R.split(h, 2 * s, 2 * s, 0), R.split(b, 2 * m, 2 * s, 1), o, false, true);
        }
        R.flush();
        R.release(0);
    }
}

// workspace of one item's merge with `kids` children at once
size_t item_bytes(int s, int kids, int cnt) {
    Runner R(nullptr, nullptr, nullptr, cnt, true);
    merge_steps(R, nullptr, s, kids, nullptr);
    return R.peak();
}

// most workspace a merge level takes before it is run in parts
constexpr size_t kMaxWorkspace = size_t(512) << 20;

struct Parts {
    int kids, items;
    size_t bytes;
};
Parts merge_parts(int cnt, int s) {
    Parts p{4, cnt, 0};
    if (item_bytes(s, 4, 1) > kMaxWorkspace) p.kids = 1;
    const size_t one = item_bytes(s, p.kids, 1);
    p.items = int(std::max<size_t>(1, std::min<size_t>(size_t(std::min(cnt, 65535)), kMaxWorkspace / one)));
    p.bytes = item_bytes(s, p.kids, p.items);
    return p;
}

}  // namespace

bool merge64_supported(int s) { return s >= 8 && s % 2 == 0 && 16LL * s <= 65536; }

size_t merge64_workspace(int cnt, int s) { return merge_parts(cnt, s).bytes; }

void merge64(cudaStream_t st, const MergeItem* items, int cnt, int s, int* info, char* ws, int* err) {
    const Parts p = merge_parts(cnt, s);
    for (int i = 0; i < cnt; i += p.items) {
        Runner R(st, ws, err, std::min(p.items, cnt - i), false);
        merge_steps(R, items + i, s, p.kids, info + i);
    }
}

}  // namespace efgb
