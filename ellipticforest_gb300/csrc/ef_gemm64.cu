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
//   * pairs with w > 7 are left out;
//   * after every 128 values of k the eight sums per entry go to two 64-bit integers (exact), and the entry
//     is rounded to a double once, at the end.
// With the row's largest entry in [2^61, 2^62) of its scale, the seven pairs of weight 8 come to 7 x 2^-62 of the two
// scales' product per k, rounding both operands to 2^-63 to one more, and a scale is up to twice the largest entry: an
// entry's error is at most 33 K 2^-62 (K 2^-57) of its row maximum times its column maximum, plus one rounding; for
// digits without a pattern it is some sqrt(K) 2^-60.  This is a bound by norms: a chain of FP64 FMAs errs by up to K 2^-53
// of the sum of its |products|, which is less where every product is far below the two maxima (entries of graded rows and
// columns).  The merges check the inverses they form with these products by their residuals, S and T follow from them.
#include <cuda_bf16.h>

#include <algorithm>
#include <climits>
#include <stdexcept>
#include <string>
#include <vector>

#include "ef_gemm64.hpp"
#include "ef_kernels.cuh"
#include "ef_launch.cuh"
#include "ef_tcgen05.cuh"

namespace efgb {

namespace {

constexpr int kDigits = 8;
constexpr int kMT = 128, kNT = 32, kKB = 64;             // tile rows, tile columns, k per block
constexpr int kPlane = kMT * kKB * 2;                    // one digit of an A block: 16 KB
constexpr int kBBlock = kDigits * kNT * kKB * 2;         // all digits of a B block: 32 KB
constexpr int kASlots = kDigits, kBSlots = 2, kSets = 2; // rings: A digits, B blocks, accumulator sets
constexpr int kFlush = 2;                                // k blocks per accumulator set (128 values of k)
constexpr int kNotFinite = 1 << 20;                      // exponent of a row that holds an infinity or NaN
constexpr int kCollect = 256, kGemmThreads = kCollect + 64;  // collecting threads, then the copy and MMA warps
constexpr int kHalf = kNT / 2;                           // columns per collecting thread
constexpr int kMaxOps = 8, kMaxGemms = 4;
enum Add : int { ADD_NONE = 0, ADD_D = 1, ADD_IDENTITY = 2 };
constexpr int kPass = kHalf / 2;                         // of them, columns per pass of the write-out
constexpr int kSums = kCollect * kPass * 16;             // a pass's integer sums on their way to rows of C
constexpr size_t kSmem = 1024 + size_t(kASlots) * kPlane + size_t(kBSlots) * kBBlock + kSums + 512;
static_assert(kBSlots == 2 && kFlush == 2, "a digit's slot is full in even blocks with parity 0, in odd ones with 1");
static_assert(kSmem <= 227 * 1024, "shared memory of one CTA");
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
    int* info;  // info[item] = 1 where a row's largest entry is 2^limit or more
    int limit;
};
struct SplitList {
    int n;
    SplitOp op[kMaxOps];
};

// Digits of one operand: a block takes 32 rows (or columns), finds their largest magnitudes and writes the
// digits of every 64 values of k as the GEMM's shared-memory image (128-byte rows, 16-byte groups swizzled),
// zeros past the operand's ends.  Memory bound: 8 B in (twice, the second time from L2), 16 B out; 5 TB/s on
// 4096 x 8192 entries (160 us).
__global__ void __launch_bounds__(256) k_split64(const __grid_constant__ SplitList L) {
    pdl_begin();
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
    // rows of this thread: columns of B by lanes (coalesced reads), rows of A by groups of eight threads;
    // either way eight consecutive k per 64
    const int rl = cols ? lane : tid >> 3, oct = cols ? warp : tid & 7, r = r0 + rl;
    const bool in = r < P.rows;
    const double* p = base + min(r, P.rows - 1) * sr + (r >= P.v.rs ? P.v.dr : 0);
    auto load = [&](int kb, double (&x)[8]) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int k = kb * kKB + 8 * oct + u;
            x[u] = in && k < K ? p[k * sk + (k >= P.v.ks ? P.v.dk : 0)] : 0.0;
        }
    };
    auto largest = [](const double (&x)[8]) {
        unsigned m = 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) m = max(m, unsigned(__double2hiint(x[u])) & 0x7fffffffu);
        return m;
    };
    double x[8], y[8];  // the first two blocks stay in registers
    load(0, x);
    load(1, y);
    unsigned mx = max(largest(x), largest(y));
    for (int kb = 2; kb < nkb; kb += 2) {
        double t[8], q[8];
        load(kb, t);
        load(kb + 1, q);
        mx = max(mx, max(largest(t), largest(q)));
    }
    if (cols) {
        s_max[warp][lane] = mx;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 8; ++w) mx = max(mx, s_max[w][lane]);
    } else {
#pragma unroll
        for (int off = 4; off > 0; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    }
    const bool finite = mx < 0x7ff00000u;
    const int E = max(int(mx >> 20), 1);  // |x| < 2^(E - 1022)
    if (in && oct == 0) {
        const int e = finite ? E - 1022 : kNotFinite;
        P.ex[(long long)b * P.estride + r] = e;
        if (P.info && e > P.limit) P.info[b] = 1;
    }
    unsigned char* out = P.planes + (long long)b * P.pstride;
    for (int kb = 0; kb < nkb; ++kb) {
        const int k0 = kb * kKB + 8 * oct;
        if (kb == 1) {
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = y[u];
        } else if (kb > 1) {
            load(kb, x);
        }
        if (!finite) {
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = 0.0;
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
    MatView c, d;  // C = (neg ? -1 : 1) A B + D or I or nothing; rows >= rs shifted by dr, columns >= ks by dk
    int neg, add;
    int mt, nt, tile0;
};
struct GemmList {
    int n, tiles;
    GemmOp op[kMaxGemms];
};

// (h + f 2^-32) 2^k as a double, rounded to nearest even, with integer instructions only (a conversion and
// two additions per entry would take the FP64 pipe longer than the whole product of a short K) and without a
// branch, so that several entries overlap.  `odd`: the result is not a normal number (see fixed_to_double_any).
__device__ __forceinline__ double fixed_to_double(long long h, unsigned f, int k, bool& odd) {
    const unsigned sign = unsigned(h >> 63);
    f = (f ^ sign) - sign;
    h = (h ^ (h >> 63)) + (sign != 0 && f == 0 ? 1 : 0);
    unsigned a2 = unsigned((unsigned long long)h >> 32), a1 = unsigned(h), a0 = f;
    int n = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {  // leading zero words
        const bool z = a2 == 0;
        n += z ? 32 : 0;
        a2 = z ? a1 : a2;
        a1 = z ? a0 : a1;
        a0 = z ? 0u : a0;
    }
    const int l = __clz(int(a2)) & 31;
    const unsigned b2 = __funnelshift_l(a1, a2, l), b1 = __funnelshift_l(a0, a1, l), b0 = a0 << l;
    const int e = 1023 + 63 - n - l + k;  // biased exponent of the leading bit
    unsigned lo = (b2 << 21) | (b1 >> 11);
    const unsigned up = (b1 & 0x7ffu) + ((b0 | (lo & 1u)) != 0 ? 1u : 0u) > 0x400u ? 1u : 0u;
    lo += up;
    const unsigned hi = (unsigned(e - 1) << 20) + (b2 >> 11) + (up != 0 && lo == 0 ? 1u : 0u);
    odd = b2 != 0 && unsigned(e - 1) > 2044u;
    return b2 == 0 ? 0.0 : __hiloint2double(int(hi | (sign & 0x80000000u)), int(lo));
}
// the same for results beyond the normal range and rows or columns that are not finite
__device__ __noinline__ double fixed_to_double_any(long long h, unsigned f, int ea, int eb) {
    if (ea >= kNotFinite || eb >= kNotFinite) return __longlong_as_double(0x7ff8000000000000LL);
    return scalbn((double)h + (double)f * 0x1p-32, ea + eb - 36);
}
__device__ __forceinline__ long long join(const int4& q) {
    return (long long)(((unsigned long long)unsigned(q.y) << 32) | unsigned(q.x));
}

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

// C tile of 128 x 32 per step, one CTA per SM walking over the tiles.  Warp 8 copies digit blocks (one bulk
// copy each, the layout is the shared-memory image), warp 9 issues the MMAs, warps 0-7 collect.  For every
// 16 values of k one MMA per digit i of A multiplies it with digits 0 .. 7 - i of B, which are consecutive
// rows of one K-major operand, into the consecutive accumulators of weights i .. 7: N = 32 (8 - i), so a
// digit of A is read from shared memory once.  Two accumulator sets of 256 TMEM columns alternate, so the
// collecting of 128 values of k (8 sums per entry: convert, multiply-add into 64 bits) hides behind the
// MMAs of the next.  Bound: the 2,304 MMA clocks per 64 values of k, with their 160 KB of digits from L2.  A
// 4096 x 4096 x 4096 product runs at 46 TFLOP/s (the FP64 pipe's 1.1), the products of an FP64 build of a
// 7-level tree of 16 x 16 leaves at 36 (17.6 ms); 128 rows and less are a chain of latencies, 10 us a launch.
__global__ void __launch_bounds__(kGemmThreads, 1) k_gemm64(const __grid_constant__ GemmList L, int* __restrict__ err) {
    extern __shared__ unsigned char g_smem[];
    unsigned char* base = g_smem + ((1024u - (smem_u32(g_smem) & 1023u)) & 1023u);
    unsigned char* bbase = base + size_t(kASlots) * kPlane;
    int4* sums = reinterpret_cast<int4*>(bbase + size_t(kBSlots) * kBBlock);
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(sums + kCollect * kPass);
    unsigned long long *a_full = bars, *a_empty = a_full + kASlots, *b_full = a_empty + kASlots,
                       *b_empty = b_full + kBSlots, *acc_full = b_empty + kBSlots, *acc_empty = acc_full + kSets,
                       *drain = acc_empty + kSets;
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(drain + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    if (tid == 0) {
        for (int i = 0; i < kASlots; ++i) { mbar_init(a_full + i, 1); mbar_init(a_empty + i, 1); }
        for (int i = 0; i < kBSlots; ++i) { mbar_init(b_full + i, 1); mbar_init(b_empty + i, 1); }
        for (int i = 0; i < kSets; ++i) { mbar_init(acc_full + i, 1); mbar_init(acc_empty + i, kCollect); }
        mbar_init(drain, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 9) {
        tmem_alloc(tmem_slot, 512u);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = *tmem_slot;
    pdl_begin();  // barriers and TMEM are set up while the digits are still being written

    // Warps 8 and 9 stay converged and one elected lane issues: a branch on the lane number would have the
    // compiler move every operand of an instruction into uniform registers through a loop over the active
    // lanes (109 clocks per MMA measured, against 16 to 128 that the MMA takes).
    if (warp == 8) {
        unsigned sa = 0, sb = 0, pa = 0, pb = 0;  // ring positions and the parity of their current round
        unsigned na = 0, nb = 0;                  // copies issued into either ring
        bool ok = true;
        for (int t = blockIdx.x; t < L.tiles && ok; t += gridDim.x) {
            const TileAt at = tile_at(L, t);
            const GemmOp& g = L.op[at.o];
            const int nkb = (g.K + kKB - 1) / kKB;
            const unsigned char* A = g.A + at.b * g.astride + (long long)at.m * nkb * (kDigits * kPlane);
            const unsigned char* B = g.B + at.b * g.bstride + (long long)at.n * nkb * kBBlock;
            for (int kb = 0; kb < nkb && ok; ++kb) {
                if (nb >= kBSlots) ok = tc_wait(b_empty + sb, pb ^ 1u, abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                if (elect_one()) {
                    mbar_expect_tx(b_full + sb, kBBlock);
                    bulk_copy(bbase + size_t(sb) * kBBlock, B, kBBlock, b_full + sb);
                }
                __syncwarp();
                B += kBBlock;
                ++nb;
                if (++sb == kBSlots) { sb = 0; pb ^= 1u; }
                for (int i = 0; i < kDigits; ++i) {
                    if (na >= kASlots) ok = tc_wait(a_empty + sa, pa ^ 1u, abort_flag);
                    if (!(ok = __all_sync(0xffffffffu, ok))) break;
                    if (elect_one()) {
                        mbar_expect_tx(a_full + sa, kPlane);
                        bulk_copy(base + size_t(sa) * kPlane, A, kPlane, a_full + sa);
                    }
                    __syncwarp();
                    A += kPlane;
                    ++na;
                    if (++sa == kASlots) { sa = 0; pa ^= 1u; }
                }
            }
        }
        if (!ok && lane == 0) {
            // let the copies still in flight land before the shared memory goes away
            volatile int never_set = 0;
            for (unsigned q = na > kASlots ? na - kASlots : 0; q < na; ++q)
                (void)tc_wait(a_full + q % kASlots, (q / kASlots) & 1u, &never_set);
            for (unsigned q = nb > kBSlots ? nb - kBSlots : 0; q < nb; ++q)
                (void)tc_wait(b_full + q % kBSlots, (q / kBSlots) & 1u, &never_set);
            atomicExch(err, 1);
        }
    } else if (warp == 9) {
        unsigned ns = 0;
        bool ok = true;
        // Operand descriptors differ in their address field only, by constants: a digit's slot is its number, and
        // the loop over the k blocks is unrolled over the B slots (an FP64 build of a 7-level tree of 16 x 16
        // leaves: 28.6 ms with slots taken round robin, 27.5 now; an MMA took 96 clocks on average against 72 of
        // the tensor cores).
        const uint64_t da0 = tc_desc(smem_u32(base)), db0 = tc_desc(smem_u32(bbase));
        int t = blockIdx.x, kb = 0, nkb = t < L.tiles ? (L.op[tile_at(L, t).o].K + kKB - 1) / kKB : 0;
        for (unsigned turn = 0; t < L.tiles && ok; ++turn) {
#pragma unroll
            for (int sb = 0; sb < kBSlots; ++sb) {
                if (t >= L.tiles || !ok) break;
                const unsigned set = ns % kSets;
                const bool fresh = kb % kFlush == 0, last = kb == nkb - 1;
                if (fresh && ns >= kSets) ok = tc_wait(acc_empty + set, (ns / kSets - 1) & 1u, abort_flag);
                if (ok) ok = tc_wait(b_full + sb, turn & 1u, abort_flag);
                const uint64_t db = db0 + uint64_t(sb * (kBBlock >> 4));
                const unsigned d = tmem + set * 256u;
#pragma unroll
                for (int i = 0; i < kDigits; ++i) {
                    if (ok) ok = tc_wait(a_full + i, unsigned(sb & 1), abort_flag);
                    if (!(ok = __all_sync(0xffffffffu, ok))) break;
                    tc_fence_after();
                    const uint64_t da = da0 + uint64_t(i * (kPlane >> 4));
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < kKB / 16; ++kk)
                            tc_mma(d + unsigned(i * kNT), da + uint64_t(2 * kk), db + uint64_t(2 * kk),
                                   tc_idesc(kMT, kNT * (kDigits - i)), i == 0 && kk == 0 ? (fresh ? 0u : 1u) : 1u);
                        tc_commit(a_empty + i);
                        if (i == kDigits - 1) {
                            tc_commit(b_empty + sb);
                            if (!fresh || last) tc_commit(acc_full + set);
                        }
                    }
                    __syncwarp();
                }
                if (!fresh || last) ++ns;
                ++kb;
                if (last) {
                    t += gridDim.x;
                    kb = 0;
                    if (t < L.tiles) nkb = (L.op[tile_at(L, t).o].K + kKB - 1) / kKB;
                }
            }
        }
        // every MMA issued has completed before TMEM is freed
        if (elect_one()) tc_commit(drain);
        __syncwarp();
        volatile int never_set = 0;
        if (!tc_wait(drain, 0u, &never_set)) ok = false;
        if (!ok && lane == 0) atomicExch(err, 1);
    } else {
        // warps w and w + 4 hold the same 32 rows (TMEM lanes 32 (w mod 4) ..), columns 0-15 and 16-31
        const int wr = warp & 3, c0 = warp < 4 ? 0 : kHalf;
        const unsigned acc0 = tmem + (unsigned(wr * 32) << 16) + unsigned(c0);
        int4* own = sums + (warp * 32) * kPass;
        unsigned ns = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < L.tiles && ok; t += gridDim.x) {
            const TileAt at = tile_at(L, t);
            const GemmOp& g = L.op[at.o];
            const int nkb = (g.K + kKB - 1) / kKB, flushes = (nkb + kFlush - 1) / kFlush;
            long long hi[kHalf], lo[kHalf];
#pragma unroll
            for (int c = 0; c < kHalf; ++c) { hi[c] = 0; lo[c] = 0; }
            for (int f = 0; f < flushes; ++f, ++ns) {
                const unsigned set = ns % kSets;
                if (!(ok = tc_wait(acc_full + set, (ns / kSets) & 1u, abort_flag))) break;
                tc_fence_after();
                // weights 0-3 into hi, 4-7 into lo; rolled over the weight, since a tile runs through this code
                // only K / 128 times and fetching straight-line code costs more than running it
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    int scale = 1 << 24;
#pragma unroll 1
                    for (int w = 4 * part; w < 4 * part + 4; ++w, scale >>= 8) {
                        float v[kHalf];
                        tmem_ld16(acc0 + set * 256u + unsigned(w * kNT), v);
#pragma unroll
                        for (int c = 0; c < kHalf; ++c) {
                            const long long q = (long long)__float2int_rn(v[c]) * scale;
                            if (part == 0) hi[c] += q;
                            else lo[c] += q;
                        }
                    }
                }
                tc_fence_before();
                mbar_arrive(acc_empty + set);
            }
            if (!ok) break;
            // the sums change hands inside the warp, eight columns at a time, so that lanes take consecutive columns
            // of four rows: this thread's row goes to shared memory with its 16-byte entries swizzled by the row
            const int row0 = at.m * kMT + 32 * wr, quad = lane >> 3;
            const int ea = g.ea[(long long)at.b * g.eastride + min(row0 + lane, g.M - 1)];
            const int add = g.add, crs = g.c.rs, drs = g.d.rs, rows = min(32, g.M - row0);
            const long long cld = g.c.ld, cdr = g.c.dr, dld = g.d.ld, ddr = g.d.dr;
            const unsigned flip = g.neg ? 0x80000000u : 0u;
#pragma unroll
            for (int ps = 0; ps < kHalf / kPass; ++ps) {
#pragma unroll
                for (int k = 0; k < kPass; ++k) {
                    const int c = ps * kPass + k;
                    const long long h = hi[c] + (lo[c] >> 32);  // the carry of lo first
                    own[lane * kPass + (k ^ (lane & 7))] = make_int4(int(h), int(h >> 32), int(lo[c]), 0);
                }
                __syncwarp();
                const int n = at.n * kNT + c0 + ps * kPass + (lane & 7);
                const bool col = n < g.N;
                const int eb = g.eb[(long long)at.b * g.ebstride + min(n, g.N - 1)];
                double* C = table_ptr(g.c.base, at.b) + g.c.off + n + (n >= g.c.ks ? g.c.dk : 0);
                double v[8], old[8];
                if (add == ADD_D) {
                    const double* D = table_ptr(g.d.base, at.b) + g.d.off + n + (n >= g.d.ks ? g.d.dk : 0);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int i = 4 * j + quad, r = row0 + i;
                        old[j] = col && i < rows ? D[r * dld + (r >= drs ? ddr : 0)] : 0.0;
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) old[j] = n == row0 + 4 * j + quad ? 1.0 : 0.0;
                }
                // all conversions before any branch: a branch per entry would run them one after another
                unsigned odd = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int i = 4 * j + quad;
                    const int4 q = own[i * kPass + ((lane & 7) ^ (i & 7))];
                    const int e1 = __shfl_sync(0xffffffffu, ea, i);
                    bool o;
                    v[j] = fixed_to_double(join(q), unsigned(q.z), e1 + eb - 36, o);  // (h + f 2^-32) 2^(e1 + eb - 36)
                    odd |= o || e1 >= kNotFinite || eb >= kNotFinite ? 1u << j : 0u;
                }
                if (__any_sync(0xffffffffu, odd != 0)) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int i = 4 * j + quad;
                        const int4 q = own[i * kPass + ((lane & 7) ^ (i & 7))];
                        const int e1 = __shfl_sync(0xffffffffu, ea, i);
                        if ((odd >> j) & 1u) v[j] = fixed_to_double_any(join(q), unsigned(q.z), e1, eb);
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = __hiloint2double(int(unsigned(__double2hiint(v[j])) ^ flip), __double2loint(v[j]));
                if (add) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = old[j] + v[j];
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int i = 4 * j + quad, r = row0 + i;
                    if (col && i < rows) C[r * cld + (r >= crs ? cdr : 0)] = v[j];
                }
                __syncwarp();
            }
        }
        if (!ok) atomicExch(err, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 9) tmem_dealloc(tmem, 512u);
}

struct InvList {
    int nv;
    MatView v[2], out[2];
};

// Inverse of one matrix of at most 32 rows per block, in place, by Gauss-Jordan steps in FP64 (row k of the
// result from the pivot row of step k): 64 threads hold 4 x 4 entries each.  The pivot of column k is the
// largest entry of the rows not used yet, compared by its leading 26 bits (the row's number in the last six,
// so one warp reduction finds both); rows are not moved but put in order when they are written.  A pivot that
// is zero or not finite sets info.  Bound by the two block barriers and the division of a step.
__global__ void __launch_bounds__(64) k_inv_small(const __grid_constant__ InvList L, int n, int* __restrict__ info) {
    pdl_begin();
    const MatView& V = L.v[blockIdx.x];
    double* A = table_ptr(V.base, blockIdx.y) + V.off;
    const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7, lane = tid & 31;
    __shared__ double s_col[2][32], s_row[2][32];
    __shared__ int s_p[32], s_k[32];
    double a[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = 4 * ty + i, c = 4 * tx + j;
            a[i][j] = r < n && c < n ? A[(long long)r * V.ld + c] : (r == c ? 1.0 : 0.0);
        }
    unsigned used = 0;
    bool bad = false;
    // the column inside a thread's four is a constant of the unrolled loop, the pivot row inside its four a chain
    // of selections: the entries stay in registers
    for (int k4 = 0; k4 < n; k4 += 4) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        const int k = k4 + kk, bf = kk & 1;
        if (k >= n) break;
        if (tx == (k >> 2)) {
#pragma unroll
            for (int i = 0; i < 4; ++i) s_col[bf][4 * ty + i] = a[i][kk];
        }
        __syncthreads();
        const unsigned h = unsigned(__double2hiint(s_col[bf][lane])) & 0x7fffffffu;
        const unsigned key = (used >> lane) & 1u || lane >= n ? 0u : ((h << 1) & ~63u) | unsigned(63 - lane);
        const unsigned best = __reduce_max_sync(0xffffffffu, key);
        const int p = 63 - int(best & 63u);  // an unused row always has a key above zero
        const double piv = s_col[bf][p];
        if (!(fabs(piv) > 0.0) || best >= 0xffe00000u) bad = true;
        used |= 1u << p;
        if (ty == (p >> 2)) {
            const double inv = 1.0 / piv;
            const int pi = p & 3;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double x = pi == 0 ? a[0][j] : pi == 1 ? a[1][j] : pi == 2 ? a[2][j] : a[3][j];
                s_row[bf][4 * tx + j] = j == kk && tx == (k >> 2) ? inv : x * inv;
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
            for (int j = 0; j < 4; ++j) a[i][j] = r == p ? rj[j] : fma(-c, rj[j], j == kk && tx == (k >> 2) ? 0.0 : a[i][j]);
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

// x 2^-e rounded to nearest, for |x| < 2^e (zero where it would be subnormal; NaN where asked)
__device__ __forceinline__ float scaled_float(double x, int e, bool nan) {
    const int hi = __double2hiint(x);
    const unsigned lo = unsigned(__double2loint(x));
    const int top = (hi & 0x7fffffff) - ((e + 896) << 20);  // float exponent and leading 20 bits of the significand
    const unsigned bits = ((unsigned(top) << 3) | (lo >> 29)) + ((lo >> 28) & 1u);
    return __uint_as_float(nan ? 0x7fc00000u : (unsigned(hi) & 0x80000000u) | (top < (1 << 20) ? 0u : bits));
}

// x 2^-e (zero below the smallest normal number, the largest power of two above the range; PLAIN: |e| is at most
// 800, so that neither happens to a normal x)
template <bool PLAIN>
__device__ __forceinline__ double scaled_double(float x, int e) {
    const unsigned b = __float_as_uint(x), u = b & 0x7fffffffu;
    const int ex = int(u >> 23) + 896 - e;
    const bool zero = u < 0x00800000u || (!PLAIN && ex < 1), large = !PLAIN && ex > 2046;
    const unsigned hi = zero ? 0u : large ? 0x7fe00000u : (u >> 3) + (unsigned(896 - e) << 20);
    return __hiloint2double(int((b & 0x80000000u) | hi), zero || large ? 0 : int(u << 29));
}

constexpr int kStartLd = 132;
constexpr size_t kStartSmem = 192 * kStartLd * sizeof(float);

// two FP32 multiply-adds per instruction: (x, y) += (a, a) * (p, q)
__device__ __forceinline__ void fma2(float& x, float& y, float a, float p, float q) {
    asm("{\n .reg .b64 d, m, n;\n mov.b64 d, {%0, %1};\n mov.b64 m, {%2, %2};\n mov.b64 n, {%3, %4};\n"
        " fma.rn.f32x2 d, m, n, d;\n mov.b64 {%0, %1}, d;\n}\n"
        : "+f"(x), "+f"(y)
        : "f"(a), "f"(p), "f"(q));
}

// FP32 inverse of one matrix of at most 128 rows per block: the start of the iteration of `invert`.  Gauss-Jordan
// in steps of 32 rows: one warp inverts the diagonal block in registers (a row per lane, pivots inside the
// block, the pivot row through shared memory), the block's row panel is multiplied by it, and all 256 threads
// update their 8 x 8 entries with 32 columns at once.  Rows are brought to magnitudes below one by powers of two
// first, so any scaling of the rows is harmless.  One block, so it is a chain of latencies: of 97,000 clocks for
// 128 rows (51 us; 61 us with a branch per converted entry), the diagonal blocks take 42,000 (320 per pivot, by
// shuffles as much), the updates 23,000 (16,400 of FP32 multiply-adds), the rest is loads, panels and stores.
__global__ void __launch_bounds__(256) k_inv_start(const __grid_constant__ InvList L, int n, int* __restrict__ info) {
    pdl_begin();
    constexpr int PB = 32, LD = kStartLd;  // panel width; row stride (16-byte rows, no bank conflicts)
    const MatView &V = L.v[blockIdx.x], &O = L.out[blockIdx.x];
    const double* A = table_ptr(V.base, blockIdx.y) + V.off;
    double* out = table_ptr(O.base, blockIdx.y) + O.off;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, lane = tid & 31;
    const int warp = tid >> 5;
    extern __shared__ __align__(16) float is_smem[];
    float (*s_all)[LD] = reinterpret_cast<float (*)[LD]>(is_smem);             // the matrix on its way in and out
    float (*s_row)[LD] = reinterpret_cast<float (*)[LD]>(is_smem + 128 * LD);  // row panel, then times the inverse block
    float (*s_colT)[LD] = reinterpret_cast<float (*)[LD]>(is_smem + 160 * LD); // column panel, transposed
    __shared__ __align__(16) float s_inv[PB][PB + 4];
    __shared__ __align__(16) float s_piv[2][PB + 4];
    __shared__ int s_e[128];
    // rows and columns of a thread: 4 t .. 4 t + 3 and 64 more, so that 16-byte reads of a row or column by the
    // 16 threads of a direction touch every bank once
    // (the loops over rows and steps stay rolled: the block runs each a few times at most, and fetching
    // straight-line code would take longer than running it)
    // (eight rows of a warp in flight; the conversions are integer steps without a branch: one per entry would
    // run them one after another)
#pragma unroll 1
    for (int r0 = warp; r0 < 128; r0 += 64) {
        double x[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int r = r0 + 8 * i, c = lane + 32 * q;
                x[i][q] = r < n && c < n ? A[(long long)r * V.ld + c] : (r == c ? 1.0 : 0.0);
            }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int r = r0 + 8 * i;
            unsigned m = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) m = max(m, unsigned(__double2hiint(x[i][q])) & 0x7fffffffu);
            m = __reduce_max_sync(0xffffffffu, m);
            const int e = max(int(m >> 20), 1) - 1022;
#pragma unroll
            for (int q = 0; q < 4; ++q) s_all[r][lane + 32 * q] = scaled_float(x[i][q], e, m >= 0x7ff00000u);
            if (lane == 0) s_e[r] = e;
        }
    }
    __syncthreads();
    float a[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
            const float4 t = *reinterpret_cast<const float4*>(&s_all[4 * ty + (i & 3) + 16 * (i & 4)][4 * tx + 16 * j]);
            a[i][j] = t.x; a[i][j + 1] = t.y; a[i][j + 2] = t.z; a[i][j + 3] = t.w;
        }
    bool bad = false;
#pragma unroll 1
    for (int k0 = 0; k0 < n; k0 += PB) {
        // rows (columns) k0 .. k0 + 31 are entries 4 .. 7 or 0 .. 3 of the threads of eight rows (columns)
        const int t0 = (k0 & 63) >> 2, hi = k0 >= 64 ? 4 : 0;
        const bool mine_r = ty >= t0 && ty < t0 + 8, mine_c = tx >= t0 && tx < t0 + 8;
        // published: the rows R with the identity for the block itself, the columns as -C with the identity in the
        // block's rows (A <- A - C R then turns them into R), the block
        if (mine_r) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = 4 * (ty - t0) + i;
#pragma unroll
                for (int j = 0; j < 8; j += 4) {
                    float4 v = hi ? make_float4(a[i + 4][j], a[i + 4][j + 1], a[i + 4][j + 2], a[i + 4][j + 3])
                                  : make_float4(a[i][j], a[i][j + 1], a[i][j + 2], a[i][j + 3]);
                    if (mine_c && j == hi) {
                        const int c = 4 * (tx - t0);
                        *reinterpret_cast<float4*>(&s_inv[r][c]) = v;
                        v = make_float4(r == c, r == c + 1, r == c + 2, r == c + 3);
                    }
                    *reinterpret_cast<float4*>(&s_row[r][4 * tx + 16 * j]) = v;
                }
            }
        }
        if (mine_c) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = 4 * (tx - t0) + j;
#pragma unroll
                for (int i = 0; i < 8; i += 4) {
                    float4 v = hi ? make_float4(-a[i][j + 4], -a[i + 1][j + 4], -a[i + 2][j + 4], -a[i + 3][j + 4])
                                  : make_float4(-a[i][j], -a[i + 1][j], -a[i + 2][j], -a[i + 3][j]);
                    if (mine_r && i == hi) {
                        const int r = 4 * (ty - t0);
                        v = make_float4(r == c, r + 1 == c, r + 2 == c, r + 3 == c);
                    }
                    *reinterpret_cast<float4*>(&s_colT[c][4 * ty + 16 * i]) = v;
                }
            }
        }
        __syncthreads();
        if (tid < 32) {
            // inverse of the 32 x 32 diagonal block: lane = row; the pivot of column k is the largest entry of the
            // rows not used yet (leading 26 bits, then the row), row k of the result comes from that row
            float d[PB];
#pragma unroll
            for (int j = 0; j < PB; j += 4) {
                const float4 t = *reinterpret_cast<const float4*>(&s_inv[lane][j]);
                d[j] = t.x; d[j + 1] = t.y; d[j + 2] = t.z; d[j + 3] = t.w;
            }
            bool used = false;
            int my_k = 0, my_p = 0;  // the step this row is the pivot of; the pivot row of step `lane`
            unsigned best = 0;
            float my_inv = 0.f;
            auto candidate = [&](float v) {
                const unsigned h = __float_as_uint(v) & 0x7fffffffu;
                my_inv = __fdividef(1.f, v);
                best = __reduce_max_sync(0xffffffffu, used ? 0u : ((h << 1) & ~63u) | unsigned(63 - lane));
            };
            candidate(d[0]);
            // The pivot row goes round through shared memory, and a step leaves the columns where they are, two to
            // an instruction; after two steps they move down two registers and the steps' own go to the end.
#pragma unroll 1
            for (int k = 0; k < PB; k += 2) {
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    const int p = 63 - int(best & 63u);
                    const bool pr = lane == p;
                    if (pr) {
                        used = true;
                        my_k = k + o;
#pragma unroll
                        for (int j = 0; j < PB; j += 4)
                            *reinterpret_cast<float4*>(&s_piv[o][j]) = make_float4(d[j], d[j + 1], d[j + 2], d[j + 3]);
                        s_piv[o][PB] = my_inv;
                    }
                    if (lane == k + o) my_p = p;
                    __syncwarp();
                    const float inv = s_piv[o][PB];
                    float r[PB];
#pragma unroll
                    for (int j = 0; j < PB; j += 4) {
                        const float4 t = *reinterpret_cast<const float4*>(&s_piv[o][j]);
                        r[j] = t.x; r[j + 1] = t.y; r[j + 2] = t.z; r[j + 3] = t.w;
                    }
                    if (!(fabsf(r[o]) > 0.f) || best >= 0xff000000u) bad = true;
                    // every row loses c times the scaled pivot row; the pivot row keeps 1 / piv of itself with
                    // c = piv - 1; the entries of the step's column count as those of a unit vector
                    const float c = (pr ? r[o] - 1.f : d[o]) * inv, own = (pr ? 1.f : 0.f) - c;
                    // the next column first, and the search for its pivot between the others
                    if (o == 0) {
                        d[1] = fmaf(-c, r[1], d[1]);
                        d[0] = own;
                        candidate(d[1]);
#pragma unroll
                        for (int j = 2; j < PB; j += 2) fma2(d[j], d[j + 1], -c, r[j], r[j + 1]);
                    } else {
                        const float first = fmaf(-c, r[0], d[0]);
                        fma2(d[2], d[3], -c, r[2], r[3]);
                        candidate(d[2]);
#pragma unroll
                        for (int j = 4; j < PB; j += 2) fma2(d[j], d[j + 1], -c, r[j], r[j + 1]);
#pragma unroll
                        for (int j = 2; j < PB; ++j) d[j - 2] = d[j];
                        d[PB - 2] = first;
                        d[PB - 1] = own;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < PB; ++j) {
                const int pj = __shfl_sync(0xffffffffu, my_p, j);
                s_inv[my_k][pj] = d[j];
            }
        }
        __syncthreads();
        // panel x inverse block: 32 x 128, 4 x 4 entries per thread
        {
            const int r0 = 4 * (tid >> 5), c0 = 4 * lane;
            float s[4][4] = {};
#pragma unroll 2
            for (int k4 = 0; k4 < PB; k4 += 4) {
                float v[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 t = *reinterpret_cast<const float4*>(&s_inv[r0 + i][k4]);
                    v[i][0] = t.x; v[i][1] = t.y; v[i][2] = t.z; v[i][3] = t.w;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float4 p = *reinterpret_cast<const float4*>(&s_row[k4 + u][c0]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        fma2(s[i][0], s[i][1], v[i][u], p.x, p.y);
                        fma2(s[i][2], s[i][3], v[i][u], p.z, p.w);
                    }
                }
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<float4*>(&s_row[r0 + i][c0]) = make_float4(s[i][0], s[i][1], s[i][2], s[i][3]);
        }
        __syncthreads();
        // the block's columns and rows start from zero
        if (mine_c) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (hi) a[i][j + 4] = 0.f;
                    else a[i][j] = 0.f;
                }
        }
        if (mine_r) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (hi) a[i + 4][j] = 0.f;
                    else a[i][j] = 0.f;
                }
        }
#pragma unroll 2
        for (int k = 0; k < PB; ++k) {
            float rj[8], ci[8];
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                const float4 t = *reinterpret_cast<const float4*>(&s_row[k][4 * tx + 16 * j]);
                rj[j] = t.x; rj[j + 1] = t.y; rj[j + 2] = t.z; rj[j + 3] = t.w;
                const float4 u = *reinterpret_cast<const float4*>(&s_colT[k][4 * ty + 16 * j]);
                ci[j] = u.x; ci[j + 1] = u.y; ci[j + 2] = u.z; ci[j + 3] = u.w;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) a[i][j] = fmaf(ci[i], rj[j], a[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; j += 4)
            *reinterpret_cast<float4*>(&s_all[4 * ty + (i & 3) + 16 * (i & 4)][4 * tx + 16 * j]) =
                make_float4(a[i][j], a[i][j + 1], a[i][j + 2], a[i][j + 3]);
    __syncthreads();
    int ec[4];  // a column of A^-1 takes the scale of that row of A
    bool plain = true;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        ec[q] = s_e[lane + 32 * q];
        plain = plain && ec[q] >= -800 && ec[q] <= 800;
    }
    plain = __all_sync(0xffffffffu, plain);
    double* o = out + (long long)warp * O.ld + lane;
    if (plain) {
#pragma unroll 2
        for (int r = warp; r < n; r += 8, o += 8LL * O.ld)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (lane + 32 * q < n) o[32 * q] = scaled_double<true>(s_all[r][lane + 32 * q], ec[q]);
    } else {
#pragma unroll 1
        for (int r = warp; r < n; r += 8, o += 8LL * O.ld)
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (lane + 32 * q < n) o[32 * q] = scaled_double<false>(s_all[r][lane + 32 * q], ec[q]);
    }
    if (tid < 32 && bad && lane == 0) info[blockIdx.y] = 1;
}

// X^{-1} from the X buffer to its place behind S in the RHS buffer (columns [8s, 12s))
__global__ void k_place_inverse(const MergeItem* __restrict__ items, int s) {
    pdl_begin();
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
    pdl_begin();
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
    pdl_begin();
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
    Runner(cudaStream_t st, char* ws, int* err, int cnt, bool dry) : st_(st), ws_(ws), err_(err), cnt_(cnt), dry_(dry), chain_(dry ? Chain::none : merge_chain(st)) {}
    size_t mark() const { return off_; }
    void release(size_t m) { off_ = m; }
    size_t peak() const { return peak_; }
    bool dry() const { return dry_; }
    Chain chain() const { return chain_; }  // see ef_launch.cuh
    int count() const { return cnt_; }
    cudaStream_t stream() const { return st_; }

    struct Digits {
        unsigned char* planes;
        long long pstride;
        int* ex;
        int estride, len, K;
    };
    // role 0: rows of A (len = M); 1: columns of B (len = N)
    Digits split(const MatView& v, int len, int K, int role, int neg0 = 0, int neg1 = 0, int* info = nullptr,
                 int limit = 0) {
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
        op = SplitOp{v, len, K, role, neg0, neg1, d.planes, d.pstride, d.ex, d.estride, blocks_, info, limit};
        // whole tiles: the rows past the end are written as zeros
        blocks_ += role ? (len + kNT - 1) / kNT : (len + kMT - 1) / kMT * (kMT / 32);
        ++sl_.n;
        return d;
    }
    // C = (neg ? -1 : 1) A B, plus C or the identity
    void gemm(const Digits& a, const Digits& b, const MatView& c, bool neg, int add) { gemm(a, b, c, neg, add, c); }
    // ..., plus D
    void gemm(const Digits& a, const Digits& b, const MatView& c, bool neg, int add, const MatView& d) {
        if (gl_.n == kMaxGemms) flush();
        GemmOp& g = gl_.op[gl_.n];
        const int mt = (a.len + kMT - 1) / kMT, nt = (b.len + kNT - 1) / kNT;
        g = GemmOp{a.planes, b.planes, a.pstride, b.pstride, a.ex, b.ex, a.estride, b.estride, a.len, b.len, a.K,
                   c, d, neg, add, mt, nt, gl_.tiles};
        gl_.tiles += mt * nt * cnt_;
        ++gl_.n;
    }
    void flush_split() {
        if (sl_.n && !dry_) {
            launch_chained(chain_, k_split64, dim3(unsigned(blocks_), unsigned(cnt_)), 256, 0, st_, sl_);
            ++g_kernel_launches;
        }
        sl_.n = 0;
        blocks_ = 0;
    }
    void flush() {
        flush_split();
        if (gl_.n && !dry_) {
            cudaFuncSetAttribute(k_gemm64, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem));
            launch_chained(chain_, k_gemm64, dim3(unsigned(std::min(gl_.tiles, sm_count()))), kGemmThreads, kSmem, st_, gl_, err_);
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
    Chain chain_;
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

// rows of the leading block of the 2 x 2 elimination of h rows
int first_part(int h) { return (h / 2 + 31) / 32 * 32; }

// Inverses of one or two h x h matrices per item, in place.  tmp: invert64_tmp(h) doubles per view.
//
// Up to 32 rows: Gauss-Jordan in FP64.  Up to 128: an FP32 inverse Y with residual E = I - A Y (~1e-7 cond) and
// Y (I + E)(I + E^2), whose residual is E^4, with accurate products (two Newton steps in three rounds of products
// instead of four); where E^2 is not below 2^-31 per entry (E^4 below 128 2^-62 = 2^-55) info is set.  Beyond,
// 2 x 2 block elimination:
//   [A B; C D]: G = A^-1 B, F = C A^-1, D <- (D - C G)^-1, B <- -G D, C <- -D F, A <- A^-1 - B F.
// Every product is an accurate GEMM, so the only FP64 roundings are those of the stored blocks.
void invert(Runner& R, const std::vector<MatView>& v, int h, const MatView& tmp, int* info) {
    const size_t n = v.size(), m0 = R.mark();
    if (h <= 32) {
        if (!R.dry()) {
            InvList L{};
            L.nv = int(n);
            for (size_t i = 0; i < n; ++i) L.v[i] = v[i];
            launch_chained(R.chain(), k_inv_small, dim3(unsigned(n), unsigned(R.count())), 64, 0, R.stream(), L, h, info);
            ++g_kernel_launches;
        }
        return;
    }
    if (h <= 128) {
        std::vector<MatView> Y, E;
        InvList L{};
        L.nv = int(n);
        for (size_t i = 0; i < n; ++i) {
            MatView y = tmp;
            y.off += 2LL * i * h * h;
            y.ld = h;
            MatView e = y;
            e.off += (long long)h * h;
            Y.push_back(y);
            E.push_back(e);
            L.v[i] = v[i];
            L.out[i] = y;
        }
        if (!R.dry()) {
            cudaFuncSetAttribute(k_inv_start, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kStartSmem));
            launch_chained(R.chain(), k_inv_start, dim3(unsigned(n), unsigned(R.count())), 256, kStartSmem, R.stream(), L, h, info);
            ++g_kernel_launches;
        }
        // E = I - A Y; Y' = Y + Y E and E^2 together; Y' + Y' E^2
        for (size_t i = 0; i < n; ++i) {
            const auto a = R.split(v[i], h, h, 0), yb = R.split(Y[i], h, h, 1);
            R.gemm(a, yb, E[i], true, ADD_IDENTITY);
        }
        R.flush();
        for (size_t i = 0; i < n; ++i) {
            const auto eb = R.split(E[i], h, h, 1), ya = R.split(Y[i], h, h, 0), ea = R.split(E[i], h, h, 0);
            R.gemm(ya, eb, Y[i], false, ADD_D);
            R.gemm(ea, eb, E[i], false, ADD_NONE);
        }
        R.flush();
        for (size_t i = 0; i < n; ++i) {
            const auto eb = R.split(E[i], h, h, 1, 0, 0, info, -31), ya = R.split(Y[i], h, h, 0);
            R.gemm(ya, eb, v[i], false, ADD_D, Y[i]);
        }
        R.flush();
        R.release(m0);
        return;
    }
    const int h1 = first_part(h), h2 = h - h1;
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
        R.gemm(aA, bB, G[i], false, ADD_NONE);
        R.gemm(c0[i], aB, F[i], false, ADD_NONE);
    }
    R.flush();
    for (size_t i = 0; i < n; ++i) R.gemm(c0[i], R.split(G[i], h2, h1, 1), D[i], true, ADD_D);
    R.flush();
    R.release(m0);
    invert(R, D, h2, below, info);
    std::vector<Runner::Digits> f0;
    for (size_t i = 0; i < n; ++i) {
        const auto dA = R.split(D[i], h2, h2, 0), dB = R.split(D[i], h2, h2, 1), gA = R.split(G[i], h1, h2, 0);
        f0.push_back(R.split(F[i], h1, h2, 1));
        R.gemm(gA, dB, B[i], true, ADD_NONE);
        R.gemm(dA, f0[i], C[i], true, ADD_NONE);
    }
    R.flush();
    for (size_t i = 0; i < n; ++i) R.gemm(R.split(B[i], h1, h2, 0), f0[i], A[i], true, ADD_D);
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
        R.gemm(a0, b0, G, false, ADD_NONE);
        R.gemm(a1, b1, at(G, s, 0), false, ADD_NONE);
        R.gemm(c0, a0b, F, false, ADD_NONE);
        R.gemm(c1, a1b, at(F, 0, s), false, ADD_NONE);
        R.flush();
        R.release(0);
        const auto c = R.split(C0, 2 * s, 2 * s, 0), g = R.split(G, 2 * s, 2 * s, 1);
        R.gemm(c, g, D, true, ADD_D);
        R.flush();
        R.release(0);
    }
    invert(R, {D}, 2 * s, below, info);
    {
        const auto dA = R.split(D, 2 * s, 2 * s, 0), dB = R.split(D, 2 * s, 2 * s, 1), g = R.split(G, 2 * s, 2 * s, 0),
                   f = R.split(F, 2 * s, 2 * s, 1);
        R.gemm(g, dB, B0, true, ADD_NONE);
        R.gemm(dA, f, C0, true, ADD_NONE);
        R.flush();
        R.gemm(R.split(B0, 2 * s, 2 * s, 0), f, A0, true, ADD_D);
        R.flush();
        R.release(0);
    }
    if (!R.dry()) {
        const dim3 rows(unsigned((m + 7) / 8), unsigned(R.count()));
        launch_chained(R.chain(), k_check_y, rows, 256, 0, R.stream(), items, s);
        launch_chained(R.chain(), k_check_r, rows, 256, 0, R.stream(), items, s, info);
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
            R.gemm(xa, tb, o, false, ADD_NONE);
        }
        R.flush();
        R.release(0);
    }
    if (!R.dry()) {
        const long long tot = 8LL * s * s;
        launch_chained(R.chain(), k_place_inverse, dim3(unsigned(std::min(2048LL, (tot + 255) / 256)), unsigned(R.count())), 256, 0, R.stream(),
                       items, s);
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
            R.gemm(R.split(h, 2 * s, 2 * s, 0), R.split(b, 2 * m, 2 * s, 1), o, false, ADD_D);
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

size_t invert64_tmp(int h) {
    if (h <= 128) return 2 * size_t(h) * h;
    const size_t h1 = first_part(h), h2 = h - h1;
    return 2 * h1 * h2 + std::max(invert64_tmp(int(h1)), invert64_tmp(int(h2)));
}

size_t invert64_workspace(int h) {
    Runner R(nullptr, nullptr, nullptr, 1, true);
    const MatView v{PtrTable{nullptr, 0}, 0, h};
    invert(R, {v}, h, v, nullptr);
    return R.peak();
}

void invert64(cudaStream_t st, double* const* A, double* const* tmp, int h, int* info, char* ws, int* err) {
    Runner R(st, ws, err, 1, false);
    invert(R, {MatView{PtrTable{A, 0}, 0, h}}, h, MatView{PtrTable{tmp, 0}, 0, h}, info);
}

}  // namespace efgb
