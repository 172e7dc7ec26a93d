// split_gemm.cu — K2/K3: the tensor-core forms of the double-precision product on sm_103a.
//
//   GB300_METHOD_SPLIT   Ozaki-style split-precision product that reaches FP64-level normwise
//                        accuracy: A and B are scaled per row / per column by powers of two and
//                        cut into BF16 planes, residues of the scaled integers modulo 2 to 15
//                        moduli (by default) or base-256 digits (explicit slice counts); the plane
//                        products run on tcgen05 tensor cores (FP32 accumulators in TMEM) in groups
//                        whose sums stay exactly representable; the group sums are reduced modulo
//                        their modulus (digits: added in int32) exactly, and only the final
//                        rounding, the exponent rescale and alpha/beta run in FP64.
//   GB300_METHOD_BF16X3  hi*hi + hi*lo + lo*hi with BF16 hi/lo parts, FP32 accumulation.
//   GB300_METHOD_BF16    one BF16 product, FP32 accumulation.
//   GB300_METHOD_AUTO    the split form when it is predicted faster than the native kernel.
//
// They replace the same CBLAS dgemm call as the native kernel (blaze/math/blas/cblas/gemm.h:
// 156-162, reached from DMatDMatMultExpr.h:2021-2037 and siblings).
//
// ---- digit arithmetic --------------------------------------------------------------------------
// (The residue form's stands at c_mod below.)
// Row i of op(A) is scaled by 2^-e_i with e_i = frexp exponent of max_p |A(i,p)|, so the scaled
// entries x satisfy |x| < 1.  Digits: d_1 = rint(x*2^7), r_1 = x*2^7 - d_1, then
// d_s = rint(r_{s-1}*2^8), r_s = r_{s-1}*2^8 - d_s (all exact in FP64; |d_s| <= 128, |r_s| <= 1/2),
// so x = sum_s d_s 2^(1-8s) + r_S 2^(1-8S).  Columns of op(B) likewise with exponents f_j.
// With planes numbered a = s-1, the pair (a, b) has weight 2^(-14-8(a+b)); all pairs with
// a + b = L form "level" L, L = 0..S-1 (the triangle s + t <= S + 1 of Ozaki's scheme).
//   Exactness: one TMEM drain group accumulates at most 16 x 64 = 1024 products of digits,
//   |product| <= 128^2 = 2^14, so every partial sum is an integer of magnitude at most 2^24, which
//   FP32 holds exactly (2^24 itself only as the group's final value, when all 1024 products are
//   largest with one sign).  The epilogue converts the FP32 integer v with cvt.rni (exact) and
//   adds it in int32.  A level's int32 sum over a k-segment is bounded by
//   n_L * Kseg * 2^14 < 2^31.
//   Error bound (elementwise, scaled units): |dC_ij| <= (S+1) K 2^(-8S); normwise
//   ||dC||_F / (||A||_F ||B||_F) <= (S+1) K 2^(-8S) ||2^e||_2 ||2^f||_2 / (||A||_F ||B||_F)
//   plus (S+3) 2^-53 for the FP64 recombination.  The slice count is the smallest S whose bound
//   meets the target (default K * 2^-53, the classical worst-case FP64 dot-product bound); it is
//   chosen on the device, so the whole product is stream-ordered without a host round trip.
//
// ---- kernel structure (tc_gemm_kernel) ---------------------------------------------------------
// Persistent pairs of CTAs (a cluster of two, one CTA per SM), each pair owning 256 x 256 output
// tiles (and a k-segment) of one level at a time.
//   warp 0      TMA producer: 128x64 A-plane box + the CTA's 128x64 half of the B-plane box per item,
//               128B swizzle, 6-stage ring of 32 KB stages.
//   warp 1      TMEM allocator; the even CTA's issues the pair's 4 x tcgen05.mma (M=256, N=256, K=16,
//               BF16->FP32) per item; tcgen05.commit releases the smem stage in both CTAs and, at the
//               end of a drain group, hands the accumulator buffer to both epilogues.  Two 256-column
//               TMEM accumulators let the MMAs of one group overlap the drain of the previous one.
//   warps 2-9   epilogue: tcgen05.ld of its 32 lanes x 128 columns; residue form: the groups' residues
//               summed in packed FP32, and at each level end a TMA store of them as bytes (16 bits for
//               the modulus 257); digit form: exact int32 sums (float modes: the FP32 tile), stored to
//               the level planes in global memory.
// A separate kernel reconstructs C from the residue planes (crt_combine_kernel) or recombines the
// level sums, C = alpha * 2^(e_i+f_j) * sum_L 2^(-14-8L) T_L + beta*C in FP64 (float modes: alpha *
// sum of segment partials + beta*C).  Every wait is bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <cmath>
#include <string>
#include <type_traits>
#include <utility>
#include <vector>

#include "../../include/gb300_blas.h"
#include "gb300_internal.h"
#include "ptx.cuh"
#include "runtime.h"
#include "profile.h"
#include "split_api.h"
#include "crt_tables.h"

namespace gb {
namespace {

constexpr int TM = 128;                 // A rows held by each CTA of a pair
constexpr int TN = 256;                 // tile cols (pair MMA N)
constexpr int TMP = 2 * TM;             // rows of a CTA pair's tile (pair MMA M = 256)
constexpr int TNH = TN / 2;             // B rows (tile columns) held by each CTA of the pair
constexpr int TK = 64;                  // k per item (one 128-byte swizzle row of bf16)
constexpr int STAGES = 6;
constexpr int A_BYTES = TM * TK * 2;    // 16 KB
constexpr int B_BYTES = TNH * TK * 2;   // 16 KB (this CTA's half of the B tile)
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int GROUP_ITEMS = 16;         // exact mode: 16 items (1024 products) per TMEM drain
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + EPI_WARPS * 32;
constexpr int MAX_SLICES = 10;
constexpr int KSEG_UNIT = 256;          // k-segments are multiples of this
constexpr int kPipeMaxQ = 2;            // column blocks of B in the host-operand pipeline
constexpr int kPipeMaxEvents = 64;      // of a pipeline of P panels and Q column blocks, P + Q + 2 P Q + 1
constexpr uint32_t MAGIC_BITS = 0x4B400000u;  // bits of 1.5 * 2^23
constexpr float MAGIC = 12582912.0f;

enum Mode : int { kExact = 0, kBf16 = 1, kBf16x3 = 2, kCrt = 3 };

// ---- moduli of the CRT (Ozaki scheme II) form ----------------------------------------------------
// Pairwise coprime moduli <= 257, largest first: a residue in the symmetric range has |r| <= 128,
// so it is exactly a BF16 and a 1024-product group of residue products stays within 2^24, where
// every partial sum is an integer exact in the FP32 accumulator (the same exactness argument as
// for the digits).  Prime factors: 257; 2; 3,5,17; 11,23; 251; 13,19; 241;
// 239; 233; 229; 227; 223; 7,31; 211; 199.  Product of all 15: about 2^118.2.
constexpr int MAX_MODULI = 15;
__constant__ uint32_t c_mod[MAX_MODULI] = {257, 256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199};
// Running products of the moduli rounded to FP64: entry N for the first N (device copy).
__constant__ double c_mod_prod[MAX_MODULI + 1] = {
    0x1.0p+0, 0x1.0100000000000p+8, 0x1.0100000000000p+16, 0x1.fffe000000000p+23,
    0x1.f9fe060000000p+31, 0x1.f01c0fe200000p+39, 0x1.deab13530e000p+47, 0x1.c29f0d31302e0p+55,
    0x1.a4b27d50ebfafp+63, 0x1.7ee6740ea6c76p+71, 0x1.568425d11b306p+79, 0x1.2fb72d886b1bep+87,
    0x1.089090a9d54d5p+95, 0x1.c085153feb9d1p+102, 0x1.71adb083af327p+110, 0x1.1f5e04365d303p+118};
// What the product of the moduli must exceed the largest |T| by: 2^1.0875, just above 2.125.
constexpr double kModMargin = 0x1.1001cb22b792cp+1;
// log2 of the running products of the moduli (host-side copy for the worst-case plan).
constexpr double kModLog2[MAX_MODULI] = {8.00562, 8.0, 7.99435, 7.98299, 7.97154, 7.94837, 7.91289, 7.90087,
                                         7.86419, 7.83920, 7.82655, 7.80090, 7.76155, 7.72110, 7.63662};

// Residues on the FP32 pipe: a 56-bit integer U = sum_i w_i 2^(14 i) (14-bit chunks, i = 0..3) is
// congruent to x = w_0 + sum_{i>0} w_i K_i with K_i = 2^(14 i) mod p in the symmetric range
// (|K_i| <= 128), so |x| <= 16383 * 385 < 2^23 and every partial sum is an exact FP32 integer.
// q = rint(x fl(1/p)) is the nearest integer to x / p: the relative error 2^-24 of fl(1/p) moves
// x / p by less than 2^23 / p * 2^-24 = 0.5 / p, the smallest distance of x / p from a half
// integer for odd p (p = 256 is exact), so r = x - p q lies in [-p/2, p/2] and |r| <= 128.
__constant__ float c_modf[MAX_MODULI] = {257.f, 256.f, 255.f, 253.f, 251.f, 247.f, 241.f, 239.f,
                                         233.f, 229.f, 227.f, 223.f, 217.f, 211.f, 199.f};
__constant__ float c_modf_inv[MAX_MODULI] = {
    0x1.fe01fe0000000p-9f, 0x1.0000000000000p-8f, 0x1.0101020000000p-8f, 0x1.03091c0000000p-8f,
    0x1.0519800000000p-8f, 0x1.0953f40000000p-8f, 0x1.0fef020000000p-8f, 0x1.12358e0000000p-8f,
    0x1.1945380000000p-8f, 0x1.1e2ef40000000p-8f, 0x1.20b4700000000p-8f, 0x1.25e2280000000p-8f,
    0x1.2e025c0000000p-8f, 0x1.3698e00000000p-8f, 0x1.49539e0000000p-8f};
__constant__ float c_mod_k14[3][MAX_MODULI] = {
    {-64.f, 0.f, 64.f, -61.f, 69.f, 82.f, -4.f, -107.f, 74.f, -104.f, 40.f, 105.f, -108.f, -74.f, 66.f},
    {-16.f, 0.f, 16.f, -74.f, -8.f, 55.f, 16.f, -23.f, -116.f, 53.f, 11.f, 98.f, -54.f, -10.f, -22.f},
    {-4.f, 0.f, 4.f, -40.f, -50.f, 64.f, -64.f, 71.f, 37.f, -16.f, -14.f, 32.f, -27.f, -104.f, -59.f}};

// Device-side result of the pre-pass: the slice count and the bound it guarantees.
struct SplitInfo {
    int slices;           // S (digit mode); residue products N (CRT mode); planes per operand otherwise
    int nonfinite;        // inputs contained Inf/NaN
    double bound;         // a-priori normwise bound of the result
    double normA, normB;  // Frobenius norms
    double scaleA, scaleB;// ||2^e||_2, ||2^f||_2
    // CRT mode
    int beta;             // rows of A are rounded to beta-bit integers
    int beta_b;           // columns of B are rounded to beta_b-bit integers (= beta unless B is sliced
                          // ahead of A, in the panel pipeline for host operands)
    double qmaxB;         // largest column sum of squares of B relative to 2^(2f)
    double qmaxA;         // largest row sum of squares of A relative to 2^(2e) (block pipeline)
};

// ---- pre-pass ------------------------------------------------------------------------------
// Row statistics of a logical R x K operand X(r,p) = X[r*sr + p*sp]: e_r = frexp exponent of
// max |X(r,:)| (kNonFinite if the row holds Inf/NaN) and q_r = sum_p (X(r,p) * 2^-e_r)^2, the
// row's sum of squares relative to 2^(2 e_r) (so that norms of huge or tiny inputs stay finite), and
// from them the plan (SplitInfo).  All of it is one launch, stats_kernel: its blocks read 32-row x 64-k
// tiles (coalesced along whichever dimension is contiguous, like slice_kernel), the last block to
// finish a row block folds the partial sums of the row block's k-chunks into (e_r, q_r) and one
// RowPartial, and the last block of all plans from those.  The counters that find the last block are
// zero before the launch; no block waits for another.
constexpr int kNonFinite = 0x7fff;

// Operands stream through shared memory in tiles of 32 rows x 64 k, a few tiles per block
// (tiles_per_block), with two buffers filled by cp.async: the copies of the next tile are in flight
// while the current one is processed.
constexpr int TILE_KT = 8;  // at most

// A row of a tile buffer: 64 elements and 16 bytes, so that rows start on different banks.
template <typename TX>
constexpr uint32_t kTileRow = 64 * sizeof(TX) + 16;

// Whether an operand's rows are contiguous and 16-byte aligned.
template <typename TX>
__device__ __forceinline__ bool rows_vec(const TX* X, int64_t sr, int64_t sp) {
    return sp == 1 && (sr * int64_t(sizeof(TX))) % 16 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
}

// Issue the copies of tile `it` (k from 64 it) into the buffer at shared address sbuf, where
// off(rr, pp) places element (rr, pp), the elements of an aligned 16 bytes side by side; zeros outside
// R x K; one commit group per tile.  The copies are coalesced along whichever index of
// X(r, p) = X[r*sr + p*sp] is contiguous: eight elements a thread, a warp reading 32 consecutive ones,
// or, where rows_vec, 16 bytes at a time.  Addresses are formed anew for
// each tile: kept across tiles they spilled from the slicing's 80 registers (725 -> 879 us at 8192^3).
template <typename TX, typename Off>
__device__ __forceinline__ void tile_issue(uint32_t sbuf, const TX* X, int64_t R, int64_t K, int64_t sr, int64_t sp,
                                           bool vec, int64_t r0, int64_t it, Off off) {
    const int t = threadIdx.x;  // 256 threads
    const bool full = r0 + 32 <= R && it * 64 + 64 <= K;  // the whole tile lies inside the matrix
    if (vec) {
        constexpr int V = 16 / sizeof(TX), CH = 64 / V, STEP = 256 / CH;  // elements, chunks a row, rows a pass
        const int rr0 = t / CH, pp = V * (t % CH);
        const int64_t left = K - it * 64 - pp;
        const int bytes = full || left >= V ? 16 : left > 0 ? int(left) * int(sizeof(TX)) : 0;
        const TX* src = X + (r0 + rr0) * sr + it * 64 + pp;
#pragma unroll
        for (int i = 0; i < 32 / STEP; ++i) {
            const int n = full || r0 + rr0 + STEP * i < R ? bytes : 0;
            cp_async16(sbuf + off(rr0 + STEP * i, pp), n ? src + STEP * i * sr : X, n);
        }
    } else {
        const int rr0 = sp == 1 ? t >> 6 : t & 31, pp0 = sp == 1 ? t & 63 : t >> 5;
        const int drr = sp == 1 ? 4 : 0, dpp = sp == 1 ? 0 : 8;
        const TX* src = X + (r0 + rr0) * sr + (it * 64 + pp0) * sp;
        const int64_t di = sp == 1 ? 4 * sr : 8 * sp;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int rr = rr0 + i * drr, pp = pp0 + i * dpp;
            const bool ok = full || (r0 + rr < R && it * 64 + pp < K);
            if constexpr (sizeof(TX) == 8) cp_async8(sbuf + off(rr, pp), ok ? src + i * di : X, ok);
            else cp_async4(sbuf + off(rr, pp), ok ? src + i * di : X, ok);
        }
    }
    cp_async_commit();
}

// The bits of a float operand's element as a double (exact).
__device__ __forceinline__ unsigned long long widened_bits(uint32_t b) {
    const uint32_t mag = b & 0x7fffffffu;
    if (mag - 1u < 0x007fffffu || mag >= 0x7f800000u)  // subnormal, Inf, NaN
        return static_cast<unsigned long long>(__double_as_longlong(double(__uint_as_float(b))));
    const uint32_t hi = (b & 0x80000000u) | (mag ? (mag >> 3) + 0x38000000u : 0u);
    return ((unsigned long long)hi << 32) | (mag << 29);
}

// 2^x in FP32 for x <= 127, 0 below the normal range.
__device__ __forceinline__ float pow2f_or0(int x) { return x < -126 ? 0.f : __uint_as_float(uint32_t(x + 127) << 23); }

// Both operands of a product go through one launch: blocks with blockIdx.y < yb0 work on A (its
// rows), the others on B (its columns), so the two passes overlap on the device.
struct OperandPair {
    const void* X[2];  // double or float elements
    int64_t R[2], sr[2], sp[2];
    int* rexp[2];
    __nv_bfloat16* planes[2];
    int64_t rpad[2];
    unsigned yb0;  // row blocks of A
};

// 64-bit shifts whose counts above 63 give zero.
__device__ __forceinline__ unsigned long long shl64(unsigned long long v, int n) {
    unsigned long long r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
}
__device__ __forceinline__ unsigned long long shr64(unsigned long long v, int n) {
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
}

// v 2^x of a zero or normal v >= 0 for x <= 0, zero below the normal range: integer operations only (an
// FP64 instruction of a warp holds its SM quarter's FP64 pipe for 64 clocks).
__device__ __forceinline__ double down2(double v, int x) {
    const int hi = __double2hiint(v);
    return (hi >> 20) + x > 0 ? __hiloint2double(hi + x * (1 << 20), __double2loint(v)) : 0.0;
}

// A float sum (zero or normal, not negative) as a double.
__device__ __forceinline__ double widened_sum(float v) {
    return __longlong_as_double(static_cast<long long>(widened_bits(__float_as_uint(v))));
}

// Summary of 32 rows (or of many): Inf/NaN flag, largest exponent E of the rows with q > 0 (kNoRows
// when none), bits of the largest q (non-negative doubles order like integers), s = sum 2^(2(e - E)) and
// nrm = sum 2^(2(e - E)) q.  A block's sums of squares are FP32; everything summed from them is FP64, with
// the scalings by powers of two done on the exponents.
constexpr int kNoRows = -100000;
struct __align__(16) RowPartial {
    int bad, E;
    long long Qbits;
    double s, nrm;
    __device__ __forceinline__ double Q() const { return __longlong_as_double(Qbits); }
};

// The sum over the calling warp's lanes (all of them get it) of zero or normal doubles v 2^x >= 0,
// x <= 0, in integers: the 53-bit significands, five bits up, aligned to the largest exponent, lose less
// than 2^-58 of the largest term each, so the sum is within 2^-53 of itself before its one rounding,
// closer than a chain of FP64 additions.  One copy of the code: a launch runs it a few times a block, from
// a cold instruction cache.
__device__ __noinline__ double warp_sum(double v, int x) {
    const int f = max((__double2hiint(v) >> 20) + x, 0), F = __reduce_max_sync(0xffffffffu, f);
    const uint32_t hi = (uint32_t(__double2hiint(v)) & 0xfffffu) | 0x100000u;
    const unsigned long long t = f ? shr64((((unsigned long long)hi << 32) | uint32_t(__double2loint(v))) << 5, F - f) : 0ull;
    const unsigned a = __reduce_add_sync(0xffffffffu, unsigned(t) & 0xfffffu);
    const unsigned b = __reduce_add_sync(0xffffffffu, unsigned(t >> 20) & 0xfffffu);
    const unsigned c = __reduce_add_sync(0xffffffffu, unsigned(t >> 40));
    unsigned long long T = a + ((unsigned long long)b << 20) + ((unsigned long long)c << 40);  // 0 or 2^57 <= T < 2^63
    if (T == 0ull) return 0.0;
    const int sh = 11 - __clzll((long long)T);  // down to 53 bits, to nearest even
    T += (1ull << (sh - 1)) - 1ull + ((T >> sh) & 1ull);
    return __longlong_as_double((long long)((T >> sh) + ((unsigned long long)(sh + F - 6) << 52)));
}

__device__ __forceinline__ RowPartial merge(const RowPartial& a, const RowPartial& b) {
    RowPartial r;
    r.bad = a.bad | b.bad;
    r.E = max(a.E, b.E);
    r.Qbits = max(a.Qbits, b.Qbits);
    r.s = down2(a.s, 2 * (a.E - r.E)) + down2(b.s, 2 * (b.E - r.E));
    r.nrm = down2(a.nrm, 2 * (a.E - r.E)) + down2(b.nrm, 2 * (b.E - r.E));
    return r;
}

// The merge over the calling warp's lanes (all of them get it).
__device__ __forceinline__ RowPartial warp_merge(const RowPartial& v) {
    constexpr unsigned all = 0xffffffffu;
    RowPartial r;
    r.bad = __any_sync(all, v.bad);
    r.E = __reduce_max_sync(all, v.E);
    const unsigned hi = unsigned(v.Qbits >> 32), top = __reduce_max_sync(all, hi);
    const unsigned lo = __reduce_max_sync(all, hi == top ? unsigned(v.Qbits) : 0u);
    r.Qbits = (long long)(((unsigned long long)top << 32) | lo);
    r.s = warp_sum(v.s, 2 * (v.E - r.E));
    r.nrm = warp_sum(v.nrm, 2 * (v.E - r.E));
    return r;
}

// What the last block of a statistics launch plans.
enum PlanKind : int { kPlanProduct = 0, kPlanSide = 1 };
struct PlanArgs {
    int kind, mode, fixed_slices, cap_planes;
    double target;
    SplitInfo* info;
};

__device__ void plan_product(const RowPartial& A, const RowPartial& B, int64_t k, const PlanArgs& plan);
__device__ void plan_side(const RowPartial& S, int64_t k, const PlanArgs& plan);

struct StatsArgs {
    OperandPair op;
    int64_t K;
    int kt, chunks;        // k-tiles per block, blocks per row block
    uint2* part;           // chunks > 1: [rows of A, then of B][chunks] of (high word and low flag, sum)
    unsigned* count;       // one counter per row block, one for the launch; zero before the launch
    RowPartial* group;     // one per row block
    PlanArgs plan;
};

// Whether this block is the last of `n` to arrive at the counter (uniform over the block).  What the
// arriving blocks wrote before is visible to the last one.
__device__ __forceinline__ bool last_to_arrive(unsigned* counter, unsigned n) {
    __shared__ unsigned last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(counter, 1u) + 1u == n ? 1u : 0u;
    __syncthreads();
    if (last != 0u) __threadfence();
    return last != 0u;
}

// One thread's part of a statistics block: over row rr = t % 32 and the eight k of group g = t / 32 in
// every tile of [tb, te), the largest high word of |x| (mx), the OR of the low words (float: of the
// magnitudes; lo) and the sum of squares in FP32 relative to the exponent of mx (sq).
//
// The sum runs relative to the largest exponent so far, `base`: f = |x| 2^(1023 - base) is the high word
// times 8 (exponent and 20 mantissa bits moved into FP32 position) minus (base - 127) 2^23, one integer
// multiply-add, valid for exponents above base - 127.  High words below that are raised to its lowest
// value, whose square is zero in FP32.  `base` moves once per tile, and the sum is rescaled exactly by a
// power of two.  An Inf/NaN shows as a largest exponent of 0x7ff.  Bound by the integer ALU (73 % active at
// 4096^3): four operations an element, the maximum and the OR two elements at a time; with `base` checked at
// every element it was seven (1 GiB of operands 215 us, now 190).
//
// A float's high word as a double is its magnitude shifted by 3 with the exponent rebased.  A zero or
// subnormal float gets exponent field 896 that way, no matter next to a row's larger values; EXACT takes
// the high words of the widened values instead.
struct ThreadStats {
    uint32_t mx, lo;
    float sq;
};
template <typename TX, bool EXACT>
__device__ __forceinline__ ThreadStats scan_tiles(unsigned char* tbuf, const TX* __restrict__ X, int64_t R, int64_t K, int64_t sr,
                                                  int64_t sp, int64_t r0, int64_t tb, int64_t te) {
    constexpr bool F32 = sizeof(TX) == 4;
    constexpr uint32_t ROWB = kTileRow<TX>, BUF = 32 * ROWB;
    const int rr = threadIdx.x & 31, g = threadIdx.x >> 5;
    const uint32_t s0 = smem_u32(tbuf);
    const bool vec = rows_vec(X, sr, sp);
    auto off = [](int r_, int p_) { return uint32_t(r_) * ROWB + uint32_t(p_) * uint32_t(sizeof(TX)); };
    uint32_t mx = 0, lo = 0;
    float sq = 0.f;
    int base = 127;  // f = |x| 2^(1023 - base); values with exponent field 0 never count
    if (tb < te) tile_issue(s0, X, R, K, sr, sp, vec, r0, tb, off);
    for (int64_t it = tb; it < te; ++it) {
        const int b = int(it - tb) & 1;
        if (it + 1 < te) tile_issue(s0 + uint32_t(b ^ 1) * BUF, X, R, K, sr, sp, vec, r0, it + 1, off);
        else cp_async_commit();  // an empty group keeps the wait count uniform
        cp_async_wait1();
        __syncthreads();
        uint32_t hi[8];
        const unsigned char* row = tbuf + b * BUF + rr * ROWB + g * 8 * uint32_t(sizeof(TX));
        if constexpr (F32) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const uint4 v = *reinterpret_cast<const uint4*>(row + 16 * q);
                const uint32_t m4[4] = {v.x & 0x7fffffffu, v.y & 0x7fffffffu, v.z & 0x7fffffffu, v.w & 0x7fffffffu};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    hi[4 * q + i] = EXACT ? uint32_t(widened_bits(m4[i]) >> 32) : (m4[i] >> 3) + 0x38000000u;
                lo |= m4[0] | m4[1];
                lo |= m4[2] | m4[3];
                mx = max(mx, max(max(hi[4 * q], hi[4 * q + 1]), max(hi[4 * q + 2], hi[4 * q + 3])));
            }
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 v = *reinterpret_cast<const uint4*>(row + 16 * q);
                hi[2 * q] = v.y & 0x7fffffffu;
                hi[2 * q + 1] = v.w & 0x7fffffffu;
                lo |= v.x | v.z;
                mx = max(mx, max(hi[2 * q], hi[2 * q + 1]));
            }
        }
        const int top = int(mx >> 20);
        if (top > base) {
            sq *= pow2f_or0(2 * (base - top));
            base = top;
        }
        const uint32_t cbias = uint32_t(base - 127) << 23, least = uint32_t(base - 126) << 20;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float f = __uint_as_float(max(hi[q], least) * 8u - cbias);
            sq = fmaf(f, f, sq);
        }
        __syncthreads();
    }
    return {mx, lo, sq};
}
// Out of line: it is rarely run, and its registers and code stay out of the kernel's way.
template <typename TX>
__device__ __noinline__ ThreadStats scan_tiles_exact(unsigned char* tbuf, const TX* X, int64_t R, int64_t K, int64_t sr,
                                                     int64_t sp, int64_t r0, int64_t tb, int64_t te) {
    return scan_tiles<TX, true>(tbuf, X, R, K, sr, sp, r0, tb, te);
}

// The statistics of both operands and the plan, in one launch: scan_tiles per thread, folded per row block
// over its k-chunks, then over the row blocks.  Small operands are bound by the launches and by the serial
// folds and FP64 functions behind them: with the row totals in a kernel of their own (atomics and a memset
// before it) and the plan in another, these steps took 23 us of a 403 x 517 x 389 product and 26 of
// 1024^3, with the gaps between four launches beside them; this kernel takes 13 and 18.
//
// A float block with a row that has nothing above 2^-86 goes over its tiles again with EXACT; all-zero rows
// are known by their OR.
template <typename TX>
__global__ void __launch_bounds__(256, 4) stats_kernel(const StatsArgs a) {
    constexpr bool F32 = sizeof(TX) == 4;
    constexpr uint32_t ROWB = kTileRow<TX>, BUF = 32 * ROWB;  // an odd count of 16-byte chunks: no bank conflicts
    constexpr uint32_t kInfHi = F32 ? 0x47f00000u : 0x7ff00000u;
    constexpr uint32_t kTinyExp = 191u, kTinyF32Exp = 937u;
    __shared__ __align__(16) unsigned char tbuf[2 * BUF];
    __shared__ uint32_t red_mx[8][32];
    __shared__ float red_sq[8][32];
    griddep_launch();  // the slicing's first tiles may come in meanwhile
    const int w = blockIdx.y < a.op.yb0 ? 0 : 1;
    const int by = w ? int(blockIdx.y - a.op.yb0) : int(blockIdx.y);
    const TX* __restrict__ X = static_cast<const TX*>(a.op.X[w]);
    const int64_t R = a.op.R[w], sr = a.op.sr[w], sp = a.op.sp[w], K = a.K;
    const int t = threadIdx.x, rr = t & 31, g = t >> 5;
    const int64_t r0 = int64_t(by) * 32;
    const int64_t ntiles = (K + 63) / 64;
    const int64_t tb = int64_t(blockIdx.x) * a.kt, te = min(ntiles, tb + a.kt);
    // a row's largest high word with the low words' flag in bit 0, and its sum of squares relative to
    // the exponent of that high word (at least 127)
    auto exponent = [](uint32_t m) { return max(127, int(m >> 21)); };
    auto fold = [&](uint32_t& m, float& s) {  // the eight groups' values of row rr
        m = 0;
        uint32_t flag = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            m = max(m, red_mx[i][rr] & ~1u);
            flag |= red_mx[i][rr] & 1u;
        }
        m |= flag;
        const int E = exponent(m);
        s = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) s = fmaf(red_sq[i][rr], pow2f_or0(2 * (exponent(red_mx[i][rr]) - E)), s);
    };
    const int64_t r = r0 + rr;
    uint32_t m = 0;
    double s = 0.0;
    auto block_rows = [&](ThreadStats v) {  // m and s of the block's tiles
        if (F32 && v.lo == 0u) {
            v.mx = 0u;
            v.sq = 0.f;
        }
        red_mx[g][rr] = (v.mx << 1) | (v.lo != 0u ? 1u : 0u);
        red_sq[g][rr] = v.sq;
        __syncthreads();
        if (g == 0) {
            float sb;
            fold(m, sb);
            s = widened_sum(sb);
        }
    };
    block_rows(scan_tiles<TX, false>(tbuf, X, R, K, sr, sp, r0, tb, te));
    if constexpr (F32)
        if (__syncthreads_or(m != 0u && m < (kTinyF32Exp << 21)))
            block_rows(scan_tiles_exact<TX>(tbuf, X, R, K, sr, sp, r0, tb, te));
    if (a.chunks > 1) {
        uint2* rowpart = a.part + ((w ? a.op.R[0] : 0) + r) * a.chunks;
        if (g == 0 && r < R) rowpart[blockIdx.x] = make_uint2(m, __float_as_uint(float(s)));
        if (!last_to_arrive(a.count + blockIdx.y, unsigned(a.chunks))) return;
        double(*const red_s)[32] = reinterpret_cast<double(*)[32]>(tbuf);  // free by now
        m = 0;
        s = 0.0;
        uint32_t flag = 0;
        if (r < R)
            for (int c = g; c < a.chunks; c += 8) {  // fixed order: the sums do not depend on which block is last
                const uint2 v = __ldcg(rowpart + c);
                const double sc = widened_sum(__uint_as_float(v.y));
                const int E = exponent(m), Ec = exponent(v.x), top = max(E, Ec);
                s = c == g ? sc : down2(s, 2 * (E - top)) + down2(sc, 2 * (Ec - top));
                m = max(m, v.x & ~1u);
                flag |= v.x & 1u;
            }
        red_mx[g][rr] = m | flag;
        red_s[g][rr] = s;
        __syncthreads();
        if (g == 0) {
            m = 0;
            flag = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                m = max(m, red_mx[i][rr] & ~1u);
                flag |= red_mx[i][rr] & 1u;
            }
            m |= flag;
            const int E = exponent(m);
            s = down2(red_s[0][rr], 2 * (exponent(red_mx[0][rr]) - E));
#pragma unroll
            for (int i = 1; i < 8; ++i) s += down2(red_s[i][rr], 2 * (exponent(red_mx[i][rr]) - E));
        }
    }
    if (g == 0) {
        int e = 0;
        double q = 0.0;
        const uint32_t hi = m >> 1;
        if (r < R && m != 0u) {
            if (hi >= kInfHi) {
                e = kNonFinite;
            } else if (hi >= (kTinyExp << 20)) {
                e = int(hi >> 20) - 1022;
                q = down2(s, -2);  // |x| 2^-e = f / 2
            } else {
                // tiny or subnormal values, whose squares left the FP32 range: the row again, exactly
                unsigned long long mb = 0;
                for (int64_t p = 0; p < K; ++p) {
                    const unsigned long long v =
                        static_cast<unsigned long long>(__double_as_longlong(double(X[r * sr + p * sp]))) & 0x7fffffffffffffffull;
                    mb = v > mb ? v : mb;
                }
                frexp(__longlong_as_double(static_cast<long long>(mb)), &e);
                double d = 0.0;
                for (int64_t p = 0; p < K; ++p) {
                    const double v = ldexp(double(X[r * sr + p * sp]), -e);
                    d = fma(v, v, d);
                }
                q = d;
            }
        }
        if (r < R) a.op.rexp[w][r] = e;
        const long long qb = __double_as_longlong(q);
        const RowPartial pr = warp_merge(RowPartial{e == kNonFinite, qb > 0 ? e : kNoRows, qb, qb > 0 ? 1.0 : 0.0, q});
        if (t == 0) a.group[blockIdx.y] = pr;
    }
    if (!last_to_arrive(a.count + gridDim.y, gridDim.y)) return;
    // the plan, from every row block: warps 0-3 sum up A's, 4-7 B's
    __shared__ RowPartial side[8];
    const RowPartial none{0, kNoRows, 0, 0.0, 0.0};
    RowPartial acc = none;
    const unsigned first = (g < 4 ? 0u : a.op.yb0) + (t & 127), end = g < 4 ? a.op.yb0 : gridDim.y;
#pragma unroll 4
    for (unsigned i = first; i < end; i += 128) {
        const uint4* v = reinterpret_cast<const uint4*>(a.group + i);
        const uint4 lo4 = __ldcg(v), hi4 = __ldcg(v + 1);
        const RowPartial pr{int(lo4.x), int(lo4.y), (long long)(((unsigned long long)lo4.w << 32) | lo4.z),
                            __hiloint2double(int(hi4.y), int(hi4.x)), __hiloint2double(int(hi4.w), int(hi4.z))};
        acc = i == first ? pr : merge(acc, pr);
    }
    acc = warp_merge(acc);
    if (rr == 0) side[g] = acc;
    __syncthreads();
    if (g != 0) return;
    const RowPartial A = warp_merge(rr < 4 ? side[rr & 7] : none), B = warp_merge(rr >= 4 && rr < 8 ? side[rr & 7] : none);
    if (a.plan.kind == kPlanProduct) plan_product(A, B, K, a.plan);
    else plan_side(a.op.yb0 ? A : B, K, a.plan);
}

// The plans: norms, slice count and bound, by one warp.  Sums come relative to the largest
// row exponent, so the ratio rho = ||2^e|| ||2^f|| / (||A|| ||B||) is finite for any finite input.
//
// On GB300 every FP64 instruction of a warp holds its SM quarter's FP64 pipe for 64 clocks whatever the
// number of active lanes, so the plan keeps FP64 work off serial chains: each function runs once with
// a different argument in each lane, and the searches test 32 candidates per instruction.

// Smallest b in [lo, hi] with ok(b), hi + 1 when there is none (ok false, then true as b grows):
// the 32 lanes of the calling warp test 32 candidates at a time.
template <typename F>
__device__ int warp_first_true(int lo, int hi, F ok) {
    const int lane = threadIdx.x & 31;
    for (int base = lo; base <= hi; base += 32) {
        const int b = base + lane;
        const unsigned m = __ballot_sync(0xffffffffu, b <= hi && ok(b));
        if (m) return base + __ffs(int(m)) - 1;
    }
    return hi + 1;
}

// Largest b in [lo, hi] with ok(b), lo - 1 when there is none (ok true, then false as b grows).
template <typename F>
__device__ int warp_last_true(int lo, int hi, F ok) {
    const int lane = threadIdx.x & 31;
    for (int base = hi; base >= lo; base -= 32) {
        const int b = base - lane;
        const unsigned m = __ballot_sync(0xffffffffu, b >= lo && ok(b));
        if (m) return base - (__ffs(int(m)) - 1);
    }
    return lo - 1;
}

// 2^x for an integer x <= 0 from the bit pattern (0 below the normal range)
__device__ __forceinline__ double pow2i(int x) {
    return x < -1022 ? 0.0 : __longlong_as_double((long long)(x + 1023) << 52);
}

// The fewest moduli, two at least and `cap` at most, whose product is at least `need`.
__device__ __forceinline__ int moduli_for(double need, int cap) {
    const int first = warp_first_true(2, MAX_MODULI, [&](int n) { return c_mod_prod[n] >= need; });
    return max(2, min(cap, first));
}

// floor(log2 |x|) of a normal x.
__device__ __forceinline__ int exponent_of(double x) { return int((__double2hiint(x) >> 20) & 0x7ff) - 1023; }

__device__ void plan_product(const RowPartial& A, const RowPartial& B, int64_t k, const PlanArgs& plan) {
    const int lane = threadIdx.x & 31, EA = A.E, EB = B.E, bad = A.bad | B.bad;
    const double QA = A.Q(), QB = B.Q(), sa = A.s, na = A.nrm, sb = B.s, nb = B.nrm;
    const int mode = plan.mode, fixed_slices = plan.fixed_slices, cap_planes = plan.cap_planes;
    const double target = plan.target;
    // Each FP64 function below runs once for the warp with a different argument in each lane
    // (the cost of one evaluation, same operations as one at a time): lanes 0-3 the norms, 4-5
    // sqrt(k s / n), 6-7 sqrt(Q (1 + 2^-10)), 8 sqrt(k), 9-10 sqrt(s / n).
    double num = 1.0, den = 1.0;  // one, not zero, in the idle lanes: zeros take the functions' slow paths
    switch (lane) {
        case 0: num = na; break;
        case 1: num = nb; break;
        case 2: num = sa; break;
        case 3: num = sb; break;
        case 4: num = double(k) * sa; den = na > 0 ? na : 1.0; break;
        case 5: num = double(k) * sb; den = nb > 0 ? nb : 1.0; break;
        case 6: num = QA * (1.0 + 0x1p-10); break;
        case 7: num = QB * (1.0 + 0x1p-10); break;
        case 8: num = double(k); break;
        case 9: num = sa; den = na > 0 ? na : 1.0; break;
        case 10: num = sb; den = nb > 0 ? nb : 1.0; break;
        default: break;
    }
    const double root = sqrt(num / den);
    const double scaled = ldexp(root, (lane == 0 || lane == 2) ? EA : EB);  // lanes 0-3
    auto from = [&](double v, int l) { return __shfl_sync(0xffffffffu, v, l); };
    const double nA_ = from(scaled, 0), nB_ = from(scaled, 1), sA_ = from(scaled, 2), sB_ = from(scaled, 3);
    const double rAk = from(root, 4), rBk = from(root, 5), sqa = from(root, 6), sqb = from(root, 7);
    const double sqk = from(root, 8), ra = from(root, 9), rb = from(root, 10);
    SplitInfo r;
    r.nonfinite = bad;
    r.normA = (na > 0) ? nA_ : 0.0;
    r.normB = (nb > 0) ? nB_ : 0.0;
    r.scaleA = (sa > 0) ? sA_ : 0.0;
    r.scaleB = (sb > 0) ? sB_ : 0.0;
    const double rho = (na > 0 && nb > 0) ? ra * rb : 0.0;
    if (mode == kCrt) {
        // operands rounded to beta-bit integers: |dA_ip| <= 2^(e_i-beta-1), so
        // ||dC||_F/(||A|| ||B||) <= 2^(-beta-1)(rA + rB) + 2^(-2beta-2) rA rB + 2^-52 with
        // rA = sqrt(k) ||2^e|| / ||A|| (and 2^-52 for the final conversion and the alpha scaling)
        const double rA = (na > 0) ? rAk : 0.0;
        const double rB = (nb > 0) ? rBk : 0.0;
        auto bnd = [&](int b) {
            return pow2i(-b - 1) * (rA + rB) + pow2i(-2 * b - 2) * rA * rB + pow2i(-52);
        };
        // the smallest beta in [1, 55] that meets the target (beta <= 55 keeps |A'| < 2^56, the
        // range of the residue extraction); below `lo` the first term alone exceeds it
        int lo = 1;
        if (rA + rB > 0.0 && target > 0x1p-1000) lo = exponent_of(rA + rB) - exponent_of(target) - 2;
        int beta = min(55, warp_first_true(max(1, min(lo, 54)), 54, [&](int b) { return bnd(b) <= target; }));
        // The scaled rows satisfy ||A'_i|| <= 2^beta sqrt(Q_A) + sqrt(k)/2 (the rounding adds
        // at most 1/2 per entry), so by Cauchy-Schwarz every exact product entry T has
        // |T| <= (2^beta sqrt(Q_A) + sqrt(k)/2)(2^beta sqrt(Q_B) + sqrt(k)/2).  The moduli's
        // product P must exceed 2.125 |T| (symmetric residues, with room for the FP32 quotient
        // estimate of the reconstruction); Q carries a 2^-10 allowance for its own rounding.
        const double hk = 0.5 * sqk;
        auto need = [&](int b) {
            const double p2 = __hiloint2double((b + 1023) << 20, 0);
            return kModMargin * fma(sqa, p2, hk) * fma(sqb, p2, hk);
        };
        // a fixed count is used as given (at least two); otherwise the fewest that carry the
        // target, within the planes the host sized for
        const int N = fixed_slices > 0 ? max(2, fixed_slices) : moduli_for(need(beta), cap_planes);
        const double have = c_mod_prod[N];
        // the moduli chosen may carry more bits than needed: round to as many bits as they allow.
        // need(b) exceeds 2 4^b sqa sqb, so no b above b0 qualifies: the largest b in (-60, b0] with
        // need(b) <= have, -60 when none
        int bhi = 55;
        if (sqa > 0 && sqb > 0) {
            const int b0 = (exponent_of(have) - exponent_of(sqa) - exponent_of(sqb)) >> 1;
            bhi = b0 < 55 ? (b0 > -60 ? b0 : -60) : 55;
        }
        beta = warp_last_true(-59, bhi, [&](int b) { return need(b) <= have; });
        r.slices = N;
        r.beta = beta;
        r.beta_b = beta;
        r.qmaxB = QB;
        // a beta the search found has need(beta) <= have; -60 (none found) was not tested.  Too
        // few moduli for even the coarsest rounding: no bound
        const bool fits = beta >= -59 || need(beta) <= have;
        r.bound = fits ? bnd(beta) : __longlong_as_double(0x7ff0000000000000ll);
    } else if (mode == kExact) {
        int S = fixed_slices;
        if (S <= 0) {
            S = MAX_SLICES;
            for (int s = 2; s <= MAX_SLICES; ++s) {
                const double b = (s + 1) * double(k) * ldexp(1.0, -8 * s) * rho + (s + 3) * ldexp(1.0, -53);
                if (b <= target) { S = s; break; }
            }
        }
        r.slices = S;
        r.bound = (S + 1) * double(k) * ldexp(1.0, -8 * S) * rho + (S + 3) * ldexp(1.0, -53);
    } else if (mode == kBf16) {
        // each operand rounded to 8 significant bits, FP32 accumulation
        r.slices = 1;
        r.bound = 2.0 * ldexp(1.0, -8) + double(k) * ldexp(1.0, -24);
    } else {
        // hi/lo split keeps 16 bits; the dropped lo*lo term and the FP32 accumulation remain
        r.slices = 2;
        r.bound = 3.0 * ldexp(1.0, -16) + double(k) * ldexp(1.0, -24);
    }
    if (lane == 0) *plan.info = r;
}

// One operand side of a block of the host pipeline (a row panel of A or a column block of B): its
// norms and largest relative sum of squares (stored in both the A and the B fields), and the
// smallest beta with 2^(-beta-1) r <= target / 2: each side takes half of the bound for its own
// rounding, so the two sides are sliced independently.  `slices` = the planes the side is sliced
// into (the host's largest modulus count).
__device__ void plan_side(const RowPartial& S, int64_t k, const PlanArgs& plan) {
    const int lane = threadIdx.x & 31;
    const double s = S.s, nrm = S.nrm;
    // lane 0 the norm, 1 the scale, 2 sqrt(k s / nrm)
    const double root = sqrt((lane == 0 ? nrm : lane == 1 ? s : double(k) * s) / (lane == 2 && nrm > 0 ? nrm : 1.0));
    const double scaled = ldexp(root, S.E);
    SplitInfo r;
    r.nonfinite = S.bad;
    r.normA = r.normB = nrm > 0 ? __shfl_sync(0xffffffffu, scaled, 0) : 0.0;
    r.scaleA = r.scaleB = s > 0 ? __shfl_sync(0xffffffffu, scaled, 1) : 0.0;
    r.qmaxA = r.qmaxB = S.Q();
    const double rr = nrm > 0 ? __shfl_sync(0xffffffffu, root, 2) : 0.0;
    int lo = 1;
    if (rr > 0.0 && plan.target > 0x1p-1000) lo = exponent_of(rr) - exponent_of(plan.target) - 1;
    r.beta = r.beta_b = min(55, warp_first_true(max(1, min(lo, 54)), 54,
                                                [&](int b) { return pow2i(-b - 1) * rr <= 0.5 * plan.target; }));
    r.slices = plan.cap_planes;
    r.bound = 0.0;
    if (lane == 0) *plan.info = r;
}

// A block (row panel i of A, column block j of B) from the two sides: the moduli that carry
// (2^beta_a sqrt(Q_A) + sqrt(k)/2)(2^beta_b sqrt(Q_B) + sqrt(k)/2) with the margin of
// plan_product, and the block's bound 2^(-beta_a-1) r_A + 2^(-beta_b-1) r_B +
// 2^(-beta_a-beta_b-2) r_A r_B + 2^-52 relative to ||A_i|| ||B_j|| (infinite when even cap_planes
// moduli are too few).
__global__ void split_block_kernel(const SplitInfo* __restrict__ ia, const SplitInfo* __restrict__ ib, int64_t k,
                                   int cap_planes, SplitInfo* out) {
    const SplitInfo A = *ia, B = *ib;
    SplitInfo r;
    r.nonfinite = A.nonfinite | B.nonfinite;
    r.normA = A.normA;
    r.scaleA = A.scaleA;
    r.qmaxA = A.qmaxA;
    r.normB = B.normB;
    r.scaleB = B.scaleB;
    r.qmaxB = B.qmaxB;
    // lanes 0, 1: r_A and r_B; 2, 3: the square roots of the Qs; 4: sqrt(k), one evaluation each
    const int lane = threadIdx.x;
    const double root = sqrt(lane == 2 ? A.qmaxA * (1.0 + 0x1p-10) : lane == 3 ? B.qmaxB * (1.0 + 0x1p-10) : double(k));
    const double ratio = lane == 0 ? (A.normA > 0 ? A.scaleA / A.normA : 0.0) : (B.normB > 0 ? B.scaleB / B.normB : 0.0);
    auto from = [&](double v, int l) { return __shfl_sync(0xffffffffu, v, l); };
    const double rA = from(root * ratio, 0), rB = from(root * ratio, 1);
    const int ba = A.beta, bb = B.beta_b;
    const double hk = 0.5 * from(root, 4);
    const double need = kModMargin * (ldexp(from(root, 2), ba) + hk) * (ldexp(from(root, 3), bb) + hk);
    const int N = moduli_for(need, cap_planes);
    const double have = c_mod_prod[N];
    r.slices = N;
    r.beta = ba;
    r.beta_b = bb;
    r.bound = need > have ? __longlong_as_double(0x7ff0000000000000ll)
                          : pow2i(-ba - 1) * rA + pow2i(-bb - 1) * rB + pow2i(-ba - bb - 2) * rA * rB + pow2i(-52);
    if (lane == 0) *out = r;
}

// The level count of a launch that covers several blocks of one panel: the largest of its blocks'
// (each block's reconstruction reads its own count of levels; the launch reads only the count).
// Infos `stride` bytes apart.
__global__ void split_max_slices_kernel(const uint8_t* __restrict__ infos, size_t stride, int count,
                                        SplitInfo* __restrict__ out) {
    if (threadIdx.x != 0) return;
    SplitInfo r = *reinterpret_cast<const SplitInfo*>(infos);
    for (int i = 1; i < count; ++i)
        r.slices = max(r.slices, reinterpret_cast<const SplitInfo*>(infos + size_t(i) * stride)->slices);
    *out = r;
}

// Summary of the blocks for the caller: the largest modulus count and bound.
__global__ void split_panels_summary_kernel(const uint8_t* __restrict__ infos, size_t stride, int count,
                                            SplitInfo* out) {
    if (threadIdx.x != 0) return;
    SplitInfo r = *reinterpret_cast<const SplitInfo*>(infos);
    for (int i = 1; i < count; ++i) {
        const SplitInfo& x = *reinterpret_cast<const SplitInfo*>(infos + size_t(i) * stride);
        r.slices = max(r.slices, x.slices);
        r.bound = fmax(r.bound, x.bound);
        r.nonfinite |= x.nonfinite;
    }
    *out = r;
}

// Digit planes: planes[a][r][p] (bf16, pitch kpad, plane stride rpad*kpad) for r < rpad, p < kpad;
// zeros outside the R x K operand.  Each block covers 32 rows x 64 k.
//
// Exact mode: for |a| < 2^e (e the row exponent) the fixed-point integer
// X = round(|a| * 2^(8S-1-e)) (round half up below the last digit) satisfies X <= 2^(8S-1); its
// balanced base-256 digits d_S..d_2 in [-128, 127] and the top digit d_1 in [0, 128] give
// |a| * 2^-e = sum_s d_s 2^(1-8s) + rho, |rho| <= 2^-8S.  Everything is integer arithmetic on the
// FP64 bit pattern (64-bit for S <= 8, 128-bit beyond); digits become BF16 bit patterns through an
// exact FP32 add.  Float modes: BF16 hi part and BF16 rounding of the remainder.
__device__ __forceinline__ uint16_t digit_bf16(int d) {
    // float(d) exactly via the 1.5*2^23 bias; |d| <= 128 has at most 8 significant bits, so the
    // upper half of the FP32 pattern is the BF16 pattern
    const float f = __int_as_float(0x4B400000 + d) - 12582912.0f;
    return uint16_t(__float_as_uint(f) >> 16);
}

// Fixed-point magnitude V = X + sum_{s<S-1} 128*256^s of one element: with it, the balanced digit of
// plane a >= 1 is byte (S-1-a) of V minus 128 and the top digit (plane 0) is V >> 8(S-1); adding the
// 128s once replaces the digit-by-digit carry chain.
template <typename U_t>
__device__ __forceinline__ U_t fixed_point_biased(unsigned long long bits, int e, int S) {
    const int eb = int((bits >> 52) & 0x7ff);
    const unsigned long long mant = bits & 0xfffffffffffffull;
    const unsigned long long M = eb ? (mant | (1ull << 52)) : mant;
    const int E = (eb ? eb : 1) - 1075;  // |a| = M * 2^E
    const int sh = E + 8 * S - 1 - e;
    U_t U;
    if (M == 0) U = 0;
    else if (sh >= 0) U = U_t(M) << sh;
    else if (sh > -64) U = U_t((M + (1ull << (-sh - 1))) >> (-sh));
    else U = 0;
    U_t B = 0;
    for (int s = 0; s < S - 1; ++s) B = (B << 8) | 0x80;
    return U + B;
}

template <typename U_t>
__device__ __forceinline__ void write_planes(const U_t (&V)[8], const bool (&neg)[8], int S, uint16_t* dst,
                                             int64_t pstride) {
    for (int a = 0; a < S; ++a) {
        const int sft = 8 * (S - 1 - a);
        __align__(16) uint16_t d[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            int v = int(uint32_t(V[q] >> sft) & (a == 0 ? 0x1ffu : 0xffu));
            if (a != 0) v -= 128;
            d[q] = digit_bf16(neg[q] ? -v : v);
        }
        *reinterpret_cast<uint4*>(dst + a * pstride) = *reinterpret_cast<const uint4*>(d);
    }
}

// |round(a * 2^sh)| for a finite double given by its bits (round half up); the result must fit in
// 56 bits, which the CRT plan guarantees (beta <= 55 and |a| < 2^e).  The mantissa, 10 bits up (below
// 2^63), goes down by n = 10 minus its exponent, from n = 64 on to zero; n is at least 8 for normal
// numbers, and only a subnormal one in a row of subnormals goes up instead.
__device__ __forceinline__ unsigned long long int_magnitude(unsigned long long bits, int sh_total) {
    const int eb = int((bits >> 52) & 0x7ff);
    const unsigned long long M = (bits & 0xfffffffffffffull) | (eb ? 1ull << 52 : 0ull);
    const int n = 1085 - max(eb, 1) - sh_total;
    if (n <= 0) return shl64(M << 10, -n);
    return shr64((M << 10) + shl64(1ull, n - 1), n);
}

// x mod p for x < 2^32 and p <= 257 with inv = floor(2^32 / p): the quotient estimate is at most
// one short, so one conditional subtraction finishes the reduction.
__device__ __forceinline__ uint32_t mod_small(uint32_t x, uint32_t p, uint32_t inv) {
    const uint32_t q = uint32_t((uint64_t(x) * inv) >> 32);
    uint32_t r = x - q * p;
    return r >= p ? r - p : r;
}

// A modulus' constants as packed pairs (k_3, k_2, k_1 = symmetric residues of 2^42, 2^28, 2^14;
// fl(1/p); -p), in shared memory: three 16-byte reads a modulus serve eight elements, and the packed
// arithmetic takes half the instructions that bound this pass.  The planes' writes bound it now (DRAM 71 %
// busy at 4096^3): 8192^3 at 12 moduli 750 us before, now 690, 6.1 TB/s; 403 x 517 x 389 20, now 7, with
// the smaller blocks of tiles_per_block.
struct __align__(16) SliceConst {
    ulonglong2 k32, k1_inv, pneg;
};

// Planes of eight consecutive elements xv of one row (row exponent e, bad: the row holds Inf/NaN)
// at dst, plane stride pstride; sl = slices (digits) or moduli (CRT), bt = beta (CRT).
template <int mode>
__device__ __forceinline__ void slice_emit(const unsigned long long (&xv)[8], int sl, int bt, int e, bool bad,
                                           const SliceConst* tab, uint16_t* __restrict__ dst, int64_t pstride) {
    if (mode == kCrt) {
        const int N = sl, beta = bt;
        // U = |round(a 2^(beta-e))| < 2^56 in signed FP32 chunks (the sign of a applied to each), two
        // elements to a packed pair.  H = 2 U + (0 or 1): the mantissa with its implicit bit, 3 bits up,
        // goes down to one bit below the rounding point, and adding one there rounds half up; counts
        // above 63 leave nothing.  A zero or subnormal element of such a row ends there too; a row of
        // numbers below 2^-960 takes the general int_magnitude.  About twenty integer
        // instructions an element.
        // (Rows with Inf / NaN have e = kNonFinite and come out as zeros.)
        uint64_t w0[4], w1[4], w2[4], w3[4];
        unsigned long long Hs[8];
        if (e < -960) {
#pragma unroll
            for (int q = 0; q < 8; ++q) Hs[q] = int_magnitude(xv[q], beta - e) << 1;
        } else {
            const int down = 1077 - beta + e;  // shift count for a biased exponent of zero
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint32_t hi = uint32_t(xv[q] >> 32), lo = uint32_t(xv[q]);
                const uint32_t vh = (__funnelshift_l(lo, hi, 3) & 0x007fffffu) | 0x00800000u;
                Hs[q] = shr64(((unsigned long long)vh << 32) | (lo << 3), down - int((hi >> 20) & 0x7ffu)) + 1ull;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint32_t c[4][2], sign[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const unsigned long long H = Hs[2 * q + h];
                const uint32_t hi = uint32_t(xv[2 * q + h] >> 32);
                const uint32_t hh = uint32_t(H >> 32), hl = uint32_t(H);
                sign[h] = hi & 0x80000000u;
                c[0][h] = 0x4B000000u | ((hl >> 1) & 0x3fffu);
                c[1][h] = 0x4B000000u | ((hl >> 15) & 0x3fffu);
                c[2][h] = 0x4B000000u | (__funnelshift_r(hl, hh, 29) & 0x3fffu);
                c[3][h] = 0x4B000000u | (hh >> 11);
            }
            // chunk c = 2^23 + w: +-(c - 2^23)
            const uint64_t sg2 = f32x2_bits(0x3f800000u | sign[0], 0x3f800000u | sign[1]);
            const uint64_t off2 = f32x2_bits(0xcb000000u ^ sign[0], 0xcb000000u ^ sign[1]);
            w0[q] = fma2(f32x2_bits(c[0][0], c[0][1]), sg2, off2);
            w1[q] = fma2(f32x2_bits(c[1][0], c[1][1]), sg2, off2);
            w2[q] = fma2(f32x2_bits(c[2][0], c[2][1]), sg2, off2);
            w3[q] = fma2(f32x2_bits(c[3][0], c[3][1]), sg2, off2);
        }
        const uint64_t magic = f32x2(MAGIC, MAGIC), nmagic = f32x2(-MAGIC, -MAGIC);
#pragma unroll 1
        for (int t = 0; t < N; ++t) {
            const ulonglong2 k32 = tab[t].k32, k1i = tab[t].k1_inv;
            const uint64_t pneg = tab[t].pneg.x;
            uint32_t d[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint64_t x = fma2(w3[q], k32.x, fma2(w2[q], k32.y, fma2(w1[q], k1i.x, w0[q])));
                const uint64_t qf = add2(fma2(x, k1i.y, magic), nmagic);
                // exact symmetric residue, an integer of at most 8 significant bits: its FP32
                // pattern's upper half is the BF16 pattern
                const uint64_t f = fma2(pneg, qf, x);
                d[q] = __byte_perm(uint32_t(f), uint32_t(f >> 32), 0x7632);
            }
            *reinterpret_cast<uint4*>(dst + t * pstride) = make_uint4(d[0], d[1], d[2], d[3]);
        }
    } else if (mode == kExact) {
        const int S = sl;
        bool neg[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) neg[q] = !bad && (xv[q] >> 63) != 0;
        if (S <= 8) {
            unsigned long long V[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) V[q] = fixed_point_biased<unsigned long long>(bad ? 0ull : xv[q], e, S);
            write_planes(V, neg, S, dst, pstride);
        } else {
            unsigned __int128 V[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) V[q] = fixed_point_biased<unsigned __int128>(bad ? 0ull : xv[q], e, S);
            write_planes(V, neg, S, dst, pstride);
        }
    } else {
        __align__(16) __nv_bfloat16 hi[8], lo[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double x = __longlong_as_double(static_cast<long long>(xv[q]));
            hi[q] = __float2bfloat16_rn(float(x));
            lo[q] = __float2bfloat16_rn(float(x - double(__bfloat162float(hi[q]))));
        }
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(hi);
        if (mode == kBf16x3) *reinterpret_cast<uint4*>(dst + pstride) = *reinterpret_cast<const uint4*>(lo);
    }
}

// Planes of 32 rows over kt k-tiles.  Thread (rr = t / 8, L = t % 8) handles elements
// 8L..8L+7 of row rr and writes 16 bytes per plane (a warp: four 128-byte row segments).  The tile
// buffer keeps rows of 528 bytes with 16-byte chunk c of a row stored at c ^ (c >> 3), so that the
// eight threads of a row read their chunks 4L + j from eight different bank groups.
template <int mode, typename TX>
__device__ __forceinline__ void slice_rows(int which, const TX* X, int64_t R, int64_t K, int64_t sr, int64_t sp,
                                           const int* rexp, const SplitInfo* info, __nv_bfloat16* planes, int64_t rpad,
                                           int64_t kpad, int by, int kt) {
    constexpr uint32_t ROWB = kTileRow<TX>, BUF = 32 * ROWB, V = 16 / sizeof(TX);
    __shared__ __align__(16) unsigned char tbuf[2 * BUF];
    __shared__ SliceConst tab[mode == kCrt ? MAX_MODULI : 1];
    const int t = threadIdx.x, rr = t >> 3, L = t & 7;
    if (mode == kCrt && t < MAX_MODULI) {  // visible after the first tile's barrier
        auto two = [](float v) { return f32x2(v, v); };
        tab[t].k32 = make_ulonglong2(two(c_mod_k14[2][t]), two(c_mod_k14[1][t]));
        tab[t].k1_inv = make_ulonglong2(two(c_mod_k14[0][t]), two(c_modf_inv[t]));
        tab[t].pneg = make_ulonglong2(two(-c_modf[t]), 0ull);
    }
    const int64_t r0 = int64_t(by) * 32, r = r0 + rr;
    const int64_t ntiles = kpad / 64;
    const int64_t tb = int64_t(blockIdx.x) * kt, te = min(ntiles, tb + kt);
    const uint32_t s0 = smem_u32(tbuf);
    auto off = [](int r_, int p_) {
        const uint32_t c = uint32_t(p_) / V;
        return uint32_t(r_) * ROWB + ((c ^ (c >> 3)) << 4) + (uint32_t(p_) % V) * uint32_t(sizeof(TX));
    };
    const int64_t pstride = rpad * kpad;
    const bool vec = rows_vec(X, sr, sp);
    if (tb < te) tile_issue(s0, X, R, K, sr, sp, vec, r0, tb, off);
    // the operand is the caller's and was there before; the plan, the exponents and the planes (which
    // an earlier product may still be reading) have to wait
    griddep_launch();
    griddep_wait();
    const int sl = (mode == kExact || mode == kCrt) ? info->slices : 0;
    const int bt = (mode == kCrt) ? (which ? info->beta_b : info->beta) : 0;
    const int e = (r < R) ? rexp[r] : 0;
    const bool bad = (mode == kExact || mode == kCrt) && e == kNonFinite;
    for (int64_t it = tb; it < te; ++it) {
        const int b = int(it - tb) & 1;
        if (it + 1 < te) tile_issue(s0 + uint32_t(b ^ 1) * BUF, X, R, K, sr, sp, vec, r0, it + 1, off);
        else cp_async_commit();  // an empty group keeps the wait count uniform
        cp_async_wait1();
        __syncthreads();
        unsigned long long xv[8];
#pragma unroll
        for (int j = 0; j < int(8 / V); ++j) {
            const uint32_t c = uint32_t(8 / V * L + j);
            const uint4 v = *reinterpret_cast<const uint4*>(tbuf + b * BUF + rr * ROWB + ((c ^ (c >> 3)) << 4));
            if constexpr (sizeof(TX) == 8) {
                xv[2 * j] = (unsigned long long)v.x | ((unsigned long long)v.y << 32);
                xv[2 * j + 1] = (unsigned long long)v.z | ((unsigned long long)v.w << 32);
            } else {
                xv[4 * j] = widened_bits(v.x);
                xv[4 * j + 1] = widened_bits(v.y);
                xv[4 * j + 2] = widened_bits(v.z);
                xv[4 * j + 3] = widened_bits(v.w);
            }
        }
        if (r < rpad)
            slice_emit<mode>(xv, sl, bt, e, bad, tab, reinterpret_cast<uint16_t*>(planes) + r * kpad + it * 64 + 8 * L,
                             pstride);
        __syncthreads();
    }
}

// The operands are indexed by the block's side where the parameters lie (__grid_constant__): each thread
// otherwise copied the 120 bytes to its stack first, 3 to 4 us of a product of a few hundred rows.
template <int MODE, typename TX>
__global__ void __launch_bounds__(256, 3) slice_kernel(const __grid_constant__ OperandPair op, int64_t K,
                                                       const SplitInfo* info, int64_t kpad, int kt) {
    const int w = blockIdx.y < op.yb0 ? 0 : 1;
    const int by = w ? int(blockIdx.y - op.yb0) : int(blockIdx.y);
    slice_rows<MODE, TX>(w, static_cast<const TX*>(op.X[w]), op.R[w], K, op.sr[w], op.sp[w], op.rexp[w], info, op.planes[w],
                         op.rpad[w], kpad, by, kt);
}

// ---- level / pair schedule ---------------------------------------------------------------------
__device__ __forceinline__ int num_levels(int mode, int S) { return (mode == kExact || mode == kCrt) ? S : 1; }
__device__ __forceinline__ int pairs_in_level(int mode, int L) {
    return mode == kExact ? L + 1 : (mode == kBf16x3 ? 3 : 1);
}
// (A plane, B plane) of pair `i` of level `L`.
__device__ __forceinline__ void pair_planes(int mode, int L, int i, int& a, int& b) {
    if (mode == kExact) { a = i; b = L - i; }
    else if (mode == kCrt) { a = L; b = L; }
    else if (mode == kBf16) { a = 0; b = 0; }
    else { a = (i == 2) ? 1 : 0; b = (i == 1) ? 1 : 0; }
}

struct TcParams {
    int mode;
    int m_tiles, n_tiles, nseg;
    int kb_per_seg;          // 64-wide k-blocks per segment
    int kb_total;            // 64-wide k-blocks in the padded K
    int64_t mpad, npad;      // padded rows of the A / B planes
    int32_t* levels;         // [nseg][nlevels][mpad][npad] int32 (float modes: fp32 bits); kCrt: the
                             // residue planes described at crt_plane
    int max_levels;          // level dimension of `levels`
    int band = 8;            // m-tiles per band of the unit order (2..32 measured alike at 8192^3)
    int tn0 = 0;             // first n-tile of this launch (a product launched in column parts)
    const SplitInfo* info;
    int* status;
    uint64_t limit_ns;
    int inject_stall;
};

struct __align__(8) TcBarriers {
    uint64_t full[STAGES];
    uint64_t empty[STAGES];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint64_t drain;
    uint32_t tmem_base;
};

// Residue (CRT) level tiles leave through a per-warp staging tile (32 rows x 128 bytes, 128-byte
// swizzle) and a TMA store: full-line writes instead of 32 rows per store instruction.
constexpr int OUT_WARP_BYTES = 32 * 128;
constexpr int OUT_BYTES = EPI_WARPS * OUT_WARP_BYTES;
constexpr size_t kTcSmem = size_t(STAGES) * STAGE_BYTES + OUT_BYTES + sizeof(TcBarriers) + 1024;

__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= uint64_t((saddr & 0x3FFFFu) >> 4);     // start address
    d |= uint64_t(1) << 16;                      // leading byte offset (unused for 128B swizzle)
    d |= uint64_t(1024 >> 4) << 32;              // stride byte offset: 8 rows x 128 B
    d |= uint64_t(1) << 46;                      // descriptor version (tcgen05)
    d |= uint64_t(2) << 61;                      // 128-byte swizzle
    return d;
}

// kind::f16 instruction descriptor: BF16 A and B (K-major), FP32 D, M = 256 (a CTA pair), N = 256.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(TN >> 3) << 17) | (uint32_t(TMP >> 4) << 24);

// Work unit u -> (level, tile m, tile n, segment): one level (a modulus, or the slice pairs of a
// digit level) of one pair tile, the level varying slowest so that concurrent pairs share the
// operand planes of one level in L2, with 8 m-tiles per band.  Units of one level have equal
// lengths, and many small units keep the last wave short.
__device__ __forceinline__ void unit_coords(const TcParams& p, int u, int& tm, int& tn, int& seg, int& L) {
    const int per_level = p.m_tiles * p.n_tiles * p.nseg;
    L = u / per_level;
    u -= L * per_level;
    seg = u % p.nseg;
    const int t = u / p.nseg;
    const int band = p.band;
    const int per_band = band * p.n_tiles;
    const int b = t / per_band, r = t % per_band;
    const int rows_in_band = min(band, p.m_tiles - b * band);
    tm = b * band + r % rows_in_band;
    tn = p.tn0 + r / rows_in_band;
}

// Residues of two FP32 integers |x| <= 2^24 modulo p: q = rint(x fl(1/p)) is within one of x / p's
// nearest integer (fl(1/p) is off by at most 2^-24 relative, x / p by at most 1 / p, so only an x
// next to a half multiple of p can round the other way), and r = x - p q, an integer of at most
// (p + 1) / 2 in magnitude, is exact.  For |x| < 2^23, r is the symmetric residue, |r| <= p / 2.  Four
// packed instructions for two outputs; converting each group sum to an integer and reducing the
// total modulo p in integers took about twelve an output, which paced every unit of few k steps
// (65536 x 256 x 256: 222 us in this kernel, now 140; 8192 x 8192 x 8192:
// 7.20 -> 6.59 ms, 2.0 PFLOP/s).
__device__ __forceinline__ uint64_t residue2(uint64_t x, uint64_t pinv2, uint64_t pneg2) {
    const uint64_t magic = f32x2(MAGIC, MAGIC), nmagic = f32x2(-MAGIC, -MAGIC);
    const uint64_t q = add2(fma2(x, pinv2, magic), nmagic);
    return fma2(pneg2, q, x);
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __maxnreg__(168)
tc_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmC0, const __grid_constant__ CUtensorMap tmC, const TcParams p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* out_stage = smem + STAGES * STAGE_BYTES;
    TcBarriers* bars = reinterpret_cast<TcBarriers*>(out_stage + OUT_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // CTA pair: both CTAs walk the same units; the even CTA issues the pair MMAs, each CTA loads its
    // 128 rows of A and its half of B and drains its own 128 TMEM lanes
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;
    const int pair = int(blockIdx.x >> 1), npairs = int(gridDim.x >> 1);

    // the epilogue's arithmetic is fixed at compile time: residues, exact integer sums or FP32 tiles
    constexpr int mode = MODE;
    griddep_launch();
    if (threadIdx.x == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        if (mode == kCrt) {
            tma_prefetch_desc(&tmC0);
            tma_prefetch_desc(&tmC);
        }
        // full: the even CTA's arm plus both CTAs' bytes; empty / acc_full: one pair-MMA commit
        // (multicast to both CTAs); acc_empty (even CTA): every epilogue warp of both CTAs
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&bars->full[s]), 1);
            mbar_init(smem_u32(&bars->empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&bars->acc_full[b]), 1);
            mbar_init(smem_u32(&bars->acc_empty[b]), 2 * EPI_WARPS);
        }
        mbar_init(smem_u32(&bars->drain), 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        __syncwarp();
        tmem_alloc_pair(smem_u32(&bars->tmem_base), 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    // barriers of both CTAs initialised before any cross-CTA arrival or copy
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    // everything above overlaps the slicing; the plan and the planes are ready from here on
    griddep_wait();
    const int S = (mode == kExact || mode == kCrt) ? p.info->slices : 1;
    const int nlev = num_levels(mode, S);
    const int units = p.m_tiles * p.n_tiles * p.nseg * nlev;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0 && !p.inject_stall) {
            fence_proxy_async();
            uint32_t it = 0;
            bool ok = true;
            for (int u = pair; u < units && ok; u += npairs) {
                int tm, tn, seg, Lu;
                unit_coords(p, u, tm, tn, seg, Lu);
                const int kb0 = seg * p.kb_per_seg;
                const int kbn = min(p.kb_per_seg, p.kb_total - kb0);
                {
                    const int L = Lu;
                    const int np = pairs_in_level(mode, L);
                    for (int kb = 0; kb < kbn && ok; ++kb) {
                        for (int i = 0; i < np; ++i, ++it) {
                            const int s = it % STAGES;
                            if (it >= STAGES &&
                                !mbar_wait(smem_u32(&bars->empty[s]), ((it / STAGES) - 1) & 1, p.status,
                                           kDevTimeoutEmpty, p.limit_ns)) {
                                ok = false;
                                break;
                            }
                            int a, b;
                            pair_planes(mode, L, i, a, b);
                            // both CTAs' bytes complete on the even CTA's full barrier, armed there
                            // for the two halves
                            const uint32_t full_local = smem_u32(&bars->full[s]);
                            if (leader) mbar_arrive_expect_tx(full_local, 2 * STAGE_BYTES);
                            const uint32_t full = mapa_shared(full_local, 0);
                            const uint32_t dst = smem_u32(smem + s * STAGE_BYTES);
                            const int32_t kx = (kb0 + kb) * TK;
                            tma_load_2d_pair(dst, &tmA, kx, int32_t(a * p.mpad + int64_t(tm) * TMP + rank * TM), full);
                            tma_load_2d_pair(dst + A_BYTES, &tmB, kx,
                                             int32_t(b * p.npad + int64_t(tn) * TN + rank * TNH), full);
                        }
                    }
                }
            }
            // drain: the last use of every stage must have landed before the pair exits (the even
            // CTA's full barriers count the bytes of both)
            if (leader) {
                const uint32_t first = it > STAGES ? it - STAGES : 0;
                for (uint32_t j = first; j < it; ++j)
                    mbar_wait_drain(smem_u32(&bars->full[j % STAGES]), (j / STAGES) & 1, p.limit_ns);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (even CTA of the pair) ----------------
        if (lane == 0 && leader) {
            uint32_t it = 0, grp = 0;
            bool ok = true, issued_any = false;
            for (int u = pair; u < units && ok; u += npairs) {
                int tm, tn, seg, Lu;
                unit_coords(p, u, tm, tn, seg, Lu);
                const int kb0 = seg * p.kb_per_seg;
                const int kbn = min(p.kb_per_seg, p.kb_total - kb0);
                {
                    const int L = Lu;
                    const int np = pairs_in_level(mode, L);
                    const int items = np * kbn;
                    const int gsize = (mode == kExact || mode == kCrt) ? GROUP_ITEMS : items;
                    for (int g0 = 0; g0 < items && ok; g0 += gsize, ++grp) {
                        const int buf = grp & 1;
                        if (grp >= 2 && !mbar_wait(smem_u32(&bars->acc_empty[buf]), ((grp >> 1) - 1) & 1, p.status,
                                                   kDevTimeoutAccEmpty, p.limit_ns)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t dcol = tmem + uint32_t(buf * TN);
                        const int gend = min(items, g0 + gsize);
                        for (int x = g0; x < gend; ++x, ++it) {
                            const int s = it % STAGES;
                            if (!mbar_wait(smem_u32(&bars->full[s]), (it / STAGES) & 1, p.status, kDevTimeoutFull,
                                           p.limit_ns)) {
                                ok = false;
                                break;
                            }
                            tc_fence_after();
                            const uint32_t a_addr = smem_u32(smem + s * STAGE_BYTES);
                            const uint64_t adesc = sw128_desc(a_addr);
                            const uint64_t bdesc = sw128_desc(a_addr + A_BYTES);
#pragma unroll
                            for (int j = 0; j < TK / 16; ++j)
                                tc_mma_f16_pair(dcol, adesc + uint64_t(2 * j), bdesc + uint64_t(2 * j), kIdesc,
                                                (x == g0 && j == 0) ? 0u : 1u);
                            tc_commit_pair_mc(smem_u32(&bars->empty[s]), 0x3);
                            issued_any = true;
                        }
                        if (!ok) break;
                        tc_commit_pair_mc(smem_u32(&bars->acc_full[buf]), 0x3);
                    }
                }
            }
            // drain: every issued MMA completes before TMEM is released
            if (issued_any) {
                tc_commit_pair_mc(smem_u32(&bars->drain), 0x1);
                mbar_wait_drain(smem_u32(&bars->drain), 0, p.limit_ns);
            }
        }
    } else {
        // ---------------- epilogue ----------------
        const int q = warp & 3;                 // TMEM lane quarter of this warp
        const int h = (warp - 2) >> 2;          // column half: 0 or 1
        const uint32_t lane_base = uint32_t(32 * q) << 16;
        uint32_t grp = 0;
        bool ok = true;
        // the even CTA's accumulator-empty barriers (the MMA issuer waits for both CTAs' drains)
        const uint32_t acc_empty0 = mapa_shared(smem_u32(&bars->acc_empty[0]), 0);
        const uint32_t acc_empty1 = mapa_shared(smem_u32(&bars->acc_empty[1]), 0);
        for (int u = pair; u < units && ok; u += npairs) {
            int tm, tn, seg, Lu;
            unit_coords(p, u, tm, tn, seg, Lu);
            const int kb0 = seg * p.kb_per_seg;
            const int kbn = min(p.kb_per_seg, p.kb_total - kb0);
            const int64_t row = int64_t(tm) * TMP + int64_t(rank) * TM + 32 * q + lane;
            {
                const int L = Lu;
                const int np = pairs_in_level(mode, L);
                const int items = np * kbn;
                const int gsize = (mode == kExact || mode == kCrt) ? GROUP_ITEMS : items;
                // kCrt: FP32 pairs, sums of the groups' residues; kExact: int32 sums; else FP32 values
                uint64_t rsum[mode == kCrt ? 64 : 1];
                uint32_t acc[mode == kCrt ? 1 : 128];
                const float pf = c_modf[mode == kCrt ? L : 0], pinv = c_modf_inv[mode == kCrt ? L : 0];
                const uint64_t pneg2 = f32x2(-pf, -pf), pinv2 = f32x2(pinv, pinv);
                if constexpr (mode == kCrt) {
#pragma unroll
                    for (int c = 0; c < 64; ++c) rsum[c] = 0ull;
                } else {
#pragma unroll
                    for (int c = 0; c < 128; ++c) acc[c] = 0u;
                }
                for (int g0 = 0; g0 < items; g0 += gsize, ++grp) {
                    const int buf = grp & 1;
                    if (!mbar_wait(smem_u32(&bars->acc_full[buf]), (grp >> 1) & 1, p.status, kDevTimeoutMma,
                                   p.limit_ns)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t base = tmem + lane_base + uint32_t(buf * TN + h * 128);
#pragma unroll
                    for (int c4 = 0; c4 < 8; ++c4) {
                        uint32_t v[16];
                        tmem_ld_32x32b_x16(base + uint32_t(c4 * 16), v);
                        tc_wait_ld();
                        if constexpr (mode == kCrt) {
                            // the group sum is an integer of at most 2^24 in magnitude, exact in
                            // FP32: its residue (below 130 in magnitude, see residue2) is added up
#pragma unroll
                            for (int c = 0; c < 8; ++c)
                                rsum[c4 * 8 + c] = add2(rsum[c4 * 8 + c],
                                                        residue2(f32x2_bits(v[2 * c], v[2 * c + 1]), pinv2, pneg2));
                        } else if constexpr (mode == kExact) {
                            // exactly converted (adding 1.5 * 2^23 would be exact only below 2^22,
                            // i.e. for groups of 256 products)
#pragma unroll
                            for (int c = 0; c < 16; ++c)
                                acc[c4 * 16 + c] += uint32_t(__float2int_rn(__uint_as_float(v[c])));
                        } else {
#pragma unroll
                            for (int c = 0; c < 16; ++c) acc[c4 * 16 + c] = v[c];
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cluster(buf ? acc_empty1 : acc_empty0);
                }
                if (!ok) break;
                // level sums -> global level plane (row-major, pitch npad)
                const int64_t plane_off = ((int64_t(seg) * p.max_levels + L) * p.mpad + row) * p.npad +
                                          int64_t(tn) * TN + h * 128;
                if constexpr (mode == kCrt) {
                    // residues as r + 128: one byte each, 16 bits for the first modulus (257, whose
                    // 129 values a side do not fit a byte).  A single group's residue may be one past
                    // the symmetric range, which matters for 257 and 255 (253 and below stay within
                    // 127, and modulo 256 the byte wraps to the same residue).
                    if (items > gsize || L == 0 || L == 2) {
#pragma unroll
                        for (int c = 0; c < 64; ++c) rsum[c] = residue2(rsum[c], pinv2, pneg2);
                    }
                    // r + 128 + 2^23 holds r + 128 in its low bits
                    const uint64_t bias2 = f32x2(128.f + 8388608.f, 128.f + 8388608.f);
                    // out through the warp's staging tile (32 rows of 128 bytes, row = lane, 16-byte
                    // chunk j of a row at j ^ (lane % 8): the TMA 128-byte swizzle) and a TMA store
                    uint8_t* stg = out_stage + (warp - 2) * OUT_WARP_BYTES;
                    const int32_t trow = int32_t(int64_t(tm) * TMP + int64_t(rank) * TM + 32 * q);
                    const int64_t seg_rows = int64_t(seg) * (p.max_levels + 1) * p.mpad;
                    if (L != 0) {
                        if (lane == 0) bulk_wait_read0();  // the previous store has read the tile
                        __syncwarp();
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            uint32_t w[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const uint64_t t = add2(rsum[j * 8 + 2 * e], bias2);
                                const uint64_t v = add2(rsum[j * 8 + 2 * e + 1], bias2);
                                w[e] = __byte_perm(__byte_perm(uint32_t(t), uint32_t(t >> 32), 0x0040),
                                                   __byte_perm(uint32_t(v), uint32_t(v >> 32), 0x0040), 0x5410);
                            }
                            *reinterpret_cast<uint4*>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                                make_uint4(w[0], w[1], w[2], w[3]);
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(&tmC, int32_t(tn * TN + h * 128),
                                         int32_t(seg_rows + int64_t(L + 1) * p.mpad) + trow, smem_u32(stg));
                            bulk_commit();
                        }
                    } else {
#pragma unroll
                        for (int ch = 0; ch < 2; ++ch) {
                            if (lane == 0) bulk_wait_read0();
                            __syncwarp();
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                uint32_t w[4];
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const uint64_t t = add2(rsum[ch * 32 + j * 4 + e], bias2);
                                    w[e] = __byte_perm(uint32_t(t), uint32_t(t >> 32), 0x5410);
                                }
                                *reinterpret_cast<uint4*>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                                    make_uint4(w[0], w[1], w[2], w[3]);
                            }
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (lane == 0) {
                                tma_store_2d(&tmC0, int32_t(tn * TN + h * 128 + ch * 64),
                                             int32_t(seg_rows / 2) + trow, smem_u32(stg));
                                bulk_commit();
                            }
                        }
                    }
                } else {
                    int32_t* dst = p.levels + plane_off;
#pragma unroll
                    for (int c = 0; c < 128; c += 4) {
                        int4 w;
                        w.x = int32_t(acc[c + 0]);
                        w.y = int32_t(acc[c + 1]);
                        w.z = int32_t(acc[c + 2]);
                        w.w = int32_t(acc[c + 3]);
                        *reinterpret_cast<int4*>(dst + c) = w;
                    }
                }
            }
        }
    }

    // the residue stores of this thread have completed
    if (warp >= 2 && lane == 0) bulk_wait0();
    tc_fence_before();
    // neither CTA leaves while the pair MMAs, copies or arrivals may still touch its memory
    cluster_sync();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        tmem_dealloc_pair(tmem, 512);
    }
}

// Round the signed 128-bit integer W to the nearest double and multiply by 2^x, with integer
// operations only whenever the result is a normal number (the usual case); sub- or overflowing
// results take the FP64 ldexp path.
__device__ __forceinline__ double int128_to_double_scaled(__int128 W, int x) {
    if (W == 0) return 0.0;
    const bool neg = W < 0;
    const unsigned __int128 U = neg ? (unsigned __int128)(-W) : (unsigned __int128)W;
    const unsigned long long hi = (unsigned long long)(U >> 64), lo = (unsigned long long)U;
    const int nbits = hi ? 128 - __clzll((long long)hi) : 64 - __clzll((long long)lo);
    unsigned long long mant;
    int shift = 0;
    if (nbits <= 53) {
        mant = lo << (53 - nbits);
        shift = nbits - 53;
    } else {
        shift = nbits - 53;
        const unsigned __int128 m = U >> shift;
        const unsigned __int128 rem = U - (m << shift);
        const unsigned __int128 half = (unsigned __int128)1 << (shift - 1);
        mant = (unsigned long long)m;
        if (rem > half || (rem == half && (mant & 1))) ++mant;
        if (mant == (1ull << 53)) {
            mant >>= 1;
            ++shift;
        }
    }
    // value = mant * 2^(shift + x), mant in [2^52, 2^53)
    const int be = 52 + shift + x + 1023;
    if (be > 0 && be < 2047) {
        const unsigned long long bits =
            (neg ? (1ull << 63) : 0ull) | ((unsigned long long)be << 52) | (mant & 0xfffffffffffffull);
        return __longlong_as_double((long long)bits);
    }
    const double v = ldexp(double(mant), shift + x);
    return neg ? -v : v;
}

// C = alpha * 2^(e_i + f_j) * sum_L 2^(-14-8L) * sum_seg T[seg][L] + beta * C   (exact mode)
// C = alpha * sum_seg P[seg] + beta * C                                         (float modes)
// Exact mode forms W = sum_L T_L * 2^(8(S-1-L)) exactly in 128-bit integers, so the only roundings
// are the conversion of W to double and the alpha/beta update (skipped when alpha == 1, beta == 0).
// Grid: x over groups of 4 consecutive columns (one 16-byte load per level plane), y over rows.
constexpr int COMBINE_COLS = 4;

// Residue planes of a residue (CRT) product, S = mpad npad elements each, row-major: per k-segment the
// plane of the first modulus in 16 bits, then one byte per element for every other modulus, all
// holding r + 128 for the symmetric residue r.  Byte offset of plane t of segment g.
__host__ __device__ __forceinline__ int64_t crt_plane(int64_t S, int max_levels, int g, int t) {
    return S * (int64_t(g) * (max_levels + 1) + (t == 0 ? 0 : t + 1));
}

// The residues of four consecutive outputs of one row: words[t] holds four bytes (the first modulus:
// two words of two 16-bit values).
template <int N>
struct CrtWords {
    uint32_t w0[2];
    uint32_t w[N];  // w[0] unused
};

// row: the plane offset of the block's row and the launch's first column, j: the thread's column from
// there; row is the same for the whole block, so the addresses are formed once per warp.
template <int N>
__device__ __forceinline__ CrtWords<N> crt_load(const uint8_t* res, int64_t S, int64_t row, uint32_t j) {
    CrtWords<N> r;
    const uint2 z = *reinterpret_cast<const uint2*>(res + 2 * row + 2u * j);
    r.w0[0] = z.x;
    r.w0[1] = z.y;
#pragma unroll
    for (int t = 1; t < N; ++t) r.w[t] = *reinterpret_cast<const uint32_t*>(res + crt_plane(S, 0, 0, t) + row + j);
    return r;
}

// With k in segments: the sums of the residues b = r + 128 of the four columns over the segments, reduced to
// [0, p) and congruent to (sum of r) + 128, as the single segment's b is.  A word of every segment (the
// first one's is in r), its columns added in 16-bit halves, 255 values of at most 256 at a time.  Byte by
// byte and column by column this took 132 us of a 1135 x 1557 x 1766 product in two segments.
template <int N>
__device__ __forceinline__ void crt_seg_sums(const CrtWords<N>& r, const uint8_t* res, int64_t S, int max_levels,
                                             int64_t off, int nseg, int t, uint32_t p, uint32_t pinv32,
                                             uint32_t (&b)[4]) {
    uint32_t s[4] = {0u, 0u, 0u, 0u};
    uint32_t u = t == 0 ? r.w0[0] : r.w[t] & 0x00ff00ffu, v = t == 0 ? r.w0[1] : (r.w[t] >> 8) & 0x00ff00ffu;
    for (int g = 1; g < nseg;) {
        const int g1 = min(nseg, (g / 255 + 1) * 255);
#pragma unroll 4
        for (; g < g1; ++g) {
            const uint8_t* q = res + crt_plane(S, max_levels, g, t);
            if (t == 0) {
                const uint2 z = *reinterpret_cast<const uint2*>(q + 2 * off);
                u += z.x;
                v += z.y;
            } else {
                const uint32_t w = *reinterpret_cast<const uint32_t*>(q + off);
                u += w & 0x00ff00ffu;
                v += (w >> 8) & 0x00ff00ffu;
            }
        }
        s[0] += u & 0xffffu;
        s[t == 0 ? 1 : 2] += u >> 16;
        s[t == 0 ? 2 : 1] += v & 0xffffu;
        s[3] += v >> 16;
        u = v = 0u;
    }
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) b[cc] = mod_small(s[cc] + 128u * (p - 1u) * uint32_t(nseg - 1), p, pinv32);
}

// The double W 2^(x) of the two's-complement integer W of LB 32-bit words (low word first), rounded to
// nearest even, where W fits `bits` bits with its sign: rows or columns with Inf / NaN (exponent
// kNonFinite) give NaN, and results that are not normal numbers take the FP64 path (ldexp).  General
// form, for outputs whose leading words are all sign: the magnitude's words move up until the top
// one is not zero.
template <int LB>
__device__ __noinline__ double words_to_double_any(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, int ei, int fj,
                                                   int scale) {
    if (ei == kNonFinite || fj == kNonFinite) return __longlong_as_double(0x7ff8000000000000ll);
    const uint32_t w[4] = {w0, w1, w2, w3};
    const uint32_t sgn = uint32_t(int32_t(w[LB - 1]) >> 31);
    uint32_t z[4] = {0u, 0u, 0u, 0u};  // the magnitude, top word first
    uint32_t carry = sgn & 1u;
#pragma unroll
    for (int i = 0; i < LB; ++i) {
        const unsigned long long t = (unsigned long long)(w[i] ^ sgn) + carry;
        z[LB - 1 - i] = uint32_t(t);
        carry = uint32_t(t >> 32);
    }
    int lead = 32 * LB - 1;  // position of the leading bit
#pragma unroll
    for (int i = 1; i < LB; ++i)
        if (z[0] == 0u) {
#pragma unroll
            for (int j = 0; j < 3; ++j) z[j] = z[j + 1];
            z[3] = 0u;
            lead -= 32;
        }
    if (z[0] == 0u) return 0.0;
    const int lz = __clz(int(z[0]));
    const uint32_t t1 = __funnelshift_l(z[1], z[0], lz);
    const uint32_t t0 = __funnelshift_l(z[2], z[1], lz) | min(__funnelshift_l(z[3], z[2], lz) | z[3], 1u);  // sticky
    unsigned long long mant = (((unsigned long long)t1 << 32) | t0) >> 11;
    mant += (t0 & 0x7ffu) + (uint32_t(mant) & 1u) > 0x400u ? 1ull : 0ull;
    const double v = ldexp(double(mant), lead - lz - 52 + ei + fj - scale);
    return sgn ? -v : v;
}

// The usual case in straight-line code: W, moved up by the constant that brings its sign bit to the top,
// has a bit that is not sign in its top word; the funnel shift that puts that bit below the sign
// leaves 64 bits whose rounding to nearest even (symmetric, so no magnitude is formed before it) is
// an integer addition, and adding the exponent's bits to the 53-bit magnitude writes it, a rounding
// carry into 2^53 moving the exponent up by itself.  About 30 instructions; with the magnitude formed
// first and the words moved up one at a time it was about 55.
template <int LB, int BITS>
__device__ __forceinline__ double words_to_double(const uint32_t (&w)[4], int ei, int fj, int scale) {
    constexpr int UP = 32 * LB - BITS;  // 0 <= UP < 32
    uint32_t z[4] = {0u, 0u, 0u, 0u};  // top word first
#pragma unroll
    for (int i = 0; i < LB; ++i) z[i] = UP == 0 ? w[LB - 1 - i] : __funnelshift_l(i + 1 < LB ? w[LB - 2 - i] : 0u, w[LB - 1 - i], UP);
    const uint32_t sgn = uint32_t(int32_t(z[0]) >> 31);
    const int lz = __clz(int(z[0] ^ sgn));  // at least 1, 32 when the top word is all sign
    const int sh = lz - 1;
    uint32_t t1 = __funnelshift_l(z[1], z[0], sh), t0 = __funnelshift_l(z[2], z[1], sh);
    if constexpr (LB > 2) t0 |= min(__funnelshift_l(z[3], z[2], sh) | (LB > 3 ? z[3] : 0u), 1u);  // sticky
    // mantissa in bits 62..10
    unsigned long long v = ((unsigned long long)t1 << 32) | t0;
    v += 0x1ffu + ((t0 >> 10) & 1u);
    // the sign bits go before the shift down: a positive carry into bit 63 is a magnitude, not a sign
    const uint32_t rl = uint32_t(v >> 10) ^ sgn, rh = (uint32_t(v >> 32) ^ sgn) >> 10;
    unsigned long long m = ((unsigned long long)rh << 32) | rl;
    m += sgn & 1u;
    const int be = BITS - 1 - lz + ei + fj - scale + 1023;  // the leading bit is bit BITS - 1 - lz of W
    if (lz < 32 && be >= 1 && be <= 2045) {
        const uint32_t hi = uint32_t(m >> 32) + (uint32_t(be - 1) << 20) + (sgn & 0x80000000u);
        return __hiloint2double(int(hi), int(uint32_t(m)));
    }
    return words_to_double_any<LB>(w[0], w[1], w[2], w[3], ei, fj, scale);
}

// Residue (CRT) reconstruction of four consecutive outputs of one row for N moduli, all constants
// compile-time (crt_tables.h).  Per super modulus x = b_p A_s + b_q B_s + K_s < 2^26 is congruent to
// the super residue u_s (one two-way byte dot product, K_s taking the 128s out), and
// W = sum_s x_s (P / P_s) in 64-bit sums of 32-bit limb products.  The multiple of P to remove is
// round(W / P), from an FP32 estimate of sum_s x_s / P_s (below 2^13, off by less than 0.01): the
// product of the scaled integers has |value| < P / 2.125, so W / P lies at least 0.029 from a half
// integer.  It is removed by adding the multiple of 2^(32 LB) - P, all modulo 2^(32 LB).
template <int N>
__device__ __forceinline__ void crt_cols(const CrtWords<N>& r, const uint8_t* res, int64_t S, int64_t off,
                                         int nseg, int max_levels, int scale, int ei, const int (&fj)[4], double (&v)[4]) {
    constexpr CrtTable T = kCrtTables[N - 2];
    constexpr int NS = T.nsup, LB = T.limbs;
    unsigned long long acc[4][4];
    float fq[4];
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        fq[cc] = 0.f;
#pragma unroll
        for (int l = 0; l < 4; ++l) acc[cc][l] = 0;
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        constexpr uint32_t one = 1u;
        const CrtSuper& Q = T.sup[s];
        const bool pair = Q.q > one;
        uint32_t x[4];
        if (nseg > 1) {
            uint32_t b[4];
            crt_seg_sums<N>(r, res, S, max_levels, off, nseg, Q.ia, Q.p, Q.pinv32, b);
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) x[cc] = b[cc] * Q.A + Q.K;
            if (pair) {
                crt_seg_sums<N>(r, res, S, max_levels, off, nseg, Q.ib, Q.q, Q.qinv32, b);
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) x[cc] += b[cc] * Q.B;
            }
        } else if (Q.ia == 0) {
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                x[cc] = ((cc & 1) ? r.w0[cc >> 1] >> 16 : r.w0[cc >> 1] & 0xffffu) * Q.A + Q.K;
                if (pair) x[cc] += __byte_perm(r.w[Q.ib], 0, 0x4440 + cc) * Q.B;
            }
        } else if (pair) {
            // bytes (p, q) of columns 0, 1 and of columns 2, 3 side by side
            const uint32_t t01 = __byte_perm(r.w[Q.ia], r.w[Q.ib], 0x5140), t23 = __byte_perm(r.w[Q.ia], r.w[Q.ib], 0x7362);
            const uint32_t AB = Q.A | (Q.B << 16);
            x[0] = __dp2a_lo(AB, t01, Q.K);
            x[1] = __dp2a_hi(AB, t01, Q.K);
            x[2] = __dp2a_lo(AB, t23, Q.K);
            x[3] = __dp2a_hi(AB, t23, Q.K);
        } else {
            x[0] = __dp2a_lo(Q.A, r.w[Q.ia], Q.K);
            x[1] = __dp2a_lo(Q.A << 16, r.w[Q.ia], Q.K);
            x[2] = __dp2a_hi(Q.A, r.w[Q.ia], Q.K);
            x[3] = __dp2a_hi(Q.A << 16, r.w[Q.ia], Q.K);
        }
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            fq[cc] = fmaf(__uint2float_rn(x[cc]), Q.finv, fq[cc]);
#pragma unroll
            for (int l = 0; l < LB; ++l)
                if (Q.M[l]) acc[cc][l] += (unsigned long long)x[cc] * Q.M[l];
        }
    }
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
        const uint32_t qm = __float_as_uint(fq[cc] + MAGIC) - MAGIC_BITS;
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        unsigned long long carry = 0;
#pragma unroll
        for (int l = 0; l < LB; ++l) {
            const unsigned long long a = acc[cc][l] + (unsigned long long)qm * T.negP[l] + carry;
            w[l] = uint32_t(a);
            carry = a >> 32;
        }
        v[cc] = words_to_double<LB, T.bits>(w, ei, fj[cc], scale);
    }
}

template <typename TC>
struct CrtCombine {
    const uint8_t* res;      // residue planes
    int64_t mpad, npad;
    int nseg, max_levels;
    int64_t row0, col0;      // first row and column of this launch in the planes, the exponents and C
    int64_t m, n;            // rows, columns of this launch
    const int *eA, *eB;
    double alpha, beta;
    TC* C;
    int64_t ldc;
    bool followed;           // by a dependent launch of this kernel on the same stream
};

// alpha v + beta c in double precision, rounded once to the result's type.  An FP64 instruction of a
// warp takes 64 clocks of its SM quarter, about half of what an output costs otherwise: a factor of one or minus
// one is a sign, and c + x needs no multiply-add.
template <typename TC>
__device__ __forceinline__ TC scaled(double v, double alpha, double beta, const TC* c) {
    double x;
    if (alpha == 1.0) x = v;
    else if (alpha == -1.0) x = -v;
    else x = alpha * v;
    if (beta == 0.0) return TC(x);
    if (beta == 1.0) return TC(double(*c) + x);
    return TC(fma(beta, double(*c), x));
}

// The rows i, i + gridDim.y, ... of four columns a thread.
template <int N, typename TC>
__device__ __forceinline__ void crt_rows(const CrtCombine<TC>& p, int scale, int64_t j0, const int (&fj)[4]) {
    const int64_t S = p.mpad * p.npad, step = int64_t(gridDim.y) * p.npad;
    const bool plain = p.alpha == 1.0 && p.beta == 0.0;
    // whole groups of four columns, 16-byte aligned in every row
    const bool vec = j0 + 4 <= p.n && (p.ldc * int64_t(sizeof(TC))) % 16 == 0 &&
                     (reinterpret_cast<uintptr_t>(p.C + p.col0) & 15) == 0;
    int64_t i = p.row0 + blockIdx.y, row = i * p.npad + p.col0;
    const int64_t end = p.row0 + p.m;
    if (i >= end) return;
    const uint32_t j = uint32_t(j0);
    while (true) {
        const int64_t inext = i + gridDim.y;
        const bool more = inext < end;
        const CrtWords<N> w = crt_load<N>(p.res, S, row, j);
        const int ei = p.eA[i];
        double v[4];
        crt_cols<N>(w, p.res, S, row + j0, p.nseg, p.max_levels, scale, ei, fj, v);
        TC* crow = p.C + i * p.ldc + p.col0 + j0;
        if (plain && vec) {
            if constexpr (sizeof(TC) == 8) {
                *reinterpret_cast<double2*>(crow) = make_double2(v[0], v[1]);
                *reinterpret_cast<double2*>(crow + 2) = make_double2(v[2], v[3]);
            } else {
                *reinterpret_cast<float4*>(crow) = make_float4(float(v[0]), float(v[1]), float(v[2]), float(v[3]));
            }
        } else {
#pragma unroll
            for (int cc = 0; cc < 4; ++cc) {
                if (j0 + cc >= p.n) break;
                crow[cc] = plain ? TC(v[cc]) : scaled(v[cc], p.alpha, p.beta, crow + cc);
            }
        }
        if (!more) return;
        i = inext;
        row += step;
    }
}

// Residue (CRT) reconstruction and epilogue: C = alpha * W 2^(e_i + f_j - scale) + beta * C.  Bound by
// instruction issue and latency (about 137 instructions an output at 13 moduli, half the issue slots
// busy; 118 MB read and 134 MB written would take 38 us of the 63 at 32768 x 256).  Byte planes, super
// residues left unreduced and a straight-line conversion to double against 16-bit planes, a reduction of
// every super residue and a branching conversion: 8.4 M outputs at 13 moduli 90 -> 63 us, 33.5 M at 12
// moduli 285 -> 184.  Eight blocks an SM (64 registers) measured like six and 4 % faster than
// five; fetching the next row's residues ahead cost the registers of
// it (66 us), two columns at a time instead of four took 40 % more instructions.
constexpr int kCombineBlocks = 8;
template <typename TC>
__global__ void __launch_bounds__(128, kCombineBlocks) crt_combine_kernel(const CrtCombine<TC> p,
                                                                          const SplitInfo* info) {
    if (p.followed) griddep_launch();
    griddep_wait();
    const int64_t j0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) * 4;
    if (j0 >= p.n) return;
    const int scale = info->beta + info->beta_b;
    int fj[4];
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) fj[cc] = (j0 + cc < p.n) ? p.eB[p.col0 + j0 + cc] : 0;
    switch (info->slices) {
#define GB_CRT_CASE(NN) \
    case NN: crt_rows<NN, TC>(p, scale, j0, fj); break;
        GB_CRT_CASE(2) GB_CRT_CASE(3) GB_CRT_CASE(4) GB_CRT_CASE(5) GB_CRT_CASE(6) GB_CRT_CASE(7)
        GB_CRT_CASE(8) GB_CRT_CASE(9) GB_CRT_CASE(10) GB_CRT_CASE(11) GB_CRT_CASE(12) GB_CRT_CASE(13)
        GB_CRT_CASE(14) GB_CRT_CASE(15)
#undef GB_CRT_CASE
        default: break;  // the plan gives 2 to 15 moduli
    }
}

// Grid of the reconstruction: rows on y, as many blocks as are resident on every SM together.
dim3 crt_combine_grid(int64_t m, int64_t n, int num_sms) {
    const int64_t x = ((n + 3) / 4 + 127) / 128;
    const int64_t y = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(m, 65535), int64_t(num_sms) * kCombineBlocks / x));
    return dim3(unsigned(x), unsigned(y));
}

// Launched the plain way, so that its pointers can be __restrict__: as a dependent launch without, the next
// row's loads waited for this row's stores (8192 x 8192 x 64 in six slices 1.79 ms a call, 1.60 so).
template <typename TC>
__global__ void __launch_bounds__(128, 8)
combine_kernel(const int32_t* __restrict__ levels, int nseg, int max_levels, int64_t mpad, int64_t npad, int mode,
               const SplitInfo* __restrict__ info, const int* __restrict__ eA, const int* __restrict__ eB, int64_t m,
               int64_t n, double alpha, double beta, TC* __restrict__ C, int64_t ldc) {
    const int64_t j0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) * COMBINE_COLS;
    if (j0 >= n) return;
    const int64_t plane = mpad * npad;
    for (int64_t i = blockIdx.y; i < m; i += gridDim.y) {
    const int64_t off = i * npad + j0;
    double v[COMBINE_COLS];
    if (mode == kExact) {
        const int S = info->slices;
        const int ei = eA[i];
        __int128 W[COMBINE_COLS] = {0, 0, 0, 0};
        for (int L = 0; L < S; ++L) {
            long long t[COMBINE_COLS] = {0, 0, 0, 0};
            for (int g = 0; g < nseg; ++g) {
                const int4 q = *reinterpret_cast<const int4*>(levels + (int64_t(g) * max_levels + L) * plane + off);
                t[0] += q.x; t[1] += q.y; t[2] += q.z; t[3] += q.w;
            }
#pragma unroll
            for (int c = 0; c < COMBINE_COLS; ++c) W[c] = (W[c] << 8) + t[c];
        }
#pragma unroll
        for (int c = 0; c < COMBINE_COLS; ++c) {
            const int64_t j = j0 + c;
            const int fj = (j < n) ? eB[j] : 0;
            if (ei == kNonFinite || fj == kNonFinite)
                v[c] = __longlong_as_double(0x7ff8000000000000ll);  // NaN: the inputs were not finite
            else
                v[c] = int128_to_double_scaled(W[c], ei + fj - 14 - 8 * (S - 1));
        }
    } else {
        float acc[COMBINE_COLS] = {0.f, 0.f, 0.f, 0.f};
        double dacc[COMBINE_COLS] = {0.0, 0.0, 0.0, 0.0};
        for (int g = 0; g < nseg; ++g) {
            const int4 q = *reinterpret_cast<const int4*>(levels + int64_t(g) * max_levels * plane + off);
            acc[0] = __int_as_float(q.x); acc[1] = __int_as_float(q.y);
            acc[2] = __int_as_float(q.z); acc[3] = __int_as_float(q.w);
#pragma unroll
            for (int c = 0; c < COMBINE_COLS; ++c) dacc[c] += double(acc[c]);
        }
#pragma unroll
        for (int c = 0; c < COMBINE_COLS; ++c) v[c] = dacc[c];
    }
    const bool plain = (alpha == 1.0 && beta == 0.0);
    TC* crow = C + i * ldc;
#pragma unroll
    for (int c = 0; c < COMBINE_COLS; ++c) {
        const int64_t j = j0 + c;
        if (j >= n) break;
        if (plain) {
            crow[j] = TC(v[c]);
        } else {
            const double x = alpha * v[c];
            crow[j] = TC(beta == 0.0 ? x : fma(beta, double(crow[j]), x));
        }
    }
    }
}

int64_t round_up(int64_t x, int64_t q) { return (x + q - 1) / q * q; }

}  // namespace

bool split_read_info(const void* info_dev, int* slices, double* bound) {
    SplitInfo h;
    if (cudaMemcpy(&h, info_dev, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return false;
    *slices = h.slices;
    *bound = h.bound;
    return true;
}

size_t split_info_bytes() { return sizeof(SplitInfo); }

void split_decode_info(const void* info_host, int* slices, double* bound) {
    SplitInfo h;
    std::memcpy(&h, info_host, sizeof(h));
    *slices = h.slices;
    *bound = h.bound;
}

// ---- host orchestration ------------------------------------------------------------------------
namespace {

// k-tiles per block of the pre-pass kernels: TILE_KT, or fewer where that would leave an SM without
// several blocks (1024^3: 128 blocks of eight tiles took 9 us for the statistics and 23 for slicing, smaller ones 7 and 16).
int tiles_per_block(int64_t tiles, int64_t row_blocks, int num_sms) {
    return int(std::max<int64_t>(1, std::min<int64_t>(TILE_KT, tiles * row_blocks / (int64_t(num_sms) * 6))));
}

// The residue planes (crt_plane) as the 2-D arrays the epilogue's TMA stores address: 16-bit rows
// (first modulus) and byte rows (the others).
bool crt_plane_maps(CUtensorMap* t16, CUtensorMap* t8, const void* planes, int nseg, int max_levels, int64_t mpad,
                    int64_t npad, std::string* err) {
    const uint64_t rows = uint64_t(nseg) * uint64_t(max_levels + 1) * uint64_t(mpad);  // of npad bytes
    return encode_tmap_2d(t16, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, planes, rows / 2, npad, npad, 32, 64,
                          CU_TENSOR_MAP_SWIZZLE_128B, err) &&
           encode_tmap_2d(t8, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, planes, rows, npad, npad, 32, 128,
                          CU_TENSOR_MAP_SWIZZLE_128B, err);
}

int native_product(const Gemm& g, const LaunchCtl& ctl, cudaStream_t st, Workspace& ws, SplitResult* out,
                   std::string* err) {
    Runtime& r = runtime();
    const NativePlan plan = native_plan(g.m, g.n, g.k, 8, r.num_sms, ctl.inject_stall != 0);
    double* w = nullptr;
    if (plan.splits > 1) {
        w = static_cast<double*>(ws.get(kSlotWork, size_t(plan.splits) * size_t(g.m) * size_t(g.n) * 8, err));
        if (!w) return GB300_ERR_NO_MEMORY;
    }
    cudaError_t e = native_gemm<double>(g, plan, w, ctl, st, err);
    if (e != cudaSuccess) {
        if (err && err->empty()) *err = cudaGetErrorString(e);
        return GB300_ERR_CUDA;
    }
    out->method_used = GB300_METHOD_NATIVE;
    out->slices = 0;
    out->error_bound = double(g.k) * 0x1p-53;
    out->info_dev = nullptr;
    return GB300_OK;
}

// The AUTO policy: the split form costs about S(S+1)/2 BF16 products plus operand passes; below a
// few million multiply-adds, or for very short k, the native kernel's single pass wins.
bool auto_uses_native(const Gemm& g) {
    const double work = double(g.m) * double(g.n) * double(g.k);
    return work < 256.0 * 256.0 * 256.0 || g.k < 64;
}

// Moduli the CRT form needs in the worst case for inner dimension k and a normwise target (<= 0:
// k*2^-53): with |a_i| < 2^e_i, ||A||_F >= ||2^e||/2, so rA, rB <= 2 sqrt(k).  Returns a count above
// MAX_MODULI when the target is out of reach (the digit form is used then).
int crt_worst_case_moduli(int64_t k, double target) {
    if (target <= 0) target = double(k) * 0x1p-53;
    const double r = 2.0 * std::sqrt(double(std::max<int64_t>(k, 1)));
    int beta = 1;
    while (beta <= 55 && (std::ldexp(1.0, -beta - 1) * 2 * r + std::ldexp(1.0, -2 * beta - 2) * r * r + 0x1p-52) > target)
        ++beta;
    if (beta > 55) return MAX_MODULI + 1;
    int kbits = 0;
    while ((int64_t(1) << kbits) < std::max<int64_t>(k, 2)) ++kbits;
    const double need = 2.0 + kbits + 2.0 * beta;
    double have = 0;
    int N = 0;
    while (N < MAX_MODULI && have < need) have += kModLog2[N++];
    return have < need ? MAX_MODULI + 1 : N;
}

struct SplitGeometry {
    int mode, m_tiles, n_tiles, nseg, kb_total, max_planes, max_levels;
    int64_t mpad, npad, kpad, kseg;
};

SplitGeometry split_geometry(const Gemm& g, const SplitRequest& req, int num_sms) {
    SplitGeometry G;
    G.mode = kExact;
    if (req.method == GB300_METHOD_BF16) G.mode = kBf16;
    else if (req.method == GB300_METHOD_BF16X3) G.mode = kBf16x3;
    else if (req.method == GB300_METHOD_SPLIT_CRT) G.mode = kCrt;
    else if ((req.method == GB300_METHOD_SPLIT || req.method == GB300_METHOD_AUTO) && req.slices <= 0 &&
             crt_worst_case_moduli(g.k, req.target_error) <= MAX_MODULI)
        G.mode = kCrt;
    G.m_tiles = int((g.m + TMP - 1) / TMP);  // tiles of a CTA pair (256 rows)
    G.n_tiles = int((g.n + TN - 1) / TN);
    G.mpad = int64_t(G.m_tiles) * TMP;
    G.npad = int64_t(G.n_tiles) * TN;
    G.kpad = round_up(g.k, TK);
    G.kb_total = int(G.kpad / TK);
    if (G.mode == kCrt)
        // at least two moduli (the reconstruction tables start at N = 2)
        G.max_planes = req.slices > 0 ? std::max(2, std::min(req.slices, MAX_MODULI))
                                      : std::max(2, std::min(MAX_MODULI, crt_worst_case_moduli(g.k, req.target_error)));
    else
        G.max_planes = (G.mode == kExact) ? (req.slices > 0 ? std::min(req.slices, MAX_SLICES) : MAX_SLICES)
                                          : (G.mode == kBf16 ? 1 : 2);
    G.max_levels = (G.mode == kExact || G.mode == kCrt) ? G.max_planes : 1;
    // k-segments: exactness (int32 level sums, sums of group residues) and parallelism for few output tiles; decided from the
    // device's SM count only, so a capped grid computes the same segments (and the same result)
    int64_t kseg = G.kpad;
    if (G.mode == kExact || G.mode == kCrt) {
        // n_L * Kseg products of at most 2^14 each must stay below 2^31 (residue form, one pair per
        // level: 128 groups' residues of at most 130, exact in FP32 by far)
        const int64_t cap = (int64_t(511) / (G.mode == kCrt ? 1 : G.max_planes)) * KSEG_UNIT;
        kseg = std::min(kseg, std::max<int64_t>(cap, KSEG_UNIT));
    }
    // Split k only when at most half the CTA pairs would have a tile, and into as many segments as
    // still fit one wave of pairs.  With more tiles a split cannot raise the occupancy (the units
    // spill into a second, partial wave) and it multiplies the residue planes the reconstruction
    // reads; at 64 tiles on 76 pairs two segments made a 512 x 8192 x 512 product 1.6 times slower.
    // A segment keeps at least one TMEM drain group of k (1024): a unit of 256 k has about 1.3 us of
    // products against about 3 us of epilogue (measured with its integer reductions), and every
    // extra segment adds residue planes for the reconstruction; 1024^3 split into four 256-k
    // segments took 59 us in the tensor-core kernel and 55 us in the reconstruction.
    const int tiles = G.m_tiles * G.n_tiles, pairs = std::max(1, num_sms / 2);
    if (2 * tiles <= pairs) {
        const int64_t want = pairs / tiles;
        constexpr int64_t kMinSeg = int64_t(GROUP_ITEMS) * TK;
        kseg = std::min(kseg, std::max<int64_t>(kMinSeg, round_up((G.kpad + want - 1) / want, KSEG_UNIT)));
    }
    // equal segments: persistent CTAs take units in a fixed stride, so unequal segments would give
    // some CTAs only the long ones
    const int64_t nseg = (G.kpad + kseg - 1) / kseg;
    G.kseg = round_up((G.kpad + nseg - 1) / nseg, TK);
    G.nseg = int((G.kpad + G.kseg - 1) / G.kseg);
    return G;
}

// Level planes of a product: int32 sums, FP32 tiles or, in the residue form, 16 bits for the first
// modulus and a byte for each other one (crt_plane).
size_t level_bytes(const SplitGeometry& G) {
    const size_t S = size_t(G.nseg) * size_t(G.mpad) * size_t(G.npad);
    return G.mode == kCrt ? S * size_t(G.max_levels + 1) : S * size_t(G.max_levels) * 4;
}

// Statistics buffers of `rows_a` rows of A and `rows_b` columns of B over k.  kSlotScaleA: exponents
// (int), SplitInfo, one RowPartial per row block; kSlotScaleB: the counters, then the chunk partials.
struct StatsLayout {
    int kt, chunks;
    int64_t blocks;  // row blocks of both
    size_t off_info, off_group, bytes_a, off_part, bytes_b;
};
StatsLayout stats_layout(int64_t rows_a, int64_t rows_b, int64_t k, int num_sms) {
    StatsLayout L;
    L.blocks = (rows_a + 31) / 32 + (rows_b + 31) / 32;
    const int64_t tiles = (k + 63) / 64;
    L.kt = tiles_per_block(tiles, L.blocks, num_sms);
    L.chunks = int((tiles + L.kt - 1) / L.kt);
    L.off_info = size_t(round_up((rows_a + rows_b) * int64_t(sizeof(int)), 256));
    L.off_group = L.off_info + (sizeof(SplitInfo) + 255) / 256 * 256;
    L.bytes_a = L.off_group + size_t(L.blocks) * sizeof(RowPartial);
    L.off_part = size_t(round_up((L.blocks + 1) * int64_t(sizeof(unsigned)), 256));
    L.bytes_b = L.off_part + (L.chunks > 1 ? size_t(rows_a + rows_b) * size_t(L.chunks) * sizeof(uint2) : 0);
    return L;
}

// Stored (row-major) shape of the operands of a logical product.
void stored_a(const Gemm& g, int64_t* rows, int64_t* cols) { *rows = g.ta ? g.k : g.m; *cols = g.ta ? g.m : g.k; }
void stored_b(const Gemm& g, int64_t* rows, int64_t* cols) { *rows = g.tb ? g.n : g.k; *cols = g.tb ? g.k : g.n; }
bool tma_ready(const void* p, int64_t ld) { return reinterpret_cast<uintptr_t>(p) % 16 == 0 && (ld * 8) % 16 == 0; }

// Whether a product runs on the native kernel, and whether there in the tiles that read their
// operands through TMA.
bool runs_native(const Gemm& g, const SplitRequest& req) {
    return g.k == 0 || req.method == GB300_METHOD_NATIVE || (req.method == GB300_METHOD_AUTO && auto_uses_native(g));
}
bool runs_tma_tiles(const Gemm& g, const SplitRequest& req, bool stall) {
    return runs_native(g, req) && native_plan(g.m, g.n, g.k, 8, runtime().num_sms, stall).tile == 0;
}

// An operand read in place: by TMA when it is 16-byte aligned in base and pitch, by every other
// kernel (single-element loads) when its base is aligned for a double.
bool read_in_place(const void* p, int64_t ld, bool tma, size_t elem = 8) {
    return tma ? tma_ready(p, ld) : reinterpret_cast<uintptr_t>(p) % elem == 0;
}

// Copy operands that cannot be read in place into the workspace.
int realign_operands(Gemm& g, bool tma, size_t elem, Workspace& ws, cudaStream_t st, std::string* err) {
    if (g.k == 0) return GB300_OK;
    for (int which = 0; which < 2; ++which) {
        const void*& p = which == 0 ? g.A : g.B;
        int64_t& ld = which == 0 ? g.lda : g.ldb;
        if (read_in_place(p, ld, tma, elem)) continue;
        int64_t rows, cols;
        if (which == 0) stored_a(g, &rows, &cols);
        else stored_b(g, &rows, &cols);
        const int64_t ldp = (cols + 1) / 2 * 2;
        void* d = ws.get(which == 0 ? kSlotA : kSlotB, size_t(rows) * size_t(ldp) * elem, err);
        if (!d) return GB300_ERR_NO_MEMORY;
        const cudaError_t e = cudaMemcpy2DAsync(d, size_t(ldp) * elem, p, size_t(ld) * elem, size_t(cols) * elem,
                                                size_t(rows), cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) {
            if (err) *err = std::string("operand realignment: ") + cudaGetErrorString(e);
            return GB300_ERR_CUDA;
        }
        p = d;
        ld = ldp;
    }
    return GB300_OK;
}

}  // namespace

void device_product_slot_needs(const Gemm& g, const SplitRequest& req, size_t need[kSlotCount]) {
    Runtime& r = runtime();
    for (int i = 0; i < kSlotCount; ++i) need[i] = 0;
    auto rounded = [](size_t b) { return b == 0 ? size_t(0) : (b + (size_t(2) << 20) - 1) & ~((size_t(2) << 20) - 1); };
    if (g.k > 0) {
        const bool tma = runs_tma_tiles(g, req, false);
        int64_t rr, cc;
        if (!read_in_place(g.A, g.lda, tma)) { stored_a(g, &rr, &cc); need[kSlotA] = rounded(size_t(rr) * size_t((cc + 1) / 2 * 2) * 8); }
        if (!read_in_place(g.B, g.ldb, tma)) { stored_b(g, &rr, &cc); need[kSlotB] = rounded(size_t(rr) * size_t((cc + 1) / 2 * 2) * 8); }
    }
    if (runs_native(g, req)) {
        const int splits = native_plan(g.m, g.n, g.k, 8, r.num_sms, false).splits;
        if (splits > 1) need[kSlotWork] = rounded(size_t(splits) * size_t(g.m) * size_t(g.n) * 8);
        return;
    }
    const SplitGeometry G = split_geometry(g, req, r.num_sms);
    need[kSlotSliceA] = rounded(size_t(G.max_planes) * size_t(G.mpad) * size_t(G.kpad) * 2);
    need[kSlotSliceB] = rounded(size_t(G.max_planes) * size_t(G.npad) * size_t(G.kpad) * 2);
    need[kSlotLevels] = rounded(level_bytes(G));
    const StatsLayout SL = stats_layout(g.m, g.n, g.k, r.num_sms);
    need[kSlotScaleA] = rounded(SL.bytes_a);
    need[kSlotScaleB] = rounded(SL.bytes_b);
}

size_t device_product_footprint(const Gemm& g, const SplitRequest& req) {
    size_t need[kSlotCount];
    device_product_slot_needs(g, req, need);
    size_t t = 0;
    for (int i = 0; i < kSlotCount; ++i) t += need[i];
    return t;
}

bool split_auto_uses_native(const Gemm& g) { return auto_uses_native(g); }

// A residue product with at least as many pair tiles as SMs runs its tensor-core work as two
// launches over the two halves of C's column tiles, and the first half's reconstruction waits on a
// second stream for the first of them.  No reconstruction block fits beside a tensor-core CTA (a quarter
// of an SM that holds three of its warps at 168 registers has 256 left), so what this hides is the
// tail: SMs that have no tensor-core unit left start on the first half at once.  65536 x 256 x 256: 403 us
// in one part, 394 in two; 8192^3 9.11 and 8.81 ms (two runs of one side differ by 2 %).  The second
// stream belongs to the pair (calling host thread, caller's stream) and has the caller's stream
// priority, so concurrent callers (user threads, or the server's slots, launched from its one
// scheduler thread on their own streams) never queue behind one another's reconstructions; the
// ordering events come from a pool.
struct PartEvents {
    cudaStream_t aux = nullptr;
    cudaEvent_t tc0 = nullptr, done0 = nullptr;
};

struct ThreadAuxStreams {
    static constexpr size_t kMax = 32;
    std::vector<std::pair<cudaStream_t, cudaStream_t>> map;  // caller's stream -> second stream
    ~ThreadAuxStreams() {
        for (auto& kv : map) cudaStreamDestroy(kv.second);  // fails harmlessly once the context is gone
    }
};

// The second stream of the calling host thread for the caller's stream `st` (created on first
// use; past kMax callers' streams the last one is shared, which orders more but stays correct).
static cudaStream_t aux_stream_for(cudaStream_t st, std::string* err) {
    static thread_local ThreadAuxStreams ts;
    for (auto& kv : ts.map)
        if (kv.first == st) return kv.second;
    if (ts.map.size() >= ThreadAuxStreams::kMax) return ts.map.back().second;
    int prio = 0;
    if (cudaStreamGetPriority(st, &prio) != cudaSuccess) {
        cudaGetLastError();
        prio = 0;
    }
    cudaStream_t s = nullptr;
    if (cudaStreamCreateWithPriority(&s, cudaStreamNonBlocking, prio) != cudaSuccess) {
        if (err) *err = "second stream creation failed";
        return nullptr;
    }
    ts.map.emplace_back(st, s);
    return s;
}

static bool part_events_get(cudaStream_t st, PartEvents* pe, std::string* err) {
    cudaStream_t aux = aux_stream_for(st, err);
    if (!aux) return false;
    Runtime& r = runtime();
    std::lock_guard<std::mutex> lk(r.part_mu);
    cudaEvent_t ev[2];
    for (int i = 0; i < 2; ++i) {
        if (!r.part_events.empty()) {
            ev[i] = r.part_events.back();
            r.part_events.pop_back();
        } else if (cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming) != cudaSuccess) {
            if (i == 1) r.part_events.push_back(ev[0]);
            if (err) *err = "part event creation failed";
            return false;
        }
    }
    pe->aux = aux;
    pe->tc0 = ev[0];
    pe->done0 = ev[1];
    return true;
}

// The events go back to the pool once every record and wait on them is enqueued (a wait takes the
// event's state when it is enqueued, so a later record by another product does not affect it).
static void part_events_put(const PartEvents& pe) {
    Runtime& r = runtime();
    std::lock_guard<std::mutex> lk(r.part_mu);
    r.part_events.push_back(pe.tc0);
    r.part_events.push_back(pe.done0);
}

namespace {
// The tensor-core forms on operands and result of type T (double or float).
template <typename T>
int tensor_product(const Gemm& g, const SplitRequest& req, const LaunchCtl& ctl, cudaStream_t st, Workspace& ws,
                   SplitResult* out, std::string* err) {
    Runtime& r = runtime();

    const SplitGeometry G = split_geometry(g, req, r.num_sms);
    const int mode = G.mode;
    const int64_t m = g.m, n = g.n, k = g.k;
    const int m_tiles = G.m_tiles, n_tiles = G.n_tiles;
    const int64_t mpad = G.mpad, npad = G.npad, kpad = G.kpad;
    const int kb_total = G.kb_total, max_planes = G.max_planes, max_levels = G.max_levels;
    const int64_t kseg = G.kseg;
    const int nseg = G.nseg;

    // device buffers
    const size_t planesA = size_t(max_planes) * size_t(mpad) * size_t(kpad);
    const size_t planesB = size_t(max_planes) * size_t(npad) * size_t(kpad);
    auto* pa = static_cast<__nv_bfloat16*>(ws.get(kSlotSliceA, planesA * 2, err));
    auto* pb = static_cast<__nv_bfloat16*>(ws.get(kSlotSliceB, planesB * 2, err));
    auto* lv = static_cast<int32_t*>(ws.get(kSlotLevels, level_bytes(G), err));
    const StatsLayout SL = stats_layout(m, n, k, r.num_sms);
    auto* stats = static_cast<uint8_t*>(ws.get(kSlotScaleA, SL.bytes_a, err));
    auto* scratch = static_cast<uint8_t*>(ws.get(kSlotScaleB, SL.bytes_b, err));
    if (!pa || !pb || !lv || !stats || !scratch) return GB300_ERR_NO_MEMORY;
    int* eA = reinterpret_cast<int*>(stats);
    int* eB = eA + m;
    auto* info = reinterpret_cast<SplitInfo*>(stats + SL.off_info);

    // operand strides of the logical R x K views
    const int64_t a_sr = g.ta ? 1 : g.lda, a_sp = g.ta ? g.lda : 1;
    const int64_t b_sr = g.tb ? g.ldb : 1, b_sp = g.tb ? 1 : g.ldb;
    OperandPair op;
    op.X[0] = g.A; op.X[1] = g.B;
    op.R[0] = m; op.R[1] = n;
    op.sr[0] = a_sr; op.sr[1] = b_sr;
    op.sp[0] = a_sp; op.sp[1] = b_sp;
    op.rexp[0] = eA; op.rexp[1] = eB;
    op.planes[0] = pa; op.planes[1] = pb;
    op.rpad[0] = mpad; op.rpad[1] = npad;
    op.yb0 = unsigned((m + 31) / 32);
    {
        StatsArgs sa;
        sa.op = op;
        sa.K = k;
        sa.kt = SL.kt;
        sa.chunks = SL.chunks;
        sa.count = reinterpret_cast<unsigned*>(scratch);
        sa.part = reinterpret_cast<uint2*>(scratch + SL.off_part);
        sa.group = reinterpret_cast<RowPartial*>(stats + SL.off_group);
        const double target = req.target_error > 0 ? req.target_error : double(k) * 0x1p-53;
        sa.plan = PlanArgs{kPlanProduct, mode, req.slices > 0 ? max_planes : 0, max_planes, target, info};
        cudaMemsetAsync(sa.count, 0, size_t(SL.blocks + 1) * sizeof(unsigned), st);
        stats_kernel<T><<<dim3(unsigned(SL.chunks), unsigned(SL.blocks)), 256, 0, st>>>(sa);
    }
    if (cudaError_t le = cudaGetLastError(); le != cudaSuccess) {
        if (err) *err = std::string("split pre-pass launch: ") + cudaGetErrorString(le);
        return GB300_ERR_CUDA;
    }
    {
        OperandPair sp2 = op;
        sp2.yb0 = unsigned(mpad / 32);
        const int64_t yb = mpad / 32 + npad / 32, tiles = kpad / 64;
        const int kt = tiles_per_block(tiles, yb, r.num_sms);
        const dim3 grid(unsigned((tiles + kt - 1) / kt), unsigned(yb));
        auto sk = mode == kCrt     ? slice_kernel<kCrt, T>
                  : mode == kExact ? slice_kernel<kExact, T>
                  : mode == kBf16  ? slice_kernel<kBf16, T>
                                   : slice_kernel<kBf16x3, T>;
        launch_dependent(sk, grid, dim3(256), 0, st, sp2, k, info, kpad, kt);
    }
    count_launches(2);
    if (cudaError_t le = cudaGetLastError(); le != cudaSuccess) {
        if (err) *err = std::string("split slicing launch: ") + cudaGetErrorString(le);
        return GB300_ERR_CUDA;
    }

    CUtensorMap tA, tB;
    if (!encode_tmap_2d(&tA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, pa, uint64_t(max_planes) * mpad, kpad, kpad, TM, TK,
                        CU_TENSOR_MAP_SWIZZLE_128B, err) ||
        !encode_tmap_2d(&tB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, pb, uint64_t(max_planes) * npad, kpad, kpad, TNH, TK,
                        CU_TENSOR_MAP_SWIZZLE_128B, err))
        return GB300_ERR_CUDA;

    CUtensorMap tC0 = tA, tC = tA;
    if (mode == kCrt && !crt_plane_maps(&tC0, &tC, lv, nseg, max_levels, mpad, npad, err)) return GB300_ERR_CUDA;

    TcParams p;
    p.mode = mode;
    p.m_tiles = m_tiles;
    p.n_tiles = n_tiles;
    p.nseg = nseg;
    p.kb_per_seg = int(kseg / TK);
    p.kb_total = kb_total;
    p.mpad = mpad;
    p.npad = npad;
    p.levels = lv;
    p.max_levels = max_levels;
    p.info = info;
    p.status = ctl.status;
    p.limit_ns = ctl.wait_limit_ns;
    p.inject_stall = ctl.inject_stall;
    // units: one level of one pair tile and k-segment (the device picks the level count, at most
    // max_levels); CTA pairs (clusters of two): at most one pair per unit, at least one pair
    const int sms = req.max_sms > 0 ? std::min(req.max_sms, r.num_sms) : r.num_sms;
    auto kern = mode == kCrt ? tc_gemm_kernel<kCrt>
                             : mode == kExact ? tc_gemm_kernel<kExact>
                                              : (mode == kBf16 ? tc_gemm_kernel<kBf16> : tc_gemm_kernel<kBf16x3>);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTcSmem));
    if (e != cudaSuccess) {
        if (err) *err = std::string("tc_gemm_kernel smem attribute: ") + cudaGetErrorString(e);
        return GB300_ERR_CUDA;
    }
    auto launch_tc = [&](int tn0, int nt) {
        TcParams q = p;
        q.tn0 = tn0;
        q.n_tiles = nt;
        const int units = m_tiles * nt * nseg * max_levels;
        const int grid = 2 * std::max(1, std::min(units, sms / 2));
        KernelTimer timer("tc_gemm", st);
        launch_dependent(kern, dim3(unsigned(grid)), dim3(THREADS), kTcSmem, st, tA, tB, tC0, tC, q);
    };
    // reconstruction of C's columns [c0, c0 + nc) on stream s, `dependent` on the launch ahead of it there
    auto launch_crt_combine = [&](int64_t c0, int64_t nc, cudaStream_t s, bool dependent) {
        const CrtCombine<T> q{reinterpret_cast<const uint8_t*>(lv), mpad, npad, nseg, max_levels, 0, c0, m, nc, eA, eB,
                              g.alpha, g.beta, static_cast<T*>(g.C), g.ldc, false};
        if (dependent) launch_dependent(crt_combine_kernel<T>, crt_combine_grid(m, nc, r.num_sms), dim3(128), 0, s, q, info);
        else crt_combine_kernel<T><<<crt_combine_grid(m, nc, r.num_sms), 128, 0, s>>>(q, info);
    };
    const bool in_parts = mode == kCrt && n_tiles >= 2 && m_tiles * n_tiles >= sms && req.max_sms <= 0;
    if (in_parts) {
        PartEvents pe;
        if (!part_events_get(st, &pe, err)) return GB300_ERR_CUDA;
        const int nt0 = n_tiles / 2;
        const int64_t c0 = int64_t(nt0) * TN;
        launch_tc(0, nt0);
        cudaEventRecord(pe.tc0, st);
        launch_tc(nt0, n_tiles - nt0);
        cudaStreamWaitEvent(pe.aux, pe.tc0, 0);
        launch_crt_combine(0, c0, pe.aux, false);
        cudaEventRecord(pe.done0, pe.aux);
        // not dependent: its blocks would be in line from the second tensor-core launch's start and take the
        // SMs before the first part's (which then ended 50 us after it at 65536 x 256 x 256: 255 us from the
        // first launch to the end of both, 246 this way)
        launch_crt_combine(c0, n - c0, st, false);
        cudaStreamWaitEvent(st, pe.done0, 0);
        part_events_put(pe);
        count_launches(2);
    } else {
        launch_tc(0, n_tiles);
        if (mode == kCrt) {
            launch_crt_combine(0, n, st, true);
        } else {
            const int64_t colgroups = (n + COMBINE_COLS - 1) / COMBINE_COLS;
            dim3 cgrid(unsigned((colgroups + 127) / 128), unsigned(std::min<int64_t>(m, 65535)));
            combine_kernel<T><<<cgrid, 128, 0, st>>>(lv, nseg, max_levels, mpad, npad, mode, info, eA, eB, m, n, g.alpha,
                                                     g.beta, static_cast<T*>(g.C), g.ldc);
        }
    }
    count_launches(2);
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        if (err) *err = std::string("split-precision launch: ") + cudaGetErrorString(e);
        return GB300_ERR_CUDA;
    }
    out->method_used = mode == kCrt ? GB300_METHOD_SPLIT_CRT
                                    : (req.method == GB300_METHOD_AUTO || req.method == GB300_METHOD_SPLIT_CRT)
                                          ? GB300_METHOD_SPLIT
                                          : req.method;
    out->slices = -1;  // filled in by the caller from the device info when synchronous
    out->error_bound = -1.0;
    out->info_dev = info;
    return GB300_OK;
}


}  // namespace

int device_product(const Gemm& g_in, const SplitRequest& req, const LaunchCtl& ctl, cudaStream_t st, Workspace& ws,
                   SplitResult* out, std::string* err) {
    Gemm g = g_in;
    const int rst = realign_operands(g, runs_tma_tiles(g, req, ctl.inject_stall != 0), 8, ws, st, err);
    if (rst != GB300_OK) return rst;
    if (runs_native(g, req)) return native_product(g, ctl, st, ws, out, err);
    return tensor_product<double>(g, req, ctl, st, ws, out, err);
}

// A float product through the FP64-accurate machinery at the float target (k 2^-24 unless the request
// sets one).  The statistics and the slicing read the float operands, whose values a double holds
// exactly, and the reconstruction's double result (with alpha and beta applied in double) is rounded
// once to float; widened copies of A, B and C beside them took 39 us of a 2048^3 product.  The
// reported bound adds 2^-24 for that rounding.
int device_product_float(const Gemm& g_in, const SplitRequest& req_in, const LaunchCtl& ctl, cudaStream_t st,
                         Workspace& ws, SplitResult* out, std::string* err) {
    Gemm g = g_in;
    const int rst = realign_operands(g, false, 4, ws, st, err);
    if (rst != GB300_OK) return rst;
    SplitRequest req = req_in;
    if (req.target_error <= 0) req.target_error = double(std::max<int64_t>(g.k, 1)) * 0x1p-24;
    const int st_ = tensor_product<float>(g, req, ctl, st, ws, out, err);
    if (st_ == GB300_OK && out->error_bound >= 0) out->error_bound += 0x1p-24;
    return st_;
}

namespace {
bool page_locked(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeHost;
}

bool pipe_init(Runtime& r, std::string* err) {
    if (r.pipe_ready) return true;
    if (cudaStreamCreateWithFlags(&r.copy_in, cudaStreamNonBlocking) != cudaSuccess ||
        cudaStreamCreateWithFlags(&r.copy_out, cudaStreamNonBlocking) != cudaSuccess) {
        if (err) *err = "copy stream creation failed";
        return false;
    }
    for (int i = 0; i < Runtime::kPipeEvents; ++i)
        if (cudaEventCreateWithFlags(&r.pipe_ev[i], cudaEventDisableTiming) != cudaSuccess) {
            if (err) *err = "event creation failed";
            return false;
        }
    r.pipe_ready = true;
    return true;
}
}  // namespace

int device_product_host_panels(const Gemm& g, const SplitRequest& req, const LaunchCtl& ctl, cudaStream_t st,
                               Workspace& ws, SplitResult* out, std::string* err) {
    Runtime& r = runtime();
    const int64_t m = g.m, n = g.n, k = g.k;
    if (k == 0 || req.method == GB300_METHOD_NATIVE || (req.method == GB300_METHOD_AUTO && auto_uses_native(g)) ||
        req.max_sms > 0 || req.slices > 0)
        return GB300_ERR_NOT_SUPPORTED;
    const SplitGeometry G = split_geometry(g, req, r.num_sms);
    if (G.mode != kCrt) return GB300_ERR_NOT_SUPPORTED;
    // blocks: row panels of about a quarter of A (at least 2048 rows) and up to kPipeMaxQ column
    // blocks of B of at least 2048 columns each, whole pair tiles.  Four column blocks at 8192^3
    // start the first block earlier (A_0 and B_0 are 256 MiB instead of 384) but measured the same
    // end to end and 1 % slower with pageable memory; loading A and B alternately in quarters over a
    // 4 x 4 grid measured 6 % slower (the copies of C back then share the link with more of the
    // copies in).
    const bool c_locked = page_locked(g.C);
    const int64_t Mp = std::max<int64_t>(2048, round_up((m + 3) / 4, TMP));
    const int P = int((m + Mp - 1) / Mp);
    const int64_t Q0 = std::max<int64_t>(1, std::min<int64_t>(kPipeMaxQ, n / 2048));
    const int64_t Nq = round_up((n + Q0 - 1) / Q0, TN);
    const int Q = int((n + Nq - 1) / Nq);
    if (P < 2 || P > 16 || Q > kPipeMaxQ) return GB300_ERR_NOT_SUPPORTED;
    if (!pipe_init(r, err)) return GB300_ERR_CUDA;
    Gemm gp = g;
    gp.m = Mp;
    gp.n = Nq;
    const SplitGeometry Gp = split_geometry(gp, req, r.num_sms);
    const int64_t mpad = Gp.mpad, kpad = Gp.kpad;
    // B planes plane-major over the whole width: plane b holds the Q * Nq columns of every column
    // block (block j at rows j * Nq..), so one tensor map addresses all blocks and one launch can
    // cover all blocks of a panel
    const int max_planes = Gp.max_planes, max_levels = Gp.max_levels, nseg = Gp.nseg;
    const int64_t npb = int64_t(Q) * Nq;

    // device copies of the operands in their stored shapes (dense pitch), C, planes, levels, statistics
    const int64_t a_rows = g.ta ? k : m, a_cols = g.ta ? m : k;
    const int64_t b_rows = g.tb ? n : k, b_cols = g.tb ? k : n;
    auto* dA = static_cast<double*>(ws.get(kSlotA, size_t(a_rows) * size_t(a_cols) * 8, err));
    auto* dB = static_cast<double*>(ws.get(kSlotB, size_t(b_rows) * size_t(b_cols) * 8, err));
    auto* dC = static_cast<double*>(ws.get(kSlotC, size_t(m) * size_t(n) * 8, err));
    // A planes of one panel: a panel's blocks all run before the next panel is sliced
    auto* pa = static_cast<__nv_bfloat16*>(ws.get(kSlotSliceA, size_t(max_planes) * size_t(mpad) * size_t(kpad) * 2, err));
    auto* pb = static_cast<__nv_bfloat16*>(ws.get(kSlotSliceB, size_t(max_planes) * size_t(npb) * size_t(kpad) * 2, err));
    // level planes of a launch over the whole width, two buffers: launch L's reconstructions (on the
    // second stream) read buffer L % 2 while launch L + 1's tensor-core work writes the other
    const size_t lv_elems = level_bytes(Gp) / size_t(mpad) / size_t(Gp.npad) * size_t(mpad) * size_t(npb) / 4;
    auto* lv = static_cast<int32_t*>(ws.get(kSlotLevels, 2 * lv_elems * 4, err));
    // exponents, then the infos; counters of every panel and column block, then the row blocks' partials
    // and the chunk partials of the one being worked on (they follow one another on st)
    const int64_t off_info = round_up((m + n) * int64_t(sizeof(int)), 256);
    const int ninfo = P + Q + P * Q + P + 1;
    const size_t info_stride = ((sizeof(SplitInfo) + 255) / 256) * 256;
    const StatsLayout LA = stats_layout(Mp, 0, k, r.num_sms), LB = stats_layout(0, Nq, k, r.num_sms);
    const size_t count_bytes = size_t(round_up((int64_t(P) * (LA.blocks + 1) + int64_t(Q) * (LB.blocks + 1)) * 4, 256));
    const size_t group_bytes = size_t(round_up(std::max(LA.blocks, LB.blocks) * int64_t(sizeof(RowPartial)), 256));
    auto part_bytes = [&](int64_t rows) {  // whatever chunks a last, shorter panel takes
        return size_t(rows) * size_t((k + 63) / 64) * sizeof(uint2);
    };
    auto* stats = static_cast<uint8_t*>(ws.get(kSlotScaleA, size_t(off_info) + size_t(ninfo) * info_stride, err));
    auto* scratch = static_cast<uint8_t*>(
        ws.get(kSlotScaleB, count_bytes + group_bytes + part_bytes(std::max(Mp, Nq)), err));
    if (!dA || !dB || !dC || !pa || !pb || !lv || !stats || !scratch) return GB300_ERR_NO_MEMORY;
    int* eA = reinterpret_cast<int*>(stats);
    int* eB = eA + m;
    auto info_at = [&](int i) { return reinterpret_cast<SplitInfo*>(stats + off_info + size_t(i) * info_stride); };
    // infos: [0, P) panels of A, [P, P+Q) blocks of B, [P+Q, P+Q+PQ) blocks of C, [P+Q+PQ,
    // P+Q+PQ+P) the launches over a whole panel (the largest level count of its blocks), last: summary
    SplitInfo* info_sum = info_at(ninfo - 1);
    const double target = req.target_error > 0 ? req.target_error : double(k) * 0x1p-53;
    // events: [0, P) A panels in, [P, P+Q) B blocks in, [P+Q, P+Q+PQ) C blocks computed, next:
    // all out, then [P+Q+PQ+1, P+Q+2PQ+1) the launches' tensor-core work done, then PQ for the first
    // row halves of the C blocks
    cudaEvent_t* ev = r.pipe_ev;
    if (P + Q + 2 * P * Q + 1 > kPipeMaxEvents) return GB300_ERR_NOT_SUPPORTED;
    static_assert(Runtime::kPipeEvents >= kPipeMaxEvents + kPipeMaxEvents / 2, "events of the row halves");
    cudaStream_t aux = aux_stream_for(st, err);
    if (!aux) return GB300_ERR_CUDA;
    auto cuda_fail = [&](const char* what, cudaError_t e) {
        if (err) *err = std::string(what) + ": " + cudaGetErrorString(e);
        return GB300_ERR_CUDA;
    };
    const double* hA = static_cast<const double*>(g.A);
    const double* hB = static_cast<const double*>(g.B);
    double* hC = static_cast<double*>(g.C);

    // ---- copies in (issued by `load` below, in its order) ----
    cudaError_t e = cudaSuccess;
    auto copy_a = [&](int i) {
        const int64_t r0 = int64_t(i) * Mp, mi = std::min(Mp, m - r0);
        if (g.ta)  // columns r0.. of the stored k x m operand
            e = cudaMemcpy2DAsync(dA + r0, size_t(a_cols) * 8, hA + r0, size_t(g.lda) * 8, size_t(mi) * 8, size_t(k),
                                  cudaMemcpyHostToDevice, r.copy_in);
        else
            e = cudaMemcpy2DAsync(dA + r0 * a_cols, size_t(a_cols) * 8, hA + r0 * g.lda, size_t(g.lda) * 8,
                                  size_t(k) * 8, size_t(mi), cudaMemcpyHostToDevice, r.copy_in);
        if (e == cudaSuccess && g.beta != 0.0)
            e = cudaMemcpy2DAsync(dC + r0 * n, size_t(n) * 8, hC + r0 * g.ldc, size_t(g.ldc) * 8, size_t(n) * 8,
                                  size_t(mi), cudaMemcpyHostToDevice, r.copy_in);
        cudaEventRecord(ev[i], r.copy_in);
    };
    auto copy_b = [&](int j) {
        const int64_t c0 = int64_t(j) * Nq, nj = std::min(Nq, n - c0);
        if (g.tb)  // rows c0.. of the stored n x k operand
            e = cudaMemcpy2DAsync(dB + c0 * b_cols, size_t(b_cols) * 8, hB + c0 * g.ldb, size_t(g.ldb) * 8,
                                  size_t(k) * 8, size_t(nj), cudaMemcpyHostToDevice, r.copy_in);
        else
            e = cudaMemcpy2DAsync(dB + c0, size_t(b_cols) * 8, hB + c0, size_t(g.ldb) * 8, size_t(nj) * 8, size_t(k),
                                  cudaMemcpyHostToDevice, r.copy_in);
        cudaEventRecord(ev[P + j], r.copy_in);
    };
    cudaMemsetAsync(scratch, 0, count_bytes, st);
    // the pre-pass launches over a panel or a column block
    auto run_stats = [&](const OperandPair& o, const StatsLayout& L, int64_t first_counter, SplitInfo* info) {
        StatsArgs sa;
        sa.op = o;
        sa.K = k;
        sa.kt = L.kt;
        sa.chunks = L.chunks;
        sa.count = reinterpret_cast<unsigned*>(scratch) + first_counter;
        sa.group = reinterpret_cast<RowPartial*>(scratch + count_bytes);
        sa.part = reinterpret_cast<uint2*>(scratch + count_bytes + group_bytes);
        sa.plan = PlanArgs{kPlanSide, kCrt, 0, max_planes, target, info};
        stats_kernel<double><<<dim3(unsigned(L.chunks), unsigned(L.blocks)), 256, 0, st>>>(sa);
    };
    auto run_slice = [&](const OperandPair& o, int64_t yb, const SplitInfo* info) {
        const int64_t tiles = kpad / 64;
        const int kt = tiles_per_block(tiles, yb, r.num_sms);
        launch_dependent(slice_kernel<kCrt, double>, dim3(unsigned((tiles + kt - 1) / kt), unsigned(yb)), dim3(256), 0, st, o, k,
                         info, kpad, kt);
    };
    const int64_t a_sr = g.ta ? 1 : a_cols, a_sp = g.ta ? a_cols : 1;
    const int64_t b_sr = g.tb ? b_cols : 1, b_sp = g.tb ? 1 : b_cols;
    OperandPair base;
    base.X[0] = dA; base.X[1] = dB;
    base.R[0] = 0; base.R[1] = 0;
    base.sr[0] = a_sr; base.sr[1] = b_sr;
    base.sp[0] = a_sp; base.sp[1] = b_sp;
    base.rexp[0] = eA; base.rexp[1] = eB;
    base.planes[0] = pa; base.planes[1] = pb;
    base.rpad[0] = mpad; base.rpad[1] = npb;
    base.yb0 = 0;
    // statistics, side scaling and planes of A's panel i (into the panel plane buffer)
    auto prep_a = [&](int i) {
        const int64_t r0 = int64_t(i) * Mp, mi = std::min(Mp, m - r0);
        OperandPair o = base;
        o.X[0] = g.ta ? dA + r0 : dA + r0 * a_cols;
        o.R[0] = mi;
        o.rexp[0] = eA + r0;
        o.yb0 = unsigned((mi + 31) / 32);
        run_stats(o, stats_layout(mi, 0, k, r.num_sms), int64_t(i) * (LA.blocks + 1), info_at(i));
        o.yb0 = unsigned(mpad / 32);
        run_slice(o, o.yb0, info_at(i));
        count_launches(2);
    };
    // statistics, side scaling and planes of B's column block j (rows j*Nq.. of the B planes)
    auto prep_b = [&](int j) {
        const int64_t c0 = int64_t(j) * Nq, nj = std::min(Nq, n - c0);
        OperandPair o = base;
        o.X[1] = g.tb ? dB + c0 * b_cols : dB + c0;
        o.R[1] = nj;
        o.rexp[1] = eB + c0;
        o.planes[1] = pb + size_t(j) * size_t(Nq) * size_t(kpad);
        o.rpad[1] = npb;
        o.yb0 = 0;
        run_stats(o, stats_layout(0, nj, k, r.num_sms), int64_t(P) * (LA.blocks + 1) + int64_t(j) * (LB.blocks + 1),
                  info_at(P + j));
        run_slice(o, Nq / 32, info_at(P + j));
        count_launches(2);
    };

    // ---- tensor maps: A panel planes, the B planes, the level planes of a launch ----
    CUtensorMap tA, tB, tC0[2], tC[2];
    if (!encode_tmap_2d(&tA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, pa, uint64_t(max_planes) * mpad, kpad, kpad, TM, TK,
                        CU_TENSOR_MAP_SWIZZLE_128B, err) ||
        !encode_tmap_2d(&tB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, pb, uint64_t(max_planes) * npb, kpad, kpad, TNH, TK,
                        CU_TENSOR_MAP_SWIZZLE_128B, err))
        return GB300_ERR_CUDA;
    for (int b = 0; b < 2; ++b)
        if (!crt_plane_maps(&tC0[b], &tC[b], lv + b * lv_elems, nseg, max_levels, mpad, npb, err)) return GB300_ERR_CUDA;
    e = cudaFuncSetAttribute(tc_gemm_kernel<kCrt>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTcSmem));
    if (e != cudaSuccess) return cuda_fail("tc_gemm_kernel smem attribute", e);

    // ---- operands in, blocks as their operands arrive, C back ----
    // Load order A_0, B_0 .. B_{Q-1}, A_1 .. A_{P-1}; after each load the blocks it completes are
    // queued (block (i, j) needs A_i and B_j), so panel i's blocks run together on the panel's
    // planes.  With page-locked memory every call returns at once; with pageable memory each copy
    // holds the host thread until it is done, and the order keeps the GPU busy meanwhile: A_i+1
    // goes in and panel i-1 comes out while panel i computes.  C goes back per block as soon as the
    // block is done (page-locked C); a pageable C goes back per panel, one linear copy when its rows
    // are exactly n elements (pitched copies into untouched pageable pages are slow, see
    // copy_to_host), else per block.
    const bool c_per_panel = !c_locked && Q > 1 && g.ldc == n;
    auto block_ev = [&](int i, int j) { return ev[P + Q + i * Q + j]; };
    auto half_ev = [&](int i, int j) { return ev[P + Q + 2 * P * Q + 1 + i * Q + j]; };
    auto half_rows = [](int64_t rows) { return (rows + 1) / 2; };
    auto copy_block_out = [&](int i, int j) {
        const int64_t r0 = int64_t(i) * Mp, mi = std::min(Mp, m - r0);
        const int64_t c0 = int64_t(j) * Nq, nj = std::min(Nq, n - c0);
        // in row halves where the copies are asynchronous; into pageable memory the host thread would wait
        // for each half, and pages touched for the first time come in slower by pieces (a first 3000 x
        // 2000 x 2500 call into a fresh C: 4.25 ms in halves, 3.7 in one copy)
        for (int h = c_locked ? 0 : 1; h < 2 && e == cudaSuccess; ++h) {
            const int64_t h0 = h && c_locked ? half_rows(mi) : 0, h1 = h ? mi : half_rows(mi);
            if (h1 == h0) continue;
            cudaStreamWaitEvent(r.copy_out, h ? block_ev(i, j) : half_ev(i, j), 0);
            e = copy_to_host(hC + (r0 + h0) * g.ldc + c0, size_t(g.ldc) * 8, dC + (r0 + h0) * n + c0, size_t(n) * 8,
                             size_t(nj) * 8, size_t(h1 - h0), r.copy_out);
        }
    };
    auto copy_panel_out = [&](int i) {
        if (!c_per_panel) {
            for (int j = 0; j < Q && e == cudaSuccess; ++j) copy_block_out(i, j);
            return;
        }
        const int64_t r0 = int64_t(i) * Mp, mi = std::min(Mp, m - r0);
        for (int j = 0; j < Q; ++j) cudaStreamWaitEvent(r.copy_out, block_ev(i, j), 0);
        e = copy_to_host(hC + r0 * g.ldc, size_t(g.ldc) * 8, dC + r0 * n, size_t(n) * 8, size_t(n) * 8, size_t(mi),
                         r.copy_out);
    };
    // Launch L (blocks j0..j1-1 of panel i, one tensor-core launch) writes level buffer L % 2 on st;
    // each block's reconstruction runs on the second stream and records the block's event, which the
    // copies of C wait on; launch L + 2 waits for launch L's reconstructions before it overwrites the
    // buffer.  A panel whose A arrives after all of B runs as one launch (fewer, fuller waves of pair
    // units than a launch per block), except the last: its blocks' copies back then start one block
    // earlier; the first panel's blocks run as their B blocks arrive.
    int nlaunch = 0;
    int launch_i[16 * kPipeMaxQ], launch_j0[16 * kPipeMaxQ], launch_j1[16 * kPipeMaxQ];
    auto tc_done_ev = [&](int l) { return ev[P + Q + P * Q + 1 + l]; };
    auto run_blocks = [&](int i, int j0, int j1) {
        const int64_t r0 = int64_t(i) * Mp, mi = std::min(Mp, m - r0);
        const int64_t c0 = int64_t(j0) * Nq, c1 = std::min(n, int64_t(j1) * Nq);
        const int l = nlaunch++;
        const int buf = l & 1;
        int32_t* lvb = lv + buf * lv_elems;
        if (l >= 2)
            for (int j = launch_j0[l - 2]; j < launch_j1[l - 2]; ++j)
                cudaStreamWaitEvent(st, block_ev(launch_i[l - 2], j), 0);
        launch_i[l] = i;
        launch_j0[l] = j0;
        launch_j1[l] = j1;
        for (int j = j0; j < j1; ++j)
            split_block_kernel<<<1, 32, 0, st>>>(info_at(i), info_at(P + j), k, max_planes, info_at(P + Q + i * Q + j));
        SplitInfo* linfo = info_at(P + Q + i * Q + j0);
        if (j1 - j0 > 1) {
            linfo = info_at(P + Q + P * Q + i);
            split_max_slices_kernel<<<1, 32, 0, st>>>(reinterpret_cast<const uint8_t*>(info_at(P + Q + i * Q + j0)),
                                                      info_stride, j1 - j0, linfo);
            count_launches(1);
        }
        TcParams tp;
        tp.mode = kCrt;
        tp.m_tiles = int((mi + TMP - 1) / TMP);
        tp.tn0 = int(c0 / TN);
        tp.n_tiles = int((c1 - c0 + TN - 1) / TN);
        tp.nseg = nseg;
        tp.kb_per_seg = int(Gp.kseg / TK);
        tp.kb_total = Gp.kb_total;
        tp.mpad = mpad;
        tp.npad = npb;
        tp.levels = lvb;
        tp.max_levels = max_levels;
        tp.info = linfo;
        tp.status = ctl.status;
        tp.limit_ns = ctl.wait_limit_ns;
        tp.inject_stall = ctl.inject_stall;
        const int units = tp.m_tiles * tp.n_tiles * nseg * max_levels;
        const int grid = 2 * std::max(1, std::min(units, r.num_sms / 2));
        {
            KernelTimer timer("tc_gemm", st);
            launch_dependent(tc_gemm_kernel<kCrt>, dim3(unsigned(grid)), dim3(THREADS), kTcSmem, st, tA, tB, tC0[buf],
                             tC[buf], tp);
        }
        cudaEventRecord(tc_done_ev(l), st);
        cudaStreamWaitEvent(aux, tc_done_ev(l), 0);
        for (int j = j0; j < j1; ++j) {
            const int64_t cj = int64_t(j) * Nq, nj = std::min(Nq, n - cj);
            // in two row halves, so that the first one's copy back starts while the second is reconstructed;
            // the second is a dependent launch, whose blocks are in line from the first one's start: behind
            // its end they came after the next panel's pre-pass, and with pageable memory the host
            // then waited longer for the panel's C (8192^3 12.4 ms a call, now 11.1)
            for (int h = 0; h < 2; ++h) {
                const int64_t h0 = h ? half_rows(mi) : 0, h1 = h ? mi : half_rows(mi);
                const CrtCombine<double> q{reinterpret_cast<const uint8_t*>(lvb), mpad, npb, nseg, max_levels, h0, cj, h1 - h0, nj,
                                           eA + r0, eB, g.alpha, g.beta, dC + r0 * n, n, h == 0};
                const dim3 grid = crt_combine_grid(h1 - h0, nj, r.num_sms);
                const SplitInfo* info = info_at(P + Q + i * Q + j);
                if (h) launch_dependent(crt_combine_kernel<double>, grid, dim3(128), 0, aux, q, info);
                else crt_combine_kernel<double><<<grid, 128, 0, aux>>>(q, info);
                if ((e = cudaGetLastError()) != cudaSuccess) return;
                cudaEventRecord(h ? block_ev(i, j) : half_ev(i, j), aux);
            }
            if (c_locked) copy_block_out(i, j);
        }
        count_launches(1 + 3 * (j1 - j0));
    };
    bool have_a[16] = {}, have_b[kPipeMaxQ] = {};
    int nb = 0;  // B blocks in
    auto load = [&](int side, int idx) {
        if (side == 0) {
            copy_a(idx);
            if (e != cudaSuccess) return;
            cudaStreamWaitEvent(st, ev[idx], 0);
            prep_a(idx);
            have_a[idx] = true;
            if (nb == Q && idx + 1 < P) run_blocks(idx, 0, Q);
            else
                for (int j = 0; j < Q && e == cudaSuccess; ++j)
                    if (have_b[j]) run_blocks(idx, j, j + 1);
        } else {
            copy_b(idx);
            if (e != cudaSuccess) return;
            cudaStreamWaitEvent(st, ev[P + idx], 0);
            prep_b(idx);
            have_b[idx] = true;
            ++nb;
            for (int i = 0; i < P && e == cudaSuccess; ++i)
                if (have_a[i]) run_blocks(i, idx, idx + 1);
        }
    };
    load(0, 0);
    for (int j = 0; j < Q && e == cudaSuccess; ++j) load(1, j);
    for (int i = 1; i < P && e == cudaSuccess; ++i) {
        load(0, i);
        if (e == cudaSuccess && !c_locked) copy_panel_out(i - 1);
    }
    if (e == cudaSuccess && !c_locked) copy_panel_out(P - 1);
    if (e != cudaSuccess) return cuda_fail("block pipeline", e);
    split_panels_summary_kernel<<<1, 32, 0, st>>>(reinterpret_cast<const uint8_t*>(info_at(P + Q)), info_stride,
                                                  P * Q, info_sum);
    count_launches(1);
    cudaEventRecord(ev[P + Q + P * Q], r.copy_out);
    cudaStreamWaitEvent(st, ev[P + Q + P * Q], 0);  // the call's work ends on st
    for (int l = std::max(0, nlaunch - 2); l < nlaunch; ++l)  // and so does the second stream's
        for (int j = launch_j0[l]; j < launch_j1[l]; ++j) cudaStreamWaitEvent(st, block_ev(launch_i[l], j), 0);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail("block pipeline", e);
    out->method_used = GB300_METHOD_SPLIT_CRT;
    out->slices = -1;
    out->error_bound = -1.0;
    out->info_dev = info_sum;
    return GB300_OK;
}

}  // namespace gb
