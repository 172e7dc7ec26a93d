// grouped.cu — K4: persistent grouped GEMM for many independent, uneven, small products
// (Blaze's StaticMatrix / HybridMatrix sizes), FP64 (DFMA) and FP32 (FFMA), one launch per batch,
// captured in a CUDA graph, with warp-tile shapes picked per size class by an autotuner.
//
// Blaze evaluates every such product separately on the CPU through its small vectorized kernel
// (blaze/math/expressions/DMatDMatMultExpr.h:864-1878, DMatTDMatMultExpr.h:1067+); it has no
// batched product, so this is a new entry point (gb300_?gemm_grouped) with the per-product CBLAS
// argument conventions.
//
// Design:
//   * Every product is brought to the row-major form (as for the single products) and tiled with
//     the warp-tile shape chosen for its (m, n, k) class: FP32 warp tiles of (8*R) x (4*C) outputs, FP64
//     tiles of at most that many, taken as flat lists of outputs (warp_tile_flat).
//   * One flat tile list, sorted by descending work (longest first), is consumed by persistent
//     warps through a global atomic counter (warp-granular work stealing): uneven products
//     balance across SMs without a per-product launch.
//   * Operands are staged in the warp's own shared memory, so a warp waits for no other.
//   * The launch (counter reset + kernel) is captured once into a CUDA graph owned by the plan;
//     running the plan is one graph launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <mutex>
#include <sstream>
#include <string>
#include <vector>

#include "../../include/gb300_blas.h"
#include "ptx.cuh"
#include "runtime.h"

namespace gb {
namespace {

// Warp-tile shapes: (R, C) -> (8R) x (4C) outputs per warp.
struct Shape {
    int R, C;
};
constexpr Shape kShapes[] = {{1, 2}, {2, 4}, {4, 4}, {2, 8}, {4, 8}, {8, 8}};
constexpr int kNumShapes = sizeof(kShapes) / sizeof(kShapes[0]);
__host__ __device__ constexpr int shape_rows(int s) { return s == 0 ? 8 : s == 1 ? 16 : s == 2 ? 32 : s == 3 ? 16 : s == 4 ? 32 : 64; }
__host__ __device__ constexpr int shape_cols(int s) { return s == 0 ? 8 : s == 1 ? 16 : s == 2 ? 16 : s == 3 ? 32 : s == 4 ? 32 : 32; }

struct DevProblem {
    const void* A;
    const void* B;
    void* C;
    int64_t lda, ldb, ldc;
    int m, n, k;
    int ta, tb;
    int shape;
    int tr, tc;  // rows and columns of its tiles (the last ones of a row or column may be smaller)
    double alpha, beta;
};

struct DevTile {
    int prob;
    int tm, tn;  // tile coordinates in units of the problem's warp tile
    int pad;
};

// FP64 warp tiles.  On this chip a multiply-add of a warp holds its SM quarter's FP64 pipe for 64
// clocks, so what a tile costs is the number of its multiply-add instructions, and loads are free.  A
// warp therefore takes its tile's outputs as one flat list, 32 at a time, whatever the tile's rows and
// columns are: output o of lane l in round u is o = l + 32 u, row o / cols, column o % cols, each lane
// reading its own A and B value from the warp's staged chunk for every multiply-add.  A product is
// split into tiles of equal parts (tr x tc, within the shape's rows and columns), which leaves at most
// 31 idle outputs a tile: 1.03 times the useful work on 10,000 products of 4 to 256 rows, columns and
// steps, against 1.22 with tiles of fixed 8 R x 4 C outputs (4.58 ms, now 3.77, 0.94 of the FP64
// peak).  The operands come in by
// cp.async, DKC k-steps ahead of the ones being used.  Every output sums k in order.
constexpr int DKC = 16;
constexpr int DPA = DKC + 1;                        // A row pitch (doubles): rows 2 banks apart
constexpr int kDStage = 32 * DPA + DKC * 17;       // doubles per buffer: 32 x 16 tiles need most, then 16 x 32
static_assert(kDStage >= 16 * DPA + DKC * 33, "16 x 32 tiles");
constexpr int kDStageBytes = 8 * 2 * kDStage * int(sizeof(double));  // per 256-thread block

// kc k-steps of the first U rounds.  U is a template argument so that no multiply-add is issued for the
// rounds a tile does not have: one that is predicated off for the whole warp holds the FP64 pipe as
// long as any other (4.75 ms against 3.93 before the epilogue was split as well).
template <int U, int UMAX>
__device__ __forceinline__ void flat_steps(const double* buf, int kc, int pb, const int (&ao)[UMAX],
                                           const int (&bo)[UMAX], double (&acc)[UMAX]) {
#pragma unroll 2
    for (int kk = 0; kk < kc; ++kk) {
        const double* a = buf + kk;
        const double* c = buf + kk * pb;
#pragma unroll
        for (int u = 0; u < U; ++u) acc[u] = fma(a[ao[u]], c[bo[u]], acc[u]);
    }
}

// The flat tile of `rows` x `cols` outputs at (i0, j0), UMAX rounds at most.
constexpr int UMAX = 16;
__device__ __forceinline__ void warp_tile_flat(const DevProblem& p, int i0, int j0, int rows, int cols, int lane,
                                               double* sw) {
    const int outs = rows * cols, U = (outs + 31) >> 5;
    const int pb = cols | 1, bbase = rows * DPA;  // B row pitch, and where B's chunk begins
    const double* A = static_cast<const double*>(p.A) + (p.ta ? int64_t(i0) : int64_t(i0) * p.lda);
    const double* B = static_cast<const double*>(p.B) + (p.tb ? int64_t(j0) * p.ldb : int64_t(j0));
    double acc[UMAX];
    int ao[UMAX], bo[UMAX];
#pragma unroll
    for (int u = 0; u < UMAX; ++u) {
        const int o = min(lane + 32 * u, outs - 1);
        const int i = o / cols;
        ao[u] = i * DPA;
        bo[u] = bbase + o - i * cols;
        acc[u] = 0.0;
    }
    // k-steps k0 .. k0 + kc - 1 of the tile's rows of A and columns of B into a buffer
    auto stage = [&](double* buf, int k0) {
        const int kc = min(DKC, p.k - k0);
        const uint32_t sa = smem_u32(buf), sb = smem_u32(buf + bbase);
        if (!p.ta) {
            const int kk = lane & (DKC - 1);
            if (kk < kc)
                for (int i = lane / DKC; i < rows; i += 32 / DKC)
                    cp_async8(sa + uint32_t(i * DPA + kk) * 8u, A + int64_t(i) * p.lda + k0 + kk, true);
        } else {
            for (int e = lane; e < rows * kc; e += 32) {
                const int kk = e / rows, i = e - kk * rows;
                cp_async8(sa + uint32_t(i * DPA + kk) * 8u, A + int64_t(k0 + kk) * p.lda + i, true);
            }
        }
        if (!p.tb) {
            for (int e = lane; e < cols * kc; e += 32) {
                const int kk = e / cols, j = e - kk * cols;
                cp_async8(sb + uint32_t(kk * pb + j) * 8u, B + int64_t(k0 + kk) * p.ldb + j, true);
            }
        } else {
            const int kk = lane & (DKC - 1);
            if (kk < kc)
                for (int j = lane / DKC; j < cols; j += 32 / DKC)
                    cp_async8(sb + uint32_t(kk * pb + j) * 8u, B + int64_t(j) * p.ldb + k0 + kk, true);
        }
    };
    if (p.k > 0) stage(sw, 0);
    cp_async_commit();
    int b = 0;
    for (int k0 = 0; k0 < p.k; k0 += DKC, b ^= 1) {
        if (k0 + DKC < p.k) stage(sw + (b ^ 1) * kDStage, k0 + DKC);
        cp_async_commit();  // an empty group keeps the wait count uniform
        cp_async_wait1();
        __syncwarp();
        const double* buf = sw + b * kDStage;
        const int kc = min(DKC, p.k - k0);
        switch (U) {
#define GB_FLAT(n) \
    case n: flat_steps<n>(buf, kc, pb, ao, bo, acc); break;
            GB_FLAT(1) GB_FLAT(2) GB_FLAT(3) GB_FLAT(4) GB_FLAT(5) GB_FLAT(6) GB_FLAT(7) GB_FLAT(8)
            GB_FLAT(9) GB_FLAT(10) GB_FLAT(11) GB_FLAT(12) GB_FLAT(13) GB_FLAT(14) GB_FLAT(15)
#undef GB_FLAT
            default: flat_steps<16>(buf, kc, pb, ao, bo, acc); break;
        }
        __syncwarp();  // the buffer is free for the chunk after next
    }
    double* C = static_cast<double*>(p.C) + int64_t(i0) * p.ldc + j0;
    const double alpha = p.alpha, beta = p.beta;
    // a loop of its own where C = A B: multiplies by one would cost as much as a k-step
    if (alpha == 1.0 && beta == 0.0) {
#pragma unroll
        for (int u = 0; u < UMAX; ++u) {
            if (lane + 32 * u >= outs) break;
            const int i = ao[u] / DPA, j = bo[u] - bbase;
            C[int64_t(i) * p.ldc + j] = acc[u];
        }
        return;
    }
#pragma unroll
    for (int u = 0; u < UMAX; ++u) {
        if (lane + 32 * u >= outs) break;
        const int i = ao[u] / DPA, j = bo[u] - bbase;
        double* c = C + int64_t(i) * p.ldc + j;
        const double v = alpha * acc[u];
        *c = (beta == 0.0) ? v : fma(beta, *c, v);
    }
}

// FP32 warp tiles of (8 R) x (4 C) outputs: lane (ly, lx) of an 8 x 4 grid owns rows ly + 8 r and the C
// contiguous columns lx C .. lx C + C - 1.  A and B are staged KC k-steps at a time in the warp's own
// shared memory by cp.async, the next chunk on its way while one is used (16 bytes a copy where base
// and leading dimension allow it, else 4), so that a chunk costs its instructions and not its latency:
// with plain loads and stores through registers a warp waited for every row, 24 us a tile of some
// 24 x 24 x 60.  One 16-byte read of an A row serves four k-steps; its chunks are rotated by the row
// so that a warp's eight rows fall on different banks.  A k-step reads a lane's B columns 16 bytes at
// a time (8 for C = 2), and its multiply-adds are packed in pairs of columns.  Rows and columns
// outside the product are never copied in and never stored, and k-steps past the end are not added:
// every output sums its k range in order.
constexpr int KC = 16;                                    // k-steps per staged chunk
constexpr int kStageA = 32 * KC;                          // up to 32 rows (FP32 tiles stop at 32 x 32)
constexpr int kStageB = KC * (32 + 4);                    // up to 32 columns, pitch PB
constexpr int kStageBuf = kStageA + kStageB;              // floats per buffer
constexpr int kStageBytes = 8 * 2 * kStageBuf * int(sizeof(float));  // per 256-thread block

// Offset of A(row, kk): 16-byte chunk kk / 4 of a row at chunk ^ (row / 2 % 4).
__device__ __forceinline__ int a_slot(int row, int kk) { return row * KC + ((((kk >> 2) ^ (row >> 1)) & 3) << 2) + (kk & 3); }

// C consecutive floats from 16-byte (or, for C = 2, 8-byte) aligned shared memory, as packed pairs.
template <int C>
__device__ __forceinline__ void lds_pairs(const float* src, uint64_t (&v)[C / 2]) {
    if constexpr (C == 2) {
        v[0] = *reinterpret_cast<const uint64_t*>(src);
    } else {
#pragma unroll
        for (int q = 0; q < C / 4; ++q) {
            const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(src + 4 * q);
            v[2 * q] = t.x;
            v[2 * q + 1] = t.y;
        }
    }
}

constexpr int PB = 36;  // B row pitch (floats)
constexpr int kAcc = 16;  // packed accumulators a lane: 4 x 8 outputs

// kc k-steps of a staged chunk.
template <int R, int C>
__device__ __forceinline__ void f32_steps(const float* As, int kc, int ly, int lx, uint64_t (&acc)[kAcc]) {
    const float* bcol = As + kStageA + lx * C;
    const int kv = kc & ~3;
#pragma unroll 1
    for (int kk = 0; kk < kv; kk += 4) {
        float4 a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = *reinterpret_cast<const float4*>(As + a_slot(ly + 8 * r, kk));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint64_t bv[C / 2];
            lds_pairs<C>(bcol + (kk + q) * PB, bv);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float x = q == 0 ? a[r].x : q == 1 ? a[r].y : q == 2 ? a[r].z : a[r].w;
                const uint64_t x2 = f32x2(x, x);
#pragma unroll
                for (int c = 0; c < C / 2; ++c) acc[r * (C / 2) + c] = fma2(x2, bv[c], acc[r * (C / 2) + c]);
            }
        }
    }
    // the last k-steps one at a time: what lies behind the end in the buffer is never added
#pragma unroll 1
    for (int kk = kv; kk < kc; ++kk) {
        uint64_t bv[C / 2];
        lds_pairs<C>(bcol + kk * PB, bv);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float x = As[a_slot(ly + 8 * r, kk)];
            const uint64_t x2 = f32x2(x, x);
#pragma unroll
            for (int c = 0; c < C / 2; ++c) acc[r * (C / 2) + c] = fma2(x2, bv[c], acc[r * (C / 2) + c]);
        }
    }
}

// C = alpha acc + beta C for the lane's rows and columns inside the product.
template <int R, int C>
__device__ __forceinline__ void f32_store(const DevProblem& p, int i0, int j0, int rows, int cols, int ly, int lx,
                                          const uint64_t (&acc)[kAcc]) {
    const float alpha = float(p.alpha), beta = float(p.beta);
    float* Cp = static_cast<float*>(p.C) + int64_t(i0) * p.ldc + j0 + lx * C;
    const int left = cols - lx * C;  // of this lane's columns
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (ly + 8 * r >= rows) break;
        float* crow = Cp + int64_t(ly + 8 * r) * p.ldc;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            if (c >= left) break;
            const float v = alpha * __uint_as_float(uint32_t(acc[r * (C / 2) + c / 2] >> ((c & 1) * 32)));
            crow[c] = (beta == 0.f) ? v : fmaf(beta, crow[c], v);
        }
    }
}

// k-steps k0 .. of the tile's rows of A and columns of B into a buffer.  One short loop per layout for
// every tile shape: copies are asynchronous, so nothing is gained by unrolling them, and code that
// is unrolled for each shape no longer fits the instruction cache (628 us for 10,000 products instead
// of 369, two thirds of the stalls waiting for instructions).
__device__ __forceinline__ void f32_stage(const DevProblem& p, const float* __restrict__ A, const float* __restrict__ B,
                                          bool va, bool vb, int rows, int cols, int k0, int lane, uint32_t sa) {
    const int kc = min(KC, p.k - k0);
    const uint32_t sb = sa + kStageA * 4u;
    if (va) {
        const int c4 = (lane & 3) * 4, bytes = min(16, (kc - c4) * 4);
        const float* src = A + int64_t(lane >> 2) * p.lda + k0 + c4;
        if (bytes > 0)
#pragma unroll 1
            for (int i = lane >> 2; i < rows; i += 8, src += 8 * p.lda) cp_async16(sa + 4u * uint32_t(a_slot(i, c4)), src, bytes);
    } else if (!p.ta) {
        const int kk = lane & 15;
        const float* src = A + int64_t(lane >> 4) * p.lda + k0 + kk;
        if (kk < kc)
#pragma unroll 2
            for (int i = lane >> 4; i < rows; i += 2, src += 2 * p.lda) cp_async4(sa + 4u * uint32_t(a_slot(i, kk)), src, true);
    } else if (lane < rows) {
        const float* src = A + int64_t(k0) * p.lda + lane;
#pragma unroll 2
        for (int kk = 0; kk < kc; ++kk, src += p.lda) cp_async4(sa + 4u * uint32_t(a_slot(lane, kk)), src, true);
    }
    if (vb) {
        const int c4 = (lane & 7) * 4, bytes = min(16, (cols - c4) * 4);
        const float* src = B + int64_t(k0 + (lane >> 3)) * p.ldb + c4;
        if (bytes > 0)
#pragma unroll 1
            for (int kk = lane >> 3; kk < kc; kk += 4, src += 4 * p.ldb) cp_async16(sb + 4u * uint32_t(kk * PB + c4), src, bytes);
    } else if (p.tb) {
        const int kk = lane & 15;
        const float* src = B + int64_t(lane >> 4) * p.ldb + k0 + kk;
        if (kk < kc)
#pragma unroll 2
            for (int j = lane >> 4; j < cols; j += 2, src += 2 * p.ldb) cp_async4(sb + 4u * uint32_t(kk * PB + j), src, true);
    } else if (cols > 16) {
        const float* src = B + int64_t(k0) * p.ldb + lane;
        if (lane < cols)
#pragma unroll 2
            for (int kk = 0; kk < kc; ++kk, src += p.ldb) cp_async4(sb + 4u * uint32_t(kk * PB + lane), src, true);
    } else {  // two k-steps a copy instruction
        const int j = lane & 15;
        const float* src = B + int64_t(k0 + (lane >> 4)) * p.ldb + j;
        if (j < cols)
#pragma unroll 2
            for (int kk = lane >> 4; kk < kc; kk += 2, src += 2 * p.ldb) cp_async4(sb + 4u * uint32_t(kk * PB + j), src, true);
    }
}

__device__ __forceinline__ void warp_tile_staged(const DevProblem& p, int tm, int tn, int lane, float* sw) {
    const int ly = lane >> 2, lx = lane & 3;
    const int i0 = tm * p.tr, j0 = tn * p.tc;
    const int rows = min(p.tr, p.m - i0), cols = min(p.tc, p.n - j0);
    const float* A = static_cast<const float*>(p.A) + (p.ta ? int64_t(i0) : int64_t(i0) * p.lda);
    const float* B = static_cast<const float*>(p.B) + (p.tb ? int64_t(j0) * p.ldb : int64_t(j0));
    // rows (or k-steps) that can be copied 16 bytes at a time
    const bool va = !p.ta && ((reinterpret_cast<uintptr_t>(A) | uintptr_t(p.lda * 4)) & 15) == 0;
    const bool vb = !p.tb && ((reinterpret_cast<uintptr_t>(B) | uintptr_t(p.ldb * 4)) & 15) == 0;
    const uint32_t s0 = smem_u32(sw);
    uint64_t acc[kAcc];
#pragma unroll
    for (int q = 0; q < kAcc; ++q) acc[q] = 0ull;
    const int chunks = (p.k + KC - 1) / KC;
#pragma unroll 1
    for (int c = -1; c < chunks; ++c) {
        if (c + 1 < chunks)
            f32_stage(p, A, B, va, vb, rows, cols, (c + 1) * KC, lane, s0 + uint32_t((c + 1) & 1) * (kStageBuf * 4u));
        cp_async_commit();  // an empty group keeps the wait count uniform
        if (c < 0) continue;
        cp_async_wait1();
        __syncwarp();
        const float* buf = sw + (c & 1) * kStageBuf;
        const int kc = min(KC, p.k - c * KC);
        switch (p.shape) {
            case 0: f32_steps<1, 2>(buf, kc, ly, lx, acc); break;
            case 1: f32_steps<2, 4>(buf, kc, ly, lx, acc); break;
            case 2: f32_steps<4, 4>(buf, kc, ly, lx, acc); break;
            case 3: f32_steps<2, 8>(buf, kc, ly, lx, acc); break;
            default: f32_steps<4, 8>(buf, kc, ly, lx, acc); break;
        }
        __syncwarp();  // the buffer is free for the chunk after next
    }
    switch (p.shape) {
        case 0: f32_store<1, 2>(p, i0, j0, rows, cols, ly, lx, acc); break;
        case 1: f32_store<2, 4>(p, i0, j0, rows, cols, ly, lx, acc); break;
        case 2: f32_store<4, 4>(p, i0, j0, rows, cols, ly, lx, acc); break;
        case 3: f32_store<2, 8>(p, i0, j0, rows, cols, ly, lx, acc); break;
        default: f32_store<4, 8>(p, i0, j0, rows, cols, ly, lx, acc); break;
    }
}

// Shapes available per element type: FP64 stops at 16x32 / 32x16 warp tiles (16 outputs per lane), whose
// staging lets an SM hold 16 warps.  FP32 stops at 32x32 (32 accumulators per lane), so that an SM holds three
// 256-thread blocks (24 warps) to cover the latency of the staging loads.
template <typename T>
__host__ __device__ constexpr int max_shape() { return sizeof(T) == 8 ? 3 : 4; }

template <typename T>
__global__ void __launch_bounds__(256, sizeof(T) == 8 ? 2 : 3)
grouped_kernel(const DevProblem* __restrict__ probs, const DevTile* __restrict__ tiles, int ntiles,
               int* __restrict__ counter, int num_sms) {
    const int lane = threadIdx.x & 31;
    // the warps' staging regions (dynamic shared memory of kStageBytes or kDStageBytes per block)
    extern __shared__ __align__(16) float stage_smem[];
    float* sw = stage_smem + (threadIdx.x >> 5) * (2 * kStageBuf);
    (void)sw;
    // A warp's first tile is fixed, the tiles being dealt out over the blocks before a block gets its second
    // one (and over the quarters of an SM: an SM's next block starts two warps on); further ones
    // are tickets.  While there are plenty, the next tile's ticket is taken a tile ahead and its description
    // read while this tile is worked on, so that neither round trip precedes a tile (small tiles are a few
    // hundred clocks of multiply-adds).  Over the last three tiles a warp a ticket is taken when it is
    // needed: one in hand would keep its tile waiting behind a long one while other warps have nothing to
    // do (28 products of 64^3 FP64, 224 tiles for as many warps: 165 us with every warp taking two).  The
    // shuffle tells the compiler that the lanes agree on t: a tile's description then lives in uniform
    // registers, without which the kernel spills 64 bytes and 10,000 FP32 products take 420 us.
    const int warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0);
    int t = ((warp + int(blockIdx.x) / num_sms * 2) & 7) * int(gridDim.x) + int(blockIdx.x);
    if (t >= ntiles) return;
    auto plenty = [&](int ticket) { return ticket < ntiles - 24 * int(gridDim.x); };
    auto take = [&] { return lane == 0 ? 8 * int(gridDim.x) + atomicAdd(counter, 1) : 0; };
    DevTile tl = tiles[t];
    int taken = plenty(t) ? take() : -1;
    while (true) {
        t = __shfl_sync(0xffffffffu, taken, 0);  // the next tile's, -1 for none in hand
        DevTile tn = tiles[min(unsigned(t), unsigned(ntiles - 1))];
        taken = t >= 0 && plenty(t) ? take() : -1;
        const DevProblem p = probs[tl.prob];
        if constexpr (sizeof(T) == 4) {
            warp_tile_staged(p, tl.tm, tl.tn, lane, sw);
        } else {
            const int i0 = tl.tm * p.tr, j0 = tl.tn * p.tc;
            const int rows = min(p.tr, p.m - i0), cols = min(p.tc, p.n - j0);
            double* sd = reinterpret_cast<double*>(stage_smem) + (threadIdx.x >> 5) * (2 * kDStage);
            warp_tile_flat(p, i0, j0, rows, cols, lane, sd);
        }
        if (t < 0) {
            t = __shfl_sync(0xffffffffu, take(), 0);
            tn = tiles[min(t, ntiles - 1)];
        }
        if (t >= ntiles) return;
        tl = tn;
    }
}

// ---- tuning table ------------------------------------------------------------------------------
constexpr int kTuneKernels = 2;  // version of the kernels and of padded_outputs that costs refer to
// Size classes: m and n bucketed by powers of two (<=8, <=16, <=32, <=64, <=128, >128), k by
// (<=16, <=64, >64).  Entry = warp-tile shape index.
constexpr int kMB = 6, kKB = 3;
int bucket_mn(int x) { return x <= 8 ? 0 : x <= 16 ? 1 : x <= 32 ? 2 : x <= 64 ? 3 : x <= 128 ? 4 : 5; }
int bucket_k(int x) { return x <= 16 ? 0 : x <= 64 ? 1 : 2; }

// How a plan picks a product's shape, per element type:
//   kPickModel   no table: the least padded work for the product's own m and n (model_shape);
//   kPickTable   a loaded table without costs: the shape stored for the product's size class;
//   kPickCost    autotuned (or a table with costs): for the product's own m, n the shape with the
//                least (padded multiply-adds) x (the time per padded multiply-add the autotuner
//                measured for that shape in the product's size class).
enum PickMode : int { kPickModel = 0, kPickTable = 1, kPickCost = 2 };

struct TuneTable {
    int shape[2][kMB][kMB][kKB];  // [dtype: 0 double, 1 float]
    float cost[2][kMB][kMB][kKB][kNumShapes] = {};  // ns per padded multiply-add, 0 = not measured
    int mode[2] = {kPickModel, kPickModel};
    double tile_w[2] = {-1.0, -1.0};  // the model's per-tile weight (the autotuner's choice; -1: default)
    bool tuned_any = false;  // the autotuner ran (or a v2 table was loaded): save as v2
};

std::mutex g_tune_mu;
TuneTable g_tune;
bool g_tune_init = false;

// Instructions of one FP32 warp tile of `rows` x `cols` used outputs (shape s, k steps): per staged
// chunk its copies and its multiply-adds, per tile its description, set-up and stores.  The small
// shapes waste little on padding but pay five times as many instructions a multiply-add as 32 x 32.
double f32_tile_cost(int s, int rows, int cols, int k) {
    const int R = shape_rows(s) / 8, C = shape_cols(s) / 4;
    const double steps = 4.0 * (R + 4.0 * (std::max(1, C / 4) + R + R * C / 2));
    const double copies = 3.5 * rows + (cols > 16 ? 112.0 : 56.0);
    return 400.0 + (k + KC - 1) / KC * (60.0 + copies) + k / double(KC) * steps;
}

// Default choice (no measurements).  FP64: the shape with the least padded work, larger tiles on ties;
// FP32: the one with the fewest instructions (f32_tile_cost), since they bound its tiles (10,000
// products: 369 us with the least padded work, 323 with this, which also holds the ticket and
// description look-ahead of grouped_kernel).
// tile_w < 0, the default: FP64 the padded outputs plus 64 a tile (k left out), FP32 f32_tile_cost (with
// k); tile_w >= 0: the padded multiply-adds (outputs x k) plus tile_w multiply-adds' worth a tile.
// FP64 (flat): a product's tiles are equal parts of at most the shape's size, each a whole number of 32
// outputs (warp_tile_flat).
struct Parts {
    int count, size;  // parts of `size`, the last one the rest
};
Parts equal_parts(int64_t x, int limit) {
    if (x <= 0) return {0, 0};
    const int64_t c = (x + limit - 1) / limit;
    const int64_t size = (x + c - 1) / c;
    return {int((x + size - 1) / size), int(size)};
}
double padded_outputs(int m, int n, int s, bool flat) {
    const int tr = shape_rows(s), tc = shape_cols(s);
    if (!flat) return std::ceil(m / double(tr)) * tr * std::ceil(n / double(tc)) * tc;
    const Parts r = equal_parts(m, tr), c = equal_parts(n, tc);
    const int lr = m - (r.count - 1) * r.size, lc = n - (c.count - 1) * c.size;
    auto warp = [](int a, int b) { return double((int64_t(a) * b + 31) / 32 * 32); };
    return double(r.count - 1) * (c.count - 1) * warp(r.size, c.size) + double(r.count - 1) * warp(r.size, lc) +
           double(c.count - 1) * warp(lr, c.size) + warp(lr, lc);
}

int model_shape(int m, int n, int nshapes, bool flat, int k = 1, double tile_w = -1.0, int max_outputs = 1 << 20) {
    int best = 0;
    double best_cost = 1e300;
    for (int s = 0; s < nshapes; ++s) {
        const double tr = shape_rows(s), tc = shape_cols(s);
        if (tr * tc > max_outputs) continue;
        const double padded = padded_outputs(m, n, s, flat);
        const double tiles = std::ceil(m / tr) * std::ceil(n / tc);
        // a small per-tile overhead favours fewer, larger tiles when the padding is equal
        const double cost = tile_w < 0 && !flat ? tiles * f32_tile_cost(s, std::min(m, int(tr)), std::min(n, int(tc)), k)
                            : tile_w < 0        ? padded + 64.0 * tiles
                                                : padded * double(std::max(k, 1)) + tile_w * tiles;
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = s;
        }
    }
    return best;
}

void tune_defaults() {
    if (g_tune_init) return;
    const int rep[kMB] = {6, 12, 24, 48, 96, 192}, rep_k[kKB] = {10, 40, 160};
    for (int d = 0; d < 2; ++d)
        for (int a = 0; a < kMB; ++a)
            for (int b = 0; b < kMB; ++b)
                for (int c = 0; c < kKB; ++c)
                    g_tune.shape[d][a][b][c] =
                        model_shape(rep[a], rep[b], d == 0 ? max_shape<double>() + 1 : max_shape<float>() + 1, d == 0, rep_k[c]);
    g_tune_init = true;
}

int pick_shape(int dtype_idx, int m, int n, int k, int mode_override = -1, int max_outputs = 1 << 20) {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    tune_defaults();
    const int nshapes = dtype_idx == 0 ? max_shape<double>() + 1 : max_shape<float>() + 1;
    const int a = bucket_mn(m), b = bucket_mn(n), c = bucket_k(k);
    switch (mode_override >= 0 ? mode_override : g_tune.mode[dtype_idx]) {
        case kPickTable: return g_tune.shape[dtype_idx][a][b][c];
        case kPickCost: {
            int best = g_tune.shape[dtype_idx][a][b][c];
            double best_cost = 1e300;
            for (int s = 0; s < nshapes; ++s) {
                const float per = g_tune.cost[dtype_idx][a][b][c][s];
                if (per <= 0.f) continue;
                const double cost = padded_outputs(m, n, s, dtype_idx == 0) * double(per);
                if (cost < best_cost) {
                    best_cost = cost;
                    best = s;
                }
            }
            return best;
        }
        default: return model_shape(m, n, nshapes, dtype_idx == 0, k, g_tune.tile_w[dtype_idx], max_outputs);
    }
}

// Whether plans pick shapes by the model.
bool uses_model(int dtype_idx, int mode_override) {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    return (mode_override >= 0 ? mode_override : g_tune.mode[dtype_idx]) == kPickModel;
}

}  // namespace

// ---- plan ----------------------------------------------------------------------------------
struct GroupedPlan {
    int elem = 8;
    int64_t count = 0;
    int64_t ntiles = 0;
    DevProblem* d_probs = nullptr;
    DevTile* d_tiles = nullptr;
    int* d_counter = nullptr;
    cudaStream_t cap_stream = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int grid = 0;
    double useful_flops = 0, padded_flops = 0;
};

namespace {

void plan_free(GroupedPlan* p) {
    if (!p) return;
    if (p->exec) cudaGraphExecDestroy(p->exec);
    if (p->graph) cudaGraphDestroy(p->graph);
    if (p->cap_stream) cudaStreamDestroy(p->cap_stream);
    if (p->d_probs) cudaFree(p->d_probs);
    if (p->d_tiles) cudaFree(p->d_tiles);
    if (p->d_counter) cudaFree(p->d_counter);
    delete p;
}

// The device problem table and the flat tile list of a batch (longest tiles first).  Every output sums its
// k range in order whatever tile it is in, so a product gets the same result bits whatever else is in
// the batch.
//
// Shapes come from the product's own (m, n, k) and the tuning state.  A list that does not fill the chip
// waits for its longest tile, which one warp works on alone: where the model picks the shapes, such a
// batch takes the smallest tiles that leave two of them or fewer on a quarter of an SM.
template <typename T>
int build_tables(const gb300_gemm_problem* probs, int64_t count, int force_shape, int policy,
                 std::vector<DevProblem>& hp, std::vector<DevTile>& ht, double& useful, double& padded,
                 std::string* err, int max_outputs = 1 << 20) {
    const int didx = sizeof(T) == 8 ? 0 : 1;
    hp.clear();
    ht.clear();
    hp.reserve(size_t(count));
    useful = padded = 0;
    for (int64_t q = 0; q < count; ++q) {
        const gb300_gemm_problem& x = probs[q];
        const bool rm = x.order == 101;
        if ((x.order != 101 && x.order != 102) || x.m < 0 || x.n < 0 || x.k < 0 || x.m > INT32_MAX ||
            x.n > INT32_MAX || x.k > INT32_MAX) {
            if (err) *err = "problem " + std::to_string(q) + ": invalid order or size";
            return GB300_ERR_INVALID_ARG;
        }
        const bool tA = x.transA != 111, tB = x.transB != 111;
        const int64_t minlda = std::max<int64_t>(1, rm ? (tA ? x.m : x.k) : (tA ? x.k : x.m));
        const int64_t minldb = std::max<int64_t>(1, rm ? (tB ? x.k : x.n) : (tB ? x.n : x.k));
        const int64_t minldc = std::max<int64_t>(1, rm ? x.n : x.m);
        if (x.lda < minlda || x.ldb < minldb || x.ldc < minldc) {
            if (err) *err = "problem " + std::to_string(q) + ": leading dimension too small";
            return GB300_ERR_INVALID_ARG;
        }
        DevProblem d;
        if (rm) {
            d.m = int(x.m); d.n = int(x.n); d.A = x.A; d.lda = x.lda; d.B = x.B; d.ldb = x.ldb;
            d.ta = tA; d.tb = tB;
        } else {
            d.m = int(x.n); d.n = int(x.m); d.A = x.B; d.lda = x.ldb; d.B = x.A; d.ldb = x.lda;
            d.ta = tB; d.tb = tA;
        }
        d.k = int(x.k);
        d.C = x.C;
        d.ldc = x.ldc;
        d.alpha = x.alpha;
        d.beta = x.beta;
        if (d.m == 0 || d.n == 0) continue;
        if (d.k == 0 || x.alpha == 0.0) d.k = 0;  // C = beta*C through the same kernel
        d.shape = force_shape >= 0 ? force_shape : pick_shape(didx, d.m, d.n, d.k, policy, max_outputs);
        d.tr = shape_rows(d.shape);
        d.tc = shape_cols(d.shape);
        if (sizeof(T) == 8) {
            d.tr = equal_parts(d.m, d.tr).size;
            d.tc = equal_parts(d.n, d.tc).size;
        }
        const int mt = int((int64_t(d.m) + d.tr - 1) / d.tr), nt = int((int64_t(d.n) + d.tc - 1) / d.tc);
        const int pid = int(hp.size());
        hp.push_back(d);
        for (int a = 0; a < mt; ++a)
            for (int b = 0; b < nt; ++b) ht.push_back(DevTile{pid, a, b, 0});
        useful += 2.0 * d.m * d.n * d.k;
        padded += 2.0 * padded_outputs(d.m, d.n, d.shape, sizeof(T) == 8) * d.k;
    }
    const size_t few = size_t(runtime().num_sms) * 8;
    if (force_shape < 0 && max_outputs == 1 << 20 && !ht.empty() && ht.size() <= few && uses_model(didx, policy)) {
        for (int cap : {64, 256, 512}) {
            size_t tiles = 0;
            for (const DevProblem& d : hp) {
                const int sh = pick_shape(didx, d.m, d.n, d.k, policy, cap);
                tiles += size_t((int64_t(d.m) + shape_rows(sh) - 1) / shape_rows(sh)) *
                         size_t((int64_t(d.n) + shape_cols(sh) - 1) / shape_cols(sh));
            }
            if (tiles <= few)
                return build_tables<T>(probs, count, force_shape, policy, hp, ht, useful, padded, err, cap);
        }
    }
    // longest first: tiles ordered by their k times tile area (descending)
    std::stable_sort(ht.begin(), ht.end(), [&](const DevTile& a, const DevTile& b) {
        const DevProblem& pa = hp[a.prob];
        const DevProblem& pb = hp[b.prob];
        const double wa = double(pa.k) * pa.tr * pa.tc;
        const double wb = double(pb.k) * pb.tr * pb.tc;
        return wa > wb;
    });
    return GB300_OK;
}

// Dynamic shared memory of a block: its warps' staging regions.
template <typename T>
int grouped_smem() {
    constexpr int bytes = sizeof(T) == 4 ? kStageBytes : kDStageBytes;
    static const bool set = [] {
        return cudaFuncSetAttribute(grouped_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
    }();
    (void)set;
    return bytes;
}

// Persistent grid for `ntiles` warp tiles: every SM's resident blocks, or a block a tile for a short list,
// which spreads it over the SMs and their quarters.
template <typename T>
int grouped_grid(int64_t ntiles, int num_sms) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, grouped_kernel<T>, 256, grouped_smem<T>());
    per_sm = std::max(per_sm, 1);
    return int(std::max<int64_t>(1, std::min<int64_t>(int64_t(num_sms) * per_sm, ntiles)));
}

template <typename T>
int plan_create(const gb300_gemm_problem* probs, int64_t count, int force_shape, GroupedPlan** out, std::string* err,
                int policy = -1) {
    Runtime& r = runtime();
    int st = ensure_init(err);
    if (st != GB300_OK) return st;
    std::vector<DevProblem> hp;
    std::vector<DevTile> ht;
    double useful = 0, padded = 0;
    st = build_tables<T>(probs, count, force_shape, policy, hp, ht, useful, padded, err);
    if (st != GB300_OK) return st;
    auto* p = new GroupedPlan();
    p->elem = sizeof(T);
    p->count = count;
    p->ntiles = int64_t(ht.size());
    p->useful_flops = useful;
    p->padded_flops = padded;
    cudaError_t e = cudaSuccess;
    if (!hp.empty()) {
        if ((e = cudaMalloc(&p->d_probs, hp.size() * sizeof(DevProblem))) != cudaSuccess ||
            (e = cudaMalloc(&p->d_tiles, ht.size() * sizeof(DevTile))) != cudaSuccess ||
            (e = cudaMemcpy(p->d_probs, hp.data(), hp.size() * sizeof(DevProblem), cudaMemcpyHostToDevice)) !=
                cudaSuccess ||
            (e = cudaMemcpy(p->d_tiles, ht.data(), ht.size() * sizeof(DevTile), cudaMemcpyHostToDevice)) != cudaSuccess) {
            plan_free(p);
            if (err) *err = std::string("grouped plan upload: ") + cudaGetErrorString(e);
            return GB300_ERR_NO_MEMORY;
        }
    }
    if ((e = cudaMalloc(&p->d_counter, sizeof(int))) != cudaSuccess ||
        (e = cudaStreamCreateWithFlags(&p->cap_stream, cudaStreamNonBlocking)) != cudaSuccess) {
        plan_free(p);
        if (err) *err = std::string("grouped plan set-up: ") + cudaGetErrorString(e);
        return GB300_ERR_NO_MEMORY;
    }
    p->grid = grouped_grid<T>(p->ntiles, r.num_sms);
    // capture: counter reset + persistent kernel
    e = cudaStreamBeginCapture(p->cap_stream, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
        cudaMemsetAsync(p->d_counter, 0, sizeof(int), p->cap_stream);
        if (p->ntiles > 0)
            grouped_kernel<T><<<p->grid, 256, grouped_smem<T>(), p->cap_stream>>>(p->d_probs, p->d_tiles,
                                                                              int(p->ntiles), p->d_counter, r.num_sms);
        e = cudaStreamEndCapture(p->cap_stream, &p->graph);
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&p->exec, p->graph, 0);
    if (e != cudaSuccess) {
        plan_free(p);
        if (err) *err = std::string("grouped graph capture: ") + cudaGetErrorString(e);
        return GB300_ERR_CUDA;
    }
    *out = p;
    return GB300_OK;
}

// ---- autotuner -----------------------------------------------------------------------------
// Fills n elements of device memory with uniform [-1, 1] values (a block of them, repeated): the FP64
// pipe runs faster on zeros.
template <typename T>
cudaError_t fill_uniform(T* d, size_t n) {
    std::vector<T> h(std::min<size_t>(n, size_t(1) << 18));
    uint64_t x = 0x2545F4914F6CDD1Dull;
    for (T& v : h) {
        x ^= x << 13; x ^= x >> 7; x ^= x << 17;
        v = T(double(int64_t(x)) * 0x1p-63);
    }
    cudaError_t e = cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
    for (size_t done = h.size(); done < n && e == cudaSuccess;) {
        const size_t c = std::min(done, n - done);
        e = cudaMemcpy(d + done, d, c * sizeof(T), cudaMemcpyDeviceToDevice);
        done += c;
    }
    return e;
}

// For every size class, time each candidate shape on a synthetic batch of that class (operands
// uniform [-1,1], sizes drawn inside the class) and keep the fastest; results can be saved to and
// loaded from a text cache ("gb300-grouped-tune v1" header, one class per line).
template <typename T>
int autotune(int didx, int effort, std::string* err) {
    const int rep_lo[kMB] = {4, 9, 17, 33, 65, 129};
    const int rep_hi[kMB] = {8, 16, 32, 64, 128, 256};
    const int k_lo[kKB] = {4, 17, 65}, k_hi[kKB] = {16, 64, 256};
    uint64_t rng = 0x9E3779B97F4A7C15ull;
    auto rnd = [&](int lo, int hi) {
        rng ^= rng << 13; rng ^= rng >> 7; rng ^= rng << 17;
        return lo + int(rng % uint64_t(hi - lo + 1));
    };
    // Each class is timed on a batch holding about `work` multiply-adds, so that a plan's run is
    // long against its launch: a batch of a few tiny products would time the launch, not the shape.
    const double work = 1.28e8 * std::max(1, effort) * (sizeof(T) == 4 ? 4.0 : 1.0);  // FP32 runs ~30x faster
    auto class_batch = [&](int a, int b, int c) {
        const double mean = 0.125 * double(rep_lo[a] + rep_hi[a]) * double(rep_lo[b] + rep_hi[b]) *
                            double(k_lo[c] + k_hi[c]);
        // (at most 16384 products: the plan's host-side set-up grows with the count)
        return int(std::max(64.0, std::min(16384.0, work / mean)));
    };
    auto footprint = [&](int a, int b, int c) {  // elements of A, B and C of one product, at most
        return size_t(rep_hi[a]) * k_hi[c] + size_t(k_hi[c]) * rep_hi[b] + size_t(rep_hi[a]) * rep_hi[b];
    };
    size_t pool = 0;
    for (int a = 0; a < kMB; ++a)
        for (int b = 0; b < kMB; ++b)
            for (int c = 0; c < kKB; ++c) pool = std::max(pool, size_t(class_batch(a, b, c)) * footprint(a, b, c));
    T* dP = nullptr;
    cudaError_t e;
    if ((e = cudaMalloc(&dP, pool * sizeof(T))) != cudaSuccess) {
        if (err) *err = std::string("autotune buffers: ") + cudaGetErrorString(e);
        return GB300_ERR_NO_MEMORY;
    }
    if ((e = fill_uniform(dP, pool)) != cudaSuccess) {
        cudaFree(dP);
        if (err) *err = std::string("autotune buffers: ") + cudaGetErrorString(e);
        return GB300_ERR_CUDA;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int table[kMB][kMB][kKB];
    float costs[kMB][kMB][kKB][kNumShapes] = {};
    for (int a = 0; a < kMB; ++a)
        for (int b = 0; b < kMB; ++b)
            for (int c = 0; c < kKB; ++c) {
                const int batch = class_batch(a, b, c);
                std::vector<gb300_gemm_problem> ps(static_cast<size_t>(batch));
                size_t off = 0;
                for (int q = 0; q < batch; ++q) {
                    gb300_gemm_problem& x = ps[size_t(q)];
                    std::memset(&x, 0, sizeof(x));
                    x.order = 101; x.transA = 111; x.transB = 111;
                    x.m = rnd(rep_lo[a], rep_hi[a]); x.n = rnd(rep_lo[b], rep_hi[b]); x.k = rnd(k_lo[c], k_hi[c]);
                    x.alpha = 1.0; x.beta = 0.0;
                    x.A = dP + off; x.lda = x.k;
                    off += size_t(x.m) * size_t(x.k);
                    x.B = dP + off; x.ldb = x.n;
                    off += size_t(x.k) * size_t(x.n);
                    x.C = dP + off; x.ldc = x.n;
                    off += size_t(x.m) * size_t(x.n);
                }
                float best_ms = 1e30f;
                int best = 0;
                for (int s = 0; s <= max_shape<T>(); ++s) {
                    GroupedPlan* p = nullptr;
                    costs[a][b][c][s] = 0.f;
                    if (plan_create<T>(ps.data(), batch, s, &p, err) != GB300_OK) continue;
                    cudaGraphLaunch(p->exec, p->cap_stream);  // warm-up
                    cudaEventRecord(e0, p->cap_stream);
                    const int reps = 5;
                    for (int it = 0; it < reps; ++it) cudaGraphLaunch(p->exec, p->cap_stream);
                    cudaEventRecord(e1, p->cap_stream);
                    cudaEventSynchronize(e1);
                    float ms = 0;
                    cudaEventElapsedTime(&ms, e0, e1);
                    count_launches(reps + 1);
                    // time per padded multiply-add (ns), the shape's efficiency in this class
                    if (p->padded_flops > 0) costs[a][b][c][s] = float(1e6 * ms / reps / (0.5 * p->padded_flops));
                    plan_free(p);
                    if (ms < best_ms) { best_ms = ms; best = s; }
                }
                table[a][b][c] = best;
            }
    cudaFree(dP);
    {
        std::lock_guard<std::mutex> lock(g_tune_mu);
        tune_defaults();
        std::memcpy(g_tune.shape[didx], table, sizeof(table));
        std::memcpy(g_tune.cost[didx], costs, sizeof(costs));
    }
    // Which way of picking shapes is faster on a mixed batch (m, n, k log-uniform over all classes): the
    // default model, the measured costs, or the model with other per-tile weights.  The batch is long
    // enough for its tail not to decide (on 2048 products the choice made 10,000 slower than the default:
    // 3.95 ms against 3.77 FP64, 0.368 against 0.322 FP32), and the default stays unless another is 1 %
    // faster, more than two runs differ.
    const int vcount = 10000;
    std::vector<gb300_gemm_problem> vs(static_cast<size_t>(vcount));
    size_t vtotal = 0;
    auto logu = [&](int lo, int hi) {
        const double u = double(rnd(0, 1 << 20)) / double(1 << 20);
        return int(std::lround(std::exp(std::log(double(lo)) + u * (std::log(double(hi)) - std::log(double(lo))))));
    };
    for (auto& x : vs) {
        std::memset(&x, 0, sizeof(x));
        x.order = 101; x.transA = 111; x.transB = 111;
        x.m = logu(4, 256); x.n = logu(4, 256); x.k = logu(4, 256);
        x.alpha = 1.0; x.beta = 0.0;
        vtotal += size_t(x.m) * size_t(x.k) + size_t(x.k) * size_t(x.n) + size_t(x.m) * size_t(x.n);
    }
    int mode = kPickModel;
    double best_w = -1.0;
    T* dV = nullptr;
    if (cudaMalloc(&dV, vtotal * sizeof(T)) == cudaSuccess && fill_uniform(dV, vtotal) == cudaSuccess) {
        size_t off = 0;
        for (auto& x : vs) {
            x.A = dV + off; x.lda = x.k; off += size_t(x.m) * size_t(x.k);
            x.B = dV + off; x.ldb = x.n; off += size_t(x.k) * size_t(x.n);
            x.C = dV + off; x.ldc = x.n; off += size_t(x.m) * size_t(x.n);
        }
        struct Candidate {
            int mode;
            double w;
            GroupedPlan* plan;
            float ms;
        };
        Candidate cands[] = {{kPickModel, -1.0, nullptr, 1e30f},  {kPickCost, -1.0, nullptr, 1e30f},
                             {kPickModel, 0.0, nullptr, 1e30f},   {kPickModel, 512.0, nullptr, 1e30f},
                             {kPickModel, 2048.0, nullptr, 1e30f}, {kPickModel, 8192.0, nullptr, 1e30f}};
        for (Candidate& c : cands) {
            {
                std::lock_guard<std::mutex> lock(g_tune_mu);
                g_tune.tile_w[didx] = c.w;
            }
            if (plan_create<T>(vs.data(), vcount, -1, &c.plan, err, c.mode) != GB300_OK) c.plan = nullptr;
        }
        for (int round = 0; round < 4; ++round)  // in turn; the first round warms up
            for (Candidate& c : cands) {
                if (!c.plan) continue;
                cudaEventRecord(e0, c.plan->cap_stream);
                for (int it = 0; it < 3; ++it) cudaGraphLaunch(c.plan->exec, c.plan->cap_stream);
                cudaEventRecord(e1, c.plan->cap_stream);
                cudaEventSynchronize(e1);
                float ms = 0;
                cudaEventElapsedTime(&ms, e0, e1);
                count_launches(3);
                if (round > 0) c.ms = std::min(c.ms, ms);
            }
        float best_ms = cands[0].ms * 0.99f;
        for (Candidate& c : cands) {
            if (c.plan) plan_free(c.plan);
            if (c.ms < best_ms) {
                best_ms = c.ms;
                mode = c.mode;
                best_w = c.w;
            }
        }
    } else {
        cudaGetLastError();
    }
    if (dV) cudaFree(dV);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_tune.mode[didx] = mode;
    g_tune.tile_w[didx] = mode == kPickModel ? best_w : -1.0;
    g_tune.tuned_any = true;
    return GB300_OK;
}

}  // namespace

// ---- lanes: grouped launches of the serving loop ---------------------------------------------
// A lane owns grow-only page-locked staging and device buffers for the problem table and tile
// list, so that a batch of small requests goes out as one plain launch (copies, counter reset,
// persistent kernel) on the lane's stream without allocating once the buffers have grown.  The
// caller waits for a lane's previous launch to finish before it launches on that lane again.
struct GroupedLane {
    cudaStream_t stream = nullptr;
    void* h_buf = nullptr;
    size_t h_bytes = 0;
    void* d_buf = nullptr;
    size_t d_bytes = 0;
    int* d_counter = nullptr;
    std::vector<void*> retired;  // outgrown staging buffers: cudaFreeHost would wait for the device
    std::vector<DevProblem> hp;
    std::vector<DevTile> ht;
};

GroupedLane* grouped_lane_create(cudaStream_t stream, std::string* err) {
    auto* l = new GroupedLane();
    l->stream = stream;
    if (cudaMalloc(&l->d_counter, sizeof(int)) != cudaSuccess) {
        cudaGetLastError();
        if (err) *err = "grouped lane: counter allocation failed";
        delete l;
        return nullptr;
    }
    return l;
}

void grouped_lane_destroy(GroupedLane* l) {
    if (!l) return;
    if (l->d_buf) cudaFreeAsync(l->d_buf, l->stream);
    if (l->stream) cudaStreamSynchronize(l->stream);
    if (l->h_buf) cudaFreeHost(l->h_buf);
    for (void* h : l->retired) cudaFreeHost(h);
    if (l->d_counter) cudaFree(l->d_counter);
    delete l;
}

int grouped_lane_launch(GroupedLane* l, const gb300_gemm_problem* probs, int64_t count, double* useful_flops,
                        std::string* err) {
    double useful = 0, padded = 0;
    int st = build_tables<double>(probs, count, -1, -1, l->hp, l->ht, useful, padded, err);
    if (st != GB300_OK) return st;
    if (useful_flops) *useful_flops = useful;
    if (l->ht.empty()) return GB300_OK;
    const size_t pb = l->hp.size() * sizeof(DevProblem), tb = l->ht.size() * sizeof(DevTile);
    const size_t off_t = (pb + 255) / 256 * 256, need = off_t + tb;
    auto grow = [](size_t n) { return (n + (size_t(1) << 20) - 1) & ~((size_t(1) << 20) - 1); };
    if (l->h_bytes < need) {
        if (l->h_buf) l->retired.push_back(l->h_buf);
        l->h_buf = nullptr;
        l->h_bytes = 0;
        if (cudaHostAlloc(&l->h_buf, grow(need), cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            if (err) *err = "grouped lane: staging allocation failed";
            return GB300_ERR_NO_MEMORY;
        }
        l->h_bytes = grow(need);
    }
    if (l->d_bytes < need) {
        // stream-ordered on the lane's stream: growing the table never waits for other streams
        if (l->d_buf) cudaFreeAsync(l->d_buf, l->stream);
        l->d_buf = nullptr;
        l->d_bytes = 0;
        if (cudaMallocAsync(&l->d_buf, grow(need), l->stream) != cudaSuccess) {
            cudaGetLastError();
            if (err) *err = "grouped lane: table allocation failed";
            return GB300_ERR_NO_MEMORY;
        }
        l->d_bytes = grow(need);
    }
    auto* h = static_cast<uint8_t*>(l->h_buf);
    std::memcpy(h, l->hp.data(), pb);
    std::memcpy(h + off_t, l->ht.data(), tb);
    auto* d = static_cast<uint8_t*>(l->d_buf);
    cudaError_t e = cudaMemcpyAsync(d, h, need, cudaMemcpyHostToDevice, l->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(l->d_counter, 0, sizeof(int), l->stream);
    if (e == cudaSuccess) {
        const int grid = grouped_grid<double>(int64_t(l->ht.size()), runtime().num_sms);
        grouped_kernel<double><<<grid, 256, grouped_smem<double>(), l->stream>>>(reinterpret_cast<const DevProblem*>(d),
                                                            reinterpret_cast<const DevTile*>(d + off_t),
                                                            int(l->ht.size()), l->d_counter, runtime().num_sms);
        count_launches(1);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        if (err) *err = std::string("grouped lane launch: ") + cudaGetErrorString(e);
        return GB300_ERR_CUDA;
    }
    return GB300_OK;
}

}  // namespace gb

// ============================================================================================
//  C-ABI
// ============================================================================================
extern "C" {

int gb300_grouped_plan_create(int elem_bytes, const gb300_gemm_problem* problems, int64_t count,
                              gb300_grouped_plan** plan) {
    if (!plan || (count > 0 && !problems) || count < 0 || (elem_bytes != 8 && elem_bytes != 4)) {
        gb::set_error(GB300_ERR_INVALID_ARG, "gb300_grouped_plan_create: invalid arguments");
        return GB300_ERR_INVALID_ARG;
    }
    gb::Runtime& r = gb::runtime();
    std::lock_guard<std::mutex> lock(r.mu);
    std::string err;
    gb::GroupedPlan* p = nullptr;
    const int st = elem_bytes == 8 ? gb::plan_create<double>(problems, count, -1, &p, &err)
                                   : gb::plan_create<float>(problems, count, -1, &p, &err);
    if (st != GB300_OK) {
        gb::set_error(st, "gb300_grouped_plan_create: " + err);
        return st;
    }
    *plan = reinterpret_cast<gb300_grouped_plan*>(p);
    gb::clear_error();
    return GB300_OK;
}

int gb300_grouped_plan_run(gb300_grouped_plan* plan, void* stream) {
    auto* p = reinterpret_cast<gb::GroupedPlan*>(plan);
    if (!p) {
        gb::set_error(GB300_ERR_INVALID_ARG, "gb300_grouped_plan_run: null plan");
        return GB300_ERR_INVALID_ARG;
    }
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : gb::runtime().stream;
    const cudaError_t e = cudaGraphLaunch(p->exec, s);
    if (e != cudaSuccess) {
        gb::set_error(GB300_ERR_CUDA, std::string("gb300_grouped_plan_run: ") + cudaGetErrorString(e));
        return GB300_ERR_CUDA;
    }
    gb::count_launches(p->ntiles > 0 ? 1 : 0);
    return GB300_OK;
}

int gb300_grouped_plan_info(const gb300_grouped_plan* plan, int64_t* tiles, double* useful_flops,
                            double* padded_flops) {
    auto* p = reinterpret_cast<const gb::GroupedPlan*>(plan);
    if (!p) return GB300_ERR_INVALID_ARG;
    if (tiles) *tiles = p->ntiles;
    if (useful_flops) *useful_flops = p->useful_flops;
    if (padded_flops) *padded_flops = p->padded_flops;
    return GB300_OK;
}

void gb300_grouped_plan_destroy(gb300_grouped_plan* plan) {
    gb::Runtime& r = gb::runtime();
    std::lock_guard<std::mutex> lock(r.mu);
    gb::plan_free(reinterpret_cast<gb::GroupedPlan*>(plan));
}

int gb300_dgemm_grouped(const gb300_gemm_problem* problems, int64_t count, void* stream) {
    gb300_grouped_plan* p = nullptr;
    int st = gb300_grouped_plan_create(8, problems, count, &p);
    if (st != GB300_OK) return st;
    st = gb300_grouped_plan_run(p, stream);
    if (st == GB300_OK) {
        cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : gb::runtime().stream;
        if (cudaStreamSynchronize(s) != cudaSuccess) st = GB300_ERR_CUDA;
    }
    gb300_grouped_plan_destroy(p);
    return st;
}

int gb300_sgemm_grouped(const gb300_gemm_problem* problems, int64_t count, void* stream) {
    gb300_grouped_plan* p = nullptr;
    int st = gb300_grouped_plan_create(4, problems, count, &p);
    if (st != GB300_OK) return st;
    st = gb300_grouped_plan_run(p, stream);
    if (st == GB300_OK) {
        cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : gb::runtime().stream;
        if (cudaStreamSynchronize(s) != cudaSuccess) st = GB300_ERR_CUDA;
    }
    gb300_grouped_plan_destroy(p);
    return st;
}

int gb300_grouped_autotune(int elem_bytes, int effort) {
    if (elem_bytes != 8 && elem_bytes != 4) {
        gb::set_error(GB300_ERR_INVALID_ARG, "gb300_grouped_autotune: elem_bytes must be 8 or 4");
        return GB300_ERR_INVALID_ARG;
    }
    gb::Runtime& r = gb::runtime();
    std::string err;
    int st;
    {
        std::lock_guard<std::mutex> lock(r.mu);
        st = gb::ensure_init(&err);
        if (st == GB300_OK)
            st = elem_bytes == 8 ? gb::autotune<double>(0, effort, &err) : gb::autotune<float>(1, effort, &err);
    }
    if (st != GB300_OK) gb::set_error(st, "gb300_grouped_autotune: " + err);
    return st;
}

// Tuning files: "gb300-grouped-tune v1" then one line per class, `dtype m-class n-class k-class
// shape`; an autotuned table is saved as "gb300-grouped-tune v2", each line followed by the measured
// ns per padded multiply-add of every shape (0: not measured), after a line "mode <double> <float>
// <weight> <weight> kernels <n>".  Loading v1 makes plans use the class shapes, loading v2 the measured
// costs, or what its mode line says.  Costs and weights belong to the kernels that they were measured on
// (what a padded multiply-add is has changed with them): a mode line of other kernels loads the class
// shapes and leaves the default choice in place.
int gb300_grouped_tuning_save(const char* path) {
    std::lock_guard<std::mutex> lock(gb::g_tune_mu);
    gb::tune_defaults();
    std::ofstream f(path);
    if (!f) {
        gb::set_error(GB300_ERR_INVALID_ARG, std::string("gb300_grouped_tuning_save: cannot write ") + path);
        return GB300_ERR_INVALID_ARG;
    }
    // untuned defaults and loaded class tables save as v1; an autotuned table as v2 with its costs
    // and the policy the autotuner chose ("mode <double> <float>")
    const bool costs = gb::g_tune.mode[0] == gb::kPickCost || gb::g_tune.mode[1] == gb::kPickCost ||
                       gb::g_tune.tuned_any;
    f << (costs ? "gb300-grouped-tune v2\n" : "gb300-grouped-tune v1\n");
    if (costs)
        f << "mode " << gb::g_tune.mode[0] << ' ' << gb::g_tune.mode[1] << ' ' << gb::g_tune.tile_w[0] << ' '
          << gb::g_tune.tile_w[1] << " kernels " << gb::kTuneKernels << '\n';
    for (int d = 0; d < 2; ++d)
        for (int a = 0; a < gb::kMB; ++a)
            for (int b = 0; b < gb::kMB; ++b)
                for (int c = 0; c < gb::kKB; ++c) {
                    f << d << ' ' << a << ' ' << b << ' ' << c << ' ' << gb::g_tune.shape[d][a][b][c];
                    if (costs)
                        for (int s = 0; s < gb::kNumShapes; ++s) f << ' ' << gb::g_tune.cost[d][a][b][c][s];
                    f << '\n';
                }
    return GB300_OK;
}

int gb300_grouped_tuning_load(const char* path) {
    std::ifstream f(path);
    std::string head;
    const bool ok_head = f && std::getline(f, head) && (head == "gb300-grouped-tune v1" || head == "gb300-grouped-tune v2");
    if (!ok_head) {
        gb::set_error(GB300_ERR_INVALID_ARG, std::string("gb300_grouped_tuning_load: not a tuning file: ") + path);
        return GB300_ERR_INVALID_ARG;
    }
    const bool v2 = head == "gb300-grouped-tune v2";
    // parse everything first: a malformed file leaves the table as it was
    gb::TuneTable t;
    {
        std::lock_guard<std::mutex> lock(gb::g_tune_mu);
        gb::tune_defaults();
        t = gb::g_tune;
    }
    std::string line;
    int modes[2] = {gb::kPickCost, gb::kPickCost};
    while (std::getline(f, line)) {
        if (line.empty()) continue;
        if (v2 && line.rfind("mode ", 0) == 0) {
            std::istringstream ms(line.substr(5));
            if (!(ms >> modes[0] >> modes[1]) || modes[0] < 0 || modes[0] > 2 || modes[1] < 0 || modes[1] > 2) {
                gb::set_error(GB300_ERR_INVALID_ARG, "gb300_grouped_tuning_load: bad mode line");
                return GB300_ERR_INVALID_ARG;
            }
            double w0 = -1.0, w1 = -1.0;
            std::string tag;
            int kernels = 0;
            ms >> w0 >> w1 >> tag >> kernels;
            if (ms && tag == "kernels" && kernels == gb::kTuneKernels) {
                t.tile_w[0] = w0;  // the model's per-tile weights
                t.tile_w[1] = w1;
            } else {
                for (int d = 0; d < 2; ++d) {
                    if (modes[d] == gb::kPickCost) modes[d] = gb::kPickModel;
                    t.tile_w[d] = -1.0;
                }
            }
            continue;
        }
        std::istringstream ls(line);
        int d, a, b, c, s;
        if (!(ls >> d >> a >> b >> c >> s) || d < 0 || d > 1 || a < 0 || a >= gb::kMB || b < 0 || b >= gb::kMB ||
            c < 0 || c >= gb::kKB || s < 0 || s > (d == 0 ? gb::max_shape<double>() : gb::max_shape<float>())) {
            gb::set_error(GB300_ERR_INVALID_ARG, "gb300_grouped_tuning_load: bad entry");
            return GB300_ERR_INVALID_ARG;
        }
        t.shape[d][a][b][c] = s;
        if (v2)
            for (int q = 0; q < gb::kNumShapes; ++q) {
                float v = 0.f;
                if (!(ls >> v) || !(v >= 0.f)) {
                    gb::set_error(GB300_ERR_INVALID_ARG, "gb300_grouped_tuning_load: bad cost");
                    return GB300_ERR_INVALID_ARG;
                }
                t.cost[d][a][b][c][q] = v;
            }
    }
    t.mode[0] = v2 ? modes[0] : gb::kPickTable;
    t.mode[1] = v2 ? modes[1] : gb::kPickTable;
    t.tuned_any = v2;
    std::lock_guard<std::mutex> lock(gb::g_tune_mu);
    gb::g_tune = t;
    return GB300_OK;
}

int gb300_grouped_shape_for(int elem_bytes, int64_t m, int64_t n, int64_t k, int* rows, int* cols) {
    const int s = gb::pick_shape(elem_bytes == 8 ? 0 : 1, int(std::min<int64_t>(m, INT32_MAX)),
                                 int(std::min<int64_t>(n, INT32_MAX)), int(std::min<int64_t>(k, INT32_MAX)));
    if (rows) *rows = gb::shape_rows(s);
    if (cols) *cols = gb::shape_cols(s);
    return s;
}

}  // extern "C"
