// trsm.cu — kernels of the triangular solve ?trsm on Blaze's seam (blaze/math/blas/cblas/trsm.h):
// the scaling of the right-hand sides by alpha and the inverses of the triangle's diagonal blocks.
// The host side (api_next.cpp) solves recursively.  It halves the triangle, solves one half,
// updates the other half's right-hand sides with one product, and solves that half.  The products
// run through the library's real or complex product, so a double solve does nearly all of its
// work on the tensor cores.  A block of at most solve_block() rows is multiplied by its inverse from
// here.  That leaf product costs 2 nb / ka of the solve's own work.  The inverses are what makes
// the leaves products.  Using them changes the rounding from that of substitution: a leaf's error
// grows with the condition number of its diagonal block, as in other blocked GPU solvers.
//
// Matrices are in row-major storage (a column-major operand is the transpose of its storage; the
// host folds that into the side, the triangle and the transposition).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <type_traits>

#include "cplx.cuh"
#include "gb300_internal.h"
#include "level23.h"
#include "ptx.cuh"
#include "runtime.h"

namespace gb {
namespace {

// X (rows x cols, pitch ld) = alpha X.
template <typename V>
__global__ void scale_kernel(int64_t rows, int64_t cols, V alpha, V* __restrict__ X, int64_t ld) {
    for (int64_t r = blockIdx.y; r < rows; r += gridDim.y)
        for (int64_t c = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; c < cols; c += int64_t(gridDim.x) * blockDim.x)
            X[r * ld + c] = Ar<V>::mul(alpha, X[r * ld + c]);
}

// Inverse of every diagonal block of the triangular matrix op(SA).  SA is ka x ka in row-major
// storage with pitch lda, and op transposes it (trans) and conjugates it (conj).  Block b covers
// rows and columns [b nb, min(ka, (b + 1) nb)).  Its inverse Y is written densely to inv + b nb nb
// with pitch nb, zeros outside the triangle included.
//
// Each block is brought to lower-triangular form L'.  L' is the block itself when op(SA) is lower;
// when it is upper (`upper`), L' is the block with its rows and columns reversed.  The inverse is
// built from the diagonal up: tri_base_kernel inverts the 16 x 16 blocks on the diagonal, and each
// level joins two neighbours of s rows into one of 2 s by two products,
//     T = L21 Y11,   Y21 = -Y22 T                              (s = 16, 32, ... nb / 2),
// T being kept where the zeros above the diagonal go in the end (tri_zero_kernel).  The products skip
// the zeros of Y11 and Y22, so the levels together take the nb^3 / 6 multiply-adds of a substitution,
// and what bounds them is the FP64 pipe (94 % active in the last level, 87 in the one before).
// Substituting column by column was bound by its chain of rows instead, 512 steps of a block-wide sum and
// two barriers: 1120 us for the four 512-row blocks of a 2048-row triangle, now 284, of which 143 are the
// multiply-adds at the full FP64 rate.
template <typename V>
struct TriArgs {
    const V* SA;
    V* inv;
    int64_t ka, lda;
    int nb, trans, conj, upper, unit;
};

// One block in lower-triangular form: L'[r][j] at P + r sr + j sj, Y[r][c] at out + r orow + c ocol.
template <typename V>
struct TriBlock {
    const V* P;
    V* out;
    int64_t sr, sj, orow, ocol;
    int rows;
    __device__ __forceinline__ TriBlock(const TriArgs<V>& a, int64_t b) {
        const int64_t b0 = b * a.nb;
        rows = int(min(int64_t(a.nb), a.ka - b0));
        sr = a.trans ? 1 : a.lda;
        sj = a.trans ? a.lda : 1;
        orow = a.nb;
        ocol = 1;
        P = a.SA + b0 * a.lda + b0;
        out = a.inv + b * a.nb * a.nb;
        if (a.upper) {
            P += int64_t(rows - 1) * (a.lda + 1);
            out += int64_t(rows - 1) * (a.nb + 1);
            sr = -sr; sj = -sj; orow = -orow; ocol = -ocol;
        }
    }
};

constexpr int kTriBase = 16;

// The inverses of two 16 x 16 diagonal blocks per warp, one in each half: lane c of a half carries
// column c of Y in registers and subtracts each finished row from all the rows below it, so that the
// multiply-adds of a row are independent of one another (a sum per row would wait for its own chain).
// A lone warp has a quarter of its SM's FP64 pipe, 64 clocks per multiply-add: 32 x 32 blocks, four
// times the instructions, took 36 us at 2048 rows, these 16 with one more level of products.
template <typename V>
__global__ void __launch_bounds__(32) tri_base_kernel(const TriArgs<V> a) {
    using A = Ar<V>;
    __shared__ V Ls[2][kTriBase][kTriBase + 1];
    griddep_launch();
    const int per = a.nb / kTriBase, c = threadIdx.x % kTriBase, h = threadIdx.x / kTriBase;
    V (&L)[kTriBase][kTriBase + 1] = Ls[h];
    const int g = int(blockIdx.x) * 2 + h;
    const TriBlock<V> t(a, g / per);
    const int r0 = (g % per) * kTriBase;
    const int n = min(kTriBase, t.rows - r0);  // below 1 past the end of the last block
    const V* P = t.P + r0 * (t.sr + t.sj);
    const bool by_row = t.sj == 1 || t.sj == -1;  // lanes along the contiguous index
#pragma unroll
    for (int i = 0; i < kTriBase; ++i) {
        const int r = by_row ? i : c, j = by_row ? c : i;
        if (j < r) L[r][j] = r < n ? (a.conj ? A::conj(P[r * t.sr + j * t.sj]) : P[r * t.sr + j * t.sj]) : A::zero();
    }
    V d = A::one();
    if (c < n && !a.unit) d = a.conj ? A::conj(P[c * (t.sr + t.sj)]) : P[c * (t.sr + t.sj)];
    L[c][c] = A::div(A::one(), d);
    __syncwarp();
    V y[kTriBase];
#pragma unroll
    for (int r = 0; r < kTriBase; ++r) y[r] = r == c ? A::one() : A::zero();
#pragma unroll
    for (int r = 0; r < kTriBase; ++r) {
        y[r] = r >= c ? A::mul(y[r], L[r][r]) : A::zero();  // a zero diagonal stays in its own columns
#pragma unroll
        for (int i = r + 1; i < kTriBase; ++i) y[i] = A::fnmadd(L[i][r], y[r], y[i]);
    }
    V* out = t.out + r0 * (t.orow + t.ocol) + c * t.ocol;
#pragma unroll
    for (int r = 0; r < kTriBase; ++r)
        if (r < n && r >= c) out[r * t.orow] = y[r];
}

// One 16 x 16 tile of T = L21 Y11 (SECOND == false; k from the tile's first column on) or of
// Y21 = -Y22 T (SECOND == true; k up to the tile's last row) for the pair of s-row halves that
// blockIdx.y picks.  A thread holds one output: on the FP64 pipe a warp's multiply-add takes 16
// clocks, far more than its two shared loads, and the next 16 k steps are in registers meanwhile.
template <typename V, bool SECOND>
__global__ void __launch_bounds__(256) tri_join_kernel(const TriArgs<V> a, int s) {
    using A = Ar<V>;
    __shared__ V As[16][17], Bs[16][17];
    griddep_launch();
    griddep_wait();
    const int pairs = a.nb / (2 * s);
    const TriBlock<V> t(a, blockIdx.y / pairs);
    const int q0 = int(blockIdx.y % pairs) * 2 * s;   // first row of the upper half
    const int n2 = min(s, t.rows - (q0 + s));         // rows of the lower half
    const int tiles = s / 16;
    // longest k ranges first
    const int ti = SECOND ? tiles - 1 - int(blockIdx.x) / tiles : int(blockIdx.x) % tiles;
    const int tj = SECOND ? int(blockIdx.x) % tiles : int(blockIdx.x) / tiles;
    const int i0 = ti * 16, j0 = tj * 16;
    if (i0 >= n2) return;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    // left operand (i, k) and right operand (k, j), T in place of the block above the diagonal
    V* const T = t.out + q0 * t.orow + (q0 + s) * t.ocol;
    const V* left = SECOND ? t.out + (q0 + s) * (t.orow + t.ocol) : t.P + (q0 + s) * t.sr + q0 * t.sj;
    const int64_t li = SECOND ? t.orow : t.sr, lk = SECOND ? t.ocol : t.sj;
    const V* right = SECOND ? T : t.out + q0 * (t.orow + t.ocol);
    const int k0 = SECOND ? 0 : j0, k1 = SECOND ? min(n2, i0 + 16) : s;
    const bool by_row = lk == 1 || lk == -1;
    const int ai = by_row ? ty : tx, ak = by_row ? tx : ty;
    V va = A::zero(), vb = A::zero();
    auto fetch = [&](int k) {
        const bool oka = i0 + ai < n2 && k + ak < k1 && (!SECOND || k + ak <= i0 + ai);
        va = oka ? left[(i0 + ai) * li + (k + ak) * lk] : A::zero();
        if (!SECOND && a.conj) va = A::conj(va);
        const bool okb = k + ty < k1 && (SECOND || k + ty >= j0 + tx);
        vb = okb ? right[(k + ty) * t.orow + (j0 + tx) * t.ocol] : A::zero();
    };
    fetch(k0);
    V acc = A::zero();
    for (int k = k0; k < k1; k += 16) {
        __syncthreads();
        As[ai][ak] = va;
        Bs[ty][tx] = vb;
        __syncthreads();
        if (k + 16 < k1) fetch(k + 16);
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) acc = A::fmadd(As[ty][kk], Bs[kk][tx], acc);
    }
    if (i0 + ty >= n2) return;
    if (SECOND) t.out[(q0 + s + i0 + ty) * t.orow + (q0 + j0 + tx) * t.ocol] = A::fnmadd(A::one(), acc, A::zero());
    else T[(i0 + ty) * t.orow + (j0 + tx) * t.ocol] = acc;
}

// Zeros above the diagonal of every inverted block.
template <typename V>
__global__ void __launch_bounds__(256) tri_zero_kernel(const TriArgs<V> a) {
    griddep_wait();
    const TriBlock<V> t(a, blockIdx.y);
    for (int r = blockIdx.x; r < t.rows; r += gridDim.x)
        for (int c = r + 1 + threadIdx.x; c < t.rows; c += blockDim.x) t.out[r * t.orow + c * t.ocol] = Ar<V>::zero();
}

}  // namespace

template <typename T, bool CPLX>
cudaError_t launch_scale(int64_t rows, int64_t cols, const T* alpha, T* X, int64_t ld, cudaStream_t st) {
    using V = typename std::conditional<CPLX, Cx<T>, T>::type;
    V al;
    std::memcpy(&al, alpha, sizeof(V));
    const int64_t x = std::max<int64_t>(1, std::min<int64_t>((cols + 255) / 256, 64));
    const int64_t y = std::max<int64_t>(1, std::min<int64_t>(rows, int64_t(runtime().num_sms) * 16 / x));
    scale_kernel<V><<<dim3(unsigned(x), unsigned(y)), 256, 0, st>>>(rows, cols, al, reinterpret_cast<V*>(X), ld);
    count_launches(1);
    return cudaGetLastError();
}

template <typename T, bool CPLX>
cudaError_t launch_tri_inverse(int64_t ka, int nb, const T* SA, int64_t lda, bool trans, bool conj, bool upper,
                               bool unit, T* inv, cudaStream_t st) {
    using V = typename std::conditional<CPLX, Cx<T>, T>::type;
    if (nb > solve_block(sizeof(V)) || nb < 2 * kTriBase || (nb & (nb - 1)) != 0) return cudaErrorInvalidValue;
    TriArgs<V> a;
    a.SA = reinterpret_cast<const V*>(SA);
    a.inv = reinterpret_cast<V*>(inv);
    a.ka = ka;
    a.lda = lda;
    a.nb = nb;
    a.trans = trans ? 1 : 0;
    a.conj = conj ? 1 : 0;
    a.upper = upper ? 1 : 0;
    a.unit = unit ? 1 : 0;
    const int64_t blocks = (ka + nb - 1) / nb, rows = std::min<int64_t>(ka, nb);
    int launches = 2;
    tri_base_kernel<V><<<unsigned(blocks * (nb / (2 * kTriBase))), 32, 0, st>>>(a);
    for (int s = kTriBase; s < rows; s *= 2, launches += 2) {
        // gridDim.y holds at most 65535 pairs: ka / 32 of them on the first level
        const dim3 grid(unsigned((s / 16) * (s / 16)), unsigned(blocks * (nb / (2 * s))));
        launch_dependent(tri_join_kernel<V, false>, grid, dim3(256), 0, st, a, s);
        launch_dependent(tri_join_kernel<V, true>, grid, dim3(256), 0, st, a, s);
    }
    launch_dependent(tri_zero_kernel<V>, dim3(unsigned(std::min<int64_t>(rows, 64)), unsigned(blocks)), dim3(256), 0, st, a);
    count_launches(launches);
    return cudaGetLastError();
}

#define GB_TRSM(T, C)                                                                                             \
    template cudaError_t launch_scale<T, C>(int64_t, int64_t, const T*, T*, int64_t, cudaStream_t);               \
    template cudaError_t launch_tri_inverse<T, C>(int64_t, int, const T*, int64_t, bool, bool, bool, bool, T*, \
                                                  cudaStream_t);
GB_TRSM(double, false)
GB_TRSM(double, true)
GB_TRSM(float, false)
GB_TRSM(float, true)
#undef GB_TRSM

}  // namespace gb
