// FP64 Cholesky factorization, right-hand-side forward solves and explicit SPD
// inverse as ONE kernel over 64 x 64 tiles ordered by data flow.
//
// The saddle solve's SPD matrix (dense.cu) of a few thousand rows is bound by
// its chain of diagonal blocks: a launch per block, panel and update left every
// block waiting for three launches (57 us for the block, 12 for the panel, 40
// for the update); the solves took a grid barrier per block and the inverse a
// launch pair per tile of its recursion. Here one block of threads (the chain) walks the diagonal
// without leaving the SM: it factors and inverts L_jj in shared memory, forms
// the tile below it, L_{j+1,j}, and takes that tile's product off the next
// diagonal block. The other blocks (workers) take everything else as tiles from
// a counter, left-looking, each tile once:
//   L_ij  = (A_ij - sum_{k<j} L_ik L_jk^T) inv(L_jj)^T          (i > j + 1)
//   the same sums for the chain's next two tiles, without the solve;
//   rows B (right-hand sides), y = B L^-T: the same tile with rows of B;
//   rows I, W = L^-T: the same tile with an identity on the left
//     (W_cj = -(sum_{c<=k<j} W_ck L_jk^T) inv(L_jj)^T, W_jj = inv(L_jj)^T);
//   inverse tiles, Ainv_ij = sum_{k>=i} W_ik W_jk^T, and their mirrors.
// Every product is C = A B^T of row-major tiles on the FP64 tensor cores
// (mma.sync m8n8k4), operands staged by 16-byte cp.async, K in ascending order:
// the result does not depend on which block took which tile.
//
// Measured against that (us): factor, order 777: 1380 -> 242, 2048: 3190 -> 575,
// 4096: 6750 -> 1330, 8192: 7100; with the explicit inverse, 777: 2220
// -> 252, 2500: 7200 -> 1010, 8192: 38500 -> 20800; one triangular solve of 15
// right-hand sides, 777: 172 -> 69, 2048: 422 -> 154. Bound: to about 3500 rows
// the chain (per 64 columns 9.7 us for the diagonal block, 8 for its two products,
// loads and flags), above it the workers' products (2.4 us each at the FP64
// tensor rate of one SM).
//
// Order and progress: tiles are numbered column by column; a tile needs only
// tiles with smaller numbers and the chain, the chain needs only tiles of
// earlier columns. The role and the numbers come from counters, so a block
// that runs never waits for one that has not started, whatever else holds the
// SMs. A finished tile raises a flag (release); readers poll the flags of up to
// 32 tiles at a time (acquire). Every wait is bounded: when it runs out, an error
// flag stops all blocks and the call returns TPE_ERR_DEVICE_TIMEOUT.
#include <math.h>

#include <algorithm>

#include "pair_math.cuh"
#include "tpe_internal.h"

namespace tpe {
namespace {

constexpr int NB = kNB;        // 64
constexpr int kThr = 256;
constexpr int kKC = 32;        // K chunk
constexpr int kPad = kKC + 4;  // row stride of a staged chunk (doubles)
constexpr int kTP = NB + 4;    // row stride of a whole tile
constexpr int kStage = NB * kPad;
constexpr int kTile = NB * kTP;
constexpr int32_t kSpin = 1 << 22;  // polls before a wait gives up (seconds)

struct Dag {
    double* L;     // n x n (rows ld apart): A on entry (lower), L on return
    double* Linv;  // nb x 64 x 64: inverses of the diagonal blocks
    double* B;     // nr rows of n: right-hand sides on entry, B L^-T on return
    double* W;     // n x n (ld), upper: L^-T (its diagonal tiles whole), or null
    double* X;     // n x n (ld), lower: L^-1, or null
    double* Ainv;  // n x n, or null
    int32_t n, nb, nr, nrb;  // nrb row blocks of right-hand sides
    int64_t ld;              // row length of L, W and X (n or more); B and Ainv have n
    double tol;
    int32_t limit;  // polls before a wait gives up
    int32_t* flag;  // [(nb + nrb + nb) x nb] tiles done, then diag, preA, preD [nb each]
    // [0] a pivot failed, [1] a wait ran out, [2] role ticket, [3] tile counter, [4] the chain's SM + 1
    int32_t* ctl;
};

__device__ __forceinline__ int32_t ld_acquire(const int32_t* p) {
    int32_t v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int32_t* p, int32_t v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}
// Two doubles of a row into shared memory (`left` columns of it remain: zeros
// beyond them; `row` is a valid address for the empty copies).
template <bool kAl>
__device__ __forceinline__ void cp_pair(double* s, const double* row, int32_t c, int32_t left) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(s);
    if (kAl && left >= 2) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(row + c));
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(left >= 1 ? row + c : row),
                     "r"(left >= 1 ? 8 : 0));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d + 8),
                     "l"(left >= 2 ? row + c + 1 : row), "r"(left >= 2 ? 8 : 0));
    }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Rows of one tile operand: row r of the tile at p + min(r, rows - 1) * ld.
struct Rows {
    const double* p;
    int64_t ld;
    int32_t rows;  // rows that exist (the rest repeat the last one and are never stored)
};

// Columns [c0, c0 + kKC) of the tile (zero from column n on) into s[64][kPad].
template <bool kAl>
__device__ __forceinline__ void load_chunk(double* s, const Rows& t, int32_t c0, int32_t n) {
    for (int idx = threadIdx.x; idx < NB * (kKC / 2); idx += kThr) {
        const int r = idx / (kKC / 2), pc = (idx % (kKC / 2)) * 2;
        cp_pair<kAl>(s + r * kPad + pc, t.p + (int64_t)min(r, t.rows - 1) * t.ld, c0 + pc, n - (c0 + pc));
    }
}
template <bool kAl>
__device__ __forceinline__ void load_tile(double* s, const Rows& t, int32_t c0, int32_t n) {
    for (int idx = threadIdx.x; idx < NB * (NB / 2); idx += kThr) {
        const int r = idx / (NB / 2), pc = (idx % (NB / 2)) * 2;
        cp_pair<kAl>(s + r * kTP + pc, t.p + (int64_t)min(r, t.rows - 1) * t.ld, c0 + pc, n - (c0 + pc));
    }
}

// The 64 x 64 product of eight warps: warp w owns rows 16 (w >> 1) .. + 16 and
// columns 32 (w & 1) .. + 32, two by four m8n8 fragments.
struct Acc {
    double v[2][4][2];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) v[i][j][0] = v[i][j][1] = 0.0;
    }
};
// acc += A B^T over kn columns (a multiple of 4), row strides lda, ldb.
__device__ __forceinline__ void mma_tile(Acc& acc, const double* A, int lda, const double* B, int ldb,
                                         int k0, int kn) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double* a = A + (16 * (w >> 1) + (lane >> 2)) * lda + (lane & 3);
    const double* b = B + (32 * (w & 1) + (lane >> 2)) * ldb + (lane & 3);
#pragma unroll 4
    for (int k = k0; k < kn; k += 4) {
        double af[2], bf[4];
#pragma unroll
        for (int i = 0; i < 2; i++) af[i] = a[8 * i * lda + k];
#pragma unroll
        for (int j = 0; j < 4; j++) bf[j] = b[8 * j * ldb + k];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) dmma(acc.v[i][j][0], acc.v[i][j][1], af[i], bf[j]);
    }
}
// f(row, column, value) for this thread's elements of the product.
template <class F>
__device__ __forceinline__ void each(const Acc& acc, F&& f) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int r = 16 * (w >> 1) + 8 * i + (lane >> 2), c = 32 * (w & 1) + 8 * j + 2 * (lane & 3);
            f(r, c, acc.v[i][j][0]);
            f(r, c + 1, acc.v[i][j][1]);
        }
}

// ---- the chain's diagonal block ----------------------------------------------

// a (64 x 64, lower) -> L in a, L^-1 in z (whole tile, zero above the diagonal).
// Factor and inverse in one sweep over the columns: right-looking on the 64 rows
// of A and, below them, the rows of the identity, which become L^-T. At column
// k only the A rows below k and the identity rows up to k are alive, 64 in all,
// so slot r holds A's row r until column r is done and the identity's row r from
// then on: 16 registers a thread (warp w: columns 8w .. 8w + 7; lane: rows lane
// and lane + 32). Warp p takes its eight columns by shuffles (one reciprocal, two
// operations and a shuffle per column) and leaves them unscaled in rows 8p .. of
// z; the warps after it then apply all eight. One pass at the end scales by
// 1/L_kk into L and L^-1. inv: 64 reciprocal pivots.
__device__ __forceinline__ void potrf64(double* a, double* z, double* inv, double tol, int32_t* bad) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double v[2][8];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int c = 0; c < 8; c += 2) {
            const int r = lane + 32 * h;
            const double2 t = *reinterpret_cast<const double2*>(a + r * kTP + 8 * w + c);
            v[h][c] = r >= 8 * w + c ? t.x : 0.0;
            v[h][c + 1] = r >= 8 * w + c + 1 ? t.y : 0.0;
        }
    for (int p = 0; p < 8; p++) {
        if (w == p) {
            const int own = (8 * p) & 31;     // lane of the panel's first row
            const int r0 = lane - 8 * p, r1 = r0 + 32;  // rows counted from the panel's first
#pragma unroll
            for (int c = 0; c < 8; c++) {
                const double x0 = v[0][c], x1 = v[1][c];
                z[(8 * p + c) * kTP + lane] = x0;
                z[(8 * p + c) * kTP + lane + 32] = x1;
                const double xs = p < 4 ? x0 : x1;
                double piv = __shfl_sync(0xffffffffu, xs, own + c);
                double l[8];
#pragma unroll
                for (int q = c + 1; q < 8; q++) l[q] = __shfl_sync(0xffffffffu, xs, own + q);
                if (!(piv > tol)) piv = 1.0;
                const double iv = recip_normal(piv);
                if (lane == 0) inv[8 * p + c] = iv;
                const double t0 = r0 == c ? iv : x0 * iv, t1 = r1 == c ? iv : x1 * iv;
#pragma unroll
                for (int q = c + 1; q < 8; q++) {
                    // slot k turns into the identity's row k
                    v[0][q] = fma(-t0, l[q], r0 == c ? 0.0 : v[0][q]);
                    v[1][q] = fma(-t1, l[q], r1 == c ? 0.0 : v[1][q]);
                }
            }
        }
        __syncthreads();
        if (w <= p) continue;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const int k = 8 * p + c;
            const double* col = z + k * kTP;
            const double iv = inv[k];
            double t0 = (lane == k ? 1.0 : col[lane]) * iv, t1 = (lane + 32 == k ? 1.0 : col[lane + 32]) * iv;
            // a row above this warp's columns and below k is neither yet
            if (lane > k && lane < 8 * w) t0 = 0.0;
            if (lane + 32 > k && lane + 32 < 8 * w) t1 = 0.0;
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
                const double2 l = *reinterpret_cast<const double2*>(col + 8 * w + q);
                v[0][q] = fma(-t0, l.x, v[0][q]);
                v[0][q + 1] = fma(-t0, l.y, v[0][q + 1]);
                v[1][q] = fma(-t1, l.x, v[1][q]);
                v[1][q + 1] = fma(-t1, l.y, v[1][q + 1]);
            }
        }
    }
    // warp w scales columns w, w + 8, ..: z[k][r] holds L_rk below and W_rk above the diagonal
    bool brk = false;
    double y[8][2], rs[8], d[8];
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int k = w + 8 * q;
        double piv = z[k * kTP + k];
        if (!(piv > tol)) {
            brk = true;
            piv = 1.0;
        }
        rs[q] = rsqrt(piv);
        d[q] = piv * rs[q];
        y[q][0] = z[k * kTP + lane] * rs[q];
        y[q][1] = z[k * kTP + lane + 32] * rs[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int k = w + 8 * q;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = lane + 32 * h;
            if (r >= k) a[r * kTP + k] = r == k ? d[q] : y[q][h];
            z[k * kTP + r] = r < k ? y[q][h] : (r == k ? rs[q] : 0.0);
        }
    }
    if (brk && lane == 0) atomicExch(bad, 1);
    __syncthreads();
}

// 64 x 64 products of the chain, eight warps of 8 rows x 64 columns; warp w < 4
// takes row group w, warp w + 4 row group 7 - w (their schedulers then carry the
// same number of the lower triangle's fragments).
__device__ __forceinline__ int row_group() {
    const int w = threadIdx.x >> 5;
    return w < 4 ? w : 11 - w;
}
struct RowAcc {
    double v[8][2];
};
// acc = A Z^T, Z lower triangular (columns m <= c of row c).
__device__ __forceinline__ void mma_lower(RowAcc& acc, const double* A, const double* Z) {
    const int lane = threadIdx.x & 31;
    const double* a = A + (8 * row_group() + (lane >> 2)) * kTP + (lane & 3);
    const double* b = Z + (lane >> 2) * kTP + (lane & 3);
#pragma unroll
    for (int j = 0; j < 8; j++) acc.v[j][0] = acc.v[j][1] = 0.0;
#pragma unroll
    for (int kg = 0; kg < 8; kg++)
#pragma unroll
        for (int k = 8 * kg; k < 8 * kg + 8; k += 4) {
            const double af = a[k];
#pragma unroll
            for (int j = kg; j < 8; j++) dmma(acc.v[j][0], acc.v[j][1], af, b[8 * j * kTP + k]);
        }
}
// acc = A A^T on the fragments at or left of the diagonal (an even number of them).
template <int NJ>
__device__ __forceinline__ void mma_syrk_n(RowAcc& acc, const double* a, const double* b) {
#pragma unroll 4
    for (int k = 0; k < NB; k += 4) {
        const double af = a[k];
#pragma unroll
        for (int j = 0; j < NJ; j++) dmma(acc.v[j][0], acc.v[j][1], af, b[8 * j * kTP + k]);
    }
}
__device__ __forceinline__ void mma_syrk(RowAcc& acc, const double* A) {
    const int lane = threadIdx.x & 31, g = row_group();
    const double* a = A + (8 * g + (lane >> 2)) * kTP + (lane & 3);
    const double* b = A + (lane >> 2) * kTP + (lane & 3);
#pragma unroll
    for (int j = 0; j < 8; j++) acc.v[j][0] = acc.v[j][1] = 0.0;
    if (g < 2)
        mma_syrk_n<2>(acc, a, b);
    else if (g < 4)
        mma_syrk_n<4>(acc, a, b);
    else if (g < 6)
        mma_syrk_n<6>(acc, a, b);
    else
        mma_syrk_n<8>(acc, a, b);
}
template <class F>
__device__ __forceinline__ void each_row(const RowAcc& acc, F&& f) {
    const int lane = threadIdx.x & 31, r = 8 * row_group() + (lane >> 2);
#pragma unroll
    for (int j = 0; j < 8; j++) {
        f(r, 8 * j + 2 * (lane & 3), acc.v[j][0]);
        f(r, 8 * j + 2 * (lane & 3) + 1, acc.v[j][1]);
    }
}

// ---- waits -------------------------------------------------------------------

// Thread 0 waits until *f is set; false when the wait ran out or another did.
__device__ __forceinline__ bool wait_one(const Dag& g, const int32_t* f, int32_t* ok) {
    if (threadIdx.x == 0) {
        int32_t it = 0, good = 1;
        while (ld_acquire(f) == 0) {
            if (++it > g.limit || ((it & 63) == 0 && ld_acquire(g.ctl + 1))) {
                atomicExch(g.ctl + 1, 1);
                good = 0;
                break;
            }
            __nanosleep(20);
        }
        *ok = good;
    }
    __syncthreads();
    const bool r = *ok != 0;
    __syncthreads();
    return r;
}

// Extends *ready (the tiles fa[k], fb[k], k < *ready, are done) beyond k, at most
// 32 more and to `end`. Whole block; false when a wait ran out.
__device__ __forceinline__ bool wait_more(const Dag& g, const int32_t* fa, const int32_t* fb, int32_t k,
                                          int32_t end, int32_t* ready) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int32_t it = 0, got;
        for (;;) {
            const bool in = k + lane < end;
            const int32_t s = !in || (ld_acquire(fa + k + lane) && ld_acquire(fb + k + lane));
            const uint32_t m = __ballot_sync(0xffffffffu, s);
            got = m == 0xffffffffu ? 32 : __ffs(~m) - 1;
            if (got > 0) break;
            int32_t stop = 0;
            if (lane == 0) stop = ++it > g.limit || ((it & 63) == 0 && ld_acquire(g.ctl + 1));
            if (__shfl_sync(0xffffffffu, stop, 0)) break;
            __nanosleep(20);
        }
        if (lane == 0) {
            if (got == 0) atomicExch(g.ctl + 1, 1);
            *ready = got == 0 ? -1 : min(end, k + got);
        }
    }
    __syncthreads();
    const bool r = *ready >= 0;
    return r;
}

// The block's stores are done: raise f (the barrier orders them before thread 0's
// fence, the fence before the flag).
__device__ __forceinline__ void raise(int32_t* f) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        st_release(f, 1);
    }
}

// ---- tiles ---------------------------------------------------------------------

struct Smem {
    double buf[4 * kStage];  // A, B chunks, two stages; then T and Linv tiles
    int32_t ok, ready, item;
};

// A whole tile's space after Smem: the chain's tile, or a worker's original tile.
__device__ __forceinline__ double* dyn_tile() {
    extern __shared__ __align__(16) double dyn[];
    return dyn + (sizeof(Smem) + 15) / 16 * 2;
}

// acc += sum over tiles k in [k0, k1) of A_k B_k^T, A_k / B_k the 64 columns from
// 64 k of the two row blocks, waiting for their flags on the way.
template <bool kAl>
__device__ __forceinline__ bool sum_tiles(const Dag& g, Smem& sm, Acc& acc, const Rows& A, const int32_t* fa,
                                          const Rows& B, const int32_t* fb, int32_t k0, int32_t k1) {
    if (k0 >= k1) return true;
    if (!wait_more(g, fa, fb, k0, k1, &sm.ready)) {
        cp_wait<0>();  // (the caller's own fetch)
        return false;
    }
    int32_t ready = sm.ready;
    auto load = [&](int st, int32_t c) {
        load_chunk<kAl>(sm.buf + (2 * st) * kStage, A, c, g.n);
        load_chunk<kAl>(sm.buf + (2 * st + 1) * kStage, B, c, g.n);
        cp_commit();
    };
    const int32_t nch = (k1 - k0) * (NB / kKC);
    load(0, k0 * NB);
    for (int32_t ch = 0; ch < nch; ch++) {
        if (ch + 1 < nch) {
            const int32_t k = k0 + (ch + 1) / (NB / kKC);
            if (k >= ready) {
                if (!wait_more(g, fa, fb, k, k1, &sm.ready)) {
                    cp_wait<0>();
                    return false;
                }
                ready = sm.ready;
            }
            load((ch + 1) & 1, k0 * NB + (ch + 1) * kKC);
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncthreads();
        mma_tile(acc, sm.buf + (2 * (ch & 1)) * kStage, kPad, sm.buf + (2 * (ch & 1) + 1) * kStage, kPad, 0, kKC);
        __syncthreads();
    }
    return true;
}

// One worker tile: row block x of column j. x in numbering order: the chain's two
// sums, rows j + 2 .., right-hand-side row blocks, rows of W.
__device__ __forceinline__ int64_t column_count(const Dag& g, int32_t c) {
    const int32_t below = g.nb - c - 1;
    return (below > 0 ? 1 + below : 0) + g.nrb + (g.W ? c + 1 : 0);
}

template <bool kAl>
__device__ __forceinline__ bool column_tile(const Dag& g, Smem& sm, int32_t j, int32_t x) {
    const int32_t nb = g.nb, n = g.n;
    const int64_t ld = g.ld;
    int32_t* diag = g.flag + (int64_t)(2 * nb + g.nrb) * nb;
    const int32_t s = min(NB, n - j * NB);  // columns of this tile
    const Rows Lj{g.L + (int64_t)j * NB * ld, ld, s};
    const int32_t* fj = g.flag + (int64_t)j * nb;
    const int32_t below = nb - j - 1;  // rows under the diagonal block
    double* O = dyn_tile();  // the tile as it is in memory, fetched ahead of the sum
    Acc acc;
    if (below > 0 && x < 2) {
        // sums of the chain's next tile (x = 0) and next diagonal block (x = 1)
        if (j == 0) return true;
        const int32_t i = j + 1, rows = min(NB, n - i * NB);
        const Rows Li{g.L + (int64_t)i * NB * ld, ld, rows};
        const int32_t* fi = g.flag + (int64_t)i * nb;
        double* out = g.L + (int64_t)i * NB * ld + (int64_t)(x == 0 ? j : i) * NB;
        load_tile<kAl>(O, Li, (x == 0 ? j : i) * NB, n);
        cp_commit();
        acc.zero();
        if (!sum_tiles<kAl>(g, sm, acc, Li, fi, x == 0 ? Lj : Li, x == 0 ? fj : fi, 0, j)) return false;
        each(acc, [&](int r, int c, double v) {
            if (r < rows && (x == 0 || c <= r)) out[r * ld + c] = O[r * kTP + c] - v;
        });
        raise(diag + nb + (x == 0 ? 0 : nb) + j);
        return true;
    }
    if (below > 0) x -= 2;
    // (a row block, its flags, its first column tile, where its tile j lives)
    Rows A;
    int32_t gid, k0 = 0;
    double* out;
    bool isw = false;
    if (x < below - 1) {
        const int32_t i = j + 2 + x;
        gid = i;
        out = g.L + (int64_t)i * NB * ld;
        A = Rows{out, ld, min(NB, n - i * NB)};
    } else if ((x -= std::max(0, below - 1)) < g.nrb) {
        gid = nb + x;
        out = g.B + (int64_t)x * NB * n;
        A = Rows{out, n, min(NB, g.nr - x * NB)};
    } else {
        const int32_t c = x - g.nrb;
        gid = nb + g.nrb + c;
        out = g.W + (int64_t)c * NB * ld;
        A = Rows{out, ld, min(NB, n - c * NB)};
        k0 = c;
        isw = true;
    }
    out += (int64_t)j * NB;
    int32_t* fg = g.flag + (int64_t)gid * nb;
    double* T = sm.buf;
    double* Z = sm.buf + kTile;
    if (isw && k0 == j) {
        // W_jj = inv(L_jj)^T, X_jj = inv(L_jj)
        if (!wait_one(g, diag + j, &sm.ok)) return false;
        load_tile<true>(Z, Rows{g.Linv + (int64_t)j * NB * NB, NB, NB}, 0, NB);
        cp_commit();
        cp_wait<0>();
        __syncthreads();
        for (int e = threadIdx.x; e < NB * NB; e += kThr) {
            const int r = e >> 6, c = e & 63;
            if (r < s && c < s) {
                out[r * ld + c] = Z[c * kTP + r];
                if (g.X) g.X[(int64_t)(j * NB + r) * ld + j * NB + c] = Z[r * kTP + c];
            }
        }
        raise(fg + j);
        return true;
    }
    if (!isw) load_tile<kAl>(O, A, j * NB, n);
    cp_commit();
    acc.zero();
    if (!sum_tiles<kAl>(g, sm, acc, A, fg, Lj, fj, k0, j)) return false;
    cp_wait<0>();
    __syncthreads();
    each(acc, [&](int r, int c, double v) {
        T[r * kTP + c] = c < s ? (isw ? 0.0 : O[r * kTP + c]) - v : 0.0;
    });
    if (!wait_one(g, diag + j, &sm.ok)) return false;
    load_tile<true>(Z, Rows{g.Linv + (int64_t)j * NB * NB, NB, NB}, 0, NB);
    cp_commit();
    cp_wait<0>();
    __syncthreads();
    RowAcc y;
    mma_lower(y, T, Z);
    each_row(y, [&](int r, int c, double v) {
        if (r < A.rows && c < s) out[r * A.ld + c] = v;
    });
    if (isw && g.X) {
        __syncthreads();
        each_row(y, [&](int r, int c, double v) { T[r * kTP + c] = v; });
    }
    if (isw && g.X) {
        __syncthreads();
        for (int e = threadIdx.x; e < NB * NB; e += kThr) {
            const int r = e >> 6, c = e & 63;  // X tile (j, c-block): row r of block j
            if (r < s) g.X[(int64_t)(j * NB + r) * ld + k0 * NB + c] = T[c * kTP + r];
        }
    }
    raise(fg + j);
    return true;
}

// The chain's wait at column j for fa and fb: polls for a while, then works on the tiles
// of the columns up to j itself (none of them needs the chain any further), one after the
// other until both flags are up, so that one running block is enough to finish. The limit counts
// the polls since the last tile. *helped: sm.buf was used.
constexpr int32_t kPatience = 8192;
template <bool kAl>
__device__ __forceinline__ bool chain_wait(const Dag& g, Smem& sm, const int32_t* fa, const int32_t* fb, int32_t j,
                                           bool* helped) {
    *helped = false;
    bool took = false;
    for (int32_t polls = 0; polls <= g.limit; polls += kPatience) {
        if (threadIdx.x == 0) {
            sm.item = -1;
            int32_t it = took ? kPatience - 1 : 0;
            auto up = [&](const int32_t* f) {
                while (ld_acquire(f) == 0) {
                    if (++it >= kPatience || ((it & 63) == 0 && ld_acquire(g.ctl + 1))) return false;
                    __nanosleep(20);
                }
                return true;
            };
            if (up(fa) && up(fb)) {
                sm.ok = 1;
            } else if (ld_acquire(g.ctl + 1)) {
                sm.ok = 0;
            } else {
                sm.ok = 2;
                int64_t end = 0;
                for (int32_t c = 0; c <= j; c++) end += column_count(g, c);
                for (int32_t x = ld_acquire(g.ctl + 3), now; x < end; x = now) {
                    now = atomicCAS(g.ctl + 3, x, x + 1);
                    if (now == x) {
                        sm.item = x;
                        break;
                    }
                }
            }
        }
        __syncthreads();
        const int32_t ok = sm.ok, x = sm.item;
        __syncthreads();
        if (ok < 2) return ok == 1;
        took = x >= 0;
        if (took) {
            int64_t y = x;
            int32_t c = 0;
            while (y >= column_count(g, c)) y -= column_count(g, c++);
            *helped = true;
            if (!column_tile<kAl>(g, sm, c, (int32_t)y)) return false;
            __syncthreads();
            polls = -kPatience;
        }
    }
    if (threadIdx.x == 0) atomicExch(g.ctl + 1, 1);
    return false;
}

// The chain: diagonal blocks, their inverses and the tiles below them.
template <bool kAl>
__device__ __forceinline__ void chain(const Dag& g, Smem& sm) {
    double* a = sm.buf;            // the diagonal block
    double* z = sm.buf + kTile;    // its inverse
    __shared__ double rcp[NB];
    double* t = dyn_tile();        // the tile below it
    int32_t* diag = g.flag + (int64_t)(2 * g.nb + g.nrb) * g.nb;
    int32_t *preA = diag + g.nb, *preD = preA + g.nb;
    // the lower triangle is what counts; past the matrix's end the identity
    auto fetch_diag = [&](int32_t j) {
        load_tile<kAl>(a, Rows{g.L + (int64_t)j * NB * g.ld, g.ld, min(NB, g.n - j * NB)}, j * NB, g.n);
        cp_commit();
    };
    auto pad_diag = [&](int32_t j) {
        const int32_t s = min(NB, g.n - j * NB);
        if (s == NB) return;
        for (int e = threadIdx.x; e < NB * NB; e += kThr) {
            const int r = e >> 6, c = e & 63;
            if (r >= s) a[r * kTP + c] = r == c ? 1.0 : 0.0;
        }
        __syncthreads();
    };
    fetch_diag(0);
    cp_wait<0>();
    __syncthreads();
    pad_diag(0);
    for (int32_t j = 0; j < g.nb; j++) {
        const int32_t r0 = j * NB, s = min(NB, g.n - r0);
        potrf64(a, z, rcp, g.tol, g.ctl);
#pragma unroll 4
        for (int e = threadIdx.x; e < NB * (NB / 2); e += kThr) {
            const int r = e / (NB / 2), c = (e % (NB / 2)) * 2;
            reinterpret_cast<double2*>(g.Linv + (int64_t)j * NB * NB)[e] =
                *reinterpret_cast<const double2*>(z + r * kTP + c);
        }
        raise(diag + j);  // (nothing reads L_jj while this kernel runs)
#pragma unroll 4
        for (int e = threadIdx.x; e < NB * NB; e += kThr) {
            const int r = e >> 6, c = e & 63;
            if (r < s && c <= r) g.L[(int64_t)(r0 + r) * g.ld + r0 + c] = a[r * kTP + c];
        }
        if (j + 1 == g.nb) break;
        const int32_t r1 = r0 + NB, rows = min(NB, g.n - r1);
        bool helped = false;
        if (j > 0 && !chain_wait<kAl>(g, sm, preA + j, preD + j, j, &helped)) return;
        __syncthreads();  // L_jj is stored: a may be overwritten
        if (helped) load_tile<true>(z, Rows{g.Linv + (int64_t)j * NB * NB, NB, NB}, 0, NB);
        load_tile<kAl>(t, Rows{g.L + (int64_t)r1 * g.ld, g.ld, rows}, r0, g.n);
        cp_commit();
        fetch_diag(j + 1);
        cp_wait<1>();
        __syncthreads();
        RowAcc acc;
        mma_lower(acc, t, z);
        __syncthreads();
        each_row(acc, [&](int r, int c, double v) {
            t[r * kTP + c] = r < rows ? v : 0.0;
            if (r < rows) g.L[(int64_t)(r1 + r) * g.ld + r0 + c] = v;
        });
        raise(g.flag + (int64_t)(j + 1) * g.nb + j);
        mma_syrk(acc, t);
        cp_wait<0>();
        __syncthreads();
        each_row(acc, [&](int r, int c, double v) {
            if (c <= r) a[r * kTP + c] -= v;
        });
        __syncthreads();
        pad_diag(j + 1);
    }
}

// Ainv tile (i, j), i >= j, and its mirror.
template <bool kAl>
__device__ __forceinline__ bool inverse_tile(const Dag& g, Smem& sm, int32_t i, int32_t j) {
    const int32_t n = g.n, nb = g.nb;
    const int32_t ri = min(NB, n - i * NB), rj = min(NB, n - j * NB);
    const int32_t* wf = g.flag + (int64_t)(nb + g.nrb) * nb;
    Acc acc;
    acc.zero();
    if (!sum_tiles<kAl>(g, sm, acc, Rows{g.W + (int64_t)i * NB * g.ld, g.ld, ri}, wf + (int64_t)i * nb,
                        Rows{g.W + (int64_t)j * NB * g.ld, g.ld, rj}, wf + (int64_t)j * nb, i, nb))
        return false;
    double* T = sm.buf;
    each(acc, [&](int r, int c, double v) { T[r * kTP + c] = v; });
    __syncthreads();
    for (int e = threadIdx.x; e < NB * NB; e += kThr) {
        const int r = e >> 6, c = e & 63;
        // a diagonal tile takes its lower half for both, so the result is symmetric
        if (r < ri && c < rj)
            g.Ainv[(int64_t)(i * NB + r) * n + j * NB + c] = T[i == j && c > r ? c * kTP + r : r * kTP + c];
        if (i != j && r < rj && c < ri) g.Ainv[(int64_t)(j * NB + r) * n + i * NB + c] = T[c * kTP + r];
    }
    __syncthreads();
    return true;
}

template <bool kAl>
__global__ void __launch_bounds__(kThr, 2) chol_dag_kernel(const Dag g) {
    extern __shared__ __align__(16) double dyn[];
    Smem& sm = *reinterpret_cast<Smem*>(dyn);
    if (threadIdx.x == 0) sm.item = atomicAdd(g.ctl + 2, 1);
    __syncthreads();
    uint32_t smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    if (sm.item == 0) {
        if (threadIdx.x == 0) atomicExch(g.ctl + 4, (int32_t)smid + 1);
        chain<kAl>(g, sm);
        if (threadIdx.x == 0) atomicExch(g.ctl + 4, 0);
        // (then a worker like the others)
    }
    int32_t j = 0;
    int64_t before = 0;  // tiles in the columns before j
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            // the chain has its SM to itself (order 3500: 1230 -> 1030 us)
            const bool off = ld_acquire(g.ctl + 4) == (int32_t)smid + 1;
            sm.item = off ? -1 : atomicAdd(g.ctl + 3, 1);
        }
        __syncthreads();
        const int64_t x = sm.item;
        if (x < 0) return;
        while (j < g.nb && x >= before + column_count(g, j)) before += column_count(g, j++);
        if (j < g.nb) {
            if (!column_tile<kAl>(g, sm, j, (int32_t)(x - before))) return;
            continue;
        }
        if (!g.Ainv) return;
        // inverse tiles row by row (the first rows have the longest sums)
        int64_t y = x - before;
        if (y >= (int64_t)g.nb * (g.nb + 1) / 2) return;
        int32_t i = (int32_t)((sqrt(8.0 * (double)y + 1.0) - 1.0) * 0.5);
        while ((int64_t)i * (i + 1) / 2 > y) i--;
        while ((int64_t)(i + 1) * (i + 2) / 2 <= y) i++;
        if (!inverse_tile<kAl>(g, sm, i, (int32_t)(y - (int64_t)i * (i + 1) / 2))) return;
    }
}

// ---- triangular solves ---------------------------------------------------------

// One triangular solve of up to 64 right-hand sides (rows of B, in place), one
// block of threads per 64 columns: y_j = (b_j - sum_{k<j} y_k L_jk^T) inv(L_jj)^T
// going down (FWD), x_j = (y_j - sum_{i>j} x_i L_ij) inv(L_jj) going up. Blocks
// take their columns from a ticket in solving order, so each waits only for
// blocks that run; the tile of L for the next step is in shared memory before the
// step's vectors are ready. Bound: the chain of columns (flag, vectors, two small
// products, store): 4.7 us each. What does not hang on it is read before the waits (the
// inverse, the block's own right-hand sides): order 2048 175 -> 154 us, 8192 790 -> 594.
// A wait that runs out sets *err and leaves NaN.
constexpr int kMaxG = 4;  // groups of 16 right-hand sides

template <bool NT>  // C[r][c] += sum_m A[r][m] B[c][m] (NT) or A[r][m] B[m][c]; warp = 8 columns
__device__ __forceinline__ void mma_rhs(double (&acc)[2 * kMaxG][2], int ng, const double* A, const double* B) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll 4
    for (int k = 0; k < NB; k += 4) {
        const double b = NT ? B[(8 * w + (lane >> 2)) * kTP + k + (lane & 3)]
                            : B[(k + (lane & 3)) * kTP + 8 * w + (lane >> 2)];
#pragma unroll
        for (int q = 0; q < 2 * kMaxG; q++)
            if (q < 2 * ng) dmma(acc[q][0], acc[q][1], A[(8 * q + (lane >> 2)) * kTP + k + (lane & 3)], b);
    }
}

template <bool kAl, bool FWD>
__global__ void __launch_bounds__(kThr)
tri_dag_kernel(const double* __restrict__ L, const double* __restrict__ Linv, int32_t n, int32_t nb, double* B,
               int32_t nr, int32_t limit, int32_t* flag, int32_t* ticket, int32_t* err) {
    extern __shared__ __align__(16) double dyn[];
    double* tile[2] = {dyn, dyn + kTile};
    double* z = dyn + 2 * kTile;
    double* v = dyn + 3 * kTile;  // 16 ng x kTP: the vectors of one column block
    __shared__ int32_t sh;
    const int ng = (nr + 15) / 16, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) sh = atomicAdd(ticket, 1);
    __syncthreads();
    const int32_t t = sh, j = FWD ? t : nb - 1 - t;
    __syncthreads();
    const int32_t s = min(NB, n - j * NB);
    // step q of this block: column block k = q (down) or nb - 1 - q (up)
    auto col = [&](int32_t q) { return FWD ? q : nb - 1 - q; };
    auto fetch = [&](int32_t q) {
        const int32_t k = col(q);
        if (FWD)
            load_tile<kAl>(tile[q & 1], Rows{L + (int64_t)j * NB * n, n, s}, k * NB, n);
        else  // rows of block k, columns of block j; rows past n meet zero vectors
            load_tile<kAl>(tile[q & 1], Rows{L + (int64_t)k * NB * n, n, min(NB, n - k * NB)}, j * NB, n);
    };
    load_tile<true>(z, Rows{Linv + (int64_t)j * NB * NB, NB, NB}, 0, NB);
    if (t > 0) fetch(0);
    cp_commit();
    // (the block's own right-hand sides are read before the waits, too)
    double acc[2 * kMaxG][2], own[2 * kMaxG][2];
#pragma unroll
    for (int q = 0; q < 2 * kMaxG; q++) {
        acc[q][0] = acc[q][1] = 0.0;
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int r = 8 * q + (lane >> 2), c = 8 * w + 2 * (lane & 3) + e;
            own[q][e] = q < 2 * ng && r < nr && c < s ? B[(int64_t)r * n + j * NB + c] : 0.0;
        }
    }
    bool bad = false;
    for (int32_t q = 0; q < t; q++) {
        if (q + 1 < t) fetch(q + 1);
        cp_commit();
        if (threadIdx.x == 0) {
            int32_t it = 0;
            sh = 1;
            while (ld_acquire(flag + q) == 0)
                if (++it > limit) {
                    atomicExch(err, 1);
                    sh = 0;
                    break;
                }
        }
        __syncthreads();
        bad = bad || sh == 0;
        const int32_t c0 = col(q) * NB, cs = min(NB, n - c0);
        for (int e = threadIdx.x; e < 16 * ng * NB; e += kThr) {
            const int r = e >> 6, c = e & 63;
            v[r * kTP + c] = r < nr && c < cs ? __ldcg(B + (int64_t)r * n + c0 + c) : 0.0;
        }
        cp_wait<1>();
        __syncthreads();
        mma_rhs<FWD>(acc, ng, v, tile[q & 1]);
        __syncthreads();
    }
    cp_wait<0>();
    // own right-hand side minus the sum, times the inverse
#pragma unroll
    for (int q = 0; q < 2 * kMaxG; q++)
        if (q < 2 * ng)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int r = 8 * q + (lane >> 2), c = 8 * w + 2 * (lane & 3) + e;
                v[r * kTP + c] = r < nr && c < s ? own[q][e] - acc[q][e] : 0.0;
                acc[q][e] = 0.0;
            }
    __syncthreads();
    mma_rhs<FWD>(acc, ng, v, z);
#pragma unroll
    for (int q = 0; q < 2 * kMaxG; q++)
        if (q < 2 * ng)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int r = 8 * q + (lane >> 2), c = 8 * w + 2 * (lane & 3) + e;
                if (r < nr && c < s) B[(int64_t)r * n + j * NB + c] = bad ? NAN : acc[q][e];
            }
    raise(flag + t);
}

}  // namespace

// See tpe_internal.h.
int32_t chol_solve(tpe_ctx* ctx, const double* L, const double* Linv, int32_t n, double* B, int32_t nr,
                   bool down) {
    const int32_t nb = (n + NB - 1) / NB;
    const cudaStream_t st = ctx->stream;
    if (!ctx->dag_err.ptr) {
        TPE_TRY(ensure(ctx, ctx->dag_err, sizeof(int32_t)));
        TPE_CUDA_TRY(cudaMemsetAsync(ctx->dag_err.ptr, 0, sizeof(int32_t), st));
    }
    TPE_TRY(ensure(ctx, ctx->dag_solve, sizeof(int32_t) * (2 * (size_t)nb + 2)));
    int32_t* ctl = ctx->dag_solve.as<int32_t>();  // two tickets, then the two directions' flags
    int32_t* err = ctx->dag_err.as<int32_t>();
    const bool al = (n & 1) == 0 && (reinterpret_cast<uintptr_t>(L) & 15) == 0;
    auto kdown = al ? tri_dag_kernel<true, true> : tri_dag_kernel<false, true>;
    auto kup = al ? tri_dag_kernel<true, false> : tri_dag_kernel<false, false>;
    const int most = (int)(sizeof(double) * (3 * kTile + 16 * kMaxG * kTP));
    TPE_CUDA_TRY(cudaFuncSetAttribute(kdown, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    TPE_CUDA_TRY(cudaFuncSetAttribute(kup, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    for (int32_t r0 = 0; r0 < nr; r0 += 16 * kMaxG) {
        const int32_t q = std::min(nr - r0, 16 * kMaxG);
        const size_t smem = sizeof(double) * (3 * kTile + 16 * (size_t)((q + 15) / 16) * kTP);
        double* b = B + (size_t)r0 * n;
        TPE_CUDA_TRY(cudaMemsetAsync(ctl, 0, sizeof(int32_t) * (2 * (size_t)nb + 2), st));
        KernelScope ks(ctx, TPE_KGROUP_TRSV, down ? 2 : 1);
        const int32_t limit = ctx->solve_polls > 0 ? ctx->solve_polls : kSpin;
        if (down) kdown<<<(unsigned)nb, kThr, smem, st>>>(L, Linv, n, nb, b, q, limit, ctl + 2, ctl, err);
        kup<<<(unsigned)nb, kThr, smem, st>>>(L, Linv, n, nb, b, q, limit, ctl + 2 + nb, ctl + 1, err);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    return TPE_OK;
}

int32_t chol_timeout(tpe_ctx* ctx) {
    TPE_CUDA_TRY(cudaMemsetAsync(ctx->dag_err.ptr, 0, sizeof(int32_t), ctx->stream));
    set_error(ctx, TPE_ERR_DEVICE_TIMEOUT, "a wait of the triangular solve ran out");
    return TPE_ERR_DEVICE_TIMEOUT;
}

// See tpe_internal.h.
int32_t chol_dag(tpe_ctx* ctx, const CholDag& c, int32_t* singular) {
    Dag g;
    g.L = c.L;
    g.Linv = c.Linv;
    g.B = c.B;
    g.W = c.W;
    g.X = c.X;
    g.Ainv = c.Ainv;
    g.n = c.n;
    g.ld = c.ld > 0 ? c.ld : c.n;
    g.nb = (c.n + NB - 1) / NB;
    g.nr = c.nr;
    g.nrb = (c.nr + NB - 1) / NB;
    g.tol = c.tol;
    g.limit = ctx->factor_polls > 0 ? ctx->factor_polls : kSpin;
    const size_t nflag = (size_t)(2 * g.nb + g.nrb) * g.nb + 3 * (size_t)g.nb;
    TPE_TRY(ensure(ctx, ctx->dag_flags, sizeof(int32_t) * (nflag + 5)));
    g.ctl = ctx->dag_flags.as<int32_t>();
    g.flag = g.ctl + 5;
    const cudaStream_t st = ctx->stream;
    TPE_CUDA_TRY(cudaMemsetAsync(g.ctl, 0, sizeof(int32_t) * (nflag + 5), st));
    auto even = [](const double* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const bool al = (c.n & 1) == 0 && (g.ld & 1) == 0 && even(c.L) && even(c.B) && even(c.W);
    auto kern = al ? chol_dag_kernel<true> : chol_dag_kernel<false>;
    const size_t smem = (sizeof(Smem) + 15) / 16 * 16 + sizeof(double) * kTile;
    TPE_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // Blocks: a worker holds its tile until the last factor of its sum is done, so the
    // columns ahead of the chain need blocks of their own; nb / 8 - 1 columns of them (nine
    // with the inverse), at most two blocks per SM. Against one column's worth (two with
    // the inverse), us: order 2048 767 -> 575, 3500 1965 -> 1030, 4096 2600 -> 1310; with
    // the inverse 1200 510 -> 357, 2500 1750 -> 1010. Below 1500 rows the chain is the
    // bound, and blocks that wait only take room from other contexts' kernels.
    const int64_t widest = g.nb + g.nrb + 1;
    const unsigned grid = ctx->factor_blocks > 0 ? (unsigned)ctx->factor_blocks : (unsigned)std::min<int64_t>(
        2 * (int64_t)ctx->num_sms, 1 + (c.Ainv ? 9 : std::max(1, g.nb / 8 - 1)) * widest);
    {
        KernelScope ks(ctx, TPE_KGROUP_CHOLESKY, 1);
        kern<<<grid, kThr, smem, st>>>(g);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    if (!singular) return TPE_OK;
    int32_t h[2] = {0, 0};
    TPE_TRY(download_on(ctx, st, h, g.ctl, sizeof(h)));
    *singular = h[0];
    return chol_dag_status(ctx, h);
}

int32_t chol_dag_status(tpe_ctx* ctx, const int32_t flags[2]) {
    if (!flags[1]) return TPE_OK;
    set_error(ctx, TPE_ERR_DEVICE_TIMEOUT, "a wait of the factorization kernel ran out");
    return TPE_ERR_DEVICE_TIMEOUT;
}

}  // namespace tpe
