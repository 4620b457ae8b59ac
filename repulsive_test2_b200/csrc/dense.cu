// Dense FP64 linear algebra of the structured saddle solve: products, residuals,
// reductions and vector helpers. The reference factors the (3V+k)^2 saddle matrix
// with Bunch-Kaufman LDL^T (src/core/sobolev/linsolve.ts:431-589). Here the only
// large factorization is the SPD V x V matrix A_rho = A + (rho/V) 1 1^T (A is
// PSD with the constants as its kernel), which needs no pivoting (chol_dag.cu).
#include <math.h>

#include "tpe_internal.h"

namespace tpe {
namespace {

// ---- C = alpha A B^T + beta C on the FP64 tensor cores ------------------------
//
// For the public product (tpe_gemm_nt_device) alone: the step's own products are chol_dag.cu's
// and ozaki.cu's.
//
// mma.sync m8n8k4 f64: 128x128 output tiles, 8 warps as 2 (rows) x 4 (cols), each
// warp 64x32 = 8x4 MMA tiles. K runs in chunks of 32 staged by 16-byte cp.async
// into two shared-memory buffers; rows are padded to 36 doubles (72 words = 8
// banks mod 32) so a fragment load (8 rows x 4 k) takes the minimum two wavefronts.
constexpr int GT = 128;
constexpr int GK = 32;
constexpr int GP = GK + 4;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
// Two doubles into 16-byte aligned shared memory from a source that may be
// only 8-byte aligned (an odd row length).
template <bool kAligned16>
__device__ __forceinline__ void cp_async_pair(void* smem, const double* gmem) {
    if (kAligned16) {
        cp_async16(smem, gmem);
    } else {
        const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s + 8), "l"(gmem + 1));
    }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Row-major operands, rows past M / N clamped (never stored), a zero-filled K tail
// and optional structure:
// kDLowerTiles computes only tiles with tile column <= tile row; kDAUpper
// (A[i][k] = 0 for k < i) starts the K loop of tile row t at 128 t, kDALower
// (A[i][k] = 0 for k > i) ends it at 128 (t + 1).
template <bool kAligned16>
__global__ void __launch_bounds__(256) dgemm_nt_kernel(const DGemmArgs g) {
    extern __shared__ double dsm[];
    const int32_t ti = blockIdx.y, tj = blockIdx.x;
    if ((g.mode & kDLowerTiles) && tj > ti) return;
    const int32_t r0 = ti * GT, c0 = tj * GT;
    int32_t kb = 0, ke = g.K;
    if (g.mode & kDAUpper) kb = min(g.K, r0);
    if (g.mode & kDALower) ke = min(g.K, r0 + GT);
    double* As = dsm;                // [2][GT][GP]
    double* Bs = dsm + 2 * GT * GP;  // [2][GT][GP]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = (warp >> 2) * 64, wc = (warp & 3) * 32;
    const int fr = lane >> 2, fk = lane & 3;
    auto load = [&](int buf, int kc) {
        for (int idx = tid; idx < GT * (GK / 2); idx += 256) {
            const int rr = idx / (GK / 2), pc = (idx % (GK / 2)) * 2;
            const int32_t k = kb + kc + pc;
            const int64_t ra = min(r0 + rr, g.M - 1), rb = min(c0 + rr, g.N - 1);
            double* da = As + (size_t)buf * GT * GP + rr * GP + pc;
            double* db = Bs + (size_t)buf * GT * GP + rr * GP + pc;
            if (k + 1 < ke) {
                cp_async_pair<kAligned16>(da, g.A + ra * g.lda + k);
                cp_async_pair<kAligned16>(db, g.B + rb * g.ldb + k);
            } else {
                da[0] = k < ke ? g.A[ra * g.lda + k] : 0.0;
                db[0] = k < ke ? g.B[rb * g.ldb + k] : 0.0;
                da[1] = 0.0;
                db[1] = 0.0;
            }
        }
        cp_async_commit();
    };
    double acc[8][4][2];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
    const int nch = ke > kb ? (ke - kb + GK - 1) / GK : 0;
    if (nch > 0) load(0, 0);
    for (int ch = 0; ch < nch; ch++) {
        if (ch + 1 < nch) {
            load((ch + 1) & 1, (ch + 1) * GK);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const double* Ab = As + (size_t)(ch & 1) * GT * GP + (wr + fr) * GP + fk;
        const double* Bb = Bs + (size_t)(ch & 1) * GT * GP + (wc + fr) * GP + fk;
#pragma unroll
        for (int kk = 0; kk < GK; kk += 4) {
            double af[8], bf[4];
#pragma unroll
            for (int i = 0; i < 8; i++) af[i] = Ab[i * 8 * GP + kk];
#pragma unroll
            for (int j = 0; j < 4; j++) bf[j] = Bb[j * 8 * GP + kk];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int32_t row = r0 + wr + 8 * i + fr;
        if (row >= g.M) continue;
        double* cp = g.C + (int64_t)row * g.ldc;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int32_t col = c0 + wc + 8 * j + 2 * fk;
#pragma unroll
            for (int e = 0; e < 2; e++) {
                if (col + e >= g.N) continue;
                double y = g.alpha * acc[i][j][e];
                if (g.beta != 0.0) y += g.beta * cp[col + e];
                cp[col + e] = y;
            }
        }
    }
}

// dst[j][i] = src[i][j] for an m x c block (row strides lds, ldd), 32 x 32 tiles.
__global__ void transpose_fp64_kernel(const double* __restrict__ src, int64_t lds, int32_t m,
                                      int32_t c, double* __restrict__ dst, int64_t ldd) {
    __shared__ double t[32][33];
    const int32_t i0 = blockIdx.y * 32, j0 = blockIdx.x * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int32_t i = i0 + r, j = j0 + threadIdx.x;
        if (i < m && j < c) t[r][threadIdx.x] = src[(int64_t)i * lds + j];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int32_t j = j0 + r, i = i0 + threadIdx.x;
        if (i < m && j < c) dst[(int64_t)j * ldd + i] = t[threadIdx.x][r];
    }
}

// M[i][j] = M[j][i] for j > i (the lower triangle mirrored onto the upper),
// one 32 x 32 tile pair per block.
__global__ void mirror_lower_kernel(double* __restrict__ M, int32_t n) {
    __shared__ double t[32][33];
    const int32_t bi = blockIdx.y, bj = blockIdx.x;  // source tile (bi, bj), bi >= bj
    if (bj > bi) return;
    const int32_t i0 = bi * 32, j0 = bj * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int32_t i = i0 + r, j = j0 + threadIdx.x;
        if (i < n && j < n) t[r][threadIdx.x] = M[(int64_t)i * n + j];
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        const int32_t row = j0 + r, col = i0 + threadIdx.x;  // (row, col) = (j, i)
        if (row < n && col < n && col > row) M[(int64_t)row * n + col] = t[threadIdx.x][r];
    }
}

// ---- reductions and vector helpers -----------------------------------------

template <int BS>
__device__ __forceinline__ double block_sum(double v) {
    __shared__ double red[BS / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < BS / 32; w++) t += red[w];
    __syncthreads();
    return t;  // valid on thread 0
}

// out[i*ny + j] = sum_t X[i][t] * Y[j][t]; one CTA per (i, j).
__global__ void __launch_bounds__(256)
gram_dots_kernel(const double* __restrict__ X, const double* __restrict__ Y, int32_t ny,
                 int64_t len, double* __restrict__ out) {
    const int32_t i = blockIdx.x / ny, j = blockIdx.x % ny;
    const double* x = X + (int64_t)i * len;
    const double* y = Y + (int64_t)j * len;
    double s = 0.0;
    for (int64_t t = threadIdx.x; t < len; t += blockDim.x) s += x[t] * y[t];
    s = block_sum<256>(s);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

__global__ void shift_copy_kernel(const double* __restrict__ A, double* __restrict__ L, int32_t n,
                                  double shift) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)n * n) return;
    const int32_t i = (int32_t)(t / n), j = (int32_t)(t % n);
    L[t] = (j <= i) ? A[t] + shift : 0.0;
}

__global__ void trace_kernel(const double* __restrict__ A, int32_t n, double* __restrict__ out) {
    double s = 0.0;
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) s += A[(int64_t)i * n + i];
    s = block_sum<256>(s);
    if (threadIdx.x == 0) *out = s;
}

__global__ void to_block_kernel(const double* __restrict__ v3, double* __restrict__ f, int32_t V) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    f[i] = v3[3 * i];
    f[V + i] = v3[3 * i + 1];
    f[2 * V + i] = v3[3 * i + 2];
}

__global__ void to_interleaved_kernel(const double* __restrict__ f, double* __restrict__ v3,
                                      int32_t V) {
    const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V) return;
    v3[3 * i] = f[i];
    v3[3 * i + 1] = f[V + i];
    v3[3 * i + 2] = f[2 * V + i];
}

__global__ void axpby_kernel(int64_t n, double a, const double* __restrict__ x, double b,
                             double* __restrict__ y) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) y[t] = a * x[t] + b * y[t];
}

// Two-stage deterministic dot / non-finite count (partials then one CTA).
__global__ void __launch_bounds__(256)
dot_partial_kernel(int64_t n, const double* __restrict__ x, const double* __restrict__ y,
                   double* __restrict__ part) {
    double s = 0.0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x)
        s += x[t] * (y ? y[t] : 1.0);
    s = block_sum<256>(s);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void __launch_bounds__(256)
nonfinite_partial_kernel(int64_t n, const double* __restrict__ x, double* __restrict__ part) {
    double s = 0.0;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x)
        s += isfinite(x[t]) ? 0.0 : 1.0;
    s = block_sum<256>(s);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void __launch_bounds__(256)
sum_kernel(const double* __restrict__ part, int32_t n, double* __restrict__ out) {
    double s = 0.0;
    for (int32_t t = threadIdx.x; t < n; t += blockDim.x) s += part[t];
    s = block_sum<256>(s);
    if (threadIdx.x == 0) *out = s;
}

// out[r] = the sum of row r (n entries), one block a row.
__global__ void __launch_bounds__(256)
row_sums_kernel(const double* __restrict__ x, int32_t n, double* __restrict__ out) {
    const double* row = x + (size_t)blockIdx.x * n;
    double s = 0.0;
    for (int32_t t = threadIdx.x; t < n; t += blockDim.x) s += row[t];
    s = block_sum<256>(s);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}

// Per-edge l2CurveNorm terms (lineSearch.ts:53-75).
__global__ void l2_terms_kernel(const double* __restrict__ vals, const double* __restrict__ pos,
                                const int2* __restrict__ edges, int32_t E,
                                double* __restrict__ terms) {
    const int32_t I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= E) return;
    const int2 e = edges[I];
    const double ex = pos[3 * e.y] - pos[3 * e.x];
    const double ey = pos[3 * e.y + 1] - pos[3 * e.x + 1];
    const double ez = pos[3 * e.y + 2] - pos[3 * e.x + 2];
    const double ell = sqrt(ex * ex + ey * ey + ez * ez);
    const double* v1 = vals + 3 * e.x;
    const double* v2 = vals + 3 * e.y;
    terms[I] = 0.5 * ell *
               (v1[0] * v1[0] + v1[1] * v1[1] + v1[2] * v1[2] +
                (v2[0] * v2[0] + v2[1] * v2[1] + v2[2] * v2[2]));
}

// x = w - sum_s Y[s] lam[s] - (mu_c / (rho sqrt(V))) in block c.
// Y^T coef for nu <= 16 coefficient vectors (coef[q]: k multipliers, then the
// 3 scaled mu), Y k x m (block layout), split over ks chunks of rows s:
// part[ks][q][t] = -sum_{s in chunk ks} Y[s][t] coef[q][s], s in order. The
// number of chunks depends on k only, so every caller sums in the same order.
constexpr int kYcMaxQ = 16;
inline int32_t ycomb_chunks(int32_t k) { return k >= 512 ? min(32, k / 256) : 1; }

__global__ void __launch_bounds__(256)
ycomb_part_kernel(const double* __restrict__ Y, int32_t k, int64_t m,
                  const double* __restrict__ coef, int32_t nu, double* __restrict__ part) {
    constexpr int kChunk = 64;
    __shared__ double cs[kChunk][kYcMaxQ];
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int32_t ks = blockIdx.y, nks = gridDim.y;
    const int32_t per = (k + nks - 1) / nks;
    const int32_t sb = ks * per, se = min(k, sb + per);
    double v[kYcMaxQ];
#pragma unroll
    for (int q = 0; q < kYcMaxQ; q++) v[q] = 0.0;
    for (int32_t s0 = sb; s0 < se; s0 += kChunk) {
        const int32_t n = min(kChunk, se - s0);
        __syncthreads();
        for (int e = threadIdx.x; e < kChunk * kYcMaxQ; e += blockDim.x) {
            const int q = e / kChunk, j = e % kChunk;
            cs[j][q] = (q < nu && j < n) ? coef[(size_t)q * (k + 3) + s0 + j] : 0.0;
        }
        __syncthreads();
        if (t < m) {
            for (int j = 0; j < n; j++) {
                const double y = Y[(int64_t)(s0 + j) * m + t];
#pragma unroll
                for (int q = 0; q < kYcMaxQ; q++)
                    if (q < nu) v[q] -= y * cs[j][q];
            }
        }
    }
    if (t >= m) return;
    for (int q = 0; q < nu; q++) part[((int64_t)ks * nu + q) * m + t] = v[q];
}

// x = w - Y^T coef - mu term (one vector, block layout; w may be null).
__global__ void combine_final_kernel(const double* __restrict__ w, const double* __restrict__ part,
                                     int32_t nks, int32_t k, const double* __restrict__ coef,
                                     int32_t V, double* __restrict__ x) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t m = 3 * (int64_t)V;
    if (t >= m) return;
    double v = w ? w[t] : 0.0;
    for (int32_t ks = 0; ks < nks; ks++) v += part[(int64_t)ks * m + t];
    v -= coef[k + (int32_t)(t / V)];
    x[t] = v;
}

// cur[idx[q]] (interleaved V x 3) += -Y^T coef[q] - mu term, flagging non-finite
// corrections in bad[idx[q]]; the same sums as combine_final_kernel with w = 0.
__global__ void proj_final_kernel(double* __restrict__ cur, int64_t stride,
                                  const double* __restrict__ part, int32_t nks, int32_t nu,
                                  int32_t k, const double* __restrict__ coef,
                                  const int32_t* __restrict__ idx, int32_t V,
                                  int32_t* __restrict__ bad) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t m = 3 * (int64_t)V;
    const int q = blockIdx.y;
    if (t >= m) return;
    double v = 0.0;
    for (int32_t ks = 0; ks < nks; ks++) v += part[((int64_t)ks * nu + q) * m + t];
    const int c = (int)(t / V);
    v -= coef[(size_t)q * (k + 3) + k + c];
    const int a = idx[q];
    if (!isfinite(v)) bad[a] = 1;
    double* p = cur + (int64_t)a * stride + 3 * (t % V) + c;
    *p = *p + v;
}

// Residual rows: top (3V): A x_c + (C^T lam)_c - rhs ; one thread per (c, i),
// grouped so each A row is read once for the three blocks; ctl = C^T lam
// (precomputed, null when k = 0). res (optional) receives rhs - (A x + C^T lam).
__global__ void __launch_bounds__(256)
residual_top_kernel(const double* __restrict__ A, int32_t V, const double* __restrict__ ctl,
                    const double* __restrict__ x, const double* __restrict__ rhs,
                    double* __restrict__ out_res, double* __restrict__ out_rhs,
                    double* __restrict__ res) {
    // one CTA per row i: 256 threads stride the row
    const int32_t i = blockIdx.x;
    const double* Ai = A + (int64_t)i * V;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int32_t j = threadIdx.x; j < V; j += blockDim.x) {
        const double a = Ai[j];
        s0 += a * x[j];
        s1 += a * x[V + j];
        s2 += a * x[2 * V + j];
    }
    s0 = block_sum<256>(s0);
    s1 = block_sum<256>(s1);
    s2 = block_sum<256>(s2);
    if (threadIdx.x == 0) {
        double r2 = 0.0, b2 = 0.0;
        double s[3] = {s0, s1, s2};
        for (int c = 0; c < 3; c++) {
            const int64_t row = (int64_t)c * V + i;
            double v = s[c];
            if (ctl) v += ctl[row];
            const double d = v - rhs[row];
            if (res) res[row] = -d;
            r2 += d * d;
            b2 += rhs[row] * rhs[row];
        }
        out_res[i] = r2;
        out_rhs[i] = b2;
    }
}

// out[row] = sum_r C[r][row] lam[r] (C k x m row-major), r in order.
__global__ void __launch_bounds__(256)
ct_lambda_kernel(const double* __restrict__ C, int32_t k, int64_t m, const double* __restrict__ lam,
                 double* __restrict__ out) {
    const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= m) return;
    double v = 0.0;
    for (int32_t r = 0; r < k; r++) v += C[(int64_t)r * m + row] * lam[r];
    out[row] = v;
}

inline int32_t grid_for(int64_t n, int bs) { return (int32_t)((n + bs - 1) / bs); }

}  // namespace

int32_t gram_dots(tpe_ctx* ctx, const double* X, int32_t nx, const double* Y, int32_t ny,
                  int64_t len, double* d_out) {
    if (nx <= 0 || ny <= 0) return TPE_OK;
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    gram_dots_kernel<<<nx * ny, 256, 0, ctx->stream>>>(X, Y, ny, len, d_out);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t row_sums(tpe_ctx* ctx, const double* x, int32_t rows, int32_t n, double* d_out) {
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    row_sums_kernel<<<rows, 256, 0, ctx->stream>>>(x, n, d_out);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t shift_copy(tpe_ctx* ctx, const double* d_A, double* d_L, int32_t n, double shift) {
    const int64_t nn = (int64_t)n * n;
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    shift_copy_kernel<<<grid_for(nn, 256), 256, 0, ctx->stream>>>(d_A, d_L, n, shift);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t trace(tpe_ctx* ctx, const double* d_A, int32_t n, double* d_out) {
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    trace_kernel<<<1, 256, 0, ctx->stream>>>(d_A, n, d_out);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t interleaved_to_block(tpe_ctx* ctx, const double* d_v3, double* d_flat, int32_t V) {
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    to_block_kernel<<<grid_for(V, 256), 256, 0, ctx->stream>>>(d_v3, d_flat, V);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t block_to_interleaved(tpe_ctx* ctx, const double* d_flat, double* d_v3, int32_t V) {
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    to_interleaved_kernel<<<grid_for(V, 256), 256, 0, ctx->stream>>>(d_flat, d_v3, V);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t axpby(tpe_ctx* ctx, int64_t n, double a, const double* x, double b, double* y) {
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    axpby_kernel<<<grid_for(n, 256), 256, 0, ctx->stream>>>(n, a, x, b, y);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

static int32_t reduce_to_host(tpe_ctx* ctx, double* part, int32_t nparts, double* out) {
    double* dst = part + nparts;
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    sum_kernel<<<1, 256, 0, ctx->stream>>>(part, nparts, dst);
    TPE_CUDA_TRY(cudaGetLastError());
    return download_on(ctx, ctx->stream, out, dst, sizeof(double));
}

int32_t dot(tpe_ctx* ctx, int64_t n, const double* x, const double* y, double* out) {
    const int32_t g = 256;
    TPE_TRY(ensure(ctx, ctx->scalars, sizeof(double) * (g + 8)));
    { KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    dot_partial_kernel<<<g, 256, 0, ctx->stream>>>(n, x, y, ctx->scalars.as<double>()); }
    TPE_CUDA_TRY(cudaGetLastError());
    return reduce_to_host(ctx, ctx->scalars.as<double>(), g, out);
}

int32_t count_nonfinite(tpe_ctx* ctx, int64_t n, const double* x, const double** d_out) {
    const int32_t g = 256;
    TPE_TRY(ensure(ctx, ctx->scalars, sizeof(double) * 600));
    double* part = ctx->scalars.as<double>();
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 2);
    nonfinite_partial_kernel<<<g, 256, 0, ctx->stream>>>(n, x, part);
    sum_kernel<<<1, 256, 0, ctx->stream>>>(part, g, part + g);
    TPE_CUDA_TRY(cudaGetLastError());
    *d_out = part + g;
    return TPE_OK;
}

int32_t l2_curve_norm(tpe_ctx* ctx, const double* d_vals, const double* d_pos, double* out) {
    const int32_t E = ctx->E;
    TPE_TRY(ensure(ctx, ctx->tmp, sizeof(double) * (size_t)(E + 8)));
    { KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    l2_terms_kernel<<<grid_for(E, 256), 256, 0, ctx->stream>>>(d_vals, d_pos,
                                                               ctx->d_edges.as<int2>(), E,
                                                               ctx->tmp.as<double>()); }
    TPE_CUDA_TRY(cudaGetLastError());
    double total = 0.0;
    TPE_TRY(dot(ctx, E, ctx->tmp.as<double>(), nullptr, &total));
    *out = sqrt(total > 0.0 ? total : 0.0);
    if (total != total) *out = NAN;
    return TPE_OK;
}

int32_t combine_solution(tpe_ctx* ctx, const double* d_w, const double* d_Y, int32_t k,
                         const double* lam, const double* mu, double rho, int32_t V, double* d_x) {
    std::vector<double> coef((size_t)k + 3, 0.0);
    for (int32_t s = 0; s < k; s++) coef[s] = lam[s];
    const double su = 1.0 / (rho * sqrt((double)V));
    for (int c = 0; c < 3; c++) coef[(size_t)k + c] = mu ? mu[c] * su : 0.0;
    TPE_TRY(ensure(ctx, ctx->scalars, sizeof(double) * (size_t)(k + 3 + 512)));
    double* dc = ctx->scalars.as<double>() + 264;
    TPE_CUDA_TRY(cudaMemcpyAsync(dc, coef.data(), sizeof(double) * coef.size(),
                                 cudaMemcpyHostToDevice, ctx->stream));
    const int64_t m = 3 * (int64_t)V;
    const int32_t nks = ycomb_chunks(k);
    TPE_TRY(ensure(ctx, ctx->ycomb_part, sizeof(double) * (size_t)nks * kYcMaxQ * m));
    double* part = ctx->ycomb_part.as<double>();
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 2);
    ycomb_part_kernel<<<dim3(grid_for(m, 256), nks), 256, 0, ctx->stream>>>(d_Y, k, m, dc, 1, part);
    combine_final_kernel<<<grid_for(m, 256), 256, 0, ctx->stream>>>(d_w, part, nks, k, dc, V, d_x);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;  // (a copy from pageable memory returns once the data is staged)
}

int32_t project_update(tpe_ctx* ctx, const double* d_Y, int32_t k, int32_t V, const double* d_coef,
                       int32_t nu, const int32_t* d_idx, double* d_cur, int64_t stride,
                       int32_t* d_bad) {
    if (nu <= 0) return TPE_OK;
    if (nu > kYcMaxQ) {
        set_error(ctx, TPE_ERR_TOO_LARGE, "project_update: at most 16 trials per update");
        return TPE_ERR_TOO_LARGE;
    }
    const int64_t m = 3 * (int64_t)V;
    const int32_t nks = ycomb_chunks(k);
    TPE_TRY(ensure(ctx, ctx->ycomb_part, sizeof(double) * (size_t)nks * kYcMaxQ * m));
    double* part = ctx->ycomb_part.as<double>();
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 2);
    ycomb_part_kernel<<<dim3(grid_for(m, 256), nks), 256, 0, ctx->stream>>>(d_Y, k, m, d_coef, nu,
                                                                            part);
    proj_final_kernel<<<dim3(grid_for(m, 256), nu), 256, 0, ctx->stream>>>(
        d_cur, stride, part, nks, nu, k, d_coef, d_idx, V, d_bad);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t saddle_residual(tpe_ctx* ctx, const double* d_A, int32_t V, const double* d_C, int32_t k,
                        const double* d_x, const double* lam, const double* d_rhs_top,
                        const double* rhs_bottom, double* out, double* d_res_top,
                        double* res_bottom, const SaddleOp* large) {
    const int64_t m = 3 * (int64_t)V;
    TPE_TRY(ensure(ctx, ctx->tmp, sizeof(double) * (size_t)(2 * V + 16 + k + m)));
    TPE_TRY(ensure(ctx, ctx->scalars, sizeof(double) * (size_t)(k + 3 + 512)));
    double* dl = ctx->scalars.as<double>() + 264;
    if (k > 0)
        TPE_CUDA_TRY(cudaMemcpyAsync(dl, lam, sizeof(double) * k, cudaMemcpyHostToDevice,
                                     ctx->stream));
    double* rr = ctx->tmp.as<double>();
    double* rb = rr + V;
    double* ctl = rb + V + 16 + k;
    if (large && k > 0) TPE_TRY(large_ct(ctx, *large, dl, ctl));
    {
        KernelScope ks(ctx, TPE_KGROUP_OTHER, k > 0 && !large ? 2 : 1);
        if (k > 0 && !large)
            ct_lambda_kernel<<<grid_for(m, 256), 256, 0, ctx->stream>>>(d_C, k, m, dl, ctl);
        residual_top_kernel<<<V, 256, 0, ctx->stream>>>(d_A, V, k > 0 ? ctl : nullptr, d_x, d_rhs_top,
                                                        rr, rb, d_res_top);
    }
    TPE_CUDA_TRY(cudaGetLastError());
    // the two norms and the bottom rows C x - rhs_bottom, read together
    double* cx = ctx->tmp.as<double>() + 2 * V;
    double* tops = cx + k;
    {
        KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
        row_sums_kernel<<<2, 256, 0, ctx->stream>>>(rr, V, tops);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    if (k > 0) {
        if (large)
            TPE_TRY(large_cx(ctx, *large, d_x, cx));
        else
            TPE_TRY(gram_dots(ctx, d_C, k, d_x, 1, 3 * (int64_t)V, cx));
    }
    std::vector<double> h((size_t)k + 2);
    TPE_TRY(download_on(ctx, ctx->stream, h.data(), cx, sizeof(double) * ((size_t)k + 2)));
    const double top_r = h[(size_t)k], top_b = h[(size_t)k + 1];
    double bot_r = 0.0, bot_b = 0.0;
    for (int32_t r = 0; r < k; r++) {
        const double b = rhs_bottom ? rhs_bottom[r] : 0.0;
        const double d = h[r] - b;
        if (res_bottom) res_bottom[r] = -d;
        bot_r += d * d;
        bot_b += b * b;
    }
    const double rn = sqrt(top_r + bot_r), bn = sqrt(top_b + bot_b);
    *out = rn / (bn > 1.0 ? bn : 1.0);
    return TPE_OK;
}

int32_t dgemm_nt(tpe_ctx* ctx, const DGemmArgs& g, cudaStream_t stream) {
    if (g.M <= 0 || g.N <= 0) return TPE_OK;
    const bool al = ((((uintptr_t)g.A) | ((uintptr_t)g.B)) & 15) == 0 && (g.lda & 1) == 0 &&
                    (g.ldb & 1) == 0;
    auto kern = al ? dgemm_nt_kernel<true> : dgemm_nt_kernel<false>;
    const size_t smem = sizeof(double) * 4 * GT * GP;
    TPE_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    dim3 grid((unsigned)((g.N + GT - 1) / GT), (unsigned)((g.M + GT - 1) / GT));
    kern<<<grid, 256, smem, stream>>>(g);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t transpose_fp64(tpe_ctx* ctx, const double* src, int64_t lds, int32_t m, int32_t c,
                       double* dst, int64_t ldd) {
    KernelScope ks(ctx, TPE_KGROUP_TRSV, 1);
    transpose_fp64_kernel<<<dim3((c + 31) / 32, (m + 31) / 32), dim3(32, 8), 0, ctx->stream>>>(
        src, lds, m, c, dst, ldd);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t mirror_lower(tpe_ctx* ctx, double* M, int32_t n) {
    KernelScope ks(ctx, TPE_KGROUP_TRSV, 1);
    const unsigned nt = (unsigned)((n + 31) / 32);
    mirror_lower_kernel<<<dim3(nt, nt), dim3(32, 8), 0, ctx->stream>>>(M, n);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

}  // namespace tpe
