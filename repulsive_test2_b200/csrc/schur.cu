// Saddle solves with a large constraint set (k rows, e.g. one edge-length row
// per edge: k = E + 3 with the barycenter), on the device.
//
// The reference eliminates the constraints inside one dense factorization of
// the (3V + k)^2 saddle matrix (src/core/sobolev/linsolve.ts:431-589, called
// from src/core/optimizer.ts:231-440). The structured solve replaces it with the
// Schur complement S = C A3^{-1} C^T (A3 = A_rho per coordinate block), which the
// small-k path forms from k x 3 solves and factors on the host. For large k that
// is k^3 host work and 3k solves; here instead:
//   Ainv = A_rho^{-1} explicitly (FP64: factor, L^-T and W W^T in one kernel,
//   chol_dag.cu). An edge-length row is one 3-vector w_s times the difference of two
//   vertices (a pin: times one), so A3^{-1} C^T on those rows is w_s times one column
//   of Gt, Gt[v][s] = Ainv[v][a_s] - Ainv[v][b_s], a third of the size; the other
//   rows (barycenter) go through a multi-RHS product with Ainv. S from differences of
//   Gt's rows; its inverse Sinv on the device makes every multiplier solve one product.
// A solution is x = w - Gt (w_s lam_s) - dense rows - mu term: one product with Gt for
// up to five trial step sizes (15 columns). The multipliers stay on the device: a
// projection iteration reads back only Phi and the norms that decide it.
// Measured per call at V = 2500, k = 2503 against the dense forms (us): the combination
// of eight trials 166 -> 2 x 28, C^T lam 658 -> 6, C x 35 -> 10, Y and S 233 -> Gt and S 43.
// (x = w - Ainv (C^T lam) needs no Gt, but rounds u |Ainv| |C^T lam| where Gt's
// differences round u |Gt| |lam|: 1e5 times more error on a loop network.)
#include <math.h>

#include <algorithm>

#include "tpe_internal.h"

namespace tpe {
namespace {

constexpr int kRhs = 16;      // columns of the right-hand-side-major products (mrhs_part)
constexpr int kPerPass = 5;   // trials (three columns each) per product with Ainv

template <int kWarps>
__device__ __forceinline__ double block_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < kWarps; w++) t += red[w];
    __syncthreads();
    return t;  // on every thread
}

// One pass over the dense rows of C. Row s: its two vertices (or one) and its
// 3-vector when it has that form, else (-1, -1) and dense[s] = 1; and the row's sums
// over each coordinate block and of absolute values.
__global__ void __launch_bounds__(256)
sparse_rows_kernel(const double* __restrict__ C, int32_t V, SparseRows sp, int32_t* __restrict__ dense) {
    const int32_t s = blockIdx.x;
    __shared__ int cnt;
    __shared__ int idx[2];
    __shared__ double val[2][3];
    __shared__ double red[8];
    if (threadIdx.x == 0) cnt = 0;
    __syncthreads();
    const double* row = C + (int64_t)s * 3 * V;
    double sum[4] = {0, 0, 0, 0};
    for (int32_t v = threadIdx.x; v < V; v += 256) {
        const double x = row[v], y = row[V + v], z = row[2 * (int64_t)V + v];
        sum[0] += x;
        sum[1] += y;
        sum[2] += z;
        sum[3] += fabs(x) + fabs(y) + fabs(z);
        if (x != 0.0 || y != 0.0 || z != 0.0) {
            const int q = atomicAdd(&cnt, 1);
            if (q < 2) {
                idx[q] = v;
                val[q][0] = x;
                val[q][1] = y;
                val[q][2] = z;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        sum[q] = block_sum<8>(sum[q], red);
        if (threadIdx.x == 0) sp.stats[4 * (int64_t)s + q] = sum[q];
    }
    if (threadIdx.x != 0) return;
    const int n = cnt;
    // vertex order, so that no sum depends on the race above
    const int f = n == 2 && idx[1] < idx[0] ? 1 : 0;
    bool ok = n == 1 || n == 2;
    if (n == 2)
        for (int d = 0; d < 3; d++) ok = ok && val[1][d] == -val[0][d];
    dense[s] = ok || n == 0 ? 0 : 1;
    sp.ab[s] = ok ? make_int2(idx[f], n == 2 ? idx[1 - f] : -1) : make_int2(-1, -1);
    for (int d = 0; d < 3; d++) sp.w[3 * (int64_t)s + d] = ok ? val[f][d] : 0.0;
}

// The same entries by vertex: off[v] .. off[v + 1] of ent, in row order (counted,
// summed, filled in any order, then placed by rank).
__global__ void col_count_kernel(SparseRows sp, int32_t k, int32_t* __restrict__ count) {
    const int32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= k) return;
    const int2 ab = sp.ab[s];
    if (ab.x >= 0) atomicAdd(&count[ab.x], 1);
    if (ab.y >= 0) atomicAdd(&count[ab.y], 1);
}
__global__ void __launch_bounds__(1024) col_scan_kernel(SparseRows sp, int32_t V, int32_t* __restrict__ count) {
    __shared__ int32_t part[1024];
    const int32_t per = (V + 1023) / 1024, b = min(V, (int32_t)threadIdx.x * per), e = min(V, b + per);
    int32_t s = 0;
    for (int32_t v = b; v < e; v++) s += count[v];
    part[threadIdx.x] = s;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const int32_t t = threadIdx.x >= o ? part[threadIdx.x - o] : 0;
        __syncthreads();
        part[threadIdx.x] += t;
        __syncthreads();
    }
    s = threadIdx.x > 0 ? part[threadIdx.x - 1] : 0;
    for (int32_t v = b; v < e; v++) {
        const int32_t c = count[v];
        sp.off[v] = s;
        count[v] = s;  // the fill's cursor
        s += c;
    }
    if (threadIdx.x == 1023) sp.off[V] = part[1023];
}
__global__ void col_fill_kernel(SparseRows sp, int32_t k, int32_t* __restrict__ cursor,
                                int32_t* __restrict__ raw) {
    const int32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= k) return;
    const int2 ab = sp.ab[s];
    if (ab.x >= 0) raw[atomicAdd(&cursor[ab.x], 1)] = 2 * s;
    if (ab.y >= 0) raw[atomicAdd(&cursor[ab.y], 1)] = 2 * s + 1;
}
__global__ void col_sort_kernel(SparseRows sp, int32_t V, const int32_t* __restrict__ raw) {
    const int32_t v = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (v >= V) return;
    const int32_t b = sp.off[v], e = sp.off[v + 1];
    for (int32_t a = b + lane; a < e; a += 32) {
        const int32_t x = raw[a];
        int32_t rank = 0;
        for (int32_t i = b; i < e; i++) rank += raw[i] < x;
        sp.ent[b + rank] = x;
    }
}

// Gt[v][s] = Ainv[v][a_s] - Ainv[v][b_s] (0 for dense rows). Differences first: they
// are exact where neighbouring columns are close.
__global__ void __launch_bounds__(256)
g_kernel(const double* __restrict__ Ainv, int32_t V, int32_t k, SparseRows sp, double* __restrict__ Gt) {
    const int32_t s = blockIdx.x * 256 + threadIdx.x;
    if (s >= k) return;
    const int2 ab = sp.ab[s];
    for (int32_t v = blockIdx.y; v < V; v += gridDim.y) {
        const double* row = Ainv + (int64_t)v * V;
        const double x = ab.x >= 0 ? row[ab.x] : 0.0;
        Gt[(int64_t)v * k + s] = ab.y >= 0 ? x - row[ab.y] : x;
    }
}

// S[r][s] = (w_r . w_s) (Gt[a_r][s] - Gt[b_r][s]) for sparse rows: 32 x 32 tiles on or
// below the diagonal, mirrored. Dense rows are s_dense_kernel's.
__global__ void __launch_bounds__(256)
s_sparse_kernel(const double* __restrict__ Gt, int32_t k, SparseRows sp, double* __restrict__ S) {
    if (blockIdx.x > blockIdx.y) return;
    __shared__ double t[32][33];
    const int32_t r0 = blockIdx.y * 32, s0 = blockIdx.x * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int32_t s = s0 + tx;
    double ws[3] = {0, 0, 0};
    if (s < k)
        for (int d = 0; d < 3; d++) ws[d] = sp.w[3 * (int64_t)s + d];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int32_t r = r0 + ty + 8 * i;
        double x = 0.0;
        if (r < k && s < k) {
            const int2 ab = sp.ab[r];
            const double* wr = sp.w + 3 * (int64_t)r;
            if (ab.x >= 0) x = Gt[(int64_t)ab.x * k + s];
            if (ab.y >= 0) x -= Gt[(int64_t)ab.y * k + s];
            x *= wr[0] * ws[0] + wr[1] * ws[1] + wr[2] * ws[2];
        }
        t[ty + 8 * i][tx] = x;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int rl = ty + 8 * i;
        const bool dg = r0 == s0;
        if (r0 + rl < k && s < k) S[(int64_t)(r0 + rl) * k + s] = dg && tx > rl ? t[tx][rl] : t[rl][tx];
        if (!dg && s0 + rl < k && r0 + tx < k) S[(int64_t)(s0 + rl) * k + r0 + tx] = t[tx][rl];
    }
}

// Dense row a = list[blockIdx.y] against the sparse rows s: both S entries from Y_a.
__global__ void s_dense_kernel(const double* __restrict__ Y, int32_t V, int32_t k, SparseRows sp,
                               const int32_t* __restrict__ dense, double* __restrict__ S) {
    const int32_t s = blockIdx.x * blockDim.x + threadIdx.x, a = sp.list[blockIdx.y];
    if (s >= k || dense[s]) return;
    const double* y = Y + (int64_t)blockIdx.y * 3 * V;
    const int2 ab = sp.ab[s];
    double acc = 0.0;
    for (int d = 0; d < 3; d++) {
        double x = 0.0;
        if (ab.x >= 0) x = y[(int64_t)d * V + ab.x];
        if (ab.y >= 0) x -= y[(int64_t)d * V + ab.y];
        acc += sp.w[3 * (int64_t)s + d] * x;
    }
    S[(int64_t)a * k + s] = acc;
    S[(int64_t)s * k + a] = acc;
}
// Two dense rows a >= b: (C_a . Y_b + C_b . Y_a) / 2.
__global__ void __launch_bounds__(256)
s_dense_pair_kernel(const double* __restrict__ C, const double* __restrict__ Y, int64_t m, int32_t k,
                    SparseRows sp, double* __restrict__ S) {
    if (blockIdx.y > blockIdx.x) return;
    __shared__ double red[8];
    const int32_t a = sp.list[blockIdx.x], b = sp.list[blockIdx.y];
    double s = 0.0;
    for (int64_t t = threadIdx.x; t < m; t += 256)
        s += C[a * m + t] * Y[blockIdx.y * m + t] + C[b * m + t] * Y[blockIdx.x * m + t];
    s = block_sum<8>(s, red);
    if (threadIdx.x == 0) S[(int64_t)a * k + b] = S[(int64_t)b * k + a] = 0.5 * s;
}

// XT[s][3 q + d] = w_s,d coef_q[s], q < n <= kPerPass; zero rows s >= k.
__global__ void coef_rhs_kernel(SparseRows sp, int32_t k, int32_t rows, const double* __restrict__ coef,
                                int32_t n, double* __restrict__ XT) {
    const int32_t s = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y;
    if (s >= rows || q >= n) return;
    const double l = s < k ? coef[(int64_t)q * (k + 3) + s] : 0.0;
    for (int d = 0; d < 3; d++) XT[(int64_t)s * kRhs + 3 * q + d] = s < k ? sp.w[3 * (int64_t)s + d] * l : 0.0;
}
// out = C^T lam, coordinate blocks: each vertex's sparse entries in row order, then
// the dense rows.
__global__ void ct_block_kernel(const double* __restrict__ C, int32_t V, SparseRows sp,
                                const double* __restrict__ lam, double* __restrict__ out) {
    const int32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= V) return;
    double t[3] = {0, 0, 0};
    for (int32_t e = sp.off[v]; e < sp.off[v + 1]; e++) {
        const int32_t x = sp.ent[e], s = x >> 1;
        const double l = x & 1 ? -lam[s] : lam[s];
        for (int d = 0; d < 3; d++) t[d] += sp.w[3 * (int64_t)s + d] * l;
    }
    for (int32_t a = 0; a < sp.nd; a++) {
        const double* row = C + (int64_t)sp.list[a] * 3 * V;
        const double l = lam[sp.list[a]];
        for (int d = 0; d < 3; d++) t[d] += row[(int64_t)d * V + v] * l;
    }
    for (int d = 0; d < 3; d++) out[(int64_t)d * V + v] = t[d];
}
// out = C x: one thread per sparse row; the first nd blocks take a dense row each.
__global__ void __launch_bounds__(256)
cx_kernel(const double* __restrict__ C, int32_t V, SparseRows sp, const int32_t* __restrict__ dense, int32_t k,
          const double* __restrict__ x, double* __restrict__ out) {
    __shared__ double red[8];
    if ((int32_t)blockIdx.x < sp.nd) {
        const int32_t a = sp.list[blockIdx.x];
        const int64_t m = 3 * (int64_t)V;
        double s = 0.0;
        for (int64_t t = threadIdx.x; t < m; t += 256) s += C[a * m + t] * x[t];
        s = block_sum<8>(s, red);
        if (threadIdx.x == 0) out[a] = s;
        return;
    }
    const int32_t r = (blockIdx.x - sp.nd) * 256 + threadIdx.x;
    if (r >= k || dense[r]) return;
    const int2 ab = sp.ab[r];
    double acc = 0.0;
    for (int d = 0; d < 3; d++) {
        double y = 0.0;
        if (ab.x >= 0) y = x[(int64_t)d * V + ab.x];
        if (ab.y >= 0) y -= x[(int64_t)d * V + ab.y];
        acc += sp.w[3 * (int64_t)r + d] * y;
    }
    out[r] = acc;
}

// XT[j][c] = rc[pos[c]][j] (pos null: c) for j < k, 0 for the rows after it; c < n <= 16.
__global__ void rc_rhs_kernel(const double* __restrict__ rc, int64_t stride, const int32_t* __restrict__ pos,
                              int32_t k, int32_t rows, int32_t n, double* __restrict__ XT) {
    const int32_t j = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (j >= rows || c >= n) return;
    XT[(int64_t)j * kRhs + c] = j < k ? rc[(pos ? pos[c] : c) * stride + j] : 0.0;
}

// One block per multiplier solve c: t = Sinv rc (its chunk sums), the 3 x 3 system
// M mu = Scu^T t - ru through M's Cholesky factor, and the second right-hand side
// rc - Scu mu into XT; mu su to coef[c][k ..]. 1024 threads, four chunks' loads at a
// time: 43 -> 20 us at k = 2503 against 256 threads and one.
__global__ void __launch_bounds__(1024)
mu_kernel(const double* __restrict__ part, int32_t nch, int32_t k, const double* __restrict__ scu,
          const double* __restrict__ mchol, double3 ru, double su, double* __restrict__ XT,
          double* __restrict__ coef) {
    __shared__ double red[32];
    const int c = blockIdx.x;
    double s[3] = {0, 0, 0};
    for (int32_t r = threadIdx.x; r < k; r += 1024) {
        const double* p = part + (int64_t)c * k + r;
        double t = 0.0;
#pragma unroll 4
        for (int32_t ch = 0; ch < nch; ch++) t += p[(int64_t)ch * kRhs * k];
        for (int d = 0; d < 3; d++) s[d] += scu[3 * (int64_t)r + d] * t;
    }
    for (int d = 0; d < 3; d++) s[d] = block_sum<32>(s[d], red);
    const double b[3] = {s[0] - ru.x, s[1] - ru.y, s[2] - ru.z};
    double y[3], mu[3];
    for (int i = 0; i < 3; i++) {
        double v = b[i];
        for (int q = 0; q < i; q++) v -= mchol[3 * i + q] * y[q];
        y[i] = v / mchol[4 * i];
    }
    for (int i = 2; i >= 0; i--) {
        double v = y[i];
        for (int q = i + 1; q < 3; q++) v -= mchol[3 * q + i] * mu[q];
        mu[i] = v / mchol[4 * i];
    }
    for (int32_t r = threadIdx.x; r < k; r += 1024) {
        double v = XT[(int64_t)r * kRhs + c];
        for (int d = 0; d < 3; d++) v -= scu[3 * (int64_t)r + d] * mu[d];
        XT[(int64_t)r * kRhs + c] = v;
    }
    if (threadIdx.x < 3) coef[(int64_t)c * (k + 3) + k + threadIdx.x] = mu[threadIdx.x] * su;
}
// coef[c][r] = the chunk sums; zero_mu: coef[c][k ..] = 0 as well.
__global__ void lam_kernel(const double* __restrict__ part, int32_t nch, int32_t k, int zero_mu,
                           double* __restrict__ coef) {
    const int32_t r = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (r < k) {
        double t = 0.0;
#pragma unroll 4
        for (int32_t ch = 0; ch < nch; ch++) t += part[((int64_t)ch * kRhs + c) * k + r];
        coef[(int64_t)c * (k + 3) + r] = t;
    } else if (r < k + 3 && zero_mu) {
        coef[(int64_t)c * (k + 3) + r] = 0.0;
    }
}

// x = w - A3^{-1} C^T coef - mu term at (d, v): the chunk sums of column c (the sparse
// rows), then the dense rows in order.
__device__ __forceinline__ double solution_at(const double* __restrict__ part, int32_t nch, int32_t V, int c,
                                              const double* __restrict__ Y, const SparseRows& sp,
                                              const double* __restrict__ coef, int32_t k, int d, int32_t v,
                                              double w) {
    double s = 0.0;
    for (int32_t ch = 0; ch < nch; ch++) s += part[((int64_t)ch * kRhs + c) * V + v];
    for (int32_t a = 0; a < sp.nd; a++) s += Y[((int64_t)a * 3 + d) * V + v] * coef[sp.list[a]];
    return (w - s) - coef[k + d];
}
__global__ void solution_kernel(const double* __restrict__ part, int32_t nch, int32_t V,
                                const double* __restrict__ Y, SparseRows sp, const double* __restrict__ w,
                                const double* __restrict__ coef, int32_t k, double* __restrict__ x) {
    const int32_t v = blockIdx.x * blockDim.x + threadIdx.x, d = blockIdx.y;
    if (v >= V) return;
    const int64_t t = (int64_t)d * V + v;
    x[t] = solution_at(part, nch, V, d, Y, sp, coef, k, d, v, w ? w[t] : 0.0);
}
// cur[idx[q]] (interleaved, rows stride apart) += the solution of coef_q, w = 0.
__global__ void update_kernel(const double* __restrict__ part, int32_t nch, int32_t V,
                              const double* __restrict__ Y, SparseRows sp, const double* __restrict__ coef,
                              int32_t k, const int32_t* __restrict__ idx, double* __restrict__ cur,
                              int64_t stride, int32_t* __restrict__ bad) {
    const int32_t v = blockIdx.x * blockDim.x + threadIdx.x, q = blockIdx.y / 3, d = blockIdx.y % 3;
    if (v >= V) return;
    const int a = idx[q];
    const double x = solution_at(part, nch, V, 3 * q + d, Y, sp, coef + (int64_t)q * (k + 3), k, d, v, 0.0);
    if (!isfinite(x)) bad[a] = 1;
    double* p = cur + (int64_t)a * stride + 3 * (int64_t)v + d;
    *p = *p + x;
}

inline unsigned blocks(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }
inline int32_t rows16(int32_t n) { return (n + 15) / 16 * 16; }

}  // namespace

int32_t large_schur_build(tpe_ctx* ctx, SaddleOp& op, const double* b_flat, bool* singular) {
    const int32_t V = op.V, k = op.k;
    const cudaStream_t st = ctx->stream;
    *singular = false;
    const int32_t nmax = std::max(V, k);
    const size_t nn = (size_t)nmax * nmax;
    const size_t half = (size_t)(nmax / 2 + kNB) * (nmax / 2 + kNB);
    TPE_TRY(ensure(ctx, ctx->mat_Ainv, sizeof(double) * (size_t)V * V));
    TPE_TRY(ensure(ctx, ctx->inv_W, sizeof(double) * nn));
    if (op.int8) {
        TPE_TRY(ensure(ctx, ctx->inv_X, sizeof(double) * nn));
        TPE_TRY(ensure(ctx, ctx->inv_T, sizeof(double) * half));
    }
    double* Ainv = ctx->mat_Ainv.as<double>();
    // op.L holds A_rho unfactored; it is overwritten
    if (op.int8) {
        bool sing = false;
        TPE_TRY(spd_inverse_int8(ctx, op.L, V, op.chol_tol, ctx->inv_X.as<double>(),
                                 ctx->inv_W.as<double>(), ctx->inv_T.as<double>(), Ainv, &sing));
        if (sing) {
            *singular = true;
            return TPE_OK;
        }
    } else {
        CholDag f;  // factor, L^-T and inverse in one kernel
        f.L = op.L;
        f.Linv = op.Linv;
        f.n = V;
        f.tol = op.chol_tol;
        f.W = ctx->inv_W.as<double>();
        f.Ainv = Ainv;
        int32_t bad = 0;
        TPE_TRY(chol_dag(ctx, f, &bad));
        if (bad) {
            *singular = true;
            return TPE_OK;
        }
    }
    op.Ainv = Ainv;
    // sparse structure of C, by row and by vertex
    const int64_t m = 3 * (int64_t)V;
    const size_t kk = (size_t)k;
    TPE_TRY(ensure(ctx, ctx->sch_nz, sizeof(double) * 7 * kk + sizeof(int32_t) * (8 * kk + 2 * (size_t)V + 1)));
    SparseRows& sp = op.sp;
    sp.w = ctx->sch_nz.as<double>();
    sp.stats = sp.w + 3 * kk;
    sp.ab = reinterpret_cast<int2*>(sp.stats + 4 * kk);
    sp.ent = reinterpret_cast<int32_t*>(sp.ab + kk);
    int32_t* raw = sp.ent + 2 * kk;
    int32_t* dense = raw + 2 * kk;
    sp.list = dense + kk;
    sp.off = sp.list + kk;
    int32_t* count = sp.off + V + 1;
    sp.nd = 0;
    TPE_CUDA_TRY(cudaMemsetAsync(count, 0, sizeof(int32_t) * (size_t)V, st));
    {
        KernelScope ks(ctx, TPE_KGROUP_OTHER, 5);
        sparse_rows_kernel<<<k, 256, 0, st>>>(op.C, V, sp, dense);
        col_count_kernel<<<blocks(k, 256), 256, 0, st>>>(sp, k, count);
        col_scan_kernel<<<1, 1024, 0, st>>>(sp, V, count);
        col_fill_kernel<<<blocks(k, 256), 256, 0, st>>>(sp, k, count, raw);
        col_sort_kernel<<<blocks(V, 8), 256, 0, st>>>(sp, V, raw);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    std::vector<int32_t> hdense(kk), drows;
    TPE_TRY(download_on(ctx, st, hdense.data(), dense, sizeof(int32_t) * kk));
    for (int32_t s = 0; s < k; s++)
        if (hdense[s]) drows.push_back(s);
    sp.nd = (int32_t)drows.size();
    sp.dense = dense;
    if (sp.nd > 0)
        TPE_CUDA_TRY(cudaMemcpyAsync(sp.list, drows.data(), sizeof(int32_t) * drows.size(),
                                     cudaMemcpyHostToDevice, st));
    // dense rows: Y_a = Ainv C_s per coordinate block, runs of up to five rows per product
    TPE_TRY(ensure(ctx, ctx->con_Y, sizeof(double) * ((size_t)sp.nd + 1) * m));
    op.Y = ctx->con_Y.as<double>();
    for (size_t a = 0; a < drows.size();) {
        size_t b = a + 1;
        while (b < drows.size() && b - a < (size_t)kPerPass && drows[b] == drows[b - 1] + 1) b++;
        TPE_TRY(mrhs_fp64(ctx, Ainv, V, op.C + (int64_t)drows[a] * m, V, 3 * (int32_t)(b - a), op.Y + a * m));
        a = b;
    }
    // the gradient right-hand side: w = A3^{-1} b
    if (b_flat) {
        TPE_TRY(finish_gradient(ctx));
        op.W = op.Y + (size_t)sp.nd * m;
        op.w_src = b_flat;
        TPE_TRY(mrhs_fp64(ctx, Ainv, V, b_flat, V, 3, op.W));
    }
    // S = C A3^{-1} C^T (k x k)
    TPE_TRY(ensure(ctx, ctx->sch_G, sizeof(double) * kk * V));
    TPE_TRY(ensure(ctx, ctx->sch_S, sizeof(double) * kk * k));
    TPE_TRY(ensure(ctx, ctx->sch_Linv, sizeof(double) * (size_t)((k + kNB - 1) / kNB) * kNB * kNB));
    TPE_TRY(ensure(ctx, ctx->sch_Sinv, sizeof(double) * kk * k));
    TPE_TRY(ensure(ctx, ctx->sch_vec, sizeof(double) * (2 * kRhs * (size_t)rows16(k) + kRhs * (kk + 3) + 3 * kk + 16)));
    double* S = ctx->sch_S.as<double>();
    op.Gt = ctx->sch_G.as<double>();
    {
        KernelScope ks(ctx, TPE_KGROUP_OTHER, sp.nd > 0 ? 4 : 2);
        const unsigned tk = blocks(k, 32);
        g_kernel<<<dim3(blocks(k, 256), (unsigned)std::min(V, 4096)), 256, 0, st>>>(Ainv, V, k, sp, op.Gt);
        s_sparse_kernel<<<dim3(tk, tk), dim3(32, 8), 0, st>>>(op.Gt, k, sp, S);
        if (sp.nd > 0) {
            s_dense_kernel<<<dim3(blocks(k, 256), (unsigned)sp.nd), 256, 0, st>>>(op.Y, V, k, sp, dense, S);
            s_dense_pair_kernel<<<dim3((unsigned)sp.nd, (unsigned)sp.nd), 256, 0, st>>>(op.C, op.Y, m, k, sp, S);
        }
        TPE_CUDA_TRY(cudaGetLastError());
    }
    double* Ls = S;  // S itself is not needed again
    if (op.int8) {
        bool sing = false;
        TPE_TRY(spd_inverse_int8(ctx, Ls, k, 0.0, ctx->inv_X.as<double>(), ctx->inv_W.as<double>(),
                                 ctx->inv_T.as<double>(), ctx->sch_Sinv.as<double>(), &sing));
        if (sing) {
            *singular = true;
            return TPE_OK;
        }
    } else {
        CholDag f;
        f.L = Ls;
        f.Linv = ctx->sch_Linv.as<double>();
        f.n = k;
        f.tol = 0.0;
        f.W = ctx->inv_W.as<double>();
        f.Ainv = ctx->sch_Sinv.as<double>();
        int32_t bad = 0;
        TPE_TRY(chol_dag(ctx, f, &bad));
        if (bad) {
            *singular = true;
            return TPE_OK;
        }
    }
    op.Sinv = ctx->sch_Sinv.as<double>();
    return TPE_OK;
}

// sch_vec: XT (two of them), coefficients of up to 16 solves, Scu and M's factor.
namespace {
double* vec_xt(tpe_ctx* ctx) { return ctx->sch_vec.as<double>(); }
double* vec_coef(tpe_ctx* ctx, const SaddleOp& op) {
    return vec_xt(ctx) + 2 * (size_t)kRhs * rows16(op.k);
}
double* vec_scu(tpe_ctx* ctx, const SaddleOp& op) { return vec_coef(ctx, op) + kRhs * ((size_t)op.k + 3); }
}  // namespace

int32_t large_set_mu(tpe_ctx* ctx, const SaddleOp& op, const double* h_scu, const double* h_mchol) {
    double* d = vec_scu(ctx, op);
    TPE_CUDA_TRY(cudaMemcpyAsync(d, h_scu, sizeof(double) * 3 * (size_t)op.k, cudaMemcpyHostToDevice, ctx->stream));
    TPE_CUDA_TRY(cudaMemcpyAsync(d + 3 * (size_t)op.k, h_mchol, sizeof(double) * 9, cudaMemcpyHostToDevice, ctx->stream));
    return TPE_OK;
}

int32_t large_sinv(tpe_ctx* ctx, const SaddleOp& op, const double* h_rc, int32_t nr, double* h_out) {
    const int32_t k = op.k;
    double* din = vec_xt(ctx);  // rows of k, then the products' rows
    double* dout = din + (size_t)kRhs * rows16(k);
    TPE_CUDA_TRY(cudaMemcpyAsync(din, h_rc, sizeof(double) * (size_t)nr * k, cudaMemcpyHostToDevice, ctx->stream));
    TPE_TRY(mrhs_fp64(ctx, op.Sinv, k, din, k, nr, dout));
    return download_on(ctx, ctx->stream, h_out, dout, sizeof(double) * (size_t)nr * k);
}

int32_t large_multipliers(tpe_ctx* ctx, const SaddleOp& op, const double* d_rc, int64_t stride,
                          const int32_t* d_pos, int32_t n, const double ru[3], double** d_coef) {
    const int32_t k = op.k;
    const cudaStream_t st = ctx->stream;
    double *XT = vec_xt(ctx), *coef = vec_coef(ctx, op), *scu = vec_scu(ctx, op);
    *d_coef = coef;
    {
        KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
        rc_rhs_kernel<<<dim3(blocks(rows16(k), 256), (unsigned)n), 256, 0, st>>>(d_rc, stride, d_pos, k, rows16(k),
                                                                             n, XT);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    const double* part = nullptr;
    int32_t nch = 0;
    TPE_TRY(mrhs_part(ctx, op.Sinv, k, k, XT, &part, &nch));
    if (op.trans_constrained) {
        {
            KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
            mu_kernel<<<(unsigned)n, 1024, 0, st>>>(part, nch, k, scu, scu + 3 * (size_t)k,
                                                   make_double3(ru[0], ru[1], ru[2]),
                                                   1.0 / (op.rho * sqrt((double)op.V)), XT, coef);
            TPE_CUDA_TRY(cudaGetLastError());
        }
        TPE_TRY(mrhs_part(ctx, op.Sinv, k, k, XT, &part, &nch));
    }
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    lam_kernel<<<dim3(blocks(k + 3, 256), (unsigned)n), 256, 0, st>>>(part, nch, k, op.trans_constrained ? 0 : 1, coef);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t large_solution(tpe_ctx* ctx, const SaddleOp& op, const double* d_coef, const double* d_w, double* d_x) {
    const int32_t V = op.V, k = op.k;
    double* XT = vec_xt(ctx);
    {
        KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
        coef_rhs_kernel<<<dim3(blocks(rows16(k), 256), 1), 256, 0, ctx->stream>>>(op.sp, k, rows16(k), d_coef, 1, XT);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    const double* part = nullptr;
    int32_t nch = 0;
    TPE_TRY(mrhs_part(ctx, op.Gt, V, k, XT, &part, &nch));
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    solution_kernel<<<dim3(blocks(V, 128), 3), 128, 0, ctx->stream>>>(part, nch, V, op.Y, op.sp, d_w, d_coef, k, d_x);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t large_update(tpe_ctx* ctx, const SaddleOp& op, const double* d_coef, int32_t nu, const int32_t* d_idx,
                     double* d_cur, int64_t stride, int32_t* d_bad) {
    const int32_t V = op.V, k = op.k;
    double* XT = vec_xt(ctx);
    for (int32_t q0 = 0; q0 < nu; q0 += kPerPass) {
        const int32_t n = std::min(nu - q0, kPerPass);
        const double* coef = d_coef + (size_t)q0 * (k + 3);
        {
            KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
            coef_rhs_kernel<<<dim3(blocks(rows16(k), 256), (unsigned)n), 256, 0, ctx->stream>>>(op.sp, k, rows16(k),
                                                                                           coef, n, XT);
            TPE_CUDA_TRY(cudaGetLastError());
        }
        const double* part = nullptr;
        int32_t nch = 0;
        TPE_TRY(mrhs_part(ctx, op.Gt, V, k, XT, &part, &nch));
        KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
        update_kernel<<<dim3(blocks(V, 128), 3 * (unsigned)n), 128, 0, ctx->stream>>>(
            part, nch, V, op.Y, op.sp, coef, k, d_idx + q0, d_cur, stride, d_bad);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    return TPE_OK;
}

int32_t large_ct(tpe_ctx* ctx, const SaddleOp& op, const double* d_lam, double* d_out) {
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    ct_block_kernel<<<blocks(op.V, 128), 128, 0, ctx->stream>>>(op.C, op.V, op.sp, d_lam, d_out);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t large_cx(tpe_ctx* ctx, const SaddleOp& op, const double* d_x, double* d_out) {
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    cx_kernel<<<op.sp.nd + blocks(op.k, 256), 256, 0, ctx->stream>>>(op.C, op.V, op.sp, op.sp.dense, op.k, d_x, d_out);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

}  // namespace tpe
