// Fractional-Sobolev Gram assembly, FP64: A = B + B0 (V x V).
//
// Reference: assembleBHighFlat / assembleBLowFlat / assembleAFlat in
// src/core/sobolev/innerProduct.ts:38-350. The reference scatters 16
// increments per ordered pair into V x V; here the same sum is written in
// matrix form and evaluated as two gathers, with no atomics:
//
//   B  = S (diag(d) - Mb) S^T,   S column I = e_{i1} - e_{i2}
//   B0 = U (diag(d0) - M0) U^T,  U column I = e_{i1} + e_{i2}
//
// with, for disjoint I != J (w_IJ = w_JI = 1/4 l_I l_J sum 1/(|d|+eps)^(2s+1),
// q_IJ = 1/4 * 1/4 l_I l_J sum (|T_I x d|+eps)^2/(|d|+eps)^4/(|d|+eps)^(2s+1)):
//   Mb[I][J] = (w_IJ + w_JI) (T_I . T_J) / (l_I l_J),   d_I  = sum_J (w_IJ + w_JI) / l_I^2
//   M0[I][J] = q_IJ + q_JI,                             d0_I = sum_J (q_IJ + q_JI)
// Kernel 1 writes the E x E pair matrix (Mb', M0') with the diagonal sums on
// its diagonal and minus signs folded in; kernel 2 forms each A[v][u] from the
// incident edges of v and u (4 entries for a closed polyline) and writes A and
// its mirror, so A is exactly symmetric as after the reference's explicit
// symmetrisation.
#include <math.h>

#include "pair_math.cuh"
#include "tpe_internal.h"

namespace tpe {
namespace {


// (|d|+eps)^(-(2 sigma + 1)) from dn = |d|+eps and its reciprocal idn;
// MODE 1: alpha = 3, beta = 6 -> exponent 7/3.
template <int MODE>
__device__ __forceinline__ double inv_dist_pow(double dn, double idn, double distExp) {
    if (MODE == 1) return inv_cbrt(dn) * (idn * idn);
    return 1.0 / pow(dn, distExp);
}

// Of one endpoint pair at squared distance x: kd = (|d|+eps)^(-(2 sigma + 1)) and
// kq = kd (|d|+eps)^-4.
template <int MODE>
__device__ __forceinline__ void dist_weights(double x, double distExp, double eps, double& kd, double& kq) {
    double s, inv, idn;
    dist_terms(x, eps, s, inv, idn);
    kd = inv_dist_pow<MODE>(s + eps, idn, distExp);
    const double i2 = idn * idn;
    kq = kd * (i2 * i2);
}

// (|T x d| + eps)^2 for the two ends d1, d2 of an edge with tangent T seen from one
// point (T x d is the same for both: the nearer one loses the least).
__device__ __forceinline__ double area_sq(double Tx, double Ty, double Tz, double dx, double dy, double dz,
                                          double eps) {
    const double cx = Ty * dz - Tz * dy, cy = Tz * dx - Tx * dz, cz = Tx * dy - Ty * dx;
    const double c2 = cx * cx + cy * cy + cz * cz;
    const double cn = (c2 > 1e-300 && c2 < 1e300 ? c2 * rsqrt_normal(c2) : sqrt(c2)) + eps;
    return cn * cn;
}

constexpr int kT = 32;  // pair tile: 32 edges I x 32 edges J

struct EdgeRec {
    double4 p1;  // endpoint 1, l^eps
    double4 p2;  // endpoint 2
    double4 T;   // unit tangent (0 below 1e-14), raw length
    int2 ij;
};

__device__ __forceinline__ void load_edge(const double4* __restrict__ ea,
                                          const double4* __restrict__ eb,
                                          const int2* __restrict__ edges, int32_t E, int32_t I,
                                          EdgeRec& r) {
    if (I >= E) {
        r.p1 = make_double4(0, 0, 0, 1);
        r.p2 = make_double4(0, 0, 0, 1);
        r.T = make_double4(0, 0, 0, 0);
        r.ij = make_int2(-1, -1);
        return;
    }
    r.p1 = ea[I];
    r.p2 = eb[I];
    r.ij = edges[I];
    const double ex = r.p2.x - r.p1.x, ey = r.p2.y - r.p1.y, ez = r.p2.z - r.p1.z;
    const double len = sqrt(ex * ex + ey * ey + ez * ez);
    if (len < 1e-14) {
        r.T = make_double4(0, 0, 0, len);
    } else {
        const double inv = 1.0 / len;
        r.T = make_double4(ex * inv, ey * inv, ez * inv, len);
    }
}

// Symmetric pair weights of one unordered pair: (w_IJ + w_JI, q_IJ + q_JI). Four
// distances and four areas (an edge against a point: the same area for its two ends).
template <int MODE>
__device__ __forceinline__ double2 pair_weight(const EdgeRec& a, const EdgeRec& b, double distExp,
                                               double eps) {
    double d[2][2][3], x[2][2], kq[2][2], sumDist = 0.0;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            d[i][j][0] = (i ? a.p2.x : a.p1.x) - (j ? b.p2.x : b.p1.x);
            d[i][j][1] = (i ? a.p2.y : a.p1.y) - (j ? b.p2.y : b.p1.y);
            d[i][j][2] = (i ? a.p2.z : a.p1.z) - (j ? b.p2.z : b.p1.z);
            x[i][j] = d[i][j][0] * d[i][j][0] + d[i][j][1] * d[i][j][1] + d[i][j][2] * d[i][j][2];
            double kd;
            dist_weights<MODE>(x[i][j], distExp, eps, kd, kq[i][j]);
            sumDist += kd;
        }
    double low = 0.0;
#pragma unroll
    for (int j = 0; j < 2; j++) {  // edge a against point j of b
        const int n = x[0][j] <= x[1][j] ? 0 : 1;
        low += area_sq(a.T.x, a.T.y, a.T.z, n ? d[1][j][0] : d[0][j][0], n ? d[1][j][1] : d[0][j][1],
                       n ? d[1][j][2] : d[0][j][2], eps) * (kq[0][j] + kq[1][j]);
    }
#pragma unroll
    for (int i = 0; i < 2; i++) {  // edge b against point i of a
        const int n = x[i][0] <= x[i][1] ? 0 : 1;
        low += area_sq(b.T.x, b.T.y, b.T.z, n ? d[i][1][0] : d[i][0][0], n ? d[i][1][1] : d[i][0][1],
                       n ? d[i][1][2] : d[i][0][2], eps) * (kq[i][0] + kq[i][1]);
    }
    const double ll = a.p1.w * b.p1.w;
    return make_double2(0.5 * ll * sumDist, 0.0625 * ll * low);
}

// One block per upper-triangular 32x32 tile (it <= jt) of the E x E pair
// matrix; 256 threads = 32 J lanes x 8 row groups of 4 I rows. Writes
// M[I][J] = (-(w_IJ+w_JI) T_I.T_J / (l_I l_J), -(q_IJ+q_JI)) coalesced along J,
// and its mirror M[J][I] through a shared-memory transpose. Row sums of the
// weights go to rowpart[slot][row] (slot = the other tile index), each slot
// written once, for the diagonal pass.
template <int MODE>
__global__ void __launch_bounds__(256)
pair_weights_kernel(const double4* __restrict__ ea, const double4* __restrict__ eb,
                    const int2* __restrict__ edges, int32_t E, double distExp, double eps,
                    double2* __restrict__ M, double2* __restrict__ rowpart) {
    __shared__ EdgeRec sI[kT], sJ[kT];
    __shared__ double2 tile[kT][kT + 1];
    __shared__ double2 colred[8][kT];
    const int64_t t = blockIdx.x;
    int32_t it = (int32_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((int64_t)it * (it + 1) / 2 > t) it--;
    while ((int64_t)(it + 1) * (it + 2) / 2 <= t) it++;
    const int32_t jt_rel = (int32_t)(t - (int64_t)it * (it + 1) / 2);
    // map the lower-triangle enumeration (it >= jt_rel) to the upper tile (row jt_rel, col it)
    const int32_t ti = jt_rel, tj = it;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (threadIdx.x < kT) load_edge(ea, eb, edges, E, ti * kT + threadIdx.x, sI[threadIdx.x]);
    else if (threadIdx.x < 2 * kT)
        load_edge(ea, eb, edges, E, tj * kT + threadIdx.x - kT, sJ[threadIdx.x - kT]);
    __syncthreads();
    const int32_t J = tj * kT + tx;
    const EdgeRec& b = sJ[tx];
    double2 colsum = make_double2(0.0, 0.0);
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int li = ty + 8 * r;
        const int32_t I = ti * kT + li;
        const EdgeRec& a = sI[li];
        double2 out = make_double2(0.0, 0.0);
        double2 w = make_double2(0.0, 0.0);
        const bool ok = I < E && J < E && I != J && a.ij.x != b.ij.x && a.ij.x != b.ij.y &&
                        a.ij.y != b.ij.x && a.ij.y != b.ij.y;
        if (ok) {
            w = pair_weight<MODE>(a, b, distExp, eps);
            const double dotT = a.T.x * b.T.x + a.T.y * b.T.y + a.T.z * b.T.z;
            out = make_double2(-w.x * dotT / (a.p1.w * b.p1.w), -w.y);
        }
        if (I < E && J < E) M[(int64_t)I * E + J] = out;
        tile[li][tx] = out;
        colsum.x += w.x;
        colsum.y += w.y;
        // row sum over this tile's J (warp = one row group)
        double2 rs = w;
        for (int o = 16; o > 0; o >>= 1) {
            rs.x += __shfl_down_sync(0xffffffffu, rs.x, o);
            rs.y += __shfl_down_sync(0xffffffffu, rs.y, o);
        }
        if (tx == 0 && I < E) rowpart[(int64_t)tj * E + I] = rs;
    }
    if (ti == tj) return;  // diagonal tile: every (I, J) was computed directly
    colred[ty][tx] = colsum;
    __syncthreads();
    // mirror: M[J][I] for I in tile ti, written along I
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int lj = ty + 8 * r;
        const int32_t Jr = tj * kT + lj;
        const int32_t Ic = ti * kT + tx;
        if (Jr < E && Ic < E) M[(int64_t)Jr * E + Ic] = tile[tx][lj];
    }
    if (ty == 0 && J < E) {
        double2 s = colred[0][tx];
        for (int g = 1; g < 8; g++) {
            s.x += colred[g][tx].x;
            s.y += colred[g][tx].y;
        }
        rowpart[(int64_t)ti * E + J] = s;
    }
}

// Diagonal of the pair matrix: (d_I, d0_I) from the per-tile row sums.
__global__ void pair_diag_kernel(const double4* __restrict__ ea, int32_t E, int32_t nt,
                                 const double2* __restrict__ rowpart, double2* __restrict__ M) {
    const int32_t I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= E) return;
    double sx = 0.0, sy = 0.0;
    for (int32_t s = 0; s < nt; s++) {
        const double2 p = rowpart[(int64_t)s * E + I];
        sx += p.x;
        sy += p.y;
    }
    const double ell = ea[I].w;
    M[(int64_t)I * E + I] = make_double2(sx / (ell * ell), sy);
}

// A[v][u] = sum_{(I,a) in inc(v)} sum_{(J,b) in inc(u)} (s_a s_b Mb'[I][J] + M0'[I][J]),
// s_0 = +1 (v is the edge's first vertex), s_1 = -1. Lower-triangle tiles only;
// each entry is written with its mirror.
__global__ void __launch_bounds__(1024, 2)
gather_A_kernel(const double2* __restrict__ M, int32_t E, const int32_t* __restrict__ inc_off,
                const int32_t* __restrict__ inc, int32_t V, int32_t tiles, double* __restrict__ A,
                double* __restrict__ B, double* __restrict__ B0) {
    // blockIdx.x enumerates lower-triangular 32x32 tiles (ti >= tj); the tile is
    // written along rows, and its mirror (tj, ti) through a shared-memory
    // transpose, so both stores are coalesced.
    __shared__ double ta[32][33], tb[32][33], t0[32][33];
    // the incidence lists of the tile's 32 rows and 32 columns, staged once
    // (vertices of degree <= kDeg; a tile with a larger degree reads them from
    // global memory as it goes)
    constexpr int kDeg = 4;
    __shared__ int32_t inc_r[32][kDeg], inc_c[32][kDeg];
    __shared__ int32_t deg_r[32], deg_c[32];
    __shared__ int big;
    const int32_t t = blockIdx.x;
    int32_t ti = (int32_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((int64_t)ti * (ti + 1) / 2 > t) ti--;
    while ((int64_t)(ti + 1) * (ti + 2) / 2 <= t) ti++;
    const int32_t tj = t - ti * (ti + 1) / 2;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int32_t v = ti * 32 + ty;
    const int32_t u = tj * 32 + tx;
    (void)tiles;
    const bool ok = v < V && u < V && u <= v;
    const int tid = ty * 32 + tx;
    if (tid == 0) big = 0;
    __syncthreads();
    if (tid < 64) {
        const int k = tid & 31;
        const bool isrow = tid < 32;
        const int32_t w = (isrow ? ti : tj) * 32 + k;
        int32_t n = 0;
        if (w < V) {
            const int32_t b = inc_off[w];
            n = inc_off[w + 1] - b;
            if (n > kDeg) big = 1;
            for (int q = 0; q < n && q < kDeg; q++) (isrow ? inc_r : inc_c)[k][q] = inc[b + q];
        }
        (isrow ? deg_r : deg_c)[k] = n;
    }
    __syncthreads();
    double sb = 0.0, s0 = 0.0;
    if (ok && !big) {
        // same sums, same order as below
        for (int p = 0; p < deg_r[ty]; p++) {
            const int32_t ip = inc_r[ty][p];
            const int32_t I = ip >> 1;
            const double sa = (ip & 1) ? -1.0 : 1.0;
            const double2* row = M + (int64_t)I * E;
            for (int q = 0; q < deg_c[tx]; q++) {
                const int32_t iq = inc_c[tx][q];
                const int32_t J = iq >> 1;
                const double sgn = (iq & 1) ? -sa : sa;
                const double2 m = row[J];
                sb += sgn * m.x;
                s0 += m.y;
            }
        }
    } else if (ok) {
        for (int32_t p = inc_off[v]; p < inc_off[v + 1]; p++) {
            const int32_t I = inc[p] >> 1;
            const double sa = (inc[p] & 1) ? -1.0 : 1.0;
            const double2* row = M + (int64_t)I * E;
            for (int32_t q = inc_off[u]; q < inc_off[u + 1]; q++) {
                const int32_t J = inc[q] >> 1;
                const double sgn = (inc[q] & 1) ? -sa : sa;
                const double2 m = row[J];
                sb += sgn * m.x;
                s0 += m.y;
            }
        }
    }
    ta[ty][tx] = sb + s0;
    tb[ty][tx] = sb;
    t0[ty][tx] = s0;
    __syncthreads();
    if (ok) {
        A[(int64_t)v * V + u] = ta[ty][tx];
        if (B) B[(int64_t)v * V + u] = tb[ty][tx];
        if (B0) B0[(int64_t)v * V + u] = t0[ty][tx];
    }
    // mirror: entry (row tj*32 + ty, column ti*32 + tx) = value (ti*32 + tx, tj*32 + ty)
    const int32_t mr = tj * 32 + ty, mc = ti * 32 + tx;
    if (mc < V && mr < V && mr < mc) {
        A[(int64_t)mr * V + mc] = ta[tx][ty];
        if (B) B[(int64_t)mr * V + mc] = tb[tx][ty];
        if (B0) B0[(int64_t)mr * V + mc] = t0[tx][ty];
    }
}

// ---- closed single loop: A straight from the pair weights -------------------
//
// When the curve is one closed loop with edge I = (I, I+1 mod V) (E = V), vertex
// v is the second vertex of edge v-1 and the first of edge v, so
//   A[v][u] = sum_{I in {v-1, v}} sum_{J in {u-1, u}} s_vI s_uJ Mb'[I][J] + M0'[I][J]
// (s = +1 for the first vertex, -1 for the second): a 2 x 2 stencil on the pair
// matrix. A warp takes kStrip columns u of A and marches down R rows v: lane j holds
// vertex u0 - 1 + j and the edge that begins there. Each row's vertex is taken once
// against the 32 lane vertices (one distance), the lane's edge against the row's
// vertex and the row's edge against the lane's vertex (one area each: an area is the
// same from both ends of the edge); the four distances and areas of an edge pair, and
// the stencil, are then sums with the neighbour lane (shuffles) and the row before
// (registers): 1 distance and 2 areas per pair where a pair on its own has 4 and 8.
// A's lower tile is written along rows, its mirror through shared memory 16 rows at a
// time; nothing of size E^2 is stored. The pair matrix's diagonal (the row sums of the
// weights over I > J, by rows and by columns) is added to A's cyclic band afterwards
// (loop_band_kernel).
//
// Bound: FP64 pipe and its latency, about 100 FP64 operations per unordered pair.
// Measured at V = 8192: 1290 us with each pair on its own; 984 with tables of distances
// and areas in shared memory (issue-bound: 690 instructions per pair); 525 in this form
// (350 instructions, FP64 pipe 44 %). The band 103 -> 20.
constexpr int kStrip = 30;   // columns per warp: 32 vertices, 31 edges
constexpr int kBatch = 16;   // rows per mirror write
constexpr int kLoopWarps = 4;

struct LoopSmem {
    double a[kBatch][33];          // A's rows
    double w[kBatch][33], q[kBatch][33];  // the weights of own pairs I > J
    double row[kBatch][8];         // the batch's vertices, tangents and l^eps
};

template <int MODE>
__global__ void __launch_bounds__(32 * kLoopWarps)
assemble_loop_kernel(const double4* __restrict__ ea, int32_t V, int32_t R, double distExp, double eps,
                     double* __restrict__ A, double2* __restrict__ rowslot, double2* __restrict__ colslot) {
    extern __shared__ __align__(16) unsigned char loop_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    LoopSmem& sm = reinterpret_cast<LoopSmem*>(loop_smem)[warp];
    const int32_t rb = blockIdx.y, cs = blockIdx.x * kLoopWarps + warp;
    const int32_t v0 = rb * R, u0 = cs * kStrip;
    if (u0 >= V || u0 >= v0 + R) return;  // (no block-wide barrier below)
    auto wrap = [&](int32_t v) -> int32_t { return v < 0 ? v + V : (v >= V ? 0 : v); };
    // edge I begins at vertex I: ea[I] = (vertex I, l^eps of edge I)
    const int32_t J = u0 - 1 + lane;  // this lane's vertex and edge (-1: the last)
    const double4 me = ea[wrap(J)];
    const bool lvalid = J < V && lane < 31;
    const double nx = __shfl_down_sync(0xffffffffu, me.x, 1), ny = __shfl_down_sync(0xffffffffu, me.y, 1),
                 nz = __shfl_down_sync(0xffffffffu, me.z, 1);
    double tx = nx - me.x, ty = ny - me.y, tz = nz - me.z;
    {
        const double len = sqrt(tx * tx + ty * ty + tz * tz);
        const double inv = len < 1e-14 ? 0.0 : 1.0 / len;
        tx *= inv;
        ty *= inv;
        tz *= inv;
    }
    const int32_t Jw = wrap(J);
    const bool own = lane >= 1 && lane <= kStrip && J < V;  // J among the strip's own columns
    double csw = 0.0, csq = 0.0;
    // the row vertex before, against this lane
    double pdx = 0, pdy = 0, pdz = 0, px2 = 1.0, pkd = 0, pkq = 0, pr = 0;
    double gprev = 0.0;
    // one row vertex: distances, and the lane's edge against it
    auto vertex = [&](double x, double y, double z, double& dx, double& dy, double& dz, double& x2, double& kd,
                      double& kq, double& r) {
        dx = x - me.x;
        dy = y - me.y;
        dz = z - me.z;
        x2 = dx * dx + dy * dy + dz * dz;
        if (MODE == 1) {
            // without a branch but for the rare case
            double ir, idn, ic;
            const bool far = inv_dist_fast(x2, eps, ir, idn);
            const bool mid = inv_cbrt_fast(fma(x2, ir, eps), ic);
            const double i2 = idn * idn;
            kd = ic * i2;
            kq = kd * (i2 * i2);
            if (!(far && mid)) dist_weights<MODE>(x2, distExp, eps, kd, kq);
        } else {
            dist_weights<MODE>(x2, distExp, eps, kd, kq);
        }
        const double kqn = __shfl_down_sync(0xffffffffu, kq, 1);
        const bool mine = kq >= kqn;  // the nearer end of the lane's edge
        r = area_sq(tx, ty, tz, mine ? dx : x - nx, mine ? dy : y - ny, mine ? dz : z - nz, eps) * (kq + kqn);
    };
    // the row edge that ends at the vertex just taken: W of (k, lane), its stencil terms
    auto edge = [&](int32_t I, bool kvalid, double Tx, double Ty, double Tz, double ell, double dx, double dy,
                    double dz, double x2, double kd, double kq, double r, double& wx, double& wy, double& w) {
        const double s = pkd + kd;
        const double sumDist = s + __shfl_down_sync(0xffffffffu, s, 1);
        const bool first = px2 <= x2;
        const double p = area_sq(Tx, Ty, Tz, first ? pdx : dx, first ? pdy : dy, first ? pdz : dz, eps) * (pkq + kq);
        const double low = (p + __shfl_down_sync(0xffffffffu, p, 1)) + (pr + r);
        const double ll = ell * me.w;
        const double dotT = Tx * tx + Ty * ty + Tz * tz;
        const int32_t gap = I < Jw ? Jw - I : I - Jw;
        const bool ok = kvalid && lvalid && gap > 1 && gap < V - 1;
        wx = ok ? -0.5 * sumDist * dotT : 0.0;
        wy = ok ? -0.0625 * ll * low : 0.0;
        w = ok ? 0.5 * ll * sumDist : 0.0;
    };
    const int32_t rows = min(R, V - v0);
    for (int32_t i0 = -1; i0 < rows; i0 += (i0 < 0 ? 1 : kBatch)) {
        // (the first round takes vertices v0 - 1 and v0 and the edge between them)
        const int32_t nb = i0 < 0 ? 1 : min(kBatch, rows - i0);
        if (i0 < 0) {
            const double4 q = ea[wrap(v0 - 1)];
            vertex(q.x, q.y, q.z, pdx, pdy, pdz, px2, pkd, pkq, pr);
        }
        // the batch's rows: edge I = v0 + i and the vertex it ends at
        __syncwarp();
        if (lane < nb) {
            const int32_t I = wrap(v0 + i0 + lane);
            const double4 b = ea[I], q = ea[wrap(v0 + i0 + lane + 1)];
            double ex = q.x - b.x, ey = q.y - b.y, ez = q.z - b.z;
            const double len = sqrt(ex * ex + ey * ey + ez * ez);
            const double inv = len < 1e-14 ? 0.0 : 1.0 / len;
            double* o = sm.row[lane];
            o[0] = q.x;
            o[1] = q.y;
            o[2] = q.z;
            o[3] = b.w;
            o[4] = ex * inv;
            o[5] = ey * inv;
            o[6] = ez * inv;
        }
        __syncwarp();
        for (int i = 0; i < nb; i++) {
            const double* o = sm.row[i];
            const int32_t I = wrap(v0 + i0 + i);
            double dx, dy, dz, x2, kd, kq, r, wx, wy, w;
            vertex(o[0], o[1], o[2], dx, dy, dz, x2, kd, kq, r);
            edge(I, true, o[4], o[5], o[6], o[3], dx, dy, dz, x2, kd, kq, r, wx, wy, w);
            pdx = dx;
            pdy = dy;
            pdz = dz;
            px2 = x2;
            pkd = kd;
            pkq = kq;
            pr = r;
            const double z = wx - __shfl_up_sync(0xffffffffu, wx, 1), y = wy + __shfl_up_sync(0xffffffffu, wy, 1);
            if (i0 >= 0) {
                const bool count = own && I > J;
                sm.a[i][lane] = (y + z) + gprev;
                sm.w[i][lane] = count ? w : 0.0;
                sm.q[i][lane] = count ? -wy : 0.0;
                csw += count ? w : 0.0;
                csq += count ? -wy : 0.0;
            }
            gprev = y - z;
        }
        if (i0 < 0) continue;
        __syncwarp();
        // A[v][u], u <= v, along rows
        for (int i = 0; i < nb; i++) {
            const int32_t v = v0 + i0 + i;
            if (own && J <= v) A[(int64_t)v * V + J] = sm.a[i][lane];
        }
        // the mirror A[u][v], u < v: 16 columns v of two rows u at a time
        for (int c = lane >> 4; c < kStrip; c += 2) {
            const int i = lane & 15;
            const int32_t u = u0 + c, v = v0 + i0 + i;
            if (i < nb && u < V && u < v) A[(int64_t)u * V + v] = sm.a[i][c + 1];
        }
        // row sums over the strip: two lanes per row
        {
            const int i = lane & 15, c0 = 1 + 15 * (lane >> 4);
            double sw = 0.0, sq = 0.0;
#pragma unroll
            for (int c = 0; c < 15; c++) {
                sw += sm.w[i][c0 + c];
                sq += sm.q[i][c0 + c];
            }
            sw += __shfl_down_sync(0xffffffffu, sw, 16);
            sq += __shfl_down_sync(0xffffffffu, sq, 16);
            if (lane < nb) rowslot[(int64_t)cs * V + v0 + i0 + i] = make_double2(sw, sq);
        }
    }
    if (own) colslot[(int64_t)rb * V + J] = make_double2(csw, csq);
}

// The pair matrix's diagonal on A's cyclic band: for each vertex v, the terms
// with I = J of the stencil: A[v][v] += Mb'_{v-1} + Mb'_v + M0'_{v-1} + M0'_v,
// A[v][v+1] = A[v+1][v] += -Mb'_v + M0'_v, with (Mb'_I, M0'_I) = (d_I / l_I^2, d0_I)
// summed from the row slots of the strips before I and the column slots of the row
// blocks that reach past it, in order within each of eight groups. Each block forms
// the diagonal entries of its 31 vertices and of the vertex before them once.
__global__ void __launch_bounds__(256) loop_band_kernel(const double4* __restrict__ ea, int32_t V, int32_t R,
                                                        const double2* __restrict__ rowslot,
                                                        const double2* __restrict__ colslot,
                                                        double* __restrict__ A) {
    __shared__ double2 part[8][32], dg[32];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int32_t b0 = blockIdx.x * 31, v = b0 - 1 + x;
    const int32_t I = v < 0 ? V - 1 : v;
    double sx = 0.0, sy = 0.0;
    if (I < V) {
        // strips whose tile (row block of I, strip) exists, and row blocks from that of I on
        const int32_t nr = min((V + kStrip - 1) / kStrip, (I / R * R + R - 1) / kStrip + 1);
        const int32_t nrb = (V + R - 1) / R, rb0 = (I / kStrip * kStrip) / R;
        for (int32_t s = y; s < nr; s += 8) {
            const double2 p = rowslot[(int64_t)s * V + I];
            sx += p.x;
            sy += p.y;
        }
        for (int32_t s = rb0 + y; s < nrb; s += 8) {
            const double2 p = colslot[(int64_t)s * V + I];
            sx += p.x;
            sy += p.y;
        }
    }
    part[y][x] = make_double2(sx, sy);
    __syncthreads();
    if (y > 0) return;
    if (I < V) {
        for (int g = 1; g < 8; g++) {
            sx += part[g][x].x;
            sy += part[g][x].y;
        }
        const double ell = ea[I].w;
        dg[x] = make_double2(sx / (ell * ell), sy);
    }
    __syncwarp();
    if (x == 0 || v >= V) return;
    const double2 dv = dg[x], dp = dg[x - 1];
    A[(int64_t)v * V + v] += (dp.x + dv.x) + (dp.y + dv.y);
    const int32_t u = v + 1 == V ? 0 : v + 1;
    const double off = -dv.x + dv.y;
    A[(int64_t)v * V + u] += off;
    A[(int64_t)u * V + v] += off;
}

}  // namespace

int32_t gather_A_launch(tpe_ctx* ctx, double* d_A, double* d_B, double* d_B0) {
    const int32_t V = ctx->V, E = ctx->E;
    const int32_t nt = (V + 31) / 32;
    const int32_t tiles = nt * (nt + 1) / 2;
    KernelScope ks(ctx, TPE_KGROUP_GATHER_A, 1);
    gather_A_kernel<<<tiles, dim3(32, 32), 0, ctx->stream>>>(
        ctx->pairM.as<double2>(), E, ctx->d_inc_off.as<int32_t>(), ctx->d_inc.as<int32_t>(), V,
        tiles, d_A, d_B, d_B0);
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

int32_t assemble_fp64(tpe_ctx* ctx, double alpha, double beta, double eps, double* d_A,
                      double* d_B, double* d_B0) {
    const int32_t E = ctx->E;
    if (ctx->closed_loop && !d_B && !d_B0) {
        // one closed loop: A straight from the pair weights (no E x E matrix)
        const int32_t V = ctx->V;
        const double s = (beta - 1.0) / alpha;
        const double distExp = 2.0 * (s - 1.0) + 1.0;
        // rows per warp: short marches where there are few warps, few first rows on large
        // curves (with the band, us: at 4 / 8 rows V = 400 25 / 28, 500 29.2 / 29.4, 777 35 / 32;
        // at 8 / 16 1000 34 / 42, 1200 43.6 / 43.5, 1400 48 / 44; at 16 / 32 1700 57 / 65, 2048
        // 68 / 66, 2600 93 / 93, 3600 148 / 139; at 32 / 64 4096 171 / 169, 6000 320 / 328, 8192
        // 564 / 551)
        const int32_t R = V >= 7000 ? 64 : V >= 1900 ? 32 : V >= 1200 ? 16 : V >= 550 ? 8 : 4;
        const int32_t ncs = (V + kStrip - 1) / kStrip, nrb = (V + R - 1) / R;
        TPE_TRY(ensure(ctx, ctx->tmp, sizeof(double2) * (size_t)(ncs + nrb) * V));
        double2* rowslot = ctx->tmp.as<double2>();
        double2* colslot = rowslot + (size_t)ncs * V;
        {
            KernelScope ks(ctx, TPE_KGROUP_PAIR_WEIGHTS, 1);
            auto kern = alpha == 3.0 && beta == 6.0 ? assemble_loop_kernel<1> : assemble_loop_kernel<0>;
            const size_t smem = sizeof(LoopSmem) * kLoopWarps;
            TPE_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            kern<<<dim3((unsigned)((ncs + kLoopWarps - 1) / kLoopWarps), (unsigned)nrb), 32 * kLoopWarps, smem,
                   ctx->stream>>>(ctx->edge_a.as<double4>(), V, R, distExp, eps, d_A, rowslot, colslot);
            TPE_CUDA_TRY(cudaGetLastError());
        }
        KernelScope ks(ctx, TPE_KGROUP_GATHER_A, 1);
        loop_band_kernel<<<(V + 30) / 31, 256, 0, ctx->stream>>>(ctx->edge_a.as<double4>(), V, R, rowslot,
                                                                 colslot, d_A);
        TPE_CUDA_TRY(cudaGetLastError());
        return TPE_OK;
    }
    TPE_TRY(ensure(ctx, ctx->pairM, sizeof(double2) * (size_t)E * E));
    const double s = (beta - 1.0) / alpha;
    const double sigma = s - 1.0;
    const double distExp = 2.0 * sigma + 1.0;
    const int mode = (alpha == 3.0 && beta == 6.0) ? 1 : 0;
    const int32_t ntp = (E + kT - 1) / kT;
    TPE_TRY(ensure(ctx, ctx->tmp, sizeof(double2) * (size_t)ntp * E));
    {
        KernelScope ks(ctx, TPE_KGROUP_PAIR_WEIGHTS, 2);
        const int64_t tiles = (int64_t)ntp * (ntp + 1) / 2;
        if (mode == 1)
            pair_weights_kernel<1><<<(unsigned)tiles, 256, 0, ctx->stream>>>(
                ctx->edge_a.as<double4>(), ctx->edge_b.as<double4>(), ctx->d_edges.as<int2>(), E,
                distExp, eps, ctx->pairM.as<double2>(), ctx->tmp.as<double2>());
        else
            pair_weights_kernel<0><<<(unsigned)tiles, 256, 0, ctx->stream>>>(
                ctx->edge_a.as<double4>(), ctx->edge_b.as<double4>(), ctx->d_edges.as<int2>(), E,
                distExp, eps, ctx->pairM.as<double2>(), ctx->tmp.as<double2>());
        pair_diag_kernel<<<(E + 255) / 256, 256, 0, ctx->stream>>>(
            ctx->edge_a.as<double4>(), E, ntp, ctx->tmp.as<double2>(), ctx->pairM.as<double2>());
        TPE_CUDA_TRY(cudaGetLastError());
    }
    return gather_A_launch(ctx, d_A, d_B, d_B0);
}

}  // namespace tpe
