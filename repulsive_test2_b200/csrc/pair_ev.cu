// All-pairs tangent-point energy and adjoint gradient by (edge, vertex) pairs, FP64.
//
// The reference sums over ordered disjoint edge pairs (I, J) and the four
// endpoint pairs of each (src/core/tangentPointEnergy.ts:50-392). Grouped by
// the vertex v of J instead, the sum is
//   E = 1/8 sum_I l_I^(1-a) sum_v M(I, v) N(I, v) (G(i1, v) + G(i2, v)),
//   N(I, v) = (|e_I x (p_I - x_v)| + eps)^a   (the same for both endpoints p_I),
//   G(i, v) = (|x_i - x_v| + eps)^-b,
//   M(I, v) = sum of l_J over the edges J at v that are disjoint from I,
// so the area is formed once per (edge, vertex) and the distance once per
// vertex pair of the thread's run of edges: 1 area and 1 + 1/R distances per
// ordered (I, v) where the edge-pair form needs 4 of each. For a vertex that no
// edge joins to I, M(I, v) is m_v, the length of all edges at v. The few near
// vertices of I (its endpoints and their neighbours, a sorted list per edge)
// are masked out of the sweep, in a copy of its inner loop for the groups of 32
// vertices that hold one; the near ones that are not endpoints are summed over
// their disjoint edges one by one afterwards.
//
// Bound: the FP64 pipe and its latency. 52 FP64 instructions per ordered (I, v)
// for the energy, 104 for the gradient; at 8192 edges the pipe is active 82 and
// 78 % of the time (three to four warps per scheduler: 120 and 168 registers). The sweep's common
// case has no branch, so that the runs of a thread's edges interleave: with the
// rare cases tested one by one the same sums took 343 and 685 us, with the masks in
// the one loop 276 and 608. Measured, 8192 edges of a closed curve: energy 699 -> 264
// us, gradient 2239 -> 575 us against the edge-pair kernels; 128 edges: 160 -> 12 and
// 239 -> 26 us. A hub's lists are dealt over the energy's chunks and over eight rows of
// the reductions (four hubs of 40 spokes, 964 edges: gradient 274 -> 126 us).
//
// Work split: a worker of 128 threads owns 128 R consecutive edges (R per
// thread, so that a run of edges shares its vertices' distances) and sweeps a
// chunk of the vertices from shared memory; R and the chunk follow the size
// (ev_split). The edge side accumulates in registers; the vertex side
// (force and length derivative of the swept vertex) is reduced over the warp by
// halving exchanges (6 shuffles for 4 values) and over the warps in a fixed
// order. Every (chunk, edge) and (edge block, vertex) partial is written once and
// summed in a fixed order: deterministic, no atomics on data.
//
// Accuracy: the cross product takes the nearer of the two endpoints, whose
// difference vector loses the least.
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "pair_math.cuh"
#include "tpe_internal.h"

namespace tpe {
namespace {

constexpr int kW = 128;      // threads of a worker
constexpr int kTile = 128;   // vertices staged at a time
constexpr int kWorkers = 3;  // workers per block of the SM-bounded form
constexpr int kGroup = kTile / 8;  // most chunks of one energy item (ev_split)
constexpr int kAcc = 7;      // per (chunk, edge): force on both endpoints, sum of M N (G1 + G2)

// The curve's records and the topology lists every kernel here reads.
struct EvTopo {
    const int2* __restrict__ ev;           // per edge: its endpoints as vertex slots
    const int32_t* __restrict__ near_off;  // per edge: its near vertex slots, sorted
    const int32_t* __restrict__ near;
    const int32_t* __restrict__ rev_off;   // per vertex slot: the edges it is near to, not on
    const int32_t* __restrict__ rev;
    const int32_t* __restrict__ inc_off;   // per vertex: incident 2 * edge + slot
    const int32_t* __restrict__ inc;
    const int32_t* __restrict__ vid;       // vertex of each slot (vertices with an edge)
    const int2* __restrict__ edges;
    int32_t E, VA;
};

// G = (|d| + eps)^-b and gI = 1 / (|d| (|d| + eps)) (0 below |d| = 1e-14) of x = |d|^2: G and
// gI on their own, since their product, -dG/d|d| / (b |d|), falls out of the double range at
// 1e38 (b = 6), well before the gradient's terms do.
template <int MODE>
__device__ __forceinline__ void dist_power(double x, double beta, double eps, double& G, double& gI) {
    double s, inv, inve;
    dist_terms(x, eps, s, inv, inve);
    if (MODE == 1) {
        const double i2 = inve * inve;
        G = i2 * i2 * i2;  // b = 6
    } else {
        G = 1.0 / pow(s + eps, beta);
    }
    gI = inve * inv;
}

// N = (|c| + eps)^a and kN = (|c| + eps)^(a-1) / |c| (0 below |c| = 1e-14).
template <int MODE>
__device__ __forceinline__ void area_power(double c2, double alpha, double eps, double& N, double& kN) {
    double rc, inv = 0.0;
    if (c2 >= 1e-28 && c2 <= 1e300) {
        inv = rsqrt_normal(c2);
        rc = c2 * inv;
    } else {  // flat, or beyond rsqrt_normal's range
        rc = sqrt(c2);
        inv = rc < 1e-14 ? 0.0 : 1.0 / rc;
    }
    const double cn = rc + eps;
    if (MODE == 1) {
        const double cn2 = cn * cn;  // a = 3
        N = cn2 * cn;
        kN = cn2 * inv;
    } else {
        N = pow(cn, alpha);
        kN = inv > 0.0 ? N / cn * inv : 0.0;
    }
}

// The same for a = 3, b = 6 where the distance is beyond 1e6 eps and the area
// above 1e-14 (and finite), without a branch; false elsewhere.
__device__ __forceinline__ bool dist_power_fast(double x, double eps, double& G, double& gI) {
    double r, inve;
    const bool ok = inv_dist_fast(x, eps, r, inve);
    const double i2 = inve * inve;
    G = i2 * i2 * i2;
    gI = inve * r;
    return ok;
}
__device__ __forceinline__ bool area_power_fast(double c2, double eps, double& N, double& kN) {
    const double inv = rsqrt_normal(c2);
    const double cn = fma(c2, inv, eps);
    const double cn2 = cn * cn;
    N = cn2 * cn;
    kN = cn2 * inv;
    return c2 >= 1e-28 && c2 <= 1e300;
}

struct V3 {
    double x, y, z;
};
__device__ __forceinline__ V3 sub(const V3& a, const V3& b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ double dot3(const V3& a, const V3& b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross3(const V3& a, const V3& b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
// a += s b
__device__ __forceinline__ void axpy3(V3& a, double s, const V3& b) {
    a.x += s * b.x;
    a.y += s * b.y;
    a.z += s * b.z;
}
// f += a x b
__device__ __forceinline__ void add_cross(V3& f, const V3& a, const V3& b) {
    f.x += a.y * b.z - a.z * b.y;
    f.y += a.z * b.x - a.x * b.z;
    f.z += a.x * b.y - a.y * b.x;
}
__device__ __forceinline__ void sub_cross(V3& f, const V3& a, const V3& b) {
    f.x -= a.y * b.z - a.z * b.y;
    f.y -= a.z * b.x - a.x * b.z;
    f.z -= a.x * b.y - a.y * b.x;
}

struct EvSmem {
    double4 sv[kTile];                 // x, y, z, m
    double acc[kW / 32][kTile][4];     // per warp: force on the swept vertex, sum of l_I^(1-a) N (G1 + G2)
    double red[kGroup][kW / 32];       // per chunk of the group and warp
    int next;
};

__device__ __forceinline__ void worker_sync(int bar) {
    asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(kW) : "memory");
}

// One edge against one vertex outside the sweep: N, G1 + G2 and the derivative
// terms (G1 g1, G2 g2: dist_power's; kc = K c with K = a (G1 + G2) kN).
template <int MODE>
struct PairTerms {
    double GS, N;
    V3 d1, d2, kc;
    double G1, G2, g1, g2;
    __device__ __forceinline__ PairTerms(const V3& p1, const V3& p2, const V3& q, double alpha,
                                         double beta, double eps) {
        d1 = sub(p1, q);
        d2 = sub(p2, q);
        const double x1 = dot3(d1, d1), x2 = dot3(d2, d2);
        double kN;
        dist_power<MODE>(x1, beta, eps, G1, g1);
        dist_power<MODE>(x2, beta, eps, G2, g2);
        const V3 e = sub(p2, p1);
        const V3 c = cross3(e, x1 <= x2 ? d1 : d2);
        area_power<MODE>(dot3(c, c), alpha, eps, N, kN);
        GS = G1 + G2;
        const double K = alpha * GS * kN;
        kc = {K * c.x, K * c.y, K * c.z};
    }
};

// M(I, v) of a near vertex slot v that is not an endpoint: the edges at v that are disjoint
// from I, m_v of them in all. One by one; at a vertex of many edges as m_v without those that
// lead to I's endpoints, where they are the smaller part (nothing cancels then).
__device__ __forceinline__ double near_length(const EvTopo& t, const double4* __restrict__ ea, int2 ei, int32_t v,
                                              double m_v) {
    const int32_t w = t.vid[v], k0 = t.inc_off[w], k1 = t.inc_off[w + 1];
    if (k1 - k0 > 8) {
        double off = 0.0;
        for (int s = 0; s < (ei.x == ei.y ? 1 : 2); s++) {
            const int32_t u = s ? ei.y : ei.x;
            for (int32_t k = t.inc_off[u]; k < t.inc_off[u + 1]; k++) {
                const int2 e = t.edges[t.inc[k] >> 1];
                if (e.x == w || e.y == w) off += ea[t.inc[k] >> 1].w;
            }
        }
        if (off < 0.5 * m_v) return m_v - off;
    }
    double m = 0.0;
    for (int32_t k = k0; k < k1; k++) {
        const int32_t J = t.inc[k] >> 1;
        if (disjoint(ei, t.edges[J])) m += ea[J].w;
    }
    return m;
}

// No edge is disjoint from this one: it has no terms, whatever its coordinates.
__device__ __forceinline__ bool lonely(const EvTopo& t, int2 ei) {
    int32_t n = 0;  // edges at its vertices
    for (int s = 0; s < (ei.x == ei.y ? 1 : 2); s++) {
        const int32_t w = s ? ei.y : ei.x;
        for (int32_t k = t.inc_off[w]; k < t.inc_off[w + 1]; k++) {
            const int2 e = t.edges[t.inc[k] >> 1];
            if (e.x == e.y ? (t.inc[k] & 1) == 0 : !(s && (e.x == ei.x || e.y == ei.x))) n++;
        }
    }
    return n == t.E;
}

// Sweeps the vertices [vb, vb + n) (n <= kTile, staged from sm.sv[s0] on) for the
// thread's R edges. CHAIN: the edges run head to tail (R + 1 vertices), else
// every edge has its own two. near_lo / near_hi bound the thread's near slots.
template <int MODE, int R, bool GRAD, bool CHAIN>
__device__ __forceinline__ void sweep(EvSmem& sm, int32_t s0, int32_t vb, int32_t n, const EvTopo& t, int32_t I0,
                                      const V3 (&P)[CHAIN ? R + 1 : 2 * R], const double (&pw)[R],
                                      int32_t near_lo, int32_t near_hi, double alpha, double beta,
                                      double eps, double (&S)[R], V3 (&F)[CHAIN ? R + 1 : 2 * R]) {
    constexpr int NV = CHAIN ? R + 1 : 2 * R;
    const int lane = threadIdx.x & 31, warp = (threadIdx.x % kW) >> 5;
    for (int32_t g0 = 0; g0 < n; g0 += 32) {
        // bit j of mask[r]: vertex vb + g0 + j is near edge r (or the edge does not exist)
        uint32_t mask[R];
        uint32_t any = 0;
        const int32_t base = vb + g0, gn = min(32, n - g0);
#pragma unroll
        for (int r = 0; r < R; r++) {
            mask[r] = I0 + r < t.E ? 0u : 0xffffffffu;
            if (I0 + r < t.E && near_hi >= base && near_lo < base + gn) {
                int32_t k = t.near_off[I0 + r];
                const int32_t end = t.near_off[I0 + r + 1];
                for (int32_t h = end; h - k > 16;) {  // (a long list: to its part from base on)
                    const int32_t mid = (k + h) >> 1;
                    if (t.near[mid] < base)
                        k = mid;
                    else
                        h = mid;
                }
                for (; k < end; k++) {
                    const int32_t d = t.near[k] - base;
                    if (d >= gn) break;
                    if (d >= 0) mask[r] |= 1u << d;
                }
            }
            any |= mask[r];
        }
        const bool careful = __any_sync(0xffffffffu, any != 0u);
        // MASKED: near pairs are left out, whatever their values (a distance of zero, a
        // coordinate that is no number)
        auto vertex = [&](auto masked, int32_t j) {
            constexpr bool MASKED = decltype(masked)::value;
            auto off = [&](int r) { return MASKED && (mask[r] >> j & 1u); };
            const double4 q4 = sm.sv[s0 + g0 + j];
            const V3 q{q4.x, q4.y, q4.z};
            V3 d[NV], c[R];
            double x[NV], G[NV], gI[NV], h[NV], c2[R], N[R], kN[R];
            // the common case without a branch, so that the runs of all R edges
            // interleave; a distance near zero or a flat triangle redoes the lane's
            bool rare = false;
#pragma unroll
            for (int a = 0; a < NV; a++) {
                d[a] = sub(P[a], q);
                x[a] = dot3(d[a], d[a]);
                if (MASKED && (CHAIN ? (a == 0 || off(a - 1)) && (a == R || off(a)) : off(a / 2))) {
                    d[a] = {0.0, 0.0, 0.0};  // (no edge of this point counts)
                    x[a] = 1.0;
                }
                if (MODE == 1)
                    rare |= !dist_power_fast(x[a], eps, G[a], gI[a]);
                else
                    dist_power<MODE>(x[a], beta, eps, G[a], gI[a]);
                h[a] = 0.0;
            }
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int a = CHAIN ? r : 2 * r, b = a + 1;
                const V3 e = sub(P[b], P[a]);
                const bool first = x[a] <= x[b];
                const V3 dn{first ? d[a].x : d[b].x, first ? d[a].y : d[b].y, first ? d[a].z : d[b].z};
                c[r] = cross3(e, dn);
                c2[r] = off(r) ? 1.0 : dot3(c[r], c[r]);
                if (MODE == 1)
                    rare |= !area_power_fast(c2[r], eps, N[r], kN[r]);
                else
                    area_power<MODE>(c2[r], alpha, eps, N[r], kN[r]);
            }
            if (rare) {
#pragma unroll
                for (int a = 0; a < NV; a++) dist_power<MODE>(x[a], beta, eps, G[a], gI[a]);
#pragma unroll
                for (int r = 0; r < R; r++) area_power<MODE>(c2[r], alpha, eps, N[r], kN[r]);
            }
            V3 Q{0.0, 0.0, 0.0};
            double Rv = 0.0;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int a = CHAIN ? r : 2 * r, b = a + 1;
                const V3 e = sub(P[b], P[a]);
                if (off(r)) continue;
                const double GS = G[a] + G[b];
                const double NG = N[r] * GS;
                S[r] += q4.w * NG;
                if (GRAD) {
                    Rv += pw[r] * NG;
                    const double mp = q4.w * pw[r];
                    const double tn = mp * N[r];
                    h[a] += tn;
                    h[b] += tn;
                    const double K = (alpha * mp) * (GS * kN[r]);
                    const V3 kc{K * c[r].x, K * c[r].y, K * c[r].z};
                    sub_cross(F[a], d[b], kc);
                    add_cross(F[b], d[a], kc);
                    add_cross(Q, e, kc);
                }
            }
            if (GRAD) {
#pragma unroll
                for (int a = 0; a < NV; a++) {
                    const double f = -beta * ((h[a] * G[a]) * gI[a]);
                    axpy3(F[a], f, d[a]);
                    axpy3(Q, -f, d[a]);
                }
                // warp sums of (Q, Rv) by halving exchanges: lane 8 k ends with value k
                const bool up = lane & 16;
                double s0 = up ? Q.x : Q.z, s1 = up ? Q.y : Rv;
                double k0 = up ? Q.z : Q.x, k1 = up ? Rv : Q.y;
                k0 += __shfl_xor_sync(0xffffffffu, s0, 16);
                k1 += __shfl_xor_sync(0xffffffffu, s1, 16);
                const bool up2 = lane & 8;
                s0 = up2 ? k0 : k1;
                k0 = up2 ? k1 : k0;
                k0 += __shfl_xor_sync(0xffffffffu, s0, 8);
                k0 += __shfl_xor_sync(0xffffffffu, k0, 4);
                k0 += __shfl_xor_sync(0xffffffffu, k0, 2);
                k0 += __shfl_xor_sync(0xffffffffu, k0, 1);
                if ((lane & 7) == 0) sm.acc[warp][g0 + j][lane >> 3] = k0;
            }
        };
        if (careful)
            for (int32_t j = 0; j < gn; j++) vertex(std::true_type{}, j);
        else
            for (int32_t j = 0; j < gn; j++) vertex(std::false_type{}, j);
    }
}

// Work item (edge block ib, vertex chunks from ch0, `group` of them) of one curve. GRAD:
// one chunk, edge_acc [ch][kAcc][E] and vert_acc [ib][VA][4]; else each chunk's energy
// (the near pairs dealt over the chunks) to part[chunk]. Several chunks have at most kTile
// vertices together, staged at once.
template <int MODE, int R, bool GRAD>
__device__ __forceinline__ void ev_item(int ib, int ch0, int group, int32_t chunk, int32_t nch, int tid, int bar,
                                        EvSmem& sm, const EvTopo& t, const double4* __restrict__ ea,
                                        const double4* __restrict__ eb,
                                        const double4* __restrict__ vr, double alpha, double beta,
                                        double eps, double* __restrict__ edge_acc,
                                        double* __restrict__ vert_acc, double* __restrict__ part) {
    const int32_t I0 = (ib * kW + tid) * R;
    V3 p1[R], p2[R];
    int2 ei[R];
    double pw[R], S[R];
    int32_t near_lo = 0x7fffffff, near_hi = -1;
    bool chain = I0 + R <= t.E;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int32_t I = min(I0 + r, t.E - 1);
        p1[r] = {ea[I].x, ea[I].y, ea[I].z};
        p2[r] = {eb[I].x, eb[I].y, eb[I].z};
        pw[r] = eb[I].w;
        ei[r] = t.ev[I];
        if (r > 0) chain = chain && ei[r - 1].y == ei[r].x;
        if (I0 + r < t.E) {
            near_lo = min(near_lo, t.near[t.near_off[I]]);
            near_hi = max(near_hi, t.near[t.near_off[I + 1] - 1]);
        }
    }
    const bool run = __all_sync(0xffffffffu, chain);
    const int32_t ch1 = min(ch0 + group, nch), last = min(t.VA, ch1 * chunk);
    int32_t s0 = 0, s1 = 0;  // the vertices in sm.sv
    V3 f1[R], f2[R];
    // the vertices [v0, v1) for the edges' points P
    auto march = [&](auto chained, const auto& P, auto& F, int32_t v0, int32_t v1) {
        for (int32_t vb = v0; vb < v1; vb += kTile) {
            const int32_t n = min(kTile, v1 - vb);
            if (vb >= s1) {
                s0 = vb;
                s1 = min(vb + kTile, last);
                worker_sync(bar);
                if (tid < s1 - s0) sm.sv[tid] = vr[s0 + tid];
                worker_sync(bar);
            }
            sweep<MODE, R, GRAD, decltype(chained)::value>(sm, vb - s0, vb, n, t, I0, P, pw, near_lo, near_hi,
                                                           alpha, beta, eps, S, F);
            if (GRAD) {
                worker_sync(bar);
                for (int k = tid; k < 4 * n; k += kW) {
                    double s = 0.0;
#pragma unroll
                    for (int w = 0; w < kW / 32; w++) s += (&sm.acc[w][0][0])[k];
                    vert_acc[((int64_t)ib * t.VA + vb) * 4 + k] = s;
                }
            }
        }
    };
    for (int32_t ch = ch0; ch < ch1; ch++) {
        const int32_t v0 = ch * chunk, v1 = min(t.VA, v0 + chunk);
#pragma unroll
        for (int r = 0; r < R; r++) S[r] = 0.0;
        if (R > 1 && run) {
            V3 P[R + 1], F[R + 1];
#pragma unroll
            for (int a = 0; a <= R; a++) {
                P[a] = a < R ? p1[a < R ? a : 0] : p2[R - 1];
                F[a] = {0.0, 0.0, 0.0};
            }
            march(std::true_type{}, P, F, v0, v1);
            // a shared vertex's force goes to the edge it begins
#pragma unroll
            for (int r = 0; r < R; r++) {
                f1[r] = F[r];
                f2[r] = {0.0, 0.0, 0.0};
            }
            f2[R - 1] = F[R];
        } else {
            V3 P[2 * R], F[2 * R];
#pragma unroll
            for (int r = 0; r < R; r++) {
                P[2 * r] = p1[r];
                P[2 * r + 1] = p2[r];
                F[2 * r] = F[2 * r + 1] = {0.0, 0.0, 0.0};
            }
            march(std::false_type{}, P, F, v0, v1);
#pragma unroll
            for (int r = 0; r < R; r++) {
                f1[r] = F[2 * r];
                f2[r] = F[2 * r + 1];
            }
        }
        if (GRAD) break;  // (one chunk)
        double en = 0.0;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int32_t I = I0 + r;
            if (I >= t.E) break;
            for (int32_t k = t.near_off[I] + ch; k < t.near_off[I + 1]; k += nch) {
                const int32_t v = t.near[k];
                if (v == ei[r].x || v == ei[r].y) continue;
                const double4 q = vr[v];
                const double m = near_length(t, ea, t.edges[I], v, q.w);
                if (m == 0.0) continue;
                const PairTerms<MODE> pt(p1[r], p2[r], {q.x, q.y, q.z}, alpha, beta, eps);
                S[r] += m * (pt.N * pt.GS);
            }
            if (isfinite(pw[r]) || !lonely(t, t.edges[I])) en += pw[r] * S[r];
        }
        for (int o = 16; o > 0; o >>= 1) en += __shfl_down_sync(0xffffffffu, en, o);
        if ((tid & 31) == 0) sm.red[ch - ch0][tid >> 5] = en;
    }
    if (GRAD) {
        double* o = edge_acc + (int64_t)ch0 * kAcc * t.E;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int32_t I = I0 + r;
            if (I >= t.E) break;
            o[I] = f1[r].x;
            o[t.E + I] = f1[r].y;
            o[2 * (int64_t)t.E + I] = f1[r].z;
            o[3 * (int64_t)t.E + I] = f2[r].x;
            o[4 * (int64_t)t.E + I] = f2[r].y;
            o[5 * (int64_t)t.E + I] = f2[r].z;
            o[6 * (int64_t)t.E + I] = S[r];
        }
        return;
    }
    worker_sync(bar);
    if (tid < ch1 - ch0) {
        double s = 0.0;
        for (int w = 0; w < kW / 32; w++) s += sm.red[tid][w];
        part[ch0 + tid] = s;
    }
}

// One item per block; blockIdx = (group of chunks, edge block, curve).
template <int MODE, int R, bool GRAD>
__global__ void __launch_bounds__(kW, GRAD && R == 2 ? 3 : 4)
ev_kernel(const double4* __restrict__ ea, const double4* __restrict__ eb,
          const double4* __restrict__ vr, EvTopo t, int32_t chunk, int32_t nch, int32_t group, double alpha,
          double beta, double eps, double* __restrict__ edge_acc, double* __restrict__ vert_acc,
          double* __restrict__ part) {
    __shared__ EvSmem sm;
    const int64_t c = blockIdx.z;
    ev_item<MODE, R, GRAD>(blockIdx.y, blockIdx.x * group, group, chunk, nch, threadIdx.x, 0, sm, t, ea + c * t.E,
                           eb + c * t.E, vr + c * t.VA, alpha, beta, eps, edge_acc, vert_acc,
                           part + (c * gridDim.y + blockIdx.y) * nch);
}

// The gradient's items on a bounded number of SMs: kWorkers independent workers
// per block (their registers fill an SM, so one block per SM) take items from a
// counter. Every item writes its own partials: the result does not depend on
// which worker took it. For the gradient that runs beside the factorization.
template <int MODE, int R>
__global__ void __launch_bounds__(kW* kWorkers, 1)
ev_persist_kernel(const double4* __restrict__ ea, const double4* __restrict__ eb,
                  const double4* __restrict__ vr, EvTopo t, int32_t chunk, int32_t nch, int32_t items,
                  double alpha, double beta, double eps, double* __restrict__ edge_acc,
                  double* __restrict__ vert_acc, int32_t* __restrict__ counter) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int w = threadIdx.x / kW, tid = threadIdx.x % kW;
    EvSmem& sm = reinterpret_cast<EvSmem*>(smem_raw)[w];
    for (;;) {
        if (tid == 0) sm.next = atomicAdd(counter, 1);
        worker_sync(1 + w);
        const int x = sm.next;
        worker_sync(1 + w);
        if (x >= items) break;
        ev_item<MODE, R, true>(x / nch, x % nch, 1, chunk, nch, tid, 1 + w, sm, t, ea, eb, vr, alpha, beta, eps,
                               edge_acc, vert_acc, nullptr);
    }
}

// Per edge: the chunks' partials summed, its near vertices added, the length
// derivative (through l^(1-a) and through M) along the tangent, to edge_f
// [6][E]; the edge's share of the energy to edge_e. 32 edges x 8 chunk lanes.
template <int MODE>
__global__ void __launch_bounds__(256)
ev_edge_kernel(const double4* __restrict__ ea, const double4* __restrict__ eb,
               const double4* __restrict__ vr, EvTopo t, int32_t nch, int32_t nib, double alpha,
               double beta, double eps, const double* __restrict__ edge_acc,
               const double* __restrict__ vert_acc, double* __restrict__ edge_f,
               double* __restrict__ edge_e) {
    __shared__ double red[8][kAcc + 1][32];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int32_t I = blockIdx.x * 32 + x;
    const bool in = I < t.E;
    const double4 a4 = ea[in ? I : 0], b4 = eb[in ? I : 0];
    const V3 p1{a4.x, a4.y, a4.z}, p2{b4.x, b4.y, b4.z};
    const double pw = b4.w;
    const int2 edge = t.edges[in ? I : 0], slot = t.ev[in ? I : 0];
    V3 f1{0.0, 0.0, 0.0}, f2 = f1;
    double S = 0.0, Rl = 0.0;
    if (in) {
        for (int32_t c = y; c < nch; c += 8) {
            const double* o = edge_acc + (int64_t)c * kAcc * t.E + I;
            f1.x += o[0];
            f1.y += o[t.E];
            f1.z += o[2 * (int64_t)t.E];
            f2.x += o[3 * (int64_t)t.E];
            f2.y += o[4 * (int64_t)t.E];
            f2.z += o[5 * (int64_t)t.E];
            S += o[6 * (int64_t)t.E];
        }
        for (int32_t k = t.near_off[I] + y; k < t.near_off[I + 1]; k += 8) {
            const int32_t v = t.near[k];
            if (v == slot.x || v == slot.y) continue;
            const double4 q = vr[v];
            const double m = near_length(t, ea, edge, v, q.w);
            if (m == 0.0) continue;
            const PairTerms<MODE> pt(p1, p2, {q.x, q.y, q.z}, alpha, beta, eps);
            S += m * (pt.N * pt.GS);
            const double mp = m * pw;
            const V3 kc{mp * pt.kc.x, mp * pt.kc.y, mp * pt.kc.z};
            sub_cross(f1, pt.d2, kc);
            add_cross(f2, pt.d1, kc);
            const double tn = -beta * (mp * pt.N);
            axpy3(f1, (tn * pt.G1) * pt.g1, pt.d1);
            axpy3(f2, (tn * pt.G2) * pt.g2, pt.d2);
        }
        // dE/dl_I through M: the edges K disjoint from I, at both of I's vertices
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int32_t v = e ? slot.y : slot.x;
            const V3 q = e ? p2 : p1;
            for (int32_t b = y; b < nib; b += 8) Rl += vert_acc[((int64_t)b * t.VA + v) * 4 + 3];
            for (int32_t k = t.rev_off[v] + y; k < t.rev_off[v + 1]; k += 8) {
                const int32_t K = t.rev[k];
                if (!disjoint(edge, t.edges[K])) continue;
                const double4 ka = ea[K], kb = eb[K];
                const PairTerms<MODE> pt({ka.x, ka.y, ka.z}, {kb.x, kb.y, kb.z}, q, alpha, beta, eps);
                Rl += kb.w * (pt.N * pt.GS);
            }
        }
    }
    const double mine[kAcc + 1] = {f1.x, f1.y, f1.z, f2.x, f2.y, f2.z, S, Rl};
#pragma unroll
    for (int q = 0; q <= kAcc; q++) red[y][q][x] = mine[q];
    __syncthreads();
    if (y != 0 || !in) return;
    double s[kAcc + 1];
#pragma unroll
    for (int q = 0; q <= kAcc; q++) {
        s[q] = mine[q];
        for (int g = 1; g < 8; g++) s[q] += red[g][q][x];
    }
    f1 = {s[0], s[1], s[2]};
    f2 = {s[3], s[4], s[5]};
    S = s[6];
    Rl = s[7];
    const V3 e = sub(p2, p1);
    const double raw = sqrt(dot3(e, e));
    if (!(isfinite(raw) && isfinite(pw)) && lonely(t, edge)) {
        f1 = f2 = {0.0, 0.0, 0.0};
        S = 0.0;
    } else if (!(raw < 1e-14)) {
        const double dl = (Rl + (1.0 - alpha) * pow(a4.w, -alpha) * S) / raw;
        axpy3(f1, -dl, e);
        axpy3(f2, dl, e);
    }
    edge_f[I] = f1.x;
    edge_f[t.E + I] = f1.y;
    edge_f[2 * (int64_t)t.E + I] = f1.z;
    edge_f[3 * (int64_t)t.E + I] = f2.x;
    edge_f[4 * (int64_t)t.E + I] = f2.y;
    edge_f[5 * (int64_t)t.E + I] = f2.z;
    edge_e[I] = !isfinite(pw) && lonely(t, edge) ? 0.0 : pw * S;
}

// grad[v] = 1/8 (its edges' forces + its own sweep partials + the edges it is near to).
// 32 vertices x 8 lanes, as the edges.
template <int MODE>
__global__ void __launch_bounds__(256)
ev_vertex_kernel(const double4* __restrict__ ea, const double4* __restrict__ eb, EvTopo t,
                 int32_t nib, int32_t V, const int32_t* __restrict__ slot_of, const double4* __restrict__ vr,
                 double alpha, double beta, double eps, const double* __restrict__ vert_acc,
                 const double* __restrict__ edge_f, double* __restrict__ grad) {
    __shared__ double red[8][3][32];
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int32_t w = blockIdx.x * 32 + x, v = w < V ? slot_of[w] : -1;
    V3 g{0.0, 0.0, 0.0};
    if (v >= 0) {
        for (int32_t b = y; b < nib; b += 8) {
            const double* o = vert_acc + ((int64_t)b * t.VA + v) * 4;
            const double2 xy = *reinterpret_cast<const double2*>(o);
            g.x += xy.x;
            g.y += xy.y;
            g.z += o[2];
        }
        const double4 q = vr[v];
        for (int32_t k = t.rev_off[v] + y; k < t.rev_off[v + 1]; k += 8) {
            const int32_t I = t.rev[k];
            const double m = near_length(t, ea, t.edges[I], v, q.w);
            if (m == 0.0) continue;
            const double4 a = ea[I], b = eb[I];
            const V3 p1{a.x, a.y, a.z}, p2{b.x, b.y, b.z};
            const PairTerms<MODE> pt(p1, p2, {q.x, q.y, q.z}, alpha, beta, eps);
            const double mp = m * b.w;
            const V3 kc{mp * pt.kc.x, mp * pt.kc.y, mp * pt.kc.z};
            add_cross(g, sub(p2, p1), kc);
            const double tn = beta * (mp * pt.N);
            axpy3(g, (tn * pt.G1) * pt.g1, pt.d1);
            axpy3(g, (tn * pt.G2) * pt.g2, pt.d2);
        }
        for (int32_t k = t.inc_off[w] + y; k < t.inc_off[w + 1]; k += 8) {
            const int32_t I = t.inc[k] >> 1, c = 3 * (t.inc[k] & 1);
            g.x += edge_f[(int64_t)c * t.E + I];
            g.y += edge_f[(int64_t)(c + 1) * t.E + I];
            g.z += edge_f[(int64_t)(c + 2) * t.E + I];
        }
    }
    red[y][0][x] = g.x;
    red[y][1][x] = g.y;
    red[y][2][x] = g.z;
    __syncthreads();
    if (y != 0 || w >= V) return;
    for (int q = 0; q < 3; q++) {
        double s = red[0][q][x];
        for (int h = 1; h < 8; h++) s += red[h][q][x];
        grad[3 * (int64_t)w + q] = 0.125 * s;
    }
}

// Edge records (as edge_prep_kernel) and vertex records (x, y, z, m) of the
// vertices with an edge, m the length (with eps) of the edges at it.
__global__ void __launch_bounds__(128)
ev_prep_kernel(const double* __restrict__ pos, EvTopo t, int32_t V, int32_t ncurves, double eps,
               double alpha, double4* __restrict__ ea, double4* __restrict__ eb,
               double4* __restrict__ vr) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    auto length = [&](const double* p, int2 e) {
        const double ex = p[3 * e.y] - p[3 * e.x], ey = p[3 * e.y + 1] - p[3 * e.x + 1],
                     ez = p[3 * e.y + 2] - p[3 * e.x + 2];
        return sqrt(ex * ex + ey * ey + ez * ez) + eps;
    };
    const int64_t ne = (int64_t)t.E * ncurves;
    if (i < ne) {
        const double* p = pos + (i / t.E) * 3 * V;
        const int2 e = t.edges[i % t.E];
        const double ell = length(p, e);
        ea[i] = make_double4(p[3 * e.x], p[3 * e.x + 1], p[3 * e.x + 2], ell);
        eb[i] = make_double4(p[3 * e.y], p[3 * e.y + 1], p[3 * e.y + 2], pow(ell, 1.0 - alpha));
        return;
    }
    i -= ne;
    if (i >= (int64_t)t.VA * ncurves) return;
    const double* p = pos + (i / t.VA) * 3 * V;
    const int32_t w = t.vid[i % t.VA];
    double m = 0.0;
    for (int32_t k = t.inc_off[w]; k < t.inc_off[w + 1]; k++) m += length(p, t.edges[t.inc[k] >> 1]);
    vr[i] = make_double4(p[3 * w], p[3 * w + 1], p[3 * w + 2], m);
}

EvTopo topo_of(const tpe_ctx* ctx) {
    EvTopo t;
    const int32_t* b = ctx->ev_lists.as<int32_t>();
    t.ev = reinterpret_cast<const int2*>(b);
    t.near_off = b + ctx->ev_at[0];
    t.near = b + ctx->ev_at[1];
    t.rev_off = b + ctx->ev_at[2];
    t.rev = b + ctx->ev_at[3];
    t.vid = b + ctx->ev_at[4];
    t.inc_off = ctx->d_inc_off.as<int32_t>();
    t.inc = ctx->d_inc.as<int32_t>();
    t.edges = ctx->d_edges.as<int2>();
    t.E = ctx->E;
    t.VA = ctx->ev_VA;
    return t;
}

// Edges per thread and vertices per item. Two edges per thread from 2048 edges
// on (1.5 distances per area and one warp reduction per two edges: 8192 edges
// 264 against 306 us for the energy, 583 against 657 for the gradient, 2048 edges 37
// against 37 and 74 against 81; four edges per thread spill). Below, one: more items, shorter chains
// (1024 edges: 21 against 23 us). Items of 8 to 128 vertices, about six per SM.
// Neither depends on how many curves a launch has: the order of an energy's sum, and with
// it its last bits, are those of the curve alone (differences of energies from launches of
// different sizes are taken). With more curves a block takes `group` chunks of one edge
// block, up to kTile vertices, one after the other.
struct EvSplit {
    int R;
    int32_t nib, chunk, nch, group;
};
EvSplit ev_split(const tpe_ctx* ctx, int32_t ncurves) {
    EvSplit s;
    const int32_t E = ctx->E, VA = ctx->ev_VA;
    s.R = E >= 2048 ? 2 : 1;
    s.nib = (E + kW * s.R - 1) / (kW * s.R);
    const int64_t want = 6 * (int64_t)ctx->num_sms;  // items
    int64_t c = ((int64_t)VA * s.nib + want - 1) / want;
    c = (c + 7) / 8 * 8;
    // at most 96 chunks (partials per edge), or items of 128 vertices where that is more
    const int64_t most = std::max<int64_t>(kTile, ((VA + 95) / 96 + kTile - 1) / kTile * kTile);
    s.chunk = (int32_t)std::min<int64_t>(std::max<int64_t>(c, 8), most);
    s.nch = (VA + s.chunk - 1) / s.chunk;
    const int64_t g = ((int64_t)s.nch * s.nib * ncurves + want - 1) / want;
    s.group = (int32_t)std::max<int64_t>(1, std::min<int64_t>(g, kTile / s.chunk));
    return s;
}

int exp_mode(double alpha, double beta) { return (alpha == 3.0 && beta == 6.0) ? 1 : 0; }

}  // namespace

// The lists of the (edge, vertex) form, built once per topology on first use:
// one device buffer of ints (ev, near_off, near, rev_off, rev, vid, slot_of).
// A topology whose near lists outgrow the edges (a hub of very high degree:
// every pair of its spokes is near), or of fewer than eight edges (a loop of four: 43 us
// against 34 for the energy, 66 against 60 for the gradient; of eight: 44 and 63 either
// way), keeps the edge-pair kernels: *ok = false.
int32_t ev_topology(tpe_ctx* ctx, bool* ok) {
    if (ctx->ev_state == 0) {
        const int32_t E = ctx->E, V = ctx->V;
        const int32_t* ed = ctx->h_edges.data();
        int64_t bound = 0;
        for (int32_t I = 0; I < E; I++)
            for (int s = 0; s < 2; s++) {
                const int32_t v = ed[2 * I + s];
                bound += ctx->h_inc_off[v + 1] - ctx->h_inc_off[v] + 1;
            }
        if (E < 8 || bound > 32 * (int64_t)E + 4096) {
            ctx->ev_state = 2;
        } else {
            std::vector<int32_t> slot((size_t)V, -1), vid;
            for (int32_t v = 0; v < V; v++)
                if (ctx->h_inc_off[v + 1] > ctx->h_inc_off[v]) {
                    slot[v] = (int32_t)vid.size();
                    vid.push_back(v);
                }
            const int32_t VA = (int32_t)vid.size();
            std::vector<int32_t> near_off((size_t)E + 1, 0), near, rev_off((size_t)VA + 1, 0), rev;
            near.reserve((size_t)bound);
            for (int32_t I = 0; I < E; I++) {
                const size_t b = near.size();
                for (int s = 0; s < 2; s++) {
                    const int32_t v = ed[2 * I + s];
                    near.push_back(slot[v]);
                    for (int32_t k = ctx->h_inc_off[v]; k < ctx->h_inc_off[v + 1]; k++) {
                        const int32_t h = ctx->h_inc[k];
                        near.push_back(slot[ed[2 * (h >> 1) + 1 - (h & 1)]]);
                    }
                }
                std::sort(near.begin() + b, near.end());
                near.erase(std::unique(near.begin() + b, near.end()), near.end());
                near_off[I + 1] = (int32_t)near.size();
            }
            auto on = [&](int32_t I, int32_t v) { return slot[ed[2 * I]] == v || slot[ed[2 * I + 1]] == v; };
            for (int32_t I = 0; I < E; I++)
                for (int32_t k = near_off[I]; k < near_off[I + 1]; k++)
                    if (!on(I, near[k])) rev_off[near[k] + 1]++;
            for (int32_t v = 0; v < VA; v++) rev_off[v + 1] += rev_off[v];
            rev.assign((size_t)rev_off[VA], 0);
            std::vector<int32_t> fill(rev_off.begin(), rev_off.end() - 1);
            for (int32_t I = 0; I < E; I++)
                for (int32_t k = near_off[I]; k < near_off[I + 1]; k++)
                    if (!on(I, near[k])) rev[fill[near[k]]++] = I;
            std::vector<int32_t> all((size_t)2 * E);
            for (int64_t i = 0; i < 2 * (int64_t)E; i++) all[i] = slot[ed[i]];
            const std::vector<int32_t>* parts[] = {&near_off, &near, &rev_off, &rev, &vid, &slot};
            for (int p = 0; p < 6; p++) {
                ctx->ev_at[p] = (int64_t)all.size();
                all.insert(all.end(), parts[p]->begin(), parts[p]->end());
            }
            TPE_TRY(ensure(ctx, ctx->ev_lists, sizeof(int32_t) * all.size()));
            TPE_CUDA_TRY(cudaMemcpyAsync(ctx->ev_lists.ptr, all.data(), sizeof(int32_t) * all.size(),
                                         cudaMemcpyHostToDevice, ctx->stream));
            TPE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
            ctx->ev_VA = VA;
            ctx->ev_state = 1;
        }
    }
    *ok = ctx->ev_state == 1;
    return TPE_OK;
}

// The edge and vertex records of ncurves position sets.
int32_t ev_prep(tpe_ctx* ctx, const double* d_pos, int32_t ncurves, double eps, double alpha) {
    TPE_TRY(ensure(ctx, ctx->ev_vert, sizeof(double4) * (size_t)ctx->ev_VA * ncurves));
    const int64_t n = ((int64_t)ctx->E + ctx->ev_VA) * ncurves;
    KernelScope ks(ctx, TPE_KGROUP_OTHER, 1);
    ev_prep_kernel<<<(unsigned)((n + 127) / 128), 128, 0, ctx->stream>>>(
        d_pos, topo_of(ctx), ctx->V, ncurves, eps, alpha, ctx->edge_a.as<double4>(),
        ctx->edge_b.as<double4>(), ctx->ev_vert.as<double4>());
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

namespace {
template <int MODE>
int32_t energy_launch(tpe_ctx* ctx, int32_t ncurves, const EvSplit& s, double alpha, double beta,
                      double eps) {
    const dim3 grid((unsigned)((s.nch + s.group - 1) / s.group), (unsigned)s.nib, (unsigned)ncurves);
    auto kern = s.R == 2 ? ev_kernel<MODE, 2, false> : ev_kernel<MODE, 1, false>;
    kern<<<grid, kW, 0, ctx->stream>>>(ctx->edge_a.as<double4>(), ctx->edge_b.as<double4>(),
                                       ctx->ev_vert.as<double4>(), topo_of(ctx), s.chunk, s.nch, s.group,
                                       alpha, beta, eps, nullptr, nullptr, ctx->partial.as<double>());
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

template <int MODE>
int32_t grad_launch(tpe_ctx* ctx, const EvSplit& s, double alpha, double beta, double eps,
                    double* d_grad, int32_t max_blocks) {
    const EvTopo t = topo_of(ctx);
    const double4 *ea = ctx->edge_a.as<double4>(), *eb = ctx->edge_b.as<double4>(),
                  *vr = ctx->ev_vert.as<double4>();
    double* acc = ctx->edge_acc.as<double>();
    double* vacc = acc + (size_t)s.nch * kAcc * t.E;
    vacc += (reinterpret_cast<uintptr_t>(vacc) >> 3) & 1;  // 16-byte rows
    double* ef = vacc + (size_t)s.nib * t.VA * 4;
    if (max_blocks > 0) {
        TPE_TRY(ensure(ctx, ctx->grad_ctr, sizeof(int32_t)));
        TPE_CUDA_TRY(cudaMemsetAsync(ctx->grad_ctr.ptr, 0, sizeof(int32_t), ctx->stream));
        const int32_t items = s.nib * s.nch;
        const size_t smem = sizeof(EvSmem) * kWorkers;
        const unsigned nb = (unsigned)std::min<int64_t>(max_blocks, (items + kWorkers - 1) / kWorkers);
        auto kern = s.R == 2 ? ev_persist_kernel<MODE, 2> : ev_persist_kernel<MODE, 1>;
        TPE_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<nb, kW * kWorkers, smem, ctx->stream>>>(ea, eb, vr, t, s.chunk, s.nch, items, alpha, beta,
                                                       eps, acc, vacc, ctx->grad_ctr.as<int32_t>());
    } else {
        const dim3 grid((unsigned)s.nch, (unsigned)s.nib, 1);
        auto kern = s.R == 2 ? ev_kernel<MODE, 2, true> : ev_kernel<MODE, 1, true>;
        kern<<<grid, kW, 0, ctx->stream>>>(ea, eb, vr, t, s.chunk, s.nch, 1, alpha, beta, eps, acc, vacc, nullptr);
    }
    TPE_CUDA_TRY(cudaGetLastError());
    ev_edge_kernel<MODE><<<(unsigned)((t.E + 31) / 32), 256, 0, ctx->stream>>>(
        ea, eb, vr, t, s.nch, s.nib, alpha, beta, eps, acc, vacc, ef, ctx->partial.as<double>());
    TPE_CUDA_TRY(cudaGetLastError());
    if (d_grad) {
        ev_vertex_kernel<MODE><<<(unsigned)((ctx->V + 31) / 32), 256, 0, ctx->stream>>>(
            ea, eb, t, s.nib, ctx->V, ctx->ev_lists.as<int32_t>() + ctx->ev_at[5], vr, alpha, beta, eps,
            vacc, ef, d_grad);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    return TPE_OK;
}
}  // namespace

// Energies of ncurves prepared curves: partials to ctx->partial, *nparts per curve.
int32_t ev_energy(tpe_ctx* ctx, int32_t ncurves, double alpha, double beta, double eps,
                  int32_t* nparts) {
    const EvSplit s = ev_split(ctx, ncurves);
    *nparts = s.nib * s.nch;
    TPE_TRY(ensure(ctx, ctx->partial, sizeof(double) * (size_t)*nparts * ncurves));
    return exp_mode(alpha, beta) ? energy_launch<1>(ctx, ncurves, s, alpha, beta, eps)
                                 : energy_launch<0>(ctx, ncurves, s, alpha, beta, eps);
}

// Gradient of the prepared curve; the edges' shares of 8 E to ctx->partial (E of them).
int32_t ev_gradient(tpe_ctx* ctx, double alpha, double beta, double eps, double* d_grad,
                    int32_t max_blocks) {
    const EvSplit s = ev_split(ctx, 1);
    const size_t n = (size_t)s.nch * kAcc * ctx->E + (size_t)s.nib * ctx->ev_VA * 4 + 6 * (size_t)ctx->E + 2;
    TPE_TRY(ensure(ctx, ctx->edge_acc, sizeof(double) * n));
    TPE_TRY(ensure(ctx, ctx->partial, sizeof(double) * (size_t)ctx->E));
    return exp_mode(alpha, beta) ? grad_launch<1>(ctx, s, alpha, beta, eps, d_grad, max_blocks)
                                 : grad_launch<0>(ctx, s, alpha, beta, eps, d_grad, max_blocks);
}

}  // namespace tpe
