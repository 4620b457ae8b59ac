// Barnes-Hut tangent-point energy: the hierarchical path for curves far larger
// than the dense O(E^2) kernels serve.
//
// The algorithm is the reference's stage-2 oracle (oracle/tpe_stage2_oracle.py):
// an edge bounding-volume tree (build_edge_bvh, :467-502) and a per-target-edge
// traversal (bh_energy, :532-589) with its admissibility rule (:556-557): a
// node of at least two edges, none of which shares a vertex with the target
// edge I, whose spatial radius over the distance from I's midpoint is at most
// theta and whose tangent radius is at most theta_t (default 1.5 theta). An
// admissible node replaces its edges by one source point at its mass-weighted
// center (bh_ordered_cluster_term, :515-529); a leaf that is not admissible is
// summed exactly. theta = 0 admits nothing and gives the exact energy.
//
// The energy's tree is built on the device (1300 to 2^19 edges, leaves up to 512; on the
// host otherwise, and for the block cluster tree), in the oracle's order of operations,
// so that it is the same tree: split on the coordinate of largest
// spread of the 6-D points (midpoint, unit tangent), stable sort, the first
// half (rounded down) to the left; node centers, tangents and masses summed as
// numpy sums them (sequential along the rows, pairwise for the mass). Node
// edges are stored as one contiguous range of a permutation of the edges, so
// "does node n contain edge J" is a range test on J's position. The device
// walks the tree once per target edge (one thread each, explicit stack) and
// writes that edge's sum and counts; the totals are reduced in a fixed order.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <thread>
#include <utility>
#include <vector>

#include "tpe_internal.h"

namespace tpe {
namespace {

constexpr double kTangentTol = 1e-14;  // TANGENT_TOL of the stage-2 oracle (:34)
constexpr int kStack = 64;             // traversal depth bound (a median tree of 2^31 edges is 32 deep)

struct Node {
    double cx, cy, cz;  // mass-weighted center of the node's edge midpoints
    double mass;        // sum of ell_eps over the node's edges
    double rx, rT;      // max distance of a midpoint (unit tangent) from the center (mean tangent)
    double tx, ty, tz;  // mass-weighted mean of the unit tangents
    int32_t begin, count;  // the node's edges: perm[begin .. begin + count)
    int32_t left, right;   // children, -1 for a leaf
    int32_t parent, pad;
};

// numpy's pairwise summation of a contiguous float64 array (np.sum).
double np_pairwise_sum(const double* a, size_t n) {
    if (n < 8) {
        double s = 0.0;
        for (size_t i = 0; i < n; i++) s += a[i];
        return s;
    }
    if (n <= 128) {
        double r[8];
        for (int j = 0; j < 8; j++) r[j] = a[j];
        size_t i = 8;
        for (; i < n - (n % 8); i += 8)
            for (int j = 0; j < 8; j++) r[j] += a[i + j];
        double res = ((r[0] + r[1]) + (r[2] + r[3])) + ((r[4] + r[5]) + (r[6] + r[7]));
        for (; i < n; i++) res += a[i];
        return res;
    }
    size_t n2 = n / 2;
    n2 -= n2 % 8;
    return np_pairwise_sum(a, n2) + np_pairwise_sum(a + n2, n - n2);
}

inline double norm3(double x, double y, double z) { return std::sqrt((x * x + y * y) + z * z); }

using Keyed = std::vector<std::pair<double, int32_t>>;

// std::stable_sort on the key, with the range cut into up to `threads` pieces
// sorted on their own threads and merged pairwise (std::merge takes from the
// first range on ties, so the order is the same stable order).
void stable_sort_keys(Keyed& a, int threads) {
    auto less = [](const std::pair<double, int32_t>& x, const std::pair<double, int32_t>& y) {
        return x.first < y.first;
    };
    const size_t n = a.size();
    int p = 1;
    while (p * 2 <= threads && n / (size_t)(p * 2) >= 16384) p *= 2;
    if (p == 1) {
        std::stable_sort(a.begin(), a.end(), less);
        return;
    }
    std::vector<size_t> cut((size_t)p + 1);
    for (int i = 0; i <= p; i++) cut[i] = n * (size_t)i / (size_t)p;
    auto run = [&](std::vector<std::thread>& th, auto&& body, int count) {
        try {
            for (int i = 0; i < count; i++) th.emplace_back(body, i);
        } catch (...) {
            for (auto& t : th) t.join();
            throw;
        }
        for (auto& t : th) t.join();
    };
    {
        std::vector<std::thread> th;
        run(th, [&](int i) { std::stable_sort(a.begin() + cut[i], a.begin() + cut[i + 1], less); }, p);
    }
    Keyed b(n);
    for (int w = 1; w < p; w *= 2) {
        std::vector<std::thread> th;
        const int pairs = p / (2 * w);
        run(th,
            [&](int j) {
                const size_t lo = cut[2 * w * j], mid = cut[2 * w * j + w], hi = cut[2 * w * (j + 1)];
                std::merge(a.begin() + lo, a.begin() + mid, a.begin() + mid, a.begin() + hi,
                           b.begin() + lo, less);
            },
            pairs);
        a.swap(b);
    }
}

struct Builder {
    const std::vector<double>& C;  // E x 3 midpoints
    const std::vector<double>& T;  // E x 3 unit tangents
    const std::vector<double>& m;  // E masses (ell_eps)
    int32_t leaf;
    int32_t* perm;                 // shared; a builder writes only its own ranges
    std::vector<Node> nodes;
    std::vector<double> tmp;
    Keyed keyed;
    int sort_threads = 1;  // threads for the sort of one node (the top levels)
    // subtrees at depth split_depth are left to other builders: (begin, count,
    // parent node, is-left) each, the parent's child link holding -2 - task
    int32_t split_depth = -1;
    struct Task {
        int32_t begin, count, parent;
        bool left;
    };
    std::vector<Task> tasks;

    int32_t rec(int32_t begin, int32_t count, int32_t depth = 0) {
        const int32_t* idx = perm + begin;
        tmp.resize((size_t)count);
        for (int32_t k = 0; k < count; k++) tmp[k] = m[idx[k]];
        const double msum = np_pairwise_sum(tmp.data(), (size_t)count);
        double c[3] = {0, 0, 0}, t[3] = {0, 0, 0};
        for (int32_t k = 0; k < count; k++) {
            const int32_t J = idx[k];
            for (int d = 0; d < 3; d++) {
                c[d] = c[d] + m[J] * C[3 * (size_t)J + d];
                t[d] = t[d] + m[J] * T[3 * (size_t)J + d];
            }
        }
        for (int d = 0; d < 3; d++) {
            c[d] = c[d] / msum;
            t[d] = t[d] / msum;
        }
        double rx = 0.0, rT = 0.0;
        for (int32_t k = 0; k < count; k++) {
            const int32_t J = idx[k];
            rx = std::max(rx, norm3(C[3 * (size_t)J] - c[0], C[3 * (size_t)J + 1] - c[1],
                                    C[3 * (size_t)J + 2] - c[2]));
            rT = std::max(rT, norm3(T[3 * (size_t)J] - t[0], T[3 * (size_t)J + 1] - t[1],
                                    T[3 * (size_t)J + 2] - t[2]));
        }
        const int32_t me = (int32_t)nodes.size();
        nodes.push_back(Node{c[0], c[1], c[2], msum, rx, rT, t[0], t[1], t[2], begin, count, -1, -1, -1, 0});
        if (count > leaf) {
            // the coordinate of largest spread (first on ties), stable sort on it
            double lo[6], hi[6];
            for (int d = 0; d < 6; d++) {
                lo[d] = INFINITY;
                hi[d] = -INFINITY;
            }
            for (int32_t k = 0; k < count; k++) {
                const int32_t J = idx[k];
                for (int d = 0; d < 6; d++) {
                    const double x = d < 3 ? C[3 * (size_t)J + d] : T[3 * (size_t)J + d - 3];
                    lo[d] = std::min(lo[d], x);
                    hi[d] = std::max(hi[d], x);
                }
            }
            int dim = 0;
            double best = hi[0] - lo[0];
            for (int d = 1; d < 6; d++)
                if (hi[d] - lo[d] > best) {
                    best = hi[d] - lo[d];
                    dim = d;
                }
            const std::vector<double>& X = dim < 3 ? C : T;
            const int dd = dim % 3;
            keyed.resize((size_t)count);
            for (int32_t k = 0; k < count; k++) keyed[k] = {X[3 * (size_t)idx[k] + dd], idx[k]};
            stable_sort_keys(keyed, sort_threads);
            for (int32_t k = 0; k < count; k++) perm[begin + k] = keyed[k].second;
            const int32_t mid = count / 2;
            int32_t l, r;
            if (depth + 1 == split_depth) {
                tasks.push_back({begin, mid, me, true});
                l = -2 - (int32_t)(tasks.size() - 1);
                tasks.push_back({begin + mid, count - mid, me, false});
                r = -2 - (int32_t)(tasks.size() - 1);
            } else {
                l = rec(begin, mid, depth + 1);
                r = rec(begin + mid, count - mid, depth + 1);
                nodes[l].parent = me;
                nodes[r].parent = me;
            }
            nodes[me].left = l;
            nodes[me].right = r;
        }
        return me;
    }
};

// |e x d|^alpha / |d|^beta, each with eps added to the length; k36: exponents 3 and 6.
template <bool k36>
__device__ __forceinline__ double term(double ex, double ey, double ez, double dx, double dy,
                                       double dz, double alpha, double beta, double eps) {
    const double cx = ey * dz - ez * dy, cy = ez * dx - ex * dz, cz = ex * dy - ey * dx;
    const double dn = sqrt((dx * dx + dy * dy) + dz * dz) + eps;
    const double cn = sqrt((cx * cx + cy * cy) + cz * cz) + eps;
    if constexpr (k36) {
        const double d2 = dn * dn;
        return cn * cn * cn / (d2 * d2 * d2);
    }
    return pow(cn, alpha) / pow(dn, beta);
}

// One thread per target edge I: its ordered sum over the tree, and the visit,
// approximated-edge and direct-pair counts.
template <bool k36>
__global__ void __launch_bounds__(128)
bh_energy_kernel(const double* __restrict__ pos, const int2* __restrict__ edges, int32_t E,
                 const Node* __restrict__ nodes, const int32_t* __restrict__ perm,
                 const int32_t* __restrict__ where, const int32_t* __restrict__ inc_off,
                 const int32_t* __restrict__ inc, double alpha, double beta, double eps,
                 double theta, double theta_t, double* __restrict__ out,
                 long long* __restrict__ counts, int32_t* __restrict__ err) {
    const int32_t I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= E) return;
    const int2 eI = edges[I];
    const double ax = pos[3 * eI.x], ay = pos[3 * eI.x + 1], az = pos[3 * eI.x + 2];
    const double bx = pos[3 * eI.y], by = pos[3 * eI.y + 1], bz = pos[3 * eI.y + 2];
    const double ex = bx - ax, ey = by - ay, ez = bz - az;
    const double ellI = sqrt((ex * ex + ey * ey) + ez * ez) + eps;
    const double pI = pow(ellI, 1.0 - alpha);
    const double mx = 0.5 * (ax + bx), my = 0.5 * (ay + by), mz = 0.5 * (az + bz);
    double val = 0.0;
    long long visits = 0, approx = 0, direct = 0;
    int32_t stack[kStack];
    int sp = 0;
    stack[sp++] = 0;
    while (sp > 0) {
        const Node nd = nodes[stack[--sp]];
        visits++;
        const double dist = sqrt(((mx - nd.cx) * (mx - nd.cx) + (my - nd.cy) * (my - nd.cy)) +
                                 (mz - nd.cz) * (mz - nd.cz));
        bool admiss = nd.count >= 2 && dist > 0.0 && nd.rx / dist <= theta && nd.rT <= theta_t;
        if (admiss) {
            // no edge of the node may share a vertex with I (I itself included)
            for (int s = 0; s < 2 && admiss; s++) {
                const int32_t v = s ? eI.y : eI.x;
                for (int32_t q = inc_off[v]; q < inc_off[v + 1]; q++) {
                    const int32_t w = where[inc[q] >> 1];
                    if (w >= nd.begin && w < nd.begin + nd.count) {
                        admiss = false;
                        break;
                    }
                }
            }
        }
        if (admiss) {
            approx += nd.count;
            const double s = term<k36>(ex, ey, ez, ax - nd.cx, ay - nd.cy, az - nd.cz, alpha, beta, eps) +
                             term<k36>(ex, ey, ez, bx - nd.cx, by - nd.cy, bz - nd.cz, alpha, beta, eps);
            val += 0.5 * pI * nd.mass * s;
        } else if (nd.left < 0) {
            for (int32_t k = nd.begin; k < nd.begin + nd.count; k++) {
                const int32_t J = perm[k];
                const int2 eJ = edges[J];
                if (J == I || eJ.x == eI.x || eJ.x == eI.y || eJ.y == eI.x || eJ.y == eI.y) continue;
                direct++;
                const double cx = pos[3 * eJ.x], cy = pos[3 * eJ.x + 1], cz = pos[3 * eJ.x + 2];
                const double dx = pos[3 * eJ.y], dy = pos[3 * eJ.y + 1], dz = pos[3 * eJ.y + 2];
                const double fx = dx - cx, fy = dy - cy, fz = dz - cz;
                const double ellJ = sqrt((fx * fx + fy * fy) + fz * fz) + eps;
                const double s = term<k36>(ex, ey, ez, ax - cx, ay - cy, az - cz, alpha, beta, eps) +
                                 term<k36>(ex, ey, ez, ax - dx, ay - dy, az - dz, alpha, beta, eps) +
                                 term<k36>(ex, ey, ez, bx - cx, by - cy, bz - cz, alpha, beta, eps) +
                                 term<k36>(ex, ey, ez, bx - dx, by - dy, bz - dz, alpha, beta, eps);
                val += 0.25 * pI * ellJ * s;
            }
        } else {
            if (sp + 2 > kStack) {
                atomicExch(err, 1);
                break;
            }
            stack[sp++] = nd.right;
            stack[sp++] = nd.left;
        }
    }
    out[I] = val;
    counts[3 * (size_t)I] = visits;
    counts[3 * (size_t)I + 1] = approx;
    counts[3 * (size_t)I + 2] = direct;
}

// Fixed-order totals in two launches: kRedPer edges a block, then the blocks' sums by one
// (224 us as one block over 131072 edges, 10 as two launches).
constexpr int kRedPer = 1024;
__global__ void __launch_bounds__(256)
bh_reduce_kernel(const double* __restrict__ val, const long long* __restrict__ counts, int32_t E,
                 double* __restrict__ total, long long* __restrict__ ctot, double scale, int32_t per) {
    __shared__ double sv[256];
    __shared__ long long sc[3][256];
    double v = 0.0;
    long long c0 = 0, c1 = 0, c2 = 0;
    const int32_t i0 = (int32_t)blockIdx.x * per, i1 = min(E, i0 + per);
    for (int32_t i = i0 + threadIdx.x; i < i1; i += 256) {
        v += val[i];
        c0 += counts[3 * (size_t)i];
        c1 += counts[3 * (size_t)i + 1];
        c2 += counts[3 * (size_t)i + 2];
    }
    sv[threadIdx.x] = v;
    sc[0][threadIdx.x] = c0;
    sc[1][threadIdx.x] = c1;
    sc[2][threadIdx.x] = c2;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            sv[threadIdx.x] += sv[threadIdx.x + s];
            for (int q = 0; q < 3; q++) sc[q][threadIdx.x] += sc[q][threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        total[blockIdx.x] = scale * sv[0];
        for (int q = 0; q < 3; q++) ctot[3 * (size_t)blockIdx.x + q] = sc[q][0];
    }
}

// ---- the same tree, built on the device ------------------------------------------------
//
// A node's halves depend on its count alone, so the tree's shape is known in advance: node
// `idx` of level l is entry 2^l - 1 + idx, its children 2i + 1 and 2i + 2. Every value is
// rounded as the host builder rounds it (no contraction, sums in the same order), so both
// give the same nodes.
//   top levels (nodes of more than kSubtree edges): per level the dimension of largest
//     spread, and a bitonic sort of (coordinate, position), which is the stable order;
//     then one launch for the statistics of all their nodes;
//   below: one block per subtree, its edges in shared memory, all levels in one launch.
// 131072 edges: a call takes 2.4 ms (23.6 with the host's tree, 19 of them its build and
// copies): 1.6 the tree, 0.7 the traversal, whose powers are products at exponents 3
// and 6 (2.35 with pow). Bound: the sort's 84 small launches, 0.9 ms, beside which the
// root's sums run, one addition after the other (0.6 ms, 9 clocks each).
constexpr int kSubtree = 1024;
constexpr int kSubThr = 512;
constexpr int kTile = 2048;  // elements sorted in shared memory at the top levels
constexpr int kSeq = 992;    // a chunk of the sequential sums (31 warps fetch, one adds)
// Below 1300 edges the host's tree with its copies is the sooner one (a call, us, device / host:
// smooth curves of 500 edges 408 / 352, 1000 568 / 484, 1500 564 / 531, 2000 587 / 598; random
// walks 814 / 792, 1459 / 1498, 2224 / 2398, 2808 / 3134).
constexpr int32_t kDeviceTreeFrom = 1300;
constexpr int32_t kDeviceTreeEdges = 1 << 19;
constexpr int kDeviceTreeLeaf = 512;
constexpr int kPairDepth = 13;  // halvings until 2^19 terms are at most 128

struct DevTree {
    const double* pos;
    const int2* edges;
    int32_t E, leaf, top;  // `top` levels above the subtrees
    double eps;
    double *X, *m;   // 6 x E (midpoint, unit tangent) and E, by edge
    int32_t* perm;   // (top + 1) x E: the edges in order at each level
    unsigned long long* key;
    int32_t* ord;    // positions, sorted with their keys
    double* sums;    // 7 per top node: the six weighted sums and the mass
    unsigned long long* spread;  // 12 per top node (tree_spread_kernel)
    Node* nodes;
    int32_t *final_perm, *where;
};

// Edges [begin, begin + count) of node idx of a level (count = 0: its parent is a leaf).
__device__ __forceinline__ int2 span_of(int32_t begin, int32_t count, int32_t leaf, int level, int32_t idx) {
    for (int q = level - 1; q >= 0; q--) {
        if (count <= leaf) return make_int2(begin, 0);
        const int32_t l = count / 2;
        if ((idx >> q) & 1) {
            begin += l;
            count -= l;
        } else {
            count = l;
        }
    }
    return make_int2(begin, count);
}

// x's place in the order of doubles (-0 as +0).
__device__ __forceinline__ unsigned long long order_key(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(__dadd_rn(x, 0.0));
    return b >> 63 ? ~b : b | (1ull << 63);
}

__device__ __forceinline__ double norm3_sq(double x, double y, double z) {
    return __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
}

__global__ void tree_edges_kernel(const DevTree t) {
    const int32_t I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= t.E) return;
    const int2 e = t.edges[I];
    double d[3];
    for (int q = 0; q < 3; q++) {
        const double a = t.pos[3 * (size_t)e.x + q], b = t.pos[3 * (size_t)e.y + q];
        d[q] = __dsub_rn(b, a);
        t.X[(size_t)q * t.E + I] = __dmul_rn(0.5, __dadd_rn(a, b));
    }
    const double ell = __dsqrt_rn(norm3_sq(d[0], d[1], d[2]));
    for (int q = 0; q < 3; q++)
        t.X[(size_t)(3 + q) * t.E + I] = ell >= kTangentTol ? __ddiv_rn(d[q], ell) : 0.0;
    t.m[I] = __dadd_rn(ell, t.eps);
    t.perm[I] = I;
}

__device__ __forceinline__ double key_value(unsigned long long k) {
    return __longlong_as_double((long long)(k >> 63 ? k & ~(1ull << 63) : ~k));
}

// Spreads of a top level's nodes: per node and coordinate the largest key and the largest
// complement (of the smallest), from zeros. kKeysPer edges a block.
constexpr int kKeysPer = 2048;
__global__ void __launch_bounds__(256) tree_spread_kernel(const DevTree t, int level) {
    const int2 s = span_of(0, t.E, t.leaf, level, blockIdx.y);
    const int32_t* perm = t.perm + (size_t)level * t.E;
    __shared__ double red[12][8];
    double lo[6], hi[6];
    for (int d = 0; d < 6; d++) {
        lo[d] = INFINITY;
        hi[d] = -INFINITY;
    }
    const int32_t k0 = s.x + blockIdx.x * kKeysPer, k1 = min(s.x + s.y, k0 + kKeysPer);
    for (int32_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        const int32_t J = perm[k];
        for (int d = 0; d < 6; d++) {
            const double x = t.X[(size_t)d * t.E + J];
            lo[d] = fmin(lo[d], x);
            hi[d] = fmax(hi[d], x);
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int d = 0; d < 6; d++) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[d] = fmin(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = fmax(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
        if (lane == 0) {
            red[d][w] = lo[d];
            red[6 + d][w] = hi[d];
        }
    }
    __syncthreads();
    if (threadIdx.x >= 12 || k0 >= k1) return;
    double x = red[threadIdx.x][0];
    for (int q = 1; q < 8; q++) x = threadIdx.x < 6 ? fmin(x, red[threadIdx.x][q]) : fmax(x, red[threadIdx.x][q]);
    const unsigned long long k = order_key(x);
    atomicMax(t.spread + 12 * ((size_t)(1 << level) - 1 + blockIdx.y) + threadIdx.x, threadIdx.x < 6 ? ~k : k);
}
// The sort keys of a top level: the coordinate of largest spread, the first on ties.
__global__ void __launch_bounds__(256) tree_keys_kernel(const DevTree t, int level) {
    const int2 s = span_of(0, t.E, t.leaf, level, blockIdx.y);
    const int32_t* perm = t.perm + (size_t)level * t.E;
    const unsigned long long* sp = t.spread + 12 * ((size_t)(1 << level) - 1 + blockIdx.y);
    int dim = 0;
    double best = 0.0;
    for (int d = 0; d < 6; d++) {
        const double width = __dsub_rn(key_value(sp[6 + d]), key_value(~sp[d]));
        if (d == 0 || width > best) {
            best = width;
            dim = d;
        }
    }
    const double* x = t.X + (size_t)dim * t.E;
    const int32_t k0 = s.x + blockIdx.x * kKeysPer, k1 = min(s.x + s.y, k0 + kKeysPer);
    for (int32_t k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        t.key[k] = order_key(x[perm[k]]);
        t.ord[k] = k;
    }
}

__device__ __forceinline__ bool after(unsigned long long ka, int32_t oa, unsigned long long kb, int32_t ob) {
    return ka > kb || (ka == kb && oa > ob);
}
// Pair p of a bitonic step (every comparison ascending, so that places beyond the end are
// as good as filled with the largest key): the mirror step of blocks of k, or distance h.
__device__ __forceinline__ int2 mirror_pair(int32_t p, int32_t k) {
    const int32_t b = p / (k / 2) * k, o = p % (k / 2);
    return make_int2(b + o, b + k - 1 - o);
}
__device__ __forceinline__ int2 distance_pair(int32_t p, int32_t h) {
    const int32_t i = p / h * 2 * h + p % h;
    return make_int2(i, i + h);
}

// One step of all nodes of a level: block k's mirror step (h = 0) or distance h.
__global__ void tree_step_kernel(const DevTree t, int level, int32_t k, int32_t h) {
    const int2 s = span_of(0, t.E, t.leaf, level, blockIdx.y);
    const int2 p = h ? distance_pair(blockIdx.x * blockDim.x + threadIdx.x, h)
                     : mirror_pair(blockIdx.x * blockDim.x + threadIdx.x, k);
    if (p.y >= s.y) return;
    const int32_t a = s.x + p.x, b = s.x + p.y;
    const unsigned long long ka = t.key[a], kb = t.key[b];
    const int32_t oa = t.ord[a], ob = t.ord[b];
    if (!after(ka, oa, kb, ob)) return;
    t.key[a] = kb, t.key[b] = ka;
    t.ord[a] = ob, t.ord[b] = oa;
}

// The steps within tiles of kTile: from nothing (k0 = 2), or the rest of merge k0.
__global__ void __launch_bounds__(kTile / 2) tree_tile_kernel(const DevTree t, int level, int32_t k0) {
    __shared__ unsigned long long key[kTile];
    __shared__ int32_t ord[kTile];
    const int2 s = span_of(0, t.E, t.leaf, level, blockIdx.y);
    const int32_t t0 = s.x + blockIdx.x * kTile, n = min(kTile, s.y - (int32_t)blockIdx.x * kTile);
    if (n <= 0) return;
    for (int32_t e = threadIdx.x; e < n; e += blockDim.x) {
        key[e] = t.key[t0 + e];
        ord[e] = t.ord[t0 + e];
    }
    auto exchange = [&](int2 p) {
        __syncthreads();
        if (p.y < n && after(key[p.x], ord[p.x], key[p.y], ord[p.y])) {
            const unsigned long long k = key[p.x];
            const int32_t o = ord[p.x];
            key[p.x] = key[p.y], key[p.y] = k;
            ord[p.x] = ord[p.y], ord[p.y] = o;
        }
    };
    if (k0 > kTile) {
        for (int32_t h = kTile / 2; h > 0; h /= 2) exchange(distance_pair(threadIdx.x, h));
    } else {
        for (int32_t k = 2; k <= kTile; k *= 2) {
            exchange(mirror_pair(threadIdx.x, k));
            for (int32_t h = k / 4; h > 0; h /= 2) exchange(distance_pair(threadIdx.x, h));
        }
    }
    __syncthreads();
    for (int32_t e = threadIdx.x; e < n; e += blockDim.x) {
        t.key[t0 + e] = key[e];
        t.ord[t0 + e] = ord[e];
    }
}

__global__ void tree_order_kernel(const DevTree t, int level) {
    const int32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < t.E) t.perm[(size_t)(level + 1) * t.E + k] = t.perm[(size_t)level * t.E + t.ord[k]];
}

// np_pairwise_sum of at most 128 terms get(0 .. n - 1).
template <class F>
__device__ __forceinline__ double pairwise_base(F&& get, int32_t n) {
    if (n < 8) {
        double s = 0.0;
        for (int32_t i = 0; i < n; i++) s = __dadd_rn(s, get(i));
        return s;
    }
    double r[8];
    for (int j = 0; j < 8; j++) r[j] = get(j);
    int32_t i = 8;
    for (; i < n - n % 8; i += 8)
        for (int j = 0; j < 8; j++) r[j] = __dadd_rn(r[j], get(i + j));
    double s = __dadd_rn(__dadd_rn(__dadd_rn(r[0], r[1]), __dadd_rn(r[2], r[3])),
                         __dadd_rn(__dadd_rn(r[4], r[5]), __dadd_rn(r[6], r[7])));
    for (; i < n; i++) s = __dadd_rn(s, get(i));
    return s;
}
// The piece at `path` (its first `depth` halvings, first one in the top bit) of np_pairwise_sum's
// recursion over n terms: (first, count), count 0 where the recursion ended before.
__device__ __forceinline__ int2 pairwise_piece(int32_t n, int32_t path, int depth) {
    int32_t at = 0;
    for (int q = depth - 1; q >= 0; q--) {
        const bool right = (path >> q) & 1;
        if (n <= 128) {
            if (right) return make_int2(at, 0);
            continue;
        }
        int32_t l = n / 2;
        l -= l % 8;
        if (right) {
            at += l;
            n -= l;
        } else {
            n = l;
        }
    }
    return make_int2(at, n);
}

// The sequential sums (y = 0) and the pairwise mass (y = 1) of each top node.
__global__ void __launch_bounds__(1024) tree_sums_kernel(const DevTree t, int32_t first) {
    extern __shared__ __align__(16) double buf[];
    const int32_t node = first + (int32_t)blockIdx.x;
    const int level = 31 - __clz(node + 1);
    const int2 s = span_of(0, t.E, t.leaf, level, node + 1 - (1 << level));
    const int32_t* perm = t.perm + (size_t)level * t.E + s.x;
    double* out = t.sums + 7 * (size_t)node;
    if (blockIdx.y == 0) {
        constexpr int kRow = kSeq + 1;
        auto fetch = [&](int32_t c) {
            const int32_t e = (int32_t)threadIdx.x - 32, k = c * kSeq + e;
            if (e < 0 || k >= s.y) return;
            const int32_t J = perm[k];
            const double mass = t.m[J];
            for (int d = 0; d < 6; d++)
                buf[((c & 1) * 6 + d) * kRow + e] = __dmul_rn(mass, t.X[(size_t)d * t.E + J]);
        };
        double sum = 0.0;
        fetch(0);
        for (int32_t c = 0; c * kSeq < s.y; c++) {
            __syncthreads();
            fetch(c + 1);
            if (threadIdx.x < 6) {
                const double* row = buf + ((c & 1) * 6 + threadIdx.x) * kRow;
                const int32_t n = min(kSeq, s.y - c * kSeq);
                int32_t k = 0;
                for (; k + 16 <= n; k += 16) {
                    double x[16];
#pragma unroll
                    for (int q = 0; q < 16; q++) x[q] = row[k + q];
#pragma unroll
                    for (int q = 0; q < 16; q++) sum = __dadd_rn(sum, x[q]);
                }
                for (; k < n; k++) sum = __dadd_rn(sum, row[k]);
            }
        }
        if (threadIdx.x < 6) out[threadIdx.x] = sum;
        return;
    }
    for (int32_t p = threadIdx.x; p < 1 << kPairDepth; p += blockDim.x) {
        const int2 r = pairwise_piece(s.y, p, kPairDepth);
        if (r.y > 0) buf[p] = pairwise_base([&](int32_t i) { return t.m[perm[r.x + i]]; }, r.y);
    }
    for (int depth = kPairDepth - 1; depth >= 0; depth--) {
        __syncthreads();
        for (int32_t p = threadIdx.x; p < 1 << depth; p += blockDim.x) {
            const int2 r = pairwise_piece(s.y, p, depth);
            if (r.y > 128) {
                const int w = 1 << (kPairDepth - depth);
                buf[p * w] = __dadd_rn(buf[p * w], buf[p * w + w / 2]);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) out[6] = buf[0];
}

__device__ __forceinline__ Node make_node(const double (&c)[6], double mass, double rx2, double rT2, int2 s,
                                          int32_t leaf, int32_t i) {
    Node nd;
    nd.cx = c[0], nd.cy = c[1], nd.cz = c[2];
    nd.tx = c[3], nd.ty = c[4], nd.tz = c[5];
    nd.mass = mass;
    nd.rx = __dsqrt_rn(rx2);  // (of the largest square: the root is monotonic)
    nd.rT = __dsqrt_rn(rT2);
    nd.begin = s.x, nd.count = s.y;
    nd.left = s.y > leaf ? 2 * i + 1 : -1;
    nd.right = s.y > leaf ? 2 * i + 2 : -1;
    nd.parent = i > 0 ? (i - 1) / 2 : -1;
    nd.pad = 0;
    return nd;
}

// Centers and radii of each top node.
__global__ void __launch_bounds__(1024) tree_top_kernel(const DevTree t) {
    const int level = 31 - __clz(blockIdx.x + 1);
    const int2 s = span_of(0, t.E, t.leaf, level, (int32_t)blockIdx.x + 1 - (1 << level));
    const int32_t* perm = t.perm + (size_t)level * t.E;
    const double* in = t.sums + 7 * (size_t)blockIdx.x;
    double c[6];
    for (int d = 0; d < 6; d++) c[d] = __ddiv_rn(in[d], in[6]);
    double r[2] = {0.0, 0.0};
    for (int32_t k = s.x + threadIdx.x; k < s.x + s.y; k += blockDim.x) {
        const int32_t J = perm[k];
        double x[6];
        for (int d = 0; d < 6; d++) x[d] = __dsub_rn(t.X[(size_t)d * t.E + J], c[d]);
        r[0] = fmax(r[0], norm3_sq(x[0], x[1], x[2]));
        r[1] = fmax(r[1], norm3_sq(x[3], x[4], x[5]));
    }
    __shared__ double red[2][32];
    for (int q = 0; q < 2; q++) {
        for (int o = 16; o > 0; o >>= 1) r[q] = fmax(r[q], __shfl_xor_sync(0xffffffffu, r[q], o));
        if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = r[q];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 0; q < 2; q++)
            for (int w = 0; w < 32; w++) r[q] = fmax(r[q], red[q][w]);
        t.nodes[blockIdx.x] = make_node(c, in[6], r[0], r[1], s, t.leaf, blockIdx.x);
    }
}

// One block per subtree of at most kSubtree edges: its nodes, level by level, and the final
// order. Shared memory: the edges' coordinates and masses, the sort's keys and positions, the
// order, and per node of a level its sums (and spreads), mass and squared radii.
struct SubSmem {
    double X[6][kSubtree], m[kSubtree];
    unsigned long long key[kSubtree];
    int32_t pos[kSubtree];         // sorted with key
    int32_t ord[2][kSubtree];      // element at each place
    double c[kSubtree][6];         // per node
    double width[kSubtree / 2][6];
    double mass[kSubtree];
    unsigned long long r2[kSubtree][2];
    int32_t dim[kSubtree / 2];
};

template <int D, class F>
__device__ double pairwise_small(F&& get, int32_t at, int32_t n) {
    if constexpr (D > 0) {
        if (n > 128) {
            int32_t l = n / 2;
            l -= l % 8;
            const double a = pairwise_small<D - 1>(get, at, l);
            return __dadd_rn(a, pairwise_small<D - 1>(get, at + l, n - l));
        }
    }
    return pairwise_base([&](int32_t i) { return get(at + i); }, n);
}

__global__ void __launch_bounds__(kSubThr) tree_sub_kernel(const DevTree t) {
    extern __shared__ __align__(16) unsigned char raw[];
    SubSmem& sm = *reinterpret_cast<SubSmem*>(raw);
    const int tid = threadIdx.x;
    const int2 root = span_of(0, t.E, t.leaf, t.top, blockIdx.x);
    const int32_t n = root.y;
    const int32_t* perm = t.perm + (size_t)t.top * t.E + root.x;
    for (int32_t e = tid; e < n; e += kSubThr) {
        const int32_t J = perm[e];
        for (int d = 0; d < 6; d++) sm.X[d][e] = t.X[(size_t)d * t.E + J];
        sm.m[e] = t.m[J];
        sm.ord[0][e] = e;
    }
    int cur = 0;
    for (int depth = 0;; depth++) {
        const int32_t nn = 1 << depth;  // nodes of this level (some may not exist)
        const int32_t* ord = sm.ord[cur];
        auto span = [&](int32_t idx) { return span_of(0, n, t.leaf, depth, idx); };
        __syncthreads();
        // sums and spreads, a thread per node and coordinate; masses, a thread per node
        // (in the upper half of the block, beside them)
        for (int32_t q = tid; tid < kSubThr / 2 && q < 6 * nn; q += kSubThr / 2) {
            const int32_t idx = q / 6, d = q % 6;
            const int2 s = span(idx);
            double sum = 0.0, lo = INFINITY, hi = -INFINITY;
#pragma unroll 4
            for (int32_t k = s.x; k < s.x + s.y; k++) {
                const int32_t e = ord[k];
                const double x = sm.X[d][e];
                sum = __dadd_rn(sum, __dmul_rn(sm.m[e], x));
                lo = fmin(lo, x);
                hi = fmax(hi, x);
            }
            sm.c[idx][d] = sum;
            if (s.y > t.leaf) sm.width[idx][d] = __dsub_rn(hi, lo);
        }
        for (int32_t idx = tid - kSubThr / 2; tid >= kSubThr / 2 && idx < nn; idx += kSubThr / 2) {
            const int2 s = span(idx);
            sm.mass[idx] = pairwise_small<5>([&](int32_t k) { return sm.m[ord[k]]; }, s.x, s.y);
            sm.r2[idx][0] = sm.r2[idx][1] = 0;
        }
        __syncthreads();
        int32_t more = 0;  // does a node of this level split
        for (int32_t q = tid; q < 6 * nn; q += kSubThr) sm.c[q / 6][q % 6] = __ddiv_rn(sm.c[q / 6][q % 6], sm.mass[q / 6]);
        for (int32_t idx = tid; idx < nn; idx += kSubThr) {
            if (span(idx).y <= t.leaf) continue;
            more = 1;
            int dim = 0;
            for (int d = 1; d < 6; d++)
                if (sm.width[idx][d] > sm.width[idx][dim]) dim = d;
            sm.dim[idx] = dim;
        }
        more = __syncthreads_or(more);
        // radii and sort keys, a thread per place
        for (int32_t k = tid; k < n; k += kSubThr) {
            int32_t idx = 0, b = 0, c = n;
            bool in = true;
            for (int q = 0; q < depth && in; q++) {
                in = c > t.leaf;
                if (!in) break;
                const int32_t l = c / 2;
                const bool right = k >= b + l;
                idx = 2 * idx + right;
                if (right) {
                    b += l;
                    c -= l;
                } else {
                    c = l;
                }
            }
            const int32_t e = ord[k];
            sm.pos[k] = k;
            if (!in) continue;
            double x[6];
            for (int d = 0; d < 6; d++) x[d] = __dsub_rn(sm.X[d][e], sm.c[idx][d]);
            const double a = norm3_sq(x[0], x[1], x[2]), g = norm3_sq(x[3], x[4], x[5]);
            if (a > 0.0) atomicMax(&sm.r2[idx][0], (unsigned long long)__double_as_longlong(a));
            if (g > 0.0) atomicMax(&sm.r2[idx][1], (unsigned long long)__double_as_longlong(g));
            if (c > t.leaf) sm.key[k] = order_key(sm.X[sm.dim[idx]][e]);
        }
        __syncthreads();
        for (int32_t idx = tid; idx < nn; idx += kSubThr) {
            const int2 s = span(idx);
            if (s.y == 0) continue;
            double c[6];
            for (int d = 0; d < 6; d++) c[d] = sm.c[idx][d];
            const int32_t i = (1 << (t.top + depth)) - 1 + ((int32_t)blockIdx.x << depth) + idx;
            t.nodes[i] = make_node(c, sm.mass[idx], __longlong_as_double((long long)sm.r2[idx][0]),
                                   __longlong_as_double((long long)sm.r2[idx][1]),
                                   make_int2(root.x + s.x, s.y), t.leaf, i);
        }
        if (!more) break;
        // sort every node that splits
        int32_t P = 2;
        while (P < (n + nn - 1) / nn) P *= 2;
        auto step = [&](int32_t k, int32_t h) {
            __syncthreads();
            for (int32_t p = tid; p < nn * (P / 2); p += kSubThr) {
                const int32_t idx = p / (P / 2);
                const int2 s = span(idx);
                if (s.y <= t.leaf) continue;
                const int2 r = h ? distance_pair(p % (P / 2), h) : mirror_pair(p % (P / 2), k);
                if (r.y >= s.y) continue;
                const int32_t a = s.x + r.x, b = s.x + r.y;
                const unsigned long long ka = sm.key[a], kb = sm.key[b];
                const int32_t pa = sm.pos[a], pb = sm.pos[b];
                if (!after(ka, pa, kb, pb)) continue;
                sm.key[a] = kb, sm.key[b] = ka;
                sm.pos[a] = pb, sm.pos[b] = pa;
            }
        };
        for (int32_t k = 2; k <= P; k *= 2) {
            step(k, 0);
            for (int32_t h = k / 4; h > 0; h /= 2) step(0, h);
        }
        __syncthreads();
        for (int32_t k = tid; k < n; k += kSubThr) sm.ord[cur ^ 1][k] = ord[sm.pos[k]];
        cur ^= 1;
    }
    for (int32_t k = tid; k < n; k += kSubThr) {
        const int32_t J = perm[sm.ord[cur][k]];
        t.final_perm[root.x + k] = J;
        t.where[J] = root.x + k;
    }
}

// Queues the build of the tree over ctx's edges at d_xyz into t (buffers set).
int32_t build_tree_device(tpe_ctx* ctx, const DevTree& t) {
    const cudaStream_t st = ctx->stream;
    const int32_t E = t.E;
    const unsigned flat = (unsigned)((E + 255) / 256);
    KernelScope ks(ctx, TPE_KGROUP_ENERGY, 2);
    const size_t smem = sizeof(double) * std::max<size_t>(12 * (kSeq + 1), (size_t)1 << kPairDepth);
    TPE_CUDA_TRY(cudaFuncSetAttribute(tree_sums_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    TPE_CUDA_TRY(cudaFuncSetAttribute(tree_sub_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(SubSmem)));
    TPE_CUDA_TRY(cudaMemsetAsync(t.spread, 0, sizeof(double) * 12 * ((size_t)1 << t.top), st));
    tree_edges_kernel<<<flat, 256, 0, st>>>(t);
    // the sums of the first levels, the longest, beside the sorting
    cudaEvent_t ev[2] = {ctx->ev_prep, ctx->ev_grad};
    const cudaStream_t side[2] = {ctx->stream2, ctx->stream3};
    const int early = std::min(t.top, 2);
    for (int l = 0; l < t.top; l++) {
        if (l < early) {
            TPE_CUDA_TRY(cudaEventRecord(ev[l], st));
            TPE_CUDA_TRY(cudaStreamWaitEvent(side[l], ev[l], 0));
            tree_sums_kernel<<<dim3(1u << l, 2), 1024, smem, side[l]>>>(t, (1 << l) - 1);
            TPE_CUDA_TRY(cudaEventRecord(ev[l], side[l]));
            ks.count(1);
        }
        const unsigned nn = 1u << l;
        const int32_t n = (E + (int32_t)nn - 1) / (int32_t)nn;
        const unsigned tiles = (unsigned)((n + kTile - 1) / kTile);
        int32_t P = kTile;
        while (P < n) P *= 2;
        const dim3 per((unsigned)((n + kKeysPer - 1) / kKeysPer), nn);
        tree_spread_kernel<<<per, 256, 0, st>>>(t, l);
        tree_keys_kernel<<<per, 256, 0, st>>>(t, l);
        tree_tile_kernel<<<dim3(tiles, nn), kTile / 2, 0, st>>>(t, l, 2);
        ks.count(4);  // (with the order)
        for (int32_t k = 2 * kTile; k <= P; k *= 2) {
            const dim3 grid((unsigned)(P / 2 / 256), nn);
            tree_step_kernel<<<grid, 256, 0, st>>>(t, l, k, 0);
            ks.count(2);
            for (int32_t h = k / 4; h >= kTile; h /= 2) {
                tree_step_kernel<<<grid, 256, 0, st>>>(t, l, k, h);
                ks.count(1);
            }
            tree_tile_kernel<<<dim3(tiles, nn), kTile / 2, 0, st>>>(t, l, k);
        }
        tree_order_kernel<<<flat, 256, 0, st>>>(t, l);
    }
    tree_sub_kernel<<<1u << t.top, kSubThr, sizeof(SubSmem), st>>>(t);
    if (t.top > early) {
        const int32_t first = (1 << early) - 1, nn = (1 << t.top) - 1 - first;
        tree_sums_kernel<<<dim3((unsigned)nn, 2), 1024, smem, st>>>(t, first);
        ks.count(1);
    }
    for (int l = 0; l < early; l++) TPE_CUDA_TRY(cudaStreamWaitEvent(st, ev[l], 0));
    if (t.top > 0) {
        tree_top_kernel<<<(1u << t.top) - 1, 1024, 0, st>>>(t);
        ks.count(1);
    }
    TPE_CUDA_TRY(cudaGetLastError());
    return TPE_OK;
}

// Edge geometry as edge_geometry computes it (tpe_stage2_oracle.py:72-82) and
// the tree over it.
struct Tree {
    std::vector<double> C, T, m;  // midpoints, unit tangents (E x 3), ell_eps (E)
    std::vector<Node> nodes;
    std::vector<int32_t> perm, where;  // edge at each position, position of each edge
};

void build_tree(const int32_t* edges, int32_t E, const double* h_xyz, double eps, int32_t leaf,
                Tree& tr) {
    tr.C.assign((size_t)3 * E, 0.0);
    tr.T.assign((size_t)3 * E, 0.0);
    tr.m.assign((size_t)E, 0.0);
    for (int32_t I = 0; I < E; I++) {
        const int32_t a = edges[2 * (size_t)I], b = edges[2 * (size_t)I + 1];
        double e[3];
        for (int d = 0; d < 3; d++) {
            e[d] = h_xyz[3 * (size_t)b + d] - h_xyz[3 * (size_t)a + d];
            tr.C[3 * (size_t)I + d] = 0.5 * (h_xyz[3 * (size_t)a + d] + h_xyz[3 * (size_t)b + d]);
        }
        const double ell = norm3(e[0], e[1], e[2]);
        for (int d = 0; d < 3; d++) tr.T[3 * (size_t)I + d] = ell >= kTangentTol ? e[d] / ell : 0.0;
        tr.m[I] = ell + eps;
    }
    tr.perm.resize((size_t)E);
    std::iota(tr.perm.begin(), tr.perm.end(), 0);
    // The top levels on this thread; below them, subtrees on their own threads
    // (disjoint ranges of the permutation, the same arithmetic), then joined.
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    int32_t split = 0;
    while ((1u << split) < std::min(hw, 16u) && ((int64_t)E >> split) > 4 * (int64_t)leaf + 4096) split++;
    Builder top{tr.C, tr.T, tr.m, leaf, tr.perm.data(), {}, {}, {}, 1, split > 0 ? split : -1, {}};
    top.sort_threads = (int)std::min(hw, 16u);
    top.rec(0, E);
    std::vector<Builder> sub;
    sub.reserve(top.tasks.size());
    for (size_t i = 0; i < top.tasks.size(); i++)
        sub.push_back(Builder{tr.C, tr.T, tr.m, leaf, tr.perm.data(), {}, {}, {}, 1, -1, {}});
    {
        // a failure inside a worker (allocation) is carried back to this thread
        std::vector<char> failed(top.tasks.size(), 0);
        std::vector<std::thread> th;
        try {
            for (size_t i = 0; i < top.tasks.size(); i++)
                th.emplace_back([&, i] {
                    try {
                        sub[i].rec(top.tasks[i].begin, top.tasks[i].count);
                    } catch (...) {
                        failed[i] = 1;
                    }
                });
        } catch (...) {
            for (auto& x : th) x.join();
            throw;
        }
        for (auto& x : th) x.join();
        for (char f : failed)
            if (f) throw std::bad_alloc();
    }
    tr.nodes.swap(top.nodes);
    for (size_t i = 0; i < sub.size(); i++) {
        const int32_t base = (int32_t)tr.nodes.size();
        for (Node nd : sub[i].nodes) {
            if (nd.left >= 0) {
                nd.left += base;
                nd.right += base;
            }
            if (nd.parent >= 0) nd.parent += base;
            tr.nodes.push_back(nd);
        }
        const Builder::Task& tk = top.tasks[i];
        tr.nodes[base].parent = tk.parent;
        (tk.left ? tr.nodes[tk.parent].left : tr.nodes[tk.parent].right) = base;
    }
    tr.where.assign((size_t)E, 0);
    for (int32_t k = 0; k < E; k++) tr.where[tr.perm[k]] = k;
}

}  // namespace

int32_t bh_energy(tpe_ctx* ctx, const double* h_xyz, const double* d_xyz, double alpha, double beta,
                  double eps, double theta, double theta_t, int32_t leaf, double* energy,
                  int64_t* stats) {
    const int32_t E = ctx->E;
    if (leaf < 1 || !(theta >= 0.0) || !(theta_t >= 0.0)) {
        set_error(ctx, TPE_ERR_BAD_ARG, "bh energy: leaf size >= 1 and theta, theta_t >= 0");
        return TPE_ERR_BAD_ARG;
    }
    if (E == 0) {
        *energy = 0.0;
        if (stats) stats[0] = stats[1] = stats[2] = 0;
        return TPE_OK;
    }
    // the device builds the tree where its scratch and the shape of a subtree allow
    const bool device = E >= kDeviceTreeFrom && E <= kDeviceTreeEdges && leaf <= kDeviceTreeLeaf;
    Tree tr;
    size_t nn = 1;
    DevTree t{};
    if (device) {
        while ((E + (1 << t.top) - 1) >> t.top > kSubtree) t.top++;
        while (((int64_t)E + (int64_t)nn - 1) / (int64_t)nn > leaf) nn *= 2;
        nn = 2 * nn - 1;
    } else {
        build_tree(ctx->h_edges.data(), ctx->E, h_xyz, eps, leaf, tr);
        nn = tr.nodes.size();
    }
    const size_t bytes_nodes = sizeof(Node) * nn, bytes_idx = sizeof(int32_t) * (size_t)E;
    size_t end = 0;
    auto place = [&](size_t bytes) {
        const size_t at = end;
        end += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t off_nodes = place(bytes_nodes), off_perm = place(bytes_idx), off_where = place(bytes_idx);
    const size_t off_val = place(sizeof(double) * (size_t)E), off_cnt = place(sizeof(long long) * 3 * (size_t)E);
    const int32_t parts = (E + kRedPer - 1) / kRedPer;
    const size_t off_tot = place(256), off_part = place(sizeof(double) * 4 * (size_t)parts);
    const size_t off_x = place(device ? sizeof(double) * 7 * (size_t)E : 0);
    const size_t off_ord = place(device ? bytes_idx * (size_t)(t.top + 2) : 0);
    const size_t off_key = place(device ? sizeof(double) * (size_t)E : 0);
    const size_t off_sums = place(device ? sizeof(double) * 7 * ((size_t)1 << t.top) : 0);
    const size_t off_spread = place(device ? sizeof(double) * 12 * ((size_t)1 << t.top) : 0);
    TPE_TRY(ensure(ctx, ctx->bh_buf, end));
    uint8_t* base = ctx->bh_buf.as<uint8_t>();
    const cudaStream_t st = ctx->stream;
    if (device) {
        t.pos = d_xyz;
        t.edges = ctx->d_edges.as<int2>();
        t.E = E;
        t.leaf = leaf;
        t.eps = eps;
        t.X = reinterpret_cast<double*>(base + off_x);
        t.m = t.X + 6 * (size_t)E;
        t.ord = reinterpret_cast<int32_t*>(base + off_ord);
        t.perm = t.ord + E;
        t.key = reinterpret_cast<unsigned long long*>(base + off_key);
        t.sums = reinterpret_cast<double*>(base + off_sums);
        t.spread = reinterpret_cast<unsigned long long*>(base + off_spread);
        t.nodes = reinterpret_cast<Node*>(base + off_nodes);
        t.final_perm = reinterpret_cast<int32_t*>(base + off_perm);
        t.where = reinterpret_cast<int32_t*>(base + off_where);
        TPE_TRY(build_tree_device(ctx, t));
    } else {
        TPE_CUDA_TRY(cudaMemcpyAsync(base + off_nodes, tr.nodes.data(), bytes_nodes, cudaMemcpyHostToDevice, st));
        TPE_CUDA_TRY(cudaMemcpyAsync(base + off_perm, tr.perm.data(), bytes_idx, cudaMemcpyHostToDevice, st));
        TPE_CUDA_TRY(cudaMemcpyAsync(base + off_where, tr.where.data(), bytes_idx, cudaMemcpyHostToDevice, st));
    }
    int32_t* err = reinterpret_cast<int32_t*>(base + off_tot + 32);
    TPE_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int32_t), st));
    {
        KernelScope ks(ctx, TPE_KGROUP_ENERGY, 3);
        (alpha == 3.0 && beta == 6.0 ? bh_energy_kernel<true> : bh_energy_kernel<false>)<<<(E + 127) / 128, 128, 0, st>>>(
            d_xyz, ctx->d_edges.as<int2>(), E, reinterpret_cast<const Node*>(base + off_nodes),
            reinterpret_cast<const int32_t*>(base + off_perm),
            reinterpret_cast<const int32_t*>(base + off_where), ctx->d_inc_off.as<int32_t>(),
            ctx->d_inc.as<int32_t>(), alpha, beta, eps, theta, theta_t,
            reinterpret_cast<double*>(base + off_val), reinterpret_cast<long long*>(base + off_cnt), err);
        TPE_CUDA_TRY(cudaGetLastError());
        double* part = reinterpret_cast<double*>(base + off_part);
        long long* cpart = reinterpret_cast<long long*>(part + parts);
        bh_reduce_kernel<<<(unsigned)parts, 256, 0, st>>>(reinterpret_cast<const double*>(base + off_val),
                                                          reinterpret_cast<const long long*>(base + off_cnt), E,
                                                          part, cpart, 1.0, kRedPer);
        bh_reduce_kernel<<<1, 256, 0, st>>>(part, cpart, parts, reinterpret_cast<double*>(base + off_tot),
                                            reinterpret_cast<long long*>(base + off_tot + 8), 0.5, parts);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    // total (8 bytes), three counts (24 bytes), the stack flag (4 bytes)
    unsigned char h[36];
    TPE_CUDA_TRY(cudaMemcpyAsync(h, base + off_tot, sizeof(h), cudaMemcpyDeviceToHost, st));
    TPE_CUDA_TRY(cudaStreamSynchronize(st));
    int32_t herr = 0;
    memcpy(&herr, h + 32, sizeof(int32_t));
    if (herr) {
        set_error(ctx, TPE_ERR_INTERNAL, "bh energy: tree deeper than the traversal stack");
        return TPE_ERR_INTERNAL;
    }
    memcpy(energy, h, sizeof(double));
    if (stats) {
        long long c[3];
        memcpy(c, h + 8, sizeof(c));
        for (int q = 0; q < 3; q++) stats[q] = (int64_t)c[q];
    }
    return TPE_OK;
}


// ---- block-cluster-tree kernel products (bct_matvec_kernel) -------------------------
//
// phi = K psi for the high- or low-order edge kernel K of the Sobolev inner
// product, the stage-2 oracle's bct_matvec_kernel (tpe_stage2_oracle.py:649-703):
// a dual traversal of the edge tree from (root, root); a block (t, s) is
// admissible when it holds at least three edges, no edge of t shares a vertex
// with an edge of s, max(rx) / distance <= theta and max(rT) <= theta_t; it then
// adds mass_I * k(t, s) * sum_{J in s} mass_J psi_J to every I in t, with k the
// node kernel (bct_kernel_node :634-643). Two leaves that are not admissible are
// summed pair by pair with the exact edge kernel (exact_edge_kernel_pair
// :706-730). Otherwise the target splits when it is not a leaf and the source is
// a leaf or no larger, else the source splits. The block list is built on the
// host (the same recursion); the device forms every node's moment
// sum_J mass_J psi_J, each target node's sum of k * moment over its admissible
// blocks, and per edge the sum over its tree ancestors plus its direct blocks.

namespace {

struct BctLists {
    std::vector<int32_t> adm_t, adm_s, dir_t, dir_s;
    std::vector<double> adm_k;
    int64_t admissible = 0, direct_blocks = 0, direct_pairs = 0;
};

double node_kernel(int kind, const Node& t, const Node& s, double eps) {
    const double dx = t.cx - s.cx, dy = t.cy - s.cy, dz = t.cz - s.cz;
    const double dn = norm3(dx, dy, dz) + eps;
    if (kind == 0) return 2.0 / std::pow(dn, 7.0 / 3.0);
    // |t_T x d| and |t_S x (-d)|
    const double c1 = norm3(t.ty * dz - t.tz * dy, t.tz * dx - t.tx * dz, t.tx * dy - t.ty * dx) + eps;
    const double c2 = norm3(s.ty * -dz - s.tz * -dy, s.tz * -dx - s.tx * -dz, s.tx * -dy - s.ty * -dx) + eps;
    return (std::pow(c1, 2.0) + std::pow(c2, 2.0)) / std::pow(dn, 4.0 + 7.0 / 3.0);
}

struct BctRec {
    const Tree& tr;
    const tpe_ctx* ctx;
    int kind;
    double eps, theta, theta_t;
    BctLists& out;

    bool shares(int32_t I, int32_t J) const {
        const int32_t* e = ctx->h_edges.data();
        return I == J || e[2 * I] == e[2 * J] || e[2 * I] == e[2 * J + 1] || e[2 * I + 1] == e[2 * J] ||
               e[2 * I + 1] == e[2 * J + 1];
    }
    // no edge of t shares a vertex with an edge of s (blocks_all_disjoint); the
    // relation is symmetric, so the smaller node's edges are looked up in the other
    bool disjoint(const Node& t0, const Node& s0) const {
        const Node& t = t0.count <= s0.count ? t0 : s0;
        const Node& s = t0.count <= s0.count ? s0 : t0;
        for (int32_t k = t.begin; k < t.begin + t.count; k++) {
            const int32_t I = tr.perm[k];
            for (int q = 0; q < 2; q++) {
                const int32_t v = ctx->h_edges[2 * (size_t)I + q];
                for (int32_t r = ctx->h_inc_off[v]; r < ctx->h_inc_off[v + 1]; r++) {
                    const int32_t w = tr.where[ctx->h_inc[r] >> 1];
                    if (w >= s.begin && w < s.begin + s.count) return false;
                }
            }
        }
        return true;
    }
    void rec(int32_t ti, int32_t si) {
        const Node& tn = tr.nodes[ti];
        const Node& sn = tr.nodes[si];
        const double dist = norm3(tn.cx - sn.cx, tn.cy - sn.cy, tn.cz - sn.cz);
        const bool well = tn.count + sn.count >= 3 && dist > 0.0 &&
                          std::max(tn.rx, sn.rx) / dist <= theta && std::max(tn.rT, sn.rT) <= theta_t &&
                          disjoint(tn, sn);
        if (well) {
            out.adm_t.push_back(ti);
            out.adm_s.push_back(si);
            out.adm_k.push_back(node_kernel(kind, tn, sn, eps));
            out.admissible++;
            return;
        }
        if (tn.left < 0 && sn.left < 0) {
            out.dir_t.push_back(ti);
            out.dir_s.push_back(si);
            out.direct_blocks++;
            for (int32_t a = tn.begin; a < tn.begin + tn.count; a++)
                for (int32_t b = sn.begin; b < sn.begin + sn.count; b++)
                    if (!shares(tr.perm[a], tr.perm[b])) out.direct_pairs++;
            return;
        }
        const bool split_t = tn.left >= 0 && (sn.left < 0 || tn.count >= sn.count);
        if (split_t) {
            rec(tn.left, si);
            rec(tn.right, si);
        } else {
            rec(ti, sn.left);
            rec(ti, sn.right);
        }
    }
};

// CSR of (key, value) pairs grouped by key, keeping the recorded order in a group.
void csr(int32_t nkeys, const std::vector<int32_t>& key, std::vector<int32_t>& off,
         std::vector<int32_t>& order) {
    off.assign((size_t)nkeys + 1, 0);
    for (int32_t k : key) off[k + 1]++;
    for (int32_t i = 0; i < nkeys; i++) off[i + 1] += off[i];
    order.assign(key.size(), 0);
    std::vector<int32_t> fill(off.begin(), off.end() - 1);
    for (size_t i = 0; i < key.size(); i++) order[fill[key[i]]++] = (int32_t)i;
}

// moment[n][c] = sum over the node's edges of mass_J psi_J[c]
__global__ void bct_moment_kernel(const Node* __restrict__ nodes, int32_t nn,
                                  const int32_t* __restrict__ perm, const double* __restrict__ mass,
                                  const double* __restrict__ psi, int32_t nr, double* __restrict__ mom) {
    const int32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const Node nd = nodes[n];
    double acc[3] = {0.0, 0.0, 0.0};
    for (int32_t k = nd.begin; k < nd.begin + nd.count; k++) {
        const int32_t J = perm[k];
        for (int c = 0; c < nr; c++) acc[c] += mass[J] * psi[(size_t)J * nr + c];
    }
    for (int c = 0; c < nr; c++) mom[(size_t)n * nr + c] = acc[c];
}

// local[t][c] = sum over t's admissible blocks (s, k) of k * moment[s][c]
__global__ void bct_local_kernel(int32_t nn, const int32_t* __restrict__ off,
                                 const int32_t* __restrict__ src, const double* __restrict__ kv,
                                 const double* __restrict__ mom, int32_t nr, double* __restrict__ loc) {
    const int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nn) return;
    double acc[3] = {0.0, 0.0, 0.0};
    for (int32_t b = off[t]; b < off[t + 1]; b++)
        for (int c = 0; c < nr; c++) acc[c] += kv[b] * mom[(size_t)src[b] * nr + c];
    for (int c = 0; c < nr; c++) loc[(size_t)t * nr + c] = acc[c];
}

__device__ __forceinline__ double exact_pair_kernel(int kind, const double* __restrict__ pos, int2 eI,
                                                    int2 eJ, double eps) {
    const double p = 7.0 / 3.0;
    const double ax = pos[3 * eI.x], ay = pos[3 * eI.x + 1], az = pos[3 * eI.x + 2];
    const double bx = pos[3 * eI.y], by = pos[3 * eI.y + 1], bz = pos[3 * eI.y + 2];
    const double cx = pos[3 * eJ.x], cy = pos[3 * eJ.x + 1], cz = pos[3 * eJ.x + 2];
    const double dx = pos[3 * eJ.y], dy = pos[3 * eJ.y + 1], dz = pos[3 * eJ.y + 2];
    const double ux = bx - ax, uy = by - ay, uz = bz - az, wx = dx - cx, wy = dy - cy, wz = dz - cz;
    const double lI = sqrt((ux * ux + uy * uy) + uz * uz), lJ = sqrt((wx * wx + wy * wy) + wz * wz);
    const double ellI = lI + eps, ellJ = lJ + eps;
    double tI[3] = {0, 0, 0}, tJ[3] = {0, 0, 0};
    if (lI >= kTangentTol) {
        tI[0] = ux / lI;
        tI[1] = uy / lI;
        tI[2] = uz / lI;
    }
    if (lJ >= kTangentTol) {
        tJ[0] = wx / lJ;
        tJ[1] = wy / lJ;
        tJ[2] = wz / lJ;
    }
    const double vi[2][3] = {{ax, ay, az}, {bx, by, bz}}, vj[2][3] = {{cx, cy, cz}, {dx, dy, dz}};
    double s1 = 0.0, s2 = 0.0;
    for (int i = 0; i < 2; i++)
        for (int j = 0; j < 2; j++) {
            const double qx = vi[i][0] - vj[j][0], qy = vi[i][1] - vj[j][1], qz = vi[i][2] - vj[j][2];
            const double dn = sqrt((qx * qx + qy * qy) + qz * qz) + eps;
            if (kind == 0) {
                s1 += 1.0 / pow(dn, p);
            } else {
                const double c1 = sqrt(((tI[1] * qz - tI[2] * qy) * (tI[1] * qz - tI[2] * qy) +
                                        (tI[2] * qx - tI[0] * qz) * (tI[2] * qx - tI[0] * qz)) +
                                       (tI[0] * qy - tI[1] * qx) * (tI[0] * qy - tI[1] * qx)) + eps;
                const double c2 = sqrt(((tJ[1] * -qz - tJ[2] * -qy) * (tJ[1] * -qz - tJ[2] * -qy) +
                                        (tJ[2] * -qx - tJ[0] * -qz) * (tJ[2] * -qx - tJ[0] * -qz)) +
                                       (tJ[0] * -qy - tJ[1] * -qx) * (tJ[0] * -qy - tJ[1] * -qx)) + eps;
                const double den = pow(dn, 4.0 + p);
                s1 += pow(c1, 2.0) / den;
                s2 += pow(c2, 2.0) / den;
            }
        }
    return kind == 0 ? 2.0 * 0.25 * ellI * ellJ * s1 : 0.25 * ellI * ellJ * (s1 + s2);
}

// per edge I: mass_I times the ancestors' local sums, plus its leaf's direct blocks
__global__ void bct_apply_kernel(int kind, const double* __restrict__ pos, const int2* __restrict__ edges,
                                 int32_t E, const Node* __restrict__ nodes,
                                 const int32_t* __restrict__ perm, const int32_t* __restrict__ leaf_of,
                                 const double* __restrict__ mass, const double* __restrict__ loc,
                                 const int32_t* __restrict__ doff, const int32_t* __restrict__ dsrc,
                                 const double* __restrict__ psi, int32_t nr, double eps,
                                 double* __restrict__ phi) {
    const int32_t I = blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= E) return;
    const int32_t leaf = leaf_of[I];
    double far[3] = {0.0, 0.0, 0.0}, near[3] = {0.0, 0.0, 0.0};
    for (int32_t n = leaf; n >= 0; n = nodes[n].parent)
        for (int c = 0; c < nr; c++) far[c] += loc[(size_t)n * nr + c];
    const int2 eI = edges[I];
    for (int32_t b = doff[leaf]; b < doff[leaf + 1]; b++) {
        const Node sn = nodes[dsrc[b]];
        for (int32_t k = sn.begin; k < sn.begin + sn.count; k++) {
            const int32_t J = perm[k];
            const int2 eJ = edges[J];
            if (J == I || eJ.x == eI.x || eJ.x == eI.y || eJ.y == eI.x || eJ.y == eI.y) continue;
            const double kij = exact_pair_kernel(kind, pos, eI, eJ, eps);
            for (int c = 0; c < nr; c++) near[c] += kij * psi[(size_t)J * nr + c];
        }
    }
    for (int c = 0; c < nr; c++) phi[(size_t)I * nr + c] = mass[I] * far[c] + near[c];
}

}  // namespace

int32_t bct_matvec(tpe_ctx* ctx, const double* h_xyz, const double* d_xyz, int32_t kind,
                   const double* h_psi, int32_t nr, double eps, double theta, double theta_t,
                   int32_t leaf, double* h_phi, int64_t* stats) {
    const int32_t E = ctx->E;
    if (leaf < 1 || !(theta >= 0.0) || !(theta_t >= 0.0) || (kind != 0 && kind != 1) ||
        (nr != 1 && nr != 3)) {
        set_error(ctx, TPE_ERR_BAD_ARG, "bct matvec: kind 0/1, 1 or 3 columns, leaf >= 1, theta >= 0");
        return TPE_ERR_BAD_ARG;
    }
    if (E == 0) {
        if (stats) stats[0] = stats[1] = stats[2] = stats[3] = 0;
        return TPE_OK;
    }
    Tree tr;
    build_tree(ctx->h_edges.data(), ctx->E, h_xyz, eps, leaf, tr);
    BctLists L;
    BctRec R{tr, ctx, kind, eps, theta, theta_t, L};
    R.rec(0, 0);
    const int32_t nn = (int32_t)tr.nodes.size();
    std::vector<int32_t> aoff, aord, doff, dord;
    csr(nn, L.adm_t, aoff, aord);
    csr(nn, L.dir_t, doff, dord);
    std::vector<int32_t> asrc(aord.size()), dsrc(dord.size());
    std::vector<double> akv(aord.size());
    for (size_t i = 0; i < aord.size(); i++) {
        asrc[i] = L.adm_s[aord[i]];
        akv[i] = L.adm_k[aord[i]];
    }
    for (size_t i = 0; i < dord.size(); i++) dsrc[i] = L.dir_s[dord[i]];
    std::vector<int32_t> leaf_of((size_t)E, 0);
    for (int32_t n = 0; n < nn; n++)
        if (tr.nodes[n].left < 0)
            for (int32_t k = tr.nodes[n].begin; k < tr.nodes[n].begin + tr.nodes[n].count; k++)
                leaf_of[tr.perm[k]] = n;
    // device layout, 256-byte aligned pieces
    size_t off = 0;
    auto piece = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) / 256 * 256;
        return o;
    };
    const size_t o_nodes = piece(sizeof(Node) * nn), o_perm = piece(sizeof(int32_t) * E),
                 o_leaf = piece(sizeof(int32_t) * E), o_mass = piece(sizeof(double) * E),
                 o_aoff = piece(sizeof(int32_t) * (nn + 1)), o_asrc = piece(sizeof(int32_t) * (asrc.size() + 1)),
                 o_akv = piece(sizeof(double) * (akv.size() + 1)), o_doff = piece(sizeof(int32_t) * (nn + 1)),
                 o_dsrc = piece(sizeof(int32_t) * (dsrc.size() + 1)), o_psi = piece(sizeof(double) * E * nr),
                 o_mom = piece(sizeof(double) * nn * nr), o_loc = piece(sizeof(double) * nn * nr),
                 o_phi = piece(sizeof(double) * E * nr);
    TPE_TRY(ensure(ctx, ctx->bh_buf, off));
    uint8_t* base = ctx->bh_buf.as<uint8_t>();
    const cudaStream_t st = ctx->stream;
    auto up = [&](size_t o, const void* h, size_t bytes) -> int32_t {
        if (bytes) TPE_CUDA_TRY(cudaMemcpyAsync(base + o, h, bytes, cudaMemcpyHostToDevice, st));
        return TPE_OK;
    };
    TPE_TRY(up(o_nodes, tr.nodes.data(), sizeof(Node) * nn));
    TPE_TRY(up(o_perm, tr.perm.data(), sizeof(int32_t) * E));
    TPE_TRY(up(o_leaf, leaf_of.data(), sizeof(int32_t) * E));
    TPE_TRY(up(o_mass, tr.m.data(), sizeof(double) * E));
    TPE_TRY(up(o_aoff, aoff.data(), sizeof(int32_t) * (nn + 1)));
    TPE_TRY(up(o_asrc, asrc.data(), sizeof(int32_t) * asrc.size()));
    TPE_TRY(up(o_akv, akv.data(), sizeof(double) * akv.size()));
    TPE_TRY(up(o_doff, doff.data(), sizeof(int32_t) * (nn + 1)));
    TPE_TRY(up(o_dsrc, dsrc.data(), sizeof(int32_t) * dsrc.size()));
    TPE_TRY(up(o_psi, h_psi, sizeof(double) * E * nr));
    const Node* dn = reinterpret_cast<const Node*>(base + o_nodes);
    const int32_t* dperm = reinterpret_cast<const int32_t*>(base + o_perm);
    const double* dmass = reinterpret_cast<const double*>(base + o_mass);
    const double* dpsi = reinterpret_cast<const double*>(base + o_psi);
    double* dmom = reinterpret_cast<double*>(base + o_mom);
    double* dloc = reinterpret_cast<double*>(base + o_loc);
    double* dphi = reinterpret_cast<double*>(base + o_phi);
    {
        KernelScope ks(ctx, TPE_KGROUP_PAIR_WEIGHTS, 3);
        bct_moment_kernel<<<(nn + 127) / 128, 128, 0, st>>>(dn, nn, dperm, dmass, dpsi, nr, dmom);
        TPE_CUDA_TRY(cudaGetLastError());
        bct_local_kernel<<<(nn + 127) / 128, 128, 0, st>>>(
            nn, reinterpret_cast<const int32_t*>(base + o_aoff), reinterpret_cast<const int32_t*>(base + o_asrc),
            reinterpret_cast<const double*>(base + o_akv), dmom, nr, dloc);
        TPE_CUDA_TRY(cudaGetLastError());
        bct_apply_kernel<<<(E + 127) / 128, 128, 0, st>>>(
            kind, d_xyz, ctx->d_edges.as<int2>(), E, dn, dperm, reinterpret_cast<const int32_t*>(base + o_leaf),
            dmass, dloc, reinterpret_cast<const int32_t*>(base + o_doff),
            reinterpret_cast<const int32_t*>(base + o_dsrc), dpsi, nr, eps, dphi);
        TPE_CUDA_TRY(cudaGetLastError());
    }
    TPE_CUDA_TRY(cudaMemcpyAsync(h_phi, dphi, sizeof(double) * E * nr, cudaMemcpyDeviceToHost, st));
    TPE_CUDA_TRY(cudaStreamSynchronize(st));
    if (stats) {
        stats[0] = L.admissible + L.direct_blocks;  // leaves of the block tree
        stats[1] = L.admissible;
        stats[2] = L.direct_blocks;
        stats[3] = L.direct_pairs;
    }
    return TPE_OK;
}

}  // namespace tpe

// The edge tree alone, on the host (no device, no context): for checking the
// builder against the stage-2 oracle's build_edge_bvh node by node.
extern "C" int32_t tpe_edge_tree(const double* xyz, int32_t V, const int32_t* edges, int32_t E,
                                 double epsilon, int32_t leaf_size, int32_t max_nodes,
                                 double* node_f, int32_t* node_i, int32_t* perm,
                                 int32_t* n_nodes) {
    try {
        if (!xyz || !edges || !node_f || !node_i || !perm || !n_nodes || V < 0 || E < 1 ||
            leaf_size < 1)
            return TPE_ERR_BAD_ARG;
        for (int64_t q = 0; q < 2 * (int64_t)E; q++)
            if (edges[q] < 0 || edges[q] >= V) return TPE_ERR_BAD_ARG;
        tpe::Tree tr;
        tpe::build_tree(edges, E, xyz, epsilon, leaf_size, tr);
        *n_nodes = (int32_t)tr.nodes.size();
        if ((int64_t)tr.nodes.size() > max_nodes) return TPE_ERR_TOO_LARGE;
        for (size_t i = 0; i < tr.nodes.size(); i++) {
            const tpe::Node& nd = tr.nodes[i];
            const double f[9] = {nd.cx, nd.cy, nd.cz, nd.tx, nd.ty, nd.tz, nd.mass, nd.rx, nd.rT};
            for (int q = 0; q < 9; q++) node_f[9 * i + q] = f[q];
            node_i[4 * i] = nd.begin;
            node_i[4 * i + 1] = nd.count;
            node_i[4 * i + 2] = nd.left;
            node_i[4 * i + 3] = nd.right;
        }
        for (int32_t k = 0; k < E; k++) perm[k] = tr.perm[k];
        return TPE_OK;
    } catch (const std::bad_alloc&) {
        return TPE_ERR_OUT_OF_MEMORY;
    } catch (...) {
        return TPE_ERR_INTERNAL;
    }
}
