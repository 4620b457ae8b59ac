// Internal declarations of libtpe: the context, device buffers and the
// launchers each .cu file provides. Not part of the ABI (include/tpe.h is).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/tpe.h"
#include "tc.h"

#define TPE_CUDA_TRY(expr)                                                              \
    do {                                                                                \
        cudaError_t _e = (expr);                                                        \
        if (_e != cudaSuccess) {                                                        \
            tpe::set_error(ctx, TPE_ERR_CUDA, std::string(#expr) + ": " +               \
                                                  cudaGetErrorString(_e));              \
            return TPE_ERR_CUDA;                                                        \
        }                                                                               \
    } while (0)

#define TPE_TRY(expr)                       \
    do {                                    \
        int32_t _s = (expr);                \
        if (_s != TPE_OK) return _s;        \
    } while (0)

namespace tpe {

// A grow-only device allocation owned by the context.
struct DevBuf {
    void* ptr = nullptr;
    size_t bytes = 0;
    template <class T>
    T* as() const { return static_cast<T*>(ptr); }
};

// Dense Cholesky block size (diagonal blocks are factored by one CTA).
constexpr int kNB = 64;
// Most right-hand sides (3 per constraint row, +3 for b) the mixed solve takes
// at factor time; larger sets use the FP64 factorization.
constexpr int kMixedMaxRhs = 48;
// Up to this many vertices the mixed mode takes the FP64 factor too (op_finalize): one
// data-flow launch where the FP32 factor and its CG take 150 to 250, and one solve where the
// CG takes 3 to 11. A step on a random walk or a jittered trefoil, FP32 against FP64 factor
// (us): V = 1024 1910 -> 1330, 2500 2810 -> 2325 and 2720 -> 1910, 4096 4614 -> 3234 and 4636
// -> 2822, 6000 6866 -> 5668 and 7209 -> 5379, 8192 10610 -> 10956 and 10269 -> 10355. A
// correction, which rough curves of 3600 and smooth ones of 3000 and more vertices need to
// reach 1e-12, adds 900 (4096) to 1400 (6000): then 5000 5340 -> 5350 and 6000 -> 5060, 6000
// 6866 -> 7100 and 7209 -> 6760. 64 curves of 256 to 1500 vertices together: 44 -> 16 ms.
constexpr int32_t kMixedDirect = 5000;
// Most step sizes one batched line-search launch projects together.
constexpr int kMaxTrials = 16;

// The rows of a large constraint Jacobian that are one 3-vector w times one vertex
// (a pin) or times the difference of two (an edge length: w at a, -w at b): row s is
// w_s (x) (e_a - e_b), b = -1 for one vertex. The same by vertex, and the list of
// the other (dense) rows. Device pointers (schur.cu).
struct SparseRows {
    int2* ab = nullptr;        // k: (a, b); (-1, -1) for a dense row
    double* w = nullptr;       // k x 3
    int32_t* off = nullptr;    // V + 1
    int32_t* ent = nullptr;    // 2 row + (0: at a, 1: at b), by vertex, in row order
    int32_t* dense = nullptr;  // k: 1 for a row of another form
    int32_t* list = nullptr;   // nd dense rows
    double* stats = nullptr;   // k x 4: sums over the coordinate blocks, sum of |.|
    int32_t nd = 0;
};

// Everything the structured saddle solve keeps between the factorization and
// later solves: the frozen operator of optimizer.ts's 'frozen' projection.
struct SaddleOp {
    bool valid = false;
    int V = 0, k = 0;
    bool trans_constrained = false;  // set contains a barycenter or point block
    bool mixed = false;              // solves use the FP32 factor + FP64 CG (mixed.cu)
    bool mixed_fallback = false;     // mixed requested, FP64 factorization used instead
    int refine_iters = 0;            // CG iterations (FP64 factor: solves) at factor time
    int refine_max_iter = 60;
    double refine_tol = 1e-12;
    double rho = 0.0;                // A_rho = A + (rho/V) 1 1^T
    // device (views into ctx buffers)
    double* A = nullptr;     // V x V original A (unfactored, for residuals)
    double* L = nullptr;     // V x V Cholesky factor of A_rho (lower, row-major)
    double* Linv = nullptr;  // nb x 64 x 64 inverses of the diagonal blocks of L
    double* C = nullptr;     // k x 3V dense constraint Jacobian
    double* Y = nullptr;     // k x 3V: Abar_rho^{-1} C^T (row s = column s of C^T; large: the nd dense rows)
    double* W = nullptr;     // 3V: Abar_rho^{-1} b for the b given at factor time (row k of Y)
    const double* w_src = nullptr;  // that b (device), or null
    // large constraint sets (schur.cu): explicit inverses on the device
    bool large = false;
    double* Ainv = nullptr;  // V x V: A_rho^{-1}
    double* Sinv = nullptr;  // k x k: (C A3^{-1} C^T)^{-1}
    SparseRows sp;
    double* Gt = nullptr;    // V x k: column s = Ainv (e_a - e_b) of sparse row s
    bool int8 = false;       // both inverses with their products on the int8 tensor cores
    double chol_tol = 0.0;   // pivot tolerance of A_rho's Cholesky
    // host: small Schur complement and its factors
    std::vector<double> Scc;   // k x k, then its Cholesky factor (lower)
    std::vector<double> Scu;   // k x 3 = C U / rho
    std::vector<double> M;     // 3 x 3 = Scu^T Scc^{-1} Scu, then its Cholesky factor
};

// FP32 tensor-core factor of the Jacobi-scaled A_rho (mixed.cu): S ~ L L^T,
// Z = L^{-1}, W = Z^T, all Vp x Vp split-FP32; T is the TRTRI scratch.
struct MixedFactor {
    bool valid = false;
    int V = 0, Vp = 0;
    double rho = 0.0;
    tc::SplitMat L, Z, W, T, T2;  // T: level scratch; T2: the top level's T^T
    tc::SplitMat Zf;              // plain FP32 view of the CG's copy of Z
    tc::SplitMat S;  // plain FP32 trailing matrix (hi only)
};

struct DevBlock {
    int32_t kind;
    int32_t row0;
    int32_t vertex;
    int32_t rows;
    double target[3];
    double L0;
    const double* ell0;  // device copy, E entries (NaN where the host array ended)
};

}  // namespace tpe

struct tpe_ctx {
    // Held by every entry point for the whole call (tpe::guarded): calls on one
    // context from several host threads run one after another. Recursive, so an
    // entry point may call another on the same context.
    std::recursive_mutex mu;
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t stream2 = nullptr;           // look-ahead stream of the factorization
    cudaStream_t stream3 = nullptr;           // the gradient, concurrent with assembly + factor
    cudaStream_t stream4 = nullptr;           // first half of the mixed inverse, beside the factor
    cudaStream_t stream5 = nullptr;           // panel remainders of the mixed factor (high priority)
    cudaEvent_t ev_prep = nullptr, ev_grad = nullptr;
    // a gradient launched on stream3 and not yet joined (step_impl / finish_gradient)
    bool grad_pending = false;
    bool grad_unlaunched = false;
    bool grad_first = false;  // before the assembly, on all SMs: the factorization needs it (step_impl)
    double grad_params[3] = {0, 0, 0};  // alpha, beta, eps
    const double* grad_pos = nullptr;
    double* grad_dE = nullptr;
    double* grad_flat = nullptr;
    const tpe_penalties* grad_pen = nullptr;
    // SMs the concurrent gradient may occupy; the rest stay free for the
    // factorization's chain of small launches (TPE_GRAD_SMS overrides)
    int32_t grad_sms = 0;
    // SMs the persistent trailing updates leave free for the chain's and the
    // panel's launches (TPE_FACTOR_FREE_SMS overrides)
    int32_t free_sms = 8;
    std::vector<cudaEvent_t> fac_events;      // dependency events (no timing)
    std::string err;
    int32_t num_sms = 0;

    // topology
    bool has_topology = false;
    int32_t V = 0, E = 0;
    // one closed loop with edge I = (I, I+1 mod V), V >= 8: Gram assembly by the
    // fused stencil kernel (assembly.cu)
    bool closed_loop = false;
    std::vector<int32_t> h_edges;     // 2E
    std::vector<int32_t> h_inc_off;   // V+1
    std::vector<int32_t> h_inc;       // 2E entries: edge*2 + slot, ascending edge order per vertex
    tpe::DevBuf d_edges, d_inc_off, d_inc;
    // lists of the (edge, vertex) pair kernels (pair_ev.cu), built on first use:
    // ev_state 0 not built, 1 in ev_lists, 2 not used for this topology
    int32_t ev_state = 0, ev_VA = 0;
    int64_t ev_at[6] = {};
    tpe::DevBuf ev_lists, ev_vert;

    // per-evaluation buffers
    tpe::DevBuf pos, pos2, pos3, edge_a, edge_b, grad, edge_acc, partial, scalars, flat0, flat1,
        flat2, flat3, dir;
    tpe::DevBuf grad_ctr;  // tile counter of the SM-bounded gradient kernel
    // large constraint sets (schur.cu)
    tpe::DevBuf mat_Ainv, inv_X, inv_W, inv_T, sch_nz, sch_G, sch_S, sch_Linv, sch_Sinv, sch_vec;
    tpe::DevBuf ref_r, ref_x;  // residual and correction of the refinement step
    tpe::DevBuf oz_planes, oz_err;  // digit planes and timeout flag of ozaki_gemm_nt
    tpe::DevBuf oz_base;            // diagonal-block inverses of spd_inverse_int8's base blocks
    tpe::DevBuf bh_buf;             // Barnes-Hut tree, permutation and per-edge sums (bh.cu)
    tpe::DevBuf dag_solve, dag_err;  // the same of the triangular solves, and their error flag
    tpe::DevBuf dag_flags;     // flags and counters of the data-flow factorization (chol_dag.cu)
    tpe::DevBuf mrhs_xt;       // right-hand-side-major input of mrhs_fp64
    tpe::DevBuf ycomb_part;    // split-over-rows partial sums of Y^T coef
    tpe::DevBuf mx_ctr;    // tile counters of the persistent trailing updates
    tpe::DevBuf pairM;                      // E x E double2 (Mb, M0) pair matrix
    tpe::DevBuf edge_m;                     // mixed-precision edge records (4 float4 per edge)
    tpe::DevBuf mat_A, mat_L, mat_Linv, mat_B, mat_B0;
    tpe::DevBuf con_C, con_Y, con_phi, con_blocks, con_ell0, con_red;
    tpe::DevBuf con_part;  // split partial reductions of the constraint rows
    tpe::DevBuf rhs, sol, tmp;
    tpe::DevBuf status;                     // device-side int flags
    tpe::DevBuf trial_raw, trial_cur;       // batched line-search trials (K x 3V each)
    tpe::SaddleOp op;
    // mixed-precision factor (mixed.cu)
    tpe::DevBuf mx_T2hi, mx_T2lo;
    tpe::DevBuf mx_d, mx_dinv, mx_S, mx_Lhi, mx_Llo, mx_Zhi, mx_Zlo, mx_Whi, mx_Wlo, mx_Thi, mx_Tlo,
        mx_vec, mx_part, mx_Zd, mx_Wd;
    tpe::MixedFactor mf;
    void* h_stage = nullptr;  // pinned staging of small device-to-host copies (download_many)
    size_t h_stage_bytes = 0;

    // settings of tpe_tune
    int64_t fail_alloc = 0;  // the growth of a device buffer that fails (1: the next one)
    int32_t mixed_direct = tpe::kMixedDirect;
    int32_t factor_polls = 0, solve_polls = 0, factor_blocks = 0;  // chol_dag.cu (0: its own)

    // instrumentation: kernel launch count and per-group CUDA-event timing
    int64_t launches = 0;
    bool profiling = false;
    double prof_ms[TPE_KGROUP_COUNT] = {};
    int64_t prof_launches[TPE_KGROUP_COUNT + 1] = {};
    struct PendingEvent {
        int group;
        cudaEvent_t a, b;
    };
    std::vector<PendingEvent> prof_pending;
    std::vector<cudaEvent_t> prof_pool;
};

namespace tpe {

// Times the launches issued while in scope under `group` (when profiling) and
// counts them; `n` = number of kernels the scope launches.
struct KernelScope {
    tpe_ctx* ctx;
    int group;
    cudaEvent_t b = nullptr;
    KernelScope(tpe_ctx* c, int g, int64_t n);
    ~KernelScope();
    void count(int64_t n);  // n more launches
};

void set_error(tpe_ctx* ctx, int32_t code, const std::string& msg);

// Runs the body of a C entry point under the context's mutex (when there is a
// context). A C++ exception (a failed host allocation, a thread that could not
// start, a mutex that could not be taken) becomes an error status, with the
// message in the context when there is one, instead of leaving through the C ABI.
template <class F>
int32_t guarded(tpe_ctx* ctx, F&& body) noexcept {
    int32_t code = TPE_ERR_INTERNAL;
    const char* msg = "unexpected host-side exception";
    try {
        std::unique_lock<std::recursive_mutex> lock;
        if (ctx) lock = std::unique_lock<std::recursive_mutex>(ctx->mu);
        return body();
    } catch (const std::bad_alloc&) {
        code = TPE_ERR_OUT_OF_MEMORY;
        msg = "host allocation failed";
    } catch (const std::length_error&) {
        code = TPE_ERR_TOO_LARGE;
        msg = "host buffer size out of range";
    } catch (const std::exception& e) {
        msg = e.what();
    } catch (...) {
    }
    try {
        set_error(ctx, code, msg);
    } catch (...) {
    }
    return code;
}
int32_t ensure(tpe_ctx* ctx, DevBuf& b, size_t bytes);

// Device-to-host copies through the context's pinned staging area: the copies
// are issued on `stream`, the stream is synchronized once, and the bytes are
// copied out on the host. Pageable copies from many host threads (the
// multi-curve batch) would queue in the driver's shared staging buffer.
struct HostCopy {
    void* host;
    const void* dev;
    size_t bytes;
};
int32_t download_many(tpe_ctx* ctx, cudaStream_t stream, const HostCopy* copies, int n);
inline int32_t download_on(tpe_ctx* ctx, cudaStream_t stream, void* host, const void* dev,
                           size_t bytes) {
    const HostCopy c{host, dev, bytes};
    return download_many(ctx, stream, &c, 1);
}

// ---- pair kernels (pair_kernels.cu) ----------------------------------------
// Per-edge records from interleaved positions: a = (p1, ell^eps), b = (p2, |e|).
int32_t edge_prep(tpe_ctx* ctx, const double* d_pos, int32_t ncurves, double eps,
                  double alpha);
// Energy of ncurves position sets (edge records already prepared) into
// d_energy[ncurves] (device).
int32_t energy_fp64(tpe_ctx* ctx, int32_t ncurves, double alpha, double beta, double eps,
                    double* d_energy);
// Energy of one curve with caller-provided scratch and stream (no context);
// edge indices are checked on the device (*bad set, energy NaN).
int32_t energy_fp64_scratch(cudaStream_t stream, const double* d_pos, const int2* d_edges,
                            int32_t V, int32_t E, double alpha, double beta, double eps,
                            double4* ea, double4* eb, double* partial, int32_t max_parts,
                            int32_t* bad, double* d_energy);
// Energy (optional) and gradient (interleaved V x 3) of one curve. max_blocks > 0
// bounds the SMs the pair kernel occupies (one block per SM).
int32_t energy_grad_fp64(tpe_ctx* ctx, double alpha, double beta, double eps, double* d_energy,
                         double* d_grad, int32_t max_blocks = 0);

// ---- (edge, vertex) pair kernels (pair_ev.cu) ---------------------------------
// The topology's lists, built on first use; *ok = false when the edge-pair
// kernels serve this topology.
int32_t ev_topology(tpe_ctx* ctx, bool* ok);
int32_t ev_prep(tpe_ctx* ctx, const double* d_pos, int32_t ncurves, double eps, double alpha);
int32_t ev_energy(tpe_ctx* ctx, int32_t ncurves, double alpha, double beta, double eps,
                  int32_t* nparts);
int32_t ev_gradient(tpe_ctx* ctx, double alpha, double beta, double eps, double* d_grad,
                    int32_t max_blocks);

// Barnes-Hut energy (bh.cu) of this context's curve: h_xyz (host) builds the
// tree, d_xyz (device, the same positions) is traversed. stats (nullable):
// visits, approximated edge references, direct pairs.
int32_t bh_energy(tpe_ctx* ctx, const double* h_xyz, const double* d_xyz, double alpha, double beta,
                  double eps, double theta, double theta_t, int32_t leaf, double* energy,
                  int64_t* stats);

// phi = K psi (E x nr, nr = 1 or 3; host arrays) for the high (kind 0) or low
// (kind 1) edge kernel by the block cluster tree (bh.cu). stats (nullable, 4):
// block-tree leaves, admissible blocks, direct blocks, direct pairs.
int32_t bct_matvec(tpe_ctx* ctx, const double* h_xyz, const double* d_xyz, int32_t kind,
                   const double* h_psi, int32_t nr, double eps, double theta, double theta_t,
                   int32_t leaf, double* h_phi, int64_t* stats);

// ---- mixed precision energy (pair_mixed.cu) ----------------------------------
// FP32 pair terms, FP64 sums: tpe_energy_batch with TPE_PRECISION_MIXED only.
int32_t edge_prep_mixed(tpe_ctx* ctx, const double* d_pos, int32_t ncurves, double eps,
                        double alpha);
int32_t energy_mixed(tpe_ctx* ctx, int32_t ncurves, double alpha, double beta, double eps,
                     double* d_energy);

// ---- assembly (assembly.cu) -----------------------------------------------
// A (and optionally B, B0) V x V row-major FP64 from prepared edge records.
int32_t assemble_fp64(tpe_ctx* ctx, double alpha, double beta, double eps, double* d_A,
                      double* d_B, double* d_B0);

// ---- dense linear algebra (dense.cu) --------------------------------------
// Lower Cholesky of an n x n row-major matrix as one data-flow kernel
// (chol_dag.cu), optionally with rows of right-hand sides (B <- B L^-T, the
// forward solves), W = L^-T (upper tiles; X = L^-1, lower tiles) and the symmetric
// inverse Ainv = W W^T. A pivot at or below tol sets *singular.
struct CholDag {
    double* L = nullptr;     // lower triangle read; L on return
    double* Linv = nullptr;  // nb x 64 x 64: inverses of L's diagonal blocks
    int32_t n = 0;
    int64_t ld = 0;  // row length of L, W and X (0: n)
    double tol = 0.0;
    double* B = nullptr;  // nr x n
    int32_t nr = 0;
    double* W = nullptr;  // n x n or null; X and Ainv need it
    double* X = nullptr;
    double* Ainv = nullptr;
};
// With singular = null nothing is read back: the caller reads the two ints at
// ctx->dag_flags ({singular, timed out}) with its next copy and passes them to
// chol_dag_status before it uses the result.
int32_t chol_dag(tpe_ctx* ctx, const CholDag& c, int32_t* singular);
int32_t chol_dag_status(tpe_ctx* ctx, const int32_t flags[2]);
// Solves (L L^T) X = B in place for nr right-hand sides stored as B[nr][n]
// (down = false: only L^T X = B). A wait that runs out leaves NaN in B and sets
// ctx->dag_err, for which the caller returns chol_timeout once it has read it.
int32_t chol_solve(tpe_ctx* ctx, const double* d_L, const double* d_Linv, int32_t n, double* d_B,
                   int32_t nr, bool down);
int32_t chol_timeout(tpe_ctx* ctx);
// out[i*ncols + j] = dot(X[i], Y[j]) over len (rows of length len): FP64, deterministic.
int32_t gram_dots(tpe_ctx* ctx, const double* X, int32_t nx, const double* Y, int32_t ny,
                  int64_t len, double* d_out);
// A_rho = A + shift (every entry) into L (lower triangle copied), and trace(A) into *d_trace.
int32_t shift_copy(tpe_ctx* ctx, const double* d_A, double* d_L, int32_t n, double shift);
// C = alpha A B^T + beta C, FP64 row-major, on the FP64 tensor cores (dense.cu).
// kDBUpper, kDBLower (B[j][k] = 0 for k < j, k > j) and kDMaskUpper (write only
// elements with column <= row) are for ozaki_gemm_nt only.
enum : int32_t {
    kDLowerTiles = 1, kDAUpper = 2, kDALower = 4, kDBUpper = 8, kDBLower = 16, kDMaskUpper = 32
};
struct DGemmArgs {
    const double* A = nullptr;
    int64_t lda = 0;
    const double* B = nullptr;
    int64_t ldb = 0;
    double* C = nullptr;
    int64_t ldc = 0;
    int32_t M = 0, N = 0, K = 0;
    double alpha = 1.0, beta = 0.0;
    int32_t mode = 0;
};
int32_t dgemm_nt(tpe_ctx* ctx, const DGemmArgs& g, cudaStream_t stream);
// The same product on the integer tensor cores (ozaki.cu): each operand row cut
// into eight 8-bit digits under a power-of-two row scale, the digit products
// exact int32 GEMMs, summed in FP64: FP64-class accuracy. Scratch: ctx->oz_planes
// (ozaki_scratch_bytes); calls on one context must share one stream. A pipeline
// timeout sets a device flag that ozaki_status reads (and clears).
size_t ozaki_scratch_bytes(int32_t M, int32_t N, int32_t K);
int32_t ozaki_reserve(tpe_ctx* ctx, size_t bytes);
int32_t ozaki_gemm_nt(tpe_ctx* ctx, const DGemmArgs& g, cudaStream_t stream,
                      int group = TPE_KGROUP_TRSV);
int32_t ozaki_status(tpe_ctx* ctx, cudaStream_t stream);
// M[j][i] = M[i][j] for j > i (n x n, row-major).
int32_t mirror_lower(tpe_ctx* ctx, double* M, int32_t n);
// dst[j][i] = src[i][j] for an m x c block (row strides lds, ldd).
int32_t transpose_fp64(tpe_ctx* ctx, const double* src, int64_t lds, int32_t m, int32_t c,
                       double* dst, int64_t ldd);
// out = A^{-1} for the SPD n x n matrix in Mat (lower triangle read; Mat is
// overwritten) with the heavy products on the integer tensor cores
// (ozaki_gemm_nt): recursive Cholesky and triangular inverse in halves down to
// blocks of at most 2048 (chol_dag there), then out = X^T X. X, W (n x n) and Tt ((n/2 + 64)^2) are scratch. A pivot at or
// below piv_tol sets *singular.
int32_t spd_inverse_int8(tpe_ctx* ctx, double* Mat, int32_t n, double piv_tol, double* X,
                         double* W, double* Tt, double* out, bool* singular);
// Y[c][i] = sum_j M[i][j] X[c][j] for c < nr <= 16: M n x n FP64 (row length n),
// X and Y nr rows of stride ldx >= n (mixed.cu: the CG's multi-RHS kernel).
int32_t mrhs_fp64(tpe_ctx* ctx, const double* M, int32_t n, const double* X, int32_t ldx,
                  int32_t nr, double* Y);
// The same for a rows x cols matrix M and X right-hand-side major (XT: (cols + 15) / 16
// * 16 rows of 16, zero rows past cols) without the last sum: part[ch][c][i], ch <
// *nch, i < rows, to be added in order.
int32_t mrhs_part(tpe_ctx* ctx, const double* M, int32_t rows, int32_t cols, const double* XT,
                  const double** part, int32_t* nch);
int32_t trace(tpe_ctx* ctx, const double* d_A, int32_t n, double* d_out);

// ---- mixed-precision solve (mixed.cu) ------------------------------------
int32_t mixed_padded_size(int32_t V);
// FP32 tensor-core factor + inverse of the Jacobi-scaled A_rho = A + (rho/V) 1 1^T
// into ctx->mf; *ok = false when the FP32 factorization broke down.
int32_t mixed_factor(tpe_ctx* ctx, const double* d_A, int32_t V, double rho, bool* ok);
// A_rho X = B for nr right-hand sides ([nr][V], FP64, may alias) by CG with the
// FP32 factor as preconditioner, to ||B - A_rho X|| <= tol ||B|| per column.
int32_t mixed_solve(tpe_ctx* ctx, const double* d_A, const double* d_B, double* d_X, int32_t nr,
                    int32_t maxit, double tol, int32_t* iters, bool* converged);

// ---- large constraint sets (schur.cu) ----------------------------------------
// Constraint sets with more rows than this take the explicit-inverse Schur path.
constexpr int32_t kLargeSchur = 64;
// Iterative refinement of the large-set gradient solve: stop at this relative
// saddle residual, or after kLargeRefineMax corrections, or when a correction
// no longer halves the residual. (At 1e-13 the int8 inverses could stop with a
// residual of 5e-14, which on a loop network left the step's energy 2e-7 off.)
constexpr double kRefineStop = 1e-14;
constexpr int32_t kLargeRefineMax = 4;
// The residual the int8-tensor-core inverses must reach within kInt8RefineMax
// corrections; else the step rebuilds them in FP64. Good inverses lose four digits or
// more of it per correction, as the FP64 ones do. Where rows span many orders of
// magnitude (digits lost under a per-row scale) a correction takes one digit or less,
// and the projection, which uses the inverses without refinement, is off with them: on
// a loop network residuals of 3.4e-7, 3.9e-12, 1.2e-12, 2.2e-13, 5.9e-14 left the
// step's energy 9e-8 off.
constexpr double kInt8ResidualGate = 1e-13;
constexpr int32_t kInt8RefineMax = 2;
// From A_rho in op.L (overwritten): op.Ainv, op.sp, op.W = A3^{-1} b when b is given,
// and op.Sinv; *singular when the Schur complement is not SPD.
int32_t large_schur_build(tpe_ctx* ctx, SaddleOp& op, const double* b_flat, bool* singular);
// out[c] = Sinv rc[c] for nr <= 16 host vectors of length k (host in and out).
int32_t large_sinv(tpe_ctx* ctx, const SaddleOp& op, const double* h_rc, int32_t nr, double* h_out);
// Scu (k x 3) and the Cholesky factor of M (3 x 3) for large_multipliers.
int32_t large_set_mu(tpe_ctx* ctx, const SaddleOp& op, const double* h_scu, const double* h_mchol);
// Multipliers of n <= 16 reduced right-hand sides d_rc + pos[c] * stride (pos null: c):
// *d_coef (n x (k + 3)): lam, then the scaled mu. ru: U^T w, the same for all.
int32_t large_multipliers(tpe_ctx* ctx, const SaddleOp& op, const double* d_rc, int64_t stride,
                          const int32_t* d_pos, int32_t n, const double ru[3], double** d_coef);
// x = w - A3^{-1} C^T lam - mu term (block layout; w may be null), and the same for nu
// coefficient vectors added to cur[idx[q]] (project_update's contract).
int32_t large_solution(tpe_ctx* ctx, const SaddleOp& op, const double* d_coef, const double* d_w, double* d_x);
int32_t large_update(tpe_ctx* ctx, const SaddleOp& op, const double* d_coef, int32_t nu, const int32_t* d_idx,
                     double* d_cur, int64_t stride, int32_t* d_bad);
// C^T lam (3V) and C x (k) from the sparse rows.
int32_t large_ct(tpe_ctx* ctx, const SaddleOp& op, const double* d_lam, double* d_out);
int32_t large_cx(tpe_ctx* ctx, const SaddleOp& op, const double* d_x, double* d_out);
// Joins the gradient running on stream3 (api.cu).
int32_t finish_gradient(tpe_ctx* ctx);

// ---- constraints (constraints.cu) -----------------------------------------
// Upload the set, returns k (stacked rows).
int32_t upload_set(tpe_ctx* ctx, const tpe_constraint* set, int32_t nblocks, int32_t* k);
// Phi (k) and per-block {norm^2, scale} (2*nblocks) into host arrays; dense C
// (k x 3V, device) when d_C != nullptr.
int32_t eval_constraints(tpe_ctx* ctx, const double* d_pos, int32_t nblocks, int32_t k,
                         double* d_C, std::vector<double>& phi, std::vector<double>& norm_scale,
                         const int32_t* d_flag = nullptr, int32_t* flag = nullptr);
// The Jacobian alone (nothing read back).
int32_t eval_jacobian(tpe_ctx* ctx, const double* d_pos, int32_t nblocks, int32_t k, double* d_C);

// Phi (d_phi: n x k) and per-block {norm^2, scale} (d_ns: n x 2 nblocks), on the
// device, for the position sets pos + idx[q] * stride, q < n (idx on the device).
int32_t eval_constraints_batch(tpe_ctx* ctx, const double* d_pos, int64_t stride,
                               const int32_t* d_idx, int32_t n, int32_t nblocks, int32_t k,
                               double* d_phi, double* d_ns);
// The frozen projection of a small set on the device, iterations it0 .. it1 - 1 of `trials`
// (<= kMaxTrials) trials at d_cur, nothing read back: state = {done, ok, iters, bad}[trials],
// norm the last ||Phi||. (The Schur factors travel as a kernel argument.)
constexpr int32_t kProjRows = 16;
struct ProjSolve {
    int32_t k, nblocks, max_iter, trans;
    double tol_abs, tol_rel, su;  // su = 1 / (rho sqrt(V))
    double Scc[kProjRows * kProjRows], Scu[kProjRows * 3], M[9];
};
int32_t project_iterations(tpe_ctx* ctx, const ProjSolve& p, const double* d_Y, int32_t it0, int32_t it1,
                           int32_t trials, double* d_cur, double* d_phi, double* d_ns, double* d_coef,
                           double* d_norm, int32_t* d_state);

// ---- small device helpers (dense.cu) --------------------------------------
int32_t interleaved_to_block(tpe_ctx* ctx, const double* d_v3, double* d_flat, int32_t V);
int32_t block_to_interleaved(tpe_ctx* ctx, const double* d_flat, double* d_v3, int32_t V);
// y = a*x + b*y (n)
int32_t axpby(tpe_ctx* ctx, int64_t n, double a, const double* x, double b, double* y);
// host result: sum(x*y) over n (deterministic)
int32_t dot(tpe_ctx* ctx, int64_t n, const double* x, const double* y, double* out);
// *d_out: the number (device, in ctx->scalars) of non-finite entries in x[n]
int32_t count_nonfinite(tpe_ctx* ctx, int64_t n, const double* x, const double** d_out);
// d_out[r] = the sum of row r of x (n entries each)
int32_t row_sums(tpe_ctx* ctx, const double* x, int32_t rows, int32_t n, double* d_out);
// l2CurveNorm of interleaved values at interleaved positions (host result)
int32_t l2_curve_norm(tpe_ctx* ctx, const double* d_vals, const double* d_pos, double* out);
// x_flat(3V) = w - sum_s Y[s] * lam[s] - U mu / rho ; lam/mu are host arrays
int32_t combine_solution(tpe_ctx* ctx, const double* d_w, const double* d_Y, int32_t k,
                         const double* lam, const double* mu, double rho, int32_t V, double* d_x);
// cur[idx[q]] (interleaved, rows stride apart) += -Y^T coef[q] - mu term for nu <= 16
// device coefficient vectors (k + 3 each), with combine_solution's sums.
int32_t project_update(tpe_ctx* ctx, const double* d_Y, int32_t k, int32_t V, const double* d_coef,
                       int32_t nu, const int32_t* d_idx, double* d_cur, int64_t stride,
                       int32_t* d_bad);
// Structured residual ||K z - rhs|| / max(1, ||rhs||) with A (V x V), C (k x 3V);
// optionally the residual vector rhs - K z itself: top (device, 3V) and bottom
// (host, k). large: C through its sparse rows.
int32_t saddle_residual(tpe_ctx* ctx, const double* d_A, int32_t V, const double* d_C, int32_t k,
                        const double* d_x, const double* lam, const double* d_rhs_top,
                        const double* rhs_bottom, double* out, double* d_res_top = nullptr,
                        double* res_bottom = nullptr, const SaddleOp* large = nullptr);

}  // namespace tpe
