// k_dyson.cu -- K3-K5: Dyson matrix assembly, batched FP64 symmetric
// eigensolve, quasiparticle / quasihole split and Koltun partial sums.
//
// Restates DysonMatrix (source/BcDor-DysonMatrix.cpp:123-532) and Calc_En
// (:542-594).  The reference calls LAPACK dsyevd for all eigenvectors but only
// uses the first D components of each (:448-470).  Here:
//   K3 k_dyson_assemble   fills the dense matrix row by row (:269-390),
//   K4a k_tridiag_small   Householder reduction A = Q T Q^T of a matrix of order
//                         <= 160 in one CTA's shared memory, with the first D rows of Q,
//       k_tridiag_df      the same for larger orders, one thread-block cluster per
//                         matrix (rows split across the CTAs),
//       k_tridiag_grid    the same for one large matrix alone, a CTA on every SM,
//       k_tridiag         in FP64 for launches of orders beyond about 2 300, and beyond those
//                         kernels' shared memory (Q's rows by k_qrows),
//   K4b..K5 (k_eig.cu)    eigenvalues and the first D eigenvector components of T,
//                         back-transformed, split by E_F, Koltun sums.
#include <algorithm>
#include <atomic>
#include <cooperative_groups.h>
#include "bd_common.cuh"
#include "bd_kernels.h"
#include "df64.cuh"
#include "lz_fixed.cuh"

namespace cg = cooperative_groups;

namespace bd {

// ---------------------------------------------------------------- K3 assembly
// Row order of the full matrix: D one-body rows, nfw forward poles, nbk backward poles.
//
// Deflation: a pole row whose every off-diagonal entry is exactly zero (no coupling to
// the orbitals, no beta to its neighbours, no fishbone entry) is an eigenvector of
// the Dyson matrix by itself: eigenvalue its diagonal, no strength.  The deflated
// tails of exhausted Lanczos chains are such rows, often most of a chain.  They are
// taken out before the eigensolve; the matrix keeps the other rows in their order.

// value of the coupling of pole i of part (0 fw, 1 bk) to orbital d
__device__ inline double dy_mcoup(const DyJob &J, int part, int i, int d) {
    const int NT = J.nden + J.D;
    if (part == 0) return J.fw_rows ? J.fw_rows[(size_t)i * NT + J.nden + d] : J.M_fw[(size_t)d * J.nfw + i];
    return J.bk_rows ? J.bk_rows[(size_t)i * NT + J.nden + d] : J.M_bk[(size_t)d * J.nbk + i];
}

__device__ inline double dy_diag(const DyJob &J, int part, int i) {
    const int NT = J.nden + J.D;
    const double *rows = part == 0 ? J.fw_rows : J.bk_rows;
    return rows ? rows[(size_t)i * NT] : (part == 0 ? J.E_fw[i] : J.E_bk[i]);
}

// whether full-matrix row r has an off-diagonal entry, apart from the fishbone
// entries of a branch's start row s-1 to the later rows (k_dyson_deflate marks
// those from the later rows' side)
__device__ inline bool dy_coupled(const DyJob &J, int r) {
    const int D = J.D;
    if (r < D) return true;
    const int part = (r < D + J.nfw) ? 0 : 1;
    const int i = r - (part == 0 ? D : D + J.nfw);
    const int np = part == 0 ? J.nfw : J.nbk;
    for (int d = 0; d < D; ++d) if (dy_mcoup(J, part, i, d) != 0.0) return true;
    const bool lz = part == 0 ? J.lanczos_fw : J.lanczos_bk;
    if (!lz) return false;
    const int NT = J.nden + D;
    const double *rows = part == 0 ? J.fw_rows : J.bk_rows;
    const int *ipiv = part == 0 ? J.ipiv_fw : J.ipiv_bk;
    if (i >= 1 && rows[(size_t)i * NT + 1] != 0.0) return true;
    if (i + 1 < np && rows[(size_t)(i + 1) * NT + 1] != 0.0) return true;
    for (int nc = 1; nc < ipiv[0]; ++nc) {
        const int s = ipiv[nc + 1];
        if (s < 1 || s >= np) continue;
        if (i >= s && rows[(size_t)i * NT + 1 + nc] != 0.0) return true;
    }
    return false;
}

// Row r >= s of a branch starting at s with a fishbone entry: row s-1 is coupled.
__device__ inline void dy_mark_branch_starts(const DyJob &J, int r, int *flag) {
    const int D = J.D;
    if (r < D) return;
    const int part = (r < D + J.nfw) ? 0 : 1;
    const int off = part == 0 ? D : D + J.nfw;
    const int i = r - off, np = part == 0 ? J.nfw : J.nbk;
    if (!(part == 0 ? J.lanczos_fw : J.lanczos_bk)) return;
    const int NT = J.nden + D;
    const double *rows = part == 0 ? J.fw_rows : J.bk_rows;
    const int *ipiv = part == 0 ? J.ipiv_fw : J.ipiv_bk;
    for (int nc = 1; nc < ipiv[0]; ++nc) {
        const int s = ipiv[nc + 1];
        if (s < 1 || s >= np) continue;
        if (i >= s && rows[(size_t)i * NT + 1 + nc] != 0.0) flag[off + s - 1] = 1;
    }
}

constexpr int kTdgMax = 256;   // CTAs of k_tridiag_grid at most
// Its smallest order: a column costs it about the same at any order below 700, the cluster kernel's
// 16 CTAs less up to orders of 350 (a solve of 300: 2.22 against 2.12 ms, 350: 2.52 and 2.55, 400: 2.83
// and 3.00, 500: 3.51 and 4.12)
constexpr int kTdgMin = 384;
// the exchange area in a job's work space (5 n^2 doubles, the spilled rows in the first n^2):
// y[2][n], row k+1 [2][n], parts of v^T A v [2][kTdgMax], the barrier's count (zeroed by
// k_dyson_deflate)
__host__ __device__ inline size_t tdg_exchange(int n) { return 4 * (size_t)n * n; }
__host__ __device__ inline size_t tdg_count(int n) { return tdg_exchange(n) + 4 * (size_t)n + 2 * kTdgMax; }

// One CTA per matrix: the compact index of every kept row (work area, ints; -1 for a
// deflated row), the compact order into the job, and the deflated rows' solutions
// [W, 0, 0 ..] staged behind R after the nc rows the eigensolver will stage.
constexpr int kDfThreads = 1024;

__global__ void __launch_bounds__(kDfThreads) k_dyson_deflate(DyJob *jobs, int njobs, double *work,
                                                              const long long *work_first) {
    const int jid = blockIdx.x;
    if (jid >= njobs) return;
    const DyJob J = jobs[jid];
    const int n = J.n, D = J.D, NS = 2 + D, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int *map = reinterpret_cast<int *>(work + work_first[jid]);
    __shared__ int wsum[kDfThreads / 32][2];
    __shared__ int s_keep, s_defl;
    if (tid == 0) {
        s_keep = 0;
        s_defl = 0;
        if (n > kTsMax) *reinterpret_cast<unsigned *>(work + work_first[jid] + tdg_count(n)) = 0u;   // k_tridiag_grid's
    }
    __syncthreads();
    double *st = J.R + (size_t)D * n;
    int nkept_total = 0;
    // first pass: keep flags (a branch's start row from its later rows' side), then
    // the count of kept rows (the deflated rows' staged positions start after them)
    for (int r = tid; r < n; r += kDfThreads) map[r] = dy_coupled(J, r);
    __syncthreads();
    for (int r = tid; r < n; r += kDfThreads) dy_mark_branch_starts(J, r, map);
    __syncthreads();
    for (int b = 0; b < n; b += kDfThreads) {
        const int r = b + tid;
        const int keep = (r < n) ? map[r] : 0;
        int x = __syncthreads_count(keep);
        nkept_total += x;
    }
    // second pass: ranks among kept / deflated rows, in row order
    for (int b = 0; b < n; b += kDfThreads) {
        const int r = b + tid;
        const int keep = (r < n) ? map[r] : 0, defl = (r < n) ? !keep : 0;
        int xk = keep, xd = defl;
        for (int o = 1; o < 32; o <<= 1) {
            const int yk = __shfl_up_sync(0xffffffffu, xk, o), yd = __shfl_up_sync(0xffffffffu, xd, o);
            if (lane >= o) { xk += yk; xd += yd; }
        }
        if (lane == 31) { wsum[warp][0] = xk; wsum[warp][1] = xd; }
        __syncthreads();
        int ok = s_keep, od = s_defl;
        for (int q = 0; q < warp; ++q) { ok += wsum[q][0]; od += wsum[q][1]; }
        if (r < n) {
            if (keep) {
                map[r] = ok + xk - 1;
            } else {
                map[r] = -1;
                const int part = (r < D + J.nfw) ? 0 : 1;
                const int i = r - (part == 0 ? D : D + J.nfw);
                double *row = st + (size_t)(nkept_total + od + xd - 1) * NS;
                row[0] = dy_diag(J, part, i);
                for (int q = 1; q < NS; ++q) row[q] = 0.0;
            }
        }
        __syncthreads();
        if (tid == kDfThreads - 1) { s_keep = ok + xk; s_defl = od + xd; }
        __syncthreads();
    }
    if (tid == 0) jobs[jid].nc = nkept_total;
}

// One thread per full-matrix row; kept rows are written at their compact index, in a
// matrix of order nc (deflated columns hold zeros in every kept row).  Only the lower
// triangle (columns up to the row's own) is written: the reductions read nothing else,
// and every entry right of the diagonal (a model-space row's pole couplings, the beta
// to the next row, a branch start's fishbone entries) is also left of it in its
// partner row.
__global__ void k_dyson_assemble(const DyJob *jobs, int njobs, const long long *row_first, long long total_rows,
                                 const double *work, const long long *work_first) {
    long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (g >= total_rows) return;
    int lo = 0, hi = njobs - 1;
    while (lo < hi) { int mid = (lo + hi + 1) >> 1; if (row_first[mid] <= g) lo = mid; else hi = mid - 1; }
    const DyJob J = jobs[lo];
    const int r = (int)(g - row_first[lo]);
    const int *map = reinterpret_cast<const int *>(work + work_first[lo]);
    const int cr = map[r];
    if (cr < 0) return;
    const int nc = J.nc, D = J.D, nfw = J.nfw, nbk = J.nbk;
    double *Ar = J.A + (size_t)cr * nc;
    for (int c = 0; c <= cr; ++c) Ar[c] = 0.0;
    auto put = [&](int c, double v) { const int cc = map[c]; if (cc >= 0 && cc <= cr) Ar[cc] = v; };
    if (r < D) {   // the model-space rows are never deflated and come first: cr == r
        for (int c = 0; c <= r; ++c) Ar[c] = J.sig1b[r * D + c] + J.sighf[r * D + c];
        return;
    }
    const int part = (r < D + nfw) ? 0 : 1;
    const int off = part == 0 ? D : D + nfw;
    const int np = part == 0 ? nfw : nbk;
    const int i = r - off;
    const bool lz = part == 0 ? J.lanczos_fw : J.lanczos_bk;
    for (int d = 0; d < D; ++d) Ar[d] = dy_mcoup(J, part, i, d);
    Ar[cr] = dy_diag(J, part, i);
    if (!lz) return;
    const int NT = J.nden + D;
    const double *rows = part == 0 ? J.fw_rows : J.bk_rows;
    const int *ipiv = part == 0 ? J.ipiv_fw : J.ipiv_bk;
    const int nbr = ipiv[0];  // branches (pivots used)
    if (i >= 1) put(r - 1, rows[(size_t)i * NT + 1]);
    // fishbone (:303-333): branch nc (1 .. nbr-1) starts at s = ipiv[nc+1];
    // row s-1 couples to every later row nr >= s with row_nr[1 + nc] (held by row nr)
    for (int nc2 = 1; nc2 < nbr; ++nc2) {
        const int s = ipiv[nc2 + 1];
        if (s < 1 || s >= np) continue;
        if (i >= s) put(off + s - 1, rows[(size_t)i * NT + 1 + nc2]);
    }
}

// ---------------------------------------------------------------- K4a Householder
constexpr int kTdThreads = 256;

__device__ inline double block_sum(double v, double *scratch) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    double s = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += scratch[q];
    return s;
}

// Symmetric Householder reduction on the lower triangle.  Row i belongs to CTA
// (i mod CL) of the cluster, so the shrinking triangle stays balanced; inside a
// CTA the warps take its rows in turn.  One step k (trailing size m = n - k - 1):
//   1. every CTA reads column k below the diagonal and forms the reflector v and
//      tau itself (identical data and order, so identical results and branches);
//   2. one pass over the own rows gives the symmetric product A v: each row's
//      dot product (warp sum) and its transposed contributions A_ij v_i to p_j,
//      gathered in per-warp shared partial vectors (shared atomics only when eight
//      copies do not fit);
//   3. the CTAs' partial vectors are summed through distributed shared memory in
//      rank order; w = tau A v - (tau^2/2)(v^T A v) v;
//   4. the own rows' lower parts get A -= v w^T + w v^T.
// Two FP64 multiply-adds per stored element and step (against three with full
// storage), two cluster barriers per step.  The reflector is kept in row k,
// columns > k (unused by the lower triangle), for the back-transformation.
//
// Shared layout (doubles): v[nmax] | p[nmax] | pc[nmax] | pt[npriv][nmax] |
// pr[nmax / CL + 1] | scratch[32]
// A deflated matrix of order beyond the launch's shared-memory layout (sized for at
// most the largest order that layout can hold): the cluster leaves together before its
// first barrier, the job reports kDyStatCapacity, and a zero tridiagonal with no
// reflectors lets the eigen kernels after it finish on it at once.
__device__ inline void tridiag_beyond_layout(const DyJob &J, int rank) {
    if (rank != 0) return;
    for (int i = threadIdx.x; i < J.nc; i += blockDim.x) { J.d[i] = 0.0; J.e[i] = 0.0; J.tau[i] = 0.0; }
    if (threadIdx.x == 0) *J.stat = kDyStatCapacity;
}

__global__ void __launch_bounds__(kTdThreads) k_tridiag(const DyJob *jobs, int njobs, int nmax, int npriv, int nlim) {
    cg::cluster_group cluster = cg::this_cluster();
    const int CL = (int)cluster.num_blocks();
    const int rank = (int)cluster.block_rank();
    const int jid = blockIdx.x / CL;
    if (jid >= njobs) return;
    const DyJob J = jobs[jid];
    const int n = J.nc;   // order after deflation
    if (n <= nlim) return;   // k_tridiag_small's or k_tridiag_df's (the whole cluster leaves together)
    if (n > nmax) { tridiag_beyond_layout(J, rank); return; }
    extern __shared__ double sm[];
    double *v = sm;
    double *p = v + nmax;
    double *pc = p + nmax;
    double *pt = pc + nmax;
    double *pr = pt + (size_t)npriv * nmax;
    double *scratch = pr + (nmax / CL + 1);
    double *A = J.A;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kWarps = kTdThreads / 32;
    const bool priv = (npriv >= kWarps);
    double *ptw = pt + (size_t)(warp % npriv) * nmax;
    for (int k = 0; k + 2 < n; ++k) {
        const int b0 = k + 1, m = n - b0;
        // 1. reflector from column k (rows > k)
        double sig = 0.0;
        for (int t = 1 + tid; t < m; t += kTdThreads) { const double x = __ldcg(A + (size_t)(b0 + t) * n + k); sig += x * x; }
        sig = block_sum(sig, scratch);
        const double alpha = __ldcg(A + (size_t)b0 * n + k);
        double tau = 0.0, beta = alpha;
        if (sig != 0.0) {
            beta = -copysign(sqrt(alpha * alpha + sig), alpha);
            tau = (beta - alpha) / beta;
            const double scal = 1.0 / (alpha - beta);
            for (int t = tid; t < m; t += kTdThreads) v[t] = (t == 0) ? 1.0 : __ldcg(A + (size_t)(b0 + t) * n + k) * scal;
        }
        if (rank == 0 && tid == 0) { J.e[k] = beta; J.tau[k] = tau; J.d[k] = __ldcg(A + (size_t)k * n + k); }
        if (sig != 0.0) {
            for (int t = tid; t < npriv * m; t += kTdThreads) pt[(size_t)(t / m) * nmax + t % m] = 0.0;
            __syncthreads();
            // 2. own rows i = first, first + CL, ...; row part and transposed part of A v
            const int first = b0 + ((rank - b0 % CL) % CL + CL) % CL;
            for (int i = first + warp * CL; i < n; i += CL * kWarps) {
                const double *Ai = A + (size_t)i * n;
                const double vi = v[i - b0];
                double rs = 0.0;
                int j = b0 + lane;
                for (; j + 96 < i; j += 128) {
                    const double a0 = __ldcg(Ai + j), a1 = __ldcg(Ai + j + 32), a2 = __ldcg(Ai + j + 64),
                                 a3 = __ldcg(Ai + j + 96);
                    const int t = j - b0;
                    rs += a0 * v[t] + a1 * v[t + 32] + a2 * v[t + 64] + a3 * v[t + 96];
                    if (priv) {
                        ptw[t] += a0 * vi; ptw[t + 32] += a1 * vi; ptw[t + 64] += a2 * vi; ptw[t + 96] += a3 * vi;
                    } else {
                        atomicAdd(ptw + t, a0 * vi); atomicAdd(ptw + t + 32, a1 * vi);
                        atomicAdd(ptw + t + 64, a2 * vi); atomicAdd(ptw + t + 96, a3 * vi);
                    }
                }
                for (; j <= i; j += 32) {
                    const double a = __ldcg(Ai + j);
                    rs += a * v[j - b0];
                    if (j < i) {
                        if (priv) ptw[j - b0] += a * vi;
                        else atomicAdd(ptw + (j - b0), a * vi);
                    }
                }
                for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
                if (lane == 0) pr[(i - first) / CL] = rs;
            }
            __syncthreads();
            // this CTA's share of A v: transposed partials plus its own rows' sums
            for (int t = tid; t < m; t += kTdThreads) {
                double s = 0.0;
                for (int q = 0; q < npriv; ++q) s += pt[(size_t)q * nmax + t];
                const int i = b0 + t;
                if (i >= first && (i - first) % CL == 0) s += pr[(i - first) / CL];
                pc[t] = s;
            }
            cluster.sync();
            // 3. p = tau A v summed over the cluster in rank order; w = p - (tau/2)(p.v) v
            double kv = 0.0;
            for (int t = tid; t < m; t += kTdThreads) {
                double s = 0.0;
                for (int r = 0; r < CL; ++r) s += cluster.map_shared_rank(pc, r)[t];
                s *= tau;
                p[t] = s;
                kv += s * v[t];
            }
            const double K = block_sum(kv, scratch);
            for (int t = tid; t < m; t += kTdThreads) p[t] -= 0.5 * tau * K * v[t];
            __syncthreads();
            // 4. A_ij -= v_i w_j + w_i v_j on the own rows, j <= i
            for (int i = first + warp * CL; i < n; i += CL * kWarps) {
                double *Ai = A + (size_t)i * n;
                const double vi = v[i - b0], wi = p[i - b0];
                int j = b0 + lane;
                for (; j + 96 <= i; j += 128) {
                    const int t = j - b0;
                    const double a0 = __ldcg(Ai + j), a1 = __ldcg(Ai + j + 32), a2 = __ldcg(Ai + j + 64),
                                 a3 = __ldcg(Ai + j + 96);
                    Ai[j] = a0 - (vi * p[t] + wi * v[t]);
                    Ai[j + 32] = a1 - (vi * p[t + 32] + wi * v[t + 32]);
                    Ai[j + 64] = a2 - (vi * p[t + 64] + wi * v[t + 64]);
                    Ai[j + 96] = a3 - (vi * p[t + 96] + wi * v[t + 96]);
                }
                for (; j <= i; j += 32) Ai[j] = __ldcg(Ai + j) - (vi * p[j - b0] + wi * v[j - b0]);
            }
            if (rank == 0)
                for (int t = tid; t < m; t += kTdThreads) A[(size_t)k * n + b0 + t] = v[t];
        }
        cluster.sync();
    }
    if (rank == 0 && tid == 0) {
        if (n >= 2) {
            J.d[n - 2] = __ldcg(A + (size_t)(n - 2) * n + (n - 2));
            J.e[n - 2] = __ldcg(A + (size_t)(n - 1) * n + (n - 2));
            J.tau[n - 2] = 0.0;
        }
        J.d[n - 1] = __ldcg(A + (size_t)(n - 1) * n + (n - 1));
        J.e[n - 1] = 0.0;
        J.tau[n - 1] = 0.0;
    }
    cluster.sync();
}

// ---------------------------------------------------------------- K4a'' clusters, one pass a column
// Orders beyond kTsMax: a cluster per matrix, row i with CTA (i mod CL), both triangles of a
// row (so a row's product needs no other CTA's partial sums), in double-float (df64.cuh).
// Rows live in shared memory, the last ones first (they stay longest); those that do not fit
// in the job's work area.  Step k (trailing rows and columns > k) takes one pass over the
// matrix instead of a product and an update: the pass applies step k-1's rank-2 update and
// multiplies by step k's column as it goes.  The column is used as it is (v is x but for a power
// of two and its first entry), so the reflector's scalars are formed by one warp beside the pass:
//   pass      a_ij -= v'_i w'_j + w'_i v'_j (v', w' of step k-1), S_i = sum_{j>k+1} a_ij x_j, two
//             rows a warp; the same product for this CTA's rows of R; warp kTdScal: |x|^2 from
//             the CTAs' partial sums, then h, v_0 and g
//   own rows  y_i = v_0 a_i,k+1 + g S_i = (A v)_i to every CTA, with the warps' partials of v^T A v;
//             cluster barrier
//   all rows  v = g x, w = h y - (h^2 / 2) (v^T A v) v; R -= h (R v) v^T (R in FP64)
//   own rows  column k+1 of the updated matrix to every CTA (x of the next step, d_{k+1} from
//             the diagonal), with the partials of its square; cluster barrier
// Bound by these two cluster barriers and the chains between them (about 4 000 cycles a
// column) up to orders of a few hundred, by the FP32 pipe (41 instructions an element)
// beyond.  Against the two passes from L2 with eight warps that this replaced, and k_qrows
// for R (one CTA, FP64, a pass of its own): order 1 000 alone on 16 CTAs 34.4 + 6.4 -> 13.0 ms,
// a batch of orders up to 205 on 8 CTAs each 1.99 + 0.96 -> 0.69 ms (0.68 with R in double-float and v
// rounded, which took an eigenvector's components 3 to 11 % further off).
namespace {

// x as hi + lo from its bits: hi the double truncated to FP32, lo the next bits of the
// significand (rounded to FP32), then renormalised; no FP64 instruction (values inside
// the FP32 range; below it, zero)
__device__ inline dfm::df df_from_bits(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int E = (int)((b >> 52) & 0x7FF) - 1023;
    if (E < -126) return dfm::df{0.0f, 0.0f};
    const unsigned s = (unsigned)(b >> 63) << 31;
    const float hi = __uint_as_float(s | ((unsigned)(E + 127) << 23) | (unsigned)((b >> 29) & 0x7FFFFFu));
    // remainder (b & (2^29 - 1)) 2^(E - 52); below 2^-126 the factor goes in two steps
    float lo = __uint2float_rn((unsigned)(b & 0x1FFFFFFFull));
    if (E - 52 >= -126) {
        lo = __fmul_rn(lo, __uint_as_float((unsigned)(E - 52 + 127) << 23));
    } else {
        lo = __fmul_rn(lo, __uint_as_float((unsigned)(E - 52 + 64 + 127) << 23));
        lo = __fmul_rn(lo, 5.42101086242752217e-20f);   // 2^-64
    }
    if (s) lo = -lo;
    return dfm::renorm(hi, lo);
}

// a pair's value, one FP64 instruction (the conversions from the words' bits)
__device__ __forceinline__ double df_value(dfm::df a) { return f32_to_double(a.h) + f32_to_double(a.l); }

__device__ inline int f32_exponent(float x) { return (int)((__float_as_uint(x) >> 23) & 255u) - 127; }
__device__ inline float pow2_f32(int e) { return __uint_as_float((unsigned)(e + 127) << 23); }

constexpr int kTdfThreads = 512, kTdfWarps = kTdfThreads / 32, kTdScal = kTdfWarps - 1;

// 8-byte slots before the resident rows: V[2], W[2], the partials kb and sb, R rows, S and
// a_{i,k+1} of own rows
__host__ __device__ inline size_t tdf_fixed(int n, int CL, int D) {
    const int nrm = (n + CL - 1) / CL;
    return (size_t)(4 + (D + CL - 1) / CL) * n + 2 * (size_t)nrm + 2 * (size_t)CL * kTdfWarps + 32;
}

__device__ __forceinline__ dfm::df scaled(dfm::df a, float g) { return dfm::df{dfm::fmul(a.h, g), dfm::fmul(a.l, g)}; }

// The reflector H = 1 - h v v^T that takes a column x = (alpha, x_1, ..) to (beta, 0, ..): v = g x
// but for v_0 = g (alpha - beta), with g a power of two that brings |x| to about one, so v holds
// x's own bits and the products A x formed before the scalars were known are A v's.  s2: |x_1:|^2;
// h is zero when there is nothing to reflect.
struct Reflector { dfm::df h, v0, beta; float g; };
__device__ __forceinline__ Reflector reflector(dfm::df al, dfm::df s2) {
    using dfm::df;
    Reflector o{df{0.0f, 0.0f}, df{0.0f, 0.0f}, al, 1.0f};
    if (s2.h != 0.0f || s2.l != 0.0f) {
        const int ea = (al.h != 0.0f) ? f32_exponent(al.h) : -1000;
        int e = max(ea, f32_exponent(s2.h) >> 1);
        e = min(max(e, -126), 126);
        o.g = pow2_f32(-e);
        const df alt = scaled(al, o.g), x2 = dfm::fma(alt, alt, scaled(scaled(s2, o.g), o.g));   // in [1, 12)
        const df r = dfm::rsqrt2(x2), nx = dfm::mul(x2, r);
        const bool ng = signbit(alt.h);
        const df u = dfm::add(ng ? dfm::neg(alt) : alt, nx);   // |alpha| + |x|
        o.h = dfm::mul(r, dfm::rcp2(u));                       // 2 / v^T v
        o.v0 = ng ? dfm::neg(u) : u;
        o.beta = scaled(ng ? nx : dfm::neg(nx), pow2_f32(e));
    }
    return o;
}

// a - (vi wj + wi vj): both products exact to ~2^-48, summed before they meet a; the same bits
// with i and j exchanged, so the two triangles stay equal
__device__ __forceinline__ dfm::df rank2(dfm::df a, dfm::df vi, dfm::df wj, dfm::df wi, dfm::df vj) {
    const float p = dfm::fmul(vi.h, wj.h), q = dfm::fmul(wi.h, vj.h);
    float e = dfm::ffma(vi.h, wj.h, -p);
    e = dfm::ffma(vi.h, wj.l, e);
    e = dfm::ffma(vi.l, wj.h, e);
    float f = dfm::ffma(wi.h, vj.h, -q);
    f = dfm::ffma(wi.l, vj.h, f);
    f = dfm::ffma(wi.h, vj.l, f);
    float s, r, t, u;
    dfm::two_sum(p, q, s, r);
    dfm::two_sum(a.h, -s, t, u);
    return dfm::renorm(t, dfm::fadd(dfm::fadd(u, a.l), -dfm::fadd(r, dfm::fadd(e, f))));
}

}  // namespace

template <int CL>
__global__ void __launch_bounds__(kTdfThreads, 1) k_tridiag_df(const DyJob *jobs, int njobs, int nlim, int smem_df,
                                                               double *work, const long long *work_first) {
    using dfm::df;
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank();
    const int jid = blockIdx.x / CL;
    if (jid >= njobs) return;
    const DyJob J = jobs[jid];
    const int n = J.nc, D = J.D;
    beside_release();
    if (n <= kTsMax || n > nlim) return;   // another kernel's (the whole cluster leaves together)
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrm = (n + CL - 1) / CL, nr = (n - rank + CL - 1) / CL;   // own rows i = rank + q CL, q < nr
    const int NRR = (D - rank + CL - 1) / CL;                            // own rows of R: d = rank + u CL (<= 0: none)
    constexpr int RW = 32 / CL;                  // own rows per warp in the own-rows phases, a lane per (row, CTA)
    extern __shared__ double sm[];
    df *V = reinterpret_cast<df *>(sm);          // [2][n]
    df *W = V + 2 * (size_t)n;                   // [2][n]
    df *kb = W + 2 * (size_t)n;                  // [kTdfWarps][CL] partials of v . y
    df *sb = kb + (size_t)CL * kTdfWarps;        // [kTdfWarps][CL] partials of |x_1:|^2
    double *R = reinterpret_cast<double *>(sb + (size_t)CL * kTdfWarps);   // [NRR][n]
    df *rs = reinterpret_cast<df *>(R + (size_t)((D + CL - 1) / CL) * n);   // [nrm] S of own rows
    df *ra = rs + nrm;                           // [nrm] a_{i,k+1}
    df *rows = reinterpret_cast<df *>(sm) + tdf_fixed(n, CL, D);
    const int room = max(0, (smem_df - (int)tdf_fixed(n, CL, D)) / n);
    const int qs = max(0, nr - room);            // own rows q >= qs in shared memory
    df *spill = reinterpret_cast<df *>(work + work_first[jid]);
    auto row = [&](int q) -> df * { return q >= qs ? rows + (size_t)(q - qs) * n : spill + (size_t)(rank + q * CL) * n; };
    __shared__ df s_sc[2];      // h, v_0 of the step
    __shared__ float s_g;       // and the power of two that scales x
    __shared__ double s_rd[8], s_c[8];   // R_d . x_{1:} of own R rows, -h R_d . v
    const df zero{0.0f, 0.0f};
    // d and e stay double-float pairs in their FP64 slots until the end: a conversion is
    // two FP64 instructions on a chain that other warps wait for
    auto put = [](double *p, df x) { *reinterpret_cast<float2 *>(p) = make_float2(x.h, x.l); };
    // the sum of cnt values by a warp, the same in every lane
    auto sum_of = [&](const df *p, int cnt) {
        df t = lane < cnt ? p[lane] : zero;
        for (int e = lane + 32; e < cnt; e += 32) t = dfm::add(t, p[e]);
        return dfm::warp_sum(t);
    };
    // this CTA's rows, both triangles, from the assembled lower one
    for (int q = warp; q < nr; q += kTdfWarps) {
        const int i = rank + q * CL;
        df *a = row(q);
        for (int j = lane; j < n; j += 32) a[j] = df_from_bits(__ldcg(J.A + (j <= i ? (size_t)i * n + j : (size_t)j * n + i)));
    }
    df sq0 = zero;
    for (int j = tid; j < n; j += kTdfThreads) {
        const df xj = df_from_bits(__ldcg(J.A + (size_t)j * n));   // x of step 0
        V[j] = xj;
        V[n + j] = zero;
        W[n + j] = zero;
        for (int u = 0; u < NRR; ++u) R[(size_t)u * n + j] = (j == rank + u * CL) ? 1.0 : 0.0;
        if (j >= 2) sq0 = dfm::fma(xj, xj, sq0);
    }
    // the squares of column 0, summed by every CTA for itself
    sq0 = dfm::warp_sum(sq0);
    if (lane == 0) sb[warp] = sq0;
    int nsb = kTdfWarps;        // partials of |x_1:|^2
    if (rank == 0 && tid == 0) put(J.d, V[0]);
    cluster.sync();   // every CTA runs, and this CTA's arrays are set
    int cur = 0;
    for (int k = 0; k + 2 < n; ++k, cur ^= 1) {
        df *x = V + (size_t)cur * n, *vp = V + (size_t)(cur ^ 1) * n;
        df *y = W + (size_t)cur * n, *wp = W + (size_t)(cur ^ 1) * n;
        const int b0 = k + 1;
        const int q0 = (unsigned)(b0 - rank + CL - 1) / CL;   // first own row >= b0 (b0 - rank + CL - 1 >= 1)
        // pass
        if (warp == kTdScal) {
            const df s2 = sum_of(sb, nsb);
            const Reflector r = reflector(x[b0], s2);
            if (lane == 0) {
                s_sc[0] = r.h;
                s_sc[1] = r.v0;
                s_g = r.g;
                if (rank == 0) put(J.e + k, r.beta);
            }
        }
        {   // the active own rows in runs of consecutive ones, one run a warp (the scalars' warp
            // after them, the first to go without); two rows at a time share the vectors' loads,
            // and the next columns' entries are loaded before this one's are used
            const int na = nr - q0;
            const int per = na / kTdfWarps, ext = na - per * kTdfWarps;
            int q = q0 + warp * per + min(warp, ext);
            const int q1 = q + per + (warp < ext ? 1 : 0);
            for (; q < q1; q += 2) {
                const bool two = q + 1 < q1;
                df *a0 = row(q);
                const int i0 = rank + q * CL;
                const df v0 = vp[i0], w0 = wp[i0];
                if (two) {
                    df *a1 = row(q + 1);
                    const df v1 = vp[i0 + CL], w1 = wp[i0 + CL];
                    df s0 = zero, s1 = zero;
                    int j = b0 + lane;
                    df p0 = j < n ? a0[j] : zero, p1 = j < n ? a1[j] : zero;
                    for (; j < n; j += 32) {
                        const int jn = min(j + 32, n - 1);
                        const df n0 = a0[jn], n1 = a1[jn];
                        const df vj = vp[j], wj = wp[j], xj = (j == b0) ? zero : x[j];
                        const df t0 = rank2(p0, v0, wj, w0, vj), t1 = rank2(p1, v1, wj, w1, vj);
                        a0[j] = t0;
                        a1[j] = t1;
                        s0 = dfm::fma(t0, xj, s0);
                        s1 = dfm::fma(t1, xj, s1);
                        if (j == b0) { ra[q] = t0; ra[q + 1] = t1; }
                        p0 = n0;
                        p1 = n1;
                    }
                    s0 = dfm::warp_sum(s0);
                    s1 = dfm::warp_sum(s1);
                    if (lane == 0) { rs[q] = s0; rs[q + 1] = s1; }
                } else {
                    df s0 = zero, s1 = zero;   // two columns at a time
                    for (int j = b0 + lane; j < n; j += 64) {
                        const bool in = j + 32 < n;
                        const int j2 = in ? j + 32 : j;
                        const df p0 = a0[j], p1 = a0[j2];
                        const df t0 = rank2(p0, v0, wp[j], w0, vp[j]), t1 = rank2(p1, v0, wp[j2], w0, vp[j2]);
                        a0[j] = t0;
                        if (in) a0[j2] = t1;
                        s0 = dfm::fma(t0, (j == b0) ? zero : x[j], s0);
                        s1 = dfm::fma(t1, in ? x[j2] : zero, s1);
                        if (j == b0) ra[q] = t0;
                    }
                    s0 = dfm::warp_sum(dfm::add(s0, s1));
                    if (lane == 0) rs[q] = s0;
                }
            }
            // R_d . x_{1:} of own R rows, from the warps before the scalars' one
            if (warp < kTdScal && kTdScal - 1 - warp < NRR) {
                const int u = kTdScal - 1 - warp;
                const double *r = R + (size_t)u * n;
                double t = 0.0;
                for (int j = b0 + 1 + lane; j < n; j += 32) t = fma(r[j], df_value(x[j]), t);
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0) s_rd[u] = t;
            }
        }
        __syncthreads();
        const df hs = s_sc[0], v0 = s_sc[1];
        const float g = s_g;
        const bool nz = (hs.h != 0.0f);
        // own rows, a lane per (row, receiving CTA): y to every CTA, partials of v . y (of the
        // warp's RW rows, the same count of warps in every CTA)
        const int wpk = min(kTdfWarps, (int)((unsigned)((n - b0 + CL - 1) / CL + RW - 1) / RW));
        const int to = lane % CL, q_ = q0 + warp * RW + lane / CL;
        if (warp == kTdScal && lane < NRR)
            s_c[lane] = -df_value(hs) * fma(df_value(v0), R[(size_t)lane * n + b0], (double)g * s_rd[lane]);
        if (warp < wpk) {
            df kv = zero;
            df *yr = cluster.map_shared_rank(y, to);
            for (int q = q_; q < nr; q += kTdfWarps * RW) {
                const int i = rank + q * CL;
                const df yi = nz ? dfm::fma(v0, ra[q], scaled(rs[q], g)) : zero;
                yr[i] = yi;
                kv = dfm::fma((i == b0) ? v0 : scaled(x[i], g), yi, kv);
            }
#pragma unroll
            for (int o = 16; o >= CL; o >>= 1) kv = dfm::add(kv, dfm::shfl_xor(kv, o));
            if (lane < CL) cluster.map_shared_rank(kb, to)[warp * CL + rank] = kv;
        }
        cluster.sync();
        // all rows: v, w; R
        {
            const df K = sum_of(kb, wpk * CL);
            const df hh = dfm::mul(hs, hs);
            const df nK = dfm::neg(dfm::mul(df{0.5f * hh.h, 0.5f * hh.l}, K));
            for (int j = b0 + tid; j < n; j += kTdfThreads) {
                const df vj = !nz ? zero : (j == b0) ? v0 : scaled(x[j], g);
                y[j] = dfm::fma(nK, vj, dfm::mul(hs, y[j]));
                x[j] = vj;
                for (int u = 0; u < NRR; ++u) R[(size_t)u * n + j] = fma(s_c[u], df_value(vj), R[(size_t)u * n + j]);
            }
        }
        __syncthreads();
        // own rows: column k+1 of the updated matrix
        if (warp < wpk) {
            const df vb = x[b0], wb = y[b0];
            df *xr = cluster.map_shared_rank(vp, to);
            df sq = zero;
            for (int q = q_; q < nr; q += kTdfWarps * RW) {
                const int i = rank + q * CL;
                const df t = rank2(row(q)[b0], x[i], wb, y[i], vb);
                if (i == b0) {
                    if (to == 0) put(J.d + b0, t);
                } else {
                    xr[i] = t;
                    if (i > b0 + 1) sq = dfm::fma(t, t, sq);
                    if (k + 3 == n && to == 0) {   // the last step: e_{n-2}, and the last diagonal entry
                        put(J.e + n - 2, t);
                        put(J.d + n - 1, rank2(row(q)[n - 1], x[i], y[i], y[i], x[i]));
                    }
                }
            }
#pragma unroll
            for (int o = 16; o >= CL; o >>= 1) sq = dfm::add(sq, dfm::shfl_xor(sq, o));
            if (lane < CL) cluster.map_shared_rank(sb, to)[warp * CL + rank] = sq;
        }
        nsb = wpk * CL;
        cluster.sync();
    }
    if (rank == 0)   // every CTA's entries are visible since the last barrier
        for (int j = tid; j < n; j += kTdfThreads) {
            auto conv = [](double *p) { const float2 f = __ldcg(reinterpret_cast<const float2 *>(p)); *p = dfm::to_double(df{f.x, f.y}); };
            conv(J.d + j);
            if (j + 1 < n) conv(J.e + j); else J.e[j] = 0.0;
        }
    for (int u = 0; u < NRR; ++u)
        for (int j = tid; j < n; j += kTdfThreads) J.R[(size_t)(rank + u * CL) * n + j] = R[(size_t)u * n + j];
}

// ---------------------------------------------------------------- K4a''' one matrix, the whole GPU
// A matrix reduced alone leaves a cluster's 16 SMs to do the pass and most of its rows in L2 (order
// 1 000: 25 000 cycles a column, two thirds of them the pass).  Here every SM takes part: a
// cooperative launch, one CTA an SM, row i with CTA (i mod H), and what the CTAs exchange goes
// through L2.  The last D CTAs have a row of R each and none of the matrix: R is FP64, and 2 n of
// its instructions a column beside a CTA's own rows would hold up the barrier (order 1 000: 5.6 ms
// for 4.7), in the time the others take for the pass they do not.  Step k, with one grid barrier:
//   pass      as k_tridiag_df's, 1 to 4 warps a row; R_d . x
//   own rows  y_i = v_0 a_i,k+1 + g S_i and the CTA's part of v^T A v; from its owner row k+1; barrier
//   all rows  v, w, R; from row k+1, which is column k+1, that column after this step's update (x
//             of the next step, d_{k+1} on the diagonal), and the sum of its squares, by every CTA
//             for itself
// Bound by the barrier and what surrounds it in a column (order 1 000, 9 900 cycles: of 9 000 in an
// earlier form the pass beside the scalars' chain was 3 000, y 1 000, the barrier 3 200, then L2, the
// sum of the parts, v and w).  Order 1 000: 13.0 ms by the cluster kernel -> 4.8.
constexpr int kTdgRowWarps = kTdfWarps - 1;   // the other: the scalars
constexpr int kTdgParts = 4;                  // warps a row at most
constexpr int kTdgPolls = 1 << 20;            // a barrier's reads before it gives up (about a second)

// 8-byte slots before the resident rows (H CTAs with rows): V[2], W, one row of R, S by parts and
// a_{i,k+1} of own rows
__host__ __device__ inline size_t tdg_fixed(int n, int H) {
    return 4 * (size_t)n + (kTdgParts + 1) * (size_t)((n + H - 1) / H) + kTdfWarps + 16;
}
__global__ void __launch_bounds__(kTdfThreads, 1) k_tridiag_grid(const DyJob *jobs, int nlim, int smem_df, double *work,
                                                                 const long long *work_first) {
    using dfm::df;
    __shared__ DyJob J;
    __shared__ int s_ok;
    const int G = gridDim.x, rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < (int)(sizeof(DyJob) / 4)) reinterpret_cast<int *>(&J)[tid] = reinterpret_cast<const int *>(jobs)[tid];
    if (tid == 0) s_ok = 1;
    __syncthreads();
    const int n = J.nc, D = J.D;
    if (n < kTdgMin || n > nlim) return;   // another kernel's (the whole grid leaves)
    const int H = G - D;   // CTAs with rows of the matrix; the others have row rank - H of R
    const bool own_r = rank >= H;
    const int nrm = (n + H - 1) / H, nr = !own_r && rank < n ? (n - rank + H - 1) / H : 0;   // own rows i = rank + q H
    extern __shared__ double sm[];
    df *V = reinterpret_cast<df *>(sm);          // [2][n]
    df *w = V + 2 * (size_t)n;                   // [n]
    double *R = reinterpret_cast<double *>(w + n);   // [n] the own row of R
    df *rs = reinterpret_cast<df *>(R + n);      // [kTdgParts][nrm] parts of S of own rows
    df *ra = rs + (size_t)kTdgParts * nrm;       // [nrm] a_{i,k+1}
    df *sb = ra + nrm;                           // [kTdfWarps] partials of |x_1:|^2
    df *rows = reinterpret_cast<df *>(sm) + tdg_fixed(n, H);
    const int room = max(0, (smem_df - (int)tdg_fixed(n, H)) / n);
    const int qs = max(0, nr - room);            // own rows q >= qs in shared memory
    double *wk = work + work_first[0];
    df *spill = reinterpret_cast<df *>(wk);
    auto row = [&](int q) -> df * { return q >= qs ? rows + (size_t)(q - qs) * n : spill + (size_t)(rank + q * H) * n; };
    df *Yx = reinterpret_cast<df *>(wk + tdg_exchange(J.n)), *Bx = Yx + 2 * (size_t)n, *Kx = Bx + 2 * (size_t)n;
    unsigned *count = reinterpret_cast<unsigned *>(wk + tdg_count(J.n));
    __shared__ df s_sc[2];              // h, v_0 of the step
    __shared__ float s_g;               // and the power of two that scales x
    __shared__ double s_rd[kTdfWarps], s_c;   // parts of R_d . x of the own R row, -h R_d . v
    __shared__ df s_k[2];               // -(h^2 / 2) v^T A v, w_{k+1}
    const df zero{0.0f, 0.0f};
    auto put = [](double *p, df x) { *reinterpret_cast<float2 *>(p) = make_float2(x.h, x.l); };
    auto far = [](const df *p) { const float2 f = __ldcg(reinterpret_cast<const float2 *>(p)); return df{f.x, f.y}; };
    for (int q = warp; q < nr; q += kTdfWarps) {
        const int i = rank + q * H;
        df *a = row(q);
        for (int j = lane; j < n; j += 32) a[j] = df_from_bits(__ldcg(J.A + (j <= i ? (size_t)i * n + j : (size_t)j * n + i)));
    }
    df sq0 = zero;
    for (int j = tid; j < n; j += kTdfThreads) {
        const df xj = df_from_bits(__ldcg(J.A + (size_t)j * n));   // x of step 0
        V[j] = xj;
        V[n + j] = zero;
        w[j] = zero;
        R[j] = (j == rank - H) ? 1.0 : 0.0;
        if (j >= 2) sq0 = dfm::fma(xj, xj, sq0);
    }
    sq0 = dfm::warp_sum(sq0);
    if (lane == 0) sb[warp] = sq0;
    if (rank == 0 && tid == 0) put(J.d, V[0]);
    __syncthreads();
    int cur = 0;
    for (int k = 0; k + 2 < n; ++k, cur ^= 1) {
        df *x = V + (size_t)cur * n, *vp = V + (size_t)(cur ^ 1) * n;
        df *yk = Yx + (size_t)cur * n, *bk = Bx + (size_t)cur * n, *kb = Kx + (size_t)cur * kTdgMax;
        const int b0 = k + 1;
        const int q0 = b0 <= rank ? 0 : (b0 - rank + H - 1) / H;   // first own row >= b0
        const int na = max(0, nr - q0);
        const int np = 4 * na <= kTdgRowWarps ? 4 : 2 * na <= kTdgRowWarps ? 2 : 1;
        // pass
        if (warp == kTdScal) {
            df s2 = lane < kTdfWarps ? sb[lane] : zero;
            s2 = dfm::warp_sum(s2);
            const Reflector r = reflector(x[b0], s2);
            if (lane == 0) {
                s_sc[0] = r.h;
                s_sc[1] = r.v0;
                s_g = r.g;
                if (rank == 0) put(J.e + k, r.beta);
            }
        } else if (own_r) {   // R_d . x_{1:}
            double t = 0.0;
            for (int j = b0 + 1 + tid; j < n; j += 32 * kTdScal) t = fma(R[j], df_value(x[j]), t);
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) s_rd[warp] = t;
        } else {
            for (int u = warp; u < na * np; u += kTdgRowWarps) {
                const int q = q0 + u / np, part = u % np, i0 = rank + q * H;
                df *a0 = row(q);
                const df v0 = vp[i0], w0 = w[i0];
                df s0 = zero, s1 = zero;   // two columns at a time
                for (int j = b0 + 32 * part + lane; j < n; j += 64 * np) {
                    const bool in = j + 32 * np < n;
                    const int j2 = in ? j + 32 * np : j;
                    const df p0 = a0[j], p1 = a0[j2];
                    const df t0 = rank2(p0, v0, w[j], w0, vp[j]), t1 = rank2(p1, v0, w[j2], w0, vp[j2]);
                    a0[j] = t0;
                    if (in) a0[j2] = t1;
                    s0 = dfm::fma(t0, (j == b0) ? zero : x[j], s0);
                    s1 = dfm::fma(t1, in ? x[j2] : zero, s1);
                    if (j == b0) ra[q] = t0;
                }
                s0 = dfm::warp_sum(dfm::add(s0, s1));
                if (lane == 0) rs[(size_t)part * nrm + q] = s0;
            }
        }
        __syncthreads();
        const df hs = s_sc[0], v0 = s_sc[1];
        const float g = s_g;
        const bool nz = (hs.h != 0.0f);
        if (warp == 0 && !own_r) {   // y of own rows, and their part of v . y
            df kv = zero;
            for (int q = q0 + lane; q < nr; q += 32) {
                const int i = rank + q * H;
                df S = rs[q];
                for (int p = 1; p < np; ++p) S = dfm::add(S, rs[(size_t)p * nrm + q]);
                const df yi = nz ? dfm::fma(v0, ra[q], scaled(S, g)) : zero;
                yk[i] = yi;
                kv = dfm::fma((i == b0) ? v0 : scaled(x[i], g), yi, kv);
            }
            kv = dfm::warp_sum(kv);
            if (lane == 0) kb[rank] = kv;
        } else if (b0 % H == rank) {   // row k+1 (not with an R row's CTA: rank < H)
            const df *a = row(q0);
            for (int j = b0 + tid - 32; j < n; j += kTdfThreads - 32) bk[j] = a[j];
        }
        // every CTA's count of this step; a CTA that waits in vain marks the job and all leave
        __syncthreads();
        if (tid == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
            const unsigned want = (unsigned)(k + 1) * (unsigned)G;
            unsigned c = 0;
            int polls = 0;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
            } while (c < want && ++polls < kTdgPolls);
            if (c < want) s_ok = 0;
        }
        __syncthreads();
        if (!s_ok) {
            if (tid == 0) atomicExch(J.stat, kDyStatBarrier);
            return;
        }
        // all rows: v, w; R; x of the next step
        {
            // all that comes from L2 first; the parts' sum and what follows from it by one warp (by every
            // warp it takes the FP32 pipe from the others: 2 700 cycles)
            constexpr int NA = 2;   // rows a thread has ahead
            df ya[NA], ba[NA];
#pragma unroll
            for (int h = 0; h < NA; ++h) {
                const int j = min(b0 + tid + h * kTdfThreads, n - 1);
                ya[h] = far(yk + j);
                ba[h] = far(bk + j);
            }
            const df vb = nz ? v0 : zero;
            if (warp == 0) {
                df ka[kTdgMax / 32];
#pragma unroll
                for (int h = 0; h < kTdgMax / 32; ++h) ka[h] = lane + 32 * h < H ? far(kb + lane + 32 * h) : zero;
                const df yb = far(yk + b0);
#pragma unroll
                for (int o = kTdgMax / 64; o > 0; o >>= 1)
#pragma unroll
                    for (int h = 0; h < o; ++h) ka[h] = dfm::add(ka[h], ka[h + o]);
                const df K = dfm::warp_sum(ka[0]);
                const df hh = dfm::mul(hs, hs);
                const df nk = dfm::neg(dfm::mul(df{0.5f * hh.h, 0.5f * hh.l}, K));
                const df wk1 = dfm::fma(nk, vb, dfm::mul(hs, yb));
                if (lane == 0) { s_k[0] = nk; s_k[1] = wk1; }
            } else if (warp == 1 && own_r) {
                double t = lane < kTdScal ? s_rd[lane] : 0.0;
                for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0) s_c = -df_value(hs) * fma(df_value(v0), R[b0], (double)g * t);
            }
            __syncthreads();   // (R_{b0} changes behind it too)
            const df nK = s_k[0], wb = s_k[1];
            df sq = zero;
            auto one_row = [&](int j, df yj, df bj) {
                const df vj = !nz ? zero : (j == b0) ? v0 : scaled(x[j], g);
                const df wj = dfm::fma(nK, vj, dfm::mul(hs, yj));
                const df t = rank2(bj, vj, wb, wj, vb);
                w[j] = wj;
                x[j] = vj;
                vp[j] = t;
                if (j > b0 + 1) sq = dfm::fma(t, t, sq);
                if (rank == 0 && j == b0) put(J.d + b0, t);
                if (rank == 0 && j == b0 + 1 && k + 3 == n) put(J.e + n - 2, t);
                if (k + 3 == n && j == n - 1 && (n - 1) % H == rank)   // the last step: the last diagonal entry
                    J.d[n - 1] = dfm::to_double(rank2(row(nr - 1)[n - 1], vj, wj, wj, vj));
                if (own_r) R[j] = fma(s_c, df_value(vj), R[j]);
            };
#pragma unroll
            for (int h = 0; h < NA; ++h)
                if (b0 + tid + h * kTdfThreads < n) one_row(b0 + tid + h * kTdfThreads, ya[h], ba[h]);
            for (int j = b0 + tid + NA * kTdfThreads; j < n; j += kTdfThreads) one_row(j, far(yk + j), far(bk + j));
            sq = dfm::warp_sum(sq);
            if (lane == 0) sb[warp] = sq;
        }
        __syncthreads();
    }
    if (rank == 0)
        for (int j = tid; j < n; j += kTdfThreads) {
            auto conv = [](double *p) { const float2 f = __ldcg(reinterpret_cast<const float2 *>(p)); *p = dfm::to_double(df{f.x, f.y}); };
            if (j + 1 < n) { conv(J.d + j); conv(J.e + j); } else J.e[j] = 0.0;
        }
    if (own_r)
        for (int j = tid; j < n; j += kTdfThreads) J.R[(size_t)(rank - H) * n + j] = R[j];
}

// the kernel for a cluster size (1, 2, 4, 8 or 16)
static auto tridiag_df_kernel(int cluster) {
    return cluster == 16 ? k_tridiag_df<16> : cluster == 8 ? k_tridiag_df<8> : cluster == 4 ? k_tridiag_df<4>
           : cluster == 2 ? k_tridiag_df<2> : k_tridiag_df<1>;
}

// ---------------------------------------------------------------- K4a' small matrices
// Matrices of order nc <= kTsMax (after deflation nearly all: the N_max = 10 channels
// reduce to 11..94) are reduced by one CTA with the matrix resident in shared memory
// (both triangles), and the first D rows of Q = H_0 ... H_{n-3} (what k_qrows forms
// for the cluster path) are updated in the same pass.  The element arithmetic is
// double-float (df64.cuh: hi + lo FP32 pairs, ~48 bits): on this GPU an FP64 FMA
// issues at 1/64 of the FP32 rate.
//
// Step k reduces column k (x = rows k+1 .. n-1, alpha = x_0) with H = I - tau v v^T,
// v = (1, s x_1 ..), s = 1 / (alpha - beta), beta = -sign(alpha) |x|.  The column is
// carried scaled by a power of two, xs = 2^-e x with max(|alpha|, |x_1:|) in [1, 2)
// (exact), so the reflector's scalars need no range checks.  Every sum the step needs
// is formed from xs without the scalars, which lets one thread form them beside the
// product instead of before it:
//   S_i = sum_{t>=1} A_{b0+i, b0+t} xs_t   (eight parts per row, over fifteen warps),
//   Q = sum_{i>=1} xs_i S_i                 (per-warp partials of the same pass),
//   A v = A_{:,0} + s S,  v^T A v = A_00 + 2 s S_0 + s^2 Q,  p = tau A v,
//   w = p - (tau^2 / 2) (v^T A v) v,  A <- A - v w^T - w v^T,  R <- R - tau (R v) v^T.
// One step, three barriers:
//   2. warp 0, lane 0: beta, tau and s from (alpha, |x_1:|^2) in double-float (Newton's
//      reciprocal and square root); warps 1..15: the parts of S and Q; the last D
//      warps also R_d[b0+1:] . xs[1:];
//   3. every thread of a trailing row t: v_t and w_t from the parts (each thread sums
//      the warp partials of Q itself, in one fixed order), and the R update;
//   4. the rank-2 update of the trailing block, each result also at its mirror
//      position; warp 0 takes column k + 1 and scales it for the next step.
constexpr int kTsThreads = 512;
constexpr int kTsParts = 8;                   // threads per row of the symmetric product
constexpr int kTsIt = kTsMax / 32;            // column entries per lane of warp 0
static_assert(kTsMax % 32 == 0, "warp 0 holds a column in kTsIt entries per lane");
static_assert(2 * kTsMax <= kTsThreads, "the R update keeps at least half the threads");

// Binary exponent of a non-zero float (denormals give -127), and 2^e for -126 <= e <= 127.
__device__ inline int f32_exp(float x) { return (int)((__float_as_uint(x) >> 23) & 255u) - 127; }
__device__ inline float f32_pow2(int e) { return __uint_as_float((unsigned)(e + 127) << 23); }

__global__ void __launch_bounds__(kTsThreads) k_tridiag_small(const DyJob *jobs, int njobs) {
    using dfm::df;
    const int jid = blockIdx.x;
    if (jid >= njobs) return;
    const DyJob J = jobs[jid];
    const int n = J.nc, D = J.D;
    if (n > kTsMax) { beside_wait(); return; }   // the cluster kernel's
    const int ld = n | 1;     // odd stride: column reads hit distinct bank pairs
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    extern __shared__ double sm[];
    df *A = reinterpret_cast<df *>(sm);      // [n][ld], both triangles
    df *v = A + (size_t)n * ld;              // [n]
    df *ph = v + n;                          // [kTsParts][n] parts of S
    df *w = ph + kTsParts * n;               // [n]
    df *xs = w + n;                          // [n] the step's scaled column
    df *R = xs + n;                          // [D][n]
    __shared__ df s_col[2][2];               // alpha and |x_1:|^2 of a column, scaled, by parity
    __shared__ int s_nz[2], s_exp[2];        // the column has a reflector; e, by parity
    __shared__ df s_sc[2];                   // tau, s of the step
    __shared__ df s_q[kTsThreads / 32];      // per-warp partials of Q
    __shared__ df s_rx[8][2];                // R_d[b0+1:] . xs[1:], R_d[b0] before the update
    for (int q = tid; q < n * n; q += kTsThreads) {
        const int i = q / n, j = q - i * n;
        if (j <= i) {   // the assembled lower triangle, mirrored
            const df x = dfm::from_double(__ldcg(J.A + q));
            A[(size_t)i * ld + j] = x;
            A[(size_t)j * ld + i] = x;
        }
    }
    for (int q = tid; q < D * n; q += kTsThreads) R[q] = df{((q % n) == (q / n)) ? 1.0f : 0.0f, 0.0f};
    __syncthreads();
    const df zero{0.0f, 0.0f};
    // Warp 0: column kc's entries below the diagonal (rows kc+1 .. n-1), alpha, the sum of
    // the other entries' squares, the power of two 2^-e that brings the larger of |alpha|
    // and that norm into [1, 2), and xs = 2^-e x, into the column's parity slots.
    auto scale_column = [&](int kc) {
        const int b = kc + 1, mc = n - b, par = kc & 1;
        df x[kTsIt];
        df s2 = zero;
#pragma unroll
        for (int it = 0; it < kTsIt; ++it) {
            const int t = lane + 32 * it;
            x[it] = (t < mc) ? A[(size_t)(b + t) * ld + kc] : zero;
            if (t >= 1) s2 = dfm::fma(x[it], x[it], s2);
        }
        s2 = dfm::warp_sum(s2);
        const df al{__shfl_sync(0xffffffffu, x[0].h, 0), __shfl_sync(0xffffffffu, x[0].l, 0)};
        const int ea = (al.h != 0.0f) ? f32_exp(al.h) : -1000;
        const int es = (s2.h != 0.0f) ? (f32_exp(s2.h) >> 1) : -1000;   // floor(e / 2)
        int e = max(ea, es);
        e = (e == -1000) ? 0 : min(max(e, -126), 126);
        const float sg = f32_pow2(-e);
#pragma unroll
        for (int it = 0; it < kTsIt; ++it) {
            const int t = lane + 32 * it;
            if (t < mc) xs[t] = df{x[it].h * sg, x[it].l * sg};
        }
        if (lane == 0) {
            s_nz[par] = (s2.h != 0.0f || s2.l != 0.0f);
            s_exp[par] = e;
            s_col[par][0] = df{al.h * sg, al.l * sg};
            s_col[par][1] = df{(s2.h * sg) * sg, (s2.l * sg) * sg};
        }
    };
    if (n >= 3 && warp == 0) scale_column(0);
    __syncthreads();
    for (int k = 0; k + 2 < n; ++k) {
        const int b0 = k + 1, m = n - b0, par = k & 1;
        if (!s_nz[par]) {                    // column already reduced: H_k = I
            if (warp == 0) {
                if (lane == 0) A[(size_t)k * ld + k + 2] = zero;   // tau (e is alpha, in place)
                if (k + 3 < n) scale_column(k + 1);
            }
            __syncthreads();
            continue;
        }
        // 2. the reflector's scalars (warp 0, lane 0) beside the parts of S and Q
        if (warp == 0) {
            if (lane == 0) {
                const df al = s_col[par][0], s2 = s_col[par][1];
                const df x2 = dfm::fma(al, al, s2);   // in [1, 12)
                const df r = dfm::rsqrt2(x2), nx = dfm::mul(x2, r);
                const bool ng = signbit(al.h);
                const df aa = ng ? dfm::neg(al) : al;
                const df tau = dfm::fma(aa, r, df{1.0f, 0.0f});   // (beta - alpha) / beta = 1 + |alpha| / |x|
                df s = dfm::rcp2(dfm::add(aa, nx));               // 1 / (alpha - beta) = sign(alpha) / (|alpha| + |x|)
                if (ng) s = dfm::neg(s);
                s_sc[0] = tau;
                s_sc[1] = s;
                s_q[0] = zero;
                // e and tau of the step into row k, right of the diagonal (never read again),
                // converted to FP64 with d at the end: FP64 instructions stay off this chain
                const float un = f32_pow2(s_exp[par]);        // beta = 2^e beta~
                const df beta = ng ? nx : dfm::neg(nx);
                A[(size_t)k * ld + k + 1] = df{beta.h * un, beta.l * un};
                A[(size_t)k * ld + k + 2] = tau;
            }
        } else {
            if (warp >= kTsThreads / 32 - D) {   // R_d[b0+1:] . xs[1:] and R_d[b0]
                const int d = kTsThreads / 32 - 1 - warp;
                df sx = zero;
                for (int t = 1 + lane; t < m; t += 32) sx = dfm::fma(R[(size_t)d * n + b0 + t], xs[t], sx);
                sx = dfm::warp_sum(sx);
                if (lane == 0) { s_rx[d][0] = sx; s_rx[d][1] = R[(size_t)d * n + b0]; }
            }
            df qa = zero;
            for (int u = tid - 32; u < kTsParts * m; u += kTsThreads - 32) {
                const int i = u / kTsParts, h = u - i * kTsParts;
                const int q0 = (m * h) / kTsParts, q1 = (m * (h + 1)) / kTsParts;
                const df *Ai = A + (size_t)(b0 + i) * ld + b0;   // the full row (the update mirrors)
                df acc0 = zero, acc1 = zero;   // two chains
                int q = q0 > 0 ? q0 : 1;
                for (; q + 1 < q1; q += 2) {
                    acc0 = dfm::fma(Ai[q], xs[q], acc0);
                    acc1 = dfm::fma(Ai[q + 1], xs[q + 1], acc1);
                }
                if (q < q1) acc0 = dfm::fma(Ai[q], xs[q], acc0);
                const df r = dfm::add(acc0, acc1);
                ph[h * n + i] = r;
                if (i >= 1) qa = dfm::fma(xs[i], r, qa);
            }
            qa = dfm::warp_sum(qa);
            if (lane == 0) s_q[warp] = qa;
        }
        __syncthreads();
        // 3. v and w of every trailing row; R <- R - tau (R v) v^T
        const df tau = s_sc[0], s = s_sc[1];
        if (tid < m) {
            const int t = tid;
            df qv[kTsThreads / 32];
#pragma unroll
            for (int q = 0; q < kTsThreads / 32; ++q) qv[q] = s_q[q];
#pragma unroll
            for (int o = kTsThreads / 64; o > 0; o >>= 1)
#pragma unroll
                for (int q = 0; q < o; ++q) qv[q] = dfm::add(qv[q], qv[q + o]);
            df p0[kTsParts], pt[kTsParts];
#pragma unroll
            for (int h = 0; h < kTsParts; ++h) { p0[h] = ph[h * n]; pt[h] = ph[h * n + t]; }
#pragma unroll
            for (int o = kTsParts / 2; o > 0; o >>= 1)
#pragma unroll
                for (int h = 0; h < o; ++h) { p0[h] = dfm::add(p0[h], p0[h + o]); pt[h] = dfm::add(pt[h], pt[h + o]); }
            // v^T A v = A_00 + s (2 S_0 + s Q); K = (tau^2 / 2) v^T A v
            const df vav = dfm::fma(s, dfm::fma(s, qv[0], dfm::add(p0[0], p0[0])), A[(size_t)b0 * ld + b0]);
            const df tk = dfm::mul(tau, tau);
            const df nK = dfm::neg(dfm::mul(df{0.5f * tk.h, 0.5f * tk.l}, vav));
            const df vt = (t == 0) ? df{1.0f, 0.0f} : dfm::mul(s, xs[t]);
            const df p = dfm::mul(tau, dfm::fma(s, pt[0], A[(size_t)(b0 + t) * ld + b0]));
            v[t] = vt;
            w[t] = dfm::fma(nK, vt, p);
        }
        // the R update on the warps that form no v and w
        const int rb = (m + 31) & ~31;
        for (int u = tid - rb; u >= 0 && u < D * m; u += kTsThreads - rb) {
            const int d = u / m, t = u - d * m;
            const df vt = (t == 0) ? df{1.0f, 0.0f} : dfm::mul(s, xs[t]);
            const df nc = dfm::neg(dfm::mul(tau, dfm::fma(s, s_rx[d][0], s_rx[d][1])));
            df &r = R[(size_t)d * n + b0 + t];
            r = dfm::fma(nc, vt, r);
        }
        __syncthreads();
        // 4. A -= v w^T + w v^T on the trailing block: warp 0 takes column k + 1 (local
        //    column 0) and then scales it for the next step; warps 1..15 the rest, rows i
        //    and m-1-i per warp so the triangle's rows balance, each result also at its mirror
        if (warp == 0) {
            for (int r = lane; r < m; r += 32) {
                df *a = A + (size_t)(b0 + r) * ld + b0;
                const df x = rank2(*a, v[r], w[0], w[r], v[0]);
                *a = x;
                A[(size_t)b0 * ld + b0 + r] = x;
            }
            __syncwarp();
            if (k + 3 < n) scale_column(k + 1);
        } else {
            for (int i1 = warp - 1; i1 < (m + 1) / 2; i1 += kTsThreads / 32 - 1) {
                const int i2 = m - 1 - i1;
                const int len = (i1 == i2) ? (i1 + 1) : (m + 1);
                // two entries per pass, both read before either is written: the entries
                // are distinct lower-triangle ones, so no write meets the other's reads
                for (int u = lane; u < len; u += 64) {
                    int r[2], c[2];
                    df x[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int uu = u + 32 * h;
                        r[h] = (uu <= i1) ? i1 : i2;
                        c[h] = (uu <= i1) ? uu : uu - i1 - 1;
                        if (uu < len && c[h] != 0) {   // column k + 1: warp 0's
                            x[h] = rank2(A[(size_t)(b0 + r[h]) * ld + b0 + c[h]], v[r[h]], w[c[h]], w[r[h]], v[c[h]]);
                        } else {
                            c[h] = 0;
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (c[h] != 0) {
                            A[(size_t)(b0 + r[h]) * ld + b0 + c[h]] = x[h];
                            A[(size_t)(b0 + c[h]) * ld + b0 + r[h]] = x[h];   // the mirror, read by the next product
                        }
                }
            }
        }
        __syncthreads();
    }
    for (int k = tid; k < n; k += kTsThreads) {   // d, e, tau in FP64 (row k: d_k, e_k, tau_k)
        const df *Ak = A + (size_t)k * ld + k;
        J.d[k] = dfm::to_double(Ak[0]);
        J.e[k] = (k + 1 < n) ? dfm::to_double(Ak[1]) : 0.0;
        J.tau[k] = (k + 2 < n) ? dfm::to_double(Ak[2]) : 0.0;
    }
    for (int q = tid; q < D * n; q += kTsThreads) J.R[q] = dfm::to_double(R[q]);
    beside_wait();
}

size_t tridiag_small_smem_bytes(int nmax, int Dmax) {
    const size_t n = (size_t)std::min(nmax, kTsMax);
    return sizeof(double) * (n * (n | 1) + (size_t)(kTsParts + 3) * n + (size_t)Dmax * n);
}

// Per-warp partial vectors that fit next to the other arrays (8 = one per warp).
int tridiag_npriv(int nmax, int cluster) {
    const size_t fixed = (size_t)3 * nmax + (size_t)(nmax / cluster + 1) + 32;
    const size_t cap = (size_t)200 * 1024 / sizeof(double);
    int np = 8;
    while (np > 1 && fixed + (size_t)np * nmax > cap) --np;
    return np;
}

size_t tridiag_smem_bytes(int nmax, int cluster) {
    return sizeof(double) * ((size_t)(3 + tridiag_npriv(nmax, cluster)) * nmax + (size_t)(nmax / cluster + 1) + 32);
}

// The largest order whose layout fits the dynamic shared memory a CTA may opt into.
// Up to the orders that leave room for two partial vectors the layout stays within
// 200 KB; beyond, it grows with the order, so the orders that fit are a prefix.
// Cached per cluster size (bd_create fills the cache, so no attribute query falls inside
// a stream capture); the GPUs a process drives are of one kind.
static std::atomic<int> g_fit_order[17];

int tridiag_fit_order(int cluster) {
    const bool cached = cluster >= 1 && cluster <= 16;
    if (cached) {
        const int v = g_fit_order[cluster].load(std::memory_order_relaxed);
        if (v) return v;
    }
    int dev = 0, optin = 0;
    cudaFuncAttributes a{};
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&a, k_tridiag) != cudaSuccess)
        return kTsMax + 1;   // the launch that follows reports the error
    const size_t limit = (size_t)optin - a.sharedSizeBytes;
    int lo = kTsMax + 1, hi = 1 << 22;
    while (lo < hi) {
        const int mid = lo + (hi - lo + 1) / 2;
        if (tridiag_smem_bytes(mid, cluster) <= limit) lo = mid; else hi = mid - 1;
    }
    if (cached) g_fit_order[cluster].store(lo, std::memory_order_relaxed);
    return lo;
}

// Shared memory of k_tridiag_df (8-byte slots, at most kTdfSlots: 224 KB) and the largest
// order it takes in a launch of orders up to nmax: as far as its vectors fit (the rows may
// spill), where all of the launch's orders leave k_tridiag room for a partial vector a warp
// (orders up to about 2 300); kTsMax, none, beyond.  There FP64 stays: double-float is twelve
// times as fast (a solve of order 2 500, 38 ms against 465) but its rounding, 2^-48 a step,
// grows with the order beside the bisection's 1e-13 |T| (eigenvector components off by 1.8e-14
// against 1.0e-15 in the median, 8.6e-11 against 3.5e-12 at the most).
constexpr int kTdfSlots = 224 * 1024 / 8;
int tridiag_df_limit(int nmax, int cluster, int D) {
    if (tridiag_npriv(std::min(nmax, tridiag_fit_order(cluster)), cluster) < kTdThreads / 32) return kTsMax;
    int lo = kTsMax, hi = 1 << 16;
    while (lo < hi) {
        const int mid = lo + (hi - lo + 1) / 2;
        if (tdf_fixed(mid, cluster, D) <= (size_t)kTdfSlots) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// CTAs of k_tridiag_grid: one on every SM (0: the device takes no cooperative launch)
static int grid_ctas() {
    static const int g = [] {
        int dev = 0, sms = 0, coop = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
            return 0;
        return std::min(sms, kTdgMax);
    }();
    return g;
}

void tridiag_fit_warm() {
    for (int c = 1; c <= 16; c <<= 1) tridiag_fit_order(c);
    allow_dynamic_smem((const void *)k_tridiag_small);
    allow_dynamic_smem((const void *)k_tridiag);
    for (int c = 1; c <= 16; c <<= 1) allow_dynamic_smem((const void *)tridiag_df_kernel(c));
    allow_dynamic_smem((const void *)k_tridiag_grid);
    grid_ctas();
}

// One matrix in the launch, of an order that k_tridiag_grid may take
static bool tridiag_on_grid(int njobs, int nmax, int nlim) {
    return njobs == 1 && std::min(nmax, nlim) >= kTdgMin && grid_ctas() > 8;
}

// Kernels launch_dyson starts for matrices of order up to nmax: deflate, assemble, the
// small-matrix reduction (the cluster one beyond kTsMax, the FP64 one and k_qrows beyond
// its limit), then launch_eig's.
int dyson_launch_count(int njobs, int nmax, int Dmax, int cluster) {
    const int nlim = tridiag_df_limit(nmax, cluster, Dmax);
    return 3 + (nmax > kTsMax && nlim > kTsMax ? 1 : 0) + (tridiag_on_grid(njobs, nmax, nlim) ? 1 : 0) + (nmax > nlim ? 2 : 0) + (nmax > kTsMax ? 8 : 7);
}

cudaError_t launch_dyson(const DyJob *d_jobs, int njobs, const long long *d_row_first, long long total_rows,
                         int nmax, int Dmax, int cluster, double *work, const long long *d_work_first, cudaStream_t st) {
    if (njobs <= 0) return cudaSuccess;
    k_dyson_deflate<<<njobs, kDfThreads, 0, st>>>(const_cast<DyJob *>(d_jobs), njobs, work, d_work_first);
    k_dyson_assemble<<<(unsigned)((total_rows + 127) / 128), 128, 0, st>>>(d_jobs, njobs, d_row_first, total_rows, work,
                                                                       d_work_first);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const size_t ssmem = tridiag_small_smem_bytes(nmax, Dmax);
    e = allow_dynamic_smem((const void *)k_tridiag_small);
    if (e != cudaSuccess) return e;
    if (nmax <= kTsMax) {
        k_tridiag_small<<<njobs, kTsThreads, ssmem, st>>>(d_jobs, njobs);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
        return launch_eig(d_jobs, njobs, d_row_first, total_rows, nmax, nmax, work, d_work_first, st);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(njobs * cluster, 1, 1);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto prepare = [&](const void *kern) {
        e = allow_dynamic_smem(kern);
        if (e == cudaSuccess && cluster > 8) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        return e == cudaSuccess;
    };
    const int nlim = tridiag_df_limit(nmax, cluster, Dmax);
    const bool grid = tridiag_on_grid(njobs, nmax, nlim);
    if (grid) {
        cudaLaunchConfig_t gc = {};
        gc.gridDim = dim3(grid_ctas(), 1, 1);
        gc.blockDim = dim3(kTdfThreads, 1, 1);
        gc.dynamicSmemBytes = kTdfSlots * 8;
        gc.stream = st;
        cudaLaunchAttribute ga[1];
        ga[0].id = cudaLaunchAttributeCooperative;
        ga[0].val.cooperative = 1;
        gc.attrs = ga;
        gc.numAttrs = 1;
        e = allow_dynamic_smem((const void *)k_tridiag_grid);
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&gc, k_tridiag_grid, d_jobs, nlim, kTdfSlots, work, d_work_first);
        if (e != cudaSuccess) return e;
    }
    if (nlim == kTsMax) {
        k_tridiag_small<<<njobs, kTsThreads, ssmem, st>>>(d_jobs, njobs);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    } else {
        // as many slots as the largest order (the full orders bound the deflated ones) needs
        // to keep all its rows, at most kTdfSlots
        const int nb = grid ? kTdgMin - 1 : std::min(nmax, nlim);
        const size_t slots = std::min((size_t)kTdfSlots, tdf_fixed(nb, cluster, Dmax) + (size_t)((nb + cluster - 1) / cluster) * nb);
        cfg.blockDim = dim3(kTdfThreads, 1, 1);
        cfg.dynamicSmemBytes = slots * 8;
        const auto kern = tridiag_df_kernel(cluster);
        if (!prepare((const void *)kern)) return e;
        e = cudaLaunchKernelEx(&cfg, kern, d_jobs, njobs, nb, (int)slots, work, d_work_first);
        if (e != cudaSuccess) return e;
        // the small orders beside it: a batch of either leaves most SMs idle (orders up to 205 in 34
        // channels: 0.65 + 0.49 ms one after the other)
        e = launch_beside(k_tridiag_small, dim3(njobs), dim3(kTsThreads), ssmem, st, d_jobs, njobs);
        if (e != cudaSuccess) return e;
    }
    if (nmax > nlim) {
        // the layout is sized for at most the largest order shared memory holds, and larger
        // deflated orders report it
        const int nb = std::min(nmax, tridiag_fit_order(cluster));
        cfg.blockDim = dim3(kTdThreads, 1, 1);
        cfg.dynamicSmemBytes = tridiag_smem_bytes(nb, cluster);
        if (!prepare((const void *)k_tridiag)) return e;
        e = cudaLaunchKernelEx(&cfg, k_tridiag, d_jobs, njobs, nb, tridiag_npriv(nb, cluster), nlim);
        if (e != cudaSuccess) return e;
    }
    return launch_eig(d_jobs, njobs, d_row_first, total_rows, nmax, nlim, work, d_work_first, st);
}

}  // namespace bd
