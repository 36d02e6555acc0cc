// k_compact.cu -- pole sets with few distinct energies, reduced in the space their
// couplings span.
//
// E is diagonal, so inside a group of poles of one energy every rotation leaves the
// problem unchanged: with M_g (D x m) the group's couplings and G_g = M_g M_g^T = L L^T,
// the poles M_g^T = Q L^T act through L alone -- D couplings of at most D rotated poles of
// that energy -- and the other m - D directions couple to nothing.  The unperturbed
// propagator's spectra have about a dozen distinct energies a channel (the oscillator
// shells) however many thousand poles they hold, so a chain of N poles is a chain of
// N' = sum_g rank(M_g) <= 12 D rotated ones: 54 instead of 4 863 for the largest channel
// at N_max = 10.  alpha, beta, g and m are inner products, the same in both.
//
//   k_lz_compact   the multi-pivot Lanczos reduction (k_lanczos's steps, FP64 vectors) of
//                  a chain in that space, one CTA with the whole basis in shared memory.
//                  A chain it cannot take is left to k_lanczos (CompactInfo::handled).
//   k_lz_expand    its stored vectors in the poles' space, v = sum_g M_g^T L^-T v'_g.
//   k_plain_rotate the plain Sigma(2) rows of the full Dyson matrix with every group of
//                  more than kKeep poles rotated the same way: its first D rows couple by L, the
//                  others not at all, and k_dyson_deflate takes those out of the matrix
//                  (N_max = 4 without Lanczos: a step of 152 ms, 111 of them spent on
//                  orthonormalising clusters of a hundred equal eigenvalues, takes 0.92).
//
// Energies that differ by rounding only (e1 + e2 - e3 of orbits of the same shells added
// in another order: over hbar omega of 5 to 40 MeV and N_max of 4 to 12 a shell's differ by at
// most 2.2 eps of the largest energy) count as one group, whose poles take the middle of it.
// All of a group lies within kMergeUlp eps, so that moves E by no more than the rounding of the
// sum; a set in which neighbours lie that close and the whole run does not is not one of such
// shells, and is left as it is.  The Gram matrices come from k_lz_groups
// (sums of FP64 products in a fixed order).  A group keeps its poles as they are when it
// has at most kKeep, or at most kGrpSmall and a pivot that loses digits (below kPivot of
// its diagonal entry); a larger group with such a pivot leaves the whole chain to
// k_lanczos.
//
// The reduction depends on a group through L only, but a Gram matrix holds L's rows to the
// rounding of their squares: where an orbital's couplings lie close to the others' (a pivot
// of the fraction p of its diagonal entry) L is off by about 1e-17 / p, and alpha and beta
// with it (1.7e-11 of the energies at p = 2e-6, where the reduction over the poles is off by
// 3e-15).  So a factor with a pivot below kLossy is formed a second time from its own poles,
// factor_again: Q = L^-1 M_g has rows that are orthonormal but for L's error, and with
// Q Q^T = L2 L2^T the product L L2 is M_g's factor to FP64's rounding of M_g (Cholesky QR
// taken twice).
#include <cfloat>
#include "bd_common.cuh"
#include "bd_kernels.h"
#include "lz_fixed.cuh"

namespace bd {

namespace {

constexpr int kCpThreads = 256;
constexpr int kCpWarps = kCpThreads / 32;
constexpr int kKeep = 12;
constexpr double kMergeUlp = 4.0;
constexpr double kPivot = 1e-6, kLossy = 0.125;
constexpr int kCpSmem = 200 * 1024;

// Lower-triangular factor of a D x D Gram matrix (lower triangle in tri), a warp; L (D x D,
// row-major, zero above the diagonal) to out.  A row without couplings (zero diagonal
// entry) gives a zero column.  0 when a pivot falls below kPivot of its diagonal entry
// or anything is not finite, and out is not to be used; 2 when one falls below kLossy of it.
__device__ int warp_cholesky(const double *tri, int D, double *out, int lane) {
    int res = 1;
    for (int e = lane; e < D * D; e += 32) {
        const int a = e / D, b = e % D;
        out[e] = (b <= a) ? tri[a * (a + 1) / 2 + b] : 0.0;
    }
    __syncwarp();
    for (int s = 0; s < D; ++s) {
        const double p = out[s * D + s], g = tri[s * (s + 1) / 2 + s];
        const bool zero = (g == 0.0);
        if (!zero && !(p > kPivot * g && p <= DBL_MAX)) return 0;   // the same in every lane
        if (!zero && p < kLossy * g) res = 2;
        // (Newton's iteration to a few ulp: FP64 square root and division are chains of their own)
        const double ri = zero ? 0.0 : rsqrt_cubic(p), r = p * ri;
        __syncwarp();
        if (lane >= s && lane < D) out[lane * D + s] = (lane == s) ? r : out[lane * D + s] * ri;
        __syncwarp();
        for (int e = lane; e < D * D; e += 32) {
            const int a = e / D, b = e % D;
            if (a > s && b > s && b <= a) out[e] = fma(-out[a * D + s], out[b * D + s], out[e]);
        }
        __syncwarp();
    }
    return res;
}

// The factor L (D x D, row-major, global) of the couplings M of poles [p0, p0 + m) formed again
// from Q = L^-1 M, by the whole CTA: a thread per pole and round, D (D + 1) FP64 instructions a
// pole.  (N_max = 10 with every subshell's orbitals close, all groups formed again: the Lanczos phase
// 0.39 -> 0.52 ms; none of them: no change.)
template <int D>
__device__ __noinline__ void factor_again(const double *M, size_t N, int p0, int m, double *L, double (*s_l)[64],
                                          double (*s_tri)[kGramEntries]) {
    constexpr int P = D * (D + 1) / 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < D * D) s_l[0][tid] = L[tid];
    if (tid < D) s_l[1][tid] = L[tid * D + tid] != 0.0 ? 1.0 / L[tid * D + tid] : 0.0;
    __syncthreads();
    double G[P];
#pragma unroll
    for (int u = 0; u < P; ++u) G[u] = 0.0;
    for (int i = tid; i < m; i += kCpThreads) {
        double y[D];
#pragma unroll
        for (int a = 0; a < D; ++a) y[a] = M[a * N + p0 + i];
#pragma unroll
        for (int a = 0; a < D; ++a) {
#pragma unroll
            for (int b = 0; b < a; ++b) y[a] = fma(-s_l[0][a * D + b], y[b], y[a]);
            y[a] *= s_l[1][a];
        }
#pragma unroll
        for (int a = 0; a < D; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b) G[a * (a + 1) / 2 + b] = fma(y[a], y[b], G[a * (a + 1) / 2 + b]);
    }
    auto add = [](double p, double q) { return p + q; };
    auto shf = [](double p, int o) { return __shfl_xor_sync(0xffffffffu, p, o); };
    constexpr int NV = P <= 4 ? 4 : P <= 8 ? 8 : P <= 16 ? 16 : 32, W = 32 / NV;
    double v[NV];
#pragma unroll
    for (int u = 0; u < NV; ++u) v[u] = u < P ? G[u < P ? u : 0] : 0.0;
    const double r = warp_sums_of<NV>(v, lane, add, shf);   // lane L: value L / W
    if (lane % W == 0 && lane / W < P) s_tri[warp][lane / W] = r;
    if constexpr (P > 32) {
        double x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = G[32 + u];
        const double r2 = warp_sums_of<4>(x, lane, add, shf);
        if (lane % 8 == 0) s_tri[warp][32 + lane / 8] = r2;
    }
    __syncthreads();
    if (tid < P) {
        double s = s_tri[0][tid];
        for (int w = 1; w < kCpWarps; ++w) s += s_tri[w][tid];
        s_tri[0][tid] = s;
    }
    __syncthreads();
    if (warp == 0 && warp_cholesky(s_tri[0], D, s_l[2], lane))
        for (int e = lane; e < D * D; e += 32) {
            const int a = e / D, b = e % D;
            double s = 0.0;
            for (int c = b; c <= a; ++c) s = fma(s_l[0][a * D + c], s_l[2][c * D + b], s);
            L[e] = s;
        }
    __syncthreads();
}

// The factors that state marks as lossy (2), S.L[g] of groups [S.start[first[g]], S.start[first[g + 1]]).
__device__ void lossy_factors(const LzChain &C, const CompactScratch &S, const int *first, int ng, const int *state,
                              double (*s_l)[64], double (*s_tri)[kGramEntries]) {
    for (int g = 0; g < ng; ++g) {
        if (state[g] != 2) continue;
        const int p0 = S.start[first[g]], m = S.start[first[g + 1]] - p0;
        double *L = S.L + (size_t)g * 64;
        switch (C.D) {
            case 1: factor_again<1>(C.M, C.N, p0, m, L, s_l, s_tri); break;
            case 2: factor_again<2>(C.M, C.N, p0, m, L, s_l, s_tri); break;
            case 3: factor_again<3>(C.M, C.N, p0, m, L, s_l, s_tri); break;
            case 4: factor_again<4>(C.M, C.N, p0, m, L, s_l, s_tri); break;
            case 5: factor_again<5>(C.M, C.N, p0, m, L, s_l, s_tri); break;
            case 6: factor_again<6>(C.M, C.N, p0, m, L, s_l, s_tri); break;
            case 7: factor_again<7>(C.M, C.N, p0, m, L, s_l, s_tri); break;
            default: factor_again<8>(C.M, C.N, p0, m, L, s_l, s_tri); break;
        }
    }
}

// Exclusive scan over one int per thread of the CTA.
__device__ __forceinline__ int scan_ints(int x, int &total, int *ws) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int v = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) ws[warp] = v;
    __syncthreads();
    int off = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < kCpWarps; ++w) {
        if (w < warp) off += ws[w];
        total += ws[w];
    }
    __syncthreads();
    return off + v - x;
}

// The merged groups of a chain (first exact group of each, s_first[0 .. n], s_first[n] = Q)
// from the exact groups' energies; returns their number, 0 when one spans more than kMergeUlp.
// One thread per exact group.
__device__ int merge_groups(const double *gE, int Q, int *s_first, int *ws) {
    const int tid = threadIdx.x;
    const double tol = kMergeUlp * DBL_EPSILON * fmax(fabs(gE[0]), fabs(gE[Q - 1]));
    const int brk = (tid < Q) ? (tid == 0 || fabs(gE[tid] - gE[tid - 1]) > tol) : 0;
    int n;
    const int pos = scan_ints(brk, n, ws);
    if (brk) s_first[pos] = tid;
    if (tid == 0) s_first[n] = Q;
    __syncthreads();
    const bool wide = tid < n && fabs(gE[s_first[tid + 1] - 1] - gE[s_first[tid]]) > tol;
    return __syncthreads_or(wide) ? 0 : n;
}

static_assert(kCpThreads >= kCpGroups, "a thread per exact group");
static_assert(kCpDim <= kFixedRun, "a chain's sums are one run");

}  // namespace

// ------------------------------------------------------------------ Lanczos
// One CTA per chain.  The steps, decisions and rows are k_lanczos's with FP64 vectors; a
// chain that would need what only the full space has (a restart vector, a direction no
// group has left) is left to k_lanczos as a whole.
//
// A step is a chain of short phases between barriers, and an FP64 instruction holds an SM
// sub-partition's FP64 unit for ~64 cycles, so FP64 is kept to what needs it (w = M p, alpha, g,
// the recurrence, 1/|w|): the sweep's dot products, |w|^2 and m are fixed-point sums (lz_fixed.cuh),
// the update is FP32 where the coefficients are rounding-sized (|c| <= 1e-9 |w|: an error below
// 2^-23 1e-9 |w|) and fixed point otherwise.  Stored vectors lie element by element: in the dot
// products a lane takes a vector and the warps split the elements, in the update a thread takes
// an element and the idle ones split the vectors, so neither sums across lanes; one warp takes
// the decision beside the other warps' sums.
// Measured (N_max = 10, 100 iterations per pivot): the reduction of all 84 chains takes
// 0.29 ms against 3.59 ms in the poles' space (N_max = 12: 0.44 against 12.2); 600 000 cycles for
// the longest chain, 54 steps in 54 coordinates and its set-up.
__global__ void __launch_bounds__(kCpThreads) k_lz_compact(const LzChain *chains, int nchains, double eta2) {
    const int cid = blockIdx.x;
    if (cid >= nchains) return;
    __shared__ LzChain C;
    if (threadIdx.x < sizeof(LzChain) / 4)
        reinterpret_cast<int *>(&C)[threadIdx.x] = reinterpret_cast<const int *>(chains + cid)[threadIdx.x];
    __syncthreads();
    if (!C.cp || !C.cp_on) return;
    const CompactScratch S = lz_compact(C.cp);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = C.N, D = C.D, L = C.L, NT = C.nden_out + C.D;
    const int Q = S.info->q;
    if (Q < 1) return;   // too many distinct energies (k_lz_groups cleared S.info->handled)
    __shared__ int ws[kCpWarps];
    __shared__ int s_first[kCpGroups + 1], s_off[kCpGroups + 1], s_state[kCpMerged];
    __shared__ int s_bad;
    __shared__ unsigned s_rng[2];
    __shared__ double s_tri[kCpWarps][kGramEntries], s_l[kCpWarps][64];
    extern __shared__ double sm[];
    if (tid == 0) { s_bad = 0; s_rng[0] = 0; s_rng[1] = 0; }
    const int ng = merge_groups(C.gE, Q, s_first, ws);
    if (ng < 1 || ng > kCpMerged) return;
    // 1. every merged group's coordinates: its own poles (kept), or the columns of L
    for (int g = warp; g < ng; g += kCpWarps) {
        const int q0 = s_first[g], q1 = s_first[g + 1];
        const int p0 = S.start[q0], m = S.start[q1] - p0;
        CompactGroup G;
        G.p0 = p0; G.m = m; G.kept = 1; G.c = m;
        if (m > kKeep) {
            for (int e = lane; e < D * (D + 1) / 2; e += 32) {
                double s = 0.0;
                for (int q = q0; q < q1; ++q) s += S.gram[(size_t)q * kGramEntries + e];
                s_tri[warp][e] = s;
            }
            __syncwarp();
            const int ok = warp_cholesky(s_tri[warp], D, s_l[warp], lane);
            if (lane == 0) s_state[g] = ok;
            if (ok) {
                G.kept = 0;
                G.c = D;
                for (int e = lane; e < D * D; e += 32) S.L[(size_t)g * 64 + e] = s_l[warp][e];
            } else if (m > kGrpSmall) {
                if (lane == 0) s_bad = 1;
            }
            __syncwarp();
        } else if (lane == 0) {
            s_state[g] = 0;
        }
        if (lane == 0) { S.grp[g] = G; s_off[g] = G.c; }
    }
    __syncthreads();
    if (s_bad) return;
    lossy_factors(C, S, s_first, ng, s_state, s_l, s_tri);
    int np;
    {
        const int x = (tid < ng) ? s_off[tid] : 0;
        const int off = scan_ints(x, np, ws);
        if (tid < ng) s_off[tid] = off;
        if (tid == 0) s_off[ng] = np;
        __syncthreads();
    }
    const int R = min(L, np);               // vectors, at most
    const int rq = (R + 4) & ~3, np4 = (np + 3) & ~3;
    const int nla = max(C.n_used - 1, 0);   // chains whose last vector later ones refer to
    // shared layout (doubles): E[np4] | M[D][np4] (two planes of integers against s_mb) | w[np4] |
    // ew[np4] | ring[2][np4] | last[nla][np4] | c[rq + 4] | sc[20] | part[256] (FixedSum) | wab[np4] (int2),
    // then ints Va[np][RS] | Vb[np][RS] (element by element: a lane a vector reads consecutive ones, a lane an
    // element ones an odd stride apart), floats cf[rq + 4], ints rowslot[L]
    const int RS = R | 1;
    const size_t need = sizeof(double) * ((size_t)(D + 6 + nla) * np4 + rq + 4 + 20 + 512) +
                        sizeof(int) * (2 * (size_t)np * RS + rq + 4 + (size_t)L);
    if (np > kCpDim || need > (size_t)kCpSmem) return;
    double *E = sm, *M = E + np4, *w = M + (size_t)D * np4;
    double *ew = w + np4, *ring = ew + np4, *lasts = ring + 2 * np4, *c = lasts + (size_t)nla * np4, *sc = c + rq + 4;
    FixedSum *part = reinterpret_cast<FixedSum *>(sc + 20);
    float *fpart = reinterpret_cast<float *>(part);
    int2 *wab = reinterpret_cast<int2 *>(part + 256);
    int *Va = reinterpret_cast<int *>(wab + np4), *Vb = Va + (size_t)np * RS;
    float *cf = reinterpret_cast<float *>(Vb + (size_t)np * RS);
    int *rowslot = reinterpret_cast<int *>(cf + rq + 4);
    static_assert(kCpThreads == 256, "part holds a sum a thread");
    unsigned me = 0, mm = 0;   // upper words of the largest |E| and |M|
    for (int g = warp; g < ng; g += kCpWarps) {
        const CompactGroup G = S.grp[g];
        const double e0 = C.E[G.p0], eg = 0.5 * (e0 + C.E[G.p0 + G.m - 1]);
        for (int i = lane; i < G.c; i += 32) {
            const double e = G.kept ? C.E[G.p0 + i] : eg;
            E[s_off[g] + i] = e;
            me = max(me, (unsigned)__double2hiint(e) & 0x7fffffffu);
            for (int d = 0; d < D; ++d) {
                const double m = G.kept ? C.M[(size_t)d * N + G.p0 + i] : S.L[(size_t)g * 64 + d * D + i];
                M[(size_t)d * np4 + s_off[g] + i] = m;
                S.M[d * kCpDim + s_off[g] + i] = m;   // for w = M p (the planes are for m)
                mm = max(mm, (unsigned)__double2hiint(m) & 0x7fffffffu);
            }
        }
    }
    int *Ma = reinterpret_cast<int *>(M), *Mb = Ma + (size_t)D * np4;
    __syncthreads();
    __shared__ int s_mb[8];
    double mv[(8 * kCpDim + kCpThreads - 1) / kCpThreads];   // (the planes take the doubles' place)
#pragma unroll
    for (int r = 0; r < (8 * kCpDim + kCpThreads - 1) / kCpThreads; ++r) {
        const int q = tid + r * kCpThreads;
        mv[r] = q < D * np ? M[(size_t)(q / np) * np4 + q % np] : 0.0;
    }
    if (warp < D) {   // a power of two above |M_d|
        float m2 = 0.0f;
        for (int i = lane; i < np; i += 32) { const float f = f32_trunc(M[(size_t)warp * np4 + i]); m2 = fmaf(f, f, m2); }
        for (int o = 16; o > 0; o >>= 1) m2 += __shfl_xor_sync(0xffffffffu, m2, o);
        bool any = false;
        for (int i = lane; i < np; i += 32) any |= M[(size_t)warp * np4 + i] != 0.0;
        any = __any_sync(0xffffffffu, any);
        if (lane == 0) {
            s_mb[warp] = bias_above((double)m2);
            if (any && m2 < 0x1p-90f) s_bad = 1;   // an orbital coupled far more weakly than the others
        }
    }
    me = __reduce_max_sync(0xffffffffu, me);
    mm = __reduce_max_sync(0xffffffffu, mm);
    if (lane == 0) { atomicMax(&s_rng[0], me); atomicMax(&s_rng[1], mm); }
    __syncthreads();
    if (s_bad || !fixed_range(s_rng[0]) || !fixed_range(s_rng[1])) return;   // (fixed-point and FP32 parts)
#pragma unroll
    for (int r = 0; r < (8 * kCpDim + kCpThreads - 1) / kCpThreads; ++r) {
        const int q = tid + r * kCpThreads;
        if (q < D * np) {
            const int2 f = fixed_of(mv[r], s_mb[q / np]);
            Ma[(size_t)(q / np) * np4 + q % np] = f.x;
            Mb[(size_t)(q / np) * np4 + q % np] = f.y;
        }
    }
    __shared__ int s_start[10], s_last[10], lslot[8], lo_[16], s_nl, s_fl;
    __shared__ double lc[16], s_n[3];   // s_n: 1/|w|, |w|, |E v|^2 of the kept vector
    __shared__ float s_f[kCpWarps], s_cm[kCpWarps];
    __shared__ double s_piv[80];   // at most 9 pivots of 8
    bool bad_piv = false;   // (a pivot of zeros is NaN here: the integers of the split would hide it)
    for (int q = tid; q < C.n_used * D && q < 80; q += kCpThreads) {
        const double p = C.piv[q];
        s_piv[q] = p;
        bad_piv |= (__double2hiint(p) & 0x7ff00000) == 0x7ff00000;
    }
    if (__syncthreads_or(bad_piv)) return;
    if (tid <= C.n_used && tid < 10) s_start[tid] = C.start[tid];
    if (tid < C.n_used && tid < 10) s_last[tid] = C.last[tid];
    // the groups' energies and unreached directions, cumulated (Q = gInfo[0])
    __shared__ int s_cum[kCpGroups];
    __shared__ double s_gE[kCpGroups];
    if (tid < Q) { s_cum[tid] = C.gInfo[1 + tid]; s_gE[tid] = C.gE[tid]; }
    __syncthreads();
    const int dtot = s_cum[Q - 1];
    auto group_of = [&](int d) {
        int lo = 0, hi = Q - 1;
        while (lo < hi) { const int mid = (lo + hi) >> 1; if (s_cum[mid] > d) hi = mid; else lo = mid + 1; }
        return lo;
    };
    constexpr double tau = 1e-48, thr_exh = 1e-20;   // k_lanczos's, FP64 vectors
    int dcur = 0, ndefl = 0, nvec = 0, extra = 0, k = -1;
    double e2v = 0.0;            // |E v|^2 of the last built vector
    int nl0 = 0;                 // vectors of the next recurrence (lo_, lc)
    bool rough = false;          // w much shorter than what it was split against: swept again
    // stored vector t as doubles: the two newest, or the last one of chain q
    auto vecd = [&](int t, int q) -> const double * { return t >= nvec - 2 ? ring + (t & 1) * np4 : lasts + (size_t)q * np4; };
    int wbias = 1023;   // exponent field of the power of two w is split against
    auto split_w = [&](int i, double x) {
        wab[i] = fixed_of(x, wbias);
    };
    // a scale that FP32 may have lost (from its upper word), and a w that is not zero
    auto weak = [](double x2) { return __double2hiint(x2) < __double2hiint(kFixedWeak); };
    auto lost = [&]() {
        bool any = false;
        for (int i = tid; i < np; i += kCpThreads) any |= (__double_as_longlong(w[i]) << 1) != 0;
        return __syncthreads_or(any) != 0;
    };
    // the update's threads: an element each, npw apart the groups that share its vectors
    const int npw = (np + 31) & ~31, tgs = kCpThreads / npw, tgp = tid / npw, ei = tid - tgp * npw;
    __syncthreads();
    for (int j = 0; j < L; ++j) {
        const bool newv = (k + 1 < C.n_used) && (j == s_start[k + 1]);
        if (newv) ++k;
        const int nq = k;
        if (tid < nq) lslot[tid] = rowslot[s_last[tid]];
        // w = M p, or E v_{j-1} less its known components
        double wn2 = 0.0, wn2_first = e2v;   // |w|^2 before the sweep, and of E v_{j-1} / M p (thresholds' scales)
        if (newv) {
            float s2 = 0.0f;
            for (int i = tid; i < np; i += kCpThreads) {
                const double *p = s_piv + k * D;
                double x = 0.0, m[8];
#pragma unroll
                for (int d = 0; d < 8; ++d) m[d] = d < D ? S.M[d * kCpDim + i] : 0.0;
#pragma unroll
                for (int d = 0; d < 8; ++d)
                    if (d < D) x = fma(m[d], p[d], x);
                w[i] = x;
                const float f = f32_trunc(x);
                s2 = fmaf(f, f, s2);
            }
            for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            if (lane == 0) s_f[warp] = s2;
            __syncthreads();
            s2 = 0.0f;
#pragma unroll
            for (int h = 0; h < kCpWarps; ++h) s2 += s_f[h];
            wn2 = wn2_first = (double)s2;
            wbias = bias_above(wn2);
            if (weak(wn2) && lost()) return;
            for (int i = tid; i < np; i += kCpThreads) split_w(i, w[i]);
        } else {
            wbias = bias_above(e2v);
            const double *v0 = ring + lo_[0];
            float s2 = 0.0f;
            for (int i = tid; i < np; i += kCpThreads) {
                double x = v0[i] * E[i];
                for (int t0 = 0; t0 < nl0; t0 += 4) {
                    double y[4], cc[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int t = min(t0 + u, nl0 - 1);
                        y[u] = ring[lo_[t] + i];
                        cc[u] = lc[t];
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) if (t0 + u < nl0) x = fma(-cc[u], y[u], x);
                }
                w[i] = x;
                split_w(i, x);
                const float f = f32_trunc(x);
                s2 = fmaf(f, f, s2);
            }
            // |w|^2, read against the swept norm and the coefficients only: FP32
            for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            if (lane == 0) s_f[warp] = s2;
            if (weak(e2v) && lost()) return;
        }
        int fl, nfull = 0;
        for (;;) {
            __syncthreads();
            // c_t = <v_t, w>, a lane a vector (no sums across lanes), the warps over groups of 32 vectors
            // and parts of the elements
            const bool want_n = !newv && nfull == 0;
            {
                const int tg = (nvec + 31) >> 5, P = tg > 0 ? kCpWarps / tg : 0;
                const int gi = tg > 0 ? warp % tg : 0, pa = tg > 0 ? warp / tg : 1, v = 32 * gi + lane;
                if (pa < P) {
                    const int i1 = (pa + 1) * np / P, vc = min(v, nvec - 1);
                    FixedSum acc{0, 0};
                    const int *va = Va + vc, *vb = Vb + vc;
#pragma unroll 4
                    for (int i = pa * np / P; i < i1; ++i) {
                        const int2 x = wab[i];
                        fixed_step(acc, va[(size_t)i * RS], vb[(size_t)i * RS], x.x, x.y);
                    }
                    part[pa * 32 * tg + v] = acc;
                }
                __syncthreads();
                float cm = 0.0f;
                for (int q = tid; q < nvec; q += kCpThreads) {
                    FixedSum x = part[q];
                    for (int r = 1; r < P; ++r) x = fixed_add(x, part[r * 32 * tg + q]);
                    const double ct = fixed_value(x, wbias);
                    c[q] = ct;
                    cm = f32_trunc(ct);
                    cf[q] = cm * 0x1p-30f;   // (against the a planes)
                }
                cm = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(cm))));
                if (lane == 0) s_cm[warp] = cm;
            }
            __syncthreads();
            float wf = 0.0f, cm = 0.0f;
#pragma unroll
            for (int q = 0; q < kCpWarps; ++q) { wf += s_f[q]; cm = fmaxf(cm, s_cm[q]); }
            if (want_n) wn2 = (double)wf;
            const bool small = want_n && (cm * 1e9f) * (cm * 1e9f) * (float)max(nvec, 1) <= wf && wf > 1e-30f;
            // the update: every element's sum by tgs threads, each its part of the vectors
            if (tgp < tgs && ei < np) {
                const int t0 = tgp * nvec / tgs, t1 = (tgp + 1) * nvec / tgs;
                const int *va = Va + (size_t)ei * RS, *vb = Vb + (size_t)ei * RS;
                if (small) {
                    float a0 = 0.0f, a1 = 0.0f;
                    int q = t0;
                    for (; q + 1 < t1; q += 2) {
                        a0 = fmaf(cf[q], (float)va[q], a0);
                        a1 = fmaf(cf[q + 1], (float)va[q + 1], a1);
                    }
                    if (q < t1) a0 = fmaf(cf[q], (float)va[q], a0);
                    fpart[tid] = a0 + a1;
                } else {
                    FixedSum acc{0, 0};
                    for (int q = t0; q < t1; ++q) {
                        const int2 ct = fixed_of(c[q], wbias);
                        fixed_step(acc, va[q], vb[q], ct.x, ct.y);
                    }
                    part[tid] = acc;
                }
            }
            __syncthreads();
            for (int i = tid; i < np; i += kCpThreads) {
                double x = w[i];
                if (small) {
                    float a = fpart[i];
                    for (int r = 1; r < tgs; ++r) a += fpart[r * npw + i];
                    x -= f32_to_double(a);
                } else {
                    FixedSum acc = part[i];
                    for (int r = 1; r < tgs; ++r) acc = fixed_add(acc, part[r * npw + i]);
                    x -= fixed_value(acc, wbias);
                }
                w[i] = x;
                split_w(i, x);   // (for |w|^2 and m; the dot products are done)
                ew[i] = E[i] * x;
            }
            __syncthreads();
            // the scalars of the updated w: <w|E|w> and <v_last(q)|E|w> in FP64, a warp each, beside <M_d|w> in
            // fixed point, four a warp; the last warp takes |w|^2, in fixed point too (w is no shorter than
            // kFixedShort allows against what it is split against), |E w|^2, a threshold's scale, in FP32, and
            // with them k_lanczos's decision, its lanes one threshold each (exhaustion first: further sweeps of
            // a w that holds nothing leave nothing)
            if (warp == kCpWarps - 1) {
                FixedSum p{0, 0};
                float s2 = 0.0f;
                int h = 0;   // (the low words' squares have one sign)
                for (int i = lane; i < np; i += 32) {
                    const int2 x = wab[i];
                    fixed_step(p, h, x.x, x.y, x.x, x.y);
                    const float f = f32_trunc(ew[i]);
                    s2 = fmaf(f, f, s2);
                }
                p = fixed_carry(p, h);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    p = fixed_add(p, fixed_shfl(p, o));
                    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
                }
                const double x2 = fixed_value(p, 2 * wbias - 1023);
                const double lim = lane == 0 ? eta2 * wn2 : (lane == 1 ? thr_exh : lane == 2 ? tau : kFixedShort) * wn2_first;
                const unsigned lt_ = __ballot_sync(0xffffffffu, x2 < lim), le = __ballot_sync(0xffffffffu, x2 <= lim);
                const long long xb = __double_as_longlong(x2);
                const bool zero = (xb << 1) == 0, fin = (xb & 0x7ff0000000000000LL) != 0x7ff0000000000000LL;
                int f;
                if ((le & 2u) || zero) f = (dcur < dtot) ? 2 : 3;
                else if (nvec > 0 && nfull + 1 < 4 && (lt_ & 1u)) f = 1;
                else if (nvec > 0 && nfull == 0 && (lt_ & 8u)) f = 4;
                else if (!(le & 4u) && fin) f = 0;
                else f = 3;   // (not finite)
                const double r = rsqrt_cubic(x2);
                const double y = (lane == 0 ? 1.0 : lane == 1 ? x2 : f32_to_double(s2) * r) * r;
                if (lane < 3) s_n[lane] = y;
                if (lane == 0) { sc[0] = x2; s_fl = f; }
            } else if (warp >= kCpWarps - 3) {
                const int d0 = 4 * (kCpWarps - 2 - warp);
                if (d0 < D) {
                    FixedSum acc[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) acc[u] = FixedSum{0, 0};
                    for (int i = lane; i < np; i += 32) {
                        const int2 x = wab[i];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (d0 + u < D) fixed_step(acc[u], Ma[(size_t)(d0 + u) * np4 + i], Mb[(size_t)(d0 + u) * np4 + i], x.x, x.y);
                    }
                    const FixedSum r = warp_sums_of<4>(acc, lane, fixed_add, fixed_shfl);
                    const int d = d0 + (lane >> 3);
                    if ((lane & 7) == 0 && d < D) sc[3 + d] = fixed_value(r, wbias + s_mb[d] - 1023);
                }
            } else {
                for (int q = warp - 1; q < nq; q += kCpWarps - 3) {   // q -1: <w|E|w>
                    const double *a = q < 0 ? w : lslot[q] >= 0 ? vecd(lslot[q], q) : nullptr;
                    double x = 0.0;
                    if (a)
                        for (int i = lane; i < np; i += 32) x = fma(a[i], ew[i], x);
                    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                    if (lane == 0) sc[q < 0 ? 1 : 3 + D + q] = x;
                }
            }
            __syncthreads();
            fl = s_fl;
            if (nfull++ > 0 && !rough) ++extra;
            rough = fl == 4;
            if (fl != 1 && fl != 4) break;
            wn2 = sc[0];   // another sweep, of the updated w
            wbias = bias_above(wn2);
            for (int i = tid; i < np; i += kCpThreads) split_w(i, w[i]);
        }
        if (fl == 3) return;   // the full space's (handled stays 0)
        if (fl == 2) {
            // exhausted: the rest of this pivot chain takes unreached directions
            const int jend = (k + 1 < C.n_used) ? min(L, s_start[k + 1]) : L;
            const int nr = jend - j;
            for (int r = tid; r < nr; r += kCpThreads) {
                const int d = dcur + r;
                const double a = s_gE[d < dtot ? group_of(d) : Q - 1];
                double *row = C.out + (size_t)(j + r) * NT;
                for (int e = 0; e < NT; ++e) row[e] = 0.0;
                row[0] = a;
                rowslot[j + r] = -1;
            }
            dcur = min(dcur + nr, dtot);
            ndefl += nr;
            j = jend - 1;
            __syncthreads();
            continue;
        }
        if (nvec >= R) return;   // (beyond the space's dimension: not reached with exact arithmetic)
        // normalise and store; the row
        const double ixb = s_n[0];
        e2v = s_n[2];
        {
            double *rg = ring + (nvec & 1) * np4, *rl = (j == s_last[k] && k < nla) ? lasts + (size_t)k * np4 : nullptr;
            for (int i = tid; i < np; i += kCpThreads) {
                const double v = w[i] * ixb;
                const int2 f = fixed_of(v, 1023);
                Va[(size_t)i * RS + nvec] = f.x;
                Vb[(size_t)i * RS + nvec] = f.y;
                rg[i] = v;
                if (rl) rl[i] = v;
                reinterpret_cast<double *>(C.V)[(size_t)nvec * np + i] = v;   // (np <= N: within the chain's store)
            }
        }
        // the row, and the next step's recurrence from it, by the last warp (the first ones hold the
        // elements)
        if (warp == kCpWarps - 1) {
            double x = 0.0;
            if (lane < NT) {
                int e = -1;   // the row's entry from sc
                if (lane == 0) e = 1;
                else if (lane == 1) e = (newv && k >= 1) ? 3 + D + (k - 1) : -1;
                else if (lane < 2 + k) e = 3 + D + (lane - 2);
                else if (lane >= C.nden_out && lane < C.nden_out + D) e = 3 + (lane - C.nden_out);
                if (e >= 0) x = sc[e] * ixb;
                if (lane == 0) x *= ixb;
                if (lane == 1 && e < 0) x = s_n[1];
                C.out[(size_t)j * NT + lane] = x;
            }
            // lane 0: v_j, lane 1: v_{j-1}, lane 2 + q: chain q's last
            int v = -1;
            if (lane == 0) v = nvec;
            else if (lane == 1) v = j >= 1 ? rowslot[j - 1] : -1;
            else if (lane < 2 + k) v = s_last[lane - 2] < j - 1 ? rowslot[s_last[lane - 2]] : -1;
            const unsigned m = __ballot_sync(0xffffffffu, v >= 0);
            if (v >= 0) {
                const int n = __popc(m & ((1u << lane) - 1u));
                lo_[n] = v >= nvec - 1 ? (v & 1) * np4 : (2 + lane - 2) * np4;   // (lasts behind the ring)
                lc[n] = x;
            }
            if (lane == 0) { rowslot[j] = nvec; s_nl = __popc(m); }
        }
        ++nvec;
        __syncthreads();
        nl0 = s_nl;
    }
    for (int q = tid; q < L; q += kCpThreads) C.rowslot[q] = rowslot[q];
    if (tid == 0) {
        atomicAdd(&C.stat[0], extra);
        atomicAdd(&C.stat[2], ndefl);
        S.info->np = np;
        S.info->ng = ng;
        S.info->nvec = nvec;
        S.info->handled = 1;
    }
    for (int g = tid; g < ng; g += kCpThreads) S.grp[g].off = s_off[g];
}

// The stored vectors of a compact chain in the poles' space, into out (slot-major, stride
// C.ld): a thread per pole, its group's L^-T v' formed by the D-term back substitution
// against the pole's own couplings (y = L^-1 M_p, then v_p = sum_c y_c v'_c).
__global__ void k_lz_expand(const LzChain C, double *out) {
    const CompactScratch S = lz_compact(C.cp);
    const int np = S.info->np, ng = S.info->ng, nvec = S.info->nvec, D = C.D;
    const double *V = reinterpret_cast<const double *>(C.V);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < C.N; i += gridDim.x * blockDim.x) {
        int lo = 0, hi = ng - 1;   // the last group starting at or before pole i
        while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (S.grp[mid].p0 <= i) lo = mid; else hi = mid - 1; }
        const CompactGroup G = S.grp[lo];
        double y[8];
        if (!G.kept) {
            const double *Lg = S.L + (size_t)lo * 64;
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                y[a] = 0.0;
                if (a < D) {
                    double s = C.M[(size_t)a * C.N + i];
#pragma unroll
                    for (int b = 0; b < a; ++b) s = fma(-Lg[a * D + b], y[b], s);
                    y[a] = (Lg[a * D + a] != 0.0) ? s / Lg[a * D + a] : 0.0;
                }
            }
        }
        for (int t = 0; t < nvec; ++t) {
            const double *vt = V + (size_t)t * np + G.off;
            double s = 0.0;
            if (G.kept) {
                s = vt[i - G.p0];
            } else {
#pragma unroll
                for (int a = 0; a < 8; ++a) if (a < D) s = fma(y[a], vt[a], s);
            }
            out[(size_t)t * C.ld + i] = s;
        }
    }
}

// ------------------------------------------------------------------ full Dyson
// One CTA per pole set (C.E, C.M sorted; C.cp from k_lz_groups): its rows for the Dyson
// matrix to io.E [N] and io.M [D][N].  A set in which no group is rotated keeps the order it
// was built in (io.E0, io.M0).
__global__ void __launch_bounds__(kCpThreads) k_plain_rotate(const LzChain *chains, const PlainIO *ios, int nchains) {
    const int cid = blockIdx.x;
    if (cid >= nchains) return;
    const LzChain C = chains[cid];
    const PlainIO io = ios[cid];
    const CompactScratch S = lz_compact(C.cp);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, N = C.N, D = C.D;
    __shared__ int ws[kCpWarps];
    __shared__ int s_first[kCpGroups + 1];
    __shared__ int s_any;
    __shared__ double s_tri[kCpWarps][kGramEntries], s_l[kCpWarps][64];
    const int Q = S.info->q;
    if (tid == 0) s_any = 0;
    __syncthreads();
    const int ng = Q > 0 ? merge_groups(C.gE, Q, s_first, ws) : 0;
    for (int g = warp; g < ng; g += kCpWarps)
        if (S.start[s_first[g + 1]] - S.start[s_first[g]] > kKeep && lane == 0) s_any = 1;
    __syncthreads();
    if (!s_any) {
        for (int i = tid; i < N; i += kCpThreads) io.E[i] = io.E0[i];
        for (size_t i = tid; i < (size_t)D * N; i += kCpThreads) io.M[i] = io.M0[i];
        return;
    }
    __shared__ int s_state[kCpGroups];
    for (int g = warp; g < ng; g += kCpWarps) {
        const int q0 = s_first[g], q1 = s_first[g + 1];
        int rot = 0;
        if (S.start[q1] - S.start[q0] > kKeep) {
            for (int e = lane; e < D * (D + 1) / 2; e += 32) {
                double s = 0.0;
                for (int q = q0; q < q1; ++q) s += S.gram[(size_t)q * kGramEntries + e];
                s_tri[warp][e] = s;
            }
            __syncwarp();
            rot = warp_cholesky(s_tri[warp], D, s_l[warp], lane);
            __syncwarp();
            if (rot)
                for (int e = lane; e < D * D; e += 32) S.L[(size_t)g * 64 + e] = s_l[warp][e];
        }
        if (lane == 0) s_state[g] = rot;
        __syncwarp();
    }
    __syncthreads();
    lossy_factors(C, S, s_first, ng, s_state, s_l, s_tri);
    for (int g = warp; g < ng; g += kCpWarps) {
        const int p0 = S.start[s_first[g]], m = S.start[s_first[g + 1]] - p0;
        const bool rot = s_state[g] != 0;
        const double *L = S.L + (size_t)g * 64;
        const double eg = 0.5 * (C.E[p0] + C.E[p0 + m - 1]);
        for (int i = lane; i < m; i += 32) {
            io.E[p0 + i] = (rot && i < D) ? eg : C.E[p0 + i];
            for (int d = 0; d < D; ++d)
                io.M[(size_t)d * N + p0 + i] = !rot ? C.M[(size_t)d * N + p0 + i] : i < D ? L[d * D + i] : 0.0;
        }
    }
}

cudaError_t launch_plain_rotate(const LzChain *d_chains, const PlainIO *d_ios, int nchains, cudaStream_t st) {
    if (nchains <= 0) return cudaSuccess;
    k_plain_rotate<<<nchains, kCpThreads, 0, st>>>(d_chains, d_ios, nchains);
    return cudaGetLastError();
}

cudaError_t launch_lz_compact(const LzChain *d_chains, int nchains, double eta, cudaStream_t st) {
    if (nchains <= 0) return cudaSuccess;
    cudaError_t e = allow_dynamic_smem((const void *)k_lz_compact);
    if (e != cudaSuccess) return e;
    k_lz_compact<<<nchains, kCpThreads, kCpSmem, st>>>(d_chains, nchains, eta * eta);
    return cudaGetLastError();
}

cudaError_t launch_lz_expand(const LzChain &chain, double *out, cudaStream_t st) {
    k_lz_expand<<<(chain.N + 127) / 128, 128, 0, st>>>(chain, out);
    return cudaGetLastError();
}

void compact_smem_init() { allow_dynamic_smem((const void *)k_lz_compact); }

}  // namespace bd
