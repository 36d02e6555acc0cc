// k_lanczos_long.cu -- the multi-pivot Lanczos reduction with FP64 vectors of long chains
// whose energies are (nearly) all distinct: dressed propagators, and caller-owned pole sets.
//
// The steps, decisions and rows are k_lanczos's.  What differs is the sweep over the stored
// vectors, which is where the time goes and which an FP64 form leaves at the FP64 unit (an
// instruction holds an SM sub-partition's for ~64 cycles).  A basis vector has |v_i| <= 1 and
// the sweep needs c_t = <v_t|w> to a fixed part of |w|, so both are fixed-point numbers here:
//   - a stored vector is two planes of 32-bit integers, v = (a 2^27 + b) 2^-57 (a of 30 bits and
//     sign, b centred): the same 8 bytes a pole as a double, an absolute error of 2^-58.  The two
//     newest vectors, which the recurrence reads, are kept as doubles besides;
//   - w is split the same way against a power of two above |w| (above |E v_{j-1}| after a
//     recurrence, of which w is a projection), and a dot product is three 32 x 32 -> 64 bit
//     multiply-adds an element, exact sums on the integer pipe (run by run of what a word holds,
//     lz_fixed.cuh): c_t is off by about 2^-57 |w|, where FP64's own sum is off by 1e-16 |w|.  w's words are
//     dithered, so that elements of one size leave no sum of their low words' products (which at the most
//     would be n 2^-62 |w|; as a fourth product an element they cost a chain of 20 000 poles 4.7 %);
//   - the update w -= sum c_t v_t runs in FP32 from the a planes alone (4 bytes a pole) where
//     every |c_t| <= kSmall |w|, which after a recurrence is the rule: its error is below 2^-23
//     kSmall sqrt(R) |w|.  Otherwise (new pivots, further sweeps) it is fixed point too.
// The recurrence, the norm, alpha, m and g stay FP64 with as few instructions as they take.
//
// What a chain needs beyond that -- a restart vector, energies or couplings outside 2^+-40, a
// vector (a weakly coupled orbital's, say) whose |w|^2 the FP32 scale does not hold (kFixedWeak),
// fewer poles than lz_long_from says -- is left to k_lanczos as a whole (C.done stays 0), which the
// host launches behind this kernel.
//
// Work split: a cluster per chain, CTA r the pole rows [r S, (r+1) S), 512 threads and an SM to
// itself; a part of four vectors a warp in the dot products, a thread per two or four poles
// everywhere else.  A step is two cluster reductions.  With an SM's whole shared memory taken by
// the slices L1 is a few KB, so what does not fit in registers costs an L2 access: the uniform
// state is read from shared memory where it is used and the loads in flight are unconditional
// (with 250 bytes a thread spilled the step below took 9.4 ms).
// Bound by the planes' traffic and the phases around it in batches (12 bytes a stored element
// and step: 2.1 M poles in 52 chains, 20 iterations a pivot, 18.3 -> 7.6 ms against 3.2 at the
// copy bandwidth; two thirds of a 41 000-pole chain's step are the sweep's loads, a fifth the
// FP64 instructions) and by the chain of phases for one chain on its 16 SMs (20 000 poles, 80
// vectors: the call 5.36 -> 2.27 ms).  FP64 dot products took 17.1 and 4.2 ms, double-float ones
// formed from the doubles' bits 12.5 and 3.1 (off by 2e-15 |w| where this is off by 5e-16, as
// FP64 is).
#include <algorithm>
#include <cfloat>
#include <cooperative_groups.h>
#include "bd_common.cuh"
#include "bd_kernels.h"
#include "lz_fixed.cuh"

namespace cg = cooperative_groups;

namespace bd {

namespace {

constexpr int kLongThreads = 512, kMaxWarps = kLongThreads / 32;
constexpr int kMaxSc = 20;             // |w|^2, <w|E|w>, 8 m, 8 g; the last: |E w|^2
constexpr float kSmall = 1e-10f;

__device__ __forceinline__ int4 ld4(const int *p) { return *reinterpret_cast<const int4 *>(p); }
__device__ __forceinline__ double2 ld2(const double *p) { return *reinterpret_cast<const double2 *>(p); }
__device__ __forceinline__ void st2(double *p, double a, double b) { *reinterpret_cast<double2 *>(p) = make_double2(a, b); }

// warps that share a vector's dot product, each a part of the elements: the vectors then divide
// among the warps more evenly (17 of them: 5 quarters a warp against 2 wholes; 5164 elements of 30
// vectors 72 000 clocks against 88 000), while a part below 512 elements is mostly remainder (1252
// elements: halves 15 000, quarters 17 000) and the parts' sums of many rows would take the room
// of the slices
__host__ __device__ inline int long_parts_max(int rmax) { return rmax <= 160 ? 4 : 1; }
__host__ __device__ inline int long_parts(int rmax, int S) { return min(long_parts_max(rmax), S >= 2048 ? 4 : 2); }
// shared memory before the slices: A[2][at most parts_max][rq] sums (FixedSum), c[rq], sp[2][kMaxSc], red[16][kMaxSc]
// (doubles), cf[rq] (floats), rowslot[rq] (ints)
__host__ __device__ inline size_t long_fixed(int rmax) {
    const size_t rq = ((size_t)rmax + 4) & ~(size_t)3;
    return sizeof(FixedSum) * 2 * long_parts_max(rmax) * rq + sizeof(double) * (rq + 2 * kMaxSc + kMaxWarps * kMaxSc) + 8 * rq;
}
// A warp's part of four dot products (the last vector again where there are fewer): elements
// [0, n) of this lane's start (n less that start), va the vectors' first planes there, pb from
// those to the second planes.
__device__ __forceinline__ void long_dots(FixedSum (&acc)[4], const int *const (&va)[4], int pb, const int *wa,
                                          int S, int n) {
#pragma unroll 1
    for (int r = 0; r < n; r += 32 * kFixedRun) {
        const int end = min(n, r + 32 * kFixedRun);
#pragma unroll 1
        for (int i = r; i < end; i += 128) {
            int4 x[4], y[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                x[u] = ld4(va[u] + i);
                y[u] = ld4(va[u] + pb + i);
            }
            const int4 a = ld4(wa + i), b = ld4(wa + S + i);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                fixed_step(acc[u], x[u].x, y[u].x, a.x, b.x);
                fixed_step(acc[u], x[u].y, y[u].y, a.y, b.y);
                fixed_step(acc[u], x[u].z, y[u].z, a.z, b.z);
                fixed_step(acc[u], x[u].w, y[u].w, a.w, b.w);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u] = fixed_carry(acc[u]);
    }
}

// Whether one of the n pivots (of D) has couplings that the ones before it span but for the part tol of
// their square: elimination in the pivots' order of their Gram matrix, from the orbitals' (G, lower
// triangle).  A warp; H holds n^2 values.
template <typename T>
__device__ bool pivots_depend(const T *G, const double *piv, int n, int D, T *H, T tol, int lane) {
    for (int e = lane; e < n * n; e += 32) {
        const double *a = piv + e / n * D, *b = piv + e % n * D;
        T s = 0;
        for (int c = 0; c < D; ++c) {
            T t = 0;
            for (int d = 0; d < D; ++d) t += G[c >= d ? c * (c + 1) / 2 + d : d * (d + 1) / 2 + c] * (T)b[d];
            s += (T)a[c] * t;
        }
        H[e] = s;
    }
    __syncwarp();
    const T own = lane < n ? H[lane * n + lane] : (T)0;
    for (int q = 0; q < n; ++q) {
        const T p = H[q * n + q];
        if (!(p > tol * __shfl_sync(0xffffffffu, own, q))) return true;   // the same in every lane
        const T inv = (T)1 / p;
        for (int e = lane; e < n * n; e += 32) {
            const int a = e / n, b = e % n;
            if (a > q && b > q) H[e] -= H[a * n + q] * inv * H[q * n + b];
        }
        __syncwarp();
    }
    return false;
}

// The CTA's sums of m_a m_b over its poles into G (shared memory), warp after warp.
template <typename T, typename Coupling>
__device__ __forceinline__ void long_gram(int S, int D, double *G, Coupling coupling) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    T g[kGramEntries];
#pragma unroll
    for (int u = 0; u < kGramEntries; ++u) g[u] = 0;
    for (int i = tid; i < S; i += kLongThreads) {
        T m[8];
#pragma unroll
        for (int d = 0; d < 8; ++d) m[d] = d < D ? coupling(d, i) : (T)0;
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b)
                if (a < D) g[a * (a + 1) / 2 + b] += m[a] * m[b];
    }
    T own[2] = {0, 0};   // entries lane and lane + 32
#pragma unroll
    for (int u = 0; u < kGramEntries; ++u)
        if (u < D * (D + 1) / 2) {
            T x = g[u];
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if (lane == (u & 31)) own[u >> 5] = x;
        }
    for (int q = 0; q < kMaxWarps; ++q) {
        if (warp == q) {
            G[lane] = (q ? G[lane] : 0.0) + (double)own[0];
            if (lane + 32 < kGramEntries) G[lane + 32] = (q ? G[lane + 32] : 0.0) + (double)own[1];
        }
        __syncthreads();
    }
}

// Whether the chain's pivots depend on one another, from their couplings: FP32 sums tell nearly all sets that
// do not, FP64 ones the rest.  The whole cluster, with the same answer; sm: 160 doubles.
__device__ __noinline__ bool couplings_depend(const LzChain &C, int S, int i0, double *sm) {
    cg::cluster_group cluster = cg::this_cluster();
    const int CL = (int)cluster.num_blocks(), lane = threadIdx.x & 31, n = min(C.n_used, 9);
    double *mine = sm, *all = sm + 36, *H = sm + 72;   // (H: 81)
    int *flag = reinterpret_cast<int *>(sm + 156);
    const double *cp = C.M + i0;
    const int own = min(S, C.N - i0);
    auto coupling = [&](int d, int i) { return i < own ? cp[(size_t)d * C.N + i] : 0.0; };
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 0) long_gram<float>(S, C.D, mine, [&](int d, int i) { return f32_trunc(coupling(d, i)); });
        else long_gram<double>(S, C.D, mine, coupling);
        cluster.sync();
        if (threadIdx.x < 36) {
            double x = 0.0;
            for (int r = 0; r < CL; ++r) x += cluster.map_shared_rank(mine, r)[threadIdx.x];
            all[threadIdx.x] = x;
        }
        cluster.sync();   // (peers have read mine)
        if (threadIdx.x < 32) {
            bool d;
            if (pass == 0) {
                float *G = reinterpret_cast<float *>(mine);
                for (int u = lane; u < 36; u += 32) G[u] = (float)all[u];
                __syncwarp();
                d = pivots_depend<float>(G, C.piv, n, C.D, reinterpret_cast<float *>(H), 1e-4f, lane);
            } else {
                d = pivots_depend<double>(all, C.piv, n, C.D, H, 1e-13, lane);
            }
            if (lane == 0) *flag = d;
        }
        __syncthreads();
        const bool dep = *flag != 0;
        __syncthreads();
        if (!dep) return false;
    }
    return true;
}

}  // namespace

// CTAs a chain where the slices are in shared memory: at one CTA an SM the GPCs hold 15 clusters of
// nine as of eight, so nine put 135 SMs to work for 120.  (Ten: 13 clusters.)
__host__ __device__ inline int long_cluster(int cluster) { return cluster == 8 ? 9 : cluster; }
__host__ __device__ inline int long_slice(int N, int cluster) { return ((N + cluster - 1) / cluster + 3) / 4 * 4; }
__host__ __device__ inline bool long_fits(int N, int cluster, int rmax, size_t smem) {
    return long_fixed(rmax) + 32 * (size_t)long_slice(N, long_cluster(cluster)) <= smem;
}

// SS: w, its split and the two newest vectors in shared memory (else in the chain's global scratch).
template <bool SS>
__global__ void __launch_bounds__(kLongThreads, 1) k_lz_long(const LzChain *chains, int nchains, int rmax, int nmin, double eta2,
                                                    int smem_bytes) {
    cg::cluster_group cluster = cg::this_cluster();
    const int CL = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), cid = blockIdx.x / CL;
    if (cid >= nchains) return;
    __shared__ LzChain C;   // (registers are short: what does not fit goes to an L1 of a few KB)
    if (threadIdx.x < sizeof(LzChain) / 4)
        reinterpret_cast<int *>(&C)[threadIdx.x] = reinterpret_cast<const int *>(chains + cid)[threadIdx.x];
    __syncthreads();
    if (!C.done || *C.done || C.N < nmin) return;   // (the whole cluster leaves together)
    if (long_fits(C.N, CL, rmax, smem_bytes) != SS) return;   // the other form's
    const int S = long_slice(C.N, CL), i0 = rank * S;
    constexpr int T = kLongThreads, NW = kMaxWarps;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    extern __shared__ double sm[];
    const int rq = (rmax + 4) & ~3;
    const int np = long_parts(rmax, S), cl2 = 32 - __clz(CL - 1);   // 2^cl2 lanes for the CTAs
    FixedSum *A = reinterpret_cast<FixedSum *>(sm);
    double *c = reinterpret_cast<double *>(A + 2 * long_parts_max(rmax) * rq), *sp = c + rq, *red = sp + 2 * kMaxSc;
    float *cf = reinterpret_cast<float *>(red + kMaxWarps * kMaxSc);
    int *rowslot = reinterpret_cast<int *>(cf + rq);
    // slices: w, the two newest vectors and w's split (two planes); E and M beside them when they
    // fit, and the earlier chains' last vectors as doubles (the recurrence and the g read them)
    double *const w = SS ? sm + long_fixed(rmax) / sizeof(double)
                         : reinterpret_cast<double *>(C.slice + (size_t)rank * C.slice_stride);
    double *const ring = w + S;
    int *const ws = reinterpret_cast<int *>(w + 3 * (size_t)S);
    __shared__ int s_oE, s_oM, s_oL, s_nl;   // where in sm, -1: not there; last vectors held
    if (tid == 0) {
        int o = (int)(long_fixed(rmax) / sizeof(double)) + (SS ? 4 * S : 0);
        const int end = smem_bytes / (int)sizeof(double);
        s_oE = s_oM = -1;
        if (end - o >= S) { s_oE = o; o += S; }
        if (end - o >= C.D * S) { s_oM = o; o += C.D * S; }
        s_oL = o;
        s_nl = min(max(C.n_used - 1, 0), (end - o) / S);
    }
    __shared__ int s_start[10], s_last[10], lslot[8], lt[16], lq[16];
    __shared__ double lc[16], s_row[32], s_tot[kMaxSc];
    __shared__ double s_n[3];   // 1/|w|, |w|, |E v|^2 of the kept vector
    __shared__ int s_fl;        // 0 keep, 1 sweep again, 2 exhausted, 3 the full space's, 4 sweep again (split too coarse)
    __shared__ unsigned s_rng[2];
    __shared__ float4 s_w2[2][NW / 4];   // the warps' parts of |w|^2, by the parity of A
    if (tid < 2) s_rng[tid] = 0;
    if (tid <= C.n_used && tid < 10) s_start[tid] = C.start[tid];
    if (tid < C.n_used && tid < 10) s_last[tid] = C.last[tid];
    __syncthreads();
    {   // energies and couplings inside 2^+-40 (the largest of each): FP32's exponents hold all that follows
        unsigned me = 0, mm = 0;
        for (int i = tid; i < S; i += T) {
            const bool in = i < min(S, C.N - i0);
            const double e = in ? C.E[i0 + i] : 0.0;
            if (s_oE >= 0) sm[s_oE + i] = e;
            me = max(me, (unsigned)__double2hiint(e) & 0x7fffffffu);
            for (int d = 0; d < C.D; ++d) {
                const double m = in ? C.M[(size_t)d * C.N + i0 + i] : 0.0;
                if (s_oM >= 0) sm[s_oM + d * S + i] = m;
                mm = max(mm, (unsigned)__double2hiint(m) & 0x7fffffffu);
            }
        }
        me = __reduce_max_sync(0xffffffffu, me);
        mm = __reduce_max_sync(0xffffffffu, mm);
        if (lane == 0) { atomicMax(&s_rng[0], me); atomicMax(&s_rng[1], mm); }
        cluster.sync();
        for (int r = 0; r < CL; ++r) {
            const unsigned *p = cluster.map_shared_rank(&s_rng[0], r);
            me = max(me, p[0]);
            mm = max(mm, p[1]);
        }
        cluster.sync();   // peers have read s_rng (a CTA that leaves frees its shared memory)
        if (!fixed_range(me) || !fixed_range(mm)) return;
    }
    const int Qg = C.gE ? C.gInfo[0] : 0;
    const int dtot = Qg > 0 ? C.gInfo[Qg] : 0;
    // Pivots that depend on one another (an orbital that couples to nothing among them) end a chain in a
    // restart vector where no unreached direction is left: k_lanczos's from the start, not after rows of it
    // here (20 000 poles, the last orbital the first less the second: 6.5 ms; 5.5 by k_lanczos alone).
    if (dtot == 0 && couplings_depend(C, S, i0, sm)) return;
    int nvec = 0;
    // planes of stored vector t: a at the address, b C.ld behind it
    int *Vg = reinterpret_cast<int *>(C.V) + i0;
    auto plane = [&](int t) -> int * { return Vg + 2 * (size_t)t * C.ld; };
    // elements i, i + 1 of vector t as doubles (q: the chain it is the last vector of, or -1)
    auto vec2 = [&](int t, int q, int i) -> double2 {
        if (t >= nvec - 2) return ld2(ring + (size_t)(t & 1) * S + i);
        if (q >= 0 && q < s_nl) return ld2(sm + s_oL + q * S + i);
        const int *p = plane(t) + i;
        const int2 x = *reinterpret_cast<const int2 *>(p), y = *reinterpret_cast<const int2 *>(p + C.ld);
        return make_double2(fixed_to_double(x.x, y.x), fixed_to_double(x.y, y.y));
    };
    auto energy2 = [&](int i) -> double2 {   // of poles i, i + 1 of the slice
        if (s_oE >= 0) return ld2(sm + s_oE + i);
        return make_double2(i < min(S, C.N - i0) ? C.E[i0 + i] : 0.0, i + 1 < min(S, C.N - i0) ? C.E[i0 + i + 1] : 0.0);
    };
    auto coupling2 = [&](int d, int i) -> double2 {
        if (s_oM >= 0) return ld2(sm + s_oM + d * S + i);
        const double *p = C.M + (size_t)d * C.N + i0 + i;
        return make_double2(i < min(S, C.N - i0) ? p[0] : 0.0, i + 1 < min(S, C.N - i0) ? p[1] : 0.0);
    };
    int wbias = 1023;   // exponent field of the power of two w is split against
    auto split_w = [&](int i, double a, double b) {
        const int2 x = fixed_dithered(a, wbias, i), y = fixed_dithered(b, wbias, i + 1);
        *reinterpret_cast<int2 *>(ws + i) = make_int2(x.x, y.x);
        *reinterpret_cast<int2 *>(ws + S + i) = make_int2(x.y, y.y);
    };
    auto group_of = [&](int d) {
        int lo = 0, hi = Qg - 1;
        while (lo < hi) { const int mid = (lo + hi) >> 1; if (C.gInfo[1 + mid] > d) hi = mid; else lo = mid + 1; }
        return lo;
    };
    constexpr double tau = 1e-48, thr_exh = 1e-20;   // k_lanczos's, FP64 vectors
    int dcur = 0, ndefl = 0, extra = 0, k = -1, dpar = 0, spar = 0, nl0 = 0;
    double e2v = 0.0;
    bool ok = true, rough = false;   // rough: w much shorter than what it was split against, swept again
    for (int j = 0; j < C.L; ++j) {
        const bool newv = (k + 1 < C.n_used) && (j == s_start[k + 1]);
        if (newv) ++k;
        const int nq = k;
        if (tid < nq) lslot[tid] = rowslot[s_last[tid]];
        // w = M p, or E v_{j-1} less its known components
        double wn2 = 0.0, wn2_first = e2v;   // |w|^2 before the sweep, and of E v_{j-1} / M p (thresholds' scales)
        if (newv) {
            double p[8];
#pragma unroll
            for (int d = 0; d < 8; ++d) p[d] = d < C.D ? C.piv[(size_t)k * C.D + d] : 0.0;
            float s2 = 0.0f;
            for (int i = 2 * tid; i < S; i += 2 * T) {
                double a = 0.0, b = 0.0;
#pragma unroll
                for (int d = 0; d < 8; ++d)
                    if (d < C.D) {
                        const double2 m = coupling2(d, i);
                        a = fma(m.x, p[d], a);
                        b = fma(m.y, p[d], b);
                    }
                st2(w + i, a, b);
                const float x = f32_trunc(a), y = f32_trunc(b);
                s2 = fmaf(y, y, fmaf(x, x, s2));
            }
            for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            if (lane == 0) red[warp * kMaxSc] = (double)s2;
            __syncthreads();
            if (tid == 0) {
                double x = 0.0;
                for (int h = 0; h < NW; ++h) x += red[h * kMaxSc];
                sp[(size_t)spar * kMaxSc] = x;
            }
            cluster.sync();
            if (warp == 0) {
                double x = lane < CL ? *cluster.map_shared_rank(sp + (size_t)spar * kMaxSc, lane) : 0.0;
                for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                if (lane == 0) s_n[0] = x;
            }
            spar ^= 1;
            __syncthreads();
            wn2 = wn2_first = s_n[0];
            wbias = bias_above(wn2);
            for (int i = 2 * tid; i < S; i += 2 * T) {
                const double2 x = ld2(w + i);
                split_w(i, x.x, x.y);
            }
        } else {
            wbias = bias_above(e2v);
            const double *v0 = ring + (size_t)(lt[0] & 1) * S;
            float s2 = 0.0f;   // |w|^2 is read against the swept norm and the coefficients only
#pragma unroll 1
            for (int b = 2 * tid; b < S; b += 4 * T) {   // two poles here and two 2 T on, loads first
                const int i[2] = {b, b + 2 * T < S ? b + 2 * T : b};
                double2 x[2], e[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) { e[h] = energy2(i[h]); x[h] = ld2(v0 + i[h]); }
#pragma unroll
                for (int h = 0; h < 2; ++h) { x[h].x *= e[h].x; x[h].y *= e[h].y; }
#pragma unroll 1
                for (int t = 0; t < nl0; ++t) {
                    const double ct = -lc[t];
                    double2 y[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) y[h] = vec2(lt[t], lq[t], i[h]);
#pragma unroll
                    for (int h = 0; h < 2; ++h) { x[h].x = fma(ct, y[h].x, x[h].x); x[h].y = fma(ct, y[h].y, x[h].y); }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    if (h == 0 || b + 2 * T < S) {
                        st2(w + i[h], x[h].x, x[h].y);
                        split_w(i[h], x[h].x, x[h].y);
                        const float p = f32_trunc(x[h].x), q = f32_trunc(x[h].y);
                        s2 = fmaf(q, q, fmaf(p, p, s2));
                    }
            }
            for (int o = 16; o > 0; o >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, o);
            if (lane == 0) reinterpret_cast<float *>(s_w2[dpar])[warp] = s2;
        }
        int fl, nfull = 0;
        for (;;) {
            __syncthreads();
            // c_t = <v_t, w> for every stored vector: np warps a vector, each its part of the
            // elements, four vectors at a time
            FixedSum *Ap = A + (size_t)dpar * np * rq;
            const bool want_n = !newv && nfull == 0;
            {
                const int part = warp % np, nw = NW / np;
                const int pe = (S / 4 + np - 1) / np * 4, e0 = min(part * pe, S), pn_ = min(pe, S - e0);
                const int *wa = ws + e0 + 4 * lane;
                for (int t0 = warp / np; t0 < nvec; t0 += 4 * nw) {
                    const int nu = min(4, (nvec - 1 - t0) / nw + 1);   // stored vectors t0, t0 + nw, ..
                    const int *va[4];
                    FixedSum acc[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int t = min(t0 + u * nw, nvec - 1);
                        va[u] = plane(t) + e0 + 4 * lane;
                        acc[u] = FixedSum{0, 0};
                    }
                    long_dots(acc, va, C.ld, wa, S, pn_ - 4 * lane);
                    const FixedSum r = warp_sums_of<4>(acc, lane, fixed_add, fixed_shfl);
                    const int u = lane >> 3;
                    if ((lane & 7) == 0 && u < nu) Ap[part * rq + t0 + u * nw] = r;
                }
            }
            if (np > 1) {   // the parts' sums here: reads of the other CTAs cost more
                __syncthreads();
                for (int t = tid; t < nvec; t += T)
                    for (int q = 1; q < np; ++q) Ap[t] = fixed_add(Ap[t], Ap[q * rq + t]);
            }
            cluster.sync();
            // the CTAs' sums, one a lane: exact, so in any order
            for (int u0 = warp * 32; u0 < nvec << cl2; u0 += T) {
                const int u = u0 + lane, t = min(u >> cl2, nvec - 1), r = u & ((1 << cl2) - 1);
                FixedSum x = r < CL ? cluster.map_shared_rank(Ap, r)[t] : FixedSum{0, 0};
                for (int o = (1 << cl2) >> 1; o > 0; o >>= 1) x = fixed_add(x, fixed_shfl(x, o));
                if (r == 0 && u < nvec << cl2) {
                    const double ct = fixed_value(x, wbias);
                    c[t] = ct;
                    cf[t] = f32_trunc(ct) * 0x1p-30f;   // (against the a planes)
                }
            }
            if (want_n && warp == NW - 1) {   // four lanes a CTA
                float x2 = 0.0f;
                for (int r = lane >> 2; r < CL; r += 8) {
                    const float4 q = cluster.map_shared_rank(&s_w2[dpar][0], r)[lane & 3];
                    x2 += (q.x + q.y) + (q.z + q.w);
                }
                for (int o = 16; o > 0; o >>= 1) x2 += __shfl_xor_sync(0xffffffffu, x2, o);
                if (lane == 0) { c[nvec] = (double)x2; cf[nvec] = x2; }
            }
            dpar ^= 1;
            __syncthreads();
            if (want_n) wn2 = c[nvec];
            // the update and, of the updated w, this thread's part of the scalars
            float cm = 0.0f;
            for (int t = lane; t < nvec; t += 32) cm = fmaxf(cm, fabsf(cf[t]));
            for (int o = 16; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
            const bool small = want_n && cm * 0x1p30f <= kSmall * sqrtf(cf[nvec]);
#pragma unroll 1
            for (int i = 4 * tid; i < S; i += 4 * T) {
                double x[4];
                {
                    const double2 p = ld2(w + i), q = ld2(w + i + 2);
                    x[0] = p.x; x[1] = p.y; x[2] = q.x; x[3] = q.y;
                }
                if (small) {
                    float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    auto step = [&](float ct, int4 v) {
                        a[0] = fmaf(ct, (float)v.x, a[0]);
                        a[1] = fmaf(ct, (float)v.y, a[1]);
                        a[2] = fmaf(ct, (float)v.z, a[2]);
                        a[3] = fmaf(ct, (float)v.w, a[3]);
                    };
                    constexpr int NB = 8;   // vectors a round
#pragma unroll 1
                    for (int t = 0; t < nvec; t += NB) {
                        int4 v[NB];
                        const int *q = Vg + 2 * (size_t)t * C.ld + i;
#pragma unroll
                        for (int r = 0; r < NB; ++r)
                            v[r] = ld4(q + 2 * (size_t)min(r, nvec - 1 - t) * C.ld);
#pragma unroll
                        for (int r = 0; r < NB; ++r)
                            step(t + r < nvec ? cf[t + r] : 0.0f, v[r]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[e] -= f32_to_double(a[e]);
                } else {
                    FixedSum a[4];
                    int h[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) a[e] = FixedSum{0, 0};
#pragma unroll 1
                    for (int r = 0; r < nvec; r += kFixedRun) {
                        const int end = min(nvec, r + kFixedRun);
#pragma unroll
                        for (int e = 0; e < 4; ++e) h[e] = 0;
#pragma unroll 2
                        for (int t = r; t < end; ++t) {
                            const int2 ct = fixed_of(c[t], wbias);
                            const int *q = plane(t) + i;
                            const int4 v = ld4(q), u = ld4(q + C.ld);
                            fixed_step(a[0], h[0], v.x, u.x, ct.x, ct.y);
                            fixed_step(a[1], h[1], v.y, u.y, ct.x, ct.y);
                            fixed_step(a[2], h[2], v.z, u.z, ct.x, ct.y);
                            fixed_step(a[3], h[3], v.w, u.w, ct.x, ct.y);
                        }
#pragma unroll
                        for (int e = 0; e < 4; ++e) a[e] = fixed_carry(a[e], h[e]);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[e] -= fixed_value(a[e], wbias);
                }
                st2(w + i, x[0], x[1]);
                st2(w + i + 2, x[2], x[3]);
            }
            // the scalars' parts, a loop of its own (the thread's same poles): registers
            double pn = 0.0, sa = 0.0, m_[8], g_[8];
            float se = 0.0f;
#pragma unroll
            for (int q = 0; q < 8; ++q) { m_[q] = 0.0; g_[q] = 0.0; }
            for (int i = 4 * tid; i < S; i += 4 * T) {
                double2 e[2], m0[2];   // (more of the couplings ahead would spill)
#pragma unroll
                for (int h = 0; h < 2; ++h) { e[h] = energy2(i + 2 * h); m0[h] = coupling2(0, i + 2 * h); }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double2 x = ld2(w + i + 2 * h);
                    const double t0 = e[h].x * x.x, t1 = e[h].y * x.y;
                    pn = fma(x.y, x.y, fma(x.x, x.x, pn));
                    sa = fma(t1, x.y, fma(t0, x.x, sa));
                    const float f0 = f32_trunc(t0), f1 = f32_trunc(t1);   // |E w|^2 is a threshold's scale
                    se = fmaf(f1, f1, fmaf(f0, f0, se));
#pragma unroll
                    for (int d = 0; d < 8; ++d)
                        if (d < C.D) {
                            const double2 m = d == 0 ? m0[h] : coupling2(d, i + 2 * h);
                            m_[d] = fma(m.y, x.y, fma(m.x, x.x, m_[d]));
                        }
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q < nq && lslot[q] >= 0) {
                            const double2 v = vec2(lslot[q], q, i + 2 * h);
                            g_[q] = fma(v.y, t1, fma(v.x, t0, g_[q]));
                        }
                }
            }
            {   // the warp's sums: values 0 |w|^2, 1 alpha, 2 + d m_d, 2 + D + q g_q, eight or all at a time;
                // |E w|^2 in FP32
                const int nv = 2 + C.D + nq;
                auto addd = [](double p, double q) { return p + q; };
                auto shfd = [](double p, int o) { return __shfl_xor_sync(0xffffffffu, p, o); };
                double v[18];
                v[0] = pn; v[1] = sa;
#pragma unroll
                for (int q = 2; q < 18; ++q) {   // (registers: every index known)
                    double x = 0.0;
#pragma unroll
                    for (int d = 0; d < 8; ++d) if (q == 2 + d && d < C.D) x = m_[d];
#pragma unroll
                    for (int h = 0; h < 8; ++h) if (q - 2 - C.D == h && h < nq) x = g_[h];
                    v[q] = x;
                }
                if (nv <= 8) {
                    const double r = warp_sums_of<8>(v, lane, addd, shfd);   // lane L: value L / 4
                    if ((lane & 3) == 0) red[warp * kMaxSc + (lane >> 2)] = r;
                } else {
                    if (nv > 16) {
                        const double r = warp_sums_of<2>(v + 16, lane, addd, shfd);
                        if ((lane & 15) == 0) red[warp * kMaxSc + 16 + (lane >> 4)] = r;
                    }
                    const double r = warp_sums_of<16>(v, lane, addd, shfd);   // lane L: value L / 2
                    if ((lane & 1) == 0) red[warp * kMaxSc + (lane >> 1)] = r;
                }
                for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
                if (lane == 0) red[warp * kMaxSc + kMaxSc - 1] = (double)se;
                __syncthreads();
                double *Sp = sp + (size_t)spar * kMaxSc;
                spar ^= 1;
                // slot by slot, sixteen lanes over the warps' partials, then over the CTAs: the FP64
                // additions of a tree are its latency, and a lane alone would add them one by one
                const int slot = tid >> 4, sl = slot < nv ? slot : kMaxSc - 1, sub = tid & 15;
                if (2 * warp <= nv) {   // whole warps (two slots each; one beyond nv repeats the last)
                    double x = red[sub * kMaxSc + sl];
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                    if (sub == 0 && slot <= nv) Sp[sl] = x;
                }
                cluster.sync();
                if (2 * warp <= nv) {
                    double x = sub < CL ? cluster.map_shared_rank(Sp, sub)[sl] : 0.0;
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                    if (sub == 0 && slot <= nv) s_tot[sl] = (sl >= 2 + C.D && sl < nv && lslot[sl - 2 - C.D] < 0) ? 0.0 : x;
                }
                __syncthreads();
                // k_lanczos's decision, by warp 0 of every CTA alike (an FP64 instruction of all the
                // CTA's warps would hold the FP64 units for hundreds of cycles; here its lanes take
                // one threshold each)
                if (warp == 0) {
                    const double x2 = s_tot[0];
                    const double lim = lane == 0 ? eta2 * wn2 : (lane == 1 ? thr_exh : lane == 2 ? tau : kFixedShort) * wn2_first;
                    const unsigned lt_ = __ballot_sync(0xffffffffu, x2 < lim), le = __ballot_sync(0xffffffffu, x2 <= lim);
                    const long long xb = __double_as_longlong(x2);
                    const bool zero = (xb << 1) == 0, fin = (xb & 0x7ff0000000000000LL) != 0x7ff0000000000000LL;
                    int f;
                    if (!zero && wn2_first < kFixedWeak) f = 3;   // split against a scale FP32 lost
                    else if ((le & 2u) || zero) f = (dcur < dtot) ? 2 : 3;   // (further sweeps leave no more)
                    else if (nvec > 0 && nfull + 1 < 4 && (lt_ & 1u)) f = 1;
                    else if (nvec > 0 && nfull == 0 && (lt_ & 8u)) f = 4;
                    else if (!(le & 4u) && fin) f = 0;
                    else f = 3;
                    const double r = rsqrt_cubic(x2);
                    const double y = (lane == 0 ? 1.0 : lane == 1 ? x2 : s_tot[kMaxSc - 1] * r) * r;
                    if (lane < 3) s_n[lane] = y;   // 1/|w|, |w|, |E v|^2
                    if (lane == 0) s_fl = f;
                }
                __syncthreads();
            }
            fl = s_fl;
            if (nfull++ > 0 && !rough) ++extra;
            rough = fl == 4;
            if (fl != 1 && fl != 4) break;
            wn2 = s_tot[0];   // another sweep, of the updated w
            wbias = bias_above(wn2);
            for (int i = 4 * tid; i < S; i += 4 * T)
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const double2 x = ld2(w + i + e);
                    split_w(i + e, x.x, x.y);
                }
        }
        if (fl == 3) { ok = false; break; }
        if (fl == 2) {
            // exhausted: the rest of this pivot chain takes unreached directions
            const int jend = (k + 1 < C.n_used) ? min(C.L, s_start[k + 1]) : C.L;
            const int nr = jend - j, NT = C.nden_out + C.D;
            for (int r = tid; r < nr; r += T) {
                const int d = dcur + r;
                if (rank == 0) {
                    double *row = C.out + (size_t)(j + r) * NT;
                    for (int e = 0; e < NT; ++e) row[e] = 0.0;
                    row[0] = (d < dtot) ? C.gE[group_of(d)] : C.gE[Qg - 1];
                }
                rowslot[j + r] = -1;
            }
            dcur = min(dcur + nr, dtot);
            ndefl += nr;
            j = jend - 1;
            __syncthreads();
            continue;
        }
        // normalise and store; the row
        const double ixb = s_n[0];
        {
            int *q = plane(nvec), *qb = q + C.ld;
            double *rg = ring + (size_t)(nvec & 1) * S;
            double *rl = (j == s_last[k] && k < s_nl) ? sm + s_oL + k * S : nullptr;
            for (int i = 4 * tid; i < S; i += 4 * T) {
                int4 a, b;
                const double2 x = ld2(w + i), y = ld2(w + i + 2);
                const double v0 = x.x * ixb, v1 = x.y * ixb, v2 = y.x * ixb, v3 = y.y * ixb;
                st2(rg + i, v0, v1);
                st2(rg + i + 2, v2, v3);
                if (rl) { st2(rl + i, v0, v1); st2(rl + i + 2, v2, v3); }
                int2 f = fixed_of(v0, 1023); a.x = f.x; b.x = f.y;
                f = fixed_of(v1, 1023); a.y = f.x; b.y = f.y;
                f = fixed_of(v2, 1023); a.z = f.x; b.z = f.y;
                f = fixed_of(v3, 1023); a.w = f.x; b.w = f.y;
                *reinterpret_cast<int4 *>(q + i) = a;
                *reinterpret_cast<int4 *>(qb + i) = b;
            }
        }
        e2v = s_n[2];
        if (tid < C.nden_out + C.D) {
            const int NT = C.nden_out + C.D;
            double x = 0.0;
            if (tid == 0) x = s_tot[1] * ixb * ixb;
            else if (tid == 1) x = (newv && k >= 1) ? s_tot[2 + C.D + (k - 1)] * ixb : s_n[1];
            else if (tid < 2 + k) x = s_tot[2 + C.D + (tid - 2)] * ixb;
            else if (tid >= C.nden_out && tid < C.nden_out + C.D) x = s_tot[2 + (tid - C.nden_out)] * ixb;
            s_row[tid] = x;
            if (rank == 0) C.out[(size_t)j * NT + tid] = x;
        }
        // the next step's recurrence, listed by the warp that holds the row
        if (warp == 0) {
            __syncwarp();
            if (lane == 0) {
                rowslot[j] = nvec;
                int n = 0;
                lt[n] = nvec; lq[n] = -1; lc[n++] = s_row[0];
                if (j >= 1 && rowslot[j - 1] >= 0) { lt[n] = rowslot[j - 1]; lq[n] = -1; lc[n++] = s_row[1]; }
                for (int q = 0; q < k; ++q)
                    if (s_last[q] < j - 1 && rowslot[s_last[q]] >= 0) { lt[n] = rowslot[s_last[q]]; lq[n] = q; lc[n++] = s_row[2 + q]; }
                lt[15] = n;
            }
        }
        ++nvec;
        __syncthreads();
        nl0 = lt[15];
    }
    if (rank == 0 && ok) {
        if (C.rowslot)
            for (int q = tid; q < C.L; q += T) C.rowslot[q] = rowslot[q];
        if (tid == 0) {
            atomicAdd(&C.stat[0], extra);
            atomicAdd(&C.stat[2], ndefl);
            *C.done = 2;
        }
    }
    cluster.sync();   // no CTA leaves while peers may still read its shared memory
}

namespace {
constexpr size_t kLongSmem = (size_t)225 * 1024;
template <bool SS>
cudaError_t launch_form(const LzChain *d_chains, int nchains, int rmax, int nmin, int cluster, double eta, cudaStream_t st) {
    if (SS) cluster = long_cluster(cluster);
    cudaError_t e = allow_dynamic_smem((const void *)k_lz_long<SS>);
    if (e == cudaSuccess && cluster > 8) e = cudaFuncSetAttribute(k_lz_long<SS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nchains * cluster, 1, 1);
    cfg.blockDim = dim3(kLongThreads, 1, 1);
    cfg.dynamicSmemBytes = kLongSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_lz_long<SS>, d_chains, nchains, rmax, nmin, eta * eta, (int)kLongSmem);
}
}  // namespace

int lanczos_long_form(int N, int rmax, int cluster) {
    return long_fixed(rmax) > kLongSmem ? 0 : long_fits(N, cluster, rmax, kLongSmem) ? 1 : 2;
}

cudaError_t launch_lanczos_long(const LzChain *d_chains, int nchains, int rmax, int nmin, int cluster, double eta, int forms,
                                cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    if (forms & 1) e = launch_form<true>(d_chains, nchains, rmax, nmin, cluster, eta, st);
    if (e == cudaSuccess && (forms & 2)) e = launch_form<false>(d_chains, nchains, rmax, nmin, cluster, eta, st);
    return e;
}

void lanczos_long_smem_init() {
    allow_dynamic_smem((const void *)k_lz_long<true>);
    allow_dynamic_smem((const void *)k_lz_long<false>);
}

}  // namespace bd
