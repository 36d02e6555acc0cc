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
//     multiply-adds an element, exact sums (they are bounded by |v| |w|) on the integer pipe: c_t
//     is off by about 2^-57 |w|, where FP64's own sum is off by 1e-16 |w|;
//   - the update w -= sum c_t v_t runs in FP32 from the a planes alone (4 bytes a pole) where
//     every |c_t| <= kSmall |w|, which after a recurrence is the rule: its error is below 2^-23
//     kSmall sqrt(R) |w|.  Otherwise (new pivots, further sweeps) it is fixed point too.
// The recurrence, the norm, alpha, m and g stay FP64 with as few instructions as they take.
//
// What a chain needs beyond that -- a restart vector, energies or couplings outside 2^+-40,
// fewer than kLzLong poles -- is left to k_lanczos as a whole (C.done stays 0), which the
// host launches behind this kernel.
//
// Work split: a cluster per chain, CTA r the pole rows [r S, (r+1) S), 512 threads and an SM to
// itself; a warp per vector in the dot products, a thread per four poles everywhere else.  A
// step is two cluster reductions.
// Bound by the planes' traffic and the phases around it in batches (12 bytes a stored element
// and step: 2.1 M poles in 52 chains, 20 iterations a pivot, 18.3 -> 10.4 ms against 3.2 at the
// copy bandwidth) and by the chain of phases for one chain on its 16 SMs (20 000 poles, 80
// vectors: the call 5.36 -> 2.36 ms).  The same kernel with FP64 dot products took 17.1 and
// 4.2 ms, with double-float ones formed from the doubles' bits 12.5 and 3.1 (off by 2e-15 |w|
// where this is off by 5e-16, as FP64 is).
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

// shared memory before the slices: A[2][rq] partials, c[rq], sp[2][kMaxSc], red[16][kMaxSc] (doubles),
// cf[rq] (floats), rowslot[lq] (ints)
__host__ __device__ inline size_t long_fixed(int rmax) {
    const size_t rq = ((size_t)rmax + 4) & ~(size_t)3;
    return sizeof(double) * (3 * rq + 2 * kMaxSc + kMaxWarps * kMaxSc) + 8 * rq;
}

}  // namespace

__global__ void __launch_bounds__(kLongThreads, 1) k_lz_long(const LzChain *chains, int nchains, int rmax, double eta2,
                                                    int smem_bytes) {
    cg::cluster_group cluster = cg::this_cluster();
    const int CL = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int cid = blockIdx.x / CL;
    if (cid >= nchains) return;
    const LzChain C = chains[cid];
    if (!C.done || *C.done || C.N < kLzLong) return;   // (the whole cluster leaves together)
    const int N = C.N, D = C.D, L = C.L, NT = C.nden_out + C.D, S = C.S, i0 = rank * S;
    const int ns = max(0, min(N, i0 + S) - i0);
    constexpr int T = kLongThreads, NW = kMaxWarps;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    extern __shared__ double sm[];
    const int rq = (rmax + 4) & ~3;
    double *A = sm, *c = A + 2 * rq, *sp = c + rq, *red = sp + 2 * kMaxSc;
    float *cf = reinterpret_cast<float *>(red + kMaxWarps * kMaxSc);
    int *rowslot = reinterpret_cast<int *>(cf + rq);
    char *free_ = reinterpret_cast<char *>(sm) + long_fixed(rmax);
    char *const end = reinterpret_cast<char *>(sm) + smem_bytes;
    // slices: w, its split (two planes) and the two newest vectors in shared memory, or in the
    // chain's global scratch; E and M beside them when they fit; then the first vectors' planes,
    // as many as fit
    double *w, *ring;
    int *ws;
    const size_t sb = sizeof(double) * (size_t)S;
    if ((size_t)(end - free_) >= 4 * sb) {
        w = reinterpret_cast<double *>(free_);
        free_ += 4 * sb;
    } else {
        w = reinterpret_cast<double *>(C.slice + (size_t)rank * C.slice_stride);
    }
    ring = w + S;
    ws = reinterpret_cast<int *>(w + 3 * (size_t)S);
    double *Es = nullptr, *Ms = nullptr;
    if ((size_t)(end - free_) >= sb) { Es = reinterpret_cast<double *>(free_); free_ += sb; }
    if ((size_t)(end - free_) >= D * sb) { Ms = reinterpret_cast<double *>(free_); free_ += D * sb; }
    // the earlier chains' last vectors as doubles (the recurrence and the g read them), the rest planes
    int nlast = min(max(C.n_used - 1, 0), (int)((size_t)(end - free_) / sb));
    double *lasts = reinterpret_cast<double *>(free_);
    free_ += nlast * sb;
    const int ccap = (int)((size_t)(end - free_) / sb);
    int *cache = reinterpret_cast<int *>(free_);
    __shared__ int s_start[10], s_last[10], lslot[8], lt[16], lq[16];
    __shared__ double lc[16], s_row[32], s_tot[kMaxSc];
    __shared__ double s_n[3];   // 1/|w|, |w|, |E v|^2 of the kept vector
    __shared__ int s_fl;        // 0 keep, 1 sweep again, 2 exhausted, 3 the full space's
    __shared__ unsigned s_rng[2];
    if (tid < 2) s_rng[tid] = 0;
    if (tid <= C.n_used && tid < 10) s_start[tid] = C.start[tid];
    if (tid < C.n_used && tid < 10) s_last[tid] = C.last[tid];
    __syncthreads();
    {   // energies and couplings inside 2^+-40 (the largest of each): FP32's exponents hold all that follows
        unsigned me = 0, mm = 0;
        for (int i = tid; i < S; i += T) {
            const bool in = i < ns;
            const double e = in ? C.E[i0 + i] : 0.0;
            if (Es) Es[i] = e;
            me = max(me, (unsigned)__double2hiint(e) & 0x7fffffffu);
            for (int d = 0; d < D; ++d) {
                const double m = in ? C.M[(size_t)d * N + i0 + i] : 0.0;
                if (Ms) Ms[(size_t)d * S + i] = m;
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
    int nvec = 0;
    // planes of stored vector t: a at the address, b pl(t) behind it
    int *Vg = reinterpret_cast<int *>(C.V) + i0;
    auto plane = [&](int t) -> int * { return t < ccap ? cache + 2 * (size_t)t * S : Vg + 2 * (size_t)t * C.ld; };
    auto pl = [&](int t) -> int { return t < ccap ? S : C.ld; };
    // elements i, i + 1 of vector t as doubles (q: the chain it is the last vector of, or -1)
    auto vec2 = [&](int t, int q, int i) -> double2 {
        if (t >= nvec - 2) return ld2(ring + (size_t)(t & 1) * S + i);
        if (q >= 0 && q < nlast) return ld2(lasts + (size_t)q * S + i);
        const int *p = plane(t) + i;
        const int2 x = *reinterpret_cast<const int2 *>(p), y = *reinterpret_cast<const int2 *>(p + pl(t));
        return make_double2(fixed_to_double(x.x, y.x), fixed_to_double(x.y, y.y));
    };
    auto energy2 = [&](int i) -> double2 {   // of poles i, i + 1 of the slice
        if (Es) return ld2(Es + i);
        return make_double2(i < ns ? C.E[i0 + i] : 0.0, i + 1 < ns ? C.E[i0 + i + 1] : 0.0);
    };
    auto coupling2 = [&](int d, int i) -> double2 {
        if (Ms) return ld2(Ms + (size_t)d * S + i);
        const double *p = C.M + (size_t)d * N + i0 + i;
        return make_double2(i < ns ? p[0] : 0.0, i + 1 < ns ? p[1] : 0.0);
    };
    int wbias = 1023;   // exponent field of the power of two w is split against
    auto split_w = [&](int i, double a, double b) {
        const int2 x = fixed_of(a, wbias), y = fixed_of(b, wbias);
        *reinterpret_cast<int2 *>(ws + i) = make_int2(x.x, y.x);
        *reinterpret_cast<int2 *>(ws + S + i) = make_int2(x.y, y.y);
    };
    auto csum = [&](const double *buf, int t) -> double {   // over the cluster, a fixed tree
        double x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) x[r] = (r < CL) ? cluster.map_shared_rank(const_cast<double *>(buf), r)[t] : 0.0;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < o; ++r) x[r] += x[r + o];
        return x[0];
    };
    const int Qg = C.gE ? C.gInfo[0] : 0;
    const int dtot = Qg > 0 ? C.gInfo[Qg] : 0;
    auto group_of = [&](int d) {
        int lo = 0, hi = Qg - 1;
        while (lo < hi) { const int mid = (lo + hi) >> 1; if (C.gInfo[1 + mid] > d) hi = mid; else lo = mid + 1; }
        return lo;
    };
    constexpr double tau = 1e-48, thr_exh = 1e-20;   // k_lanczos's, FP64 vectors
    int dcur = 0, ndefl = 0, extra = 0, k = -1, dpar = 0, spar = 0, nl0 = 0;
    double e2v = 0.0;
    bool ok = true;
    for (int j = 0; j < L; ++j) {
        const bool newv = (k + 1 < C.n_used) && (j == s_start[k + 1]);
        if (newv) ++k;
        const int nq = k;
        if (tid < nq) lslot[tid] = rowslot[s_last[tid]];
        // w = M p, or E v_{j-1} less its known components
        double wn2 = 0.0, wn2_first = e2v;   // |w|^2 before the sweep, and of E v_{j-1} / M p (thresholds' scales)
        if (newv) {
            double p[8];
#pragma unroll
            for (int d = 0; d < 8; ++d) p[d] = d < D ? C.piv[(size_t)k * D + d] : 0.0;
            float s2 = 0.0f;
            for (int i = 2 * tid; i < S; i += 2 * T) {
                double a = 0.0, b = 0.0;
#pragma unroll
                for (int d = 0; d < 8; ++d)
                    if (d < D) {
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
            if (tid == 0) s_n[0] = csum(sp + (size_t)spar * kMaxSc, 0);
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
            for (int i = 2 * tid; i < S; i += 2 * T) {
                const double2 e = energy2(i), x = ld2(v0 + i);
                double a = x.x * e.x, b = x.y * e.y;
#pragma unroll 4
                for (int t = 0; t < nl0; ++t) {
                    const double2 y = vec2(lt[t], lq[t], i);
                    const double ct = lc[t];
                    a = fma(-ct, y.x, a);
                    b = fma(-ct, y.y, b);
                }
                st2(w + i, a, b);
                split_w(i, a, b);
            }
        }
        int fl, nfull = 0;
        for (;;) {
            __syncthreads();
            // c_t = <v_t, w> for every stored vector, a warp each, four at a time; after a
            // recurrence also |w|^2 as item nvec (read against the swept norm and the
            // coefficients only: FP32)
            double *Ap = A + (size_t)dpar * rq;
            dpar ^= 1;
            const bool want_n = !newv && nfull == 0;
            const int items = nvec + (want_n ? 1 : 0);
            constexpr int NU = 4;
            for (int t0 = warp; t0 < items; t0 += NU * NW) {
                const int nu = min(NU, (nvec - 1 - t0 + NW) / NW);   // stored vectors t0, t0 + NW, ..
                if (nu > 0) {
                    const int *va[NU], *vb[NU];
#pragma unroll
                    for (int u = 0; u < NU; ++u) {
                        const int t = min(t0 + u * NW, nvec - 1);
                        va[u] = plane(t);
                        vb[u] = va[u] + pl(t);
                    }
                    FixedSum acc[NU];
#pragma unroll
                    for (int u = 0; u < NU; ++u) acc[u] = FixedSum{0, 0};
                    for (int i = 4 * lane; i < S; i += 128) {
                        int4 x[NU], y[NU];
#pragma unroll
                        for (int u = 0; u < NU; ++u) if (u < nu) { x[u] = ld4(va[u] + i); y[u] = ld4(vb[u] + i); }
                        const int4 a = ld4(ws + i), b = ld4(ws + S + i);
#pragma unroll
                        for (int u = 0; u < NU; ++u)
                            if (u < nu) {
                                fixed_step(acc[u], x[u].x, y[u].x, a.x, b.x);
                                fixed_step(acc[u], x[u].y, y[u].y, a.y, b.y);
                                fixed_step(acc[u], x[u].z, y[u].z, a.z, b.z);
                                fixed_step(acc[u], x[u].w, y[u].w, a.w, b.w);
                            }
                    }
                    const FixedSum r = warp_sums_of<NU>(acc, lane, fixed_add, fixed_shfl);
                    const int u = lane >> 3;
                    if ((lane & 7) == 0 && u < nu) Ap[t0 + u * NW] = fixed_value(r, wbias);
                }
                if (want_n && (nvec - t0) % NW == 0 && nvec >= t0 && nvec < t0 + NU * NW) {
                    float x2 = 0.0f;
                    for (int i = 2 * lane; i < S; i += 64) {
                        const double2 x = ld2(w + i);
                        const float a = f32_trunc(x.x), b = f32_trunc(x.y);
                        x2 = fmaf(b, b, fmaf(a, a, x2));
                    }
                    for (int o = 16; o > 0; o >>= 1) x2 += __shfl_xor_sync(0xffffffffu, x2, o);
                    if (lane == 0) Ap[nvec] = (double)x2;
                }
            }
            cluster.sync();
            for (int t = tid; t < items; t += T) {
                const double x = csum(Ap, t);
                c[t] = x;
                cf[t] = t < nvec ? f32_trunc(x) * 0x1p-30f : f32_trunc(x);   // (against the a planes)
            }
            __syncthreads();
            if (want_n) wn2 = c[nvec];
            // the update and, of the updated w, this thread's part of the scalars
            float cm = 0.0f;
            for (int t = lane; t < nvec; t += 32) cm = fmaxf(cm, fabsf(cf[t]));
            for (int o = 16; o > 0; o >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
            const bool small = want_n && cm * 0x1p30f <= kSmall * sqrtf(cf[nvec]);
            double pn = 0.0, sa = 0.0, m_[8], g_[8];
            float se = 0.0f;
#pragma unroll
            for (int q = 0; q < 8; ++q) { m_[q] = 0.0; g_[q] = 0.0; }
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
                    int t = 0;
                    const int tc = min(ccap, nvec);
                    for (; t < tc; ++t) step(cf[t], ld4(cache + 2 * (size_t)t * S + i));
                    for (; t + 7 < nvec; t += 8) {
                        int4 v[8];
#pragma unroll
                        for (int r = 0; r < 8; ++r) v[r] = ld4(Vg + 2 * (size_t)(t + r) * C.ld + i);
#pragma unroll
                        for (int r = 0; r < 8; ++r) step(cf[t + r], v[r]);
                    }
                    for (; t < nvec; ++t) step(cf[t], ld4(Vg + 2 * (size_t)t * C.ld + i));
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[e] -= (double)a[e];
                } else {
                    FixedSum a[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) a[e] = FixedSum{0, 0};
#pragma unroll 2
                    for (int t = 0; t < nvec; ++t) {
                        const int2 ct = fixed_of(c[t], wbias);
                        const int *q = plane(t) + i;
                        const int4 v = ld4(q), u = ld4(q + pl(t));
                        fixed_step(a[0], v.x, u.x, ct.x, ct.y);
                        fixed_step(a[1], v.y, u.y, ct.x, ct.y);
                        fixed_step(a[2], v.z, u.z, ct.x, ct.y);
                        fixed_step(a[3], v.w, u.w, ct.x, ct.y);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) x[e] -= fixed_value(a[e], wbias);
                }
                st2(w + i, x[0], x[1]);
                st2(w + i + 2, x[2], x[3]);
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const double2 ee = energy2(i + e);
                    const double t0 = ee.x * x[e], t1 = ee.y * x[e + 1];
                    pn = fma(x[e + 1], x[e + 1], fma(x[e], x[e], pn));
                    sa = fma(t1, x[e + 1], fma(t0, x[e], sa));
                    const float f0 = f32_trunc(t0), f1 = f32_trunc(t1);   // |E w|^2 is a threshold's scale
                    se = fmaf(f1, f1, fmaf(f0, f0, se));
#pragma unroll
                    for (int d = 0; d < 8; ++d)
                        if (d < D) {
                            const double2 m = coupling2(d, i + e);
                            m_[d] = fma(m.y, x[e + 1], fma(m.x, x[e], m_[d]));
                        }
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (q < nq && lslot[q] >= 0) {
                            const double2 v = vec2(lslot[q], q, i + e);
                            g_[q] = fma(v.y, t1, fma(v.x, t0, g_[q]));
                        }
                }
            }
            {   // the warp's sums: values 0 |w|^2, 1 alpha, 2 + d m_d, 2 + D + q g_q, eight or all at a time;
                // |E w|^2 in FP32
                const int nv = 2 + D + nq;
                auto addd = [](double p, double q) { return p + q; };
                auto shfd = [](double p, int o) { return __shfl_xor_sync(0xffffffffu, p, o); };
                double v[18];
                v[0] = pn; v[1] = sa;
#pragma unroll
                for (int q = 2; q < 18; ++q) {   // (registers: every index known)
                    double x = 0.0;
#pragma unroll
                    for (int d = 0; d < 8; ++d) if (q == 2 + d && d < D) x = m_[d];
#pragma unroll
                    for (int h = 0; h < 8; ++h) if (q - 2 - D == h && h < nq) x = g_[h];
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
                    if (sub == 0 && slot <= nv) s_tot[sl] = (sl >= 2 + D && sl < nv && lslot[sl - 2 - D] < 0) ? 0.0 : x;
                }
                __syncthreads();
                // k_lanczos's decision, by warp 0 of every CTA alike (an FP64 instruction of all the
                // CTA's warps would hold the FP64 units for hundreds of cycles; here its lanes take
                // one threshold each)
                if (warp == 0) {
                    const double x2 = s_tot[0];
                    const double lim = lane == 0 ? eta2 * wn2 : (lane == 1 ? thr_exh : tau) * wn2_first;
                    const unsigned lt_ = __ballot_sync(0xffffffffu, x2 < lim), le = __ballot_sync(0xffffffffu, x2 <= lim);
                    const long long xb = __double_as_longlong(x2);
                    const bool zero = (xb << 1) == 0, fin = (xb & 0x7ff0000000000000LL) != 0x7ff0000000000000LL;
                    int f;
                    if ((le & 2u) || zero) f = (dcur < dtot) ? 2 : 3;   // (further sweeps leave no more)
                    else if (nvec > 0 && nfull + 1 < 4 && (lt_ & 1u)) f = 1;
                    else if (!(le & 4u) && fin) f = 0;
                    else f = 3;
                    const double r = rsqrt_newton(x2);
                    const double y = (lane == 0 ? 1.0 : lane == 1 ? x2 : s_tot[kMaxSc - 1] * r) * r;
                    if (lane < 3) s_n[lane] = y;   // 1/|w|, |w|, |E v|^2
                    if (lane == 0) s_fl = f;
                }
                __syncthreads();
            }
            fl = s_fl;
            if (nfull++ > 0) ++extra;
            if (fl != 1) break;
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
            const int jend = (k + 1 < C.n_used) ? min(L, s_start[k + 1]) : L;
            const int nr = jend - j;
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
            int *q = plane(nvec), *qb = q + pl(nvec);
            double *rg = ring + (size_t)(nvec & 1) * S;
            double *rl = (j == s_last[k] && k < nlast) ? lasts + (size_t)k * S : nullptr;
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
                if (nvec < ccap) {   // (the host reads the basis back from V)
                    *reinterpret_cast<int4 *>(Vg + 2 * (size_t)nvec * C.ld + i) = a;
                    *reinterpret_cast<int4 *>(Vg + 2 * (size_t)nvec * C.ld + C.ld + i) = b;
                }
            }
        }
        e2v = s_n[2];
        if (tid < NT) {
            double x = 0.0;
            if (tid == 0) x = s_tot[1] * ixb * ixb;
            else if (tid == 1) x = (newv && k >= 1) ? s_tot[2 + D + (k - 1)] * ixb : s_n[1];
            else if (tid < 2 + k) x = s_tot[2 + D + (tid - 2)] * ixb;
            else if (tid >= C.nden_out && tid < C.nden_out + D) x = s_tot[2 + (tid - C.nden_out)] * ixb;
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
            for (int q = tid; q < L; q += T) C.rowslot[q] = rowslot[q];
        if (tid == 0) {
            atomicAdd(&C.stat[0], extra);
            atomicAdd(&C.stat[2], ndefl);
            *C.done = 2;
        }
    }
    cluster.sync();   // no CTA leaves while peers may still read its shared memory
}

size_t lanczos_long_smem(int S, int rmax, bool have_slices) {
    const size_t cap = (size_t)216 * 1024, fixed = long_fixed(rmax);
    return fixed + (have_slices ? 0 : 32 * (size_t)S) <= cap ? cap : 0;
}

cudaError_t launch_lanczos_long(const LzChain *d_chains, int nchains, int rmax, int cluster, double eta, size_t smem,
                                cudaStream_t st) {
    if (nchains <= 0 || smem == 0) return cudaSuccess;
    cudaError_t e = allow_dynamic_smem((const void *)k_lz_long);
    if (e == cudaSuccess && cluster > 8) e = cudaFuncSetAttribute(k_lz_long, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nchains * cluster, 1, 1);
    cfg.blockDim = dim3(kLongThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_lz_long, d_chains, nchains, rmax, eta * eta, (int)smem);
}

void lanczos_long_smem_init() { allow_dynamic_smem((const void *)k_lz_long); }

}  // namespace bd
