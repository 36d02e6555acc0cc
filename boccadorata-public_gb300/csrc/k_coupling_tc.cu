// k_coupling_tc.cu -- the 2p1h / 2h1p couplings M of the second-order self-energy on
// the tensor cores, for the mixed-precision form on a dressed propagator.
//
// Restates the contraction of Build_Dynamic_SlfEn_2ndOrder
// (source/BcDor-Self_energy_ext_Op_c.cpp:425-481 forward, :484-539 backward), which
// k_poles (k_sigma2.cu) keeps in the reference's FP64 order for the plain form.  For a
// block (I, Jab, ia, ib, ig) and a pole t = (na, nb, ng) of fragments,
//   M[d][t] = x4(t) sum_{p = (alpha, beta), gamma} V'[d][p][gamma] x2(p; na, nb) f_ng[gamma],
// a GEMM of the block's V' (rows d, columns (p, gamma)) with the matrix
// B[(p, gamma)][t] = x4(t) x2(p; t) f_ng[gamma].  B depends on (ia, ib, ig, nJab) and the
// propagator only, so the blocks of every channel that share those are stacked into one
// operand of 128 rows (their D rows each): one tile is one 128 x N x K product, N the
// block's poles padded to 16, K = pairs x orbitals of ig.
//
// Each tile, both directions at once (the forward poles' columns, then the backward ones':
// they share A): a CTA of four warps stages A (V') and B in shared memory in the canonical
// no-swizzle K-major layout (8-row x 16-byte core matrices), 16 K columns at a time; every
// value is split into two TF32 parts, hi + lo, and thread 0 issues three tcgen05.mma
// (kind::tf32, M = 128) per 8 columns, hi*hi + hi*lo + lo*hi, accumulating in FP32 in
// tensor memory (about 2^-21 relative per product, against the FP32 Lanczos vectors'
// 2^-24 rounding); their completion comes back through an mbarrier (tcgen05.commit).
// Then each warp reads its 32 rows from tensor memory (tcgen05.ld) and writes M, and the
// CTA forms the poles' energies (FP64, the reference's operations: the same bits as
// k_poles) and S2 = sum_d M^2.  Every FP64 -> FP32 conversion of the staging is done on
// the integer pipe (the double's bits truncated): the FP64 unit issues at 1/64 of FP32.
// A tile is a few dozen MMAs, so its time is the staging and the chains in front of it: a
// thread (two, four) per row with the row's address and the columns' offsets looked up once,
// the rows' table from a scan over the blocks, no row or column staged that nobody reads.
// Sigma(2) phase of a dressed step, N_max = 8, one fragment: 5.2 -> 1.0 ms (64 columns a round:
// 1.9, 32: 1.2); two fragments 5.7 -> 1.1; N_max = 4: 0.30 -> 0.09.
#include "bd_common.cuh"
#include "bd_kernels.h"

namespace bd {

namespace {

constexpr int kTcRows = 128;     // MMA M: rows of a tile
constexpr int kTcKc = 16;        // K columns staged per round (a tile is short: the rounds of eight CTAs an SM overlap)
constexpr int kTcThreads = 128;  // four warps: one per 32 lanes of tensor memory
constexpr int kTcKMax = 64 * 8;  // columns at most: 64 (alpha, beta) pairs, 8 orbitals

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor of tcgen05: start address, leading (K direction) and
// stride (8-row groups) byte offsets, all in 16-byte units; version 1, no swizzle.
__device__ __forceinline__ uint64_t mma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Element (r, k) of a K-major tile of kTcKc columns: [r / 8][k / 4][r % 8][k % 4] (floats).
__device__ __forceinline__ int tc_off(int r, int k) { return (((r >> 3) * (kTcKc / 4) + (k >> 2)) * 8 + (r & 7)) * 4 + (k & 3); }

// x truncated to FP32 from its bits (|x| inside the FP32 normal range, else 0 or the
// largest float): no FP64 instruction
__device__ __forceinline__ float f64_to_f32(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7FF) - 1023 + 127;
    const unsigned s = (unsigned)(b >> 63) << 31;
    if (e <= 0) return __uint_as_float(s);
    if (e >= 255) return __uint_as_float(s | 0x7F7FFFFFu);
    return __uint_as_float(s | ((unsigned)e << 23) | (unsigned)((b >> 29) & 0x7FFFFFu));
}

// FP32 to FP64 from the bits (exact; zero and normal values)
__device__ __forceinline__ double f32_to_f64(float x) {
    const unsigned u = __float_as_uint(x);
    const unsigned e = (u >> 23) & 0xFF;
    if (e == 0) return __longlong_as_double((long long)((unsigned long long)(u >> 31) << 63));
    return __longlong_as_double((long long)(((unsigned long long)(u >> 31) << 63) |
                                            ((unsigned long long)(e - 127 + 1023) << 52) |
                                            ((unsigned long long)(u & 0x7FFFFFu) << 29)));
}

__device__ __forceinline__ float tf32_rna(float x) {
    unsigned r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

// x = hi + lo, both TF32 (the rest is below 2^-21 |x|)
__device__ __forceinline__ void tf32_split(float x, float &hi, float &lo) {
    hi = tf32_rna(x);
    lo = tf32_rna(__fsub_rn(x, hi));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(bar)));
    asm volatile("fence.mbarrier_init.release.cluster;");
}

// wait for the completion of the given phase, at most `limit` polls (false: gave up)
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, int phase, int limit) {
    uint32_t done = 0;
    for (int it = 0; it < limit && !done; ++it)
        asm volatile("{\n .reg .pred q;\n mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n selp.u32 %0, 1, 0, q;\n}"
                     : "=r"(done) : "r"(smem_addr(bar)), "r"(phase));
    return done != 0;
}

// D (tensor memory) [+]= A B^T, both operands K-major in shared memory (descriptors)
__device__ __forceinline__ void tc_mma_tf32(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                 " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}"
                 :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// the MMAs issued so far by this thread arrive on the mbarrier when they complete
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_addr(bar)));
}

// sixteen 32-bit columns of this warp's 32 lanes of tensor memory
__device__ __forceinline__ void tc_ld16(uint32_t a, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(a));
    asm volatile("tcgen05.wait::ld.sync.aligned;");
}

// fragments (na, nb, ng) of pole t of a block, as k_poles enumerates them
__device__ __forceinline__ void pole_frags(const S2Block &B, int t, int nAa, int nAb, int nG, int &na, int &nb, int &ng) {
    ng = t % nG;
    int q = t / nG;
    if (B.ia == B.ib) {
        na = 0;
        while (na < nAa && q >= nAa - na - B.nJab) { q -= nAa - na - B.nJab; ++na; }
        nb = na + B.nJab + q;
    } else {
        na = q / nAb;
        nb = q % nAb;
    }
}

}  // namespace

__global__ void __launch_bounds__(kTcThreads) k_poles_tc(DevProblem P, const S2Block *blk, const int *tile_blk,
                                                         const int4 *tiles, int ntiles, const ChanSig *cs,
                                                         const double *vp, TcOut fw, TcOut bk, int dirs, int *err) {
    const int tile = blockIdx.x;
    if (tile >= ntiles) return;
    const int4 T4 = tiles[tile];   // first entry in tile_blk, blocks, rows
    const int b_first = T4.x, nblk = T4.y, rows = T4.z;
    const S2Block B0 = blk[tile_blk[b_first]];
    // poles of each block of the tile, forward and backward (dirs: which of the two)
    const int Tn[2] = {(dirs & 1) ? B0.nfw : 0, (dirs & 2) ? B0.nbk : 0};
    if (Tn[0] <= 0 && Tn[1] <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int NS = P.nspb;
    const int ia = B0.ia, ib = B0.ib, ig = B0.ig;
    const int noa = P.no[ia], nob = P.no[ib], nog = P.no[ig];
    const int col0[2] = {0, (Tn[0] + 15) & ~15};   // first column of each direction
    const int Np = col0[1] + ((Tn[1] + 15) & ~15);

    extern __shared__ __align__(1024) unsigned char smc[];
    float *Ahi = reinterpret_cast<float *>(smc);           // [kTcRows][kTcKc] K-major core matrices
    float *Alo = Ahi + kTcRows * kTcKc;
    float *Bhi = Alo + kTcRows * kTcKc;                    // [Np][kTcKc]
    float *Blo = Bhi + Np * kTcKc;
    __shared__ __align__(16) int s_k[kTcKMax];                            // column k: offset in a row of V' | gamma << 16 | alpha << 20 | beta << 24, or -1
    __shared__ short s_rblk[kTcRows], s_rd[kTcRows];        // block (in the tile) and d of every row
    __shared__ int s_wsum[kTcThreads / 32];
    __shared__ uint32_t s_taddr;
    __shared__ __align__(8) uint64_t s_bar;

    const int npair = ia == ib ? noa * (noa + 1) / 2 - B0.nJab * noa : noa * nob;   // (alpha, beta), beta >= alpha + nJab for ia == ib
    const int K = npair * nog;
    const int ncols = Np <= 32 ? 32 : Np <= 64 ? 64 : Np <= 128 ? 128 : 256;
    if (tid == 0) mbar_init(&s_bar);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_addr(&s_taddr)), "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // the rows of the tile's blocks, a block each: their first rows by a scan over the blocks' D
    {
        const int Dq = tid < nblk ? P.no[blk[tile_blk[b_first + tid]].ch] : 0;
        int v = Dq;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane == 31) s_wsum[warp] = v;
        __syncthreads();
        int r = v - Dq;
        for (int w = 0; w < warp; ++w) r += s_wsum[w];
        for (int d = 0; d < Dq && r + d < kTcRows; ++d) { s_rblk[r + d] = (short)tid; s_rd[r + d] = (short)d; }
    }
    // the columns
    const int Kp = min((K + 7) & ~7, kTcKMax);
    for (int k = tid; k < Kp; k += kTcThreads) {
        int v = -1;
        if (k < K) {
            const int p = k / nog, gam = k - p * nog;
            int a, b;
            if (ia == ib) {
                int q = p;
                a = 0;
                while (q >= noa - a - B0.nJab) { q -= noa - a - B0.nJab; ++a; }
                b = a + B0.nJab + q;
            } else {
                a = p / nob;
                b = p - a * nob;
            }
            v = ((a * nob + b) * nog + gam) | gam << 16 | a << 20 | b << 24;
        }
        s_k[k] = v;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t taddr = s_taddr;
    const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(Np >> 3) << 17) |
                           ((uint32_t)(kTcRows >> 4) << 24);   // F32 += TF32 x TF32, K-major, M = 128, N = Np
    // A's staging: one, two or four threads per row, each with its row's V' and excluded gamma
    const int RP = rows <= 32 ? 32 : rows <= 64 ? 64 : 128, r_ = tid % RP, part = tid / RP, nparts = kTcThreads / RP;
    const double *vrow = nullptr;
    int excl = -1;
    if (r_ < rows) {
        const S2Block &Bb = blk[tile_blk[b_first + s_rblk[r_]]];
        const int d = s_rd[r_];
        vrow = vp + Bb.vp_first + (size_t)d * noa * nob * nog;
        if (Bb.nJgd) excl = P.orb_start[Bb.ch] + d - P.orb_start[ig];
    }
    bool ok = true;
    int phase = 0;
    for (int kc0 = 0; kc0 < K; kc0 += kTcKc) {
        const int kn = min(kTcKc, Kp - kc0);   // columns of this round, a multiple of 8
        // A: V' of every row's block at columns k = (p, gamma) (the reference's excluded
        // gamma == d terms as zeros), split into TF32 hi + lo, four columns at a time.  Rows
        // beyond the tile's stay as they are: they only reach accumulators nobody reads.
        if (r_ < rows)
            for (int kk = 4 * part; kk < kn; kk += 4 * nparts) {
                const int4 kv = *reinterpret_cast<const int4 *>(s_k + kc0 + kk);
                double x[4];
                const int ke[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) x[e] = (ke[e] >= 0 && ((ke[e] >> 16) & 15) != excl) ? __ldg(vrow + (ke[e] & 0xffff)) : 0.0;
                float hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) tf32_split(f64_to_f32(x[e]), hi[e], lo[e]);
                *reinterpret_cast<float4 *>(Ahi + tc_off(r_, kk)) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<float4 *>(Alo + tc_off(r_, kk)) = make_float4(lo[0], lo[1], lo[2], lo[3]);
            }
        // B: column t = pole (na, nb, ng) of a direction, row k = (p, gamma): x4 x2(p) f_ng[gamma]
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            const int T = Tn[dir];
            const int *nA = dir == 0 ? P.np : P.nh, *nGv = dir == 0 ? P.nh : P.np;
            const int *sA = dir == 0 ? P.p_start : P.h_start, *sG = dir == 0 ? P.h_start : P.p_start;
            const double *fA = dir == 0 ? P.fqp : P.fqh, *fG = dir == 0 ? P.fqh : P.fqp;
            const int kq = kn >> 2;
            for (int u = tid; u < T * kq; u += kTcThreads) {
                const int t = u / kq, kk = 4 * (u - t * kq);
                int na, nb, ng;
                pole_frags(B0, t, nA[ia], nA[ib], nGv[ig], na, nb, ng);
                const double *fa = fA + (size_t)(sA[ia] + na) * NS, *fb = fA + (size_t)(sA[ib] + nb) * NS;
                const double *fg = fG + (size_t)(sG[ig] + ng) * NS;
                float hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int kv = s_k[kc0 + kk + e];
                    float x = 0.0f;
                    if (kv >= 0) {
                        const int gam = (kv >> 16) & 15, a = (kv >> 20) & 15, b = (kv >> 24) & 15;
                        float x2 = f64_to_f32(__ldg(fa + a)) * f64_to_f32(__ldg(fb + b));
                        if (ia == ib) {
                            x2 += (B0.nJab ? -1.0f : 1.0f) * f64_to_f32(__ldg(fa + b)) * f64_to_f32(__ldg(fb + a));
                            if (a == b) x2 *= 0.70710678118654752f;
                            if (na == nb) x2 *= 0.70710678118654752f;
                        }
                        x = x2 * f64_to_f32(__ldg(fg + gam));
                    }
                    tf32_split(x, hi[e], lo[e]);
                }
                const int o = tc_off(col0[dir] + t, kk);
                *reinterpret_cast<float4 *>(Bhi + o) = make_float4(hi[0], hi[1], hi[2], hi[3]);
                *reinterpret_cast<float4 *>(Blo + o) = make_float4(lo[0], lo[1], lo[2], lo[3]);
            }
        }
        asm volatile("fence.proxy.async.shared::cta;");   // the staged tiles, to the tensor cores
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (tid == 0) {
            const int nstep = kn / 8;
            const uint32_t sbo = (kTcKc / 4) * 128;   // next 8-row group
            for (int s = 0; s < nstep; ++s) {
                const uint32_t off = (uint32_t)s * 256;   // two 128-byte core matrices of K per step
                const uint64_t ah = mma_desc(smem_addr(Ahi) + off, 128, sbo), al = mma_desc(smem_addr(Alo) + off, 128, sbo);
                const uint64_t bh = mma_desc(smem_addr(Bhi) + off, 128, sbo), bl = mma_desc(smem_addr(Blo) + off, 128, sbo);
                const uint32_t acc0 = (kc0 > 0 || s > 0) ? 1u : 0u;
                tc_mma_tf32(taddr, ah, bh, idesc, acc0);
                tc_mma_tf32(taddr, ah, bl, idesc, 1u);
                tc_mma_tf32(taddr, al, bh, idesc, 1u);
            }
            tc_commit(&s_bar);
        }
        // the products are done before the tiles are staged again (bounded wait; the CTA
        // agrees on the outcome, so it leaves the loop together)
        const bool done = mbar_wait(&s_bar, phase, 1 << 22);
        phase ^= 1;
        ok = __syncthreads_and(done) != 0 && ok;
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (!ok) break;
    }
    if (!ok && lane == 0) atomicExch(err, 1);
    // every row's accumulators: warp w reads lanes 32w .. 32w + 31, sixteen columns at a time
    const int r = 32 * warp + lane;
    const bool has_row = r < rows;
    const S2Block &Br = blk[tile_blk[b_first + (has_row ? s_rblk[r] : 0)]];
    const ChanSig Cr = cs[Br.ch];
    if (32 * warp < rows)
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            const int T = Tn[dir], Nr = dir == 0 ? Cr.nfw : Cr.nbk;
            double *Mrow = (dir == 0 ? fw.M : bk.M) + (dir == 0 ? Cr.mfw_off : Cr.mbk_off) + (size_t)(has_row ? s_rd[r] : 0) * Nr +
                           ((dir == 0 ? Br.fw_first : Br.bk_first) - (dir == 0 ? Cr.fw_off : Cr.bk_off));
            for (int c0 = 0; c0 < T; c0 += 16) {
                uint32_t v[16];
                if (ok && K > 0) {
                    tc_ld16(taddr + ((uint32_t)(32 * warp) << 16) + (uint32_t)(col0[dir] + c0), v);
                } else {
#pragma unroll
                    for (int q = 0; q < 16; ++q) v[q] = 0u;
                }
                if (has_row)
#pragma unroll
                    for (int q = 0; q < 16; ++q)
                        if (c0 + q < T) Mrow[c0 + q] = f32_to_f64(__uint_as_float(v[q]));
            }
        }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(taddr), "r"(ncols));
    // energies (the reference's FP64 operations) and S2 = sum_d M^2 of every pole of the tile
    __threadfence_block();
    for (int dir = 0; dir < 2; ++dir) {
        const int T = Tn[dir];
        const int *nA = dir == 0 ? P.np : P.nh, *nGv = dir == 0 ? P.nh : P.np;
        const int *sA = dir == 0 ? P.p_start : P.h_start, *sG = dir == 0 ? P.h_start : P.p_start;
        const double *eA = dir == 0 ? P.ep : P.eh, *eG = dir == 0 ? P.eh : P.ep;
        for (int u = tid; u < nblk * T; u += kTcThreads) {
            const int q = u / T, t = u - q * T;
            const S2Block &Bq = blk[tile_blk[b_first + q]];
            const ChanSig Cq = cs[Bq.ch];
            int na, nb, ng;
            pole_frags(B0, t, nA[ia], nA[ib], nGv[ig], na, nb, ng);
            const long long g = (dir == 0 ? Bq.fw_first : Bq.bk_first) + t;
            (dir == 0 ? fw.E : bk.E)[g] = __dsub_rn(__dadd_rn(eA[sA[ia] + na], eA[sA[ib] + nb]), eG[sG[ig] + ng]);
            const int Nq = dir == 0 ? Cq.nfw : Cq.nbk;
            const double *Mq = (dir == 0 ? fw.M : bk.M) + (dir == 0 ? Cq.mfw_off : Cq.mbk_off) + (g - (dir == 0 ? Cq.fw_off : Cq.bk_off));
            float s2 = 0.0f;
            for (int d = 0; d < Cq.D; ++d) { const float m = f64_to_f32(Mq[(size_t)d * Nq]); s2 = fmaf(m, m, s2); }
            (dir == 0 ? fw.S2 : bk.S2)[g] = f32_to_f64(s2);
        }
    }
}

}  // namespace bd

namespace bd {

size_t tc_smem_bytes(int np) {
    return sizeof(float) * ((size_t)2 * kTcRows * kTcKc + (size_t)2 * np * kTcKc);
}

cudaError_t launch_poles_tc(const DevProblem &P, const S2Block *blk, const int *tile_blk, const int4 *tiles,
                            int ntiles, const ChanSig *cs, const double *vp, const TcOut &fw, const TcOut &bk,
                            int dirs, int *err, size_t smem, cudaStream_t st) {
    if (ntiles <= 0) return cudaSuccess;
    cudaError_t e = allow_dynamic_smem((const void *)k_poles_tc);
    if (e != cudaSuccess) return e;
    k_poles_tc<<<ntiles, kTcThreads, smem, st>>>(P, blk, tile_blk, tiles, ntiles, cs, vp, fw, bk, dirs, err);
    return cudaGetLastError();
}

void tc_smem_init() { allow_dynamic_smem((const void *)k_poles_tc); }

}  // namespace bd
