// lz_fixed.cuh -- fixed-point sweeps of the FP64 Lanczos reductions (k_lanczos_long.cu,
// k_compact.cu): a basis vector's elements are at most one in size and the sweep's
// coefficients are needed to a fixed part of |w|, so both become pairs of 32-bit integers and
// a dot product an exact 64-bit integer sum.  GB300 issues FP64 at 1/64 of the FP32 rate.
#pragma once
#include <cuda_runtime.h>

namespace bd {

// x 2^-(bias - 1023) as (a 2^27 + b) 2^-57, |x| at most 2^(bias - 1023), to nearest and with b
// in [-2^26, 2^26): E v_{j-1} and v_{j-1} have their signs in common, so truncated bits or a
// dropped product of one sign would add up.  bias is the exponent field of one.
__device__ __forceinline__ int2 fixed_of(double x, int bias) {
    const int hi = __double2hiint(x);
    const unsigned lo = (unsigned)__double2loint(x);
    const unsigned long long m = ((unsigned long long)((hi & 0xfffff) | 0x100000) << 32 | lo) << 6;
    // one bit more than kept; + half a unit, + half of a's unit
    const unsigned long long f = (m >> min((unsigned)(bias - ((hi >> 20) & 0x7ff)), 63u)) + (1 + (1 << 27));
    const int a = (int)(f >> 28), b = ((int)(f >> 1) & 0x7ffffff) - (1 << 26);
    return hi < 0 ? make_int2(-a, -b) : make_int2(a, b);
}
// The same value with a rounded up or down by element i's place in a sequence that fills the unit interval
// evenly, b in (-2^27, 2^27): over elements of one size b is zero in the mean, where to nearest it is the
// same word n times.
__device__ __forceinline__ int2 fixed_dithered(double x, int bias, int i) {
    const int hi = __double2hiint(x);
    const unsigned lo = (unsigned)__double2loint(x);
    const unsigned long long m = ((unsigned long long)((hi & 0xfffff) | 0x100000) << 32 | lo) << 6;
    const unsigned long long f = (m >> min((unsigned)(bias - ((hi >> 20) & 0x7ff)), 63u)) + 1;
    const int a = (int)((f + ((unsigned)i * 0x9e3779b9u >> 4)) >> 28), b = (int)((unsigned)(f >> 1) - ((unsigned)a << 27));
    return hi < 0 ? make_int2(-a, -b) : make_int2(a, b);
}
// (s + l 2^-27) 2^-60 for sums s of a a' and l of what is below.  A thread's l is in [0, 2^27) at last, the rest
// carried into s, so 2^36 threads' sums can be added as they are.
struct FixedSum { long long s, l; };
// A thread's running sums of a a' and of a b' + b a'.  Where the low words of all elements have one sign (vectors
// of elements of one size) the second does not cancel: it grows by up to 3 2^56 |v| |w| sqrt(n) and would wrap
// beyond n of some thousand.  A run of at most kFixedRun elements keeps it inside its word.  The products b b'
// are left out: below n 2^-62 together for one sign, sqrt(n) 2^-63 with one factor dithered.
constexpr int kFixedRun = 1024;
__device__ __forceinline__ void fixed_step(FixedSum &acc, int va, int vb, int wa, int wb) {
    acc.s += (long long)va * wa;
    acc.l += (long long)va * wb;
    acc.l += (long long)vb * wa;
}
// with the upper words of b b' (units of 2^32 2^-114), for a vector against itself, where they have one sign, and
// where a sum is short
__device__ __forceinline__ void fixed_step(FixedSum &acc, int &h, int va, int vb, int wa, int wb) {
    fixed_step(acc, va, vb, wa, wb);
    h += __mulhi(vb, wb);
}
// what a run has summed, carried
__device__ __forceinline__ FixedSum fixed_carry(FixedSum r, int h = 0) {
    const long long l = r.l + ((long long)h << 5);
    return FixedSum{r.s + (l >> 27), l & 0x7ffffff};
}
// Times 2^(bias - 1023), rounded, from its bits: the FP64 forms of this are six instructions of
// ~64 cycles in every warp of a sweep.
__device__ __forceinline__ double fixed_value(FixedSum r, int bias) {
    long long t = r.s + (r.l >> 27);             // value t + f 2^-27
    unsigned f = (unsigned)r.l & 0x7ffffffu;
    const bool neg = t < 0;
    if (neg) {
        t = -t - (f != 0);
        f = (0u - f) & 0x7ffffffu;
    }
    unsigned long long m = (unsigned long long)t, lo = (unsigned long long)f << 37;   // m, then lo behind it
    int z = __clzll((long long)m);
    if (z == 64) {
        m = lo;
        lo = 0;
        z = __clzll((long long)m);
        if (z == 64) return 0.0;
        m <<= z;
        z += 64;
    } else if (z > 0) {
        m = (m << z) | (lo >> (64 - z));
    }
    // the leading bit, at bit 63, less itself, and half a unit; the carry goes to the exponent
    const unsigned long long q = (((m & 0x7fffffffffffffffull) + (1u << 10)) >> 11) +
                                 ((unsigned long long)(unsigned)(bias + 3 - z) << 52);
    return __longlong_as_double((long long)(q | (neg ? 0x8000000000000000ull : 0)));
}
// a stored element as a double (abs. error 2^-58, or half a unit in the last place), from its bits
__device__ __forceinline__ double fixed_to_double(int a, int b) {
    const long long q = ((long long)a << 27) + b;   // v 2^57, |q| <= 2^57
    const unsigned long long m = (unsigned long long)(q < 0 ? -q : q);
    const int z = __clzll((long long)m);   // 6 .. 64
    // the leading bit at bit 63, less itself, and half a unit; the carry goes to the exponent
    const unsigned long long f = ((m << (z & 63)) & 0x7fffffffffffffffull) + (1u << 10);
    const unsigned long long r = (f >> 11) + ((unsigned long long)(unsigned)(1023 + 6 - z) << 52);
    return __longlong_as_double(m == 0 ? 0 : (long long)(r | (q < 0 ? 0x8000000000000000ull : 0)));
}
// a normal float as a double, from its bits; what FP32 has as denormal is zero
__device__ __forceinline__ double f32_to_double(float x) {
    const unsigned u = __float_as_uint(x), m = u & 0x7fffffffu;
    if (m < 0x00800000u) return 0.0;
    return __hiloint2double((int)((u & 0x80000000u) | ((m >> 3) + (896u << 20))), (int)(m << 29));
}

// x to FP32 from its bits, truncated; below 2^-126 zero
__device__ __forceinline__ float f32_trunc(double x) {
    const unsigned hi = (unsigned)__double2hiint(x);
    const unsigned b = (hi & 0x80000000u) | ((__funnelshift_l((unsigned)__double2loint(x), hi, 3) - (384u << 23)) & 0x7fffffffu);
    return (hi & 0x7fffffffu) >= 897u << 20 ? __uint_as_float(b) : 0.0f;
}

// 1/sqrt(x), x > 0: the FP32 seed (2^-23) and one third-order step, five FP64 instructions where
// two Newton steps with their conversions and comparisons are eleven
__device__ __forceinline__ double rsqrt_cubic(double x) {
    const unsigned e = (unsigned)__double2hiint(x) >> 20;
    if (e < 1023 - 120 || e > 1023 + 120) return 1.0 / sqrt(x);
    const double y = f32_to_double(__frsqrt_rn(f32_trunc(x)));
    const double r = fma(-x * y, y, 1.0);
    return fma(y * r, fma(0.375, r, 0.5), y);
}

// 1/q: the FP32 seed and one third-order step, three FP64 instructions
__device__ __forceinline__ double rcp_cubic(double q) {
    const unsigned e = ((unsigned)__double2hiint(q) >> 20) & 0x7ffu;
    if (e < 1023 - 120 || e > 1023 + 120) return 1.0 / q;
    const double y = f32_to_double(__frcp_rn(f32_trunc(q)));
    const double r = fma(-q, y, 1.0);
    return fma(y, fma(r, r, r), y);
}

// whether a set of values whose largest has this upper word (sign cleared) keeps to the
// exponents FP32 has room for (2^+-40)
__device__ __forceinline__ bool fixed_range(unsigned hi) { return hi >= (1023u - 40) << 20 && hi <= (1023u + 40) << 20; }
// After a recurrence w is split against |E v_{j-1}|: where it is below 2^-6 of that (its square
// below this part of the other's), the sums are too coarse for it and the sweep is repeated, split
// against |w| itself.
constexpr double kFixedShort = 0x1p-12;
// |E v_{j-1}|^2 and |M p|^2, the scales of the split and the thresholds, are FP32 sums of squares: below
// this they lose elements to FP32's range (squares under 2^-149), down to a scale of zero for a w that is
// not, and the split puts nothing in its place.
constexpr double kFixedWeak = 0x1p-90;
// the exponent field of a power of two above |x|, from |x|^2
__device__ __forceinline__ int bias_above(double x2) {
    return ((__double2hiint(x2) >> 20) - 1023 + 2048) / 2 - 1024 + 1023 + 1;
}

// Warp sums of NV values at once: lane L ends with the total of value L >> (5 - log2 NV).
template <int NV, typename T, typename Add, typename Shf>
__device__ __forceinline__ T warp_sums_of(T *v, int lane, Add add, Shf shf) {
#pragma unroll
    for (int lev = 0; lev < 5; ++lev) {
        const int o = 16 >> lev;
        const int n = NV >> (lev + 1);
        if (n >= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < (NV >> 1); ++i)
                if (i < n) {
                    const T send = up ? v[i] : v[i + n];
                    const T keep = up ? v[i + n] : v[i];
                    v[i] = add(keep, shf(send, o));
                }
        } else {
            v[0] = add(v[0], shf(v[0], o));
        }
    }
    return v[0];
}

__device__ __forceinline__ FixedSum fixed_add(FixedSum p, FixedSum q) { return FixedSum{p.s + q.s, p.l + q.l}; }
__device__ __forceinline__ FixedSum fixed_shfl(FixedSum p, int o) {
    return FixedSum{__shfl_xor_sync(0xffffffffu, p.s, o), __shfl_xor_sync(0xffffffffu, p.l, o)};
}

}  // namespace bd
