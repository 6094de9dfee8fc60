// FP64 window sums in integer arithmetic, for the GPU and (in tests) the host.
//
// The FP64 unit does two fused multiply-adds a clock and SM; 32 x 32 + 64-bit
// integer ones run at 24 to 32. For a sum of products sum_k w_k v_k, weights and
// values become 57-bit fixed-point numbers relative to a bound on each (the
// plan's largest weight; the largest of the values summed together), split as
// hi 2^29 + lo with lo in [-2^28, 2^28). Per product
//   (wh 2^29 + wl) (vh 2^29 + vl) = HH 2^58 + X 2^29 + (dropped) wl vl,
// HH = sum wh vh, X = sum wh vl + wl vh in 64 bits, exactly, for up to 32 terms:
// three integer operations in place of one that takes as long as twelve. What is
// dropped or rounded is below 2^-56 of the product of the two bounds a term,
// where FP64 rounds each partial sum to 2^-53 of itself. So a sum keeps FP64's bits
// while its larger terms come near the bounds: a window's middle weights do, and
// the values' bound is a local one, of 16 rows of a column block (trafo) or the 32
// nodes of a chunk (adjoint).
// Measured against sums in extended precision (planes of 32^2 to 128^2; polar and
// random nodes; values of one size, strong in the centre, a peak over a floor, and
// over 16 decades): the trafo is off by 1.4e-16 to 3.7e-16 of its norm, with FP64
// sums by 1.5e-16 to 4.0e-16, its outer nodes by 0.92 to 1.00 times what FP64 sums
// leave there; the adjoint by 2.3e-16 to 3.8e-16, with FP64 sums by 2.4e-16 to
// 4.5e-16 (values of 16 decades at random: up to 2 % more than FP64 sums).
#pragma once
#include "intdiv.cuh"

namespace nudim {

struct alignas(8) Fixed {
    int hi, lo;
};
struct alignas(16) FixedC {  // complex
    Fixed re, im;
};

NUDIM_HD Fixed split_fixed(int64_t V)
{
    const int hi = (int)((V + (1ll << 28)) >> 29);
    return Fixed{hi, (int)((uint32_t)V - ((uint32_t)hi << 29))};
}

NUDIM_HD int exp_of(double x) { return (int)(bits_of(x) >> 52) & 0x7ff; }

// x as fixed point under the exponent field E >= x's own: x = V 2^(E - 1079)
NUDIM_HD Fixed to_fixed(double x, int E)
{
    const uint64_t v = bits_of(x);
    const int e = exp_of(x), s = E - e;
    uint64_t m = ((v & 0xfffffffffffffull) | (1ull << 52)) << 4;
    m = s < 62 && e ? (m + ((1ull << s) >> 1)) >> s : 0ull;
    return split_fixed((int64_t)v < 0 ? -(int64_t)m : (int64_t)m);
}

// a / 2^s (rounded), s >= 0: of a number under field E the same under field E + s
NUDIM_HD Fixed fixed_shift(Fixed a, int s)
{
    const int64_t V = (int64_t)a.hi * (1ll << 29) + a.lo;
    s = s < 62 ? s : 62;
    return split_fixed((V + ((1ll << s) >> 1)) >> s);
}

// 2^s a, s <= 2, exactly: not split anew (the parts grow; 14 products of such
// weights still fit FixedSum's 64 bits)
NUDIM_HD Fixed fixed_scaled(Fixed a, int s)
{
    return Fixed{(int)((uint32_t)a.hi << s), (int)((uint32_t)a.lo << s)};
}

// the product of two numbers under exponent field E, under field 2 E - 1022
NUDIM_HD Fixed fixed_product(Fixed a, Fixed b)
{
    const int64_t x = (int64_t)a.hi * b.lo + (int64_t)a.lo * b.hi;
    return split_fixed(2 * ((int64_t)a.hi * b.hi) + ((x + (1ll << 27)) >> 28));
}

// HH and X of a real weight's products with complex values
struct FixedSum {
    int64_t hr, xr, hi, xi;
    NUDIM_HD void init() { hr = xr = hi = xi = 0; }
    NUDIM_HD void add(Fixed w, const FixedC &v)
    {
        mad(hr, w.hi, v.re.hi);
        mad(xr, w.hi, v.re.lo);
        mad(xr, w.lo, v.re.hi);
        mad(hi, w.hi, v.im.hi);
        mad(xi, w.hi, v.im.lo);
        mad(xi, w.lo, v.im.hi);
    }
    // (written out: the compiler carries what it knows of a factor's range into
    // a 64 x 64-bit product; the adjoint's pass took 314 us against 261)
    static NUDIM_HD void mad(int64_t &s, int a, int b)
    {
#if defined(__CUDA_ARCH__)
        asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(s) : "r"(a), "r"(b));
#else
        s += (int64_t)a * b;
#endif
    }
    // in units of fixed_scale(weights' field, values' field)
    NUDIM_HD double re() const { return (double)(hr + ((xr + (1ll << 28)) >> 29)); }
    NUDIM_HD double im() const { return (double)(hi + ((xi + (1ll << 28)) >> 29)); }
};

// The largest exponent fields of values that the integer sums take. Beyond them
// (infinities, NaN, values whose scale would leave the normal numbers) the FP64
// unit sums; 0 (all zero or subnormal) sums to zero.
NUDIM_HD bool fixed_range(int E) { return E == 0 || (E > 300 && E < 1700); }

NUDIM_HD double fixed_scale(int Ew, int Ev)  // 2^(Ew + Ev - 2100)
{
    return Ev ? double_of((uint64_t)(Ew + Ev - 1077) << 52) : 0.0;
}

// A weight again; field 0: the plan's weights stayed FP64.
NUDIM_HD double fixed_value(const double *p, int Ew)
{
    if (!Ew) return *p;
    const uint64_t v = bits_of(*p);  // hi in the low word
    const int64_t V = ((int64_t)(int32_t)(uint32_t)v << 29) + (int32_t)(uint32_t)(v >> 32);
    return (double)V * double_of((uint64_t)(Ew - 56) << 52);
}

}  // namespace nudim
