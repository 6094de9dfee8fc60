// intdiv.cuh -- correctly rounded FP64 quotients in integer arithmetic.
//
// This GPU's FP64 pipe takes two lanes a clock and SM; its 32-bit integer
// units take 64 and more.  A quotient costs the FP64 pipe eight or more fused
// multiply-adds, so the stencils whose FP64 results are held to IEEE rounding
// spend most of their time dividing.  These functions give the same bits
// (round to nearest even) from integer products: an approximation of the
// quotient to well beyond 53 bits, and where its last bits leave the rounding
// open, the sign of the exact remainder (a low 64-bit product).  Newton's
// iteration for the reciprocal, seeded by the hardware's FP32 approximation.
//
// Host and device run the same code (the seed excepted: any within 2^-21
// does), so the CPU tests hold it against the host's division.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define NUDIM_HD __host__ __device__ __forceinline__
#else
#define NUDIM_HD inline
#endif

namespace nudim {

NUDIM_HD uint64_t bits_of(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    return b;
#endif
}

NUDIM_HD double double_of(uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)b);
#else
    double x;
    std::memcpy(&x, &b, 8);
    return x;
#endif
}

NUDIM_HD uint64_t mul_hi(uint64_t a, uint64_t b)
{
#if defined(__CUDA_ARCH__)
    return __umul64hi(a, b);
#else
    return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// approximately 1 / f for a normal f in [1/2, 1), as FP32 bits
NUDIM_HD uint32_t seed_rcp(uint32_t f)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
    return __float_as_uint(r);
#else
    float x;
    std::memcpy(&x, &f, 4);
    x = 1.0f / x;
    uint32_t b;
    std::memcpy(&b, &x, 4);
#if defined(NUDIM_SEED_SHIFT)
    b += NUDIM_SEED_SHIFT;  // tests: another approximation
#endif
    return b;
#endif
}

// approximately 1 / sqrt(f) for a normal f in [1/4, 1), as FP32 bits
NUDIM_HD uint32_t seed_rsqrt(uint32_t f)
{
#if defined(__CUDA_ARCH__)
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
    return __float_as_uint(r);
#else
    float x;
    std::memcpy(&x, &f, 4);
    x = 1.0f / std::sqrt(x);
    uint32_t b;
    std::memcpy(&b, &x, 4);
#if defined(NUDIM_SEED_SHIFT)
    b += NUDIM_SEED_SHIFT;
#endif
    return b;
#endif
}

// One Newton step for 2^116 / s (s in [2^52, 2^53), y = 2^53 / s in (1, 2] as
// y 2^63) from y1, y in 48 bits (y 2^47) within 2^-41: the residual 1 - s y1 is
// the low 64 bits of the product, exactly.
NUDIM_HD uint64_t recip_step(uint64_t s, uint64_t y1)
{
    const int64_t E = -(int64_t)(s * y1);  // 2^-100
    const int32_t e1 = (int32_t)(E >> 29); // 2^-71
    const int64_t c1 = ((int64_t)e1 * (int32_t)(uint32_t)(y1 >> 17)) >> 38;
    return (y1 << 16) + (uint64_t)c1;
}

// 2^116 / s for s in (2^52, 2^53), in units of 1: y = 2^53 / s in (1, 2) as
// y 2^63, within 3 units.  Two Newton steps: the seed's error 2^-21 goes to
// 2^-42 (the residual 1 - d y0 from a 64 x 32-bit product) and below 2^-71
// (from the low 64 bits of s y1, exact since |1 - d y1| < 2^-41).
NUDIM_HD uint64_t recip63(uint64_t s)
{
    const uint64_t D = s << 11;  // d = D / 2^64 in (1/2, 1)
    const uint32_t dh = (uint32_t)(D >> 32), dl = (uint32_t)D;
    uint32_t r = seed_rcp(0x3f000000u + ((dh - 0x80000000u) >> 8));
    r = r < 0x3fffffffu ? r : 0x3fffffffu;
    r = r > 0x3f800000u ? r : 0x3f800000u;
    const uint32_t y0 = (r << 8) | 0x80000000u;  // 1.31
    const uint64_t p = (uint64_t)dh * y0 + (((uint64_t)dl * y0) >> 32);
    const int32_t e0 = (int32_t)((int64_t)(0x8000000000000000ull - p) >> 11);  // 2^-52
    const int64_t c0 = ((int64_t)e0 * (int32_t)(y0 >> 1)) >> 19;
    const uint64_t y1 = (((uint64_t)y0 << 32) + (uint64_t)c0) >> 16;  // 1.47
    return recip_step(s, y1);
}

// The diffusion coefficient 1 / (1 + g^2 / b) as the reference's operations
// round it: RN(1 / RN(1 + RN(RN(g g) / b))).  b > 0 is the square of an FP32
// value (48 significant bits), so no quotient a / b lies on a rounding
// boundary or within 2^-49 of an ulp of one.
struct DiffDiv {
    uint64_t mb, rb;  // b's 53-bit significand and floor(2^116 / mb) (2^64 - 1 if that is 2^64)
    int eb;           // b = mb 2^(eb - 52)
    int lim;          // exponents of g^2 below this: g^2 and g^2 / b are finite
    double b;
};

inline bool diff_div_init(double b, DiffDiv *d)
{
    const uint64_t v = bits_of(b);
    const int e = (int)(v >> 52);  // sign 0
    if (!(b > 0) || e < 1023 - 200 || e > 1023 + 200) return false;
    d->b = b;
    d->mb = (v & 0xfffffffffffffull) | (1ull << 52);
    d->eb = e - 1023;
    d->lim = d->eb < 0 ? 1000 + d->eb : 1000;
    const unsigned __int128 q = ((unsigned __int128)1 << 116) / d->mb;
    d->rb = q >> 64 ? ~0ull : (uint64_t)q;
    return true;
}

// The flux RN(c g) with that coefficient c; false for values whose square or
// quotient comes near overflow (2^400 and more), infinities and NaN, which the
// caller divides.  No branches: the loop around it overlaps several of these.
// 1 + q is the FP64 unit's: the sum's shifts take the integer units longer.
NUDIM_HD bool diff_flux_int(double g, const DiffDiv &k, double *out)
{
    const uint64_t v = bits_of(g);
    // ---- a = RN(g g), significand ma, exponent ea; h: the top 64 bits of the
    // square, whose rest is zero exactly when X is a multiple of 2^32
    const uint64_t X = (v << 11) | (1ull << 63);
    uint64_t h = mul_hi(X, X);
    int ea = 2 * ((int)(v >> 52 & 0x7ff) - 1023) + 1;
    if (!(h >> 63)) {
        h <<= 1;
        ea--;
    }
    uint64_t ma = h >> 11;
    const uint32_t hl = (uint32_t)h & 2047u, more = (uint32_t)X ? 1u : ((uint32_t)ma & 1u);
    ma += hl + more > 1024u;
    // ---- q = RN(a / b), b's significand brought to [ma / 2, ma]: the quotient
    // mq in [2^52, 2^53) from 2^10 a / b, low by less than 3; the last bit from
    // the sign of 2 (2^52 ma - mq mb) - mb, right also where the approximation
    // has missed an integer.  (ma = 2^53 is not below any mb.)
    int eq = ea - k.eb;
    if (ma < k.mb) {
        ma <<= 1;
        eq--;
    }
    uint64_t mq = mul_hi(ma << 10, k.rb) >> 10;
    mq += (int64_t)((ma << 53) - (2 * mq + 1) * k.mb) > 0;
    const bool ok = ea < k.lim;
    eq = eq > -1000 ? eq : -1000;  // 1 + q = 1 all the same
    // ---- s = RN(1 + q) = S 2^(e - 52)
#if defined(__CUDA_ARCH__)
    const uint64_t sv = bits_of(__dadd_rn(1.0, double_of(((uint64_t)(uint32_t)(eq + 1022) << 52) + mq)));
#else
    const uint64_t sv = bits_of(1.0 + double_of(((uint64_t)(uint32_t)(eq + 1022) << 52) + mq));
#endif
    const uint64_t S = (sv & 0xfffffffffffffull) | (1ull << 52);
    // ---- c = RN(1 / s): 2^105 / S = y / 2^11, y within 3; the last bit from
    // the sign of 2^106 - S (2 c + 1).  (S = 2^52: c = 2^53 - 1 + 1.)
    uint64_t c = recip63(S) >> 11;
    c += (int64_t)(S * (2 * c + 1)) < 0;
    // ---- RN(c g), c 2^(-53 - e) times g's significand: p in [2^62, 2^63) after
    // at most one doubling, `rest` whatever follows it.  A zero or subnormal g
    // has c = 1.
    const uint64_t cs = c << 10;
    uint64_t p = mul_hi(cs, X);
    const uint32_t rest = cs * X != 0;
    const int eg = (int)(v >> 52) & 0x7ff;
    int ep = eg + 1022 - (int)(sv >> 52);
    if (!(p >> 62)) {
        p <<= 1;
        ep--;
    }
    uint64_t m = p >> 10;
    m += ((uint32_t)p & 1023u) + (rest | ((uint32_t)m & 1u)) > 512u;
    const uint64_t r = ((uint64_t)(uint32_t)ep << 52) + m;
    *out = double_of(eg ? (v & 0x8000000000000000ull) | r : v);
    return ok;
}

// ---------------------------------------------------------------- a / b, sqrt
// A divisor ready for several quotients: b = n 2^(e - 52), n in [2^52, 2^53),
// y = 2^116 / n within 4.
struct IntDivisor {
    uint64_t n, y;
    int e;
};

// b positive and normal
NUDIM_HD IntDivisor int_divisor(double b)
{
    const uint64_t v = bits_of(b);
    IntDivisor d;
    d.n = (v & 0xfffffffffffffull) | (1ull << 52);
    d.e = (int)(v >> 52 & 0x7ff) - 1023;
    d.y = recip63(d.n);
    return d;
}

// RN(t / b); false where t is not finite or the quotient not a normal number
// or zero (the caller divides).
NUDIM_HD bool int_div(double t, const IntDivisor &d, double *out)
{
    const uint64_t v = bits_of(t);
    const int et = (int)(v >> 52) & 0x7ff;
    uint64_t m = (v & 0xfffffffffffffull) | (1ull << 52);
    int eq = et - d.e;
    if (m < d.n) {
        m <<= 1;
        eq--;
    }
    uint64_t q = mul_hi(m << 10, d.y) >> 10;
    q += (int64_t)((m << 53) - (2 * q + 1) * d.n) > 0;
    const bool zero = (v << 1) == 0;
    const uint64_t r = ((uint64_t)(uint32_t)(eq - 1) << 52) + q;
    *out = double_of(zero ? v : (v & 0x8000000000000000ull) | r);
    return zero || ((unsigned)(et - 1) < 2046u && (unsigned)(eq - 1) < 2045u);
}

// RN(z z), 0 where that is below 2^-998; false where z is not finite or the
// square near overflow.
NUDIM_HD bool int_square(double z, double *out)
{
    const uint64_t v = bits_of(z);
    const int e = (int)(v >> 52) & 0x7ff;
    const uint64_t X = (v << 11) | (1ull << 63);
    uint64_t h = mul_hi(X, X);  // the square's top 64 bits; the rest 0 if X is a multiple of 2^32
    int eq = 2 * e - 1023;
    if (h >> 63) eq++;
    else h <<= 1;
    uint64_t m = h >> 11;
    m += ((uint32_t)h & 2047u) + ((uint32_t)X ? 1u : ((uint32_t)m & 1u)) > 1024u;
    *out = double_of(e < 1023 - 499 ? 0 : ((uint64_t)(uint32_t)(eq - 1) << 52) + m);
    return e < 1023 + 500;
}

// RN(z z) for any z: what int_square leaves (near overflow) or flushes (below
// 2^-998: harmless under the norm's 1e-8, but a sum of such squares is not 0)
// is the FP64 unit's.
NUDIM_HD double square_rn(double z)
{
    double q;
    if (!int_square(z, &q) || (!bits_of(q) && bits_of(z) << 1)) {
#if defined(__CUDA_ARCH__)
        q = __dmul_rn(z, z);
#else
        q = z * z;
#endif
    }
    return q;
}

// RN(sqrt(s)) for a positive normal s, as a divisor.  With s = d 4^h, d in [1/4,
// 1): y0 ~ 1 / sqrt(d) from the FP32 seed, one Newton step (within 2^-42), then
// the square root from the 48 leading bits n1 of d y1 and the exact residual
// d - n1^2 (within 2^-63); the last bit from the sign of 4 d - (2 n + 1)^2; and
// the reciprocal of the rounded root by one more step.
NUDIM_HD IntDivisor int_sqrt(double s)
{
    const uint64_t v = bits_of(s);
    int e = (int)(v >> 52) - 1022;  // s = (1/2 .. 1) 2^e
    uint64_t D = (v << 11) | (1ull << 63);
    if (e & 1) {
        D >>= 1;
        e++;
    }
    const uint32_t dh = (uint32_t)(D >> 32);
    // d to FP32: leading bits under the exponent of [1/2, 1) or [1/4, 1/2)
    const uint32_t f = dh >> 31 ? 0x3f000000u + ((dh - 0x80000000u) >> 8)
                                : 0x3e800000u + ((dh - 0x40000000u) >> 7);
    uint32_t r = seed_rsqrt(f);
    r = r < 0x3fffffffu ? r : 0x3fffffffu;
    r = r > 0x3f800000u ? r : 0x3f800000u;
    const uint32_t a0 = (r & 0x7fffffu) | 0x800000u;  // y0, 1.23
    const uint32_t y0 = a0 << 8;                      // 1.31
    // 1 - d y0^2 in 2^-62
    const int64_t E = (int64_t)((1ull << 62) - mul_hi(D, ((uint64_t)a0 * a0) << 16));
    const int32_t e0 = (int32_t)(E >> 11);  // 2^-51
    const int64_t c0 = ((int64_t)e0 * (int32_t)(y0 >> 1)) >> 19;
    const uint64_t y1 = ((uint64_t)y0 << 32) + (uint64_t)c0;  // 1.63
    const uint64_t n1 = mul_hi(D, y1) >> 15;                  // sqrt(d), 48 bits
    // d - n1^2 in 2^-96, times y / 2: in 2^-64
    const int64_t R = (int64_t)((D << 32) - n1 * n1);
    const int64_t cr = ((int64_t)(int32_t)(R >> 24) * (int32_t)(uint32_t)(y1 >> 33)) >> 39;
    const uint64_t N = (n1 << 16) + (uint64_t)cr;
    IntDivisor d;
    d.n = N >> 11;
    d.n += (int64_t)((D << 44) - (2 * d.n + 1) * (2 * d.n + 1)) > 0;
    d.e = (e >> 1) - 1;
    // a root that rounds up to the next power of two
    const bool carry = d.n >> 53 != 0;
    d.y = recip_step(d.n, y1 >> 16);
    if (carry) {
        d.n = 1ull << 52;
        d.e++;
        d.y = ~0ull;
    }
    return d;
}

// ---------------------------------------------------------------- FP32 g / b
// RN(2^64 g / b) from y = RN(1 / b), b in [1e-15, 1e15], |g| below 2^10: two
// corrections (the first brings the quotient within one ulp, and from there one
// more with RN(1 / b) rounds correctly: Markstein 1990).  The factor keeps the
// residuals of the smallest g exact.
NUDIM_HD float quotient64(float g, float b, float y)
{
#if defined(__CUDA_ARCH__)
    const float h = __fmul_rn(g, 0x1p64f);
    float q = __fmul_rn(h, y);
    q = __fmaf_rn(__fmaf_rn(-q, b, h), y, q);
    return __fmaf_rn(__fmaf_rn(-q, b, h), y, q);
#else
    const float h = g * 0x1p64f;
    float q = h * y;
    q = std::fma(std::fma(-q, b, h), y, q);
    return std::fma(std::fma(-q, b, h), y, q);
#endif
}

NUDIM_HD double double_of(const IntDivisor &d)
{
    return double_of(((uint64_t)(uint32_t)(d.e + 1022) << 52) + d.n);
}

}  // namespace nudim
