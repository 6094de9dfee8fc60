// fft_regs.cuh -- small DFTs in registers and the four-step factorisation the
// FFT passes are built from.
#pragma once

#include "common.cuh"

namespace nudim {

template <typename T>
__device__ __forceinline__ cplx_t<T> cmul(cplx_t<T> a, cplx_t<T> b)
{
    return mkc<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// a + b, a - b: FP32 as paired instructions (the same rounding)
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b)
{
    return __ffma2_rn(b, make_float2(-1.f, -1.f), a);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b)
{
    return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b)
{
    return make_double2(a.x - b.x, a.y - b.y);
}

// e^{DIR 2 pi i k / 16}, k < 16, from cos(2 pi k / 16) for k = 0..4
template <typename T, int DIR> __device__ __forceinline__ cplx_t<T> w16(int k)
{
    constexpr double c[5] = {1.0, 0.92387953251128675613, 0.70710678118654752440,
                             0.38268343236508977173, 0.0};
    double cs, sn;
    int q = k & 3, h = k >> 2;  // k = 4h + q: rotate (cos, sin) of q by h quarter turns
    double cq = c[q], sq = c[4 - q];
    switch (h & 3) {
    case 0: cs = cq; sn = sq; break;
    case 1: cs = -sq; sn = cq; break;
    case 2: cs = -cq; sn = -sq; break;
    default: cs = sq; sn = -cq; break;
    }
    return mkc<T>((T)cs, (T)(DIR * sn));
}

template <typename T, int DIR>
__device__ __forceinline__ void dft2(cplx_t<T> &a0, cplx_t<T> &a1)
{
    cplx_t<T> t = a0;
    a0 = cadd(t, a1);
    a1 = csub(t, a1);
}

template <typename T, int DIR>
__device__ __forceinline__ void dft4(cplx_t<T> &x0, cplx_t<T> &x1, cplx_t<T> &x2, cplx_t<T> &x3)
{
    using C = cplx_t<T>;
    const C a0 = cadd(x0, x2), a1 = csub(x0, x2), a2 = cadd(x1, x3), a3 = csub(x1, x3);
    x0 = cadd(a0, a2);
    x2 = csub(a0, a2);
    // forward: X1 = a1 - i a3, X3 = a1 + i a3; inverse: the other way
    if (DIR < 0) {
        x1 = mkc<T>(a1.x + a3.y, a1.y - a3.x);
        x3 = mkc<T>(a1.x - a3.y, a1.y + a3.x);
    } else {
        x1 = mkc<T>(a1.x - a3.y, a1.y + a3.x);
        x3 = mkc<T>(a1.x + a3.y, a1.y - a3.x);
    }
}

// the same with x1 = x2 = 0
template <typename T, int DIR>
__device__ __forceinline__ void dft4_ends(cplx_t<T> &x0, cplx_t<T> &x1, cplx_t<T> &x2,
                                          cplx_t<T> &x3)
{
    using C = cplx_t<T>;
    const C a = x0, d = x3;
    x0 = cadd(a, d);
    x2 = csub(a, d);
    // forward: X1 = a + i d, X3 = a - i d; inverse: the other way
    const C r = mkc<T>(a.x - d.y, a.y + d.x), q = mkc<T>(a.x + d.y, a.y - d.x);
    x1 = DIR < 0 ? r : q;
    x3 = DIR < 0 ? q : r;
}

// R-point DFT of a[0..R) in registers.  Output X[p] is left in a[out(p)]:
// R = 16 and 8 are split as R1 = 4 inner DFTs over m = R2 m1 + m2, the
// twiddles e^{DIR 2 pi i m2 p1 / R} and R2-point outer DFTs, X[p1 + 4 p2] in
// a[R2 p1 + p2].
template <int R> __device__ __forceinline__ constexpr int dft_out(int p)
{
    return R == 16 ? 4 * (p & 3) + (p >> 2) : R == 8 ? 2 * (p & 3) + (p >> 2) : p;
}

// ENDS (R = 8, 16): only the first and last quarter of a is nonzero.
template <typename T, int DIR, int R, bool ENDS = false>
__device__ __forceinline__ void dft_regs(cplx_t<T> *a)
{
    if (R == 2) {
        dft2<T, DIR>(a[0], a[1]);
    } else if (R == 4) {
        dft4<T, DIR>(a[0], a[1], a[2], a[3]);
    } else if (R == 8) {
#pragma unroll
        for (int m2 = 0; m2 < 2; m2++) {
            if (ENDS) dft4_ends<T, DIR>(a[m2], a[2 + m2], a[4 + m2], a[6 + m2]);
            else dft4<T, DIR>(a[m2], a[2 + m2], a[4 + m2], a[6 + m2]);
        }
#pragma unroll
        for (int p1 = 1; p1 < 4; p1++) a[2 * p1 + 1] = cmul<T>(a[2 * p1 + 1], w16<T, DIR>(2 * p1));
#pragma unroll
        for (int p1 = 0; p1 < 4; p1++) dft2<T, DIR>(a[2 * p1], a[2 * p1 + 1]);
    } else {
#pragma unroll
        for (int m2 = 0; m2 < 4; m2++) {
            if (ENDS) dft4_ends<T, DIR>(a[m2], a[4 + m2], a[8 + m2], a[12 + m2]);
            else dft4<T, DIR>(a[m2], a[4 + m2], a[8 + m2], a[12 + m2]);
        }
#pragma unroll
        for (int p1 = 1; p1 < 4; p1++)
#pragma unroll
            for (int m2 = 1; m2 < 4; m2++)
                a[4 * p1 + m2] = cmul<T>(a[4 * p1 + m2], w16<T, DIR>(m2 * p1));
#pragma unroll
        for (int p1 = 0; p1 < 4; p1++)
            dft4<T, DIR>(a[4 * p1], a[4 * p1 + 1], a[4 * p1 + 2], a[4 * p1 + 3]);
    }
}

// ================================================================ four-step register FFT
// n = R1 x R2 points with one shared-memory exchange: input index l = j +
// R2 m (j < R2, m < R1), pass 1 an R1-point DFT over m per j (registers),
// twiddle W_n^{j k1}, exchange, pass 2 an R2-point DFT over j per k1, output
// index k = k1 + R1 k2 (the classical four-step factorisation of the DFT).
// R = 32 DFTs in registers split as two 16-point DFTs (dft_regs<16>) and a
// radix-2 step with the twiddles W_32^p.
template <typename T, int DIR> __device__ __forceinline__ cplx_t<T> w32(int p)
{
    // cos(2 pi p / 32), p = 0..8
    constexpr double c[9] = {1.0,
                             0.98078528040323044913,
                             0.92387953251128675613,
                             0.83146961230254523708,
                             0.70710678118654752440,
                             0.55557023301960222474,
                             0.38268343236508977173,
                             0.19509032201612826785,
                             0.0};
    const int q = p & 7, h = p >> 3;  // p = 8h + q: rotate by h quarter turns
    double cs, sn;
    const double cq = c[q], sq = c[8 - q];
    switch (h & 3) {
    case 0: cs = cq; sn = sq; break;
    case 1: cs = -sq; sn = cq; break;
    case 2: cs = -cq; sn = -sq; break;
    default: cs = sq; sn = -cq; break;
    }
    return mkc<T>((T)cs, (T)(DIR * sn));
}

// W_24^p = e^{DIR 2 pi i p / 24}, p = 0..23
template <typename T, int DIR> __device__ __forceinline__ cplx_t<T> w24(int p)
{
    // cos(2 pi q / 24), q = 0..6
    constexpr double c[7] = {1.0,
                             0.96592582628906828675,
                             0.86602540378443864676,
                             0.70710678118654752440,
                             0.5,
                             0.25881904510252076235,
                             0.0};
    const int q = p % 6, h = p / 6;  // p = 6h + q: rotate by h quarter turns
    double cs, sn;
    const double cq = c[q], sq = c[6 - q];
    switch (h & 3) {
    case 0: cs = cq; sn = sq; break;
    case 1: cs = -sq; sn = cq; break;
    case 2: cs = -cq; sn = -sq; break;
    default: cs = sq; sn = -cq; break;
    }
    return mkc<T>((T)cs, (T)(DIR * sn));
}

// R-point DFT (R = 16, 24 or 32) of a[0..R) in registers; X[p] is left in
// a[fs_out<R>(p)].  R = 24: three 8-point DFTs over a[3u + v], the twiddles
// W_24^{v p8} and 3-point DFTs over v, X[p8 + 8q] in a[3 p8 + q].
template <int R> __device__ __forceinline__ constexpr int fs_out(int p)
{
    return R == 16   ? dft_out<16>(p)
           : R == 24 ? 3 * (p & 7) + (p >> 3)
                     : (p < 16 ? 2 * dft_out<16>(p) : 2 * dft_out<16>(p - 16) + 1);
}

// ENDS: only the first and last quarter of a is nonzero (a zero-padded line's
// inputs at stride n / R), which spares half of the first stage.
template <typename T, int DIR, int R, bool ENDS = false>
__device__ __forceinline__ void fs_dft(cplx_t<T> *a)
{
    using C = cplx_t<T>;
    if constexpr (R == 16) {
        dft_regs<T, DIR, 16, ENDS>(a);
    } else if constexpr (R == 24) {
        C e[3][8];
#pragma unroll
        for (int v = 0; v < 3; v++)
#pragma unroll
            for (int u = 0; u < 8; u++) e[v][u] = a[3 * u + v];
#pragma unroll
        for (int v = 0; v < 3; v++) dft_regs<T, DIR, 8, ENDS>(e[v]);
        // X[p8 + 8q] = sum_v (W_24^{v p8} E_v[p8]) W_3^{v q}
        const T h3 = (T)0.86602540378443864676;  // sqrt(3) / 2
#pragma unroll
        for (int p8 = 0; p8 < 8; p8++) {
            const C x0 = e[0][dft_out<8>(p8)];
            C x1 = e[1][dft_out<8>(p8)], x2 = e[2][dft_out<8>(p8)];
            if (p8) {
                x1 = cmul<T>(x1, w24<T, DIR>(p8));
                x2 = cmul<T>(x2, w24<T, DIR>(2 * p8));
            }
            const C sm = cadd(x1, x2), df = csub(x1, x2);
            const C mid = mkc<T>(x0.x - (T)0.5 * sm.x, x0.y - (T)0.5 * sm.y);
            // DIR i (sqrt(3)/2) (x1 - x2)
            const C rot = mkc<T>(-(T)DIR * h3 * df.y, (T)DIR * h3 * df.x);
            a[3 * p8] = cadd(x0, sm);
            a[3 * p8 + 1] = cadd(mid, rot);
            a[3 * p8 + 2] = csub(mid, rot);
        }
    } else {
        C e[16], o[16];
#pragma unroll
        for (int u = 0; u < 16; u++) {
            e[u] = a[2 * u];
            o[u] = a[2 * u + 1];
        }
        dft_regs<T, DIR, 16, ENDS>(e);
        dft_regs<T, DIR, 16, ENDS>(o);
        // X[p] = E[p] + W32^p O[p], X[p + 16] = E[p] - W32^p O[p]
#pragma unroll
        for (int p = 0; p < 16; p++) {
            const C ev = e[dft_out<16>(p)];
            C ov = o[dft_out<16>(p)];
            if (p) ov = cmul<T>(ov, w32<T, DIR>(p));
            a[2 * dft_out<16>(p)] = cadd(ev, ov);
            a[2 * dft_out<16>(p) + 1] = csub(ev, ov);
        }
    }
}

template <int R1, int R2> __host__ __device__ constexpr int fs_col_stride()
{
    // R1 x (R2 + 1) rounded up to 4 mod 16 elements
    return ((R1 * (R2 + 1) + 11) / 16) * 16 + 4;
}

}  // namespace nudim
