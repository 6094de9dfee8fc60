// toeplitz.cu -- CGNR's normal operator T = A^H W A as a convolution, and the
// CG around it.
//
// (T p)[k] = sum_k' K[k - k'] p[k'], K[m] = sum_j w_j e^{2 pi i m x_j}, |m| < N.
// Embedded in an nt x nt circulant with nt >= 2N - 1 (so no wrap reaches a kept
// output) it is a pointwise product of DFTs.  A CG step is three passes over
// the planes:
//
//   rows      p = z + beta p and f += alpha p_old as the row is loaded, then the
//             nt-point FFT of the zero-padded row              -> H [N0][nt]
//   columns   nt-point FFT, product with khat (the kernel's DFT / nt^2, real),
//             inverse FFT, the N0 rows kept, in place; p^H T p = sum khat |P|^2
//             (Parseval) falls out of the product, so alpha = |z|^2 / p^H T p is
//             known before the product is back in coefficient space
//   rows      inverse FFT, crop, z -= alpha T p, |z|^2 for beta
//
// so T p itself is never stored and no pass of its own updates a vector: 7
// vectors and 8 half-padded spectra move per step instead of 12 and 8.  The
// row FFTs are four-step (fft_regs.cuh): nt = R1 x R2 with one shared-memory
// exchange; the column FFTs three-step.  N is even, so a line's N <= nt / 2 inputs and kept outputs lie in
// the first and last quarters: the first stages skip the zeros between and the
// last stages form only what is kept.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include <cuda_pipeline.h>

#include "engine.cuh"
#include "fft_regs.cuh"

namespace nudim {

namespace {

template <int R1, int R2> __host__ __device__ constexpr int row_stride() { return R1 * (R2 + 1); }

// dots: 4 doubles per plane, {|z|^2, alpha, beta, -}
enum RowMode {
    TR_COMPLEX, // f (complex) in
    TR_REAL,    // a real start value in, f written
    TR_FIRST,   // p = z
    TR_CG       // f += alpha p, p = z + beta p
};

// ================================================================ row pass
// R2 threads per row (a warp, or half of one), 128 / R2 rows per CTA; the
// exchange stays within the warp.  Bound by memory: TR_CG moves five vectors and
// the spectra, 96 planes of 384 x 384 at 6.8 TB/s (116 us).
template <typename T, int MODE, int R1, int R2>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 4 : 2)
k_toep_rows(const void *src, cplx_t<T> *f, cplx_t<T> *p,
            const cplx_t<T> *z, const double *dots, int N0, int N1,
            const cplx_t<T> *__restrict__ tw, int plane0, cplx_t<T> *H)
{
    await_last();
    using C = cplx_t<T>;
    constexpr int nt = R1 * R2, RPC = 128 / R2, Q = R1 / 4;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int line = threadIdx.x / R2, j = threadIdx.x - line * R2;
    C *S = (C *)smraw + line * row_stride<R1, R2>();
    const int b = blockIdx.y, gb = plane0 + b, a = blockIdx.x * RPC + line;
    const bool live = a < N0;
    const size_t row = ((size_t)gb * N0 + (live ? a : 0)) * N1;
    T alpha = 0, beta = 0;
    if (MODE == TR_CG) {
        alpha = (T)dots[4 * gb + 1];
        beta = (T)dots[4 * gb + 2];
    }
    C x[R1];
    // inputs l = j + R2 m in the first (k = l) and last (k = l - nt) quarter;
    // coefficient k is at column k + N1 / 2
    constexpr int NV = 2 * Q;
    C v[NV], w[MODE == TR_CG ? NV : 1], u[MODE == TR_CG ? NV : 1];
    auto col = [&](int i) { return j + R2 * (i < Q ? i : i - NV) + N1 / 2; };
    auto in = [&](int i) { return live && col(i) >= 0 && col(i) < N1; };
#pragma unroll
    for (int i = 0; i < NV; i++) {
        v[i] = mkc<T>(0, 0);
        if (MODE == TR_CG) w[i] = u[i] = mkc<T>(0, 0);
        if (in(i)) {
            const size_t o = row + col(i);
            if (MODE == TR_COMPLEX) v[i] = ((const C *)src)[o];
            else if (MODE == TR_REAL) v[i] = mkc<T>(((const T *)src)[o], T(0));
            else v[i] = z[o];
            if (MODE == TR_CG) {
                w[i] = p[o];
                u[i] = f[o];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NV; i++) {
        if (MODE == TR_CG) {
            u[i] = mkc<T>(u[i].x + alpha * w[i].x, u[i].y + alpha * w[i].y);
            v[i] = mkc<T>(beta * w[i].x + v[i].x, beta * w[i].y + v[i].y);
        }
        if (in(i)) {
            const size_t o = row + col(i);
            if (MODE == TR_REAL) f[o] = v[i];
            if (MODE == TR_FIRST || MODE == TR_CG) p[o] = v[i];
            if (MODE == TR_CG) f[o] = u[i];
        }
    }
#pragma unroll
    for (int m = 0; m < R1; m++)
        x[m] = m < Q ? v[m] : m >= R1 - Q ? v[m - (R1 - NV)] : mkc<T>(0, 0);
    fs_dft<T, -1, R1, true>(x);
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) {
        C t = x[fs_out<R1>(k1)];
        if (k1) t = cmul<T>(t, tw[j * k1]);
        S[k1 * (R2 + 1) + j] = t;
    }
    __syncwarp();
    if (!live) return;
    C *Hrow = H + ((size_t)b * N0 + a) * nt;
    for (int k1 = j; k1 < R1; k1 += R2) {
        C y[R2];
#pragma unroll
        for (int jj = 0; jj < R2; jj++) y[jj] = S[k1 * (R2 + 1) + jj];
        fs_dft<T, -1, R2>(y);
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) Hrow[k1 + R1 * k2] = y[fs_out<R2>(k2)];
    }
}

// The inverse row pass: g = the row's inverse FFT, cropped.  RESID: z = z - g
// (z holds A^H W y, g = T f); otherwise z -= alpha g.  Partial |z|^2 per CTA.
template <typename T, bool RESID, int R1, int R2>
__global__ void __launch_bounds__(128, sizeof(T) == 4 ? 4 : 2)
k_toep_irows(const cplx_t<T> *H, cplx_t<T> *z,
             const double *dots, int N0, int N1, const cplx_t<T> *__restrict__ tw,
             int plane0, double *part, int part_stride)
{
    await_last();
    using C = cplx_t<T>;
    constexpr int nt = R1 * R2, RPC = 128 / R2;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double sh[32];
    const int line = threadIdx.x / R2, j = threadIdx.x - line * R2;
    C *S = (C *)smraw + line * row_stride<R1, R2>();
    const int b = blockIdx.y, gb = plane0 + b, a = blockIdx.x * RPC + line;
    const bool live = a < N0;
    const C *Hrow = H + ((size_t)b * N0 + (live ? a : 0)) * nt;
    const T alpha = RESID ? T(1) : (T)dots[4 * gb + 1];
    C x[R1];
#pragma unroll
    for (int m = 0; m < R1; m++) x[m] = live ? Hrow[j + R2 * m] : mkc<T>(0, 0);
    fs_dft<T, +1, R1>(x);
#pragma unroll
    for (int k1 = 0; k1 < R1; k1++) {
        C v = x[fs_out<R1>(k1)];
        if (k1) {
            C w = tw[j * k1];
            w.y = -w.y;
            v = cmul<T>(v, w);
        }
        S[k1 * (R2 + 1) + j] = v;
    }
    __syncwarp();
    T s = 0;
    if (live) {
        C *zr = z + ((size_t)gb * N0 + a) * N1;
        for (int k1 = j; k1 < R1; k1 += R2) {
            // output k1 + R1 k2 (mod nt) is column + N1 / 2: the first and last
            // quarter of k2
            constexpr int Q2 = R2 / 4;
            C zv[2 * Q2], y[R2];
            auto col = [&](int i) { return k1 + R1 * (i < Q2 ? i : i - 2 * Q2) + N1 / 2; };
#pragma unroll
            for (int i = 0; i < 2 * Q2; i++) {
                zv[i] = mkc<T>(0, 0);
                if (col(i) >= 0 && col(i) < N1) zv[i] = zr[col(i)];
            }
#pragma unroll
            for (int jj = 0; jj < R2; jj++) y[jj] = S[k1 * (R2 + 1) + jj];
            fs_dft<T, +1, R2>(y);
#pragma unroll
            for (int i = 0; i < 2 * Q2; i++) {
                const C g = y[fs_out<R2>(i < Q2 ? i : i + R2 - 2 * Q2)];
                if (col(i) >= 0 && col(i) < N1) {
                    const C v = mkc<T>(zv[i].x - alpha * g.x, zv[i].y - alpha * g.y);
                    zr[col(i)] = v;
                    s += v.x * v.x + v.y * v.y;
                }
            }
        }
    }
    const double d = block_sum_t<T>(s, sh);
    if (threadIdx.x == 0) part[(size_t)gb * part_stride + blockIdx.x] = d;
}

// ================================================================ column pass
// One CTA per tile of 4 columns of one plane, R1 threads per column, the FFTs in
// two steps, nt = R1 x R2, row l = j + R2 m: thread j < R2 does the R1-point DFT
// over m (only the first and last quarter of the rows is nonzero) and the
// twiddles W_nt^{j k1}; thread k1 the R2-point DFT over j, the product with khat
// at the frequencies k1 + R1 k2 and the R2-point inverse DFT, with the conjugate
// twiddles; thread j again the R1-point inverse DFT over k1 for the rows that
// are kept.  The middle step works in place (row k1 of the column's buffer), so
// one buffer and two barriers do; rows of R2 + 1 and columns of 4 mod 16
// elements keep every access on distinct banks.  khat's columns and the
// twiddles come through shared memory, copied in while the first step runs.
//
// Bound by latency (IPC 0.44 at 20 warps per SM).  R1 = 32 outside and the
// shorter DFT in the middle (where its input and product would both be live)
// leave registers for five CTAs per SM.  96 planes of 384 x 768: 244 us, against
// 287 for 24 x 32 with a 32-point middle (three CTAs), 314 for that as a
// persistent kernel, 238-260 for three steps of 8-, 8- and 12-point DFTs (twice
// the exchanges: bound by shared memory).
template <typename T, int R1, int R2> struct ColShape {
    static constexpr int nt = R1 * R2, RS = R2 + 1, CS = ((R1 * RS + 11) / 16) * 16 + 4;
    static constexpr size_t bytes = sizeof(cplx_t<T>) * (4 * CS + R1 * RS) + sizeof(T) * 4 * nt;
};

template <typename T, int R1, int R2>
__global__ void __launch_bounds__(4 * R1, sizeof(T) == 4 ? (R1 == 16 ? 10 : 5) : (R1 == 16 ? 4 : 2))
k_toep_cols(cplx_t<T> *H, int N0, const cplx_t<T> *__restrict__ tw,
            const T *__restrict__ khat, double *part, int part_stride, int plane0,
            bool dot)
{
    await_last();
    using C = cplx_t<T>;
    constexpr int nt = R1 * R2, RS = ColShape<T, R1, R2>::RS, CS = ColShape<T, R1, R2>::CS;
    constexpr int Q = R1 / 4, NT = 4 * R1;
    static_assert(R1 >= R2, "R1 threads per column");
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ T wsum[NT / 32];
    const int c = threadIdx.x & 3, j = threadIdx.x >> 2;
    T *kh = (T *)smraw;                       // [frequency row][column]
    C *tws = (C *)(kh + 4 * nt);              // W_nt^{j k1} at k1 RS + j
    C *S = tws + R1 * RS + c * CS;
    const int cb = blockIdx.x, b = blockIdx.y;
    for (int i = threadIdx.x; i < nt; i += NT) {
        const int k1 = i / R2, jj = i - k1 * R2;
        if constexpr (sizeof(C) == 16)
            __pipeline_memcpy_async(tws + k1 * RS + jj, tw + k1 * jj, 16);
        else
            __pipeline_memcpy_async(tws + k1 * RS + jj, tw + k1 * jj, 8);
    }
    __pipeline_commit();
    for (int i = threadIdx.x; i < nt * 4 * (int)sizeof(T) / 16; i += NT)
        __pipeline_memcpy_async((char *)kh + 16 * i, (const char *)(khat + (size_t)cb * nt * 4) + 16 * i,
                                16);
    __pipeline_commit();
    C *Hb = H + (size_t)b * N0 * nt + (size_t)cb * 4 + c;
    const int half = N0 / 2;
    C x[R1];
    if (j < R2) {
#pragma unroll
        for (int m = 0; m < R1; m++) {
            x[m] = mkc<T>(0, 0);
            if (m < Q || m >= R1 - Q) {
                const int a = j + R2 * (m < Q ? m : m - R1) + half;
                if (a >= 0 && a < N0) x[m] = Hb[(size_t)a * nt];
            }
        }
        fs_dft<T, -1, R1, true>(x);
    }
    __pipeline_wait_prior(1);
    __syncthreads();  // the twiddles
    if (j < R2) {
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) {
            C t = x[fs_out<R1>(k1)];
            if (k1) t = cmul<T>(t, tws[k1 * RS + j]);
            S[k1 * RS + j] = t;
        }
    }
    __pipeline_wait_prior(0);
    __syncthreads();
    T sum = 0;
    {
        const int k1 = j;
        C *s = S + k1 * RS, y[R2];
        const T *kp = kh + 4 * k1 + c;
#pragma unroll
        for (int i = 0; i < R2; i++) y[i] = s[i];
        fs_dft<T, -1, R2>(y);
        C z[R2];
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) {
            const C v = y[fs_out<R2>(k2)];
            const T k = kp[4 * R1 * k2];
            z[k2] = mkc<T>(k * v.x, k * v.y);
            sum += z[k2].x * v.x + z[k2].y * v.y;
        }
        fs_dft<T, +1, R2>(z);
#pragma unroll
        for (int t2 = 0; t2 < R2; t2++) {
            C v = z[fs_out<R2>(t2)];
            if (t2) {
                C w = tws[k1 * RS + t2];
                w.y = -w.y;  // inverse: e^{+2 pi i k1 t2 / nt}
                v = cmul<T>(v, w);
            }
            s[t2] = v;
        }
    }
    if (dot) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
        if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = sum;
    }
    __syncthreads();
    if (dot && threadIdx.x == 0) {
        double d = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; w++) d += (double)wsum[w];
        part[(size_t)(plane0 + b) * part_stride + cb] = d;
    }
    if (j < R2) {
#pragma unroll
        for (int k1 = 0; k1 < R1; k1++) x[k1] = S[k1 * RS + j];
        fs_dft<T, +1, R1>(x);
#pragma unroll
        for (int i = 0; i < 2 * Q; i++) {
            const int t1 = i < Q ? i : i + R1 - 2 * Q;
            const int a = j + R2 * (i < Q ? i : i - 2 * Q) + half;
            if (a >= 0 && a < N0) Hb[(size_t)a * nt] = x[fs_out<R1>(t1)];
        }
    }
}

// ================================================================ scalars
// One block per plane sums the partials in order: STEP 0 |z|^2; 1 alpha = |z|^2 /
// sum; 2 beta = sum / |z|^2 and the new |z|^2.
template <typename T, int STEP>
__global__ void __launch_bounds__(128)
k_cg_scalar(const double *part, int nparts, int stride, int plane0,
            double *dots)
{
    await_last();
    __shared__ double sh[32];
    const int gb = plane0 + blockIdx.x;
    const double *src = part + (size_t)gb * stride;
    double v = 0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) v += src[i];
    v = block_sum(v, sh);
    if (threadIdx.x == 0) {
        double *d = dots + 4 * (size_t)gb;
        if (STEP == 1) d[1] = (double)(T)(d[0] / v);
        if (STEP == 2) d[2] = (double)(T)(v / d[0]);
        if (STEP != 1) d[0] = v;
    }
}

// f += alpha p after the last step
template <typename T>
__global__ void __launch_bounds__(256)
k_cg_last(cplx_t<T> *f, const cplx_t<T> *p,
          const double *dots, int N, int plane0)
{
    await_last();
    const int gb = plane0 + blockIdx.y;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)N) return;
    const T alpha = (T)dots[4 * gb + 1];
    const size_t o = (size_t)gb * N + i;
    const cplx_t<T> pv = p[o];
    cplx_t<T> fv = f[o];
    fv.x += alpha * pv.x;
    fv.y += alpha * pv.y;
    f[o] = fv;
}

// ================================================================ setup kernels
// The operator's kernel in FP64 from the polar set's factored form: node
// (a, i) = r_i (sg_a, cg_a) and weight w_i, so K[m] = sum_a G(m0 sg_a + m1
// cg_a) with G(s) = sum_i w_i e^{2 pi i r_i s}.  G is tabulated at s_k =
// (k - K0) delta (one thread per k, the radii summed in order) and read back
// by 8-point Lagrange interpolation: G has at most half a turn per unit of s
// (|r| <= 1/2), so delta = 1/32 leaves ~1e-11 relative error.
__global__ void k_toep_gtable(const double *__restrict__ r, const double *__restrict__ w, int np,
                              double delta, int K0, int Ns, double2 *__restrict__ G)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Ns) return;
    const double sv = (k - K0) * delta;
    double re = 0, im = 0;
    for (int i = 0; i < np; i++) {
        double sn, cs;
        sincospi(2.0 * r[i] * sv, &sn, &cs);
        const double wi = w ? w[i] : 1.0;
        re = fma(wi, cs, re);
        im = fma(wi, sn, im);
    }
    G[k] = make_double2(re, im);
}

// circ[l0][l1] = K[m] for the signed indices m = (l0, l1) (mod nt) with
// |m0| < N0, |m1| < N1, else 0; the lines summed in order.  The weights are
// real, so K[-m] = conj(K[m]): a thread takes the m of rows l0 <= nt/2 (for
// row 0 and row nt/2 the columns l1 <= nt/2) and also writes -m; every entry
// is written once.
__global__ void k_toep_circ(const double2 *__restrict__ G, double delta, int K0,
                            const double *__restrict__ sg, const double *__restrict__ cg, int A,
                            int N0, int N1, int nt, double2 *__restrict__ circ)
{
    const int h = nt / 2;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)(h + 1) * nt) return;
    const int l0 = (int)(i / nt), l1 = (int)(i - (size_t)l0 * nt);
    if ((l0 == 0 || l0 == h) && l1 > h) return;  // the mirror of a column l1 < h
    const int m0 = l0 < h ? l0 : l0 - nt, m1 = l1 < h ? l1 : l1 - nt;
    double re = 0, im = 0;
    if (m0 > -N0 && m0 < N0 && m1 > -N1 && m1 < N1) {
        // reciprocals of the Lagrange weights' denominators for the nodes
        // -3..4: 1 / prod_{l != j} (j - l)
        constexpr double rden[8] = {-1.0 / 5040, 1.0 / 720, -1.0 / 240, 1.0 / 144,
                                    -1.0 / 144,  1.0 / 240, -1.0 / 720, 1.0 / 5040};
        const double inv = 1.0 / delta;
        for (int a = 0; a < A; a++) {
            const double u = fma((double)m0, sg[a], (double)m1 * cg[a]) * inv + K0;
            const double fu = floor(u);
            const double t = u - fu;  // in [0, 1): nodes at t - (j - 3)
            const int k0 = (int)fu - 3;
            double d[8], pre[8], suf[8];
#pragma unroll
            for (int j = 0; j < 8; j++) d[j] = t - (j - 3);
            pre[0] = 1.0;
#pragma unroll
            for (int j = 1; j < 8; j++) pre[j] = pre[j - 1] * d[j - 1];
            suf[7] = 1.0;
#pragma unroll
            for (int j = 6; j >= 0; j--) suf[j] = suf[j + 1] * d[j + 1];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const double wj = pre[j] * suf[j] * rden[j];
                const double2 gv = G[k0 + j];
                re = fma(wj, gv.x, re);
                im = fma(wj, gv.y, im);
            }
        }
    }
    circ[i] = make_double2(re, im);
    const int r0 = l0 ? nt - l0 : 0, r1 = l1 ? nt - l1 : 0;  // -m (mod nt)
    if (r0 != l0 || r1 != l1) circ[(size_t)r0 * nt + r1] = make_double2(re, -im);
}

// The circulant's DFT (row-major nt x nt, FP64) divided by nt^2, in the
// order k_toep_cols reads it: [block of 4 columns][frequency row][column].
template <typename T>
__global__ void k_toep_layout(const double2 *__restrict__ F, int nt, T *__restrict__ khat)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)nt * nt) return;
    const int l0 = (int)(i / nt), l1 = (int)(i - (size_t)l0 * nt);
    const double sc = 1.0 / ((double)nt * (double)nt);
    khat[((size_t)(l1 >> 2) * nt + l0) * 4 + (l1 & 3)] = (T)(F[i].x * sc);
}

// ================================================================ launches
template <typename T, int R1, int R2> struct ToepLaunch {
    using C = cplx_t<T>;
    static constexpr int nt = R1 * R2, RPC = 128 / R2;
    static constexpr size_t smem_row = sizeof(C) * RPC * row_stride<R1, R2>();
    // the column pass's split: the shorter DFT in the middle
    static constexpr int C1 = R1 > R2 ? R1 : R2, C2 = nt / C1;
    static constexpr size_t smem_col = ColShape<T, C1, C2>::bytes;

    static int init()
    {
#define NUDIM_LIMIT(k, b)                                                                        \
    NUDIM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(b)))
        NUDIM_LIMIT((k_toep_rows<T, TR_COMPLEX, R1, R2>), smem_row);
        NUDIM_LIMIT((k_toep_rows<T, TR_REAL, R1, R2>), smem_row);
        NUDIM_LIMIT((k_toep_rows<T, TR_FIRST, R1, R2>), smem_row);
        NUDIM_LIMIT((k_toep_rows<T, TR_CG, R1, R2>), smem_row);
        NUDIM_LIMIT((k_toep_irows<T, true, R1, R2>), smem_row);
        NUDIM_LIMIT((k_toep_irows<T, false, R1, R2>), smem_row);
        NUDIM_LIMIT((k_toep_cols<T, C1, C2>), smem_col);
#undef NUDIM_LIMIT
        return NUDIM_OK;
    }

    // One operator pass over planes [p0, p0 + nb): the rows in `mode`, the
    // columns, the inverse rows; the scalars each step leaves.
    static int pass(NfftDev<T> &pl, int mode, bool resid, const void *src, C *f, C *p, C *z,
                    double *part, int part_stride, double *dots, int p0, int nb, C *H,
                    cudaStream_t st)
    {
        const int N0 = pl.N0, N1 = pl.N1;
        const double c = sizeof(C), v = (double)nb * N0 * N1 * c, h = (double)nb * N0 * nt * c;
        const dim3 g(ceil_div(N0, RPC), nb);
        {
            ProfScope ps(pl.ctx, PK_TOEPLITZ, st,
                         (mode == TR_CG ? 5 : mode == TR_COMPLEX ? 1 : 2) * v + h);
#define NUDIM_ROWS(M)                                                                            \
    launch_early(k_toep_rows<T, M, R1, R2>, g, 128, smem_row, st, src, f, p, z, dots, N0, N1, \
        pl.twT, p0, H)
            if (mode == TR_COMPLEX) NUDIM_ROWS(TR_COMPLEX);
            else if (mode == TR_REAL) NUDIM_ROWS(TR_REAL);
            else if (mode == TR_FIRST) NUDIM_ROWS(TR_FIRST);
            else NUDIM_ROWS(TR_CG);
#undef NUDIM_ROWS
            NUDIM_LAUNCH_CHECK();
        }
        {
            ProfScope ps(pl.ctx, PK_TOEPLITZ, st, 2 * h + sizeof(T) * (double)nt * nt);
            launch_early(k_toep_cols<T, C1, C2>, dim3(nt / 4, nb), 4 * C1, smem_col, st, H, N0,
                         pl.twT, pl.khat, part, part_stride, p0, !resid);
            NUDIM_LAUNCH_CHECK();
            if (!resid) {
                launch_early(k_cg_scalar<T, 1>, nb, 128, 0, st, part, nt / 4, part_stride, p0,
                             dots);
                NUDIM_LAUNCH_CHECK();
            }
        }
        {
            ProfScope ps(pl.ctx, PK_TOEPLITZ, st, h + 2 * v);
            if (resid)
                launch_early(k_toep_irows<T, true, R1, R2>, g, 128, smem_row, st, H, z, dots, N0,
                             N1, pl.twT, p0, part, part_stride);
            else
                launch_early(k_toep_irows<T, false, R1, R2>, g, 128, smem_row, st, H, z, dots, N0,
                             N1, pl.twT, p0, part, part_stride);
            NUDIM_LAUNCH_CHECK();
            if (resid) launch_early(k_cg_scalar<T, 0>, nb, 128, 0, st, part, (int)g.x, part_stride,
                                    p0, dots);
            else launch_early(k_cg_scalar<T, 2>, nb, 128, 0, st, part, (int)g.x, part_stride, p0,
                              dots);
            NUDIM_LAUNCH_CHECK();
        }
        return NUDIM_OK;
    }
};

}  // namespace

// ================================================================ Toeplitz operator
// K on the circulant in FP64 (k_toep_gtable, k_toep_circ), its nt x nt DFT
// (cuFFT, FP64, once per plan; real, as K[-m] = conj K[m]), divided by nt^2 and
// laid out in the column pass's read order in the plan's precision.
template <typename T> int NfftDev<T>::toeplitz_init(const PolarGeom &g, cudaStream_t st)
{
    if (!toeplitz_fits()) {
        set_error("Toeplitz operator: needs the fused four-step path on a square grid of 256, 512 "
                  "or 1024 points");
        return NUDIM_EINVAL;
    }
    if (g.A <= 0 || (size_t)g.A * N1 != (size_t)M || !g.r || !g.sg || !g.cg) {
        set_error("Toeplitz operator: the nodes must be A lines of N1 radii");
        return NUDIM_EINVAL;
    }
    if (toeplitz) return NUDIM_OK;
    const double two_pi = 6.283185307179586;
    // the smallest supported circulant that holds |m| < N without wrap
    // (NUDIM_TOEPLITZ_GRID=nfft keeps the NFFT grid's size)
    const char *eg = getenv("NUDIM_TOEPLITZ_GRID");
    const bool small = !(eg && !strcmp(eg, "nfft"));
    const int nt = (small && 2 * N0 - 1 <= 768 && n0 > 768) ? 768 : n0;
    const size_t nn = (size_t)nt * nt;
    // G's table: |s| <= |m0| + |m1| < N0 + N1
    const double delta = 1.0 / 32;
    const int K0 = (int)std::ceil((N0 + N1) / delta) + 8, Ns = 2 * K0 + 1;
    std::vector<C> htw(nt);
    for (int k = 0; k < nt; k++) {
        const double a = -two_pi * (double)k / nt;
        htw[k] = mkc<T>((T)std::cos(a), (T)std::sin(a));
    }
    void *dr = nullptr, *dw = nullptr, *dsg = nullptr, *dcg = nullptr, *dG = nullptr, *dc = nullptr;
    void *kh = nullptr, *dtw = nullptr;
    // temporaries released stream-ordered after their last use; on failure
    // the kept buffers too
    auto done = [&](int e) {
        for (void *q : {dr, dw, dsg, dcg, dG, dc})
            if (q) cudaFreeAsync(q, st);
        if (e) {
            for (void *q : {kh, dtw})
                if (q) cudaFreeAsync(q, st);
        }
        return e;
    };
    int rc = upload_async(&dr, g.r, sizeof(double) * N1, st);
    if (!rc && g.wr) rc = upload_async(&dw, g.wr, sizeof(double) * N1, st);
    if (!rc) rc = upload_async(&dsg, g.sg, sizeof(double) * g.A, st);
    if (!rc) rc = upload_async(&dcg, g.cg, sizeof(double) * g.A, st);
    if (!rc) rc = upload_async(&dtw, htw.data(), sizeof(C) * htw.size(), st);
    if (rc) return done(rc);
    if (cudaMallocAsync(&dG, sizeof(double2) * Ns, st) != cudaSuccess ||
        cudaMallocAsync(&dc, sizeof(double2) * nn, st) != cudaSuccess ||
        cudaMallocAsync(&kh, sizeof(T) * nn, st) != cudaSuccess) {
        set_error("Toeplitz operator: out of device memory");
        return done(NUDIM_ECUDA);
    }
    k_toep_gtable<<<(unsigned)ceil_div(Ns, 128), 128, 0, st>>>((const double *)dr,
                                                               (const double *)dw, N1, delta, K0,
                                                               Ns, (double2 *)dG);
    ++g_launches;
    k_toep_circ<<<(unsigned)ceil_div((long)(nt / 2 + 1) * nt, 128), 128, 0, st>>>(
        (const double2 *)dG, delta, K0, (const double *)dsg, (const double *)dcg, g.A, N0, N1, nt,
        (double2 *)dc);
    ++g_launches;
    if (cudaGetLastError() != cudaSuccess) {
        set_error("Toeplitz operator: setup kernel launch failed");
        return done(NUDIM_ECUDA);
    }
    cufftHandle h;
    if ((rc = ctx_fft2d(ctx, nt, nt, 1, NUDIM_FP64, &h))) return done(rc);
    if (cufftSetStream(h, st) != CUFFT_SUCCESS) {
        set_error("Toeplitz operator: cufftSetStream failed");
        return done(NUDIM_ECUDA);
    }
    if ((rc = fft_exec<double>(h, (double2 *)dc, CUFFT_FORWARD))) return done(rc);
    k_toep_layout<T><<<(unsigned)ceil_div((long)nn, 256), 256, 0, st>>>((const double2 *)dc, nt,
                                                                         (T *)kh);
    ++g_launches;
    if (cudaGetLastError() != cudaSuccess) {
        set_error("Toeplitz operator: setup kernel launch failed");
        return done(NUDIM_ECUDA);
    }
    NUDIM_TRY((ToepLaunch<T, 32, 32>::init()));
    NUDIM_TRY((ToepLaunch<T, 24, 32>::init()));
    NUDIM_TRY((ToepLaunch<T, 32, 16>::init()));
    NUDIM_TRY((ToepLaunch<T, 16, 16>::init()));
    done(NUDIM_OK);
    khat = (T *)kh;
    nT = nt;
    twT = (C *)dtw;
    bytes += sizeof(T) * nn + sizeof(C) * nt;
    toeplitz = true;
    return NUDIM_OK;
}

// CGNR's iterations in coefficient space (see cgnr_run): z holds A^H W y, f the
// start value (or f_real, or nothing: f is zero and part the adjoint's |z|^2
// partials).
template <typename T>
int NfftDev<T>::toeplitz_cg(int nplanes, C *f, const T *f_real, bool f_zero, int iters, C *z, C *p,
                            double *part, int part_stride, double *dots, cudaStream_t st)
{
    if (!toeplitz) {
        set_error("Toeplitz operator not initialised");
        return NUDIM_ESTATE;
    }
    if (part_stride < nT / 4) {
        set_error("Toeplitz operator: partial buffer too small");
        return NUDIM_EINVAL;
    }
    // (all planes at once where the budget allows: chunks small enough for the
    // spectra to stay in L2 were slower, 96 planes of 384^2 in chunks of 16 6.3
    // against 5.1 ms per iteration)
    const int chunk = fused_chunk(nplanes, (size_t)N0 * nT);
    void *wsv;
    NUDIM_TRY(workspace(sizeof(C) * (size_t)N0 * nT * chunk, &wsv));
    C *H = (C *)wsv;
    auto pass = [&](int mode, bool resid, int p0, int nb) -> int {
        const void *src = f_real ? (const void *)f_real : (const void *)f;
        switch (nT) {
        case 1024:
            return ToepLaunch<T, 32, 32>::pass(*this, mode, resid, src, f, p, z, part, part_stride,
                                               dots, p0, nb, H, st);
        case 768:
            return ToepLaunch<T, 24, 32>::pass(*this, mode, resid, src, f, p, z, part, part_stride,
                                               dots, p0, nb, H, st);
        case 512:
            return ToepLaunch<T, 32, 16>::pass(*this, mode, resid, src, f, p, z, part, part_stride,
                                               dots, p0, nb, H, st);
        default:
            return ToepLaunch<T, 16, 16>::pass(*this, mode, resid, src, f, p, z, part, part_stride,
                                               dots, p0, nb, H, st);
        }
    };
    const int N = N0 * N1;
    for (int p0 = 0; p0 < nplanes; p0 += chunk) {
        const int nb = std::min(chunk, nplanes - p0);
        if (f_zero) {
            launch_early(k_cg_scalar<T, 0>, nb, 128, 0, st, part, crop_blocks(), part_stride, p0,
                         dots);
            NUDIM_LAUNCH_CHECK();
        } else {
            NUDIM_TRY(pass(f_real ? TR_REAL : TR_COMPLEX, true, p0, nb));
        }
        for (int it = 0; it < iters; it++) NUDIM_TRY(pass(it ? TR_CG : TR_FIRST, false, p0, nb));
        if (iters > 0) {
            ProfScope ps(ctx, PK_CGVEC, st, 3.0 * sizeof(C) * (double)N * nb);
            launch_early(k_cg_last<T>, dim3(ceil_div(N, 256), nb), 256, 0, st, f, p, dots, N, p0);
            NUDIM_LAUNCH_CHECK();
        }
    }
    return NUDIM_OK;
}

template int NfftDev<double>::toeplitz_init(const PolarGeom &, cudaStream_t);
template int NfftDev<float>::toeplitz_init(const PolarGeom &, cudaStream_t);
template int NfftDev<double>::toeplitz_cg(int, double2 *, const double *, bool, int, double2 *,
                                          double2 *, double *, int, double *, cudaStream_t);
template int NfftDev<float>::toeplitz_cg(int, float2 *, const float *, bool, int, float2 *,
                                         float2 *, double *, int, double *, cudaStream_t);

}  // namespace nudim
