// denoise.cu -- TV-discrete (and its height-window variant) and the in-place
// 2D anisotropic diffusion of denoise.c, on [z][y][x] volumes.
//
// Arithmetic uses round-to-nearest intrinsics (no contraction) so that the
// FP64 form reproduces the reference's per-voxel C arithmetic exactly; only
// the two global sums of TV are summed in a different (tree) order.  The
// FP32 form uses fused multiply-adds, rsqrt and fast division where noted.
#include "engine.cuh"
#include "intdiv.cuh"

#include <cuda_pipeline.h>

#include <cstdlib>
#include <cstring>
#include <type_traits>

namespace nudim {

// ================================================================ TV
// denoise.c:67-151 / 153-249 called as total_variation_discrete(img, lam,
// niter, nz, np, np): the reference's i runs over Z, j over Y, k over X.
//
// One TV iteration is two launches:
//   k_tv_grad   the gradient g of every voxel and the two global sums
//               (G = sum g^2, N = sum of squares of the negative voxels).  The four
//               quotients of a voxel's gradient have the norms of the voxel
//               itself and of its three upper neighbours: each voxel's norm
//               is formed once, and the neighbours get its quotients (the
//               same operations on the same values as four norms per voxel).  A block owns a 32 x 16 (x, y) tile and a
//               run of Z-planes and marches along Z: per plane the tile with
//               a one-cell halo in shared memory (clamped neighbours: index
//               -1 -> 0, n -> n-1, the reference's boundary rules, whose
//               differences are zero), copied in asynchronously two or three
//               planes ahead; what the lower neighbours need goes through
//               shared memory (FP64: the Y and X terms, FP32: the reciprocal
//               norm), the Z part waits for the next plane; the row and
//               column beyond the tile are formed by 48 threads more.
//               The block that finishes last sums the per-block partials in
//               block order (deterministic) and leaves step[0] = sqrt(G),
//               step[1] = lam sqrt(N) in the volume's precision (the two
//               square roots once: in the blocks that use them they held the
//               FP64 unit 1.6 us a block);
//   k_tv_update u -= step[1] (g / step[0]).
// FP64: the square root and the quotients in integer arithmetic (intdiv.cuh;
// same bits), 15 operations of the FP64 unit a voxel left of about 110.
constexpr int kTvTX = 32, kTvTY = 16, kTvSX = kTvTX + 2, kTvSY = kTvTY + 2;
constexpr int kTvRows = kTvTY / 8;  // rows per thread (256 threads = 8 warps of 32 x)

// A voxel's terms from its differences to the lower neighbours (denoise.c:
// 84-122): (z + y + x) / norm and each difference / norm, norm = sqrt(1e-8 +
// z^2 + y^2 + x^2).
template <typename T> struct TvTerms {
    T sum, z, y, x;
};

__device__ __noinline__ TvTerms<double> tv_terms_divided(double z, double y, double x)
{
    const double n = rn_sqrt(
        rn_add(rn_add(rn_add(1e-8, rn_mul(z, z)), rn_mul(y, y)), rn_mul(x, x)));
    return {rn_div(rn_add(rn_add(z, y), x), n), rn_div(z, n), rn_div(y, n), rn_div(x, n)};
}

__device__ __forceinline__ TvTerms<double> tv_terms(double z, double y, double x)
{
    double z2, y2, x2;
    bool ok = int_square(z, &z2);
    ok &= int_square(y, &y2);
    ok &= int_square(x, &x2);
    const IntDivisor n = int_sqrt(rn_add(rn_add(rn_add(1e-8, z2), y2), x2));
    TvTerms<double> t;
    ok &= int_div(rn_add(rn_add(z, y), x), n, &t.sum);
    ok &= int_div(z, n, &t.z);
    ok &= int_div(y, n, &t.y);
    ok &= int_div(x, n, &t.x);
    if (!ok) t = tv_terms_divided(z, y, x);
    return t;
}

// FP32: t / sqrt(...) as t * rsqrt(...) with fused multiply-adds (a few ulp per
// term, against one for IEEE sqrt and division; the TV loop's own amplification
// of rounding dominates).
__device__ __forceinline__ float tv_inv(float z, float y, float x)
{
    return rsqrtf(__fmaf_rn(x, x, __fmaf_rn(y, y, __fmaf_rn(z, z, 1e-8f))));
}

// An update's la (g / b), b the gradient's norm, rounded as the division and the
// product round (intdiv.cuh; |g| is below 5).
__device__ __noinline__ double tv_divided(double a, double b) { return rn_div(a, b); }

template <typename T> struct TvNorm;
template <> struct TvNorm<float> {
    float b, y, la;  // la: the factor, times 2^-64 where y is not 0
    __device__ void init(float v, float l)
    {
        b = v;
        y = v > 1e-15f && v < 1e15f && l > 0x1p-60f ? __frcp_rn(v) : 0.f;
        la = y == 0.f ? l : l * 0x1p-64f;
    }
    __device__ __forceinline__ float step(float g) const
    {
        if (y == 0.f) return rn_mul(la, rn_div(g, b));  // the same for the whole launch
        return rn_mul(la, quotient64(g, b, y));
    }
};
template <> struct TvNorm<double> {
    double b, la;
    IntDivisor d;
    bool ok;
    __device__ void init(double v, double l)
    {
        b = v;
        la = l;
        ok = v > 1e-300 && v < 1e300;
        d = int_divisor(ok ? v : 1.0);
    }
    __device__ __forceinline__ double step(double g) const
    {
        double q;
        if (!(int_div(g, d, &q) && ok)) q = tv_divided(g, b);
        return rn_mul(la, q);
    }
};

// A thread's running sums of squares (gradients, negative voxels), a voxel at a
// time: plain in the FP64 form, compensated in the FP32 form (a thread sums two
// terms per plane of its Z-run; each addition's rounding error
// exactly, by Knuth's two-sum), the two sums as a pair.
template <typename T> struct TvAcc;
template <> struct TvAcc<double> {
    double g = 0, n = 0;
    __device__ __forceinline__ void add_sq(double a, double b)
    {
        g = rn_add(g, square_rn(a));
        n = rn_add(n, square_rn(b));
    }
    __device__ __forceinline__ double grad() const { return g; }
    __device__ __forceinline__ double neg() const { return n; }
};
template <> struct TvAcc<float> {
    float2 s = make_float2(0.f, 0.f), e = make_float2(0.f, 0.f);
    __device__ __forceinline__ void add_sq(float a, float b)
    {
        // (a product as a fused multiply-add to -0 stays a product: the
        // compiler would fold it into the additions)
        const float2 m1 = make_float2(-1.f, -1.f), z = make_float2(-0.f, -0.f);
        const float2 v = make_float2(a, b), x = __ffma2_rn(v, v, z);
        const float2 t = __fadd2_rn(s, x), c = __ffma2_rn(m1, s, t);
        const float2 d = __ffma2_rn(m1, c, t);
        e = __fadd2_rn(e, __fadd2_rn(__ffma2_rn(m1, d, s), __ffma2_rn(m1, c, x)));
        s = t;
    }
    __device__ __forceinline__ float grad() const { return rn_add(s.x, e.x); }
    __device__ __forceinline__ float neg() const { return rn_add(s.y, e.y); }
};

// Blocks per SM that the cut into Z-runs (and so the order of the sums) assumes;
// and that the kernel runs at (registers).
template <typename T> constexpr int kTvSumBlocks = sizeof(T) == 4 ? 4 : 3;

// block_sum_t of two values of a block of 256 with one pair of barriers (the same
// sums)
template <typename T> __device__ __forceinline__ double2 block_sum2(T a, T b, double2 *sh)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    __syncthreads();
    if (lane == 0) sh[wid] = make_double2((double)a, (double)b);
    __syncthreads();
    double2 v = make_double2(0, 0);
    if (wid == 0) {
        if (threadIdx.x < 8) v = sh[threadIdx.x];
        // (from 4 on: at 16 and 8 the other lanes' zeros would be added)
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            v.x += __shfl_down_sync(0xffffffffu, v.x, o);
            v.y += __shfl_down_sync(0xffffffffu, v.y, o);
        }
    }
    return v;
}

// sqrt of a sum on one thread at the end of a pass, where nothing hides the FP64
// unit's latency: in integers (16 x 48 x 40, 40 steps: 404 -> 390 us)
__device__ __forceinline__ double tv_root(double s)
{
    return s > 1e-300 && s < 1e300 ? double_of(int_sqrt(s)) : sqrt(s);
}

// The two sums: FP64 products and sums in the FP64 form; FP32 products and
// compensated per-thread sums, FP32 warp sums and FP64 across warps and
// blocks in the FP32 form, one partial per tile and run of zc planes.  Grid (x
// tiles, y tiles, groups of `rep` consecutive runs of `runs`);
// 256 threads, thread (ty, tx) owns the columns (j0 + ty + 8 r, k0 + tx),
// r < kTvRows.  done: a zeroed counter (the last block resets it).
//
// FUSED: the previous iteration's update is applied as the tile is read
// (u' = u - step_in[1] (g_in / step_in[0]) on every tile and halo cell, with
// k_tv_update's operations), the owned cells' u' are written to u_out and the gradient of u' to g: one pass reads u and g_in and
// writes u' and g (4 values per voxel instead of the 5 of a gradient and an
// update).  u_out and g must not alias u and g_in (other blocks still read
// their halos).  I: the index within a plane.
template <typename T, bool FUSED, typename I>
__global__ void __launch_bounds__(256, kTvSumBlocks<T>)
k_tv_grad(const T *u, T *g, double *part,
          unsigned *done, double *step, int nz, int ny, int nx,
          int zc, int runs, int rep, int height, int ylo, int yhi, const T *g_in,
          const double *step_in, double lam, T *u_out)
{
    constexpr int kCells = kTvSY * kTvSX, kSlots = (kCells + 255) / 256;
    constexpr bool FLOAT = sizeof(T) == 4;
    constexpr int NS = FLOAT ? 4 : 3;  // planes of the ring: p, p + 1, and those in flight
    constexpr int US = FLOAT ? 4 : 6;  // steps per loop turn (ring slot and parity constant)
    __shared__ T pl[NS][kTvSY][kTvSX];
    __shared__ T plg[FUSED ? NS : 1][FUSED ? kCells : 1];
    // of the tile's voxels and of the row and column beyond, by plane parity:
    // FP64 the Y and X terms, FP32 the reciprocal norm (in py, one wider)
    __shared__ T py[2][kTvTY + 1][kTvTX + FLOAT], px[2][FLOAT ? 1 : kTvTY][kTvTX + 1];
    __shared__ double2 sh[32];
    __shared__ int s_last;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int k0 = blockIdx.x * kTvTX, j0 = blockIdx.y * kTvTY;
    const int z0 = blockIdx.z * rep * zc, z1 = min(nz, z0 + rep * zc);
    const int k = k0 + tx;
    bool own[kTvRows], inb[kTvRows];
#pragma unroll
    for (int r = 0; r < kTvRows; r++) {
        const int j = j0 + ty + 8 * r;
        inb[r] = k < nx && j < ny;
        own[r] = inb[r] && (!height || (j >= ylo && j <= yhi));
    }
    const size_t P = (size_t)ny * nx;
    const I my = (I)(j0 + ty) * nx + k, my8 = my + (I)8 * nx;  // this thread's voxels
    // this thread's halo-tile cells (threadIdx + 256 s), their clamped in-plane
    // offsets and (FUSED) whether the update applies to their row
    I off[kSlots];
    bool upd[kSlots];
#pragma unroll
    for (int s = 0; s < kSlots; s++) {
        const int c = threadIdx.x + 256 * s, yy = c / kTvSX, xx = c - yy * kTvSX;
        const int gj = min(max(j0 + yy - 1, 0), ny - 1), gk = min(max(k0 + xx - 1, 0), nx - 1);
        off[s] = (I)gj * nx + gk;
        upd[s] = c < kCells && (!height || (gj >= ylo && gj <= yhi));
    }
    T *const cells = &pl[0][0][0] + threadIdx.x, *const gcells = &plg[0][0] + threadIdx.x;
    // the planes of the run in order (the first and last clamped to the volume)
    // into ring slot `sl`; past the run's end only the group's count goes on
    const T *fu = u + (size_t)max(z0 - 1, 0) * P, *fg = g_in + (size_t)max(z0 - 1, 0) * P;
    int fq = z0 - 1;
    auto fetch = [&](int sl) {
        if (fq <= z1) {
#pragma unroll
            for (int s = 0; s < kSlots; s++)
                if (s + 1 < kSlots || threadIdx.x < kCells - 256 * (kSlots - 1)) {
                    __pipeline_memcpy_async(cells + sl * kCells + 256 * s, fu + off[s], sizeof(T));
                    if (FUSED)
                        __pipeline_memcpy_async(gcells + sl * kCells + 256 * s, fg + off[s],
                                                sizeof(T));
                }
            if (fq >= 0 && fq + 1 < nz) {
                fu += P;
                fg += P;
            }
            fq++;
        }
        __pipeline_commit();
    };
    await_last();
    TvNorm<T> norm;
    // u' in slot `sl`: each thread its own cells, so its own copies' arrival is
    // all it waits for
    auto ready = [&](int sl) {
        if (FUSED) {
#pragma unroll
            for (int s = 0; s < kSlots; s++)
                if (upd[s]) {
                    T *v = cells + sl * kCells + 256 * s;
                    *v = rn_sub(*v, norm.step(gcells[sl * kCells + 256 * s]));
                }
        }
    };
    // the voxel beyond the tile that this thread forms: row kTvTY (warp 0),
    // column kTvTX (half of warp 1)
    const bool extra = threadIdx.x < kTvTX + kTvTY;
    const int ey = threadIdx.x < kTvTX ? kTvTY : threadIdx.x - kTvTX;
    const int ex = threadIdx.x < kTvTX ? threadIdx.x : kTvTX;
    for (int q = 0; q < NS; q++) fetch(q);  // planes z0 - 1 .. z0 + NS - 2
    __pipeline_wait_prior(NS - 2);
    if (FUSED) {
        norm.init((T)step_in[0], (T)step_in[1]);
    }
    ready(0);
    ready(1);
    __syncthreads();
    // the plane below, and the finished plane's parts waiting for the next: its
    // own (FP64 quotient; FP32 sum of differences and reciprocal norm), its upper
    // neighbours' (FP64 terms; FP32 differences and reciprocal norms)
    T below[kTvRows], cen[kTvRows], hs[kTvRows], hi[kTvRows], hy[kTvRows], hx[kTvRows];
    T dy[kTvRows], dx[kTvRows], ebelow = T(0);
#pragma unroll
    for (int r = 0; r < kTvRows; r++) {
        below[r] = pl[0][ty + 8 * r + 1][tx + 1];
        cen[r] = hs[r] = hi[r] = hy[r] = hx[r] = dy[r] = dx[r] = T(0);
    }
    if (extra) ebelow = pl[0][ey + 1][ex + 1];
    TvAcc<T> acc;
    // a finished run's partial sums
    const unsigned nblk = gridDim.x * gridDim.y * runs;
    int run = blockIdx.z * rep, next = z0 + zc;
    auto emit = [&]() {
        const unsigned bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * run);
        const double2 b = block_sum2<T>(acc.grad(), acc.neg(), sh);
        if (threadIdx.x == 0) {
            part[bid] = b.x;
            part[nblk + bid] = b.y;
        }
        acc = TvAcc<T>();
        run++;
        next += zc;
    };
    T *gp = g + (size_t)z0 * P, *up = FUSED ? u_out + (size_t)z0 * P : nullptr;
    static_assert(kTvRows == 2, "two rows a thread");
    auto finish = [&](T g0, T g1) {  // the finished plane's gradient
        if (own[0]) gp[my] = g0;
        if (own[1]) gp[my8] = g1;
        gp += P;
        acc.add_sq(own[0] ? g0 : T(0), own[0] && cen[0] < T(0) ? cen[0] : T(0));
        acc.add_sq(own[1] ? g1 : T(0), own[1] && cen[1] < T(0) ? cen[1] : T(0));
    };
    // one step: plane p in slot (S + 1) mod NS
    auto advance = [&](int p, auto sc) {
        constexpr int S = decltype(sc)::value, sl = (S + 1) % NS, pb = S & 1;
        const T(*q)[kTvSX] = pl[sl];
        T c[kTvRows];
#pragma unroll
        for (int r = 0; r < kTvRows; r++) c[r] = q[ty + 8 * r + 1][tx + 1];
        if constexpr (FLOAT) {
            // two voxels at once, each operation paired.  The own quotient
            // joins the sum unrounded, the neighbours' are rounded products
            // (multiply-adds to -0, which the compiler does not fold on)
            auto f2 = [](float a, float b) { return make_float2(a, b); };
            auto prod = [&](float2 a, float2 b) { return __ffma2_rn(a, b, f2(-0.f, -0.f)); };
            auto sub = [&](float2 a, float2 b) { return __fadd2_rn(a, f2(-b.x, -b.y)); };
            const float2 c2 = f2(c[0], c[1]);
            const float2 tz = sub(c2, f2(below[0], below[1]));
            const float2 ty2 = sub(c2, f2(q[ty][tx + 1], q[ty + 8][tx + 1]));
            const float2 tx2 = sub(c2, f2(q[ty + 1][tx], q[ty + 9][tx]));
            const float2 s = __ffma2_rn(
                tx2, tx2, __ffma2_rn(ty2, ty2, __ffma2_rn(tz, tz, f2(1e-8f, 1e-8f))));
            const float2 inv = f2(rsqrtf(s.x), rsqrtf(s.y));
            if (p > z0) {
                // the plane below is complete with this plane's Z difference and norm
                const float2 hz = prod(tz, inv);
                float2 g2 = __ffma2_rn(f2(hs[0], hs[1]), f2(hi[0], hi[1]), f2(-hz.x, -hz.y));
                g2 = sub(g2, prod(f2(dy[0], dy[1]), f2(hy[0], hy[1])));
                g2 = sub(g2, prod(f2(dx[0], dx[1]), f2(hx[0], hx[1])));
                finish(g2.x, g2.y);
            }
            const float2 h = __fadd2_rn(__fadd2_rn(tz, ty2), tx2);
            hs[0] = h.x;
            hs[1] = h.y;
            hi[0] = inv.x;
            hi[1] = inv.y;
            py[pb][ty][tx] = inv.x;
            py[pb][ty + 8][tx] = inv.y;
            if (extra) {
                const float ce = q[ey + 1][ex + 1];
                py[pb][ey][ex] = tv_inv(rn_sub(ce, ebelow), rn_sub(ce, q[ey][ex + 1]),
                                        rn_sub(ce, q[ey + 1][ex]));
                ebelow = ce;
            }
        } else {
            TvTerms<T> t[kTvRows];
#pragma unroll
            for (int r = 0; r < kTvRows; r++)
                t[r] = tv_terms(rn_sub(c[r], below[r]), rn_sub(c[r], q[ty + 8 * r][tx + 1]),
                                rn_sub(c[r], q[ty + 8 * r + 1][tx]));
            if (p > z0)
                finish(rn_sub(rn_sub(rn_sub(hs[0], t[0].z), hy[0]), hx[0]),
                       rn_sub(rn_sub(rn_sub(hs[1], t[1].z), hy[1]), hx[1]));
#pragma unroll
            for (int r = 0; r < kTvRows; r++) {
                hs[r] = t[r].sum;
                py[pb][ty + 8 * r][tx] = t[r].y;
                px[pb][ty + 8 * r][tx] = t[r].x;
            }
            if (extra && p < z1) {
                const T ce = q[ey + 1][ex + 1];
                const TvTerms<T> te = tv_terms(rn_sub(ce, ebelow), rn_sub(ce, q[ey][ex + 1]),
                                               rn_sub(ce, q[ey + 1][ex]));
                if (ey == kTvTY) py[pb][kTvTY][ex] = te.y;
                else px[pb][ey][kTvTX] = te.x;
                ebelow = ce;
            }
        }
        if (p == z1) return;
        if (!FLOAT && p == next) emit();  // (FP32 blocks have one run)
#pragma unroll
        for (int r = 0; r < kTvRows; r++) {
            if (FUSED && inb[r]) up[r ? my8 : my] = c[r];
            cen[r] = below[r] = c[r];
        }
        if (FUSED) up += P;
        __pipeline_wait_prior(NS - 3);  // plane p + 1 is here
        ready((sl + 1) % NS);
        __syncthreads();
        fetch(S % NS);  // plane p + NS - 1 over plane p - 1, which has no reader left
#pragma unroll
        for (int r = 0; r < kTvRows; r++) {
            hy[r] = py[pb][ty + 8 * r + 1][tx];
            if constexpr (FLOAT) {
                hx[r] = py[pb][ty + 8 * r][tx + 1];
                dy[r] = rn_sub(q[ty + 8 * r + 2][tx + 1], c[r]);
                dx[r] = rn_sub(q[ty + 8 * r + 1][tx + 2], c[r]);
            } else {
                hx[r] = px[pb][ty + 8 * r][tx + 1];
            }
        }
    };
    for (int p = z0; p <= z1; p += US) {
        advance(p, std::integral_constant<int, 0>());
        if (p + 1 <= z1) advance(p + 1, std::integral_constant<int, 1>());
        if (p + 2 <= z1) advance(p + 2, std::integral_constant<int, 2>());
        if (p + 3 <= z1) advance(p + 3, std::integral_constant<int, 3>());
        if constexpr (US == 6) {
            if (p + 4 <= z1) advance(p + 4, std::integral_constant<int, 4>());
            if (p + 5 <= z1) advance(p + 5, std::integral_constant<int, 5>());
        }
    }
    __pipeline_wait_prior(0);
    emit();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(done, 1u) == gridDim.x * gridDim.y * gridDim.z - 1;
    }
    __syncthreads();
    if (!s_last) return;
    // the last block: every block's partials are visible (fence before the
    // count); sum them in block order, the same order whichever block is last,
    // and leave the step's two numbers, a square root each on two warps
    __threadfence();
    double2 b = make_double2(0, 0);
    for (int t = threadIdx.x; t < (int)nblk; t += blockDim.x) {
        b.x += __ldcg(part + t);
        b.y += __ldcg(part + nblk + t);
    }
    b = block_sum2<double>(b.x, b.y, sh);
    if (threadIdx.x == 0) {
        sh[0] = b;
        *done = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) step[0] = (double)(T)tv_root(sh[0].x);
    if (threadIdx.x == 32) step[1] = (double)(T)(lam * tv_root(sh[0].y));
}

template <typename T, int N> struct alignas(sizeof(T) * N) TvVec {
    T v[N];
};

// u_out = u - (lam * sqrt(dA)) * (g / sqrt(sum g^2))   (denoise.c:125-142),
// VEC voxels per access; u_out may be u.  step: the norm and the factor, as the
// gradient pass left them.
template <typename T, typename I, int VEC>
__global__ void __launch_bounds__(256)
k_tv_update(const T *u, T *u_out, const T *g, const double *step,
            int nz, int ny, int nx, int height, int ylo, int yhi)
{
    await_last();
    TvNorm<T> tn;
    tn.init((T)step[0], (T)step[1]);
    const I nv = (I)nz * ny * nx / VEC, stride = (I)gridDim.x * blockDim.x;
    for (I t = (I)blockIdx.x * blockDim.x + threadIdx.x; t < nv; t += stride) {
        TvVec<T, VEC> x = reinterpret_cast<const TvVec<T, VEC> *>(u)[t];
        const TvVec<T, VEC> y = reinterpret_cast<const TvVec<T, VEC> *>(g)[t];
#pragma unroll
        for (int e = 0; e < VEC; e++) {
            if (height) {
                int j = (int)(((t * VEC + e) / (I)nx) % (I)ny);
                if (j < ylo || j > yhi) continue;
            }
            x.v[e] = rn_sub(x.v[e], tn.step(y.v[e]));
        }
        reinterpret_cast<TvVec<T, VEC> *>(u_out)[t] = x;
    }
}

// Per-block partial sums of k_tv_grad (two per block; at most one block per
// tile and plane) and the completion counter.
int tv_part_count(int nz, int ny, int nx)
{
    return 2 * ceil_div(nx, kTvTX) * ceil_div(ny, kTvTY) * nz + 2;
}

// Fused passes (FP32 default) or a gradient and a separate update per
// iteration (FP64 default: the FP64 gradient is bound by the FP64 pipe, and
// the folded update made it slower than the two launches); NUDIM_TV=
// fused|unfused selects one.  The same values bit for bit; read at every call.
template <typename T> static bool tv_unfused()
{
    const char *e = getenv("NUDIM_TV");
    if (e && !strcmp(e, "unfused")) return true;
    if (e && !strcmp(e, "fused")) return false;
    return sizeof(T) == 8;
}

// I: the index of a voxel in the volume; G: within a plane
template <typename T, typename I, typename G>
static int tv_launch(T *u, T *grad, double *part, int part_cap, double *scal, size_t V, int nz,
                     int ny, int nx, float lam, int niter, int height, int ylo, int yhi,
                     T *u2, T *g2, cudaStream_t st)
{
    int dev = 0, sms = 0;
    NUDIM_CUDA(cudaGetDevice(&dev));
    NUDIM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // Z-runs, one partial sum each: about two resident waves of blocks, runs of
    // at least 4 planes (each run re-reads two planes beyond its ends)
    const long tiles = (long)ceil_div(nx, kTvTX) * ceil_div(ny, kTvTY);
    const long want = 2L * sms * kTvSumBlocks<T>;
    const int most = (int)std::max(1L, std::min((long)nz / 4, (long)ceil_div(want, tiles)));
    const int zc = ceil_div(nz, most), runs = ceil_div(nz, zc);
    // FP64: as many consecutive runs per block as leave one wave (a block forms
    // the terms of a plane beyond its last run: 128^3, two runs a block 6.4 -> 5.1
    // ms)
    const int rep = sizeof(T) == 8
                        ? (int)std::max(1L, (tiles * runs + sms * kTvSumBlocks<T> - 1) /
                                                (sms * kTvSumBlocks<T>))
                        : 1;
    const dim3 gg(ceil_div(nx, kTvTX), ceil_div(ny, kTvTY), ceil_div(runs, rep));
    const long nb = tiles * runs;
    if (part_cap < 2 * nb + 1) {
        set_error("tv_run: partial buffer too small");
        return NUDIM_EINVAL;
    }
    unsigned *done = reinterpret_cast<unsigned *>(part + 2 * nb);
    NUDIM_CUDA(cudaMemsetAsync(done, 0, sizeof(unsigned), st));
    constexpr int W = 16 / sizeof(T);
    const long nu1 = std::min((long)ceil_div((long)V, 256), (long)sms * 8);
    const long nuw = std::min((long)ceil_div((long)(V / W), 256), (long)sms * 8);
    auto wide = [&](const T *a, const T *b, const T *c) {
        return V % W == 0 && (reinterpret_cast<uintptr_t>(a) % 16) == 0 &&
               (reinterpret_cast<uintptr_t>(b) % 16) == 0 &&
               (reinterpret_cast<uintptr_t>(c) % 16) == 0;
    };
    // u_out = u - step(g, scal): the widest access that divides the volume and
    // the pointers' alignment
    auto update = [&](const T *uin, T *uout, const T *gv, const double *sc) -> int {
        if (wide(uin, uout, gv))
            launch_early(k_tv_update<T, I, W>, (int)nuw, 256, 0, st, uin, uout, gv, sc, nz, ny, nx,
                         height, ylo, yhi);
        else
            launch_early(k_tv_update<T, I, 1>, (int)nu1, 256, 0, st, uin, uout, gv, sc, nz, ny, nx,
                         height, ylo, yhi);
        NUDIM_LAUNCH_CHECK();
        return NUDIM_OK;
    };
    if (niter <= 0) return NUDIM_OK;
    if (!u2 || !g2 || niter < 2 || tv_unfused<T>()) {
        for (int it = 0; it < niter; it++) {
            k_tv_grad<T, false, G><<<gg, 256, 0, st>>>(u, grad, part, done, scal, nz, ny, nx, zc,
                                                    runs, rep, height, ylo, yhi, nullptr, nullptr,
                                                    (double)lam, nullptr);
            NUDIM_LAUNCH_CHECK();
            NUDIM_TRY(update(u, u, grad, scal));
        }
        return NUDIM_OK;
    }
    // fused: the gradient of u, then niter - 1 passes that update with the
    // previous gradient and take the next one (volumes and gradients alternate
    // between (u, grad) and (u2, g2), the sums between scal[0..1] and
    // scal[2..3]), then the last update into u
    k_tv_grad<T, false, G><<<gg, 256, 0, st>>>(u, grad, part, done, scal, nz, ny, nx, zc, runs, rep,
                                            height, ylo, yhi, nullptr, nullptr, (double)lam, nullptr);
    NUDIM_LAUNCH_CHECK();
    T *cu = u, *cg = grad;
    double *cs = scal;
    for (int it = 1; it < niter; it++) {
        T *nu = cu == u ? u2 : u, *ng = cg == grad ? g2 : grad;
        double *ns = cs == scal ? scal + 2 : scal;
        launch_early(k_tv_grad<T, true, G>, gg, 256, 0, st, cu, ng, part, done, ns, nz, ny, nx, zc,
                     runs, rep, height, ylo, yhi, cg, cs, (double)lam, nu);
        NUDIM_LAUNCH_CHECK();
        cu = nu;
        cg = ng;
        cs = ns;
    }
    return update(cu, u, cg, cs);
}

template <typename T>
int tv_run(T *u, T *grad, double *part, int part_cap, double *scal, int nz, int ny, int nx,
           float lam, int niter, int height, int ylo, int yhi, cudaStream_t st, T *u2, T *g2)
{
    size_t V = (size_t)nz * ny * nx;
    if (V == 0 || niter <= 0) return NUDIM_OK;
    // 32-bit voxel indices while index + grid stride stays below 2^32, within a
    // plane while the plane does
    const bool plane32 = (size_t)ny * nx <= ((size_t)1 << 32);
    auto run = V < ((size_t)1 << 31) ? tv_launch<T, unsigned, unsigned>
               : plane32             ? tv_launch<T, size_t, unsigned>
                                     : tv_launch<T, size_t, size_t>;
    return run(u, grad, part, part_cap, scal, V, nz, ny, nx, lam, niter, height, ylo, yhi, u2, g2,
               st);
}

// ================================================================ diffusion
// One cell of denoise.c:320-378.  FP64: the reference's 1 / (1 + g^2 / K^2)
// with IEEE operations in its order (bit-identical).  FP32 form: the same
// coefficient as K^2 / (K^2 + g^2) with a fast division (relative error a few
// ulp per cell).
__device__ __forceinline__ double diff_coef(double g, double Ksq)
{
    return rn_div(1.0, rn_add(1.0, rn_div(rn_mul(g, g), Ksq)));
}
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float diff_coef(float g, float Ksq)
{
    return Ksq * rcp_approx(fmaf(g, g, Ksq));
}

template <typename T>
__device__ __forceinline__ T diff_cell(T cv, T nN, T nS, T nE, T nW, T lambda, T Ksq)
{
    T gN = rn_sub(nN, cv), gS = rn_sub(nS, cv), gE = rn_sub(nE, cv), gW = rn_sub(nW, cv);
    T cN = diff_coef(gN, Ksq), cS = diff_coef(gS, Ksq), cE = diff_coef(gE, Ksq),
      cW = diff_coef(gW, Ksq);
    if (sizeof(T) == 4) {
        // FP32 form: the same sum with fused multiply-adds
        T sum = cN * gN;
        sum = fma(cS, gS, sum);
        sum = fma(cE, gE, sum);
        sum = fma(cW, gW, sum);
        return fma(lambda, sum, cv);
    }
    T sum = rn_add(rn_add(rn_add(rn_mul(cN, gN), rn_mul(cS, gS)), rn_mul(cE, gE)),
                   rn_mul(cW, gW));
    return rn_add(cv, rn_mul(lambda, sum));
}

// Per Z-plane, `niter` Gauss-Seidel sweeps in (y, x) order, updated in
// place.  Cell (y, x) of sweep s reads its N and W neighbours from sweep s
// and its S and E neighbours from sweep s-1, so the sweeps run as a
// pipelined anti-diagonal wavefront: at step t sweep s updates diagonal
// d = t - 2s.  Every cell sees the neighbour values of the sequential loops.
// This form works in global memory (any plane size).
template <typename T>
__global__ void __launch_bounds__(1024)
k_diffusion(T *u, int ny, int nx, int nxb, double lambda_d, double ksq_d, int niter,
            const int *__restrict__ only)
{
    if (only && !only[blockIdx.x]) return;
    T *U = u + (size_t)blockIdx.x * ny * nx;
    const T lambda = (T)lambda_d, Ksq = (T)ksq_d;
    int D = ny + nx - 1, L = min(ny, nx);
    int nsteps = D + 2 * (niter - 1);
    for (int t = 0; t < nsteps; t++) {
        int s_hi = min(niter - 1, t / 2);
        int a = t - (D - 1);
        int s_lo = a > 0 ? (a + 1) / 2 : 0;
        int nact = s_hi - s_lo + 1;
        for (int w = threadIdx.x; w < nact * L; w += blockDim.x) {
            int s = s_lo + w / L, c = w - (w / L) * L;
            int d = t - 2 * s;
            int y0 = max(0, d - (nx - 1)), y1 = min(ny - 1, d);
            int y = y0 + c;
            if (y > y1) continue;
            int x = d - y;
            int jp = (y == ny - 1) ? ny - 1 : y + 1, jm = (y == 0) ? 0 : y - 1;
            int ip = (x == nxb - 1) ? nxb - 1 : x + 1, im = (x == 0) ? 0 : x - 1;
            T cv = U[(size_t)y * nx + x];
            T e = ip < nx ? U[(size_t)y * nx + ip] : T(0);
            U[(size_t)y * nx + x] = diff_cell<T>(cv, U[(size_t)jm * nx + x],
                                                 U[(size_t)jp * nx + x], e,
                                                 U[(size_t)y * nx + im], lambda, Ksq);
        }
        __syncthreads();
    }
}

// The same wavefront with the live band in shared memory.  Sweeps run in
// groups of G; inside a group sweep g updates anti-diagonal d = t - 2g at
// step t, so only diagonals [t - 2G + 1, t + 1] are live: they sit in a ring
// of R = 2G + 2 diagonal slots (slot = d mod R, cell (y, x) of diagonal d at
// position y - y0(d)).  During step t diagonal t + 2 is fetched into
// registers (its slot held diagonal t + 2 - R, written back at step t - 1)
// and diagonal t - 2G + 1, final for the group, is written back: one barrier
// per step.  The cells of a step are dealt out as 128-cell segments of the
// active diagonals, one warp per segment, from a task table (segment prefix
// counts and ring slots) that warp 0 builds for step t + 1 during step t.
// Requires min(ny, nx) <= kDiffPf * blockDim.x.
constexpr int kDiffPf = 4;
constexpr int kDiffMaxG = 64;  // sweeps per group (task tables in shared memory)

template <typename T>
__global__ void __launch_bounds__(1024)
k_diffusion_ring(T *u, int ny, int nx, int nxb, double lambda_d, double ksq_d, int niter,
                 int G, int R, const int *__restrict__ only)
{
    if (only && !only[blockIdx.x]) return;
    extern __shared__ __align__(16) unsigned char smraw[];
    T *ring = (T *)smraw;
    T *U = u + (size_t)blockIdx.x * ny * nx;
    const T lambda = (T)lambda_d, Ksq = (T)ksq_d;
    const int D = ny + nx - 1, L = min(ny, nx);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    // per step (double-buffered), for active diagonal k (sweep g_lo + k):
    // prefix count of its 128-cell tasks, d, y0(d), len(d), and the ring offsets
    // of diagonals d, d - 1, d + 1
    constexpr int TC = 128;
    __shared__ int s_pre[2][kDiffMaxG + 1], s_meta[2][2];
    __shared__ int4 s_dg[2][kDiffMaxG];   // d, y0, len, ring offset of d
    __shared__ int2 s_nb[2][kDiffMaxG];   // ring offsets of d - 1 (d itself when d == 0) and d + 1
    auto y0 = [&](int d) { return max(0, d - (nx - 1)); };
    auto len = [&](int d) { return min(d, ny - 1) - y0(d) + 1; };
    // warp 0: the task table of step t of a group of gc sweeps into buffer b
    auto build_table = [&](int t, int gc, int b) {
        const int g_hi = min(gc - 1, t / 2), a = t - (D - 1);
        const int g_lo = a > 0 ? (a + 1) / 2 : 0, nact = g_hi - g_lo + 1;
        int carry = 0;
        for (int base = 0; base < nact; base += 32) {
            const int k = base + lane;
            int c = 0;
            if (k < nact) {
                const int d = t - 2 * (g_lo + k), nd = len(d), sd = d % R;
                c = (nd + TC - 1) / TC;
                s_dg[b][k] = make_int4(d, y0(d), nd, sd * L);
                s_nb[b][k] = make_int2(d > 0 ? (sd == 0 ? R - 1 : sd - 1) * L : sd * L,
                                       (sd == R - 1 ? 0 : sd + 1) * L);
            }
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (k < nact) s_pre[b][k + 1] = carry + incl;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) {
            s_pre[b][0] = 0;
            s_meta[b][0] = nact;
            s_meta[b][1] = g_lo;
        }
    };
    auto slot = [&](int d) { return ring + (size_t)(d % R) * L; };
    auto cell = [&](int d, int i) -> size_t {
        int a = y0(d);
        return (size_t)(a + i) * nx + (d - a - i);
    };
    for (int s0 = 0; s0 < niter; s0 += G) {
        const int gc = min(G, niter - s0);
        const int nsteps = D + 2 * (gc - 1);
        for (int d = 0; d < 2 && d < D; d++) {
            T *s = slot(d);
            for (int i = threadIdx.x; i < len(d); i += blockDim.x) s[i] = U[cell(d, i)];
        }
        if (warp == 0) build_table(0, gc, 0);
        __syncthreads();
        for (int t = 0; t < nsteps; t++) {
            // fetch diagonal t + 2
            const int dn = t + 2;
            const int nn = dn < D ? len(dn) : 0;
            // slots a diagonal of this plane can use (uniform: a real branch)
            const int npf = (L + blockDim.x - 1) / blockDim.x;
            T pf[kDiffPf];
#pragma unroll
            for (int k = 0; k < kDiffPf; k++) {
                if (k >= npf) break;
                int i = threadIdx.x + k * blockDim.x;
                pf[k] = i < nn ? U[cell(dn, i)] : T(0);
            }
            // the next step's task table (warp 0), then this step's tasks:
            // 128-cell segments of the active diagonals, dealt out to the warps
            const int tb = t & 1;
            if (warp == 0 && t + 1 < nsteps) build_table(t + 1, gc, tb ^ 1);
            {
                const int *pre = s_pre[tb];
                const int nact = s_meta[tb][0], ntask = pre[nact];
                // this warp's contiguous share of the tasks; k: the diagonal of
                // the first one (binary search over the prefix counts)
                const int t_beg = (int)((long)ntask * warp / nwarps);
                const int t_end = (int)((long)ntask * (warp + 1) / nwarps);
                int k = 0;
                for (int lo = 0, hi = nact - 1; lo <= hi;) {
                    int mid = (lo + hi) >> 1;
                    if (pre[mid + 1] <= t_beg) lo = mid + 1, k = lo;
                    else hi = mid - 1;
                }
                for (int task = t_beg; task < t_end; task++) {
                    while (pre[k + 1] <= task) k++;
                    const int4 dg = s_dg[tb][k];
                    const int2 nb = s_nb[tb][k];
                    const int d = dg.x, yd = dg.y, nd = dg.z;
                    // rows of diagonal d's neighbours: y0(d - 1) and y0(d + 1)
                    const int ym = d > nx - 1 ? yd - 1 : 0, yp = d + 1 > nx - 1 ? yd + 1 : 0;
                    T *sc = ring + dg.w;
                    const T *sm = ring + nb.x, *sp = ring + nb.y;
                    const int i0 = (task - pre[k]) * TC;
                    const T *mb = sm + (yd - ym), *pb = sp + (yd - yp);
#pragma unroll
                    for (int h = 0; h < TC / 32; h++) {
                        const int g0 = i0 + h * 32, g1 = min(nd, g0 + 32) - 1, i = g0 + lane;
                        // an interior group of 32 cells: each has its four plain
                        // neighbours (y in [1, ny-2], x in [1, nx-2] and x != nxb - 1,
                        // the column the reference clamps): cell i's N and W sit at
                        // i - 1, i of diagonal d - 1 from yd - ym, its S and E at i + 1,
                        // i of diagonal d + 1 from yd - yp.  Along a diagonal y grows
                        // and x falls.
                        const int xmax = d - yd - g0, xmin = d - yd - g1;
                        const bool inner = g0 <= g1 && yd + g0 >= 1 && yd + g1 <= ny - 2 &&
                                           xmin >= 1 && xmax <= nx - 2 &&
                                           !(xmin <= nxb - 1 && nxb - 1 <= xmax);
                        if (__all_sync(0xffffffffu, inner)) {  // warp-uniform: a real branch
                            if (i <= g1) {
                                T cv = sc[i];
                                sc[i] = diff_cell<T>(cv, mb[i - 1], pb[i + 1], pb[i], mb[i], lambda,
                                                     Ksq);
                            }
                        } else if (i <= g1) {
                            int y = yd + i, x = d - y;
                            T cv = sc[i];
                            T nN = cv, nS = cv, nW = cv, nE = cv;
                            if (y > 0) nN = sm[(y - 1) - ym];
                            if (x > 0) nW = sm[y - ym];
                            if (y < ny - 1) nS = sp[(y + 1) - yp];
                            int ip = (x == nxb - 1) ? nxb - 1 : x + 1;
                            if (ip != x) nE = ip < nx ? sp[y - yp] : T(0);
                            sc[i] = diff_cell<T>(cv, nN, nS, nE, nW, lambda, Ksq);
                        }
                    }
                }
            }
            if (nn > 0) {
                T *s = slot(dn);
#pragma unroll
                for (int k = 0; k < kDiffPf; k++) {
                    if (k >= npf) break;
                    int i = threadIdx.x + k * blockDim.x;
                    if (i < nn) s[i] = pf[k];
                }
            }
            const int df = t - 2 * gc + 1;  // final for this group
            if (df >= 0 && df < D) {
                const T *s = slot(df);
                for (int i = threadIdx.x; i < len(df); i += blockDim.x) U[cell(df, i)] = s[i];
            }
            __syncthreads();
        }
        {
            const T *s = slot(D - 1);
            for (int i = threadIdx.x; i < len(D - 1); i += blockDim.x) U[cell(D - 1, i)] = s[i];
        }
        __syncthreads();
    }
}

// The same ring of diagonals with the work dealt out by rows instead of task
// tables.  A slot holds a diagonal at its rows' positions (cell (y, d - y) of
// diagonal d at position y of slot d mod R, slots ny values long), so a cell's
// N and W sit at y - 1 and y of slot d - 1 and its S and E at y + 1 and y of
// slot d + 1.  At step t sweep g updates row y's cell on diagonal t - 2g.  A
// warp owns 32 consecutive rows and one of TPR sweep classes (g = class mod
// TPR): at a given sweep its lanes touch consecutive positions of one slot
// (no bank conflicts), and no per-step table or search is needed.  (Tried
// and slower, measured: classes re-dealt per step to the rows a step has,
// and two cells per iteration with paired FP32 arithmetic.)  Prefetch of
// diagonal t + 2, write-back of the group's final diagonal and one barrier
// per step as in k_diffusion_ring.  Requires min(ny, nx) <= kDiffPf *
// blockDim.x, blockDim.x a multiple of 32 TPR and, FP32, blockDim.x <= 768
// (two CTAs per SM).
template <typename T> struct DiffNb {
    T c, n, w, s, e;
};

template <typename T, int TPR>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 768 : 1024, sizeof(T) == 4 ? 2 : 1)
k_diffusion_rows(T *u, int ny, int nx, int nxb, double lambda_d, double ksq_d, int niter,
                 int G, int R)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    T *ring = (T *)smraw;
    T *U = u + (size_t)blockIdx.x * ny * nx;
    const T lambda = (T)lambda_d, Ksq = (T)ksq_d;
    const int D = ny + nx - 1, L = min(ny, nx);
    auto y0 = [&](int d) { return max(0, d - (nx - 1)); };
    auto len = [&](int d) { return min(d, ny - 1) - y0(d) + 1; };
    // position i (row y0(d) + i) of diagonal d in the ring, and in the plane
    auto slot = [&](int d) { return ring + (size_t)(d % R) * ny + y0(d); };
    auto cell = [&](int d, int i) -> size_t {
        int a = y0(d);
        return (size_t)(a + i) * nx + (d - a - i);
    };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cls = warp % TPR;
    const int yfirst = (warp / TPR) * 32 + lane, ystride = blockDim.x / TPR;
    const int dstep = (2 * TPR) % R;  // ring slots between sweeps g and g + TPR
    // one cell's values: (y, x) of the diagonal in slot sd.  The reference's
    // clamps (denoise.c:343-351): a clamped neighbour is the cell itself,
    // x + 1 == nx reads 0.0; the reads a clamp replaces stay inside their
    // slots and are discarded.
    auto load = [&](int sd, int y, int x, bool hasN, bool hasS, int yN, int yS) {
        const int sm = sd == 0 ? R - 1 : sd - 1, sp = sd == R - 1 ? 0 : sd + 1;
        const T *rc = ring + sd * ny, *rm = ring + sm * ny, *rp = ring + sp * ny;
        DiffNb<T> v;
        v.c = rc[y];
        const T vN = rm[yN], vW = rm[y], vS = rp[yS], vE = rp[y];
        v.n = hasN ? vN : v.c;
        v.w = x > 0 ? vW : v.c;
        v.s = hasS ? vS : v.c;
        v.e = x == nxb - 1 ? v.c : (x + 1 < nx ? vE : T(0));
        return v;
    };
    for (int s0 = 0; s0 < niter; s0 += G) {
        const int gc = min(G, niter - s0);
        const int nsteps = D + 2 * (gc - 1);
        for (int d = 0; d < 2 && d < D; d++) {
            T *sd = slot(d);
            for (int i = threadIdx.x; i < len(d); i += blockDim.x) sd[i] = U[cell(d, i)];
        }
        __syncthreads();
        for (int t = 0; t < nsteps; t++) {
            // fetch diagonal t + 2 (stored after this step's cells)
            const int dn = t + 2;
            const int nn = dn < D ? len(dn) : 0;
            const int npf = (L + blockDim.x - 1) / blockDim.x;
            T pf[kDiffPf];
#pragma unroll
            for (int k = 0; k < kDiffPf; k++) {
                if (k >= npf) break;
                const int i = threadIdx.x + k * blockDim.x;
                pf[k] = i < nn ? U[cell(dn, i)] : T(0);
            }
            if (cls < gc)
                for (int y = yfirst; y <= t && y < ny; y += ystride) {
                    // this class's sweeps with a cell in row y: x = t - y - 2g
                    // in [0, nx - 1] and g < gc
                    const int ghi = min(gc - 1, (t - y) >> 1);
                    int glo = t - y - nx + 2;
                    glo = glo > 0 ? glo >> 1 : 0;
                    int g = glo + ((cls - glo) % TPR + TPR) % TPR;
                    const bool hasN = y > 0, hasS = y < ny - 1;
                    const int yN = hasN ? y - 1 : y, yS = hasS ? y + 1 : y;
                    int d = t - 2 * g, sd = d % R;
                    for (; g <= ghi; g += TPR) {
                        const DiffNb<T> a = load(sd, y, d - y, hasN, hasS, yN, yS);
                        ring[sd * ny + y] = diff_cell<T>(a.c, a.n, a.s, a.e, a.w, lambda, Ksq);
                        d -= 2 * TPR;
                        sd -= dstep;
                        if (sd < 0) sd += R;
                    }
                }
            if (nn > 0) {
                T *sd = slot(dn);
#pragma unroll
                for (int k = 0; k < kDiffPf; k++) {
                    if (k >= npf) break;
                    const int i = threadIdx.x + k * blockDim.x;
                    if (i < nn) sd[i] = pf[k];
                }
            }
            const int df = t - 2 * gc + 1;  // final for this group
            if (df >= 0 && df < D) {
                const T *sd = slot(df);
                for (int i = threadIdx.x; i < len(df); i += blockDim.x) U[cell(df, i)] = sd[i];
            }
            __syncthreads();
        }
        {
            const T *sd = slot(D - 1);
            for (int i = threadIdx.x; i < len(D - 1); i += blockDim.x) U[cell(D - 1, i)] = sd[i];
        }
        __syncthreads();
    }
}

// The row form with two rows per thread: rows (2r, 2r + 1) meet a diagonal d
// at adjacent positions of its slot, so one thread updates both cells of a
// sweep together: their centres, the W of the first (= N of the second) and
// the second's W, the first's E and S (= E of the second) and the second's S
// come from three 8-byte and two 4-byte shared-memory loads instead of ten,
// the two results go out as one 8-byte store, and the FP32 arithmetic of the
// pair runs as paired instructions (each the same IEEE operation as
// diff_cell's, so the results are bit-identical).  A pair whose second row
// or either cell is off the plane writes that position's old value back (the
// position belongs to no cell of the diagonal; only this thread writes it).
// A warp owns 64 rows and one of TPR sweep classes.  Slots are S >= ny + 1
// values (S even: the pairs' 8-byte accesses stay aligned).  Requires
// min(ny, nx) <= kDiffPf * blockDim.x, blockDim.x a multiple of 32 TPR and,
// FP32, blockDim.x <= 768.
template <typename T, int TPR>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 768 : 1024, sizeof(T) == 4 ? 2 : 1)
k_diffusion_pairs(T *u, int ny, int nx, int nxb, double lambda_d, double ksq_d, int niter,
                  int G, int R, int S, const int *__restrict__ only)
{
    if (only && !only[blockIdx.x]) return;
    extern __shared__ __align__(16) unsigned char smraw[];
    T *ring = (T *)smraw;  // R slots of S >= ny + 1 values (S even)
    T *U = u + (size_t)blockIdx.x * ny * nx;
    const T lambda = (T)lambda_d, Ksq = (T)ksq_d;
    const int D = ny + nx - 1, L = min(ny, nx);
    auto y0 = [&](int d) { return max(0, d - (nx - 1)); };
    auto len = [&](int d) { return min(d, ny - 1) - y0(d) + 1; };
    auto slot = [&](int d) { return ring + (size_t)(d % R) * S + y0(d); };
    auto cell = [&](int d, int i) -> size_t {
        int a = y0(d);
        return (size_t)(a + i) * nx + (d - a - i);
    };
    using T2 = typename std::conditional<sizeof(T) == 4, float2, double2>::type;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cls = warp % TPR;
    const int pfirst = (warp / TPR) * 32 + lane, pstride = blockDim.x / TPR;
    const int dstep = (2 * TPR) % R;
    const int npairs = (ny + 1) >> 1;
    for (int s0 = 0; s0 < niter; s0 += G) {
        const int gc = min(G, niter - s0);
        const int nsteps = D + 2 * (gc - 1);
        for (int d = 0; d < 2 && d < D; d++) {
            T *sd = slot(d);
            for (int i = threadIdx.x; i < len(d); i += blockDim.x) sd[i] = U[cell(d, i)];
        }
        __syncthreads();
        for (int t = 0; t < nsteps; t++) {
            const int dn = t + 2;
            const int nn = dn < D ? len(dn) : 0;
            const int npf = (L + blockDim.x - 1) / blockDim.x;
            T pf[kDiffPf];
#pragma unroll
            for (int k = 0; k < kDiffPf; k++) {
                if (k >= npf) break;
                const int i = threadIdx.x + k * blockDim.x;
                pf[k] = i < nn ? U[cell(dn, i)] : T(0);
            }
            if (cls < gc)
                for (int pr = pfirst; pr < npairs && 2 * pr <= t; pr += pstride) {
                    const int y = 2 * pr;  // rows y, y + 1
                    // sweeps of this class with a cell in row y or y + 1:
                    // x = t - y - 2g in [0, nx] (row y + 1 has x - 1) and g < gc
                    const int ghi = min(gc - 1, (t - y) >> 1);
                    const int over = t - y - nx;  // x <= nx  <=>  g >= over / 2
                    const int glo = over > 0 ? (over + 1) >> 1 : 0;
                    int g = glo + ((cls - glo) % TPR + TPR) % TPR;
                    const bool hasN = y > 0, hasS1 = y + 1 < ny - 1;
                    const int yN = hasN ? y - 1 : y + 1;  // in-slot when clamped
                    const int yS = y + 2 < S ? y + 2 : y;
                    int d = t - 2 * g, sd = d % R;
                    for (; g <= ghi; g += TPR) {
                        const int x = d - y;  // row y + 1: x - 1
                        const int sm = sd == 0 ? R - 1 : sd - 1, sp = sd == R - 1 ? 0 : sd + 1;
                        T *rc = ring + sd * S;
                        const T *rm = ring + sm * S, *rp = ring + sp * S;
                        const T2 c = *reinterpret_cast<const T2 *>(rc + y);
                        const T2 m = *reinterpret_cast<const T2 *>(rm + y);  // W0 = N1, W1
                        const T2 q = *reinterpret_cast<const T2 *>(rp + y);  // E0, S0 = E1
                        const T mN = rm[yN], pS = rp[yS];
                        // row y: N = rm[y-1], W = rm[y], S = rp[y+1], E = rp[y]
                        // row y+1: N = rm[y], W = rm[y+1], S = rp[y+2], E = rp[y+1]
                        const int x1 = x - 1;
                        T n0 = hasN ? mN : c.x, w0 = x > 0 ? m.x : c.x, s0v = q.y;
                        T e0 = x == nxb - 1 ? c.x : (x + 1 < nx ? q.x : T(0));
                        if (y == ny - 1) s0v = c.x;  // last row (odd ny): S clamps to itself
                        T n1 = m.x, w1 = x1 > 0 ? m.y : c.y, s1 = hasS1 ? pS : c.y;
                        T e1 = x1 == nxb - 1 ? c.y : (x1 + 1 < nx ? q.y : T(0));
                        T u0, u1;
                        if constexpr (sizeof(T) == 4) {
                            auto f2 = [](float a, float b) { return make_float2(a, b); };
                            auto sub = [](float2 a, float2 b) {
                                return __fadd2_rn(a, make_float2(-b.x, -b.y));
                            };
                            const float2 cc = f2(c.x, c.y), k2 = f2(Ksq, Ksq);
                            const float2 gN = sub(f2(n0, n1), cc), gS = sub(f2(s0v, s1), cc),
                                         gE = sub(f2(e0, e1), cc), gW = sub(f2(w0, w1), cc);
                            auto coef = [&](float2 gg) {
                                const float2 dd = __ffma2_rn(gg, gg, k2);
                                return __fmul2_rn(k2, f2(rcp_approx(dd.x), rcp_approx(dd.y)));
                            };
                            float2 sum = __fmul2_rn(coef(gN), gN);
                            sum = __ffma2_rn(coef(gS), gS, sum);
                            sum = __ffma2_rn(coef(gE), gE, sum);
                            sum = __ffma2_rn(coef(gW), gW, sum);
                            const float2 uu = __ffma2_rn(f2(lambda, lambda), sum, cc);
                            u0 = uu.x;
                            u1 = uu.y;
                        } else {
                            u0 = diff_cell<T>(c.x, n0, s0v, e0, w0, lambda, Ksq);
                            u1 = diff_cell<T>(c.y, n1, s1, e1, w1, lambda, Ksq);
                        }
                        // a cell off the plane keeps its slot's old value
                        if (x > nx - 1) u0 = c.x;
                        if (x1 < 0 || y + 1 >= ny) u1 = c.y;
                        T2 o;
                        o.x = u0;
                        o.y = u1;
                        *reinterpret_cast<T2 *>(rc + y) = o;
                        d -= 2 * TPR;
                        sd -= dstep;
                        if (sd < 0) sd += R;
                    }
                }
            if (nn > 0) {
                T *sd = slot(dn);
#pragma unroll
                for (int k = 0; k < kDiffPf; k++) {
                    if (k >= npf) break;
                    const int i = threadIdx.x + k * blockDim.x;
                    if (i < nn) sd[i] = pf[k];
                }
            }
            const int df = t - 2 * gc + 1;
            if (df >= 0 && df < D) {
                const T *sd = slot(df);
                for (int i = threadIdx.x; i < len(df); i += blockDim.x) U[cell(df, i)] = sd[i];
            }
            __syncthreads();
        }
        {
            const T *sd = slot(D - 1);
            for (int i = threadIdx.x; i < len(D - 1); i += blockDim.x) U[cell(D - 1, i)] = sd[i];
        }
        __syncthreads();
    }
}

// The wavefront form: strips (strips.cu, the default where its range and the
// scratch allow), pairs (k_diffusion_pairs, FP32 otherwise), rows
// (k_diffusion_rows) or task tables (k_diffusion_ring, FP64 otherwise);
// NUDIM_DIFFUSION=strips|pairs|rows|tables selects one.  FP64: all give the
// same cells bit for bit; FP32: the last three, while the strips pair their
// coefficients' denominators.  Read at every launch (a captured graph keeps the
// form it was captured with).
enum DiffForm { DF_STRIPS, DF_PAIRS, DF_ROWS, DF_TABLES };
template <typename T> static DiffForm diffusion_form()
{
    const char *e = getenv("NUDIM_DIFFUSION");
    if (e && !strcmp(e, "strips")) return DF_STRIPS;
    if (e && !strcmp(e, "tables")) return DF_TABLES;
    if (e && !strcmp(e, "rows")) return DF_ROWS;
    if (e && !strcmp(e, "pairs")) return DF_PAIRS;
    return DF_STRIPS;
}

template <typename T>
size_t diffusion_scratch(int nz, int ny, int nx, float lambda, float kappa, int niter)
{
    if (nz <= 0 || diffusion_form<T>() != DF_STRIPS ||
        !strips_fits<T>(ny, nx, niter, lambda, (double)kappa * (double)kappa))
        return 0;
    return strips_scratch<T>(nz, ny, nx, niter);
}

template <typename T>
int diffusion_run(T *u, int nz, int ny, int nx, int nx_bound, float lambda, float kappa,
                  int niter, void *scratch, cudaStream_t st)
{
    if (niter <= 0 || nz <= 0) return NUDIM_OK;
    double ksq = (double)kappa * (double)kappa;
    DiffForm form = diffusion_form<T>();
    const int *only = nullptr;  // pairs form: the planes the strips left to it
    if (form == DF_STRIPS && scratch && strips_fits<T>(ny, nx, niter, lambda, ksq)) {
        NUDIM_TRY(strips_run<T>(u, nz, ny, nx, nx_bound, lambda, ksq, niter, scratch, st));
        if (sizeof(T) == 8) return NUDIM_OK;
        only = (const int *)scratch;
    }
    if (form == DF_STRIPS) form = sizeof(T) == 8 ? DF_TABLES : DF_PAIRS;
    int L = ny < nx ? ny : nx;
    int P = std::min(1024, (L + 31) & ~31);
    // FP32 on planes up to 512 wide: two CTAs per SM; otherwise one CTA with
    // up to 160 KB of ring
    bool two = sizeof(T) == 4 && P <= 512;
    const size_t budget = two ? ((size_t)108 << 10) : ((size_t)160 << 10);
    const int cap = sizeof(T) == 4 ? 768 : 1024;
    if (form == DF_PAIRS) {
        // two rows per thread: slots of S = ny + 1 rounded up to even values;
        // TPR sweep classes (a power of two) so that 64-row warps x classes
        // fill up to 768 (FP32, two CTAs per SM) or 1024 threads
        const int S = (ny + 2) & ~1, Pp = (((ny + 1) >> 1) + 31) & ~31;
        int G = (int)((budget / (sizeof(T) * (size_t)S) - 2) / 2);
        if (G > niter) G = niter;
        if (G > kDiffMaxG) G = kDiffMaxG;
        int tpr = 1;
        while (tpr < 8 && 2 * tpr * Pp <= cap && 2 * tpr <= G) tpr *= 2;
        const int threads = std::min(cap, tpr * Pp);
        if (G >= 1 && L <= kDiffPf * threads) {
            const int R = 2 * G + 2;
            const size_t smem = sizeof(T) * (size_t)R * S;
#define NUDIM_DIFF_PAIRS(TP)                                                                    \
    do {                                                                                        \
        NUDIM_CUDA(cudaFuncSetAttribute(k_diffusion_pairs<T, TP>,                               \
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, 160 << 10)); \
        k_diffusion_pairs<T, TP><<<nz, threads, smem, st>>>(u, ny, nx, nx_bound, (double)lambda, \
                                                             ksq, niter, G, R, S, only);        \
    } while (0)
            if (tpr == 8) NUDIM_DIFF_PAIRS(8);
            else if (tpr == 4) NUDIM_DIFF_PAIRS(4);
            else if (tpr == 2) NUDIM_DIFF_PAIRS(2);
            else NUDIM_DIFF_PAIRS(1);
#undef NUDIM_DIFF_PAIRS
            NUDIM_LAUNCH_CHECK();
            return NUDIM_OK;
        }
    }
    if (form == DF_ROWS) {
        // one row per thread: slots of ny values; TPR sweep classes so that
        // 32-row warps x classes fill up to 768 or 1024 threads
        int G = (int)((budget / (sizeof(T) * (size_t)ny) - 2) / 2);
        if (G > niter) G = niter;
        if (G > kDiffMaxG) G = kDiffMaxG;
        const int Py = (ny + 31) & ~31;
        int tpr = 1;
        while (tpr < 8 && 2 * tpr * Py <= cap && 2 * tpr <= G) tpr *= 2;
        const int threads = std::min(cap, tpr * Py);
        if (G >= 1 && L <= kDiffPf * threads) {
            const int R = 2 * G + 2;
            const size_t smem = sizeof(T) * (size_t)R * ny;
#define NUDIM_DIFF_ROWS(TP)                                                                     \
    do {                                                                                        \
        NUDIM_CUDA(cudaFuncSetAttribute(k_diffusion_rows<T, TP>,                                \
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, 160 << 10)); \
        k_diffusion_rows<T, TP><<<nz, threads, smem, st>>>(u, ny, nx, nx_bound, (double)lambda,  \
                                                            ksq, niter, G, R);                  \
    } while (0)
            if (tpr == 8) NUDIM_DIFF_ROWS(8);
            else if (tpr == 4) NUDIM_DIFF_ROWS(4);
            else if (tpr == 2) NUDIM_DIFF_ROWS(2);
            else NUDIM_DIFF_ROWS(1);
#undef NUDIM_DIFF_ROWS
            NUDIM_LAUNCH_CHECK();
            return NUDIM_OK;
        }
    }
    int threads = two ? 2 * P : 1024;
    int G = (int)((budget / (sizeof(T) * (size_t)L) - 2) / 2);
    if (G > niter) G = niter;
    if (G > kDiffMaxG) G = kDiffMaxG;
    if (G >= 1 && L <= kDiffPf * threads) {
        int R = 2 * G + 2;
        size_t smem = sizeof(T) * (size_t)R * L;
        NUDIM_CUDA(cudaFuncSetAttribute(k_diffusion_ring<T>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        160 << 10));
        k_diffusion_ring<T><<<nz, threads, smem, st>>>(u, ny, nx, nx_bound, (double)lambda, ksq,
                                                        niter, G, R, only);
    } else {
        k_diffusion<T><<<nz, 1024, 0, st>>>(u, ny, nx, nx_bound, (double)lambda, ksq, niter,
                                     only);
    }
    NUDIM_LAUNCH_CHECK();
    return NUDIM_OK;
}

template int tv_run<double>(double *, double *, double *, int, double *, int, int, int, float,
                            int, int, int, int, cudaStream_t, double *, double *);
template int tv_run<float>(float *, float *, double *, int, double *, int, int, int, float, int,
                           int, int, int, cudaStream_t, float *, float *);
template int diffusion_run<double>(double *, int, int, int, int, float, float, int, void *,
                                   cudaStream_t);
template int diffusion_run<float>(float *, int, int, int, int, float, float, int, void *,
                                  cudaStream_t);
template size_t diffusion_scratch<double>(int, int, int, float, float, int);
template size_t diffusion_scratch<float>(int, int, int, float, float, int);

}  // namespace nudim
