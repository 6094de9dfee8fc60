// strips.cu -- the in-place 2D anisotropic diffusion of denoise.c:320-378 as a
// register-resident wavefront.
//
// Cell (y, x) of sweep s reads its N and W neighbours from sweep s and its S,
// E and own values from sweep s - 1, so the sweeps run as a pipelined
// anti-diagonal wavefront: at step t sweep s updates diagonal x + y = t - 2s.
// A lane owns a strip of R adjacent rows, a warp 32 R rows of one plane for Q
// consecutive sweeps.  At a step the lane's cells lie on one diagonal (row i at
// column d - y0 - i), so they are independent of each other, and every
// neighbour is a register: a cell's W is its row's result of the previous
// step, its N the row above's; its E is what the previous sweep produced for
// the row one step ago, its own value what it produced two steps ago, its S
// the row below's E.  Between Q sweeps of a thread nothing leaves the
// registers; between lanes two shuffles per sweep and step carry the strip's
// edges; between warps (sweep groups) R values per lane and step go through
// shared memory, double-buffered, with one barrier per step.
//
// K = Q x warps x CTAs of a cluster sweeps are live at once.  A plane goes
// through the K-sweep pipeline `rounds` times without a break: it is kept
// skewed in a scratch S[(x + y) mod P][row] (P >= nx slots), so that a step
// reads and writes one slot's consecutive rows; the pipeline's last warp writes
// slot d mod P and its first warp reads the slot again P - 2 (K - 1) steps
// later.  The plane is skewed into S when its turn comes and out of it at the
// end (32 x 32 tiles through shared memory, coalesced on both sides).
//
// Bound: issue and the FMA, ALU and special-function pipes together (25
// instructions a cell, of 38 cycles a warp's 32 cells take on a scheduler; the
// boundary columns' selects are a quarter of them).  256 x 384 x 384, 80
// sweeps: 4.40 ms against 12.1 ms for the shared-memory pairs form.
// The cell's four coefficients K^2 / (K^2 + g^2) are summed in pairs over a
// common denominator, gN/dN + gS/dS = (gN dS + gS dN) / (dN dS): one reciprocal
// for two coefficients (four per cell bound the loop by the special-function
// unit at 4 cells per clock and SM: 5.30 ms).  The distance from FP64 results,
// against that of the pairs form with its reciprocal per neighbour: median 0.99,
// geometric mean 1.00 times it over 150 volumes of 9 thousand to 11 million voxels
// (ragged, planes of 32 to 384 a side; lambda 1/4), 1.02 on 256 x 384 x 384, 0.7 where lambda
// is 0.4; one reciprocal refined by a step of Newton's iteration 1.01 there, at
// 4.61 ms.  FP64 by the integer units (66 % of their
// rate) and the FP64 unit (67 %), see intdiv.cuh.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "engine.cuh"
#include "intdiv.cuh"
#include "strip_shape.h"

namespace cg = cooperative_groups;

namespace nudim {

namespace {

__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// 1 << s, 0 for s >= 32 (also for a negative s taken as unsigned)
__device__ __forceinline__ unsigned bit_at(int s)
{
    unsigned r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(1u), "r"((unsigned)s));
    return r;
}

// The FP32 pair forms products of two denominators: |values| below kMaxF keep
// them finite (differences 2 kMaxF, denominators 4 kMaxF^2, product 16 kMaxF^4
// < 2^128; the sweeps move a value by at most 2 lambda K each), K^2 >= kMinKsq
// keeps them normal.  Planes beyond it go to the one-denominator-at-a-time form.
constexpr float kMaxF = 1e9f;
constexpr double kMinKsq = 1e-17, kMaxKsq = 1e18;

template <typename T> struct CellArgs;
template <> struct CellArgs<float> {
    float lk, ksq;  // lambda K^2, K^2
};
template <> struct CellArgs<double> {
    double lambda;
    DiffDiv div;
};

// Cells of two adjacent rows.  The differences are scalar:
// the rows' N and S are not a register pair, and pairing rows (i, i + R/2),
// whose N and S are, took more moves than it saved (256 x 384 x 384: 8 % slower).
__device__ __forceinline__ void cell2(float c0, float c1, float n0, float n1, float s0, float s1,
                                      float e0, float e1, float w0, float w1,
                                      const CellArgs<float> &k, float &u0, float &u1)
{
    const float2 k2 = make_float2(k.ksq, k.ksq);
    const float2 gN = make_float2(n0 - c0, n1 - c1), gS = make_float2(s0 - c0, s1 - c1);
    const float2 gE = make_float2(e0 - c0, e1 - c1), gW = make_float2(w0 - c0, w1 - c1);
    const float2 dN = __ffma2_rn(gN, gN, k2), dS = __ffma2_rn(gS, gS, k2);
    const float2 dE = __ffma2_rn(gE, gE, k2), dW = __ffma2_rn(gW, gW, k2);
    const float2 a = __ffma2_rn(gN, dS, __fmul2_rn(gS, dN)), p = __fmul2_rn(dN, dS);
    const float2 b = __ffma2_rn(gE, dW, __fmul2_rn(gW, dE)), q = __fmul2_rn(dE, dW);
    const float2 rp = make_float2(rcp_approx(p.x), rcp_approx(p.y));
    const float2 rq = make_float2(rcp_approx(q.x), rcp_approx(q.y));
    const float2 sum = __ffma2_rn(b, rq, __fmul2_rn(a, rp));
    const float2 u = __ffma2_rn(make_float2(k.lk, k.lk), sum, make_float2(c0, c1));
    u0 = u.x;
    u1 = u.y;
}

// FP64: the reference's operations in its order, each rounded as IEEE rounds
// it; the fluxes in integer arithmetic (intdiv.cuh), with the FP64 unit's
// divisions for the values that does not take.
__device__ __noinline__ double flux_divided(double g, double ksq)
{
    return rn_mul(rn_div(1.0, rn_add(1.0, rn_div(rn_mul(g, g), ksq))), g);
}

__device__ __forceinline__ double cell1(double c, double n, double s, double e, double w,
                                        const CellArgs<double> &k)
{
    const double g[4] = {rn_sub(n, c), rn_sub(s, c), rn_sub(e, c), rn_sub(w, c)};
    double f[4];
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 4; j++) ok &= diff_flux_int(g[j], k.div, f + j);
    if (!ok) {
        f[0] = flux_divided(g[0], k.div.b);
        f[1] = flux_divided(g[1], k.div.b);
        f[2] = flux_divided(g[2], k.div.b);
        f[3] = flux_divided(g[3], k.div.b);
    }
    return rn_add(c, rn_mul(k.lambda, rn_add(rn_add(rn_add(f[0], f[1]), f[2]), f[3])));
}

__device__ __forceinline__ void cell2(double c0, double c1, double n0, double n1, double s0,
                                      double s1, double e0, double e1, double w0, double w1,
                                      const CellArgs<double> &k, double &u0, double &u1)
{
    u0 = cell1(c0, n0, s0, e0, w0, k);
    u1 = cell1(c1, n1, s1, e1, w1, k);
}

template <typename T, int V> struct alignas(sizeof(T) * V) Vec {
    T v[V];
};
// values per 16-byte (R a multiple) or 8-byte access
template <typename T, int R> __host__ __device__ constexpr int vec_of()
{
    return sizeof(T) == 4 ? (R % 4 == 0 ? 4 : 2) : (R % 2 == 0 ? 2 : 1);
}

template <typename T, int V> __device__ __forceinline__ Vec<T, V> ldcg_vec(const T *p)
{
    Vec<T, V> r;
    if constexpr (sizeof(Vec<T, V>) == 16) {
        const int4 w = __ldcg(reinterpret_cast<const int4 *>(p));
        __builtin_memcpy(&r, &w, 16);
    } else {
        const int2 w = __ldcg(reinterpret_cast<const int2 *>(p));
        __builtin_memcpy(&r, &w, 8);
    }
    return r;
}

template <typename T> struct StripArgs {
    int nz, ny, nx, nxb;
    int rounds, W, B, P;  // warps per band and CTA, bands of 32 R rows, slots of the scratch
    int check;            // mark the planes out of range (a call's first launch)
    CellArgs<T> cell;
};

template <typename T, int R, int Q, bool FULL, bool CL>
__global__ void __launch_bounds__(512, 1)
k_diffusion_strips(T *__restrict__ u, T *__restrict__ scratch, int *__restrict__ flags,
                   StripArgs<T> a)
{
    constexpr int V = vec_of<T, R>(), NV = R / V;
    constexpr bool FLOAT = sizeof(T) == 4;
    using Vt = Vec<T, V>;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
    const int b = wi / a.W, w = wi - b * a.W, NW = a.W * a.B;
    int rank = 0, C = 1;
    if (CL) {
        rank = (int)cg::this_cluster().block_rank();
        C = (int)cg::this_cluster().num_blocks();
    }
    const int cluster = blockIdx.x / C, nclusters = gridDim.x / C;
    auto sync = [&]() {
        if (CL) cg::this_cluster().sync();
        else __syncthreads();
    };
    const int NR = 32 * R * a.B, P = a.P;
    const int K = Q * a.W * C, sw = Q * (rank * a.W + w);  // live sweeps; this warp's first
    const int y0 = 32 * R * b + R * lane;                  // this lane's first row
    T *S = scratch + (size_t)cluster * P * NR;
    // exchange buffers [2][band x warp][NV][32], then the bands' edges
    Vt *ex = reinterpret_cast<Vt *>(smraw);
    T *eN = reinterpret_cast<T *>(ex + (size_t)2 * NW * NV * 32);  // [2][NW][Q]
    T *eS = eN + 2 * NW * Q;                                       // [2][NW][Q]
    const bool first = rank == 0 && w == 0, last = rank == C - 1 && w == a.W - 1;
    // where this warp's results go: the next warp's input, or the next CTA's
    // first warp's
    Vt *out = ex + (size_t)(b * a.W + w + 1) * NV * 32 + lane;
    if (CL && w == a.W - 1 && !last)
        out = cg::this_cluster().map_shared_rank(ex, rank + 1) + (size_t)(b * a.W) * NV * 32 + lane;
    const Vt *in = ex + (size_t)(b * a.W + w) * NV * 32 + lane;
    const int exbuf = NW * NV * 32;
    unsigned mS = 0;  // rows whose S is clamped (the plane's last row)
    if (a.ny - 1 - y0 >= 0 && a.ny - 1 - y0 < R) mS = 1u << (a.ny - 1 - y0);
    // columns x with a special E: x == nxb - 1 (itself), else x == nx - 1 (0.0)
    const int xc = a.nxb <= a.nx ? a.nxb - 1 : -1, xz = a.nxb == a.nx ? -1 : a.nx - 1;
    const int span = a.rounds * P;
    const int nsteps = span - P + a.nx + a.ny - 2 + 2 * (K - 1) + 2;

    for (int pl = cluster; pl < a.nz; pl += nclusters) {
        T *U = u + (size_t)pl * a.ny * a.nx;
        // ---- skew the plane into S: slot x + y mod P, 32 x 32 tiles
        {
            T *tile = reinterpret_cast<T *>(smraw) + wi * 32 * 33;
            const int tr = NR / 32, tiles = tr * ((P + 31) / 32);
            bool big = false;
            for (int k = wi + NW * rank; k < tiles; k += NW * C) {
                const int g0 = (k / tr) * 32, r0 = (k % tr) * 32;
                int x = (g0 + lane - r0) % P;
                if (x < 0) x += P;
#pragma unroll 8
                for (int j = 0; j < 32; j++) {
                    T v = T(0);
                    if (r0 + j < a.ny && x < a.nx) v = U[(size_t)(r0 + j) * a.nx + x];
                    if (FLOAT && !(fabs(v) < T(kMaxF))) big = true;
                    tile[j * 33 + lane] = v;
                    x = x ? x - 1 : P - 1;
                }
                __syncwarp();
#pragma unroll 8
                for (int j = 0; j < 32; j++)
                    if (g0 + j < P) S[(size_t)(g0 + j) * NR + r0 + lane] = tile[lane * 33 + j];
                __syncwarp();
            }
            if (FLOAT && a.check && __any_sync(0xffffffffu, big) && lane == 0)
                atomicOr(flags + pl, 1);
            __threadfence();
            sync();
        }
        if (FLOAT && __ldcg(flags + pl)) {  // not this form's plane: left untouched
            sync();
            continue;
        }
        // X[q]: what stage q - 1 (q = 0: the input) produced one and two steps
        // ago, in the roles of the step's parity; the last stage needs one
        T X[Q][2][R], L[R];
        T pf[R], pfS = T(0);
#pragma unroll
        for (int i = 0; i < R; i++) {
#pragma unroll
            for (int q = 0; q < Q; q++) X[q][0][i] = X[q][1][i] = T(0);
            L[i] = T(0);
            pf[i] = T(0);
        }
        auto fetch = [&](int slot) {
            const T *src = S + (size_t)slot * NR + y0;
#pragma unroll
            for (int k = 0; k < NV; k++) {
                const Vt v = ldcg_vec<T, V>(src + k * V);
#pragma unroll
                for (int e = 0; e < V; e++) pf[k * V + e] = v.v[e];
            }
            if (a.B > 1 && lane == 31 && b + 1 < a.B) pfS = __ldcg(S + (size_t)slot * NR + y0 + R);
        };
        if (first) fetch(0);
        int slot_in = P > 1 ? 1 : 0;  // next slot to fetch
        // diagonal of this warp's first sweep minus y0, modulo P
        int cnt = (-1 - 2 * sw - y0) % P;
        if (cnt < 0) cnt += P;
        int d_out = -1 - 2 * (K - 1);  // diagonal the pipeline's last sweep is at
        int d_in = -1 - 2 * sw;           // ... this warp's first sweep
        int slot_out = d_out % P;
        if (slot_out < 0) slot_out += P;

        // One step, the exchange buffer `par` in and the other out.  ph: which of
        // X's two is the newest; the FP32 loop alternates it, the FP64 loop
        // (whose step is long) moves the values and keeps one copy of the code.
        auto step = [&](auto phc, int par) {
            constexpr int ph = decltype(phc)::value, pp = ph ^ 1;
            const int bi = par ? exbuf : 0, bo = par ? 0 : exbuf;
            // the warp has cells on its diagonals, or will in the next step
            const bool busy = d_in + 1 >= 32 * R * b && d_in - 2 * (Q - 1) - 32 * R * (b + 1) < span;
            // this step's input becomes the newest (over the oldest)
            T inS = T(0);
            if (!FLOAT)
#pragma unroll
                for (int i = 0; i < R; i++) X[0][pp][i] = X[0][ph][i];
            if (first) {
#pragma unroll
                for (int i = 0; i < R; i++) X[0][ph][i] = pf[i];
                inS = pfS;
                fetch(slot_in);
                slot_in = slot_in + 1 == P ? 0 : slot_in + 1;
            } else if (busy) {
#pragma unroll
                for (int k = 0; k < NV; k++) {
                    const Vt v = in[bi + k * 32];
#pragma unroll
                    for (int e = 0; e < V; e++) X[0][ph][k * V + e] = v.v[e];
                }
                if (a.B > 1 && lane == 31 && b + 1 < a.B)
                    inS = ex[bi + (size_t)((b + 1) * a.W + w) * NV * 32].v[0];
            }
            if (busy)
#pragma unroll
            for (int q = Q - 1; q >= 0; q--) {
                // E: newest of the stage before, C: the one before it.  For
                // q >= 1 the stage before has not yet run this step: its
                // newest is the previous step's
                const T *E = q == 0 ? X[0][ph] : X[q][pp];
                const T *Cc = q == 0 ? X[0][pp] : X[q][ph];
                // own results of the previous step, and where this step's go
                // (the last stage writes over its own, bottom row first)
                const T *O = q == Q - 1 ? L : X[q + 1][pp];
                T *D = q == Q - 1 ? L : X[q + 1][ph];
                T nTop = __shfl_up_sync(0xffffffffu, O[R - 1], 1);
                T sBot = __shfl_down_sync(0xffffffffu, E[0], 1);
                if (a.B > 1) {
                    const int eb = par ? NW * Q : 0;
                    if (lane == 0 && b > 0) nTop = eN[eb + ((b - 1) * a.W + w) * Q + q];
                    if (lane == 31 && b + 1 < a.B)
                        sBot = q == 0 ? inS : eS[eb + ((b + 1) * a.W + w) * Q + q];
                }
                if (y0 == 0) nTop = Cc[0];
                int cq = cnt - 2 * q;
                if (cq < 0) cq += P;
                int ce = cq - xc, cz = cq - xz;
                if (ce < 0) ce += P;
                if (cz < 0) cz += P;
                const unsigned mW = bit_at(cq), mE = xc >= 0 ? bit_at(ce) : 0u,
                               mZ = xz >= 0 ? bit_at(cz) : 0u;
#pragma unroll
                for (int i = R - 2; i >= 0; i -= 2) {
                    const T c0 = Cc[i], c1 = Cc[i + 1];
                    T n0 = i ? O[i - 1] : nTop, n1 = O[i];
                    T s0 = E[i + 1], s1 = i + 2 < R ? E[i + 2] : sBot;
                    T w0 = mW & (1u << i) ? c0 : O[i], w1 = mW & (2u << i) ? c1 : O[i + 1];
                    T e0 = mZ & (1u << i) ? T(0) : E[i], e1 = mZ & (2u << i) ? T(0) : E[i + 1];
                    if (mE & (1u << i)) e0 = c0;
                    if (mE & (2u << i)) e1 = c1;
                    if (!FULL && (mS & (1u << i))) s0 = c0;
                    if ((!FULL || i + 2 == R) && (mS & (2u << i))) s1 = c1;
                    T u0, u1;
                    cell2(c0, c1, n0, n1, s0, s1, e0, e1, w0, w1, a.cell, u0, u1);
                    D[i] = u0;
                    D[i + 1] = u1;
                }
                if (a.B > 1) {
                    const int eb = par ? 0 : NW * Q;
                    if (lane == 31) eN[eb + (b * a.W + w) * Q + q] = D[R - 1];
                    if (lane == 0 && q + 1 < Q) eS[eb + (b * a.W + w) * Q + q + 1] = D[0];
                }
            }
            if (!busy) {
            } else if (!last) {
#pragma unroll
                for (int k = 0; k < NV; k++) {
                    Vt v;
#pragma unroll
                    for (int e = 0; e < V; e++) v.v[e] = L[k * V + e];
                    out[bo + k * 32] = v;
                }
            } else {
                // the rows whose cell lies in this plane's rounds
                T *dst = S + (size_t)slot_out * NR + y0;
                const int x = d_out - y0;
                if (x - (R - 1) >= 0 && x < span) {
#pragma unroll
                    for (int k = 0; k < NV; k++) {
                        Vt v;
#pragma unroll
                        for (int e = 0; e < V; e++) v.v[e] = L[k * V + e];
                        *reinterpret_cast<Vt *>(dst + k * V) = v;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < R; i++)
                        if (x - i >= 0 && x - i < span) dst[i] = L[i];
                }
            }
            cnt = cnt + 1 == P ? 0 : cnt + 1;
            d_out++;
            d_in++;
            slot_out = slot_out + 1 == P ? 0 : slot_out + 1;
            sync();
        };
        if constexpr (FLOAT) {
            for (int n = 0; n < nsteps; n += 2) {
                step(std::integral_constant<int, 0>(), 0);
                step(std::integral_constant<int, 1>(), 1);
            }
        } else {
            for (int n = 0; n < nsteps; n++) step(std::integral_constant<int, 0>(), n & 1);
        }
        // ---- and out of S again
        {
            T *tile = reinterpret_cast<T *>(smraw) + wi * 32 * 33;
            const int tr = NR / 32, tiles = tr * ((P + 31) / 32);
            for (int k = wi + NW * rank; k < tiles; k += NW * C) {
                const int g0 = (k / tr) * 32, r0 = (k % tr) * 32;
                if (r0 >= a.ny) continue;
#pragma unroll 8
                for (int j = 0; j < 32; j++)
                    if (g0 + j < P)
                        tile[lane * 33 + j] = __ldcg(S + (size_t)(g0 + j) * NR + r0 + lane);
                __syncwarp();
                int x = (g0 + lane - r0) % P;
                if (x < 0) x += P;
#pragma unroll 8
                for (int j = 0; j < 32; j++) {
                    if (g0 + lane < P && r0 + j < a.ny && x < a.nx)
                        U[(size_t)(r0 + j) * a.nx + x] = tile[j * 33 + lane];
                    x = x ? x - 1 : P - 1;
                }
                __syncwarp();
            }
            sync();
        }
    }
}

template <typename T, int R, int Q> size_t strips_smem(int W, int B)
{
    const size_t ex = sizeof(T) * (size_t)2 * W * B * R * 32 + sizeof(T) * 4 * (size_t)W * B * Q;
    const size_t tile = sizeof(T) * 32 * 33 * (size_t)W * B;
    return ex > tile ? ex : tile;
}

template <typename T, int R, int Q>
int launch_strips(T *u, T *scratch, int *flags, const StripArgs<T> &a, int C, int clusters,
                  cudaStream_t st)
{
    const size_t smem = strips_smem<T, R, Q>(a.W, a.B);
    const bool full = a.ny == 32 * R * a.B;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * C);
    cfg.blockDim = dim3(32 * a.W * a.B);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = C > 1 ? 1 : 0;
#define NUDIM_STRIPS(FU, CLU)                                                                     \
    do {                                                                                         \
        NUDIM_CUDA(cudaFuncSetAttribute(k_diffusion_strips<T, R, Q, FU, CLU>,                    \
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, 160 << 10)); \
        NUDIM_CUDA(cudaLaunchKernelEx(&cfg, k_diffusion_strips<T, R, Q, FU, CLU>, u, scratch,    \
                                      flags, a));                                                \
    } while (0)
    if (C > 1) {
        if (full) NUDIM_STRIPS(true, true);
        else NUDIM_STRIPS(false, true);
    } else {
        if (full) NUDIM_STRIPS(true, false);
        else NUDIM_STRIPS(false, false);
    }
#undef NUDIM_STRIPS
    NUDIM_LAUNCH_CHECK();
    return NUDIM_OK;
}

int sm_count()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 152;  // a footprint asked for where no GPU is: the target's
    return sms;
}

bool cell_args(double lambda, double ksq, CellArgs<float> *c)
{
    c->ksq = (float)ksq;
    c->lk = (float)lambda * (float)ksq;
    return true;
}
bool cell_args(double lambda, double ksq, CellArgs<double> *c)
{
    c->lambda = lambda;
    return diff_div_init(ksq, &c->div);
}

// strips of RR rows, if the form has them in this precision
template <typename T, int RR>
int launch_rows(const StripShape &s, T *u, T *S, int *flags, const StripArgs<T> &a, cudaStream_t st)
{
    if constexpr (sizeof(T) == 8) {
        if constexpr (RR <= 2) return launch_strips<T, RR, 1>(u, S, flags, a, s.C, s.clusters, st);
        set_error("diffusion: no strip of %d rows", RR);
        return NUDIM_EINVAL;
    } else {
        return s.Q == 2 ? launch_strips<T, RR, 2>(u, S, flags, a, s.C, s.clusters, st)
                        : launch_strips<T, RR, 1>(u, S, flags, a, s.C, s.clusters, st);
    }
}

}  // namespace

// The form's range.  FP32: |lambda| small enough that the sweeps keep values
// within the pair form's bounds (a sweep moves a value by at most 2 |lambda| K).
template <typename T>
bool strips_fits(int ny, int nx, int niter, double lambda, double ksq)
{
    if (ny < 1 || nx < 1 || nx > kStripsMaxNx || ny > kBandRows<T> * 16 || niter < 1) return false;
    CellArgs<T> c;
    if (sizeof(T) == 8) return cell_args(lambda, ksq, &c);
    return ksq >= kMinKsq && ksq <= kMaxKsq &&
           std::fabs(lambda) * std::sqrt(ksq) * 2 * niter < 0.1 * kMaxF;
}

// scratch of strips_run: a flag per plane, then a skewed plane per cluster
template <typename T> size_t strips_scratch(int nz, int ny, int nx, int niter)
{
    size_t most = 0;
    for (int left = niter; left > 0;) {
        const StripShape s = strip_shape<T>(nz, ny, nx, left, sm_count());
        most = std::max(most, sizeof(T) * (size_t)s.clusters * s.P * 32 * s.R * s.B);
        left -= strip_rounds(s, ny, nx, left) * s.k;
    }
    return most + strips_flag_bytes(nz);
}

template <typename T>
int strips_run(T *u, int nz, int ny, int nx, int nxb, double lambda, double ksq, int niter,
               void *scratch, cudaStream_t st)
{
    int *flags = (int *)scratch;
    T *S = (T *)((char *)scratch + strips_flag_bytes(nz));
    StripArgs<T> a;
    if (!cell_args(lambda, ksq, &a.cell)) {
        set_error("diffusion: kappa out of the strip form's range");
        return NUDIM_EINVAL;
    }
    if (sizeof(T) == 4) NUDIM_CUDA(cudaMemsetAsync(flags, 0, strips_flag_bytes(nz), st));
    for (int left = niter; left > 0;) {
        const StripShape s = strip_shape<T>(nz, ny, nx, left, sm_count());
        const int rounds = strip_rounds(s, ny, nx, left);
        a.nz = nz;
        a.ny = ny;
        a.nx = nx;
        a.nxb = nxb;
        a.rounds = rounds;
        a.W = s.W;
        a.B = s.B;
        a.P = s.P;
        a.check = left == niter;
        int rc = NUDIM_EINVAL;
        switch (s.R) {
        case 2: rc = launch_rows<T, 2>(s, u, S, flags, a, st); break;
        case 4: rc = launch_rows<T, 4>(s, u, S, flags, a, st); break;
        case 6: rc = launch_rows<T, 6>(s, u, S, flags, a, st); break;
        case 8: rc = launch_rows<T, 8>(s, u, S, flags, a, st); break;
        case 10: rc = launch_rows<T, 10>(s, u, S, flags, a, st); break;
        case 12: rc = launch_rows<T, 12>(s, u, S, flags, a, st); break;
        default: set_error("diffusion: no strip of %d rows", s.R);
        }
        NUDIM_TRY(rc);
        left -= rounds * s.k;
    }
    return NUDIM_OK;
}

template bool strips_fits<float>(int, int, int, double, double);
template bool strips_fits<double>(int, int, int, double, double);
template size_t strips_scratch<float>(int, int, int, int);
template size_t strips_scratch<double>(int, int, int, int);
template int strips_run<float>(float *, int, int, int, int, double, double, int, void *,
                               cudaStream_t);
template int strips_run<double>(double *, int, int, int, int, double, double, int, void *,
                                cudaStream_t);

}  // namespace nudim
