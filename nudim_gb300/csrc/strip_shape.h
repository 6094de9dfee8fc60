// strip_shape.h -- how the strip form of the diffusion (strips.cu) cuts a launch.
// Host code: the CPU tests compile it by itself.
#pragma once

#include <algorithm>

namespace nudim {

// How a launch cuts its planes: strips of R rows (even), B bands of 32 R rows, W
// warps per band and CTA of Q sweeps each, C CTAs of a cluster per plane: k =
// Q W C live sweeps.
struct StripShape {
    int R, B, W, Q, C, k, P, clusters;
};

// rows of a band: strips of up to 12 (FP32) or 2 (FP64) rows
template <typename T> constexpr int kBandRows = sizeof(T) == 4 ? 384 : 64;

// The next launch's shape with `left` sweeps to go.
//
// FP32: 16 live sweeps (or what 16 warps hold): more of them waste more on the
// pipeline's ends, fewer leave the SM idle (256 x 384 x 384: 8 sweeps 4.60, 10
// 5.28, 16 4.40, 20 5.84 ms).  Two sweeps a warp halve the exchange and let two
// CTAs share an SM; with a plane per SM or fewer, one sweep a warp on twice the
// warps (64 x 128 x 128: 386 -> 335 us, 96 x 384 x 384 2.65 -> 2.28 ms; 256
// planes of 384 x 384: 4.40 -> 4.56 ms the other way round).  Where four CTAs a
// plane still find an SM each and the strips are at least 6 rows, a cluster of
// four with 40 live sweeps (33 x 151 x 203: 715 -> 592 us; 16 x 64 x 64, strips
// of 2 rows: 145 -> 208 us, the cluster's barrier at each step costs more than
// the rest of the step).
//
// FP64: the step is long (integer and FP64 units; 64 x 128 x 128: 38.0 ms for
// the tables form with the FP64 unit's divisions, 4.0 here) and a plane on one
// SM leaves the others idle, so a plane takes a cluster of as many CTAs as
// bring the turns per SM down (64 planes: 1 CTA 7.32 ms, 2 3.97, 4 3.94, 8 3.96;
// 32: 4 2.63, 8 2.55; equal turns: the smaller one), strips of 2 rows on up to
// 16 warps (strips of 4 on half the warps: 6.6 against 5.3 ms, one warp's
// dependent instructions bound it), 16 live sweeps; 40 where there are fewer
// planes than clusters of 8 (9 x 100 x 130: 1.93 -> 1.70 ms).
template <typename T> StripShape strip_shape(int nz, int ny, int nx, int left, int sms)
{
    StripShape s;
    s.B = (ny + kBandRows<T> - 1) / kBandRows<T>;
    const int r = (ny + 32 * s.B - 1) / (32 * s.B);
    s.R = r + (r & 1);
    s.C = 1;
    if (sizeof(T) == 8) {
        s.Q = 1;
        auto turns = [&](long long c) { return (nz * c + sms - 1) / sms; };
        for (int c = 2; c <= 8 && 2 * c <= left; c *= 2)
            if (turns(c) * s.C < turns(s.C) * c) s.C = c;
        const int most = s.C == 8 && turns(8) == 1 && left >= 40 ? 40 : 16;
        s.W = std::max(1, std::min({16 / s.B, most / s.C, left / s.C}));
        for (int w = s.W; 2 * w > s.W; w--)
            if (left % (w * s.C) == 0) {
                s.W = w;
                break;
            }
        s.k = s.W * s.C;
    } else if (s.B == 1 && s.R >= 6 && nz <= sms / 4 && left >= 40) {
        s.C = 4;
        s.k = 40;
        s.Q = 1;
    } else {
        s.k = std::min(left, std::min(16, 16 / s.B * 2));
        if (s.k % 2 && s.k * s.B > 16) s.k--;
        s.Q = s.k % 2 || (nz <= sms && s.B == 1) ? 1 : 2;
    }
    s.W = s.k / (s.Q * s.C);
    // the ring outlasts the pipeline: a slot is written 2 (k - 1) steps after it
    // was read, and read again a step before it comes round.  And a strip's rows
    // lie at R different columns modulo P, so that one of them at most is at a
    // boundary column: a mask is one bit.
    s.P = std::max({nx, 2 * s.k + 4, s.R});
    const int per = std::max(1, 16 / (s.W * s.B));  // CTAs an SM holds (128 registers)
    s.clusters = std::max(1, std::min(nz, sms * per / s.C));
    return s;
}

// Rounds of the next launch, k sweeps each.  The kernel counts a launch's steps
// and diagonals, rounds P + nx + ny + 2 k of them, in 32 bits.
constexpr int kStripsMaxNx = 1 << 28;
inline int strip_rounds(const StripShape &s, int ny, int nx, int left)
{
    const long long most = ((1ll << 30) - nx - ny - 2 * s.k) / s.P;
    return (int)std::min<long long>(left / s.k, most);
}

}  // namespace nudim
