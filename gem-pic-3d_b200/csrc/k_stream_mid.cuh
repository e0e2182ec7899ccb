// Pieces of the streaming push (k_plasma.cu) that a host harness runs on the CPU as well (tests/stream_mid_check.cu): gamma and
// the time of a half-cell, the TSC of the Fourier y grid and the gather of the midpoint fields.
#pragma once
#include <type_traits>
#include "g3d_plasma.hpp"

namespace g3d {

// gamma = sqrt(a) from r, the reciprocal root of a to a unit in its last place (which the push needs as well): a r is off by up
// to 1.5 units, and a Newton step on the residual (exact in the FMA) leaves the root's own rounding. gamma + p_z needs that: for
// a particle that runs backwards the sum cancels, to 1 / (2 |p_z|) of two numbers of size |p_z|, and with a r alone it lost
// half as many bits again and from |p_z| ~ 5e7 on came out zero or negative. (A root beside the reciprocal root is some 20
// instructions; this is three.) Never below |p_z| when a >= p_z^2.
G3D_HD double gamma_root(double a, double r) {
    const double t = a * r;
    return fma(fma(-t, t, a), 0.5 * r, t);
}
// dt = 2 hl / ((1 - v_z)_0 + (1 - v_z)_1) with 1 - v_z = N / D, over the common denominator; D = 0 (gamma + p_z below the
// resolution of FP64): the time is zero, as with the quotients N / D = infinity
G3D_HD double halfcell_time(double hl, double N0, double D0, double N1, double D1) {
    const double den = N0 * D1 + N1 * D0;
    return den > 0 ? 2 * hl * D0 * D1 / den : 0.0;
}
// The streaming push's TSC on a periodic grid: the cell coordinate t = x / d and the nearest node in FP64 (x spans the
// box, so the index needs the double), the offset from that node and the three weights in W.
// x may lie outside the box: the first index is wrapped (its two neighbours by a compare), and as a particle is rarely
// more than a cell outside, the remainder (some twenty instructions) is behind a branch.
template <class W>
G3D_HD void tsc_stream(double x, double inv_d, int n, int idx[3], W w[3]) {
    const double t = x * inv_d;
    const double c = floor(t + 0.5);
    const W f = W(t - c);
    w[0] = W(0.5) * (W(0.5) - f) * (W(0.5) - f);
    w[1] = W(0.75) - f * f;
    w[2] = W(0.5) * (W(0.5) + f) * (W(0.5) + f);
    int b = int(c) - 1;
    if (unsigned(b) >= unsigned(n)) { b %= n; if (b < 0) b += n; }
    const int b1 = b + 1 == n ? 0 : b + 1;
    idx[0] = b; idx[1] = b1; idx[2] = b1 + 1 == n ? 0 : b1 + 1;
}
// The gather half-way through the half-cell (zeta = the slice midpoint, a particle crossing the whole half-cell):
// TSC in x and y of the interleaved midpoint fields, two (FP32) or three (FP64) vector loads per point (Fourier y). W: the type
// of the offsets and weights; the products and the sums are in the form's own precision.
template <bool F32, class W>
G3D_HD void sgather_mid(const StreamArgs& c, double x, double y, double E[3], double B[3]) {
    typedef typename std::conditional<F32, float, double>::type R;
    int ix[3], jn[3]; W wx[3], wn[3];
    tsc_stream<W>(x, c.inv_dx, c.g.nx, ix, wx);
    tsc_stream<W>(y, c.inv_dy, c.g.ny, jn, wn);
    R a[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const int k0 = jn[j] * c.g.nx;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int k = k0 + ix[i];
            const R w = R(wx[i] * wn[j]);
            if constexpr (F32) {
                const float4* p = static_cast<const float4*>(c.Fmid) + 2 * k;
                const float4 u = p[0], v = p[1];
                a[0] += w * u.x; a[1] += w * u.y; a[2] += w * u.z; a[3] += w * u.w; a[4] += w * v.x; a[5] += w * v.y;
            } else {
                const double2* p = static_cast<const double2*>(c.Fmid) + 3 * k;
                const double2 u = p[0], v = p[1], q = p[2];
                a[0] += w * u.x; a[1] += w * u.y; a[2] += w * v.x; a[3] += w * v.y; a[4] += w * q.x; a[5] += w * q.y;
            }
        }
    }
    E[0] = double(a[0]); E[1] = double(a[1]); E[2] = double(a[2]);
    B[0] = double(a[3]); B[1] = double(a[4]); B[2] = double(a[5]);
}
// The weights of the push: FP32 in the mixed form's common variant, whose fields are FP32 throughout; FP64, with only their
// products rounded to FP32, where the mixed form adds an analytic wave or an external element (evaluated in FP64), and in the FP64
// form. The choice costs the common variant nothing (step of 256 x 256 x 2048 mixed 255.5 and 255.1 ms without and with it).
template <bool F32, bool LASER>
G3D_HD void sgather_midpoint(const StreamArgs& c, double x, double y, double E[3], double B[3]) {
    if constexpr (F32 && !LASER) {
        if (!c.ext.any()) { sgather_mid<F32, float>(c, x, y, E, B); return; }
    }
    sgather_mid<F32, double>(c, x, y, E, B);
}

}  // namespace g3d
