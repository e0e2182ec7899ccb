// The bound field's potential psi = (rho + gamma^-2 d_zeta^2 rho / k_perp^2) / k_perp^2 of the slice charge (the Fourier-y
// lambda of src/sim_fields.cpp:176-201) at one slice, in both forms. rho of a slice is w_lo, w_hi of its two half-cells and
// the second difference takes three slices, so psi is a combination of four half-cells' j_z whose six weights depend on
// the slice alone: a CTA makes them once, and a mode costs four loads and one quotient. (Six loads and seven quotients
// before, two of them in the weights: inside the sponge's first columns kernel 424 -> 235 us at 128 x 128 x 1024.)
#pragma once
#include "g3d_ctx.hpp"

namespace g3d {

// T: the storage of j_z (ns + 1 half-cell planes); jg: its two ghost half-cells below and above the slab, or null (zero)
template <class T>
struct BoundPsi {
    const T* h[4];               // half-cells l - 1 .. l + 2
    double r1, r2, e[4];         // rho = r1 h1 + r2 h2; gamma^-2 d_zeta^2 rho = sum e h
    __device__ __forceinline__ BoundPsi(const Geo& g, const T* jz, const T* jg, int l, double g2) {
        const int n = g.a + l;
        double s[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int hk = l - 1 + k;
            const bool below = hk < 0, above = hk > g.ns;
            s[k] = (below || above) && !jg ? 0.0 : 1.0;
            const int hc = below ? 0 : above ? g.ns : hk;        // without a ghost: a plane of this slice's rho, weight zero
            h[k] = jg && below ? jg : jg && above ? jg + g.nkh : jz + long(hc) * g.nkh;
        }
        const double hm = g.hcg[n + 1], hp = g.hcg[n + 2];
        const double cm = 2 / ((hm + hp) * hm), cp = 2 / ((hm + hp) * hp);
        const double lm = n > 0 ? g.wlo[n - 1] : 0.0, um = n > 0 ? g.whi[n - 1] : 0.0;
        const double lp = n < g.N - 1 ? g.wlo[n + 1] : 0.0, up = n < g.N - 1 ? g.whi[n + 1] : 0.0;
        r1 = s[1] * g.wlo[n]; r2 = s[2] * g.whi[n];
        e[0] = s[0] * g2 * (cm * lm);
        e[1] = s[1] * g2 * (cm * um - (cm + cp) * g.wlo[n]);
        e[2] = s[2] * g2 * (cp * lp - (cm + cp) * g.whi[n]);
        e[3] = s[3] * g2 * (cp * up);
    }
    __device__ __forceinline__ cpx at(long i, double k2) const {
        const cpx a = widen(__ldg(h[0] + i)), b = widen(__ldg(h[1] + i)), c = widen(__ldg(h[2] + i)), d = widen(__ldg(h[3] + i));
        const double ik2 = k2 > 0 ? 1 / k2 : 0.0;
        const cpx rho = r1 * b + r2 * c, d2 = e[0] * a + e[1] * b + (e[2] * c + e[3] * d);
        return ik2 * (rho + ik2 * d2);
    }
};

}  // namespace g3d
