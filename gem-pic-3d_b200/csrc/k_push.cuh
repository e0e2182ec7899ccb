// Device functions of the beam push shared by the push (k_push.cu) and its adjoint (k_adjoint.cu), so that the
// adjoint recomputes the forward trajectory with the same arithmetic: the gather of the grid fields (TSC in x
// and y, linear in zeta; reference gather, src/sim_kernels.hpp:44-72) and the right-hand side of the
// characteristics (rhs, sim_kernels.hpp:75-92). FT is the element type of the real-space fields: float (the
// reference's F) or double (the exact fields of the gradient check).
#pragma once
#include "g3d_plasma.hpp"
#include "k_external.cuh"

namespace g3d {

struct PushArgs {
    const float* __restrict__ F;
    const double* __restrict__ Fd;        // exact fields (FP64 copy of F) or null
    Geo g;
    LaserDev laser;
    double X0, Y0, zc, dz_push, push_phase, zhand, zmax, ylo, yhi, s1, vz_min, hmin;
    int freeze, self;
    ExtDev ext;                           // external magnetic elements (none: nu = nm = 0)
};

struct St { double x, y, zeta, px, py, pz; };

PushArgs push_args(Ctx& c, double s1);          // the arguments of the push to the plane s1 (k_push.cu)

template <class FT>
__device__ __forceinline__ void gather(const PushArgs& c, const FT* __restrict__ Fp, double x, double y, double zeta, double E[3],
                                       double B[3]) {
    E[0] = E[1] = E[2] = B[0] = B[1] = B[2] = 0;
    if (!c.self) return;
    const Geo& g = c.g;
    int n; double fz;
    g.zax.locate(zeta, n, fz);
    if (n == g.a - 1 && fz > 1 - 1e-9) { n = g.a; fz = 0; }    // on the lowest slice (rounding of locate)
    const int fl = n - g.a;
    if (fl < 0 || fl > g.ns) return;
    int ix[3], jn[3]; double wx[3], wn[3];
    tsc_periodic(x, g.dx, g.nx, ix, wx);
    const long nk = g.nk;
    if (!g.yf) {                       // free-hand y: E_y, B_x, B_z on the half-nodes, nothing beyond the walls
        int jh[3]; double wh[3];
        tsc_y(g.yax, y, jn, wn, jh, wh);
        for (int comp = 0; comp < 6; ++comp) {
            const FT* p0 = Fp + (long(comp) * (g.ns + 2) + fl) * nk;
            const FT* p1 = p0 + nk;
            const bool hf = is_half(comp);
            const int* jj = hf ? jh : jn;
            const double* wy = hf ? wh : wn;
            double v = 0;
            for (int j = 0; j < 3; ++j) {
                if (jj[j] < 0 || jj[j] >= g.ny) continue;
                for (int i = 0; i < 3; ++i) {
                    const long k = long(jj[j]) * g.nx + ix[i];
                    v += wx[i] * wy[j] * ((1 - fz) * double(__ldg(p0 + k)) + fz * double(__ldg(p1 + k)));
                }
            }
            if (comp < 3) E[comp] = v; else B[comp - 3] = v;
        }
        return;
    }
    tsc_periodic(y, g.dy, g.ny, jn, wn);
#pragma unroll
    for (int comp = 0; comp < 6; ++comp) {
        const FT* p0 = Fp + (long(comp) * (g.ns + 2) + fl) * nk;
        const FT* p1 = p0 + nk;
        double v = 0;
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const long k = long(jn[j]) * g.nx + ix[i];
                v += wx[i] * wn[j] * ((1 - fz) * double(__ldg(p0 + k)) + fz * double(__ldg(p1 + k)));
            }
        if (comp < 3) E[comp] = v; else B[comp - 3] = v;
    }
}

// The gather from a held stencil (Fourier y, float F): the 3 x 3 x 2 points of the six components are loaded into shared
// memory when the particle's first point or half-cell is another than the held one, and the gathers that follow take them
// from there. The four stages of a sub-step, and mostly the sub-steps of a push, stay inside one cell and half-cell, so
// a push loads them once or twice instead of four times per sub-step.
constexpr int PUSH_NT = 128;             // threads of the push kernel
struct HeldStencil {
    int fl = -1, ix = -1, jn = -1;        // first plane and first point held (none: -1)
    int n = -1;                           // the half-cell the zeta axis was last located in, between z0 and z1
    double z0 = 0, z1 = 0;
    float* f;                             // this thread's slots of shared memory: per component the nine points of plane fl, then
                                          // of fl + 1, a CTA of PUSH_NT threads' slots side by side
    __device__ __forceinline__ float& at(int comp, int q) { return f[(comp * 18 + q) * PUSH_NT]; }
};
__device__ __forceinline__ void gather(const PushArgs& c, const float* __restrict__ Fp, HeldStencil& H, double x, double y,
                                       double zeta, double E[3], double B[3]) {
    E[0] = E[1] = E[2] = B[0] = B[1] = B[2] = 0;
    if (!c.self) return;
    const Geo& g = c.g;
    int n; double fz;
    if (H.n >= 0 && zeta >= H.z0 && zeta < H.z1) {       // inside the located cell: the axis' own fraction
        n = H.n;
        fz = (zeta - H.z0) / (H.z1 - H.z0);
    } else {
        g.zax.locate(zeta, n, fz);
        H.n = -1;
        if (!g.zax.uniform && n >= 0 && n < g.N - 1) { H.n = n; H.z0 = g.zax.X[n]; H.z1 = g.zax.X[n + 1]; }
    }
    if (n == g.a - 1 && fz > 1 - 1e-9) { n = g.a; fz = 0; }    // on the lowest slice (rounding of locate)
    const int fl = n - g.a;
    if (fl < 0 || fl > g.ns) return;
    int ix[3], jn[3]; double wx[3], wn[3];
    tsc_periodic(x, g.dx, g.nx, ix, wx);
    tsc_periodic(y, g.dy, g.ny, jn, wn);
    if (fl != H.fl || ix[0] != H.ix || jn[0] != H.jn) {
        const long nk = g.nk;
#pragma unroll
        for (int j = 0; j < 3; ++j)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const float* p = Fp + long(fl) * nk + (jn[j] * g.nx + ix[i]);
#pragma unroll
                for (int comp = 0; comp < 6; ++comp) {
                    const float* q = p + long(comp) * (g.ns + 2) * nk;
                    H.at(comp, 3 * j + i) = __ldg(q); H.at(comp, 9 + 3 * j + i) = __ldg(q + nk);
                }
            }
        H.fl = fl; H.ix = ix[0]; H.jn = jn[0];
    }
    double v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double w = wx[i] * wn[j], w0 = (1 - fz) * w, w1 = fz * w;
#pragma unroll
            for (int comp = 0; comp < 6; ++comp)
                v[comp] += w0 * double(H.at(comp, 3 * j + i)) + w1 * double(H.at(comp, 9 + 3 * j + i));
        }
#pragma unroll
    for (int k = 0; k < 3; ++k) { E[k] = v[k]; B[k] = v[3 + k]; }
}
// no stencil held: the plain gather
struct NoStencil {};
template <class FT>
__device__ __forceinline__ void gather(const PushArgs& c, const FT* __restrict__ Fp, NoStencil&, double x, double y, double zeta,
                                       double E[3], double B[3]) {
    gather(c, Fp, x, y, zeta, E, B);
}

template <class FT, class Hold>
__device__ __forceinline__ bool rhs(const PushArgs& c, const FT* __restrict__ Fp, Hold& H, const St& Y, double z, double qm, St& d) {
    const double g = sqrt(1 + Y.px * Y.px + Y.py * Y.py + Y.pz * Y.pz);
    if (Y.pz < 0.3 * g) return false;
    const double gm = (1 + Y.px * Y.px + Y.py * Y.py) / (g + Y.pz);
    double E[3], B[3], Ee[3], Be[3];
    gather(c, Fp, H, wrap_periodic(Y.x, c.g.Lx), c.g.yf ? wrap_periodic(Y.y, c.g.Ly) : Y.y, Y.zeta, E, B);
    c.laser.field(Y.x + c.X0, z, z - (Y.zeta - c.zc), Ee, Be);
#pragma unroll
    for (int k = 0; k < 3; ++k) { E[k] += Ee[k]; B[k] += Be[k]; }
    if (c.ext.any()) add_external(c.ext, Y.x + c.X0, Y.y + c.Y0, z, B);
    const double ip = 1 / Y.pz;
    d.x = Y.px * ip; d.y = Y.py * ip; d.zeta = -gm * ip;
    d.px = qm * (g * E[0] + Y.py * B[2] - Y.pz * B[1]) * ip;
    d.py = qm * (g * E[1] + Y.pz * B[0] - Y.px * B[2]) * ip;
    d.pz = qm * (g * E[2] + Y.px * B[1] - Y.py * B[0]) * ip;
    return true;
}
// The next sub-step from z towards s1: at most dz_push, at most push_phase of the laser phase, and a zeta
// advance of at most hmin/2 (reference push_one, src/sim_kernels.hpp:110-125)
__device__ __forceinline__ double substep(const PushArgs& c, const St& Y, double z, double s1) {
    double ds = c.dz_push < s1 - z ? c.dz_push : s1 - z;
    {
        const double g = sqrt(1 + Y.px * Y.px + Y.py * Y.py + Y.pz * Y.pz);
        const double lz = 0.5 * c.hmin * Y.pz * (g + Y.pz) / (1 + Y.px * Y.px + Y.py * Y.py);
        if (lz < ds) ds = (s1 - z) / ceil((s1 - z) / lz);
    }
    if (c.laser.on) {
        const double g = sqrt(1 + Y.px * Y.px + Y.py * Y.py + Y.pz * Y.pz);
        const double hl = g - Y.px * c.laser.kx - Y.pz * c.laser.kz;
        const double lim = c.push_phase * Y.pz / (c.laser.kL * (hl > 1e-12 ? hl : 1e-12));
        if (lim < ds) ds = (s1 - z) / ceil((s1 - z) / lim);
    }
    if (c.ext.any()) ds = external_step(c.ext, z, ds);       // the external elements resolved
    return ds;
}
__device__ __forceinline__ St axpy(const St& a, double h, const St& b) {
    return St{a.x + h * b.x, a.y + h * b.y, a.zeta + h * b.zeta, a.px + h * b.px, a.py + h * b.py, a.pz + h * b.pz};
}

// One RK4 sub-step of length ds from z (reference push_one, src/sim_kernels.hpp:126-143); k1 + 2 k2 + 2 k3 + k4
// summed left to right as each stage completes (fewer live registers). False: the particle is too slow
// (rhs), and Y is left unchanged.
template <class FT, class Hold>
__device__ __forceinline__ bool rk4_step(const PushArgs& c, const FT* __restrict__ Fp, Hold& H, St& Y, double z, double ds, double qm) {
    St k{0, 0, 0, 0, 0, 0}, acc = k;
    // with external elements the first and last stages take the field just inside the sub-step, which ends on the
    // elements' breakpoints, where the field or its derivative jumps
    const double e = c.ext.any() ? 1e-9 * ds : 0.0;
    // one copy of the stage's code: four inlined ones hold twice the registers and four times the instructions
#pragma unroll 1
    for (int stage = 0; stage < 4; ++stage) {
        const double a = stage == 0 ? 0.0 : stage == 3 ? ds : 0.5 * ds, za = stage == 0 ? z + e : stage == 3 ? z + ds - e : z + 0.5 * ds;
        if (!rhs(c, Fp, H, axpy(Y, a, k), za, qm, k)) return false;
        acc = axpy(acc, stage == 0 || stage == 3 ? 1.0 : 2.0, k);
    }
    const double w = ds / 6;
    Y.x += w * acc.x; Y.y += w * acc.y; Y.zeta += w * acc.zeta;
    Y.px += w * acc.px; Y.py += w * acc.py; Y.pz += w * acc.pz;
    return true;
}
template <class FT>
__device__ __forceinline__ bool rk4_step(const PushArgs& c, const FT* __restrict__ Fp, St& Y, double z, double ds, double qm) {
    NoStencil none;
    return rk4_step(c, Fp, none, Y, z, ds, qm);
}

}  // namespace g3d
