// The co-moving start field per mode (Simulation::comoving_field, src/sim_fields.cpp:44-151) in both forms (T: the storage
// of j_z, E_z, B_z): the tridiagonal system of -(k_perp^2 + gamma^-2 d_zeta^2) psi = rho along zeta, then
// R = -(1 + beta) i k psi, E_z = B_z = 0.
//
// One thread per mode sweeping the slices twice (k_comoving, k_comoving_mixed) is a chain of 2 ns quotients whatever the
// grid: 0.98 ms for the 2,112 modes x 512 slices of a 64 x 64 grid. Here a CTA solves a mode by parallel cyclic reduction
// in shared memory (ceil(log2 ns) halvings; the system is diagonally dominant). beta = 1 (gamma^-2 = 0, the second solve of
// every start) has no off-diagonals: a pointwise quotient. The two solves of that grid's start: 1.96 -> 0.12 ms. The sweep
// stays for windows of many modes, which fill the chip with chains, and for rows that do not fit shared memory (pcr_modes).
#pragma once
#include <type_traits>
#include "g3d_ctx.hpp"

namespace g3d {

template <class T>
__device__ __forceinline__ void comoving_store(long o, double kx, double ky, double opb, cpx psi, cpx* Rx, cpx* Ry, T* Ez, T* Bz) {
    Rx[o] = -opb * ik(kx, psi);
    Ry[o] = -opb * ik(ky, psi);
    Ez[o] = narrow<T>(C(0)); Bz[o] = narrow<T>(C(0));
}
// gamma^-2 = 0: k_perp^2 psi = rho
template <class T>
__global__ void k_comoving_c(Geo g, const T* __restrict__ jz, cpx* __restrict__ Rx, cpx* __restrict__ Ry, T* __restrict__ Ez,
                             T* __restrict__ Bz, double beta) {
    const long nk = g.nkh, n = long(g.ns) * nk;
    for (long o = long(blockIdx.x) * blockDim.x + threadIdx.x; o < n; o += long(gridDim.x) * blockDim.x) {
        const long l = o / nk, i = o - l * nk;
        const double kx = g.kxd[int((g.m0 + i) % g.H)], ky = g.kyd[int((g.m0 + i) / g.H)], dg = kx * kx + ky * ky;
        const cpx rhs = (1 / beta) * (g.wlo[g.a + l] * widen(jz[o]) + g.whi[g.a + l] * widen(jz[o + nk]));
        comoving_store(o, kx, ky, 1 + beta, dg == 0 ? C(0) : rhs / dg, Rx, Ry, Ez, Bz);
    }
}
// One CTA per mode; the rows are kept divided by their diagonal: (a, 1, c) and the right-hand side d
constexpr int PCR_NT = 256;
constexpr size_t pcr_smem(int ns) { return size_t(8) * ns * sizeof(double); }        // two buffers of a, c, d
constexpr int PCR_MAX_NS = 3200;
// The modes up to which the reduction is the faster one. Its work per mode grows as ns log ns and, from some 1,000 slices on, its
// shared memory leaves one to three CTAs per SM; the sweep costs its chain whatever the modes are, until they fill the memory
// (the mixed form's sweep also allocates its intermediate and waits). Call of comoving_field, sweep / reduction:
//   FP64   up to 1,024 slices: 12,416 modes 1.23 to 1.52, 18,624 1.01 to 1.23 | 24,768 0.93 to 1.01, 33,024 0.73 to 0.83;
//          beyond: 8,320 modes 1.37 to 1.72, 12,416 0.98 to 1.27 | 18,624 0.71 to 0.95, 33,024 0.43 to 0.61
//   mixed  up to 1,024: 24,768 modes 1.39 to 1.63, 33,024 1.21 to 1.76 | 49,408 0.84 to 1.11, 65,792 0.95 to 1.42;
//          beyond: 12,416 modes 1.22 to 1.78, 18,624 0.87 to 1.30 | 24,768 0.81, 33,024 0.56 to 0.90
// (256 x 256 x 2048: FP64 10.4 -> 4.7 ms, mixed 10.2 -> 6.6 by the sweep.)
template <class T>
constexpr long pcr_modes(int ns) {
    constexpr bool f32 = std::is_same<T, cpxf>::value;
    return ns > PCR_MAX_NS ? 0 : ns <= 1024 ? (f32 ? 40000 : 20000) : (f32 ? 20000 : 13000);
}
template <class T>
__global__ void __launch_bounds__(PCR_NT) k_comoving_pcr(Geo g, const T* __restrict__ jz, cpx* __restrict__ Rx, cpx* __restrict__ Ry,
                                                         T* __restrict__ Ez, T* __restrict__ Bz, double beta, double gm2) {
    extern __shared__ double pcr[];
    const int ns = g.ns, tid = threadIdx.x;
    const long nk = g.nkh, i = blockIdx.x;
    const double kx = g.kxd[int((g.m0 + i) % g.H)], ky = g.kyd[int((g.m0 + i) / g.H)];
    double* A[2] = {pcr, pcr + 4 * ns};                      // a, c, Re d, Im d of ns rows each
    for (int l = tid; l < ns; l += PCR_NT) {
        const long o = long(l) * nk + i;
        const int n = g.a + l;
        const double hm = g.hcg[n + 1], hp = g.hcg[n + 2];
        const double dg = kx * kx + ky * ky + gm2 * 2 / (hm * hp);
        const cpx rhs = (1 / beta) * (g.wlo[n] * widen(jz[o]) + g.whi[n] * widen(jz[o + nk]));
        double* p = A[0];
        p[l] = l > 0 ? -gm2 * 2 / ((hm + hp) * hm) / dg : 0.0;
        p[ns + l] = l + 1 < ns ? -gm2 * 2 / ((hm + hp) * hp) / dg : 0.0;
        p[2 * ns + l] = rhs.x / dg; p[3 * ns + l] = rhs.y / dg;
    }
    __syncthreads();
    int cur = 0;
    for (int s = 1; s < ns; s *= 2, cur ^= 1) {
        const double* p = A[cur];
        double* q = A[cur ^ 1];
        for (int l = tid; l < ns; l += PCR_NT) {
            const double a = p[l], c = p[ns + l];
            double b = 1, dx = p[2 * ns + l], dy = p[3 * ns + l], na = 0, nc = 0;
            if (l >= s) {
                const int m = l - s;
                na = -a * p[m]; b -= a * p[ns + m]; dx -= a * p[2 * ns + m]; dy -= a * p[3 * ns + m];
            }
            if (l + s < ns) {
                const int m = l + s;
                nc = -c * p[ns + m]; b -= c * p[m]; dx -= c * p[2 * ns + m]; dy -= c * p[3 * ns + m];
            }
            const double ib = 1 / b;
            q[l] = na * ib; q[ns + l] = nc * ib; q[2 * ns + l] = dx * ib; q[3 * ns + l] = dy * ib;
        }
        __syncthreads();
    }
    const double* p = A[cur];
    for (int l = tid; l < ns; l += PCR_NT)
        comoving_store(long(l) * nk + i, kx, ky, 1 + beta, C(p[2 * ns + l], p[3 * ns + l]), Rx, Ry, Ez, Bz);
}
// true when one of the two above took the solve; else (gm2 > 0 and too many modes or slices) it is left to the sweep
template <class T>
static bool comoving_parallel(Ctx& c, const Geo& g, const T* jz, cpx* Rx, cpx* Ry, T* Ez, T* Bz, double beta, double gm2) {
    if (g.nkh <= 0) return true;
    if (gm2 != 0 && (!(gm2 > 0) || g.nkh > pcr_modes<T>(g.ns))) return false;
    const int tok = c.prof_begin("comoving");
    if (gm2 == 0) {
        const long b = (long(g.ns) * g.nkh + 255) / 256;
        k_comoving_c<T><<<unsigned(b < 148 * 16 ? b : 148 * 16), 256, 0, c.stream>>>(g, jz, Rx, Ry, Ez, Bz, beta);
        c.check_launch("k_comoving_c");
    } else {
        smem_attr(reinterpret_cast<const void*>(k_comoving_pcr<T>), pcr_smem(PCR_MAX_NS));
        k_comoving_pcr<T><<<unsigned(g.nkh), PCR_NT, pcr_smem(g.ns), c.stream>>>(g, jz, Rx, Ry, Ez, Bz, beta, gm2);
        c.check_launch("k_comoving_pcr");
    }
    c.prof_end(tok);
    return true;
}

}  // namespace g3d
