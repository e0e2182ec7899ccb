// Sponge and real-space fields (Simulation::sponge_and_real_fields, src/sim_fields.cpp:156-307, Fourier y),
// the window shift (src/sim_setup.cpp:249-281), the half <-> full spectrum layouts and small elementwise kernels.
//
// The spectra are kept for k_x = 0 .. nx/2 (H columns): every field is real, so X(-k) = conj X(k).
// A transverse 2-D transform is a pass along y over the H columns (k_*_cols) and a pass along x over the
// rows (k_*_rows), where a row's other half follows from X(nx - k_x) = conj X(k_x) of the y-transformed data.
//
// Sponge: the radiation part R - R_b of the forward field (R_b = (1 + beta) E_perp of the slice charge,
// psi = (rho + gamma^-2 d_zeta^2 rho / k^2) / k^2) is multiplied in real space by maskx(x) masky(y):
//   k_sp_cols_inv  bound field psi -> W3, U = R_x - R_bx and V = R_y - R_by, inverse FFT along y
//   k_sp_rows      per row: u + i v by one inverse FFT along x, 1/(nx ny), the mask, one forward FFT along x,
//                  split back into the half spectra of u and v
//   k_sp_cols_fwd  forward FFT along y, + R_b
// Real fields: k_rf_cols combines R and L into the components' spectra (E_x = (R_x + L_x)/2, ...) and transforms them along
// y (a pair per CTA); k_rf_rows transforms E_x + i E_y, B_x + i B_y, E_z + i B_z along x, row by row, into the six float
// components of F.
#include "g3d_ctx.hpp"
#include "k_fft.cuh"
#include "k_fftr.cuh"
#include "k_dispatch.cuh"
#include "k_tma.cuh"
#include "k_psi.cuh"
#include "k_slice_rows.cuh"

namespace g3d {

namespace {
constexpr int NT = 128;    // threads of the row kernels
constexpr int CW = 8;      // columns per tile of the column kernels
}  // namespace

// ---------------------------------------------------------------- sponge, pass 1: columns (psi, pack, inverse y)
template <int NY>
__global__ void __launch_bounds__(CW * FftShape<NY>::T) k_sp_cols_inv(Geo g, const cpx* __restrict__ Rx, const cpx* __restrict__ Ry,
                                                                      const cpx* __restrict__ jz, const cpx* __restrict__ jg,
                                                                      cpx* __restrict__ U, cpx* __restrict__ V,
                                                                      cpx* __restrict__ PSI, double g2, double opb) {
    using S = FftShape<NY>;
    extern __shared__ cpx sm[];
    cpx* s0 = sm;
    cpx* s1 = sm + ColTile<NY, CW>::size;
    const int l = blockIdx.y, c0 = blockIdx.x * CW, tid = threadIdx.x, nthr = CW * S::T;
    const int H = g.H;
    const long base = long(l) * g.nkh;
    const BoundPsi<cpx> bp(g, jz, jg, l, g2);
    #pragma unroll
    for (int u_ = 0; u_ < (NY * CW + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * CW) break;
        const int p = e / CW, c = e - p * CW, kxi = c0 + c;
        cpx u = C(0), v = C(0);
        if (kxi < H) {
            const long i = long(p) * H + kxi, o = base + i;
            const double kx = g.kxd[kxi], ky = g.kyd[p];
            const cpx psi = bp.at(i, kx * kx + ky * ky);
            PSI[o] = psi;
            u = Rx[o] - (-opb * ik(kx, psi));
            v = Ry[o] - (-opb * ik(ky, psi));
        }
        s0[ColTile<NY, CW>::at(p, c)] = conj(u);
        s1[ColTile<NY, CW>::at(p, c)] = conj(v);
    }
    __syncthreads();
    const int c = tid % CW, t = tid / CW;
    {
        decltype(s0) const ls_[2] = {s0, s1};
        fft_lines<NY, 2>(ls_, RowAddr{c * ColTile<NY, CW>::RS}, t, g.twy);
    }
    #pragma unroll
    for (int u_ = 0; u_ < (NY * CW + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * CW) break;
        const int p = e / CW, cc = e - p * CW, kxi = c0 + cc;
        if (kxi >= H) continue;
        const long o = base + long(p) * H + kxi;
        U[o] = conj(s0[ColTile<NY, CW>::at(p, cc)]);
        V[o] = conj(s1[ColTile<NY, CW>::at(p, cc)]);
    }
}

// The same with the tiles of R_x, R_y (maps 0, 1) loaded by the TMA (k_tma.cuh); psi per element as above.
template <int NY>
__global__ void __launch_bounds__(8 * FftShape<NY>::T) k_sp_cols_inv_tma(Geo g, const __grid_constant__ TileMaps maps,
                                                                        const cpx* __restrict__ jz, const cpx* __restrict__ jg,
                                                                        cpx* __restrict__ U, cpx* __restrict__ V,
                                                                        cpx* __restrict__ PSI, double g2, double opb,
                                                                        TmaWait wt) {
    using S = FftShape<NY>;
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int ok;
    const int l = blockIdx.y, c0 = blockIdx.x * 8, tid = threadIdx.x, nthr = 8 * S::T;
    const int H = g.H;
    const long base = long(l) * g.nkh;
    cpx* s0 = reinterpret_cast<cpx*>(smraw + ((128 - (smem_addr(smraw) & 127)) & 127));
    cpx* s1 = s0 + NY * 8;
    const int idx[2] = {0, 1};
    cpx* const dst[2] = {s0, s1};
    const BoundPsi<cpx> bp(g, jz, jg, l, g2);
    if (!tma_tiles<NY>(maps, idx, 2, dst, c0, l * g.ny, &bar, &ok, wt)) return;
    #pragma unroll
    for (int u_ = 0; u_ < (NY * 8 + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * 8) break;
        const int p = e / 8, c = e - p * 8, kxi = c0 + c;
        cpx u = C(0), v = C(0);
        if (kxi < H) {
            const long i = long(p) * H + kxi, o = base + i;
            const double kx = g.kxd[kxi], ky = g.kyd[p];
            const cpx psi = bp.at(i, kx * kx + ky * ky);
            PSI[o] = psi;
            u = s0[e] - (-opb * ik(kx, psi));
            v = s1[e] - (-opb * ik(ky, psi));
        }
        s0[e] = conj(u);
        s1[e] = conj(v);
    }
    __syncthreads();
    const int c = tid % 8, t = tid / 8;
    {
        decltype(s0) const ls_[2] = {s0, s1};
        fft_lines<NY, 2>(ls_, TileCol{c}, t, g.twy);
    }
    #pragma unroll
    for (int u_ = 0; u_ < (NY * 8 + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * 8) break;
        const int p = e / 8, cc = e - p * 8, kxi = c0 + cc;
        if (kxi >= H) continue;
        const long o = base + long(p) * H + kxi;
        U[o] = conj(s0[e]);
        V[o] = conj(s1[e]);
    }
}

// ---------------------------------------------------------------- sponge, pass 2: rows (inverse x, mask, forward x)
// The line stays in registers from the load through both transforms (k_fftr.cuh).
template <int NX>
__global__ void __launch_bounds__(NT, 3) k_sp_rows(Geo g, cpx* __restrict__ U, cpx* __restrict__ V) {
    using S = FftRegPlan<NX>;
    constexpr int LPC = NT / S::T, H = NX / 2 + 1;
    extern __shared__ cpx sm[];
    const int l = blockIdx.y, r = threadIdx.x / S::T, t = threadIdx.x % S::T, row = blockIdx.x * LPC + r;
    const bool on = row < g.ny;
    const long o = long(l) * g.nkh + long(on ? row : 0) * H;
    cpx* const line = sm + r * row_stride<NX>();
    cpx v[S::E];
#pragma unroll
    for (int j = 0; j < S::E; ++j) {
        const int k = t + S::T * j;
        const bool up = k > NX / 2;
        const long i = o + (up ? NX - k : k);
        v[j] = pair_conj(up, U[i], V[i]);
    }
    fft_reg<NX>(v, line, t, g.twx);
    const double s = g.yf ? 1.0 / double(g.nk) : 1.0 / double(g.nx);   // free-hand y: rows only, 1/nx
    const double mn = s * g.masky_n[on ? row : 0], mh = s * g.masky_h[on ? row : 0];
#pragma unroll
    for (int j = 0; j < S::E; ++j) {                                   // u + i v in real space, masked
        const double mx = g.maskx[t + S::T * j];
        v[j] = C(mx * mn * v[j].x, -(mx * mh * v[j].y));
    }
    fft_reg<NX>(v, line, t, g.twx);
    split_pair<NX>(v, line, t, [&](int k, cpx a, cpx b) {
        if (on) { U[o + k] = a; V[o + k] = b; }
    });
}

// ---------------------------------------------------------------- sponge, pass 3: columns (forward y, + R_b)
template <int NY>
__global__ void __launch_bounds__(CW * FftShape<NY>::T) k_sp_cols_fwd(Geo g, const cpx* __restrict__ U, const cpx* __restrict__ V,
                                                                      const cpx* __restrict__ PSI, cpx* __restrict__ Rx,
                                                                      cpx* __restrict__ Ry, double opb) {
    using S = FftShape<NY>;
    extern __shared__ cpx sm[];
    cpx* s0 = sm;
    cpx* s1 = sm + ColTile<NY, CW>::size;
    const int l = blockIdx.y, c0 = blockIdx.x * CW, tid = threadIdx.x, nthr = CW * S::T;
    const int H = g.H;
    const long base = long(l) * g.nkh;
    #pragma unroll
    for (int u_ = 0; u_ < (NY * CW + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * CW) break;
        const int p = e / CW, c = e - p * CW, kxi = c0 + c;
        cpx u = C(0), v = C(0);
        if (kxi < H) { const long o = base + long(p) * H + kxi; u = U[o]; v = V[o]; }
        s0[ColTile<NY, CW>::at(p, c)] = u; s1[ColTile<NY, CW>::at(p, c)] = v;
    }
    __syncthreads();
    const int c = tid % CW, t = tid / CW;
    {
        decltype(s0) const ls_[2] = {s0, s1};
        fft_lines<NY, 2>(ls_, RowAddr{c * ColTile<NY, CW>::RS}, t, g.twy);
    }
    #pragma unroll
    for (int u_ = 0; u_ < (NY * CW + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * CW) break;
        const int p = e / CW, cc = e - p * CW, kxi = c0 + cc;
        if (kxi >= H) continue;
        const long o = base + long(p) * H + kxi;
        const cpx psi = PSI[o];
        Rx[o] = s0[ColTile<NY, CW>::at(p, cc)] - opb * ik(g.kxd[kxi], psi);
        Ry[o] = s1[ColTile<NY, CW>::at(p, cc)] - opb * ik(g.kyd[p], psi);
    }
}

// The same with the tiles of U, V, PSI (maps 0, 1, 2) loaded by the TMA (k_tma.cuh).
template <int NY>
__global__ void __launch_bounds__(8 * FftShape<NY>::T) k_sp_cols_fwd_tma(Geo g, const __grid_constant__ TileMaps maps,
                                                                        cpx* __restrict__ Rx, cpx* __restrict__ Ry, double opb,
                                                                        TmaWait wt) {
    using S = FftShape<NY>;
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int ok;
    const int l = blockIdx.y, c0 = blockIdx.x * 8, tid = threadIdx.x, nthr = 8 * S::T;
    const int H = g.H;
    const long base = long(l) * g.nkh;
    cpx* s0 = reinterpret_cast<cpx*>(smraw + ((128 - (smem_addr(smraw) & 127)) & 127));
    cpx* s1 = s0 + NY * 8;
    cpx* s2 = s1 + NY * 8;
    const int idx[3] = {0, 1, 2};
    cpx* const dst[3] = {s0, s1, s2};
    if (!tma_tiles<NY>(maps, idx, 3, dst, c0, l * g.ny, &bar, &ok, wt)) return;
    const int c = tid % 8, t = tid / 8;
    {
        decltype(s0) const ls_[2] = {s0, s1};
        fft_lines<NY, 2>(ls_, TileCol{c}, t, g.twy);
    }
    #pragma unroll
    for (int u_ = 0; u_ < (NY * 8 + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * 8) break;
        const int p = e / 8, cc = e - p * 8, kxi = c0 + cc;
        if (kxi >= H) continue;
        const long o = base + long(p) * H + kxi;
        const cpx psi = s2[e];
        Rx[o] = s0[e] - opb * ik(g.kxd[kxi], psi);
        Ry[o] = s1[e] - opb * ik(g.kyd[p], psi);
    }
}

// ---------------------------------------------------------------- real fields: columns (inverse y of the six spectra)
// Two fields per CTA (blockIdx.z) keep the shared memory small enough for several CTAs per SM, so loads of one CTA overlap
// the transforms of another. COMB: the pairs (R_x, L_x), (R_y, L_y), (E_z, B_z) come out as the real fields' own
// spectra, (R + L)/2 and (R - L)/2: W0..W5 = E_x, E_y, B_x, B_y, E_z, B_z, so that each line of the rows kernel is two
// components of F. Else (one slice of the plasma march, whose rows combine) as they are: R_x, R_y, L_x, L_y, E_z, B_z.
template <bool COMB, class T>
__device__ __forceinline__ void rf_combine(int pr, T& a, T& b) {
    typedef typename RealOf<T>::type Re;
    if (!COMB || pr == 2) return;
    const T s = Re(0.5) * (a + b), d = pr == 0 ? Re(0.5) * (a - b) : Re(0.5) * (b - a);   // B_y = (R_x - L_x)/2, B_x = (L_y - R_y)/2
    a = s; b = d;
}
template <int NY, int CWT, bool COMB>
__global__ void __launch_bounds__(CWT * FftShape<NY>::T) k_rf_cols(Geo g, const cpx* __restrict__ Rx, const cpx* __restrict__ Ry,
                                                                  const cpx* __restrict__ Lx, const cpx* __restrict__ Ly,
                                                                  const cpx* __restrict__ Ez, const cpx* __restrict__ Bz,
                                                                  cpx* __restrict__ W0, cpx* __restrict__ W1, cpx* __restrict__ W2,
                                                                  cpx* __restrict__ W3, cpx* __restrict__ W4, cpx* __restrict__ W5,
                                                                  int l0) {
    using S = FftShape<NY>;
    extern __shared__ cpx sm[];
    const int l = l0 + blockIdx.y, c0 = blockIdx.x * CWT, tid = threadIdx.x, nthr = CWT * S::T, pr = blockIdx.z;
    const int H = g.H;
    const long base = long(l) * g.nkh;
    const cpx* in0 = pr == 2 ? Ez : COMB ? (pr == 0 ? Rx : Ry) : (pr == 0 ? Rx : Lx);
    const cpx* in1 = pr == 2 ? Bz : COMB ? (pr == 0 ? Lx : Ly) : (pr == 0 ? Ry : Ly);
    cpx* out0 = pr == 2 ? W4 : COMB ? (pr == 0 ? W0 : W1) : (pr == 0 ? W0 : W2);
    cpx* out1 = pr == 2 ? W5 : COMB ? (pr == 0 ? W3 : W2) : (pr == 0 ? W1 : W3);
    cpx* s0 = sm;
    cpx* s1 = sm + ColTile<NY, CWT>::size;
    #pragma unroll
    for (int u_ = 0; u_ < (NY * CWT + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * CWT) break;
        const int p = e / CWT, c = e - p * CWT, kxi = c0 + c;
        const long o = base + long(p) * H + kxi;
        cpx a = C(0), b = C(0);
        if (kxi < H) { a = in0[o]; b = in1[o]; }
        rf_combine<COMB>(pr, a, b);
        s0[ColTile<NY, CWT>::at(p, c)] = conj(a);
        s1[ColTile<NY, CWT>::at(p, c)] = conj(b);
    }
    __syncthreads();
    const int c = tid % CWT, t = tid / CWT;
    {
        decltype(s0) const ls_[2] = {s0, s1};
        fft_lines<NY, 2>(ls_, RowAddr{c * ColTile<NY, CWT>::RS}, t, g.twy);
    }
    #pragma unroll
    for (int u_ = 0; u_ < (NY * CWT + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * CWT) break;
        const int p = e / CWT, cc = e - p * CWT, kxi = c0 + cc;
        if (kxi >= H) continue;
        const long o = base + long(p) * H + kxi;
        out0[o] = conj(s0[ColTile<NY, CWT>::at(p, cc)]);
        out1[o] = conj(s1[ColTile<NY, CWT>::at(p, cc)]);
    }
}

// The same transforms of the whole window with the tiles loaded by the TMA (k_tma.cuh): the 8-column tiles of the
// pair land row-major in shared memory, are combined (COMB above) and conjugated in place, transformed along their columns (stride 8) and
// written back conjugated; maps 0..5 are R_x, R_y, L_x, L_y, E_z, B_z.
template <int NY>
__global__ void __launch_bounds__(8 * FftShape<NY>::T) k_rf_cols_tma(Geo g, const __grid_constant__ TileMaps maps,
                                                                    cpx* __restrict__ W0, cpx* __restrict__ W1,
                                                                    cpx* __restrict__ W2, cpx* __restrict__ W3,
                                                                    cpx* __restrict__ W4, cpx* __restrict__ W5, int l0,
                                                                    TmaWait wt) {
    using S = FftShape<NY>;
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int ok;
    const int l = l0 + blockIdx.y, c0 = blockIdx.x * 8, tid = threadIdx.x, nthr = 8 * S::T, pr = blockIdx.z;
    const int H = g.H;
    const long base = long(l) * g.nkh;
    cpx* s0 = reinterpret_cast<cpx*>(smraw + ((128 - (smem_addr(smraw) & 127)) & 127));
    cpx* s1 = s0 + NY * 8;
    cpx* out0 = pr == 0 ? W0 : pr == 1 ? W1 : W4;
    cpx* out1 = pr == 0 ? W3 : pr == 1 ? W2 : W5;
    const int idx[2] = {pr == 2 ? 4 : pr, pr == 2 ? 5 : pr + 2};
    cpx* const dst[2] = {s0, s1};
    if (!tma_tiles<NY>(maps, idx, 2, dst, c0, l * g.ny, &bar, &ok, wt)) return;
    for (int e = tid; e < NY * 8; e += nthr) {
        cpx a = s0[e], b = s1[e];
        rf_combine<true>(pr, a, b);
        s0[e] = conj(a); s1[e] = conj(b);
    }
    __syncthreads();
    const int c = tid % 8, t = tid / 8;
    {
        decltype(s0) const ls_[2] = {s0, s1};
        fft_lines<NY, 2>(ls_, TileCol{c}, t, g.twy);
    }
    #pragma unroll
    for (int u_ = 0; u_ < (NY * 8 + nthr - 1) / nthr; ++u_) {
        const int e = tid + u_ * nthr;
        if (e >= NY * 8) break;
        const int p = e / 8, cc = e - p * 8, kxi = c0 + cc;
        if (kxi >= H) continue;
        const long o = base + long(p) * H + kxi;
        out0[o] = conj(s0[e]);
        out1[o] = conj(s1[e]);
    }
}

// ---------------------------------------------------------------- real fields: rows (inverse x, F)
// One line per group of threads (blockIdx.z): E_x + i E_y, B_x + i B_y or E_z + i B_z of a row, from global memory through
// registers to F (k_fftr.cuh). COMB: the input are the rows of R_x, R_y, L_x, L_y, E_z, B_z (free-hand y, no columns pass)
// and are combined here. (One slice of the plasma march: k_rf_row_slice, k_slice_rows.cuh.)
template <int NX, class T, bool COMB>
__global__ void __launch_bounds__(NT, 3) k_rf_rows(Geo g, const T* __restrict__ tw, const T* __restrict__ W0, const T* __restrict__ W1,
                                                  const T* __restrict__ W2, const T* __restrict__ W3, const T* __restrict__ W4,
                                                  const T* __restrict__ W5, float* __restrict__ F, double* __restrict__ Fd) {
    typedef typename RealOf<T>::type Re;
    using S = FftRegPlan<NX>;
    constexpr int LPC = NT / S::T, H = NX / 2 + 1;
    extern __shared__ __align__(16) unsigned char smr[];
    const int l = blockIdx.y, pr = blockIdx.z, r = threadIdx.x / S::T, t = threadIdx.x % S::T, row = blockIdx.x * LPC + r;
    const bool on = row < g.ny;
    const long o = long(l) * g.nkh + long(on ? row : 0) * H;
    const T* a0 = pr == 0 ? W0 : pr == 1 ? (COMB ? W1 : W2) : W4;       // COMB: line 0 R_x, R_y and L_x, L_y; line 1 R_y, R_x
    const T* b0 = pr == 0 ? W1 : pr == 1 ? (COMB ? W0 : W3) : W5;
    const T* a1 = pr == 0 ? W2 : W3;                                   // and L_y, L_x
    const T* b1 = pr == 0 ? W3 : W2;
    T v[S::E];
#pragma unroll
    for (int j = 0; j < S::E; ++j) {
        const int k = t + S::T * j;
        const bool up = k > NX / 2;
        const long i = o + (up ? NX - k : k);
        T a = __ldg(a0 + i), b = __ldg(b0 + i);
        if (COMB && pr < 2) {
            const T c = __ldg(a1 + i), d = __ldg(b1 + i);
            if (pr == 0) { a = Re(0.5) * (a + c); b = Re(0.5) * (b + d); }      // E_x, E_y
            else { a = Re(0.5) * (c - a); b = Re(0.5) * (b - d); }              // B_x = (L_y - R_y)/2, B_y = (R_x - L_x)/2
        }
        v[j] = pair_conj(up, a, b);
    }
    fft_reg<NX>(v, reinterpret_cast<T*>(smr) + r * row_stride<NX>(), t, tw);
    if (!on) return;
    const Re s = g.yf ? Re(1) / Re(g.nk) : Re(1) / Re(g.nx);            // free-hand y: rows only, 1/nx
    const long fpl = long(g.ns + 2) * g.nk, idx = long(l) * g.nk + long(row) * NX;
    const int ca = pr == 0 ? 0 : pr == 1 ? 3 : 2, cb = pr == 0 ? 1 : pr == 1 ? 4 : 5;
#pragma unroll
    for (int j = 0; j < S::E; ++j) {
        const long i = idx + t + S::T * j;
        const Re x = s * v[j].x, y = -(s * v[j].y);
        F[ca * fpl + i] = float(x); F[cb * fpl + i] = float(y);
        if (Fd) { Fd[ca * fpl + i] = double(x); Fd[cb * fpl + i] = double(y); }    // exact fields: before the rounding
    }
}
template <int NX, class T, bool COMB>
static void rf_rows(Ctx& c, const T* tw, const T* W0, const T* W1, const T* W2, const T* W3, const T* W4, const T* W5, double* Fd) {
    constexpr int LPC = NT / FftRegPlan<NX>::T;
    const size_t smem = size_t(LPC) * row_stride<NX>() * sizeof(T);
    auto kern = k_rf_rows<NX, T, COMB>;
    smem_attr(reinterpret_cast<const void*>(kern), smem);
    const int tok = c.prof_begin("real_rows");
    kern<<<dim3(unsigned((c.ny + LPC - 1) / LPC), unsigned(c.ns), 3), NT, smem, c.stream>>>(c.geo(), tw, W0, W1, W2, W3, W4, W5, c.F.p, Fd);
    c.check_launch("k_rf_rows");
    c.prof_end(tok);
}
void launch_rf_rows_f(Ctx& c) {                       // the mixed form's (k_mixed.cu)
    auto& m = c.mx;
    G3D_DISPATCH_N(c.nx, NX, (rf_rows<NX, cpxf, false>(c, m.twx.p, m.W[0].p, m.W[1].p, m.W[2].p, m.W[3].p, m.W[4].p, m.W[5].p, nullptr)));
}

// ---------------------------------------------------------------- launchers
template <class K>
static void allow_smem(K kern, size_t smem) {
    smem_attr(reinterpret_cast<const void*>(kern), smem);
}
static unsigned col_tiles(const Ctx& c) { return unsigned((c.H + CW - 1) / CW); }

template <int NY>
static void sp_cols_inv(Ctx& c) {
    if constexpr (NY <= 256 && (NY & (NY - 1)) == 0) {
        const cpx* p[2] = {c.Rx.p, c.Ry.p};
        if (c.use_tma && c.tma_spi.get(p, 2, c.H, long(c.ns) * c.ny, c.ny)) {
            const size_t smem = size_t(2) * NY * 8 * sizeof(cpx) + 128;
            allow_smem(k_sp_cols_inv_tma<NY>, smem);
            const int tok = c.prof_begin("sponge_cols_inv");
            k_sp_cols_inv_tma<NY><<<dim3(col_tiles(c), unsigned(c.ns)), 8 * FftShape<NY>::T, smem, c.stream>>>(
                c.geo(), c.tma_spi.maps, c.jkz.p, c.jzg.p, c.W[0].p, c.W[1].p, c.W[3].p, c.gm2_b, 1 + c.beta_b, c.tma_wait());
            c.check_launch("k_sp_cols_inv_tma");
            c.prof_end(tok);
            return;
        }
    }
    const size_t smem = size_t(2) * ColTile<NY, CW>::size * sizeof(cpx);
    allow_smem(k_sp_cols_inv<NY>, smem);
    const int tok = c.prof_begin("sponge_cols_inv");
    k_sp_cols_inv<NY><<<dim3(col_tiles(c), unsigned(c.ns)), CW * FftShape<NY>::T, smem, c.stream>>>(
        c.geo(), c.Rx.p, c.Ry.p, c.jkz.p, c.jzg.p, c.W[0].p, c.W[1].p, c.W[3].p, c.gm2_b, 1 + c.beta_b);
    c.check_launch("k_sp_cols_inv");
    c.prof_end(tok);
}
template <int NX>
static void sp_rows(Ctx& c) {
    constexpr int LPC = NT / FftRegPlan<NX>::T;
    const size_t smem = size_t(LPC) * row_stride<NX>() * sizeof(cpx);
    allow_smem(k_sp_rows<NX>, smem);
    const int tok = c.prof_begin("sponge_rows");
    k_sp_rows<NX><<<dim3(unsigned((c.ny + LPC - 1) / LPC), unsigned(c.ns)), NT, smem, c.stream>>>(c.geo(), c.W[0].p, c.W[1].p);
    c.check_launch("k_sp_rows");
    c.prof_end(tok);
}
template <int NY>
static void sp_cols_fwd(Ctx& c) {
    if constexpr (NY <= 256 && (NY & (NY - 1)) == 0) {
        const cpx* p[3] = {c.W[0].p, c.W[1].p, c.W[3].p};
        if (c.use_tma && c.tma_spf.get(p, 3, c.H, long(c.ns) * c.ny, c.ny)) {
            const size_t smem = size_t(3) * NY * 8 * sizeof(cpx) + 128;
            allow_smem(k_sp_cols_fwd_tma<NY>, smem);
            const int tok = c.prof_begin("sponge_cols_fwd");
            k_sp_cols_fwd_tma<NY><<<dim3(col_tiles(c), unsigned(c.ns)), 8 * FftShape<NY>::T, smem, c.stream>>>(
                c.geo(), c.tma_spf.maps, c.Rx.p, c.Ry.p, 1 + c.beta_b, c.tma_wait());
            c.check_launch("k_sp_cols_fwd_tma");
            c.prof_end(tok);
            return;
        }
    }
    const size_t smem = size_t(2) * ColTile<NY, CW>::size * sizeof(cpx);
    allow_smem(k_sp_cols_fwd<NY>, smem);
    const int tok = c.prof_begin("sponge_cols_fwd");
    k_sp_cols_fwd<NY><<<dim3(col_tiles(c), unsigned(c.ns)), CW * FftShape<NY>::T, smem, c.stream>>>(
        c.geo(), c.W[0].p, c.W[1].p, c.W[3].p, c.Rx.p, c.Ry.p, 1 + c.beta_b);
    c.check_launch("k_sp_cols_fwd");
    c.prof_end(tok);
}
void launch_sponge(Ctx& c) {
    G3D_DISPATCH_N(c.ny, NY, sp_cols_inv<NY>(c));
    G3D_DISPATCH_N(c.nx, NX, sp_rows<NX>(c));
    G3D_DISPATCH_N(c.ny, NY, sp_cols_fwd<NY>(c));
}

// What W holds is asked for by the caller: COMB, the whole window, whose rows kernel takes the components; else one slice (of the
// plasma march, whose rows combine), in tiles of 2 columns, so that 3 x 65 CTAs spread the slice's latency over the SMs.
template <int NY, bool COMB>
static void rf_cols_w(Ctx& c, int l0, int nl) {
    constexpr int CWT = COMB ? CW : 2;
    const size_t smem = size_t(2) * ColTile<NY, CWT>::size * sizeof(cpx);
    allow_smem(k_rf_cols<NY, CWT, COMB>, smem);
    const int tok = c.prof_begin(COMB ? "real_cols" : "real_cols_slice");
    k_rf_cols<NY, CWT, COMB><<<dim3(unsigned((c.H + CWT - 1) / CWT), unsigned(nl), 3), CWT * FftShape<NY>::T, smem, c.stream>>>(
        c.geo(), c.Rx.p, c.Ry.p, c.Lx.p, c.Ly.p, c.Ez.p, c.Bz.p, c.W[0].p, c.W[1].p, c.W[2].p, c.W[3].p, c.W[4].p, c.W[5].p, l0);
    c.check_launch("k_rf_cols");
    c.prof_end(tok);
}
// the tensor maps of R_x, R_y, L_x, L_y, E_z, B_z for tiles of 8 columns x ny rows, made once per set of buffers;
// false where the TMA path does not apply (ny > 256, or the encoder is unavailable)
static bool rf_maps(Ctx& c) {
    const cpx* p[6] = {c.Rx.p, c.Ry.p, c.Lx.p, c.Ly.p, c.Ez.p, c.Bz.p};
    return c.tma_rf.get(p, 6, c.H, long(c.ns) * c.ny, c.ny);
}
template <int NY>
static void rf_cols_tma(Ctx& c) {
    const size_t smem = size_t(2) * NY * 8 * sizeof(cpx) + 128;
    allow_smem(k_rf_cols_tma<NY>, smem);
    const int tok = c.prof_begin("real_cols");
    k_rf_cols_tma<NY><<<dim3(unsigned((c.H + 7) / 8), unsigned(c.ns), 3), 8 * FftShape<NY>::T, smem, c.stream>>>(
        c.geo(), c.tma_rf.maps, c.W[0].p, c.W[1].p, c.W[2].p, c.W[3].p, c.W[4].p, c.W[5].p, 0, c.tma_wait());
    c.check_launch("k_rf_cols_tma");
    c.prof_end(tok);
}
template <int NY>
static void rf_cols(Ctx& c) {
    if constexpr (NY <= 256 && (NY & (NY - 1)) == 0) {
        if (c.use_tma && rf_maps(c)) { rf_cols_tma<NY>(c); return; }
    }
    rf_cols_w<NY, true>(c, 0, c.ns);
}
void launch_real_fields(Ctx& c) {
    G3D_DISPATCH_N(c.ny, NY, rf_cols<NY>(c));
    G3D_DISPATCH_N(c.nx, NX, (rf_rows<NX, cpx, false>(c, c.twx.p, c.W[0].p, c.W[1].p, c.W[2].p, c.W[3].p, c.W[4].p, c.W[5].p, c.Fd.p)));
}
// free-hand y: the spectra are already real in y; one inverse transform along x per row of R, L and E_z + i B_z
void launch_real_fields_fh(Ctx& c) {
    G3D_DISPATCH_N(c.nx, NX, (rf_rows<NX, cpx, true>(c, c.twx.p, c.Rx.p, c.Ry.p, c.Lx.p, c.Ly.p, c.Ez.p, c.Bz.p, c.Fd.p)));
}
void launch_real_fields_slice_fh(Ctx& c, int l, FmidOut fm) {
    G3D_DISPATCH_N(c.nx, NX, (rf_row_slice<NX, cpx, false>(c, c.twx.p, c.Rx.p, c.Ry.p, c.Lx.p, c.Ly.p, c.Ez.p, c.Bz.p, l, l, c.Fd.p, fm)));
}
// the sponge's row pass alone (inverse x, mask, forward x) on W0, W1: the free-hand y sponge
void launch_sp_rows(Ctx& c) { G3D_DISPATCH_N(c.nx, NX, sp_rows<NX>(c)); }
// E and B of one slice (plane l) in real space (Simulation::real_fields_slice, src/sim_plasma.cpp:200-220). cols: the
// columns too (into plane l of W); else they are in plane 0 of W, where k_pass_cols left them
void launch_real_fields_slice(Ctx& c, int l, FmidOut fm, bool cols) {
    if (cols) G3D_DISPATCH_N(c.ny, NY, (rf_cols_w<NY, false>(c, l, 1)));
    const cpx* W[6] = {c.W[0].p, c.W[1].p, c.W[2].p, c.W[3].p, c.W[4].p, c.W[5].p};
    const int lw = cols ? l : 0;
    if (c.Fd.p && fm.out && !fm.f32 && !fm.fh)         // exact fields: unrounded midpoint fields
        G3D_DISPATCH_N(c.nx, NX, (rf_row_slice<NX, cpx, true>(c, c.twx.p, W[0], W[1], W[2], W[3], W[4], W[5], l, lw, c.Fd.p, fm)))
    else
        G3D_DISPATCH_N(c.nx, NX, (rf_row_slice<NX, cpx, false>(c, c.twx.p, W[0], W[1], W[2], W[3], W[4], W[5], l, lw, c.Fd.p, fm)))
}

// ---------------------------------------------------------------- half <-> full spectrum layouts
// full[p][j][ix] = half[p][j][ix] (ix <= nx/2), conj(half[p][(ny - j) % ny][nx - ix]) (ix > nx/2; free-hand y:
// conj(half[p][j][nx - ix]))
__global__ void k_half_to_full(Geo g, const cpx* __restrict__ half, cpx* __restrict__ full, long planes) {
    const long n = planes * g.nk;
    for (long idx = long(blockIdx.x) * blockDim.x + threadIdx.x; idx < n; idx += long(gridDim.x) * blockDim.x) {
        const long pl = idx / g.nk, i = idx - pl * g.nk;
        const int ixx = int(i % g.nx), j = int(i / g.nx);
        const long hb = pl * g.nkh;
        const int jm = g.yf ? (g.ny - j) % g.ny : j;      // free-hand y: y is real space, only k_x mirrors
        full[idx] = ixx <= g.nx / 2 ? half[hb + long(j) * g.H + ixx]
                                    : conj(half[hb + long(jm) * g.H + (g.nx - ixx)]);
    }
}
__global__ void k_full_to_half(Geo g, const cpx* __restrict__ full, cpx* __restrict__ half, long planes) {
    const long n = planes * g.nkh;
    for (long idx = long(blockIdx.x) * blockDim.x + threadIdx.x; idx < n; idx += long(gridDim.x) * blockDim.x) {
        const long pl = idx / g.nkh, i = idx - pl * g.nkh;
        const int kx = int(i % g.H), j = int(i / g.H);
        half[idx] = full[pl * g.nk + long(j) * g.nx + kx];
    }
}

// ---------------------------------------------------------------- elementwise
__global__ void k_axpy_c(cpx* __restrict__ y, const cpx* __restrict__ x, double a, long n) {
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x) y[i] = y[i] + a * x[i];
}
__global__ void k_copy_c(cpx* __restrict__ y, const cpx* __restrict__ x, long n) {
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += long(gridDim.x) * blockDim.x) y[i] = x[i];
}
static unsigned ew_blocks(long n) {
    long b = (n + 255) / 256;
    return unsigned(b < 148 * 16 ? (b < 1 ? 1 : b) : 148 * 16);
}
void launch_half_to_full(Ctx& c, const cpx* half, cpx* full, long planes) {
    k_half_to_full<<<ew_blocks(planes * c.nk), 256, 0, c.stream>>>(c.geo(), half, full, planes);
    c.check_launch("k_half_to_full");
}
void launch_full_to_half(Ctx& c, const cpx* full, cpx* half, long planes) {
    k_full_to_half<<<ew_blocks(planes * c.nkh), 256, 0, c.stream>>>(c.geo(), full, half, planes);
    c.check_launch("k_full_to_half");
}
void launch_zero_c(Ctx& c, cpx* p, size_t n) { if (n) G3D_CUDA(cudaMemsetAsync(p, 0, n * sizeof(cpx), c.stream)); }
void launch_axpy_c(Ctx& c, cpx* y, const cpx* x, double a, size_t n) {
    if (!n) return;
    const int tok = c.prof_begin("axpy");
    k_axpy_c<<<ew_blocks(long(n)), 256, 0, c.stream>>>(y, x, a, long(n));
    c.check_launch("k_axpy_c");
    c.prof_end(tok);
}
void launch_copy_c(Ctx& c, cpx* y, const cpx* x, size_t n) {
    if (!n) return;
    const int tok = c.prof_begin("copy");
    k_copy_c<<<ew_blocks(long(n)), 256, 0, c.stream>>>(y, x, long(n));
    c.check_launch("k_copy_c");
    c.prof_end(tok);
}

// ---------------------------------------------------------------- window shift
// Spectra: exact phase factor exp(i (k_x s_x + k_y s_y)) with the shift tables kxs, kys (Nyquist kept).
__global__ void k_rotate(Geo g, cpx* __restrict__ p, long n, double sx, double sy, int nys) {
    const long nk = g.nkh;
    for (long idx = long(blockIdx.x) * blockDim.x + threadIdx.x; idx < n; idx += long(gridDim.x) * blockDim.x) {
        const long i = idx % nk;
        const double ph = g.kxs[i % g.H] * sx + (nys ? g.kys[i / g.H] * sy : 0.0);
        p[idx] = p[idx] * C(cos(ph), sin(ph));
    }
}
// Real fields: index roll of every plane.
__global__ void k_roll(Geo g, const float* __restrict__ f, float* __restrict__ t, long n, int nxs, int nys) {
    const long nk = g.nk;
    for (long idx = long(blockIdx.x) * blockDim.x + threadIdx.x; idx < n; idx += long(gridDim.x) * blockDim.x) {
        const long i = idx % nk, base = idx - i;
        const int ixx = int(i % g.nx), j = int(i / g.nx);
        const int sxx = ((ixx + nxs) % g.nx + g.nx) % g.nx, syy = ((j + nys) % g.ny + g.ny) % g.ny;
        t[idx] = f[base + long(syy) * g.nx + sxx];
    }
}
__global__ void k_shift_parts(PartsDev P, long np, double sx, double sy) {
    for (long i = long(blockIdx.x) * blockDim.x + threadIdx.x; i < np; i += long(gridDim.x) * blockDim.x) {
        P.x[i] -= sx; P.y[i] -= sy;
    }
}
void launch_rotate(Ctx& c, cpx* p, size_t n, double sx, double sy, int nys) {
    if (!n) return;
    k_rotate<<<ew_blocks(long(n)), 256, 0, c.stream>>>(c.geo(), p, long(n), sx, sy, nys);
    c.check_launch("k_rotate");
}
void launch_shift(Ctx& c, int nxs, int nys, double sx, double sy) {
    const Geo g = c.geo();
    if (c.np) {
        k_shift_parts<<<ew_blocks(c.np), 256, 0, c.stream>>>(c.parts, c.np, sx, sy);
        c.check_launch("k_shift_parts");
    }
    if (!c.P.self_fields) return;
    for (DevBuf<cpx>* a : {&c.Rx, &c.Ry, &c.Ez, &c.Bz, &c.j0x, &c.j0y}) {
        if (!a->n) continue;                     // the mixed form keeps E_z, B_z, j0 in complex64 (k_mixed.cu)
        k_rotate<<<ew_blocks(long(a->n)), 256, 0, c.stream>>>(g, a->p, long(a->n), sx, sy, nys);
        c.check_launch("k_rotate");
    }
    DevBuf<float> tmp;
    tmp.alloc(c.F.n, c.stream);
    k_roll<<<ew_blocks(long(c.F.n)), 256, 0, c.stream>>>(g, c.F.p, tmp.p, long(c.F.n), nxs, nys);
    c.check_launch("k_roll");
    std::swap(c.F.p, tmp.p);
    G3D_CUDA(cudaStreamSynchronize(c.stream));
}

}  // namespace g3d
