// The rows of the real fields of one slice of the plasma march, in both forms (T: complex128 or complex64): what
// k_rf_rows and k_rf_rows_f do for the whole window, laid out for a launch that has one plane to work on.
//
// One CTA per row, a thread per point, the three line transforms (R_x + i R_y, L_x + i L_y, E_z + i B_z) side by side on
// threads of their own. A plane of 256 x 256 is 256 CTAs of 8 warps here against 64 CTAs of 4 in the whole-window
// layout (64 x 64: 64 against 4), where each thread moved 8 points of three lines one after the other; the launch is a
// short chain of latencies (loads, transform, stores) and no byte count, so what shortens it is less work per thread.
// Per launch with the events' own ~5 us: 256 x 256 mixed 12.2 -> 9.2 us,
// FP64 13.6 -> 10.5 us, 64 x 64 FP64 14.0 -> 8.0 us.
#pragma once
#include "g3d_ctx.hpp"
#include "k_fft.cuh"
#include "k_pdl.cuh"

namespace g3d {

// W0..W5: the half rows (k_x = 0 .. NX/2) of plane lw; F (and Fd, when kept): plane l of every component.
// XM (exact fields with midpoint fields, FP64 Fourier y): the midpoint fields from the FP64 values of both slices (Fd).
template <int NX, class T, bool XM>
__global__ void __launch_bounds__(slice_row_threads<NX>()) k_rf_row_slice(Geo g, const T* __restrict__ tw, Handed<T> W0, Handed<T> W1,
                                                                         Handed<T> W2, Handed<T> W3, Handed<T> W4, Handed<T> W5,
                                                                         float* __restrict__ F, int l, int lw,
                                                                         double* __restrict__ Fd, FmidOut fm) {
    typedef typename RealOf<T>::type Re;
    using S = FftShape<NX>;
    constexpr int NTH = slice_row_threads<NX>(), RS = row_stride<NX>(), H = NX / 2 + 1;
    constexpr int EI = (H + NTH - 1) / NTH, EO = (NX + NTH - 1) / NTH;
    extern __shared__ __align__(16) unsigned char smr[];
    T* a[3] = {reinterpret_cast<T*>(smr), reinterpret_cast<T*>(smr) + RS, reinterpret_cast<T*>(smr) + 2 * RS};
    T* stw = reinterpret_cast<T*>(smr) + 3 * RS;
    const int row = blockIdx.x, tid = threadIdx.x;
    const long fpl = long(g.ns + 2) * g.nk, k0 = long(row) * NX, base = long(lw) * g.nkh + long(row) * H;
    // the other slice was written long before the columns kernel this one follows: loaded while that still runs
    float oth[XM ? 1 : EO][6];                                      // the midpoint fields' other slice
    double othd[XM ? EO : 1][6];
    if (fm.out) {
#pragma unroll
        for (int u = 0; u < EO; ++u) {
            const int p = tid + u * NTH;
            if (p >= NX) continue;
            if constexpr (XM) {
#pragma unroll
                for (int comp = 0; comp < 6; ++comp) othd[u][comp] = Fd[comp * fpl + long(fm.other) * g.nk + k0 + p];
            } else {
                fmid_load(fm, F, fpl, g.nk, k0 + p, oth[u]);
            }
        }
    }
    stage_twiddles<NX>(stw, tw, tid, NTH);
    pdl_wait();
    pdl_next();
    const Handed<T> in[6] = {W0, W1, W2, W3, W4, W5};
    T v[EI][6];
#pragma unroll
    for (int u = 0; u < EI; ++u) {
        const int p = tid + u * NTH;
#pragma unroll
        for (int f = 0; f < 6; ++f) v[u][f] = p < H ? in[f][base + p] : mk<T>(0, 0);
    }
#pragma unroll
    for (int u = 0; u < EI; ++u) {
        const int p = tid + u * NTH;
        if (p >= H) continue;
        // the full row of x + i y from its half: position p, and its mirror from the conjugates; conjugated (inverse)
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            const T x = v[u][2 * f], y = v[u][2 * f + 1];
            a[f][p + (p >> 3)] = mk<T>(x.x - y.y, -(x.y + y.x));
            if (p > 0 && p < NX / 2) { const int q = NX - p; a[f][q + (q >> 3)] = mk<T>(x.x + y.y, x.y - y.x); }
        }
    }
    __syncthreads();
    {
        static_assert(3 * S::T <= NTH, "a line of each pair per thread group");
        const int grp = tid / S::T;
        T* const ls_[1] = {a[grp < 3 ? grp : 0]};
        fft_lines_slice<NX, 1>(ls_, RowAddr{0}, tid % S::T, stw, grp < 3);
    }
    __syncthreads();
    const Re s = g.yf ? Re(1) / Re(g.nk) : Re(1) / Re(g.nx);        // free-hand y: rows only, 1/nx
#pragma unroll
    for (int u = 0; u < EO; ++u) {
        const int p = tid + u * NTH;
        if (p >= NX) continue;
        const int q = p + (p >> 3);
        const T z1 = s * conj(a[0][q]), z2 = s * conj(a[1][q]), z3 = s * conj(a[2][q]);
        const long idx = long(l) * g.nk + k0 + p;
        const Re dv[6] = {Re(0.5) * (z1.x + z2.x), Re(0.5) * (z1.y + z2.y), z3.x,      // E_x, E_y, E_z
                          Re(0.5) * (z2.y - z1.y), Re(0.5) * (z1.x - z2.x), z3.y};     // B_x, B_y, B_z
        float fv[6];
#pragma unroll
        for (int comp = 0; comp < 6; ++comp) { fv[comp] = float(dv[comp]); F[comp * fpl + idx] = fv[comp]; }
        if constexpr (XM) {
            double2* o = reinterpret_cast<double2*>(fm.out) + 3 * (k0 + p);
            o[0] = make_double2(0.5 * (dv[0] + othd[u][0]), 0.5 * (dv[1] + othd[u][1]));
            o[1] = make_double2(0.5 * (dv[2] + othd[u][2]), 0.5 * (dv[3] + othd[u][3]));
            o[2] = make_double2(0.5 * (dv[4] + othd[u][4]), 0.5 * (dv[5] + othd[u][5]));
        } else if (fm.out) {
            fmid_store(fm, k0 + p, fv, oth[u]);
        }
        if (fm.rec_f && (XM || std::is_same<T, cpxf>::value)) {      // the adjoint's record of the slice
            double* R = *fm.rec_f + fm.rec_off + k0 + p;
#pragma unroll
            for (int comp = 0; comp < 6; ++comp) R[comp * g.nk] = XM ? double(dv[comp]) : double(fv[comp]);
        }
        if (Fd) {                                      // exact fields: the same values before the rounding
#pragma unroll
            for (int comp = 0; comp < 6; ++comp) Fd[comp * fpl + idx] = double(dv[comp]);
        }
    }
}

template <int NX, class T, bool XM>
static void rf_row_slice(Ctx& c, const T* tw, const T* W0, const T* W1, const T* W2, const T* W3, const T* W4, const T* W5, int l, int lw,
                         double* Fd, const FmidOut& fm) {
    const size_t smem = (size_t(3) * row_stride<NX>() + NX) * sizeof(T);
    auto kern = k_rf_row_slice<NX, T, XM>;
    smem_attr(reinterpret_cast<const void*>(kern), smem);
    const int tok = c.prof_begin("real_rows_slice");
    launch_pdl(c.stream, kern, unsigned(c.ny), slice_row_threads<NX>(), smem, c.geo(), tw, Handed<T>{W0}, Handed<T>{W1},
               Handed<T>{W2}, Handed<T>{W3}, Handed<T>{W4}, Handed<T>{W5}, c.F.p, l, lw, Fd, fm);
    c.check_launch("k_rf_row_slice");
    c.prof_end(tok);
}

}  // namespace g3d
