// Batched FFT of the library's lengths with a line's values in registers at both ends, for the whole-window row kernels.
//
// The Stockham passes of k_fft.cuh with larger radices: a line is worked by T = N / E threads and thread t holds the values
// x[t + T j], j < E, before and after the transform (the first pass of radix R reads x[q N/R + t + T u], the last one writes
// y[r N/R + t + T u], and N/R is a multiple of T in both, so each is that set). Between passes the values cross shared
// memory once: 64, 128 and 256 points take two passes (8 x 8, 16 x 8, 16 x 16) and one crossing, where the in-place
// transform of k_fft.cuh takes two or three crossings and its callers two more, to bring a line in and out. The callers
// here load and store global memory straight from these registers (T consecutive lanes hold T consecutive points). The
// row kernels were bound by shared-memory traffic, not by DRAM.
#pragma once
#include "k_fft.cuh"

namespace g3d {

template <int N> struct FftRegPlan;            // E values per thread, the radices of the passes
#define G3D_FFTR_PLAN(N_, E_, ...)                                     \
    template <> struct FftRegPlan<N_> {                                \
        static constexpr int E = E_, T = N_ / E_;                      \
        static constexpr int R[4] = {__VA_ARGS__};                     \
    };
G3D_FFTR_PLAN(4, 4, 4, 1, 1, 1)
G3D_FFTR_PLAN(8, 8, 8, 1, 1, 1)
G3D_FFTR_PLAN(16, 8, 8, 2, 1, 1)
G3D_FFTR_PLAN(32, 8, 8, 4, 1, 1)
G3D_FFTR_PLAN(64, 8, 8, 8, 1, 1)
G3D_FFTR_PLAN(128, 16, 16, 8, 1, 1)
G3D_FFTR_PLAN(256, 16, 16, 16, 1, 1)
G3D_FFTR_PLAN(512, 8, 8, 8, 8, 1)
G3D_FFTR_PLAN(24, 12, 12, 2, 1, 1)
G3D_FFTR_PLAN(48, 12, 12, 4, 1, 1)
G3D_FFTR_PLAN(96, 12, 12, 4, 2, 1)
G3D_FFTR_PLAN(192, 12, 12, 4, 4, 1)
G3D_FFTR_PLAN(384, 12, 12, 4, 4, 2)
#undef G3D_FFTR_PLAN

// exp(-2 pi i m / R) for the inner twiddles of the composite radices (R = 12: m <= 6; R = 16: m <= 9)
template <int R, int M, class T>
__device__ __forceinline__ T root_of_unity() {
    typedef typename RealOf<T>::type Re;
    constexpr double c12[7] = {1.0, 0.86602540378443864676, 0.5, 0.0, -0.5, -0.86602540378443864676, -1.0};
    constexpr double s12[7] = {0.0, 0.5, 0.86602540378443864676, 1.0, 0.86602540378443864676, 0.5, 0.0};
    constexpr double c16[10] = {1.0, 0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0,
                                -0.38268343236508977173, -0.70710678118654752440, -0.92387953251128675613, -1.0,
                                -0.92387953251128675613};
    constexpr double s16[10] = {0.0, 0.38268343236508977173, 0.70710678118654752440, 0.92387953251128675613, 1.0,
                                0.92387953251128675613, 0.70710678118654752440, 0.38268343236508977173, 0.0,
                                -0.38268343236508977173};
    static_assert(R == 12 || R == 16, "composite radix");
    if constexpr (R == 12) return mk<T>(Re(c12[M]), Re(-s12[M]));
    else return mk<T>(Re(c16[M]), Re(-s16[M]));
}
// length R = A x 4 (12, 16) in registers: X[k1 + A k2] = sum_n2 W_4^(n2 k2) W_R^(n2 k1) sum_n1 W_A^(n1 k1) x[4 n1 + n2]
template <int R, int K1, int N2, class T>
__device__ __forceinline__ void inner_twiddle(T& v) {
    if constexpr (K1 * N2 > 0) v = v * root_of_unity<R, K1 * N2, T>();
}
template <int A, int N2, class T>
__device__ __forceinline__ void composite_column(T* v) {
    T a[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) a[n1] = v[4 * n1 + N2];
    dft<A>(a);
    inner_twiddle<4 * A, 1, N2>(a[1]);
    inner_twiddle<4 * A, 2, N2>(a[2]);
    if constexpr (A > 3) inner_twiddle<4 * A, 3, N2>(a[3]);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) v[4 * k1 + N2] = a[k1];
}
template <int R, class T>
__device__ __forceinline__ void dft_any(T* v) {
    if constexpr (R == 12 || R == 16) {
        constexpr int A = R / 4;
        composite_column<A, 0>(v); composite_column<A, 1>(v); composite_column<A, 2>(v); composite_column<A, 3>(v);
        T o[R];
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            T b[4] = {v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]};
            dft4(b);
#pragma unroll
            for (int k2 = 0; k2 < 4; ++k2) o[k1 + A * k2] = b[k2];
        }
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = o[k];
    } else {
        dft<R>(v);
    }
}
// position p of a line in shared memory: a pad slot per first radix (8 or 16), so that the first pass's stores (stride R) and
// the next one's loads (consecutive) meet no bank twice; a line takes row_stride<N>() slots at most
template <int N>
__device__ __forceinline__ int fftr_at(int p) { return p + (p >> (FftRegPlan<N>::R[0] == 16 ? 4 : 3)); }
template <int N> constexpr bool fftr_in_warp() { return FftRegPlan<N>::T <= 32; }
template <int N>
__device__ __forceinline__ void fftr_sync() {
    if constexpr (fftr_in_warp<N>()) __syncwarp();
    else __syncthreads();
}
// pass P at stride L of the line's values v (v[j] = x[t + T j]); sm: the line's row_stride<N>() values of shared memory
template <int N, int P, int L, class T>
__device__ __forceinline__ void fftr_passes(T* v, T* sm, int t, const T* __restrict__ tw) {
    using S = FftRegPlan<N>;
    constexpr int R = S::R[P], E = S::E, TT = S::T, BPT = E / R, M = N / (L * R);
    constexpr bool last = L * R == N;
    if constexpr (L > 1) {                     // the pass before left y in shared memory
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = sm[fftr_at<N>(t + TT * j)];
    }
    // butterfly b = t + T u takes x[q N/R + b], i.e. v[q (N/R)/T + u]
    T o[E];
#pragma unroll
    for (int u = 0; u < BPT; ++u) {
        T w[R];
#pragma unroll
        for (int q = 0; q < R; ++q) w[q] = v[q * BPT + u];
        if constexpr (L > 1) {
            const int k = (t + TT * u) % L;
#pragma unroll
            for (int q = 1; q < R; ++q) w[q] = w[q] * __ldg(&tw[q * k * M]);
        }
        dft_any<R>(w);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if constexpr (last) o[r * BPT + u] = w[r];        // y[r N/R + b]
            else o[u * R + r] = w[r];
        }
    }
    if constexpr (last) {
#pragma unroll
        for (int j = 0; j < E; ++j) v[j] = o[j];
    } else {
        fftr_sync<N>();                                       // the line's reads of this shared memory are done
#pragma unroll
        for (int u = 0; u < BPT; ++u) {
            const int b = t + TT * u, j = b / L, k = b - j * L;
#pragma unroll
            for (int r = 0; r < R; ++r) sm[fftr_at<N>((j * R + r) * L + k)] = o[u * R + r];
        }
        fftr_sync<N>();
        fftr_passes<N, P + 1, L * R>(v, sm, t, tw);
    }
}
// the forward transform of a line, v[j] = x[t + T j] in and out; every thread of the warp (of the CTA for lines longer than a
// warp) calls it
template <int N, class T>
__device__ __forceinline__ void fft_reg(T* v, T* sm, int t, const T* __restrict__ tw) {
    fftr_passes<N, 0, 1>(v, sm, t, tw);
}

// z(k) = a(k) + i b(k) of two real fields' half spectra (k_x = 0 .. N/2), conjugated for an inverse transform: a, b the values
// at k, or for k > N/2 (up) those at N - k, whose conjugates stand there
template <class T>
__device__ __forceinline__ T pair_conj(bool up, T a, T b) {
    return up ? mk<T>(a.x + b.y, a.y - b.x) : mk<T>(a.x - b.y, -(a.y + b.x));
}
// The forward spectrum v of a + i b (a, b real, v[j] = z(t + T j)) split by symmetry into the half spectra of a and b:
// put(k, A(k), B(k)) for k = 0 .. N/2 of this thread. sm: the line's shared memory.
template <int N, class T, class Put>
__device__ __forceinline__ void split_pair(const T* v, T* sm, int t, Put put) {
    using S = FftRegPlan<N>;
    typedef typename RealOf<T>::type Re;
    fftr_sync<N>();
#pragma unroll
    for (int j = 0; j < S::E; ++j) sm[fftr_at<N>(t + S::T * j)] = v[j];
    fftr_sync<N>();
#pragma unroll
    for (int j = 0; j <= S::E / 2; ++j) {
        const int k = t + S::T * j;
        if (j == S::E / 2 && t != 0) continue;               // k = N/2 alone
        const T z = v[j], zm = conj(sm[fftr_at<N>(k == 0 ? 0 : N - k)]);
        const T d = z - zm;
        put(k, Re(0.5) * (z + zm), Re(0.5) * mk<T>(d.y, -d.x));
    }
}

}  // namespace g3d
