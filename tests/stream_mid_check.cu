// Host check of pieces of the streaming push (gem-pic-3d_b200/csrc/k_stream_mid.cuh); compiled by tests/test_stream_mid.py with
// nvcc and run on the CPU (no GPU). Prints one line per check.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "k_stream_mid.cuh"

using namespace g3d;

// The weight the gather gives to a node: the midpoint fields are 1 at that node and 0 elsewhere, so no sum rounds. Largest
// relative error over the nine nodes against the weights in FP64, over random positions.
template <bool F32, bool LASER>
static double weight_error(bool ext) {
    const int nx = 24, ny = 16;
    StreamArgs c{};
    c.g.nx = nx; c.g.ny = ny; c.g.dx = 0.3; c.g.dy = 0.21;
    c.inv_dx = 1 / c.g.dx; c.inv_dy = 1 / c.g.dy;
    c.ext.nu = ext ? 1 : 0;
    std::vector<double> F(size_t(nx) * ny * 6, 0.0);             // 48 bytes a point, of which the FP32 form uses 32
    c.Fmid = F.data();
    std::mt19937_64 rng(5);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    double worst = 0;
    for (int k = 0; k < 4000; ++k) {
        const double x = (-0.5 + 2 * U(rng)) * nx * c.g.dx, y = (-0.5 + 2 * U(rng)) * ny * c.g.dy;      // some outside the box
        int ix[3], jn[3];
        double wx[3], wy[3];
        tsc_stream<double>(x, c.inv_dx, nx, ix, wx);
        tsc_stream<double>(y, c.inv_dy, ny, jn, wy);
        auto w = [](double t, int q) -> double {
            const double f = t - std::floor(t + 0.5);
            return q == 0 ? 0.5 * (0.5 - f) * (0.5 - f) : q == 1 ? 0.75 - f * f : 0.5 * (0.5 + f) * (0.5 + f);
        };
        for (int j = 0; j < 3; ++j)
            for (int i = 0; i < 3; ++i) {
                const double want = w(x * c.inv_dx, i) * w(y * c.inv_dy, j);
                if (want < 1e-4) continue;                      // towards the stencil's edge the offset's own rounding counts
                const int p = jn[j] * nx + ix[i];
                double E[3], B[3];
                float* f = reinterpret_cast<float*>(F.data()) + 8 * size_t(p);
                double* d = F.data() + 6 * size_t(p);
                for (int q = 0; q < 6; ++q) { if (F32) f[q] = 1.f; else d[q] = 1.0; }
                sgather_midpoint<F32, LASER>(c, x, y, E, B);
                for (int q = 0; q < 6; ++q) { if (F32) f[q] = 0.f; else d[q] = 0.0; }
                for (int q = 0; q < 3; ++q)
                    worst = std::max({worst, double(std::fabs(E[q] - want) / want), double(std::fabs(B[q] - want) / want)});
            }
    }
    return worst;
}

// The half-cell's time of a particle that runs backwards with p_z = -P, its reciprocal roots off by a unit in the last place:
// gamma + p_z not below zero, the time finite and not negative, and its error no larger than the one of the textbook form
// (roots and quotients, over the same draws).
static bool backwards(double P, double& err, double& err_ref) {
    std::mt19937_64 rng(9);
    std::normal_distribution<double> G(0.0, 0.3);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    bool ok = true;
    err = err_ref = 0;
    for (int k = 0; k < 3000; ++k) {
        double N[2], D[2], omv[2], ex[2];
        for (int s = 0; s < 2; ++s) {
            const double px = k % 3 ? G(rng) : 0.0, py = k % 3 ? G(rng) : 0.0, pz = -P * (1 + 0.2 * U(rng));
            N[s] = 1 + px * px + py * py;
            const double a = N[s] + pz * pz, r = 1 / std::sqrt(a);
            const double g = gamma_root(a, k % 2 ? std::nextafter(r, 0.0) : std::nextafter(r, 2.0)), gr = std::sqrt(a);
            ok = ok && g + pz >= 0;
            D[s] = g * (g + pz);
            omv[s] = N[s] / (gr * (gr + pz));
            ex[s] = 1 + std::fabs(pz) / std::sqrt(1 + px * px + py * py + pz * pz);       // 1 - v_z, nothing cancels
        }
        const double dt = halfcell_time(0.2, N[0], D[0], N[1], D[1]), ref = 2 * 0.2 / (omv[0] + omv[1]), want = 2 * 0.2 / (ex[0] + ex[1]);
        ok = ok && std::isfinite(dt) && dt >= 0;
        err = std::max(err, std::fabs(dt - want) / want);
        err_ref = std::max(err_ref, std::fabs(ref - want) / want);
    }
    return ok;
}

int main() {
    // FP64 weights: the product's one rounding to FP32, 2^-24, and FP64 roundings (the offset of a weight of 1e-4: 1e-13)
    const double one = std::ldexp(1.0, -24) * (1 + 1e-5);
    struct { const char* what; double err, bound; } r[] = {
        {"fp64", weight_error<false, false>(false), 1e-12},
        {"mixed, wave", weight_error<true, true>(false), one},
        {"mixed, external element", weight_error<true, false>(true), one},
        {"mixed, wave and external element", weight_error<true, true>(true), one},
        // FP32 weights: offset, square, factor and product each round once, and the offset's error grows by 2 |w'| f / w <= 15
        // at a weight of 1e-2 squared
        {"mixed", weight_error<true, false>(false), 64 * std::ldexp(1.0, -24)},
    };
    int bad = 0;
    for (const auto& q : r) {
        std::printf("weights, %s: largest relative error %.3e (bound %.3e)\n", q.what, q.err, q.bound);
        bad += !(q.err <= q.bound);
    }
    for (double P : {0.01, 1.0, 30.0, 1e3, 1e5, 1e7, 4e7, 6e7, 1e8, 1e10, 1e30}) {
        double err, ref;
        const bool ok = backwards(P, err, ref);
        const bool good = ok && err <= 1.02 * ref + 4e-16;              // the other form's products and quotients round otherwise
        std::printf("time at p_z = -%g: %s, largest relative error %.3e (roots and quotients %.3e)\n", P, ok ? "sound" : "NOT SOUND", err, ref);
        bad += !good;
    }
    return bad;
}
