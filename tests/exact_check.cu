// exact_check.cu -- the exact fold (mc_exact.cu) against big integers on the
// host, and the ordered fold on columns of a few histories.  Columns chosen
// where the 128-bit window can go wrong: both signs, values far below the
// largest of a slice, subnormals, squares that overflow, underflow or become
// subnormal, the largest doubles, values that are left out; history counts
// at the edges of a vector and of a slice.  Prints "ok" or what differs.
#include <cfloat>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "mc_exact.cu"
#include "mc_fold.cuh"

static double column(int kind, std::mt19937_64 &g, uint32_t h)
{
    std::uniform_real_distribution<double> u(0.0, 1.0);
    switch (kind) {
    case 0: return u(g);
    case 1: return u(g) < 0.02 ? u(g) * 1e-3 : 0.0;
    case 2: return u(g) - 0.5;
    case 3: return (u(g) < 0.5 ? -1.0 : 1.0) * std::ldexp(1.0 + u(g), (int)(g() % 80) - 40);
    case 4: return std::ldexp(u(g) - 0.5, -1060);
    case 5: return (g() & 1 ? -1.0 : 1.0) * (h % 97 == 3 ? std::ldexp(u(g), 300) : std::ldexp(u(g), -300));
    case 6: return std::ldexp(u(g) - 0.5, 600);
    case 7: return std::ldexp(u(g), -530 - (int)(g() % 12));
    case 8: return (g() & 1 ? -1.0 : 1.0) * DBL_MAX * (1.0 - 0.5 * u(g));
    case 9: return g() & 1 ? -0.0 : 0.0;
    case 10: return h == 5 ? 1e300 : (h == 4099 ? -1e300 : u(g));
    case 11: return (g() & 1 ? -1.0 : 1.0) * 4.9e-324 * (double)(g() % 5);
    case 12: return h % 50 == 7 ? INFINITY : (h % 50 == 8 ? NAN : u(g) - 0.5);
    default: return h % 2 ? -0.75 : 0.75;
    }
}
constexpr int kKinds = 14;

// v 2^1074 into an integer of 32-bit digits (carried on the way)
static void host_add(std::vector<__int128> &a, double v)
{
    if (v == 0.0 || !std::isfinite(v)) return;
    int e;
    const double f = std::frexp(std::fabs(v), &e);              // v = f 2^e
    unsigned long long m = (unsigned long long)std::ldexp(f, 53);
    int p = e - 53 + 1074;
    if (p < 0) { m >>= -p; p = 0; }                             // (a subnormal's low bits are zero)
    const unsigned __int128 x = (unsigned __int128)m << (p & 31);
    for (int i = 0; i < 3; ++i) {
        const __int128 d = (__int128)((x >> (32 * i)) & 0xFFFFFFFFu);
        a[p / 32 + i] += v < 0.0 ? -d : d;
    }
}

int main()
{
    int bad = 0;
    for (uint32_t n : {1u, 2u, 3u, 7u, 8u, 9u, 17u, 4095u, 4096u, 4097u, 9001u}) {
        std::mt19937_64 g(n);
        const size_t ld = mc::hist_rows(n);
        std::vector<double> h(ld * kKinds, 0.0), zero(2 * kKinds, 0.0), tree(2 * kKinds), ord(2 * kKinds);
        std::vector<long long> ex((size_t)kKinds * 2 * mc::kExactLimbs, 0);
        for (int b = 0; b < kKinds; ++b)
            for (uint32_t i = 0; i < n; ++i) h[b * ld + i] = column(b, g, i);
        double *dh, *ds;
        long long *de;
        if (cudaMalloc(&dh, h.size() * 8) != cudaSuccess || cudaMalloc(&ds, 4 * kKinds * 8) != cudaSuccess ||
            cudaMalloc(&de, ex.size() * 8) != cudaSuccess) return 2;
        cudaMemcpy(dh, h.data(), h.size() * 8, cudaMemcpyHostToDevice);
        cudaMemset(ds, 0, 4 * kKinds * 8);
        cudaMemset(de, 0, ex.size() * 8);
        // the exact sums twice, once with the tree sums; the ordered fold once
        if (mc::launch_fold_exact(dh, n, ld, kKinds, de, ds, ds + kKinds, 0) != cudaSuccess ||
            mc::launch_fold_exact(dh, n, ld, kKinds, de, nullptr, nullptr, 0) != cudaSuccess ||
            mc::launch_exact_normalize(de, kKinds, 0) != cudaSuccess) return 2;
        mc::k_fold_ordered<<<dim3(kKinds, 2), mc::kFoldThreads>>>(dh, n, ld, ds + 2 * kKinds, ds + 3 * kKinds);
        cudaMemcpy(tree.data(), ds, 2 * kKinds * 8, cudaMemcpyDeviceToHost);
        cudaMemcpy(ord.data(), ds + 2 * kKinds, 2 * kKinds * 8, cudaMemcpyDeviceToHost);
        if (cudaMemcpy(ex.data(), de, ex.size() * 8, cudaMemcpyDeviceToHost) != cudaSuccess) { std::printf("CUDA error\n"); return 2; }
        cudaFree(dh);
        cudaFree(ds);
        cudaFree(de);
        for (int b = 0; b < kKinds; ++b)
            for (int w = 0; w < 2; ++w) {
                std::vector<__int128> want(mc::kExactLimbs + 4, 0);
                double serial = 0.0, size = 0.0;
                for (uint32_t i = 0; i < n; ++i) {
                    const double v = h[b * ld + i], x = w ? v * v : v;
                    host_add(want, std::isfinite(v) ? x : 0.0);
                    host_add(want, std::isfinite(v) ? x : 0.0);
                    serial += x;
                    size += std::fabs(x);
                }
                for (int j = 0; j + 1 < mc::kExactLimbs; ++j) {
                    const __int128 c = want[j] >> 32;
                    want[j] -= c << 32;
                    want[j + 1] += c;
                }
                for (int j = 0; j < mc::kExactLimbs; ++j)
                    if ((__int128)ex[((size_t)b * 2 + w) * mc::kExactLimbs + j] != want[j]) {
                        std::printf("n %u column %d %s: limb %d differs\n", n, b, w ? "squares" : "sum", j);
                        ++bad;
                        break;
                    }
                const double o = ord[w * kKinds + b], t = tree[w * kKinds + b];
                if (std::memcmp(&o, &serial, 8) != 0 && !(std::isnan(o) && std::isnan(serial))) {
                    std::printf("n %u column %d: ordered %a want %a\n", n, b, o, serial);
                    ++bad;
                }
                // n terms in any order: (n - 1) 2^-53 of the sum of their sizes, twice that for two orders
                if (std::isfinite(size) && !(std::fabs(t - serial) <= 2.0 * n * 0x1p-53 * size)) {
                    std::printf("n %u column %d: tree %a serial %a\n", n, b, t, serial);
                    ++bad;
                }
            }
    }
    if (!bad) std::printf("ok\n");
    return bad != 0;
}
