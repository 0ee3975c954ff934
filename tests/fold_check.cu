// fold_check.cu -- k_fold_ordered against the serial chain it restates.
// Columns chosen where the scan can go wrong: sums that cross binades, ties
// to even in both parities, signed sums about zero, subnormals, zeros, terms
// larger than the sum, infinities and NaN; history counts at the edges of a
// thread's, a block's and several steps' share.  Prints "ok" or what differs.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "mc_fold.cuh"

static double column(int kind, std::mt19937_64 &g, uint32_t h)
{
    std::uniform_real_distribution<double> u(0.0, 1.0);
    switch (kind) {
    case 0: return u(g);
    case 1: return u(g) < 0.02 ? u(g) * 1e-3 : 0.0;
    case 2: return u(g) - 0.5;
    case 3: return h == 0 ? 0x1p53 : (u(g) < 0.5 ? 1.0 : 3.0);              // ties at u = 2
    case 4: return (u(g) < 0.5 ? -1.0 : 1.0) * std::ldexp(1.0 + (g() & 3) * 0.25, (int)(g() % 80) - 40);
    case 5: return std::ldexp(u(g), -1060);                                 // subnormal terms
    case 6: return h % 3000 == 2999 ? 1e6 * u(g) : u(g) * 1e-9;             // jumps of binades
    case 7: return h == 4097 ? INFINITY : (h == 4200 ? -INFINITY : u(g));   // then NaN
    case 8: return h == 0 ? -0x1p53 : (u(g) < 0.5 ? -1.0 : (u(g) < 0.5 ? 1.0 : -3.0));
    case 9: return h % 2 ? -0.75 : 0.75;                                    // back to zero each time
    case 10: return (h / 700) % 2 ? -u(g) : u(g);                           // rises and falls through zero
    case 11: return std::ldexp(u(g) - 0.5, 600);                            // squares overflow
    default: return 0.0;
    }
}

int main()
{
    int bad = 0;
    for (int nb : {1, 13}) {
        for (uint32_t n : {1u, 7u, 8u, 9u, 4095u, 4096u, 4097u, 8193u, 30011u}) {
            for (int start = 0; start < 2; ++start) {
                std::mt19937_64 g(n + nb);
                const size_t ld = (n + 7) & ~7u;
                std::vector<double> h(ld * nb, 0.0), s0(nb), q0(nb);
                for (int b = 0; b < nb; ++b) {
                    s0[b] = start ? (b % 2 ? -3.25 : 1.0) : 0.0;
                    q0[b] = start ? 0.5 : 0.0;
                    const int kind = nb == 1 ? (int)(n % 12) : b;
                    for (uint32_t i = 0; i < n; ++i) h[b * ld + i] = column(kind, g, i);
                }
                std::vector<double> s = s0, q = q0, rs(nb), rq(nb);
                for (int b = 0; b < nb; ++b)
                    for (uint32_t i = 0; i < n; ++i) {
                        const double v = h[b * ld + i];
                        s[b] += v;
                        const double w = v * v;
                        q[b] += w;
                    }
                double *dh, *ds;
                if (cudaMalloc(&dh, h.size() * 8) != cudaSuccess || cudaMalloc(&ds, 2 * nb * 8) != cudaSuccess) return 2;
                cudaMemcpy(dh, h.data(), h.size() * 8, cudaMemcpyHostToDevice);
                cudaMemcpy(ds, s0.data(), nb * 8, cudaMemcpyHostToDevice);
                cudaMemcpy(ds + nb, q0.data(), nb * 8, cudaMemcpyHostToDevice);
                mc::k_fold_ordered<<<dim3(nb, 2), mc::kFoldThreads>>>(dh, n, ld, ds, ds + nb);
                cudaMemcpy(rs.data(), ds, nb * 8, cudaMemcpyDeviceToHost);
                cudaMemcpy(rq.data(), ds + nb, nb * 8, cudaMemcpyDeviceToHost);
                if (cudaGetLastError() != cudaSuccess) { std::printf("CUDA error\n"); return 2; }
                cudaFree(dh);
                cudaFree(ds);
                for (int b = 0; b < nb; ++b) {
                    const bool es = std::memcmp(&s[b], &rs[b], 8) == 0 || (std::isnan(s[b]) && std::isnan(rs[b]));
                    const bool eq = std::memcmp(&q[b], &rq[b], 8) == 0 || (std::isnan(q[b]) && std::isnan(rq[b]));
                    if (!es || !eq) {
                        std::printf("nb %d n %u start %d column %d: sum %a want %a, squares %a want %a\n", nb, n, start,
                                    b, rs[b], s[b], rq[b], q[b]);
                        ++bad;
                    }
                }
            }
        }
    }
    if (!bad) std::printf("ok\n");
    return bad != 0;
}
