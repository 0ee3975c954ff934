// plain_check.cu -- the FP32 bounds and decisions of the FP64 kernels as the
// plain mode has them, built with FMA contraction: each decision against the
// FP64 one of the same build, over random and edge inputs.  (fp64_check.cu
// holds the replay mode's, built without.)  Prints "ok" or what differs.
#include <cstdio>
#include <vector>

#include "mc_history_kernels.cuh"

using namespace mc;

enum { E_DIV, E_BRANCH, E_CAND, E_DIST, E_OUT, E_N };

__global__ void k_check(DevTables T, int n_surf, uint64_t n, unsigned long long *err)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const U4 a = philox((uint32_t)i, (uint32_t)(i >> 32), 1, 2, 3, 4), e = philox((uint32_t)i, (uint32_t)(i >> 32), 2, 2, 3, 4);
        const U4 c = philox((uint32_t)i, (uint32_t)(i >> 32), 3, 2, 3, 4);
        auto pick = [&](uint32_t lo, uint32_t hi) -> uint64_t {
            const uint64_t v = (((uint64_t)hi << 32) | lo) >> 12;
            if ((i & 15) != 0) return v;
            const uint64_t at[4] = {0, (1ull << 52) - 1, 1ull << 51, 1ull << 50};   // the ends, quadrants, and their neighbours
            return (at[v & 3] + ((v >> 2) % 5) - 2) & ((1ull << 52) - 1);
        };
        const uint64_t v1 = pick(a.x, a.y), v2 = pick(a.z, a.w), v3 = pick(e.x, e.y), v4 = pick(e.z, e.w), v5 = pick(c.x, c.y);
        const double u1 = u01_bits(v1), u2 = u01_bits(v2), u3 = u01_bits(v3);
        {
            const double d = dfrom((dbits(u2) & 0x000FFFFFFFFFFFFFull) | ((uint64_t)(1023 - 150 + c.z % 300) << 52));
            const double x = dfrom((dbits(u1) & 0x800FFFFFFFFFFFFFull) | ((uint64_t)(1023 - 250 + c.w % 500) << 52) | ((uint64_t)(c.z & 1) << 63));
            const double hi = 1.0 / d;
            if (dbits(div_by(x, d, Recip64{hi, __fma_rn(-d, hi, 1.0) * hi})) != dbits(x / d)) atomicAdd(err + E_DIV, 1ull);
        }
        // free-gas candidates from y = 1e-3 (far below thermal) to 1e5
        {
            const double speed = exp(-7.0 + 18.5 * ((double)v5 * 0x1p-52));
            const float y32 = f32_of(speed);
            int is = branch_test(v4, y32);
            if (is >= 0 && (is != 0) != (u01_bits(v4) < 2.0 / (2.0 + kPiSqrt * speed))) atomicAdd(err + E_BRANCH, 1ull);
            for (int w = 0; w < 2; ++w) {
                // the acceptance draw near its limit half of the time
                uint64_t va = (((uint64_t)c.w << 20) ^ e.x) & ((1ull << 52) - 1);
                if (i & 1) {
                    const double x = w ? sqrt(-log(u1 * u2)) : sqrt(-log(u2) - log(u3) * cos(kPiHalf * u1) * cos(kPiHalf * u1));
                    const double acc = sqrt(speed * speed + x * x - 2.0 * speed * x * mu_bits(v4)) / (speed + x);
                    va = (uint64_t)fmin(fmax(acc * (1.0 + ((double)c.z * 0x1p-32 - 0.5) * 4e-4) * 0x1p52, 0.0), 0x1p52 - 1.0);
                }
                is = candidate_test(w != 0, v1, v2, v3, v4, va, y32);
                if (is >= 0 && (is != 0) != candidate_accepted<false>(w != 0, v1, v2, v3, v4, va, 1.0, speed)) atomicAdd(err + E_CAND, 1ull);
            }
        }
        // surfaces: points near to and far from them, unit directions and others
        {
            const int s = (int)(c.w % (uint32_t)n_surf);
            const double far = (i & 2) ? 100.0 : 12.0;
            double x = far * (2.0 * u1 - 1.0), y = far * (2.0 * u2 - 1.0), z = far * (2.0 * u3 - 1.0);
            double u = mu_bits(v4), v = mu_bits(v5), w = mu_bits(v1);
            const double len = (i & 4) ? sqrt(u * u + v * v + w * w) : ((i & 64) ? 0.05 : 1.0);   // of length 1, up to 1.7 or 35
            u /= len; v /= len; w /= len;
            if (i & 8) {           // onto the surface, then off it by a nudge
                const double d = surface_distance(T, s, x, y, z, u, v, w);
                if (d < 1e6) {
                    const double o = d + ((i & 16) ? kEpsF : -kEpsF) * ((i & 32) ? 1.0 : 1e3);
                    x += u * o; y += v * o; z += w * o;
                }
            }
            const float reach = (float)exp(-14.0 + 20.0 * ((double)(c.x >> 8) * 0x1p-24));
            const float2 b = distance_bounds(T, s, x, y, z, u, v, w, reach);
            const double d = surface_distance(T, s, x, y, z, u, v, w), dd = d >= kMaxF ? (double)kInfF : d;
            if (!(b.x == kInfF ? (dd == (double)kInfF || d > (double)reach) : ((double)b.x <= dd && dd <= (double)b.y))) atomicAdd(err + E_DIST, 1ull);
            for (int sense = -1; sense <= 1; ++sense)
                if (outside(T, s, sense, x, y, z) != (surface_eval(T, s, x, y, z) * sense < 0)) atomicAdd(err + E_OUT, 1ull);
        }
    }
}

int main()
{
    // planes, general planes, spheres and cylinders, centred and not
    std::vector<int> type;
    std::vector<double> k;
    auto add = [&](int t, std::vector<double> c) { type.push_back(t); c.resize(8, 0.0); k.insert(k.end(), c.begin(), c.end()); };
    for (int t = 0; t < 3; ++t) { add(t, {0.0}); add(t, {7.25}); add(t, {-90.0}); add(t, {1e-9}); }
    add(3, {1.0, 0.5, -0.25, 6.0}); add(3, {-1.0, 0.2, 0.1, 6.0});
    for (double r : {0.5, 10.0, 30.0, 70.0}) {
        add(4, {0.0, 0.0, 0.0, r, r * r}); add(4, {3.0, -40.0, 0.1, r, r * r});
        add(5, {0.0, 0.0, r, r * r}); add(5, {5.0, -1.0, r, r * r});
        add(6, {0.5, 0.0, r, r * r});
        add(7, {0.0, 0.0, r, r * r}); add(7, {0.5, -20.0, r, r * r});
    }
    DevTables T{};
    int *dt;
    double *dk;
    unsigned long long *de, e[E_N] = {};
    if (cudaMalloc(&dt, type.size() * 4) != cudaSuccess || cudaMalloc(&dk, k.size() * 8) != cudaSuccess ||
        cudaMalloc(&de, sizeof(e)) != cudaSuccess) return 2;
    cudaMemcpy(dt, type.data(), type.size() * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(dk, k.data(), k.size() * 8, cudaMemcpyHostToDevice);
    cudaMemset(de, 0, sizeof(e));
    T.surf_type = dt;
    T.surf_coef = dk;
    k_check<<<608, 128>>>(T, (int)type.size(), 40000000ull, de);
    if (cudaMemcpy(e, de, sizeof(e), cudaMemcpyDeviceToHost) != cudaSuccess) { std::printf("CUDA error\n"); return 2; }
    const char *what[] = {"division", "branch", "candidate", "distance bounds", "outside"};
    bool bad = false;
    for (int i = 0; i < E_N; ++i)
        if (e[i]) { std::printf("%s: %llu wrong\n", what[i], e[i]); bad = true; }
    if (!bad) std::printf("ok\n");
    return bad;
}
