// sphere_direction_check.cu -- sphere_beyond against surface_distance for
// directions that are not unit vectors (a source's direction is taken as
// given, and a particle keeps it until its first collision): lengths from 1/2
// to 128, points, tangents and flights as in sphere_check.cu.  Prints "ok" or
// the count.
#include <cstdio>

#include "mc_event_kernels.cuh"

using namespace mc;
using namespace mc::ev;

__global__ void k_check(uint64_t n, unsigned long long *cnt)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const U4 a = philox((uint32_t)i, (uint32_t)(i >> 32), 1, 2, 3, 4), b = philox((uint32_t)i, (uint32_t)(i >> 32), 2, 2, 3, 4);
        const U4 c = philox((uint32_t)i, (uint32_t)(i >> 32), 3, 2, 3, 4);
        auto u01 = [](uint32_t x) { return ((float)(x >> 8) + 0.5f) * 0x1p-24f; };
        const float r = exp2f(20.f * u01(a.x) - 10.f);
        const float at = (c.x & 3) == 0 ? 0.f : ((c.x & 4) ? 1.f : -1.f) * 3.f * r * u01(c.y);   // centre off the origin
        // radial position: uniform to 2 r, or 2^-1 .. 2^-24 from the surface
        float rho = 2.f * r * u01(a.y);
        if (c.x & 8) rho = r * (1.f + ((c.x & 16) ? 1.f : -1.f) * exp2f(-24.f * u01(a.y)));
        const float m = 2.f * u01(a.z) - 1.f, ph = 6.2831853f * u01(a.w), q = sqrtf(fmaxf(0.f, 1.f - m * m));
        PState p = {};
        const int kb = (int)(c.z >> 2) % 9; const float K = exp2f((float)kb - 1.f);   // direction's length
        float nx = q * cosf(ph), ny = q * sinf(ph), nz = m;
        p.x = at + rho * nx; p.y = rho * ny; p.z = rho * nz;
        // direction: at a cosine to the outward normal that is uniform, 0, or that of the tangent to the sphere
        float w = 2.f * u01(b.x) - 1.f;
        const int dk = c.z & 3;
        if (dk == 1) w = 0.f;
        if (dk == 2 && rho > r) w = -sqrtf(fmaxf(0.f, (1.f - r / rho) * (1.f + r / rho))) / K * (1.f + (u01(b.x) - 0.5f) * exp2f(-24.f * u01(b.y)));
        const float ps = 6.2831853f * u01(b.z), sw = sqrtf(fmaxf(0.f, 1.f - w * w));
        // two vectors across the normal
        float tx = -ny, ty = nx, tz = 0.f;
        if (q < 0.1f) { tx = 0.f; ty = -nz; tz = ny; }
        const float it = rsqrtf(tx * tx + ty * ty + tz * tz);
        tx *= it; ty *= it; tz *= it;
        const float sx = ny * tz - nz * ty, sy = nz * tx - nx * tz, sz = nx * ty - ny * tx;
        p.u = K * (w * nx + sw * (cosf(ps) * tx + sinf(ps) * sx));
        p.v = K * (w * ny + sw * (cosf(ps) * ty + sinf(ps) * sy));
        p.w = K * (w * nz + sw * (cosf(ps) * tz + sinf(ps) * sz));
        const float k[5] = {at, 0.f, 0.f, r, r * r};
        const float d = surface_distance(4, k, p, false);
        float l = 4.f * r * u01(b.w);
        if ((c.w & 3) == 1 && d < 1e30f) l = d * (1.f + ((c.w & 4) ? 1.f : -1.f) * exp2f(-24.f * u01(c.y)));
        if ((c.w & 3) == 2) l = r * exp2f(40.f * u01(b.w) - 20.f);
        if ((c.w & 63) == 3) l = 0.9f * FLT_MAX;
        if (sphere_beyond(k, p, l) && l > d) atomicAdd(cnt + kb, 1ull);
    }
}

int main()
{
    unsigned long long *d, h[9], n = 0;
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 2;
    k_check<<<152 * 4, 128>>>(1ull << 27, d);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    for (int i = 0; i < 9; ++i) {
        if (h[i]) printf("length 2^%d: reached although passed over: %llu\n", i - 1, h[i]);
        n += h[i];
    }
    if (!n) printf("ok\n");
    return n ? 1 : 0;
}
