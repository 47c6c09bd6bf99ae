// Device check of the node update's short forms (stencil.cuh), whose decisions
// rest on the GPU's approximate single-precision square root and division:
// fm_update and fm_update_upstream against the general octant form, bit for
// bit, in both precisions.  Nodes where the decisions are close: keys that
// differ by 1e-15 to 1e-1 of each other, second neighbours next to the first
// ones, keys far above the others, unset neighbours and neighbours outside the
// grid, equal and very unequal spacings, both orders.
//
//   nvcc -gencode arch=compute_103a,code=sm_103a -std=c++17 -fmad=false update_device_check.cu -o check && ./check
#include <cstdio>

#include "../parallel-fast-marching-method_gb300/csrc/stencil.cuh"

using fm3dt::Lim;
using fm3dt::Spacing;

struct Rng {
    unsigned long long x;
    __device__ unsigned long long bits()              // splitmix64 (Steele, Lea, Flood 2014)
    {
        unsigned long long z = (x += 0x9e3779b97f4a7c15ull);
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        return z ^ (z >> 31);
    }
    __device__ int below(int n) { return (int)(bits() % (unsigned)n); }
    __device__ double u() { return (double)(bits() >> 11) * 0x1p-53; }
};

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }
__device__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }

template <typename R>
__global__ void check(int n, unsigned long long seed, unsigned *bad)
{
    const R INF = Lim<R>::inf(), nan = INF - INF;
    const double near[6] = {1e-1, 3e-3, 3e-4, 1e-6, 1e-12, 1e-15};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        Rng g{seed + 0x632be59bd9b4e019ull * (unsigned long long)i};
        const double base = g.below(2) ? (sizeof(R) == 8 ? 600.0 : 60.0) : 0.5, ep = near[g.below(6)];
        const double c0 = g.u(), far = g.below(4) ? 1.0 : pow(10.0, 3.0 * g.u());
        const double cs[4] = {0.0, c0, c0 * (1 + ep * (g.u() - 0.5)), g.below(2) ? g.u() : c0 * (1 + ep * (g.u() - 0.5))};
        R t1[6], t2[6];
        const unsigned inb = g.below(4) ? 63u : (unsigned)g.below(64);
        for (int d = 0; d < 6; ++d) {
            const double k = cs[g.below(4)] * (g.below(4) ? 1.0 : far);
            t1[d] = g.below(15) ? R(base + k) : INF;
            const int z = g.below(3);
            t2[d] = z == 0 ? R(fmax(0.0, base + k - 0.8 * g.u() * (g.below(5) ? 1.0 : far)))
                  : z == 1 ? R(fmax(0.0, base + k + (g.u() - 0.5) * ep)) : INF;
            if (!((inb >> d) & 1u)) {
                t1[d] = g.below(2) ? INF : nan;
                t2[d] = g.below(2) ? INF : nan;
            }
        }
        Spacing<R> sp;
        for (int a = 0; a < 3; ++a) {
            sp.h[a] = R(g.below(4) ? 0.5 + 2.5 * g.u() : g.below(2) ? 1.0 : 0.05 + 8.0 * g.u());
            sp.w[a] = R(1) / (sp.h[a] * sp.h[a]);
        }
        const R s = R(0.1 + g.u());
        const int order2 = g.below(2);
        const R want = fm3dt::fm_update_octants<R>(s, t1, t2, inb, sp, order2);
        if (!same(want, fm3dt::fm_update<R>(s, t1, t2, inb, sp, order2))) atomicAdd(bad, 1u);
        // upstream only: down, and the lateral sides a sweep comes from
        const int dX = 2 + g.below(2), dZ = 4 + g.below(2);
        for (int d = 0; d < 6; ++d) {
            const bool out = !((inb >> d) & 1u);
            if (d == 0 || d == (dX ^ 1) || d == (dZ ^ 1) || out) t1[d] = INF;
            if (out) t2[d] = INF;
        }
        auto in = [&](int d) { return ((inb >> d) & 1u) != 0; };
        const R up = fm3dt::fm_update_octants<R>(s, t1, t2, inb, sp, order2);
        const R got = fm3dt::fm_update_upstream<R>(s, t1[1], t2[1], t1[dX], t2[dX], t1[dZ], t2[dZ], in(1), in(0), in(dX),
                                                   in(dX ^ 1), in(dZ), in(dZ ^ 1), sp, order2);
        if (!same(up, got)) atomicAdd(bad + 1, 1u);
    }
}

int main()
{
    const int n = 1 << 22;
    unsigned *bad = nullptr, h[4];
    if (cudaMalloc(&bad, sizeof h) != cudaSuccess || cudaMemset(bad, 0, sizeof h) != cudaSuccess) return 3;
    check<float><<<2048, 128>>>(n, 1, bad);
    check<double><<<2048, 128>>>(n, 2, bad + 2);
    if (cudaMemcpy(h, bad, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    std::printf("of %d: single update %u, upstream %u differ; double update %u, upstream %u\n", n, h[0], h[1], h[2], h[3]);
    return h[0] || h[1] || h[2] || h[3];
}
