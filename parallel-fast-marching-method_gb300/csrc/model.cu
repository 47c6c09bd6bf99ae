// model.cu -- kernel (a): cubic B-spline gridder of the velocity nodes onto
// the propagation grid (fm3dt_parallel.f90 gridder, F:6989-7038), and the
// slowness field the solver reads.
//
// Compiled without FMA contraction so that every double-precision value is
// rounded exactly like the reference's left-to-right Fortran arithmetic.
#include "internal.h"

namespace fm3dt {

__device__ __forceinline__ void bspline4(double u, double w[4])
{
    // F:7002-7005
    const double u2 = u * u, u3 = u * u * u;
    const double om = 1.0 - u;
    w[0] = om * om * om / 6.0;
    w[1] = (4.0 - 6.0 * u2 + 3.0 * u3) / 6.0;
    w[2] = (1.0 + 3.0 * u + 3.0 * u2 - 3.0 * u3) / 6.0;
    w[3] = u3 / 6.0;
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// Velocity indices that would fall outside 0..nv+1 are clamped (the
// reference reads outside its array there; inputs that cover the grid, as
// the .vtx convention intends, never clamp).
//
// The reference's triple sum (F:7006-7035) is separable as it is written: the
// innermost sum (over r nodes) depends on the node's layer and the velocity
// column, the next (over theta) on layer, row and phi node, the outer one on
// the node.  Each is formed once, in the reference's order -- the same
// operations, hence the same bits -- in three passes, from weights formed
// once per axis index: 8 double-precision operations per node instead of
// ~170 with 3 divisions.  One thread per node over the whole sum was bound by
// the double-precision pipe (2 lanes per SM and cycle): 7.07 ms on 195 x 227
// x 227 nodes from 18 x 22 x 22 velocity nodes, 12.2 ms on 259^3, and 0.09 /
// 0.18 ms for the slowness.  Now 0.34 / 0.54 ms with the slowness fused in, 93%
// of it the last pass, still on that pipe (its division for the most part).
struct SplineAxis {
    double w[4];
    long long c;          // first of the four velocity nodes
};

// weights of every padded index of an axis (r, then theta, then phi; index i
// stands for the reference's i - 1)
__global__ void spline_axes_kernel(Geom g, SplineAxis *__restrict__ ax)
{
    const int PZ = g.nnz + 3, PX = g.nnx + 3, PR = g.nnr + 3;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < PR + PX + PZ; q += gridDim.x * blockDim.x) {
        SplineAxis a;
        if (q < PR) {
            const int k = q - 1;
            const int ri = (int)floor((g.gor - g.rgor + (double)(k - 1) * g.dnr) / g.dvr) + 1;
            const double distr = -(g.rgor - (double)(k - 1) * g.dnr) + (g.gor - (double)(ri - 1) * g.dvr);
            bspline4(distr / g.dvr, a.w);
            a.c = ri - 1;
        } else if (q < PR + PX) {
            const int j = q - PR - 1;
            const double xpos = g.rgox + (double)(j - 1) * g.dnx - g.gox;
            const int xi = (int)floor(xpos / g.dvx) + 1;
            bspline4((xpos - (double)(xi - 1) * g.dvx) / g.dvx, a.w);
            a.c = xi - 1;
        } else {
            const int i = q - PR - PX - 1;
            const double zpos = g.rgoz + (double)(i - 1) * g.dnz - g.goz;
            const int zi = (int)floor(zpos / g.dvz) + 1;
            bspline4((zpos - (double)(zi - 1) * g.dvz) / g.dvz, a.w);
            a.c = zi - 1;
        }
        ax[q] = a;
    }
}

// sums over r: rs[k][c][b] for padded layer k and velocity column (theta
// node b, phi node c)
__global__ void spline_r_kernel(Geom g, const SplineAxis *__restrict__ ax, const double *__restrict__ velv,
                                double *__restrict__ rs)
{
    const int ncol = (g.nvx + 2) * (g.nvz + 2);
    const long long total = (long long)ncol * (g.nnr + 3);
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(q / ncol), col = (int)(q - (long long)k * ncol);
        const SplineAxis &a = ax[k];
        const double *v = velv + (size_t)(g.nvr + 2) * col;
        double sum = 0.0;
        for (int k1 = 0; k1 < 4; ++k1) sum = sum + a.w[k1] * __ldg(v + clampi((int)a.c + k1, 0, g.nvr + 1));
        rs[q] = sum;
    }
}

// sums over theta: xs[k][j][c] for padded layer k, row j and phi node c
__global__ void spline_x_kernel(Geom g, const SplineAxis *__restrict__ ax, const double *__restrict__ rs,
                                double *__restrict__ xs)
{
    const int NVX = g.nvx + 2, NVZ = g.nvz + 2, PX = g.nnx + 3;
    const long long total = (long long)(g.nnr + 3) * PX * NVZ;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < total;
         q += (long long)gridDim.x * blockDim.x) {
        const long long kj = q / NVZ;
        const int c = (int)(q - kj * NVZ), k = (int)(kj / PX), j = (int)(kj - (long long)k * PX);
        const SplineAxis &a = ax[g.nnr + 3 + j];
        const double *v = rs + ((size_t)k * NVZ + c) * NVX;
        double sum = 0.0;
        for (int j1 = 0; j1 < 4; ++j1) sum = sum + a.w[j1] * v[clampi((int)a.c + j1, 0, g.nvx + 1)];
        xs[q] = sum;
    }
}

// sums over phi, one warp per (layer, row) of nodes; and the slowness
// 1/velocity of the interior nodes (F:642), in the solver's precision, phi
// fastest; velf: the velocity in single precision, for the rays' weights
template <typename R>
__global__ void spline_z_kernel(Geom g, const SplineAxis *__restrict__ ax, const double *__restrict__ xs,
                                double *__restrict__ veln, float *__restrict__ velf, R *__restrict__ s)
{
    const int NVZ = g.nvz + 2, PX = g.nnx + 3, PZ = g.nnz + 3;
    const long long rows = (long long)(g.nnr + 3) * PX;
    for (long long kj = blockIdx.x * (long long)blockDim.y + threadIdx.y; kj < rows;
         kj += (long long)gridDim.x * blockDim.y) {
        const int k = (int)(kj / PX), j = (int)(kj - (long long)k * PX);
        const double *v = xs + (size_t)kj * NVZ;
        const bool in = k >= 2 && k < g.nnr + 2 && j >= 2 && j < g.nnx + 2;
        R *sr = s + ((size_t)(k - 2) * g.nnx + (j - 2)) * g.nnz;      // (used when in)
        for (int i = threadIdx.x; i < PZ; i += 32) {
            const SplineAxis &a = ax[g.nnr + 3 + PX + i];
            double sum = 0.0;
            for (int i1 = 0; i1 < 4; ++i1) sum = sum + a.w[i1] * v[clampi((int)a.c + i1, 0, g.nvz + 1)];
            veln[(size_t)kj * PZ + i] = sum;
            velf[(size_t)kj * PZ + i] = (float)sum;
            if (in && i >= 2 && i < g.nnz + 2) sr[i - 2] = (R)(1.0 / sum);
        }
    }
}

static int grid_for(long long n, int block)
{
    long long b = (n + block - 1) / block;
    if (b > 152LL * 64) b = 152LL * 64;
    return (int)(b < 1 ? 1 : b);
}

size_t gridder_scratch(const Geom &g)
{
    const size_t axes = (size_t)(g.nnr + g.nnx + g.nnz + 9) * (sizeof(SplineAxis) / sizeof(double));
    return axes + (size_t)(g.nnr + 3) * (g.nvz + 2) * ((g.nvx + 2) + (size_t)(g.nnx + 3));
}

void launch_gridder(const Geom &g, const double *velv, double *veln, float *velf, void *s, int prec, double *scratch,
                    cudaStream_t st)
{
    const int na = g.nnr + g.nnx + g.nnz + 9;
    SplineAxis *ax = (SplineAxis *)scratch;
    double *rs = scratch + (size_t)na * (sizeof(SplineAxis) / sizeof(double));
    const long long nr = (long long)(g.nnr + 3) * (g.nvx + 2) * (g.nvz + 2);
    double *xs = rs + nr;
    spline_axes_kernel<<<(na + 63) / 64, 64, 0, st>>>(g, ax);
    spline_r_kernel<<<grid_for(nr, 128), 128, 0, st>>>(g, ax, velv, rs);
    spline_x_kernel<<<grid_for((long long)(g.nnr + 3) * (g.nnx + 3) * (g.nvz + 2), 256), 256, 0, st>>>(g, ax, rs, xs);
    const dim3 block(32, 4);
    const int grid = grid_for((long long)(g.nnr + 3) * (g.nnx + 3), 4);
    if (prec == FM3DT_FP64)
        spline_z_kernel<double><<<grid, block, 0, st>>>(g, ax, xs, veln, velf, (double *)s);
    else
        spline_z_kernel<float><<<grid, block, 0, st>>>(g, ax, xs, veln, velf, (float *)s);
}

}  // namespace fm3dt
