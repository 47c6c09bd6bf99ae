// rays.cu -- kernel (d): ray back-tracing down the traveltime gradient and
// Frechet-row assembly (fm3dt_parallel.f90 parallel_rpaths, F:7250-7777, and
// the writer's row merge, F:6503-6599).
//
// One lane traces one (event, receiver) ray over the whole grid, so the
// reference's ray hand-off between subdomains (F:6464-6501) and the partial
// rows it creates disappear; the global outer faces stop a ray exactly where
// the reference's boundary subdomains stop it (clip to the first face
// crossed, F:7474-7541).  The ray path is double precision like the
// reference's (with the single-precision field, each step's direction is
// formed in single precision, see rays_kernel); the row's weights are single
// precision and accumulate in the same order as the reference's REAL(4) fdm
// (F:7722-7732), including its quirks:
// the segment clipped at the grid face is integrated with the full nominal
// step length (dinc from vrat*dpl), and the start-point B-spline weights of a
// sub-segment that follows a velocity-cell crossing keep the indices of the
// new cell (F:7647-7652, 7717-7732).
// Compiled without FMA contraction.
#include "internal.h"

namespace fm3dt {

// Single-precision Frechet weights: the row is accumulated in REAL(4), so its
// weights need no more; the FP64 pipe (a small fraction of FP32 throughput on
// this GPU) is kept for the ray path itself, whose end points must match.
__device__ __forceinline__ void bsplf(float u, float w[4])
{
    const float sixth = 1.0f / 6.0f;
    const float u2 = u * u, u3 = u * u * u;
    const float om = 1.0f - u;
    w[0] = om * om * om * sixth;
    w[1] = (4.0f - 6.0f * u2 + 3.0f * u3) * sixth;
    w[2] = (1.0f + 3.0f * u + 3.0f * u2 - 3.0f * u3) * sixth;
    w[3] = u3 * sixth;
}

__device__ __forceinline__ float vel_at(const Geom &g, const float *vel, int iz, int ix, int ir)
{
    return __ldg(vel + (size_t)(iz + 1) + (size_t)(g.nnz + 3) * ((size_t)(ix + 1) + (size_t)(g.nnx + 3) * (size_t)(ir + 1)));
}

// trilinear velocity at a point of propagation cell (ipz,ipx,ipr) (F:7629-7641),
// in single precision (it only weights the Frechet row; the velocity comes
// rounded to it, which saves its conversions on the double-precision pipe: eight
// a point); inr/inx/inz: reciprocals
// of the node spacings
__device__ float trilinf(const Geom &g, const float *velf, int ipz, int ipx, int ipr, float drr, float drx, float drz,
                         float dnr, float dnx, float dnz, float inr, float inx, float inz)
{
    float vel = 0.0f;
    for (int k = 1; k <= 2; ++k)
        for (int l = 1; l <= 2; ++l)
            for (int m = 1; m <= 2; ++m) {
                float produ = (1.0f - fabsf(((float)(m - 1) * dnz - drz) * inz));
                produ = produ * (1.0f - fabsf(((float)(l - 1) * dnx - drx) * inx));
                produ = produ * (1.0f - fabsf(((float)(k - 1) * dnr - drr) * inr));
                if (ipz - 1 + m <= g.nnz + 1 && ipx - 1 + l <= g.nnx + 1 && ipr - 1 + k <= g.nnr + 1)
                    vel = vel + vel_at(g, velf, ipz - 1 + m, ipx - 1 + l, ipr - 1 + k) * produ;
            }
    return vel;
}

constexpr int kRayBlock = 64;

// What a ray's arithmetic shares.  With the single-precision (offset) field the
// direction of each step -- gradient, its norm, sin(colatitude) -- is formed in
// single precision (G = float), and cells are located by multiplying with the
// spacings' reciprocals; positions, crossings and clipping stay in double.
// With the double-precision field everything is the reference's double
// arithmetic (G = double, divisions).
template <typename R>
struct RayGrid {
    static constexpr bool kFast = sizeof(R) == sizeof(float);
    const Geom &g;
    const float *velf;
    float fnr, fnx, fnz, inr, inx, inz;
    double inr_, inx_, inz_, ivr_, ivx_, ivz_;
    __device__ RayGrid(const RayArgs &a) : g(a.g), velf(a.velf)
    {
        fnr = (float)g.dnr; fnx = (float)g.dnx; fnz = (float)g.dnz;
        inr = 1.0f / fnr; inx = 1.0f / fnx; inz = 1.0f / fnz;
        inr_ = 1.0 / g.dnr; inx_ = 1.0 / g.dnx; inz_ = 1.0 / g.dnz;
        ivr_ = 1.0 / g.dvr; ivx_ = 1.0 / g.dvx; ivz_ = 1.0 / g.dvz;
    }
    // floor(x / d) + 1, in the double-precision form by the reciprocal i where
    // the product is clearly not next to a whole number (the quotient is at
    // most some thousands: the product is within 1e-11 of it)
    static __device__ __forceinline__ int cell(double x, double d, double i)
    {
        const double q = x * i;
        const int c = __double2int_rd(q);
        if (kFast) return c + 1;
        // (the fraction in [2^-30, 1 - 2^-20): by its high word)
        const unsigned f = (unsigned)__double2hiint(q - (double)c);
        if (f - 0x3e100000u < 0x3feffffeu - 0x3e100000u) return c + 1;
        return (int)floor(x / d) + 1;
    }
    __device__ __forceinline__ int cellr(double v) const { return cell(g.rgor - v, g.dnr, inr_); }
    __device__ __forceinline__ int cellx(double v) const { return cell(v - g.rgox, g.dnx, inx_); }
    __device__ __forceinline__ int cellz(double v) const { return cell(v - g.rgoz, g.dnz, inz_); }
    __device__ __forceinline__ int vcellr(double v) const { return cell(g.gor - v, g.dvr, ivr_); }
    __device__ __forceinline__ int vcellx(double v) const { return cell(v - g.gox, g.dvx, ivx_); }
    __device__ __forceinline__ int vcellz(double v) const { return cell(v - g.goz, g.dvz, ivz_); }

    // The cell a ray starts in (F:7320-7333), formed and checked in double
    // precision so that a non-finite or huge coordinate is rejected (false),
    // not converted.
    __device__ bool start(double r, double x, double z, int &ipr, int &ipx, int &ipz) const
    {
        double fpr = floor((g.rgor - r) / g.dnr) + 1.0;
        double fpx = floor((x - g.rgox) / g.dnx) + 1.0;
        double fpz = floor((z - g.rgoz) / g.dnz) + 1.0;
        if (fpr == (double)g.nnr) fpr -= 1.0;
        if (fpx == (double)g.nnx) fpx -= 1.0;
        if (fpz == (double)g.nnz) fpz -= 1.0;
        if (!(fpr >= 1.0 && fpr < (double)g.nnr && fpx >= 1.0 && fpx < (double)g.nnx && fpz >= 1.0 &&
              fpz < (double)g.nnz))
            return false;
        ipr = (int)fpr;
        ipx = (int)fpx;
        ipz = (int)fpz;
        return true;
    }

    // One step from (rgr, rgx, rgz) in cell (ipr, ipx, ipz) down the gradient
    // (F:7382-7541): the new point and its cell; true when the ray ends there,
    // clipped at the first face of the grid it crosses.
    __device__ __forceinline__ bool step(const R *Te, double rgr, double rgx, double rgz, int &ipr, int &ipx, int &ipz,
                                         double &nr, double &nx, double &nz) const
    {
        using G = R;
        const double dpl = g.dnr;        // F:7290
        const R *T0 = Te + ((size_t)(ipr - 1) * g.nnx + (ipx - 1)) * g.nnz + (ipz - 1);
        const size_t up = (size_t)g.nnx * g.nnz;
        // t<r><x><z>
        const G t000 = (G)T0[0], t001 = (G)T0[1], t010 = (G)T0[g.nnz], t011 = (G)T0[g.nnz + 1];
        const G t100 = (G)T0[up], t101 = (G)T0[up + 1], t110 = (G)T0[up + g.nnz], t111 = (G)T0[up + g.nnz + 1];
        G dtr = 0;
        int temp = 0;
        if (t100 < t000) { dtr = dtr + t100 - t000; temp++; }
        if (t101 < t001) { dtr = dtr + t101 - t001; temp++; }
        if (t111 < t011) { dtr = dtr + t111 - t011; temp++; }
        if (t110 < t010) { dtr = dtr + t110 - t010; temp++; }
        if (temp != 0) dtr = dtr / ((G)temp * (G)g.dnr);
        const G rcell = (G)(g.earth + g.rgor - (double)(ipr - 1) * g.dnr);
        G dtx = t010 - t000;
        dtx = dtx + t011 - t001;
        dtx = dtx + t111 - t101;
        dtx = dtx + t110 - t100;
        dtx = dtx / ((G)4 * rcell * (G)g.dnx);
        const G sx = sin((G)rgx);
        G dtz = t001 - t000;
        dtz = dtz + t111 - t110;
        dtz = dtz + t011 - t010;
        dtz = dtz + t101 - t100;
        dtz = dtz / ((G)4 * rcell * sx * (G)g.dnz);
        const G crad = (G)(g.earth + rgr);
        const G rd1 = sqrt(dtr * dtr + dtx * dtx + dtz * dtz);
        nr = rgr + (double)((G)dpl * dtr / rd1);
        nx = rgx - (double)((G)dpl * dtx / (crad * rd1));
        nz = rgz - (double)((G)dpl * dtz / (crad * sx * rd1));
        const int ipro = ipr, ipxo = ipx, ipzo = ipz;
        ipr = cellr(nr);
        ipx = cellx(nx);
        ipz = cellz(nz);
        const bool swr = (ipr < 1 || ipr >= g.nnr);
        const bool swx = (ipx < 1 || ipx >= g.nnx);
        const bool swz = (ipz < 1 || ipz >= g.nnz);
        if (!(swr || swx || swz)) return false;
        int sw = 0;
        double atio = 0.0;
        if (swr) {
            double ri;
            if (ipr < 1) { ri = g.rgor; ipr = 1; }
            else { ri = g.rgor - (double)(g.nnr - 1) * g.dnr; ipr = g.nnr - 1; }
            atio = (ri - rgr) / (nr - rgr);
            sw = 1;
        }
        if (swx) {
            double xi;
            if (ipx < 1) { xi = g.rgox; ipx = 1; }
            else { xi = g.rgox + (double)(g.nnx - 1) * g.dnx; ipx = g.nnx - 1; }
            const double r1 = (xi - rgx) / (nx - rgx);
            if (sw == 1) { if (r1 < atio) { atio = r1; sw = 2; } }
            else { atio = r1; sw = 2; }
        }
        if (swz) {
            double zi;
            if (ipz < 1) { zi = g.rgoz; ipz = 1; }
            else { zi = g.rgoz + (double)(g.nnz - 1) * g.dnz; ipz = g.nnz - 1; }
            const double r1 = (zi - rgz) / (nz - rgz);
            if (sw != 0) { if (r1 < atio) { atio = r1; sw = 3; } }
            else { atio = r1; sw = 3; }
        }
        if (sw == 1) { ipx = ipxo; ipz = ipzo; }
        else if (sw == 2) { ipr = ipro; ipz = ipzo; }
        else if (sw == 3) { ipr = ipro; ipx = ipxo; }
        nz = rgz + atio * (nz - rgz);
        nx = rgx + atio * (nx - rgx);
        nr = rgr + atio * (nr - rgr);
        return true;
    }

    // Where a step crosses into other velocity cells (F:7543-7620): the
    // crossings' fractions of the step in order (then 1), the axis of each
    // (1 r, 2 theta, 3 phi), and the number of sub-segments.
    __device__ __forceinline__ int crossings(double br, double bx, double bz, double nr, double nx, double nz, int ivro,
                                             int ivxo, int ivzo, int ivr, int ivx, int ivz, double (&vrat)[4],
                                             int (&chp)[4]) const
    {
        int nhp = 0;
        if (ivr != ivro) {
            const double ri = (ivr > ivro) ? g.gor - (double)(ivr - 1) * g.dvr : g.gor - (double)ivr * g.dvr;
            vrat[0] = (ri - br) / (nr - br);
            chp[0] = 1;
            nhp = 1;
        }
        if (ivx != ivxo) {
            const double xi = (ivx > ivxo) ? g.gox + (double)(ivx - 1) * g.dvx : g.gox + (double)ivx * g.dvx;
            const double r1 = (xi - bx) / (nx - bx);
            nhp++;
            if (nhp == 1) { vrat[0] = r1; chp[0] = 2; }
            else if (r1 >= vrat[0]) { vrat[1] = r1; chp[1] = 2; }
            else { vrat[1] = vrat[0]; chp[1] = chp[0]; vrat[0] = r1; chp[0] = 2; }
        }
        if (ivz != ivzo) {
            const double zi = (ivz > ivzo) ? g.goz + (double)(ivz - 1) * g.dvz : g.goz + (double)ivz * g.dvz;
            const double r1 = (zi - bz) / (nz - bz);
            nhp++;
            if (nhp == 1) { vrat[0] = r1; chp[0] = 3; }
            else if (nhp == 2) {
                if (r1 >= vrat[0]) { vrat[1] = r1; chp[1] = 3; }
                else { vrat[1] = vrat[0]; chp[1] = chp[0]; vrat[0] = r1; chp[0] = 3; }
            } else {
                if (r1 >= vrat[1]) { vrat[2] = r1; chp[2] = 3; }
                else if (r1 >= vrat[0]) { vrat[2] = vrat[1]; chp[2] = chp[1]; vrat[1] = r1; chp[1] = 3; }
                else { vrat[2] = vrat[1]; chp[2] = chp[1]; vrat[1] = vrat[0]; chp[1] = chp[0]; vrat[0] = r1; chp[0] = 3; }
            }
        }
        vrat[nhp] = 1.0;
        chp[nhp] = 0;
        return nhp + 1;
    }

    // The B-spline weights (r, theta, phi) of a point in a velocity cell, and
    // its 1/v^2, v trilinear in its propagation cell.
    __device__ __forceinline__ void point(double pr, double px, double pz, int cr, int cx, int cz, int vr, int vx, int vz,
                                          float *u, float *v, float *w, float &iv2) const
    {
        const double drr = (g.rgor - pr) - (double)(cr - 1) * g.dnr;
        const double drx = (px - g.rgox) - (double)(cx - 1) * g.dnx;
        const double drz = (pz - g.rgoz) - (double)(cz - 1) * g.dnz;
        const float vel = trilinf(g, velf, cz, cx, cr, (float)drr, (float)drx, (float)drz, fnr, fnx, fnz, inr, inx, inz);
        iv2 = 1.0f / (vel * vel);
        bsplf((float)(((g.gor - pr) - (double)(vr - 1) * g.dvr) * ivr_), u);
        bsplf((float)(((px - g.gox) - (double)(vx - 1) * g.dvx) * ivx_), v);
        bsplf((float)(((pz - g.goz) - (double)(vz - 1) * g.dvz) * ivz_), w);
    }
    __device__ __forceinline__ bool support(int vr, int vx, int vz) const
    {
        return !(vz - 1 < 0 || vz + 2 > g.nvz + 1 || vx - 1 < 0 || vx + 2 > g.nvx + 1 || vr - 1 < 0 || vr + 2 > g.nvr + 1);
    }
};

constexpr int kRayMaxSteps = 100000;        // F:7262

// Many rays: one thread a ray.  The velocity and weights at a step's start are
// those of the step before at its end where the two points are the same to
// the bit, which they nearly always are (the reference forms both), and so
// are its velocity cells: ~60 double-precision operations a step instead of
// ~120, the pipe that bounds it.
template <typename R>
__global__ void __launch_bounds__(kRayBlock) rays_kernel(RayArgs a)
{
    __shared__ float ray_acc[64 * kRayBlock];
    const RayGrid<R> rg(a);
    const Geom &g = rg.g;
    // the rays of a.nlist listed events (a.events), or of all a.nev events;
    // a ray's row, end point and flag index is its event's row e * nrc + i
    const int total = (a.events ? a.nlist : a.nev) * a.nrc;
    const size_t N = (size_t)g.nnx * g.nnz * g.nnr;
    const size_t nmp = (size_t)(g.nvr + 2) * (g.nvx + 2) * (g.nvz + 2);
    const double dpl = g.dnr;        // F:7290
    for (int qq = blockIdx.x * blockDim.x + threadIdx.x; qq < total; qq += gridDim.x * blockDim.x) {
        const int kk = qq / a.nrc, i = qq - kk * a.nrc;
        const int e = a.events ? a.events[kk] : kk;
        const int q = e * a.nrc + i;
        const R *Te = (const R *)a.T + (size_t)e * N;
        float *fdm = a.fdm ? a.fdm + nmp * (size_t)q : nullptr;
        // The row's sums for the velocity cell whose 4 x 4 x 4 B-spline
        // support the ray is in (one slot per support node, in shared memory,
        // this thread's slots strided by the block size so that a warp's
        // threads hit 32 different banks); added to the row when the ray
        // moves to another cell and at its end.  In the row each node's value
        // is the REAL(4) sum of its terms in ray order, grouped per cell visit.
        float *acc = ray_acc + threadIdx.x;
        int acc_r = -1, acc_x = -1, acc_z = -1;
        for (int t = 0; t < 64; ++t) acc[t * kRayBlock] = 0.0f;
        auto flush = [&]() {
            if (acc_r < 0) return;
            const size_t zstride = (size_t)(g.nvr + 2) * (size_t)(g.nvx + 2);
            // a row of four nodes (along phi) at a time: four independent
            // loads, then the four sums stored
#pragma unroll 1
            for (int nm = 0; nm < 16; ++nm) {
                const int n = nm >> 2, m = nm & 3;
                float *p = fdm + (size_t)(acc_r - 1 + n) +
                           (size_t)(g.nvr + 2) * ((size_t)(acc_x - 1 + m) + (size_t)(g.nvx + 2) * (size_t)(acc_z - 1));
                const float o0 = p[0], o1 = p[zstride], o2 = p[2 * zstride], o3 = p[3 * zstride];
                float *c = acc + (nm * 4) * kRayBlock;
                p[0] = c[0] + o0;
                p[zstride] = c[kRayBlock] + o1;
                p[2 * zstride] = c[2 * kRayBlock] + o2;
                p[3 * zstride] = c[3 * kRayBlock] + o3;
                c[0] = 0.0f;
                c[kRayBlock] = 0.0f;
                c[2 * kRayBlock] = 0.0f;
                c[3 * kRayBlock] = 0.0f;
            }
        };
        int st = 0;
        double rgr = a.rcr[i], rgx = a.rcx[i], rgz = a.rcz[i];
        int ipr = 0, ipx = 0, ipz = 0;
        const bool inside = rg.start(rgr, rgx, rgz, ipr, ipx, ipz);
        int steps = 0;
        if (!inside && a.flags) atomicMin(&a.flags[1], q);
        if (inside) {
            bool same = false;                           // (ui, vi, wi, iv2) hold the step's start
            int ivro = 0, ivxo = 0, ivzo = 0;
            if (fdm) {
                ivro = rg.vcellr(rgr);
                ivxo = rg.vcellx(rgx);
                ivzo = rg.vcellz(rgz);
            }
            float ui[4], vi[4], wi[4], iv2 = 0.0f;
            for (int jstep = 1; jstep <= kRayMaxSteps; ++jstep) {
                ++steps;
                const int ipro = ipr, ipxo = ipx, ipzo = ipz;
                double nr, nx, nz;
                const bool stop = rg.step(Te, rgr, rgx, rgz, ipr, ipx, ipz, nr, nx, nz);
                if (fdm) {
                    const int ivr = rg.vcellr(nr), ivx = rg.vcellx(nx), ivz = rg.vcellz(nz);
                    double vrat[4];
                    int chp[4];
                    const int nhp = rg.crossings(rgr, rgx, rgz, nr, nx, nz, ivro, ivxo, ivzo, ivr, ivx, ivz, vrat, chp);
                    if (!same) rg.point(rgr, rgx, rgz, ipro, ipxo, ipzo, ivro, ivxo, ivzo, ui, vi, wi, iv2);
                    same = rgr + (nr - rgr) == nr && rgx + (nx - rgx) == nx && rgz + (nz - rgz) == nz;
                    int ivrt = ivro, ivxt = ivxo, ivzt = ivzo;
                    for (int k = 0; k < nhp; ++k) {
                        const float iv2o = iv2;
                        float uio[4], vio[4], wio[4];
#pragma unroll
                        for (int m = 0; m < 4; ++m) { uio[m] = ui[m]; vio[m] = vi[m]; wio[m] = wi[m]; }
                        if (k > 0) {
                            if (chp[k - 1] == 1) ivrt = ivr;
                            else if (chp[k - 1] == 2) ivxt = ivx;
                            else if (chp[k - 1] == 3) ivzt = ivz;
                        }
                        const double rigz = rgz + vrat[k] * (nz - rgz);
                        const double rigx = rgx + vrat[k] * (nx - rgx);
                        const double rigr = rgr + vrat[k] * (nr - rgr);
                        rg.point(rigr, rigx, rigz, rg.cellr(rigr), rg.cellx(rigx), rg.cellz(rigz), ivrt, ivxt, ivzt, ui, vi,
                                 wi, iv2);
                        const double dinc = (k == 0) ? vrat[k] * dpl : (vrat[k] - vrat[k - 1]) * dpl;
                        const float hd = (float)(0.5 * dinc);
                        if (!rg.support(ivrt, ivxt, ivzt)) {
                            st = 1;
                            continue;
                        }
                        // a sub-segment in another support cell: the current
                        // cell's sums go to the row first
                        if (ivrt != acc_r || ivxt != acc_x || ivzt != acc_z) {
                            flush();
                            acc_r = ivrt; acc_x = ivxt; acc_z = ivzt;
                        }
#pragma unroll 1
                        for (int n = 0; n < 4; ++n)
#pragma unroll
                            for (int m = 0; m < 4; ++m) {
                                const float uv = ui[n] * vi[m] * iv2, uvo = uio[n] * vio[m] * iv2o;
#pragma unroll
                                for (int l = 0; l < 4; ++l) {
                                    const float a1 = -(uv * wi[l] + uvo * wio[l]) * hd;
                                    float &c = acc[((n * 4 + m) * 4 + l) * kRayBlock];
                                    c = a1 + c;
                                }
                            }
                    }
                    ivro = ivr; ivxo = ivx; ivzo = ivz;
                }
                rgr = nr; rgx = nx; rgz = nz;
                if (stop) break;
            }
        }
        if (fdm) flush();
        if (st && a.flags) atomicMin(&a.flags[0], q);
        if (a.endpoints) {
            a.endpoints[3 * (size_t)q] = rgr;
            a.endpoints[3 * (size_t)q + 1] = rgx;
            a.endpoints[3 * (size_t)q + 2] = rgz;
        }
        if (a.nsteps) a.nsteps[q] = steps;
    }
}

// Few rays: a warp traces RPW of them, lane i the path of ray i, STEPS steps at
// a time; then the whole warp works off those steps' Frechet terms.  The path
// is a serial chain (eight loads of the field, a direction, the next cell),
// so nothing else stays on it: its positions go to shared memory, and the
// terms' work -- crossings, velocities, weights, mostly double precision and
// loads -- is done by one lane a step, 32 steps at once.  Only the sums are in
// ray order again: 64 support nodes, two a lane.  A thread doing all of it in
// turn took ~14 us a step (2,400 rays on 256^3: 5.0 ms, now 1.1; in double
// precision 2,400 on 96x112x112 3.1 ms, now 1.4), a warp being given one
// double-precision operation in 64 cycles, whether 1 or 32 lanes need it --
// which is why many rays are traced one a lane (rays_kernel).
template <int RPW>
struct RayShape {
    static constexpr int STEPS = 128 / RPW;      // steps of a ray at a time
    static constexpr int ITEMS = STEPS * RPW;
    // points (12 weights and 1/v^2: 13 words, odd, no bank conflicts) that 32
    // steps may have; with more crossings than that, 16 steps at once
    static constexpr int POOL = 96;
};

template <typename R, int RPW>
__global__ void __launch_bounds__(32) rays_shared_kernel(RayArgs a)
{
    using S = RayShape<RPW>;
    constexpr int STEPS = S::STEPS, ITEMS = S::ITEMS;
    __shared__ double s_pos[3][(STEPS + 1) * RPW];       // step-major: a ray's start and its steps' ends
    __shared__ long long s_ip[STEPS * RPW];              // the cell each step starts in
    __shared__ int s_steps[RPW];                         // steps taken
    __shared__ float s_acc[RPW][64];
    __shared__ long long s_cur[RPW];                     // the velocity cell the sums belong to (-1: none)
    __shared__ float s_last[RPW][13];                    // the end point of a ray's last step
    __shared__ long long s_lv[RPW];                      // ... its velocity cell (-1: no step yet)
    __shared__ bool s_lsame[RPW];                        // ... whether it is the step's end to the bit
    __shared__ float s_w[S::POOL][13], s_hd[S::POOL];    // points; half length of the sub-segment that ends there
    __shared__ long long s_vc[S::POOL];                  // ... and its velocity cell (-1: support outside)
    __shared__ int s_n[32], s_first[32];                 // sub-segments of a step, its first point | its start is a point
    const RayGrid<R> rg(a);
    const Geom &g = rg.g;
    const int lane = threadIdx.x;
    const int total = (a.events ? a.nlist : a.nev) * a.nrc;
    const size_t N = (size_t)g.nnx * g.nnz * g.nnr;
    const size_t nmp = (size_t)(g.nvr + 2) * (g.nvx + 2) * (g.nvz + 2);
    const double dpl = g.dnr;        // F:7290
    // three cell indices in a word (21 bits each, so that none below zero --
    // outside the velocity grid -- makes the word negative)
    constexpr int kMask = (1 << 21) - 1, kBias = 1 << 20;
    auto pack = [](int r, int x, int z) -> long long {
        return ((long long)((r + kBias) & kMask) << 42) | ((long long)((x + kBias) & kMask) << 21) | ((z + kBias) & kMask);
    };
    auto unpack = [](long long v, int &r, int &x, int &z) {
        r = (int)(v >> 42) - kBias;
        x = ((int)(v >> 21) & kMask) - kBias;
        z = ((int)v & kMask) - kBias;
    };
    const bool rows = a.fdm != nullptr;

    // this lane's ray
    const int qq = blockIdx.x * RPW + lane;
    const bool mine = lane < RPW && qq < total;
    const int kk = mine ? qq / a.nrc : 0, i = mine ? qq - kk * a.nrc : 0;
    const int e = a.events ? a.events[kk] : kk;
    const int q = e * a.nrc + i;
    const R *Te = (const R *)a.T + (size_t)e * N;
    double rgr = 0.0, rgx = 0.0, rgz = 0.0;
    bool live = false;
    int ipr = 0, ipx = 0, ipz = 0, steps = 0;
    if (mine) {
        rgr = a.rcr[i];
        rgx = a.rcx[i];
        rgz = a.rcz[i];
        live = rg.start(rgr, rgx, rgz, ipr, ipx, ipz);
        if (!live && a.flags) atomicMin(&a.flags[1], q);
    }
    if (rows) {
        for (int t = lane; t < 64 * RPW; t += 32) (&s_acc[0][0])[t] = 0.0f;
        for (int t = lane; t < RPW; t += 32) s_cur[t] = s_lv[t] = -1;
    }
    unsigned outside = 0;                                // rays whose support left the velocity grid
    // a ray's sums, two a lane, into its row (the REAL(4) sum of its terms in
    // ray order, grouped per visit of a velocity cell): node (n, m, l) of the
    // 4 x 4 x 4 support is slot (n * 4 + m) * 4 + l
    auto flush = [&](float *row, long long cur, float &c0, float &c1) {
        if (cur < 0) return;
        int vr, vx, vz;
        unpack(cur, vr, vx, vz);
        float *p0 = row + (size_t)(vr - 1 + (lane >> 4)) +
                    (size_t)(g.nvr + 2) * ((size_t)(vx - 1 + ((lane >> 2) & 3)) + (size_t)(g.nvx + 2) * (size_t)(vz - 1 + (lane & 3)));
        const float o0 = p0[0], o1 = p0[2];
        p0[0] = c0 + o0;
        p0[2] = c1 + o1;
        c0 = c1 = 0.0f;
        __syncwarp();
    };
    while (__any_sync(0xffffffffu, live)) {
        // the path
        int n = 0;
        if (rows && lane < RPW) {
            s_pos[0][lane] = rgr;
            s_pos[1][lane] = rgx;
            s_pos[2][lane] = rgz;
        }
        for (int j = 0; j < STEPS && live; ++j) {
            ++steps;
            if (rows) s_ip[j * RPW + lane] = pack(ipr, ipx, ipz);
            double nr, nx, nz;
            live = !rg.step(Te, rgr, rgx, rgz, ipr, ipx, ipz, nr, nx, nz) && steps < kRayMaxSteps;
            rgr = nr; rgx = nx; rgz = nz;
            n = j + 1;
            if (rows) {
                s_pos[0][n * RPW + lane] = rgr;
                s_pos[1][n * RPW + lane] = rgx;
                s_pos[2][n * RPW + lane] = rgz;
            }
        }
        if (!rows) continue;
        if (lane < RPW) s_steps[lane] = n;
        __syncwarp();
        // the terms, 32 steps at a time, ray by ray
        long long cur = -1;
        float c0 = 0.0f, c1 = 0.0f, uv0 = 0.0f, uv1 = 0.0f, z = 0.0f;
        const int n0 = lane >> 4, m = 4 + ((lane >> 2) & 3), l = 8 + (lane & 3);
        auto take = [&](const float *w) {
            const float v = w[m], iv2 = w[12];
            uv0 = w[n0] * v * iv2;
            uv1 = w[n0 + 2] * v * iv2;
            z = w[l];
        };
        for (int base = 0; base < ITEMS; base += 32) {
            // one lane a step: where it crosses into other velocity cells
            const int ray = (base + lane) / STEPS, st = (base + lane) % STEPS, at = st * RPW + ray;
            int nhp = 0;
            bool own_start = false;                      // its start is a point of its own
            double br = 0.0, bx = 0.0, bz = 0.0, nr = 0.0, nx = 0.0, nz = 0.0, vrat[4];
            int ivr = 0, ivx = 0, ivz = 0, ivro = 0, ivxo = 0, ivzo = 0, chp[4];
            bool same = false;                           // its last point is its end, to the bit
            if (st < s_steps[ray]) {
                br = s_pos[0][at]; bx = s_pos[1][at]; bz = s_pos[2][at];
                nr = s_pos[0][at + RPW]; nx = s_pos[1][at + RPW]; nz = s_pos[2][at + RPW];
                ivr = rg.vcellr(nr); ivx = rg.vcellx(nx); ivz = rg.vcellz(nz);
                same = br + (nr - br) == nr && bx + (nx - bx) == nx && bz + (nz - bz) == nz;
            }
            // the start's cells and point: those of the step before (of an
            // earlier lane, or kept from the last steps taken)
            {
                const unsigned prev = 0xffffffffu;
                ivro = __shfl_up_sync(prev, ivr, 1);
                ivxo = __shfl_up_sync(prev, ivx, 1);
                ivzo = __shfl_up_sync(prev, ivz, 1);
                bool psame = __shfl_up_sync(prev, same ? 1 : 0, 1);
                if (lane == 0 || st == 0) {
                    // (s_lv: -1 before a ray's first step)
                    const long long v = s_lv[ray];
                    unpack(v, ivro, ivxo, ivzo);
                    psame = v >= 0 && s_lsame[ray];
                    if (st < s_steps[ray] && v < 0) {
                        ivro = rg.vcellr(br); ivxo = rg.vcellx(bx); ivzo = rg.vcellz(bz);
                    }
                }
                own_start = !psame;
            }
            if (st < s_steps[ray])
                nhp = rg.crossings(br, bx, bz, nr, nx, nz, ivro, ivxo, ivzo, ivr, ivx, ivz, vrat, chp);
            __syncwarp();
            if (nhp && (lane == 31 || st + 1 == s_steps[ray])) {
                s_lv[ray] = pack(ivr, ivx, ivz);
                s_lsame[ray] = same;
            }
            // points of the pool: this lane's first, and how many in all
            const int need = nhp ? nhp + (own_start ? 1 : 0) : 0;
            int off = need;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, off, o);
                if (lane >= o) off += y;
            }
            const int all = __shfl_sync(0xffffffffu, off, 31), half = __shfl_sync(0xffffffffu, off, 15);
            off -= need;
            const int parts = all <= S::POOL ? 1 : 2;
            for (int part = 0; part < parts; ++part) {
                const int j0 = part * 16, j1 = parts == 1 ? 32 : j0 + 16;
                if (lane >= j0 && lane < j1) {
                    const int f0 = part ? off - half : off;
                    s_n[lane] = nhp;
                    s_first[lane] = f0 * 2 + (own_start ? 1 : 0);
                    auto point = [&](int k, double pr, double px, double pz, int cr, int cx, int cz, int vr, int vx, int vz) {
                        float *w = s_w[k];
                        rg.point(pr, px, pz, cr, cx, cz, vr, vx, vz, w, w + 4, w + 8, w[12]);
                    };
                    int slot = f0;
                    if (nhp && own_start) {
                        int cr, cx, cz;
                        unpack(s_ip[at], cr, cx, cz);
                        point(slot++, br, bx, bz, cr, cx, cz, ivro, ivxo, ivzo);
                    }
                    int ivrt = ivro, ivxt = ivxo, ivzt = ivzo;
                    for (int k = 0; k < nhp; ++k) {
                        if (k > 0) {
                            if (chp[k - 1] == 1) ivrt = ivr;
                            else if (chp[k - 1] == 2) ivxt = ivx;
                            else if (chp[k - 1] == 3) ivzt = ivz;
                        }
                        double rigz = nz, rigx = nx, rigr = nr;
                        if (k < nhp - 1 || !same) {
                            rigz = bz + vrat[k] * (nz - bz);
                            rigx = bx + vrat[k] * (nx - bx);
                            rigr = br + vrat[k] * (nr - br);
                        }
                        point(slot, rigr, rigx, rigz, rg.cellr(rigr), rg.cellx(rigx), rg.cellz(rigz), ivrt, ivxt, ivzt);
                        const double dinc = (k == 0) ? vrat[k] * dpl : (vrat[k] - vrat[k - 1]) * dpl;
                        s_hd[slot] = (float)(0.5 * dinc);
                        s_vc[slot++] = rg.support(ivrt, ivxt, ivzt) ? pack(ivrt, ivxt, ivzt) : -1;
                    }
                }
                __syncwarp();
                // the sums, in order
                for (int j = j0; j < j1; ++j) {
                    const int jr = (base + j) / STEPS;
                    if ((base + j) % STEPS == 0) {
                        c0 = s_acc[jr][lane];
                        c1 = s_acc[jr][lane + 32];
                        cur = s_cur[jr];
                        take(s_last[jr]);
                    }
                    const int jn = s_n[j];
                    if (jn) {
                        int slot = s_first[j] >> 1;
                        if (s_first[j] & 1) take(s_w[slot++]);
                        for (int k = 0; k < jn; ++k, ++slot) {
                            const float uvo0 = uv0, uvo1 = uv1, zo = z;
                            take(s_w[slot]);
                            const long long vc = s_vc[slot];
                            if (vc < 0) {
                                outside |= 1u << jr;
                                continue;
                            }
                            // a sub-segment in another support cell: the
                            // current cell's sums go to the row first
                            if (vc != cur) {
                                const int rq = __shfl_sync(0xffffffffu, q, jr);
                                flush(a.fdm + nmp * (size_t)rq, cur, c0, c1);
                                cur = vc;
                            }
                            const float hd = s_hd[slot];
                            c0 = -(uv0 * z + uvo0 * zo) * hd + c0;
                            c1 = -(uv1 * z + uvo1 * zo) * hd + c1;
                        }
                        // (the ray's last point so far)
                        if ((base + j) % STEPS == STEPS - 1 && lane < 13) s_last[jr][lane] = s_w[slot - 1][lane];
                    }
                    if ((base + j) % STEPS == STEPS - 1) {
                        s_acc[jr][lane] = c0;
                        s_acc[jr][lane + 32] = c1;
                        if (lane == 0) s_cur[jr] = cur;
                    }
                }
                __syncwarp();
            }
        }
    }
    if (rows) {
        for (int ray = 0; ray < RPW; ++ray) {
            float c0 = s_acc[ray][lane], c1 = s_acc[ray][lane + 32];
            const int rq = __shfl_sync(0xffffffffu, q, ray);
            flush(a.fdm + nmp * (size_t)rq, s_cur[ray], c0, c1);
        }
    }
    if (!mine) return;
    if (((outside >> lane) & 1u) && a.flags) atomicMin(&a.flags[0], q);
    if (a.endpoints) {
        a.endpoints[3 * (size_t)q] = rgr;
        a.endpoints[3 * (size_t)q + 1] = rgx;
        a.endpoints[3 * (size_t)q + 2] = rgz;
    }
    if (a.nsteps) a.nsteps[q] = steps;
}

// Rows: count and compact entries with |f| >= 1e-6 (F:7739-7765).  One block
// per row; the block scans the row in column order, V consecutive columns per
// thread (V = 4: 16-byte loads, when the row length keeps every row 16-byte
// aligned), so that enough loads are in flight to stream the dense rows at
// HBM speed.
template <int V>
struct RowVec;
template <>
struct RowVec<1> {
    static __device__ __forceinline__ void load(const float *p, float (&v)[1]) { v[0] = __ldcs(p); }
};
template <>
struct RowVec<4> {
    static __device__ __forceinline__ void load(const float *p, float (&v)[4])
    {
        const float4 x = __ldcs(reinterpret_cast<const float4 *>(p));
        v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    }
};

template <int V>
__global__ void row_counts_kernel(const float *__restrict__ fdm, int nrows, int nmp, int64_t *__restrict__ counts)
{
    const float ftol = 1.0e-6f;
    __shared__ int red[2][32];
    const int nv = nmp / V;                      // whole vectors (nmp % V == 0)
    int it = 0;
    for (int row = blockIdx.x; row < nrows; row += gridDim.x, it ^= 1) {
        const float *f = fdm + (size_t)row * nmp;
        int c = 0;
#pragma unroll 2
        for (int q = threadIdx.x; q < nv; q += blockDim.x) {
            float v[V];
            RowVec<V>::load(f + (size_t)q * V, v);
#pragma unroll
            for (int j = 0; j < V; ++j) c += fabsf(v[j]) >= ftol ? 1 : 0;
        }
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        // (two buffers: a row's sums are not overwritten by the next row's
        // before thread 0 has read them)
        if ((threadIdx.x & 31) == 0) red[it][threadIdx.x >> 5] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            int sum = 0;
            for (int w = 0; w < (int)(blockDim.x + 31) / 32; ++w) sum += red[it][w];
            counts[row] = sum;
        }
    }
}

template <int V>
__global__ void row_compact_kernel(const float *__restrict__ fdm, int nrows, int nmp,
                                   const int64_t *__restrict__ row_ptr, int32_t *__restrict__ cols,
                                   float *__restrict__ vals)
{
    const float ftol = 1.0e-6f;
    __shared__ int wsum[2][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    const int nv = nmp / V;
    int it = 0;
    for (int row = blockIdx.x; row < nrows; row += gridDim.x) {
        const float *f = fdm + (size_t)row * nmp;
        int64_t base = row_ptr[row];
        for (int c0 = 0; c0 < nv; c0 += blockDim.x, it ^= 1) {
            const int q = c0 + threadIdx.x;
            float v[V];
            int k = 0;
            if (q < nv) {
                RowVec<V>::load(f + (size_t)q * V, v);
#pragma unroll
                for (int j = 0; j < V; ++j) k += fabsf(v[j]) >= ftol ? 1 : 0;
            }
            // the thread's first slot: the kept entries of the lower threads
            // of its warp, then of the lower warps
            int incl = k;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) wsum[it][wid] = incl;
            __syncthreads();
            int before = 0, total = 0;
            for (int w = 0; w < nw; ++w) {
                const int x = wsum[it][w];
                before += w < wid ? x : 0;
                total += x;
            }
            if (k > 0) {
                int64_t pos = base + before + incl - k;
#pragma unroll
                for (int j = 0; j < V; ++j)
                    if (fabsf(v[j]) >= ftol) {
                        cols[pos] = q * V + j + 1;
                        vals[pos] = v[j];
                        ++pos;
                    }
            }
            base += total;
            // (the next chunk writes the other wsum buffer; the one after it
            // this buffer again, after the next chunk's barrier, which every
            // thread reaches only after reading this one)
        }
    }
}

// Row pointers from row counts: row_ptr[0] = 0, row_ptr[i+1] = row_ptr[i] +
// counts[i].  Each block scans a chunk of kScanChunk rows and writes its total;
// one block then turns the totals into chunk offsets in order (any number of
// chunks, with a running carry) and the chunks add their offset.
constexpr int kScanThreads = 1024;
constexpr int kScanChunk = kScanThreads;

__device__ int64_t block_exclusive_scan(int64_t v, int64_t *total)
{
    __shared__ int64_t warp_sums[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int64_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
        const int nw = blockDim.x >> 5;
        int64_t w = lane < nw ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) warp_sums[lane] = w;
    }
    __syncthreads();
    const int64_t before = (wid > 0 ? warp_sums[wid - 1] : 0) + x - v;
    *total = warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
    return before;
}

__global__ void __launch_bounds__(kScanThreads) scan_chunks_kernel(const int64_t *__restrict__ counts, int n,
                                                                   int64_t *__restrict__ row_ptr,
                                                                   int64_t *__restrict__ chunk_tot)
{
    const int i = blockIdx.x * kScanChunk + threadIdx.x;
    const int64_t v = i < n ? counts[i] : 0;
    int64_t tot;
    const int64_t ex = block_exclusive_scan(v, &tot);
    if (i < n) row_ptr[i + 1] = ex + v;          // inclusive within the chunk
    if (threadIdx.x == 0) chunk_tot[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kScanThreads) scan_totals_kernel(int64_t *__restrict__ chunk_tot, int nchunks)
{
    __shared__ int64_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int c0 = 0; c0 < nchunks; c0 += kScanThreads) {
        const int c = c0 + threadIdx.x;
        const int64_t v = c < nchunks ? chunk_tot[c] : 0;
        int64_t tot;
        const int64_t ex = block_exclusive_scan(v, &tot);
        if (c < nchunks) chunk_tot[c] = carry + ex;  // offset of chunk c
        __syncthreads();
        if (threadIdx.x == 0) carry += tot;
        __syncthreads();
    }
}

__global__ void scan_add_kernel(int n, int64_t *__restrict__ row_ptr, const int64_t *__restrict__ chunk_off)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) row_ptr[0] = 0;
    if (i < n) row_ptr[i + 1] += chunk_off[i / kScanChunk];
}

int scan_chunks(int nrows) { return (nrows + kScanChunk - 1) / kScanChunk; }

void launch_row_scan(const int64_t *counts, int nrows, int64_t *row_ptr, int64_t *chunk_tmp, cudaStream_t st)
{
    if (nrows <= 0) return;
    const int nc = scan_chunks(nrows);
    scan_chunks_kernel<<<nc, kScanThreads, 0, st>>>(counts, nrows, row_ptr, chunk_tmp);
    scan_totals_kernel<<<1, kScanThreads, 0, st>>>(chunk_tmp, nc);
    scan_add_kernel<<<(nrows + 255) / 256, 256, 0, st>>>(nrows, row_ptr, chunk_tmp);
}

// Which kernel, by the number of rays (rays of 135 / 100 steps, in ms, with 2
// and 8 rays a warp and one a thread):
//   single precision  2,400: 0.61 1.10 1.98   9,600: 1.72 1.29 2.09   38,400: 6.35 3.55 2.94
//   double precision  2,400: 1.45 1.38 2.14   9,600: 5.78 2.03 2.36   19,200: 10.8 4.36 2.61
template <typename R>
static void launch_rays_of(const RayArgs &a, int total, cudaStream_t st)
{
    const bool fast = sizeof(R) == sizeof(float);
    if (total <= (fast ? 6000 : 1800))
        rays_shared_kernel<R, 2><<<(total + 1) / 2, 32, 0, st>>>(a);
    else if (total <= (fast ? 25000 : 12000))
        rays_shared_kernel<R, 8><<<(total + 7) / 8, 32, 0, st>>>(a);
    else
        rays_kernel<R><<<(total + kRayBlock - 1) / kRayBlock, kRayBlock, 0, st>>>(a);
}

void launch_rays(const RayArgs &a, cudaStream_t st)
{
    const int total = (a.events ? a.nlist : a.nev) * a.nrc;
    if (total <= 0) return;
    if (a.prec == FM3DT_FP64)
        launch_rays_of<double>(a, total, st);
    else
        launch_rays_of<float>(a, total, st);
}

void launch_row_counts(const float *fdm, int nrows, int nmp, int64_t *counts, cudaStream_t st)
{
    if (nrows <= 0) return;
    const int grid = nrows < 152 * 16 ? nrows : 152 * 16;
    if (nmp % 4 == 0)
        row_counts_kernel<4><<<grid, 256, 0, st>>>(fdm, nrows, nmp, counts);
    else
        row_counts_kernel<1><<<grid, 256, 0, st>>>(fdm, nrows, nmp, counts);
}

void launch_row_compact(const float *fdm, int nrows, int nmp, const int64_t *row_ptr, int32_t *cols, float *vals,
                        cudaStream_t st)
{
    if (nrows <= 0) return;
    const int grid = nrows < 152 * 16 ? nrows : 152 * 16;
    if (nmp % 4 == 0)
        row_compact_kernel<4><<<grid, 256, 0, st>>>(fdm, nrows, nmp, row_ptr, cols, vals);
    else
        row_compact_kernel<1><<<grid, 256, 0, st>>>(fdm, nrows, nmp, row_ptr, cols, vals);
}

}  // namespace fm3dt
