// front.cuh -- the main sweep of a solve: every event once, upward from its
// boundary frame and along its lateral directions, in one launch.
//
// One warp owns a block of SX x SZ (theta, phi) columns over the whole height.
// At step t lane (x', z') (swept coordinates) computes the node of layer
// t - x' - z' (counted from the bottom) by fm_update_upstream.  The field is
// unset before this sweep, so only the three upstream neighbours matter, and
// all six values of a node are at hand in the warp:
//   down    the lane's own last two values (registers);
//   theta   lane x'-1's last value (one shuffle), and behind it the value that
//           lane used for the same layer one step before (one shuffle);
//   phi     the same from lane z'-1;
//   lanes at x' = 0 or z' = 0 take the two columns of the block upstream.
// A layer's slowness, halo columns and spacings are copied (cp.async)
// four steps ahead, coalesced, by the whole warp, into shared-memory rings
// from which lanes use them up to SX + SZ - 2 steps later; values leave
// through such a ring as well, a layer at a time.  (Loaded and stored by the
// lanes themselves, a step's 32 nodes lie in 32 different sectors; prefetched
// through registers, each step's register moves wait for the load of the
// step before: 408 us for one 64^3 event.)
//
// Blocks wait for each other by the data: the field is filled with ones
// (a NaN no update gives) before the launch, every node is written once, and
// a halo load that still reads ones is repeated.  No flag, no fence, and a
// block follows the ones upstream at a distance of a dozen layers, so the
// critical path is nnr + ~14 (blocks along theta + phi) steps, not that many
// times the height.  Warps take blocks from a counter, a group of events at a
// time and hyperplane by hyperplane in a group, so the blocks a block waits
// for were taken before it by warps that run: every wait ends (and is bounded
// all the same).  One block per warp and CTA: a launch of higher priority gets
// its slots as blocks end.
//
// SKEW: a halo column's value for layer r is read by the step that uses it
// first (r + z' or r + x', not r), and every value is stored when computed, so a
// block trails the one before it along theta by 3 steps and along phi by 7
// (and an L2 round trip) instead of 10; but a step's loads and stores then
// touch up to 56 sectors one by one instead of 14.  For solves whose blocks are all
// resident at once, which the critical path bounds: one 64^3 event 189 us
// against 228; eight 256^3 events 2.41 ms against 1.69 without it.
//
// What bounds it: instruction issue when there are events enough to fill the
// SMs (84% of the issue slots; 9.5 warp instructions a node with 128 layers, 9.8
// with 96), else the step's latency (~0.5 us) along the critical path.  Against one launch per
// hyperplane of blocks in height segments, with rings of whole layers and
// their halos: 500 events on 192x224x224 77.8 -> 42.4 ms, 256 on 128^3 10.3 ->
// 5.5 ms, eight on 256^3 4.26 -> 1.67 ms, one on 64^3 0.52 -> 0.19 ms; in double
// precision 32 events on 128^3 30.5 -> 9.0 ms, one on 64^3 3.4 -> 0.89 ms (both with
// the screened update).
#pragma once
#include "halo_layers.h"
#include "stream.cuh"

namespace fm3dt {

// A halo value not yet written: sign bit set (no time has it) -- all ones, or
// the start value of a boundary node without a time (holes_kernel).
__device__ __forceinline__ bool front_unwritten(float v) { return __float_as_int(v) < 0; }
__device__ __forceinline__ bool front_unwritten(double v) { return __double2hiint(v) < 0; }
// such a node's start value (NaN of all ones: none)
__device__ __forceinline__ float front_value(float v) { return fabsf(v); }
__device__ __forceinline__ double front_value(double v) { return fabs(v); }
// (from L2: the writer is another SM)
__device__ __forceinline__ float front_load(const float *p)
{
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];\n" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double front_load(const double *p)
{
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];\n" : "=d"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void front_store(float *p, float v)
{
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;\n" ::"l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void front_store(double *p, double v)
{
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;\n" ::"l"(p), "d"(v) : "memory");
}

template <typename R, int SX, int SZ, bool SKEW>
__global__ void __launch_bounds__(32) front_kernel(FrontArgs<R> a)
{
    static_assert(SX * SZ == 32, "one warp per column block");
    constexpr int LAG = SX + SZ - 2;               // steps from a layer's first node to its last
    constexpr int AHEAD = 4;                       // steps a layer's copies are issued ahead
    // layers t - LAG .. t + AHEAD, and one more: a lane may be a step ahead
    constexpr int RING = LAG + AHEAD + 2 <= 16 ? 16 : 32;
    constexpr int NH = 2 * SZ + 4 * SX;            // halo columns (theta, phi), then hz and wz of the block's rows
    constexpr int PER = (NH + 31) / 32;
    __shared__ R s_slow[RING][32], s_out[SKEW ? 1 : RING][32], s_halo[RING][NH];
    const FieldArgs<R> &f = a.f;
    const R INF = Lim<R>::inf();
    const int lane = threadIdx.x;
    const int xs = lane / SZ, zs = lane % SZ;
    unsigned item = 0;
    if (lane == 0) item = atomicAdd(a.next, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= a.count) return;
    // group of events, block in it (hyperplane order), event
    const unsigned gsize = (unsigned)a.nblocks * (unsigned)a.group;
    const int k0 = (int)(item / gsize) * a.group;
    const unsigned rem = item % gsize;
    const unsigned ge = (unsigned)min(a.group, a.nev - k0);
    const int packed = a.blocks[rem / ge];
    const int k = k0 + (int)(rem % ge);
    const int e = a.events ? a.events[k] : k;
    const int dir = a.dir[e];
    const bool sx = dir & 1, sz = (dir >> 1) & 1;
    const int bxp = (packed >> 12) & 0xfff, bzp = packed & 0xfff;
    const int x0 = (sx ? bxp : a.nbx - 1 - bxp) * SX, z0 = (sz ? bzp : a.nbz - 1 - bzp) * SZ;
    const int gx = sx ? x0 + xs : x0 + SX - 1 - xs, gz = sz ? z0 + zs : z0 + SZ - 1 - zs;
    const bool colv = gx < f.nnx && gz < f.nnz;
    const size_t layer = (size_t)f.nnx * f.nnz;
    const int nnr = f.nnr;
    R *Tb = f.T + (size_t)e * layer * nnr + (size_t)(nnr - 1) * layer;      // bottom layer
    const size_t own = colv ? (size_t)gx * f.nnz + gz : 0;
    // this lane's share of the halo and spacings of a layer: where it is in
    // the bottom layer, its step from layer to layer; unset outside the grid
    const R *hp[PER];
    long long hstep[PER];
    bool hfield[PER], hok[PER];
    int hlate[PER];                                 // steps this column is read behind layer t (SKEW)
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        int q = lane + 32 * j, hx = 0, hz = 0;
        hfield[j] = q < 2 * SZ + 2 * SX;
        if (q < 2 * SZ) {
            const int d = q / SZ, i = q % SZ;
            hx = sx ? x0 - 1 - d : x0 + SX + d;
            hz = sz ? z0 + i : z0 + SZ - 1 - i;
        } else if (hfield[j]) {
            const int d = (q - 2 * SZ) / SX, i = (q - 2 * SZ) % SX;
            hx = sx ? x0 + i : x0 + SX - 1 - i;
            hz = sz ? z0 - 1 - d : z0 + SZ + d;
        } else {
            const int i = (q - 2 * SZ - 2 * SX) % SX;
            hx = sx ? x0 + i : x0 + SX - 1 - i;
        }
        hlate[j] = !SKEW || !hfield[j] ? 0 : (q < 2 * SZ ? q % SZ : (q - 2 * SZ) % SX);
        hok[j] = q < NH && hx >= 0 && hx < f.nnx && hz >= 0 && hz < f.nnz;
        if (hfield[j]) {
            hstep[j] = (long long)layer;
            hp[j] = Tb + (hok[j] ? (long long)hx * f.nnz + hz : 0) + hlate[j] * hstep[j];
        } else {
            hp[j] = (q < 2 * SZ + 3 * SX ? f.hz : f.wz) + (size_t)(nnr - 1) * f.nnx + (hok[j] ? hx : 0);
            hstep[j] = f.nnx;
        }
    }
    const R *sp = f.s + (size_t)(nnr - 1) * layer + own;
    R *op = Tb + own;
    const bool fixed0 = colv && f.frozen[(size_t)e * layer + own] != 0;
    // (a boundary node without a time holds its start value, marked unwritten)
    const R bottom = colv ? front_value(*op) : INF;
    // neighbours inside the grid (the sweep's upstream and downstream sides)
    const bool xlo = gx > 0, xhi = gx < f.nnx - 1, zlo = gz > 0, zhi = gz < f.nnz - 1;
    const bool inXu = sx ? xlo : xhi, inXd = sx ? xhi : xlo, inZu = sz ? zlo : zhi, inZd = sz ? zhi : zlo;
    // (unset halo columns, and what lies below the grid, stay so)
    for (int row = 0; row < RING; ++row)
#pragma unroll
        for (int j = 0; j < PER; ++j)
            if (lane + 32 * j < NH) s_halo[row][lane + 32 * j] = INF;
    // the copies that step t uses first
    auto fetch = [&](int t) {
        const int row = t & (RING - 1);
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            if (hok[j] && halo_layer_in(t, hlate[j], nnr))
                cp_async_elem(&s_halo[row][lane + 32 * j], hp[j]);
            hp[j] -= hstep[j];
        }
        if (colv && t < nnr) cp_async_elem(&s_slow[row][lane], sp);
        sp -= layer;
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
#pragma unroll
    for (int t = 0; t < AHEAD; ++t) fetch(t);
    R v1 = INF, v2 = INF, Xp = INF, Zp = INF;      // own last two values; neighbours' values used last
    Spacing<R> spc;
    spc.h[0] = f.hr;
    spc.w[0] = f.wr;
    const R *hxp = f.hx + (nnr - 1), *wxp = f.wx + (nnr - 1);
    const int delay = xs + zs;
    R hxn = __ldg(hxp), wxn = __ldg(wxp);
    const int steps = nnr + LAG;
    for (int t = 0; t < steps; ++t) {
        // step t + AHEAD's copies on their way; step t's are here, or not yet
        // written (a copy may also have hit an older line in L1): then polled
        // in L2
        fetch(t + AHEAD);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(AHEAD) : "memory");
        {
            R *halo = s_halo[t & (RING - 1)];
            unsigned polls = 0;
            for (;;) {
                bool wait = false;
#pragma unroll
                for (int j = 0; j < PER; ++j)
                    wait = wait || (hok[j] && hfield[j] && front_unwritten(halo[lane + 32 * j]));
                if (!__any_sync(0xffffffffu, wait)) break;
                if (wait_gives_up(++polls, a.err)) {
                    // (none is left in the ring: rows of layers above the
                    // grid are not copied anew, and a value unwritten there
                    // would be polled before the field)
#pragma unroll
                    for (int j = 0; j < PER; ++j)
                        if (hok[j] && hfield[j] && front_unwritten(halo[lane + 32 * j])) halo[lane + 32 * j] = INF;
                    break;
                }
                // (hp stands AHEAD + 1 layers above)
#pragma unroll
                for (int j = 0; j < PER; ++j)
                    if (hok[j] && hfield[j] && front_unwritten(halo[lane + 32 * j]))
                        halo[lane + 32 * j] = front_load(hp[j] + (AHEAD + 1) * hstep[j]);
            }
        }
        // (a ring holds more layers than a step reads, so that a lane one step
        // ahead writes none of them: this barrier a step is enough)
        __syncwarp();
        const int rp = t - delay, row = rp & (RING - 1), hrow = SKEW ? t & (RING - 1) : row;
        R X = __shfl_up_sync(0xffffffffu, v1, SZ), X2 = __shfl_up_sync(0xffffffffu, Xp, SZ);
        R Z = __shfl_up_sync(0xffffffffu, v1, 1), Z2 = __shfl_up_sync(0xffffffffu, Zp, 1);
        if (xs == 0) {
            X = s_halo[hrow][zs];
            X2 = s_halo[hrow][SZ + zs];
        }
        if (zs == 0) {
            Z = s_halo[hrow][2 * SZ + xs];
            Z2 = s_halo[hrow][2 * SZ + SX + xs];
        }
        Xp = X;
        Zp = Z;
        if (colv && rp >= 0 && rp < nnr) {
            spc.h[1] = hxn;
            spc.w[1] = wxn;
            spc.h[2] = s_halo[row][2 * SZ + 2 * SX + xs];
            spc.w[2] = s_halo[row][2 * SZ + 3 * SX + xs];
            // (the next layer's, a step ahead)
            const int up = rp + 1 < nnr ? -(rp + 1) : 0;
            hxn = __ldg(hxp + up);
            wxn = __ldg(wxp + up);
            R v = fm_update_upstream<R>(s_slow[row][lane], v1, v2, X, X2, Z, Z2, true, rp < nnr - 1, inXu, inXd,
                                        inZu, inZd, spc, f.order2);
            if (rp == 0) v = fixed0 ? bottom : fm_min(v, bottom);
            v2 = v1;
            v1 = v;
            if (SKEW) {
                front_store(op, v);
                op -= layer;
            } else {
                s_out[row][lane] = v;
            }
        }
        // layer t - LAG is complete
        if (!SKEW && t >= LAG) {
            if (colv) front_store(op, s_out[(t - LAG) & (RING - 1)][lane]);
            op -= layer;
        }
    }
}

// Boundary nodes without a time, next to fixed ones: a start value from the
// fixed lateral neighbours of all four quadrants, left in the field marked
// unwritten (sign bit set) for the main sweep, which takes the lesser of it
// and its own.  The certification always has these nodes recomputed.
template <typename R>
__global__ void __launch_bounds__(256) holes_kernel(FieldArgs<R> f, int nev)
{
    const size_t layer = (size_t)f.nnx * f.nnz;
    const R INF = Lim<R>::inf();
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < layer * nev; q += (size_t)gridDim.x * blockDim.x) {
        if (f.frozen[q]) continue;
        const int e = (int)(q / layer), c = (int)(q - (size_t)e * layer);
        const int gx = c / f.nnz, gz = c - gx * f.nnz;
        R *Tb = f.T + ((size_t)e * f.nnr + (f.nnr - 1)) * layer;
        auto fixed_at = [&](int x, int z) -> R {
            if (x < 0 || x >= f.nnx || z < 0 || z >= f.nnz) return INF;
            const size_t p = (size_t)x * f.nnz + z;
            return f.frozen[(size_t)e * layer + p] ? Tb[p] : INF;
        };
        const auto p = Tile<R, 1, 4, 8>::params_global(f, f.nnr - 1, gx, gz);
        R v = INF;
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            const int dx = (k & 1) ? 1 : -1, dz = (k & 2) ? 1 : -1;      // the sides taken as upstream
            auto in = [](int i, int n) { return i >= 0 && i < n; };
            v = fm_min(v, fm_update_upstream<R>(p.s, INF, INF, fixed_at(gx + dx, gz), fixed_at(gx + 2 * dx, gz),
                                                fixed_at(gx, gz + dz), fixed_at(gx, gz + 2 * dz), false, true,
                                                in(gx + dx, f.nnx), in(gx - dx, f.nnx), in(gz + dz, f.nnz),
                                                in(gz - dz, f.nnz), p.sp, f.order2));
        }
        Tb[c] = -v;
    }
}

template <typename R>
void launch_holes(const FieldArgs<R> &f, int nev, cudaStream_t st)
{
    const long long n = (long long)f.nnx * f.nnz * nev;
    holes_kernel<R><<<(int)std::min<long long>((n + 255) / 256, 152LL * 16), 256, 0, st>>>(f, nev);
}

template <typename R, int SX, int SZ>
void launch_front(const FrontArgs<R> &a, cudaStream_t st)
{
    if (a.skew)
        front_kernel<R, SX, SZ, true><<<a.count, 32, 0, st>>>(a);
    else
        front_kernel<R, SX, SZ, false><<<a.count, 32, 0, st>>>(a);
}

template <typename R, int SX, int SZ>
int occupancy_front()
{
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, front_kernel<R, SX, SZ, false>, 32, 0);
    return nb;
}

}  // namespace fm3dt
