// stream.cuh -- streaming sweeps after the main one (front.cuh): the extra
// sweeps of near-tie events, re-sweeps of events that still change on many
// tiles, and the verifying sweep.  A sweep is only a good start for the
// rounds, which reach the same fixed point from any start.
//
// One warp takes a block of SX x SZ (theta, phi) columns over the whole height,
// upward, lane (x', z') (swept coordinates) updating layer t - x' - z' at step t
// with the full update, so each node sees its upstream neighbours' new values
// and its downstream neighbours' old ones.  As in the main sweep the values of
// the block's own columns pass through registers and shuffles (upstream: the
// neighbour lane's last value, and the value it used one step before;
// downstream: the neighbour lane's old values one and two layers up, which are
// the old values of this lane's layer), and layers of the field, the slowness
// and the halo columns come in coalesced and wait in shared-memory rings for
// the lanes that use them up to SX + SZ - 2 steps later.
//
// A sweep is one launch.  Warps take blocks from a counter, group of events by
// group and hyperplane by hyperplane; a block follows the two upstream of it
// step by step: each publishes, every step or two, a word with the steps it has
// made and the chunks of layers it has changed (a release store), and a block
// reads the halo of a step -- each column at the layer of the lane beside it --
// only when both upstream words say it is final (an acquire load; the halo
// columns come from L2).  The blocks a block waits for were taken before it by
// warps that run, so every wait ends; it is bounded all the same.
//
// Tracked sweeps (the near-tie chain) run only where something can change: a
// node is recomputed to the same bits unless a stencil neighbour changed since
// it was last computed.  Per block and sweep a word holds the chunks (1 <<
// act_shift layers) in which a node changed.  A step runs when one of its nodes
// lies in a chunk that changed in the previous sweep in the block itself (or
// the chunk above or below: neighbours up to two layers away) or a lateral
// neighbour (the same chunk: lateral neighbours share the layer), or earlier in
// this sweep in the block itself or an upstream neighbour -- which the
// published word tells before the step.  Quiet chunks are passed by without
// loading them.
//
// What bounds it with few events is the chain: nnr steps and a block's lag for
// every hyperplane of blocks, SX steps along theta and SZ along phi (and the
// publication's).  With many (141 near ties on 96x112x112) it is throughput, by
// the blocks and steps that run: 55-63% of the issue slots in the sweeps that
// run most blocks, from the 15.5 warps an SM that 128 registers allow, which
// wait for their own instructions; DRAM 2-6%.
// With whole layers instead of steps in the words, a block lagged SX + SZ - 1
// steps along either: two double-precision events on 192x224x224 131 -> 120.5 ms,
// 32 on 128^3 22.9 -> 21.4, 500 single-precision ones on 192x224x224 94.5 ->
// 93.3, three requests on 97^3 0.87 -> 0.85.
#pragma once
#include "solver.cuh"

namespace fm3dt {

// Queue tile w with flag bits `bits` unless it holds them already (flags only
// gain bits while a sweep runs, so a stale read costs one needless atomic);
// the node's new value is made visible before the flag that sends its tile
// to a round.
template <typename R>
__device__ __forceinline__ void stream_queue(const StreamArgs<R> &a, int w, int bits)
{
    const int want = bits | kQueued;
    if ((__ldcg(a.flag + w) & want) == want) return;
    __threadfence();
    if (!(atomicOr(&a.flag[w], want) & kQueued)) a.list[atomicAdd(a.count_out, 1)] = w;
}

// A node changed in a flag-mode sweep (a verification sweep, a re-sweep, the
// near-tie events' last extra sweep): its tile recomputes every node,
// and each face neighbour whose 2-deep halo holds the node recomputes the
// nodes next to that face (the flag bits of the rounds).
template <typename R>
__device__ void stream_mark(const StreamArgs<R> &a, int e, int gr, int gx, int gz)
{
    const int ti = gr / a.tr, tj = gx / a.tx, tk = gz / a.tz;
    const int ri = gr - ti * a.tr, xi = gx - tj * a.tx, zi = gz - tk * a.tz;
    const int sl = a.ntx * a.ntz;
    const int w = e * a.tiles_per_event + (ti * a.ntx + tj) * a.ntz + tk;
    stream_queue(a, w, kFull);
    if (ri < 2 && ti > 0) stream_queue(a, w - sl, kFaceDown);
    if (ri >= a.tr - 2 && ti < a.ntr - 1) stream_queue(a, w + sl, kFaceUp);
    if (xi < 2 && tj > 0) stream_queue(a, w - a.ntz, kFaceXp);
    if (xi >= a.tx - 2 && tj < a.ntx - 1) stream_queue(a, w + a.ntz, kFaceXm);
    if (zi < 2 && tk > 0) stream_queue(a, w - 1, kFaceZp);
    if (zi >= a.tz - 2 && tk < a.ntz - 1) stream_queue(a, w + 1, kFaceZm);
}

// Polls of a halo value or an upstream word (an L2 round trip each, about a
// second in all) before the error flag is raised and the block goes on.
#ifndef FM_WAIT_POLLS
#define FM_WAIT_POLLS (1u << 20)
#endif

// Whether a warp's wait ends unanswered after `polls` polls (the same in all
// lanes): its limit is reached, or another wait's was, looked for every 64th
// poll.  The lanes take one read of the error word: lanes that saw it change
// between their reads would part, and wait for each other in the votes and
// shuffles ahead.
__device__ __forceinline__ bool wait_gives_up(unsigned polls, int *err)
{
    if (!(polls > FM_WAIT_POLLS ||
          ((polls & 63u) == 0u && (__shfl_sync(0xffffffffu, *(volatile int *)err, 0) & 16))))
        return false;
    atomicOr(err, 16);
    return true;
}
// Steps between two publications of a block's word.  Each costs a fence, and
// delays the blocks downstream by as many steps each.  A step in double precision
// is long against a fence: 1 (two events on 192x224x224 with 1, 2, 3 steps 120.5,
// 122.3, 123.6 ms).  Single precision: 2 (500 events on 192x224x224 with 1, 2, 3
// steps 94.1, 93.4, 93.5 ms).
template <typename R> constexpr int kPublish = sizeof(R) == 8 ? 1 : 2;
// In a block's word: the steps it tells of were passed by, so that the layers
// below are final (a running block is LAG layers behind its leading lane).
constexpr unsigned kPassed = 1u << 31;
// Quiet steps ahead that are worth the reload of the rings.
constexpr int kRelayJump = 6;

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_u64(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.release.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void st_relaxed_u64(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}

// Chunk c of a mask and the chunks above and below it.
__device__ __forceinline__ unsigned chunk_spread(unsigned m) { return m | (m << 1) | (m >> 1); }

// Resident one-warp CTAs the registers must allow: in single precision 16 (128
// registers, no spills; warps mostly follow each other, so a shorter step counts
// for more than another warp).  500 events on 192x224x224 with 14, 16, 18, 20
// resident 92.3, 92.4, 93.3, 93.3 ms, with +-5% contrast 200, 198.5, 208, 206.5;
// three requests on 97^3 0.83, 0.82, 0.845, 0.86.  In double precision 12.
template <typename R> struct RelayBlocks { static constexpr int value = 16; };
template <> struct RelayBlocks<double> { static constexpr int value = 12; };

template <typename R, int SX, int SZ>
__global__ void __launch_bounds__(32, RelayBlocks<R>::value) relay_kernel(StreamArgs<R> a)
{
    static_assert(SX * SZ == 32, "one warp per column block");
    constexpr int LAG = SX + SZ - 2;
    constexpr int AHEAD = 3;                        // steps a step's copies are issued ahead
    // rows t - LAG .. t + AHEAD (the own columns two layers higher), and one
    // more: a lane may be a step ahead
    constexpr int RING = LAG + AHEAD + 2 <= 16 ? 16 : 32;
    constexpr int NF = 2 * SZ + 2 * SX;             // halo columns of the upstream (downstream) sides
    constexpr int NU = NF + 2 * SX;                 // ... and hz, wz of the block's rows
    constexpr int PU = (NU + 31) / 32, PD = (NF + 31) / 32;
    __shared__ R s_own[RING][32], s_slow[RING][32], s_up[RING][NU], s_dn[RING][NF];
    const FieldArgs<R> &f = a.f;
    const R INF = Lim<R>::inf();
    const int lane = threadIdx.x, xs = lane / SZ, zs = lane % SZ, delay = xs + zs;
    const int nnr = f.nnr;
    const long long layer = (long long)f.nnx * f.nnz;
    const bool track = a.act_cur != nullptr, skip = track && a.act_prev != nullptr;
    const int sh = a.act_shift;
    for (;;) {
        __syncwarp();
        unsigned item = 0;
        if (lane == 0) item = atomicAdd(a.next, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= a.count) return;
        const unsigned gsize = (unsigned)a.nblocks * (unsigned)a.group;
        const int k0 = (int)(item / gsize) * a.group;
        const unsigned rem = item % gsize;
        const unsigned ge = (unsigned)min(a.group, a.nev - k0);
        const int packed = a.blocks[rem / ge];
        const int k = k0 + (int)(rem % ge);
        const int e = a.events ? a.events[k] : k;
        int dir = a.dir[e];
        if (a.flip & 4) dir ^= ((dir >> 2) & 1) | (((dir >> 3) & 1) << 1);
        dir ^= a.flip & 3;
        const bool sx = dir & 1, sz = (dir >> 1) & 1;
        const int bxp = (packed >> 12) & 0xfff, bzp = packed & 0xfff;
        const int bx = sx ? bxp : a.nbx - 1 - bxp, bz = sz ? bzp : a.nbz - 1 - bzp;
        const int x0 = bx * SX, z0 = bz * SZ;
        const int gx = sx ? x0 + xs : x0 + SX - 1 - xs, gz = sz ? z0 + zs : z0 + SZ - 1 - zs;
        const bool colv = gx < f.nnx && gz < f.nnz;
        const size_t slot = ((size_t)k * a.nbx + bx) * a.nbz + bz;
        // bottom layer; a layer L counted from it lies L * layer before
        R *Tb = f.T + (size_t)e * layer * nnr + (nnr - 1) * layer;
        const long long own = colv ? (long long)gx * f.nnz + gz : 0;
        const R *Sb = f.s + (nnr - 1) * layer + own;
        const bool fixed0 = colv && f.frozen[(size_t)e * layer + own] != 0;
        // this lane's halo columns (upstream, downstream) in the bottom layer
        const R *up[PU], *dn[PD];
        long long ustep[PU];
        int late[PU];                                // steps after which a halo column is taken
        bool uok[PU], dok[PD];
#pragma unroll
        for (int j = 0; j < PU; ++j) {
            const int q = lane + 32 * j;
            int hx, hz = 0;
            if (q < 2 * SZ) {
                hx = sx ? x0 - 1 - q / SZ : x0 + SX + q / SZ;
                hz = sz ? z0 + q % SZ : z0 + SZ - 1 - q % SZ;
            } else {
                const int p = q - 2 * SZ, i = p % SX;
                hx = sx ? x0 + i : x0 + SX - 1 - i;
                if (p < 2 * SX) hz = sz ? z0 - 1 - p / SX : z0 + SZ + p / SX;
            }
            uok[j] = q < NU && hx >= 0 && hx < f.nnx && hz >= 0 && hz < f.nnz;
            ustep[j] = q < NF ? layer : f.nnx;
            late[j] = q < 2 * SZ ? q % SZ : q < NF ? (q - 2 * SZ) % SX : 0;
            up[j] = q < NF ? Tb : (q < NF + SX ? f.hz : f.wz) + (long long)(nnr - 1) * f.nnx;
            if (uok[j]) up[j] += q < NF ? (long long)hx * f.nnz + hz : hx;
        }
#pragma unroll
        for (int j = 0; j < PD; ++j) {
            const int q = lane + 32 * j;
            int hx, hz;
            if (q < 2 * SZ) {
                hx = sx ? x0 + SX + q / SZ : x0 - 1 - q / SZ;
                hz = sz ? z0 + q % SZ : z0 + SZ - 1 - q % SZ;
            } else {
                const int p = q - 2 * SZ;
                hx = sx ? x0 + p % SX : x0 + SX - 1 - p % SX;
                hz = sz ? z0 + SZ + p / SX : z0 - 1 - p / SX;
            }
            dok[j] = q < NF && hx >= 0 && hx < f.nnx && hz >= 0 && hz < f.nnz;
            dn[j] = Tb + (dok[j] ? (long long)hx * f.nnz + hz : 0);
        }
        const unsigned inl = (gx > 0 ? 4u : 0u) | (gx < f.nnx - 1 ? 8u : 0u) | (gz > 0 ? 16u : 0u) |
                             (gz < f.nnz - 1 ? 32u : 0u);
        // lanes 0 and 1: the words of the blocks upstream along theta and phi
        const unsigned long long *upw = nullptr;
        if (lane == 0 && bxp > 0) upw = a.prog + ((size_t)k * a.nbx + (sx ? bx - 1 : bx + 1)) * a.nbz + bz;
        if (lane == 1 && bzp > 0) upw = a.prog + ((size_t)k * a.nbx + bx) * a.nbz + (sz ? bz - 1 : bz + 1);
        const int steps = nnr + LAG;
        const bool up0 = bxp > 0 || bzp > 0;
        int avail = up0 ? 0 : nnr;                   // layers final upstream
        int ready = up0 ? 0 : steps;                 // steps whose halo is final
        unsigned um = 0;                             // chunks changed upstream, as far as known
        // waits until L layers and step t's halo are final
        auto need = [&](int L, int t) {
            unsigned polls = 0;
            while (avail < L || ready <= t) {
                const unsigned long long w = upw ? ld_acquire_u64(upw) : (unsigned long long)(kPassed | (unsigned)steps);
                const int n = (int)((unsigned)w & ~kPassed);
                const int la = min(nnr, (unsigned)w & kPassed ? n : n - LAG), ra = n >= steps ? steps : n - (lane ? SZ : SX) + 1;
                avail = max(avail, min(__shfl_sync(0xffffffffu, la, 0), __shfl_sync(0xffffffffu, la, 1)));
                ready = max(ready, min(__shfl_sync(0xffffffffu, ra, 0), __shfl_sync(0xffffffffu, ra, 1)));
                const unsigned m = (unsigned)(w >> 32);
                um = __shfl_sync(0xffffffffu, m, 0) | __shfl_sync(0xffffffffu, m, 1);
                if (avail >= L && ready > t) break;
                if (wait_gives_up(++polls, a.err)) {
                    avail = nnr;
                    ready = steps;
                }
                __nanosleep(20);
            }
            __syncwarp();
        };
        // the chunks that can change
        unsigned act = ~0u, chg = 0;
        if (skip) {
            unsigned m = 0;
            if (lane < 5) {
                const int x_ = bx + (lane == 1 ? -1 : lane == 2 ? 1 : 0), z_ = bz + (lane == 3 ? -1 : lane == 4 ? 1 : 0);
                if (x_ >= 0 && x_ < a.nbx && z_ >= 0 && z_ < a.nbz)
                    m = __ldcg(a.act_prev + ((size_t)k * a.nbx + x_) * a.nbz + z_);
                if (lane == 0) m = chunk_spread(m);
            }
            act = __reduce_or_sync(0xffffffffu, m);
        }
        R hu[PU];                                    // the next step's upstream halo, the next layer's spacings
        R v1 = INF, v2 = INF, Xp = INF, Zp = INF, u1 = INF, u2 = INF;
        auto load_up = [&](int t) {
            need(0, t);
#pragma unroll
            for (int j = 0; j < PU; ++j) {
                const int L = t - late[j];
                hu[j] = uok[j] && L >= 0 && L < nnr ? __ldcg(up[j] - L * ustep[j]) : INF;
            }
        };
        auto store_up = [&](int t) {
#pragma unroll
            for (int j = 0; j < PU; ++j)
                if (lane + 32 * j < NU) s_up[t & (RING - 1)][lane + 32 * j] = hu[j];
        };
        auto copy_own = [&](int L) {
            if (L >= 0 && L < nnr && colv) cp_async_elem(&s_own[L & (RING - 1)][lane], Tb + own - L * layer);
        };
        auto copy_rest = [&](int L) {
            if (L < 0 || L >= nnr) return;
            if (colv) cp_async_elem(&s_slow[L & (RING - 1)][lane], Sb - L * layer);
#pragma unroll
            for (int j = 0; j < PD; ++j)
                if (lane + 32 * j < NF) {
                    R *d = &s_dn[L & (RING - 1)][lane + 32 * j];
                    if (dok[j])
                        cp_async_elem(d, dn[j] - L * layer);
                    else
                        *d = INF;
                }
        };
        // everything step t reads, from memory (the layers of earlier steps
        // have been computed, or left as they are)
        auto seat = [&](int t) {
            __syncwarp();
            for (int L = max(0, t - LAG + 2); L < t + AHEAD + 2; ++L) copy_own(L);
            for (int L = max(0, t - LAG); L < t + AHEAD; ++L) copy_rest(L);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            // (the spacings' rows; a step's halo is its own)
            for (int L = max(0, t - LAG); L < min(t, nnr); ++L)
#pragma unroll
                for (int j = 0; j < PU; ++j)
                    if (lane + 32 * j >= NF && lane + 32 * j < NU)
                        s_up[L & (RING - 1)][lane + 32 * j] = uok[j] ? __ldg(up[j] - L * ustep[j]) : INF;
            load_up(t);
            const int rp = t - delay;
            auto at = [&](int L, bool in, long long c) -> R {
                return colv && in && L >= 0 && L < nnr ? __ldcg(Tb + c - L * layer) : INF;
            };
            v1 = at(rp - 1, true, own);
            v2 = at(rp - 2, true, own);
            Xp = at(rp - 1, inl & (sx ? 4u : 8u), own + (sx ? -f.nnz : f.nnz));
            Zp = at(rp - 1, inl & (sz ? 16u : 32u), own + (sz ? -1 : 1));
            u1 = at(rp, true, own);
            u2 = at(rp + 1, true, own);
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncwarp();
        };
        int published = 0;
        bool dirty = false;                          // values stored since the last publication
        auto publish = [&](int done, unsigned passed) {
            __syncwarp();
            if (lane == 0) {
                const unsigned long long w = (unsigned long long)(passed | (unsigned)done) | (unsigned long long)chg << 32;
                // (with nothing stored there is nothing to release)
                if (dirty)
                    st_release_u64(a.prog + slot, w);
                else
                    st_relaxed_u64(a.prog + slot, w);
            }
            dirty = false;
            published = done;
        };
        bool seated = false, ran = false;
        int first = 0;                               // lowest layer of the current run of steps
        int t = 0;
        while (t < steps) {
            if (skip) {
                const unsigned range = (~0u << (max(0, t - LAG) >> sh)) & (0xffffffffu >> (31 - (min(t, nnr - 1) >> sh)));
                if (!((act | um) & range)) {
                    // quiet as far as known: on to the next chunk that changes
                    // or that upstream has not left (chunks above the leading
                    // one; with none, to the end)
                    const int c = t < nnr ? (t >> sh) + 1 : 32;
                    need(t < nnr ? min(nnr, c << sh) : nnr, -1);
                    if (!((act | um) & range)) {
                        const int known = avail >= nnr ? 32 : avail >> sh;
                        const unsigned above = c < 32 ? (act | um) & (~0u << c) : 0u;
                        const int to = min(above ? __ffs(above) - 1 : 32, max(c, known));
                        const int tn = (to << sh) < nnr ? to << sh : steps;
                        if (!seated || tn - t >= kRelayJump) {
                            // (copies of the last steps may still be on their
                            // way into the rings, which are filled anew: two
                            // copies to one place come in no order)
                            if (seated) asm volatile("cp.async.wait_all;\n" ::: "memory");
                            seated = false;
                            t = tn;
                            if (t < steps) publish(t, kPassed);
                            continue;
                        }
                    }
                }
            }
            if (!seated) {
                seat(t);
                seated = ran = true;
                first = t;
            }
            // step t: layer t's halo into its ring, layer t + 1's on its way
            store_up(t);
            if (t + 1 < steps) load_up(t + 1);
            copy_own(t + AHEAD + 2);
            copy_rest(t + AHEAD);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            asm volatile("cp.async.wait_group %0;\n" ::"n"(AHEAD) : "memory");
            __syncwarp();
            const int rp = t - delay, row = rp & (RING - 1);
            const R old = u1;
            u1 = u2;
            u2 = colv && rp + 2 >= 0 && rp + 2 < nnr ? s_own[(rp + 2) & (RING - 1)][lane] : INF;
            R t1[6], t2[6];
            t1[1] = v1; t2[1] = v2;                  // r+1 (the layer below)
            t1[0] = u1; t2[0] = u2;                  // r-1
            t1[2] = __shfl_up_sync(0xffffffffu, v1, SZ);
            t2[2] = __shfl_up_sync(0xffffffffu, Xp, SZ);
            t1[4] = __shfl_up_sync(0xffffffffu, v1, 1);
            t2[4] = __shfl_up_sync(0xffffffffu, Zp, 1);
            t1[3] = __shfl_down_sync(0xffffffffu, u1, SZ);
            t2[3] = __shfl_down_sync(0xffffffffu, u2, (2 * SZ) & 31);
            t1[5] = __shfl_down_sync(0xffffffffu, u1, 1);
            t2[5] = __shfl_down_sync(0xffffffffu, u2, 2);
            if (xs == 0) {
                t1[2] = s_up[t & (RING - 1)][zs];
                t2[2] = s_up[t & (RING - 1)][SZ + zs];
            }
            if (zs == 0) {
                t1[4] = s_up[t & (RING - 1)][2 * SZ + xs];
                t2[4] = s_up[t & (RING - 1)][2 * SZ + SX + xs];
            }
            if (xs == SX - 1) t1[3] = s_dn[row][zs];
            if (xs >= SX - 2) t2[3] = s_dn[row][(xs - (SX - 2)) * SZ + zs];
            if (zs == SZ - 1) t1[5] = s_dn[row][2 * SZ + xs];
            if (zs >= SZ - 2) t2[5] = s_dn[row][2 * SZ + (zs - (SZ - 2)) * SX + xs];
            Xp = t1[2];
            Zp = t1[4];
            bool changed = false;
            if (colv && rp >= 0 && rp < nnr) {
                const int gr = nnr - 1 - rp;
                R v = old;
                // (layers below the run's first were passed by, and are final)
                if (rp >= first && !(rp == 0 && fixed0)) {
                    Spacing<R> sp;
                    sp.h[0] = f.hr;
                    sp.w[0] = f.wr;
                    sp.h[1] = __ldg(f.hx + gr);
                    sp.w[1] = __ldg(f.wx + gr);
                    sp.h[2] = s_up[row][NF + xs];
                    sp.w[2] = s_up[row][NF + SX + xs];
                    // (theta and phi neighbours may change places: a node's
                    // octants are the same either way)
                    const unsigned inb = (gr > 0 ? 1u : 0u) | (rp > 0 ? 2u : 0u) |
                                         (sx ? inl & 12u : ((inl & 4u) << 1) | ((inl & 8u) >> 1)) |
                                         (sz ? inl & 48u : ((inl & 16u) << 1) | ((inl & 32u) >> 1));
                    v = fm_update<R>(s_slow[row][lane], t1, t2, inb, sp, f.order2);
                    if (fbits(v) != fbits(old)) {
                        changed = true;
                        Tb[own - rp * layer] = v;
                        if (a.flag) stream_mark(a, e, gr, gx, gz);
                    }
                }
                v2 = v1;
                v1 = v;
            }
            if (track) {
                const unsigned m = __reduce_or_sync(0xffffffffu, changed ? 1u << (rp >> sh) : 0u);
                chg |= m;
                act |= chunk_spread(m);
                dirty = dirty || m;
            } else {
                dirty = dirty || __any_sync(0xffffffffu, changed);
            }
            ++t;
            if (t >= published + kPublish<R> && t < steps) publish(t, 0u);
        }
        if (lane == 0) {
            if (track) a.act_cur[slot] = chg;
            if (skip && a.act_items) atomicAdd(a.act_items + (ran ? 0 : 1), 1ull);
        }
        publish(steps, kPassed);
    }
}

template <typename R, int SX, int SZ>
struct StreamKernels {
    static void sweep(int grid, const StreamArgs<R> &a, cudaStream_t st)
    {
        relay_kernel<R, SX, SZ><<<grid, 32, 0, st>>>(a);
    }
    static int occ()
    {
        int nb = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, relay_kernel<R, SX, SZ>, 32, 0);
        return nb;
    }
};

#define FM_STREAM_SWITCH(idx, CALL)       \
    switch (idx) {                        \
        case 0: CALL(4, 8); break;        \
        default: CALL(2, 16); break;      \
    }

}  // namespace fm3dt
