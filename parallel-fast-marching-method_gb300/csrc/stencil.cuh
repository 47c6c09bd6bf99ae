// stencil.cuh -- the upwind eikonal node update shared by every solver kernel.
//
// Restates the octant update of fm3dt_parallel.f90 fouds2_all (F:635-1004,
// mixed order) and fouds1_all (F:535-633, first order) in a generic form.
// For each of the eight octants (one direction per axis r, theta, phi) whose
// three neighbours all lie inside the grid (F:710-712), the axes whose
// neighbour is upwind contribute one term of
//     sum_a ((k_a*T - beta_a) / H_a)^2 = s^2,
// with k=1, beta=t1, H=h for a first-order axis and k=3, beta=4*t1-t2, H=2h
// for a second-order axis (F:712-982 enumerate the same cases by hand).  The
// quadratic keeps the reference's root choice and its clamp of a negative
// discriminant to zero (F:991-993); the node takes the minimum over octants
// (F:995-1000).  An axis is second order when its second neighbour is inside
// the grid, upwind and earlier than the first (F:645-707).
//
// Upwind set.  In the reference's fast marching a neighbour is used when it is
// alive, i.e. already final and earlier than the node being computed.  A
// block-parallel iterative solver has no heap order, so "alive" is restated
// as the fixed-point condition t1 < T: each octant adds its neighbours in
// ascending order of t1 and keeps the largest set whose solution T exceeds
// every used t1 (the causal Godunov solve).  At convergence the used set is
// exactly the set of neighbours earlier than the node, which is the set the
// reference's heap has popped when it computes the node.
//
// "Unset" is +infinity here (the reference uses 0.0, which an offset time can
// legitimately equal).  The unknown is solved relative to the earliest used
// neighbour, so every coefficient is a difference of nearby times; this keeps
// single-precision offset times accurate.
#pragma once

#ifndef FM_HD
#ifdef __CUDACC__
#define FM_HD __host__ __device__ __forceinline__
#else
#define FM_HD inline
#endif
#endif

namespace fm3dt {

template <typename R> struct Lim;
template <> struct Lim<double> {
    static FM_HD double inf() { return __builtin_huge_val(); }
};
template <> struct Lim<float> {
    static FM_HD float inf() { return __builtin_huge_valf(); }
};

template <typename R> FM_HD R fm_sqrt(R x);
template <> FM_HD double fm_sqrt<double>(double x) {
#ifdef __CUDA_ARCH__
    return __dsqrt_rn(x);
#else
    return __builtin_sqrt(x);
#endif
}
template <> FM_HD float fm_sqrt<float>(float x) {
#ifdef __CUDA_ARCH__
    return __fsqrt_rn(x);
#else
    return __builtin_sqrtf(x);
#endif
}

// Minimum and maximum as the hardware min/max instructions.  They differ from
// a compare-and-select only for NaN and for a +0/-0 pair; in-grid times are
// never NaN and never -0 (offsets from an event's earliest time start at +0,
// and sums of non-negative terms stay +0 or above), so the results are the
// same bits.
template <typename R> FM_HD R fm_min(R a, R b);
template <typename R> FM_HD R fm_max(R a, R b);
#ifdef __CUDA_ARCH__
template <> FM_HD float fm_min<float>(float a, float b) { return fminf(a, b); }
template <> FM_HD double fm_min<double>(double a, double b) { return fmin(a, b); }
template <> FM_HD float fm_max<float>(float a, float b) { return fmaxf(a, b); }
template <> FM_HD double fm_max<double>(double a, double b) { return fmax(a, b); }
#else
template <> FM_HD float fm_min<float>(float a, float b) { return __builtin_fminf(a, b); }
template <> FM_HD double fm_min<double>(double a, double b) { return __builtin_fmin(a, b); }
template <> FM_HD float fm_max<float>(float a, float b) { return __builtin_fmaxf(a, b); }
template <> FM_HD double fm_max<double>(double a, double b) { return __builtin_fmax(a, b); }
#endif

// The two keys of a conditional swap, in order (p: the second is smaller).
// Single precision takes min and max, which do not wait for the comparison;
// double precision keeps the selects, which run on the integer pipe rather
// than the narrow double-precision one.
template <typename R> FM_HD void fm_order_keys(bool p, R &ki, R &kj);
template <> FM_HD void fm_order_keys<float>(bool, float &ki, float &kj)
{
    const float lo = fm_min<float>(ki, kj);
    kj = fm_max<float>(ki, kj);
    ki = lo;
}
template <> FM_HD void fm_order_keys<double>(bool p, double &ki, double &kj)
{
    const double lo = p ? kj : ki;
    kj = p ? ki : kj;
    ki = lo;
}

// Explicit fused multiply-add.  The solver is compiled without automatic
// contraction, so every kernel instantiation (and the host) evaluates the
// stencil with exactly the same roundings; otherwise the compiler may fuse
// differently per instantiation and the iteration map -- hence its fixed
// point -- would differ in the last bits between tile shapes.
template <typename R> FM_HD R fm_fma(R a, R b, R c);
template <> FM_HD double fm_fma<double>(double a, double b, double c) { return __builtin_fma(a, b, c); }
template <> FM_HD float fm_fma<float>(float a, float b, float c) { return __builtin_fmaf(a, b, c); }

// Square root and quotient of the quadratic's root.  Single precision on the
// device uses the hardware approximations (deterministic, <= 2 ulp on a
// time increment of order 0.1-1 s, far below the float spacing of the
// offset times themselves); double precision is IEEE-rounded.
template <typename R> struct Fast;
template <> struct Fast<double> {
    static FM_HD double sqrt(double x) { return fm_sqrt<double>(x); }
    static FM_HD double div(double a, double b) { return a / b; }
};
template <> struct Fast<float> {
    static FM_HD float sqrt(float x) {
#ifdef __CUDA_ARCH__
        float r;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
        return r;
#else
        return __builtin_sqrtf(x);
#endif
    }
    static FM_HD float div(float a, float b) {
#ifdef __CUDA_ARCH__
        return __fdividef(a, b);
#else
        return a / b;
#endif
    }
};

// Per-node grid spacings: h[a] and 1/h[a]^2 for axes r, theta, phi.
template <typename R> struct Spacing {
    R h[3];
    R w[3];
};

// Neighbour directions: 0 = r-1 (up), 1 = r+1 (down), 2 = x-1, 3 = x+1,
// 4 = z-1, 5 = z+1.
//
// t1[d]: neighbour value (+inf if unset; +inf or NaN when bit d of inb is
//        clear, i.e. outside the grid)
// t2[d]: second neighbour value (+inf if unset; +inf or NaN outside the grid)
// sp:    spacings at the centre node
// s:     slowness at the centre node
// order2: 1 for the mixed-order scheme (fom=1), 0 for first order (fom=0)
// Returns the candidate time (+inf when no neighbour is set).
//
// Each direction is written in first-order form ((T - tau)/g)^2 with
// tau = t1, g = h (first order) or tau = t1 + (t1 - t2)/3, g = 2h/3 (second
// order, the same equation as the reference's (3T - 4 t1 + t2)/(2h) term),
// relative to tmin, the earliest in-grid neighbour.  Every octant sorts its
// three terms by t1 and adds them while t1 < T (the causal solve).
//
// This is the general form; fm_update below takes it only where its shorter
// form does not hold.
template <typename R>
FM_HD R fm_update_octants(R s, const R t1[6], const R t2[6], unsigned inb, const Spacing<R> &sp, int order2)
{
    const R INF = Lim<R>::inf();
    // (a neighbour outside the grid holds +inf or NaN, which the hardware
    // minimum passes over: no mask needed)
    R tmin = INF;
#pragma unroll
    for (int d = 0; d < 6; ++d) tmin = fm_min(tmin, t1[d]);
    if (!(tmin < INF)) return INF;
    const R s2 = s * s;
    R key[6], e[6], g[6], w[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        const int a = d >> 1;
        const bool o2 = order2 && (t2[d] < t1[d]);
        const R dt = t1[d] - tmin;
        // (an octant is evaluated only when its three neighbours are in the
        // grid, so an outside direction's key is never read)
        key[d] = dt;
        e[d] = o2 ? fm_fma<R>(t1[d] - t2[d], R(1.0 / 3.0), dt) : dt;
        g[d] = o2 ? sp.h[a] * R(2.0 / 3.0) : sp.h[a];
        w[d] = o2 ? sp.w[a] * R(2.25) : sp.w[a];
    }
    R best = INF;
    // Each octant sorts its three terms by key, stably (ties keep the order
    // r, theta, phi).  The lateral pair is sorted once and shared by the two
    // octants that differ only in the radial direction, and the radial term
    // is then inserted in front: two compare-and-swaps per octant instead of
    // three, and the same order as a full three-term network (a stable sort's
    // result is unique).  Both octants of a pair are sorted before either
    // solves, so that their sorts form one straight run of code.  An octant
    // with a neighbour outside the grid is evaluated all the same (from
    // whatever its keys hold) and left out of the minimum by a select rather
    // than branched around.  The minimum over octants does not depend on the
    // order they are visited in.
    // conditional swaps as selects (a branch around four moves costs more)
#define FM_CSWAP(i, j)                                                        \
    {                                                                         \
        const bool p_ = k##j < k##i;                                          \
        fm_order_keys<R>(p_, k##i, k##j);                                     \
        R q_ = p_ ? e##j : e##i; e##j = p_ ? e##i : e##j; e##i = q_;          \
        q_ = p_ ? g##j : g##i; g##j = p_ ? g##i : g##j; g##i = q_;            \
        q_ = p_ ? w##j : w##i; w##j = p_ ? w##i : w##j; w##i = q_;            \
    }
    // the causal two- and three-term solves of a sorted octant, from its
    // one-term solution x
    auto solve = [&](R k1, R k2, R e0, R e1, R e2, R w0, R w1, R w2, R x) -> R {
        if (k1 < x) {
            R a = w0 + w1;
            const R we0 = w0 * e0, we1 = w1 * e1;
            R b = we0 + we1;
            R c = fm_fma<R>(we0, e0, fm_fma<R>(we1, e1, -s2));
            R disc = fm_fma<R>(b, b, -(a * c));
            x = Fast<R>::div(b + Fast<R>::sqrt(fm_max<R>(disc, R(0))), a);
            if (k2 < x) {
                const R we2 = w2 * e2;
                a += w2;
                b += we2;
                c = fm_fma<R>(we2, e2, c);
                disc = fm_fma<R>(b, b, -(a * c));
                x = Fast<R>::div(b + Fast<R>::sqrt(fm_max<R>(disc, R(0))), a);
            }
        }
        return x;
    };
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int dx = 2 + ((q >> 1) & 1), dz = 4 + (q & 1);
        R ka = key[dx], ea = e[dx], ga = g[dx], wa = w[dx];
        R kb = key[dz], eb = e[dz], gb = g[dz], wb = w[dz];
        FM_CSWAP(a, b)
        // terms 0-2: the octant with the upper (r-1) neighbour; 3-5: the
        // lower (r+1) one; om*: the neighbours each needs inside the grid
        const unsigned omu = 1u | (1u << dx) | (1u << dz), omd = 2u | (1u << dx) | (1u << dz);
        R k0 = key[0], e0 = e[0], g0 = g[0], w0 = w[0];
        R k1 = ka, e1 = ea, g1 = ga, w1 = wa;
        R k2 = kb, e2 = eb, g2 = gb, w2 = wb;
        R k3 = key[1], e3 = e[1], g3 = g[1], w3 = w[1];
        R k4 = ka, e4 = ea, g4 = ga, w4 = wa;
        R k5 = kb, e5 = eb, g5 = gb, w5 = wb;
        FM_CSWAP(0, 1)
        FM_CSWAP(3, 4)
        FM_CSWAP(1, 2)
        FM_CSWAP(4, 5)
        // (an octant with no neighbour set has e0 = +inf: its x = +inf leaves
        // best as it is, and no further term passes k < x)
        const R xu = fm_fma<R>(s, g0, e0), xd = fm_fma<R>(s, g3, e3);
        const R vu = solve(k1, k2, e0, e1, e2, w0, w1, w2, xu);
        best = (inb & omu) == omu ? fm_min(best, vu) : best;
        const R vd = solve(k4, k5, e3, e4, e5, w3, w4, w5, xd);
        best = (inb & omd) == omd ? fm_min(best, vd) : best;
    }
#undef FM_CSWAP
    return tmin + best;
}

// The least value, relative to tmin, of the causal solves of the seven subsets
// of three sides (one an axis), with four quadratic solves instead of the eight
// octants' sixteen: the singletons are one FMA each, the three pairs one solve
// each, and the triple's first two terms are one of the pairs (the same order and
// the same operations as the octants', hence the same bits), so only its
// three-term solve is added.  The four solves are straight-line code with
// selects at the end: a sweep's few warps wait on each other, and three pairs
// solved side by side are a third of the chain of three branches (main sweep of
// one 64^3 event 300 -> 228 us; of 500 events on 192x224x224, bound by issue,
// 50.6 -> 42.4 ms: 341 -> 295 instructions a step).  Sums of two are the same in
// either order; only the innermost FMA of a pair's c depends on which term
// comes first.
//
// t1, t2: the sides' first and second neighbour values; tmin: the least of t1;
// n / f: whether each side, and the opposite one, lies inside the grid.
template <typename R>
FM_HD R fm_subsets(R s, const R t1[3], const R t2[3], R tmin, bool n0, bool f0, bool n1, bool f1, bool n2, bool f2,
                   const Spacing<R> &sp, int order2)
{
    const R INF = Lim<R>::inf();
    const R s2 = s * s;
    // (with an unset neighbour, or all of them, differences are +inf or NaN:
    // no comparison lets them in, and an unset tmin is selected at the end)
    R k[3], e[3], w[3], we[3], x1[3], q[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const bool o2 = order2 && (t2[a] < t1[a]);
        const R dt = t1[a] - tmin;
        k[a] = dt;
        e[a] = o2 ? fm_fma<R>(t1[a] - t2[a], R(1.0 / 3.0), dt) : dt;
        const R g = o2 ? sp.h[a] * R(2.0 / 3.0) : sp.h[a];
        w[a] = o2 ? sp.w[a] * R(2.25) : sp.w[a];
        x1[a] = fm_fma<R>(s, g, e[a]);        // the one-term solution
        we[a] = w[a] * e[a];
        q[a] = fm_fma<R>(we[a], e[a], -s2);
    }
    // causal solves of the pairs DX, DZ, XZ (i before j in axis order, sorted
    // stably): the two-term step exactly as fm_update's
    R A[3], B[3], C[3], xp[3];
    bool both[3];
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        const int i = n == 2 ? 1 : 0, j = n == 0 ? 1 : 2;
        const bool p = k[j] < k[i];
        A[n] = w[i] + w[j];
        B[n] = we[i] + we[j];
        const R cj = fm_fma<R>(we[j], e[j], q[i]), ci = fm_fma<R>(we[i], e[i], q[j]);
        C[n] = p ? cj : ci;
        const R disc = fm_fma<R>(B[n], B[n], -(A[n] * C[n]));
        const R x = Fast<R>::div(B[n] + Fast<R>::sqrt(fm_max<R>(disc, R(0))), A[n]);
        const R xf = p ? x1[j] : x1[i];
        both[n] = (p ? k[i] : k[j]) < xf;
        xp[n] = both[n] ? x : xf;
    }
    // the triple: L, the last of a stable sort, and the pair without it
    const bool zx = k[2] < k[1];                            // Z before X
    const bool dl = fm_max(k[1], k[2]) < k[0];              // D last
    const R kL = dl ? k[0] : (zx ? k[1] : k[2]);
    const R eL = dl ? e[0] : (zx ? e[1] : e[2]);
    const R wL = dl ? w[0] : (zx ? w[1] : w[2]);
    const R weL = dl ? we[0] : (zx ? we[1] : we[2]);
    const R A2 = dl ? A[2] : (zx ? A[1] : A[0]);
    const R B2 = dl ? B[2] : (zx ? B[1] : B[0]);
    const R C2 = dl ? C[2] : (zx ? C[1] : C[0]);
    const R x2 = dl ? xp[2] : (zx ? xp[1] : xp[0]);
    const bool on2 = dl ? both[2] : (zx ? both[1] : both[0]);
    const R A3 = A2 + wL, B3 = B2 + weL, C3 = fm_fma<R>(weL, eL, C2);
    const R disc = fm_fma<R>(B3, B3, -(A3 * C3));
    const R x3 = Fast<R>::div(B3 + Fast<R>::sqrt(fm_max<R>(disc, R(0))), A3);
    const R xt = on2 && kL < x2 ? x3 : x2;
    // subsets whose octant lies inside the grid (upstream side on the axes in
    // the subset, downstream side on the others).  (At the bottom layer, D
    // unset and r-1 inside, n0 may be passed as true: the octants with D then
    // give what those with r-1 give.)
    R best = INF;
    best = n0 && f1 && f2 ? fm_min(best, x1[0]) : best;
    best = f0 && n1 && f2 ? fm_min(best, x1[1]) : best;
    best = f0 && f1 && n2 ? fm_min(best, x1[2]) : best;
    best = n0 && n1 && f2 ? fm_min(best, xp[0]) : best;
    best = n0 && f1 && n2 ? fm_min(best, xp[1]) : best;
    best = f0 && n1 && n2 ? fm_min(best, xp[2]) : best;
    best = n0 && n1 && n2 ? fm_min(best, xt) : best;
    return best;
}

// The node update of a sweep from an unset field, where every neighbour
// downstream of the sweep (up, r-1, and the lateral directions the sweep runs
// toward) is still unset when the node is computed.  Then only the three
// upstream neighbours -- down (r+1) and the lateral ones the sweep comes
// from, here D, X and Z -- can enter an octant, and each of the eight octants
// is the causal solve of the upstream terms it contains: the octant that
// takes the upstream side on the axes of a subset S of {D, X, Z} and the
// downstream side on the others solves S (its downstream terms are +inf,
// sort last and never pass k < x).  So this returns fm_update's value, bit
// for bit, with +inf at the downstream neighbours: the same keys, the same
// stable order within each subset (key, then axis r, theta, phi), the same
// arithmetic, and an octant counted when its three neighbours lie inside the
// grid.
//
// tD/tD2, tX/tX2, tZ/tZ2: upstream first and second neighbour values;
// in*: whether each upstream (u) and downstream (d) neighbour lies inside the
// grid (inD: r+1, inU: r-1).
template <typename R>
FM_HD R fm_update_upstream(R s, R tD, R tD2, R tX, R tX2, R tZ, R tZ2, bool inD, bool inU, bool inXu, bool inXd,
                           bool inZu, bool inZd, const Spacing<R> &sp, int order2)
{
    const R INF = Lim<R>::inf();
    const R t1[3] = {tD, tX, tZ}, t2[3] = {tD2, tX2, tZ2};
    const R tmin = fm_min(fm_min(tD, tX), tZ);
    const R best = fm_subsets<R>(s, t1, t2, tmin, inD, inU, inXu, inXd, inZu, inZd, sp, order2);
    return tmin < INF ? tmin + best : INF;
}

// The node update's short form (false: it does not hold).  On each axis the earlier neighbour is the near side, the
// other the far side.  Where every far side is first order and its key at
// least B (1 + kNear), B the least value of the near sides' seven subsets, and
// no near side with a key of B (1 - kNear) or more is second order, the eight
// octants' least value is B, bit for bit: adding a first-order causal term
// with key k to an octant's solve gives a root above k (the quadratic is below
// s^2 at k, or its vertex lies above k), so an octant that takes a far side
// ends above B (1 + kNear) less the solve's rounding (at most ~7e-4 of it in
// single precision, a discriminant near zero losing half its digits), and
// one that takes none is the solve of its near sides, which is a subset's.
// (An unset or outside far side is never taken.)  The seven subsets are four
// quadratics in straight-line code, the octants up to sixteen behind
// branches; in a sweep or a round nearly every node takes the short form.
constexpr float kNear = 1.0f / 256.0f;

template <typename R>
FM_HD bool fm_update_near(R s, const R t1[6], const R t2[6], unsigned inb, const Spacing<R> &sp, int order2, R &out)
{
    const R INF = Lim<R>::inf();
    R n1[3], n2[3], f1[3], f2[3];
    bool nin[3], fin[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const bool ia = (inb >> (2 * a)) & 1u, ib = (inb >> (2 * a + 1)) & 1u;
        const R ta = ia ? t1[2 * a] : INF, tb = ib ? t1[2 * a + 1] : INF;
        const bool p = tb < ta;
        n1[a] = p ? tb : ta;
        f1[a] = p ? ta : tb;
        n2[a] = p ? t2[2 * a + 1] : t2[2 * a];
        f2[a] = p ? t2[2 * a] : t2[2 * a + 1];
        nin[a] = p ? ib : ia;
        fin[a] = p ? ia : ib;
    }
    const R tmin = fm_min(fm_min(n1[0], n1[1]), n1[2]);
    out = INF;
    if (!(tmin < INF)) return true;
    const R best = fm_subsets<R>(s, n1, n2, tmin, nin[0], fin[0], nin[1], fin[1], nin[2], fin[2], sp, order2);
    const R hi = fm_fma<R>(best, R(kNear), best), lo = fm_fma<R>(best, R(-kNear), best);
    bool ok = best < INF;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        ok = ok && f1[a] - tmin >= hi && !(order2 && f2[a] < f1[a] && f1[a] < INF);
        ok = ok && !(order2 && n2[a] < n1[a] && n1[a] - tmin >= lo && n1[a] < INF);
    }
    out = tmin + best;
    return ok;
}

template <typename R>
FM_HD R fm_update(R s, const R t1[6], const R t2[6], unsigned inb, const Spacing<R> &sp, int order2)
{
    R v;
    return fm_update_near<R>(s, t1, t2, inb, sp, order2, v) ? v : fm_update_octants<R>(s, t1, t2, inb, sp, order2);
}

// ---------------------------------------------------------------------------
// Double precision, screened in single precision
// ---------------------------------------------------------------------------
//
// This GPU's double-precision pipe retires two lanes per SM and cycle, a
// sixty-fourth of the single-precision rate, and bounds every double-precision
// kernel: fm_update's eight octants take ~550 such operations a node (sixteen
// quadratics, each with a square root and a division of ~8 operations).  The
// node takes the least octant, so the octants are first solved in single
// precision, and only those that can be the least -- one or two, mostly -- are
// solved in double: the operations of the general update in its order, so
// the same bits, ~60 double-precision operations a node.  Rounds of a two-event
// 192x224x224 solve: 544 -> 161 ms, extra sweeps 146 -> 69 ms; the upstream-only
// update of a 64^3 main sweep (latency of one warp's chain) 3.4 -> 1.9 ms.
//
// An octant's screened value stands when every decision on the way to it is
// clear: each key differs from the solution it is compared with by more than
// kScreen of it, no discriminant is below 1/32 of its positive part, and no
// two keys so near that the sort could go the other way lead to different
// terms.  Terms are formed relative to tmin, discriminants as
//     a s^2 - sum_{i<j} w_i w_j (e_i - e_j)^2
// (the same b^2 - a c without its cancellation), so a value that stands is
// within ~1e-5 of the double-precision one (sqrt and division are within a few
// ulp, and a discriminant's relative error is at most ~32 times its terms');
// kScreen is twenty times that.  With m the least value that stands, an octant
// is solved in double unless it stands above m (1 + 2 kScreen), or starts
// there: its solution lies above its earliest key, every e being at least its
// key and the root above their weighted mean.  An octant whose three terms
// clearly all enter skips the pair's root too (it only decides that).
constexpr float kScreen = 1.0f / 4096.0f;

FM_HD unsigned long long fm_ubits(double v)
{
#ifdef __CUDA_ARCH__
    return (unsigned long long)__double_as_longlong(v);
#else
    unsigned long long b;
    __builtin_memcpy(&b, &v, sizeof b);
    return b;
#endif
}
// a < b of times (zero or above, +inf when unset; a NaN of either sign, as
// copied from outside the grid, is above all), on the integer pipe
FM_HD bool fm_less(double a, double b) { return fm_ubits(a) < fm_ubits(b); }

// A time difference (zero or above, or +inf) rounded down to single
// precision, on the integer pipe.
FM_HD float fm_narrow(double v)
{
    const unsigned long long b = fm_ubits(v);
    int h = (int)(b >> 32) - (896 << 20);            // exponent bias 1023 -> 127
    unsigned lo = (unsigned)b >> 29;
    if (h < 0) { h = 0; lo = 0; }
    if (h >= (255 << 20)) { h = 255 << 20; lo = 0; }
    const unsigned f = ((unsigned)h << 3) | lo;
#ifdef __CUDA_ARCH__
    return __uint_as_float(f);
#else
    float r;
    __builtin_memcpy(&r, &f, sizeof r);
    return r;
#endif
}

// One term of an octant in single precision: key, e, weight, one-term solution.
struct ScreenTerm {
    float k, e, w, x;
};

// The double-precision causal solve of one octant: terms in axis order, dt
// the keys, dd = t1 - t2 where the axis is second order (o2), h and w the
// spacings; three: all three terms are known to enter.  fm_update's
// operations in its order.
FM_HD double fm_octant(double s, const double dt[3], const double dd[3], unsigned o2, const Spacing<double> &sp,
                       bool three)
{
    double e[3], w[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const bool o = (o2 >> a) & 1u;
        e[a] = o ? fm_fma<double>(dd[a], 1.0 / 3.0, dt[a]) : dt[a];
        w[a] = o ? sp.w[a] * 2.25 : sp.w[a];
    }
    // the lateral pair in order, then the radial term inserted (ties keep the
    // order r, theta, phi)
    const bool p = fm_less(dt[2], dt[1]);
    const double kA = p ? dt[2] : dt[1], eA = p ? e[2] : e[1], wA = p ? w[2] : w[1];
    const double kB = p ? dt[1] : dt[2], eB = p ? e[1] : e[2], wB = p ? w[1] : w[2];
    const bool p1 = fm_less(kA, dt[0]);
    const double e0 = p1 ? eA : e[0], w0 = p1 ? wA : w[0];
    const double kM = p1 ? dt[0] : kA, eM = p1 ? e[0] : eA, wM = p1 ? w[0] : wA;
    const bool p2 = fm_less(kB, kM);
    const double k1 = p2 ? kB : kM, e1 = p2 ? eB : eM, w1 = p2 ? wB : wM;
    const double k2 = p2 ? kM : kB, e2 = p2 ? eM : eB, w2 = p2 ? wM : wB;
    // the first term's axis
    const double hf = p1 ? (p ? sp.h[2] : sp.h[1]) : sp.h[0];
    const bool of = ((p1 ? (p ? o2 >> 2 : o2 >> 1) : o2) & 1u) != 0;
    double x = fm_fma<double>(s, of ? hf * (2.0 / 3.0) : hf, e0);
    if (three || fm_less(k1, x)) {
        const double s2 = s * s;
        double a = w0 + w1;
        const double we0 = w0 * e0, we1 = w1 * e1;
        double b = we0 + we1;
        double c = fm_fma<double>(we0, e0, fm_fma<double>(we1, e1, -s2));
        if (!three) {
            const double disc = fm_fma<double>(b, b, -(a * c));
            x = (b + Fast<double>::sqrt(disc > 0.0 ? disc : 0.0)) / a;
            three = fm_less(k2, x);
        }
        if (three) {
            const double we2 = w2 * e2;
            a += w2;
            b += we2;
            c = fm_fma<double>(we2, e2, c);
            const double disc = fm_fma<double>(b, b, -(a * c));
            x = (b + Fast<double>::sqrt(disc > 0.0 ? disc : 0.0)) / a;
        }
    }
    return x;
}

// A pair's screened solve: its value x, whether its second term enters (on)
// and whether the value stands (ok); Q = w_i w_j (e_i - e_j)^2.
struct ScreenPair {
    float x, Q;
    bool on, ok;
};

FM_HD ScreenPair fm_screen_pair(float s2, const ScreenTerm &u, const ScreenTerm &v)
{
    ScreenPair r;
    const float A = u.w + v.w, B = fm_fma<float>(u.w, u.e, v.w * v.e), d = u.e - v.e;
    r.Q = u.w * v.w * d * d;
    const float D = fm_fma<float>(A, s2, -r.Q);
    const float x = Fast<float>::div(B + Fast<float>::sqrt(fm_max(D, 0.0f)), A);
    const float xf = v.k < u.k ? v.x : u.x, kl = fm_max(u.k, v.k), kf = fm_min(u.k, v.k);
    r.on = kl < xf;
    const bool clear = r.on ? kl < xf * (1.0f - kScreen) && D >= A * s2 * (1.0f / 32.0f) : kl > xf * (1.0f + kScreen);
    // (keys that the sort could exchange: the second has to enter either way)
    const bool tie = kl * (1.0f - kScreen) <= kf && !(kl * (1.0f + kScreen) < fm_min(u.x, v.x));
    r.ok = clear && !tie;
    r.x = r.on ? x : xf;
    return r;
}

// A triple's, from its pairs: x, whether it stands, whether all three terms
// enter.  (Which pair comes first matters for the decisions only; sums and
// discriminant are the same in any order.)
FM_HD bool fm_screen_triple(float s2, const ScreenTerm &a, const ScreenTerm &b, const ScreenTerm &c, const ScreenPair &ab,
                            const ScreenPair &ac, const ScreenPair &bc, float &x, bool &three)
{
    const float bcmax = fm_max(b.k, c.k);
    const bool al = bcmax < a.k, cb = c.k < b.k;             // a last; c before b
    const float kL = fm_max(a.k, bcmax), kM = al ? bcmax : fm_max(a.k, fm_min(b.k, c.k));
    const float x2 = al ? bc.x : (cb ? ac.x : ab.x);
    const bool on2 = al ? bc.on : (cb ? ac.on : ab.on);
    bool ok = al ? bc.ok : (cb ? ac.ok : ab.ok);
    const float A = a.w + b.w + c.w, B = fm_fma<float>(a.w, a.e, fm_fma<float>(b.w, b.e, c.w * c.e));
    const float D = fm_fma<float>(A, s2, -(ab.Q + ac.Q + bc.Q));
    const float x3 = Fast<float>::div(B + Fast<float>::sqrt(fm_max(D, 0.0f)), A);
    const bool on3 = on2 && kL < x2;
    if (on2)
        ok = ok && (on3 ? kL < x2 * (1.0f - kScreen) && D >= A * s2 * (1.0f / 32.0f) : kL > x2 * (1.0f + kScreen)) &&
             !(kL * (1.0f - kScreen) <= kM);
    x = on3 ? x3 : x2;
    three = on3 && ok;
    return ok;
}

// The seven subsets of three terms, screened (bits: 0 D, 1 X, 2 Z, 3 DX, 4 DZ,
// 5 XZ, 6 DXZ): those that can be the least among the ones in `in`; three:
// DXZ's three terms clearly enter.
FM_HD unsigned fm_screen7(float s, const ScreenTerm t[3], unsigned in, bool &three)
{
    const float INF = Lim<float>::inf();
    const float s2 = s * s;
    const ScreenPair p[3] = {fm_screen_pair(s2, t[0], t[1]), fm_screen_pair(s2, t[0], t[2]),
                             fm_screen_pair(s2, t[1], t[2])};
    float xt;
    const bool ok = fm_screen_triple(s2, t[0], t[1], t[2], p[0], p[1], p[2], xt, three);
    const float k0 = fm_min(fm_min(t[0].k, t[1].k), t[2].k);
    const float lo[7] = {t[0].x, t[1].x, t[2].x, p[0].ok ? p[0].x : fm_min(t[0].k, t[1].k),
                         p[1].ok ? p[1].x : fm_min(t[0].k, t[2].k), p[2].ok ? p[2].x : fm_min(t[1].k, t[2].k), ok ? xt : k0};
    const bool stands[7] = {true, true, true, p[0].ok, p[1].ok, p[2].ok, ok};
    float m = INF;
#pragma unroll
    for (int j = 0; j < 7; ++j) m = ((in >> j) & 1u) && stands[j] ? fm_min(m, lo[j]) : m;
    const float cut = m * (1.0f + 2.0f * kScreen);
    unsigned need = 0;
#pragma unroll
    for (int j = 0; j < 7; ++j) need |= lo[j] <= cut && lo[j] < INF ? 1u << j : 0u;
    return need & in;
}

// The least of the subsets in `need`, solved in double precision.
FM_HD double fm_solve7(double s, const double dt[3], const double dd[3], unsigned o2, const Spacing<double> &sp,
                       unsigned need, bool three)
{
    const double INF = Lim<double>::inf();
    double best = INF;
    while (need) {
        const unsigned bit = need & (0u - need);
        need ^= bit;
        // D in 0, 3, 4, 6; X in 1, 3, 5, 6; Z in 2, 4, 5, 6
        const double kt[3] = {(bit & 0x59u) ? dt[0] : INF, (bit & 0x6au) ? dt[1] : INF, (bit & 0x74u) ? dt[2] : INF};
        const double v = fm_octant(s, kt, dd, o2, sp, bit == 0x40u && three);
        best = fm_less(v, best) ? v : best;
    }
    return best;
}

// Which subsets' octants lie inside the grid: each takes the near side on its
// axes and the far side on the others (n, f: bit a of each).
FM_HD unsigned fm_inside7(unsigned n, unsigned f)
{
    unsigned in = 0;
    const unsigned sets[7] = {1u, 2u, 4u, 3u, 5u, 6u, 7u};
#pragma unroll
    for (int j = 0; j < 7; ++j) in |= (((n & sets[j]) | (f & ~sets[j])) & 7u) == 7u ? 1u << j : 0u;
    return in;
}

// One side's term: keys and differences in double, the screen's in single.
FM_HD void fm_side(float s, double t1, double t2, double tmin, double h, double w, int order2, double &dt, double &dd,
                   bool &o2, ScreenTerm &t)
{
    o2 = order2 && fm_less(t2, t1);
    dt = t1 - tmin;
    dd = o2 ? t1 - t2 : 0.0;
    const float hf = fm_narrow(h), wf = fm_narrow(w);
    t.k = fm_narrow(dt);
    t.e = o2 ? fm_fma<float>(fm_narrow(dd), 1.0f / 3.0f, t.k) : t.k;
    t.w = o2 ? wf * 2.25f : wf;
    t.x = fm_fma<float>(s, o2 ? hf * (2.0f / 3.0f) : hf, t.e);
}

// fm_update in double precision: all eight octants screened, in straight-line
// code that shares the twelve pairs (an octant's value is its triple's), then
// those that can be the least solved in double.  (The short form with a
// fallback loses here: along a near tie's axis a warp seldom has all lanes
// in it, and both forms run -- rounds and extra sweeps of the two-event
// 192x224x224 solve 192 and 93 ms against 157 and 57.)
template <>
FM_HD double fm_update<double>(double s, const double t1[6], const double t2[6], unsigned inb,
                               const Spacing<double> &sp, int order2)
{
    const double INF = Lim<double>::inf();
    const float INFF = Lim<float>::inf();
    double tmin = INF;
#pragma unroll
    for (int d = 0; d < 6; ++d) tmin = fm_less(t1[d], tmin) ? t1[d] : tmin;
    if (!fm_less(tmin, INF)) return INF;
    const float sf = fm_narrow(s), s2 = sf * sf;
    double dt[6], dd[6];
    unsigned o2 = 0;
    ScreenTerm t[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        bool o;
        fm_side(sf, t1[d], t2[d], tmin, sp.h[d >> 1], sp.w[d >> 1], order2, dt[d], dd[d], o, t[d]);
        o2 |= o ? 1u << d : 0u;
    }
    // pairs of sides: radial with theta, radial with phi, theta with phi
    ScreenPair rx[4], rz[4], xz[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        rx[q] = fm_screen_pair(s2, t[q & 1], t[2 + (q >> 1)]);
        rz[q] = fm_screen_pair(s2, t[q & 1], t[4 + (q >> 1)]);
        xz[q] = fm_screen_pair(s2, t[2 + (q & 1)], t[4 + (q >> 1)]);
    }
    // octant q: bit 0 the radial side, bit 1 theta, bit 2 phi; the least value
    // each can have, as far as the screen tells
    float lo[8], m = INFF;
    unsigned three = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int r = q & 1, x = (q >> 1) & 1, z = q >> 2;
        const unsigned om = (1u << r) | (4u << x) | (16u << z);
        float v;
        bool th;
        const bool ok = fm_screen_triple(s2, t[r], t[2 + x], t[4 + z], rx[r | x << 1], rz[r | z << 1], xz[x | z << 1], v, th);
        const float k0 = fm_min(fm_min(t[r].k, t[2 + x].k), t[4 + z].k);
        const bool in = (inb & om) == om;
        lo[q] = in ? (ok ? v : k0) : INFF;
        m = in && ok ? fm_min(m, v) : m;
        three |= th ? 1u << q : 0u;
    }
    // (an octant outside the grid, or with no neighbour set, has lo = +inf)
    const float cut = m * (1.0f + 2.0f * kScreen);
    unsigned need = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) need |= lo[q] <= cut && lo[q] < INFF ? 1u << q : 0u;
    double best = INF;
    while (need) {
        const unsigned bit = need & (0u - need);
        need ^= bit;
        const bool r = (bit & 0xaau) != 0, x = (bit & 0xccu) != 0, z = (bit & 0xf0u) != 0;
        const double kt[3] = {r ? dt[1] : dt[0], x ? dt[3] : dt[2], z ? dt[5] : dt[4]};
        const double kd[3] = {r ? dd[1] : dd[0], x ? dd[3] : dd[2], z ? dd[5] : dd[4]};
        const unsigned oo = ((o2 >> (r ? 1 : 0)) & 1u) | (((o2 >> (x ? 3 : 2)) & 1u) << 1) |
                            (((o2 >> (z ? 5 : 4)) & 1u) << 2);
        const double v = fm_octant(s, kt, kd, oo, sp, (three & bit) != 0);
        best = fm_less(v, best) ? v : best;
    }
    return tmin + best;
}

template <>
FM_HD double fm_update_upstream<double>(double s, double tD, double tD2, double tX, double tX2, double tZ, double tZ2,
                                        bool inD, bool inU, bool inXu, bool inXd, bool inZu, bool inZd,
                                        const Spacing<double> &sp, int order2)
{
    const double INF = Lim<double>::inf();
    double tmin = fm_less(tX, tD) ? tX : tD;
    tmin = fm_less(tZ, tmin) ? tZ : tmin;
    if (!fm_less(tmin, INF)) return INF;
    const double t1[3] = {tD, tX, tZ}, t2[3] = {tD2, tX2, tZ2};
    const float sf = fm_narrow(s);
    double dt[3], dd[3];
    unsigned o2 = 0;
    ScreenTerm t[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        bool o;
        fm_side(sf, t1[a], t2[a], tmin, sp.h[a], sp.w[a], order2, dt[a], dd[a], o, t[a]);
        o2 |= o ? 1u << a : 0u;
    }
    bool three;
    const unsigned n = (inD ? 1u : 0u) | (inXu ? 2u : 0u) | (inZu ? 4u : 0u);
    const unsigned f = (inU ? 1u : 0u) | (inXd ? 2u : 0u) | (inZd ? 4u : 0u);
    const unsigned need = fm_screen7(sf, t, fm_inside7(n, f), three);
    return tmin + fm_solve7(s, dt, dd, o2, sp, need, three);
}

}  // namespace fm3dt
