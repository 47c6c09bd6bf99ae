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
template <typename R>
FM_HD R fm_update(R s, const R t1[6], const R t2[6], unsigned inb, const Spacing<R> &sp, int order2)
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
// grid.  It evaluates the seven subsets with four quadratic solves instead of
// the eight octants' sixteen: the singletons are one FMA each, the three pairs
// one solve each, and the triple's first two terms are one of the pairs (the
// same order and the same operations, hence the same bits), so only its
// three-term solve is added.  The four solves are straight-line code with
// selects at the end: a sweep's few warps wait on each other, and three pairs
// solved side by side are a third of the chain of three branches (main sweep of
// one 64^3 event 300 -> 228 us; of 500 events on 192x224x224, bound by issue,
// 50.6 -> 42.4 ms: 341 -> 295 instructions a step).  Sums of two are the same in
// either order; only the innermost FMA of a pair's c depends on which term
// comes first.
//
// tD/tD2, tX/tX2, tZ/tZ2: upstream first and second neighbour values;
// in*: whether each upstream (u) and downstream (d) neighbour lies inside the
// grid (inD: r+1, inU: r-1).
template <typename R>
FM_HD R fm_update_upstream(R s, R tD, R tD2, R tX, R tX2, R tZ, R tZ2, bool inD, bool inU, bool inXu, bool inXd,
                           bool inZu, bool inZd, const Spacing<R> &sp, int order2)
{
    const R INF = Lim<R>::inf();
    const R tmin = fm_min(fm_min(tD, tX), tZ);
    const R s2 = s * s;
    // (with an unset neighbour, or all of them, differences are +inf or NaN:
    // no comparison lets them in, and an unset tmin is selected at the end)
    R k[3], e[3], w[3], we[3], x1[3], q[3];
    {
        const R t1[3] = {tD, tX, tZ}, t2[3] = {tD2, tX2, tZ2};
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
    // unset and r-1 inside, inD may be passed as true: the octants with D then
    // give what those with r-1 give.)
    R best = INF;
    best = inD && inXd && inZd ? fm_min(best, x1[0]) : best;
    best = inU && inXu && inZd ? fm_min(best, x1[1]) : best;
    best = inU && inXd && inZu ? fm_min(best, x1[2]) : best;
    best = inD && inXu && inZd ? fm_min(best, xp[0]) : best;
    best = inD && inXd && inZu ? fm_min(best, xp[1]) : best;
    best = inU && inXu && inZu ? fm_min(best, xp[2]) : best;
    best = inD && inXu && inZu ? fm_min(best, xt) : best;
    return tmin < INF ? tmin + best : INF;
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

// One term of an octant: key, e, spacing and weight, in single precision.
struct ScreenTerm {
    float k, e, g, w;
};

// An octant's (or subset's) screened value: x; whether it stands; whether all
// three terms enter; its earliest key.
struct Screened {
    float x, k0;
    bool stands, three;
};

FM_HD void fm_screen_swap(ScreenTerm &a, ScreenTerm &b)
{
    const bool p = b.k < a.k;
    const ScreenTerm t = a;
    a.k = p ? b.k : a.k; a.e = p ? b.e : a.e; a.g = p ? b.g : a.g; a.w = p ? b.w : a.w;
    b.k = p ? t.k : b.k; b.e = p ? t.e : b.e; b.g = p ? t.g : b.g; b.w = p ? t.w : b.w;
}

// a, b, c sorted by key
FM_HD Screened fm_screen(float s, float s2, const ScreenTerm &a, const ScreenTerm &b, const ScreenTerm &c)
{
    Screened r;
    r.k0 = a.k;
    const float x0 = fm_fma<float>(s, a.g, a.e);
    float x = x0;
    bool three = false;
    // the second term clearly out, or clearly in whichever of the first two
    // comes first
    bool in2 = b.k < x0;
    bool ok = in2 ? b.k < x0 * (1.0f - kScreen) : b.k > x0 * (1.0f + kScreen);
    const bool near01 = b.k * (1.0f - kScreen) <= a.k;
    ok = ok && !(near01 && !(b.k * (1.0f + kScreen) < fm_min(x0, fm_fma<float>(s, b.g, b.e))));
    if (in2) {
        const float A = a.w + b.w, B = fm_fma<float>(a.w, a.e, b.w * b.e);
        const float d01 = a.e - b.e, q01 = a.w * b.w * d01 * d01;
        const float D = A * s2 - q01;
        x = Fast<float>::div(B + Fast<float>::sqrt(fm_max(D, 0.0f)), A);
        ok = ok && D >= A * s2 * (1.0f / 32.0f);
        three = c.k < x;
        ok = ok && (three ? c.k < x * (1.0f - kScreen) : c.k > x * (1.0f + kScreen));
        const bool near12 = c.k * (1.0f - kScreen) <= b.k;
        ok = ok && !(near12 && (b.e != b.k || c.e != c.k));
        if (three) {
            const float A3 = A + c.w, B3 = fm_fma<float>(c.w, c.e, B);
            const float d02 = a.e - c.e, d12 = b.e - c.e;
            const float D3 = A3 * s2 - (q01 + c.w * (a.w * d02 * d02 + b.w * d12 * d12));
            x = Fast<float>::div(B3 + Fast<float>::sqrt(fm_max(D3, 0.0f)), A3);
            ok = ok && D3 >= A3 * s2 * (1.0f / 32.0f);
        }
    }
    r.x = x;
    r.stands = ok;                                    // (false for NaN)
    r.three = three && ok;
    return r;
}

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

template <>
FM_HD double fm_update<double>(double s, const double t1[6], const double t2[6], unsigned inb,
                               const Spacing<double> &sp, int order2)
{
    const double INF = Lim<double>::inf();
    double tmin = INF;
#pragma unroll
    for (int d = 0; d < 6; ++d) tmin = fm_less(t1[d], tmin) ? t1[d] : tmin;
    if (!fm_less(tmin, INF)) return INF;
    float hf[3], wf[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        hf[a] = fm_narrow(sp.h[a]);
        wf[a] = fm_narrow(sp.w[a]);
    }
    const float sf = fm_narrow(s), s2f = sf * sf;
    double dt[6], dd[6];
    unsigned o2 = 0;
    ScreenTerm t[6];
#pragma unroll
    for (int d = 0; d < 6; ++d) {
        const int a = d >> 1;
        const bool o = order2 && fm_less(t2[d], t1[d]);
        dt[d] = t1[d] - tmin;
        dd[d] = o ? t1[d] - t2[d] : 0.0;
        o2 |= o ? 1u << d : 0u;
        t[d].k = fm_narrow(dt[d]);
        t[d].e = o ? fm_fma<float>(fm_narrow(dd[d]), 1.0f / 3.0f, t[d].k) : t[d].k;
        t[d].g = o ? hf[a] * (2.0f / 3.0f) : hf[a];
        t[d].w = o ? wf[a] * 2.25f : wf[a];
    }
    // octant q: bit 0 the radial side, bit 1 theta, bit 2 phi
    float lo[8];           // least value the octant can have, as far as the screen tells
    unsigned three = 0;
    float m = Lim<float>::inf();
#pragma unroll
    for (int lat = 0; lat < 4; ++lat) {
        ScreenTerm a = t[2 + (lat & 1)], b = t[4 + (lat >> 1)];
        fm_screen_swap(a, b);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int q = r | (lat << 1);
            const unsigned om = (1u << r) | (4u << (lat & 1)) | (16u << (lat >> 1));
            ScreenTerm x = t[r], y = a, z = b;
            fm_screen_swap(x, y);
            fm_screen_swap(y, z);
            const Screened v = fm_screen(sf, s2f, x, y, z);
            const bool in = (inb & om) == om;
            lo[q] = in ? (v.stands ? v.x : v.k0) : Lim<float>::inf();
            m = in && v.stands ? fm_min(m, v.x) : m;
            three |= v.three ? 1u << q : 0u;
        }
    }
    // (an octant outside the grid, or with no neighbour set, has lo = +inf)
    const float cut = m * (1.0f + 2.0f * kScreen);
    unsigned need = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) need |= lo[q] <= cut && lo[q] < Lim<float>::inf() ? 1u << q : 0u;
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

// The upstream-only update, screened likewise over its seven subsets (bit 0
// down, bit 1 theta, bit 2 phi).
template <>
FM_HD double fm_update_upstream<double>(double s, double tD, double tD2, double tX, double tX2, double tZ, double tZ2,
                                        bool inD, bool inU, bool inXu, bool inXd, bool inZu, bool inZd,
                                        const Spacing<double> &sp, int order2)
{
    const double INF = Lim<double>::inf();
    const float INFF = Lim<float>::inf();
    double tmin = fm_less(tX, tD) ? tX : tD;
    tmin = fm_less(tZ, tmin) ? tZ : tmin;
    if (!fm_less(tmin, INF)) return INF;
    const double t1[3] = {tD, tX, tZ}, t2[3] = {tD2, tX2, tZ2};
    const float sf = fm_narrow(s), s2f = sf * sf;
    double dt[3], dd[3];
    unsigned o2 = 0;
    ScreenTerm t[3];
    float x1[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const bool o = order2 && fm_less(t2[a], t1[a]);
        dt[a] = t1[a] - tmin;
        dd[a] = o ? t1[a] - t2[a] : 0.0;
        o2 |= o ? 1u << a : 0u;
        const float h = fm_narrow(sp.h[a]), w = fm_narrow(sp.w[a]);
        t[a].k = fm_narrow(dt[a]);
        t[a].e = o ? fm_fma<float>(fm_narrow(dd[a]), 1.0f / 3.0f, t[a].k) : t[a].k;
        t[a].g = o ? h * (2.0f / 3.0f) : h;
        t[a].w = o ? w * 2.25f : w;
        x1[a] = fm_fma<float>(sf, t[a].g, t[a].e);
    }
    float lo[7];
    unsigned three = 0;
    float m = INFF;
    // singles stand as they are
    const bool c1[3] = {inD && inXd && inZd, inU && inXu && inZd, inU && inXd && inZu};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = c1[a] ? x1[a] : INFF;
        m = fm_min(m, lo[a]);
    }
    const ScreenTerm none = {INFF, INFF, 1.0f, 1.0f};
    const bool c2[4] = {inD && inXu && inZd, inD && inXd && inZu, inU && inXu && inZu, inD && inXu && inZu};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        // DX, DZ, XZ, DXZ
        ScreenTerm x = t[j == 2 ? 1 : 0], y = t[j == 0 || j == 3 ? 1 : 2], z = j == 3 ? t[2] : none;
        if (j == 3) fm_screen_swap(y, z);
        fm_screen_swap(x, y);
        if (j == 3) fm_screen_swap(y, z);
        const Screened v = fm_screen(sf, s2f, x, y, z);
        lo[3 + j] = c2[j] ? (v.stands ? v.x : v.k0) : INFF;
        m = c2[j] && v.stands ? fm_min(m, v.x) : m;
        if (j == 3 && v.three) three = 1;
    }
    const float cut = m * (1.0f + 2.0f * kScreen);
    unsigned need = 0;
#pragma unroll
    for (int j = 0; j < 7; ++j) need |= lo[j] <= cut && lo[j] < INFF ? 1u << j : 0u;
    double best = INF;
    while (need) {
        const unsigned bit = need & (0u - need);
        need ^= bit;
        // D in 0, 3, 4, 6; X in 1, 3, 5, 6; Z in 2, 4, 5, 6
        const double kt[3] = {(bit & 0x59u) ? dt[0] : INF, (bit & 0x6au) ? dt[1] : INF, (bit & 0x74u) ? dt[2] : INF};
        const double v = fm_octant(s, kt, dd, o2, sp, bit == 0x40u && three);
        best = fm_less(v, best) ? v : best;
    }
    return tmin + best;
}

}  // namespace fm3dt
