// Host check of the double-precision node update's single-precision screen
// (stencil.cuh): fm_update<double> and fm_update_upstream<double> against a
// plain restatement that solves every octant in double precision, bit for
// bit, where the screen's decisions are close: keys that differ by 1e-15 to
// 1e-1 of each other, second neighbours next to the first ones, keys far
// above the others, times of several hundred seconds, unset neighbours and
// neighbours outside the grid, equal and very unequal spacings, both orders.
//
//   g++ -O2 -std=c++17 -ffp-contract=off screened_update_check.cpp -o check && ./check cases seed
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "../parallel-fast-marching-method_gb300/csrc/stencil.cuh"

using fm3dt::Spacing;

static double plain(double s, const double t1[6], const double t2[6], unsigned inb, const Spacing<double> &sp,
                    int order2)
{
    double tmin = INFINITY, best = INFINITY;
    for (int d = 0; d < 6; ++d)
        if (((inb >> d) & 1u) && t1[d] < tmin) tmin = t1[d];
    if (!(tmin < INFINITY)) return INFINITY;
    for (int o = 0; o < 8; ++o) {
        double k[3], e[3], g[3], w[3];
        bool in = true;
        for (int a = 0; a < 3; ++a) {
            const int d = 2 * a + ((o >> a) & 1);
            in = in && ((inb >> d) & 1u);
            const bool o2 = order2 && t2[d] < t1[d];
            k[a] = t1[d] - tmin;
            e[a] = o2 ? std::fma(t1[d] - t2[d], 1.0 / 3.0, k[a]) : k[a];
            g[a] = o2 ? sp.h[a] * (2.0 / 3.0) : sp.h[a];
            w[a] = o2 ? sp.w[a] * 2.25 : sp.w[a];
        }
        if (!in) continue;
        for (const auto &p : {std::pair<int, int>{0, 1}, {1, 2}, {0, 1}})
            if (k[p.second] < k[p.first]) {
                std::swap(k[p.first], k[p.second]); std::swap(e[p.first], e[p.second]);
                std::swap(g[p.first], g[p.second]); std::swap(w[p.first], w[p.second]);
            }
        double x = std::fma(s, g[0], e[0]);
        double A = w[0], B = w[0] * e[0], C = 0.0;
        for (int n = 1; n < 3 && k[n] < x; ++n) {
            const double we = w[n] * e[n];
            C = n == 1 ? std::fma(B, e[0], std::fma(we, e[1], -(s * s))) : std::fma(we, e[2], C);
            A += w[n];
            B += we;
            const double disc = std::fma(B, B, -(A * C));
            x = (B + std::sqrt(disc > 0.0 ? disc : 0.0)) / A;
        }
        if (x < best) best = x;
    }
    return tmin + best;
}

int main(int argc, char **argv)
{
    const long n = argc > 1 ? std::atol(argv[1]) : 100000;
    std::mt19937_64 rng(argc > 2 ? std::atol(argv[2]) : 1);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    const double near[6] = {1e-1, 3e-3, 3e-4, 1e-6, 1e-12, 1e-15};
    long bad = 0, bad_up = 0;
    for (long it = 0; it < n; ++it) {
        const double base = (rng() & 1) ? 600.0 : 3.0, ep = near[rng() % 6];
        const double c0 = U(rng), far = (rng() & 3) ? 1.0 : std::pow(10.0, 3.0 * U(rng));
        const double cs[4] = {0.0, c0, c0 * (1 + ep * (U(rng) - 0.5)), (rng() & 1) ? U(rng) : c0 * (1 + ep * (U(rng) - 0.5))};
        double t1[6], t2[6];
        for (int d = 0; d < 6; ++d) {
            const double k = cs[rng() % 4] * (rng() % 4 ? 1.0 : far);
            t1[d] = rng() % 15 ? base + k : INFINITY;
            const int z = (int)(rng() % 3);
            t2[d] = z == 0 ? base + k - 0.8 * U(rng) * (rng() % 5 ? 1.0 : far) : z == 1 ? base + k + (U(rng) - 0.5) * ep : INFINITY;
            if (t2[d] < 0.0) t2[d] = 0.0;
        }
        const unsigned inb = rng() % 4 ? 63u : (unsigned)(rng() & 63);
        for (int d = 0; d < 6; ++d)
            if (!((inb >> d) & 1u)) {
                t1[d] = (rng() & 1) ? INFINITY : (rng() & 1) ? NAN : -NAN;
                t2[d] = (rng() & 1) ? INFINITY : NAN;
            }
        Spacing<double> sp;
        for (int a = 0; a < 3; ++a) {
            sp.h[a] = (rng() & 3) ? 0.5 + 2.5 * U(rng) : (rng() & 1) ? 1.0 : 0.05 + 8.0 * U(rng);
            sp.w[a] = 1.0 / (sp.h[a] * sp.h[a]);
        }
        const double s = 0.1 + U(rng);
        const int order2 = (int)(rng() & 1);
        double want = plain(s, t1, t2, inb, sp, order2), got = fm3dt::fm_update<double>(s, t1, t2, inb, sp, order2);
        bad += std::memcmp(&want, &got, sizeof want) != 0;
        // upstream only: down, and the lateral sides a sweep comes from
        const int dX = 2 + (int)(rng() & 1), dZ = 4 + (int)(rng() & 1);
        for (const int d : {1, 0, dX, dX ^ 1, dZ, dZ ^ 1}) {
            if (d == 0 || d == (dX ^ 1) || d == (dZ ^ 1) || !((inb >> d) & 1u)) t1[d] = INFINITY;
            if (!((inb >> d) & 1u)) t2[d] = INFINITY;
        }
        want = plain(s, t1, t2, inb, sp, order2);
        auto in = [&](int d) { return ((inb >> d) & 1u) != 0; };
        got = fm3dt::fm_update_upstream<double>(s, t1[1], t2[1], t1[dX], t2[dX], t1[dZ], t2[dZ], in(1), in(0), in(dX),
                                                in(dX ^ 1), in(dZ), in(dZ ^ 1), sp, order2);
        bad_up += std::memcmp(&want, &got, sizeof want) != 0;
    }
    std::printf("update mismatches %ld, upstream mismatches %ld of %ld\n", bad, bad_up, n);
    return bad || bad_up;
}
