// Host check of the halo reads of the main sweep (front.cuh front_kernel).
//
// One warp's wait loop over its halo ring is restated: each step copies the
// halo layers used AHEAD steps later into a ring row (halo_layers.h says which
// layers the grid has), then polls the columns whose value is unwritten.  The
// blocks upstream write their columns' first `upto` layers and then never
// again, so a wait gives up, and leaves unset what it waited for.  No copy and
// no poll may read a layer the grid does not have, the sweep has to end, and
// the values it uses have to be settled ones.  If a wait that gives up leaves
// its row as it is, the same loop reads layers above the grid, so the check can
// tell.
//
//   g++ -O2 -std=c++17 halo_layers_check.cpp -o check && ./check
#include <algorithm>
#include <cstdio>
#include <vector>

#include "../parallel-fast-marching-method_gb300/csrc/halo_layers.h"

namespace {

constexpr int kAhead = 4, kPolls = 3;
enum { kUnset, kUnwritten, kWritten };

struct Found {
    long long reads = 0, outside = 0, used = 0, unsettled = 0;
};

// the columns of one side (n of them) of a block of sx x sz columns
void sweep(int sx, int sz, bool skew, int n, int nnr, int upto, bool clear, Found &f)
{
    const int lag = sx + sz - 2, ring = lag + kAhead + 2 <= 16 ? 16 : 32;
    std::vector<int> rows(ring * n, kUnset);
    bool gave_up = false;
    auto read = [&](int layer) {
        ++f.reads;
        if (layer < 0 || layer >= nnr) ++f.outside;
        return layer < upto ? kWritten : kUnwritten;
    };
    auto late = [&](int q) { return skew ? q : 0; };
    auto fetch = [&](int t) {
        for (int q = 0; q < n; ++q)
            if (fm3dt::halo_layer_in(t, late(q), nnr)) rows[(t % ring) * n + q] = read(t - late(q));
    };
    for (int t = 0; t < kAhead; ++t) fetch(t);
    for (int t = 0; t < nnr + lag; ++t) {
        fetch(t + kAhead);
        for (int polls = 0;;) {
            bool wait = false;
            for (int q = 0; q < n; ++q) wait = wait || rows[(t % ring) * n + q] == kUnwritten;
            if (!wait) break;
            // (the error that another wait raised is seen every other poll)
            const bool give_up = ++polls > kPolls || (polls % 2 == 0 && gave_up);
            for (int q = 0; q < n; ++q) {
                int &v = rows[(t % ring) * n + q];
                if (v != kUnwritten) continue;
                if (!give_up)
                    v = read(t - late(q));
                else if (clear)
                    v = kUnset;
            }
            if (give_up) {
                gave_up = true;
                break;
            }
        }
        // what lane (column q, d columns into the block) reads in step t
        for (int q = 0; q < n; ++q) {
            const int rp = t - q;
            if (rp < 0 || rp >= nnr) continue;
            ++f.used;
            if (rows[((skew ? t : rp) % ring) * n + q] == kUnwritten) ++f.unsettled;
        }
    }
}

}  // namespace

int main()
{
    const int shapes[2][2] = {{4, 8}, {2, 16}};
    Found with, without;
    for (auto &s : shapes)
        for (int skew = 0; skew < 2; ++skew)
            for (int side = 0; side < 2; ++side)
                for (int nnr = 1; nnr <= 70; ++nnr)
                    for (int upto = 0; upto <= nnr; ++upto) {
                        sweep(s[0], s[1], skew, s[side], nnr, upto, true, with);
                        sweep(s[0], s[1], skew, s[side], nnr, upto, false, without);
                    }
    std::printf("%lld reads, %lld outside, %lld values used, %lld unsettled; left as they are, %lld outside\n", with.reads,
                with.outside, with.used, with.unsettled, without.outside);
    return with.outside == 0 && with.unsettled == 0 && without.outside > 0 ? 0 : 1;
}
