// Locator (prefix table) against a scan of all leaves: random forests, some refined to
// the finest level along one path, periodic or not; points inside, on edges and outside.
#include <cstdio>
#include <random>

#include "../forestclaw_b200/csrc/fcb_forest.hpp"

using fcb::Leaf;
using fcb::QuadForest;

static int scan(const QuadForest& f, int32_t x, int32_t y) {
    if (!f.wrap(x, y)) return -1;
    for (size_t p = 0; p < f.leaves.size(); ++p) {
        const Leaf& l = f.leaves[p];
        const int64_t h = QuadForest::width(l.level);
        if (x >= l.x && y >= l.y && x < l.x + h && y < l.y + h) return (int)p;
    }
    return -2;
}

template <class WHICH>
static void refine(QuadForest& f, WHICH which) {
    std::vector<Leaf> out;
    for (size_t p = 0; p < f.leaves.size(); ++p) {
        const Leaf& l = f.leaves[p];
        if (l.level < QuadForest::kMaxLevel && which(p)) {
            const int32_t h = QuadForest::width(l.level + 1);
            for (int k = 0; k < 4; ++k) out.push_back(QuadForest::make(l.level + 1, l.x + (k & 1) * h, l.y + (k >> 1) * h));
        } else {
            out.push_back(l);
        }
    }
    f.leaves = out;
}

int main() {
    std::mt19937 r(1);
    long bad = 0, points = 0;
    for (int it = 0; it < 60; ++it) {
        QuadForest f;
        f.periodic_x = r() & 1;
        f.periodic_y = r() & 1;
        f.uniform((int)(r() % 4));
        for (int k = 0; k < 1 + it % 5; ++k) refine(f, [&](size_t) { return r() % 5 == 0; });
        if (it % 7 == 0)
            for (int k = 0; k < 26; ++k) {
                const size_t mid = f.leaves.size() / 2;
                refine(f, [&](size_t p) { return p == mid; });
            }
        const QuadForest::Locator at(f);
        for (int k = 0; k < 1000; ++k) {
            int32_t x = (int32_t)(r() % (QuadForest::kRoot + 200)) - 100, y = (int32_t)(r() % (QuadForest::kRoot + 200)) - 100;
            if (k % 2) {
                const Leaf& l = f.leaves[r() % f.leaves.size()];
                const int32_t h = QuadForest::width(l.level);
                x = l.x + ((int)(r() % 3) - 1) * ((r() & 1) ? h : 1);
                y = l.y + ((int)(r() % 3) - 1) * ((r() & 1) ? h : 1);
            }
            ++points;
            bad += at.locate(x, y) != scan(f, x, y);
        }
        // the balanced forest has neighbours of at most one level's difference everywhere
        // (neighbors() throws otherwise)
        f.balance();
        const QuadForest::Locator bal(f);
        for (size_t p = 0; p < f.leaves.size(); ++p) f.neighbors((int)p, bal);
    }
    std::printf("%ld wrong of %ld\n", bad, points);
    return bad != 0;
}
