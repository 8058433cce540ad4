// The search of va_autotune over the launch shapes of the two sweeps.  Host code
// without CUDA, so it is checked on its own (tests/test_tune.py).
#pragma once

#include <algorithm>
#include <vector>

namespace va {

// A sweep's launch shape: threads per block and resident blocks per SM, or (0, 0),
// the default shape with what comes with it (resting).
struct Shape {
    int block = 0, bps = 0;
    int threads() const { return block * bps; }
};
struct ShapePair {
    Shape fwd, bwd;
};

// The pair of shapes that the sweeps together run fastest in.
// run(fwd, bwd, tf, tb) times one pair and returns whether that worked.
//
// Not the best of each sweep by itself: the forward's shape decides how the
// records lie that the backward reads.  262,144 double-word Van der Pol instances:
// forward 2.69 ms with 640 threads per SM, 2.82 with 512, but the backward at the
// same shape of its own 2.32 after the one and 2.20 after the other.  So every
// shape is first timed for both sweeps at once, then the pairs of each sweep's
// three best, no two with the same number of threads per SM, and the default.  The
// default stays unless a pair is 1% faster, twice what two runs of it differ by.
template <class Run>
bool tune_pair(const std::vector<Shape> &shapes, Run run, ShapePair &best)
{
    constexpr int kBest = 3;
    struct Timed {
        Shape s;
        float f, b;
    };
    best = ShapePair{};
    float base_f, base_b; // the second time: the first also orders the batch by its lengths
    for (int k = 0; k < 2; k++)
        if (!run(Shape{}, Shape{}, base_f, base_b))
            return false;
    float best_t = 0.99f * (base_f + base_b);
    std::vector<Timed> all;
    for (const Shape &s : shapes) {
        Timed t{s, 0.0f, 0.0f};
        if (!run(s, s, t.f, t.b))
            return false;
        all.push_back(t);
    }
    auto top = [&](auto less) {
        std::vector<Timed> sorted(all);
        std::stable_sort(sorted.begin(), sorted.end(), less);
        std::vector<Shape> out{Shape{}};
        for (const Timed &t : sorted)
            if ((int)out.size() <= kBest && std::none_of(out.begin(), out.end(), [&](const Shape &o) {
                    return o.threads() == t.s.threads();
                }))
                out.push_back(t.s);
        return out;
    };
    const std::vector<Shape> fs = top([](const Timed &x, const Timed &y) { return x.f < y.f; });
    const std::vector<Shape> bs = top([](const Timed &x, const Timed &y) { return x.b < y.b; });
    for (const Shape &f : fs)
        for (const Shape &b : bs) {
            if (!f.block && !b.block)
                continue;
            float tf, tb;
            if (!run(f, b, tf, tb))
                return false;
            if (tf + tb < best_t) {
                best_t = tf + tb;
                best = {f, b};
            }
        }
    return true;
}

} // namespace va
