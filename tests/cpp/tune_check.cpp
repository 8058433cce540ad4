// tune_pair (va_tune.h) on made-up times.  Prints one line per case: the chosen
// shapes and how many pairs were timed.
#include <cstdio>

#include "../../vectorizedadjoint_gb300/csrc/va_tune.h"

using va::Shape;

static std::vector<Shape> shapes()
{
    std::vector<Shape> v;
    for (int block : {64, 128, 256})
        for (int bps = 1; block * bps <= 640; bps++)
            v.push_back({block, bps});
    return v;
}

template <class F>
static void report(const char *name, F time)
{
    int runs = 0;
    va::ShapePair p;
    const bool ok = va::tune_pair(
        shapes(), [&](Shape f, Shape b, float &tf, float &tb) { return runs++, time(f, b, tf, tb); }, p);
    std::printf("%s %d %d %d %d %d %s\n", name, p.fwd.block, p.fwd.bps, p.bwd.block, p.bwd.bps, ok,
                runs <= (int)shapes().size() + 17 ? "few" : "many");
}

static float far(int threads, int from) { return 0.002f * (threads > from ? threads - from : from - threads); }

int main()
{
    // the forward's best shape by itself (640 threads) costs the backward more than it gains
    report("coupled", [](Shape f, Shape b, float &tf, float &tb) {
        const int ft = f.block ? f.threads() : 640, bt = b.block ? b.threads() : 512;
        tf = ft == 640 ? 2.70f : 2.75f + far(ft, 512);
        tb = (ft == 640 ? 2.32f : 2.20f) + far(bt, 512);
        return true;
    });
    // nothing is faster than the default by more than 1%
    report("default", [](Shape f, Shape b, float &tf, float &tb) {
        tf = f.block ? 1.0f + far(f.threads(), 256) : 1.005f;
        tb = b.block ? 1.0f + far(b.threads(), 384) : 1.005f;
        return true;
    });
    // each sweep has a best shape of its own
    report("apart", [](Shape f, Shape b, float &tf, float &tb) {
        tf = f.block ? 1.0f + far(f.threads(), 256) : 1.5f;
        tb = b.block ? 1.0f + far(b.threads(), 384) : 1.5f;
        return true;
    });
    // the default forward with another backward
    report("half", [](Shape f, Shape b, float &tf, float &tb) {
        tf = f.block ? 1.2f : 1.0f;
        tb = b.block ? 1.0f + far(b.threads(), 128) : 1.5f;
        return true;
    });
    int left = 5;
    report("fails", [&](Shape, Shape, float &tf, float &tb) {
        tf = tb = 1.0f;
        return left-- > 0;
    });
    return 0;
}
