// split_digits_in_place (va_contract.cuh) against split_digits on the host: the
// same digits with their weights, for normalised double-words.  Prints the number
// of pairs that differ and of pairs tried.
#include <cmath>
#include <cstdio>
#include <random>

#include "../../vectorizedadjoint_gb300/csrc/va_contract.cuh"

static long tried, differ;

static void check(double x, int e)
{
    const float hi = (float)x, lo = (float)(x - (double)hi);
    if (!(std::fabs((double)hi + (double)lo) < std::ldexp(1.0, e)))
        return;
    float d[4], w[4];
    const va::DigitScale sc = va::digit_scale(e);
    va::split_digits<4>(hi, lo, sc, d);
    va::split_digits_in_place(hi, lo, sc, w);
    bool same = true;
    for (int s = 0; s < 4; s++)
        same = same && w[s] == std::ldexp(d[s], -8 * s);
    tried++;
    differ += same ? 0 : 1;
}

int main()
{
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    for (int e : {-120, -119, -118, -60, -1, 0, 1, 37, 100}) {
        const double top = std::ldexp(1.0, e);
        for (int k = 0; k < 200000; k++) {
            check(u(rng) * top, e);
            check(u(rng) * top * std::ldexp(1.0, -(int)(rng() % 60)), e); // far below the column's maximum
        }
        // halves and steps of every digit, and what lies next to them
        for (int s = 0; s < 4; s++)
            for (int n = -300; n <= 300; n++)
                for (double off : {0.0, 0x1p-20, -0x1p-20, 0x1p-34, -0x1p-34, 0x1p-44, -0x1p-44})
                    check(std::ldexp(n * 0.5, e - 8 * (s + 1)) + off * top, e);
        check(std::nextafter(top, 0.0), e);
        check(-std::nextafter(top, 0.0), e);
        check(0.0, e);
        check(-0.0, e);
    }
    std::printf("%ld %ld\n", differ, tried);
    return 0;
}
