// A model with a function `rate` of its own (a chemist's rate law, the
// signature of the library's internal one) against the same model without it:
// one back step on the host, the same bits.  Prints "same".
#include <cstdio>
#include <cstring>

#include "../../include/va_model.cuh"

struct Plain {
    static constexpr int N = 2, P = 1, PG = 1;
    template <class S>
    __host__ __device__ static void rhs(const S *x, const S *p, S, S *f)
    {
        f[0] = p[0] * x[1] - x[0] * x[0];
        f[1] = x[0] * x[0] - p[0] * x[1];
    }
    template <class S>
    __host__ __device__ static void vjp(const S *w, const S *x, const S *p, S, S *gx, S *gp)
    {
        const S d = w[1] - w[0];
        gx[0] = S(2) * x[0] * d;
        gx[1] = -(p[0] * d);
        gp[0] = -(x[1] * d);
    }
};
struct WithRate : Plain {
    template <class S>
    __host__ __device__ static S rate(const S *x, const S *p)
    {
        return p[0] * x[1];
    }
};

template <class M, class Tab>
static void run(double *out)
{
    const double y[2] = {0.7, 1.3}, p[1] = {0.9};
    double lam[2] = {1.0, -0.4}, mu[1] = {0.2};
    va::back_step<M, Tab, double>(y, 0.5, 0.125, p, lam, mu);
    out[0] = lam[0], out[1] = lam[1], out[2] = mu[0];
}

int main()
{
    double a[9], b[9];
    run<Plain, va::TabDopri5>(a);
    run<WithRate, va::TabDopri5>(b);
    run<Plain, va::TabCK54>(a + 3);
    run<WithRate, va::TabCK54>(b + 3);
    run<Plain, va::TabRKF78>(a + 6);
    run<WithRate, va::TabRKF78>(b + 6);
    std::puts(std::memcmp(a, b, sizeof a) ? "different" : "same");
    return 0;
}
