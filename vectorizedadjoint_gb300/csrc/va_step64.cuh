// One FP64 step, forward and backward, with its products on the integer pipe
// (va_int64.cuh).  The FP64 unit is left to the additions.
//
// What bounds it: an FP64 instruction holds its quadrant's FP64 unit for 64
// cycles, and an attempt of Dormand-Prince on Van der Pol is ~100 products
// and ~75 sums (a back step ~130 and ~100), so the one-thread FP64 sweeps
// are bound by the FP64 instruction count at every batch size.  A product in
// integers issues in ~45 cycles beside the sums.
//
// Not every product: with all of them in integers the FP64 unit waits for the
// integer pipe and the instruction fetch.  Left to the FP64 unit: the forward's
// right-hand side of the one-lane models (a chain of products, short of
// independent work; 65,536 Van der Pol instances forward 3.94 -> 3.81 ms) and
// the second product of each K-bar term (backward 5.22 -> 4.58; the recompute's
// right-hand sides as well 4.99, the coefficients c h as well 5.1; the error's
// terms of one component 4.17 forward).
//
// The operations and their order are those of attempt_pair and back_step; every sum is the FP64 instruction and every product the
// correctly rounded one, so the results have the same bits.  For the 5(4)
// pairs: no a_mj is zero, and a zero b_m or e_m is left out of the sums as it
// is in attempt_pair.
//
// Range.  The products need operands whose significand and exponent can be
// taken apart (no infinities, NaNs or subnormals) and results that are
// normal.  Every value that enters a product from outside the product chain
// is noted in a MulRange; the chains below multiply at most four noted values
// before the next one is noted, so with all of them within 2^-240 .. 2^240 (or
// zero) no product leaves the normal range.  Otherwise the functions return
// false and the caller takes the step over with FP64 instructions throughout
// (attempt_pair, back_step): the same result, or the same
// infinities and NaNs.
#pragma once

#include <type_traits>

#include "va_int64.cuh"

namespace va {

constexpr int kChainRange = 240;

// the model's parameters into the range, once per step (rhs64 and vjp64, the
// model's functions with integer products, take them as noted)
template <class M>
__host__ __device__ __forceinline__ void note_params64(const double (&p)[M::P], MulRange &r)
{
#pragma unroll
    for (int k = 0; k < M::P; k++)
        r.note(f64_hi(p[k]), f64_lo(p[k]));
}
// the right-hand side of a forward stage
template <class M>
__host__ __device__ __forceinline__ void forward_rhs64(const double *x, const double *p, double t, double *f,
                                                       MulRange &r)
{
    if constexpr (M::kForwardRhsFp64)
        M::template rhs<double>(x, p, t, f);
    else
        M::rhs64(x, p, f, r);
}

// Whether every lane that carries the instance stayed in range (a lane-group
// model, whose functions exchange components, answers for its group).
template <class M, class = void>
struct Uniform64 {
    __host__ __device__ static bool all(bool ok) { return ok; }
};
template <class M>
struct Uniform64<M, std::void_t<decltype(M::TPI)>> {
    __device__ static bool all(bool ok) { return M::all(ok); }
};
template <class M>
__host__ __device__ __forceinline__ bool uniform64(bool ok)
{
    return Uniform64<M>::all(ok);
}

// c h for a tableau coefficient c, as a second factor
__host__ __device__ __forceinline__ MulR coef_right(double c, const MulR &h)
{
    return mul_right_in(mul_rn(mul_left_in(c), h));
}

// X_m = y + sum_{j<m} (a_mj dt) K_j (form_stage); the 5(4) pairs have no zero a_mj
template <class Tab, int N>
__host__ __device__ __forceinline__ void form_stage64(int m, const double (&y)[N], const MulL (&K)[Tab::S][N],
                                                      const MulR &h, double (&X)[N])
{
#pragma unroll
    for (int i = 0; i < N; i++)
        X[i] = y[i];
#pragma unroll
    for (int j = 0; j < Tab::S - 1; j++)
        if (j < m) {
            const MulR c = coef_right(Tab::a(m, j), h);
#pragma unroll
            for (int i = 0; i < N; i++)
                X[i] = X[i] + mul_rn(K[j][i], c);
        }
}

// attempt_pair's step for double stages: y_new, k_new and the error norm.
// False: out of range.
template <class M, class Tab>
__host__ __device__ __forceinline__ bool attempt64(const double (&y)[M::N], const double (&k0)[M::N],
                                                   const double (&p)[M::P], double t, double dt, double atol,
                                                   double rtol, double (&ynew)[M::N], double (&knew)[M::N],
                                                   double &err)
{
    constexpr int N = M::N, NS = Tab::S;
    MulRange r;
    note_params64<M>(p, r);
    const MulR h = mul_right(dt, r);
    MulL K[NS][N];
#pragma unroll
    for (int i = 0; i < N; i++)
        K[0][i] = mul_left(k0[i], r);
#pragma unroll
    for (int m = 1; m < NS; m++) {
        double X[N], f[N];
        form_stage64<Tab, N>(m, y, K, h, X);
        forward_rhs64<M>(X, p, t + Tab::c(m) * dt, f, r);
#pragma unroll
        for (int i = 0; i < N; i++)
            K[m][i] = mul_left(f[i], r);
    }
#pragma unroll
    for (int i = 0; i < N; i++)
        ynew[i] = y[i];
#pragma unroll
    for (int j = 0; j < NS; j++)
        if (Tab::b(j) != 0.0) {
            const MulR c = coef_right(Tab::b(j), h);
#pragma unroll
            for (int i = 0; i < N; i++)
                ynew[i] = ynew[i] + mul_rn(K[j][i], c);
        }
    double e[N];
    bool first = true;
#pragma unroll
    for (int j = 0; j < NS; j++)
        if (Tab::e(j) != 0.0) {
            const MulR c = coef_right(Tab::e(j), h);
#pragma unroll
            for (int i = 0; i < N; i++) {
                const double term = mul_rn(K[j][i], c);
                e[i] = first ? term : e[i] + term;
            }
            first = false;
        }
    if constexpr (Tab::FSAL) {
        forward_rhs64<M>(ynew, p, t + dt, knew, r);
        const MulR c = coef_right(Tab::E_NEW, h);
#pragma unroll
        for (int i = 0; i < N; i++)
            e[i] = e[i] + mul_rn(mul_left(knew[i], r), c);
    }
    // odeint's rel_error + norm_inf: one quotient per component, then max
    const MulR ah = {h.h, h.l, h.e & 0x7fffffffu};
    const MulL rt = mul_left(rtol, r);
    err = 0.0;
#pragma unroll
    for (int i = 0; i < N; i++) {
        const MulL ak = {K[0][i].h, K[0][i].l, K[0][i].e & 0x7fffffffu};
        const double s = fabs(y[i]) + mul_rn(ak, ah);
        err = max_nonneg64(err, quotient64(fabs(e[i]), atol + mul_rn(rt, mul_right(s, r))));
    }
    return !r.beyond(kChainRange) && !is_nan64(err);
}

// back_step for double stages: lambda_n in ybar, mu's new sums in ms.  False:
// out of range.
template <class M, class Tab>
__host__ __device__ __forceinline__ bool back_step64(const double (&y)[M::N], double hh,
                                                     const double (&p)[M::P], const double (&lam)[M::N],
                                                     const double (&mu)[M::PG], double (&ybar)[M::N],
                                                     double (&ms)[M::PG])
{
    constexpr int N = M::N, P = M::PG, NS = Tab::S;
    MulRange r;
    note_params64<M>(p, r);
    const MulR h = mul_right(hh, r);
    double X[NS][N];
    {
        MulL K[NS][N];
#pragma unroll
        for (int m = 0; m < NS; m++) {
            form_stage64<Tab, N>(m, y, K, h, X[m]);
            if (m < NS - 1) {
                double f[N];
                M::rhs64(X[m], p, f, r);
#pragma unroll
                for (int i = 0; i < N; i++)
                    K[m][i] = mul_left(f[i], r);
            }
        }
    }
    double Kbar[NS][N];
    MulL l[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
        ybar[i] = lam[i];
        l[i] = mul_left(lam[i], r);
    }
#pragma unroll
    for (int k = 0; k < P; k++)
        ms[k] = mu[k];
#pragma unroll
    for (int m = 0; m < NS; m++) {
        const MulR bh = coef_right(Tab::b(m), h);
#pragma unroll
        for (int i = 0; i < N; i++)
            Kbar[m][i] = Tab::b(m) != 0.0 ? mul_rn(l[i], bh)
                                          : f64_from_bits((uint64_t)((l[i].e ^ h.e) & 0x80000000u) << 32);
    }
#pragma unroll
    for (int m = NS - 1; m >= 0; m--) {
        double gx[N], gp[P];
        M::vjp64(Kbar[m], X[m], p, gx, gp, r);
#pragma unroll
        for (int i = 0; i < N; i++) {
            ybar[i] += gx[i];
            if (m == 0)
                continue;
            const MulL g = mul_left(gx[i], r);
#pragma unroll
            for (int k = 0; k < NS - 1; k++)
                if (k < m)
                    Kbar[k][i] += mul_rn(g, mul_right_in(Tab::a(m, k))) * hh;
        }
#pragma unroll
        for (int k = 0; k < P; k++)
            ms[k] += gp[k];
    }
    return !r.beyond(kChainRange);
}

} // namespace va
