// Right-hand sides and hand-written vector-Jacobian products of the built-in
// models (N states, P parameters read by the RHS, PG parameter gradients).  They take the place of the user functor the reference records
// with AADC (lib/include/AadData.hpp:124-171) and of the JIT reverse code it
// replays in AadData::VectorTimesJacobians (AadData.hpp:291-330): every
// model gives f(x, p, t) and (J_x^T w, J_p^T w) at the same point.
//
// The argument order (x, p, t) keeps the reference functor's
// (x, dxdt, params, t) meaning (examples/VanDerPol/main.cpp:38-43).  S is the
// stage arithmetic type: double for the FP64 path, float for the mixed path,
// dword for the double-word path.  The double-word forms write each sum of
// products through the compensated accumulator (dacc) instead of a
// double-word multiply followed by a double-word add: the same O(u^2)
// accuracy in about half the FP32 operations.  The FP64 forms keep the
// reference's operation order (the FP64 path is compared bit for bit).
// rhs64 and vjp64 are the double forms with their products on the integer pipe
// (va_step64.cuh): the same operations in the same order, at most four noted
// values multiplied together (kForwardRhsFp64: the forward takes rhs).
// Parameter layouts follow the reference examples.
#pragma once

#include <type_traits>

#include "va_dword.cuh"
#include "va_int64.cuh"

namespace va {

template <class S>
constexpr bool is_dw = std::is_same<S, dword>::value;

// exact product by -2 of a double-word
__host__ __device__ __forceinline__ dword dw_m2(dword v) { return dword(-2.0f * v.hi, -2.0f * v.lo); }

// 1 - x^2 in double-word
__host__ __device__ __forceinline__ dword dw_one_minus_sq(dword x)
{
    dacc r{1.0f, 0.0f};
    dacc_fma(r, -x, x);
    return dacc_get(r);
}

// c + a b in double-word
__host__ __device__ __forceinline__ dword dw_fma(dword a, dword b, dword c)
{
    dacc r = dacc_of(c);
    dacc_fma(r, a, b);
    return dacc_get(r);
}

// Van der Pol, Lienard form: x0' = x1, x1' = mu (1 - x0^2) x1 - x0.  p = (mu).
struct ModelVdP {
    static constexpr int N = 2, P = 1, PG = 1;
    template <class S>
    __host__ __device__ __forceinline__ static void rhs(const S *x, const S *p, S t, S *f)
    {
        (void)t;
        f[0] = x[1];
        if constexpr (is_dw<S>)
            f[1] = dw_fma(p[0] * dw_one_minus_sq(x[0]), x[1], -x[0]);
        else
            f[1] = p[0] * (S(1) - x[0] * x[0]) * x[1] - x[0];
    }
    template <class S>
    __host__ __device__ __forceinline__ static void vjp(const S *w, const S *x, const S *p, S t, S *gx, S *gp)
    {
        (void)t;
        const S mu = p[0];
        if constexpr (is_dw<S>) {
            const dword a = dw_one_minus_sq(x[0]);
            gx[0] = w[1] * dw_fma(dw_m2(mu * x[0]), x[1], dword(-1.0f, 0.0f));
            gx[1] = dw_fma(w[1], mu * a, w[0]);
            gp[0] = w[1] * (a * x[1]);
        } else {
            gx[0] = w[1] * (S(-2) * mu * x[0] * x[1] - S(1));
            gx[1] = w[0] + w[1] * (mu * (S(1) - x[0] * x[0]));
            gp[0] = w[1] * ((S(1) - x[0] * x[0]) * x[1]);
        }
    }
    static constexpr bool kForwardRhsFp64 = true;
    __host__ __device__ __forceinline__ static void rhs64(const double *x, const double *p, double *f, MulRange &r)
    {
        const double a = 1.0 - mul_rn(mul_left(x[0], r), mul_right_in(x[0]));
        f[0] = x[1];
        f[1] = mul_rn(mul_left_in(mul_rn(mul_left_in(a), mul_right_in(p[0]))), mul_right(x[1], r)) - x[0];
    }
    __host__ __device__ __forceinline__ static void vjp64(const double *w, const double *x, const double *p,
                                                          double *gx, double *gp, MulRange &r)
    {
        const MulR x1 = mul_right(x[1], r), mu = mul_right_in(p[0]);
        const MulL w1 = mul_left(w[1], r), x0 = mul_left(x[0], r);
        const double a = 1.0 - mul_rn(x0, mul_right_in(x[0]));
        const MulL al = mul_left_in(a);
        const double mx = mul_rn(mul_m2(x0), mu); // -2 mu x0
        gx[0] = mul_rn(w1, mul_right_in(mul_rn(mul_left_in(mx), x1) - 1.0));
        gx[1] = w[0] + mul_rn(w1, mul_right_in(mul_rn(al, mu)));
        gp[0] = mul_rn(w1, mul_right_in(mul_rn(al, x1)));
    }
    // vjp's outputs as w[kVjpW] W_o (+ w[0] for o = kVjpAdd)
    static constexpr int kVjpW = 1, kVjpAdd = 1;
    __host__ __device__ __forceinline__ static void vjp_weights(const double *x, const double *p, double *W)
    {
        const double a = 1.0 - x[0] * x[0];
        W[0] = -2.0 * p[0] * x[0] * x[1] - 1.0;
        W[1] = p[0] * a;
        W[2] = a * x[1];
    }
};

// Van der Pol as in the reference example (examples/VanDerPol/main.cpp:41-42):
// x0' = x1, x1' = mu ((1 - x0^2) x1 - x0).
struct ModelVdPPetsc {
    static constexpr int N = 2, P = 1, PG = 1;
    template <class S>
    __host__ __device__ __forceinline__ static void rhs(const S *x, const S *p, S t, S *f)
    {
        (void)t;
        f[0] = x[1];
        if constexpr (is_dw<S>)
            f[1] = p[0] * dw_fma(dw_one_minus_sq(x[0]), x[1], -x[0]);
        else
            f[1] = p[0] * ((S(1) - x[0] * x[0]) * x[1] - x[0]);
    }
    template <class S>
    __host__ __device__ __forceinline__ static void vjp(const S *w, const S *x, const S *p, S t, S *gx, S *gp)
    {
        (void)t;
        const S mu = p[0];
        if constexpr (is_dw<S>) {
            const dword a = dw_one_minus_sq(x[0]);
            gx[0] = w[1] * (mu * dw_fma(dw_m2(x[0]), x[1], dword(-1.0f, 0.0f)));
            gx[1] = dw_fma(w[1], mu * a, w[0]);
            gp[0] = w[1] * dw_fma(a, x[1], -x[0]);
        } else {
            gx[0] = w[1] * (mu * (S(-2) * x[0] * x[1] - S(1)));
            gx[1] = w[0] + w[1] * (mu * (S(1) - x[0] * x[0]));
            gp[0] = w[1] * ((S(1) - x[0] * x[0]) * x[1] - x[0]);
        }
    }
    static constexpr bool kForwardRhsFp64 = true;
    __host__ __device__ __forceinline__ static void rhs64(const double *x, const double *p, double *f, MulRange &r)
    {
        const double a = 1.0 - mul_rn(mul_left(x[0], r), mul_right_in(x[0]));
        f[0] = x[1];
        f[1] = mul_rn(mul_left_in(mul_rn(mul_left_in(a), mul_right(x[1], r)) - x[0]), mul_right_in(p[0]));
    }
    __host__ __device__ __forceinline__ static void vjp64(const double *w, const double *x, const double *p,
                                                          double *gx, double *gp, MulRange &r)
    {
        const MulR x1 = mul_right(x[1], r), mu = mul_right_in(p[0]);
        const MulL w1 = mul_left(w[1], r), x0 = mul_left(x[0], r);
        const double a = 1.0 - mul_rn(x0, mul_right_in(x[0]));
        const MulL al = mul_left_in(a);
        const double ax = mul_rn(al, x1); // (1 - x0^2) x1
        const double c = mul_rn(mul_left_in(mul_rn(mul_m2(x0), x1) - 1.0), mu);
        gx[0] = mul_rn(w1, mul_right_in(c));
        gx[1] = w[0] + mul_rn(w1, mul_right_in(mul_rn(al, mu)));
        gp[0] = mul_rn(w1, mul_right_in(ax - x[0]));
    }
    static constexpr int kVjpW = 1, kVjpAdd = 1;
    __host__ __device__ __forceinline__ static void vjp_weights(const double *x, const double *p, double *W)
    {
        const double a = 1.0 - x[0] * x[0];
        W[0] = p[0] * (-2.0 * x[0] * x[1] - 1.0);
        W[1] = p[0] * a;
        W[2] = a * x[1] - x[0];
    }
};

// Damped harmonic oscillator x'' + 2 zeta omega x' + omega^2 x = 0 as a first
// order system; p = (omega, zeta).  (The reference example
// examples/HarmonicOscillator/main.cpp:11-30 uses fixed k = 1 and a friction
// parameter; this is the (omega, zeta) form of the same family.)
struct ModelDHO {
    static constexpr int N = 2, P = 2, PG = 2;
    template <class S>
    __host__ __device__ __forceinline__ static void rhs(const S *x, const S *p, S t, S *f)
    {
        (void)t;
        f[0] = x[1];
        if constexpr (is_dw<S>) {
            dacc r = dacc_mul(-(p[0] * p[0]), x[0]);
            dacc_fma(r, dw_m2(p[1] * p[0]), x[1]);
            f[1] = dacc_get(r);
        } else {
            f[1] = -p[0] * p[0] * x[0] - S(2) * p[1] * p[0] * x[1];
        }
    }
    template <class S>
    __host__ __device__ __forceinline__ static void vjp(const S *w, const S *x, const S *p, S t, S *gx, S *gp)
    {
        (void)t;
        const S om = p[0], ze = p[1];
        if constexpr (is_dw<S>) {
            gx[0] = w[1] * -(om * om);
            gx[1] = dw_fma(w[1], dw_m2(ze * om), w[0]);
            dacc r = dacc_mul(dw_m2(om), x[0]);
            dacc_fma(r, dw_m2(ze), x[1]);
            gp[0] = w[1] * dacc_get(r);
            gp[1] = w[1] * (dw_m2(om) * x[1]);
        } else {
            gx[0] = w[1] * (-om * om);
            gx[1] = w[0] + w[1] * (S(-2) * ze * om);
            gp[0] = w[1] * (S(-2) * om * x[0] - S(2) * ze * x[1]);
            gp[1] = w[1] * (S(-2) * om * x[1]);
        }
    }
    static constexpr bool kForwardRhsFp64 = true;
    __host__ __device__ __forceinline__ static void rhs64(const double *x, const double *p, double *f, MulRange &r)
    {
        const MulL om = mul_left_in(p[0]), ze = mul_left_in(p[1]);
        const MulR omr = mul_right_in(p[0]);
        const double k = mul_rn(mul_neg(om), omr), c = mul_rn(mul_m2(ze), omr); // -om om, -2 ze om
        f[0] = x[1];
        f[1] = mul_rn(mul_left(x[0], r), mul_right_in(k)) + mul_rn(mul_left(x[1], r), mul_right_in(c));
    }
    __host__ __device__ __forceinline__ static void vjp64(const double *w, const double *x, const double *p,
                                                          double *gx, double *gp, MulRange &r)
    {
        const MulL om = mul_left_in(p[0]), ze = mul_left_in(p[1]), w1 = mul_left(w[1], r);
        const MulR omr = mul_right_in(p[0]), x0 = mul_right(x[0], r), x1 = mul_right(x[1], r);
        gx[0] = mul_rn(w1, mul_right_in(mul_rn(mul_neg(om), omr)));
        gx[1] = w[0] + mul_rn(w1, mul_right_in(mul_rn(mul_m2(ze), omr)));
        gp[0] = mul_rn(w1, mul_right_in(mul_rn(mul_m2(om), x0) + mul_rn(mul_m2(ze), x1)));
        gp[1] = mul_rn(w1, mul_right_in(mul_rn(mul_m2(om), x1)));
    }
    static constexpr int kVjpW = 1, kVjpAdd = 1;
    __host__ __device__ __forceinline__ static void vjp_weights(const double *x, const double *p, double *W)
    {
        const double om = p[0], ze = p[1];
        W[0] = -om * om;
        W[1] = -2.0 * ze * om;
        W[2] = -2.0 * om * x[0] - 2.0 * ze * x[1];
        W[3] = -2.0 * om * x[1];
    }
};

// Exponential decay y' = -k y; p = (k).  Its discrete adjoint has a closed
// form for a frozen step sequence, which the tests use.
struct ModelDecay {
    static constexpr int N = 1, P = 1, PG = 1;
    template <class S>
    __host__ __device__ __forceinline__ static void rhs(const S *x, const S *p, S t, S *f)
    {
        (void)t;
        f[0] = -p[0] * x[0];
    }
    template <class S>
    __host__ __device__ __forceinline__ static void vjp(const S *w, const S *x, const S *p, S t, S *gx, S *gp)
    {
        (void)t;
        gx[0] = -p[0] * w[0];
        gp[0] = -x[0] * w[0];
    }
    static constexpr bool kForwardRhsFp64 = true;
    __host__ __device__ __forceinline__ static void rhs64(const double *x, const double *p, double *f, MulRange &r)
    {
        f[0] = mul_rn(mul_neg(mul_left_in(p[0])), mul_right(x[0], r));
    }
    __host__ __device__ __forceinline__ static void vjp64(const double *w, const double *x, const double *p,
                                                          double *gx, double *gp, MulRange &r)
    {
        const MulR wr = mul_right(w[0], r);
        gx[0] = mul_rn(mul_neg(mul_left_in(p[0])), wr);
        gp[0] = mul_rn(mul_neg(mul_left(x[0], r)), wr);
    }
    static constexpr int kVjpW = 0, kVjpAdd = -1;
    __host__ __device__ __forceinline__ static void vjp_weights(const double *x, const double *p, double *W)
    {
        W[0] = -p[0];
        W[1] = -x[0];
    }
};

} // namespace va
