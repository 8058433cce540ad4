// Host build of the integer forms of IEEE double arithmetic
// (csrc/va_int64.cuh, csrc/va_stepfactor.cuh) for tests/test_int64.py.
#include "../../vectorizedadjoint_gb300/csrc/va_stepfactor.cuh"

extern "C" {
// out[i] = a[i] * b[i]; ok[i]: both operands accepted
void i64_mul(int n, const double *a, const double *b, double *out, unsigned char *ok)
{
    for (int i = 0; i < n; i++) {
        va::MulRange r;
        out[i] = va::mul_rn(va::mul_left(a[i], r), va::mul_right(b[i], r));
        ok[i] = !r.beyond(480);
    }
}
void i64_div(int n, const double *a, const double *b, double *out, unsigned char *ok)
{
    for (int i = 0; i < n; i++)
        ok[i] = va::div_rn_pos(a[i], b[i], out[i]);
}
// the integer step factor alone: ok[i] = decided
void i64_pow(int k, int n, const double *x, double *out, unsigned char *ok)
{
    for (int i = 0; i < n; i++)
        ok[i] = k == 3 ? va::step_pow_int<3>(x[i], out[i])
              : k == 5 ? va::step_pow_int<5>(x[i], out[i])
              : k == 6 ? va::step_pow_int<6>(x[i], out[i]) : va::step_pow_int<8>(x[i], out[i]);
}
// bit 0: v > c, 1: v <= c, 2: NaN, 3: finite
void i64_cmp(int n, const double *v, double c, unsigned char *out)
{
    for (int i = 0; i < n; i++)
        out[i] = (va::greater_pos64(v[i], c) ? 1 : 0) | (va::less_equal_pos64(v[i], c) ? 2 : 0) |
                 (va::is_nan64(v[i]) ? 4 : 0) | (va::is_finite64(v[i]) ? 8 : 0);
}
}
