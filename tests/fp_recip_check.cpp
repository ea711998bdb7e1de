// Host check of fp_recip.h: the reciprocal and the quotient against the
// compiler's IEEE division, over random operands of many exponents, operands
// around powers of two, and the ends of the range.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>
#include <vector>

#include "fp_recip.h"

static int64_t ordered(double v)
{
    int64_t b;
    std::memcpy(&b, &v, sizeof b);
    return b < 0 ? INT64_MIN - b : b;
}
static int64_t ulps(double a, double b)
{
    if (std::isnan(a) || std::isnan(b)) return std::isnan(a) && std::isnan(b) ? 0 : INT64_MAX;
    return std::llabs(ordered(a) - ordered(b));
}

int main()
{
    std::mt19937_64 rng(7);
    auto mantissa = [&]() { return 1.0 + (double)(rng() >> 12) * 0x1p-52; };
    auto number = [&](int e) { return std::ldexp(mantissa() * (rng() & 1 ? 1 : -1), (int)(rng() % (2 * e + 1)) - e); };
    std::vector<double> special = {0.0, -0.0, 1.0, -1.0, 3.0, std::numeric_limits<double>::infinity(),
                                   -std::numeric_limits<double>::infinity(), std::nan(""),
                                   std::numeric_limits<double>::min(), std::numeric_limits<double>::denorm_min(),
                                   std::numeric_limits<double>::max(), 0x1p-1030, 0x1p-1025, 0x1p1000};
    for (int e : {-1022, -901, -800, -799, -101, -100, -99, -1, 0, 1, 99, 100, 101, 799, 800, 801, 1023})
        for (double m : {1.0, 1.0 + 0x1p-52, 2.0 - 0x1p-52, 1.5, 4.0 / 3}) special.push_back(std::ldexp(m, e));
    long long unequal = 0, total = 0;
    auto check = [&](double a, double b) {
        const double want = a / b, got = mhfem::quotient(a, b);
        const int64_t d = ulps(got, want);
        ++total;
        unequal += d != 0;
        if (d > 1) {
            std::printf("%a / %a: %a, not %a\n", a, b, got, want);
            std::exit(1);
        }
        if (ulps(mhfem::quotient_product(a, b, mhfem::recip_newton(b)), want) > 2) {
            std::printf("%a / %a: %a without correction, not %a\n", a, b,
                        mhfem::quotient_product(a, b, mhfem::recip_newton(b)), want);
            std::exit(1);
        }
        if (ulps(mhfem::recip_newton(b), 1.0 / b) > 1) {
            std::printf("1 / %a: %a\n", b, mhfem::recip_newton(b));
            std::exit(1);
        }
    };
    for (double a : special)
        for (double b : special) check(a, b);
    for (double a : special)
        for (int k = 0; k < 2000; ++k) {
            check(a, number(110));
            check(number(900), a);
        }
    for (int k = 0; k < 4000000; ++k) check(number(60), number(60));
    for (int k = 0; k < 1000000; ++k) check(number(1020), number(1020));
    std::printf("%lld of %lld unequal\n", unequal, total);
    return unequal * 1000 > total;
}
