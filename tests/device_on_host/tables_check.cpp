// tables_check.cpp -- the table functions (ysg_tables.cuh) against extended
// precision, on the CPU: every twiddle argument up to rows of 2^18 samples,
// dense angles over [0, 4], exponents over [-700, 700] and around zero.
// Prints the largest error in units of the last place of the 64-bit result;
// exit status 0 if none exceeds 0.502: half a unit of the final rounding, and
// up to 2^-9 for the series, the two-double operations (a few 2^-100) and the
// comparison's own 64-bit mantissa (2^-12).
#include "block_on_host.h"

#include "ysg_tables.cuh"

using namespace ysg;

static double units(double got, long double want, double floor_)
{
    const double w = std::max(std::fabs((double)want), floor_);
    return (double)(std::fabs((long double)got - want) / (std::nextafter(w, INFINITY) - w));
}

int main()
{
    double es = 0.0, ec = 0.0, ee = 0.0;
    auto angle = [&](double a) {
        double s, c;
        table_sincos(a, &s, &c);
        es = std::max(es, units(s, sinl(a), 0x1p-1000));
        ec = std::max(ec, units(c, cosl(a), 0x1p-1000));
    };
    const double pi_d = (double)3.14159265358979323846f;
    for (int st = 0; st < 18; st++)
        for (int m = 0; m < (1 << st); m++) angle((double)m * (pi_d / (double)(1 << st)));
    for (int i = 0; i <= 400000; i++) angle(1.0e-5 * i);
    auto power = [&](double a) { ee = std::max(ee, units(table_exp(a), expl(a), 0x1p-1074)); };
    for (int i = -350000; i <= 350000; i++) power(0.002 * i - 1.0e-5);
    for (int i = -200000; i <= 200000; i++) power(1.0e-5 * i);
    for (double a : {0.0, 1e-300, -1e-300, 1e-17, -1e-17, 709.7, -745.0, 800.0, -800.0}) {
        const double g = table_exp(a);
        const bool far = std::fabs(a) >= 700.0;             // the library's own result
        if (far ? g != std::exp(a) : units(g, expl(a), 0x1p-1000) > 0.502) ee = 1e9;
    }
    if (!std::isnan(table_exp(NAN))) ee = 1e9;
    std::printf("sin %.5f cos %.5f exp %.5f\n", es, ec, ee);
    return es <= 0.502 && ec <= 0.502 && ee <= 0.502 ? 0 : 1;
}
