// The cell functions of bspline_math.cuh on the host: for every coordinate, finite or not, a cell inside
// the basis; for NaN an offset that stays NaN, so that what is evaluated there is NaN.
#include <cmath>
#include <cstdio>
#include <limits>
#include <vector>

#include "../../ddc_b200/csrc/bspline_math.cuh"

int main()
{
    int failures = 0, cases = 0;
    double const inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    for (int periodic = 0; periodic < 2; ++periodic)
        for (int nc : {1, 7, 1000, 1 << 20}) {
            ddcb::BasisDesc b {};
            b.degree = 3;
            b.periodic = periodic;
            b.uniform = 1;
            b.ncells = nc;
            b.rmin = -0.3;
            b.rmax = 1.7;
            b.length = b.rmax - b.rmin;
            b.step = b.length / nc;
            b.inv_step = 1.0 / b.step;
            std::vector<double> xs {nan, -nan, inf, -inf, 1e308, -1e308, 3e9 * b.length, b.rmin, b.rmax, std::nextafter(b.rmax, -inf),
                                    std::nextafter(b.rmin, inf), 0.7, -0.0};
            for (double x0 : xs) {
                double const x = periodic ? ddcb::periodic_wrap(b, x0) : x0;
                double off1 = 0.0, off2 = 0.0;
                int const c1 = ddcb::uniform_cell(b, x, off1), c2 = ddcb::uniform_cell_select(b, x, off2);
                bool ok = c1 >= 0 && c1 < nc && c1 == c2;
                if (std::isnan(x)) ok = ok && std::isnan(off1) && std::isnan(off2);
                else ok = ok && off1 == off2 && off1 >= 0.0 && off1 <= 1.0;
                ++cases;
                if (!ok) {
                    ++failures;
                    std::printf("FAIL nc=%d periodic=%d x=%g: cells %d %d offsets %g %g\n", nc, periodic, x0, c1, c2, off1, off2);
                }
            }
        }
    std::printf("%d cases, %d failures\n", cases, failures);
    return failures != 0;
}
