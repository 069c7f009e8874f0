"""The preparation kernels' exp(x) (nsdg_exp64.cuh), its arithmetic on the host
against extended precision: the stated 0.55 ulp over the whole range it takes,
and the arguments around zero, around the ends of its range and beyond."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include "nsdg_exp64.cuh"
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <random>
using nsdg::sf::exp64;
static long double ulps(double x)
{
    const long double exact = expl(static_cast<long double>(x));
    int e;
    frexpl(exact, &e);
    return fabsl(exp64(x) - exact) / ldexpl(1.0L, e - 53);
}
int main(int argc, char** argv)
{
    if (!std::strcmp(argv[1], "range")) {
        const double lo = std::atof(argv[2]), hi = std::atof(argv[3]);
        std::mt19937_64 gen(17);
        std::uniform_real_distribution<double> U(lo, hi);
        long double worst = 0;
        for (int i = 0; i < 1000000; ++i)
            worst = std::max(worst, ulps(U(gen)));
        // the table's steps: arguments where n changes, from both sides
        for (int j = static_cast<int>(lo * 92); j < static_cast<int>(hi * 92); ++j) {
            const double x = (j + 0.5) * 0x1.62e42fefa39efp-7;
            if (x > lo && x < hi)
                for (double y : { x, std::nextafter(x, -1e3), std::nextafter(x, 1e3) })
                    worst = std::max(worst, ulps(y));
        }
        std::printf("%.6Lf\n", worst);
        return 0;
    }
    const double inf = std::numeric_limits<double>::infinity();
    const double below = std::nextafter(700.0, 0.0), above = std::nextafter(700.0, 1e3);
    int bad = exp64(0.0) != 1.0 || exp64(-0.0) != 1.0 || exp64(0x1p-1074) != 1.0 || exp64(-0x1p-1074) != 1.0
        || exp64(0x1p-54) != 1.0 || exp64(-0x1p-55) != 1.0;
    for (double x : { below, 700.0, above, -below, -700.0, -above, 709.0, -708.0, -745.0 })
        bad |= std::fabs(exp64(x) - std::exp(x)) > 2e-16 * 2 * std::exp(x) ? 2 : 0;
    bad |= exp64(inf) != inf || exp64(-inf) != 0.0 || exp64(710.0) != inf || exp64(-1e5) != 0.0 ? 4 : 0;
    bad |= exp64(std::numeric_limits<double>::quiet_NaN()) == exp64(std::numeric_limits<double>::quiet_NaN()) ? 8 : 0;
    std::printf("%d\n", bad);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("exp64")
    (d / "a.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-x", "c++", "-I",
                    str(ROOT / "nextsimdg_gb300" / "csrc"), str(d / "a.cpp"), "-o", str(d / "a")], check=True)
    return d / "a"


@pytest.mark.parametrize("lo,hi", [(-20, 0), (-1e-3, 1e-3), (-1e-10, 1e-10), (-699.99, -600), (600, 699.99), (-60, 60)])
def test_within_its_stated_error(program, lo, hi):
    """Half an ulp for the last sum, 0.04 for the series' remainder, and below a
    hundredth each for the roundings of r, of p and of t.x p + t.y, which are at
    most 2^-7.5 of the result."""
    assert float(subprocess.check_output([str(program), "range", str(lo), str(hi)])) <= 0.55


def test_special_arguments(program):
    assert int(subprocess.check_output([str(program), "special"])) == 0
