"""P/(8 alpha Delta) with the numerator as a pair of floats (the mixed stress
kernels' default form): on the host, its error against extended precision is
no larger than the FP64 Newton form's."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include "nsdg_visc_ff.hpp"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace nsdg_ff;
int main(int argc, char** argv)
{
    const double lo = std::atof(argv[1]), hi = std::atof(argv[2]), dmin = 2e-9;
    std::mt19937_64 gen(5);
    std::uniform_real_distribution<double> U(0, 1);
    float h, l;
    splitSquare(dmin, h, l);
    long double s2 = 0, sp = 0, mp = 0;
    const long n = 1000000;
    for (long i = 0; i < n; ++i) {
        const float inv = static_cast<float>(std::pow(10.0, lo + (hi - lo) * U(gen)));
        const double pa = std::pow(10.0, -6 + 14 * U(gen));
        const float s = static_cast<float>(1.0 / std::sqrt(static_cast<double>(inv + h)));
        const float y0 = floatOf(bitsOf(s) + static_cast<int>(U(gen) * 5) - 2); // rsqrtf: within 2 ulp
        const float ph = static_cast<float>(pa), pl = static_cast<float>(pa - static_cast<double>(ph));
        const long double ex = pa / sqrtl(static_cast<long double>(inv) + static_cast<long double>(dmin) * dmin);
        const long double u = std::ldexp(1.0, std::ilogb(static_cast<double>(ex)) - 23);
        const long double e2 = (viscNewton64(inv, pa, dmin, y0) - ex) / u, ep = (viscPair(inv, ph, pl, h, l, y0) - ex) / u;
        s2 += e2 * e2;
        sp += ep * ep;
        mp = fabsl(ep) > mp ? fabsl(ep) : mp;
    }
    std::printf("%.12Lf %.12Lf %.12Lf\n", sqrtl(s2 / n), sqrtl(sp / n), mp);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("visc_pair")
    (d / "a.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "nextsimdg_gb300" / "csrc"),
                    str(d / "a.cpp"), "-o", str(d / "a")], check=True)
    return d / "a"


@pytest.mark.parametrize("lo,hi", [(-36, -20), (-20, -14), (-14, -4)])
def test_no_further_from_the_exact_value_than_the_fp64_form(program, lo, hi):
    """Both round an approximation within 2^-41 to the nearest float: RMS 1/sqrt(12)
    ulp, equal to 1e-6 of it, and at most half an ulp plus 2^-41 / 2^-24."""
    rms64, rms_pair, worst = map(float, subprocess.check_output([str(program), str(lo), str(hi)]).split())
    assert rms_pair <= rms64 * (1 + 1e-6)
    assert worst <= 0.5 + 2.0 ** -17
