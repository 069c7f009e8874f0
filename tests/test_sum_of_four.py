"""The sum of four divergence shares at a node of the mixed BBM path
(nsdg_ff::sumOfFour): against the same sum in FP64, rounded to FP32."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SOURCE = r"""
#include "nsdg_visc_ff.hpp"
#include <cstdio>
#include <cstdlib>
#include <random>
int main(int, char** argv)
{
    const int spread = std::atoi(argv[1]);
    std::mt19937_64 gen(9);
    std::uniform_real_distribution<double> U(-1, 1);
    long differ = 0;
    double worst = 0;
    const long n = 1000000;
    for (long i = 0; i < n; ++i) {
        float x[4];
        double s = 0, most = 0;
        for (int k = 0; k < 4; ++k) {
            x[k] = static_cast<float>(std::ldexp(U(gen), -static_cast<int>(gen() % (spread + 1))));
            if (i % 8 == 7 && k == 3) // cancels to a rest
                x[3] = static_cast<float>(-s + std::ldexp(U(gen), -20));
            if (i % 5 == 4 && k > static_cast<int>(i % 3))
                x[k] = 0.f;
            s += x[k];
            most = std::max(most, std::fabs(static_cast<double>(x[k])));
        }
        const float r = static_cast<float>(s), q = nsdg_ff::sumOfFour(x[0], x[1], x[2], x[3]);
        differ += r != q;
        // beyond half a unit of the result
        const double half = std::ldexp(1.0, std::ilogb(std::fabs(s) + 1e-300) - 24);
        worst = std::max(worst, (std::fabs(q - s) - half) / most);
    }
    std::printf("%.9f %.3e\n", static_cast<double>(differ) / n, worst);
}
"""


@pytest.mark.parametrize("spread", [0, 8, 30])
def test_rounds_as_the_fp64_sum(tmp_path, spread):
    """The sums are exact up to the rest of the errors' sum, below 2 4 2^-24 2^-24
    3 < 2^-43 of the largest term, and the tie's decision moves a midpoint by
    2^-22 of half a unit: beyond half a unit by less than 2^-43, so that the result
    differs from the FP64 sum's rounding only within that of a midpoint."""
    (tmp_path / "a.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "nextsimdg_gb300" / "csrc"),
                    str(tmp_path / "a.cpp"), "-o", str(tmp_path / "a")], check=True)
    differ, worst = map(float, subprocess.check_output([str(tmp_path / "a"), str(spread)]).split())
    assert worst <= 2.0 ** -43
    assert differ <= 1e-4
