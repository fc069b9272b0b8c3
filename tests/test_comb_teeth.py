"""The comb index that the comb's plan takes from a running weight
(storm_comb.cuh, compiled here for the host) against the reference's walk from
tooth to tooth (population/CombPopulationControl.hpp:203-222), from ordinary
weights down to the smallest doubles, where the reciprocal of a tooth's weight
is no longer finite.  In a process of its own with a time limit: a search that
does not end fails instead of holding up the tests."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "storm_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "storm_comb.cuh"
using namespace storm;
int main(int argc, char **argv) {
    const double unit = std::strtod(argv[1], nullptr);
    const int spread = std::atoi(argv[2]);
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> u(0.0, 1.0);
    for (uint64_t nin : {1, 2, 7, 50, 999})
        for (uint64_t n : {nin + 1, nin + 2, 3 * nin, 3 * nin + 500}) {
            if (n <= nin) continue;
            std::vector<double> w(n);
            double W = 0.0;
            for (double &x : w) W += x = unit * std::ceil(spread * u(g));
            const double e = W / static_cast<double>(nin), r = (static_cast<double>(g() >> 12) + 0.5) * 0x1p-52;
            const CombTeeth t = comb_teeth(r, e, nin);
            uint64_t k = 0;
            double cum = 0.0;
            for (double x : w) {
                while ((cum + x) > (static_cast<double>(k) + r) * e) ++k;
                cum += x;
                if (teeth_index(t, cum) != static_cast<double>(k)) {
                    std::printf("nin %llu n %llu weight %g: %g, not %llu\n", (unsigned long long)nin, (unsigned long long)n,
                                cum, teeth_index(t, cum), (unsigned long long)k);
                    return 1;
                }
            }
            // numbers that are no running weight of the cell end as well
            for (double P : {-1.0, 0.0, 1e300, HUGE_VAL, double(NAN)}) (void)teeth_index(t, P);
        }
    // and so do teeth that no cell has
    for (double e : {0.0, -1.0, 4.9e-324, HUGE_VAL, double(NAN)})
        for (double P : {-1.0, 1e-320, 1.0, 1e300, HUGE_VAL, double(NAN)})
            if (!(teeth_index(comb_teeth(0.5, e, 50), P) <= 102.0)) return 2;
    return 0;
}
"""


@pytest.mark.parametrize("spread", [1, 3, 1000000])
@pytest.mark.parametrize("unit", ["1.0", "1e25", "1e-200", "1e-271", "1e-290", "1e-307", "5.6e-309", "1e-309", "1e-315",
                                  "4.94065645841246544e-324"])
def test_comb_index_is_the_walks(tmp_path_factory, unit, spread):
    d = tmp_path_factory.getbasetemp() / "comb_teeth"
    exe = d / "teeth"
    if not exe.exists():
        d.mkdir(exist_ok=True)
        (d / "teeth.cpp").write_text(PROGRAM)
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(d / "teeth.cpp"), "-o", str(exe)],
                       check=True)
    r = subprocess.run([str(exe), unit, str(spread)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
