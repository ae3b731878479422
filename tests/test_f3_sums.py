"""The three-term FP32 sums (csrc/f3.cuh), on the CPU: a C++ program built from the header adds the
same numbers in three FP32 terms and in FP64 and compares both with the exact sum (128-bit
fixed point).  Three terms must be no further off than FP64, term by term and in the tree of a warp."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pasc_inference_gb300", "csrc")

SRC = r"""
#include "f3.cuh"
#include <math.h>
#include <stdio.h>
#include <random>
#include <vector>
using namespace pasc;
// exact: values are multiples of 2^-60 below 2^40
typedef __int128 fix;
static fix fixed(double v) { return (fix)ldexp(v, 60); }
static double off(double v, fix exact) { return fabs(ldexp((double)(fixed(v) - exact), -60)); }
int main()
{
    std::mt19937_64 g(7);
    double worst = 0.0, worst64 = 0.0;
    for (int kind = 0; kind < 4; kind++)
        for (int n : {1, 2, 3, 10, 32, 1000, 100000}) {
            std::vector<float> v(n);
            std::uniform_real_distribution<double> u(0.0, 1.0);
            for (float &x : v) {
                // positive; both signs; sizes over 2^24; a large pair that cancels below
                double r = u(g);
                if (kind >= 1) r = 2.0 * r - 1.0;
                if (kind == 2) r = ldexp(r, (int)(24 * u(g)) - 12);
                x = (float)ldexp(floor(ldexp(r, 36)), -36);
            }
            if (kind == 3 && n >= 3) v[0] = 1048576.f, v[n - 1] = -1048576.f;
            fix exact = 0;
            double s = 0.0;
            F3 t{0.f, 0.f, 0.f};
            for (float x : v) exact += fixed(x), s += (double)x, t = f3_add(t, x);
            // the same terms pair by pair
            std::vector<F3> w;
            for (float x : v) w.push_back(F3{x, 0.f, 0.f});
            while (w.size() > 1) {
                std::vector<F3> h;
                for (size_t i = 0; i + 1 < w.size(); i += 2) h.push_back(f3_add(w[i], w[i + 1]));
                if (w.size() & 1) h.push_back(w.back());
                w = h;
            }
            const double half_ulp = 0.5 * (nextafter(fabs(s), 1e300) - fabs(s)) + ldexp(1.0, -60);
            const double e1 = off(f3_value(t), exact), e2 = off(f3_value(w[0]), exact), e64 = off(s, exact);
            // no further off than the FP64 sum, or than FP64's nearest number to the exact one
            if (e1 > fmax(e64, 1.01 * half_ulp) || e2 > fmax(e64, 1.01 * half_ulp)) {
                printf("kind %d n %d: %g %g fp64 %g\n", kind, n, e1, e2, e64);
                return 1;
            }
            worst = fmax(worst, e1), worst64 = fmax(worst64, e64);
        }
    // not finite where the sum leaves FP32, so that a caller can tell
    F3 t{3e38f, 0.f, 0.f};
    if (isfinite(f3_add(t, 3e38f).a) || isfinite(f3_add(F3{1.f, 0.f, 0.f}, INFINITY).a)) return 2;
    printf("ok %g %g\n", worst, worst64);
}
"""


def test_three_terms_are_no_further_off_than_fp64(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "f3.cpp", tmp_path / "f3"
    src.write_text(SRC)
    subprocess.check_call([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
