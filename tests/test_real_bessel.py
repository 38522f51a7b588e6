"""The real spherical Bessel recurrences (special.cuh, mstm_bessel_real), which
run on host and device alike, against the same recurrences in 80-bit arithmetic
up to the largest order asked for: 216, an origin order of 200 and a sphere of 16.

Bound: a step rounds the factor (2 k + 1) / z and its result, 1.1e-16 each and
independent from step to step: 432 of them add up to 2.3e-15 (one deviation),
the values at order 0 and 1 and the scale of j bring three roundings more; 8e-15
is past three deviations.  The error is of the envelope sqrt(j^2 + y^2) for
orders below z and of j and y themselves above.
"""
import os
import subprocess

from mstm_b200 import build as B

SRC = r"""
#include "special.cuh"
#include <cmath>
#include <cstdio>
#include <vector>
typedef long double ld;
int main()
{
    double worst = 0.0;
    unsigned long long seed = 1;
    for (int n : {1, 7, 16, 32, 64, 100, 160, 216})
        for (int t = 0; t < 60; t++) {
            seed = seed * 6364136223846793005ull + 1442695040888963407ull;
            const double u = (double)(seed >> 11) / 9007199254740992.0;
            const double z = t < 5 ? n + 0.5 * (t - 2) + 0.01 : 0.05 * std::exp(u * std::log(400.0 / 0.05));
            std::vector<zd> h(n + 2);
            if (!mstm_bessel_real(n, mk(z, 0.0), h.data())) continue;
            const ld x = z;
            std::vector<ld> y(n + 2), j(n + 2);
            y[0] = -cosl(x) / x;
            y[1] = (y[0] - sinl(x)) / x;
            for (int k = 1; k < n; k++) y[k + 1] = (2 * k + 1) / x * y[k] - y[k - 1];
            ld a = 0.0L, b = 1e-2000L;
            for (int k = n + 60 + (int)z + 20 * (int)std::cbrt(n + z); k >= 1; k--) {
                if (k <= n) j[k] = b;
                const ld c = (2 * k + 1) / x * b - a;
                a = b;
                b = c;
            }
            // orders 0 and 1 from the Wronskian j_1 y_0 - j_0 y_1 = 1 / z^2
            const ld s = 1 / (x * x) / (a * y[0] - b * y[1]);
            j[0] = b;
            for (int k = 0; k <= n; k++) {
                j[k] *= s;
                const ld e = hypotl(j[k], y[k]), dj = fabsl(h[k].x - j[k]) / (z > k ? e : fabsl(j[k])), dy = fabsl(h[k].y - y[k]) / (z > k ? e : fabsl(y[k]));
                if (!(dj <= worst)) worst = (double)dj;
                if (!(dy <= worst)) worst = (double)dy;
            }
        }
    std::printf("%.3e\n", worst);
}
"""


def test_errors_up_to_the_largest_order(tmp_path):
    src, exe = tmp_path / "bes.cu", tmp_path / "bes"
    src.write_text(SRC)
    subprocess.check_call([B.nvcc(), "-O2", "-std=c++17", "-I", B.CSRC, str(src), "-o", str(exe)])
    assert os.path.exists(exe)
    worst = float(subprocess.check_output([str(exe)], text=True))
    assert 0.0 < worst <= 8e-15, worst
