"""The quotients by a shared divisor of the FP64 step (Divisor in
sphere_b200/csrc/sph_device.cuh): RN(a r) with r = RN(1 / b), one FMA for the
remainder and one for the correction (P. Markstein, IBM J. Res. Dev. 34(1),
1990), the division itself where a, r or the product is near the ends of the
range, and a zero with its sign.  The FP64 form's parity rests on these being
the correctly rounded quotients; here the same steps in C, compiled without
contraction, against IEEE division: random operands over the whole exponent
range, quotients next to the ends of a binade, special values on both
sides."""
import os
import shutil
import subprocess

import pytest

C_SOURCE = r"""
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
static uint64_t s = 88172645463325252ull;
static uint64_t rnd(void) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double bits(uint64_t b) { double d; memcpy(&d, &b, 8); return d; }
static double mkd(uint64_t mant, int e)
{
    return bits(((uint64_t)(e + 1023) << 52) | (mant & ((1ull << 52) - 1)));
}
static double shared_div(double a, double b)
{
    const double r = 1.0 / b;
    const int ok = fabs(r) > 0x1p-1000 && fabs(r) < 0x1p+1000;
    const double q0 = a * r;
    const double aq = fabs(q0);
    if (ok && aq > 0x1p-900 && aq < 0x1p+1000 && fabs(a) > 0x1p-900)
        return fma(fma(-q0, b, a), r, q0);
    if (ok && a == 0.0) return q0;
    return a / b;
}
static long bad = 0, n = 0;
static void check(double a, double b)
{
    const double x = a / b, y = shared_div(a, b);
    ++n;
    if (memcmp(&x, &y, 8) != 0 && !(isnan(x) && isnan(y))) {
        if (bad < 5) printf("a=%a b=%a: %a vs %a\n", a, b, x, y);
        ++bad;
    }
}
int main(void)
{
    for (int t = 0; t < 4000000; ++t) check(bits(rnd()), bits(rnd()));
    for (int t = 0; t < 2000; ++t) {
        double b = mkd(rnd(), (int)(rnd() % 200) - 100);
        if (t % 4 == 0) b = mkd((1ull << 52) - 1 - (rnd() % 8), (int)(rnd() % 10) - 8);
        if (t % 4 == 1) b = mkd(rnd() % 16, (int)(rnd() % 10) - 8);
        for (int k = 0; k < 3000; ++k) {
            const uint64_t m = rnd();
            double a;
            if (k % 4 == 0) a = mkd(m, (int)(rnd() % 200) - 100);
            else if (k % 4 == 1) a = mkd((1ull << 52) - 1 - (m % 64), (int)(rnd() % 40) - 20) * b;
            else if (k % 4 == 2) a = mkd(m % 64, (int)(rnd() % 40) - 20) * b;
            else a = mkd(m, (int)(rnd() % 10));
            if (k & 4) a = nextafter(a, (m & 1) ? INFINITY : -INFINITY);
            check((m & 2) ? -a : a, b);
        }
    }
    const double sp[] = {0.0, -0.0, 5e-324, -5e-324, 1e-320, 1e-308, -1e-300, 0x1p-900, 0x1p-901,
                         0x1p1000, 0x1p1023, 1e300, INFINITY, -INFINITY, NAN, 1.0, -3.0, 1.7976931348623157e308};
    const int ns = sizeof sp / sizeof sp[0];
    for (int i = 0; i < ns; ++i)
        for (int j = 0; j < ns; ++j) check(sp[i], sp[j]);
    printf("%ld %ld\n", n, bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_shared_divisor_quotients_are_correctly_rounded(tmp_path):
    src = os.path.join(str(tmp_path), "shared_div.c")
    exe = os.path.join(str(tmp_path), "shared_div")
    with open(src, "w") as fh:
        fh.write(C_SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-o", exe, src, "-lm"], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    n, bad = (int(v) for v in out.stdout.split()[-2:])
    assert n == 4000000 + 2000 * 3000 + 18 * 18
    assert out.returncode == 0 and bad == 0, out.stdout
