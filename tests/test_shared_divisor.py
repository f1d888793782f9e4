"""The quotients by a shared divisor of the FP64 step (Divisor in
sphere_b200/csrc/sph_divisor.cuh, whose comment has the argument): RN(a r)
with r = RN(1 / b), one FMA for the remainder and one for the correction, the
division itself where a, r or the product is near the ends of the range, and a
zero with its sign.  The FP64 form's parity rests on these being the correctly
rounded quotients; here the header itself, compiled for the CPU without
contraction, against IEEE division: random operands over the whole exponent
range, quotients next to the ends of a binade, special values on both sides,
quotients as near to a midpoint of two numbers as 53-bit operands allow, and
operands whose first product is farthest off."""
import os
import random
import shutil
import struct
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sphere_b200", "csrc")

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "sph_divisor.cuh"
static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double bits(uint64_t b) { double d; memcpy(&d, &b, 8); return d; }
static double mkd(uint64_t mant, int e)
{
    return bits(((uint64_t)(e + 1023) << 52) | (mant & ((1ull << 52) - 1)));
}
static long bad = 0, n = 0;
static void check(double a, double b)
{
    const double x = a / b, y = sph::Divisor(b).div(a);
    ++n;
    if (memcmp(&x, &y, 8) != 0 && !(std::isnan(x) && std::isnan(y))) {
        if (bad < 5) printf("a=%a b=%a: %a vs %a\n", a, b, x, y);
        ++bad;
    }
}
int main(int argc, char **argv)
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
    // the pairs of the file
    if (FILE *f = fopen(argv[argc - 1], "rb")) {
        double ab[2];
        while (fread(ab, 8, 2, f) == 2) check(ab[0], ab[1]);
        fclose(f);
    }
    printf("%ld %ld\n", n, bad);
    return bad != 0;
}
"""


def _next_to_midpoints(rng, count):
    """Pairs (a, b) of 53-bit integers with a / b the least distance from a
    midpoint: a 2^(53 or 54) = m b + d with m odd and d = +-1, +-3 (b odd)."""
    out = []
    while len(out) < count:
        # odd divisors over the binade, half of them near its upper end, where
        # the correction's margin is smallest
        b = (1 << 53) - 1 - 2 * rng.getrandbits(rng.randint(1, 40)) if len(out) % 2 else \
            (1 << 52) | rng.getrandbits(52) | 1
        for e in (53, 54):
            inv = pow(b, -1, 1 << e)
            for d in (1, -1, 3, -3):
                m = (-d * inv) % (1 << e)
                while m < 1 << 53:
                    m += 1 << e
                if m >= 1 << 54:
                    continue
                a = (m * b + d) >> e
                if 1 << 52 <= a < 1 << 53 and (a << e) == m * b + d and (e == 53) == (a >= b):
                    out.append((a, b))
    return out


def _first_product_far_off():
    """Both operands near the upper end of the binade, a < b."""
    top = (1 << 53) - 1
    return [(top - i, top - j) for j in range(0, 200) for i in range(j + 1, j + 40)]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_shared_divisor_quotients_are_correctly_rounded(tmp_path):
    src = os.path.join(str(tmp_path), "shared_div.cpp")
    exe = os.path.join(str(tmp_path), "shared_div")
    pairs = os.path.join(str(tmp_path), "pairs")
    with open(src, "w") as fh:
        fh.write(SOURCE)
    ab = _next_to_midpoints(random.Random(1), 60000) + _first_product_far_off()
    with open(pairs, "wb") as fh:
        for a, b in ab:
            fh.write(struct.pack("<2d", float(a), float(b)))
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", exe, src], check=True)
    out = subprocess.run([exe, pairs], capture_output=True, text=True, timeout=120)
    n, bad = (int(v) for v in out.stdout.split()[-2:])
    assert n == 4000000 + 2000 * 3000 + 18 * 18 + len(ab)
    assert out.returncode == 0 and bad == 0, out.stdout
