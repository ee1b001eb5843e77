"""The FP64 helpers of sw2d_f64math.cuh over the whole exponent range: a
quotient that overflows, underflows or is subnormal, and operands at the ends
of the range, give the bits of the plain IEEE expression, as they do in the
middle of it (test_step64.py)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include "sw2d_f64math.cuh"
#include <cstdio>
#include <random>
using namespace sw2d;
static std::mt19937_64 R(29);
static bool eq(double a, double b) { return d_bits(a) == d_bits(b) || (a != a && b != b); }
static long bad = 0;
static void expect(bool ok, const char *what, double a, double b) {
    if (!ok && bad++ < 10) printf("%s %a %a\n", what, a, b);
}
static double at(int field) {  // a double of that exponent field (0: subnormal), either sign
    return d_from_bits((R() & 0x800fffffffffffffull) | ((unsigned long long)field << 52));
}
static void both(double a, double b) {
    expect(eq(d_div(a, b), a / b), "div", a, b);
    const double d = std::fabs(b);
    if (d > 0 && d < HUGE_VAL) {
        const double q = d_div_known(a, known_divisor(d));
        expect(q == a / d || (q != q && a != a), "div_known", a, d);  // a zero of either sign is itself
    }
}
int main() {
    for (int i = 0; i < 2000000; i++) both(at((int)(R() % 2047)), at((int)(R() % 2047)));
    // the differences of the exponents at which a quotient leaves the normal range
    for (int d = -1100; d <= 1100; d++)
        for (int k = 0; k < 40; k++) {
            const int lo = d < 0 ? 1 - d : 1, hi = d < 0 ? 2046 : 2046 - d;
            if (lo > hi) continue;
            const int fb = lo + (int)(R() % (unsigned)(hi - lo + 1));
            both(at(fb + d), at(fb));
        }
    for (int f = 0; f < 2047; f++)
        for (int k = 0; k < 200; k++) {
            const double a = at(f);
            expect(eq(d_sqrt(a), std::sqrt(a)), "sqrt", a, 0);
            expect(eq(d_half(a), 0.5 * a), "half", a, 0);
            const double b = at(f);
            expect(d_lt(a, b) == (a < b), "lt", a, b);
        }
    printf("bad %ld\n", bad);
    return bad != 0;
}
"""


def test_helpers_give_the_plain_bits_at_every_exponent(tmp_path):
    src, exe = tmp_path / "range.cpp", tmp_path / "range"
    src.write_text(CHECK)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "sw2d-gpu_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
