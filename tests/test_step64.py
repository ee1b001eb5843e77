"""The FP64 step kernel's helpers and decompositions.

  * On the CPU: the short divisions, roots, comparisons and the friction power
    of sw2d_f64math.cuh (which compiles as host C++) give the bits of the plain
    IEEE expressions and of the oracle's power, on random operands, operands
    with extreme mantissas, quotients and roots next to rounding midpoints, and
    zeros, infinities, NaN and subnormals.
  * On the GPU: every tile build gives the oracle's bits where it can go wrong:
    grids at and around the tile edges, a thin film on rough ground (dry-bed
    rules and momentum side by side), NODATA cells, roughness as a raster, a
    scalar and none, every kind of forcing, the open south edge.
"""
import os
import subprocess

import numpy as np
import pytest

from helpers import make_pair, same, set_forcing

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include "sw2d_f64math.cuh"
#include <cstdio>
#include <cstdlib>
#include <random>
using namespace sw2d;
extern "C" double orc_pow43(double);
extern "C" double orc_log(double);
static std::mt19937_64 R(17);
static double rnd(int lo, int hi) {
    unsigned long long m = R() & 0xfffffffffffffull;
    switch (R() % 8) {
    case 0: m &= 0xffull << 44; break;
    case 1: m |= 0xfffffffffff00ull; break;
    case 2: m = R() % 16; break;
    }
    return d_from_bits(((unsigned long long)(lo + (int)(R() % (unsigned)(hi - lo + 1)) + 1023) << 52) | m);
}
static bool eq(double a, double b) { return a == b || (a != a && b != b); }
static long bad = 0, taken = 0;
static void expect(bool ok, const char *what, double a, double b) {
    if (!ok && bad++ < 10) printf("%s %a %a\n", what, a, b);
}
static void pair(double a, double b) {
    expect(eq(d_div(a, b), a / b), "div", a, b);
    expect(d_lt(a, b) == (a < b), "lt", a, b);
}
static void one(double a) {
    expect(eq(d_sqrt(a), std::sqrt(a)), "sqrt", a, 0);
    expect(eq(d_half(a), 0.5 * a), "half", a, 0);
    expect(d_clamp0(a) == std::fmax(a, 0.0), "clamp", a, 0);
    expect(d_ge_pos(a, d_bits(1e-4)) == (a >= 1e-4), "ge", a, 0);
    expect(d_gt_zero(a) == (a > 0) && d_lt_zero(a) == (a < 0), "sign", a, 0);
    expect(d_is_nan(a) == (a != a) && d_is_finite(a) == (std::fabs(a) <= 1.7976931348623157e308), "class", a, 0);
}
int main(int, char **argv) {
    const long n = atol(argv[1]);
    PowTables *T = new PowTables;
    for (int k = 0; k < 128; k++) {
        const double c = 1.0 + k * 0.0078125;
        T->inv[k] = 1.0 / c;
        T->logc[k] = orc_log(c);
    }
    for (int j = 0; j < 64; j++) {
        const double y = (double)j * (0x1.62e42p-1 / 64.0) + (double)j * (0x1.fdf473de6af28p-22 / 64.0);
        const double kf = std::floor(y * 0x1.71547652b82fep+0 + 0.5);
        const double r = (y - kf * 0x1.62e42p-1) - kf * 0x1.fdf473de6af28p-22;
        double p = 1.0 / 6227020800.0;
        const double c[] = {1.0 / 479001600.0, 1.0 / 39916800.0, 1.0 / 3628800.0, 1.0 / 362880.0, 1.0 / 40320.0,
                            1.0 / 5040.0, 1.0 / 720.0, 1.0 / 120.0, 1.0 / 24.0, 1.0 / 6.0, 0.5, 1.0, 1.0};
        for (double q : c) p = p * r + q;
        T->exp2j[j] = std::ldexp(p, (int)kf);
    }
    for (int e = -kPowE; e < kPowE; e++) {
        T->ehi[e + kPowE] = (double)e * 0x1.62e42p-1;
        T->elo[e + kPowE] = (double)e * 0x1.fdf473de6af28p-22;
    }
    for (int k = -kPowN; k < kPowN; k++) {
        T->nhi[k + kPowN] = (double)k * (0x1.62e42p-1 / 64.0);
        T->nlo[k + kPowN] = (double)k * (0x1.fdf473de6af28p-22 / 64.0);
    }
    for (long i = 0; i < n; i++) {
        const double a = rnd(-40, 40) * ((R() & 1) ? 1 : -1), b = rnd(-20, 20), d = rnd(-8, 8);
        pair(a, b);
        expect(d_div_known(a, known_divisor(d)) == a / d, "div_known", a, d);
        one(a);
        one(std::fabs(a));
        const double m = rnd(0, 0), near = d_fma(b, m, b * 0x1p-53 * m * 0.5);  // a quotient by a midpoint
        for (int t = -1; t <= 1; t++) {
            const double x = d_from_bits(d_bits(near) + (unsigned long long)(long long)t);
            pair(x, b);
            expect(d_div_known(x, known_divisor(b)) == x / b, "div_known", x, b);
        }
        const double s = rnd(-20, 20);
        one(d_from_bits(d_bits(s * s) + R() % 5 - 2));
        bool ok;
        const double h = rnd(-14, 8), pw = d_pow43_fast(h, T, &ok);
        expect(ok && pw == orc_pow43(h), "pow", h, pw);
        const double pi = d_pow43_int(h, T, &ok);
        taken += ok;
        expect(!ok || pi == orc_pow43(h), "pow_int", h, pi);
        expect(std::fabs((double)d_abs_float(a) - std::fabs(a)) <= std::fabs(a) * 0x1p-23, "float", a, 0);
    }
    const double sp[] = {0.0, -0.0, HUGE_VAL, -HUGE_VAL, std::nan(""), 5e-324, -5e-324, 1e-310, 1e-300, 1e300, -1e300,
                         1e-4, 1.0, -1.0};
    for (double a : sp) {
        one(a);
        for (double b : sp) pair(a, b);
    }
    expect(taken > n / 2, "pow_int covers too few", (double)taken, 0);
    printf("bad %ld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.parametrize("seed_ulps", [-2, 0, 2])
def test_f64_helpers_give_the_plain_bits(oracle_mod, tmp_path, seed_ulps):
    """With exact FP32 seeds and with seeds off by more than the device's
    approximations are (one ulp)."""
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(CHECK)
    so = os.path.join(ROOT, "oracle", "_build", "liboracle.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-DSW2D_SEED_ULPS={seed_ulps}", "-I",
                    os.path.join(ROOT, "sw2d-gpu_gb300", "csrc"), str(src), so, "-Wl,-rpath," + os.path.dirname(so),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), "200000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


TILES = [(16, 32), (8, 32), (8, 16), (4, 16), (4, 8)]


def _film(rows, cols, seed, holes):
    rng = np.random.default_rng(seed)
    z = 0.05 * np.arange(rows)[::-1, None] + rng.uniform(0.0, 0.2, (rows, cols))
    h = np.where(rng.random((rows, cols)) < 0.3, 0.0, rng.uniform(0.0, 0.15, (rows, cols)))
    if holes:
        z[rng.random(z.shape) < 0.06] = -9999.0
    return z, h, rng


@pytest.mark.gpu
@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("shape", [(1, 1), (3, 7), (4, 8), (5, 9), (16, 32), (17, 33), (33, 65), (70, 41)])
def test_step64_tiles_match_the_oracle(oracle_mod, sw2d_mod, tile, shape):
    """Bit for bit, friction included: the kernel and the oracle round the same
    operations."""
    rows, cols = shape
    for form in range(4):
        z, h, rng = _film(rows, cols, 100 * rows + cols + form, holes=form == 1)
        n = rng.choice([0.0, 0.03, 0.12], (rows, cols)) if form in (0, 1) else None
        kw = dict(INT=0.2, INF=0.1, LWL=0.3, EV_WL_min=0.01) if form == 3 else {}
        o, g = make_pair(oracle_mod, sw2d_mod, rows, cols, 4.0, z, h, n=n, manning=0.05 if form == 3 else 0.0,
                         south_open=form % 2, dt_mode=0 if form == 3 else 1, dt=0.05 if form == 3 else 1.0, dy=3.0,
                         tile=tile, **kw)
        if form == 2:
            set_forcing(oracle_mod, o, g, storm={"peak": 200.0, "x0": 0.0, "y0": 0.0, "vx": 1.0, "vy": 1.0,
                                                 "sigma": 40.0})
        elif form == 3:
            cells = np.array([0, rows * cols - 1], dtype=np.int32)
            set_forcing(oracle_mod, o, g, rain_kind=1, rain=np.array([4.0, 9.0, 2.0]), rain_dt=50.7,
                        ev=np.array([0.5, 0.7]), ev_dt=60.3, sources=cells,
                        src_q=np.array([[0.02, 0.01], [0.05, 0.0]]), dtoq=70.1)
        else:
            set_forcing(oracle_mod, o, g, rain_kind=2, rain=np.array([120.0]), rain_dt=3600.0)
        assert o.advance(40, 1e9) == g.advance(40, 1e9) == 40
        a, b = o.state(), g.state()
        for k in ("h", "um", "vn"):
            assert same(a[k], b[k]), (form, k, np.max(np.abs(a[k] - b[k])))
        bo, bg = o.budget(), g.budget()
        assert bg["cmax"] == bo["cmax"] and bg["t"] == a["t"]
        for k in ("rain_in", "source_in", "evap_out", "outflow", "clamp_gain"):
            assert bg[k] == pytest.approx(bo[k], rel=1e-12, abs=1e-14), k  # sums in another order
        g.close()


@pytest.mark.gpu
def test_step64_tile_rule(sw2d_mod):
    """The smallest tile that gives at most one CTA per SM; a caller's tile is
    kept."""
    for rows, cols, kw, name in ((64, 64, {}, "4,8"), (117, 131, {}, "8,16"), (512, 512, {}, "16,32"),
                                 (64, 64, dict(tile_h=8, tile_w=32), "8,32")):
        with sw2d_mod.Solver(rows=rows, cols=cols, dx=1.0, dy=1.0, **kw) as g:
            assert g.describe().startswith("step_kernel<double,%s>" % name), g.describe()


@pytest.mark.gpu
@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("shape", [(16, 32), (37, 70)])
def test_step64_every_flux_at_once(oracle_mod, sw2d_mod, tile, shape):
    """Deep water moving everywhere: all four fluxes of every element are
    formed, so a warp's list is flushed before its last block of elements."""
    rows, cols = shape
    rng = np.random.default_rng(rows)
    z = rng.uniform(0.0, 0.1, shape)
    h = rng.uniform(2.0, 3.0, shape)
    o, g = make_pair(oracle_mod, sw2d_mod, rows, cols, 4.0, z, h, n=rng.uniform(0.02, 0.1, shape), dt=0.1, tile=tile)
    assert o.advance(20, 1e9) == g.advance(20, 1e9) == 20
    a, b = o.state(), g.state()
    assert np.count_nonzero(a["um"]) >= (rows - 1) * cols and np.count_nonzero(a["vn"]) >= rows * (cols - 1)
    for k in ("h", "um", "vn"):
        assert same(a[k], b[k]), (k, np.max(np.abs(a[k] - b[k])))
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("tile", [(14, 32), (12, 32), (10, 32), (6, 32)])
@pytest.mark.parametrize("shape", [(1, 33), (6, 32), (15, 31), (41, 66)])
def test_step64_tiles_between_match_the_oracle(oracle_mod, sw2d_mod, tile, shape):
    """The tile heights between 4 and 16, as above: film with NODATA cells,
    storm, rain with evaporation and point sources; rows that the tile divides,
    one less, one more."""
    test_step64_tiles_match_the_oracle(oracle_mod, sw2d_mod, tile, shape)


@pytest.mark.gpu
def test_step64_tile_rule_fills_the_sms(sw2d_mod):
    """Where no SM, or no SM more than two, CTAs: the smallest tile that leaves
    it so (152 SMs)."""
    for rows, cols, name in ((150, 150, "6,32"), (180, 256, "10,32"), (200, 256, "12,32"), (256, 256, "14,32"),
                             (256, 512, "14,32"), (300, 500, "16,32"), (256, 300, "16,32"), (1013, 900, "16,32")):
        with sw2d_mod.Solver(rows=rows, cols=cols, dx=1.0, dy=1.0) as g:
            assert g.describe().startswith("step_kernel<double,%s>" % name), g.describe()
