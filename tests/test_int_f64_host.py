"""FP64 arithmetic on the integer units (``life_gb300/csrc/int_f64.cuh``) and
the site collisions that use it (``collide_bgk_int``, ``collide_cm_int`` in
``collide_cm.cuh``), compiled here for the host (nvcc, host code only: no GPU is
used) and compared bit for bit with IEEE arithmetic and with the written-out
collisions: products of normal operands and zeros, ties and long carries; sums
with a power of two; the moment sums over the accepted range of populations;
whole sites over the accepted range, at its edges and at rest. Values just
outside the range must be refused."""
import os
import shutil
import subprocess
import tempfile

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "life_gb300", "csrc")

DRIVER = r"""
#include "collide_cm.cuh"
#include <cstdint>
#include <cstdio>
#include <cstdlib>
using namespace life;

static uint64_t state;
static uint64_t rnd() {
    uint64_t z = (state += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
static double unit() { return (double)(rnd() >> 11) * 0x1p-53; }
static long long bad = 0;
static void same(const char* what, double got, double want, double a, double b) {
    if (div_bits(got) != div_bits(want) && bad++ < 8) printf("%s(%a, %a) = %a, not %a\n", what, a, b, got, want);
}
// a double of exponent e with random, sparse or dense significands
static double number(int e) {
    uint64_t m = rnd() & 0xfffffffffffffull;
    const int cut = (int)(rnd() % 53);
    switch (rnd() % 4) {
        case 0: m &= ~0ull << cut; break;
        case 1: m |= ((1ull << cut) - 1); break;
        default: break;
    }
    return bits_double((rnd() & 0x8000000000000000ull) | (uint64_t)(1023 + e) << 52 | (m & 0xfffffffffffffull));
}
static double velocity() {
    static const double edge[] = {0.0, -0.0, 0.05, -0.05, 0x1p-60, -0x1p-60, 0x1.fffffffffffffp-4, -0x1.fffffffffffffp-4, 0x1p-4};
    switch (rnd() % 4) {
        case 0: return edge[rnd() % 9];
        case 1: return number(-4 - (int)(rnd() % 57));
        default: return 0.2 * (unit() - 0.5);
    }
}

int main(int argc, char** argv) {
    state = strtoull(argv[1], nullptr, 10);
    const long long n = atoll(argv[2]);
    const double cs = 1.0 / std::sqrt(3.0);
    volatile double cs2v = cs * cs;
    const double cs4 = cs * cs * cs * cs;
    long long refused = 0;
    for (long long q = 0; q < n; q++) {
        const double a = rnd() % 32 ? number((int)(rnd() % 600) - 300) : (rnd() & 1 ? 0.0 : -0.0);
        const double b = rnd() % 32 ? number((int)(rnd() % 600) - 300) : 0.0;
        same("mul", mul_int<kZeroAny>(a, b), a * b, a, b);
        if (b != 0.0) same("mul<A>", mul_int(a, b), a == 0.0 ? 0.0 : a * b, a, b);
        if (a != 0.0 && b != 0.0) same("mul<nz>", mul_int<kNonZero>(a, b), a * b, a, b);
        const double x = rnd() % 32 ? number(-1 - (int)(rnd() % 80)) : (rnd() & 1 ? 0.0 : -0.0);
        same("1 +", add_pow2_int<0>(x), 1.0 + x, 1.0, x);
        same("2 +", add_pow2_int<1>(2.0 * x), 2.0 + 2.0 * x, 2.0, 2.0 * x);
        same("1/2 +", add_pow2_int<-1>(0.5 * x), 0.5 + 0.5 * x, 0.5, 0.5 * x);

        double f[9], r, mx, my, ri, mxi, myi;
        const int kind = (int)(rnd() % 4);
        for (int v = 0; v < 9; v++) {
            const double w = v == 0 ? 4.0 / 9.0 : (v < 5 ? 1.0 / 9.0 : 1.0 / 36.0);
            f[v] = kind == 0 ? std::fabs(number(-1 - (int)(rnd() % 8))) : w * (1.0 + (kind == 1 ? 0.6 : 0.01) * (unit() - 0.5));
        }
        if (kind == 2) { f[2] = f[1]; f[4] = f[3]; f[6] = f[5]; f[8] = f[7]; }
        if (!populations_in_range(f)) bad++;
        moment_sums(f, r, mx, my);
        moment_sums_int(f, ri, mxi, myi);
        same("rho", ri, r, f[0], f[1]);
        same("mx", mxi, mx, f[1], f[2]);
        same("my", myi, my, f[3], f[4]);

        const double ux = velocity(), uy = rnd() % 16 ? velocity() : (rnd() & 1 ? ux : -ux);
        const double omega = rnd() % 16 ? 0.5 + 1.45 * unit() : 1.0;
        if (!site_range_ok(ux, uy, omega)) bad++;
        double want[9], got[9];
        collide_bgk<true>(f, r, ux, uy, 0.0, 0.0, omega, want);
        collide_bgk_int(f, r, ux, uy, omega, got);
        for (int v = 0; v < 9; v++) same("bgk", got[v], want[v], ux, uy);
        collide_cm<true>(f, r, ux, uy, 0.0, 0.0, omega, cs, want);
        collide_cm_int(f, r, ux, uy, 1.0 - omega, cs2v, cs4, got);
        for (int v = 0; v < 9; v++) same("cm", got[v], want[v], ux, uy);

        // one value out of range
        double g[9];
        for (int v = 0; v < 9; v++) g[v] = f[v];
        static const double out[] = {0.0, -0.1, 0x1.fffffffffffffp-9, 1.0, 0x1p-1040, 1.0 / 0.0, 0.0 / 0.0};
        g[rnd() % 9] = out[rnd() % 7];
        static const double uout[] = {0x1p-3, -0x1p-3, 0x1.fffffffffffffp-61, 0x1p-1040, 1.0 / 0.0, 0.0 / 0.0};
        if (populations_in_range(g) || site_range_ok(uout[rnd() % 6], uy, omega) || site_range_ok(ux, uout[rnd() % 6], omega) ||
            site_range_ok(ux, uy, 0.0) || site_range_ok(ux, uy, -1.0) || site_range_ok(ux, uy, 4.0))
            bad++;
        else
            refused++;
    }
    printf("%lld %lld\n", refused, bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def driver():
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    d = tempfile.mkdtemp(prefix="int_f64_")
    src, exe = os.path.join(d, "int_f64_host.cu"), os.path.join(d, "int_f64_host")
    with open(src, "w") as fh:
        fh.write(DRIVER)
    inc = os.path.join(os.path.dirname(CSRC), "..", "include")
    cmd = [nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "--fmad=false",
           "-Xcompiler", "-ffp-contract=off", "-I", CSRC, "-I", inc, src, "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    yield exe
    shutil.rmtree(d, ignore_errors=True)


@pytest.mark.parametrize("seed", [3, 777, 20261205])
def test_integer_arithmetic_equals_ieee(driver, seed):
    n = 2000000
    res = subprocess.run([driver, str(seed), str(n)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr
    refused, bad = map(int, res.stdout.split()[-2:])
    assert bad == 0, res.stdout
    assert refused == n
