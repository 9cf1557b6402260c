"""The moment sums and collisions on the integer units (``int_f64.cuh``,
``collide_cm.cuh``) at the upper end of the accepted range: populations just below 1,
all nine alike, densities on both sides of 8 (where a sum in units of 2^-60 passes
2^63) and up to 9, compared bit for bit with the written-out forms. Compiled here for
the host (no GPU is used)."""
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
    long long above = 0, below = 0;
    static const double alike[] = {0x1.fffffffffffffp-1, 0.9, 0.95, 8.0 / 9.0, 0x1.c71c71c71c71dp-1, 0.875, 0x1.bffffffffffffp-1};
    for (long long q = 0; q < n; q++) {
        double f[9], r, mx, my, ri, mxi, myi;
        const int kind = (int)(rnd() % 4);
        const double a = alike[rnd() % 7];
        for (int v = 0; v < 9; v++) {
            // alike; in [7/8, 1); about 8/9 (a density near 8); dense significands below 1
            f[v] = kind == 0 ? a : kind == 1 ? 0.875 + 0.125 * unit() : kind == 2 ? 8.0 / 9.0 + 0x1p-40 * (unit() - 0.5)
                                                                                  : std::fabs(number(-1));
        }
        if (kind == 2) f[rnd() % 9] += (unit() - 0.5) * (rnd() & 1 ? 0x1p-4 : 0x1p-44);
        if (!populations_in_range(f)) bad++;
        moment_sums(f, r, mx, my);
        moment_sums_int(f, ri, mxi, myi);
        (r >= 8.0 ? above : below)++;
        same("rho", ri, r, f[0], f[1]);
        same("mx", mxi, mx, f[1], f[2]);
        same("my", myi, my, f[3], f[4]);
        const double ux = velocity(), uy = velocity(), omega = 0.05 + 1.9 * unit();
        double want[9], got[9];
        collide_bgk<true>(f, r, ux, uy, 0.0, 0.0, omega, want);
        collide_bgk_int(f, ri, ux, uy, omega, got);
        for (int v = 0; v < 9; v++) same("bgk", got[v], want[v], ux, uy);
        collide_cm<true>(f, r, ux, uy, 0.0, 0.0, omega, cs, want);
        collide_cm_int(f, ri, ux, uy, 1.0 - omega, cs2v, cs4, got);
        for (int v = 0; v < 9; v++) same("cm", got[v], want[v], ux, uy);
    }
    printf("%lld %lld %lld\n", above, below, bad);
    return 0;
}
"""


@pytest.fixture(scope="module")
def driver():
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    d = tempfile.mkdtemp(prefix="int_f64_upper_")
    src, exe = os.path.join(d, "int_f64_upper.cu"), os.path.join(d, "int_f64_upper")
    with open(src, "w") as fh:
        fh.write(DRIVER)
    inc = os.path.join(os.path.dirname(CSRC), "..", "include")
    cmd = [nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "--fmad=false",
           "-Xcompiler", "-ffp-contract=off", "-I", CSRC, "-I", inc, src, "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    yield exe
    shutil.rmtree(d, ignore_errors=True)


@pytest.mark.parametrize("seed", [5, 20261206])
def test_sums_up_to_nine(driver, seed):
    n = 1000000
    res = subprocess.run([driver, str(seed), str(n)], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr
    above, below, bad = map(int, res.stdout.split()[-3:])
    assert above > n // 5 and below > n // 5
    assert bad == 0, res.stdout
