"""The one-population form of the FP64 central-moment collision
(``cm_population`` in ``life_gb300/csrc/collide_cm.cuh``, used where a warp's
lanes hold the nine populations of a site) takes the power-of-two factors out
of the written-out polynomials of ``collide_cm`` and serves every direction
with one expression. Both are compiled here for the host (nvcc, host code
only: no GPU is used) and compared bit for bit on seeded sites: velocities
and moments of a flow, exact zeros of either sign, equal and opposite
components, and magnitudes down to the edge of the range that
``cm_factored_ok`` accepts, with and without a force. Outside that range the
guard must refuse.
"""
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

static uint64_t state;
static uint64_t rnd() {
    uint64_t z = (state += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
static double unit() { return (double)(rnd() >> 11) * 0x1p-53; }
static double velocity(int kind, int sub) {
    static const double pool[] = {0.0, -0.0, 0.05, -0.05, 0.25, 0x1p-60, -0x1p-59};
    if (kind == 0) return pool[rnd() % 7];
    const double s = rnd() & 1 ? 1.0 : -1.0;
    if (kind == 1) return s * unit() * std::ldexp(1.0, -(int)(rnd() % 59));
    if (kind == 2 && sub) return s * std::ldexp(1.0 + unit(), -70 - (int)(rnd() % 200));
    return s * 0.15 * unit();
}

int main(int argc, char** argv) {
    state = strtoull(argv[1], nullptr, 10);
    const long long n = atoll(argv[2]);
    const double cs = 1.0 / std::sqrt(3.0);
    long long bad = 0, refused = 0;
    for (long long q = 0; q < n; q++) {
        double f[9], r, mx, my;
        for (int v = 0; v < 9; v++) f[v] = (v == 0 ? 4.0 / 9.0 : (v < 5 ? 1.0 / 9.0 : 1.0 / 36.0)) * (1.0 + 0.1 * (unit() - 0.5));
        life::moment_sums(f, r, mx, my);
        const int kind = (int)(rnd() % 4);
        double ux = velocity(kind, rnd() & 1), uy = velocity(kind, rnd() & 1);
        if (rnd() % 16 == 0) uy = rnd() & 1 ? ux : -ux;
        const bool forced = rnd() & 1;
        double Fx = forced ? (unit() - 0.5) * 1e-4 : 0.0, Fy = forced && (rnd() & 3) ? (unit() - 0.5) * 1e-6 : 0.0;
        const double omega = 0.6 + 1.3 * unit();
        double want[9];
        life::collide_cm<false>(f, r, ux, uy, Fx, Fy, omega, cs, want);
        // the two sums of collide_cm, term by term
        double k4 = 0.0, k5 = 0.0;
        for (int v = 0; v < 9; v++) {
            const double cx = life::cx_of(v) - ux, cy = life::cy_of(v) - uy;
            const double t4 = f[v] * (cx * cx - cy * cy), t5 = f[v] * cx * cy;
            k4 = v == 0 ? t4 : k4 + t4;
            k5 = v == 0 ? t5 : k5 + t5;
        }
        life::CmSite c;
        life::cm_site<false>(c, r, ux, uy, Fx, Fy, life::pos_zero(k4), life::pos_zero(k5), omega, cs);
        const bool small = (ux != 0.0 && std::fabs(ux) < 0x1p-60) || (uy != 0.0 && std::fabs(uy) < 0x1p-60);
        if (life::cm_factored_ok(c) == small) bad++;
        if (!life::cm_factored_ok(c)) {
            refused++;
            continue;
        }
        for (int v = 0; v < 9; v++) {
            const double got = life::cm_population(life::cx_of(v), life::cy_of(v), c, Fx != 0.0 || Fy != 0.0);
            if (life::div_bits(got) != life::div_bits(want[v])) {
                if (bad < 5) printf("v %d ux %a uy %a F %a %a: %a / %a\n", v, ux, uy, Fx, Fy, got, want[v]);
                bad++;
            }
        }
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
    d = tempfile.mkdtemp(prefix="cm_factored_")
    src, exe = os.path.join(d, "cm_factored_host.cu"), os.path.join(d, "cm_factored_host")
    with open(src, "w") as fh:
        fh.write(DRIVER)
    inc = os.path.join(os.path.dirname(CSRC), "..", "include")
    cmd = [nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "--fmad=false",
           "-Xcompiler", "-ffp-contract=off", "-I", CSRC, "-I", inc, src, "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    yield exe
    shutil.rmtree(d, ignore_errors=True)


@pytest.mark.parametrize("seed", [5, 1234, 20261205])
def test_one_population_form_equals_the_written_out_collision(driver, seed):
    res = subprocess.run([driver, str(seed), "1000000"], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stderr
    refused, bad = map(int, res.stdout.split()[-2:])
    assert refused > 10000
    assert bad == 0, res.stdout
