"""Which form the boundary sites of a step take (``wall_plan.h``, compiled here for
the host): nine lanes a site while they are few, one thread a site with shared
products for straight no-slip and velocity walls and the outlet, and one thread a
site in the general form once the sites that the shared products cannot take
(pressure and free-slip walls, any wall under a force) are many, alone or in a
batch. Every boundary site is in exactly one place of the launch."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "life_gb300", "csrc")

DRIVER = r"""
#include "wall_plan.h"
#include <cstdio>
#include <cstdlib>
using namespace life;
int main(int argc, char** argv) {
    // nx ny left right bottom top prec cm force others_sites others_slow outlet_form
    long long v[12];
    for (int k = 0; k < 12; k++) v[k] = atoll(argv[k + 1]);
    LatDev L{};
    L.Nx = (int)v[0]; L.Ny = (int)v[1];
    for (int k = 0; k < 4; k++) L.wall[k] = (int)v[2 + k];
    L.prec = (int)v[6]; L.cm = (int)v[7]; L.Fx0 = v[8] ? 1e-6 : 0.0;
    L.others_sites = v[9]; L.others_slow = (int)v[10]; L.outlet_form = (int)v[11];
    const WallPlan p = wall_plan(L);
    printf("%d %d %d %d %d %d %d\n", p.general, p.lanes, p.straight, p.lane_sites, p.lane_warps, p.warps, slow_wall_sites(L));
    return 0;
}
"""
FLUID, WALL, VELOCITY, FREESLIP, PRESSURE, CONVECTIVE = range(6)
F64, F32, F16 = range(3)


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("wall_plan")
    src, exe = d / "wall_plan.cpp", d / "wall_plan"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-O1", "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return str(exe)


def plan(driver, nx, ny, walls, prec=F32, cm=0, force=0, others=(0, 0), outlet=1):
    args = [nx, ny, *walls, prec, cm, force, *others, outlet]
    out = subprocess.run([driver] + [str(int(a)) for a in args], capture_output=True, text=True, check=True).stdout
    return dict(zip(("general", "lanes", "straight", "lane_sites", "lane_warps", "warps", "slow"), map(int, out.split())))


CHANNEL = (VELOCITY, CONVECTIVE, WALL, WALL)
SLIP = (VELOCITY, CONVECTIVE, FREESLIP, FREESLIP)
OPEN = (VELOCITY, PRESSURE, WALL, WALL)
PERIODIC = (FLUID, FLUID, WALL, WALL)


@pytest.mark.parametrize("nx,ny,walls,kw,form", [
    (400, 100, CHANNEL, {}, "lanes"),                                  # few sites
    (1501, 703, CHANNEL, {}, "straight"),
    (400, 100, CHANNEL, dict(others=(1000, 0)), "straight"),           # in a batch
    (1501, 703, SLIP, {}, "both"),                                     # 2998 slow sites
    (20000, 64, CHANNEL, {}, "straight"),
    (20000, 64, SLIP, {}, "general"),
    (20000, 64, SLIP, dict(cm=1), "general"),
    (20000, 64, SLIP, dict(prec=F16), "general"),
    (20000, 64, PERIODIC, dict(force=1), "general"),
    (20000, 64, PERIODIC, dict(force=1, prec=F64), "general"),
    (64, 20000, OPEN, {}, "general"),
    (1000, 100, PERIODIC, dict(force=1), "lanes"),
    (3201, 64, SLIP, {}, "both"), (3202, 64, SLIP, {}, "general"),     # 6398, 6400 slow sites
    (2401, 64, SLIP, dict(cm=1), "both"), (2402, 64, SLIP, dict(cm=1), "general"),
    (1751, 64, SLIP, dict(prec=F64), "both"), (1752, 64, SLIP, dict(prec=F64), "general"),
    (499, 100, PERIODIC, dict(force=1, prec=F64), "lanes"), (500, 100, PERIODIC, dict(force=1, prec=F64), "general"),
    (299, 100, PERIODIC, dict(force=1, prec=F64, cm=1), "lanes"),
    (300, 100, PERIODIC, dict(force=1, prec=F64, cm=1), "general"),
    (502, 100, SLIP, dict(others=(10 ** 6, 2999)), "both"), (502, 100, SLIP, dict(others=(10 ** 6, 3000)), "general"),
    (502, 100, CHANNEL, dict(others=(10 ** 6, 10 ** 6)), "straight"),  # nothing slow of its own
])
def test_form(driver, nx, ny, walls, kw, form):
    p = plan(driver, nx, ny, walls, **kw)
    got = "general" if p["general"] else {(True, False): "lanes", (False, True): "straight", (True, True): "both"}[
        (p["lanes"] > 0, p["straight"] > 0)]
    assert got == form, p


@pytest.mark.parametrize("walls", [CHANNEL, SLIP, OPEN, PERIODIC, (WALL,) * 4, (FLUID,) * 4])
@pytest.mark.parametrize("nx,ny", [(4, 4), (35, 34), (1501, 703), (7000, 40)])
@pytest.mark.parametrize("kw", [{}, dict(force=1), dict(others=(1, 0)), dict(outlet=0)])
def test_every_site_once(driver, nx, ny, walls, kw):
    p = plan(driver, nx, ny, walls, **kw)
    sites = [nx - 2, nx - 2, ny - 2, ny - 2]
    types = [walls[2], walls[3], walls[0], walls[1]]
    if p["general"]:
        assert p["warps"] * 32 >= 2 * nx + 2 * (ny - 2) > (p["warps"] - 1) * 32
        return
    assert p["lanes"] & p["straight"] == 0
    assert p["lanes"] | p["straight"] == sum(1 << e for e in range(4) if types[e] != FLUID)
    assert p["lane_sites"] == 4 + sum(sites[e] for e in range(4) if p["lanes"] >> e & 1)
    assert p["lane_warps"] == -(-p["lane_sites"] // 3)
    assert p["warps"] == p["lane_warps"] + sum(-(-sites[e] // 32) for e in range(4) if p["straight"] >> e & 1)
