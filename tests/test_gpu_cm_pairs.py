"""Central moments with two sites a thread in packed FP32 (the TMA-staged step
kernel of lattices of 2^22 sites or more): the same bits as one site a thread
(LIFE_STEP_KERNEL=site) and as the separate kernels (LIFE_CASE_HOSTLOOP=1),
from a flow in which every site moves, at odd and even widths (a last pair
with one site outside), one column past a tile, with and without a force."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r"""
import hashlib, sys
import numpy as np
sys.path.insert(0, '.')
from life_gb300.case import CaseParams, CONVECTIVE, FLUID, VELOCITY, WALL
from life_gb300.lib import Case
kind, Nx, Ny, prec = sys.argv[1], int(sys.argv[2]), int(sys.argv[3]), int(sys.argv[4])
omega = 1.0 / 0.56
kw = dict(Nx=Nx, Ny=Ny, height_p=Ny - 1.0, rho_p=1.0, nu_p=(1.0 / omega - 0.5) / 3.0, omega=omega,
          central_moments=True, precision=prec, wall_bottom=WALL)
if kind == 'cavity':
    p = CaseParams(wall_left=WALL, wall_right=WALL, wall_top=VELOCITY, uxInlet_p=0.1, **kw)
elif kind == 'channel':
    p = CaseParams(wall_left=VELOCITY, wall_right=CONVECTIVE, wall_top=WALL, uxInlet_p=0.05, **kw)
else:
    p = CaseParams(wall_left=FLUID, wall_right=FLUID, wall_top=WALL, gravityX=2e-6, gravityY=-1e-6, **kw)
rng = np.random.default_rng(Nx)
with Case(p) as c:
    w = np.array([16, 4, 4, 4, 4, 1, 1, 1, 1]) / 36.0
    cv = np.array([[0, 0], [1, 0], [-1, 0], [0, 1], [0, -1], [1, 1], [-1, -1], [1, -1], [-1, 1]], dtype=float)
    f = w * (1.0 + 0.05 * rng.standard_normal((Nx, Ny, 9)))
    rho = f.sum(axis=2)
    c.set_fields(0, rho, (f @ cv) / rho[:, :, None], f)
    c.step(20)
    fl = c.fields(("rho", "u"))
assert np.isfinite(fl["u"]).all()
print("DIGEST", hashlib.sha256(fl["rho"].tobytes() + fl["u"].tobytes()).hexdigest())
"""


def digest(args, env):
    res = subprocess.run([sys.executable, "-c", CODE] + [str(a) for a in args], cwd=ROOT, capture_output=True,
                         text=True, env=dict(os.environ, **env))
    assert res.returncode == 0, res.stderr[-2000:]
    return [ln for ln in res.stdout.splitlines() if ln.startswith("DIGEST")][-1]


@pytest.mark.parametrize("prec", [1, 2])
@pytest.mark.parametrize("kind,Nx,Ny", [("cavity", 2049, 2048), ("channel", 2050, 2051), ("forced", 2176, 2047)])
def test_pairs_bit_identical(kind, Nx, Ny, prec):
    from life_gb300.build import build
    build()
    args = (kind, Nx, Ny, prec)
    pairs = digest(args, {"LIFE_STEP_KERNEL": "tma"})
    assert pairs == digest(args, {"LIFE_STEP_KERNEL": "site"}), "two sites a thread vs one"
    assert pairs == digest(args, {"LIFE_CASE_HOSTLOOP": "1"}), "one launch vs separate kernels"
