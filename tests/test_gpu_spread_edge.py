"""The spread beside the boundary sites (rigid bodies whose support stays off the
edges of the lattice) and after them (support on an edge): captured steps
against steps launched one after another from the host, bit for bit, with the
support one site off an edge, on it and cut by it, and after markers were moved
onto an edge between captured runs."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = r"""
import hashlib, sys
sys.path.insert(0, '.'); sys.path.insert(0, 'tests/golden')
from cases import lattice_case
from life_gb300.case import CONVECTIVE, VELOCITY, WALL, Circle
from life_gb300.lib import Case
x, y, prec, shift = float(sys.argv[1]), float(sys.argv[2]), int(sys.argv[3]), float(sys.argv[4])
p = lattice_case(96, 48, 1.0 / 0.6, 100, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=WALL, wall_top=WALL,
                 uxInlet_p=0.05, precision=prec)
with Case(p, [Circle(x, y, 4.0)]) as c:
    c.step(100)
    if shift:
        m = c.markers()
        m['pos'][:, 1] += shift
        c.set_markers(m['pos'], m['vel'], m['force'])
        c.step(100)
    fl = c.fields()
    mk = c.markers()
print("DIGEST", hashlib.sha256(fl["rho"].tobytes() + fl["u"].tobytes() + mk["force"].tobytes()).hexdigest())
"""


def digest(args, env):
    res = subprocess.run([sys.executable, "-c", CODE] + [str(a) for a in args], cwd=ROOT, capture_output=True,
                         text=True, env=dict(os.environ, **env))
    assert res.returncode == 0, res.stderr[-2000:]
    return [ln for ln in res.stdout.splitlines() if ln.startswith("DIGEST")][-1]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("x,y,shift", [(40.0, 24.0, 0.0), (40.0, 6.5, 0.0), (40.0, 5.4, 0.0), (40.0, 4.0, 0.0),
                                       (90.0, 24.0, 0.0), (40.0, 7.0, -2.0)])
def test_beside_equals_after(x, y, shift, prec):
    from life_gb300.build import build
    build()
    args = (x, y, prec, shift)
    assert digest(args, {}) == digest(args, {"LIFE_CASE_HOSTLOOP": "1"})
