"""The spread of bodies with more markers than one range holds, and of bodies whose
marker counts lie around a range's: forces and fields bit for bit against the oracle,
with another body's markers reaching the same sites."""
import math

import numpy as np
import pytest

from cases import lattice_case
from life_gb300.case import CONVECTIVE, VELOCITY, WALL, Circle, Filament
from life_gb300.lib import Case
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu

STEPS = 7


def channel(nx, ny, cm=False):
    return lattice_case(nx, ny, 1.0 / 0.6, STEPS, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=WALL,
                        wall_top=WALL, uxInlet_p=0.05, ux0_p=0.05, central_moments=cm)


def rigid(x, y, length, angle, k):
    return Filament(x=x, y=y, length=length, height=1.0, angle_deg=angle, flexible=False, n_elements=None, clamped=True,
                    rho=1.0, E=1.0, ID=k)


@pytest.mark.parametrize("cm", [False, True], ids=["bgk", "cm"])
@pytest.mark.parametrize("markers", [127, 128, 129, 256, 257, 300])
def test_long_bodies(markers, cm):
    # a filament of about so many markers, crossed by a second one and near a circle
    nx = int(markers + 40)
    p = channel(nx, 64, cm)
    bodies = [rigid(15.0, 20.3, float(markers - 1), 0.0, 0), rigid(nx / 2.0, 12.2, 30.0, 80.0, 1),
              Circle(x=nx / 2.0 + 20.0, y=30.4, radius=9.6, ID=2)]
    o = Oracle(p, bodies)
    o.step(STEPS)
    want, wm = o.fields(), o.markers()
    with Case(p, bodies) as c:
        c.step(STEPS)
        got, gm = c.fields(), c.markers()
    for k in ("f", "rho", "u", "force_ibm"):
        assert np.array_equal(got[k], want[k]), k
    assert np.array_equal(gm["force"], wm["force"])


def test_large_circle():
    p = channel(200, 180)
    bodies = [Circle(x=95.3, y=90.2, radius=62.0)]
    o = Oracle(p, bodies)
    o.step(STEPS)
    want = o.fields()
    with Case(p, bodies) as c:
        assert c.n_markers > 2 * 128 and c.n_markers > math.pi * 2 * 60
        c.step(STEPS)
        got = c.fields()
    for k in ("f", "rho", "u", "force_ibm"):
        assert np.array_equal(got[k], want[k]), k
