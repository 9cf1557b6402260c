"""Straight walls and the convective outlet with one thread a site (the form
that cases of a batch take) against nine lanes a site (a small case alone): bit
for bit, at edge lengths around the warp size and the smallest lattice, for
both collisions and all storage forms, with a moving lid, a ramped inlet, and a
flow fast enough that sites leave the range of the thread form's integer
arithmetic (the general code)."""
import numpy as np
import pytest

from cases import lattice_case

pytestmark = pytest.mark.gpu

SIZES = [(4, 4), (5, 34), (34, 5), (35, 66), (67, 33), (130, 36)]


def _cases(cm, prec, speed):
    from life_gb300.case import CONVECTIVE, VELOCITY, WALL
    out = []
    for nx, ny in SIZES:
        out.append(lattice_case(nx, ny, 1.0 / 0.62, 12, wall_left=WALL, wall_right=WALL, wall_bottom=WALL,
                                wall_top=VELOCITY, uxInlet_p=speed, uyInlet_p=0.0, central_moments=cm, precision=prec))
        out.append(lattice_case(nx, ny, 1.0 / 0.58, 12, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=WALL,
                                wall_top=VELOCITY, uxInlet_p=speed, inlet_ramp=20.0, central_moments=cm, precision=prec))
    return [(p, []) for p in out]


@pytest.mark.parametrize("speed", [0.04, 0.2])
@pytest.mark.parametrize("prec", [0, 1, 2], ids=["f64", "f32", "f16"])
@pytest.mark.parametrize("cm", [False, True], ids=["bgk", "cm"])
def test_thread_form_equals_lane_form(cm, prec, speed):
    from life_gb300.build import build
    build()
    from life_gb300.lib import Batch, Case
    items = _cases(cm, prec, speed)
    with Batch(items) as b:
        b.step(12)
        got = [b.case(k).fields() for k in range(len(items))]
    for k, (p, bodies) in enumerate(items):
        with Case(p, bodies) as c:
            c.step(12)
            ref = c.fields()
        for key in ("rho", "u", "f"):
            assert np.array_equal(got[k][key], ref[key], equal_nan=True), (k, p.Nx, p.Ny, key)
