"""Boundary sites with one thread each in the general form (what a batch with many
sites on pressure and free-slip walls or under a force takes) against nine lanes a
site (a small case alone): bit for bit, for every condition, at edge lengths around
the warp size and the smallest lattice, both collisions and all storage forms."""
import numpy as np
import pytest

from cases import golden_cases, lattice_case
from life_gb300.case import CONVECTIVE, FREESLIP, PRESSURE, VELOCITY, WALL
from life_gb300.lib import Batch, Case

pytestmark = pytest.mark.gpu

SIZES = [(4, 4), (5, 34), (34, 5), (35, 66), (67, 33)]
STEPS = 11


def small_cases(cm, prec):
    kw = dict(central_moments=cm, precision=prec)
    out = []
    for nx, ny in SIZES:
        om = 1.0 / 0.6
        out.append(lattice_case(nx, ny, om, STEPS, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=FREESLIP,
                                wall_top=FREESLIP, uxInlet_p=0.04, ux0_p=0.03, **kw))
        out.append(lattice_case(nx, ny, om, STEPS, wall_left=VELOCITY, wall_right=PRESSURE, wall_bottom=WALL,
                                wall_top=FREESLIP, uxInlet_p=0.04, inlet_ramp=20.0, **kw))
        out.append(lattice_case(nx, ny, om, STEPS, wall_left=PRESSURE, wall_right=PRESSURE, wall_bottom=WALL,
                                wall_top=PRESSURE, ux0_p=0.02, **kw))
        out.append(lattice_case(nx, ny, om, STEPS, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=WALL,
                                wall_top=WALL, uxInlet_p=0.04, gravityX=1e-5, gravityY=-2e-5, **kw))
        out.append(lattice_case(nx, ny, om, STEPS, wall_bottom=WALL, wall_top=FREESLIP, womersley=4.0, dpdx=1e-5,
                                gravityY=-1e-5, **kw))
    golden = golden_cases()
    for name in ("channel_convective_freeslip_cm", "pressure_top_corners", "womersley_gravity_cm", "periodic_womersley"):
        out.append(golden[name][0].replace(**kw))
    return [(p, []) for p in out]


def filler(prec, cm):
    """A case whose walls and sites make the batch take the general form."""
    p = lattice_case(6000, 14, 1.0 / 0.6, STEPS, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=FREESLIP,
                     wall_top=FREESLIP, uxInlet_p=0.03, precision=prec, central_moments=cm)
    return p, []


@pytest.mark.parametrize("prec", [0, 1, 2], ids=["f64", "f32", "f16"])
@pytest.mark.parametrize("cm", [False, True], ids=["bgk", "cm"])
def test_general_form_equals_lane_form(cm, prec):
    items = small_cases(cm, prec)
    with Batch(items + [filler(prec, cm)]) as b:
        b.step(STEPS)
        got = [b.case(k).fields() for k in range(len(items))]
    for k, (p, bodies) in enumerate(items):
        with Case(p, bodies) as c:
            c.step(STEPS)
            want = c.fields()
        for key in ("rho", "u", "f"):
            assert np.array_equal(got[k][key], want[key], equal_nan=True), (k, p.Nx, p.Ny, key)


def test_outlet_term_from_its_kernel():
    """A lattice large enough for the one-launch step, in a batch: the general form
    reads the outlet's speed term that a kernel has formed."""
    p = lattice_case(2100, 2000, 1.0 / 0.6, 4, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=FREESLIP,
                     wall_top=FREESLIP, uxInlet_p=0.04, ux0_p=0.03, precision=1)
    with Batch([(p, []), filler(1, False)]) as b:
        b.step(4)
        got = b.case(0).fields(("rho", "u"))
    with Case(p, []) as c:
        c.step(4)
        want = c.fields(("rho", "u"))
    for key in want:
        assert np.array_equal(got[key], want[key]), key
