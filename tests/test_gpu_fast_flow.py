"""FP64 lattices whose flow is faster than the integer products' range (1/8 in a
component), in part of the sites and in all of them: alone and in a batch, bit for
bit against the oracle."""
import numpy as np
import pytest

from cases import lattice_case
from life_gb300.case import CONVECTIVE, VELOCITY, WALL
from life_gb300.lib import Batch, Case
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu

STEPS = 9


def cases(cm):
    kw = dict(central_moments=cm, precision=0)
    om = 1.0 / 0.6
    return [
        lattice_case(67, 33, om, STEPS, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=WALL, wall_top=WALL,
                     uxInlet_p=0.2, ux0_p=0.2, **kw),
        lattice_case(33, 40, om, STEPS, wall_left=WALL, wall_right=WALL, wall_bottom=WALL, wall_top=VELOCITY,
                     uxInlet_p=0.3, **kw),
        lattice_case(35, 31, om, STEPS, ux0_p=0.14, uy0_p=-0.17, **kw),           # periodic
        lattice_case(64, 32, om, STEPS, ux0_p=0.125, uy0_p=0.0, **kw),            # at the range's edge
        lattice_case(64, 32, om, STEPS, wall_bottom=WALL, wall_top=WALL, ux0_p=-0.1249999, **kw),
    ]


@pytest.mark.parametrize("cm", [False, True], ids=["bgk", "cm"])
def test_fast_flow_equals_oracle(cm):
    ps = cases(cm)
    want = []
    for p in ps:
        o = Oracle(p, [])
        o.step(STEPS)
        want.append(o.fields())
    assert max(float(np.abs(w["u"]).max()) for w in want) > 0.2
    for p, w in zip(ps, want):
        with Case(p, []) as c:
            c.step(STEPS)
            got = c.fields()
        for k in ("f", "rho", "u"):
            assert np.array_equal(got[k], w[k]), (p.Nx, p.Ny, k)
    with Batch([(p, []) for p in ps]) as b:
        b.step(STEPS)
        for q, w in enumerate(want):
            got = b.case(q).fields()
            for k in ("f", "rho", "u"):
                assert np.array_equal(got[k], w[k]), (q, k)
