"""A state loaded at another time step than the case has reached: the inlet ramp and
the oscillating pressure gradient are those of the new time, also when the case has
step graphs and a table of later (or much later) steps' values. Bit for bit against a
fresh case."""
import numpy as np
import pytest

from cases import lattice_case
from life_gb300.case import CONVECTIVE, VELOCITY, WALL
from life_gb300.lib import Batch, Case

pytestmark = pytest.mark.gpu


def problems():
    ramp = lattice_case(48, 24, 1.0 / 0.6, 100, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=WALL,
                        wall_top=WALL, uxInlet_p=0.05, inlet_ramp=200.0)
    wom = lattice_case(48, 24, 1.0 / 0.6, 100, wall_bottom=WALL, wall_top=WALL, womersley=3.0, dpdx=1e-5)
    return [ramp, wom]


def load(c, t, st):
    c.set_fields(t, st["rho"], st["u"], st["f"], st["force_ibm"])


def fresh(p, t, st, steps):
    with Case(p, []) as c:
        load(c, t, st)
        c.step(steps)
        return c.fields()


@pytest.mark.parametrize("first", [0, 4096, 100000])
@pytest.mark.parametrize("which", [0, 1])
def test_back_in_time(which, first):
    p = problems()[which]
    with Case(p, []) as c:
        c.step(20)
        st = c.fields()
        load(c, first, st)
        c.step(80)  # (step graphs, and a table from `first` on)
        for t, steps in ((0, 3), (0, 90), (37, 70), (100, 5), (first, 66), (0, 70)):
            load(c, t, st)
            c.step(steps)
            want = fresh(p, t, st, steps)
            got = c.fields()
            for k in ("rho", "u", "f"):
                assert np.array_equal(got[k], want[k]), (t, steps, k)


def test_cases_of_a_batch():
    ps = problems()
    with Batch([(p, []) for p in ps]) as b:
        b.step(10)
        st = [b.case(k).fields() for k in range(2)]
        b.step(5000)
        for k in range(2):
            load(b.case(k), 0, st[k])
        b.step(40)
        for k in range(2):
            want, got = fresh(ps[k], 0, st[k], 40), b.case(k).fields()
            for key in ("rho", "u", "f"):
                assert np.array_equal(got[key], want[key]), (k, key)
