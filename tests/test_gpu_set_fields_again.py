"""A state loaded (``set_fields``) into a case that has already stepped: the steps
after it equal those of a fresh case given the same state, bit for bit, whatever
the case did before. The runs before it are of odd length and long enough that
step graphs exist, so the list of support sites that the next step fills is not
the one that its graph was captured with unless the loading sets it right; the
state is loaded many times over with a single step after each, so a list that is
not emptied would keep growing; and the body is moved before a load, so a force
left on sites that it no longer reaches would show."""
import numpy as np
import pytest

from cases import lattice_case
from life_gb300.case import CONVECTIVE, VELOCITY, WALL, Circle
from life_gb300.lib import Batch, Case

pytestmark = pytest.mark.gpu

ALL = ("rho", "u", "f", "force_ibm")


def problem(prec=0, cm=False, x=30.0):
    p = lattice_case(96, 48, 1.0 / 0.6, 100, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=WALL, wall_top=WALL,
                     uxInlet_p=0.05, precision=prec, central_moments=cm)
    return p, [Circle(x, 24.2, 6.0)]


def start_state(p, bodies):
    with Case(p, bodies) as c:
        c.step(40)
        return c.fields(ALL)


def load(c, st):
    c.set_fields(0, st["rho"], st["u"], st["f"], st["force_ibm"])


def result(c):
    fl = c.fields(ALL)
    fl["force"] = c.markers()["force"]
    return fl


def fresh(p, bodies, st, steps, shift=0.0):
    with Case(p, bodies) as c:
        if shift:
            move(c, shift)
        load(c, st)
        c.step(steps)
        return result(c)


def move(c, shift):
    m = c.markers()
    m["pos"][:, 0] += shift
    c.set_markers(m["pos"], m["vel"], m["force"])


def same(got, want):
    for k in want:
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("prec,cm", [(0, False), (0, True), (1, False), (2, True)])
@pytest.mark.parametrize("before", [0, 1, 2, 101, 102])
def test_loaded_state_steps_like_a_fresh_case(before, prec, cm):
    p, bodies = problem(prec, cm)
    st = start_state(p, bodies)
    one, many = fresh(p, bodies, st, 1), fresh(p, bodies, st, 70)
    with Case(p, bodies) as c:
        if before:
            c.step(before)
        for _ in range(12):
            load(c, st)
            c.step(1)
        same(result(c), one)
        load(c, st)
        c.step(70)
        same(result(c), many)
        c.step(1)  # (an odd run, with graphs)
        load(c, st)
        c.step(70)
        same(result(c), many)


@pytest.mark.parametrize("before", [1, 101, 102])
def test_no_force_stays_where_the_body_was(before):
    p, bodies = problem()
    st = start_state(p, bodies)
    want = fresh(p, bodies, st, 3, shift=20.0)
    with Case(p, bodies) as c:
        c.step(before)
        move(c, 20.0)
        load(c, st)
        c.step(3)
        same(result(c), want)


def test_cases_of_a_batch():
    ps = [problem(0, False), problem(0, True, 50.0)]
    st = [start_state(*q) for q in ps]
    want = [fresh(*q, s, 5) for q, s in zip(ps, st)]
    with Batch(ps) as b:
        b.step(7)
        for _ in range(6):
            for k in range(2):
                load(b.case(k), st[k])
            b.step(5)
        for k in range(2):
            same(result(b.case(k)), want[k])
