"""Fields read into page-locked host arrays (written by the export kernel
itself) equal the fields read into ordinary ones (staged on the device): every
storage form and collision, lattices whose sizes are not multiples of the
export tile, periodic and boundary-condition walls, bodies near a wall, and
arrays that start at an odd offset (which take the staged way)."""
import numpy as np
import pytest

from cases import golden_cases, lattice_case
from life_gb300.case import CONVECTIVE, FREESLIP, VELOCITY, WALL
from life_gb300.lib import Case

pytestmark = pytest.mark.gpu

NAMES = ["cavity_bgk", "channel_convective_freeslip_cm", "periodic_womersley", "womersley_gravity_cm",
         "pressure_top_corners", "cylinder_rigid_cm", "honami_like_cm"]


def pinned(shape):
    import torch
    return torch.full(shape, np.nan, dtype=torch.float64, pin_memory=True).numpy()


def check(p, bodies, steps, shift=0):
    n = p.Nx * p.Ny
    with Case(p, bodies) as c:
        c.step(steps)
        want = c.fields(("rho", "u", "force_ibm"))
        got = {"rho": pinned((n + shift,))[shift:], "force_ibm": pinned((n, 2)),
               "u": pinned((2 * n + shift,))[shift:].reshape(n, 2)}
        c.fields(("rho", "u", "force_ibm"), out=got)
        for k in want:
            assert np.array_equal(got[k], want[k]), k
        only = pinned((n, 2))
        c.fields(("u",), out={"u": only})
        assert np.array_equal(only, want["u"])


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("name", NAMES)
def test_pinned_fields_equal_staged_fields(name, precision):
    p, bodies = golden_cases()[name]
    check(p.replace(precision=precision), bodies, 21)


@pytest.mark.parametrize("nx,ny", [(4, 4), (31, 33), (32, 32), (65, 7), (1029, 1023)])
def test_pinned_fields_at_tile_edges(nx, ny):
    p = lattice_case(nx, ny, 1.0 / 0.6, 5, wall_left=VELOCITY, wall_right=CONVECTIVE, wall_bottom=WALL,
                     wall_top=FREESLIP, uxInlet_p=0.04, ux0_p=0.03)
    check(p, [], 5)


def test_arrays_at_an_odd_offset():
    p, bodies = golden_cases()["cylinder_rigid_cm"]
    check(p, bodies, 5, shift=1)
