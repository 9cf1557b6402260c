"""Fields read into host arrays that the caller registered itself (page-locked from
end to end, with sizes that are no multiple of a page and starts inside one) equal
the fields read into ordinary arrays."""
import numpy as np
import pytest

from cases import golden_cases
from life_gb300.lib import Case

pytestmark = pytest.mark.gpu


def test_registered_arrays():
    import torch
    torch.zeros(1, device="cuda")
    rt = torch.cuda.cudart()
    p, bodies = golden_cases()["cylinder_rigid_cm"]
    n = p.Nx * p.Ny
    with Case(p, bodies) as c:
        c.step(21)
        want = c.fields(("rho", "u", "force_ibm"))
        big = {"rho": np.full(n, np.nan), "u": np.full((n, 2), np.nan), "force_ibm": np.full((n, 2), np.nan)}
        for a in big.values():
            assert int(rt.cudaHostRegister(a.ctypes.data, a.nbytes, 0)) == 0
        try:
            c.fields(("rho", "u", "force_ibm"), out=big)
        finally:
            for a in big.values():
                assert int(rt.cudaHostUnregister(a.ctypes.data)) == 0
        for k in want:
            assert np.array_equal(big[k], want[k]), k
