"""Narrow-band epsilon systems (lines of markers): the band elimination with its
window in registers (bands of up to five), its interchanges, the pipelined one
for wider bands and both orders of the backward solve, against the textbook
dense LU in numpy FP64 (``test_gpu_epsilon_sparse``), bit for bit. The spacing
sets the band (3 / spacing), the jitter makes the systems so ill-conditioned
that rows are interchanged; sizes start at one marker and cross the window, the
forward solve's batches and the backward solve's chunks."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_epsilon_sparse import _dense, _system

pytestmark = pytest.mark.gpu

SPACINGS = {0.8: 3, 0.55: 5, 0.45: 6, 0.36: 8, 0.22: 13}


def _line(n, spacing, jitter, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = 6.0 + spacing * np.arange(n) + jitter * spacing * rng.uniform(-0.45, 0.45, n)
    y = 9.3 + jitter * rng.uniform(-0.4, 0.4, n)
    return [(float(a), float(b)) for a, b in zip(x, y)]


@pytest.mark.parametrize("jitter", [0.0, 1.0])
@pytest.mark.parametrize("spacing", sorted(SPACINGS))
def test_band_elimination_is_the_dense_lu(spacing, jitter):
    import torch
    from life_gb300.build import build
    build()
    from life_gb300.lib import lib
    swaps = 0
    for n in (1, 2, 5, 6, 7, 12, 31, 33, 80, 121):
        pos, nsupp, si, sj, sd, ds, A = _system(_line(n, spacing, jitter, 100 + n))
        want, s = _dense(A)
        swaps += s
        dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (pos, nsupp, si, sj, sd, ds)]
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        rc = lib().life_ibm_epsilon(*[C.c_void_p(a.data_ptr()) for a in dev], n, 1.0, C.c_void_p(out.data_ptr()), None)
        assert rc == 0, lib().life_last_error()
        assert np.array_equal(out.cpu().numpy(), want), n
    if jitter and spacing <= 0.55:
        assert swaps > 20
