"""The epsilon solve of marker sets whose system is sparse but not a narrow
band (closed rings, bodies that touch, scattered markers): the device's sparse
elimination against the textbook dense LU with partial pivoting and transposed
solve in numpy FP64, element by element in the same order, bit for bit. Ring
sizes lie on both sides of the shared-memory capacity (one mask word to nine);
the scattered sets need row interchanges (asserted)."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _delta(r):
    a = abs(r)
    if a > 1.5:
        return 0.0
    if a > 0.5:
        return (5.0 - 3.0 * a - math.sqrt(-3.0 * ((1.0 - a) * (1.0 - a)) + 1.0)) / 6.0
    return (1.0 + math.sqrt(1.0 - 3.0 * (a * a))) / 3.0


def _ring(n, x, y):
    r = n / (2.0 * math.pi)
    return [(x + r * math.cos(2.0 * math.pi * k / n), y + r * math.sin(2.0 * math.pi * k / n)) for k in range(n)]


def _scatter(n, box, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    while len(out) < n:
        x, y = rng.uniform(4.0, 4.0 + box, 2)
        if all(math.hypot(x - a, y - b) > 0.6 for a, b in out):
            out.append((float(x), float(y)))
    return out


def _markers(kind):
    name, n = kind
    if name == "ring":
        return _ring(n, n / 5.0 + 6.3, n / 5.0 + 6.1)
    if name == "tail":  # a ring and the two sides of a tail behind it
        ring = _ring(n, 20.3, 20.4)
        x0 = max(x for x, _ in ring) + 0.7
        return ring + [(x0 + 0.9 * k, 18.55) for k in range(n // 2)] + [(x0 + 0.9 * k, 22.2) for k in range(n // 2)]
    return _scatter(n, 1.15 * math.sqrt(n), 11 + n)


def _system(pts):
    n = len(pts)
    nsupp, si, sj, sd = np.zeros(n, np.int32), np.zeros((n, 9), np.int32), np.zeros((n, 9), np.int32), np.zeros((n, 9))
    for k, (x, y) in enumerate(pts):
        q = 0
        ix, iy = math.floor(x + 0.5), math.floor(y + 0.5)
        for i in range(ix - 2, ix + 3):
            for j in range(iy - 2, iy + 3):
                if abs(x - i) < 1.5 and abs(y - j) < 1.5 and q < 9:
                    si[k, q], sj[k, q], sd[k, q] = i, j, _delta(x - i) * _delta(y - j)
                    q += 1
        nsupp[k] = q
    pos = np.array(pts)
    dd = (pos[:, None, 0] - pos[None, :, 0]) ** 2 + (pos[:, None, 1] - pos[None, :, 1]) ** 2
    np.fill_diagonal(dd, np.inf)
    ds = np.minimum(np.sqrt(dd.min(axis=1)), 10.0)
    A = np.zeros((n, n))
    for i in range(n):
        for j in range(n):
            if abs(pos[i, 0] - pos[j, 0]) < 3.0 and abs(pos[i, 1] - pos[j, 1]) < 3.0:
                acc = 0.0
                for s in range(nsupp[i]):
                    acc += float(sd[i, s]) * (_delta(pts[j][0] - int(si[i, s])) * _delta(pts[j][1] - int(sj[i, s])))
                A[i, j] = acc * float(ds[j])
    return pos, nsupp, si, sj, sd, ds, A


def _dense(A):
    """Textbook LU of M = A^T and the transposed solve of a vector of ones."""
    M, n = A.T.copy(), len(A)
    piv, swaps = list(range(n)), 0
    for j in range(n):
        jp = j + int(np.argmax(np.abs(M[j:, j])))
        piv[j] = jp
        if jp != j:
            M[[j, jp]] = M[[jp, j]]
            swaps += 1
        M[j + 1:, j] *= 1.0 / M[j, j]
        M[j + 1:, j + 1:] += M[j + 1:, j:j + 1] * -M[j:j + 1, j + 1:]
    y = np.ones(n)
    for k in range(n):
        y[k] = y[k] / M[k, k]
        y[k + 1:] -= M[k, k + 1:] * y[k]
    for i in range(n - 1, -1, -1):
        t = y[i]
        for k in range(i + 1, n):
            t = t - M[k, i] * y[k]
        y[i] = t
    for i in range(n - 1, -1, -1):
        y[i], y[piv[i]] = y[piv[i]], y[i]
    return y, swaps


@pytest.mark.parametrize("kind", [("ring", 31), ("ring", 33), ("ring", 96), ("ring", 140), ("ring", 165), ("ring", 270),
                                  ("tail", 40), ("tail", 64), ("scatter", 60), ("scatter", 130)], ids=str)
def test_sparse_elimination_is_the_dense_lu(kind):
    import torch
    from life_gb300.build import build
    build()
    from life_gb300.lib import lib
    pos, nsupp, si, sj, sd, ds, A = _system(_markers(kind))
    want, swaps = _dense(A)
    assert np.all(np.isfinite(want))
    if kind[0] == "scatter":
        assert swaps > 0
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (pos, nsupp, si, sj, sd, ds)]
    out = torch.zeros(len(ds), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rc = lib().life_ibm_epsilon(*[C.c_void_p(a.data_ptr()) for a in dev], len(ds), 1.0, C.c_void_p(out.data_ptr()), None)
    assert rc == 0, lib().life_last_error()
    assert np.array_equal(out.cpu().numpy(), want)
