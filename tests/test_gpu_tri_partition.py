"""The partitioned tridiagonal solve (partition_solve in csrc/gas.cu) at the
edges of its rows a thread, its warps and the block sizes, against dgtsv."""
import numpy as np
import pytest

from oracle import vdi_oracle as vo

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def V():
    import vdropimpact_b200 as V
    return V


SIZES = [2, 3, 4, 5, 63, 64, 65, 127, 255, 256, 257, 511, 512, 513, 1023, 1025, 2047, 2048, 2049, 2050, 4094, 4095]


@pytest.mark.parametrize("margin", [0.0, 1e-3, 10.0])
@pytest.mark.parametrize("n", SIZES)
def test_dominant_systems(V, n, margin):
    """Rows dominant by a margin (0: just dominant, an M-matrix whose
    solutions grow as n^2). Elimination without pivoting of such a system is
    backward stable row by row, so x differs by at most a small multiple of
    eps times |A^-1| |A| |x|; for an M-matrix that is A^-1 |A| |x|, evaluated
    here. The reduction's log2(n) steps are allowed 4 roundings each."""
    rng = np.random.default_rng(n)
    a, c = -rng.uniform(0.5, 1, n), -rng.uniform(0.5, 1, n)
    a[0] = c[-1] = 0.0
    b = np.abs(a) + np.abs(c) + margin
    b[0] += 0.5      # nonsingular at margin 0
    d = rng.standard_normal(n)
    t = V.TriSolve(n)
    t.a[:], t.b[:], t.c[:], t.d[:] = a, b, c, d
    x = t.solve_lapack()
    assert not t.pivoted
    xr, info = vo.dgtsv(a[1:], b, c[:-1], d)
    assert info == 0
    ax = np.abs(b) * np.abs(xr)
    ax[1:] += np.abs(a[1:]) * np.abs(xr[:-1])
    ax[:-1] += np.abs(c[:-1]) * np.abs(xr[1:])
    bound, _ = vo.dgtsv(a[1:], b, c[:-1], ax)
    assert np.all(np.abs(x - xr) <= EPS * (8 + 4 * np.log2(n)) * (bound + np.abs(xr)))
