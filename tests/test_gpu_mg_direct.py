"""The exact solve of a separable finest level (csrc/mg_direct.cuh) where it
can go wrong: row lengths that are powers of two and others (chirp form),
the edges of the FFT's first radix, of the chunks of a column and of the
kernels' variants, and the smallest and largest grids it takes."""
import numpy as np
import pytest

from oracle import vdi_oracle as vo

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def V():
    import vdropimpact_b200 as V
    return V


def _solve(V, kind, m, n, dx, dy, b, prec="fp64", z0=None):
    import torch
    s = {"mac": V.MgsMac, "fem": V.MgsFem, "neumann": V.MgsMacNeumann}[kind](m, n, dx, dy)
    s.b.copy_(torch.from_numpy(b))
    if z0 is not None:
        s.z.copy_(torch.from_numpy(z0))
    v, rel = s.solve_v_cycle(rtol=1e-10, precision=prec)
    return s, v, rel


# rows of 2 to 8 points short of and past a chunk (8 and 16 rows), columns of
# 8 to 512 points: radix 2, 4 and 8 first passes, chirp lengths odd and even
SMALL = [(8, 2), (9, 8), (16, 9), (17, 16), (32, 17), (33, 7), (64, 31), (63, 64), (96, 65), (128, 33), (130, 24),
         (251, 40), (256, 130), (512, 20), (600, 37)]


@pytest.mark.parametrize("kind", ["mac", "fem", "neumann"])
@pytest.mark.parametrize("m,n", SMALL)
def test_exact_solve_small(V, kind, m, n):
    """Against a sparse LU solve. Rounding bounds the difference by about
    eps times the condition number of the operator, below 10 (m^2 + n^2) with
    the cells' aspect ratio, from a starting iterate that is not zero."""
    if kind == "fem":
        m, n = m + 1, n + 1
    rng = np.random.default_rng(m * 1000 + n)
    dx, dy = 1.0 / m, 1.3 / m
    b = rng.standard_normal((n, m))
    if kind == "mac":
        A = vo.mac_matrix(m, n, 1 / dx ** 2, 1 / dy ** 2)
    elif kind == "fem":
        A = vo.fem_matrix(m, n, dx, dy)
    else:
        A = vo.mac_matrix(m, n, 1 / dx ** 2, 1 / dy ** 2, neumann_bottom=True)
        b += 0.4
    b = b.ravel()
    z0 = rng.standard_normal(m * n)
    s, v, rel = _solve(V, kind, m, n, dx, dy, b, z0=z0)
    # the exact solve ends it, counted as a V-cycle per 1.25 decades (FEM 2.5)
    # that the residual had to fall; one V-cycle more may follow where the
    # rounding of this far-off start, eps |A z0|, exceeds the tolerance
    bp = b - b.mean() if kind == "neumann" else b
    r0 = np.linalg.norm(bp - A @ z0) / np.linalg.norm(bp)
    count = int(np.ceil(np.log10(r0 / 1e-10) / (2.5 if kind == "fem" else 1.25)))
    assert rel <= 1e-10 and count <= v <= count + (10 * EPS * r0 > 1e-10)
    z = s.z.cpu().numpy()
    if kind == "neumann":
        import scipy.sparse as sp
        one = sp.csr_matrix(np.ones((m * n, 1)))
        K = sp.bmat([[sp.csr_matrix(A), one], [one.T, None]]).tocsc()
        zx = vo.DirectSolver(K).solve(np.concatenate([b - b.mean(), [0.]]))[:-1]
    else:
        zx = vo.DirectSolver(A).solve(b)
    err = np.max(np.abs(z - zx)) / np.max(np.abs(zx))
    # the exact solve alone meets it; 1e-10 of residual from V-cycles would
    # not on the larger of these grids
    assert err <= EPS * 100 * (m * m + n * n), err


# a power-of-two row with chunks of 16 rows; the 4-mode block (more than 1024
# rows); a 1024-thread transform (8192 points, chirp form); chunks of 32 rows;
# one row too long for the exact solve (V-cycles alone)
LARGE = [("mac", 1024, 1024), ("mac", 64, 1500), ("fem", 257, 1026), ("fem", 1501, 30), ("mac", 2049, 64),
         ("fem", 4097, 65), ("mac", 32, 2100), ("mac", 4100, 32)]


@pytest.mark.parametrize("kind,m,n", LARGE)
def test_exact_solve_large(V, kind, m, n):
    """The residual of the returned iterate, evaluated by the library's own
    residual entry point, and its agreement with the V-cycles alone."""
    rng = np.random.default_rng(m + n)
    b = rng.standard_normal(m * n)
    s, v, rel = _solve(V, kind, m, n, 1.0 / m, 1.2 / m, b)
    _, nr = s.residual()
    assert rel <= 1e-10
    assert nr <= 1e-10 * np.linalg.norm(b) * (1 + 1e-6)


@pytest.mark.parametrize("prec", ["fp64", "mixed", "hybrid"])
@pytest.mark.parametrize("kind,m,n", [("mac", 200, 100), ("mac", 256, 128), ("fem", 201, 101), ("fem", 257, 129)])
def test_exact_solve_matches_vcycles(V, kind, m, n, prec, monkeypatch):
    """The same solve with the exact solve turned off: both to the 1e-10
    residual, and no more cycles counted with it."""
    b = np.random.default_rng(7).standard_normal(m * n)
    res = []
    for on in (True, False):
        if not on:
            monkeypatch.setenv("VDI_MG_DIRECT", "0")
        s, v, rel = _solve(V, kind, m, n, 1.0 / m, 1.0 / m, b, prec)
        monkeypatch.delenv("VDI_MG_DIRECT", raising=False)
        assert rel <= 1e-10
        res.append((v, s.z.cpu().numpy()))
    (va, za), (vb, zb) = res
    assert va <= vb
    assert np.max(np.abs(za - zb)) <= 1e-7 * np.max(np.abs(zb))


def test_cap_below_the_equivalent_runs_vcycles(V):
    """A cap below the V-cycles an exact solve stands for is kept: the solve
    stops at it, as it does without the exact solve."""
    m, n = 256, 128
    b = V.projection_source(m, n, 3)
    with pytest.raises(V.VdiError) as e:
        s = V.MgsMac(m, n, 1. / m, 1. / m)
        import torch
        s.b.copy_(torch.from_numpy(b))
        s.solve_v_cycle(rtol=1e-10, max_vcycles=3)
    assert e.value.status == 5 and "3 V-cycles" in str(e.value)


def test_sweep_after_the_exact_solve(V):
    """A smooth source on a fine grid, whose exact solution rounded to FP64
    lies near the tolerance: whichever of the exact solve, the sweep and the
    V-cycles ends it, host-driven and replayed solves are the same."""
    import torch
    m, n = 1300, 1100
    b = torch.from_numpy(V.projection_source(m, n, 3)).cuda()
    s = V.MgsMac(m, n, 1. / m, 1. / m)
    s.b.copy_(b)
    out = []
    for _ in range(3):
        s.z.zero_()
        out.append((s.solve_v_cycle(rtol=1e-10), s.z.clone()))
    assert out[0][0][1] <= 1e-10
    for r, z in out[1:]:
        assert r == out[0][0] and torch.equal(z, out[0][1])
