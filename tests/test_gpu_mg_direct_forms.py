"""The exact solve (csrc/mg_direct.cuh) and the SOR passes (csrc/
mg_relax.cuh) over the forms they accept: every size of chunk, block and
transform, stretched cells, arrays off 16-byte alignment, a start so far off
that V-cycles have to follow, and couplings on either side of the rule that
selects SOR.

A solve that the exact solve ends reports exactly the V-cycles it stands for
(one per 1.25 decades, FEM 2.5); V-cycles behind it would add to that."""
import ctypes as C
import math

import numpy as np
import pytest

from oracle import vdi_oracle as vo

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def V():
    import vdropimpact_b200 as V
    return V


def _system(V, kind, m, n, dx, dy):
    return {"mac": V.MgsMac, "fem": V.MgsFem, "neumann": V.MgsMacNeumann}[kind](m, n, dx, dy)


def _matrix(kind, m, n, dx, dy):
    if kind == "fem":
        return vo.fem_matrix(m, n, dx, dy)
    return vo.mac_matrix(m, n, 1 / dx ** 2, 1 / dy ** 2, neumann_bottom=kind == "neumann")


def _count(kind, r0=1.0, rtol=1e-10):
    return math.ceil(math.log10(r0 / rtol) / (2.5 if kind == "fem" else 1.25))


# chunks of 8 rows in blocks of 8 modes (to 512 rows) and 4 (to 1024), of 16
# (to 2048) and 32 rows; transforms of 8192 points in powers of two and in the
# chirp form
@pytest.mark.parametrize("kind,m,n", [
    ("mac", 64, 512), ("mac", 64, 513), ("mac", 1024, 1024), ("mac", 64, 1025), ("fem", 257, 1026), ("mac", 64, 1500),
    ("fem", 33, 2049), ("mac", 32, 2049), ("mac", 32, 2100), ("fem", 4097, 65), ("fem", 1501, 30), ("mac", 2049, 64),
    ("neumann", 2000, 40), ("mac", 8192, 16)])
def test_large_sizes_end_with_the_exact_solve(V, kind, m, n):
    """White noise from zero: what rounding leaves, eps times |A| |z| (1e3 to
    1e4 |b| here), is far below the tolerance, so the exact solve alone ends
    it. The residual is checked against the oracle's matrix."""
    import torch
    dx, dy = 1.0 / m, 1.2 / m
    b = np.random.default_rng(m + n).standard_normal(m * n)
    if kind == "neumann":
        b -= b.mean()
    s = _system(V, kind, m, n, dx, dy)
    s.b.copy_(torch.from_numpy(b))
    s.z.zero_()
    v, rel = s.solve_v_cycle(rtol=1e-10)
    assert rel <= 1e-10 and v == _count(kind)
    r = b - _matrix(kind, m, n, dx, dy) @ s.z.cpu().numpy()
    assert np.linalg.norm(r) <= 1e-10 * (1 + 1e-6) * np.linalg.norm(b)


# below and above the sqrt(2) at which the FEM operator's couplings to the
# upper and lower (dx over dy) and side neighbours (dy over dx) change sign
@pytest.mark.parametrize("aspect", [0.05, 0.5, 0.7, 1.5, 2.0, 20.0])
@pytest.mark.parametrize("m,n", [(64, 33), (97, 40), (130, 24)])
@pytest.mark.parametrize("kind", ["mac", "fem", "neumann"])
def test_stretched_cells(V, kind, m, n, aspect):
    """Against a sparse LU solve, to 100 eps times the condition number: the
    largest eigenvalue is at most 4 (1/dx^2 + 1/dy^2), the smallest about
    pi^2 over the square of the longer side, twice the height where the bottom
    is fixed (the FEM's mass factors between 1/3 and 1 only lower the ratio of
    the two parts; a factor of 3 covers them)."""
    import torch
    if kind == "fem":
        m, n = m + 1, n + 1
    dx, dy = 1.0 / m, aspect / m
    b = np.random.default_rng(m * 100 + n).standard_normal(m * n)
    if kind == "neumann":
        b -= b.mean()
    s = _system(V, kind, m, n, dx, dy)
    s.b.copy_(torch.from_numpy(b))
    s.z.zero_()
    v, rel = s.solve_v_cycle(rtol=1e-10)
    assert rel <= 1e-10 and v == _count(kind)
    A = _matrix(kind, m, n, dx, dy)
    if kind == "neumann":
        import scipy.sparse as sp
        one = sp.csr_matrix(np.ones((m * n, 1)))
        zx = vo.DirectSolver(sp.bmat([[sp.csr_matrix(A), one], [one.T, None]]).tocsc()).solve(np.append(b, 0.))[:-1]
    else:
        zx = vo.DirectSolver(A).solve(b)
    cond = 3 * 4 * (1 / dx ** 2 + 1 / dy ** 2) * max(m * dx, 2 * n * dy) ** 2 / math.pi ** 2
    assert np.max(np.abs(s.z.cpu().numpy() - zx)) <= 100 * EPS * cond * np.max(np.abs(zx))


@pytest.mark.parametrize("kind,m,n,c", [("MAC", 128, 66, 1 / 128), ("FEM", 129, 66, 1 / 128), ("VISC_U", 132, 50, 0.4),
                                        ("VISC_V", 132, 50, 0.02)])
def test_arrays_off_16_byte_alignment(kind, m, n, c):
    """The same bits, host-driven and replayed, as with aligned arrays: only
    the width of the accesses differs. (0.02: one pass, copied back.)"""
    import torch
    from vdropimpact_b200 import _abi
    L = _abi.lib()
    src = torch.from_numpy(np.random.default_rng(m).standard_normal(m * n)).cuda()
    out = {}
    for off_b, off_z in ((0, 0), (1, 0), (0, 1), (1, 1)):
        h = C.c_void_p()
        _abi.check(L.vdi_mg_create(getattr(_abi, "VDI_MG_" + kind), m, n, c, c, 1, None, C.byref(h)), "vdi_mg_create")
        b = torch.empty(m * n + 1, dtype=torch.float64, device="cuda")[off_b:off_b + m * n]
        z = torch.empty(m * n + 1, dtype=torch.float64, device="cuda")[off_z:off_z + m * n]
        assert b.data_ptr() % 16 == 8 * off_b and z.data_ptr() % 16 == 8 * off_z
        b.copy_(src)
        for call in range(2):
            z.zero_()
            r = _abi.VdiMgResult()
            torch.cuda.synchronize()
            _abi.check(L.vdi_mg_solve(h, C.c_void_p(b.data_ptr()), C.c_void_p(z.data_ptr()), 1e-10, 200, 0,
                                      C.byref(r)), "vdi_mg_solve")
            out[off_b, off_z, call] = (r.vcycles, r.rel_res, z.clone())
        L.vdi_mg_destroy(h)
    v, rel, z = out[0, 0, 0]
    assert rel <= 1e-10 and (kind[:4] == "VISC" or v == _count(kind.lower()))
    for w in out.values():
        assert w[:2] == (v, rel) and torch.equal(w[2], z)


@pytest.mark.parametrize("kind", ["mac", "fem", "neumann"])
@pytest.mark.parametrize("m,n", [(128, 64), (100, 50)])
def test_vcycles_after_the_exact_solve(V, kind, m, n):
    """From 1e8 times noise the exact solve leaves eps |A z0|, 1e-8 of |b| and
    more, which a sweep (MAC, Neumann) does not bring to 1e-10: V-cycles follow,
    in the captured loop as host-driven."""
    import torch
    if kind == "fem":
        m, n = m + 1, n + 1
    rng = np.random.default_rng(m)
    b, z0 = rng.standard_normal(m * n), 1e8 * rng.standard_normal(m * n)
    if kind == "neumann":
        b -= b.mean()
        z0 -= z0.mean()     # V-cycles keep the mean, whose rounding would stay
    A = _matrix(kind, m, n, 1. / m, 1. / m)
    s = _system(V, kind, m, n, 1. / m, 1. / m)
    s.b.copy_(torch.from_numpy(b))
    out = []
    for _ in range(3):
        s.z.copy_(torch.from_numpy(z0))
        out.append((s.solve_v_cycle(rtol=1e-10), s.z.clone()))
    (v, rel), z = out[0]
    r0 = np.linalg.norm(b - A @ z0) / np.linalg.norm(b)
    assert rel <= 1e-10 and v > _count(kind, r0)
    assert np.linalg.norm(b - A @ z.cpu().numpy()) <= 1e-10 * (1 + 1e-3) * np.linalg.norm(b)
    for r, zz in out[1:]:
        assert r == (v, rel) and torch.equal(zz, z)


@pytest.mark.parametrize("vf,sor", [(7.5, True), (7.7, False)])
def test_couplings_beside_the_line_of_the_relaxation(V, monkeypatch, vf, sor):
    """omega - 1 is 0.5975 at vfx = vfy = 7.5 and 0.6015 at 7.7, the line 0.6:
    with VDI_MG_SOR=0 the bits differ below it and are the same above."""
    import torch
    m, n = 128, 64
    b = np.random.default_rng(3).standard_normal(m * n)
    out = []
    for _ in range(2):
        s = V.ViscoImpl(m, n, True, True, vf, vf)
        s.b.copy_(torch.from_numpy(b))
        s.z.zero_()
        out.append((s.solve_v_cycle(rtol=1e-10), s.z.clone()))
        monkeypatch.setenv("VDI_MG_SOR", "0")
    assert torch.equal(out[0][1], out[1][1]) != sor
    A = vo.visco_matrix(m, n, vf, vf, True, True)
    for (v, rel), z in out:
        assert rel <= 1e-10 and np.linalg.norm(b - A @ z.cpu().numpy()) <= 1e-10 * (1 + 1e-6) * np.linalg.norm(b)
