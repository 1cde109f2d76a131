"""The SOR solver of the viscous systems (csrc/mg_relax.cuh) at the edges of
its strips (44 columns), chunks and iterations (4 rows), on even and odd row
lengths, and on either side of the rule that selects it."""
import numpy as np
import pytest

from oracle import vdi_oracle as vo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def V():
    import vdropimpact_b200 as V
    return V


def _system(V, m, n, x_sym, horiz, vf):
    import torch
    s = V.ViscoImpl(m, n, x_sym, horiz, vf, 1.1 * vf)
    b = np.random.default_rng(m * 100 + n).standard_normal(m * n)
    s.b.copy_(torch.from_numpy(b))
    return s, b, vo.visco_matrix(m, n, vf, 1.1 * vf, x_sym, horiz)


SIZES = [(3, 8), (4, 4), (8, 3), (43, 7), (44, 8), (45, 9), (54, 21), (88, 24), (89, 25), (133, 60), (640, 70)]


@pytest.mark.parametrize("x_sym,horiz", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("m,n", SIZES)
def test_sor_solve(V, m, n, x_sym, horiz):
    """The operator's inverse is bounded by 1 in the maximum norm and its
    condition number by 1 + 4 (vfx + vfy) < 5, so a solve to 1e-10 of ||b||_2
    lies within 5e-10 of the exact one in the 2-norm."""
    s, b, A = _system(V, m, n, x_sym, horiz, 0.4)
    v, rel = s.solve_v_cycle(rtol=1e-10)
    z = s.z.cpu().numpy()
    assert rel <= 1e-10 and 1 <= v <= 6
    assert np.linalg.norm(b - A @ z) <= 1e-10 * (1 + 1e-6) * np.linalg.norm(b)
    zx = vo.DirectSolver(A).solve(b)
    assert np.linalg.norm(z - zx) <= 5e-10 * np.linalg.norm(zx)


@pytest.mark.parametrize("vf", [0.0, 0.01, 0.4, 2.0, 3.5, 4.2, 40.0])
def test_sor_and_vcycles_meet_the_tolerance(V, vf):
    """Weak couplings (one pass, whose result is copied back), strong ones,
    and past the rule's line (V-cycles); repeated solves replay the same."""
    import torch
    s, b, A = _system(V, 130, 67, True, True, vf)
    out = []
    for _ in range(3):
        s.z.zero_()
        out.append((s.solve_v_cycle(rtol=1e-10), s.z.clone()))
    z = out[0][1].cpu().numpy()
    assert np.linalg.norm(b - A @ z) <= 1e-10 * (1 + 1e-6) * np.linalg.norm(b)
    for r, zz in out[1:]:
        assert r == out[0][0] and torch.equal(zz, out[0][1])


def test_sor_ends_at_once(V):
    """A zero source gives a zero solution, a converged start is left as it
    is, and a cap ends the solve with its error."""
    import torch
    s, b, A = _system(V, 100, 50, True, False, 0.4)
    s.solve_v_cycle(rtol=1e-12)
    z = s.z.clone()
    assert s.solve_v_cycle(rtol=1e-10)[0] == 0 and torch.equal(s.z, z)
    s.z.zero_()
    with pytest.raises(V.VdiError) as e:
        s.solve_v_cycle(rtol=1e-12, max_vcycles=1)
    assert e.value.status == 5
    s.b.zero_()
    s.z.fill_(3.0)
    assert s.solve_v_cycle() == (0, 0.0) and float(s.z.abs().max()) == 0.0
    s.b[7] = float("nan")
    with pytest.raises(V.VdiError) as e:
        s.solve_v_cycle()
    assert e.value.status == 8
