"""Viscous systems whose rows are too long for the SOR passes' partial sums
(csrc/mg_relax.cuh) keep their V-cycles."""
import numpy as np
import pytest

from oracle import vdi_oracle as vo

pytestmark = pytest.mark.gpu


# 10909 and 10932 strips of 44 columns: 2728 blocks, within the third of 8192
# partial sums that a pass may use, and 2734, past it
@pytest.mark.parametrize("m", [479996, 481000])
def test_long_rows(m):
    """The condition number 1 + 4 (vfx + vfy) < 5 bounds the error of a solve
    to 1e-10; the residual is checked against the oracle's matrix."""
    import torch
    import vdropimpact_b200 as V
    n, vf = 8, 0.4
    s = V.ViscoImpl(m, n, True, False, vf, vf)
    b = np.random.default_rng(m).standard_normal(m * n)
    s.b.copy_(torch.from_numpy(b))
    s.z.zero_()
    _, rel = s.solve_v_cycle(rtol=1e-10)
    A = vo.visco_matrix(m, n, vf, vf, True, False)
    assert rel <= 1e-10
    assert np.linalg.norm(b - A @ s.z.cpu().numpy()) <= 1e-10 * (1 + 1e-6) * np.linalg.norm(b)
