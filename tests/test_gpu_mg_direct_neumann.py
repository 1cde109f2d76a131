"""The exact solve's choice among the solutions of the pure-Neumann system."""
import numpy as np
import pytest

from oracle import vdi_oracle as vo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,scale", [(100, 50, 1e4), (256, 128, 1e4), (64, 1025, 1e4), (40, 2100, 1e4), (128, 64, 1e8)])
def test_start_far_off(m, n, scale):
    """From a mean-free start much larger than the solution, the correction
    must not carry a constant of the start's size into z: its rounding, eps
    times scale times the operator's diagonal 4 m^2, would stay above 1e-10 of
    |b| through every V-cycle (1e-9 and more here)."""
    import torch
    import vdropimpact_b200 as V
    rng = np.random.default_rng(m)
    b = rng.standard_normal(m * n)
    b -= b.mean()
    z0 = rng.standard_normal(m * n)
    z0 -= z0.mean()
    s = V.MgsMacNeumann(m, n, 1. / m, 1. / m)
    s.b.copy_(torch.from_numpy(b))
    out = []
    for _ in range(2):          # host-driven, then replayed
        s.z.copy_(torch.from_numpy(scale * z0))
        out.append((s.solve_v_cycle(rtol=1e-10), s.z.clone()))
    (_, rel), z = out[0]
    assert rel <= 1e-10
    assert out[1][0] == out[0][0] and torch.equal(out[1][1], z)
    A = vo.mac_matrix(m, n, float(m * m), float(m * m), neumann_bottom=True)
    r = b - A @ z.cpu().numpy()
    assert np.linalg.norm(r) <= 1e-10 * (1 + 1e-3) * np.linalg.norm(b)
