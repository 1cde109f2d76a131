"""V-cycles on grids of more tiles than the 8192 partial sums that smaller
grids share: the residual norm's sums need a place for every tile."""
import pytest

pytestmark = pytest.mark.gpu


def test_fem_8193x4097():
    """187 x 94 tiles of 44 x 44 nodes, on rows too long for the exact solve.
    The norm that ends the solve is the tiles' sum; the residual entry point
    adds it up over other blocks."""
    import torch
    import vdropimpact_b200 as V
    m, n = 8193, 4097
    s = V.MgsFem(m, n, 1.0 / (m - 1), 1.0 / (m - 1))
    g = torch.Generator(device="cuda").manual_seed(5)
    s.b.copy_(torch.randn(m * n, dtype=torch.float64, device="cuda", generator=g))
    s.z.zero_()
    v, rel = s.solve_v_cycle(rtol=1e-8)
    _, nr = s.residual()
    ref = float(torch.linalg.vector_norm(s.b))
    assert 1 <= v and rel <= 1e-8
    # A z rounds to eps |A| |z|, about 2e-12 of ||b|| for the 2e3 ||b|| that
    # the slowest modes of white noise make of z
    assert abs(nr / ref - rel) <= 1e-11
