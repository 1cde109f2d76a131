"""What solves report and are capped by where the exact solve (csrc/
mg_direct.cuh) or the SOR passes (csrc/mg_relax.cuh) stand in for V-cycles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def V():
    import vdropimpact_b200 as V
    return V


@pytest.mark.parametrize("m,n", [(256, 128), (1024, 512)])
@pytest.mark.parametrize("vf", [0.4, 2.0, 3.75, 7.5])
@pytest.mark.parametrize("rtol", [1e-4, 1e-10])
def test_a_cap_that_vcycles_meet_is_met(V, monkeypatch, m, n, vf, rtol):
    """A pair of passes (eight sweeps) gains a factor (omega - 1)^8, 0.02 or
    less where SOR is used, and a V-cycle 0.1 to 0.01 at the same couplings:
    with the V-cycles' own count as the cap the passes meet the tolerance."""
    import torch
    b = V.projection_source(m, n, 3) + 0.01 * np.random.default_rng(3).standard_normal(m * n)

    def solve(cap):
        s = V.ViscoImpl(m, n, True, True, vf, vf)
        s.b.copy_(torch.from_numpy(b))
        out = []
        for _ in range(2):          # host-driven, then replayed
            s.z.copy_(s.b)
            out.append(s.solve_v_cycle(rtol=rtol, max_vcycles=cap))
        assert out[0] == out[1] and out[0][1] <= rtol
        return out[0][0]

    monkeypatch.setenv("VDI_MG_SOR", "0")
    count = solve(200)
    monkeypatch.delenv("VDI_MG_SOR")
    assert 1 <= solve(count) <= count


def test_launches_of_solves_that_end_at_the_first_check(V):
    """A tolerance of 1 ends every solve of a first step at its first check,
    but a viscous solve's pair of passes is launched all the same. Against a
    step whose solves run (the exact solve's four kernels in place of the FEM
    check, two launches a counted pair) everything else is equal."""
    import os
    cfg = open(os.path.join(os.path.dirname(__file__), "golden", "ld_vis100.cfg")).read()
    cfg = "\n".join([q for q in cfg.splitlines() if not q.startswith("grid_points")] + ["grid_points 64 32"]) + "\n"

    def step(rtol):
        f = V.Fluid2D(cfg, mg_rtol=rtol)
        f.init_fields()
        f.stats(reset=True)
        f.step_forward(f.frame_dt(), 1)
        st = f.stats()
        f.close()
        return st

    idle, busy = step(1.0), step(1e-12)
    assert set(idle["vcycles"].values()) == {0} and set(idle["solves"].values()) == {1}
    pairs = [busy["vcycles"][k] for k in ("VX", "VY")]
    assert min(pairs) >= 1
    assert busy["kernel_launches"] - idle["kernel_launches"] == (4 - 1) + sum(2 * (q - 1) for q in pairs)


@pytest.mark.parametrize("kind,m,n", [("mac", 100, 50), ("mac", 128, 64), ("fem", 101, 51), ("fem", 129, 65),
                                      ("neumann", 100, 50), ("neumann", 256, 128)])
@pytest.mark.parametrize("scale", [0.0, 1.0, 1e4, 1e8])
def test_a_cap_that_vcycles_meet_is_met_by_exact_solves(V, monkeypatch, kind, m, n, scale):
    """From starts near and far off, with every cap from the V-cycles' own
    count on: below the exact solve's count (and what has to follow it) the
    V-cycles run, above it there is room for both. (The far-off Neumann starts
    that V-cycles alone do not bring to 1e-10 have no such cap.)"""
    import torch
    rng = np.random.default_rng(m)
    b, z0 = rng.standard_normal(m * n), scale * rng.standard_normal(m * n)
    if kind == "neumann":
        b -= b.mean()
        z0 -= z0.mean()
        if scale == 1e8:
            pytest.skip("V-cycles stop at the rounding of the mean")

    def solver():
        s = {"mac": V.MgsMac, "fem": V.MgsFem, "neumann": V.MgsMacNeumann}[kind](m, n, 1. / m, 1. / m)
        s.b.copy_(torch.from_numpy(b))
        return s

    def solve(s, cap):
        s.z.copy_(torch.from_numpy(z0))
        return s.solve_v_cycle(rtol=1e-10, max_vcycles=cap)

    monkeypatch.setenv("VDI_MG_DIRECT", "0")
    count = solve(solver(), 200)[0]
    monkeypatch.delenv("VDI_MG_DIRECT")
    s = solver()
    for cap in range(count, count + 40):
        v, rel = solve(s, cap)
        assert rel <= 1e-10 and v <= cap, cap
