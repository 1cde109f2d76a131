"""The FEM solve inside a step. Its source holds the gas pressure on the
bottom row, so an iterate that meets 1e-10 of ||b|| is not determined to
1e-10 in the rows above, and v follows it through the pressure gradient: a
step at such a tolerance gives the fields of earlier runs only with the
V-cycles of the asked precision. At 1e-12 either solver gives them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def V():
    import vdropimpact_b200 as V
    return V


def _cfg(m, n, nu, vel):
    return (f"grid_points {m} {n}\nL_nd 45\nh0_nd 15\nt_end_nd 100\nframes 250\ntmult 8e-3\nnul_cSt {nu}\n"
            f"rhol 997.96\nR 1.5e-3\nV {vel}\ngamma 1.4\nsigma 72e-3\nmug 1.820775e-5\nPamb 1e5\n"
            "gas_layer_model\nimplicit_visc\n")


def _run(V, cfg, prec, graph, rtol, steps):
    f = V.Fluid2D(cfg, mg_rtol=rtol, mg_precision=prec, mg_guess="quadratic", graph=graph)
    f.init_fields()
    f.step_forward(f.frame_dt(), steps)
    a, st = f.state(), f.stats()
    f.close()
    return a, st


# full domains, whose pressure has no symmetry axis to anchor it
@pytest.mark.parametrize("m,n,nu,vel,prec,graph,rtol,steps", [
    (512, 256, 16.20974755, 0.43549018, "mixed", False, 1e-10, 4),
    (1024, 512, 71.17801490, 0.49289703, "hybrid", True, 1e-10, 6),
    (200, 100, 5.0, 0.45, "fp64", True, 1e-12, 5),
    (512, 256, 16.20974755, 0.43549018, "mixed", False, 1e-12, 4),
])
def test_step_keeps_the_fields_of_vcycle_solves(V, monkeypatch, m, n, nu, vel, prec, graph, rtol, steps):
    """Against the same steps with the exact solve turned off everywhere: at
    1e-10 as many FEM V-cycles, and u, v and p within 1e-9 in the 2-norm and
    4e-8 at every point (of the larger of the value and the field's RMS), ten
    and four hundred times the looser tolerance."""
    cfg = _cfg(m, n, nu, vel)
    a, sa = _run(V, cfg, prec, graph, rtol, steps)
    monkeypatch.setenv("VDI_MG_DIRECT", "0")
    b, sb = _run(V, cfg, prec, graph, rtol, steps)
    if rtol > 1e-12:
        assert sa["vcycles"]["FEM"] == sb["vcycles"]["FEM"]
    for k in ("u", "v", "p"):
        x, y = np.asarray(a[k]), np.asarray(b[k])
        nr = np.linalg.norm(y)
        d = np.abs(x - y)
        assert np.linalg.norm(x - y) <= 1e-9 * nr, (k, np.linalg.norm(x - y) / nr)
        assert np.max(d / np.maximum(nr / np.sqrt(y.size), np.abs(y))) <= 4e-8, k
