"""A system is created on a device that has room for its V-cycles but not for
the tables and the modal array of the exact solve, and runs V-cycles."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_creation_without_room_for_the_exact_solve(monkeypatch):
    """4096 x 2048 cells: the exact solve's allocation takes 88 MB (67 for the
    modal array, 21 of tables); 48 MB are left for it beyond what the V-cycles
    took when they alone were set up."""
    import torch
    import vdropimpact_b200 as V
    from vdropimpact_b200 import _abi
    L = _abi.lib()
    m, n = 4096, 2048
    g = torch.Generator(device="cuda").manual_seed(1)
    b = torch.randn(m * n, dtype=torch.float64, device="cuda", generator=g)
    z = torch.zeros_like(b)

    def create():
        h = C.c_void_p()
        _abi.check(L.vdi_mg_create(_abi.VDI_MG_MAC, m, n, 1. / m, 1. / m, 0, None, C.byref(h)), "vdi_mg_create")
        return h

    def solve(h):
        r = _abi.VdiMgResult()
        z.zero_()
        torch.cuda.synchronize()
        _abi.check(L.vdi_mg_solve(h, C.c_void_p(b.data_ptr()), C.c_void_p(z.data_ptr()), 1e-10, 200, 0, C.byref(r)),
                   "vdi_mg_solve")
        return r.vcycles, z.clone()

    # the V-cycles alone: their memory, their kernels loaded, their solution
    monkeypatch.setenv("VDI_MG_DIRECT", "0")
    before = torch.cuda.mem_get_info()[0]
    h = create()
    need = before - torch.cuda.mem_get_info()[0]
    vcycles, want = solve(h)
    L.vdi_mg_destroy(h)
    monkeypatch.delenv("VDI_MG_DIRECT")

    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - need - (48 << 20), dtype=torch.uint8, device="cuda")
    try:
        h = create()
    finally:
        del fill
        torch.cuda.empty_cache()
    v, got = solve(h)
    L.vdi_mg_destroy(h)
    assert v == vcycles and torch.equal(got, want)
