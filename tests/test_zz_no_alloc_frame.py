"""The allocation-free entry point serves a caller whose stack limit is the frame
that include/stx.h has given for it: 2624 bytes at 9 species and 3360 at 14 in its
first form, less now."""
import ctypes as C

import pytest

import helpers as H

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

import test_zz_no_alloc as T  # noqa: E402
from stx.native import StxGrid, load_stx  # noqa: E402


@pytest.mark.parametrize("mech,limit", [("h2air_9sp", 2624), ("h2air_9sp", 2208), ("keromnes_14sp", 3360),
                                        ("keromnes_14sp", 2928)])
def test_documented_frame_is_enough(mech, limit):
    dev = torch.device("cuda", torch.cuda.current_device())
    case = H.synthetic_case(n=(10, 8, 6), mech=mech, seed=23, T0=1300.0, amp_T=200.0)
    tabs = T.DeviceTables(case, dev)
    w, wa = torch.from_numpy(case.w.copy()).to(dev), torch.from_numpy(case.w_aux.copy()).to(dev)
    wa[case.J("Z")] = 0.5
    w0 = w.clone()
    grid, par = StxGrid(), case.params_struct()
    grid.nx, grid.ny, grid.nz, grid.ng = case.nx, case.ny, case.nz, case.ng
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    torch.cuda.synchronize()
    try:
        assert T.set_stack_limit(limit) == limit
        rc = T._bind(load_stx())(C.byref(par), C.byref(tabs.t), C.byref(grid), None, C.c_void_p(w.data_ptr()),
                                 C.c_void_p(wa.data_ptr()), None, 1e-7, 0.0, 1e-7, 0, C.c_void_p(status.data_ptr()))
        torch.cuda.synchronize()
    finally:
        T.set_stack_limit(T.STACK_BYTES)
    assert rc == 0
    assert torch.isfinite(w).all() and not torch.equal(w, w0)
