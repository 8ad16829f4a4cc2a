"""The chemistry's launch is the one that the context's tuning names.

chem_ctas_per_sm = 0 leaves it to the grid's size (a warp per cell up to 8192
cells); 1 and up and -1 name the thread-per-cell kernel at any size, which is
seen from the launched kernels' names.  All give the same bits.
"""
import ctypes as C

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from stx.native import check  # noqa: E402
from stx.solver import Solver  # noqa: E402

DT = 2e-7
BASE = {"sweep_kind": [0, 0, 0], "weno_list": [1, 1, 1]}


def _kernels(fn):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    return [e.key for e in prof.key_averages() if "k_rok4" in e.key]


@pytest.mark.parametrize("n,small", [((16, 16, 8), True), ((32, 16, 16), True), ((32, 17, 16), False)])
def test_tuning_names_the_kernel(n, small):
    case = H.synthetic_case(n=n, seed=31, T0=1300.0, amp_T=400.0)
    s = Solver(case)
    s.update_ghost(1)
    s.compute_aux(1, 1)
    w0 = s.w.clone()

    def rok4():
        check(s.lib.stx_rosenbrock_krylov(s.ctx, s.stream, C.c_void_p(s.w.data_ptr()), C.c_void_p(s.w_aux.data_ptr()),
                                          None, DT, 0.0, DT, 0), "rok4")

    out = []
    for ctas in (0, 1, s.tuning()["chem_ctas_max"], -1):
        s.set_tuning(dict(BASE, chem_ctas_per_sm=ctas))
        s.w.copy_(w0)
        names = _kernels(rok4)
        assert len(names) == 1 and ("k_rok4_w<" in names[0]) == (small and ctas == 0), (ctas, names)
        out.append(case.interior(s.host_w()).copy())
    assert not np.array_equal(out[0], case.interior(w0.cpu().numpy()))
    for o in out[1:]:
        assert np.array_equal(o, out[0])
    s.close()


def test_autotune_times_the_warp_kernel_on_small_grids():
    """2048 hot cells: a warp per cell takes a third of a thread per cell's time, so it stays the choice."""
    case = H.synthetic_case(n=(16, 16, 8), seed=31, T0=1300.0, amp_T=400.0)
    s = Solver(case)
    s.update_ghost(1)
    s.compute_aux(1, 1)
    names = _kernels(lambda: s.autotune(dt_chem=DT))
    assert any("k_rok4_w<" in k for k in names) and any("k_rok4<" in k for k in names), names
    assert s.tuning()["chem_ctas_per_sm"] == 0
    s.close()
