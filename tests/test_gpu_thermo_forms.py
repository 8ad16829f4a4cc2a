"""The two-range form of the property polynomials against the general one.

A mechanism whose polynomials have two ranges and the powers 0..4 takes the fast
T(e), cp and enthalpy paths; any other takes the general ones.  The same
mechanism with a third range, a copy of its second one, gives the general paths
the same polynomials, and both forms round every operation alike: the recovery,
the flux divergences and a chemistry window have the same bits.  The 9-species
mechanism has one middle temperature for all species, the 14-species one several.
"""
import ctypes as C
import dataclasses

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from stx import case as CS  # noqa: E402
from stx.native import check  # noqa: E402
from stx.solver import Solver  # noqa: E402


def _third_range(case):
    tb = case.tb
    assert tb.nsetcv == 2 and (tb.indx_cp_l, tb.indx_cp_r) == (0, 4)
    grow = lambda a: np.concatenate([a, a[:, :, 1:]], axis=2)
    tb = dataclasses.replace(tb, nsetcv=3, trange=np.concatenate([tb.trange, tb.trange[:, 2:] + 500.0], axis=1),
                             cp_coeff=grow(tb.cp_coeff), cv_coeff=grow(tb.cv_coeff))
    out = CS.Case(case.cfg, tb)
    out.w[:], out.w_aux[:] = case.w, case.w_aux
    return out


@pytest.mark.parametrize("form", ["fp64", "mixed"])
@pytest.mark.parametrize("mech,thr", [("h2air_9sp", 0.02), ("h2air_9sp", -0.2), ("keromnes_14sp", 0.02),
                                      ("keromnes_14sp", -0.2)])
def test_two_range_form_equals_general_form(mech, thr, form):
    case = H.synthetic_case(n=(19, 13, 9), mech=mech, seed=11, T0=1350.0, amp_T=1400.0, amp_u=120.0,
                            sensor_threshold=thr)
    T = case.interior(case.w_aux)[case.J("T")]
    assert T.min() < case.tb.trange[:, 1].min() and T.max() > case.tb.trange[:, 1].max()
    out = []
    for c in (case, _third_range(case)):
        s = Solver(c)
        s.set_precision(form)
        s.update_ghost(1)
        s.compute_aux(1, 1)
        p = lambda t: C.c_void_p(t.data_ptr())
        res = [("w_aux", s.w_aux.clone())]
        for d, fn in enumerate((s.lib.stx_euler_x, s.lib.stx_euler_y, s.lib.stx_euler_z)):
            check(fn(s.ctx, s.stream, p(s.w_aux), p(s.fl), 1, (c.nx, c.ny, c.nz)[d], 1 if d == 0 else 0), "euler")
            res.append(("euler", s.fl.clone()))
        for mode in (1, 2):
            s.fl.zero_()
            check(s.lib.stx_visflx(s.ctx, s.stream, p(s.w_aux), p(s.fl), mode), "visflx")
            res.append(("visflx", s.fl.clone()))
        w0 = s.w.clone()
        for simpler in (0, 1):
            s.fl_sav.zero_()
            s.w.copy_(w0)
            check(s.lib.stx_rosenbrock_krylov(s.ctx, s.stream, p(s.w), p(s.w_aux), p(s.fl_sav), 1e-7, 0.0, 1e-7,
                                              simpler), "rok4")
            res.append(("rok4", s.w.clone()))
            assert not torch.equal(s.w, w0)
        torch.cuda.synchronize()
        out.append(res)
        s.close()
    for (name, a), (_, b) in zip(*out):
        assert torch.isfinite(a).all(), name
        for m in range(a.shape[0]):
            assert torch.equal(a[m], b[m]), (name, m)
