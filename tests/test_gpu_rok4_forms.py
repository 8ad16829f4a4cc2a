"""The forms of the ROK4 cell update against one another.

A grid of up to 8192 cells takes a warp per cell and a larger one a thread per
cell, with the same operations in the same order: the same cells give the same
bits.  A mechanism whose reactions all fit the packed records takes them;
otherwise the sparse stoichiometry lists serve it.  Both are run on the same
cells: without the Strang splitting's shared exponential the bits are the same,
with it the rates differ by rounding.
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

from driver import OracleSolver  # noqa: E402
from stx import case as CS  # noqa: E402
from stx import mech as M  # noqa: E402
from stx.native import check  # noqa: E402
from stx.solver import Solver  # noqa: E402

DT = 2e-7


def _source(case, simpler, seed=7):
    """A prepared solver and its fl_sav (the simpler splitting's residual)."""
    s = Solver(case)
    s.update_ghost(1)
    s.compute_aux(1, 1)
    rng = np.random.default_rng(seed)
    scale = np.abs(case.interior(s.host_w())).max(axis=(1, 2, 3)) * 1e3
    fs = torch.from_numpy(rng.standard_normal(tuple(s.fl_sav.shape)) * scale[:, None, None, None]).to(s.device)
    return s, fs if simpler else None


def _rok4(s, fs, simpler):
    check(s.lib.stx_rosenbrock_krylov(s.ctx, s.stream, C.c_void_p(s.w.data_ptr()), C.c_void_p(s.w_aux.data_ptr()),
                                      None if fs is None else C.c_void_p(fs.data_ptr()), DT, 0.0, DT, simpler), "rok4")
    torch.cuda.synchronize()
    return s.case.interior(s.host_w())


@pytest.mark.parametrize("n", [(16, 16, 8), (13, 9, 7), (32, 16, 16)])
@pytest.mark.parametrize("simpler", [0, 1])
def test_warp_per_cell_equals_thread_per_cell(n, simpler):
    """A small box, and the same box repeated until the thread-per-cell kernel takes it."""
    small = H.synthetic_case(n=n, seed=31, T0=1300.0, amp_T=400.0)
    s, fs = _source(small, simpler)
    rep = -(-8193 // (n[0] * n[1] * n[2]))
    big = H.synthetic_case(n=(n[0], n[1], n[2] * rep), seed=31, T0=1300.0, amp_T=400.0)
    b = Solver(big)
    b.compute_aux(1, 1)
    for src, dst in ((s.w, b.w), (s.w_aux, b.w_aux)):
        big.interior(dst)[:] = small.interior(src).repeat(1, rep, 1, 1)
    fb = None if fs is None else fs.repeat(1, rep, 1, 1).contiguous()
    got, ref = _rok4(s, fs, simpler), _rok4(b, fb, simpler)
    for q in range(rep):
        assert np.array_equal(got, ref[:, q * n[2]:(q + 1) * n[2]]), q
    s.close()
    b.close()


def _padded(case):
    """The case with one more, inert reaction (A = 0) whose stoichiometry fits no record."""
    tb = case.tb
    row = lambda a, v: np.concatenate([a, np.full((1,) + a.shape[1:], v, a.dtype)])
    rc, pc = row(tb.r_coeffs, 0), row(tb.p_coeffs, 0)
    rc[-1, 0], pc[-1, 1] = 1.5, 1.5
    tb = dataclasses.replace(tb, nr=tb.nr + 1, reac_ty=row(tb.reac_ty, 0), is_rev=row(tb.is_rev, 0),
                             arr_a=row(tb.arr_a, 0), arr_b=row(tb.arr_b, 0), arr_ea=row(tb.arr_ea, 0),
                             falloff=row(tb.falloff, 0), tb_eff=row(tb.tb_eff, 0), r_coeffs=rc, p_coeffs=pc,
                             kc_tab=np.concatenate([tb.kc_tab, np.ones_like(tb.kc_tab[:, :1])], axis=1))
    return CS.Case(case.cfg, tb)


@pytest.mark.parametrize("n", [(8, 6, 5), (32, 20, 16)])
@pytest.mark.parametrize("simpler", [0, 1])
def test_records_equal_sparse_lists(n, simpler):
    case = H.synthetic_case(n=n, seed=33, T0=1300.0, amp_T=400.0)
    other = _padded(case)
    other.w[:], other.w_aux[:] = case.w, case.w_aux
    (s, fs), (o, fo) = _source(case, simpler), _source(other, simpler)
    got, ref = _rok4(s, fs, simpler), _rok4(o, fo, simpler)
    if simpler:
        assert np.array_equal(got, ref)
    else:
        # A rounding of the rates, 1e-16, enters the finite-difference Jacobian
        # divided by its step of 1e-8, and an adaptive window carries that: 1e-8
        # of the species' scale.
        for m in range(case.nv):
            H.assert_close(got[m], ref[m], 1e-8, f"w[{m}]", floor=np.abs(ref[m]).max())
    s.close()
    o.close()


def _with_reaction(case, reac, prod, A, kc=None, b=0.0, ER=0.0):
    """The case with one more reaction, reac and prod: {species: molecules}; kc: its equilibrium constant
    (None: irreversible); ER: E/R in K."""
    tb = case.tb
    row = lambda a, v: np.concatenate([a, np.full((1,) + a.shape[1:], v, a.dtype)])
    rc, pc = row(tb.r_coeffs, 0), row(tb.p_coeffs, 0)
    for c, side in ((rc, reac), (pc, prod)):
        for k, n in side.items():
            c[-1, tb.names.index(k)] = n
    aa, ab, ae = row(tb.arr_a, 0), row(tb.arr_b, 0), row(tb.arr_ea, 0)
    aa[-1, 0], ab[-1, 0], ae[-1, 0] = A, b, ER * CS.M.R_UNIV
    tb = dataclasses.replace(tb, nr=tb.nr + 1, reac_ty=row(tb.reac_ty, 0), is_rev=row(tb.is_rev, int(kc is not None)),
                             arr_a=aa, arr_b=ab, arr_ea=ae, falloff=row(tb.falloff, 0), tb_eff=row(tb.tb_eff, 0),
                             r_coeffs=rc, p_coeffs=pc,
                             kc_tab=np.concatenate([tb.kc_tab, np.full_like(tb.kc_tab[:, :1], kc or 1.0)], axis=1))
    return _like(case, tb)


def _like(case, tb):
    out = CS.Case(case.cfg, tb)
    out.w[:], out.w_aux[:] = case.w, case.w_aux
    return out


# sides of two and three molecules: a species that counts twice before and after a
# single one, three different ones, and three alike (which no record holds), with
# rates that compare with the mechanism's own
SIDES = [({"H2": 2, "O2": 1}, {"H2O": 2}, 1e10, None), ({"O": 2, "H2": 1}, {"OH": 2}, 1e16, None),
         ({"OH": 2}, {"O": 2, "H2": 1}, 1e13, 1e-3), ({"H": 1, "O2": 1, "N2": 1}, {"HO2": 1, "N2": 1}, 1e11, None),
         ({"OH": 3}, {"H2O": 1, "HO2": 1}, 1e19, None), ({"H2O": 1, "HO2": 1}, {"OH": 3}, 1e13, 1e-6)]


@pytest.mark.parametrize("n", [(8, 6, 5), (32, 20, 16)])
@pytest.mark.parametrize("reac,prod,A,kc", SIDES)
def test_every_form_of_a_side_has_the_bits_of_the_lists(reac, prod, A, kc, n):
    """The simpler splitting (no shared exponential), warp and thread per cell."""
    base = H.synthetic_case(n=n, seed=35, T0=1300.0, amp_T=400.0)
    case = _with_reaction(base, reac, prod, A, kc)
    lists = _like(case, _padded(case).tb)
    (z, fz), (s, fs), (o, fo) = _source(base, 1), _source(case, 1), _source(lists, 1)
    plain, got, ref = _rok4(z, fz, 1), _rok4(s, fs, 1), _rok4(o, fo, 1)
    assert not np.array_equal(plain, got)            # the reaction counts
    assert np.array_equal(got, ref)
    for x in (z, s, o):
        x.close()


@pytest.mark.parametrize("reac,prod,A,kc", SIDES)
@pytest.mark.parametrize("simpler", [0, 1])
def test_every_form_of_a_side_in_the_warp_and_the_thread_kernel(reac, prod, A, kc, simpler):
    case = _with_reaction(H.synthetic_case(n=(8, 6, 5), seed=35, T0=1300.0, amp_T=400.0), reac, prod, A, kc)
    s, fs = _source(case, simpler)
    w0 = s.w.clone()
    out = []
    for ctas in (0, 1):
        s.set_tuning({"sweep_kind": [0, 0, 0], "weno_list": [1, 1, 1], "chem_ctas_per_sm": ctas})
        s.w.copy_(w0)
        out.append(_rok4(s, fs, simpler).copy())
    assert np.array_equal(out[0], out[1])
    s.close()


@pytest.mark.parametrize("n", [(8, 6, 5), (32, 20, 16)])
@pytest.mark.parametrize("simpler", [0, 1])
def test_rates_beyond_the_records_temperatures_take_the_lists(simpler, n):
    """A = 1e-307, b = 22, E/R = -728000 K: 5e4 at 1300 K, where b ln T - E / (R T) is
    717 and its exponential overflows.  The records' lower limit, 1840 K here, leaves
    such cells to the power and the exponential of the lists."""
    base = H.synthetic_case(n=n, seed=37, T0=1300.0, amp_T=0.0)
    case = _with_reaction(base, {"H2": 1, "O2": 1}, {"OH": 2}, 1e-307, b=22.0, ER=-728000.0)
    lists = _like(case, _padded(case).tb)
    (z, fz), (s, fs), (o, fo) = _source(base, simpler), _source(case, simpler), _source(lists, simpler)
    plain, got, ref = _rok4(z, fz, simpler), _rok4(s, fs, simpler), _rok4(o, fo, simpler)
    assert np.isfinite(ref).all() and not np.array_equal(plain, ref)
    assert np.array_equal(got, ref)
    for x in (z, s, o):
        x.close()


# one cp range boundary for all species and plain, three-body and Troe reactions (9, 11);
# several boundaries, Lindemann and a side with a repeated species (14, and 13 without He)
MECHS = ["h2air_9sp", "flame_11sp", "keromnes_13sp", "keromnes_14sp"]


@pytest.fixture
def any_mech(monkeypatch):
    full = H.mechanism

    def pick(name):
        if name != "keromnes_13sp":
            return full(name)
        m = full("keromnes_14sp")
        return M.restrict_species(m, [x for x in m.names if x != "HE"])

    monkeypatch.setattr(H, "mechanism", pick)


def _tune(s, ctas):
    s.set_tuning({"sweep_kind": [0, 0, 0], "weno_list": [1, 1, 1], "chem_ctas_per_sm": ctas})


@pytest.mark.parametrize("mech", MECHS)
@pytest.mark.parametrize("simpler", [0, 1])
def test_every_mechanism_warp_thread_and_lists(any_mech, mech, simpler):
    """431 cells (no multiple of a warp or a CTA): the warp kernel, the thread kernel's
    persistent and plain launches and, without the shared exponential, the lists."""
    case = H.synthetic_case(n=(431, 1, 1), mech=mech, seed=39, T0=1350.0, amp_T=1400.0)
    s, fs = _source(case, simpler)
    w0 = s.w.clone()
    out = []
    for ctas in (0, 1, -1):
        _tune(s, ctas)
        s.w.copy_(w0)
        out.append(_rok4(s, fs, simpler).copy())
    assert not np.array_equal(out[0], case.interior(w0.cpu().numpy())) and np.isfinite(out[0]).all()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    o, fo = _source(_like(case, _padded(case).tb), simpler)
    for ctas in (0, 1):
        _tune(o, ctas)
        o.w.copy_(w0)
        ref = _rok4(o, fo, simpler)
        if simpler:
            assert np.array_equal(out[0], ref)
        else:                            # the bound of test_records_equal_sparse_lists
            for m in range(case.nv):
                H.assert_close(out[0][m], ref[m], 1e-8, f"w[{m}]", floor=np.abs(ref[m]).max())
    s.close()
    o.close()


@pytest.mark.parametrize("mech", MECHS)
@pytest.mark.parametrize("ctas", [0, 1, -1])
@pytest.mark.parametrize("simpler", [0, 1])
def test_every_kernel_against_the_oracle(any_mech, mech, ctas, simpler):
    """A short window of each kernel against the FP64 oracle, to 1e-9 of a component
    (one or two steps: rounding enters through exp, pow and log10 alone)."""
    case = H.synthetic_case(n=(10, 8, 6), mech=mech, seed=10, T0=1300.0, amp_T=200.0)
    s = Solver(case)
    o = OracleSolver(case, threads=8)
    o.update_ghost(1)
    o.compute_aux(1, 1)
    o.fl_sav[:] = 1e-3 * np.random.default_rng(12).standard_normal(o.fl_sav.shape)
    s.w.copy_(torch.from_numpy(o.w))
    s.w_aux.copy_(torch.from_numpy(o.w_aux))
    s.fl_sav.copy_(torch.from_numpy(o.fl_sav))
    _tune(s, ctas)
    p = lambda a: C.c_void_p(a.ctypes.data)
    w0 = case.interior(o.w).copy()
    o.lib.ox_rosenbrock_krylov(o.ctx, p(o.w), p(o.w_aux), p(o.fl_sav), DT, 0.0, DT, simpler)
    wg, wo = _rok4(s, s.fl_sav, simpler), case.interior(o.w)
    assert not np.array_equal(wo, w0)
    for m in range(case.nv):
        H.assert_close(wg[m], wo[m], 1e-9, f"w[{m}]", floor=1e-9 * np.abs(wo[:case.ns]).max() if m < case.ns else None)
    s.close()
    o.close()
