"""The logarithm and the Arrhenius form of the packed reaction records
(csrc/stx_rates.cuh), compiled for the host, against 50-digit values."""
import ctypes as C
import decimal
import os
import subprocess

import numpy as np
import pytest

import helpers as H

CSRC = os.path.join(H.REPO, "prop-streams2_b200", "csrc")
U = 2.0 ** -53
D = decimal.Decimal

SRC = r'''
#include "stx_rates.cuh"
extern "C" void logs(int n, const double *x, double *hi, double *lo) {
  for (int i = 0; i < n; i++) log_dd(x[i], hi[i], lo[i]);
}
extern "C" double rate(double A, double b, double nE, double T, double rt) {
  double h, l;
  log_dd(T, h, l);
  return arrhenius_dd(A, b, nE, h, l, rt);
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("rates")
    (d / "r.cpp").write_text(SRC)
    so = str(d / "r.so")
    # the chemistry's arithmetic: no contraction beyond the written fma
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, "-o", so,
                    str(d / "r.cpp")], check=True)
    lib = C.CDLL(so)
    lib.rate.restype = C.c_double
    lib.rate.argtypes = [C.c_double] * 5
    return lib


@pytest.fixture(autouse=True)
def digits():
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        yield


def _temperatures():
    rng = np.random.default_rng(3)
    edges = [1.0, np.nextafter(1.0, 2.0), 2.0 ** 0.5, np.nextafter(2.0 ** 0.5, 2.0), 2.0, 1023.9999999999999, 1024.0,
             1e6]
    edges += [np.nextafter(2.0 ** k, 0.0) for k in range(1, 20)] + [2.0 ** (k + 0.5) for k in range(19)]
    return np.concatenate([edges, np.exp(rng.uniform(0.0, np.log(1e6), 2000)), rng.uniform(200.0, 5500.0, 1000)])


def test_log_in_two_doubles(lib):
    """Within the 4e-18 that the header states, over 1 to 1e6."""
    T = np.ascontiguousarray(_temperatures())
    hi, lo = np.empty_like(T), np.empty_like(T)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    lib.logs(T.size, p(T), p(hi), p(lo))
    err = [abs(D(float(h)) + D(float(l)) - D(float(t)).ln()) for t, h, l in zip(T, hi, lo)]
    assert max(err) < D("4e-18"), (max(err), T[int(np.argmax([float(e) for e in err]))])
    assert np.all(np.abs(lo) <= np.spacing(hi) + 4e-18)         # hi is ln T rounded


@pytest.mark.parametrize("mech", ["h2air_9sp", "keromnes_14sp", "shock_tube_9sp"])
def test_arrhenius_form(lib, mech):
    """Every rate of the shipped mechanisms, 200 to 3500 K, against A T^b exp(q) with
    q = nE rt exact.  Roundings: that of nE rt (|q| U), of the exponential (2 U with
    an error below one ulp), of the correction and of the product (U each), and the
    logarithm's 4e-18 b; one U beside them for the second order."""
    tb = H.tables(mech, 101325.0)
    rng = np.random.default_rng(4)
    T = np.concatenate([[200.0, 298.15, 1000.0, 3500.0], rng.uniform(200.0, 3500.0, 12)])
    worst = 0.0
    for col in (0, 1):
        for A, b, E in zip(tb.arr_a[:, col], tb.arr_b[:, col], tb.arr_ea[:, col]):
            if A == 0.0:
                continue
            for t in T:
                rt = 1.0 / (H.CS.M.R_UNIV * t)
                got = lib.rate(A, b, -E, t, rt)
                q = D(float(-E)) * D(rt)
                ref = D(float(A)) * (D(float(b)) * D(float(t)).ln() + q).exp()
                err = float(abs(D(got) / ref - 1))
                worst = max(worst, err / ((abs(float(q)) + 5.0) * U))
                assert err <= (abs(float(q)) + 5.0) * U, (mech, A, b, E, t, err)
    assert worst > 0.05              # the bound is not slack by orders of magnitude
