"""The device thermodynamics (csrc/thermo.cuh), compiled for the host, against the known
answers of the reference's own self-tests and against the oracle's restatement.

tests/host_thermo.cu builds the evaluator that athad_thermo_eval runs on the GPU (k_thermo.cu)
for the host, so the same source is checked on a machine without a GPU.  Known answers: each
self-test assertion's tolerance (tests/golden/thermo_kat.json).  Against the oracle, over the
model's range: 1e-14 relative, both sides on the host's libm; the remaining few ulp come from
the device code's arrangement of the curves (the GPU test allows 1e-13 for CUDA's
exp/log/pow).

Skipped where nvcc is not installed.
"""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from oracle_binding import lib as oracle_lib
from thermo_checks import (DEW, DQ_DT, SUBL_P, check_against_the_oracle_over_the_model_range,
                           check_mixture_and_lapse_known_answers, check_saturation_known_answers)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

pytestmark = pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not installed")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("host_thermo") / "libhost_thermo.so")
    cmd = [NVCC, "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr",
           "-gencode", "arch=compute_100a,code=sm_100a",
           "-I", os.path.join(ROOT, "athad_cond_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
           os.path.join(ROOT, "tests", "host_thermo.cu"), "-o", out]
    subprocess.run(cmd, check=True, capture_output=True)
    lib = ctypes.CDLL(out)
    dp = ctypes.POINTER(ctypes.c_double)
    lib.host_thermo_eval.argtypes = [ctypes.c_int, ctypes.c_int, dp, dp]

    def ev(fn, *cols):
        cols = [np.atleast_1d(np.asarray(c, dtype=np.float64)) for c in cols]
        n = max(len(c) for c in cols)
        x = np.ascontiguousarray(np.stack([np.broadcast_to(c, (n,)) for c in cols], axis=1))
        assert x.shape[1] == lib.host_thermo_arity(fn)
        out = np.empty(n)
        assert lib.host_thermo_eval(fn, n, x.ctypes.data_as(dp), out.ctypes.data_as(dp)) == 0
        return out
    return ev


def test_saturation_known_answers_host_build(host):
    check_saturation_known_answers(host)


def test_mixture_and_lapse_known_answers_host_build(host):
    check_mixture_and_lapse_known_answers(host)


def test_host_build_matches_the_oracle_over_the_model_range(host):
    check_against_the_oracle_over_the_model_range(host, tol=1e-14)


def test_dew_point_over_liquid_water_is_unbiased(host):
    """The dew point against the root in extended precision: its mean error over pressures from
    the triple point to 300 bar is rounding, not the rounded logarithm of a constant (which moved
    it by a quarter to half an ulp everywhere).  0.1 ulp is ten standard errors of the mean of
    4000 errors of half an ulp."""
    L = np.longdouble
    rng = np.random.default_rng(20261208)
    e = np.exp(rng.uniform(np.log(6.2), np.log(2.0e5), 4000))
    got = host(DEW, e)

    def f_and_slope(T):     # ln p_sat - ln e and its derivative (SaturationH2O.h:68-93)
        th = 1 - T / L(647.096)
        terms = [(-7.85951783, L(1)), (1.84408259, L(1.5)), (-11.7866497, L(3)), (22.6807411, L(3.5)),
                 (-15.9618719, L(4)), (1.80122502, L(7.5))]
        S = sum(L(c) * th ** x for c, x in terms)
        dS = sum(L(c) * x * th ** (x - 1) for c, x in terms)
        cS = L(647.096) / T * S
        return np.log(L(220640.0) / L(e)) + cS, (-cS - dS) / T
    T = L(got)
    for _ in range(3):
        f, slope = f_and_slope(T)
        T = T - f / slope
    ulps = (L(got) - T) / L(np.spacing(got))
    assert abs(float(np.mean(ulps))) <= 0.1, float(np.mean(ulps))
    assert float(np.max(np.abs(ulps))) <= 4.0


def test_saturation_slope_at_vanishing_pressures(host):
    """dq_sat/dT where the squares of the pressures underflow: the oracle's values, which are
    formed from the ratio of the two pressures."""
    T = np.linspace(14.0, 18.0, 41)
    p = 10.0 * host(SUBL_P, T)
    assert (p > 0.0).all() and (p * p == 0.0).any()
    got = host(DQ_DT, T, p, 0.034)
    want = np.array([oracle_lib().or_dqsat_dT(t, q, 0.034) for t, q in zip(T, p)])
    assert np.isfinite(want).all() and (want > 0.0).all()
    assert (np.abs(got - want) <= 1e-11 * want).all()
