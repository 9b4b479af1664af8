"""The FP64 path's block fixed-point transforms (csrc/fxfft.cuh) against
extended-precision transforms, and the FP64 step and its adjoint at the
lengths whose radix plans differ (16, 32, 128, 1024).

Tolerance of one 2D transform: each of its two 1D transforms rounds its
outputs to doubles (at most 2^-53 relative, 2^-53.8 in the mean square) and
carries the fixed-point noise of a spectrum with a single large value, whose
integers keep 53 bits below the growth bound: eight inputs of a last
butterfly rounded at half a unit, sqrt(8/12) 2^-53.  Together below
sqrt(2) (2^-53.8 + 2^-53.3) < 2^-51.9; the test allows 2^-51.8."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.fft as sfft

from oracle.qgybj_adjoint import Adjoint
from qgybj import Simulation
from qgybj.config import CONFIGS, scaled
from tests.helpers import oracle_for, random_masked, rel_l2

pytestmark = pytest.mark.gpu

TOL = 2.0 ** -51.8


def _sim(n, n3=2):
    return Simulation(dict(n1=n, n2=n, n3=n3, dz=1.0 / n3, Bu=1.0, Ro=0.1, W2F=1.0, delt=1e-3, gamma=1e-3, a_ell_ut=np.ones(n3)),
                      "fp64")


def _realit(k, n):
    k = k.copy()
    m = np.arange(1, n // 2)
    k[..., n - m, 0] = np.conj(k[..., m, 0])
    return k


def _spectrum(kind, n):
    rng = np.random.default_rng(n)
    z = rng.standard_normal((1, n, n // 2 + 1)) + 1j * rng.standard_normal((1, n, n // 2 + 1))
    k2 = np.arange(n // 2 + 1)[None, :] ** 2 + np.fft.fftfreq(n, 1.0 / n)[:, None] ** 2
    if kind == "steep":
        z = z / (1 + k2) ** 3
    elif kind == "gauss":            # columns down to subnormal values
        z = z * np.exp(-k2 / 18.0)
    elif kind == "one":
        z = np.where(k2 == 13, z, 0)
    elif kind == "tiny":             # every input subnormal or close to it
        z = z * 1e-306
    elif kind == "huge":
        z = z * 1e300
    z[0, 0, 0] = z[0, 0, 0].real
    z[0, n // 2, 0] = z[0, n // 2, 0].real
    return np.ascontiguousarray(z)


@pytest.mark.parametrize("kind", ["white", "steep", "gauss", "one", "tiny", "huge"])
@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 512, 1024])
def test_transforms_against_extended_precision(n, kind):
    if n >= 512 and kind not in ("white", "steep"):
        pytest.skip("the long extended-precision transforms are slow")
    k = _spectrum(kind, n)
    with np.errstate(over="ignore", under="ignore"), _sim(n) as sim:
        ex = sfft.irfft2(_realit(k, n).astype(np.clongdouble), s=(n, n), norm="forward")
        sc = np.abs(ex).max()
        got = sim.fft_c2r(k)
        assert not got[..., n:].any()
        # at the smallest scales a result is no finer than the subnormals' spacing
        floor = float(n * np.longdouble(5e-324) / (np.linalg.norm((ex / sc).astype(float)) * sc)) if kind == "tiny" else 0.0
        err = np.linalg.norm(((got[..., :n] - ex) / sc).astype(float)) / np.linalg.norm((ex / sc).astype(float))
        assert err <= TOL + floor, err
        r = np.zeros((1, n, n + 2))
        r[..., :n] = ex.astype(float)
        fx = sfft.rfft2(r[..., :n].astype(np.longdouble), norm="forward")
        sc = np.abs(fx).max()
        err = np.linalg.norm(((sim.fft_r2c(r) - fx) / sc).astype(complex)) / np.linalg.norm((fx / sc).astype(complex))
        floor = float(n * np.longdouble(5e-324) / (np.linalg.norm((fx / sc).astype(complex)) * sc)) if kind == "tiny" else 0.0
        assert err <= TOL + floor, err


def test_nonfinite_zero_and_overflowing_inputs():
    n = 64
    with _sim(n) as sim:
        k = np.zeros((2, n, n // 2 + 1), dtype=complex)
        assert not sim.fft_c2r(k).any() and not sim.fft_r2c(np.zeros((2, n, n + 2))).any()
        k[0, 3, 5] = np.nan
        out = sim.fft_c2r(k)[..., :n]
        assert np.isnan(out[0]).all() and not out[1].any()
        k[0, 3, 5] = np.inf
        assert not np.isfinite(sim.fft_c2r(k)[0, :, :n]).any()
        k[0] = 1e306       # the sums exceed the largest double at the origin
        assert np.isinf(sim.fft_c2r(k)[0, 0, 0])


@pytest.mark.parametrize("n,n3", [(16, 5), (32, 3), (64, 7), (128, 4), (256, 3), (1024, 2)])
def test_fp64_step_and_transpose(n, n3):
    model, st, ic, params = oracle_for(scaled(CONFIGS["c4"], n, n3))
    adj = Adjoint(model)
    X = tuple(adj.mask(a + 0.05 * random_masked(n, n3, 60 + i) / (1 + model.kh2f)) for i, a in
              enumerate((st.q, st.qo, st.BR, st.BI, st.BRo, st.BIo)))
    lam = tuple(random_masked(n, n3, 80 + i) for i in range(6))
    with Simulation(params, "fp64") as sim:
        Xn, lo = sim.adjoint_step(X, lam, euler_first=False)
    for a, b in zip(Xn, adj.step(X, False)):
        assert rel_l2(a, b) <= 1e-12, rel_l2(a, b)
    for a, b in zip(lo, adj.step_T(X, False, lam)):
        assert rel_l2(a, b) <= 1e-11, rel_l2(a, b)
