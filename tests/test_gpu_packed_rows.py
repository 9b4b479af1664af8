"""The FP64 transforms carry two real rows in one complex transform.  Each row keeps the precision of its own scale, whatever the
other one holds, and no spectrum of one leaves the integers' range.

Tolerances: the bound of one 2D transform derived in test_gpu_fixed_point.py (2^-51.8 of a result's norm) applies to each row by
itself; a masked product adds two more transforms and its own roundings (2^-49)."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.fft as sfft

from oracle import qgybj_oracle as orc
from qgybj import Simulation
from qgybj.config import CONFIGS, dealias_mask, scaled
from tests.helpers import oracle_for, random_masked, rel_l2
from tests.test_gpu_fixed_point import _realit, _spectrum

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -51.8


def _sim(n, **kw):
    return Simulation(dict(n1=n, n2=n, n3=2, dz=0.5, Bu=1.0, Ro=0.1, W2F=1.0, delt=1e-3, gamma=1e-3, a_ell_ut=np.ones(2), **kw),
                      "fp64")


def _noise(n, seed):
    """A physical row set with a k^-2 spectrum in x, independent from row to row, and no mean."""
    rng = np.random.default_rng(seed)
    k = np.arange(n // 2 + 1)
    z = (rng.standard_normal((n, n // 2 + 1)) + 1j * rng.standard_normal((n, n // 2 + 1))) / (1.0 + k * k)
    z[:, 0] = 0.0
    z[:, -1] = 0.0
    return np.fft.irfft(z, n=n, axis=1) * n


def _err(got, exact):
    sc = np.abs(exact).max()
    return np.linalg.norm(((got - exact) / sc).astype(complex)) / np.linalg.norm((exact / sc).astype(complex))


@pytest.mark.parametrize("size", [1e-3, 1e-9, 1e3])
@pytest.mark.parametrize("n", [16, 64, 256, 512, 1024])
def test_a_small_row_beside_a_uniform_one(n, size):
    # the even rows uniform, the odd ones a small (large) k^-2 row without mean
    r = np.zeros((1, n, n + 2))
    r[0, 0::2, :n] = 1.0
    r[0, 1::2, :n] = size * _noise(n, 3)[1::2]
    fx = sfft.rfft(r[0, :, :n].astype(np.longdouble), norm="forward")
    with _sim(n) as sim:
        # the rows' own spectra, from the 2D ones (past kx = 0, where the uniform rows' columns are)
        got = sfft.ifft(sim.fft_r2c(r)[0].astype(np.clongdouble), axis=0, norm="forward")
        assert _err(got[1::2, 1:], fx[1::2, 1:]) <= TOL
        assert np.abs(got[0::2, 1:]).max() <= TOL
        # back: kx = 0 holds a uniform value on the even rows alone (its coefficients at ky = 0 and n/2)
        k = random_masked(n, 1, 5)
        k[..., 0] = 0.0
        k *= size
        k[0, 0, 0] = k[0, n // 2, 0] = 0.5
        ex = sfft.irfft2(k.astype(np.clongdouble), s=(n, n), norm="forward")
        got = sim.fft_c2r(k)[..., :n]
        for s in (0, 1):
            assert _err(got[:, s::2], ex[:, s::2]) <= TOL, s


@pytest.mark.parametrize("period", [32, 64, 128])
def test_square_waves_beside_zero_rows_at_1024(period):
    # amplitudes across one binade, each in its own pair of rows; such a row's spectrum is the largest that the passes of this
    # length leave (radix 8 after radix 2)
    n = 1024
    f = np.where(((np.arange(n) / period + 0.25) % 1.0) < 0.5, 1.0, -1.0)
    r = np.zeros((1, n, n + 2))
    amp = np.linspace(1.0, 2.0, n // 4, endpoint=False)
    r[0, 0::2, :n] = np.concatenate([amp, -amp])[:, None] * f
    fx = sfft.rfft2(r[..., :n].astype(np.longdouble), norm="forward")
    with _sim(n) as sim:
        assert _err(sim.fft_r2c(r), fx) <= TOL
        # and as a product of the routine-level calls, u q with q = 1 and v = 0
        k = np.fft.rfft2(r[..., :n], norm="forward")
        one, zero = np.zeros_like(k), np.zeros_like(k)
        one[0, 0, 0] = 1.0
        nq = sim.convol_waqg(k, zero, one, zero, zero)[0]
    ex = np.where(dealias_mask(n)[None], 1j * np.arange(n // 2 + 1) * fx, 0)
    assert _err(nq, ex) <= 2.0 ** -49


@pytest.mark.parametrize("n,n3", [(32, 3), (64, 4), (256, 2), (512, 2)])
def test_step_with_a_uniform_wave_and_a_small_imaginary_part(n, n3):
    """The shipped initial condition: BR uniform, BI zero or small.  Without advection, the modes of BR with k > 0 after a step
    come from zeta BI alone, whose rows are carried beside those of zeta BR, 1e9 times as large."""
    model, _, ic, params = oracle_for(scaled(CONFIGS["c4"], n, n3), linear=1)
    BI = 1e-9 * random_masked(n, n3, 7) / (1 + model.kh2f)
    BI[:, 0, 0] = 0.0
    BR = np.zeros_like(BI)
    BR[:, 0, 0] = 1.0
    st = orc.initial_state(model, ic.psi, BR, BI, apply_sumB=False)
    with Simulation(params, "fp64", flags={"linear": 1}) as sim:
        for f, a in (("psi", ic.psi), ("BR", BR), ("BI", BI)):
            sim.set_state(f, a)
        sim.init_state(False, True)
        sim.step(euler_first=True)
        got = sim.get_state("BR")
    exp = model.step_euler(st).BR.copy()
    got[:, 0, 0] = exp[:, 0, 0] = 0.0
    assert rel_l2(got, exp) <= 1e-12


@pytest.mark.parametrize("kind", ["one", "gauss", "tiny", "huge"])
@pytest.mark.parametrize("n", [512, 1024])
def test_peaked_and_scaled_spectra_at_long_lengths(n, kind):
    """A few modes, columns down to subnormal values, and the ends of the exponents' range, against 64-bit-mantissa transforms (or
    longer) at the lengths whose divisions leave the fewest bits."""
    k = _spectrum(kind, n)
    with np.errstate(over="ignore", under="ignore"), _sim(n) as sim:
        ex = sfft.irfft2(_realit(k, n).astype(np.clongdouble), s=(n, n), norm="forward")
        floor = float(n * np.longdouble(5e-324) / np.linalg.norm((ex / np.abs(ex).max()).astype(float)) / np.abs(ex).max())
        assert _err(sim.fft_c2r(k)[..., :n], ex) <= TOL + (floor if kind == "tiny" else 0)
        r = np.zeros((1, n, n + 2))
        r[..., :n] = ex.astype(float)
        fx = sfft.rfft2(r[..., :n].astype(np.longdouble), norm="forward")
        floor = float(n * np.longdouble(5e-324) / np.linalg.norm((fx / np.abs(fx).max()).astype(complex)) / np.abs(fx).max())
        assert _err(sim.fft_r2c(r), fx) <= TOL + (floor if kind == "tiny" else 0)
