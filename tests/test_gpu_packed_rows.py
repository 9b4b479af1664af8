"""The FP64 transforms carry two real rows in one complex transform: no spectrum of one leaves the integers' range.

Tolerances: the bound of one 2D transform derived in test_gpu_fixed_point.py (2^-51.8 of a result's norm); a masked product adds two
more transforms and its own roundings (2^-49)."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.fft as sfft

from qgybj import Simulation
from qgybj.config import dealias_mask

pytestmark = pytest.mark.gpu
TOL = 2.0 ** -51.8


def _sim(n, **kw):
    return Simulation(dict(n1=n, n2=n, n3=2, dz=0.5, Bu=1.0, Ro=0.1, W2F=1.0, delt=1e-3, gamma=1e-3, a_ell_ut=np.ones(2), **kw),
                      "fp64")


def _err(got, exact):
    sc = np.abs(exact).max()
    return np.linalg.norm(((got - exact) / sc).astype(complex)) / np.linalg.norm((exact / sc).astype(complex))


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
