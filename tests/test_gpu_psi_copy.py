"""q = init_q(psi) comes from the psi that the handle holds, however the host set it: in parts, again after a run, on some levels
only.  The mixed path keeps an FP64 copy of what the host set; the other levels are the resident (FP32) ones."""
from __future__ import annotations

import numpy as np
import pytest

from qgybj import Ensemble, Simulation
from qgybj.config import CONFIGS, make_initial_condition, model_parameters, scaled
from tests.helpers import random_masked

pytestmark = pytest.mark.gpu


def _run(n, n3):
    rc = scaled(CONFIGS["c1"], n, n3)
    ic = make_initial_condition(rc)
    return ic, model_parameters(rc, ic.delt)


def _q(sim, psi, level0=0):
    sim.set_state("psi", psi, level0)
    sim.init_state(False, True)
    return sim.get_state("q")


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,n3,lo,nl", [(32, 7, 3, 1), (64, 9, 0, 4), (16, 2, 1, 1), (32, 33, 20, 13)])
def test_q_follows_the_resident_psi(precision, n, n3, lo, nl):
    ic, params = _run(n, n3)
    new = random_masked(n, nl, 4) / (1 + np.arange(n // 2 + 1)) ** 2
    zero = np.zeros_like(ic.psi)
    with Simulation(params, precision) as sim, Simulation(params, precision) as ref:
        # before any other psi: the rest of the field is zero
        part = zero.copy()
        part[lo:lo + nl] = new
        assert np.array_equal(_q(sim, new, lo), _q(ref, part))
        # the whole field in two parts
        sim.set_state("psi", ic.psi[lo:], lo)
        if lo:
            sim.set_state("psi", ic.psi[:lo], 0)
        sim.init_state(False, True)
        assert np.array_equal(sim.get_state("q"), _q(ref, ic.psi))
        for f in ("BR", "BI"):
            sim.set_state(f, getattr(ic, f))
        sim.init_state(True, True)
        sim.steps_async(3, True)
        sim.synchronize()
        # some levels again after a run: the others are the run's
        now = sim.get_state("psi")
        assert not np.array_equal(now, ic.psi)
        now[lo:lo + nl] = new
        assert np.array_equal(_q(sim, new, lo), _q(ref, now))
        # set, and replaced by a step's
        sim.set_state("psi", ic.psi)
        sim.step()
        now = sim.get_state("psi")
        sim.init_state(False, True)
        assert np.array_equal(sim.get_state("q"), _q(ref, now))


def test_members_of_a_stack():
    ic, params = _run(32, 6)
    new = random_masked(32, 2, 8)
    ens = Ensemble([params] * 3, precision="mixed")
    with Simulation(params, "mixed") as ref:
        for m in ens.members:
            for f in ("psi", "BR", "BI"):
                m.set_state(f, getattr(ic, f))
        for m in ens.members:
            m.init_state(True, True)
        ens.step(2, euler_first=True)
        ens.synchronize()
        now = [m.get_state("psi") for m in ens.members]
        ens.members[1].set_state("psi", new, 3)
        for k, m in enumerate(ens.members):
            m.init_state(False, True)
            want = now[k].copy()
            if k == 1:
                want[3:5] = new
            assert np.array_equal(m.get_state("q"), _q(ref, want)), k
    ens.close()
