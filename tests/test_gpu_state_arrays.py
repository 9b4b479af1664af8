"""State I/O through pointers of any alignment and kind: a device or page-locked array that the kernels cannot read as 16-byte
values goes through a staging copy, with the same results."""
from __future__ import annotations

import numpy as np
import pytest

from qgybj import Simulation
from qgybj._lib import FIELDS, check, lib, ptr
from qgybj.config import CONFIGS, make_initial_condition, model_parameters, scaled
from tests.helpers import random_masked

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,n3", [(16, 2), (32, 5), (64, 33), (256, 3)])
def test_state_through_every_kind_of_array(precision, n, n3):
    import torch
    rc = scaled(CONFIGS["c0"], n, n3)
    params = model_parameters(rc, make_initial_condition(rc).delt)
    a = random_masked(n, n3, 5)
    nv = a.size * 2

    def view(kind, shift):
        """nv doubles, `shift` doubles past a 16-byte boundary."""
        f = torch.full((nv + 2,), 7.0, dtype=torch.float64, pin_memory=kind == "pinned",
                       device="cuda" if kind == "device" else "cpu")
        v = f[shift:shift + nv]
        assert v.data_ptr() % 16 == 8 * shift
        return v

    with Simulation(params, precision) as sim:
        for f in ("psi", "BR", "BI"):
            sim.set_state(f, a)
        sim.init_state(True, True)
        want = {f: sim.get_state(f) for f in ("q", "psi", "AR", "CR")}
        for kind in ("device", "pinned", "pageable"):
            for shift in (0, 1):
                src = view(kind, shift)
                src.copy_(torch.from_numpy(a.view(np.float64).reshape(-1)))
                torch.cuda.synchronize()
                for f in ("psi", "BR", "BI"):
                    check(lib().qg_set_state(sim.h, FIELDS[f], ptr(src), 0, n3), sim.h)
                sim.init_state(True, True)
                for f, w in want.items():
                    out = view(kind, shift)
                    check(lib().qg_get_state(sim.h, FIELDS[f], ptr(out), 0, n3), sim.h)
                    assert np.array_equal(out.cpu().numpy().view(np.complex128).reshape(a.shape), w), (kind, shift, f)
                    # a range of levels, its ends untouched
                    part = view(kind, shift)
                    check(lib().qg_get_state(sim.h, FIELDS[f], ptr(part), 1, 1), sim.h)
                    got = part.cpu().numpy()
                    m = nv // n3
                    assert np.array_equal(got[:m].view(np.complex128).reshape(a.shape[1:]), w[1]) and (got[m:] == 7.0).all()
