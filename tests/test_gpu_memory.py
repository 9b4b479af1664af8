"""Device memory that a handle can do without: it is created and runs where that part does not fit, with the same results, and gives
back what it keeps unused before a later call fails."""
from __future__ import annotations

import gc

import numpy as np
import pytest

from qgybj import Simulation
from qgybj._lib import check, lib, ptr
from qgybj.config import CONFIGS, dealias_mask, make_initial_condition, model_parameters, scaled
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


class _Leave:
    """Device memory taken so that `free` bytes are left."""

    def __init__(self, free):
        import torch
        self.held = torch.empty(_free() - free, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *a):
        import torch
        del self.held
        torch.cuda.empty_cache()


def _free():
    import torch
    gc.collect()               # (handles that an earlier test left to it)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("precision,size,tol", [("fp64", 16, 1e-12), ("mixed", 8, 1e-5)])
def test_a_handle_without_the_memory_it_can_do_without(precision, size, tol):
    """The kept y-inverse planes of B, the solves' forward values and their per-column factors."""
    import torch
    torch.zeros(1, device="cuda")
    n, n3 = 256, 128
    rc = scaled(CONFIGS["c1"], n, n3)
    ic = make_initial_condition(rc)
    params = model_parameters(rc, ic.delt)

    def run(sim):
        for f in ("psi", "BR", "BI"):
            sim.set_state(f, getattr(ic, f))
        sim.init_state(True, True)
        sim.steps_async(3, True)
        sim.synchronize()
        return [sim.get_state(f) for f in ("q", "psi", "BR", "BI", "AR", "AI")]

    with Simulation(params, precision) as sim:      # (loads the kernels)
        want = run(sim)
    free = _free()
    with Simulation(params, precision) as sim:
        used = free - _free()
    KX, KXP = 85, 88
    planes = n3 * 2 * n * KXP * size
    forward = 6 * n3 * (2 * KX - 1) * KXP * 8
    factors = 6 * n3 * int(dealias_mask(n).sum()) * 8
    room = _Leave(used - forward - factors - planes // 2)
    with room:
        sim = Simulation(params, precision)
    with sim:
        got = run(sim)
    assert all(rel_l2(a, b) <= tol for a, b in zip(got, want))


def test_the_unused_copy_of_psi_makes_room():
    import torch
    n, n3 = 512, 64
    rc = scaled(CONFIGS["c1"], n, n3)
    ic = make_initial_condition(rc)
    params = model_parameters(rc, ic.delt)
    out = torch.empty((n3, n, n), dtype=torch.float32, device="cuda")
    psi = torch.from_numpy(ic.psi).cuda()
    torch.cuda.synchronize()
    with Simulation(params, "mixed") as sim:
        def dump():
            check(lib().qg_dump_psi(sim.h, ptr(out), 0, n3, 1.0, 1.0), sim.h)
            return out.cpu().numpy()
        sim.set_state("psi", psi)
        sim.init_state(True, True)
        planes = 6 * n3 * n * ((n // 2 + 1 + 7) // 8 * 8) * 8        # of the transforms, 415 MB
        copy = n3 * 341 * 176 * 16                                    # of the FP64 psi, 61 MB
        with _Leave(planes - copy // 2):
            a = dump()
        # and it comes back with the next psi
        sim.set_state("psi", psi)
        sim.init_state(True, True)
        assert np.array_equal(a, dump())
