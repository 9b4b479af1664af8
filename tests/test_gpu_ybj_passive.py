"""Regular YBJ with passive waves: neither sigma nor A is computed, and the step needs no memory for them."""
from __future__ import annotations

import pytest

from qgybj.config import CONFIGS, scaled
from tests.test_gpu_parity import compare, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-5)])
@pytest.mark.parametrize("flags", [{"ybj_plus": 0, "passive_scalar": 1}, {"ybj_plus": 0, "passive_scalar": 1, "fixed_flow": 1},
                                   {"ybj_plus": 0, "passive_scalar": 1, "no_feedback": 1}])
def test_regular_ybj_with_passive_waves(flags, precision, tol):
    rc = scaled(CONFIGS["c0"], 32, 8)
    model, st, sim = pair(rc, precision, dict(flags))
    st = model.run(st, 4, first=True)
    sim.steps_async(4, True)
    sim.synchronize()
    compare(sim, st, tol)
    sim.close()
