"""The device functions that divide through tabulated reciprocals (step_kernels.cuh: div_by, Divisor) against the hardware's
division: the same bits over the exponents that the solves and A_z meet, for zeros of both signs, infinities and NaN; where the
quotient or the dividend is subnormal or nearly so (below 2^-969, where the residual underflows), within the last place."""
from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "qg-ybjp-model_gb300" / "csrc"


@pytest.fixture(scope="module")
def division(tmp_path_factory):
    so = tmp_path_factory.mktemp("division") / "division_check.so"
    subprocess.run([shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", str(CSRC), "-I", str(ROOT / "include"), str(ROOT / "tests" / "division_check.cu"), "-o", str(so)],
                   check=True, capture_output=True)
    L = C.CDLL(str(so))
    L.division_random.restype = C.c_longlong
    L.division_random.argtypes = [C.c_ulonglong, C.c_longlong, C.c_int, C.c_int]
    L.division_list.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 5
    return L


def _list(L, one, a, d):
    import torch
    with np.errstate(all="ignore"):
        arr = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (a, d, 1.0 / d)]
    out = [torch.empty(len(a), dtype=torch.float64, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    assert L.division_list(len(a), one, *[x.data_ptr() for x in arr + out]) == 0
    return [x.cpu().numpy() for x in out]


def _same(q, exact):
    return (q.view(np.int64) == exact.view(np.int64)) | (np.isnan(q) & np.isnan(exact))


@pytest.mark.parametrize("e0,e1", [(1003, 1043), (723, 1323), (1023, 1023)])
def test_random_quotients(division, e0, e1):
    # (2^28 of them; one lies within 2^-50 of an ulp of a midpoint with a probability below 2^-20)
    assert division.division_random(12345 + e0, 1 << 28, e0, e1) == 0


def _operands():
    big, tiny, sub = np.finfo(float).max, np.finfo(float).tiny, 5e-324
    one = 1.0 + 2.0 ** -52
    return np.array([0.0, 1.0, one, 2.0 - 2.0 ** -52, 3.0, 1e-300, 1e300, big, tiny, tiny * one, sub, 12345 * sub, tiny - sub,
                     np.inf, np.nan, 2.0 ** -969, 2.0 ** -970, 2.0 ** -1000, 1.0 / 3.0, 2.0 ** 1000])


DIVISORS = [-1.0, -0.25, -2.0 ** 40, -(2.0 - 2.0 ** -52), -(1.0 + 2.0 ** -52), -3.0, -1.7e5, -2.0, 1.0 / 3.0, 1.0 / 256, 7e-5, 1e-3]


@pytest.mark.parametrize("one", [0, 1])
@pytest.mark.parametrize("d", DIVISORS)
def test_edges(division, d, one):
    a = np.concatenate([_operands(), -_operands()])
    with np.errstate(all="ignore"):
        q, exact = _list(division, one, a, np.full_like(a, d))
    small = np.isfinite(a) & (a != 0) & ((np.abs(a) < 2.0 ** -969) | (np.abs(exact) < np.finfo(float).tiny))
    assert _same(q, exact)[~small].all(), (a[~small][~_same(q, exact)[~small]], d)
    assert (np.abs(q.view(np.int64) - exact.view(np.int64))[small] <= 1).all()
