"""Routine-level calls on device arrays: kernels use the caller's arrays in place where they can (16-byte aligned memory of the
device), and staging copies otherwise.  Both routes and host arrays run the same kernels on the same values, so the outputs are
the same bytes; in-place transforms (the Fortran host's equivalenced arrays) give them too.  Numerics against the oracle at the
tile edges: n = 16 (one row pair per few threads) to 256, one level and several."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import qgybj_oracle as orc
from qgybj import Simulation
from qgybj._lib import check, lib, ptr
from qgybj.config import CONFIGS, make_initial_condition, model_parameters, scaled
from tests.helpers import oracle_params, random_masked, random_physical, rel_l2

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-12, "mixed": 2e-6}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,nz", [(16, 1), (32, 5), (64, 4), (128, 3), (256, 2)])
def test_device_arrays_in_place_and_staged(precision, n, nz):
    import torch
    rc = scaled(CONFIGS["c0"], n, max(nz, 4))
    params = model_parameters(rc, make_initial_condition(rc).delt)
    model = orc.Model(oracle_params(params))
    sim = Simulation(params, precision)
    L = lib()
    psi, q = random_masked(n, nz, 3), random_masked(n, nz, 4)
    BR, BI = random_masked(n, nz, 5, masked=False), random_masked(n, nz, 6, masked=False)
    uk, vk = model.compute_velo(psi)
    rp = np.zeros((nz, n, n + 2))
    rp[:, :, :n] = random_physical(n, nz, 1)

    def dev(a, shift):
        """A copy of a on the device, `shift` doubles past a 16-byte boundary (its storage is kept by the view)."""
        flat = torch.zeros(a.size * (2 if a.dtype == np.complex128 else 1) + 2, dtype=torch.float64, device="cuda")
        v = flat[shift:shift + flat.numel() - 2]
        v.copy_(torch.from_numpy(np.ascontiguousarray(a).view(np.float64).reshape(-1)))
        torch.cuda.synchronize()
        return v

    def host(v, like):
        return v.cpu().numpy().view(like.dtype).reshape(like.shape)

    def call(fn, ins, outs, shift, extra=()):
        a, o = [dev(x, shift) for x in ins], [dev(np.full_like(x, 7.0), shift) for x in outs]
        check(fn(sim.h, *[ptr(x) for x in a], *[ptr(x) for x in o], *extra), sim.h)
        return [host(v, x) for v, x in zip(o, outs)]

    spec = np.zeros((nz, n, n // 2 + 1), dtype=np.complex128)
    cases = {
        "r2c": (L.qg_fft_r2c, [rp], [spec], [sim.fft_r2c(rp)]),
        "c2r": (L.qg_fft_c2r, [BR], [rp], [sim.fft_c2r(BR)]),
        "convol": (L.qg_convol_waqg, [uk, vk, q, BR, BI], [spec] * 3, sim.convol_waqg(uk, vk, q, BR, BI)),
        "refraction": (L.qg_refraction_waqg, [BR, BI, psi], [spec] * 2, sim.refraction_waqg(BR, BI, psi)),
        "qw": (L.qg_compute_qw, [BR, BI], [spec], [sim.compute_qw(BR, BI)]),
    }
    for name, (fn, ins, outs, want) in cases.items():
        for shift in (0, 1):
            got = call(fn, ins, outs, shift, (nz,))
            assert all(np.array_equal(a, b) for a, b in zip(got, want)), (name, shift)
    exp = list(model.convol_waqg(uk, vk, q, BR, BI)) + list(model.refraction_waqg(BR, BI, psi)) + [model.compute_qw(BR, BI)]
    got = list(cases["convol"][3]) + list(cases["refraction"][3]) + list(cases["qw"][3])
    for a, b in zip(got, exp):
        assert rel_l2(a, b) < TOL[precision]
    # in place, as a host with equivalenced real and complex arrays calls them
    buf = dev(rp, 0)
    check(L.qg_fft_r2c(sim.h, ptr(buf), ptr(buf), nz), sim.h)
    assert np.array_equal(host(buf, spec), cases["r2c"][3][0])
    buf = dev(BR, 0)
    check(L.qg_fft_c2r(sim.h, ptr(buf), ptr(buf), nz), sim.h)
    assert np.array_equal(host(buf, rp), cases["c2r"][3][0])
    # an output over an input
    a = [dev(x, 0) for x in (uk, vk, q, BR, BI)]
    o = [a[2], dev(spec, 0), dev(spec, 0)]
    check(L.qg_convol_waqg(sim.h, *[ptr(x) for x in a], *[ptr(x) for x in o], nz), sim.h)
    assert np.array_equal(host(o[0], spec), cases["convol"][3][0])
    sim.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,n3", [(32, 5), (64, 33)])
def test_solvers_on_device_arrays(precision, n, n3):
    import torch
    rc = scaled(CONFIGS["c0"], n, n3)
    params = model_parameters(rc, make_initial_condition(rc).delt)
    sim = Simulation(params, precision)
    L = lib()
    b = random_masked(n, n3, 8, masked=False)
    psi, (A, C), w = sim.psi_solver(b), sim.A_solver_ybj_plus(b), sim.omega_equation(b)
    d = torch.from_numpy(b).cuda()
    o = [torch.full_like(d, 7.0) for _ in range(4)]
    torch.cuda.synchronize()
    check(L.qg_psi_solver(sim.h, ptr(d), ptr(o[0])), sim.h)
    check(L.qg_A_solver_ybj_plus(sim.h, ptr(d), ptr(o[1]), ptr(o[2])), sim.h)
    check(L.qg_omega_equation(sim.h, ptr(d), ptr(o[3])), sim.h)
    for got, want in zip(o, (psi, A, C, w)):
        assert np.array_equal(got.cpu().numpy(), want)
    # in place: the solve reads all of its input first
    check(L.qg_omega_equation(sim.h, ptr(d), ptr(d)), sim.h)
    assert np.array_equal(d.cpu().numpy(), w)
    sim.close()
