"""The work that users of this framework have it do, as cases that can be timed and checked.

Every case goes through the public entry points (``qgybj.Simulation``, ``qgybj.Ensemble`` and the C-ABI that they bind) with arrays
held on the GPU, as a host program that keeps its data there does.  Kinds of case:

  run        a model run from an initial condition: psi and B uploaded, initialised, a forward Euler step, leapfrog steps, the FP64
             energy integrals and the fields read back (the whole of a short run; the benchmark's FP64 and mixed precisions)
  ensemble   members of three sizes advanced together, their fields read back
  adjoint    J and its gradient by the checkpointed reverse sweep (FP64)
  transforms the routine-level r2c and c2r of a stack of levels, for a host that keeps its own time loop
  products   the routine-level nonlinear terms (advection, refraction, wave feedback) of a stack of levels
  solvers    the routine-level vertical inversions q* -> psi and B -> A
  output     what a run writes every few steps: real-space psi and LA, vertical velocity

``exact`` restates each of them in plain torch, in 64 bits.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qg-ybjp-model_gb300"))

GAMMA = float(np.float32(1e-3))
FIELDS = ("q", "psi", "BR", "BI", "AR", "AI")


def listed():
    return [
        # the smallest runs: a parameter sweep's 64^2 x 32 members, where launches and latency count
        dict(name="run_mixed_64x32", kind="run", precision="mixed", n=64, n3=32, strat="exponential", steps=100),
        # an ordinary size with a level count that no tile divides
        dict(name="run_mixed_128x50", kind="run", precision="mixed", n=128, n3=50, strat="constant", steps=50),
        # the benchmark's mixed-precision run
        dict(name="run_mixed_512x256", kind="run", precision="mixed", n=512, n3=256, strat="exponential", steps=10),
        # the reference's own precision: its small CPU configuration ...
        dict(name="run_fp64_64x64", kind="run", precision="fp64", n=64, n3=64, strat="constant", steps=40),
        # ... the drop-in configuration of 256^2 x 128 ...
        dict(name="run_fp64_256x128", kind="run", precision="fp64", n=256, n3=128, strat="exponential", steps=4),
        # ... and the benchmark's size in FP64, the largest work here
        dict(name="run_fp64_512x256", kind="run", precision="fp64", n=512, n3=256, strat="exponential", steps=2),
        # an uneven ensemble
        dict(name="ensemble_mixed", kind="ensemble", precision="mixed", m64=6, m128=4, m256=2, steps=5),
        # the gradient of the adjoint configuration (fewer steps than its 50)
        dict(name="adjoint_fp64_128x64", kind="adjoint", precision="fp64", n=128, n3=64, strat="constant", steps=8, every=4),
        # a host's own loop: both transforms of 37 levels
        dict(name="transforms_fp64_256x37", kind="transforms", precision="fp64", n=256, nz=37),
        # the nonlinear terms of 45 levels
        dict(name="products_fp64_128x45", kind="products", precision="fp64", n=128, nz=45),
        # the vertical inversions of the 256^2 x 128 configuration
        dict(name="solvers_fp64_256x128", kind="solvers", precision="fp64", n=256, n3=128, strat="exponential"),
        # a dump of a mixed-precision run
        dict(name="output_mixed_512x60", kind="output", precision="mixed", n=512, n3=60, strat="exponential"),
    ]


def _levels(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "ensemble", "adjoint", "transforms", "products", "solvers", "output"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "ensemble":
        return dict(kind=kind, precision=precision, m64=rng.randint(1, 8), m128=rng.randint(0, 5), m256=rng.randint(0, 2),
                    steps=rng.randint(1, 6))
    n = rng.choice([32, 64, 128, 256, 512])
    if kind in ("transforms", "products"):
        return dict(kind=kind, precision=precision, n=n, nz=_levels(rng, 1, 100 if n < 512 else 40))
    strat = rng.choice(["constant", "exponential"])
    n3 = _levels(rng, 5, 200 if n < 512 else 120)
    case = dict(kind=kind, precision=precision, n=n, n3=n3, strat=strat)
    if kind == "run":
        # at most about half of the largest listed run's cell-steps
        case["steps"] = max(1, min(rng.randint(1, 60), int(6.0e7 * (1 if precision == "fp64" else 8) / (n * n * n3))))
    elif kind == "adjoint":
        case.update(precision="fp64", n=min(n, 128), n3=min(n3, 64), steps=rng.randint(1, 8), every=rng.randint(1, 4))
    return case


# ---------------------------------------------------------------------------------------------------------------- inputs
def _grid(n, dev):
    kx = torch.arange(n // 2 + 1, device=dev, dtype=torch.float64)[None, :]
    j = torch.arange(n, device=dev, dtype=torch.float64)
    ky = torch.where(j > n // 2, j - n, j)
    ky[n // 2] = 0.0
    ky = ky[:, None]
    kh2 = kx * kx + ky * ky
    thr = float(int(n / 3.0 + 0.5)) - 0.5
    mask = kh2 <= thr * thr
    mask[n // 2, :] = False
    mask[n // 2 + 1:, 0] = False
    return kx, ky, kh2, mask, int(thr)


def _profile(strat, n3):
    za = np.arange(1, n3 + 1) / n3
    return np.ones(n3) if strat == "constant" else np.exp((za - 1.0) / 0.2)


def _baroclinic(a):
    """First baroclinic mode of the discrete vertical operator with coefficients a (Neumann ends), mean square 1."""
    n3 = len(a)
    d = np.zeros(n3)
    d[:-1] -= a[:-1]
    d[1:] -= a[:-1]
    m = np.diag(d) + np.diag(a[:-1], 1) + np.diag(a[:-1], -1)
    v = np.linalg.eigh(m)[1][:, -2]
    v = v / math.sqrt(float(np.mean(v * v)))
    return v if v[0] > 0 else -v


def _c2r(k, n):
    """The reference's c2r: the kx = 0 column completed from its ky > 0 half, then unnormalised."""
    idx = torch.arange(1, n // 2, device=k.device)
    col = k[..., :, 0].clone()
    col[..., n - idx] = col[..., idx].conj()
    k = torch.cat([col[..., None], k[..., 1:]], dim=-1)
    return torch.fft.irfft2(k, s=(n, n), dim=(-2, -1), norm="forward")


def _r2c(r):
    return torch.fft.rfft2(r, dim=(-2, -1), norm="forward")


def _model(case, n, n3, strat, Ro=0.1, k0=6.0, depth=0.1):
    """Host tables of a run: profiles and scalars (the time step follows from the initial condition)."""
    n2 = _profile(strat, n3)
    return dict(n1=n, n2=n, n3=n3, dz=1.0 / n3, Bu=1.0, Ro=Ro, W2F=1.0, gamma=GAMMA, nuh2=0.0, ilap1=2, ilap2=6, nuh2w=0.0,
                ilap1w=2, ilap2w=6, nuz=0.0, a_ell_ut=1.0 / n2, r_2ut=n2), k0, depth


def _initial(par, k0, depth, seed, dev):
    """Random-phase eddies (barotropic and first baroclinic) and a surface wave, uniform plus a random-phase part; sets the
    time step and the hyperdiffusion that goes with it."""
    n, n3 = par["n1"], par["n3"]
    kx, ky, kh2, mask, K = _grid(n, dev)
    gen = torch.Generator(device="cpu").manual_seed(1000003 * int(seed) + 97 * n + n3)
    k0 = min(k0, K / 3.0)

    def phases():
        p = torch.rand((n, n // 2 + 1), generator=gen, dtype=torch.float64).to(dev) * (2 * math.pi)
        return torch.polar(torch.ones_like(p), p)

    sel = mask & (kh2 > 0)
    amp = torch.where(sel, torch.exp(-0.5 * kh2 / (k0 * k0)) / torch.sqrt(kh2.clamp(min=1.0)), torch.zeros_like(kh2))
    vert = torch.from_numpy(_baroclinic(np.asarray(par["a_ell_ut"]))).to(dev)
    psi = (amp * phases())[None] + vert[:, None, None] * (amp * phases())[None]
    z2 = (kh2 * kh2)[None] * (psi.real ** 2 + psi.imag ** 2)
    psi = psi / torch.sqrt((2.0 * z2.sum(dim=(1, 2)) - z2[:, 0, 0]).mean())
    u = _c2r(-1j * ky * psi, n)
    v = _c2r(1j * kx * psi, n)
    umax = float(torch.sqrt((u * u + v * v).max()))
    zs = (torch.arange(1, n3 + 1, device=dev, dtype=torch.float64) - 0.5) / n3
    prof = torch.exp(-((1.0 - zs) / depth) ** 2)[:, None, None]
    norm = 0.2 / math.sqrt(2.0 * float((amp * amp).sum()))
    BR = prof * (amp * phases())[None] * norm
    BI = prof * (amp * phases())[None] * norm
    BR[:, 0, 0] = prof[:, 0, 0].to(BR.dtype)
    BI[:, 0, 0] = 0.0
    # the advective limit, and at most 0.4 of the leapfrog limit of the fastest wave dispersion (2/Ro)
    delt = min(0.2 * (2 * math.pi / n) / umax, 0.2 * par["Ro"])
    nuh = 0.1 / (delt * float(K) ** 4)
    par.update(delt=delt, nuh1=nuh, nuh1w=nuh)
    return psi.contiguous(), BR.contiguous(), BI.contiguous()


def _spectra(n, nz, count, seed, dev):
    """Dense half spectra of developed fields: k^-2 tails over every retained mode."""
    kx, ky, kh2, mask, K = _grid(n, dev)
    gen = torch.Generator(device=dev).manual_seed(7919 * int(seed) + 31 * n + nz)
    amp = torch.where(mask, 1.0 / (1.0 + kh2), torch.zeros_like(kh2))
    out = []
    for _ in range(count):
        re, im = (torch.randn((nz, n, n // 2 + 1), generator=gen, device=dev, dtype=torch.float64) for _ in range(2))
        out.append((torch.complex(re, im) * amp).contiguous())
    return out


def _empty(nz, n, dev):
    return torch.empty((nz, n, n // 2 + 1), dtype=torch.complex128, device=dev)


def _inputs(case, seed, dev):
    """What prepare() and exact() start from."""
    kind = case["kind"]
    if kind == "ensemble":
        members = []
        rng = np.random.RandomState(int(seed) % (1 << 31))
        for n, n3, count in ((64, 32, case["m64"]), (128, 64, case["m128"]), (256, 128, case["m256"])):
            for _ in range(count):
                par, k0, depth = _model(case, n, n3, "exponential", Ro=float(rng.uniform(0.05, 0.2)), k0=8.0,
                                        depth=float(rng.uniform(0.05, 0.2)))
                members.append((par, _initial(par, k0, depth, int(seed) + 31 * len(members), dev)))
        return members
    if kind in ("transforms", "products"):
        n, nz = case["n"], case["nz"]
        par, k0, depth = _model(case, n, max(2, nz), "constant")
        par.update(delt=1e-3, nuh1=0.0, nuh1w=0.0)
        if kind == "transforms":
            r = _c2r(_spectra(n, nz, 1, seed, dev)[0], n)
            pad = torch.zeros((nz, n, n + 2), dtype=torch.float64, device=dev)
            pad[..., :n] = r
            return par, [pad] + _spectra(n, nz, 1, int(seed) + 1, dev)
        return par, _spectra(n, nz, 4, seed, dev)
    par, k0, depth = _model(case, case["n"], case["n3"], case["strat"])
    return par, _initial(par, k0, depth, seed, dev)


def prepare(case, seed):
    import qgybj
    dev = torch.device("cuda")
    kind = case["kind"]
    state = {"case": case}
    if kind == "ensemble":
        members = _inputs(case, seed, dev)
        torch.cuda.synchronize()
        ens = qgybj.Ensemble([p for p, _ in members], precision=case["precision"])
        groups = {}
        for m, (par, (psi, BR, BI)) in zip(ens.members, members):
            m.set_state("psi", psi)
            m.set_state("BR", BR)
            m.set_state("BI", BI)
            m.init_state(True, True)
            groups.setdefault(par["n1"], []).append(m)
        ens.step(1, euler_first=True)
        ens.synchronize()
        out = {n: torch.empty((len(ms), 4, ms[0].n3, n, n // 2 + 1), dtype=torch.complex128, device=dev) for n, ms in groups.items()}
        state.update(ens=ens, groups=groups, out=out)
        return state
    par, arrays = _inputs(case, seed, dev)
    torch.cuda.synchronize()
    # the column solves' block shape that the benchmark configurations name for 256^2 levels and more
    sim = qgybj.Simulation(par, case["precision"], solve_columns=16 if case.get("n", 0) >= 256 else 0)
    state.update(sim=sim, arrays=arrays)
    n = case["n"]
    if kind == "run":
        state["out"] = {f: _empty(case["n3"], n, dev) for f in FIELDS}
    elif kind == "adjoint":
        psi, BR, BI = arrays
        sim.set_state("psi", psi)
        sim.set_state("BR", BR)
        sim.set_state("BI", BI)
        sim.init_state(True, True)
        state["x0"] = [sim.get_state(f, out=_empty(case["n3"], n, dev)) for f in ("q", "BR", "BI")]
        state["out"] = [_empty(case["n3"], n, dev) for _ in range(3)]
    elif kind == "transforms":
        nz = case["nz"]
        state["out"] = [_empty(nz, n, dev), torch.empty((nz, n, n + 2), dtype=torch.float64, device=dev)]
    elif kind == "products":
        state["out"] = [_empty(case["nz"], n, dev) for _ in range(6)]
        # velocities as compute_velo gives them
        kx, ky, _, mask, _ = _grid(n, dev)
        psi = arrays[0]
        state["uv"] = [torch.where(mask, -1j * ky * psi, 0j).contiguous(), torch.where(mask, 1j * kx * psi, 0j).contiguous()]
    elif kind == "solvers":
        psi, BR, BI = arrays
        sim.set_state("psi", psi)
        sim.set_state("BR", BR)
        sim.set_state("BI", BI)
        sim.init_state(True, True)
        state["x0"] = [sim.get_state(f, out=_empty(case["n3"], n, dev)) for f in ("q", "BR")]
        state["out"] = [_empty(case["n3"], n, dev) for _ in range(3)]
    elif kind == "output":
        psi, BR, BI = arrays
        sim.set_state("psi", psi)
        sim.set_state("BR", BR)
        sim.set_state("BI", BI)
        sim.init_state(True, True)
        state["out"] = [torch.empty((case["n3"], n, n), dtype=torch.float32, device=dev) for _ in range(3)] + [_empty(case["n3"], n, dev)]
    torch.cuda.synchronize()
    return state


def run(state):
    import qgybj
    from qgybj._lib import check, ptr
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        state["ens"].step(case["steps"])
        state["ens"].synchronize()
        for n, ms in state["groups"].items():
            for i, m in enumerate(ms):
                for f, name in enumerate(("q", "psi", "BR", "BI")):
                    m.get_state(name, out=state["out"][n][i, f])
        return list(state["out"].values())
    sim, L = state["sim"], qgybj.lib()
    if kind == "run":
        psi, BR, BI = state["arrays"]
        sim.set_state("psi", psi)
        sim.set_state("BR", BR)
        sim.set_state("BI", BI)
        sim.init_state(True, True)
        sim.steps_async(case["steps"], euler_first=True)
        sim.synchronize()
        energy = sim.diagnostics_fp64()
        for f in FIELDS:
            sim.get_state(f, out=state["out"][f])
        return {"energy": np.array([energy[k] for k in ("wke", "wpe", "wce", "ke", "pe", "zeta2", "omegah2")]), "fields": state["out"]}
    out = state["out"]
    if kind == "adjoint":
        J = ctypes.c_double()
        check(L.qg_adjoint_run(sim.h, *[ptr(a) for a in state["x0"]], case["steps"], case["every"], 0, ctypes.byref(J),
                               *[ptr(a) for a in out]), sim.h)
        return {"J": np.array([J.value]), "gradient": out}
    if kind == "transforms":
        check(L.qg_fft_r2c(sim.h, ptr(state["arrays"][0]), ptr(out[0]), case["nz"]), sim.h)
        check(L.qg_fft_c2r(sim.h, ptr(state["arrays"][1]), ptr(out[1]), case["nz"]), sim.h)
        return out
    if kind == "products":
        psi, q, BR, BI = (ptr(a) for a in state["arrays"])
        u, v = (ptr(a) for a in state["uv"])
        check(L.qg_convol_waqg(sim.h, u, v, q, BR, BI, ptr(out[0]), ptr(out[1]), ptr(out[2]), case["nz"]), sim.h)
        check(L.qg_refraction_waqg(sim.h, BR, BI, psi, ptr(out[3]), ptr(out[4]), case["nz"]), sim.h)
        check(L.qg_compute_qw(sim.h, BR, BI, ptr(out[5]), case["nz"]), sim.h)
        return out
    if kind == "solvers":
        check(L.qg_psi_solver(sim.h, ptr(state["x0"][0]), ptr(out[0])), sim.h)
        check(L.qg_A_solver_ybj_plus(sim.h, ptr(state["x0"][1]), ptr(out[1]), ptr(out[2])), sim.h)
        return out
    n3 = case["n3"]
    check(L.qg_dump_psi(sim.h, ptr(out[0]), 0, n3, 0.1, 2.0e5), sim.h)
    check(L.qg_dump_la(sim.h, ptr(out[1]), ptr(out[2]), 0, n3, 2.5, 1), sim.h)
    check(L.qg_omega(sim.h, ptr(out[3])), sim.h)
    return out


# ------------------------------------------------------------------------------------------------------------------ work
def _retained(n):
    thr = float(int(n / 3.0 + 0.5)) - 0.5
    k = int(thr)
    return sum(2 * int(math.sqrt(thr * thr - x * x)) + 1 for x in range(1, k + 1)) + k + 1, k


def _fft_flops(n, K, columns, rows):
    """One level: `columns` column transforms of each retained kx and `rows` packed row transforms of each y (5 N log2 N)."""
    return 5.0 * n * math.log2(n) * (columns * (K + 1) + rows * n)


def work(case):
    kind = case["kind"]
    w = 8.0 if case["precision"] == "mixed" else 16.0       # bytes of a resident complex value

    def steps(n, n3, count, passes=22.0, cols=16, rows=11):
        # a step's field passes over the retained modes, its transforms, products and vertical solves
        modes, K = _retained(n)
        return count * n3 * passes * modes * w, count * n3 * (_fft_flops(n, K, cols, rows) + 14.0 * n * n + 80.0 * modes)

    def dense(n, n3, fields):
        return fields * n3 * n * (n // 2 + 1) * 16.0

    if kind == "ensemble":
        b = f = 0.0
        for n, n3, m in ((64, 32, case["m64"]), (128, 64, case["m128"]), (256, 128, case["m256"])):
            x, y = steps(n, n3, case["steps"])
            b, f = b + m * (x + dense(n, n3, 4) + 4 * _retained(n)[0] * n3 * w), f + m * y
        return {"bytes": b, "flops": f}
    n = case["n"]
    modes, K = _retained(n)
    if kind == "run":
        n3 = case["n3"]
        b, f = steps(n, n3, case["steps"])
        # inputs and initialisation, integrals, six dense fields out
        return {"bytes": b + (3 * 16.0 + 12 * w + 5 * w + 6 * w) * modes * n3 + dense(n, n3, 6), "flops": f + 100.0 * modes * n3}
    if kind == "adjoint":
        n3, s = case["n3"], case["steps"]
        # the forward sweep, one recomputation of each segment, the transposed steps at 1.55 of a step's transforms
        fwd = steps(n, n3, 2 * s - -(-s // case["every"]))
        back = steps(n, n3, s, passes=35.0, cols=28, rows=17)
        return {"bytes": fwd[0] + back[0] + 6 * modes * 16.0 * n3 + dense(n, n3, 3), "flops": fwd[1] + back[1]}
    if kind in ("transforms", "products"):
        nz = case["nz"]
        full = n // 2 + 1
        per = 5.0 * n * math.log2(n) * (full + n / 2)       # one 2D transform of real data
        if kind == "transforms":
            return {"bytes": 2 * nz * (n * (n + 2) * 8.0 + n * full * 16.0), "flops": 2 * nz * per}
        # 6 inputs (u, v, psi, q, BR, BI) and 6 outputs; 10 transforms to physical space and 10 back
        return {"bytes": (6 * modes + 6 * n * full) * nz * 16.0, "flops": nz * (20 * per + 14.0 * n * n)}
    n3 = case["n3"]
    if kind == "solvers":
        return {"bytes": 2 * modes * n3 * 16.0 + dense(n, n3, 3), "flops": 4 * 6.0 * modes * n3 + 4 * modes * n3}
    per = 5.0 * n * math.log2(n) * (K + 1 + n / 2)
    return {"bytes": 5 * modes * n3 * w + 3 * n3 * n * n * 4.0 + dense(n, n3, 1), "flops": n3 * (8 * per + 3.0 * n * n + 20.0 * modes)}


# ----------------------------------------------------------------------------------------------------------------- exact
class _Exact:
    """The reference's step in plain torch, FP64 (all operations on new tensors, so that autograd can pass through it)."""

    def __init__(self, par, dev):
        self.p, self.n, self.n3 = par, par["n1"], par["n3"]
        n, dt = self.n, par["delt"]
        self.kx, self.ky, self.kh2, self.mask, _ = _grid(n, dev)
        # integrating factors: the powers and their sum in single precision, as the reference writes them
        k4 = lambda k: torch.from_numpy(np.array([np.float32(int(abs(x)) ** 4) for x in k.reshape(-1).tolist()])).to(dev)  # noqa: E731
        s = (k4(self.kx)[None, :] + k4(self.ky)[:, None]).double()
        f = dt * (par["nuh1"] * s)
        self.e1, self.e2 = torch.exp(-f), torch.exp(-2 * f)
        self.a = [float(x) for x in par["a_ell_ut"]]
        self.dev = dev

    def m(self, x):
        return torch.where(self.mask, x, torch.zeros((), dtype=x.dtype, device=x.device))

    def solve(self, rhs, k2, scale):
        """DGTSV's elimination, one system per column (the real and imaginary parts as two real right-hand sides)."""
        a, n3 = self.a, self.n3
        live = self.mask & (self.kh2 > 0)
        k2 = torch.where(live, k2, torch.ones_like(k2))[..., None]
        out_type, rhs = rhs.dtype, torch.view_as_real(rhs)
        d = [-(a[0] + k2)] + [-((a[i] + a[i - 1]) + k2) for i in range(1, n3 - 1)] + [-(a[n3 - 2] + k2)]
        b = [scale * rhs[0]]
        for i in range(n3 - 1):
            f = a[i] / d[i]
            d[i + 1] = d[i + 1] - f * a[i]
            b.append(scale * rhs[i + 1] - f * b[i])
        x = [None] * n3
        x[n3 - 1] = b[n3 - 1] / d[n3 - 1]
        for i in range(n3 - 2, -1, -1):
            x[i] = (b[i] - a[i] * x[i + 1]) / d[i]
        return torch.where(live, torch.view_as_complex(torch.stack(x)), torch.zeros((), dtype=out_type, device=rhs.device))

    def psi(self, q):
        dz = self.p["dz"]
        return self.solve(q, self.kh2 * dz * dz, dz * dz)

    def A(self, B):
        dz = self.p["dz"]
        return self.solve(B, self.kh2 * dz * dz / 4.0, dz * dz * self.p["Bu"])

    def qw(self, BR, BI):
        n, kx, ky = self.n, self.kx, self.ky
        C = lambda x: _c2r(x, n)  # noqa: E731
        p1 = C(self.m(1j * ky * BR)) * C(self.m(1j * kx * BI)) - C(self.m(1j * kx * BR)) * C(self.m(1j * ky * BI))
        p2 = C(BR) ** 2 + C(BI) ** 2
        return self.m(_r2c(p1) - 0.25 * self.kh2 * _r2c(p2)) * self.p["Ro"] * self.p["W2F"]

    def advect(self, u, v, X):
        x = _c2r(X, self.n)
        return self.m(1j * self.kx * _r2c(u * x) + 1j * self.ky * _r2c(v * x))

    def start(self, psi, BR, BI):
        p, a, n3 = self.p, self.a, self.n3
        live = self.mask & (self.kh2 > 0)
        # the vertical mean, summed level by level from the bottom
        BR = torch.where(live, BR - sum(BR[i] for i in range(n3)) / n3, BR)
        BI = torch.where(live, BI - sum(BI[i] for i in range(n3)) / n3, BI)
        k = self.kh2 * p["dz"] * p["dz"]
        q = [a[0] * psi[1] - (a[0] + k) * psi[0]]
        for i in range(1, n3 - 1):
            q.append(a[i] * psi[i + 1] - ((a[i] + a[i - 1]) + k) * psi[i] + a[i - 1] * psi[i - 1])
        q.append(-(a[n3 - 2] + k) * psi[n3 - 1] + a[n3 - 2] * psi[n3 - 2])
        q = self.m(torch.stack(q)) / (p["dz"] * p["dz"])
        return dict(q=q, qo=q, BR=BR, BI=BI, BRo=BR, BIo=BI, psi=psi, AR=self.A(BR), AI=self.A(BI))

    def step(self, s, first):
        p = self.p
        n, kh2, dt, g = self.n, self.kh2, p["delt"], p["gamma"]
        c = 0.5 / (p["Bu"] * p["Ro"])
        u, v = _c2r(self.m(-1j * self.ky * s["psi"]), n), _c2r(self.m(1j * self.kx * s["psi"]), n)
        zeta = _c2r(self.m(-kh2 * s["psi"]), n)
        nq = self.advect(u, v, s["q"])
        tr = self.advect(u, v, s["BR"]) + c * kh2 * s["AI"] - 0.5 * self.m(_r2c(zeta * _c2r(s["BI"], n)))
        ti = self.advect(u, v, s["BI"]) - c * kh2 * s["AR"] + 0.5 * self.m(_r2c(zeta * _c2r(s["BR"], n)))
        new = {}
        for x, t in (("q", nq), ("BR", tr), ("BI", ti)):
            o = s[x + "o"]
            if first:
                new[x] = self.m((s[x] - dt * t) * self.e1)
                new[x + "o"] = s[x]
            else:
                new[x] = self.m(o * self.e2 - 2 * dt * t * self.e1)
                new[x + "o"] = self.m(s[x] + g * (o - 2 * s[x] + new[x]))
        new["psi"] = self.psi(self.m(new["q"] - self.qw(new["BR"], new["BI"])))
        new["AR"], new["AI"] = self.A(new["BR"]), self.A(new["BI"])
        return new

    def energy(self, s):
        p, n3, dz, Bu = self.p, self.n3, self.p["dz"], self.p["Bu"]
        r2 = torch.from_numpy(np.asarray(p["r_2ut"])).to(self.dev)[:, None, None]
        sq = lambda x: x.real ** 2 + x.imag ** 2  # noqa: E731
        on = self.mask.double()
        b = torch.zeros_like(s["psi"])
        b[:-1] = (s["psi"][1:] - s["psi"][:-1]) / dz
        cz = torch.zeros(s["psi"].shape, dtype=torch.float64, device=self.dev)
        for A in (s["AR"], s["AI"]):
            cz[:-1] += sq((A[1:] - A[:-1]) / dz)
        half = torch.ones_like(on)
        half[0, 0] = 0.5
        k2 = self.kh2 * on
        e = [((sq(s["BR"]) + sq(s["BI"])) * on * half).sum(), (0.5 / (r2 * Bu) * k2 * cz).sum(),
             (0.125 / (Bu * Bu) * k2 * k2 * (sq(s["AR"]) + sq(s["AI"]))).sum(), (k2 * sq(s["psi"])).sum(),
             (Bu / r2 * sq(b) * on * half).sum(), (2 * k2 * k2 * sq(s["psi"])).sum(), (2 * k2 * sq(b)).sum()]
        return np.array([float(x) / n3 for x in e])

    def omega(self, psi):
        n, n3, dz, kx, ky, kh2 = self.n, self.n3, self.p["dz"], self.kx, self.ky, self.kh2
        up = torch.cat([psi[1:], psi[-1:]])
        mid = self.m(0.5 * (up + psi))
        rz = self.m((up - psi) / dz)
        C = lambda x: _c2r(x, n)  # noqa: E731
        rhs = _r2c(2.0 * (C(1j * kx * rz) * C(-1j * ky * kh2 * mid) - C(1j * ky * rz) * C(-1j * kx * kh2 * mid)))
        live = self.mask & (kh2 > 0)
        k2 = torch.where(live, kh2, torch.ones_like(kh2)) * (dz * dz)
        d = [-(2.0 + k2 / self.a[i]) for i in range(n3 - 1)]
        b = [dz * dz * rhs[0]]
        for i in range(n3 - 2):
            f = 1.0 / d[i]
            d[i + 1] = d[i + 1] - f
            b.append(dz * dz * rhs[i + 1] - f * b[i])
        w = [None] * (n3 - 1) + [torch.zeros_like(psi[0])]
        w[n3 - 2] = b[n3 - 2] / d[n3 - 2]
        for i in range(n3 - 3, -1, -1):
            w[i] = (b[i] - w[i + 1]) / d[i]
        return torch.where(live, torch.stack(w), torch.zeros((), dtype=psi.dtype, device=self.dev))


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    kind = case["kind"]
    if kind == "ensemble":
        groups = {}
        for par, x in _inputs(case, seed, dev):
            E = _Exact(par, dev)
            s = E.start(*x)
            for i in range(case["steps"] + 1):
                s = E.step(s, i == 0)
            groups.setdefault(par["n1"], []).append(torch.stack([s[f] for f in ("q", "psi", "BR", "BI")]))
        return [torch.stack(g) for g in groups.values()]
    par, arrays = _inputs(case, seed, dev)
    E = _Exact(par, dev)
    n = case["n"]
    if kind == "transforms":
        back = torch.zeros((case["nz"], n, n + 2), dtype=torch.float64, device=dev)
        back[..., :n] = _c2r(arrays[1], n)
        return [_r2c(arrays[0][..., :n]), back]
    if kind == "products":
        psi, q, BR, BI = arrays
        u, v = _c2r(E.m(-1j * E.ky * psi), n), _c2r(E.m(1j * E.kx * psi), n)
        zeta = _c2r(E.m(-E.kh2 * psi), n)
        return [E.advect(u, v, x) for x in (q, BR, BI)] + [E.m(_r2c(zeta * _c2r(x, n))) for x in (BR, BI)] + [E.qw(BR, BI)]
    s = E.start(*arrays)
    if kind == "run":
        for i in range(case["steps"]):
            s = E.step(s, i == 0)
        return {"energy": E.energy(s), "fields": {f: s[f] for f in FIELDS}}
    if kind == "solvers":
        A = E.A(s["BR"])
        C = torch.zeros_like(A)
        C[:-1] = (A[1:] - A[:-1]) / par["dz"]
        return [E.psi(s["q"]), A, C]
    if kind == "output":
        la = [_c2r(E.m(s[b] + 0.25 * E.kh2 * s[a] / par["Bu"]), n) * 2.5 for b, a in (("BR", "AR"), ("BI", "AI"))]
        return [_c2r(s["psi"], n) * 0.1 * 2.0e5] + la + [E.omega(s["psi"])]
    x0 = [s[f].detach().clone().requires_grad_(True) for f in ("q", "BR", "BI")]
    q, BR, BI = x0
    s = dict(q=q, qo=q, BR=BR, BI=BI, BRo=BR, BIo=BI, psi=E.psi(E.m(q - E.qw(BR, BI))), AR=E.A(BR), AI=E.A(BI))
    for i in range(case["steps"]):
        s = E.step(s, i == 0)
    window = torch.zeros((case["n3"], n, n), dtype=torch.float64, device=dev)
    zs = (np.arange(case["n3"]) + 0.5) / case["n3"]
    window[int(np.argmax(zs >= 0.8)):, n // 4:3 * n // 4, n // 4:3 * n // 4] = 1.0
    J = 0.0
    for b, a in (("BR", "AR"), ("BI", "AI")):
        la = _c2r(E.m(s[b] + 0.25 * E.kh2 * s[a] / par["Bu"]), n)
        J = J + 0.5 * (window * la * la).sum()
    J.backward()
    return {"J": np.array([float(J.detach())]), "gradient": [torch.where(E.mask, x.grad, torch.zeros_like(x.grad)) for x in x0]}
