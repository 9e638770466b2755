"""What users of this library have it do, as timed cases.

The library's work is one explicit step of a compressible flow solver: the CFL
query, two transport stages, the Peng-Robinson HEM flash of every cell after
each, and the adjoint of that step; beside it the flash is called on its own
batches. A case is one of seven kinds:

  step      SSPRK2 + HEM steps of the N2O impingement box through `Flow.step`
            (one captured graph a step), FP64 or mixed precision, HLL or HLLC,
            inviscid, viscous, WALE, with or without the WALE scalar closure
  flash     a device-resident batch of pure N2O states through `GpuHem.run_device`
  recover   the same flash on the caller's host arrays through `GpuHem.run`
  mixture   the four-species air / N2O / isopropanol flash on host arrays
  solver    one step as an existing solver drives the C ABI: host arrays in and
            out of every call (CFL query, upload, advance, download, flash)
  adjoint   HEM steps recorded with autograd and their gradient
  box       the two-species ideal-gas box (blast): steps and their gradient
  mesh      an SSPRK2 step of an ideal-gas mixture on a general (oblique) mesh
            through the device entries of the face-graph operator

Sizes are those of the repository's configurations (40^3 to 160^3 cells, batches
of 1,500 to 4,096,000 states) and odd ones between them. Inputs are made here
from the seed; the N2O states by the Peng-Robinson relations below.
"""
import ctypes as C
import functools
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
PACKAGE = "spuma_multiphysics_b200"


def _package():
    if PACKAGE not in sys.modules:
        home = ROOT / "spuma-multiphysics_b200"
        spec = importlib.util.spec_from_file_location(PACKAGE, home / "__init__.py",
                                                      submodule_search_locations=[str(home)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[PACKAGE] = module
        spec.loader.exec_module(module)
    return sys.modules[PACKAGE]


_package()
from spuma_multiphysics_b200 import _abi as A, _lib, adjoint as AD, cases as K, thermo_data as TD  # noqa: E402
from spuma_multiphysics_b200.flow import Flow  # noqa: E402
from spuma_multiphysics_b200.hem import GpuHem  # noqa: E402

DT = 1e-8                                    # the impingement case's step
VISCOUS = dict(viscosity=1.821e-5, conductivity=0.02587)
CW = 0.325
EDGE = 0.08                                  # the longest edge of the impingement box


# ------------------------------------------------------------------ the cases
def listed():
    step = dict(kind="step", precision="fp64", flux="hll", wale=True, viscous=True, prandtl=0.0)
    return [
        # the small configuration: a step is a few dozen short launches
        dict(step, name="step_40", nx=40, ny=40, nz=40, steps=8, warm=20),
        # the production configuration
        dict(step, name="step_160", nx=160, ny=160, nz=160, steps=2, warm=4),
        # the mixed form at the configuration it is checked at
        dict(step, name="step_80_mixed", nx=80, ny=80, nz=80, steps=4, warm=12, precision="mixed"),
        # a box with no round dimension, HLLC and the turbulent heat flux
        dict(step, name="step_ragged_hllc", nx=101, ny=67, nz=83, steps=4, warm=8, flux="hllc", prandtl=0.9),
        # one device batch of the standalone flash workload: saturated and single-phase states
        dict(kind="flash", name="flash_4096000", n=4096000, share=0.6, seeds="exact"),
        # a middling batch whose seeds are one fixed gas state (a first recovery)
        dict(kind="flash", name="flash_65537_fixed", n=65537, share=0.6, seeds="fixed"),
        # the smallest call: a host batch of a worker's own cells
        dict(kind="recover", name="recover_1500", n=1500, share=0.6, seeds="exact"),
        # the production gas: hot mixtures and cold N2O-rich air that condenses
        dict(kind="mixture", name="mixture_20011", n=20011),
        # an existing solver's calls on host arrays
        dict(kind="solver", name="solver_64", nx=64, ny=64, nz=64),
        # the gradient of two recorded steps of the viscous WALE case
        dict(kind="adjoint", name="adjoint_96", nx=96, ny=96, nz=96, steps=2),
        # the gradient of ten steps of the ideal-gas blast box, one checkpoint
        dict(kind="box", name="blast_64", nx=64, ny=64, nz=64, steps=10),
        # four species on a general mesh
        dict(kind="mesh", name="mesh_4_species", nx=64, ny=50, nz=48, species=4, wale=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dims(rng, lo, hi):
    """Box dimensions of about lo..hi cells, up to twice as long as wide."""
    side = _log(rng, lo, hi) ** (1 / 3)
    return tuple(max(12, int(side * 2 ** rng.uniform(-.5, .5))) for _ in range(3))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "flash", "flash", "recover", "mixture", "solver", "adjoint", "box",
                       "mesh"])
    if kind == "step":
        nx, ny, nz = _dims(rng, 20000, 1500000)
        wale = rng.random() < .7
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=4, warm=rng.randrange(2, 20),
                    precision=rng.choice(["fp64", "fp64", "mixed"]), flux=rng.choice(["hll", "hll", "hllc"]),
                    wale=wale, viscous=wale or rng.random() < .5, prandtl=rng.choice([0.0, .85]) if wale else 0.0)
    if kind in ("flash", "recover"):
        return dict(kind=kind, n=_log(rng, 300, 2500000 if kind == "flash" else 300000),
                    share=round(rng.uniform(.1, .9), 3), seeds=rng.choice(["exact", "fixed"]))
    if kind == "mixture":
        return dict(kind=kind, n=_log(rng, 250, 20000))
    if kind == "solver":
        nx, ny, nz = _dims(rng, 8000, 500000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz)
    if kind == "adjoint":
        nx, ny, nz = _dims(rng, 20000, 800000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randrange(1, 4))
    if kind == "box":
        nx, ny, nz = _dims(rng, 8000, 260000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randrange(2, 11))
    nx, ny, nz = _dims(rng, 8000, 200000)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, species=rng.randrange(1, 5), wale=rng.random() < .7)


def _cells(case):
    return case["n"] if "n" in case else case["nx"] * case["ny"] * case["nz"]


# ------------------------------------------------- Peng-Robinson N2O in torch
R = TD.GAS_CONSTANT


def _nasa(sp, T):
    """cp/R, h/RT, s/R of species sp at T (NASA9 regions)."""
    a = torch.tensor(sp["nasa9"], dtype=torch.float64, device=T.device)
    inner = torch.tensor(sp["ranges"][1:-1], dtype=torch.float64, device=T.device)
    a = a[torch.bucketize(T.detach(), inner, right=True)].movedim(-1, 0)
    i, l = 1 / T, torch.log(T)
    cp = a[0] * i * i + a[1] * i + a[2] + T * (a[3] + T * (a[4] + T * (a[5] + T * a[6])))
    h = -a[0] * i * i + a[1] * l * i + a[2] + T * (a[3] / 2 + T * (a[4] / 3 + T * (a[5] / 4 + T * a[6] / 5))) + a[7] * i
    s = -a[0] * i * i / 2 - a[1] * i + a[2] * l + T * (a[3] + T * (a[4] / 2 + T * (a[5] / 3 + T * a[6] / 4))) + a[8]
    return cp, h, s


class _Fluid:
    """One Peng-Robinson species: the properties at (T, rho), the volume roots at
    (T, p) and the saturation line."""

    def __init__(self, sp):
        self.sp, self.a, self.b, self.W = sp, sp["a"], sp["b"], sp["W"]
        self.k = TD.kappa(sp["omega"])
        self.Tc = self.a * TD.OMEGA_B / (self.b * TD.OMEGA_A * R)
        self.pc = TD.OMEGA_B * R * self.Tc / self.b
        self.omega = sp["omega"]

    def _attraction(self, T):
        root = torch.sqrt(T / self.Tc)
        f = 1 + self.k * (1 - root)
        df = -self.k / (2 * self.Tc * root)
        return self.a * f * f, 2 * self.a * f * df, 2 * self.a * (df * df - f * df / (2 * T))

    def at(self, T, rho):
        b, V = self.b, self.W / rho
        aa, da, d2a = self._attraction(T)
        den = V * V + 2 * b * V - b * b
        p = R * T / (V - b) - aa / den
        pV = -R * T / (V - b) ** 2 + 2 * aa * (V + b) / den ** 2
        pT = R / (V - b) - da / den
        L = torch.log((V + (1 + math.sqrt(2)) * b) / (V + (1 - math.sqrt(2)) * b)) / (2 * math.sqrt(2) * b)
        cp0, h0, s0 = _nasa(self.sp, T)
        e = R * T * (h0 - 1) + L * (T * da - aa)
        s = R * (s0 - torch.log(R * T / (TD.ONE_ATM * (V - b)))) + L * da
        cv = R * (cp0 - 1) + L * T * d2a
        cp = cv - T * pT * pT / pV
        g = e + p * V - T * s
        return dict(p=p, e=e / self.W, s=s / self.W, cv=cv / self.W, cp=cp / self.W, g=g, V=V, rho=rho,
                    kT=-1 / (V * pV), alpha=-pT / (V * pV))

    def root(self, T, p, gas):
        """Largest (gas) or smallest molar volume of the cubic at (T, p): the closed
        form, then Newton."""
        aa, b, v0 = self._attraction(T)[0], self.b, R * T / p
        c2, c1, c0 = b - v0, aa / p - 2 * v0 * b - 3 * b * b, b * b * v0 + b ** 3 - aa * b / p
        P, Q = c1 - c2 * c2 / 3, 2 * c2 ** 3 / 27 - c2 * c1 / 3 + c0
        disc = Q * Q / 4 + P ** 3 / 27
        r, m = torch.sqrt(torch.clamp(disc, min=0)), torch.sqrt(torch.clamp(-P / 3, min=1e-300))
        cbrt = lambda x: torch.sign(x) * x.abs() ** (1 / 3)
        theta = torch.acos(torch.clamp(-Q / (2 * m ** 3), -1, 1)) / 3
        V = torch.where(disc > 0, cbrt(r - Q / 2) - cbrt(r + Q / 2),
                        2 * m * torch.cos(theta if gas else theta + 2 * math.pi / 3)) - c2 / 3
        for _ in range(4):
            V = V - (((V + c2) * V + c1) * V + c0) / ((3 * V + 2 * c2) * V + c1)
        return V

    def tp(self, T, p, gas):
        return self.at(T, self.W / self.root(T, p, gas))

    def saturation(self, T):
        """(p, gas, liquid) where the roots' Gibbs energies agree, by Newton in p."""
        p = self.pc * torch.exp(5.373 * (1 + self.omega) * (1 - self.Tc / T))
        for _ in range(14):
            g, l = self.tp(T, p, True), self.tp(T, p, False)
            gap = g["V"] - l["V"]
            p = torch.where(gap > 1e-6 * g["V"], torch.maximum(p - (g["g"] - l["g"]) / gap, .5 * p), p)
        return p, self.tp(T, p, True), self.tp(T, p, False)


N2O = _Fluid(TD.N2O)


def _mixture_state(T, p, x, g, l):
    """The state fields of vapour quality x of the phases g and l (x 1 or 0: one phase)."""
    v = x / g["rho"] + (1 - x) / l["rho"]
    rho = 1 / v
    mg, ml = x * rho, (1 - x) * rho
    mean = lambda k: x * g[k] + (1 - x) * l[k]
    vp = -(mg / g["rho"] * g["kT"] + ml / l["rho"] * l["kT"])
    vt = mg / g["rho"] * g["alpha"] + ml / l["rho"] * l["alpha"]
    cp = mean("cp")
    cv = cp + T * vt * vt / vp / rho
    sound = torch.sqrt(-1 / (rho * rho * (vp / rho + T * (vt / rho) ** 2 / cp)))
    zero = torch.zeros_like(rho)
    return dict(p=p, T=T, rho=rho, e=mean("e"), entropy=mean("s"), soundFrozen=sound, gasMass=mg, liquidMass=ml,
                cp=cp, cv=cv, rhoGas=torch.where(mg > 0, g["rho"], zero), rhoLiquid=torch.where(ml > 0, l["rho"], zero))


def _flash_states(case, seed, device):
    """The generating states of a flash batch: `share` saturated two-phase cells (T
    uniform in 220-305 K, vapour quality uniform) and single-phase cells (p
    log-uniform in 1-80 bar, T uniform in 200-320 K, the largest root), shuffled."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    n = case["n"]
    n2 = int(round(case["share"] * n))
    u = torch.rand((3, n), generator=g, dtype=torch.float64)
    order = torch.randperm(n, generator=g).to(device)
    u = u.to(device)
    T2, x2 = 220 + 85 * u[0, :n2], u[1, :n2]
    T1, p1 = 200 + 120 * u[0, n2:], torch.exp(math.log(1e5) + math.log(80.0) * u[2, n2:])
    p2, g2, l2 = N2O.saturation(T2)
    one = N2O.tp(T1, p1, True)
    two, single = _mixture_state(T2, p2, x2, g2, l2), _mixture_state(T1, p1, torch.ones_like(T1), one, one)
    return {k: torch.cat([two[k], single[k]])[order] for k in two}, order


def _records(s, fixed):
    """THERMO_DTYPE seeds of generating states s: those states, or one gas state."""
    n = len(s["rho"])
    out = np.zeros(n, dtype=A.THERMO_DTYPE)
    host = {k: s[k].cpu().numpy() for k in ("p", "T", "rho", "liquidMass")}
    out["rho"] = host["rho"]
    if fixed:
        out["p"], out["T"] = 40e5, 293.15
    else:
        out["p"], out["T"] = host["p"], host["T"]
        out["liquidMass"][:, 0] = host["liquidMass"]
        out["activeLiquids"] = host["liquidMass"] > 0
    return out


_COLUMN = {name: A.THERMO_DTYPE.fields[name][1] // 8 for name in (
    "p", "T", "rho", "e", "entropy", "soundFrozen", "soundEquilibrium", "alphaGas", "alphaLiquid", "rhoGas",
    "rhoLiquid", "liquidMass", "gasMass", "cp", "cv")}
_PHASE = A.THERMO_DTYPE.fields["activeLiquids"][1] // 4


def _fields(states):
    """The thermo records (a uint8 tensor, or a THERMO_DTYPE array), whole and field by
    field, so that each field is compared on its own scale."""
    raw = states if isinstance(states, torch.Tensor) else torch.from_numpy(states.view(np.uint8))
    d = raw.view(torch.float64).view(-1, A.THERMO_DTYPE.itemsize // 8)
    out = {name: d[:, c] for name, c in _COLUMN.items()}
    out["record"] = d
    out["phase"] = raw.view(torch.int32).view(-1, A.THERMO_DTYPE.itemsize // 4)[:, _PHASE]
    return out


class _Held:
    """What a program keeps between calls; its handles are released with it."""

    def __init__(self, case, close=(), **kept):
        self.case, self._close = case, close
        self.__dict__.update(kept)

    def __del__(self):
        if torch.cuda.is_available():
            torch.cuda.synchronize()
        for c in self._close:
            c()


# ------------------------------------------------------- the impingement flow
@functools.lru_cache(maxsize=2)
def _impingement_mesh(nx, ny, nz):
    """The box with its two circular inlets on x = 0 and y = 0 (transmissive elsewhere)."""
    h = EDGE / max(nx, ny, nz)
    kinds = []
    for side, (fast, slow) in enumerate(((ny, nz), (ny, nz), (nx, nz), (nx, nz), (nx, ny), (nx, ny))):
        k = np.full(fast * slow, 2)
        if side in (0, 2):
            j, i = np.indices((slow, fast))
            k[(((i.ravel() + .5) * h - .006) ** 2 + ((j.ravel() + .5) * h - .5 * nz * h) ** 2) < .0025 ** 2] = 3
        kinds.append(k)
    return K.box_faces((nx, ny, nz), h, kinds)


def _impingement(case, seed):
    """The arguments of `Flow`: still N2O gas at 40 bar and 293.15 K with 1% density
    noise, liquid at 56.01325 bar in the inlets."""
    faces, volume = _impingement_mesh(case["nx"], case["ny"], case["nz"])
    n = len(volume)
    g = torch.Generator(device="cuda").manual_seed(seed)
    T0 = torch.full((1,), 293.15, dtype=torch.float64, device="cuda")
    rho0 = N2O.tp(T0, torch.full_like(T0, 40e5), True)["rho"]
    rho = rho0 * (1 + .01 * (2 * torch.rand(n, generator=g, dtype=torch.float64, device="cuda") - 1))
    gas = N2O.at(T0.expand(n), rho)
    q = torch.zeros((n, 5), dtype=torch.float64, device="cuda")
    q[:, 0], q[:, 4] = rho, rho * gas["e"]
    guess = np.zeros(n, dtype=A.THERMO_DTYPE)
    guess["p"], guess["T"], guess["rho"] = gas["p"].cpu().numpy(), 293.15, rho.cpu().numpy()
    liq = N2O.tp(T0, torch.full_like(T0, 56.01325e5), False)
    rl, el = liq["rho"].item(), liq["e"].item()
    fixed_guess = np.zeros(1, dtype=A.THERMO_DTYPE)
    fixed_guess["p"], fixed_guess["T"], fixed_guess["rho"] = 56.01325e5, 293.15, rl
    fixed_guess["liquidMass"][:, 0] = rl
    fixed_guess["activeLiquids"] = 1
    return faces, volume, q.cpu().numpy(), guess, np.array([[rl, 0, 0, 0, rl * el]]), fixed_guess


def _flow(case, seed):
    options = dict(VISCOUS) if case.get("viscous", True) else {}
    if case.get("wale", True):
        options["wale_cw"] = CW
    if case.get("prandtl"):
        options["turbulent_prandtl"] = case["prandtl"]
    return Flow(*_impingement(case, seed), precision=case.get("precision", "fp64"), flux=case.get("flux", "hll"),
                **options)


def _prepare_step(case, seed):
    flow = _flow(case, seed)
    for _ in range(case["warm"]):
        flow.step(DT)
    flow.check(DT)
    start = [t.clone() for t in (flow.qn, flow.sn, flow.tr)]
    return _Held(case, close=(flow.close,), flow=flow, start=start)


def _run_step(s):
    """`steps` steps from the state in hand (so every pass does the same work)."""
    flow = s.flow
    with torch.cuda.stream(flow.stream):
        for dst, src in zip((flow.qn, flow.sn, flow.tr), s.start):
            dst.copy_(src)
    for _ in range(s.case["steps"]):
        flow.step(DT)
    return {"q": flow.qn, "state": _fields(flow.sn), "transport": flow.tr, "ledger": flow.boundary,
            "cfl": flow.dt_cfl, "success": flow.success_stages}


def _prepare_adjoint(case, seed):
    flow = _flow(case, seed)
    for _ in range(4):
        flow.step(DT)
    flow.check(DT)
    stepper = AD.HemStep(flow)
    q0 = flow.qn.clone()
    torch.cuda.synchronize()
    s0 = stepper.recover(q0, flow.sn)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    weight = torch.randn(q0.shape, generator=g, dtype=torch.float64, device="cuda")
    weight[:, flow.cells:] = 0
    return _Held(case, close=(flow.close,), stepper=stepper, q0=q0, s0=s0, weight=weight)


def _run_adjoint(s):
    q0 = s.q0.detach().requires_grad_(True)
    q, state = AD.hem_rollout(s.stepper, q0, s.s0, s.case["steps"], DT, s.case["steps"])
    (grad,) = torch.autograd.grad(q, q0, s.weight)
    return {"q": q.detach(), "state": _fields(state), "gradient": grad}


# ------------------------------------------------- a solver on the host entries
def _prepare_solver(case, seed):
    lib = _lib.load()
    faces, volume, q0, guess, fixed_q, fixed_guess = _impingement(case, seed)
    n = len(volume)
    hem = GpuHem(capacity=n)
    e0 = lambda q: np.ascontiguousarray(q[:, 4] - .5 * (q[:, 1:4] ** 2).sum(1) / q[:, 0])
    hem.run(np.ascontiguousarray(q0[:, 0]), e0(q0), guess)
    hem.run(np.ascontiguousarray(fixed_q[:, 0]), e0(fixed_q), fixed_guess)
    fixed_tr = np.zeros(1, dtype=A.STATE_DTYPE)
    assert lib.reactive_b200_host_transport_states_v3(fixed_guess.ctypes.data, 1, None, 0, 1, fixed_tr.ctypes.data,
                                                      None) == 0
    cfg = A.Config(n, 1, 5, len(faces), 1, VISCOUS["viscosity"], VISCOUS["conductivity"], 0.0, 1.1, 1.6e11, 0)
    opts = A.OptionsV2(1, C.sizeof(A.OptionsV2), 256, 0, b"0" * 64)
    err = C.create_string_buffer(2048)
    h = lib.reactive_transport_create_v2(1, C.byref(cfg), C.byref(opts), A.dptr(volume),
                                         faces.ctypes.data_as(C.POINTER(A.Face)), A.dptr(fixed_q),
                                         fixed_tr.ctypes.data_as(C.POINTER(A.State)), None, None, err, len(err))
    assert h, err.value
    h = C.c_void_p(h)
    wale = A.WaleOptions(1, C.sizeof(A.WaleOptions), CW)
    assert lib.reactive_transport_set_wale_v1(h, C.byref(wale)) == 0
    pins = []

    def pinned(like):
        t = torch.empty(like.nbytes, dtype=torch.uint8, pin_memory=True)
        pins.append(t)
        out = t.numpy().view(like.dtype).reshape(like.shape)
        out[...] = like
        return out

    return _Held(case, close=(hem.close, lambda: lib.reactive_transport_destroy(h)), lib=lib, t=h, hem=hem, n=n,
                 pins=pins, q0=pinned(q0), start=pinned(guess), q=pinned(q0), states=pinned(guess),
                 seeds=pinned(guess), tr=pinned(np.zeros(n, dtype=A.STATE_DTYPE)), prim=pinned(np.zeros((n, 4))),
                 rho=pinned(np.zeros(n)), e=pinned(np.zeros(n)), ok=pinned(np.zeros(n, dtype=np.int32)),
                 version=0, attempt=0)


def _run_solver(s):
    """One step: the step-start arrays stay as they are, the results go to the others."""
    lib, t, n = s.lib, s.t, s.n
    dt = C.c_double()

    def check(rc):
        if rc:
            raise RuntimeError(lib.reactive_transport_error(t).decode())

    def query(states, q):
        check(lib.reactive_b200_host_transport_states_v3(states.ctypes.data, n, A.dptr(q), 5, 1, s.tr.ctypes.data,
                                                         s.prim.ctypes.data))
        check(lib.reactive_transport_stable_step_primitives(
            t, s.prim.ctypes.data_as(C.POINTER(A.Primitive)), s.tr.ctypes.data_as(C.POINTER(A.State)), .5, DT,
            C.byref(dt)))
        return dt.value

    steps = [query(s.start, s.q0)]
    s.attempt += 1
    check(lib.reactive_transport_begin_attempt(t, b"0" * 64, s.attempt))
    s.version += 1
    check(lib.reactive_transport_upload_conserved(t, A.dptr(s.q0), s.version))
    ledger = np.zeros((2, 5))
    for stage, out in enumerate((s.seeds, s.states)):
        check(lib.reactive_b200_host_copy_v3(out.ctypes.data, s.start.ctypes.data, out.nbytes))
        before = A.Token(s.attempt, stage, s.version)
        s.version += 1
        after = A.Token(s.attempt, stage + 1, s.version)
        check(lib.reactive_transport_advance_resident_v2(t, before, after, s.tr.ctypes.data_as(C.POINTER(A.State)),
                                                         None, None, None, DT, A.dptr(ledger[stage])))
        check(lib.reactive_transport_download_conserved(t, after, A.dptr(s.q)))
        check(lib.reactive_b200_host_recovery_inputs_v3(A.dptr(s.q), n, 5, 1, A.dptr(s.rho), A.dptr(s.e)))
        s.hem.run(s.rho, s.e, out, s.ok)
        if stage == 0:
            steps.append(query(out, s.q))
    check(lib.reactive_transport_end_attempt(t, s.attempt, 1))
    return {"q": s.q, "state": _fields(s.states), "ledger": ledger, "cfl": steps, "success": s.ok}


# ------------------------------------------------------------------- the flash
def _prepare_flash(case, seed):
    s, _ = _flash_states(case, seed, "cuda")
    n = case["n"]
    cons = torch.zeros((5, n), dtype=torch.float64, device="cuda")
    cons[0], cons[4] = s["rho"], s["rho"] * s["e"]
    seeds = torch.from_numpy(_records(s, case["seeds"] == "fixed").view(np.uint8)).cuda()
    # a moving fluid: the recovery removes the kinetic energy
    g = torch.Generator(device="cuda").manual_seed(seed + 7)
    cons[1:4] = cons[0] * 20 * torch.randn((3, n), generator=g, dtype=torch.float64, device="cuda")
    cons[4] += .5 * (cons[1:4] ** 2).sum(0) / cons[0]
    return _Held(case, hem=GpuHem(capacity=n), cons=cons, seeds=seeds, out=seeds.clone(),
                 tr=torch.zeros((n, 7), dtype=torch.float64, device="cuda"),
                 ok=torch.zeros(n, dtype=torch.int32, device="cuda"))


def _run_flash(s):
    n = s.case["n"]
    s.hem.run_device(s.cons, n, n, 5, s.seeds, s.out, s.tr, s.ok, torch.cuda.current_stream().cuda_stream)
    return {"state": _fields(s.out), "transport": s.tr, "success": s.ok}


def _prepare_recover(case, seed):
    s, _ = _flash_states(case, seed, "cuda")
    host = lambda t: np.ascontiguousarray(t.cpu().numpy())
    return _Held(case, hem=GpuHem(capacity=case["n"]), q=host(s["rho"]), e=host(s["rho"] * s["e"]),
                 seeds=_records(s, case["seeds"] == "fixed"))


def _run_recover(s):
    out = s.seeds.copy()
    ok, _ = s.hem.run(s.q, s.e, out)
    return {"state": _fields(out), "success": ok}


def _prepare_mixture(case, seed):
    """Half hot mixtures of all four species (all gas), half cold N2O-rich air (some
    condenses), each state at its own (T, p, Y) on the gas root."""
    n = case["n"]
    lib = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(seed)
    m = 2 * n + 64
    rand = lambda *shape: torch.rand(shape, generator=g, dtype=torch.float64, device="cuda")
    hot = torch.arange(m, device="cuda") % 2 == 0
    Y = -torch.log(rand(m, 4))
    air = 1 - (.6 + .38 * rand(m))
    cold = torch.stack([.767 * air, .233 * air, 1 - air, torch.zeros_like(air)], 1)
    Y = torch.where(hot[:, None], Y / Y.sum(1, keepdim=True), cold)
    T = torch.where(hot, 330 + 570 * rand(m), 230 + 70 * rand(m))
    u = rand(m)
    p = torch.where(hot, torch.exp(math.log(1e5) + math.log(200.0) * u), 5e5 + 4.5e6 * u)
    model = TD.production_model(analytic_jacobian=0)
    table = torch.frombuffer(bytearray(C.string_at(C.addressof(model.phase[0]), C.sizeof(A.Table))),
                             dtype=torch.uint8).cuda()
    out = torch.zeros((m, 19), dtype=torch.float64, device="cuda")
    status, phase = (torch.full((m,), -9, dtype=torch.int32, device="cuda") for _ in range(2))
    err = C.create_string_buffer(512)
    assert lib.reactive_b200_mixture_properties_v3(
        table.data_ptr(), m, T.data_ptr(), p.data_ptr(), Y.contiguous().data_ptr(), 1, 1, out.data_ptr(),
        status.data_ptr(), phase.data_ptr(), torch.cuda.current_stream().cuda_stream, err, len(err)) == 0, err.value
    torch.cuda.synchronize()
    keep = torch.nonzero(status == 0)[:, 0][:n]
    assert len(keep) == n
    rho, e = out[keep, 4], out[keep, 5]
    guess = np.zeros(n, dtype=A.THERMO_DTYPE)
    guess["p"], guess["T"], guess["rho"] = p[keep].cpu().numpy(), T[keep].cpu().numpy(), rho.cpu().numpy()
    return _Held(case, hem=GpuHem(model=TD.model_bytes(model), capacity=n),
                 q=np.ascontiguousarray((rho[:, None] * Y[keep]).cpu().numpy()),
                 e=np.ascontiguousarray((rho * e).cpu().numpy()), seeds=guess)


# ---------------------------------------------------------- ideal-gas mixtures
@functools.lru_cache(maxsize=2)
def _blast_mesh(nx, ny, nz):
    return K.box_faces((nx, ny, nz), 1e-3)


def _ideal_energy(species, T):
    """(e, cv, r) of each species at T, stacked."""
    e, cv, r = [], [], []
    for sp in species:
        cp, h, _ = _nasa(sp, T)
        rk = R / sp["W"]
        e.append(rk * T * (h - 1))
        cv.append(rk * (cp - 1))
        r.append(torch.full_like(T, rk))
    return torch.stack(e), torch.stack(cv), torch.stack(r)


def _blast_state(case, seed, device):
    """q (6, cells) of a sphere of N2O at 10 bar in N2 at 1 bar, 300 K, with 0.5%
    density noise, and the step (0.3 of an acoustic CFL step)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    g = torch.Generator(device="cpu").manual_seed(seed)
    noise = torch.rand(nx * ny * nz, generator=g, dtype=torch.float64).to(device)
    k, j, i = torch.meshgrid(*(torch.arange(d, device=device, dtype=torch.float64) for d in (nz, ny, nx)),
                             indexing="ij")
    r2 = (i + .5 - nx / 2) ** 2 + (j + .5 - ny / 2) ** 2 + (k + .5 - nz / 2) ** 2
    inside = (r2 < (.25 * min(nx, ny, nz)) ** 2).reshape(-1)
    ri, ro = R / TD.N2O["W"], R / TD.N2["W"]
    rho = torch.where(inside, 10e5 / (ri * 300), 1e5 / (ro * 300)) * (1 + .005 * (2 * noise - 1))
    T = torch.where(inside, 10e5 / (rho * ri), 1e5 / (rho * ro))
    e, _, _ = _ideal_energy((TD.N2O, TD.N2), T)
    zero = torch.zeros_like(rho)
    q = torch.stack([torch.where(inside, rho, zero), torch.where(inside, zero, rho), zero, zero, zero,
                     rho * torch.where(inside, e[0], e[1])])
    return q, .3 * .5 * 1e-3 / (3 * 1.1 * 370)


def _blast_weight(case, seed, device):
    g = torch.Generator(device="cpu").manual_seed(seed + 1)
    return torch.randn((6, _cells(case)), generator=g, dtype=torch.float64).to(device)


def _prepare_box(case, seed):
    faces, volume = _blast_mesh(case["nx"], case["ny"], case["nz"])
    box = AD.IdealGasBox(faces, volume, (TD.N2O, TD.N2))
    q0, dt = _blast_state(case, seed, "cuda")
    return _Held(case, close=(box.close,), box=box, q0=q0, dt=dt, weight=_blast_weight(case, seed, "cuda"))


def _run_box(s):
    q0 = s.q0.detach().requires_grad_(True)
    q = AD.rollout(s.box, q0, s.case["steps"], s.dt, 10)
    (grad,) = torch.autograd.grad(q, q0, s.weight)
    return {"q": q.detach(), "gradient": grad}


# ------------------------------------------------------------ a general mesh
MESH_SPECIES = (TD.N2, TD.O2, TD.N2O, TD.IC3H7OH)


@functools.lru_cache(maxsize=2)
def _general_mesh(nx, ny, nz):
    """A hexahedral mesh with oblique face normals, stretched faces and unequal cells:
    fixed states on -x, transmissive +x, slip walls in y, transmissive in z."""
    faces, volume = K.box_faces((nx, ny, nz), 1e-3, (3, 2, 1, 1, 2, 2))
    faces = faces.copy()
    rng = np.random.default_rng(17)
    n = faces["normal"] + .05 * rng.normal(size=faces["normal"].shape)
    faces["normal"] = n / np.linalg.norm(n, axis=1)[:, None]
    faces["area"] *= rng.uniform(.9, 1.1, len(faces))
    faces["distance"] *= rng.uniform(.9, 1.1, len(faces))
    inner = faces["kind"] == 0
    faces["ownerWeight"][inner] = rng.uniform(.45, .55, int(inner.sum()))
    return faces, volume * rng.uniform(.9, 1.1, len(volume))


def _mesh_state(case, seed, device):
    """q (ns + 4, cells + 1): gas at about 1 bar and 320 K moving at about 20 m/s; the
    last column is the inflow state."""
    n, ns = _cells(case) + 1, case["species"]
    g = torch.Generator(device="cpu").manual_seed(seed)
    u = torch.rand((2 + ns, n), generator=g, dtype=torch.float64).to(device)
    v = torch.randn((3, n), generator=g, dtype=torch.float64).to(device)
    T = 310 + 20 * u[0]
    Y = .2 + u[2:]
    Y = Y / Y.sum(0)
    e, _, r = _ideal_energy(MESH_SPECIES[:ns], T)
    rho = 1e5 * (.95 + .1 * u[1]) / ((Y * r).sum(0) * T)
    m = 20 * v * rho
    return torch.cat([Y * rho, m, ((Y * e).sum(0) * rho + .5 * (m * m).sum(0) / rho)[None]])


MESH_DT = 1e-7


def _prepare_mesh(case, seed):
    lib = _lib.load()
    faces, volume = _general_mesh(case["nx"], case["ny"], case["nz"])
    n, ns = len(volume), case["species"]
    nv = ns + 4
    q = _mesh_state(case, seed, "cuda")
    err = C.create_string_buffer(2048)
    table = TD.gas_table(MESH_SPECIES[:ns])
    gas = lib.reactive_ideal_gas_create_v3(table, len(table), 200.0, 1400.0, 1e-13, err, len(err))
    assert gas, err.value
    gas = C.c_void_p(gas)
    fixed = torch.zeros((1, 7), dtype=torch.float64, device="cuda")
    seed_T, T = (torch.full((n + 1,), 300.0, dtype=torch.float64, device="cuda") for _ in range(2))
    fq = q[:, n:].contiguous()
    assert lib.reactive_ideal_gas_run_device_v3(gas, fq.data_ptr(), 1, 1, nv, seed_T.data_ptr(), T.data_ptr(),
                                                fixed.data_ptr(), None, 0, err, len(err)) == 0
    torch.cuda.synchronize()
    cfg = A.Config(n, ns, nv, len(faces), 1, VISCOUS["viscosity"], VISCOUS["conductivity"], 0.0, 1.1, 1.6e11, 0)
    fixed_q = np.ascontiguousarray(fq.T.cpu().numpy())
    fixed_tr = fixed.cpu().numpy().view(A.STATE_DTYPE)
    h = lib.reactive_transport_create(1, C.byref(cfg), A.dptr(volume), faces.ctypes.data_as(C.POINTER(A.Face)),
                                      A.dptr(fixed_q), fixed_tr.ctypes.data_as(C.POINTER(A.State)), None, None, err,
                                      len(err))
    assert h, err.value
    h = C.c_void_p(h)
    if case["wale"]:
        wale = A.WaleOptions(1, C.sizeof(A.WaleOptions), CW)
        assert lib.reactive_transport_set_wale_v1(h, C.byref(wale)) == 0
    return _Held(case, close=(lambda: lib.reactive_transport_destroy(h), lambda: lib.reactive_ideal_gas_destroy_v3(gas)),
                 lib=lib, t=h, gas=gas, n=n, nv=nv, q0=q, qn=q.clone(), q1=q.clone(), tr=torch.cat([fixed] * (n + 1)),
                 seed_T=seed_T, T=T, ok=torch.zeros(n, dtype=torch.int32, device="cuda"), err=err,
                 boundary=torch.zeros((2, nv), dtype=torch.float64, device="cuda"),
                 cfl=torch.zeros(2, dtype=torch.float64, device="cuda"))


def _run_mesh(s):
    lib, stream = s.lib, torch.cuda.current_stream().cuda_stream
    s.qn.copy_(s.q0)
    for stage, (src, dst) in enumerate(((s.qn, s.q1), (s.q1, s.qn))):
        rc = lib.reactive_ideal_gas_run_device_v3(s.gas, src.data_ptr(), s.n + 1, s.n, s.nv, s.seed_T.data_ptr(),
                                                  s.T.data_ptr(), s.tr.data_ptr(), s.ok.data_ptr(), stream, s.err,
                                                  len(s.err))
        rc = rc or lib.reactive_transport_stage_cfl_device_v3(
            s.t, src.data_ptr(), dst.data_ptr(), s.tr.data_ptr(), MESH_DT, stage, s.boundary[stage].data_ptr(), .5,
            1.0, s.cfl[stage:].data_ptr(), stream)
        if rc:
            raise RuntimeError(s.err.value.decode() or lib.reactive_transport_error(s.t).decode())
    return {"q": s.qn, "stage": s.q1, "transport": s.tr, "ledger": s.boundary, "cfl": s.cfl, "success": s.ok}


_PREPARE = dict(step=_prepare_step, adjoint=_prepare_adjoint, solver=_prepare_solver, flash=_prepare_flash,
                recover=_prepare_recover, mixture=_prepare_mixture, box=_prepare_box, mesh=_prepare_mesh)
_RUN = dict(step=_run_step, adjoint=_run_adjoint, solver=_run_solver, flash=_run_flash, recover=_run_recover,
            mixture=_run_recover, box=_run_box, mesh=_run_mesh)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state.case["kind"]](state)


# ------------------------------------------------------------------- the work
def work(case):
    """Bytes: a step moves 504 B a cell (two stages and two recoveries, each reading
    its inputs and writing its results once; 472 inviscid), a flash its 40 B row, the
    24 B of the seed it starts from and the 176 + 56 + 4 B it returns (host batches:
    two doubles and the record in, record and flag out), a gradient the forward and
    the adjoint state of both stages again. Operations: about 200 a face and 3 faces
    a cell and stage (twice that for the reverse pass); a single-phase recovery needs
    two (T, rho) evaluations of about 150, a two-phase one about five
    iterations of two phases."""
    n, kind = _cells(case), case["kind"]
    stage, recover, saturated = 600.0, 300.0, 2500.0
    if kind == "step":
        bytes_ = 504 if case["viscous"] or case["wale"] else 472
        return {"bytes": bytes_ * n * case["steps"], "flops": 2 * (stage + recover) * n * case["steps"]}
    if kind in ("flash", "recover"):
        size = 300 if kind == "flash" else 16 + 176 + 176 + 4
        return {"bytes": size * n, "flops": (case["share"] * saturated + (1 - case["share"]) * recover) * n}
    if kind == "mixture":
        return {"bytes": (40 + 176 + 176 + 4) * n, "flops": 4 * saturated * n}
    if kind == "solver":
        # the step's own arrays between host and device: q up once and down twice, the
        # transport states of both queries, two flash batches
        return {"bytes": (504 + 3 * 40 + 2 * 56 + 2 * (16 + 2 * 176 + 4)) * n, "flops": 2 * (stage + recover) * n}
    if kind == "adjoint":
        return {"bytes": 3 * 504 * n * case["steps"], "flops": 4 * 2 * (stage + recover) * n * case["steps"]}
    nv = 6 if kind == "box" else case["species"] + 4
    closure, states = 120.0 * (nv - 4), 2 * 48 + 2 * 32
    if kind == "box":
        return {"bytes": 3 * (8 * 5 * nv + states) * n * case["steps"],
                "flops": 4 * 2 * (300 + closure) * n * case["steps"]}
    return {"bytes": (2 * 3 * 80 + 8 * 5 * nv + states) * n, "flops": 2 * (stage + 60 * nv + closure) * n}


def tolerance(case):
    """What another correct form of the same precision shows. The recovery stops at
    volume and energy residuals of 1e-9 (mixture: the chemical one at 1e-7), which
    bounds the states two orders of the same sums reach; transport and closures are 64-bit sums
    (1e-13 a step); the mixed form's faces are FP32, whose rounding enters the state
    through dt / V. Cells within rounding of a phase boundary can change their label."""
    kind = case["kind"]
    if kind in ("box", "mesh"):
        return {"rel": 1e-10, "max": 1e-7, "differ": 0.0}
    if kind == "step" and case["precision"] == "mixed":
        return {"rel": 4e-7, "max": 1e-3, "differ": 1e-5}
    if kind == "adjoint":
        return {"rel": 1e-7, "max": 1e-3, "differ": 1e-5}
    if kind == "mixture":
        return {"rel": 1e-7, "max": 1e-4, "differ": 1e-4}
    return {"rel": 1e-8, "max": 1e-3, "differ": 1e-5}


# ------------------------------------------------------------- 64-bit results
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _exact_flash(case, seed):
    """The equilibrium of each cell. A saturated cell is its generating state; so is a
    single-phase one, unless its gas is supersaturated: then the saturated state with
    its volume and energy, by bisection in T."""
    s, order = _flash_states(case, seed, _device())
    n2 = int(round(case["share"] * case["n"]))
    Tc = N2O.Tc
    rho, e = s["rho"], s["e"]
    cold = (order >= n2) & (s["T"] < Tc - .5)
    T = s["T"][cold]
    ps = N2O.saturation(T)[0]
    gaslike = s["rho"][cold] < N2O.tp(T, ps, False)["rho"] * .999
    sub = torch.nonzero(cold)[:, 0][gaslike & (s["p"][cold] > ps)]
    if len(sub):
        v, u = 1 / rho[sub], e[sub]
        lo, hi = s["T"][sub].clone(), torch.full_like(v, Tc - .2)

        def mix(t):
            p, g, l = N2O.saturation(t)
            x = (v - 1 / l["rho"]) / (1 / g["rho"] - 1 / l["rho"])
            return p, g, l, x

        for _ in range(46):
            t = .5 * (lo + hi)
            _, g, l, x = mix(t)
            low = (x * g["e"] + (1 - x) * l["e"]) < u
            lo, hi = torch.where(low, t, lo), torch.where(low, hi, t)
        t = .5 * (lo + hi)
        p, g, l, x = mix(t)
        found = _mixture_state(t, p, x, g, l)
        for k in s:
            s[k] = s[k].clone()
            s[k][sub] = found[k]
    # a single phase below the critical temperature and above the critical density is a liquid
    dense = (order >= n2) & (s["T"] < Tc) & (rho > N2O.W / (.30740130869870383 * R * Tc / N2O.pc))
    s["gasMass"] = torch.where(dense, torch.zeros_like(rho), s["gasMass"])
    s["rhoGas"] = torch.where(dense, torch.zeros_like(rho), s["rhoGas"])
    out = dict.fromkeys(list(_COLUMN) + ["record", "phase"])
    for k in ("p", "T", "rho", "e", "entropy", "soundFrozen", "gasMass", "cp", "cv", "rhoGas"):
        out[k] = s[k]
    result = {"state": out, "success": None}
    if case["kind"] == "flash":
        result["transport"] = torch.stack([s["p"], s["T"], rho, s["cv"], s["soundFrozen"], s["gasMass"],
                                           torch.zeros_like(rho)], 1)
    return result


def _closure(species, q, T0=300.0):
    """Ideal-gas states of q: T by Newton, one more step recorded for the gradient."""
    ns = len(species)
    rho = q[:ns].sum(0)
    Y = q[:ns] / rho
    e_in = (q[ns + 3] - .5 * (q[ns:ns + 3] ** 2).sum(0) / rho) / rho
    with torch.no_grad():
        T = torch.full_like(rho, T0)
        for _ in range(12):
            e, cv, _ = _ideal_energy(species, T)
            T = T - ((Y * e).sum(0) - e_in) / (Y * cv).sum(0)
    e, cv, r = _ideal_energy(species, T)
    T = T - ((Y * e).sum(0) - e_in) / (Y * cv).sum(0).detach()
    _, cv, _ = _ideal_energy(species, T)
    cv, r = (Y * cv).sum(0), (Y * r).sum(0)
    return dict(p=rho * r * T, T=T, rho=rho, cv=cv, c=torch.sqrt((cv + r) / cv * r * T))


def _operator(faces, volume, q, s, ns, viscosity=0.0, conductivity=0.0, cw=None, wave=1.1):
    """Rate, boundary sums and CFL denominators of the finite-volume operator on any
    mesh: q (nv, cells + fixed), s its states, HLL, Green-Gauss traction, WALE."""
    dev, cells = q.device, len(volume)
    at = lambda k: torch.from_numpy(np.ascontiguousarray(faces[k])).to(dev)
    L, nb, kind, n = at("owner"), at("neighbour"), at("kind"), at("normal").T
    area, dist, w = at("area"), at("distance"), at("ownerWeight")
    Rt = torch.where(nb >= 0, nb, torch.where(kind == 3, cells + at("fixed"), L))
    inner, slip = nb >= 0, kind == 1
    V = torch.from_numpy(volume).to(dev)
    u = q[ns:ns + 3] / q[:ns].sum(0)
    uL, uR = u[:, L], u[:, Rt]
    qR = q[:, Rt]
    uR = torch.where(slip, uL - 2 * (uL * n).sum(0) * n, uR)
    mR = qR[ns:ns + 3]
    qR = torch.cat([qR[:ns], torch.where(slip, mR - 2 * (mR * n).sum(0) * n, mR), qR[ns + 3:]])
    a, b = (uL * n).sum(0), (uR * n).sum(0)
    cL, cR, pL, pR = wave * s["c"][L], wave * s["c"][Rt], s["p"][L], s["p"][Rt]
    zero = torch.zeros_like(a)
    lo = torch.minimum(zero, torch.minimum(a - cL, b - cR))
    hi = torch.maximum(zero, torch.maximum(a + cL, b + cR))
    inv = 1 / (hi - lo)
    flux = hi * (a - lo) * inv * q[:, L] + lo * (hi - b) * inv * qR
    mom = (hi * pL - lo * pR) * inv * n
    energy = (hi * pL * a - lo * pR * b) * inv
    rhoL, rhoR = s["rho"][L], s["rho"][Rt]
    mu = torch.full_like(a, viscosity)
    if viscosity > 0 or cw:
        into = lambda x, f: torch.zeros(x.shape[:-1] + (cells,), dtype=x.dtype, device=dev).index_add(-1, f, x)
        face = ((w * uL + (1 - w) * uR)[:, None] * n * area).reshape(9, -1)
        G = (into(face, L) - into(face[:, inner], nb[inner])) / V
        if cw:
            g = G.reshape(3, 3, -1)
            S, sq = .5 * (g + g.transpose(0, 1)), torch.einsum("ikc,kjc->ijc", g, g)
            eye = torch.eye(3, dtype=q.dtype, device=dev)[..., None]
            D = .5 * (sq + sq.transpose(0, 1)) - eye * (sq[0, 0] + sq[1, 1] + sq[2, 2]) / 3
            ss, dd = (S * S).sum((0, 1)), (D * D).sum((0, 1))
            nut = (cw * V ** (1 / 3)) ** 2 * dd ** 1.5 / (ss ** 2.5 + dd ** 1.25)
            mu = mu + w * rhoL * nut[L] + (1 - w) * rhoR * nut[torch.where(inner, nb, L)]
        g = torch.where(inner, w * G[:, L] + (1 - w) * G[:, torch.where(inner, nb, L)], G[:, L]).reshape(3, 3, -1)
        target = (uR - uL) / (torch.where(slip, 2.0, 1.0) * dist)
        g = g + n[None] * (target - (g * n[None]).sum(1))[:, None]
        div = g[0, 0] + g[1, 1] + g[2, 2]
        t = mu * ((g * n[None]).sum(1) + (g * n[:, None]).sum(0) - 2 / 3 * div * n)
        t = torch.where(slip, (t * n).sum(0) * n, t)
        energy = energy - (t * (w * uL + (1 - w) * uR)).sum(0)
        mom = mom - t
    energy = energy - torch.where(slip, zero, conductivity * (s["T"][Rt] - s["T"][L]) / dist)
    F = torch.cat([flux[:ns], flux[ns:ns + 3] + mom, (flux[ns + 3] + energy)[None]]) * area
    out = lambda x, f: torch.zeros((x.shape[0], cells), dtype=x.dtype, device=dev).index_add(1, f, x)
    rate = (out(F[:, inner], nb[inner]) - out(F, L)) / V
    D = torch.maximum(torch.maximum(4 * mu / (3 * rhoL), 4 * mu / (3 * rhoR)),
                      conductivity / torch.minimum(rhoL * s["cv"][L], rhoR * s["cv"][Rt]))
    speed = (torch.maximum(a.abs() + cL, b.abs() + cR) + 2 * D / dist) * area
    total = out(speed[None], L)[0] + out(speed[inner][None], nb[inner])[0]
    return rate, F[:, ~inner].sum(1), (V / total).min()


def _exact_box(case, seed):
    dev = _device()
    faces, volume = _blast_mesh(case["nx"], case["ny"], case["nz"])
    q0, dt = _blast_state(case, seed, dev)
    q0 = q0.requires_grad_(True)
    rate = lambda q: _operator(faces, volume, q, _closure((TD.N2O, TD.N2), q), 2)[0]
    q = q0
    for _ in range(case["steps"]):
        q1 = q + dt * rate(q)
        q = .5 * q + .5 * (q1 + dt * rate(q1))
    (grad,) = torch.autograd.grad(q, q0, _blast_weight(case, seed, dev))
    return {"q": q.detach(), "gradient": grad}


def _exact_mesh(case, seed):
    dev, ns = _device(), case["species"]
    faces, volume = _general_mesh(case["nx"], case["ny"], case["nz"])
    q0 = _mesh_state(case, seed, dev)
    n = len(volume)
    species = MESH_SPECIES[:ns]
    q, out, ledger, cfl = q0, [], [], []
    for stage in range(2):
        s = _closure(species, q)
        rate, boundary, step = _operator(faces, volume, q, s, ns, **VISCOUS, cw=CW if case["wale"] else None)
        new = q[:, :n] + MESH_DT * rate
        if stage:
            new = .5 * q0[:, :n] + .5 * new
        q = torch.cat([new, q0[:, n:]], 1)
        out.append(q)
        ledger.append(boundary)
        cfl.append(.5 * step)
    tr = torch.stack([s["p"], s["T"], s["rho"], s["cv"], s["c"], s["rho"], torch.zeros_like(s["p"])], 1)
    return {"q": out[1], "stage": out[0], "transport": tr, "ledger": torch.stack(ledger), "cfl": torch.stack(cfl),
            "success": None}


def exact(case, seed):
    """None for the whole steps with the HEM flash and the mixture flash: their phase
    searches in plain torch, over the warm-up steps too, take minutes; their parts
    (flash, operator, gradient) have exact results in the other kinds. None for a
    fixed seed: it leaves some compressed liquids unrecovered, which keep the seed."""
    kind = case["kind"]
    if kind in ("flash", "recover"):
        return _exact_flash(case, seed) if case["seeds"] == "exact" else None
    if kind == "box":
        return _exact_box(case, seed) if _cells(case) * case["steps"] <= 2700000 else None
    return _exact_mesh(case, seed) if kind == "mesh" else None
