"""Performance cases of the time-step engine: what a program using it has it do.

Every case goes through the public entry points (``Model``, ``Ensemble`` and the
device-pointer calls of the C ABI).  A case is a plain dict:

* ``op``: ``step`` (advance the resident state), ``rates`` (one right-hand side of a
  device state), ``project`` (one pressure projection of a device state), ``fields``
  (physical fields from the host into the state and back), ``ensemble`` (one step of
  several size classes);
* ``flow``: ``les`` (rough wall below, free slip above, Smagorinsky model) or ``dns``
  (closed channel between smooth walls);
* ``n1``, ``n2``, ``n3``: resolution; ``precision``: ``fp64`` or ``mixed``;
* ``members``: independent members in one handle; ``steps`` and ``method`` of one pass;
* ``eta``: vertical stretching (0: uniform); ``flux``: constant mean flow instead of
  constant forcing.

Results of the double-precision form are returned as the engine holds them.  The
mixed form computes its transforms in single precision, so a program keeps its
results as single-precision snapshots, and so do these cases.
"""

import importlib
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "boundarylayerdynamics.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

DT = 1e-4
RE_INV = {"les": 1e-5, "dns": 1.0 / 180}
SIZE = {"les": (2 * math.pi, math.pi, 1.0), "dns": (4 * math.pi, 2 * math.pi, 2.0)}
Z0, KAPPA, CS, CENTRELINE = 1e-4, 0.4, 0.1, 18.0


def _case(name, op, flow, n1, n2, n3, precision, steps=1, members=1, method="SSPRK33", eta=0.0, flux=False):
    c = dict(op=op, flow=flow, n1=n1, n2=n2, n3=n3, precision=precision, steps=steps, members=members, method=method,
             eta=eta, flux=flux)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest simulations (tests, tutorials, parameter scans): launches and latency only
        _case("les16_step_fp64", "step", "les", 16, 16, 8, "fp64"),
        # the small LES of the benchmark, one step at a time as an interactive program or an
        # outer loop with its own time-step control makes it
        _case("les64_step_fp64", "step", "les", 64, 64, 32, "fp64"),
        # the same grid as the server advances it: ten steps per call between admissions
        _case("les64_tick_mixed", "step", "les", 64, 64, 32, "mixed", steps=10),
        # one right-hand side of a device state, as a program with its own integrator asks for it
        _case("les96_rates_fp64", "rates", "les", 96, 96, 48, "fp64"),
        # sizes that nobody tuned: neither square nor powers of two and three, stretched grid,
        # two-stage method, prescribed mass flux
        _case("les_ragged_step_fp64", "step", "les", 100, 84, 37, "fp64", steps=2, method="SSPRK22", eta=0.6, flux=True),
        # the headline workload: closed-channel DNS, both precision forms
        _case("dns192_step_fp64", "step", "dns", 192, 192, 96, "fp64", steps=2),
        _case("dns192_step_mixed", "step", "dns", 192, 192, 96, "mixed", steps=2),
        # the projection alone on a device state (an embedding program's own stages)
        _case("dns192_project_fp64", "project", "dns", 192, 192, 96, "fp64"),
        # a production LES in double precision
        _case("les256_step_fp64", "step", "les", 256, 256, 128, "fp64"),
        # the largest member of the benchmark
        _case("les512_step_mixed", "step", "les", 512, 512, 256, "mixed"),
        # the 64-member uneven ensemble: 24 x 64^2x32, 24 x 96^2x48, 16 x 128^2x64
        _case("ensemble64_step_mixed", "ensemble", "les", 64, 64, 32, "mixed", members=64),
        # initial conditions and snapshots: physical fields on the host into the state and back
        _case("fields128_fp64", "fields", "les", 128, 128, 64, "fp64"),
    ]


def _only(n, primes):
    for p in primes:
        while n % p == 0:
            n //= p
    return n == 1


def _horizontal(rng, hi, primes):
    """A resolution whose default physical size 2 kmax + 2 has these prime factors only; odd ones among them."""
    while True:
        n = int(round(math.exp(rng.uniform(math.log(16), math.log(hi)))))
        if _only(2 * ((n - 1) // 2) + 2, primes):
            return n


def draw(rng):
    op = rng.choice(["step", "step", "step", "step", "rates", "project", "fields", "ensemble"])
    flow = "les" if op == "ensemble" else rng.choice(["les", "dns"])
    precision = "fp64" if op in ("project", "fields") else rng.choice(["fp64", "mixed"])
    if op == "ensemble":   # the size classes are multiples of 64^2x32, 96^2x48, 128^2x64
        return _case("", op, flow, 64, 64, rng.randrange(16, 49), precision, members=rng.randrange(4, 65))
    # the Smagorinsky model and the host fields live on the default grid; the channel takes any size
    primes = (2, 3) if op == "fields" else (2, 3, 5, 7) if flow == "les" else tuple(range(2, 300))
    while True:
        n1, n2 = _horizontal(rng, 300, primes), _horizontal(rng, 300, primes)
        n3 = int(round(math.exp(rng.uniform(math.log(6), math.log(150)))))
        members = rng.choice([1, 1, 1, 2, 5, 12]) if op == "step" else 1
        if n1 * n2 * n3 * members <= 256 * 256 * 128:
            break
    steps = rng.choice([1, 1, 2, 5]) if op == "step" and n1 * n2 * n3 * members < 1 << 20 else 1
    return _case("", op, flow, n1, n2, n3, precision, steps=steps, members=members,
                 method=rng.choice(["SSPRK33", "SSPRK33", "SSPRK22", "Euler"]) if op == "step" else "SSPRK33",
                 eta=rng.choice([0.0, 0.0, 0.5, 0.8]), flux=rng.random() < 0.3)


# ------------------------------------------------------------------------------- inputs
def _groups(case):
    """(case of one size class, members) of an ensemble: 3/8, 3/8 and 1/4 of the members."""
    m = case["members"]
    a, b = (3 * m) // 8, (3 * m) // 8
    out = []
    for num, den, count in ((1, 1, a), (3, 2, b), (2, 1, m - a - b)):
        out.append(dict(case, op="step", n1=case["n1"] * num // den, n2=case["n2"] * num // den,
                        n3=case["n3"] * num // den, members=count))
    return out


def _mapping(case):
    """vmap and its derivative on zeta in [0, 1] (host floats)."""
    l3, eta = SIZE[case["flow"]][2], case["eta"]
    if not eta:
        return (lambda z: z * l3), (lambda z: l3)
    s, h = math.sin(eta * math.pi / 2), eta * math.pi / 2
    if case["flow"] == "dns":
        return (lambda z: l3 / 2 * (1 + math.sin((2 * z - 1) * h) / s)), (lambda z: l3 * h / s * math.cos((2 * z - 1) * h))
    return (lambda z: l3 * (1 + math.sin((z - 1) * h) / s)), (lambda z: l3 * h / s * math.cos((z - 1) * h))


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _physical(case, seed, member=0):
    """Physical fields (u, v, w) on the default grid (n3, P2, P1): log law or laminar profile plus noise."""
    n3 = case["n3"]
    P1, P2 = 2 * ((case["n1"] - 1) // 2) + 2, 2 * ((case["n2"] - 1) // 2) + 2
    vmap, _ = _mapping(case)
    dev = _device()
    g = torch.Generator(device=dev)
    g.manual_seed(seed * 1009 + member)
    zc = torch.tensor([vmap((2 * i + 1) / (2 * n3)) for i in range(n3)], dtype=torch.float64, device=dev)[:, None, None]
    zi = torch.tensor([vmap(i / n3) for i in range(1, n3)], dtype=torch.float64, device=dev)[:, None, None]

    def noise(nz):
        if case["flow"] == "les":
            return torch.rand((nz, P2, P1), dtype=torch.float64, device=dev, generator=g).mul_(0.2).sub_(0.1)
        return torch.randn((nz, P2, P1), dtype=torch.float64, device=dev, generator=g).mul_(0.05 * CENTRELINE)

    if case["flow"] == "les":
        pc, pi = torch.log(zc / Z0) / KAPPA, torch.log(zi / Z0) / KAPPA
        return noise(n3).add_(1).mul_(pc), noise(n3).mul_(pc), noise(n3 - 1).mul_(pi)
    return noise(n3).add_(CENTRELINE * (1 - (zc - 1) ** 2)), noise(n3), noise(n3 - 1)


def _spectral(q, n1, n2):
    """The resolved modes of physical layers on the default grid, (nz, 2 k2max + 1, k1max + 1)."""
    k1m, k2m = (n1 - 1) // 2, (n2 - 1) // 2
    out = torch.empty((q.shape[0], 2 * k2m + 1, k1m + 1), dtype=torch.complex128, device=q.device)
    for z in range(0, q.shape[0], 32):
        x = torch.fft.rfft2(q[z:z + 32], norm="forward")
        out[z:z + 32, :k2m + 1] = x[:, :k2m + 1, :k1m + 1]
        if k2m:
            out[z:z + 32, k2m + 1:] = x[:, x.shape[1] - k2m:, :k1m + 1]
    # real fields: the k1 = 0 column is Hermitian and its mean real
    out[:, 0, 0] = out[:, 0, 0].real.to(out.dtype)
    if k2m:
        out[:, k2m + 1:, 0] = out[:, 1:k2m + 1, 0].flip(1).conj()
    return out


def _state_fields(case, seed, member=0):
    return [_spectral(q, case["n1"], case["n2"]) for q in _physical(case, seed, member)]


class _DeviceArray:
    """A float64 array at a device address for torch (the engine owns the memory)."""

    def __init__(self, address, shape, owner):
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(address, False), version=3)
        self.owner = owner


def _views(model, base):
    """vel1, vel2, vel3 of all members in the packed device state `base` (float64, last axis re/im)."""
    n3, K2, K1, B = model.n3, model.K2, model.K1, model.members
    s = base.view(B, 3 * n3 - 1, K2, K1, 2)
    return [s[:, :n3], s[:, n3:2 * n3], s[:, 2 * n3:]]


def _resident(model):
    n = model.members * (3 * model.n3 - 1) * model.K2 * model.K1 * 2
    return torch.as_tensor(_DeviceArray(model.device_state_ptr(), (n,), model), device="cuda")


def _model(case):
    bld = importlib.import_module("BoundaryLayerDynamics")
    les = case["flow"] == "les"
    lower = bld.RoughWall(Z0, KAPPA) if les else bld.SmoothWall()
    upper = bld.FreeSlipBoundary() if les else bld.SmoothWall()
    domain = bld.Domain(SIZE[case["flow"]], lower, upper, bld.SinusoidalMapping(case["eta"]) if case["eta"] else None)
    source = dict(constant_flux=10.0) if case["flux"] else dict(constant_forcing=1.0)
    sgs = bld.StaticSmagorinskyModel(Cs=CS) if les else None
    return bld.Model((case["n1"], case["n2"], case["n3"]), domain,
                     bld.incompressible_flow(RE_INV[case["flow"]], sgs_model=sgs, **source),
                     precision=case["precision"], members=case["members"])


def _loaded(case, seed):
    """A model with its seeded state resident (before the initial projection) and the state as a tensor."""
    model = _model(case)
    base = _resident(model)
    for m in range(case["members"]):
        for v, q in zip(_views(model, base), _state_fields(case, seed, m)):
            v[m].copy_(torch.view_as_real(q))
    torch.cuda.synchronize()
    return model, base


def prepare(case, seed):
    if case["op"] == "ensemble":
        parts = [_loaded(c, seed + 17 * i) for i, c in enumerate(_groups(case))]
        ens = importlib.import_module("BoundaryLayerDynamics.ensemble").Ensemble([m for m, _ in parts])
        ens.prepare()
        return dict(case=case, ensemble=ens, bases=[b for _, b in parts])
    if case["op"] == "fields":
        host = [q.cpu().numpy() for q in _physical(case, seed)]
        return dict(case=case, model=_model(case), host=host)
    model, base = _loaded(case, seed)
    if case["op"] == "step":
        model.prepare()      # initial projection and slope, as evolve begins
        return dict(case=case, model=model, base=base)
    # the device-pointer calls are ordered on the program's own stream and buffers
    state = dict(case=case, model=model, base=base.clone(), out=torch.zeros_like(base), stream=torch.cuda.Stream())
    torch.cuda.synchronize()
    return state


# ------------------------------------------------------------------------------ one pass
def _outputs(model, base, precision):
    v = dict(zip(("vel1", "vel2", "vel3"), _views(model, base)))
    return v if precision == "fp64" else {k: q.to(torch.float32) for k, q in v.items()}


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "ensemble":
        state["ensemble"].step(case["steps"], DT, case["method"])
        return [_outputs(m, b, case["precision"]) for m, b in zip(state["ensemble"].models, state["bases"])]
    model = state["model"]
    if op == "step":
        model.step(case["steps"], DT, case["method"])
        return _outputs(model, state["base"], case["precision"])
    if op == "fields":
        for f, q in zip(("vel1", "vel2", "vel3"), state["host"]):
            model.set_field(f, q)
        return {f: model.get_field(f) for f in ("vel1", "vel2", "vel3")}
    capi = importlib.import_module("BoundaryLayerDynamics._capi")
    stream, base = state["stream"], state["base"]
    with torch.cuda.stream(stream):
        if op == "rates":
            capi.check(model._lib.bld_compute_rates_device(model._h, base.data_ptr(), state["out"].data_ptr(),
                                                           stream.cuda_stream))
            return _outputs(model, state["out"], case["precision"])
        # a projection of a projected state is the same state: repeated passes do the same work
        capi.check(model._lib.bld_apply_projections_device(model._h, base.data_ptr(), stream.cuda_stream))
        return _outputs(model, base, case["precision"])


# ------------------------------------------------- bytes and operations of one pass
def _quadratic(k):
    """Physical points for exact quadratic products (3/2 rule)."""
    return 3 * k + 2


def work(case):
    if case["op"] == "ensemble":
        parts = [work(c) for c in _groups(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n1, n2, n3, B = case["n1"], case["n2"], case["n3"], case["members"]
    k1, k2 = (n1 - 1) // 2, (n2 - 1) // 2
    F = (k1 + 1) * (2 * k2 + 1)
    S = B * (3 * n3 - 1) * F * 16          # the state: read once and written once
    P1, P2 = 2 * k1 + 2, 2 * k2 + 2

    def transforms(p1, p2, count):         # real 2-d transforms of one layer each
        return count * 2.5 * p1 * p2 * math.log2(p1 * p2)

    solve = B * n3 * F * 30                # divergence, two sweeps, gradient
    if case["op"] == "fields":
        phys = (3 * n3 - 1) * P1 * P2 * 8
        return {"bytes": 2 * phys, "flops": 2 * (3 * n3 - 1) * transforms(P1, P2, 1)}
    if case["op"] == "project":
        return {"bytes": 2 * S + n3 * F * 8, "flops": solve}
    q1, q2 = _quadratic(k1), _quadratic(k2)
    rhs = B * n3 * (transforms(q1, q2, 9) + 20 * q1 * q2 + 3 * 30 * F)
    if case["flow"] == "les":
        rhs += B * n3 * (transforms(P1, P2, 17) + 100 * P1 * P2)
    if case["op"] == "rates":
        return {"bytes": 2 * S, "flops": rhs}
    stages = {"SSPRK33": 3, "SSPRK22": 2, "Euler": 1}[case["method"]]
    return {"bytes": 2 * S * case["steps"], "flops": case["steps"] * stages * (rhs + solve)}


# ------------------------------------- the same in 64 bits, written with torch alone
class _Flow:
    """The equations on the staggered Fourier grid: rates, projection and integrators."""

    def __init__(self, case):
        self.case, self.les = case, case["flow"] == "les"
        dev, n3 = _device(), case["n3"]
        L1, L2, self.L3 = SIZE[case["flow"]]
        k1m, k2m = (case["n1"] - 1) // 2, (case["n2"] - 1) // 2
        self.k1m, self.k2m, self.n3 = k1m, k2m, n3
        t = lambda v: torch.tensor(v, dtype=torch.float64, device=dev)
        k2 = list(range(k2m + 1)) + list(range(-k2m, 0))
        self.d1 = (t(range(k1m + 1)) * (2 * math.pi / L1))[None, None, :]
        self.d2 = (t(k2) * (2 * math.pi / L2))[None, :, None]
        vmap, dv = _mapping(case)
        self.vmap = vmap
        ext = [n3 / dv(i / n3) for i in range(n3 + 1)]
        ac = [n3 / dv((2 * i + 1) / (2 * n3)) for i in range(n3)]
        col = lambda v: t(v)[:, None, None]
        self.ext, self.ac, self.ai = col(ext), col(ac), col(ext[1:n3])
        self.nu = RE_INV[case["flow"]]
        # tridiagonal pressure matrices
        diag = torch.zeros((n3, 1, 1), dtype=torch.float64, device=dev)
        diag[1:] -= self.ai
        diag[:-1] -= self.ai
        diag = diag - (self.d1 ** 2 + self.d2 ** 2) / self.ac
        diag[-1, 0, 0] = -3 * ext[n3 - 1]
        self.gamma = torch.empty_like(diag)
        self.gamma[0] = 1 / diag[0]
        for z in range(1, n3):
            self.gamma[z] = 1 / (diag[z] - self.gamma[z - 1] * self.ai[z - 1] ** 2)
        del diag
        if self.les:
            dx = (L1 / (2 * k1m + 2)) * (L2 / (2 * k2m + 2))
            length = lambda zs: [(lambda a, b: (a ** -2 + b ** -2) ** -0.5)(
                CS * (dx * dv(z) / n3) ** (1 / 3), KAPPA * vmap(z)) for z in zs]
            self.lc2 = col(length([(2 * i + 1) / (2 * n3) for i in range(n3)])) ** 2
            self.li2 = col(length([i / n3 for i in range(1, n3)])) ** 2
            first = vmap(1 / (2 * n3))
            lg = math.log(first / Z0)
            self.strain_lo, self.stress_lo = 1 / (2 * first * lg), -(KAPPA / lg) ** 2

    def grid(self, q, P1, P2):
        """Modes (nz, K2, K1) to the physical grid (nz, P2, P1)."""
        out = torch.empty((q.shape[0], P2, P1), dtype=torch.float64, device=q.device)
        for z in range(0, q.shape[0], 32):
            h = torch.zeros((min(32, q.shape[0] - z), P2, P1 // 2 + 1), dtype=torch.complex128, device=q.device)
            h[:, :self.k2m + 1, :self.k1m + 1] = q[z:z + 32, :self.k2m + 1]
            if self.k2m:
                h[:, P2 - self.k2m:, :self.k1m + 1] = q[z:z + 32, self.k2m + 1:]
            out[z:z + 32] = torch.fft.irfft2(h, s=(P2, P1), norm="forward")
        return out

    def modes(self, p):
        P2 = p.shape[1]
        out = torch.empty((p.shape[0], 2 * self.k2m + 1, self.k1m + 1), dtype=torch.complex128, device=p.device)
        for z in range(0, p.shape[0], 32):
            x = torch.fft.rfft2(p[z:z + 32], norm="forward")
            out[z:z + 32, :self.k2m + 1] = x[:, :self.k2m + 1, :self.k1m + 1]
            if self.k2m:
                out[z:z + 32, self.k2m + 1:] = x[:, P2 - self.k2m:, :self.k1m + 1]
        return out

    def advection(self, u, v, w):
        i1, i2, ai = 1j * self.d1, 1j * self.d2, self.ai
        # any physical grid that holds the products exactly gives the same modes
        P1, P2 = (2 * ((3 * k + 3) // 2) for k in (self.k1m, self.k2m))
        g = lambda q: self.grid(q, P1, P2)
        o1 = g(i2 * w - ai * (v[1:] - v[:-1]))
        o2 = g(ai * (u[1:] - u[:-1]) - i1 * w)
        o3 = g(i1 * v - i2 * u)
        u, v, w = g(u), g(v), g(w)
        r1, r2 = o3 * v, -o3 * u
        q = 0.5 * o2 * w
        r1[:-1] -= q
        r1[1:] -= q
        q = 0.5 * o1 * w
        r2[:-1] += q
        r2[1:] += q
        r3 = 0.5 * (o2 * (u[:-1] + u[1:]) - o1 * (v[:-1] + v[1:]))
        return self.modes(r1), self.modes(r2), self.modes(r3)

    def smagorinsky(self, u, v, w):
        i1, i2, ai, ac, n = 1j * self.d1, 1j * self.d2, self.ai, self.ac, self.n3
        P1, P2 = 2 * self.k1m + 2, 2 * self.k2m + 2
        g = lambda q: self.grid(q, P1, P2)
        s11, s22 = g(i1 * u), g(i2 * v)
        s12 = (g(i2 * u) + g(i1 * v)) / 2
        up, vp, wp = g(u), g(v), g(w)
        s13 = (ai * (up[1:] - up[:-1]) + g(i1 * w)) / 2
        s23 = (ai * (vp[1:] - vp[:-1]) + g(i2 * w)) / 2
        pad = lambda q, lo, hi: torch.cat([lo, q, hi])
        zero = torch.zeros_like(up[:1])
        wx = pad(wp, zero, zero)
        s33 = ac * (wx[1:] - wx[:-1])
        sc = s11 ** 2 + s22 ** 2 + s33 ** 2 + 2 * s12 ** 2
        si = 2 * s13 ** 2 + 2 * s23 ** 2
        for s, c in ((s11, 1), (s22, 1), (s33, 1), (s12, 2)):
            si += c * ((s[1:] + s[:-1]) / 2) ** 2
        for s, q in ((s13, up), (s23, vp)):
            x = pad(s, zero, zero)
            m = ((x[1:] + x[:-1]) / 2) ** 2
            m[0] = (self.strain_lo * q[0]) ** 2
            sc += 2 * m
        nc, ni = self.lc2 * torch.sqrt(2 * sc), self.li2 * torch.sqrt(2 * si)
        t11, t22, t33, t12 = (2 * nc * s for s in (s11, s22, s33, s12))
        t13, t23 = 2 * ni * s13, 2 * ni * s23
        speed = torch.sqrt(up[:1] ** 2 + vp[:1] ** 2)
        x13 = pad(t13, -self.stress_lo * up[:1] * speed, zero)
        x23 = pad(t23, -self.stress_lo * vp[:1] * speed, zero)
        m = self.modes
        m12 = m(t12)
        r1 = i1 * m(t11) + i2 * m12 + m(ac * (x13[1:] - x13[:-1]))
        r2 = i1 * m12 + i2 * m(t22) + m(ac * (x23[1:] - x23[:-1]))
        r3 = i1 * m(t13) + i2 * m(t23) + m(ai * (t33[1:] - t33[:-1]))
        return r1, r2, r3

    def rates(self, q):
        out = []
        horizontal = -(self.d1 ** 2 + self.d2 ** 2)
        for f, s in enumerate(q):
            if f == 2:
                below, above = torch.zeros_like(s[:1]), torch.zeros_like(s[:1])
                mid, a = self.ai, self.ac           # alpha at the I nodes and at the C nodes between them
            else:
                below = (-15 * s[:1] + 5 * s[1:2] - s[2:3]) / 5
                above = ((21 * s[-1:] + 3 * s[-2:-1] - s[-3:-2]) / 23 if self.les else
                         (-15 * s[-1:] + 5 * s[-2:-1] - s[-3:-2]) / 5)
                mid, a = self.ac, self.ext
            x = torch.cat([below, s, above])
            out.append(self.nu * (mid * (a[1:] * (x[2:] - s) - a[:-1] * (s - x[:-2])) + horizontal * s))
        if not self.case["flux"]:
            out[0][:, 0, 0] += 1.0
        for part in (self.advection, self.smagorinsky) if self.les else (self.advection,):
            for o, r in zip(out, part(*q)):
                o += r
        return out

    def project(self, q):
        u, v, w = q
        i1, i2, ai, n = 1j * self.d1, 1j * self.d2, self.ai, self.n3
        p = (i1 * u + i2 * v) / self.ac
        p[:-1] += w
        p[1:] -= w
        p[-1, 0, 0] = 0
        p[0] *= self.gamma[0]
        for z in range(1, n):
            p[z] = self.gamma[z] * (p[z] - ai[z - 1] * p[z - 1])
        for z in range(n - 2, -1, -1):
            p[z] -= self.gamma[z] * ai[z] * p[z + 1]
        u, v, w = u - i1 * p, v - i2 * p, w - ai * (p[1:] - p[:-1])
        if self.case["flux"]:
            mean = (u[:, 0, 0].real / (self.ac[:, 0, 0] * self.L3)).sum()
            u[:, 0, 0] += 10.0 - mean
        return [u, v, w]

    def step(self, q, dt, method):
        mix = lambda *terms: [sum(c * s[f] for c, s in terms) for f in range(3)]
        t = self.project(mix((1, q), (dt, self.rates(q))))
        if method == "Euler":
            return t
        if method == "SSPRK22":
            return self.project(mix((0.5, q), (0.5, t), (dt / 2, self.rates(t))))
        t = self.project(mix((0.75, q), (0.25, t), (dt / 4, self.rates(t))))
        return self.project(mix((1 / 3, q), (2 / 3, t), (2 * dt / 3, self.rates(t))))


def _exact(case, seed):
    flow, members = _Flow(case), []
    for m in range(case["members"]):
        q = _state_fields(case, seed, m)
        if case["op"] == "rates":
            q = flow.rates(q)
        else:
            q = flow.project(q)
            for _ in range(case["steps"] if case["op"] == "step" else 0):
                q = flow.step(q, DT, case["method"])
        members.append([torch.view_as_real(s) for s in q])
    return {f: torch.stack([m[i] for m in members]) for i, f in enumerate(("vel1", "vel2", "vel3"))}


def exact(case, seed):
    if case["op"] == "ensemble":
        return [_exact(c, seed + 17 * i) for i, c in enumerate(_groups(case))]
    if case["op"] != "fields":
        return _exact(case, seed)
    # the default grid's highest wave has no place among the resolved modes, the rest comes back
    k1m, k2m, out = (case["n1"] - 1) // 2, (case["n2"] - 1) // 2, {}
    for f, q in zip(("vel1", "vel2", "vel3"), _physical(case, seed)):
        x = torch.fft.rfft2(q, norm="forward")
        x[:, k2m + 1] = 0
        x[:, :, k1m + 1] = 0
        out[f] = torch.fft.irfft2(x, s=q.shape[1:], norm="forward").cpu().numpy()
    return out
