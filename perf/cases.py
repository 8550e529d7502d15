"""Work that users of the framework have it do, as measurable cases.

Every case goes through a public entry point: ``Model.simulate``,
``core.simulate_ensemble``, ``core.EnsemblePlan`` with its device outputs,
``core.generate_clusters``, ``adjoint.EnsembleAdjoint`` and
``core.simulate_dom_batch``.  The workloads are the framework's own benchmark
configurations and the ensembles of the reference's notebooks (single
particles and dimers by the ten thousand), with windows short enough that two
correct runs stay comparable: stochastic trajectories amplify differences.

Results of the FP64 precision are returned as FP64.  The mixed precisions
evaluate the field and the stage maps in FP32, and the gradient is an FP32
computation: their results are kept as FP32, the precision they are good for.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from magpy_gb300 import Model, _lib, core
from magpy_gb300.adjoint import EnsembleAdjoint, sar_grad_M

MS, TEMPERATURE, K_ANIS = 4e5, 300.0, 2e4
AMPLITUDE, FREQUENCY = 1e4, 3e5


def _case(kind, n, members, steps, dt, precision="fp64", implicit=False, alpha=0.1, samples=3,
          shape="sine", renorm=False, thermal_spread=False):
    return dict(kind=kind, n=n, members=members, steps=steps, dt=dt, precision=precision,
                implicit=implicit, alpha=alpha, samples=samples, shape=shape, renorm=renorm,
                thermal_spread=thermal_spread)


def listed():
    return [
        # one Model.simulate call with its defaults (implicit midpoint, FP64) on
        # one particle: what a user tries first; latency
        dict(_case("model", 1, 1, 250, 1e-12, implicit=True, samples=51), name="one_particle"),
        # the notebooks' dimer ensembles with the defaults of EnsembleModel
        # (implicit midpoint, FP64)
        dict(_case("ensemble", 2, 10000, 10, 1e-12, implicit=True), name="dimers_implicit"),
        # the notebooks' Heun dimers with renormalisation, in mixed precision
        dict(_case("plan", 2, 50000, 1000, 1e-13, "mixed", shape="constant", renorm=True),
             name="dimers_heun_mixed"),
        # single-particle relaxation, E = 1000, FP64 Heun: the benchmark's first
        # configuration (a window of its 1e5 steps)
        dict(_case("ensemble", 1, 1000, 2000, 1e-13, samples=21, shape="constant"),
             name="singles_heun"),
        # the interacting 64-particle cluster in the reference's own arithmetic
        dict(_case("ensemble", 64, 512, 50, 5e-14), name="cluster64_heun"),
        # a cluster of its own for every member: geometry drawn on the GPU, then
        # mixed-precision Heun (the tensor cores need one shared geometry)
        dict(_case("random", 27, 1000, 400, 5e-14, "mixed"), name="random27_heun_mixed"),
        # the same with the default integrator, odd sizes
        dict(_case("random", 13, 700, 100, 2e-13, "mixed", implicit=True),
             name="random13_implicit_mixed"),
        # the benchmark's headline: 4096 members of one 64-particle cluster,
        # dipolar field on the tensor cores (a 2000-step window)
        dict(_case("plan", 64, 4096, 2000, 5e-14, "mixed_tc"), name="cluster64_heun_tc"),
        # the largest group of the uneven batch: 125 particles on a thread-block
        # cluster of CTAs
        dict(_case("plan", 125, 1638, 1000, 1e-13, "mixed_tc"), name="cluster125_heun_tc"),
        # 512 particles, implicit midpoint on the tensor cores: the benchmark's
        # large interacting cluster
        dict(_case("plan", 512, 512, 40, 2e-13, "mixed_tc", implicit=True, alpha=0.01),
             name="cluster512_implicit_tc"),
        # gradient of the dissipated energy and the final magnetisation: forward
        # with checkpoints and the backward sweep (the benchmark's 27 particles)
        dict(_case("gradient", 27, 2048, 512, 5e-14, "mixed", samples=9), name="gradient27"),
        # two-state model of a polydisperse batch (DOModel), one field cycle
        dict(_case("two_state", 1, 8192, 1, 1e-10, samples=21), name="two_state"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "singles", "dimers_implicit", "dimers_heun", "cluster_fp64",
                       "random_heun", "random_implicit", "tc_small", "tc_large", "tc_implicit",
                       "gradient", "two_state"])
    shape = rng.choice(["sine", "square", "constant"])
    if kind == "model":
        return _case("model", _log_int(rng, 1, 12), 1, _log_int(rng, 20, 200),
                     rng.choice([2e-13, 1e-12]), implicit=rng.random() < 0.7, samples=11,
                     shape=shape)
    if kind == "singles":
        return _case("ensemble", 1, _log_int(rng, 16, 16000), _log_int(rng, 50, 600), 1e-13,
                     samples=_log_int(rng, 2, 40), shape=shape, renorm=rng.random() < 0.3,
                     thermal_spread=rng.random() < 0.3, implicit=rng.random() < 0.3)
    if kind == "dimers_implicit":
        return _case("ensemble", _log_int(rng, 2, 9), _log_int(rng, 16, 4000),
                     _log_int(rng, 4, 12), 1e-12, implicit=True, shape=shape,
                     thermal_spread=rng.random() < 0.3)
    if kind == "dimers_heun":
        return _case("plan", _log_int(rng, 1, 12), _log_int(rng, 100, 8000),
                     _log_int(rng, 100, 1000), 1e-13, "mixed", shape=shape,
                     renorm=rng.random() < 0.5)
    if kind == "cluster_fp64":
        return _case("ensemble", _log_int(rng, 8, 90), _log_int(rng, 8, 300),
                     _log_int(rng, 8, 40), 5e-14, shape=shape)
    if kind == "random_heun":
        return _case("random", _log_int(rng, 2, 70), _log_int(rng, 30, 1000),
                     _log_int(rng, 50, 300), 5e-14, "mixed", shape=shape)
    if kind == "random_implicit":
        return _case("random", _log_int(rng, 2, 50), _log_int(rng, 30, 400),
                     _log_int(rng, 10, 60), 2e-13, "mixed", implicit=True, shape=shape)
    if kind == "tc_small":
        return _case("plan", _log_int(rng, 9, 64), _log_int(rng, 200, 4096),
                     _log_int(rng, 200, 1500), 5e-14, "mixed_tc", shape=shape)
    if kind == "tc_large":
        return _case("plan", _log_int(rng, 65, 520), _log_int(rng, 64, 512),
                     _log_int(rng, 20, 150), 1e-13, "mixed_tc", shape=shape)
    if kind == "tc_implicit":
        return _case("plan", _log_int(rng, 16, 300), _log_int(rng, 32, 512),
                     _log_int(rng, 8, 40), 2e-13, "mixed_tc", implicit=True,
                     alpha=rng.choice([0.01, 0.1]), shape=shape)
    if kind == "gradient":
        return _case("gradient", _log_int(rng, 1, 60), _log_int(rng, 64, 2000),
                     _log_int(rng, 64, 500), 5e-14, "mixed", samples=9)
    return _case("two_state", 1, _log_int(rng, 1, 8000), 1, 1e-10, samples=_log_int(rng, 5, 60),
                 shape=rng.choice(["sine", "square"]))


def _lattice(n, rng, pitch=22e-9):
    """n sites of a cubic lattice nearest its centre, each moved by up to 1 nm."""
    side = int(math.ceil((2.0 * n) ** (1 / 3))) + 2
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    g = g - (side - 1) / 2.0
    g = g[np.argsort(np.sum(g * g, axis=1), kind="stable")[:n]]
    return g * pitch + rng.uniform(-1e-9, 1e-9, (n, 3))


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    n, E = case["n"], case["members"]
    radius = np.exp(rng.normal(np.log(7.5e-9), 0.1, n))
    axes = rng.normal(size=(n, 3))
    axes /= np.linalg.norm(axes, axis=1, keepdims=True)
    d = dict(radius=radius, anisotropy=np.full(n, K_ANIS), axes=axes, m0=axes.copy(),
             location=_lattice(n, rng), seeds=rng.integers(0, 2 ** 31 - 1, size=E))
    d["temperature"] = (rng.uniform(280.0, 320.0, E) if case["thermal_spread"]
                        else np.full(E, TEMPERATURE))
    return d


def _end_time(case):
    return case["dt"] * (case["steps"] - 0.5)


def _field(case):
    return case["shape"], AMPLITUDE, FREQUENCY


def _ensemble_args(case, d):
    args = (case["members"], d["radius"], d["anisotropy"], d["axes"], d["m0"], d["location"], MS,
            case["alpha"], TEMPERATURE, case["renorm"], True, case["implicit"], case["dt"],
            _end_time(case), case["samples"], d["seeds"], *_field(case))
    kw = dict(precision=case["precision"])
    if case["thermal_spread"]:
        kw["per_member"] = {"temperature": d["temperature"]}
    return args, kw


class _DeviceArray:
    """A device pointer of the library as a __cuda_array_interface__ object."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr="<f8",
                                             version=3, strides=None)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "two_state":
        rng = np.random.default_rng(seed)
        radius = np.exp(rng.normal(np.log(8e-9), 0.2, case["members"]))
        return dict(case=case, volume=4 / 3 * np.pi * radius ** 3,
                    p0=np.tile([1.0, 0.0], (case["members"], 1)))
    d = _inputs(case, seed)
    s = dict(case=case, inputs=d)
    if kind == "model":
        s["model"] = Model(d["radius"], d["anisotropy"], d["axes"], d["m0"], d["location"], MS,
                           case["alpha"], TEMPERATURE, case["shape"], FREQUENCY, AMPLITUDE)
    elif kind == "plan":
        args, kw = _ensemble_args(case, d)
        s["plan"] = core.EnsemblePlan(*args, **kw)
        ptr = [ctypes.c_void_p() for _ in range(3)]
        _lib.check(_lib.lib().magpy_plan_device_outputs(s["plan"].handle,
                                                        *[ctypes.byref(p) for p in ptr], None,
                                                        None))
        rows = (case["samples"], case["members"] * case["n"])
        s["out"] = [torch.as_tensor(_DeviceArray(p.value, rows, s["plan"]), device="cuda")
                    for p in ptr]
    elif kind == "gradient":
        s["adjoint"] = EnsembleAdjoint(
            case["members"], d["radius"], d["anisotropy"], d["axes"], d["m0"], d["location"], MS,
            case["alpha"], TEMPERATURE, case["dt"], _end_time(case), case["samples"], d["seeds"],
            case["shape"], AMPLITUDE, FREQUENCY, checkpoint_every=256)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "two_state":
        return core.simulate_dom_batch(state["p0"], state["volume"], K_ANIS, TEMPERATURE, MS, 0.1,
                                       case["dt"], 1.0 / FREQUENCY, case["samples"], *_field(case))
    d = state["inputs"]
    if kind == "model":
        r = state["model"].simulate(_end_time(case), case["dt"], case["samples"],
                                    seed=int(d["seeds"][0]), implicit_solve=case["implicit"])
        return dict(time=r.time, field=r.field,
                    **{c: np.stack([getattr(r, c)[i] for i in range(r.N)]) for c in "xyz"})
    if kind == "ensemble":
        args, kw = _ensemble_args(case, d)
        a = core.simulate_ensemble(*args, **kw)
        return dict(time=a.time, field=a.field, x=a.mx, y=a.my, z=a.mz, status=a.status,
                    steps=a.steps)
    if kind == "plan":
        state["plan"].run()
        return {c: t.to(torch.float32) for c, t in zip("xyz", state["out"])}
    if kind == "random":
        g = core.generate_clusters(case["members"], case["n"], d["seeds"], 7.5e-9, 0.1,
                                   packing_fraction=0.2)
        a = core.simulate_ensemble(
            case["members"], g["radius"], np.full(g["radius"].shape, K_ANIS),
            g["anisotropy_axis"], g["magnetisation_direction"], g["location"], MS, case["alpha"],
            TEMPERATURE, False, True, case["implicit"], case["dt"], _end_time(case),
            case["samples"], d["seeds"], *_field(case), per_member_geometry=True,
            precision=case["precision"])
        return dict(radius=g["radius"], axes=g["anisotropy_axis"], location=g["location"],
                    status=g["status"],
                    **{c: m.astype(np.float32) for c, m in zip("xyz", (a.mx, a.my, a.mz))})
    time, field, M = state["adjoint"].forward()
    w = sar_grad_M(field)
    w[-1] += 1e-4
    theta, reduced = state["adjoint"].backward(w)
    return dict(time=time, field=field, M=M.astype(np.float32),
                **{"d" + k: theta[i:i + 1].astype(np.float32)
                   for i, k in enumerate(("K", "alpha", "H0"))},
                **{"dreduced%d" % i: reduced[i:i + 1].astype(np.float32) for i in range(5)})


def work(case):
    n, E, K, S = case["n"], case["members"], case["steps"], case["samples"]
    if case["kind"] == "two_state":
        # the steps an adaptive integration takes at least (its step is capped at
        # a thousandth of the run), 6 evaluations of about 60 operations each
        return {"bytes": 8.0 * E * (10 + 3 * S), "flops": 1000.0 * E * 6 * 60}
    # Heun: 251 operations a particle and two dipolar sums; an implicit step: at
    # least the guess and two Newton iterations; a gradient: forward, recompute, reverse
    per = {True: 3 * (200.0 + 18 * n), False: 251.0 + 36 * n}[case["implicit"]]
    if case["kind"] == "gradient":
        per = 3 * 251.0 + 4 * 36 * n
    inputs = n * (E if case["kind"] == "random" else 1) * 11 * 8.0 + 8.0 * E
    return {"bytes": inputs + 3 * 8.0 * S * E * n, "flops": per * E * n * K}


# ---------------------------------------------------------------------------
# the same numbers in 64 bits, in plain torch
# ---------------------------------------------------------------------------
KB, MU0, GYROMAG = 1.38064852e-23, 1.25663706e-6, 1.76086e11
MASK = 0xFFFFFFFF


def _philox_normals(seeds, n, step, device):
    """[E][n][3] standard normals of one step: Philox-4x32-10 on (step, pair)."""
    pairs = (n + 1) // 2
    E = seeds.numel()
    c = [torch.full((E, pairs), step & MASK, dtype=torch.int64, device=device),
         torch.full((E, pairs), step >> 32, dtype=torch.int64, device=device),
         torch.arange(pairs, device=device).expand(E, pairs),
         torch.full((E, pairs), 0x5D12, dtype=torch.int64, device=device)]
    k0, k1 = (seeds & MASK)[:, None], ((seeds >> 32) & MASK)[:, None]
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & MASK) ^ c[1] ^ k0, p1 & MASK, ((p0 >> 32) & MASK) ^ c[3] ^ k1,
             p0 & MASK]
        k0, k1 = (k0 + 0x9E3779B9) & MASK, (k1 + 0xBB67AE85) & MASK
    lo = lambda a, b: ((a & 0x7FF) << 11) | (b & 0x7FF)  # noqa: E731
    u21 = lambda w: ((w >> 11).double() + 0.5) * 2.0 ** -21  # noqa: E731
    u22 = lambda w: (w.double() + 0.5) * 2.0 ** -22  # noqa: E731

    def pair(ur, ut):
        r, a = torch.sqrt(-2.0 * torch.log(ur)), 2 * math.pi * ut - math.pi
        return r * torch.cos(a), r * torch.sin(a)

    a0, a1 = pair(u21(c[0]), u21(c[1]))
    b0, b1 = pair(u21(c[2]), u21(c[3]))
    z0, z1 = pair(u22(lo(c[0], c[1])), u22(lo(c[2], c[3])))
    w = torch.stack([torch.stack([a0, a1, z0], -1), torch.stack([b0, b1, z1], -1)], 2)
    return w.reshape(E, 2 * pairs, 3)[:, :n]


def _waveform(shape, t, f):
    if shape == "constant":
        return 1.0
    if shape == "sine":
        return math.sin(2 * math.pi * f * t)
    return -1.0 if int(t * f * 2) % 2 else 1.0


def _unit_field(axes, location, volumes, pref):
    """Dipolar matrix [..., 3n, 3n] of unit prefactor and of reduced distances."""
    n = location.shape[-2]
    v_av = volumes.mean(-1, keepdim=True)
    r = (location[..., None, :, :] - location[..., :, None, :]) / (v_av ** (1 / 3))[..., None, None]
    dist = r.norm(dim=-1)
    eye = torch.eye(n, dtype=torch.bool, device=location.device)
    dist = torch.where(eye, torch.ones_like(dist), dist)
    u = r / dist[..., None]
    p = pref * (volumes / v_av)[..., None, :] / dist ** 3
    p = torch.where(eye, torch.zeros_like(p), p)
    d = p[..., None, None] * (3 * u[..., :, None] * u[..., None, :]
                              - torch.eye(3, dtype=torch.float64, device=location.device))
    return d.transpose(-3, -2).reshape(*location.shape[:-2], 3 * n, 3 * n)


class _Exact:
    """Members e0..e1 of a case in reduced units; K, alpha, H0 may carry gradients."""

    def __init__(self, case, d, K, alpha, H0, sl=slice(None)):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        f = lambda v: torch.as_tensor(np.asarray(v), dtype=torch.float64, device=dev)  # noqa: E731
        one = (lambda v: f(v)[sl]) if case["kind"] == "random" else f
        self.case, self.alpha, self.device = case, alpha, dev
        self.seeds = torch.as_tensor(d["seeds"], dtype=torch.int64, device=dev)[sl]
        E, n = self.seeds.numel(), case["n"]
        vol = 4.0 / 3.0 * math.pi * one(d["radius"]) ** 3
        hk = 2 * K / MU0 / MS
        self.factor = GYROMAG * MU0 * hk / (1 + alpha * alpha)
        self.dt = case["dt"] * self.factor
        self.sq = self.dt ** 0.5
        self.happ, self.f = H0 / hk, FREQUENCY / self.factor
        T = f(d["temperature"])[sl][:, None]
        self.sr = (alpha * KB * T / (K * vol) / (1 + alpha * alpha)) ** 0.5
        self.sr = self.sr.expand(E, n)[..., None]
        self.axes = one(d["axes"])
        self.x = one(d["m0"]).expand(E, n, 3)
        self.D = None
        if n > 1:
            self.D = _unit_field(self.axes, one(d["location"]), vol, MU0 * MS * MS / 8 / math.pi / K)
        end = _end_time(case) * float(self.factor)
        S, dt = case["samples"], float(self.dt)
        self.at = [0]
        for s in range(1, S):
            thr = s * (end / (S - 1))
            k = max(int(thr / dt) - 1, self.at[-1], 1)
            while not k * dt > thr:
                k += 1
            self.at.append(k)

    def field(self, m, h):
        out = (m * self.axes).sum(-1, keepdim=True) * self.axes
        if self.D is not None:
            flat = m.reshape(m.shape[0], -1)
            dip = (flat @ self.D.T if self.D.dim() == 2
                   else torch.einsum("eij,ej->ei", self.D, flat))
            out = out + dip.reshape(m.shape)
        return torch.cat([out[..., :2], out[..., 2:] + h], -1)

    def stage(self, m, v):
        c = torch.linalg.cross(m, v)
        return -c - self.alpha * torch.linalg.cross(m, c)

    def step(self, x, k):
        t = k * float(self.dt)
        w = self.sr * self.sq * _philox_normals(self.seeds, self.case["n"], k, self.device)
        h = lambda s: self.happ * _waveform(self.case["shape"], s, float(self.f))  # noqa: E731
        if self.case["implicit"]:
            hm, y = h(t + float(self.dt) / 2), x
            for _ in range(40):
                new = x + 0.5 * self.stage(y, self.dt * self.field(y, hm) + w)
                far, y = float((new - y).abs().max()), new
                if far < 1e-15:
                    break
            return 2 * y - x
        f1 = self.stage(x, self.dt * self.field(x, h(t)) + w)
        xt = x + f1
        f2 = self.stage(xt, self.dt * self.field(xt, h(t + float(self.dt))) + w)
        x = x + 0.5 * (f1 + f2)
        return x / x.norm(dim=-1, keepdim=True) if self.case["renorm"] else x

    def samples(self):
        """The state at each sample, [S] of [E][n][3] in A/m."""
        x, got, k = self.x, [self.x], 0
        for s in range(1, len(self.at)):
            while k < self.at[s] - 1:
                k += 1
                x = self.step(x, k)
            got.append(x)
        return [g * MS for g in got]

    def times(self):
        S = len(self.at)
        end = _end_time(self.case)
        t = np.arange(S) * (end / (S - 1))
        fr = float(self.f) * float(self.factor)
        return t, np.array([AMPLITUDE * _waveform(self.case["shape"], v, fr) for v in t])


def exact(case, seed):
    kind = case["kind"]
    if kind == "two_state":
        return None  # the adaptive integrator's own samples are its answer
    d = _inputs(case, seed)
    n, E, S = case["n"], case["members"], case["samples"]
    if kind == "gradient":
        return _exact_gradient(case, d)
    if kind == "random":
        g = core.generate_clusters(E, n, d["seeds"], 7.5e-9, 0.1, packing_fraction=0.2)
        d = dict(d, radius=g["radius"], axes=g["anisotropy_axis"],
                 m0=g["magnetisation_direction"], location=g["location"])
    with torch.no_grad():
        x = _Exact(case, d, K_ANIS, case["alpha"], AMPLITUDE)
        m = torch.stack(x.samples())  # [S][E][n][3]
        t, field = x.times()
    if kind == "model":
        return dict(time=t, field=field,
                    **{c: m[:, 0, :, i].T.cpu().numpy() for i, c in enumerate("xyz")})
    rows = {c: m[..., i].reshape(S, E * n) for i, c in enumerate("xyz")}
    if kind == "plan":
        return rows
    rows = {c: v.cpu().numpy() for c, v in rows.items()}
    if kind == "ensemble":
        tile = lambda v: np.tile(v, (E, 1))  # noqa: E731
        return dict(time=tile(t), field=tile(field), **rows, status=None, steps=None)
    return dict(radius=None, axes=None, location=None, status=None, **rows)


def _exact_gradient(case, d):
    n, E = case["n"], case["members"]
    theta = [torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True)
             for v in (K_ANIS, case["alpha"], AMPLITUDE)]
    x = _Exact(case, d, K_ANIS, case["alpha"], AMPLITUDE)
    t, field = x.times()
    w = sar_grad_M(field)
    w[-1] += 1e-4
    total, grads = np.zeros(case["samples"]), np.zeros(3)
    chunk = max(1, int(2e7 / (n * case["steps"])))  # what the graph of a chunk holds
    for e0 in range(0, E, chunk):
        x = _Exact(case, d, *theta, slice(e0, min(E, e0 + chunk)))
        M = torch.stack([g[..., 2].sum() / E for g in x.samples()])
        J = (M * torch.as_tensor(w, device="cuda")).sum()
        grads += [float(g) for g in torch.autograd.grad(J, theta)]
        total += M.detach().cpu().numpy()
    return dict(time=t, field=field, M=total,
                **{"d" + k: grads[i:i + 1] for i, k in enumerate(("K", "alpha", "H0"))},
                **{"dreduced%d" % i: None for i in range(5)})
