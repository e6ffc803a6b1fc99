"""What a user of langevina_b200 has it do, as cases to be timed.

``listed()`` names twelve of them, ``draw()`` gives more of the same ranges,
``prepare()`` makes what a program holds before the call, ``run()`` is one pass
through the public entry points, ``work()`` what that pass cannot do without,
and ``exact()`` its outputs from plain torch in 64 bits.

Kinds of case:

- ``stepper``: a run segment.  A stored configuration is loaded, the evolver
  takes ``steps`` steps with a measurement every ``every`` steps, and the
  configuration is read back.
- ``adjoint``: a differentiable run and its gradients, one lattice.
- ``ensemble``: many lattices of uneven sizes started from Gaussian draws,
  stepped together, their averages and configurations read back.
- ``ensemble_adjoint``: differentiable runs of all lattices of an ensemble.
- ``snapshots``: stored configurations measured again, results on the host.
- ``x2k``: a history of walls to k space and into the frame of the mean field.
- ``correlator``: time correlators of a history.
"""
import ctypes as C
import math

import numpy as np
import torch

from langevina_b200 import Measurer, ModelA, ModelAData, _lib as L, postprocess
from langevina_b200.adjoint import diff_observables

COEF = dict(mass0=-4.813, lam=4.0, chi=5.0, gamma=1.0, diffusion=1.0 / 3.0)
EVOLVERS = {"PV2HBSplit": L.PV2HBSPLIT, "PV2HBSplitNoDiffuse": L.PV2HBSPLIT_NODIFFUSE,
            "EulerLangevinHB": L.EULER_LANGEVIN_HB, "ChargeHB": L.CHARGE_HB, "IdealPV2": L.IDEAL_PV2,
            "ModelAEulerMaruyama": L.MODELA_EM, "IdealEulerMaruyama": L.IDEAL_EM}
CTR0 = 1000  # noise counter a run segment resumes from


def _stepper(N, evolver, steps, every, inner=1, outer=1, dt=0.04, H=0.003, gauss=False):
    return dict(kind="stepper", N=N, evolver=evolver, inner=inner, outer=outer, steps=steps, every=every, dt=dt, H=H,
                gauss=gauss)


def listed():
    return [
        # the smallest lattice of the tests' workloads: Model A relaxation by heat-bath sweeps, bound by launches
        dict(_stepper(32, "EulerLangevinHB", 20, 10, dt=0.04, H=0.01), name="heat_bath_32"),
        # the ordinary production run: full Model G on 64^3, measured every ten steps
        dict(_stepper(64, "PV2HBSplit", 10, 10, H=0.006), name="model_g_64"),
        # a side that no tile divides, at the default save frequency
        dict(_stepper(90, "PV2HBSplit", 6, 3, 2, 3), name="model_g_90"),
        # the large lattice of the benchmark, default composer
        dict(_stepper(256, "PV2HBSplit", 10, 10, 2, 3), name="model_g_256"),
        # Euler-Maruyama Model A on a middling lattice
        dict(_stepper(160, "ModelAEulerMaruyama", 20, 10, dt=0.02), name="euler_maruyama_160"),
        # parameter gradients: forward and backward of a Model A run at the benchmark's size
        dict(kind="adjoint", N=48, evolver="em", steps=100, avg_begin=50, ckpt=25, dt=0.02, H=0.01,
             name="adjoint_em_48"),
        # gradients through the rotation step as well, on a side that no tile divides
        dict(kind="adjoint", N=40, evolver="ideal_em", steps=40, avg_begin=20, ckpt=10, dt=0.02, H=0.01,
             name="adjoint_ideal_em_40"),
        # an ensemble of independent events of four sizes
        dict(kind="ensemble", n20=8, n32=32, n48=8, n64=4, inner=2, outer=3, steps=60, dt=0.04, H=0.006,
             name="ensemble_mixed"),
        # batched gradients
        dict(kind="ensemble_adjoint", n32=8, n24=4, steps=200, avg_begin=100, ckpt=50, dt=0.02, H=0.003,
             name="ensemble_adjoint_32"),
        # saved configurations measured again
        dict(kind="snapshots", N=120, count=3, name="snapshots_120"),
        # the walls of a 256^3 run's history
        dict(kind="x2k", N=256, T=1024, name="x2k_256"),
        # correlators of the k walls of one axis of that history
        dict(kind="correlator", T=2000, series=11 * 129, ntmax=250, cplx=True, decim=1, conn=False,
             name="correlator_k"),
    ]


def _log_even(rng, lo, hi):
    return 2 * round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2))))


def draw(rng):
    kind = rng.choice(["stepper"] * 5 + ["adjoint", "adjoint", "ensemble", "ensemble_adjoint", "snapshots", "x2k",
                                         "correlator", "correlator"])
    if kind == "stepper":
        ev = rng.choice(["PV2HBSplit"] * 4 + ["PV2HBSplitNoDiffuse", "EulerLangevinHB", "EulerLangevinHB", "ChargeHB",
                                              "IdealPV2", "ModelAEulerMaruyama", "IdealEulerMaruyama"])
        N = _log_even(rng, 16, 240)
        if rng.random() < 0.4:
            N = max(32, N // 32 * 32)
        inner, outer = rng.choice([(1, 1), (2, 3)]) if ev.startswith("PV2HBSplit") else (1, 1)
        every = rng.choice([2, 3, 5])
        return _stepper(N, ev, every * (2 if N < 160 else 1), every, inner, outer, dt=rng.choice([0.02, 0.04]),
                        H=rng.choice([0.003, 0.006, 0.01]), gauss=ev == "EulerLangevinHB" and rng.random() < 0.3)
    if kind == "adjoint":
        steps = rng.randint(10, 60)
        return dict(kind=kind, N=_log_even(rng, 16, 72), evolver=rng.choice(["em", "em", "ideal", "ideal_em"]),
                    steps=steps, avg_begin=steps // 2, ckpt=rng.randint(3, 20), dt=0.02, H=rng.choice([0.003, 0.01]))
    if kind == "ensemble":
        inner, outer = rng.choice([(1, 1), (2, 3)])
        return dict(kind=kind, n20=rng.randint(0, 16), n32=rng.randint(1, 40), n48=rng.randint(0, 8),
                    n64=rng.randint(0, 4), inner=inner, outer=outer, steps=rng.randint(10, 50), dt=0.04, H=0.006)
    if kind == "ensemble_adjoint":
        steps = rng.randint(40, 200)
        return dict(kind=kind, n32=rng.randint(1, 10), n24=rng.randint(0, 6), steps=steps, avg_begin=steps // 2,
                    ckpt=rng.randint(4, 20), dt=0.02, H=0.003)
    if kind == "snapshots":
        return dict(kind=kind, N=_log_even(rng, 24, 160), count=rng.randint(1, 3))
    if kind == "x2k":
        N = _log_even(rng, 24, 640)
        return dict(kind=kind, N=N, T=max(4, int(rng.uniform(0.1, 1.0) * 250000 / N)))
    T = int(math.exp(rng.uniform(math.log(100), math.log(4000))))
    ntmax = rng.randint(max(1, T // 20), max(2, T // 5))
    series = max(1, int(math.exp(rng.uniform(math.log(0.02), 0.0)) * 6e8 / (T * ntmax)))
    return dict(kind=kind, T=T, series=min(series, 4257), ntmax=ntmax, cplx=rng.random() < 0.6,
                decim=rng.choice([1, 1, 1, 2, 5]), conn=rng.random() < 0.3)


# ---- inputs -----------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _normal(shape, gen):
    return torch.randn(shape, dtype=torch.float64, device=gen.device, generator=gen)


def _configuration(N, gen):
    """A configuration [N, N, N, 10] as a run near its transition has it: phi a mean field of 0.3 along the first
    direction with smooth fluctuations, <phi^2> = 1, and charges of variance chi without zero mode."""
    phi = _normal((4, N, N, N), gen)
    k2 = 2.0 - 2.0 * torch.cos(2.0 * math.pi * torch.arange(N, dtype=torch.float64, device=gen.device) / N)
    k2 = k2[:, None, None] + k2[None, :, None] + k2[None, None, :N // 2 + 1]
    phi = torch.fft.irfftn(torch.fft.rfftn(phi, dim=(1, 2, 3)) / torch.sqrt(k2 + 0.05), s=(N, N, N), dim=(1, 2, 3))
    phi *= math.sqrt(0.91 / 4.0) / phi.square().mean().sqrt()
    phi[0] += 0.3
    q = math.sqrt(COEF["chi"]) * _normal((6, N, N, N), gen)
    q -= q.mean(dim=(1, 2, 3), keepdim=True)
    return torch.cat([phi, q]).permute(1, 2, 3, 0).contiguous()


def _series(case, gen):
    """[T, series] with the memory of a measured history: x(t+1) = 0.9 x(t) + noise, by blocks of independent starts."""
    T, ns, w = case["T"], case["series"], 2 if case["cplx"] else 1
    x = _normal((T, ns * w), gen)
    for t in range(1, T):
        x[t].add_(x[t - 1], alpha=0.9)
    x += 0.5
    return torch.view_as_complex(x.reshape(T, ns, 2)) if case["cplx"] else x


def _walls(case, gen):
    w = 0.05 * _normal((case["T"], 3, 11, case["N"]), gen)
    w[:, :, 0] += 0.3
    w[:, :, 10] += 1.0
    return w


def _seed(seed, r=0):
    return (int(seed) * 7919 + 31 * r + 5) & 0x7FFFFFFF


def _replicas(case):
    return [N for N in (64, 48, 32, 24, 20) for _ in range(case.get(f"n{N}", 0))]


# ---- states -----------------------------------------------------------------
def _model(N, H, seed):
    m = ModelA(ModelAData(dict(NX=N, mass0=COEF["mass0"], H=H, chi=COEF["chi"], gamma=COEF["gamma"],
                               diffusion=COEF["diffusion"], seed=_seed(seed), **{"lambda": COEF["lam"]})))
    L.check(m.lib.lgv_set_stream(m.handle, C.c_void_p(torch.cuda.current_stream().cuda_stream)), "lgv_set_stream")
    return m


class _Ensemble:
    def __init__(self, sizes, H, seed):
        self.lib = L.load()
        ps = (L.lgv_params * len(sizes))(*[L.make_params(N, H=H, seed=_seed(seed, r), **COEF)
                                           for r, N in enumerate(sizes)])
        h = C.c_void_p()
        L.check(self.lib.lgv_ensemble_create(len(sizes), ps, C.byref(h)), "lgv_ensemble_create")
        self.handle = h
        self("set_stream", C.c_void_p(torch.cuda.current_stream().cuda_stream))

    def __call__(self, name, *args):
        L.check(getattr(self.lib, "lgv_ensemble_" + name)(self.handle, *args), "lgv_ensemble_" + name)

    def __del__(self):
        try:
            self.lib.lgv_ensemble_destroy(self.handle)
        except Exception:
            pass


def prepare(case, seed):
    kind, gen = case["kind"], _generator(seed)
    s = dict(case=case)
    if kind == "stepper":
        s["model"] = _model(case["N"], case["H"], seed)
        if case["gauss"]:
            s["model"].set_hb_proposal(True)
        s["u"] = _configuration(case["N"], gen)
        s["out"] = torch.empty_like(s["u"])
        n = int(s["model"].lib.lgv_measure_size(case["N"]))
        s["meas"] = torch.empty((case["steps"] // case["every"], n), dtype=torch.float64, device="cuda")
    elif kind == "adjoint":
        s["model"] = _model(case["N"], case["H"], seed)
        s["u"] = _configuration(case["N"], gen)
        s["out"] = torch.empty_like(s["u"])
        s["theta"] = torch.tensor([COEF["mass0"], COEF["lam"], case["H"], COEF["gamma"]], dtype=torch.float64)
    elif kind in ("ensemble", "ensemble_adjoint"):
        sizes = _replicas(case)
        s["ens"] = _Ensemble(sizes, case["H"], seed)
        s["avg"] = np.zeros((len(sizes), 11))
        s["all"] = torch.empty(sum(10 * N ** 3 for N in sizes), dtype=torch.float64, pin_memory=True)
        s["host"] = s["all"].split([10 * N ** 3 for N in sizes])  # one buffer, each replica's part of it
        if kind == "ensemble_adjoint":
            s["w"] = np.ones((len(sizes), 2))
            s["obs"], s["grad"] = np.zeros((len(sizes), 2)), np.zeros((len(sizes), 4))
            s["start"] = [_configuration(N, gen).cpu().pin_memory() for N in sizes]
    elif kind == "snapshots":
        s["model"] = _model(case["N"], 0.003, seed)
        s["u"] = [_configuration(case["N"], gen) for _ in range(case["count"])]
        s["measurers"] = [Measurer(s["model"]) for _ in range(case["count"])]
    elif kind == "x2k":
        s["walls"] = _walls(case, gen)
    else:
        s["a"] = _series(case, gen)
        s["b"] = s["a"].conj().resolve_conj() if case["cplx"] else s["a"]
    return s


# ---- one pass ---------------------------------------------------------------
def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _load(m, u):
    L.check(m.lib.lgv_set_state_device(m.handle, _ptr(u)), "lgv_set_state_device")
    m.set_counter(CTR0)


def _store(m, u):
    L.check(m.lib.lgv_get_state_device(m.handle, _ptr(u)), "lgv_get_state_device")
    return u


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "stepper":
        m = s["model"]
        _load(m, s["u"])
        for i in range(case["steps"] // case["every"]):
            L.check(m.lib.lgv_step(m.handle, EVOLVERS[case["evolver"]], case["inner"], case["outer"], case["dt"], 0.0,
                                   case["every"]), "lgv_step")
            L.check(m.lib.lgv_measure_device(m.handle, _ptr(s["meas"][i])), "lgv_measure_device")
        return dict(state=_store(m, s["out"]), measured=s["meas"])
    if kind == "adjoint":
        m = s["model"]
        _load(m, s["u"])
        theta = s["theta"].clone().requires_grad_(True)
        obs = diff_observables(m, theta, case["dt"], case["steps"], case["avg_begin"], case["ckpt"],
                               evolver=case["evolver"])
        obs.sum().backward()
        return dict(obs=obs.detach(), grad=theta.grad, state=_store(m, s["out"]))
    if kind == "ensemble":
        e = s["ens"]
        e("set_counter", CTR0)
        e("initialize", L.INIT_PHI_GAUSSIAN, 0.5)
        e("initialize", L.INIT_CHARGES_GAUSSIAN, 0.0)
        e("step", L.PV2HBSPLIT, case["inner"], case["outer"], case["dt"], 0.0, case["steps"])
        e("oaverage", L.ptr(s["avg"]))
        for r, u in enumerate(s["host"]):
            e("get_state", r, _ptr(u))
        return dict(averages=s["avg"], states=s["all"])
    if kind == "ensemble_adjoint":
        e = s["ens"]
        for r, u in enumerate(s["start"]):
            e("set_state", r, _ptr(u))
        e("set_counter", CTR0)
        e("diff_forward", case["dt"], 0.0, case["steps"], case["avg_begin"], case["ckpt"], L.ptr(s["obs"]))
        e("diff_backward", L.ptr(s["w"]), L.ptr(s["grad"]))
        for r, u in enumerate(s["host"]):
            e("get_state", r, _ptr(u))
        return dict(obs=s["obs"], grad=s["grad"], states=s["all"])
    if kind == "snapshots":
        out = []
        for u, meas in zip(s["u"], s["measurers"]):
            L.check(s["model"].lib.lgv_set_state_device(s["model"].handle, _ptr(u)), "lgv_set_state_device")
            out.append(meas.measure().arrays())
        return out
    if kind == "x2k":
        wk = postprocess.x2k(s["walls"])
        return dict(k=wk, rotated=postprocess.x2k_rotated(wk))
    c, err = postprocess.computeOtOtp(s["a"], s["b"], conn=case["conn"], nTMax=case["ntmax"], decim=case["decim"])
    return dict(c=c, err=err)


# ---- what a pass cannot do without -------------------------------------------
# floating-point operations per site: an ideal step, a heat-bath sweep, the six
# faces of a charge step (three links per site, six charges), an
# Euler-Maruyama step, its adjoint, the ideal step's adjoint, one measurement
FLOPS = dict(ideal=250.0, hb=90.0, charge=270.0, em=170.0, em_adj=230.0, ideal_adj=700.0, meas=60.0)


def _measure_doubles(N):
    return 11 + 75 * N + 234 * (N // 2 + 1)


def _step_flops(evolver, inner, outer):
    f = FLOPS
    split = outer * (f["ideal"] + inner * f["hb"])
    return {"PV2HBSplit": split + f["charge"], "PV2HBSplitNoDiffuse": split, "EulerLangevinHB": f["hb"],
            "ChargeHB": f["charge"], "IdealPV2": f["ideal"], "ModelAEulerMaruyama": f["em"],
            "IdealEulerMaruyama": f["ideal"] + f["em"]}[evolver]


def work(case):
    """Each input read once and each output written once: the configuration in and out, the measurements out."""
    kind = case["kind"]
    if kind == "stepper":
        V, nm = case["N"] ** 3, case["steps"] // case["every"]
        return dict(bytes=160.0 * V + 8.0 * nm * _measure_doubles(case["N"]),
                    flops=V * (case["steps"] * _step_flops(case["evolver"], case["inner"], case["outer"])
                               + nm * FLOPS["meas"]))
    if kind == "adjoint":
        V, ev = case["N"] ** 3, case["evolver"]
        per = 3 * FLOPS["em"] + FLOPS["em_adj"] if ev != "ideal" else 0.0
        per += 3 * FLOPS["ideal"] + FLOPS["ideal_adj"] if ev != "em" else 0.0
        return dict(bytes=160.0 * V + 48.0, flops=V * case["steps"] * per)
    if kind == "ensemble":
        V = sum(N ** 3 for N in _replicas(case))
        return dict(bytes=80.0 * V, flops=V * case["steps"] * _step_flops("PV2HBSplit", case["inner"], case["outer"]))
    if kind == "ensemble_adjoint":
        V = sum(N ** 3 for N in _replicas(case))
        return dict(bytes=160.0 * V, flops=V * case["steps"] * (3 * FLOPS["em"] + FLOPS["em_adj"]))
    if kind == "snapshots":
        V = case["N"] ** 3
        return dict(bytes=case["count"] * (80.0 * V + 8.0 * _measure_doubles(case["N"])),
                    flops=case["count"] * FLOPS["meas"] * V)
    if kind == "x2k":
        rows, N, NK = 33.0 * case["T"], case["N"], case["N"] // 2 + 1
        # an FFT's count, and 60 per rotated mode
        return dict(bytes=rows * 8 * (N + 2 * NK) + 3.0 * case["T"] * 13 * NK * 16,
                    flops=rows * 2.5 * N * math.log2(N) + 60.0 * 3 * case["T"] * NK)
    n, w = float(case["T"]) * case["series"], 2 if case["cplx"] else 1
    terms = sum((case["T"] - t + case["decim"] - 1) // case["decim"] for t in range(case["ntmax"])) * case["series"]
    return dict(bytes=8.0 * w * (2 * n + case["ntmax"] * case["series"]), flops=terms * (8.0 if case["cplx"] else 2.0))


# ---- the same in plain torch, 64 bits ------------------------------------------
def _i64(x):
    x &= (1 << 64) - 1
    return x - (1 << 64) if x >> 63 else x


GOLDEN, MUL1, MUL2 = 0x9E3779B97F4A7C15, 0xBF58476D1CE4E5B9, 0x94D049BB133111EB


def _mix_int(z):
    z &= (1 << 64) - 1
    z = (z ^ (z >> 30)) * MUL1 & ((1 << 64) - 1)
    z = (z ^ (z >> 27)) * MUL2 & ((1 << 64) - 1)
    return z ^ (z >> 31)


def _srl(x, n):
    return (x >> n) & ((1 << (64 - n)) - 1)


def _words(sk, w):
    """splitmix64 outputs w of the sequence seeded with sk."""
    z = (w + 1) * _i64(GOLDEN) + _i64(sk)
    z = (z ^ _srl(z, 30)) * _i64(MUL1)
    z = (z ^ _srl(z, 27)) * _i64(MUL2)
    return z ^ _srl(z, 31)


def _key(seed):
    return _mix_int(int(seed) + GOLDEN)


def _sub(key, ctr):
    return _mix_int(key + (ctr + 1) * GOLDEN)


def _draws(sk, n, count):
    """The first `count` outputs of the xoroshiro128+ streams of sites n."""
    a, b = _words(sk, 2 * n), _words(sk, 2 * n + 1)
    out = []
    for _ in range(count):
        out.append(a + b)
        b = b ^ a
        a, b = ((a << 55) | _srl(a, 9)) ^ b ^ (b << 14), (b << 36) | _srl(b, 28)
    return out


def _u53(r):
    return _srl(r, 11).to(torch.float64) * 2.0 ** -53


def _normals(sk, n, count):
    r, z = _draws(sk, n, count), []
    for ra, rb in zip(r[::2], r[1::2]):
        rho, ang = torch.sqrt(-2.0 * torch.log(1.0 - _u53(ra))), 2.0 * math.pi * _u53(rb)
        z += [rho * torch.cos(ang), rho * torch.sin(ang)]
    return torch.stack(z)


AXIS = (-1, -2, -3)  # x, y, z of an array [..., k, j, i]


def _nbr_sum(f):
    return sum(torch.roll(f, s, a) for a in AXIS for s in (1, -1))


class _Lattice:
    """One lattice advanced in plain torch."""

    def __init__(self, N, H, seed, ctr=CTR0, gauss=False):
        self.N, self.H, self.key, self.ctr, self.gauss = N, H, _key(_seed(*seed)), ctr, gauss
        self.n = torch.arange(N ** 3, dtype=torch.int64, device=_device()).reshape(N, N, N)
        i = torch.arange(N, device=_device())
        self.par = (i[:, None, None] + i[None, :, None] + i[None, None, :]) & 1
        self.mass, self.lam, self.gamma = COEF["mass0"], COEF["lam"], COEF["gamma"]

    def load(self, u):
        f = u.permute(3, 0, 1, 2)
        self.phi, self.q = f[:4].clone(), f[4:].clone()

    def store(self):
        return torch.cat([self.phi, self.q]).permute(1, 2, 3, 0).contiguous()

    def initialize(self):
        self.phi = 0.5 * _normals(_sub(self.key, self.ctr), self.n, 4)
        z = math.sqrt(COEF["chi"]) * _normals(_sub(self.key, self.ctr + 1), self.n, 6)
        self.q = z - z.mean(dim=(1, 2, 3), keepdim=True)
        self.ctr += 2

    def _rotate(self, phi, q, k):
        def qexp(v):
            x2 = (v * v).sum(0)
            x = torch.sqrt(x2)
            return torch.cat([torch.cos(x)[None], -(torch.sin(x) / x) * v])

        def mul(a, b):
            return torch.stack([a[0] * b[0] - (a[1] * b[1] + a[2] * b[2] + a[3] * b[3]),
                                a[2] * b[3] - b[2] * a[3] + b[0] * a[1] + a[0] * b[1],
                                a[3] * b[1] - a[1] * b[3] + b[0] * a[2] + a[0] * b[2],
                                a[1] * b[2] - b[1] * a[2] + b[0] * a[3] + a[0] * b[3]])

        h = 0.5 * k
        return mul(qexp(-h * (q[3:] + q[:3])), mul(phi, qexp(h * (q[3:] - q[:3]))))

    def ideal(self, dt):
        k, a2 = dt / 2.0 / COEF["chi"], 1.0  # lattice spacing one
        p = self._rotate(self.phi, self.q, k)
        S = _nbr_sum(p)
        J = [a2 * (p[0] * S[c + 1] - p[c + 1] * S[0]) - self.H * p[c + 1] for c in range(3)]
        J += [a2 * (p[1 + (s + 1) % 3] * S[1 + (s + 2) % 3] - p[1 + (s + 2) % 3] * S[1 + (s + 1) % 3])
              for s in range(3)]
        self.q = self.q + dt * torch.stack(J)
        self.phi = self._rotate(p, self.q, k)

    def heat_bath(self, dt):
        sk = _sub(self.key, self.ctr)
        r = _draws(sk, self.n, 5)
        if self.gauss:
            v = _normals(sk, self.n, 4)
        else:
            v = torch.stack([(2.0 * _u53(x) - 1.0) * math.sqrt(3.0) for x in r[:4]])
        acc, lam2 = _u53(r[4]), 0.5 * (6.0 + self.mass)
        for parity in range(2):
            po = self.phi
            heff = _nbr_sum(po)
            heff[0] += self.H
            pn = po + math.sqrt(2.0 * dt * self.gamma) * v
            so, sn = (po * po).sum(0), (pn * pn).sum(0)
            dS = -((heff * pn).sum(0) - (heff * po).sum(0)) + lam2 * (sn - so) + self.lam / 4 * (sn * sn - so * so)
            yes = (self.par == parity) & ((dS < 0) | (acc < torch.exp(-dS)))
            self.phi = torch.where(yes, pn, po)
        self.ctr += 1

    def charges(self, dt):
        w = _mix_int(_sub(self.key, self.ctr) + GOLDEN)
        order = [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)][(w & 0xFFFFFFFF) % 6]
        eo = (1, 0) if w >> 63 else (0, 1)
        rms, chi = math.sqrt(2.0 * dt * (COEF["diffusion"] * COEF["chi"])), COEF["chi"]
        for p in range(6):
            axis, sk = AXIS[order[p // 2]], _sub(self.key, self.ctr + 1 + p)
            site = self.par == eo[p % 2]
            for c in range(6):
                word = _words(sk, 6 * self.n + c)
                lo, hi = (word & 0xFFFFFFFF).to(torch.float64), _srl(word, 32).to(torch.float64)
                q = rms * (((lo + 0.5) * 2.0 ** -31 - 1.0) * math.sqrt(3.0))
                a, b = self.q[c], torch.roll(self.q[c], -1, axis)
                da, db = a - q, b + q
                dS = (da * da + db * db - a * a - b * b) * (1.0 / (2.0 * chi))
                q = torch.where(site & ((dS < 0) | ((hi + 0.5) * 2.0 ** -32 < torch.exp(-dS))), q, 0.0)
                self.q[c] = self.q[c] - q + torch.roll(q, 1, axis)
        self.ctr += 7

    def euler(self, dt):
        xi = _normals(_sub(self.key, self.ctr), self.n, 4)
        p = self.phi
        F = -_nbr_sum(p) + (6.0 + self.mass) * p + self.lam * (p * p).sum(0) * p
        F = F - self.H * torch.tensor([1.0, 0, 0, 0], dtype=torch.float64, device=p.device)[:, None, None, None]
        self.phi = p - dt * self.gamma * F + (2.0 * self.gamma * dt) ** 0.5 * xi
        self.ctr += 1

    def step(self, evolver, inner, outer, dt):
        if evolver.startswith("PV2HBSplit"):
            for _ in range(outer):
                self.ideal(dt / outer)
                for _ in range(inner):
                    self.heat_bath(dt / (inner * outer))
            if evolver == "PV2HBSplit":
                self.charges(dt)
        elif evolver == "EulerLangevinHB":
            self.heat_bath(dt)
        elif evolver == "ChargeHB":
            self.charges(dt)
        else:
            if evolver.startswith("Ideal"):
                self.ideal(dt)
            if evolver.endswith("EulerMaruyama"):
                self.euler(dt)

    def measure(self):
        """The measurement as a dict of the measurer's arrays, x, y and z axes of each."""
        phi, q = self.phi, self.q
        p2 = (phi * phi).sum(0)
        sigma = torch.sqrt(p2)
        n = phi / sigma
        phase = torch.cat([sigma[None], n, _contract(n, q), _contract(n, q[[3, 4, 5, 0, 1, 2]]), (sigma * sigma)[None]])
        obs = torch.cat([phi, q, p2[None]])
        out = {"OAverage": obs.mean(dim=(1, 2, 3))}
        for ax, dims in (("X", (1, 2)), ("Y", (1, 3)), ("Z", (2, 3))):
            for name, f in ((f"wall{ax}", obs), (f"wall{ax}Phase", phase)):
                out[name] = f.mean(dim=dims)
                out[name + "_k"] = torch.view_as_real(torch.fft.rfft(out[name], dim=-1) / self.N)
            w = torch.view_as_complex(out[f"wall{ax}_k"])
            d = w[:4, 0] / torch.sqrt((w[:4, 0].abs() ** 2).sum())
            d = d[:, None].expand(4, w.shape[1])
            along = (d * w[:4]).sum(0)
            rot = torch.cat([along[None], w[:4] - d * along, _contract(d, w[4:10]),
                             _contract(d, w[[7, 8, 9, 4, 5, 6]]), w[10:11]])
            out[f"wall{ax}_k_rotated"] = torch.view_as_real(rot)
        return out


def _contract(n, r):
    return torch.stack([-(n[1] * r[0]) - n[2] * r[1] - n[3] * r[2],
                        n[0] * r[0] + n[3] * r[4] - n[2] * r[5],
                        n[0] * r[1] - n[3] * r[3] + n[1] * r[5],
                        n[0] * r[2] + n[2] * r[3] - n[1] * r[4]])


def _packed(m):
    """A measurement in the order lgv_measure_device packs it."""
    names = ["OAverage"] + [f"wall{ax}{tail}" for tail in ("", "_k", "_k_rotated", "Phase", "Phase_k") for ax in "XYZ"]
    return torch.cat([m[k].reshape(-1) for k in names])


def _gradients(lat, evolver, steps, avg_begin, dt):
    """Observables and gradients of a differentiable run by autograd; leaves the final state in `lat`."""
    theta = torch.tensor([lat.mass, lat.lam, lat.H, lat.gamma], dtype=torch.float64, device=_device(),
                         requires_grad=True)
    lat.mass, lat.lam, lat.H, lat.gamma = theta
    o = [0.0, 0.0]
    for n in range(steps):
        lat.step({"em": "ModelAEulerMaruyama", "ideal": "IdealPV2", "ideal_em": "IdealEulerMaruyama"}[evolver], 1, 1, dt)
        if n >= avg_begin:
            a = lat.phi.mean(dim=(1, 2, 3))
            o = [o[0] + a[0], o[1] + lat.N ** 3 * (a[1:] ** 2).sum()]
    obs = torch.stack([x / (steps - avg_begin) for x in o])
    obs.sum().backward()
    lat.phi, lat.q = lat.phi.detach(), lat.q.detach()
    return obs.detach(), theta.grad


def exact(case, seed):
    kind, gen = case["kind"], _generator(seed)
    if kind == "stepper":
        lat = _Lattice(case["N"], case["H"], (seed,), gauss=case["gauss"])
        lat.load(_configuration(case["N"], gen))
        meas = []
        for n in range(1, case["steps"] + 1):
            lat.step(case["evolver"], case["inner"], case["outer"], case["dt"])
            if n % case["every"] == 0:
                meas.append(_packed(lat.measure()))
        return dict(state=lat.store(), measured=torch.stack(meas))
    if kind == "adjoint":
        lat = _Lattice(case["N"], case["H"], (seed,))
        lat.load(_configuration(case["N"], gen))
        obs, grad = _gradients(lat, case["evolver"], case["steps"], case["avg_begin"], case["dt"])
        return dict(obs=obs, grad=grad, state=lat.store())
    if kind == "ensemble":
        avg, states = [], []
        for r, N in enumerate(_replicas(case)):
            lat = _Lattice(N, case["H"], (seed, r))
            lat.initialize()
            for _ in range(case["steps"]):
                lat.step("PV2HBSplit", case["inner"], case["outer"], case["dt"])
            avg.append(lat.measure()["OAverage"])
            states.append(lat.store().reshape(-1))
        return dict(averages=torch.stack(avg), states=torch.cat(states))
    if kind == "ensemble_adjoint":
        obs, grad, states = [], [], []
        for r, N in enumerate(_replicas(case)):
            lat = _Lattice(N, case["H"], (seed, r))
            lat.load(_configuration(N, gen))
            o, g = _gradients(lat, "em", case["steps"], case["avg_begin"], case["dt"])
            obs.append(o)
            grad.append(g)
            states.append(lat.store().reshape(-1))
        return dict(obs=torch.stack(obs), grad=torch.stack(grad), states=torch.cat(states))
    if kind == "snapshots":
        out = []
        for _ in range(case["count"]):
            lat = _Lattice(case["N"], 0.003, (seed,))
            lat.load(_configuration(case["N"], gen))
            out.append(lat.measure())
        return out
    if kind == "x2k":
        w = _walls(case, gen)
        wk = torch.fft.rfft(w, dim=-1) / case["N"]
        d = wk[:, :, :4, :1].real
        d = (d / d.square().sum(2, keepdim=True).sqrt()).movedim(2, 0)
        f = wk.movedim(2, 0)
        along = (d * f[:4]).sum(0)
        rot = torch.cat([along[None], f[:4] - d * along, _contract(d, f[4:10]), _contract(d, f[[7, 8, 9, 4, 5, 6]])])
        return dict(k=torch.view_as_real(wk), rotated=torch.view_as_real(rot.movedim(0, 2).contiguous()))
    a = _series(case, gen)
    b = a.conj().resolve_conj() if case["cplx"] else a
    T, c = case["T"], []
    off = a.mean(0) * b.mean(0) if case["conn"] else 0.0
    for t in range(case["ntmax"]):
        c.append((a[:T - t:case["decim"]] * b[t::case["decim"]]).mean(0) - off)
    c = torch.stack(c)
    return dict(c=c, err=torch.zeros_like(c))
