"""The performance cases of the particle step: what a user's program calls, over the range of its sizes.

`listed()` names the fixed cases, `draw(rng)` gives one more of the same ranges, `prepare` makes a case's
inputs and the handle that a program keeps, `run` is one pass through the public entry points, `work` is
the bytes and operations a pass cannot do without, and `exact` computes the results of the first pass in
64 bits with plain torch and numpy.

Kinds of case:
  step    one RK4 step of a particle population (first_repo_gb300.pstep). `drive` says how it is called:
          "run" (fields bound once, pstep_run), "staged" (the solver's own call order: velocity and
          temperature bound in every stage, the deposits and the energy mean read after each), or "owner"
          (the program owns the particle vectors: upload, prime, step, download)
  gas     one coupled time step of the box gas solver with its particles (first_repo_gb300.gas)
  train   Adam steps of the correction's network (first_repo_gb300.mlp)
  forward the network's outputs for a table of samples
"""
from __future__ import annotations

import math

import numpy as np
import torch

from first_repo_gb300 import gas, learn, mlp, pstep

PI = 3.141592653589793
L = 2 * PI
DT = 1e-3
PRE = (0.5, 0.5, 1.0, 1.0 / 6.0)
POST = (1.0 / 6.0, 1.0 / 3.0, 1.0 / 3.0, 1.0 / 6.0)
FIELDS = ("C", "RHS_RU_x", "RHS_RU_y", "RHS_RU_z", "RHS_Part_Temp")
GAS_FIELDS = ("RU_x", "RU_y", "RU_z", "Rho", "P", "T", "RHS_Part_Temp")
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _step(name, n, count, precision, drive, **more):
    case = dict(kind="step", n=n, count=count, precision=precision, drive=drive, clustered=False, blobs=64,
                order="storage", correction=False, tau_each=False, gravity=False, twc=True)
    case.update(more)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # a small test box on the mixed-precision form: launches and latency count
        _step("fp32_box64", 64, 1 << 15, "fp32", "run"),
        # a grid that is not a multiple of 16, a ragged population, per-particle tau_p and gravity, called
        # stage by stage as the solver does
        _step("fp32_box104_staged", 104, 1_300_003, "fp32", "staged", clustered=True, tau_each=True, gravity=True),
        # a production run at moderate resolution, clustered, per-particle tau_p
        _step("fp32_box256", 256, 1 << 24, "fp32", "run", clustered=True, tau_each=True),
        # the headline: the largest box with the learned correction (bench.py's box512_corrected)
        _step("fp32_box512_corrected", 512, 1 << 27, "fp32", "run", clustered=True, correction=True),
        # a host code that owns the particle vectors and hands them over every step
        _step("fp32_box160_owner", 160, 4_000_001, "fp32", "owner", clustered=True),
        # the double-precision drop-in behind the solver's particle class: a small box ...
        _step("fp64_box64_staged", 64, 1 << 15, "fp64", "staged", order="reference"),
        # ... a box of odd size whose fields have to equal the solver's bit for bit ...
        _step("fp64_box90_sums", 90, 400_001, "fp64", "run", order="sums", clustered=True, gravity=True),
        # ... and a production box (config.py's box256_clustered)
        _step("fp64_box256_staged", 256, 1 << 24, "fp64", "staged", order="reference", clustered=True),
        # the runs that the correction's training data come from: isolated particles in gas at rest
        dict(name="gas_quiescent128", kind="gas", n=128, count=512, precision="fp32", quiescent=True),
        # the solver's own coupled run in a small turbulent box, double precision
        dict(name="gas_box64", kind="gas", n=64, count=1 << 15, precision="fp64", quiescent=False),
        # training the correction's network at its own batch size
        dict(name="train_8192", kind="train", rows=1 << 20, batch=8192, steps=100),
        # evaluating the network on a recorded data set
        dict(name="forward_1m", kind="forward", rows=(1 << 20) + 3),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("fp32", "fp32", "fp32", "fp64", "fp64", "gas", "train", "forward"))
    if kind == "fp32":
        n = 8 * int(round(_log(rng, 4, 32)))  # 32 .. 256
        count = int(min(_log(rng, 0.02, 2.0) * n ** 3, 1 << 24)) | 1
        return _step(None, n, count, "fp32", rng.choice(("run", "staged", "owner")), clustered=rng.random() < 0.7,
                     blobs=rng.choice((8, 64)), correction=rng.random() < 0.4, tau_each=rng.random() < 0.4,
                     gravity=rng.random() < 0.3, twc=rng.random() < 0.9)
    if kind == "fp64":
        n = int(round(_log(rng, 20, 200)))
        count = int(min(_log(rng, 0.05, 2.0) * n ** 3, 1 << 23)) | 1
        return _step(None, n, count, "fp64", rng.choice(("run", "staged")), clustered=rng.random() < 0.7,
                     blobs=rng.choice((8, 64)), order=rng.choice(("reference", "reference", "storage", "sums")),
                     tau_each=rng.random() < 0.3, gravity=rng.random() < 0.3, twc=rng.random() < 0.9)
    if kind == "gas":
        n = rng.choice((32, 64, 128))
        return dict(kind="gas", n=n, count=int(_log(rng, 100, 0.25 * n ** 3)), precision=rng.choice(("fp32", "fp64")),
                    quiescent=False)
    if kind == "train":
        return dict(kind="train", rows=int(_log(rng, 1 << 14, 1 << 20)), batch=128 * int(round(_log(rng, 1, 256))),
                    steps=rng.choice((20, 50, 100)))
    return dict(kind="forward", rows=int(_log(rng, 1, 1 << 22)))


# ---------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _ghost(a):
    n = a.shape[0]
    g = torch.empty((n + 2,) * 3, dtype=a.dtype, device=a.device)
    g[1:-1, 1:-1, 1:-1] = a
    g[1:-1, 1:-1, 0], g[1:-1, 1:-1, -1] = a[:, :, -1], a[:, :, 0]
    g[1:-1, 0], g[1:-1, -1] = g[1:-1, -2], g[1:-1, 1]
    g[0], g[-1] = g[-2], g[1]
    return g


def _velocity(n, gen):
    """Random-phase solenoidal modes in shells 1..8 with E(k) ~ k^-5/3 and u_rms = 1, on the cell faces [z, y, x]."""
    top = min(8, n // 2 - 1)
    k = torch.arange(-top, top + 1, device=DEVICE, dtype=torch.float64)
    kz, ky, kx = torch.meshgrid(k, k, k[top:], indexing="ij")
    k2 = kx ** 2 + ky ** 2 + kz ** 2
    amp = torch.where((k2 > 0) & (k2 <= top * top), k2.clamp_min(1.0) ** (-11.0 / 12.0), torch.zeros_like(k2))
    vec = torch.randn((3,) + tuple(k2.shape), generator=gen, device=DEVICE, dtype=torch.complex128) * amp
    along = (kx * vec[0] + ky * vec[1] + kz * vec[2]) / k2.clamp_min(1.0)
    vec = vec - along * torch.stack((kx, ky, kz))
    half = PI / n  # cell centres lie half a cell up from the faces
    shift = torch.exp(1j * torch.stack((ky + kz, kx + kz, kx + ky)) * half)
    at = torch.remainder(k, n).long()
    out = []
    for d in range(3):
        spec = torch.zeros((n, n, n // 2 + 1), dtype=torch.complex128, device=DEVICE)
        spec[at[:, None, None], at[None, :, None], at[None, None, top:]] = vec[d] * shift[d]
        out.append(torch.fft.irfftn(spec, s=(n, n, n)))
    rms = math.sqrt(sum(float(u.square().mean()) for u in out) / 3.0)
    return [u / rms for u in out]


def _temperature(n, gen):
    """1 + 0.05 N(0,1) smoothed by a 3-cell box filter."""
    t = torch.randn((n, n, n), generator=gen, device=DEVICE, dtype=torch.float64)
    for d in range(3):
        t = (t + torch.roll(t, 1, d) + torch.roll(t, -1, d)) / 3.0
    return 1.0 + 0.05 * t / t.std()


def _positions(n, count, clustered, blobs, gen):
    """Uniform positions, or half of them in Gaussian blobs of sigma = 4 cells; numbered along the grid, as a
    restart written from a sorted run numbers them."""
    x = torch.rand((3, count), generator=gen, device=DEVICE, dtype=torch.float64) * n
    if clustered:
        m = count // 2
        centre = torch.rand((3, blobs), generator=gen, device=DEVICE, dtype=torch.float64) * n
        pick = torch.randint(0, blobs, (m,), generator=gen, device=DEVICE)
        for d in range(3):
            x[d, :m] = centre[d][pick] + 4.0 * torch.randn(m, generator=gen, device=DEVICE, dtype=torch.float64)
        x.remainder_(n)
        x.clamp_(0.0, n * (1.0 - 1e-12))
    cell = (x[2].int() * n + x[1].int()) * n + x[0].int()
    by = torch.argsort(cell)
    del cell
    return torch.stack([x[d][by] * (L / n) for d in range(3)])


def _face_gather(n, x, faces):
    """The gas velocity at the particles: linear along each component's own axis (ghosted faces)."""
    g = n + 2
    xi = [x[d] * (n / L) for d in range(3)]
    c = [t.floor().clamp(0, n - 1) for t in xi]
    at = ((c[2].long() + 1) * g + c[1].long() + 1) * g + c[0].long() + 1
    out = []
    for d in range(3):
        f, w = faces[d].reshape(-1), xi[d] - c[d]
        out.append(w * f[at + g ** d] + (1 - w) * f[at])
    return out


def _box(n, count, gravity, twc, dp_dx=0.1, mass_loading=0.2):
    """The step's scalars for tau_p 0.1, tau_T 0.15 and heating rate 1 in a box of side 2 pi."""
    dp = dp_dx * L / n
    mp = mass_loading * L ** 3 / count
    cvp = 0.15 * 2.0 * PI * dp / mp
    return dict(n=n, l=L, dt=DT, tp=0.1, mp=mp, dp=dp, nu=2.0, k=1.0, epsilonp=1.0,
                i0=mp * cvp / (0.25 * PI * dp * dp), cvp=cvp, gx=0.0, gy=0.0, gz=-0.5 if gravity else 0.0,
                particle_gravity=int(gravity), twc=int(twc))


def _step_inputs(case, seed):
    n, gen = case["n"], _generator(seed)
    faces = [_ghost(u) for u in _velocity(n, gen)]
    temp = _ghost(_temperature(n, gen))
    x = _positions(n, case["count"], case["clustered"], case["blobs"], gen)
    # in mid-run: the particles lag the gas a little
    v = torch.stack(_face_gather(n, x, faces)) * 0.9
    for d in range(3):
        v[d] += 0.05 * torch.randn(case["count"], generator=gen, device=DEVICE, dtype=torch.float64)
    t = 1.0 + 0.02 * torch.rand(case["count"], generator=gen, device=DEVICE, dtype=torch.float64)
    tau = None
    if case["tau_each"]:
        tau = 0.01 * torch.exp(math.log(100.0) * torch.rand(case["count"], generator=gen, device=DEVICE,
                                                            dtype=torch.float64))
    cfg = _box(n, case["count"], case["gravity"], case["twc"], *((0.5, 1.0) if case["correction"] else ()))
    return dict(cfg=cfg, faces=faces, temp=temp, x=x, v=v, t=t, tau=tau)


def _gas_inputs(case, seed):
    n, count, gen = case["n"], case["count"], _generator(seed)
    rng = np.random.default_rng(seed)
    dx = L / n
    if case["quiescent"]:
        # one box of the training runs: isolated particles on a lattice, each held at its slip by a body force
        re_cell = math.exp(rng.uniform(math.log(1.0), math.log(20.0)))
        nu = min(0.05, 0.05 / re_cell) * dx * dx / DT
        k_gas = 3.5 * nu / 0.7
        side = int(round(count ** (1 / 3)))
        sites = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij")).reshape(3, -1) * (n // side)
        x = (sites + n // side // 2 + rng.uniform(0.0, 1.0, (3, count))) * dx
        dp = rng.uniform(0.05, 1.0, count) * dx
        q = rng.uniform(0.0, 2.0, count)
        d = rng.normal(size=(3, count))
        v = re_cell * rng.uniform(0.2, 1.0, count) * nu / dx * d / np.linalg.norm(d, axis=0)
        tau = 1000.0 * dp * dp / (18.0 * nu)
        itth = 2.0 * PI * dp * k_gas
        heat_is = 1.0 / (0.15 * itth)
        props = dict(tau_p=tau, mass_ratio=1000.0 * PI * dp ** 3 / 6.0, itth=itth, heat_is=heat_is, alpha=q / heat_is,
                     accel=list(v / tau))
        cfg = dict(n=n, l=L, dt=DT, tp=1.0, mp=1.0, dp=float(dp.mean()), nu=2.0, k=k_gas, epsilonp=1.0, i0=0.0,
                   cvp=1.0, gx=0.0, gy=0.0, gz=0.0, particle_gravity=0, twc=1)
        zero = torch.zeros((n,) * 3, dtype=torch.float64, device=DEVICE)
        gcfg = dict(mu0=nu, k=k_gas, mp=1.0, epsilon=1e-10, cooling=1)
        return dict(cfg=cfg, gcfg=gcfg, ru=[zero] * 3, rho=zero + 1.0, x=torch.from_numpy(x).to(DEVICE),
                    v=torch.from_numpy(v).to(DEVICE), t=torch.from_numpy(1.0 + 0.15 * q).to(DEVICE), props=props)
    u = _velocity(n, gen)
    x = _positions(n, count, True, 8, gen)
    v = torch.stack(_face_gather(n, x, [_ghost(a) for a in u])) * 0.9
    t = 1.0 + 0.02 * torch.rand(count, generator=gen, device=DEVICE, dtype=torch.float64)
    cfg = _box(n, n ** 3 // 8, False, True)  # mass loading 0.2 at one particle in eight cells
    gcfg = dict(mu0=0.02, k=0.02, mp=cfg["mp"], epsilon=1e-7, cooling=0)
    rho = 1.0 / _temperature(n, gen)
    ru = [0.5 * (rho + torch.roll(rho, 1, 2 - d)) * u[d] for d in range(3)]
    return dict(cfg=cfg, gcfg=gcfg, ru=ru, rho=rho, x=x, v=v, t=t, props=None)


def _gas_config(case, inp):
    c, g = inp["cfg"], inp["gcfg"]
    return dict(n=case["n"], l=L, dt=DT, cp=3.5, cv=2.5, rho0=1.0, u0=0.0, a_force=0.0, gx=0.0, gy=0.0, gz=0.0,
                iterations=30, twc=c["twc"], p0=1.0, **g)


def _table(rows, seed):
    """Normalised features and targets as the training runs record them (in [-1, 1], targets O(1) of them)."""
    gen = torch.Generator().manual_seed(int(seed))
    x = 2.0 * torch.rand((rows, 10), generator=gen) - 1.0
    x[:, 3:6] = torch.nn.functional.normalize(torch.randn((rows, 3), generator=gen), dim=1)
    y = torch.stack([torch.sin(2 * x[:, d]) * (1.0 + 0.5 * x[:, 6]) + 0.3 * x[:, 3 + d] for d in range(3)]
                    + [torch.tanh(x[:, 7]) + 0.5 * x[:, 8] * x[:, 9]], dim=1)
    return x, y


# ---------------------------------------------------------------- prepare and run
class _State:
    """What a program keeps between passes; the handle goes with it."""


def _flags(case):
    return {"storage": 0, "reference": pstep.TRACK_ORDER,
            "sums": pstep.TRACK_ORDER | pstep.REFERENCE_SUMS}[case["order"]]


def _upload(s):
    s.ps.load(*s.x, *s.v, s.t, s.ids)
    if s.tau is not None:
        s.ps.set_tau_p(s.tau)


def _particle_buffers(s, count, by_id):
    s.raw = torch.empty((7, count), dtype=torch.float64, device=DEVICE)
    s.flag = torch.empty(count, dtype=torch.int32, device=DEVICE)
    s.by_id = by_id
    if by_id:
        s.at = torch.empty(count, dtype=torch.int64, device=DEVICE)
        s.out = torch.empty_like(s.raw)


def _read_particles(s):
    """The particle vectors; the mixed form returns them in storage order, so a program files them by id."""
    s.ps.download(*s.raw, s.flag)
    if not s.by_id:
        return s.raw, s.flag
    s.at.copy_(s.flag)
    s.out.scatter_(1, s.at.expand(7, -1), s.raw)
    return s.out, None


def _prepare_step(case, seed):
    inp = _step_inputs(case, seed)
    s = _State()
    s.case, s.faces, s.temp, s.x, s.v, s.t, s.tau = case, inp["faces"], inp["temp"], inp["x"], inp["v"], inp["t"], inp["tau"]
    n, count = case["n"], case["count"]
    fp32 = case["precision"] == "fp32"
    s.ids = torch.arange(count, dtype=torch.int32, device=DEVICE)
    s.ps = pstep.ParticleStep(inp["cfg"], count, pstep.FP32 if fp32 else pstep.FP64, 0 if fp32 else _flags(case))
    if case["correction"]:
        rhop = 6 * inp["cfg"]["mp"] / (PI * inp["cfg"]["dp"] ** 3)
        s.ps.set_correction(learn.load_model(), rhop * inp["cfg"]["dp"] ** 2 / (18 * inp["cfg"]["tp"]))
    _particle_buffers(s, count, fp32)
    s.fields = [torch.empty((n + 2,) * 3, dtype=torch.float64, device=DEVICE) for _ in FIELDS]
    if case["drive"] != "owner":
        _upload(s)
        s.ps.bind_velocity(*s.faces)
        s.ps.bind_temperature(s.temp)
        s.ps.prime()
        s.x = s.v = s.t = s.ids = None
    return s


def _run_step(s):
    ps, drive, means = s.ps, s.case["drive"], []
    if drive == "owner":
        _upload(s)
        ps.bind_velocity(*s.faces)
        ps.bind_temperature(s.temp)
        ps.prime()
    if drive == "staged":
        for k in range(4):
            ps.bind_velocity(*s.faces)
            ps.interp_advance_deposit(k)
            for name, out in zip(FIELDS[:4], s.fields):
                ps.field(name, out)
            ps.wrap()
            ps.bind_temperature(s.temp)
            ps.stage_temp()
            ps.field(FIELDS[4], s.fields[4])
            means.append(ps.energy_mean())
            ps.end_stage()
        ps.end_step()
    else:
        ps.run(1)
        for name, out in zip(FIELDS, s.fields):
            ps.field(name, out)
    arrays, flag = _read_particles(s)
    return {"fields": s.fields, "particles": arrays, "flag": flag, "means": means}


def _prepare_gas(case, seed):
    inp = _gas_inputs(case, seed)
    s = _State()
    s.case = case
    count, fp32 = case["count"], case["precision"] == "fp32"
    s.ps = pstep.ParticleStep(inp["cfg"], count, pstep.FP32 if fp32 else pstep.FP64, 0 if fp32 else pstep.TRACK_ORDER)
    s.ps.load(*inp["x"], *inp["v"], inp["t"], torch.arange(count, dtype=torch.int32, device=DEVICE))
    if inp["props"]:
        s.ps.set_props(**inp["props"])
    s.gas = gas.GasStep(_gas_config(case, inp), s.ps)
    s.gas.init(*[a.cpu().numpy() for a in inp["ru"]], inp["rho"].cpu().numpy())
    _particle_buffers(s, count, fp32)
    s.fields = [torch.empty((case["n"] + 2,) * 3, dtype=torch.float64, device=DEVICE) for _ in GAS_FIELDS]
    return s


def _run_gas(s):
    s.gas.step()
    for name, out in zip(GAS_FIELDS, s.fields):
        s.gas.field_to(name, out.data_ptr())
    arrays, flag = _read_particles(s)
    return {"fields": s.fields, "particles": arrays, "flag": flag, "p0": s.gas.p0()}


def prepare(case, seed):
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    if case["kind"] == "gas":
        return _prepare_gas(case, seed)
    s = _State()
    s.case, s.seed = case, int(seed)
    x, y = _table(case["rows"], seed)
    if case["kind"] == "train":
        s.net = mlp.Mlp(seed=int(seed))
        s.net.set_data(x.numpy(), y.numpy())
    else:
        s.net = mlp.Mlp(seed=int(seed))
        s.x = x.to(DEVICE)
        s.y = torch.empty((case["rows"], 4), dtype=torch.float32, device=DEVICE)
    return s


def run(s):
    kind = s.case["kind"]
    if kind == "step":
        return _run_step(s)
    if kind == "gas":
        return _run_gas(s)
    if kind == "train":
        loss = s.net.train(s.case["steps"], s.case["batch"], 1e-3, s.seed)
        return {"loss": loss, "params": s.net.params}
    s.net._check(s.net.L.pmlp_forward(s.net.h, s.x.data_ptr(), s.case["rows"], s.y.data_ptr(), 1))
    return s.y


def work(case):
    kind = case["kind"]
    if kind == "train":
        rows, per = case["batch"] * case["steps"], 10 * 64 + 64 * 64 + 64 * 4
        return {"bytes": rows * 14 * 4 + case["steps"] * 6 * 4 * 5000, "flops": rows * per * 6}
    if kind == "forward":
        return {"bytes": case["rows"] * 14 * 4, "flops": case["rows"] * 2 * (10 * 64 + 64 * 64 + 64 * 4)}
    n, count = case["n"], case["count"]
    cells, word = (n + 2) ** 3, 4 if case["precision"] == "fp32" else 8
    # particles: seven words, the heating rate and the id in and out, and the vectors that come back
    particle = count * (2 * (8 * word + 4) + 7 * 8 + 4)
    if kind == "gas":
        # four stages: momentum, density, pressure and the deposits in and out
        return {"bytes": particle + 4 * cells * 8 * 2 * 10, "flops": count * 1000 + 4 * cells * 400}
    stages = 4 if case["drive"] == "staged" else 1
    flops = count * 4 * 260 + (count * 2 * (10 * 64 + 64 * 64 + 64 * 4) if case["correction"] else 0)
    return {"bytes": particle + stages * cells * (4 * word + 5 * 8), "flops": flops}


# ---------------------------------------------------------------- the same results in 64 bits
class _Particles:
    """The particle stage of the solver in plain 64-bit torch (periodic box, one rank)."""

    def __init__(self, cfg, x, v, t, tau=None, props=None):
        n = cfg["n"]
        self.c, self.n, self.g = cfg, n, n + 2
        self.base = [*x, *v, t]
        dev = dict(dtype=torch.float64, device=x.device)
        p = {k: torch.as_tensor(np.asarray(a), **dev) for k, a in (props or {}).items() if k != "accel"}
        self.itp = 1.0 / (tau if tau is not None else p["tau_p"] if props else torch.tensor(cfg["tp"], **dev))
        self.mass = p.get("mass_ratio", 1.0)
        self.itth = p.get("itth", cfg["nu"] * PI * cfg["dp"] * cfg["k"])
        self.heat = p.get("heat_is", 1.0 / (cfg["mp"] * cfg["cvp"]))
        self.alpha = p.get("alpha", 0.25 * cfg["epsilonp"] * PI * cfg["dp"] ** 2 * cfg["i0"])
        grav = [cfg["particle_gravity"] * cfg[k] for k in ("gx", "gy", "gz")]
        self.acc = [torch.as_tensor(a, **dev) for a in props["accel"]] if props else grav

    def node(self, x):
        xi = [a * (self.n / L) for a in x]
        r = [(a + 0.5).floor() for a in xi]
        w = [a - b + 0.5 for a, b in zip(xi, r)]
        return ((r[2].long() + 1) * self.g + r[1].long() + 1) * self.g + r[0].long() + 1, w

    def corners(self, x):
        at, w = self.node(x)
        for o in range(8):
            o3 = (o & 1, (o >> 1) & 1, o >> 2)
            f = [(1 - w[d]) if o3[d] else w[d] for d in range(3)]
            yield at - (o3[0] + self.g * (o3[1] + self.g * o3[2])), f[0] * f[1] * f[2]

    def heating(self, x, t, temp):
        flat = temp.reshape(-1)
        return (sum(w * flat[at] for at, w in self.corners(x)) - t) * self.itth

    def prime(self, temp):
        self.now, self.np1 = list(self.base), list(self.base)
        self.rhs_t = self.heating(self.base[:3], self.base[6], temp)

    def stage(self, k, faces, temp):
        pre, post, cur = DT * PRE[k], DT * POST[k], self.now
        ug = _face_gather(self.n, cur[:3], faces)
        self.rhs = [(ug[d] - cur[3 + d]) * self.itp for d in range(3)]
        rate = cur[3:6] + [self.rhs[d] + self.acc[d] for d in range(3)] + [(self.rhs_t + self.alpha) * self.heat]
        self.np1 = [a + post * r for a, r in zip(self.np1, rate)]
        new = list(self.np1) if k == 3 else [b + pre * r for b, r in zip(self.base, rate)]
        self.dep = cur[:3]
        for d in range(3):
            over = (new[d] < 0).double() - (new[d] > L).double()
            new[d], self.np1[d] = new[d] + L * over, self.np1[d] + L * over
            self.base[d] = self.base[d] + L * over
        self.rhs_t = self.heating(new[:3], new[6], temp)
        self.now = new

    def end_step(self):
        self.base, self.now = list(self.np1), list(self.np1)

    def deposit(self, x, val):
        f = torch.zeros(self.g ** 3, dtype=torch.float64, device=x[0].device)
        for at, w in self.corners(x):
            f.index_add_(0, at, w if val is None else w * val)
        return f.view(self.g, self.g, self.g)

    def momentum(self, d):
        f = torch.zeros(self.g ** 3, dtype=torch.float64, device=self.dep[0].device)
        xi = [a * (self.n / L) for a in self.dep]
        c = [a.floor().clamp(0, self.n - 1) for a in xi]
        at = ((c[2].long() + 1) * self.g + c[1].long() + 1) * self.g + c[0].long() + 1
        r, w = self.rhs[d] * self.mass, xi[d] - c[d]
        f.index_add_(0, at, (1 - w) * r)
        f.index_add_(0, at + self.g ** d, w * r)
        return f.view(self.g, self.g, self.g)

    @staticmethod
    def fold(f):
        """What lies in the ghost layers goes to its periodic image, z first; the layers keep their partial sums."""
        inner = slice(1, -1)
        f[-2], f[1] = f[-2] + f[0], f[1] + f[-1]
        f[inner, -2], f[inner, 1] = f[inner, -2] + f[inner, 0], f[inner, 1] + f[inner, -1]
        f[inner, inner, -2], f[inner, inner, 1] = (f[inner, inner, -2] + f[inner, inner, 0],
                                                   f[inner, inner, 1] + f[inner, inner, -1])
        return f

    def fields(self, partial_ghosts):
        c = self.fold(self.deposit(self.dep, None))
        out = [c if partial_ghosts else _ghost(c[1:-1, 1:-1, 1:-1])]
        for d in range(3):
            out.append(_ghost(self.fold(self.momentum(d))[1:-1, 1:-1, 1:-1]) if self.c["twc"] else torch.zeros_like(c))
        out.append(_ghost(self.fold(self.deposit(self.now[:3], self.rhs_t))[1:-1, 1:-1, 1:-1]))
        return out


def _exact_step(case, seed):
    if case["correction"] or case["count"] > 1 << 25:
        return None  # the corrected gas values are the 16-bit network's; the largest population takes too long
    inp = _step_inputs(case, seed)
    fp32 = case["precision"] == "fp32"
    p = _Particles(inp["cfg"], inp["x"], inp["v"], inp["t"], inp["tau"])
    p.prime(inp["temp"])
    means = []
    for k in range(4):
        p.stage(k, inp["faces"], inp["temp"])
        if case["drive"] == "staged":
            means.append(float(p.rhs_t.sum()) / case["n"] ** 3)
    fields = p.fields(not fp32)
    p.end_step()
    # in the solver's own particle order the vectors have a value here only by id
    return {"fields": fields, "particles": torch.stack(p.base) if fp32 else None, "flag": None, "means": means}


def _exact_gas(case, seed):
    inp = _gas_inputs(case, seed)
    c, n = _gas_config(case, inp), case["n"]
    idx, vcell, gas_r = n / L, (L / n) ** 3, c["cp"] - c["cv"]
    up = lambda a, d: torch.roll(a, -1, 2 - d)  # noqa: E731
    down = lambda a, d: torch.roll(a, 1, 2 - d)  # noqa: E731
    face = lambda a, d: (a + down(a, d)) * 0.5  # noqa: E731
    grad = lambda a: [(a - down(a, d)) * idx for d in range(3)]  # noqa: E731
    div = lambda f: sum((up(f[d], d) - f[d]) * idx for d in range(3))  # noqa: E731
    del2 = lambda a: sum((up(a, d) - 2 * a + down(a, d)) * idx * idx for d in range(3))  # noqa: E731
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=DEVICE)
    one = 2.0 * idx * idx * (1 - torch.cos(k * (2 * PI / n)))
    den = one[:, None, None] + one[None, :, None] + one[None, None, :]
    den[0, 0, 0] = 1.0
    ru, rho = list(inp["ru"]), inp["rho"]
    ru_int, ru_np1, rho_np1, pres = list(ru), list(ru), rho, torch.zeros_like(rho)
    p0 = p0_np1 = c["p0"]
    rho_face = [face(rho, d) for d in range(3)]
    part = _Particles(inp["cfg"], inp["x"], inp["v"], inp["t"], None, inp["props"])
    part.prime(_ghost(p0 / gas_r / rho))
    inner = slice(1, -1)
    heat = part.fold(part.deposit(part.base[:3], part.rhs_t))[inner, inner, inner]
    for s in range(4):
        pre, post = DT * PRE[s], DT * POST[s]
        rate = div(ru_int)
        rho_np1 = rho_np1 - post * rate
        rho_new = rho_np1 if s == 3 else rho - pre * rate
        dp0 = 0.0 if c["cooling"] else -gas_r / c["cv"] * float(heat.mean())
        p0_np1 += post * dp0
        p0_new = p0_np1 if s == 3 else p0 + pre * dp0
        u = [ru_int[d] / rho_face[d] for d in range(3)]
        temp = p0_new / gas_r / rho_new
        part.stage(s, [_ghost(a) for a in u], _ghost(temp))
        _, fx, fy, fz, heat = [a[inner, inner, inner] for a in part.fields(False)]
        dil = grad(div(u))
        rhs = [-c["mp"] / vcell * f + c["mu0"] / 3.0 * dil[d] + c["mu0"] * del2(u[d]) for d, f in enumerate((fx, fy, fz))]
        for e in range(3):
            rhs[e] = rhs[e] - div([face(u[e], d) * face(ru_int[d], e) for d in range(3)])
        ru_np1 = [a + post * r for a, r in zip(ru_np1, rhs)]
        ru_new = list(ru_np1) if s == 3 else [a + pre * r for a, r in zip(ru, rhs)]
        source = heat - heat.mean() if c["cooling"] else heat
        dil = c["k"] / c["cp"] * del2(1.0 / rho_new) - gas_r / (c["cp"] * p0_new * vcell) * source
        rho_face = [face(rho_new, d) for d in range(3)]
        pois = (div([ru_new[d] / rho_face[d] for d in range(3)]) - dil) / pre
        pois = pois - pois.mean()
        coef = [1.0 / a for a in rho_face]
        centre = -1.0 / (sum((coef[d] + up(coef[d], d)) * 0.5 for d in range(3)) / 3.0)
        for _ in range(c["iterations"]):
            g = grad(pres)
            r = (div([g[d] * coef[d] for d in range(3)]) - pois) * centre
            add = -torch.fft.ifftn(torch.fft.fftn(r) / den).real
            pres = pres + add
            if float(add.abs().max()) <= c["epsilon"]:
                break
        g = grad(pres)
        ru_np1 = [a - post * b for a, b in zip(ru_np1, g)]
        ru_new = list(ru_np1) if s == 3 else [a - pre * b for a, b in zip(ru_new, g)]
        ru_int = ru_new
    part.end_step()
    ru = [a - a.mean() for a in ru_np1]
    fields = [_ghost(a) for a in (*ru, rho_np1, pres, temp, heat)]
    return {"fields": fields, "particles": torch.stack(part.base) if case["precision"] == "fp32" else None,
            "flag": None, "p0": p0_np1}


def _network(p, x):
    z = x @ p[0].T + p[1]
    z = torch.nn.functional.silu(z) @ p[2].T + p[3]
    return torch.nn.functional.silu(z) @ p[4].T + p[5]


def _weights(flat):
    """The layers of a parameter table (padding left out)."""
    f = torch.from_numpy(flat.astype(np.float64)).to(DEVICE)
    return [f[:1024].view(64, 16)[:, :10].clone(), f[1024:1088].clone(), f[1088:5184].view(64, 64).clone(),
            f[5184:5248].clone(), f[5248:6272].view(16, 64)[:4].clone(), f[6272:6276].clone()]


def _mix(z):
    with np.errstate(over="ignore"):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _first_weights(seed):
    """The start values: uniform in +-1/sqrt(fan_in), drawn one after the other from the seed."""
    flat, s = np.zeros(6288, dtype=np.float32), np.array([seed], dtype=np.uint64)
    a1, a2 = np.float64(np.float32(1) / np.sqrt(np.float32(10))), np.float64(0.125)
    at = [(o * 16 + j, a1) for o in range(64) for j in range(10)] + [(1024 + o, a1) for o in range(64)]
    at += [(1088 + e, a2) for e in range(4096 + 64)] + [(5248 + e, a2) for e in range(256)]
    at += [(6272 + o, a2) for o in range(4)]
    for place, bound in at:
        s = _mix(s)
        flat[place] = (2.0 * (float(s[0] >> np.uint64(11)) / 9007199254740992.0) - 1.0) * bound
    return flat


def _exact_train(case, seed):
    x, y = (a.double().to(DEVICE) for a in _table(case["rows"], seed))
    p = [a.requires_grad_(True) for a in _weights(_first_weights(seed))]
    opt = torch.optim.Adam(p, lr=1e-3, betas=(0.9, 0.999), eps=1e-8)
    slot = np.arange(case["batch"], dtype=np.uint64)
    loss = []
    for step in range(case["steps"]):
        with np.errstate(over="ignore"):
            h = _mix(np.uint64(seed) ^ _mix(np.uint64(step) * np.uint64(0x100000001) + slot))
        row = torch.from_numpy((h % np.uint64(case["rows"])).astype(np.int64)).to(DEVICE)
        opt.zero_grad()
        err = (_network(p, x[row]) - y[row]).square().mean()
        err.backward()
        opt.step()
        loss.append(float(err.detach()))
    flat = torch.zeros(6288, dtype=torch.float64, device=DEVICE)
    flat[:1024].view(64, 16)[:, :10] = p[0].detach()
    flat[1024:1088], flat[1088:5184], flat[5184:5248] = p[1].detach(), p[2].detach().reshape(-1), p[3].detach()
    flat[5248:6272].view(16, 64)[:4] = p[4].detach()
    flat[6272:6276] = p[5].detach()
    return {"loss": torch.tensor(loss, dtype=torch.float64), "params": flat}


def exact(case, seed):
    if case["kind"] == "step":
        return _exact_step(case, seed)
    if case["kind"] == "gas":
        return _exact_gas(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    x, _ = _table(case["rows"], seed)
    return _network(_weights(_first_weights(seed)), x.double().to(DEVICE))
