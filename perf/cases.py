"""The workloads by which this framework's speed is judged.

Every case is a piece of work that a user's program has the framework do,
through the public entry points (``rot2d3c_gb300``, its closure and its torch
operator): RK4 steps of one run at the grid sizes of the reference's
configurations, in both precisions; a batch of uneven runs; the diagnostics of
one output time; the large-eddy run with the learned closure; the closure
network's training and its vector-Jacobian product; and the layout-compatible
2-D transforms.  ``listed`` gives the twelve fixed ones, ``draw`` another one of
the same ranges, ``exact`` the results of plain torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import rot2d3c_gb300 as R
from rot2d3c_gb300 import closure as CL
from rot2d3c_gb300.torch_ops import ClosureNet

CIN = [8, 32, 32, 32, 32, 32]
COUT = [32, 32, 32, 32, 32, 2]


def listed():
    return [
        # the reference's 256^2 configuration in FP64: a short, latency-bound run between two outputs
        dict(name="step_f64_256", kind="step", n=256, prec=64, steps=20, cfl=0.5, iflow=0, nu=1e-3, omega=1.0),
        # the reference's default forcing (random in time, iflow 3) on a mid-size FP64 grid
        dict(name="step_f64_1024_rand", kind="step", n=1024, prec=64, steps=7, cfl=0.5, iflow=3, nu=5e-5, omega=1.0),
        # the drop-in path at production size, one step per call, fixed time step
        dict(name="step_f64_4096", kind="step", n=4096, prec=64, steps=1, cfl=0.0, iflow=0, nu=1e-5, omega=10.0),
        # the direct simulation that the closure is trained on
        dict(name="step_f32_2048", kind="step", n=2048, prec=32, steps=10, cfl=0.5, iflow=0, nu=2e-5, omega=1.0),
        # the FP32 path at production size
        dict(name="step_f32_4096", kind="step", n=4096, prec=32, steps=5, cfl=0.0, iflow=0, nu=1e-5, omega=10.0),
        # the largest grid that the framework takes
        dict(name="step_f32_8192", kind="step", n=8192, prec=32, steps=2, cfl=0.5, iflow=0, nu=5e-6, omega=10.0),
        # all diagnostics of one output time: budgets, spectrum, transfers, a physical field
        dict(name="diag_f64_2048", kind="diag", n=2048, prec=64, nu=2e-5, omega=1.0),
        # a parameter study: runs of three sizes advanced together, their states read at the end
        dict(name="ensemble_f32", kind="ensemble", groups="256x12,512x5,1024x2", prec=32, steps=100, cfl=0.5),
        # the large-eddy run with the network before every second step
        dict(name="les_256", kind="les", n=256, steps=20, every=2, cfl=0.5),
        # one training step of the closure network at its usual batch
        dict(name="cnn_train_256_b32", kind="train", h=256, w=256, batch=32),
        # the network inside a torch program, on a grid that no tile size divides evenly
        dict(name="cnn_vjp_72x112_b3", kind="vjp", h=72, w=112, batch=3),
        # the layout-compatible transforms on device buffers, there and back
        dict(name="fft_f64_2048", kind="fft", n=2048, prec=64),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "step", "diag", "ensemble", "les", "train", "vjp", "fft"])
    prec = rng.choice([64, 32])
    if kind == "step":
        n = 2 ** rng.randint(4, 12 if prec == 64 else 13)
        # no more work than the listed 4096^2 FP64 step or the two 8192^2 FP32 steps
        most = max(1, min(40, (4096 if prec == 64 else 11585) ** 2 // n ** 2))
        return dict(kind=kind, n=n, prec=prec, steps=rng.randint(1, most), cfl=rng.choice([0.0, 0.3, 0.5]),
                    iflow=rng.choice([0, 0, 3]), nu=round(0.2 * n ** -1.3, 8), omega=round(rng.uniform(0, 20), 3))
    if kind == "diag":
        n = 2 ** rng.randint(5, 11)
        return dict(kind=kind, n=n, prec=prec, nu=round(0.2 * n ** -1.3, 8), omega=round(rng.uniform(0, 20), 3))
    if kind == "ensemble":
        top = rng.randint(6, 9)
        groups = ",".join("%dx%d" % (2 ** (top - i), rng.randint(1, 9) * 2 ** i) for i in range(rng.randint(1, 3)))
        return dict(kind=kind, groups=groups, prec=prec, steps=rng.randint(5, 40), cfl=rng.choice([0.3, 0.5]))
    if kind == "les":
        every = rng.choice([1, 2, 3])
        return dict(kind=kind, n=2 ** rng.randint(6, 9), steps=every * rng.randint(2, 8), every=every,
                    cfl=rng.choice([0.3, 0.5]))
    if kind in ("train", "vjp"):
        if rng.random() < 0.5:  # square grids of a large-eddy run
            h = w = rng.choice([64, 128, 256])
        else:
            h, w = 8 * rng.randint(2, 30), 16 * rng.randint(1, 20)
        return dict(kind=kind, h=h, w=w, batch=rng.randint(1, max(1, min(31, 2_000_000 // (h * w)))))
    return dict(kind="fft", n=2 ** rng.randint(4, 12), prec=prec)


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _wave(n):
    """(kx [n/2+1, 1], ky [1, n]) of a spectral plane [kx][ky]."""
    ka = torch.cat([torch.arange(n // 2), torch.arange(n // 2) - n // 2]).double().cuda()
    kx = ka[: n // 2 + 1].clone()
    return kx[:, None], ka[None, :]


def _two(n):
    two = torch.full((n // 2 + 1, 1), 2.0, dtype=torch.float64, device="cuda")
    two[0] = 1.0
    return two


def _field(n, kmin, kmax, slope, kin, energy, gen):
    """A random-phase field with |a(k)| ~ k**slope on kmin <= |k| <= kmax and
    sum(two ka2**kin |a|^2)/n^4 = energy, Hermitian on kx = 0."""
    kx, ky = _wave(n)
    k2 = kx ** 2 + ky ** 2
    on = (k2 >= kmin * kmin) & (k2 <= kmax * kmax)
    amp = torch.where(on, k2.clamp(min=1.0) ** (0.5 * slope), 0.0)
    a = torch.polar(amp, 2 * math.pi * torch.rand(k2.shape, dtype=torch.float64, device="cuda", generator=gen))
    j = torch.arange(1, n // 2, device="cuda")
    a[0, n - j] = a[0, j].conj()
    a[0, 0] = 0.0
    a[0, n // 2] = 0.0
    a[n // 2] = 0.0
    e = (_two(n) * k2 ** kin * a.abs() ** 2).sum() / float(n) ** 4
    return a * torch.sqrt(energy / e)


def _fields(n, seed, kmax=None):
    """psi, vz with kinetic energies 1/2 and spectra up to the dealiasing
    cutoff (or kmax), and a forcing of unit energy around shell 5."""
    g = _gen(seed)
    kmax = min(kmax or n, n / 3.0)
    f1 = min(6.0, n / 4.0)
    return (_field(n, 1.0, kmax, -3.0, 1, 0.5, g), _field(n, 1.0, kmax, -2.0, 0, 0.5, g),
            _field(n, f1 - 2.0, f1, 0.0, 1, 1.0, g), _field(n, f1 - 2.0, f1, 0.0, 0, 1.0, g))


def _params(n, nu, omega, iflow=0, cfl=0.5):
    kup = min(6.0, n // 4)
    return dict(n=n, nu=nu, nuv=nu, hnu=0.1, hnuv=0.1, nn=1, mm=2, nnv=1, mmv=2, omega=omega, iflow=iflow,
                cfl=cfl or 0.5, kup=kup, kdn=kup, fp0=0.02, fz0=0.02)


def _prec(case):
    return R.FP64 if case["prec"] == 64 else R.FP32


def _host(*t):
    return [x.cpu().numpy() for x in t]


class _Dev:
    """A context's device plane as torch sees it; holds the context, whose
    memory it is, for as long as a tensor of it lives."""

    def __init__(self, ctx, which):
        self.ctx = ctx
        self.__cuda_array_interface__ = dict(shape=(ctx.n // 2 + 1, ctx.n), version=3, strides=None,
                                             typestr="<c16" if ctx.precision == R.FP64 else "<c8",
                                             data=(ctx.dev_ptr(which), False))


def _plane(ctx, which):
    owner = _Dev(ctx, which)
    t = torch.as_tensor(owner, device="cuda")
    t.owner = owner
    return t


def _fixed_dt(n):
    return min(1e-3, 0.4096 / n)


def _case_fields(case, seed):
    # the production-size fixed-step runs start from scales up to shell 100, the others from a full spectrum
    return _fields(case["n"], seed, 100.0 if case.get("cfl") == 0.0 else None)


def _context(case, seed):
    ps, vz, fp, fz = _host(*_case_fields(case, seed))
    p = _params(case["n"], case["nu"], case["omega"], case.get("iflow", 0), case.get("cfl", 0.5))
    c = R.Context(R.make_params(**p), _prec(case))
    c.set_state(ps, vz)
    if p["iflow"] == 0:
        c.set_forcing(fp, fz)
    c.set_time(0.0)
    return c, p


def _groups(case):
    return [tuple(int(v) for v in g.split("x")) for g in case["groups"].split(",")]


def _run_params(case, i, n):
    return _params(n, 0.2 * n ** -1.3 * (1 + 0.1 * (i % 5)), 0.5 * (i % 7))


def _net_params(seed):
    """The network's parameter vector: layer by layer weights [9][cin][cout], biases [cout]."""
    g = _gen(seed)
    out = []
    for l, (ci, co) in enumerate(zip(CIN, COUT)):
        b = math.sqrt(6.0 / (9 * ci))
        out.append((torch.rand(9 * ci * co, device="cuda", generator=g) * 2 - 1) * b)
        out.append((torch.rand(co, device="cuda", generator=g) - 0.5) * 0.1)
    return torch.cat(out)


def _net_batch(case, seed):
    """Inputs and targets of the closure network: smooth fields and noise of
    different magnitudes per channel, as its eight channels have."""
    g = _gen(seed)
    b, h, w = case["batch"], case["h"], case["w"]
    scale = torch.tensor([20.0, 1.0, 1.0, 1.0, 400.0, 400.0, 15.0, 15.0], device="cuda")
    x = torch.randn((b, h, w, 8), device="cuda", generator=g)
    x = (x + x.roll(1, 1) + x.roll(1, 2) + x.roll(2, 1)) / 2 * scale
    y = torch.randn((b, h, w, 2), device="cuda", generator=g) * torch.tensor([30.0, 2.0], device="cuda")
    y = y + x[..., :2] * torch.tensor([1.0, 2.0], device="cuda")
    norm = (np.zeros(8, np.float32), scale.cpu().numpy(), np.zeros(2, np.float32), np.array([36.0, 2.8], np.float32))
    return x, y, norm


def _les_norm(ps, vz, n):
    """Mean and spread of the network's inputs and outputs for a large-eddy run, from its first state."""
    x = _inputs64(ps, vz, n)
    sd = x.reshape(-1, 8).std(0).float().cpu().numpy()
    return np.zeros(8, np.float32), sd, np.zeros(2, np.float32), np.array([0.5, 0.05], np.float32) * sd[:2]


def _band(n):
    kc = n // 3
    w = np.zeros((2, n // 2 + 1), np.float32)
    w[:, 2 * kc // 3:kc + 1] = 1.0
    return w


# ------------------------------------------------------------------ the work
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "step":
        c, _ = _context(case, seed)
        s.update(ctx=c, psi=_plane(c, 0), vz=_plane(c, 1), seed=[int(seed) % 30011 + 1], seed1=[0])
        if case["iflow"] == 3:
            c.forcing_init(s["seed"], s["seed1"])
    elif kind == "diag":
        s["ctx"], _ = _context(case, seed)
    elif kind == "ensemble":
        groups, i = [], 0
        for n, runs in _groups(case):
            groups.append((n, [R.make_params(**_run_params(case, i + r, n)) for r in range(runs)]))
            i += runs
        e = R.Ensemble(groups, _prec(case))
        for r, n in enumerate(e.ns):
            ps, vz, fp, fz = _host(*_fields(n, seed * 1000 + r))
            e.set_state(r, ps, vz)
            e.set_forcing(r, fp, fz)
            e.set_time(r, 0.0)
        s["ens"] = e
    elif kind == "les":
        n = case["n"]
        f = _fields(n, seed)
        c = R.Context(R.make_params(**_params(n, 2e-5, 1.0)), R.FP32)
        ps, vz, fp, fz = _host(*f)
        c.set_state(ps, vz)
        c.set_forcing(fp, fz)
        c.set_time(0.0)
        net = CL.CNN(n, n, 1, 1)
        net.set_params(_net_params(seed).cpu().numpy())
        net.set_normalization(*_les_norm(f[0], f[1], n))
        CL.set_band(c, _band(n))
        s.update(ctx=c, net=net, psi=_plane(c, 0), vz=_plane(c, 1))
    elif kind == "train":
        x, y, norm = _net_batch(case, seed)
        net = CL.CNN(case["h"], case["w"], case["batch"], 1)
        net.set_params(_net_params(seed).cpu().numpy())
        net.set_normalization(*norm)
        for k in range(2):  # the optimiser's moments, as a running training has them
            net.train_step(x.roll(k + 1, 1), y.roll(k + 1, 1), case["batch"], 5e-4)
        s.update(net=net, x=x, y=y)
    elif kind == "vjp":
        x, y, norm = _net_batch(case, seed)
        m = ClosureNet(case["h"], case["w"], case["batch"], 1)
        m.set_normalization(*norm)
        with torch.no_grad():
            m.params.copy_(_net_params(seed))
        s.update(model=m, x=x.requires_grad_(True), gout=y / 1000)
    else:
        n = case["n"]
        s.update(x=torch.randn((n, n), dtype=torch.float64, device="cuda", generator=_gen(seed)),
                 stream=torch.cuda.Stream(),
                 fwd=R.FFTPlan(n, R.R2C, _prec(case)), inv=R.FFTPlan(n, R.C2R, _prec(case)),
                 spec=torch.empty((n // 2 + 1, n), dtype=torch.complex128, device="cuda"),
                 back=torch.empty((n, n), dtype=torch.float64, device="cuda"))
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        mode, v = (R.DT_CFL, case["cfl"]) if case["cfl"] else (R.DT_FIXED, _fixed_dt(case["n"]))
        t, dt = s["ctx"].advance(case["steps"], mode, v, s["seed"], s["seed1"])
        return dict(psi=s["psi"], vz=s["vz"], time=t, dt=dt)
    if kind == "diag":
        c = s["ctx"]
        b = c.cond_check(0.0)
        ek, ezk = c.spectrum()
        return dict(budget=b[:25], extrema=b[25:], ek=ek, ezk=ezk, transfers=np.stack(c.transfers()),
                    vorticity=c.get_field(R.FIELD_WW))
    if kind == "ensemble":
        e = s["ens"]
        t = e.advance(case["steps"], R.DT_CFL, case["cfl"])
        return dict(times=t, states=[v for r in range(e.nruns) for v in e.get_state(r)])
    if kind == "les":
        t, dt = CL.closure_advance(s["ctx"], s["net"], case["steps"], R.DT_CFL, case["cfl"], every=case["every"])
        return dict(psi=s["psi"], vz=s["vz"], time=t, dt=dt)
    if kind == "train":
        loss = s["net"].train_step(s["x"], s["y"], case["batch"], 5e-4)
        return dict(loss=loss, params=s["net"].get_params())
    if kind == "vjp":
        m, x = s["model"], s["x"]
        out = m(x)
        gx, gp = torch.autograd.grad(out, (x, m.params), s["gout"])
        return dict(out=out.detach(), gx=gx, gp=gp)
    st = s["stream"].cuda_stream
    s["fwd"].r2c_dev(s["x"].data_ptr(), s["spec"].data_ptr(), st)
    s["inv"].c2r_dev(s["spec"].data_ptr(), s["back"].data_ptr(), st)
    return dict(spec=s["spec"], back=s["back"])


def _step_work(n, prec):
    """One RK4 step: per substep 8 M column and 4 n row transforms (two real
    rows to a complex one; 5 n log2 n operations each); the state read and
    written once and the forcing read once, on the retained modes."""
    m = n // 3 + 1
    flops = 4 * (8 * m + 4 * n) * 5 * n * math.log2(n)
    return 6 * m * (2 * (n // 3) + 1) * (16 if prec == 64 else 8), flops


def work(case):
    kind = case["kind"]
    if kind == "step":
        b, f = _step_work(case["n"], case["prec"])
        return dict(bytes=b, flops=f * case["steps"])
    if kind == "ensemble":
        b = f = 0.0
        for n, runs in _groups(case):
            sb, sf = _step_work(n, case["prec"])
            # the states also go to the host in 64 bits
            b += runs * (sb + 2 * (n // 2 + 1) * n * 16)
            f += runs * sf * case["steps"]
        return dict(bytes=b, flops=f)
    if kind == "diag":
        n = case["n"]
        c = (n // 2 + 1) * n * (16 if case["prec"] == 64 else 8)
        # psi, vz, fp, fz read; the field out in 64 bits; two brackets, two extrema and one field of transforms
        return dict(bytes=4 * c + 8 * n * n, flops=(8 * (n // 3 + 1) + 4 * n + 3 * n) * 5 * n * math.log2(n))
    macs = 9 * sum(a * b for a, b in zip(CIN, COUT))
    if kind == "les":
        n = case["n"]
        b, f = _step_work(n, 32)
        evals = case["steps"] // case["every"]
        return dict(bytes=b, flops=f * case["steps"] + evals * (2 * macs * n * n + 10 * n * 5 * n * math.log2(n)))
    if kind in ("train", "vjp"):
        px = case["batch"] * case["h"] * case["w"]
        nparam = macs + sum(COUT)
        # inputs, targets or output gradients; parameters, moments; output and input gradients of the vjp
        return dict(bytes=px * (40 if kind == "train" else 80) + nparam * (24 if kind == "train" else 8),
                    flops=6.0 * macs * px)
    n = case["n"]
    return dict(bytes=8 * (2 * n * n + 4 * (n // 2 + 1) * n), flops=2 * (n // 2 + n // 2 + 1) * 5 * n * math.log2(n))


# ------------------------------------------------------------------ the same in plain torch, 64 bits
def _c2r(a, n):
    return torch.fft.irfft(torch.fft.ifft(a, dim=-1), n=n, dim=-2) * float(n) ** 2  # [x][y]


def _r2c(r):
    return torch.fft.fft(torch.fft.rfft(r, dim=-2), dim=-1)


class _Solver:
    """The RK4 step on states [..., kx, ky] (a batch of runs of one n with
    their own coefficients)."""

    def __init__(self, plist):
        p0 = plist[0]
        self.n = n = p0["n"]
        self.kx, self.ky = _wave(n)
        self.k2 = self.kx ** 2 + self.ky ** 2
        self.mask = self.k2 <= (n / 3.0) ** 2
        self.keep = self.mask & (self.k2 >= 1)
        k2 = self.k2.clamp(min=1.0)
        self.ik2 = 1.0 / k2

        def col(key):
            return torch.tensor([p[key] for p in plist], dtype=torch.float64, device="cuda")[:, None, None]
        self.w2 = 2 * col("omega")
        self.d1 = col("nu") * k2 ** p0["nn"] + col("hnu") * self.ik2 ** p0["mm"]
        self.d2 = col("nuv") * k2 ** p0["nnv"] + col("hnuv") * self.ik2 ** p0["mmv"]
        kc = n / 3.0
        self.visc = (col("nu") * kc ** (2 * p0["nn"]) + col("nuv") * kc ** (2 * p0["nnv"]) + self.w2).reshape(-1)

    def grad(self, a):
        a = torch.where(self.mask, a, 0.0)
        return _c2r(1j * self.kx * a, self.n), _c2r(1j * self.ky * a, self.n)

    def brackets(self, a, b):
        ax, ay = self.grad(a)
        wx, wy = self.grad(-self.k2 * a)
        bx, by = self.grad(b)
        s = 1.0 / float(self.n) ** 4
        return _r2c((ax * wy - ay * wx) * s), _r2c((ax * by - ay * bx) * s)

    def dt(self, psi, cfl):
        ax, ay = self.grad(psi)
        u = (ax * ax + ay * ay).flatten(-2).amax(-1).sqrt() / float(self.n) ** 2
        return cfl / (self.n / 3.0 * u + self.visc)

    def step(self, psi, vz, fp, fz, dt, tau=None):
        c1, c2 = psi, vz
        for o in (4, 3, 2, 1):
            h = (dt / o)[:, None, None]
            b5, b6 = self.brackets(c1, c2)
            if tau is not None:
                b5, b6 = b5 + tau[0], b6 + tau[1]
            d1, d2 = 1j * self.ky * c1, 1j * self.ky * c2
            n1 = (psi + ((-b5 + self.w2 * d2) * self.ik2 + fp) * h) / (1 + self.d1 * h)
            n2 = (vz + (b6 + self.w2 * d1 + fz) * h) / (1 + self.d2 * h)
            c1, c2 = torch.where(self.keep, n1, 0.0), torch.where(self.keep, n2, 0.0)
        return c1, c2


def _randu(seed):
    """The reference's generator: (new seed, draw in [-1, 1))."""
    mask = 123459876
    s = seed ^ mask
    k = int(s / 127773)
    s = 16807 * (s - k * 127773) - 2836 * k
    s = (s + 2 ** 31) % 2 ** 32 - 2 ** 31
    if s < 0:
        s += 2147483647
    r = (np.float32(1.0) / np.float32(2147483647)) * np.float32(s)
    return s ^ mask, float((r - np.float32(0.5)) * np.float32(2.0))


def _rand_force(p, f0, kin, dt, seed):
    """(forcing plane, new seed) of one draw of the random forcing."""
    n = p["n"]
    seed, r = _randu(seed)
    theta = r * math.pi
    phase = _randu(seed + 1)[1] * math.pi
    kx, ky = math.floor(p["kup"] * math.cos(theta) + 0.5), math.floor(p["kup"] * math.sin(theta) + 0.5)
    amp = math.sqrt(2 * f0) / (math.sqrt(dt) * p["kup"] ** kin) * float(n) ** 2
    v = complex(amp * math.cos(phase), amp * math.sin(phase))
    f = torch.zeros((n // 2 + 1, n), dtype=torch.complex128, device="cuda")
    if ky != 0 and -n // 2 <= kx < n // 2:
        f[abs(ky), kx % n] = v
    elif ky == 0 and 1 <= kx < n // 2:
        f[0, kx], f[0, n - kx] = v, v.conjugate()
    return f, seed


def _inputs64(ps, vz, n):
    """The network's inputs [n][n][8] of a state."""
    kx, ky = _wave(n)
    k2 = kx ** 2 + ky ** 2
    m = k2 <= (n / 3.0) ** 2
    w = k2 * ps
    f = [w, vz * m, 1j * kx * ps * m, 1j * ky * ps * m, 1j * kx * w * m, 1j * ky * w * m, 1j * kx * vz * m,
         1j * ky * vz * m]
    return torch.stack([_c2r(v, n).T / float(n) ** 2 for v in f], -1)


def _net64(x, params):
    """The network on standardised inputs [b][h][w][8]."""
    off = 0
    for l, (ci, co) in enumerate(zip(CIN, COUT)):
        w = params[off:off + 9 * ci * co].reshape(9, ci, co)
        b = params[off + 9 * ci * co:off + 9 * ci * co + co]
        off += 9 * ci * co + co
        y = b
        for t in range(9):
            y = y + x.roll((1 - t // 3, 1 - t % 3), (1, 2)) @ w[t]
        x = torch.nn.functional.gelu(y) if l < 5 else y
    return x


def _dev64(a):
    return torch.as_tensor(np.asarray(a), device="cuda").double()


def _exact_step(case, seed):
    p = _params(case["n"], case["nu"], case["omega"], case["iflow"], case["cfl"])
    psi, vz, fp, fz = (v[None] for v in _case_fields(case, seed))
    sv = _Solver([p])
    t, dt = 0.0, torch.tensor([_fixed_dt(case["n"])], dtype=torch.float64, device="cuda")
    sd, sd1 = int(seed) % 30011 + 1, int(seed) % 30011 + 2
    if case["iflow"] == 3:  # the draw of the forcing's set-up
        _, sd = _rand_force(p, p["fp0"], 1, 1.0, sd)
        _, sd1 = _rand_force(p, p["fz0"], 0, 1.0, sd1)
        # a fixed-step run keeps time steps of its own; the forcing follows them
    for _ in range(case["steps"]):
        if case["cfl"]:
            dt = sv.dt(psi, case["cfl"])
        if case["iflow"] == 3:
            fp, sd = _rand_force(p, p["fp0"], 1, float(dt), sd)
            fz, sd1 = _rand_force(p, p["fz0"], 0, float(dt), sd1)
        t += float(dt)
        psi, vz = sv.step(psi, vz, fp, fz, dt)
    return dict(psi=psi[0], vz=vz[0], time=t, dt=float(dt))


def _exact_diag(case, seed):
    n = case["n"]
    p = _params(n, case["nu"], case["omega"])
    psi, vz, fp, fz = _fields(n, seed)
    sv = _Solver([p])
    k2, two, s = sv.k2, _two(n), 1.0 / float(n) ** 4
    pos = k2 >= 1

    def powk(kin):
        return k2.clamp(min=1.0) ** kin

    def energy(a, kin):
        w = torch.where(pos, powk(kin), 0.0 if kin else 1.0)
        return float((two * w * a.abs() ** 2).sum() * s)

    def inner(a, b, kin):
        w = torch.where(sv.mask & pos, powk(kin), 0.0)
        if kin == 0:
            w = torch.where(sv.mask, 1.0, 0.0).double()
        return float((two * w * (b * a.conj()).real).sum() * s)
    nn, mm, nnv, mmv = p["nn"], p["mm"], p["nnv"], p["mmv"]
    band = (k2 <= 2.01 * p["kup"] ** 2) & (k2 >= p["kup"] ** 2)
    b = [0.0, energy(psi, 1), energy(vz, 0), inner(psi, fp, 1), inner(vz, fz, 0), p["nu"] * energy(psi, nn + 1),
         p["nuv"] * energy(vz, nnv), p["hnu"] * energy(psi, 1 - mm), p["hnuv"] * energy(vz, -mmv),
         2 * p["omega"] * inner(vz, 1j * sv.ky * psi, 0), float((two * band * k2 * psi.abs() ** 2).sum() * s),
         float((two * band * vz.abs() ** 2).sum() * s),
         0.0, energy(psi, 2), inner(psi, fp, 2), p["nu"] * energy(psi, nn + 2), p["hnu"] * energy(psi, 2 - mm),
         0.0, -inner(vz, psi, 1), -inner(vz, fp, 1), -inner(psi, fz, 1), -p["nu"] * inner(vz, psi, nn + 1),
         -p["nuv"] * inner(psi, vz, nnv + 1), -p["hnu"] * inner(vz, psi, 1 - mm), -p["hnuv"] * inner(psi, vz, 1 - mmv)]
    w = _c2r(-k2 * psi, n)
    v = _c2r(torch.where(sv.mask, vz, 0.0), n)
    ext = [0.0, float(w.max()), float(w.min()), float(v.max()), float(v.min())]
    nb = n // 2 + 1
    kmn = torch.floor(torch.sqrt(k2) + 0.5).long()
    ok = (kmn > 0) & (kmn <= nb)
    idx = torch.where(ok, kmn - 1, 0).reshape(-1)

    def shells(f):
        f = torch.where(ok, two * f, 0.0).reshape(-1)
        return (torch.zeros(nb, dtype=torch.float64, device="cuda").index_add_(0, idx, f) * s).cpu().numpy()
    b5, b6 = (x[0] for x in sv.brackets(psi[None], vz[None]))
    tr = [shells(k2 * (psi * b5.conj()).real), shells((psi * b5.conj()).real), shells(-(vz * b6.conj()).real)]
    return dict(budget=np.array(b), extrema=np.array(ext), ek=shells(k2 * psi.abs() ** 2),
                ezk=shells(vz.abs() ** 2), transfers=np.stack(tr), vorticity=-w.T / float(n) ** 2)


def _exact_ensemble(case, seed):
    times, states, i = [], [], 0
    for n, runs in _groups(case):
        f = [_fields(n, seed * 1000 + i + r) for r in range(runs)]
        psi, vz, fp, fz = (torch.stack([x[k] for x in f]) for k in range(4))
        sv = _Solver([_run_params(case, i + r, n) for r in range(runs)])
        t = torch.zeros(runs, dtype=torch.float64, device="cuda")
        for _ in range(case["steps"]):
            dt = sv.dt(psi, case["cfl"])
            t += dt
            psi, vz = sv.step(psi, vz, fp, fz, dt)
        times.append(t)
        states += [v for r in range(runs) for v in (psi[r], vz[r])]
        i += runs
    return dict(times=torch.cat(times), states=states)


def _exact_les(case, seed):
    n = case["n"]
    psi, vz, fp, fz = _fields(n, seed)
    im, isd, om, osd = (_dev64(v) for v in _les_norm(psi, vz, n))
    w = _net_params(seed).double()
    sv = _Solver([_params(n, 2e-5, 1.0)])
    band = _dev64(_band(n))[:, torch.floor(torch.sqrt(sv.k2) + 0.5).long().clamp(max=n // 2)]
    psi, vz, fp, fz = (v[None] for v in (psi, vz, fp, fz))
    t = 0.0
    for k in range(case["steps"]):
        if k % case["every"] == 0:
            x = (_inputs64(psi[0], vz[0], n) - im) / isd
            y = _net64(x[None], w)[0] * osd + om
            tau = [_r2c(y[..., c].T) * band[c] for c in range(2)]
        dt = sv.dt(psi, case["cfl"])
        t += float(dt)
        psi, vz = sv.step(psi, vz, fp, fz, dt, tau)
    return dict(psi=psi[0], vz=vz[0], time=t, dt=float(dt))


def _exact_train(case, seed):
    x, y, norm = _net_batch(case, seed)
    im, isd, om, osd = (_dev64(v) for v in norm)
    w = _net_params(seed).double()
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    for k, shift in enumerate((1, 2, 0)):
        w.requires_grad_(True)
        xs, ys = (x.roll(shift, 1).double() - im) / isd, (y.roll(shift, 1).double() - om) / osd
        loss = ((_net64(xs, w) - ys) ** 2).mean()
        g, = torch.autograd.grad(loss, w)
        with torch.no_grad():
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            w = w - 5e-4 * (m / (1 - 0.9 ** (k + 1))) / (torch.sqrt(v / (1 - 0.999 ** (k + 1))) + 1e-8)
    return dict(loss=float(loss), params=w)


def _exact_vjp(case, seed):
    x, y, norm = _net_batch(case, seed)
    im, isd, om, osd = (_dev64(v) for v in norm)
    w = _net_params(seed).double().requires_grad_(True)
    x = x.double().requires_grad_(True)
    out = _net64((x - im) / isd, w) * osd + om
    gx, gp = torch.autograd.grad(out, (x, w), (y / 1000).double())
    return dict(out=out.detach(), gx=gx, gp=gp)


def exact(case, seed):
    kind = case["kind"]
    if kind == "fft":
        n = case["n"]
        x = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=_gen(seed))
        return dict(spec=_r2c(x.T), back=x * float(n) ** 2)
    return dict(step=_exact_step, diag=_exact_diag, ensemble=_exact_ensemble, les=_exact_les, train=_exact_train,
                vjp=_exact_vjp)[kind](case, seed)
