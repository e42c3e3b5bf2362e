"""The work a program has this library do: DNS integrations of one field and of ensembles, f^T(u), the request
server, whole-FlowField transforms and the batched tau solve.

A DNS case advances host FlowField buffers through DNS.advance, the call of a time-stepping program
(simulateflow's loop); its state has taken its start-up steps already.  Mixed-precision results carry the
rounding of single-precision transforms: such a program keeps its snapshots on the GPU in single precision.
"""

import math

import numpy as np
import torch

from channelflow_gb300 import DNS, DNSFlags, Ensemble, Grid, tau_solve_batched
from channelflow_gb300 import dns as D
from channelflow_gb300.dsi import TimeStep, ft
from channelflow_gb300.flowfield import FlowField, Spectral
from channelflow_gb300.server import Server

PI = math.pi
WARM = 4  # steps a DNS has taken before the timed call: past the start-up steps of every scheme

# flow: box (Lx, Lz), Reynolds number scale and base flow; the boxes are those of the repository's workloads
COUETTE_BOX = (2 * PI / 1.14, 2 * PI / 2.5)
CHANNEL_BOX = (4 * PI, 2 * PI)
SCHEMES = {"CNFE1": D.CNFE1, "CNAB2": D.CNAB2, "CNRK2": D.CNRK2, "SMRK2": D.SMRK2, "SBDF2": D.SBDF2,
           "SBDF3": D.SBDF3, "SBDF4": D.SBDF4}
FORMS = {"rotational": D.Rotational, "convection": D.Convection, "divergence": D.Divergence,
         "skew": D.SkewSymmetric}


def _dns(name, Nx, Ny, Nz, flow, scheme, form, precision, steps, fields=1, kind="dns"):
    return {"name": name, "kind": kind, "Nx": Nx, "Ny": Ny, "Nz": Nz, "flow": flow, "scheme": scheme, "form": form,
            "precision": precision, "steps": steps, "fields": fields}


def listed():
    return [
        # the smallest call: one step of a minimal-flow-unit Couette DNS, fields handed over every step
        _dns("couette_32_fp64_step", 32, 33, 32, "couette", "SBDF3", "rotational", "fp64", 1),
        # one output interval (dT = 1) of the same flow in mixed precision
        _dns("couette_32_mixed_interval", 32, 33, 32, "couette", "SBDF3", "rotational", "mixed", 50),
        # one f^T(u) of a Newton-Krylov search: a DNS built, 200 steps, the field back
        _dns("ft_couette_32x35_fp64", 32, 35, 32, "couette", "SBDF3", "rotational", "fp64", 200, kind="ft"),
        # plane Poiseuille turbulence at constant bulk velocity, both precisions
        _dns("poiseuille_128_mixed", 128, 97, 128, "poiseuille", "CNAB2", "rotational", "mixed", 20),
        _dns("poiseuille_128_fp64", 128, 97, 128, "poiseuille", "SBDF3", "rotational", "fp64", 10),
        # 64 trajectories of an edge-tracking / ensemble study advanced together
        _dns("ensemble_48_mixed", 48, 49, 48, "couette", "SBDF3", "rotational", "mixed", 10, fields=64,
             kind="ensemble"),
        # gradient forms on ragged, non-power-of-two grids
        _dns("skew_72x57x90_fp64", 72, 57, 90, "couette", "SBDF3", "skew", "fp64", 10),
        _dns("convection_60x65x84_mixed", 60, 65, 84, "poiseuille", "SMRK2", "convection", "mixed", 5),
        # a tall, wide channel grid: the largest single field
        _dns("channel_192x129x160_fp64", 192, 129, 160, "poiseuille", "SBDF3", "rotational", "fp64", 5),
        # 12 requests of different grids, Reynolds numbers and horizons through the request server
        {"name": "serve_mixed_12", "kind": "serve", "requests": 12, "steps": 100, "precision": "mixed"},
        # a velocity field to physical space and a physical field to spectral space, on the GPU
        {"name": "transforms_128_fp64", "kind": "transforms", "Nx": 128, "Ny": 97, "Nz": 128},
        # TauSolver::solve for every mode of a 48x49x48 field, from and to host profiles
        {"name": "tau_solve_48", "kind": "tau", "Nx": 48, "Ny": 49, "Nz": 48},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fft_len(rng, lo, hi):
    """An even length between lo and hi without prime factors above 13."""
    while True:
        n = 2 * _log_int(rng, lo // 2, hi // 2)
        m = n
        for p in (2, 3, 5, 7, 11, 13):
            while m % p == 0:
                m //= p
        if m == 1:
            return n


def draw(rng):
    kind = rng.choice(["dns"] * 6 + ["ft", "ensemble", "transforms", "tau", "serve"])
    if kind == "serve":
        precision = rng.choice(["mixed", "fp64"])
        return {"kind": kind, "requests": rng.randint(3, 11 if precision == "mixed" else 5),
                "steps": rng.randint(40, 100), "precision": precision}
    if kind == "transforms":
        return {"kind": kind, "Nx": _fft_len(rng, 24, 128), "Ny": 2 * _log_int(rng, 8, 48) + 1,
                "Nz": _fft_len(rng, 24, 128)}
    if kind == "tau":
        return {"kind": kind, "Nx": _fft_len(rng, 16, 64), "Ny": 2 * _log_int(rng, 8, 48) + 1,
                "Nz": _fft_len(rng, 16, 64)}
    top = {"dns": 160, "ft": 36, "ensemble": 48}[kind]
    form = rng.choice(["rotational"] * 3 + ["convection", "divergence", "skew"])
    precision = "fp64" if kind == "ft" else rng.choice(["fp64", "mixed"])
    # Ny up to 129: single-precision transforms lose digits of the pressure with Ny, mixed runs stay below 100;
    # the low-viscosity channel with the multistep schemes, whose pressure does not feed back from step to step
    ny = _log_int(rng, 8, 24 if kind != "dns" else 40 if form != "rotational" else 48 if precision == "mixed" else 64)
    flow = rng.choice(["couette", "poiseuille"])
    scheme = rng.choice(["SBDF3", "SBDF2", "SBDF4"] + (["CNAB2", "SMRK2"] if flow == "couette" else []))
    c = _dns("", _fft_len(rng, 20, top), 2 * ny + 1, _fft_len(rng, 20, top), flow, scheme, form, precision,
             rng.randint(30, 100) if kind == "ft" else rng.randint(1, 4 if form != "rotational" else 10),
             fields=rng.randint(3, 32) if kind == "ensemble" else 1, kind=kind)
    while work(c)["flops"] > 2e10 and c["steps"] > 1:  # no more than the largest listed field's work
        c["steps"] //= 2
    del c["name"]
    return c


# ---- flags and inputs ------------------------------------------------------------------------------------------


def _flow(case):
    """(box, flags) of a case: dt falls with the grid spacing, so that every grid runs at a moderate CFL number."""
    nx = case["Nx"]
    if case["flow"] == "couette":
        fl = DNSFlags(nu=1 / 400, dt=0.02 * min(1.0, 48 / nx), baseflow=D.LaminarBase, ulowerwall=-1.0, uupperwall=1.0)
        box = COUETTE_BOX
    else:
        fl = DNSFlags(nu=1 / 4000, dt=0.64 / max(nx, 64), baseflow=D.LaminarBase, constraint=D.BulkVelocity,
                      Ubulk=2 / 3)
        box = CHANNEL_BOX
    fl.timestepping, fl.nonlinearity = SCHEMES[case["scheme"]], FORMS[case["form"]]
    return box, fl


def _coef(n, gen, lead, ncut):
    """Random Chebyshev coefficients (lead + (n,)) with spectral decay 0.7^n, the last ones zero."""
    c = torch.randn(lead + (n, 2), generator=gen, dtype=torch.float64, device="cuda")
    c = torch.view_as_complex(c) * 0.7 ** torch.arange(n, dtype=torch.float64, device="cuda")
    c[..., ncut:] = 0
    return c


def _perturbation(Nx, Ny, Nz, box, seed, norm, fields=1, zero_mean_u=False):
    """Divergence-free, no-slip fields (fields, 3, Ny, Nx, Nz//2+1) with Fourier decay 0.5^(|kx|+|kz|) and the
    given L2 norms: v and the wall-normal vorticity from random coefficients, u and w from continuity."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    ch = _Cheb(Ny)
    Kx, Kz = Nx // 3 - 1, Nz // 3 - 1
    kx = torch.arange(-Kx, Kx + 1, device="cuda")
    kz = torch.arange(0, Kz + 1, device="cuda")
    al, ga = (2 * PI / box[0]) * kx[:, None].double(), (2 * PI / box[1]) * kz[None, :].double()
    decay = 0.5 ** (kx.abs()[:, None] + kz[None, :]).double()
    lead = (fields, 2 * Kx + 1, Kz + 1)
    w1 = 1 - ch.y ** 2
    mul = lambda c, w: (c @ ch.T.t().to(c.dtype) * w) @ ch.F.t().to(c.dtype)  # noqa: E731
    v = mul(_coef(Ny, gen, lead, Ny - 4) * decay[..., None], w1 * w1)
    eta = mul(_coef(Ny, gen, lead, Ny - 2) * decay[..., None], w1)
    k2 = (al * al + ga * ga)
    k2[Kx, 0] = 1
    vy = v @ ch.D.t().to(v.dtype)
    u = (al[..., None] * (1j * vy) - ga[..., None] * (1j * eta)) / k2[..., None]
    w = (ga[..., None] * (1j * vy) + al[..., None] * (1j * eta)) / k2[..., None]
    for a, s in ((u, 1), (v, 0), (w, 1)):  # kz = 0: Hermitian in kx; the mean profiles are real, without v
        a[:, :Kx, 0] = a[:, Kx + 1:, 0].flip(1).conj()
        a[:, Kx, 0] = s * mul(_coef(Ny, gen, (fields,), Ny - 2), w1).real.to(a.dtype)
    if zero_mean_u:
        m = u[:, Kx, 0] @ ch.mean.to(u.dtype)
        u[:, Kx, 0] -= m[:, None] / (2 / 3) * (ch.F @ w1).to(u.dtype)
    s = torch.stack((u, v, w), 1)  # fields, 3, kx, kz, n
    cz = torch.where(kz == 0, 1.0, 2.0).double()
    sq = sum(torch.einsum("fixzn,nm,fixzm,z->f", p, ch.W, p, cz) for p in (s.real, s.imag))
    s = s * (torch.as_tensor(norm, dtype=torch.float64, device="cuda") / sq.sqrt())[:, None, None, None, None]
    out = torch.zeros((fields, 3, Ny, Nx, Nz // 2 + 1), dtype=torch.complex128, device="cuda")
    out[:, :, :, kx % Nx, :Kz + 1] = s.permute(0, 1, 4, 2, 3)
    return out


def _initial(case, seed):
    box, fl = _flow(case)
    f = case["fields"]
    bulk = fl.constraint == D.BulkVelocity
    norm = [0.3] * f if bulk else np.random.default_rng(seed).uniform(0.05, 0.3, size=f)
    return _perturbation(case["Nx"], case["Ny"], case["Nz"], box, seed, norm, f, bulk)


def _requests(case, seed):
    """The requests of a serving case: (dns case, flags, steps, field)."""
    r = np.random.default_rng(seed)
    shapes = np.random.default_rng(7)  # the mix of grids is the case's, the fields and Reynolds numbers the seed's
    out = []
    for k in range(case["requests"]):
        nx, nz = (int(v) for v in shapes.choice([32, 48, 64], size=2))
        c = {"Nx": nx, "Ny": int(shapes.choice([33, 49])), "Nz": nz, "flow": "couette" if k % 2 else "poiseuille",
             "scheme": "SBDF3", "form": "rotational", "fields": 1}
        steps = int(case["steps"] * shapes.uniform(0.5, 1.0))
        box, fl = _flow(c)
        fl.dt = 0.01
        fl.nu = 1 / float(r.uniform(300, 2000))
        u = _perturbation(nx, c["Ny"], nz, COUETTE_BOX, seed * 1000 + k, [0.1], 1, k % 2 == 0)[0]
        out.append((c, fl, steps, u))
    return out


def _tau_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    Kx, Kz = case["Nx"] // 3 - 1, case["Nz"] // 3 - 1
    kx, kz = (a.ravel().astype(np.int32) for a in np.meshgrid(np.arange(-Kx, Kx + 1), np.arange(Kz + 1), indexing="ij"))
    R = [_coef(case["Ny"], gen, (len(kx),), case["Ny"]) for _ in range(3)]
    for r in R:
        r[(kx == 0) & (kz == 0)] = r[(kx == 0) & (kz == 0)].real.to(r.dtype)
    return kx, kz, R


TAU = {"lambda_t": (11 / 6) / 0.02, "nu": 1 / 400}


# ---- the framework's entry points ------------------------------------------------------------------------------


class _DeviceArray:
    """A FlowField's device buffer for torch (the field stays alive while a tensor refers to it)."""

    def __init__(self, field):
        import ctypes
        p = ctypes.c_void_p()
        if field._lib.cfgpu_flowfield_data(field._h, ctypes.byref(p)):
            raise RuntimeError("cfgpu_flowfield_data")
        self.field = field
        self.__cuda_array_interface__ = {"shape": (field.Nd, field.Ny, field.Nx, field.Nzpad), "typestr": "<f8",
                                         "data": (p.value, False), "version": 3}


def _buffer(shape, src, pinned):
    """A host FlowField buffer holding src: plain memory, or page-locked for snapshots that go to the GPU."""
    t = torch.zeros(shape, dtype=torch.complex128, pin_memory=pinned)
    if src is not None:
        t.copy_(src.reshape(shape))
    return t.numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "tau":
        kx, kz, R = _tau_inputs(case, seed)
        return {"kind": kind, "case": case, "kx": kx, "kz": kz, "R": [r.cpu().numpy() for r in R]}
    if kind == "transforms":
        Nx, Ny, Nz = case["Nx"], case["Ny"], case["Nz"]
        fields = [FlowField(Nx, Ny, Nz, 3, *CHANNEL_BOX) for _ in range(2)]
        u = _perturbation(Nx, Ny, Nz, CHANNEL_BOX, seed, [0.1])[0]
        fields[0].set_spectral(u.cpu().numpy())
        fields[1].set_physical(_physical(_perturbation(Nx, Ny, Nz, CHANNEL_BOX, seed + 1, [0.1])[0], Nz).cpu().numpy())
        return {"kind": kind, "fields": fields, "views": [torch.as_tensor(_DeviceArray(f), device="cuda") for f in fields]}
    if kind == "serve":
        reqs = [(Grid(c["Nx"], c["Ny"], c["Nz"], *COUETTE_BOX), fl, steps, u.cpu().numpy())
                for c, fl, steps, u in _requests(case, seed)]
        return {"kind": kind, "server": Server(max_bytes=8 << 30, slots=8, precision=case["precision"]),
                "requests": reqs, "mixed": case["precision"] == "mixed"}
    box, fl = _flow(case)
    g = Grid(case["Nx"], case["Ny"], case["Nz"], *box)
    u0 = _initial(case, seed)
    if kind == "ft":
        T = case["steps"] * fl.dt
        ts = TimeStep(dt=fl.dt, dtmin=fl.dt, dtmax=fl.dt, dT=T, CFLmin=0.0, CFLmax=1.0, variable=False)
        return {"kind": kind, "grid": g, "flags": fl, "timestep": ts, "T": T, "u": u0[0].cpu().numpy()}
    mixed, f = case["precision"] == "mixed", case["fields"]
    lead = (f,) if kind == "ensemble" else ()
    u = _buffer(lead + (3, g.Ny, g.Nx, g.Mz), u0, mixed)
    q = _buffer(lead + (1, g.Ny, g.Nx, g.Mz), None, mixed)
    dns = (Ensemble(g, fl, f, precision=case["precision"]) if kind == "ensemble"
           else DNS(u, g, fl, precision=case["precision"]))
    dns.advance(u, q, WARM)
    return {"kind": kind, "dns": dns, "u": u, "q": q, "steps": case["steps"], "mixed": mixed}


def run(state):
    kind = state["kind"]
    if kind == "dns" or kind == "ensemble":
        u, q = state["u"], state["q"]
        state["dns"].advance(u, q, state["steps"])
        if not state["mixed"]:
            return u, q
        return tuple(torch.from_numpy(a).to("cuda").to(torch.complex64) for a in (u, q))
    if kind == "ft":
        return ft(state["u"], state["grid"], state["flags"], state["timestep"], state["T"])
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(*r) for r in state["requests"]]
        srv.run()
        out = []
        for i in ids:
            status, u, _ = srv.poll(i)
            if u is None:
                raise RuntimeError("request %d ended with status %d" % (i, status))
            srv.release(i)
            out.append(u.astype(np.complex64) if state["mixed"] else u)
        return out
    if kind == "transforms":
        for f in state["fields"]:  # one field each way in every pass
            if f.state() == (Spectral, Spectral):
                f.makePhysical()
            else:
                f.makeSpectral()
        return [torch.view_as_complex(v.unflatten(-1, (-1, 2))) if f.xzstate == Spectral else v[..., :f.Nz]
                for f, v in zip(state["fields"], state["views"])]
    c = state["case"]
    return tau_solve_batched(c["Ny"], state["kx"], state["kz"], *COUETTE_BOX, -1.0, 1.0, TAU["lambda_t"], TAU["nu"],
                             *state["R"])


# ---- algorithmic work ------------------------------------------------------------------------------------------


def _step_work(c):
    nx, ny, nz = c["Nx"], c["Ny"], c["Nz"]
    modes = (2 * (nx // 3) - 1) * (nz // 3)
    A = modes * ny
    sw = 4 if c["precision"] == "mixed" else 8
    sub = 3 if c["scheme"] in ("SMRK2", "CNRK2") else 1
    order = {"SBDF2": 2, "SBDF3": 3, "SBDF4": 4}.get(c["scheme"], 1)
    old_u, old_n = (order - 1, order - 1) if order > 1 else (0, 1)
    nt = {"rotational": 9, "convection": 15, "divergence": 9, "skew": 21}[c["form"]]  # transforms
    transform = 2.5 * nx * ny * nz * math.log2(nx * ny * nz)
    # u (and the schemes' older u, N) in, u, q and N out; q in where the scheme has an implicit pressure
    by = sub * (16 * A * (3 + 3 * old_u + 4 + (1 if order == 1 else 0)) + 2 * sw * A * (3 * old_n + 3))
    return by * c["fields"], sub * (nt * transform + 150 * A) * c["fields"]


def work(case):
    kind = case["kind"]
    if kind == "serve":
        tot = [0.0, 0.0]
        shapes = np.random.default_rng(7)
        for _ in range(case["requests"]):
            nx, nz = (int(v) for v in shapes.choice([32, 48, 64], size=2))
            ny = int(shapes.choice([33, 49]))
            steps = int(case["steps"] * shapes.uniform(0.5, 1.0))
            b, f = _step_work({"Nx": nx, "Ny": ny, "Nz": nz, "precision": case["precision"], "scheme": "SBDF3",
                               "form": "rotational", "fields": 1})
            tot[0] += b * steps
            tot[1] += f * steps
        return {"bytes": tot[0], "flops": tot[1]}
    if kind == "transforms":
        nx, ny, nz = case["Nx"], case["Ny"], case["Nz"]
        return {"bytes": 2 * 2 * 3 * 8 * nx * ny * (nz + 2), "flops": 6 * 2.5 * nx * ny * nz * math.log2(nx * ny * nz)}
    if kind == "tau":
        A = (2 * (case["Nx"] // 3) - 1) * (case["Nz"] // 3) * case["Ny"]
        return {"bytes": 16 * A * 7, "flops": 150 * A}
    b, f = _step_work(case)
    return {"bytes": b * case["steps"], "flops": f * case["steps"]}


# ---- the same results in 64 bits -------------------------------------------------------------------------------


def _physical(u, nz):
    """makePhysical: (..., Ny, Nx, Mz) spectral -> (..., Ny, Nx, nz)."""
    T = _Cheb(u.shape[-3]).T.to(u.dtype)
    y = torch.einsum("jn,...nxz->...jxz", T, u)
    return torch.fft.irfft2(y, s=(u.shape[-2], nz)) * (u.shape[-2] * nz)


def _spectral(p):
    s = torch.fft.rfft2(p) / (p.shape[-2] * p.shape[-1])
    return torch.einsum("nj,...jxz->...nxz", _Cheb(p.shape[-3]).F.to(s.dtype), s)


class _Cheb:
    """Chebyshev matrices on [-1, 1]: T coefficients -> Gauss-Lobatto values, F its inverse, D the derivative,
    W the L2 weights, mean the y average."""

    def __init__(self, N):
        j = np.arange(N)
        T = np.cos(PI * (np.outer(j, j) % (2 * (N - 1))) / (N - 1))
        e = np.where((j == 0) | (j == N - 1), 0.5, 1.0)
        Dm = np.zeros((N, N))
        for n in range(N):
            Dm[n, n + 1::2] = 2 * j[n + 1::2]
        Dm[0] /= 2
        m, n = j[:, None], j[None, :]
        with np.errstate(divide="ignore", invalid="ignore"):
            W = (1 - m * m - n * n) / ((1 + m - n) * (1 - m + n) * (1 + m + n) * (1 - m - n))
        W[(m + n) % 2 == 1] = 0
        mean = np.where(j % 2 == 0, 1.0 / (1.0 - np.where(j % 2 == 0, j, 0) ** 2), 0.0)
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
        self.N, self.T, self.F, self.D, self.W, self.mean = (
            N, t(T), t(T * np.outer(e, e) * (2 / (N - 1))), t(Dm), t(W), t(mean))
        self.y = t(np.cos(PI * j / (N - 1)))
        self.at_b, self.at_a = t(np.ones(N)), t(np.where(j % 2 == 0, 1.0, -1.0))


class _Helmholtz:
    """nu u'' - lam u = f with u(+-1) given, Chebyshev tau, for many lam: the integrated (tridiagonal in each
    parity) equations, inverted densely."""

    def __init__(self, N, lam, nu):
        n_ = np.arange(N)
        self.par = []
        for p in (0, 1):
            n = n_[p::2]
            P = len(n)
            B = np.zeros((P, P))
            for i in range(1, P):
                k = n[i]
                B[i, i - 1] = (2 if k == 2 else 1) / (4 * k * (k - 1))
                if k <= N - 3:
                    B[i, i] = -1 / (2 * (k * k - 1))
                if i + 1 < P and k + 2 <= N - 3:
                    B[i, i + 1] = 1 / (4 * k * (k + 1))
            B = torch.as_tensor(B, dtype=torch.float64, device="cuda")
            A = -lam[:, None, None] * B
            i = torch.arange(P, device="cuda")
            A[:, i, i] += nu
            A[:, 0, :] = 1
            inv = torch.linalg.inv(A)
            self.par.append((inv @ B, inv[:, :, 0]))
        self.N = N

    def __call__(self, f, ua=0.0, ub=0.0):
        """f (modes, N, columns) real."""
        u = torch.empty_like(f)
        for p, (G, bc) in enumerate(self.par):
            u[:, p::2] = G @ f[:, p::2]
            if ua or ub:
                u[:, p::2] += bc[:, :, None] * ((ub + ua) / 2 if p == 0 else (ub - ua) / 2)
        return u


class _Tau:
    """TauSolver of many modes: influence-matrix and tau-corrected Stokes solves; complex (modes, N, columns)."""

    def __init__(self, kx, kz, box, lam, nu, N):
        ch = self.ch = _Cheb(N)
        self.ax, self.az = 2 * PI * kx / box[0], 2 * PI * kz / box[1]
        self.lam, self.nu, M = lam, nu, len(kx)
        self.zero = (kx == 0) & (kz == 0)
        self.pH, self.vH = _Helmholtz(N, self.ax ** 2 + self.az ** 2, 1.0), _Helmholtz(N, lam, nu)
        z = torch.zeros((M, N, 1), dtype=torch.float64, device="cuda")
        self.Pp, self.Pm = self.pH(z, 0.0, 1.0), self.pH(z, 1.0, 0.0)
        self.vp, self.vm = self.vH(ch.D @ self.Pp), self.vH(ch.D @ self.Pm)
        ends = torch.stack((ch.at_b, ch.at_a)) @ ch.D
        self.ends = ends
        I = torch.cat((ends @ self.vp, ends @ self.vm), 2)
        I[self.zero] = torch.eye(2, dtype=torch.float64, device="cuda")
        self.inv = torch.linalg.inv(I)
        Nb = N - 1
        n0 = [Nb - 1 if k == 0 else 0 if k == Nb else 2 * (Nb - 1) if k % 2 == 0 else 2 * Nb for k in range(N)]
        P0 = self.pH(torch.as_tensor(n0, dtype=torch.float64, device="cuda")[None, :, None].expand(M, N, 1).contiguous())
        dP0 = ch.D @ P0
        v0 = self.vH(dP0)
        self.P0, self.v0 = self._influence(P0, v0)
        self.s0 = self._residual(self.v0, dP0)

    def _influence(self, P, v):
        d = -self.inv @ (self.ends @ v)
        P = P + self.Pp * d[:, :1] + self.Pm * d[:, 1:]
        v = v + self.vp * d[:, :1] + self.vm * d[:, 1:]
        return P, v

    def _residual(self, v, rest):
        r = self.lam[:, None, None] * v + rest - self.nu * (self.ch.D @ (self.ch.D @ v))
        return r[:, -2:]

    def pv(self, r, Ry):
        D = self.ch.D
        P = self.pH(r)
        v = self.vH(D @ P - Ry)
        P2, v2 = self._influence(P, v)
        s = self._residual(v2, D @ P2 - Ry) / (1 - self.s0)
        sNb1, sNb = s[:, :1], s[:, 1:]
        even = (torch.arange(self.ch.N, device="cuda") % 2 == 0)[None, :, None]
        P2 = P2 + torch.where(even, sNb1, sNb) * self.P0
        v2 = v2 + torch.where(even, sNb, sNb1) * self.v0
        P2[self.zero], v2[self.zero] = P[self.zero], 0
        return P2, v2

    def solve(self, Rx, Ry, Rz):
        C = Rx.shape[2]
        ri = lambda c: torch.cat((c.real, c.imag), 2)  # noqa: E731
        cx = lambda r: torch.complex(r[..., :C].contiguous(), r[..., C:].contiguous())  # noqa: E731
        ax, az = self.ax[:, None, None], self.az[:, None, None]
        D = self.ch.D.to(Rx.dtype)
        P, v = (cx(a) for a in self.pv(ri(D @ Ry + 1j * (ax * Rx + az * Rz)), ri(Ry)))
        u, w = (cx(self.vH(ri(1j * a * P - R))) for a, R in ((ax, Rx), (az, Rz)))
        return u, v, w, P


class _Exact:
    """One DNS (its fields advanced together) in 64 bits: arrays (fields, components, Ny, kx, kz) of the solved modes."""

    MULTI = {D.SBDF1: (1.0, [-1.0], [1.0]), D.SBDF2: (1.5, [-2.0, 0.5], [2.0, -1.0]),
             D.SBDF3: (11 / 6, [-3.0, 1.5, -1 / 3], [3.0, -3.0, 1.0]),
             D.SBDF4: (25 / 12, [-4.0, 3.0, -4 / 3, 0.25], [4.0, -6.0, 4.0, -1.0])}
    CNAB = {D.CNAB2: ([0.5], [0.5], [1.5], [-0.5]),
            D.SMRK2: ([29 / 96, -3 / 40, 1 / 6], [37 / 160, 5 / 24, 1 / 6], [8 / 15, 5 / 12, 3 / 4],
                      [0.0, -17 / 60, -5 / 12])}
    RK = ([0.0, -5 / 9, -153 / 128], [1 / 3, 15 / 16, 8 / 15], [1 / 6, 5 / 24, 1 / 8])

    def __init__(self, case, box, fl):
        self.Nx, self.Ny, self.Nz, self.fl, self.box = case["Nx"], case["Ny"], case["Nz"], fl, box
        Kx, Kz = self.Nx // 3 - 1, self.Nz // 3 - 1
        self.kx = torch.cat((torch.arange(Kx + 1), torch.arange(-Kx, 0))).cuda()
        self.kz = torch.arange(Kz + 1).cuda()
        self.ch = ch = _Cheb(self.Ny)
        self.ax = (2 * PI / box[0] * self.kx.double())[:, None]
        self.az = (2 * PI / box[1] * self.kz.double())[None, :]
        self.U = torch.zeros(self.Ny, dtype=torch.float64, device="cuda")
        self.bulk = fl.constraint == D.BulkVelocity
        if self.bulk:  # laminar profile of the bulk velocity, walls at rest
            self.U[0], self.U[2] = 0.75 * fl.Ubulk, -0.75 * fl.Ubulk
        else:  # walls at -1 and 1, no pressure gradient
            self.U[1] = 1.0
        self.umean = fl.Ubulk - float(self.U @ ch.mean) if self.bulk else 0.0
        self.Uyy = ch.D @ (ch.D @ self.U)
        self.tau = {}
        self.method, self.hist, self.fj1, self.Q = fl.timestepping, [], None, None
        self.started = 0
        self.need = {D.SBDF2: 1, D.SBDF3: 2, D.SBDF4: 3, D.CNAB2: 1}.get(self.method, 0)

    def tau_of(self, lam_t):
        if lam_t not in self.tau:
            kx, kz = (a.reshape(-1).double() for a in torch.meshgrid(self.kx, self.kz, indexing="ij"))
            k2 = (2 * PI * kx / self.box[0]) ** 2 + (2 * PI * kz / self.box[1]) ** 2
            self.tau[lam_t] = _Tau(kx, kz, self.box, lam_t + self.fl.nu * k2, self.fl.nu, self.Ny)
        return self.tau[lam_t]

    def modes(self, full):
        return full[..., self.kx % self.Nx, :len(self.kz)].contiguous()

    def full(self, s):
        out = torch.zeros(s.shape[:-2] + (self.Nx, self.Nz // 2 + 1), dtype=s.dtype, device="cuda")
        out[..., self.kx % self.Nx, :len(self.kz)] = s
        return out

    def dy(self, a):
        return torch.einsum("nm,...mxz->...nxz", self.ch.D.to(a.dtype), a)

    def phys(self, s):
        return _physical(self.full(s), self.Nz)

    def spec(self, p):
        return self.modes(_spectral(p))

    def nonlinear(self, u):
        u = u.clone()
        u[:, 0, :, 0, 0] += self.U
        dx, dy, dz = (lambda a: 1j * self.ax * a), self.dy, (lambda a: 1j * self.az * a)
        p = self.phys(u)
        form = self.fl.nonlinearity
        if form == D.Rotational:
            a, b, c = u[:, 0], u[:, 1], u[:, 2]
            o = self.phys(torch.stack((dy(c) - dz(b), dz(a) - dx(c), dx(b) - dy(a)), 1))
            return self.spec(torch.stack([o[:, (i + 1) % 3] * p[:, (i + 2) % 3] - o[:, (i + 2) % 3] * p[:, (i + 1) % 3]
                                          for i in range(3)], 1))
        out = []
        if form in (D.Convection, D.SkewSymmetric):
            conv = sum(p[:, j:j + 1] * self.phys(d(u)) for j, d in enumerate((dx, dy, dz)))
            out.append(self.spec(conv))
        if form in (D.Divergence, D.SkewSymmetric):
            s = [self.spec(p * p[:, j:j + 1]) for j in range(3)]
            out.append(dx(s[0]) + dy(s[1]) + dz(s[2]))
        return sum(out) / len(out)

    def linear(self, u, q):
        nu, P = self.fl.nu, q[:, 0]
        k2 = self.ax ** 2 + self.az ** 2
        out = nu * (self.dy(self.dy(u)) - k2 * u) - torch.stack((1j * self.ax * P, self.dy(P), 1j * self.az * P), 1)
        out[:, 0, :, 0, 0] += nu * self.Uyy
        if self.bulk:
            ends = (self.ch.at_b - self.ch.at_a) @ self.ch.D / 2
            for i, base in ((0, self.U), (2, None)):
                m = u[:, i, :, 0, 0].real + (base if base is not None else 0)
                out[:, i, 0, 0, 0] -= nu * (m @ ends)
        return out

    def solve(self, R, lam_t):
        t = self.tau_of(lam_t)
        R = R.clone()
        F = R.shape[0]
        R[:, :, :, 0, 0] = R[:, :, :, 0, 0].real.to(R.dtype)
        R[:, 0, :, 0, 0] += self.fl.nu * self.Uyy
        cols = [R[:, i].permute(2, 3, 1, 0).reshape(-1, self.Ny, F) for i in range(3)]
        u, v, w, P = t.solve(*cols)
        if self.bulk:  # a mean pressure gradient holds the bulk velocities
            one = torch.zeros((1, self.Ny, 1), dtype=torch.float64, device="cuda")
            one[0, 0] = self.fl.nu
            H = _Helmholtz(self.Ny, t.lam[:1], self.fl.nu)
            c = H(one)[0, :, 0]
            for a, m in ((u, self.umean), (w, 0.0)):
                a[0] += c[:, None] * ((m - self.ch.mean @ a[0].real) / (self.ch.mean @ c))[None, :]
        back = lambda a: a.reshape(len(self.kx), len(self.kz), self.Ny, F).permute(3, 2, 0, 1)  # noqa: E731
        un, qn = torch.stack([back(a) for a in (u, v, w)], 1).contiguous(), back(P)[:, None].contiguous()
        for a in (un, qn):
            a[..., 0, 0] = a[..., 0, 0].real.to(a.dtype)
        return un, qn

    def _cnab(self, u, q, method, fj1):
        dt = self.fl.dt
        for a, b, g, z in zip(*self.CNAB[method]):
            f = self.nonlinear(u)
            R = u / (b * dt) + (a / b) * self.linear(u, q) - (g / b) * f
            if z:
                R -= (z / b) * fj1
            u, q = self.solve(R, 1 / (b * dt))
            fj1 = f
        return u, q, fj1

    def advance(self, u, q, n):
        dt, m = self.fl.dt, self.method
        for _ in range(n):
            if self.started < self.need:  # start-up: this scheme's history, one SMRK2 step
                f = self.nonlinear(u)
                self.hist.insert(0, (u, f))
                self.fj1 = f
                u, q, _ = self._cnab(u, q, D.SMRK2, None)
                self.started += 1
            elif m in self.MULTI:
                eta, al, be = self.MULTI[m]
                self.hist.insert(0, (u, self.nonlinear(u)))
                R = sum((-a / dt) * h[0] - b * h[1] for a, b, h in zip(al, be, self.hist))
                self.hist = self.hist[:len(al) - 1]
                u, q = self.solve(R, eta / dt)
            elif m in self.CNAB:
                u, q, self.fj1 = self._cnab(u, q, m, self.fj1)
            else:
                for A, B, C in zip(*self.RK):
                    self.Q = -self.nonlinear(u) + (A * self.Q if A else 0)
                    u, q = self.solve(self.linear(u, q) + u / (C * dt) + (B / C) * self.Q, 1 / (C * dt))
        return u, q


def _exact_run(case, box, fl, u0, steps):
    e = _Exact(case, box, fl)
    u = e.modes(u0)
    u, q = e.advance(u, torch.zeros_like(u[:, :1]), steps)
    return e.full(u), e.full(q)


def exact(case, seed):
    kind = case["kind"]
    if kind == "tau":
        kx, kz, R = _tau_inputs(case, seed)
        tx, tz = (torch.as_tensor(k, device="cuda").double() for k in (kx, kz))
        k2 = (2 * PI * tx / COUETTE_BOX[0]) ** 2 + (2 * PI * tz / COUETTE_BOX[1]) ** 2
        t = _Tau(tx, tz, COUETTE_BOX, TAU["lambda_t"] + TAU["nu"] * k2, TAU["nu"], case["Ny"])
        return [a[:, :, 0] for a in t.solve(*(r[:, :, None] for r in R))]
    if kind == "transforms":
        Nx, Ny, Nz = case["Nx"], case["Ny"], case["Nz"]
        a, b = (_perturbation(Nx, Ny, Nz, CHANNEL_BOX, s, [0.1])[0] for s in (seed, seed + 1))
        return [_physical(a, Nz), _spectral(_physical(b, Nz))]
    if kind == "serve":
        return [_exact_run(c, COUETTE_BOX, fl, u[None], steps)[0][0].cpu() for c, fl, steps, u in _requests(case, seed)]
    box, fl = _flow(case)
    u, q = _exact_run(case, box, fl, _initial(case, seed), case["steps"] + (0 if kind == "ft" else WARM))
    if kind == "ft":
        return u[0], None
    return (u, q) if kind == "ensemble" else (u[0], q[0])
