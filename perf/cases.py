"""The work that users of this framework have it do, as measurable cases.

A case goes through the public Python interface (`Simulation`, `Ensemble`) as a
run script or an analysis script does: advance a state some RK4 steps, evaluate
the right-hand side once, filter fields, or analyse a frame.  `prepare` makes
the context and the inputs, `run` is one pass, `exact` the same result in plain
torch, 64 bits.
"""
import functools
import importlib
import math

import torch

hqt = importlib.import_module("ads4-holographic-quantum-turbulence_b200")

VY7 = -2 * math.pi * 7 / 20  # the driven script's flow (kk = 7)


# ---- the cases --------------------------------------------------------------
def _case(do, nx, ny, nz, **kw):
    # L is the box length along x; the spacing along y is the same
    c = {"do": do, "nx": nx, "ny": ny, "nz": nz, "L": nx / 2, "mu": 6.0, "vy": 0.0, "dt": 0.02,
         "winding": True, "precision": "fp64", "vortices": 0, "steps": 1}
    c.update(kw)
    return c


def _box(case):
    """Box lengths (Lx, Ly); a frame's box is square, whatever its grid."""
    return case["L"], case["L"] * (1 if case["do"] == "frame" else case["ny"] / case["nx"])


def listed():
    return [
        # the reference's smoke test: four steps of a tiny grid on host
        # arrays, as the MEX gateway calls it; latency and launches count
        _case("host_step", 33, 33, 10, name="smoke33", L=16.0, vy=VY7, steps=4),
        # the run that a CPU can follow (parity runs, trying parameters out)
        _case("step", 64, 64, 21, name="cpu64", L=50.0, steps=10),
        # the reference's driven flow, the grid that the headline is quoted on
        _case("step", 301, 301, 21, name="driven301", L=100.0, vy=VY7, steps=10),
        # the same in mixed precision
        _case("step", 301, 301, 21, name="driven301_mixed", L=100.0, vy=VY7, steps=4,
              precision="mixed"),
        # vortex-lattice decay on a power-of-two grid (no winding removal)
        _case("step", 512, 512, 25, name="lattice512", L=128.0, dt=0.01, winding=False,
              vortices=400, steps=4),
        # the large single run, in mixed precision
        _case("step", 1024, 1024, 33, name="large1024_mixed", L=256.0, dt=0.01, steps=2,
              precision="mixed"),
        # the reference's largest grid (nx = 1001, L = 500, its own nz = 20)
        _case("step", 1001, 1001, 20, name="large1001", L=500.0, vy=VY7, steps=1),
        # a grid that nobody tuned for: uneven, 2*5^3 by 2^2*3^2*5 points
        _case("step", 250, 180, 20, name="uneven250x180", vy=VY7, steps=5),
        # a parameter scan: 32 runs of 128, 192 and 256 points, nz 17, 21, 25
        _case("ensemble", 128, 256, 25, name="ensemble32", runs=32, steps=2),
        # one evaluation of F1..F4 for a user's own integrator
        _case("rhs", 301, 301, 21, name="rhs301", L=100.0, vy=VY7),
        # the Fourier filter on four real fields
        _case("filter", 256, 256, 21, name="filter256", L=128.0, fields=4),
        # one frame of the analysis scripts: boundary fields, velocity, vortex
        # count and energy spectrum
        _case("frame", 512, 512, 25, name="frame512", L=128.0, vortices=400),
    ]


# grids in use: the configurations' and tests' own, and round numbers of points
_GRIDS = (33, 48, 64, 96, 100, 128, 150, 192, 200, 250, 256, 300, 301, 320, 384, 400, 500, 512,
          600, 640, 750, 768, 800, 1000, 1001, 1024)
_MOST = 1024 * 1024 * 33  # sites of the largest listed grid


def _points(rng):
    """A line length, spread over its logarithm: two in three a grid in use,
    else any number, odd ones among them."""
    n = int(round(math.exp(rng.uniform(math.log(32.0), math.log(1024.0)))))
    if rng.random() < 2 / 3:
        return min(_GRIDS, key=lambda g: abs(math.log(g / n)))
    return min(n, 640)


def draw(rng):
    do = rng.choice(["step", "step", "step", "step", "mixed", "host_step", "rhs", "filter",
                     "frame", "ensemble"])
    nx = _points(rng)
    ny = nx if rng.random() < 0.6 else _points(rng)
    nz = rng.choice([8, 10, 12, 16, 17, 20, 21, 21, 24, 25, 30, 33])
    kw = {"vy": rng.choice([0.0, VY7, round(rng.uniform(-2.5, -0.5), 3)]),
          "mu": rng.choice([6.0, 6.0, 5.0, 8.0, round(rng.uniform(4.5, 8.0), 3)]),
          "dt": rng.choice([0.01, 0.02]), "winding": rng.random() < 0.7}
    sites = nx * ny * nz
    steps = max(1, min(10, _MOST // (4 * sites)))
    if do == "mixed":
        return _case("step", nx, ny, nz, precision="mixed", steps=min(steps, 4), **kw)
    if do == "host_step":
        return _case(do, nx, ny, nz, steps=min(steps, 4), **kw)
    if do == "rhs":
        return _case(do, nx, ny, nz, vy=kw["vy"], mu=kw["mu"])
    if do == "filter":
        return _case(do, nx, ny, nz, fields=rng.choice([1, 2, 3, 4]))
    if do == "frame":
        return _case(do, nx, ny, nz, vortices=2 * rng.randint(2, 40))
    if do == "ensemble":
        lo = min(nx, 192)
        return _case(do, lo, min(256, max(lo, ny)), min(nz, 25), runs=rng.randint(2, 12), steps=2)
    return _case("step", nx, ny, nz, steps=steps, **kw)


def _members(case):
    """The runs of an ensemble: grids of 128, 192, 256 points within nx..ny and
    nz of 17, 21, 25 up to nz (the smallest of each where none fits), mu in
    [4.5, 8]."""
    grids = [n for n in (128, 192, 256) if case["nx"] <= n <= case["ny"]] or [case["nx"]]
    nzs = [n for n in (17, 21, 25) if n <= case["nz"]] or [case["nz"]]
    out = []
    for i in range(case["runs"]):
        n, nz = grids[(7 * i + i // 3) % len(grids)], nzs[(5 * i + i // 2) % len(nzs)]
        mu = 4.5 + 3.5 * ((0.37 + 0.618034 * i) % 1.0)
        out.append(_case("step", n, n, nz, L=n / 2, mu=round(mu, 2)))
    return out


# ---- inputs -----------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _columns(mu, vy, nz):
    """Radial columns of the stationary state, as `seed.init_driven` lays them
    out over the plane: Psi, A_t, A_x, A_y on nz points and the charge."""
    one = hqt.seed.init_driven(1, 1, nz, hqt.seed.stationary_profile(mu, vy), noise="none")
    return [torch.from_numpy(a[0, 0].copy()) for a in one[:4]] + [float(one[4][0, 0, 0])]


def _plane(case, g):
    """What Psi is multiplied by at each (y, x): complex noise of 1e-3, and for
    a vortex run the phases and density dips of vortices at random places, half
    of each sign."""
    nx, ny = case["nx"], case["ny"]
    Lx, Ly = _box(case)
    n = torch.randn(2, ny, nx, dtype=torch.float64, device="cuda", generator=g)
    p = torch.complex(1 + 1e-3 * n[0], 1e-3 * n[1])
    if case["vortices"]:
        at = torch.rand(2, case["vortices"], dtype=torch.float64, device="cuda", generator=g)
        x = torch.arange(nx, dtype=torch.float64, device="cuda") * (Lx / nx)
        y = torch.arange(ny, dtype=torch.float64, device="cuda") * (Ly / ny)
        dip = torch.zeros(ny, nx, dtype=torch.float64, device="cuda")
        phase = torch.zeros_like(dip)
        for i in range(case["vortices"]):
            ux, uy = x[None, :] - at[0, i] * Lx, y[:, None] - at[1, i] * Ly
            # periodic in x by the sine, in y by two image rows each way
            for m in (-2, -1, 0, 1, 2):
                s = torch.sin(torch.complex(ux + 0 * uy, uy - m * Ly + 0 * ux) * (math.pi / Lx))
                phase += (1 if i % 2 == 0 else -1) * torch.angle(s)
            dx = torch.remainder(ux + Lx / 2, Lx) - Lx / 2
            dy = torch.remainder(uy + Ly / 2, Ly) - Ly / 2
            dip += torch.exp(-(dx * dx + dy * dy) / 9.0)
        p = p * torch.polar(1 - dip, phase)
    return p


def _state(case, seed):
    """Z1..Z4 and rhoi as CUDA tensors of shape (nz, ny, nx)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + 17)
    psi, at, ax, ay, rho = _columns(case["mu"], case["vy"], case["nz"])
    shape = (case["nz"], case["ny"], case["nx"])

    def flow():
        # a uniform flow with a small smooth disturbance, zero at the boundary
        k = torch.randint(1, 4, (2,), device="cuda", generator=g)
        x = torch.arange(case["nx"], dtype=torch.float64, device="cuda") / case["nx"]
        y = torch.arange(case["ny"], dtype=torch.float64, device="cuda") / case["ny"]
        s = torch.sin(2 * math.pi * (k[0] * x[None, :] + k[1] * y[:, None]))
        r = torch.linspace(1, 0, case["nz"], dtype=torch.float64, device="cuda")
        return r[:, None, None] * (0.3 + 1e-3 * s[None])

    col = [c.to("cuda")[:, None, None] for c in (psi, at, ax, ay)]
    Z1 = (col[0] * _plane(case, g)[None]).contiguous()
    Z2 = (col[1] + torch.zeros(shape, dtype=torch.float64, device="cuda")).contiguous()
    Z3 = (col[2] + flow()).contiguous()
    Z4 = (col[3] + flow()).contiguous()
    return [Z1, Z2, Z3, Z4, torch.full(shape, rho, dtype=torch.float64, device="cuda")]


def _host(t):
    """A device tensor as the column-major [x, y, z] host array."""
    return t.cpu().numpy().T


def _sim(case):
    Lx, Ly = _box(case)
    return hqt.Simulation(case["nx"], case["ny"], case["nz"], Lx=Lx, Ly=Ly,
                          mu=case["mu"], vy=case["vy"], dt=case["dt"],
                          remove_winding=case["winding"], precision=case["precision"])


def prepare(case, seed):
    do = case["do"]
    if do == "ensemble":
        members = _members(case)
        sims = [_sim(m) for m in members]
        first = [_state(m, 100 * seed + i) for i, m in enumerate(members)]
        # the ensemble before its members, the order they are released in
        return {"case": case, "ens": hqt.Ensemble(sims), "sims": sims, "first": first,
                "now": [[t.clone() for t in s] for s in first]}
    state = {"case": case, "sim": _sim(case)}
    first = _state(case, seed)
    if do == "host_step":
        state["first"] = [_host(t) for t in first]
    elif do == "filter":
        g = torch.Generator(device="cuda")
        g.manual_seed(7919 * int(seed) + 3)
        x = torch.randn(case["fields"], case["nz"], case["ny"], case["nx"], dtype=torch.float64,
                        device="cuda", generator=g)
        # the fields that are filtered: a profile and a disturbance
        state["x"] = first[1][None] + 1e-2 * x
        state["out"] = torch.empty_like(state["x"])
    else:
        state["first"] = first
        if do == "step":
            state["now"] = [t.clone() for t in first]
    return state


# ---- one pass ---------------------------------------------------------------
def run(state):
    """One pass.  A run of steps starts from the prepared fields, which the
    call then advances in place."""
    case = state["case"]
    do = case["do"]
    if do == "step":
        torch._foreach_copy_(state["now"], state["first"])
        info = state["sim"].step_device(*state["now"], nsteps=case["steps"])
        return {"fields": state["now"], "steps": info.steps_done, "winding": info.last_winding}
    if do == "host_step":
        fields, info = state["sim"].step(*state["first"], nsteps=case["steps"])
        return {"fields": list(fields), "steps": info.steps_done, "winding": info.last_winding}
    if do == "ensemble":
        torch._foreach_copy_([t for s in state["now"] for t in s],
                             [t for s in state["first"] for t in s])
        infos = state["ens"].step_device(state["now"], nsteps=case["steps"])
        # ten runs at most come back, spread over the set
        at = range(0, len(infos), -(-len(infos) // 10))
        return {"fields": [state["now"][i] for i in at], "steps": [infos[i].steps_done for i in at]}
    if do == "rhs":
        F1, F2, F3, F4 = state["sim"].rhs_device(*state["first"][:4])
        return {"F1": F1, "F2": F2, "F3": F3, "F4": F4}
    if do == "filter":
        return state["sim"].filter_device(state["x"], out=state["out"])
    sim = state["sim"]
    O, vx, vy, n = sim.boundary_fields_device(state["first"][0])
    k, E, Ec, Ei = sim.energy_spectrum_device(O)
    return {"O": O, "vx": vx, "vy": vy, "count": n, "k": k, "E": E, "Ec": Ec, "Ei": Ei}


def work(case):
    """Bytes that a pass cannot do without (each array read once and written
    once; a step also touches its RK accumulators once a stage) and the
    operations of its line transforms and column products."""
    if case["do"] == "ensemble":
        each = [work(dict(m, steps=case["steps"])) for m in _members(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    sites = nx * ny * nz
    lines = 5 * (math.log2(nx) + math.log2(ny))  # one complex transform each way, a site
    if case["do"] in ("step", "host_step"):
        each = 4 * (6.5 * lines + 12 * 4 * nz) + 6 * lines + 12 * nz
        return {"bytes": 368.0 * sites * case["steps"], "flops": each * sites * case["steps"]}
    if case["do"] == "rhs":
        return {"bytes": (40.0 + 32.0) * sites + 8 * nx * ny,
                "flops": (6.5 * lines + 12 * 4 * nz) * sites}
    if case["do"] == "filter":
        return {"bytes": 16.0 * sites * case["fields"], "flops": 1.0 * lines * sites * case["fields"]}
    return {"bytes": 16.0 * sites + 32.0 * nx * ny, "flops": 8.0 * sites + 10 * lines * nx * ny}


# ---- the same in plain torch, 64 bits ----------------------------------------
def _chebyshev(nz):
    """Points z = 1 (horizon) .. 0 (boundary), d/dz on them and the inverse of
    its leading block, from the differences in sine form."""
    f64 = {"dtype": torch.float64}
    j = torch.arange(nz, **f64)
    x = torch.sin(math.pi * (nz - 1 - 2 * j) / (2 * (nz - 1)))
    th = j * math.pi / (nz - 1)
    d = 2 * torch.sin((th[None] + th[:, None]) / 2) * torch.sin((th[None] - th[:, None]) / 2)
    # the lower half by the flip, where the differences are exact
    h = nz // 2
    d = torch.cat([d[:h], -torch.flip(d[:nz - h], (0, 1))])
    c = (-1.0) ** j
    c[0] *= 2
    c[-1] *= 2
    D = c[:, None] / c[None] / (d + torch.eye(nz, **f64))
    D = D - torch.diag(torch.diag(D))
    D = 2 * (D - torch.diag(D.sum(1)))
    return (x + 1) / 2, D, torch.linalg.inv(D[:nz - 1, :nz - 1])


def _wave(n, L):
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
    if n % 2 == 0:
        k[n // 2] = 0
    return k * (2 * math.pi / L)


class _Plain:
    """The step of one run, after `tevol_driven_cluster.m:60-142`."""

    def __init__(self, case):
        self.c = case
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        z, D, I = _chebyshev(nz)
        self.z, self.D, self.I = z.cuda()[:, None, None], D.cuda(), I.cuda()
        self.kx, self.ky = (_wave(n, L) for n, L in zip((nx, ny), _box(case)))

        def band(n):
            f = torch.zeros(n, dtype=torch.bool, device="cuda")
            f[math.floor(n / 3 + 0.5) - 1:math.floor(2 * n / 3 + 0.5)] = True
            return f
        self.keep = (~(band(ny)[:, None] | band(nx)[None])).double()

    def x(self, a):
        d = torch.fft.ifft(1j * self.kx * torch.fft.fft(a, dim=2), dim=2)
        return d if a.is_complex() else d.real

    def y(self, a):
        d = torch.fft.ifft(1j * self.ky[:, None] * torch.fft.fft(a, dim=1), dim=1)
        return d if a.is_complex() else d.real

    def zd(self, a):
        if a.is_complex():
            return torch.complex(self.zd(a.real), self.zd(a.imag))
        return (self.D @ a.reshape(a.shape[0], -1)).view(a.shape)

    def zr(self, a):
        if a.is_complex():
            return torch.complex(self.zr(a.real), self.zr(a.imag))
        out = torch.zeros_like(a)
        out[:-1] = (self.I @ a[:-1].reshape(a.shape[0] - 1, -1)).view_as(out[:-1])
        return out

    def rhs(self, p, at, ax, ay):
        f = 1 - self.z ** 3
        px, py, pz = self.x(p), self.y(p), self.zd(p)
        div = self.x(ax) + self.y(ay)
        F1 = self.zr(1j * at * pz + 0.5j * p * self.zd(at) + 0.5 * f * self.zd(pz)
                     - 1.5 * self.z ** 2 * pz - 0.5 * (self.z + ax * ax + ay * ay) * p
                     + 0.5 * (self.x(px) + self.y(py)) - 0.5j * p * div - 1j * (ax * px + ay * py))
        curl = self.x(ay) - self.y(ax)
        dens = p.real ** 2 + p.imag ** 2
        F3 = self.zr(0.5 * self.zd(self.x(at) + f * self.zd(ax)) - 0.5 * self.y(curl)
                     + (p.conj() * px).imag - ax * dens)
        F4 = self.zr(0.5 * self.zd(self.y(at) + f * self.zd(ay)) + 0.5 * self.x(curl)
                     + (p.conj() * py).imag - ay * dens)
        return F1, self.zd(div)[-1], F3, F4

    def filt(self, a):
        return torch.fft.ifft2(self.keep * torch.fft.fft2(a)).real

    def step(self, p, at, ax, ay, rho):
        h, ny = self.c["dt"], self.c["ny"]
        q = (p, ax, ay)
        k, sums, dq = None, [0, 0, 0], 0
        for s, w in ((0, 1), (0.5, 2), (0.5, 2), (1, 1)):
            y = q if k is None else tuple(a + s * b for a, b in zip(q, k))
            F1, F2, F3, F4 = self.rhs(y[0], at, y[1], y[2])
            k = [h * F1, h * F3, h * F4]
            for a in k:
                a[-1] = 0
            sums = [a + (w / 6) * b for a, b in zip(sums, k)]
            dq = dq + (w / 6) * h * F2
            del F1, F3, F4, y
        p, ax, ay = (a + b for a, b in zip(q, sums))
        rho = rho - dq
        cons = self.zd(self.x(ax) + self.y(ay)) - 2 * (p.conj() * self.zd(p)).imag
        at = self.zr(self.zr(cons) - rho) + self.c["mu"]
        p[-1], ax[-1], at[-1], ay[-1] = 0, 0, self.c["mu"], -self.c["vy"]
        wind = 0
        if self.c["winding"]:
            O = self.zd(p)[-1]
            turn = torch.angle(torch.roll(O, -1, 0) / O).sum(0).mean() / (2 * math.pi)
            wind = int(math.floor(abs(float(turn)) + 0.5)) * (1 if turn >= 0 else -1)
            j = torch.arange(ny, dtype=torch.float64, device="cuda") / ny
            p = p * torch.polar(torch.ones_like(j), -2 * math.pi * wind * j)[:, None]
        p = torch.complex(self.filt(p.real), self.filt(p.imag))
        return (p, self.filt(at), self.filt(ax), self.filt(ay), rho), wind


def _steps(case, fields):
    plain, wind = _Plain(case), 0
    for _ in range(case["steps"]):
        fields, wind = plain.step(*fields)
    return list(fields), wind


def exact(case, seed):
    do = case["do"]
    if do == "ensemble":
        members = _members(case)
        at = range(0, len(members), -(-len(members) // 10))
        done = [_steps(dict(members[i], steps=case["steps"]), _state(members[i], 100 * seed + i))[0]
                for i in at]
        return {"fields": [d[:4] + [d[4].contiguous()] for d in done],
                "steps": [case["steps"]] * len(done)}
    if do == "filter":
        return _Plain(case).filt(prepare(case, seed)["x"])
    first = _state(case, seed)
    if do in ("step", "host_step"):
        fields, wind = _steps(case, first)
        fields[4] = fields[4].contiguous()
        if do == "host_step":
            fields = [_host(t) for t in fields]
        return {"fields": fields, "steps": case["steps"], "winding": wind}
    plain = _Plain(case)
    if do == "rhs":
        F1, F2, F3, F4 = plain.rhs(*first[:4])
        return {"F1": F1, "F2": F2, "F3": F3, "F4": F4}
    O = plain.zd(first[0])[-1]
    a = O.abs()
    w = a / a.amax(1, keepdim=True)
    flow = []
    for d in (plain.x, plain.y):
        dO, da = d(O[None])[0], d(a[None])[0]
        flow.append(w * (-1j * (dO - da * O / a) / O).real)
    # a mode on the edge of a shell falls on either side of it by rounding: the
    # spectrum has no value that another arithmetic gives too
    return {"O": O, "vx": flow[0], "vy": flow[1], "count": None, "k": None, "E": None,
            "Ec": None, "Ei": None}
