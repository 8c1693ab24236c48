"""The work a user of this framework has it do, as cases that can be timed and compared.

The users are: someone who steps a lattice through the reference's kernel interface; someone who runs
one wall (the command line's time loop: chunks of steps in the averaging phase, in each storage type
and in both streaming patterns); someone who runs many walls together (both batch modes); the viewer
payload taken every few hundred steps; the solve server's turnover of a resident wall; and the
checkpoint's way through host memory.  Domains are the two families of stonewall.params, in H:
"baseline" 20 x 4 x 4 and "reference" 20 x 4 x 8 (plus one level), with other lengths among the drawn
ones, as the command line's --up, --down, --span and --height give them.

A case's state starts from populations made here (power-law inlet profile, a few long waves, 2 % noise
and a small non-equilibrium part; stones at rest) on a stone mask made here, so that exact() can step
the same inputs in float64 without the package.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "jeju-stonewall-lbm_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

CX = (0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0)
CY = (0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1)
CZ = (0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1)
OPP = (0,) + tuple(i + 1 if i % 2 else i - 1 for i in range(1, 19))
MIRZ = (0, 1, 2, 3, 4, 6, 5, 7, 8, 9, 10, 13, 14, 11, 12, 17, 18, 15, 16)
WEIGHT = (1 / 3,) + (1 / 18,) * 6 + (1 / 36,) * 12
BYTES = {"f32": 4, "f16": 2, "bf16": 2, "f64": 8}
TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "f64": torch.float64}
NU_SPONGE = 0.05
ACC_EVERY = 5


def _case(name, kind, H, dtype, steps=0, pattern="ab", mode="", domain="baseline", up=None, down=None, span=4.0,
          height=None, porosity=0.2, Re=1e4, walls=""):
    base = domain == "baseline"
    return dict(name=name, kind=kind, H=H, dtype=dtype, steps=steps, pattern=pattern, mode=mode, domain=domain,
                up=up if up is not None else (5.0 if base else 4.0),
                down=down if down is not None else (15.0 if base else 16.0), span=span,
                height=height if height is not None else (4.0 if base else 8.0), porosity=porosity, Re=Re, walls=walls)


def listed():
    return [
        # one eager step of a very small lattice through launch(k_step, ...), the reference's own call:
        # the smallest call there is, all launch and host latency
        _case("launch_step_tiny_f32", "launch", 5, "f32", steps=1, Re=400.0),
        # a quick look at a wall (--H 16): the smallest solve in use, float32 as the reference stores it
        _case("solve_f32_h16", "solve", 16, "f32", steps=100),
        # the headline wall, 800 x 160 x 160, in float32
        _case("solve_f32_h40", "solve", 40, "f32", steps=50),
        # the same wall in fp16 shifted storage, what the batches and the server run
        _case("solve_f16_h40", "solve", 40, "f16", steps=50),
        # a small wall whose rows are no multiple of 32 cells (420 x 84 x 84), fp16
        _case("solve_f16_h21", "solve", 21, "f16", steps=100),
        # float64 storage: the precision run that the other storage types are held against
        _case("solve_f64_h24", "solve", 24, "f64", steps=50),
        # in place (one lattice), fp16: walls of which twice as many have to fit the memory
        _case("solve_aa_f16_h32", "solve", 32, "f16", steps=50, pattern="aa"),
        # many walls together as the server advances them: one graph of per-wall chains, H from the batch study
        _case("batch_graph_f16", "batch", 40, "f16", steps=50, mode="graph", walls="16,24,32,40,16,24,32,40"),
        # many small walls in the persistent kernel, a batch's default mode, float32
        _case("batch_persistent_f32", "batch", 24, "f32", steps=50, mode="persistent", walls="12,16,20,24,15,18"),
        # a viewer frame of the command line's default wall (800 x 160 x 321): two planes and the Q-criterion
        _case("payload_f32_h40", "payload", 40, "f32", domain="reference"),
        # the server retires a finished solve (statistics on the GPU) and admits the next request
        _case("turnover_f16_h32", "turnover", 32, "f16"),
        # a state taken to host memory and back in the reference's layout, as checkpoints are
        _case("checkpoint_f32_h24", "checkpoint", 24, "f32"),
    ]


def draw(rng):
    """One more case of the same ranges: H over 8 to 40, domain lengths as the command line takes them."""
    kind = rng.choice(["solve"] * 6 + ["batch", "batch", "payload", "turnover", "checkpoint", "launch"])
    logint = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    more = dict(up=round(rng.uniform(3.0, 6.0), 2), down=round(rng.uniform(8.0, 15.0), 2),
                span=round(rng.uniform(2.0, 4.0), 2), porosity=round(rng.uniform(0.0, 0.5), 2))
    more["height"] = round(rng.uniform(3.0, 4.0), 2)
    if kind == "solve":
        dtype = rng.choice(["f32", "f32", "f16", "f16", "f16", "f64", "bf16"])
        pattern = rng.choice(["ab", "ab", "aa"])
        return _case("", kind, logint(8, 24 if dtype == "f64" else 40), dtype, steps=50,
                     pattern=pattern, **more)
    if kind == "batch":
        dtype, mode = rng.choice(["f32", "f16"]), rng.choice(["graph", "persistent"])
        hs = sorted(logint(8, 32) for _ in range(rng.randint(2, 8)))
        return _case("", kind, max(hs), dtype, steps=50, mode=mode, walls=",".join(map(str, hs)), **more)
    if kind == "payload":
        more["height"] = round(rng.uniform(5.0, 8.0), 2)
        return _case("", kind, logint(8, 40), rng.choice(["f32", "f16"]), domain="reference", **more)
    if kind == "launch":
        return _case("", kind, logint(4, 12), rng.choice(["f32", "f16"]), steps=1, Re=400.0, **more)
    return _case("", kind, logint(8, 32 if kind == "turnover" else 24), rng.choice(["f32", "f16"]), **more)


# ---------------------------------------------------------------- inputs
class _Wall:
    """Grid, physics and stone mask of one wall (numpy, from the case and the seed alone)."""

    def __init__(self, case, seed, H=None):
        H = self.H = int(H if H is not None else case["H"])
        base = case["domain"] == "baseline"
        self.nx = int(round((case["up"] + case["down"]) * H))
        self.ny = int(round(case["span"] * H))
        self.nz = int(round(case["height"] * H)) + (0 if base else 1)
        self.X0, self.T = int(round(case["up"] * H)), max(2, int(round((0.75 if base else 0.3) * H)))
        zeta = np.arange(self.nz) - 0.5
        if base:
            self.UH, self.cs, prof = 0.05, 0.1, 0.05 * np.clip(zeta / H, 0, None) ** (1 / 7)
        else:
            self.UH, self.cs = 0.08 * (1 / 3) ** (1 / 7), 0.16
            prof = 0.08 * np.clip(zeta / (3.0 * H), 0, 1) ** (1 / 7)
        self.uin = prof.astype(np.float32)
        self.uin[0] = 0.0
        self.nu0 = self.UH * H / case["Re"]
        self.x_sponge = self.nx - 3 * H
        self.cells = self.nx * self.ny * self.nz
        self.flag = self._stones(np.random.default_rng(seed), case["porosity"])

    def _stones(self, rng, porosity):
        """Ellipsoids dropped into the wall box until 1 - porosity of it is stone; y is periodic."""
        H, T, ny = self.H, self.T, self.ny
        hz = min(H, self.nz - 1)
        box = np.zeros((T, ny, hz), bool)
        if porosity <= 0.01:
            box[:] = True
        x, z = np.arange(T)[:, None, None] + 0.5, np.arange(hz)[None, None, :] + 0.5
        filled, want = int(box.sum()), (1.0 - porosity) * box.size
        while filled < want:
            semi = np.maximum(rng.uniform(0.15, 0.3, 3) * H, 1.0)
            cx, cy, cz = rng.uniform(0, T), rng.uniform(0, ny), rng.uniform(0, hz)
            half = min(int(semi[1]) + 1, (ny - 1) // 2)
            ys = int(cy) + np.arange(-half, half + 1)
            y = (ys + 0.5)[None, :, None]
            inside = ((x - cx) / semi[0]) ** 2 + ((y - cy) / semi[1]) ** 2 + ((z - cz) / semi[2]) ** 2 <= 1.0
            at = np.ix_(np.arange(T), ys % ny, np.arange(hz))
            old = box[at]
            filled += int((inside & ~old).sum())
            box[at] = old | inside
        flag = np.zeros((self.nx, ny, self.nz), np.uint8)
        flag[self.X0:self.X0 + T, :, 1:1 + hz][box] = 1
        flag[:, :, 0] = 2
        return flag


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _velocity(w, seed, real):
    """A velocity field (3, nx, ny, nz): the inlet profile, a wake behind the wall, long waves and 2 % noise."""
    dev = _device()
    rng = np.random.default_rng(seed + 7)
    gen = torch.Generator(device=dev).manual_seed(seed)
    x = torch.arange(w.nx, dtype=real, device=dev)[:, None, None]
    y = torch.arange(w.ny, dtype=real, device=dev)[None, :, None]
    z = torch.arange(w.nz, dtype=real, device=dev)[None, None, :]
    uin = torch.from_numpy(w.uin).to(dev, real)[None, None, :]
    u = torch.empty((3, w.nx, w.ny, w.nz), dtype=real, device=dev)
    wake = torch.where((x > w.X0) & (z < 1.2 * w.H), 0.7 * torch.exp(-(x - w.X0) / (5.0 * w.H)), torch.zeros_like(x))
    for k in range(3):
        wave = torch.zeros((1, 1, 1), dtype=real, device=dev)
        for _ in range(2):
            a, b, c = (int(v) for v in rng.integers(1, 5, 3))
            ph = float(rng.uniform(0, 6.28))
            wave = wave + torch.sin(6.283185307 * (a * x / w.nx + b * y / w.ny + c * z / w.nz) + ph)
        noise = torch.randn((w.nx, w.ny, w.nz), generator=gen, dtype=real, device=dev)
        u[k] = uin * ((1.0 - wake if k == 0 else 0.0) + 0.05 * wave + 0.02 * noise)
    u[:, torch.from_numpy(w.flag).to(dev) != 0] = 0.0
    return u


def _populations(w, seed, dtype):
    """f in the reference layout (19, nx, ny, nz), float32 (float64 for f64 storage), on the GPU."""
    real = torch.float64 if dtype == "f64" else torch.float32
    dev = _device()
    u = _velocity(w, seed, real)
    gen = torch.Generator(device=dev).manual_seed(seed + 1)
    usq = 1.5 * (u * u).sum(0)
    f = torch.empty((19, w.nx, w.ny, w.nz), dtype=real, device=dev)
    for i in range(19):
        cu = 3.0 * (CX[i] * u[0] + CY[i] * u[1] + CZ[i] * u[2])
        off = torch.randn((w.nx, w.ny, w.nz), generator=gen, dtype=real, device=dev)
        f[i] = WEIGHT[i] * (1.0 + cu + 0.5 * cu * cu - usq + 1e-4 * off)
    return f


def _solver(w, case, f0, n_total=40000, n_spin=0):
    from stonewall.solver import WallSolver
    s = WallSolver(w.flag, w.uin, w.nu0, w.cs, w.x_sponge, n_total, n_spin=n_spin, nu_sponge=NU_SPONGE,
                   dtype=case["dtype"], pattern=case["pattern"], acc_every=ACC_EVERY)
    s.state.assign(f0)
    return s


def prepare(case, seed):
    import warnings
    warnings.simplefilter("ignore")              # bf16 storage warns about its bias
    kind = case["kind"]
    if kind == "batch":
        from stonewall.batch import Batch
        b = Batch(dtype=case["dtype"], chunk=50, mode=case["mode"])
        flags = []
        for k, H in enumerate(case["walls"].split(",")):
            w = _Wall(case, seed * 100 + k, int(H))
            b.add(_solver(w, case, _populations(w, seed * 100 + k, case["dtype"])))
            flags.append((torch.from_numpy(w.flag).cuda(), torch.from_numpy(w.uin).cuda()))
        max(b.members, key=lambda m: m.grid.cells).autotune()    # as the server tunes a storage type, once
        return dict(case=case, batch=b, flags=flags)
    w = _Wall(case, seed)
    if kind == "launch":
        from stonewall.fields import Flags, ForceSeries, Grid, Lattice
        from stonewall.kernels import DeviceVector, tables_host
        g = Grid(w.nx, w.ny, w.nz)
        return dict(case=case, w=w, grid=g, flag=Flags(g, w.flag), uin=DeviceVector(w.uin), tables=tables_host(),
                    f=[Lattice(g, case["dtype"]).assign(_populations(w, seed, case["dtype"])),
                       Lattice(g, case["dtype"]).zero_()], force=ForceSeries(40000, w.nz), t=0)
    if kind == "turnover":
        # a finished solve on the GPU (its force series and sums), and the next request with its mask
        from stonewall.params import baseline_params
        from stonewall.serve import Request
        old = _solver(w, case, _populations(w, seed, case["dtype"]), n_total=20000)
        rng = np.random.default_rng(seed + 3)
        t = np.arange(old.n_total)[:, None, None]
        row = rng.uniform(0.5, 1.5, (1, w.nz, 2)) * 1e-2 * w.ny
        row[:, w.H + 1:] = 0.0
        force = row * (1.0 + 0.1 * np.sin(t / 97.0) + 0.05 * rng.standard_normal((old.n_total, w.nz, 2)))
        old.force.assign(force)
        old.t, old.n_acc = old.n_total, old.n_total // ACC_EVERY
        mean = _velocity(w, seed + 5, torch.float64) - 0.2 * w.UH
        sums = torch.empty((4, w.nz, w.ny, old.grid.pitch), dtype=torch.float64, device="cuda").zero_()
        sums[0, :, :, :w.nx] = float(old.n_acc)
        sums[1:, :, :, :w.nx] = old.n_acc * mean.permute(0, 3, 2, 1)
        old.acc.data.copy_(sums.ravel())
        old.params = baseline_params(w.H, old.n_total)
        old.params.X0, old.params.ny = w.X0, w.ny
        nxt = _Wall(case, seed + 1)
        p = baseline_params(nxt.H, 20000)
        p.nx, p.ny, p.nz, p.X0, p.T, p.uin, p.x_sponge = nxt.nx, nxt.ny, nxt.nz, nxt.X0, nxt.T, nxt.uin, nxt.x_sponge
        req = Request(rid=0, t_arrive=0.0, H=nxt.H, porosity=case["porosity"], U=0.05, steps=20000,
                      dtype=case["dtype"], seed=1000 + seed)
        return dict(case=case, old=old, req=req, p=p, flag=nxt.flag)
    s = _solver(w, case, _populations(w, seed, case["dtype"]))
    if kind == "solve":
        s.autotune()                             # as the command line does before its time loop
        return dict(case=case, w=w, s=s, flag=(torch.from_numpy(w.flag).cuda(), torch.from_numpy(w.uin).cuda()))
    if kind == "checkpoint":
        from stonewall.fields import Lattice
        return dict(case=case, s=s, other=Lattice(s.grid, case["dtype"]).zero_())
    ds = max(1, int(round(w.H / 13)))            # the command line's choices for a frame
    x0 = max(1, w.X0 - int(round(0.5 * w.H)))
    dims = (min(int(round(9.0 * w.H)), w.nx - 1 - x0) // ds, w.ny // ds, min(int(round(2.5 * w.H)), w.nz - 1) // ds)
    return dict(case=case, s=s, y_mid=w.ny // 2, z_half=int(round(0.5 * w.H)) + 1, x0=x0, ds=ds, dims=dims,
                scale=(w.H / w.UH) ** 2)


# ---------------------------------------------------------------- one pass
def _cells(t, k, g, nx):
    """A field's tensor [k, nz, ny, nx] without the padding columns of its rows."""
    return t.view(k, g.nz, g.ny, g.pitch)[..., :nx]


def _results(s, t0, n):
    """What a user takes from a solve on the GPU: the populations, the steps' wall forces and the sums of
    (rho, u), the latter two in float32 as the result files hold them."""
    g = s.grid
    return dict(f=_cells(s.state.data.view(TORCH[_NAMES[s.dtype]]), 19, g, g.nx),
                force=s.force.data[t0:t0 + n].to(torch.float32) * 2.0 ** -40,
                sums=_cells(s.acc.data, 4, g, g.nx).to(torch.float32))


_NAMES = {0: "f32", 1: "f64", 2: "f16", 3: "bf16"}


def run(state):
    case = state["case"]
    kind, n = case["kind"], case["steps"]
    if kind == "solve":
        s = state["s"]
        if s.t + n > s.n_total:                  # the solve is complete: the next one on the same buffers
            s.reload(*state["flag"])
        t0 = s.t
        s.advance(n)
        return _results(s, t0, n)
    if kind == "batch":
        b = state["batch"]
        if b.members[0].t + n > b.members[0].n_total:
            for m, fl in zip(b.members, state["flags"]):
                m.reload(*fl)
        t0 = b.members[0].t
        b.advance(n)
        return [_results(m, t0, n) for m in b.members]
    if kind == "launch":
        from stonewall.kernels import k_step, launch
        w, g = state["w"], state["grid"]
        f_in, f_out = state["f"]
        cx, cy, cz, wt, opp, mirz = state["tables"]
        if state["t"] == state["force"].n_steps:
            state["force"].data.zero_()
            state["t"] = 0
        t = state["t"]
        launch(k_step, (g.nx, g.ny, g.nz), [f_in, f_out, state["flag"], state["uin"], cx, cy, cz, wt, opp, mirz,
                                            g.nx, g.ny, g.nz, w.nu0, w.cs, w.x_sponge, NU_SPONGE, state["force"], t])
        state["f"].reverse()
        state["t"] = t + 1
        return dict(f=_cells(f_out.data.view(TORCH[case["dtype"]]), 19, g, g.nx), force=state["force"].data[t])
    if kind == "payload":
        s = state["s"]
        xz, xy = s.snapshot(state["y_mid"], state["z_half"])
        q = s.q_frame(state["x0"], state["ds"], state["dims"], state["scale"], macro_ready=True)
        return dict(xz=xz, xy=xy, q=q)
    if kind == "turnover":
        from stonewall.serve import make_solver, solve_stats
        stats = solve_stats(state["old"])
        new = make_solver(state["req"], state["p"], state["flag"], pattern=case["pattern"])
        g = new.grid
        return dict(stats=stats, f=_cells(new.state.data.view(TORCH[case["dtype"]]), 19, g, g.nx),
                    classes=new.flags.tiles)
    f = state["s"].state_numpy(np.float64 if case["dtype"] == "f64" else np.float32)
    state["other"].assign(f)
    g = state["s"].grid
    return dict(host=f, f=_cells(state["other"].data.view(TORCH[case["dtype"]]), 19, g, g.nx))


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes and operations of one pass: a step reads and writes every population of every cell once (and on
    an accumulating step the four float64 sums), about 300 operations a cell; the other kinds move each
    field they take once and each they give once."""
    def cells(H):
        extra = 0 if case["domain"] == "baseline" else 1
        return (int(round((case["up"] + case["down"]) * H)) * int(round(case["span"] * H))
                * (int(round(case["height"] * H)) + extra))
    kind, size, n = case["kind"], BYTES[case["dtype"]], case["steps"]
    if kind in ("solve", "batch"):
        c = sum(cells(int(h)) for h in case["walls"].split(",")) if kind == "batch" else cells(case["H"])
        return dict(bytes=c * (n * 38 * size + math.ceil(n / ACC_EVERY) * 64), flops=c * n * 300)
    c = cells(case["H"])
    if kind == "launch":
        return dict(bytes=c * 38 * size, flops=c * 300)
    if kind == "payload":
        return dict(bytes=c * 19 * size, flops=c * 60)
    if kind == "turnover":
        nz = int(round(case["height"] * case["H"]))
        # the force series and the recirculation box once; the new mask, two lattices and the sums once
        return dict(bytes=20000 * nz * 16 + c * (2 + 38 * size + 32), flops=c * 150)
    return dict(bytes=c * 19 * (2 * size + 8), flops=c * 19)


# ---------------------------------------------------------------- the same in float64
class _Exact:
    """The time step on [19, nz, ny, nx] float64 tensors, written from its equations."""

    def __init__(self, w, f0):
        dev = f0.device
        self.w = w
        self.flag = torch.from_numpy(w.flag).to(dev).permute(2, 1, 0).contiguous()
        self.fluid = self.flag == 0
        self.f = [f0, torch.zeros_like(f0)]
        self.uin = torch.from_numpy(w.uin).to(dev, torch.float64)[:, None]
        x = torch.arange(w.nx, device=dev, dtype=torch.float64)
        s = torch.clamp(x - w.x_sponge, min=0.0) / (w.nx - w.x_sponge)
        self.tau0 = 3.0 * (w.nu0 + NU_SPONGE * s * s) + 0.5
        self.sums = torch.zeros((4,) + tuple(self.flag.shape), dtype=torch.float64, device=dev)
        self.force = []
        ground = torch.full_like(self.flag[:1], 2)
        self.src = [self._shift(self.flag, self.flag[-1:], ground, i) for i in range(19)]

    @staticmethod
    def _shift(a, top, below, i):
        """a at the pull source of population i: z clamped to `top` / `below`, y periodic, outlet copy."""
        if CZ[i] == 1:
            a = torch.cat((below, a[:-1]))
        elif CZ[i] == -1:
            a = torch.cat((a[1:], top))
        if CY[i]:
            a = torch.roll(a, CY[i], 1)
        if CX[i] == 1:
            a = torch.cat((a[..., :1], a[..., :-1]), 2)
        elif CX[i] == -1:
            a = torch.cat((a[..., 1:], a[..., -1:]), 2)
        return a

    def step(self, accumulate):
        f, out = self.f
        pull = []
        pulls = self.fluid.clone()
        pulls[..., 0] = False                    # the inlet column does not pull
        fx = torch.zeros(f.shape[1], dtype=torch.float64, device=f.device)
        fz = torch.zeros_like(fx)
        for i in range(19):
            v = f[0] if i == 0 else self._shift(f[i], f[MIRZ[i]][-1:], f[i][:1], i)
            if i:
                own = f[OPP[i]]
                if CX[i] or CZ[i]:
                    hit = torch.where((self.src[i] == 1) & pulls, own - WEIGHT[i], torch.zeros_like(own)).sum((1, 2))
                    fx -= 2.0 * CX[i] * hit
                    fz -= 2.0 * CZ[i] * hit
                v = torch.where(self.src[i] != 0, own, v)
            pull.append(v)
        self.force.append(torch.stack((fx, fz), 1))
        rho = sum(pull)
        m = [sum(c[i] * pull[i] for i in range(19) if c[i]) for c in (CX, CY, CZ)]
        u = [a / rho for a in m]
        C = (CX, CY, CZ)
        neq = {}
        for a in range(3):
            for b in range(a, 3):
                p = sum(C[a][i] * C[b][i] * pull[i] for i in range(19) if C[a][i] * C[b][i])
                neq[a, b] = p - (rho / 3.0 if a == b else 0.0) - m[a] * u[b]
        del pull
        norm = torch.sqrt(sum(v * v * (1.0 if a == b else 2.0) for (a, b), v in neq.items()))
        cs2 = 18.0 * math.sqrt(2.0) * self.w.cs * self.w.cs
        tau = 0.5 * (self.tau0 + torch.sqrt(self.tau0 * self.tau0 + cs2 * norm / rho))
        keep = 1.0 - 1.0 / tau
        usq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
        for i in range(19):
            cu = 3.0 * (CX[i] * u[0] + CY[i] * u[1] + CZ[i] * u[2])
            q = sum(v * (C[a][i] * C[b][i] * (1.0 if a == b else 2.0) - (1.0 / 3.0 if a == b else 0.0))
                    for (a, b), v in neq.items())
            val = WEIGHT[i] * (rho * (1.0 + cu + 0.5 * cu * cu - usq) + 4.5 * keep * q)
            cu0 = 3.0 * CX[i] * self.uin
            val[..., 0] = WEIGHT[i] * (1.0 + cu0 + 0.5 * cu0 * cu0 - 1.5 * self.uin * self.uin)
            out[i] = torch.where(self.fluid, val, out[i])
        if accumulate:
            rho[..., 0] = 1.0
            u[0][..., 0] = self.uin
            u[1][..., 0] = 0.0
            u[2][..., 0] = 0.0
            for k, v in enumerate([rho] + u):
                self.sums[k] += torch.where(self.fluid, v, torch.zeros_like(v))
        self.f.reverse()


def _stored(f, dtype):
    """f (19, nx, ny, nz) as the storage type holds it, in float64 and [19, nz, ny, nx]."""
    if dtype in ("f16", "bf16"):
        g = torch.empty_like(f, dtype=torch.float64)
        for i in range(19):
            w32 = np.float32(WEIGHT[i])
            g[i] = (f[i] - float(w32)).to(TORCH[dtype]).double() + float(w32)
        f = g
    return f.double().permute(0, 3, 2, 1).contiguous()


def _weights(f, dtype):
    """Populations as the output holds them: f - w in the shifted types."""
    if dtype in ("f16", "bf16"):
        return f - torch.tensor(np.float32(WEIGHT), dtype=torch.float64, device=f.device)[:, None, None, None]
    return f


def _exact_solve(w, case, seed, n):
    e = _Exact(w, _stored(_populations(w, seed, case["dtype"]), case["dtype"]))
    for t in range(n):
        e.step(case["kind"] != "launch" and t % ACC_EVERY == 0)
    return e


def _pcg(s):
    m = 0xFFFFFFFF
    b = (s * 747796405 + 2891336453) & m
    c = ((((b >> ((b >> 28) + 4)) ^ b) & m) * 277803737) & m
    return (c >> 22) ^ c


def _exact_init(w, seed, dtype):
    """The start of a solve (k_init with Gaussian noise of 2 %), [19, nz, ny, nx]."""
    dev = _device()
    x = torch.arange(w.nx, device=dev)[None, None, :]
    y = torch.arange(w.ny, device=dev)[None, :, None]
    z = torch.arange(w.nz, device=dev)[:, None, None]
    st = _pcg((seed + _pcg((((x * 7919 + y) * 7907) + z) & 0xFFFFFFFF)) & 0xFFFFFFFF)
    r = []
    for _ in range(4):
        st = _pcg(st)
        r.append((st >> 8).double() / 16777216.0)
    a, b = torch.sqrt(-2.0 * torch.log(1.0 - r[0])), 2.0 * math.pi * r[1]
    c, d = torch.sqrt(-2.0 * torch.log(1.0 - r[2])), 2.0 * math.pi * r[3]
    u0 = torch.from_numpy(w.uin).to(dev, torch.float64)[:, None, None]
    noise = float(np.float32(0.02))
    u = [u0 * (1.0 + noise * a * torch.cos(b)), u0 * noise * a * torch.sin(b), u0 * noise * c * torch.cos(d)]
    fluid = torch.from_numpy(w.flag).to(dev).permute(2, 1, 0) == 0
    u = [torch.where(fluid, v, torch.zeros_like(v)) for v in u]
    usq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
    f = torch.empty((19,) + tuple(usq.shape), dtype=torch.float64, device=dev)
    for i in range(19):
        cu = 3.0 * (CX[i] * u[0] + CY[i] * u[1] + CZ[i] * u[2])
        f[i] = WEIGHT[i] * (1.0 + cu + 0.5 * cu * cu - usq)
    return _weights(f, dtype)


def exact(case, seed):
    kind, dtype, n = case["kind"], case["dtype"], case["steps"]
    pack = lambda e: dict(f=_weights(e.f[0], dtype), force=torch.stack(e.force), sums=e.sums)  # noqa: E731
    if kind == "batch":
        return [pack(_exact_solve(_Wall(case, seed * 100 + k, int(H)), case, seed * 100 + k, n))
                for k, H in enumerate(case["walls"].split(","))]
    w = _Wall(case, seed)
    if kind == "solve":
        return pack(_exact_solve(w, case, seed, n))
    if kind == "launch":
        e = _exact_solve(w, case, seed, 1)
        f = _weights(e.f[0], dtype)
        return dict(f=torch.where(e.fluid, f, torch.zeros_like(f)), force=None)
    if kind == "turnover":
        return dict(stats=None, f=_exact_init(_Wall(case, seed + 1), 1000 + seed, dtype), classes=None)
    f = _stored(_populations(w, seed, dtype), dtype)
    if kind == "checkpoint":
        return dict(host=f.permute(0, 3, 2, 1).contiguous(), f=_weights(f, dtype))
    fluid = torch.from_numpy(w.flag).to(f.device).permute(2, 1, 0) == 0
    rho = f.sum(0)
    u = torch.stack([sum(c[i] * f[i] for i in range(19) if c[i]) / rho for c in (CX, CY, CZ)])
    u = torch.where(fluid, u, torch.zeros_like(u))
    return dict(xz=u[:, :, w.ny // 2, :].permute(0, 2, 1).contiguous(),
                xy=u[:, int(round(0.5 * w.H)) + 1].permute(0, 2, 1).contiguous(), q=None)
