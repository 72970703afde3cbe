"""The work that programs have this package do, as timed cases.

A pass of a "step" case is a run segment as a solver program makes it: the
state goes up from page-locked host arrays, the boundary conditions are
applied, the time steps run (in one call, or one call per step where the
program reads the forces every step) and the centred fields come back into
page-locked arrays.  An "adjoint" pass is one evaluation of the gradient of the
mean force over K steps; a "mask" pass rebuilds the immersed body at an angle
and reads it back.  Sizes are those of the package's own configurations (the
40^3 and 128^3 cavities, the NACA 0012 and 0015 LES grids, the cylinder of the
adjoint), of its tests, and ragged ones between them.

``exact`` evaluates the same scheme with plain torch in 64 bits.
"""
import math

import numpy as np
import torch

F64 = torch.float64
KIND = {"no-slip": 0, "Neumann": 1, "Dirichlet": 2, "periodic": 3}


def f4(x):
    """A literal stored from a default real, as the solver's configurations have them."""
    return float(np.float32(x))


# ------------------------------------------------------------------ cases
def listed():
    cav = dict(kind="step", body="none", les=False, stretch=1.0, per_step=False, amp=0.2)
    foil = dict(kind="step", body="naca", les=True, stretch=12.0, per_step=False, amp=0.02)
    return [
        # the smallest grids of the tests and of interactive use: launches and latency only
        dict(cav, name="cavity 12x10x8 fp64", nx=12, ny=10, nz=8, mixed=False, Re=100.0, dt=1e-3, steps=4, per_step=True),
        # the reference's default cavity at full precision, forces read after every step
        dict(cav, name="cavity 40 fp64", nx=40, ny=40, nz=40, mixed=False, Re=100.0, dt=1e-3, steps=10, per_step=True),
        # odd sizes on a stretched grid, as a user's own geometry has them
        dict(cav, name="cavity 61x47x53 mixed", nx=61, ny=47, nz=53, mixed=True, Re=400.0, dt=1e-3, steps=10, stretch=4.0),
        # the headline cavity: start-up segment, mixed precision and plain FP64
        dict(cav, name="cavity 128 mixed", nx=128, ny=128, nz=128, mixed=True, Re=1000.0, dt=5e-4, steps=20),
        dict(cav, name="cavity 128 fp64", nx=128, ny=128, nz=128, mixed=False, Re=1000.0, dt=5e-4, steps=20),
        # the NACA 0012 LES case (impulsive start), mixed and FP64
        dict(foil, name="naca0012 les mixed", nx=64, ny=192, nz=256, mixed=True, Re=1000.0, dt=1e-3, steps=1, t=0.12, aoa=5.0),
        dict(foil, name="naca0012 les fp64", nx=64, ny=192, nz=256, mixed=False, Re=1000.0, dt=1e-3, steps=1, t=0.12, aoa=5.0),
        # the largest configured grid, the NACA 0015 LES case (12.6 M cells)
        dict(foil, name="naca0015 les mixed", nx=128, ny=256, nz=384, mixed=True, Re=5000.0, dt=5e-4, steps=1, t=0.15, aoa=10.0),
        dict(foil, name="naca0015 les fp64", nx=128, ny=256, nz=384, mixed=False, Re=5000.0, dt=5e-4, steps=1, t=0.15, aoa=10.0),
        # gradients of the cylinder's drag with a body force: the adjoint leg, both precisions
        dict(kind="adjoint", name="cylinder adjoint mixed", nx=32, ny=96, nz=96, mixed=True, Re=100.0, dt=5e-3, steps=10, every=5),
        dict(kind="adjoint", name="cylinder adjoint fp64 32x60x72", nx=32, ny=60, nz=72, mixed=False, Re=100.0, dt=5e-3, steps=8, every=3),
        # a body turned between two segments: ray casting on the NACA 0012 grid
        dict(kind="mask", name="mask naca0012", nx=64, ny=192, nz=256, t=0.12, aoa=5.0, npts=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cavity", "cavity", "foil", "adjoint", "mask"])
    if kind == "cavity":
        n = _log(rng, 9, 150)
        nx, ny, nz = (max(8, int(n * rng.uniform(0.75, 1.3))) for _ in range(3))
        return dict(kind="step", body="none", les=rng.random() < 0.25, stretch=rng.choice([1.0, 1.0, 4.0]),
                    per_step=rng.random() < 0.4, amp=rng.uniform(0.05, 0.3), nx=nx, ny=ny, nz=nz, mixed=rng.random() < 0.5,
                    Re=float(_log(rng, 100, 1000)), dt=f4(5e-4), steps=rng.randint(2, 10))
    if kind == "foil":
        nx = rng.choice([16, 24, 33, 48, 64, 96, 128])
        ny, nz = _log(rng, 96, 250), _log(rng, 120, 380)
        return dict(kind="step", body="naca", les=rng.random() < 0.7, stretch=rng.uniform(8.0, 12.0), per_step=False,
                    amp=rng.uniform(0.005, 0.03), nx=nx, ny=ny, nz=nz, mixed=rng.random() < 0.5, Re=float(_log(rng, 500, 5000)),
                    dt=5e-4, steps=1, t=rng.choice([0.12, 0.15]), aoa=rng.uniform(1.0, 12.0))
    if kind == "adjoint":
        return dict(kind="adjoint", nx=rng.randint(8, 40), ny=_log(rng, 40, 100), nz=_log(rng, 40, 100), mixed=rng.random() < 0.5,
                    Re=100.0, dt=5e-3, steps=rng.randint(3, 10), every=rng.randint(2, 6))
    return dict(kind="mask", nx=rng.randint(16, 128), ny=_log(rng, 90, 256), nz=_log(rng, 120, 384), t=rng.choice([0.12, 0.15]),
                aoa=rng.uniform(1.0, 12.0), npts=_log(rng, 100, 400))


# ------------------------------------------------------------ grid, body, state
def _nodes(n, length, centre, ratio):
    """n cells over [0, length], `ratio` times finer at `centre` than far from it."""
    if ratio <= 1.0:
        return np.linspace(0.0, length, n + 1)
    x = np.linspace(0.0, length, 20001)
    density = 1.0 + (ratio - 1.0) * np.exp(-((x - centre) / (0.08 * length)) ** 2)
    c = np.concatenate([[0.0], np.cumsum(0.5 * (density[1:] + density[:-1]))])
    return np.interp(np.linspace(0.0, c[-1], n + 1), c, x)


def _geometry(case):
    """(lengths, centres, ratios) of the three axes: x the span, y the normal, z the stream."""
    if case["kind"] == "adjoint":
        return (4.0, 12.0, 12.0), (2.0, 6.0, 4.0), (1.0, 1.0, 1.0)
    if case["kind"] == "mask" or case["body"] == "naca":
        return (1.0, 8.0, 16.0), (0.5, 4.0, 4.5), (1.0, case.get("stretch", 12.0), case.get("stretch", 12.0))
    return (1.0, 1.0, 1.0), (0.5, 0.0, 1.0), (1.0, case["stretch"], case["stretch"])


def _grid(case):
    """Node coordinates (index -1..n+3) and metrics iD, Ds (index -1..n+2) of a user's grid."""
    g = {}
    lengths, centres, ratios = _geometry(case)
    for ax, n, L, c, r in zip("xyz", (case["nx"], case["ny"], case["nz"]), lengths, centres, ratios):
        x = _nodes(n, L, c, r)
        h = np.diff(x)
        h = np.concatenate([[h[0], h[0]], h, [h[-1]] * 3])          # cells -1..n+3
        g["iD" + ax] = h[:n + 4].copy()
        g["D" + ax + "s"] = (0.5 * (h[:-1] + h[1:]))[:n + 4].copy()
        X = np.concatenate([[x[0] - 2 * h[0], x[0] - h[0]], x, [x[-1] + h[-1], x[-1] + 2 * h[-1]]])
        g[ax.upper()] = X                                           # nodes -1..n+3
    return g


def _foil(t, npts):
    """Closed symmetric four-digit section, leading edge -> upper -> trailing edge -> lower."""
    x = 0.5 * (1.0 - np.cos(np.pi * np.arange(npts) / (npts - 1)))
    y = 5.0 * t * (0.2969 * np.sqrt(x) - 0.1260 * x - 0.3516 * x ** 2 + 0.2843 * x ** 3 - 0.1036 * x ** 4)
    return np.concatenate([x, x[::-1]]), np.concatenate([y, -y[::-1]])


CENTRE = (4.0137, 4.0071)          # (zc, yc) of the airfoil


def _walls(case):
    """Wall kinds and Dirichlet values of the case."""
    if case["kind"] == "step" and case["body"] == "none":           # the lid moves in x
        return {"North": ("Dirichlet", "no-slip", "no-slip")}, {}
    return ({"West": ("periodic",) * 3, "East": ("periodic",) * 3, "South": ("Neumann",) * 3, "North": ("Neumann",) * 3,
             "Back": ("Dirichlet",) * 3, "Front": ("Neumann",) * 3}, {"Back": (0.0, 0.0, 1.0)})


def _state(case, seed):
    """Halo arrays u, v, w, p (index order k, j, i: Fortran order for the solver) on the GPU: the discrete
    curl of a few smooth random modes (no divergence, as a run's own fields have none), of amplitude `amp`,
    on rest or on the uniform inflow, and p = 0."""
    r = np.random.default_rng(seed)
    n = (case["nx"], case["ny"], case["nz"])
    amp, lengths, g = case.get("amp", 0.02), _geometry(case)[0], _grid(case)
    vel = [torch.zeros(n[2] + 4, n[1] + 4, n[0] + 4, dtype=F64, device="cuda") for _ in range(3)]
    for q in range(9):
        c = q % 3                                   # component of the vector potential
        a, b = (c + 1) % 3, (c + 2) % 3             # its curl: +d/da in component b, -d/db in component a
        F, D, m = [], [], [int(r.integers(1, 4)) for _ in range(3)]
        for ax in range(3):
            i = np.arange(-1, n[ax] + 3)
            F.append(np.sin(np.pi * m[ax] * i / n[ax]) if ax != c else np.cos(np.pi * m[ax] * (i - 0.5) / n[ax]))
            D.append((F[ax] - np.sin(np.pi * m[ax] * (i - 1) / n[ax])) / g["iD" + "xyz"[ax]])
        size = 0.3 * amp * float(r.uniform(0.5, 1.0)) / math.pi
        for comp, d, sign in ((b, a, -size * lengths[a] / m[a]), (a, b, size * lengths[b] / m[b])):
            x = [torch.tensor(D[ax] if ax == d else F[ax], device="cuda") for ax in range(3)]
            vel[comp] += sign * x[2][:, None, None] * x[1][:, None] * x[0]
    if case["kind"] == "adjoint" or case["body"] == "naca":
        vel[2] += 1.0
    return vel + [torch.zeros_like(vel[0])]


def _force(case, seed):
    """Body force of the adjoint cases, (nx, ny, nz) each, standard deviation 1e-3."""
    r = np.random.default_rng(seed + 7919)
    return [np.asfortranarray(r.normal(0.0, 1e-3, (case["nx"], case["ny"], case["nz"]))) for _ in range(3)]


def _pinned(t):
    """A page-locked Fortran-order array with the values of t (index order k, j, i)."""
    h = torch.empty(t.shape, dtype=F64, pin_memory=True)
    h.copy_(t)
    return h.numpy().T


# ------------------------------------------------------------ prepare, run
def prepare(case, seed):
    from ntustcfdlab_b200.abi import FP64, MIXED, make_params
    from ntustcfdlab_b200.solver import Solver
    bc, val = _walls(case)
    lengths = _geometry(case)[0]
    p = make_params(case["nx"], case["ny"], case["nz"], Re=case.get("Re", 1000.0), dt=f4(case.get("dt", 1e-3)),
                    precision=MIXED if case.get("mixed") else FP64, LES=1 if case.get("les") else 0, Cs=f4(0.1), bc=bc,
                    bc_value=val, lx=lengths[0])
    st = {"case": case, "solver": Solver(p, _grid(case))}
    s = st["solver"]
    if case["kind"] == "mask":
        st["foil"] = _foil(case["t"], case["npts"])
        st["aoa"] = case["aoa"] + float(np.random.default_rng(seed).uniform(-1.0, 1.0))
        st["eta"] = _pinned(torch.zeros(case["nz"] + 4, case["ny"] + 4, case["nx"] + 4, dtype=F64))
        return st
    if case["kind"] == "adjoint":
        s.build_mask_cylinder(4.0, 6.0, 0.5)
        s.set_body_force(*_force(case, seed))
    elif case["body"] == "naca":
        s.build_mask_polygon(*_foil(case["t"], 256), case["aoa"], *CENTRE)
    st["state"] = [_pinned(f) for f in _state(case, seed)]
    st["out"] = [_pinned(torch.zeros(case["nz"], case["ny"], case["nx"], dtype=F64)) for _ in range(4)]
    return st


def run(st):
    from ntustcfdlab_b200.abi import dptr
    case, s = st["case"], st["solver"]
    if case["kind"] == "mask":
        s.build_mask_polygon(*st["foil"], st["aoa"], *CENTRE)
        s._check(s.lib.ntcfd_get_mask(s.h, dptr(st["eta"])))
        return {"eta": st["eta"]}
    s.set_state(*st["state"])
    s.boundary_conditions()
    if case["kind"] == "adjoint":
        r = s.adjoint(case["steps"], case["every"], w_drag=1.0, w_lift=0.5, inflow=("Back", 2, 1))
        return {"J": r["J"], "dU": r["dJ_dU"], "dtheta": r["dJ_dtheta"], "df": r["dJ_df"],
                "sweeps": [i.sor_iters for i in r["info"]]}
    if case["per_step"]:
        info = [s.step(1)[0][0] for _ in range(case["steps"])]
    else:
        info = s.step(case["steps"])[0]
    s.output_async(st["out"])
    pre, uc, vc, wc = s.output_wait()
    return {"pre": pre, "uc": uc, "vc": vc, "wc": wc, "sweeps": np.array([i.sor_iters for i in info]),
            "drag": np.array([i.cDrag for i in info]), "lift": np.array([i.cLift for i in info])}


def work(case):
    """What a pass cannot do without: the state in and the fields out once, u, v, w and p read and written
    in every step, and the arithmetic of a step (some 430 operations in the predictor, 60 elsewhere) with one
    SOR sweep (15); the number of sweeps is the flow's.  An adjoint repeats the steps and transposes them."""
    n = case["nx"] * case["ny"] * case["nz"]
    halo = (case["nx"] + 4) * (case["ny"] + 4) * (case["nz"] + 4)
    if case["kind"] == "mask":
        return {"bytes": 8.0 * halo, "flops": 20.0 * case["ny"] * case["nz"] * 2 * case["npts"]}
    k = case["steps"] * (3 if case["kind"] == "adjoint" else 1)
    io = 8.0 * (4 * halo + (3 if case["kind"] == "adjoint" else 4) * n)
    return {"bytes": io + 64.0 * n * k, "flops": 505.0 * n * k}


# ------------------------------------------------------------ the same in 64 bits
class _Scheme:
    """The projection step on tensors f[k+1, j+1, i+1], i, j, k = -1..n+2."""

    def __init__(self, case):
        self.n = (case["nx"], case["ny"], case["nz"])
        g = _grid(case)
        t = lambda a: torch.tensor(a, dtype=F64, device="cuda")
        self.iD = [t(g["iD" + a]) for a in "xyz"]
        self.Ds = [t(g["D" + a + "s"]) for a in "xyz"]
        self.node = [t(g[a]) for a in "XYZ"]
        self.dt, self.nu = f4(case["dt"]) if "dt" in case else 0.0, 1.0 / case.get("Re", 1.0)
        self.les, self.lx = case.get("les", False), _geometry(case)[0][0]
        bc, val = _walls(case)
        names = ("West", "East", "South", "North", "Back", "Front")
        self.bc = [[KIND[k] for k in bc.get(w, ("no-slip",) * 3)] for w in names]
        self.val = [[t(v) for v in val.get(w, (1.0, 1.0, 1.0))] for w in names]
        c = lambda i, j: 1.0 / (i * j)
        at = lambda a, o, ax: a[2 + o:2 + o + self.n[ax]]
        self.cp = [self.line(c(at(self.iD[a], 0, a), at(self.Ds[a], 0, a)), a) for a in range(3)]
        self.cm = [self.line(c(at(self.iD[a], 0, a), at(self.Ds[a], -1, a)), a) for a in range(3)]
        self.rd = 1.0 / sum(self.cp[a] + self.cm[a] for a in range(3))
        self.rd = self.rd.expand(self.n[2], self.n[1], self.n[0])
        i = [torch.arange(1, m + 1, device="cuda") for m in self.n]
        self.red = ((i[0] + i[1][:, None] + i[2][:, None, None]) % 2 == 0)
        self.eta = torch.zeros(self.n[2], self.n[1], self.n[0], dtype=F64, device="cuda")
        self.fb = None

    def line(self, v, ax):
        return v.view([-1 if a == ax else 1 for a in (2, 1, 0)])

    def sh(self, f, *offs):
        """The interior of f shifted by unit steps: offs = (axis, steps) pairs."""
        o = [0, 0, 0]
        for ax, d in offs:
            o[ax] += d
        return f[tuple(slice(2 + o[a], 2 + o[a] + self.n[a]) for a in (2, 1, 0))]

    def at(self, v, ax, d):
        return self.line(v[2 + d:2 + d + self.n[ax]], ax)

    def quick(self, f, c, ax, t, d):
        """QUICK value at the face between cells d and d+1 (relative), upwinded on t."""
        if ax == c:
            h = self.at(self.iD[ax], ax, d + 1)
            A, B = 0.125 * h * h / self.at(self.Ds[ax], ax, d), 0.125 * h * h / self.at(self.Ds[ax], ax, d + 1)
            r = [1.0 / self.at(self.iD[ax], ax, d + q) for q in range(3)]
        else:
            h = self.at(self.Ds[ax], ax, d)
            A, B = 0.125 * h * h / self.at(self.iD[ax], ax, d), 0.125 * h * h / self.at(self.iD[ax], ax, d + 1)
            r = [1.0 / self.at(self.Ds[ax], ax, d - 1 + q) for q in range(3)]
        fm, f0, f1, f2 = (self.sh(f, (ax, d + q)) for q in (-1, 0, 1, 2))
        mid = 0.5 * (f0 + f1)
        return torch.where(t > 0, mid - A * ((f1 - f0) * r[1] - (f0 - fm) * r[0]), mid - B * ((f2 - f1) * r[2] - (f1 - f0) * r[1]))

    def predictor(self, vel, nut):
        nue = self.nu if nut is None else self.nu + nut
        out = []
        for c in range(3):
            f = vel[c]
            f0 = self.sh(f)
            r = f0
            for ax in range(3):
                V = vel[ax]
                t1 = 0.5 * (self.sh(V) + self.sh(V, (c, 1)))
                t2 = 0.5 * (self.sh(V, (ax, -1)) + self.sh(V, (c, 1), (ax, -1)))
                flux = t1 * self.quick(f, c, ax, t1, 0) - t2 * self.quick(f, c, ax, t2, -1)
                fp, fm = self.sh(f, (ax, 1)), self.sh(f, (ax, -1))
                if ax == c:
                    w = 1.0 / self.at(self.Ds[ax], ax, 0)
                    diff = (fp - f0) / self.at(self.iD[ax], ax, 1) - (f0 - fm) / self.at(self.iD[ax], ax, 0)
                else:
                    w = 1.0 / self.at(self.iD[ax], ax, 0)
                    diff = (fp - f0) / self.at(self.Ds[ax], ax, 0) - (f0 - fm) / self.at(self.Ds[ax], ax, -1)
                r = r - self.dt * flux * w + nue * self.dt * diff * w
            out.append(r if self.fb is None else r + self.dt * self.fb[c])
        return out

    def smagorinsky(self, vel, Cs):
        """Eddy viscosity with the reference's storage association of the halo arrays."""
        nx, ny, nz = self.n
        i, j, k = (torch.arange(1, m + 1, device="cuda") for m in self.n)
        off = (i - 1) + (j[:, None] - 1) * nx + (k[:, None, None] - 1) * nx * ny
        grads = []
        for c in range(3):
            flat = vel[c].reshape(-1)
            D = [self.at(self.Ds[a] if a == c else self.iD[a], a, 0) for a in range(3)]
            rd = lambda o: torch.where((o >= 0) & (o < flat.numel()), flat[o.clamp(0, flat.numel() - 1)], 0.0)
            grads.append([0.5 * (rd(off + s) - rd(off - s)) / D[a] for a, s in enumerate((1, nx, nx * ny))])
        S = sum(2 * grads[a][a] ** 2 for a in range(3))
        S = S + (grads[0][1] + grads[1][0]) ** 2 + (grads[0][2] + grads[2][0]) ** 2 + (grads[1][2] + grads[2][1]) ** 2
        vol = self.at(self.iD[0], 0, 0) * self.at(self.iD[1], 1, 0) * self.at(self.iD[2], 2, 0)
        return (Cs * vol ** float(np.float32(1) / np.float32(3))) ** 2 * S.abs().sqrt()

    def nbsum(self, p):
        return sum(self.cp[a] * self.sh(p, (a, 1)) + self.cm[a] * self.sh(p, (a, -1)) for a in range(3))

    def sor(self, p, b, omega=1.5, zeta=f4(1e-4), itmax=3000):
        """Red-black SOR in place on the interior of p (ghosts frozen); the sweep count."""
        x = self.sh(p)
        for it in range(1, itmax + 1):
            top = 0.0
            for colour in (self.red, ~self.red):
                d = torch.where(colour, torch.addcmul(-b, self.rd, self.nbsum(p)) - x, 0.0)
                x.add_(d, alpha=omega)
                top = torch.maximum(d.abs().max(), top) if torch.is_tensor(top) else d.abs().max()
            if float(top) <= zeta:
                break
        return it

    def conditions(self, vel, p):
        """The boundary conditions on copies of the fields."""
        vel, p = [f.clone() for f in vel], p.clone()
        for ax in range(3):
            n = self.n[ax]

            def pl(f, i):
                return f.select(2 - ax, i + 1)

            def put(f, i, v):
                pl(f, i).copy_(v.clone() if torch.is_tensor(v) and v.dim() else v)

            for c in range(3):
                f, lo, hi = vel[c], self.bc[2 * ax][c], self.bc[2 * ax + 1][c]
                vlo, vhi = self.val[2 * ax][c], self.val[2 * ax + 1][c]
                if c == ax:
                    v = (torch.zeros_like(pl(f, 1)), pl(f, 1), vlo.expand_as(pl(f, 1)), pl(f, n))[lo].clone()
                else:
                    v = (-pl(f, 1), pl(f, 1), 2 * vlo - pl(f, 1), pl(f, n))[lo].clone()
                if ax == 2 and c == 1 and lo == 1:
                    v = pl(f, 0).clone()
                put(f, 0, v)
                put(f, -1, pl(f, n - 1) if lo == 3 else v)
                if hi == 3:
                    put(f, n + 1, pl(f, 1))
                    put(f, n + 2, pl(f, 2))
                elif c == ax:
                    v = (torch.zeros_like(pl(f, 1)), pl(f, n - 1), vhi.expand_as(pl(f, 1)))[hi].clone()
                    for q in (n, n + 1, n + 2):
                        put(f, q, v)
                else:
                    v = (-pl(f, n), pl(f, n), 2 * vhi - pl(f, n))[hi].clone()
                    put(f, n + 1, v)
                    put(f, n + 2, v)
            per = self.bc[2 * ax][ax] == 3
            for dst, src in ((0, n if per else 1), (-1, n - 1 if per else 1), (n + 1, 1 if per else n), (n + 2, 2 if per else n)):
                put(p, dst, pl(p, src))
        return vel, p

    def force(self, F):
        """Guarded Simpson sums of a cell force over z, y and x."""
        nx, ny, nz = self.n
        k = torch.arange(nz, device="cuda")
        wz = self.Ds[2][2:2 + nz] * (4.0 + (k > 0).double() + (k < nz - 1).double()) / 6.0
        line = (F * wz[:, None, None]).sum(0)                                    # (ny, nx)
        for n, D in ((ny, self.Ds[1]), (nx, self.Ds[0])):
            z = torch.zeros_like(line[:1])
            w = D[1:n + 3].view(-1, *[1] * (line.dim() - 1))
            e = torch.cat([z, line, z])
            s = (e[:-2] * w[:-2] + 4.0 * line * w[1:-1] + e[2:] * w[2:]) / 6.0
            line = torch.where(line != 0, s, 0.0).sum(0)
        return -2.0 * line / self.lx

    def rhs(self, vel, star):
        """b' from the predicted velocity (the faces at index 0 are the state's)."""
        full = []
        div = 0.0
        for c in range(3):
            f = vel[c].clone()
            f[tuple(slice(2, 2 + self.n[a]) for a in (2, 1, 0))] = star[c]
            full.append(f)
            div = div + (star[c] - self.sh(f, (c, -1))) / self.at(self.iD[c], c, 0)
        return self.rd * div / self.dt

    def project(self, p, star):
        """Velocity after projection and forcing, and the two force integrals."""
        new, F = [], []
        for c in range(3):
            u1 = star[c] - self.dt * (self.sh(p, (c, 1)) - self.sh(p)) / self.at(self.Ds[c], c, 0)
            u2 = (1.0 - self.eta) * u1
            new.append(u2)
            F.append((u2 - u1) / self.dt)
        return new, self.force(F[2]), self.force(F[1])

    def commit(self, vel, new):
        out = []
        for c in range(3):
            f = vel[c].clone()
            f[tuple(slice(2, 2 + self.n[a]) for a in (2, 1, 0))] = new[c]
            out.append(f)
        return out

    def step(self, vel, p, solve):
        nut = self.smagorinsky(vel, f4(0.1)) if self.les else None
        star = self.predictor(vel, nut)
        p, it = solve(p, self.rhs(vel, star))
        new, drag, lift = self.project(p, star)
        vel = self.commit(vel, new)
        centred = [0.5 * (self.sh(vel[c]) + self.sh(vel[c], (c, -1))) for c in range(3)]
        pre = self.sh(p).clone()
        vel, p = self.conditions(vel, p)
        return vel, p, it, drag, lift, pre, centred

    # ---- bodies
    def extrude(self, e):
        self.eta = e[:, :, None].expand(self.n[2], self.n[1], self.n[0])

    def parity(self, Yn, Zn, Yc, Zc, py, pz, strict):
        """Odd crossings of the ray from (Yc, Zc), slopes taken from the nodes (Yn, Zn)."""
        cnt = torch.zeros_like(Yc, dtype=torch.int64)
        for m in range(len(py) - 1):
            a0, a1, z0, z1 = py[m], py[m + 1], pz[m], pz[m + 1]
            past = Zc > max(z0, z1) if strict else Zc >= max(z0, z1)
            before = Zc < min(z0, z1)
            down, up = (a0 >= Yc) & (a1 <= Yc), (a0 <= Yc) & (a1 >= Yc)
            slope = (a1 - a0) / (z1 - z0) if z1 != z0 else math.copysign(math.inf, a1 - a0)
            hit_d = (Yn - a1) / (Zn - z1) > slope
            hit_u = (Yn - a0) / (Zn - z0) > slope
            cnt += (down & (before | (~past & hit_d))).long() + (up & (before | (~past & hit_u))).long()
        return cnt % 2 == 1

    def polygon(self, z, y, aoa, zc, yc):
        nx, ny, nz = self.n
        c, s = math.cos(-aoa * math.pi / 180), math.sin(-aoa * math.pi / 180)
        z0 = z - 0.25
        z1 = c * z0 - s * y
        y1 = s * z1 + c * y
        pz, py = [float(v) for v in z1 + zc + 0.25], [float(v) for v in y1 + yc]
        Y, Z = self.node[1], self.node[2]
        Yl, Yh = Y[2:2 + ny].expand(nz, ny), Y[3:3 + ny].expand(nz, ny)
        Zl, Zh = Z[2:2 + nz, None].expand(nz, ny), Z[3:3 + nz, None].expand(nz, ny)
        e = self.parity(Yl, Zl, (Yl + Yh) / 2, (Zl + Zh) / 2, py, pz, False).double()
        Yi, Zi = Y.cpu().numpy()[2:], Z.cpu().numpy()[2:]
        cut = sorted({(int(np.searchsorted(Zi, a, "right")) - 1, int(np.searchsorted(Yi, b, "right")) - 1) for a, b in zip(pz, py)})
        cut = torch.tensor([q for q in cut if 0 <= q[0] < nz and 0 <= q[1] < ny], device="cuda")
        l = torch.arange(50, device="cuda", dtype=F64)
        kk, jj = cut[:, 0], cut[:, 1]
        y0, dy, z0_, dz = Yl[kk, jj], (Yh - Yl)[kk, jj], Zl[kk, jj], (Zh - Zl)[kk, jj]
        ya = (y0[:, None] + l * dy[:, None] / 50)[:, :, None].expand(-1, 50, 50)
        yb = (y0[:, None] + (l + 1) * dy[:, None] / 50)[:, :, None].expand(-1, 50, 50)
        za = (z0_[:, None] + l * dz[:, None] / 50)[:, None, :].expand(-1, 50, 50)
        zb = (z0_[:, None] + (l + 1) * dz[:, None] / 50)[:, None, :].expand(-1, 50, 50)
        odd = self.parity(ya, za, (ya + yb) / 2, (za + zb) / 2, py, pz, True)
        e[kk, jj] = odd.double().sum((1, 2)) / 50 / 50
        self.extrude(e)

    def cylinder(self, zc, yc, r):
        """50 x 50 sub-cells near the surface, with the single-precision steps of the reference."""
        nx, ny, nz = self.n
        f = lambda x: x.float()
        Y, Z = self.node[1], self.node[2]
        hy, hz, hx = self.iD[1][2:2 + ny], self.iD[2][2:2 + nz, None], self.iD[0][2]
        diag = f((hx ** 2 + hy ** 2 + hz ** 2).sqrt() / 2).double()
        dist = f((((Z[2:2 + nz] + Z[3:3 + nz]) / 2 - zc)[:, None] ** 2 + ((Y[2:2 + ny] + Y[3:3 + ny]) / 2 - yc) ** 2).sqrt()).double()
        m = torch.arange(50, device="cuda", dtype=torch.float32)

        def mid(X, h, n):
            d = f(h.reshape(-1) / 50)[:, None]
            x = X[2:2 + n, None]
            return (f(x + (m * d).double()) + f(x + ((m + 1) * d).double())).double() / 2

        sy, sz = mid(Y, hy, ny) - yc, mid(Z, hz, nz) - zc
        e = (dist <= r).double()
        for k, j in ((dist - r).abs() < diag).nonzero().tolist():
            e[k, j] = float(f((sz[k][None] ** 2 + sy[j][:, None] ** 2).sqrt()).double().le(r).sum()) / 2500
        e = e.float().double()
        self.extrude(e)


class _Solve(torch.autograd.Function):
    """The pressure solve; its derivative is that of the converged system (conjugate gradients)."""

    @staticmethod
    def forward(ctx, p, b, S):
        q = p.clone()
        S.sweeps.append(S.sor(q, b))
        ctx.S = S
        return q

    @staticmethod
    def backward(ctx, g):
        S = ctx.S
        vol = S.at(S.iD[0], 0, 0) * S.at(S.iD[1], 1, 0) * S.at(S.iD[2], 2, 0)
        pad = torch.zeros_like(g)
        inner = S.sh(pad)

        def A(x):
            inner.copy_(x)
            return vol * (x / S.rd - S.nbsum(pad))

        lam = S.sh(g).clone()
        z = torch.zeros_like(lam)
        r = lam.clone()
        d = r * S.rd / vol
        q, rz = d.clone(), (r * d).sum()
        stop = 1e-13 * float(lam.abs().max())
        for it in range(4000):
            Aq = A(q)
            a = rz / (q * Aq).sum()
            z += a * q
            r -= a * Aq
            if it % 20 == 0 and float(r.abs().max()) <= stop:
                break
            d = r * S.rd / vol
            rz, old = (r * d).sum(), rz
            q = d + rz / old * q
        y = vol * z / S.rd                                  # adjoint of the row p = rd sum c p - b'
        gp = g.clone()
        S.sh(gp).zero_()
        for a in range(3):                                  # the frozen ghosts next to the interior
            ax, n = 2 - a, S.n[a]
            inside = [slice(2, 2 + S.n[q]) for q in (2, 1, 0)]
            for i, row, coef in ((0, 0, S.cm[a]), (n + 1, n - 1, S.cp[a])):
                idx = list(inside)
                idx[ax] = i + 1
                gp[tuple(idx)] += (coef * S.rd * y).select(ax, row)
        return gp, -y, None


def exact(case, seed):
    S = _Scheme(case)
    if case["kind"] == "mask":
        aoa = case["aoa"] + float(np.random.default_rng(seed).uniform(-1.0, 1.0))
        S.polygon(*_foil(case["t"], case["npts"]), aoa, *CENTRE)
        out = torch.zeros(case["nz"] + 4, case["ny"] + 4, case["nx"] + 4, dtype=F64, device="cuda")
        S.sh(out).copy_(S.eta)
        return {"eta": out.permute(2, 1, 0).cpu().numpy()}
    fields = _state(case, seed)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed, S, fields)
    if case["body"] == "naca":
        S.polygon(*_foil(case["t"], 256), case["aoa"], *CENTRE)

    def solve(p, b):
        p = p.clone()
        return p, S.sor(p, b)

    vel, p = S.conditions(fields[:3], fields[3])
    sweeps, drag, lift = [], [], []
    for _ in range(case["steps"]):
        vel, p, it, d, l, pre, cen = S.step(vel, p, solve)
        sweeps.append(it)
        drag.append(float(d))
        lift.append(float(l))
    host = lambda f: f.permute(2, 1, 0).cpu().numpy()
    return {"pre": host(pre), "uc": host(cen[0]), "vc": host(cen[1]), "wc": host(cen[2]), "sweeps": None,
            "drag": np.array(drag), "lift": np.array(lift)}


def _exact_adjoint(case, seed, S, fields):
    S.cylinder(4.0, 6.0, 0.5)
    S.fb = [torch.tensor(np.ascontiguousarray(f.T), device="cuda").requires_grad_() for f in _force(case, seed)]
    S.sweeps = []
    vel, p = S.conditions(fields[:3], fields[3])
    back = [S.val[4][c].requires_grad_() for c in range(3)]
    J = 0.0
    for _ in range(case["steps"]):
        vel, p, _, d, l, _, _ = S.step(vel, p, lambda p, b: (_Solve.apply(p, b, S), 0))
        J = J + (d + 0.5 * l) / case["steps"]
    grads = torch.autograd.grad(J, S.fb + back)
    # U = 1, theta = 0: w = U cos(theta), v = U sin(theta)
    return {"J": float(J.detach()), "dU": float(grads[5]), "dtheta": float(grads[4]),
            "df": [f.permute(2, 1, 0).cpu().numpy() for f in grads[:3]], "sweeps": None}
