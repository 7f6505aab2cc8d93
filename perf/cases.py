"""What the engine is timed on: the runs its users make, through the public
binding (lbmx.Lattice, lbmx.Batch, lbmx.Tangent, lbmx_autograd) and, where a
program hands the engine its own pinned or device buffers, the C entry points.

listed() names the runs, draw() gives more of the same ranges, prepare() makes
what a program holds before the call, run() is one call with its readback,
work() the bytes and operations it cannot do without, and exact() the same
outputs in 64 bits from a plain torch restatement of the model at the end of
this file.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-lbm_gb300"))
import lbmx  # noqa: E402
import lbmx_autograd  # noqa: E402

OPS = {"bgk": lbmx.BGK, "mrt": lbmx.MRT, "cm": lbmx.CM, "cm_opt": lbmx.CM_OPT}
STORAGE = {"f32": lbmx.F32, "f16": lbmx.F16_OFFSET, "bf16": lbmx.BF16_OFFSET}
BYTES = {"f32": 4, "f16": 2, "bf16": 2}


def listed():
    return [
        # a small lattice watched after every step: one launch and one readback
        dict(name="cavity64_bgk_one_step", kind="cavity", nx=64, ny=64, op="bgk", storage="f32", steps=1),
        # the Taylor-Green validation flow: a lattice far smaller than L2, periodic both ways
        dict(name="taylor_green256_bgk", kind="vortex", nx=256, ny=256, op="bgk", storage="f32", steps=100),
        # the benchmark cavity with the sums of every step recorded, as a monitored run does
        dict(name="cavity1024_mrt_series", kind="series", nx=1024, ny=1024, op="mrt", storage="f32", steps=200),
        # the same cavity in 16-bit storage, plain steps
        dict(name="cavity1024_mrt_f16", kind="cavity", nx=1024, ny=1024, op="mrt", storage="f16", steps=200),
        # the HBM-bound cavity, FP32 and 16-bit storage
        dict(name="cavity8192_mrt_f32", kind="cavity", nx=8192, ny=8192, op="mrt", storage="f32", steps=20),
        dict(name="cavity8192_mrt_f16", kind="cavity", nx=8192, ny=8192, op="mrt", storage="f16", steps=20),
        # an open channel at a ragged size: Zou-He inlet and outlet, bounce-back walls
        dict(name="channel1021x517_cm", kind="channel", nx=1021, ny=517, op="cm", storage="f32", steps=60, markers=0),
        # flow past a cylinder with immersed-boundary markers, drag and lift of every step
        dict(name="cylinder2048x512_bgk", kind="channel", nx=2048, ny=512, op="bgk", storage="f32", steps=100,
             markers=256),
        # the body-force channel with the adaptive operator: grid averages before every collision
        dict(name="poiseuille4096_cm_opt", kind="poiseuille", nx=4096, ny=1024, op="cm_opt", storage="f32", steps=20),
        # an ensemble of cavities of mixed sizes in one batch
        dict(name="ensemble32_mrt_f16", kind="ensemble", count=32, lo=64, hi=768, op="mrt", storage="f16", steps=64),
        # a gradient of the outlet flux by the adjoint: forward and backward
        dict(name="adjoint2048x1024_cm", kind="adjoint", nx=2048, ny=1024, op="cm", storage="f32", steps=20, every=10),
        # the derivative of the cylinder's drag by the inlet velocity
        dict(name="tangent2048x512_bgk", kind="tangent", nx=2048, ny=512, op="bgk", storage="f32", steps=20,
             markers=256),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def lattice(largest_side, updates, most_steps):
        nx, ny = log(48, largest_side), log(48, largest_side)
        return dict(nx=nx, ny=ny, steps=max(1, min(log(1, most_steps), updates // (nx * ny))))

    kind = rng.choice(["cavity", "cavity", "vortex", "series", "channel", "channel", "cylinder", "poiseuille",
                       "ensemble", "adjoint", "tangent"])
    op = rng.choice(["bgk", "mrt", "cm"])
    storage = rng.choice(["f32", "f32", "f16", "bf16"])
    if kind in ("cavity", "vortex"):
        return dict(kind=kind, op=op, storage=storage, **lattice(8192, 1 << 30, 200))
    if kind == "series":
        return dict(kind=kind, op=op, storage=storage, **lattice(2048, 1 << 28, 200))
    if kind == "channel":
        return dict(kind=kind, op=op, storage=storage, markers=0, **lattice(4096, 1 << 28, 200))
    if kind == "cylinder":
        c = lattice(2048, 1 << 27, 100)
        c.update(nx=max(c["nx"], 160), ny=max(c["ny"], 96))
        return dict(kind="channel", op=op, storage=storage, markers=rng.randint(32, 256), **c)
    if kind == "poiseuille":
        return dict(kind=kind, op=rng.choice(["cm_opt", "cm", "mrt"]), storage="f32", **lattice(4096, 1 << 27, 40))
    if kind == "ensemble":
        lo = log(48, 256)
        return dict(kind=kind, count=rng.randint(4, 32), lo=lo, hi=lo * rng.randint(1, 3), op=op, storage=storage,
                    steps=log(4, 64))
    if kind == "adjoint":
        c = lattice(2048, 1 << 26, 40)
        return dict(kind=kind, op=op, storage="f32", every=rng.randint(1, c["steps"]), **c)
    c = lattice(2048, 1 << 25, 40)
    c.update(nx=max(c["nx"], 160), ny=max(c["ny"], 96))
    return dict(kind="tangent", op=rng.choice(["bgk", "mrt"]), storage="f32", markers=rng.randint(32, 256), **c)


# ---------------------------------------------------------------- inputs
def rates(op, omega):
    """The operators' relaxation rates, as the repository's test cases set them."""
    if op == "mrt":
        return [0.0, 1.0, 1.4, 0.0, 1.2, 0.0, 1.9, omega, omega]
    if op in ("cm", "cm_opt"):
        return [0.0, 0.0, 0.0, 1.0, omega, omega, 1.0, 1.0, 1.0]
    return [omega] * 9


def viscosity(kind):
    return {"channel": 0.032, "tangent": 0.032, "poiseuille": 0.02, "adjoint": 0.02, "vortex": 0.01}.get(kind, 0.05)


def setup(case, nx, ny):
    """The flow's parameters and flags: the same for every seed."""
    kind = case["kind"]
    omega = 1.0 / (3.0 * viscosity(kind) + 0.5)
    c = dict(nx=nx, ny=ny, op=case["op"], omega=omega, S=rates(case["op"], omega), periodic=(False, False), u_bc=0.0,
             wall_u=(0.0, 0.0), body=(0.0, 0.0))
    fl = np.zeros((ny, nx), np.uint8)
    if kind in ("cavity", "series", "ensemble"):
        fl[0, :] = fl[:, 0] = fl[:, -1] = lbmx.HALFWAY_BB
        fl[-1, 1:-1] = lbmx.MOVING_WALL_BB
        fl[-1, 0] = fl[-1, -1] = lbmx.HALFWAY_BB
        c["wall_u"] = (0.1, 0.0)
    elif kind == "vortex":
        c["periodic"] = (True, True)
    elif kind in ("channel", "tangent"):
        fl[:, 0] = lbmx.ZOU_HE_PARABOLIC_LEFT
        fl[:, -1] = lbmx.ZOU_HE_PRESSURE_RIGHT
        fl[0, :] = fl[-1, :] = lbmx.BOUNCE_BACK
        c["u_bc"] = 0.05
    else:
        fl[0, :] = fl[-1, :] = lbmx.BOUNCE_BACK if kind == "poiseuille" else lbmx.HALFWAY_BB
        c["periodic"] = (True, False)
        c["body"] = (float(np.float32(8.0 * viscosity(kind) * 0.05 / (ny * ny))), 0.0)
    c["flags"] = fl
    return c


def fields(case, nx, ny, seed):
    """A flow under way: a base flow of its kind and eddies of several sizes, rho near 1."""
    g = torch.Generator().manual_seed(seed)
    x = torch.arange(nx, device="cuda", dtype=torch.float32) * (2 * math.pi / nx)
    y = torch.arange(ny, device="cuda", dtype=torch.float32) * (2 * math.pi / ny)
    rho = torch.ones((ny, nx), device="cuda")
    u = torch.zeros((2, ny, nx), device="cuda")
    if case["kind"] in ("channel", "tangent", "poiseuille", "adjoint"):
        h = torch.arange(ny, device="cuda", dtype=torch.float32) / (ny - 1)
        u[0] += (0.2 * h * (1 - h))[:, None]
    for m in range(6):
        r = torch.rand(5, generator=g).tolist()
        kx, ky = 1 + int(r[0] * 2 ** m) % 24, 1 + int(r[1] * 2 ** m) % 24
        amp, px, py = 0.02 * (0.5 + r[2]) / (m + 1), 2 * math.pi * r[3], 2 * math.pi * r[4]
        u[0] += amp * torch.outer(torch.cos(ky * y + py), torch.sin(kx * x + px))
        u[1] -= amp * torch.outer(torch.sin(ky * y + py), torch.cos(kx * x + px))
        rho += 0.02 * amp * torch.outer(torch.sin(ky * y + px), torch.sin(kx * x + py))
    return rho, u


def marker_ring(case, seed):
    """A cylinder of markers a quarter down the channel, its centre the seed's;
    the tangent's bodies all sit at one place, as its benchmark has them."""
    r = min(32.0, case["ny"] / 8.0)
    j = np.random.RandomState(seed % (1 << 31)).uniform(-0.5, 0.5, 2) if case["kind"] == "channel" else (0.0, 0.0)
    a = 2 * np.pi * np.arange(case["markers"]) / case["markers"]
    cx, cy = 0.25 * min(case["nx"], 1024) + j[0], 0.5 * case["ny"] + j[1]
    return np.stack([cx + r * np.cos(a), cy + r * np.sin(a)], axis=1).astype(np.float32)


def porous_field(case, seed):
    """Brinkman solid fractions in [0, 1]: smooth patches of solid."""
    _, u = fields(dict(case, kind="cavity"), case["nx"], case["ny"], seed + 7)
    return (0.5 + 12.0 * u[0]).clamp_(0.0, 1.0)


def flux_weights(case):
    w = torch.zeros((3, case["ny"], case["nx"]), device="cuda")
    w[1, :, -1] = 1.0 / case["steps"]
    return w


def sides_of(case, seed):
    r = np.random.RandomState(1234 + case["count"])
    return [int(s) for s in np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"] + 1), case["count"]))]


def make_lattice(case, nx, ny, seed):
    c = setup(case, nx, ny)
    L = lbmx.Lattice(nx, ny, op=OPS[c["op"]], omega=c["omega"], S=c["S"], periodic=c["periodic"],
                     storage=STORAGE[case["storage"]], u_bc=c["u_bc"], wall_u=c["wall_u"], body_force=c["body"])
    L.set_flags(c["flags"])
    rho, u = fields(case, nx, ny, seed)
    torch.cuda.synchronize()  # the lattice reads them on a stream of its own
    L.init(rho, u)
    return L


def prepare(case, seed):
    kind, nx, ny = case["kind"], case.get("nx"), case.get("ny")
    s = dict(case=case, kind=kind, steps=case["steps"])
    if kind == "ensemble":
        sides = sides_of(case, seed)
        s["lattices"] = [make_lattice(case, n, n, seed + 100 * k) for k, n in enumerate(sides)]
        s["batch"] = lbmx.Batch(s["lattices"])
        ends = np.cumsum([0] + [n * n for n in sides])
        s["rho"], s["u"] = torch.empty(int(ends[-1]), device="cuda"), torch.empty(2 * int(ends[-1]), device="cuda")
        s["views"] = [(s["rho"][a:b], s["u"][2 * a:2 * b]) for a, b in zip(ends[:-1], ends[1:])]
        return s
    if kind == "adjoint":
        c = setup(case, nx, ny)
        a = lbmx.Adjoint(nx, ny, op=OPS[c["op"]], omega=c["omega"], S=c["S"], periodic=c["periodic"], flags=c["flags"],
                         checkpoint_every=case["every"], body_force=c["body"])
        rho, u = fields(case, nx, ny, seed)
        w = flux_weights(case)
        s["gamma"] = porous_field(case, seed).requires_grad_()
        s["omega"] = torch.tensor(c["omega"], dtype=torch.float32, requires_grad=True)
        s["force"] = torch.tensor(c["body"], dtype=torch.float32, requires_grad=True)
        torch.cuda.synchronize()
        a.set_state(rho, u)
        a.set_objective(w, 1)
        s["adjoint"] = a
        return s
    if kind == "tangent":
        c = setup(case, nx, ny)
        t = lbmx.Tangent(nx, ny, lbmx.TANGENT_U_BC, op=OPS[c["op"]], omega=c["omega"], S=c["S"], flags=c["flags"],
                         u_bc=c["u_bc"])
        rho, u = fields(case, nx, ny, seed)
        torch.cuda.synchronize()
        t.set_state(rho, u)
        t.set_markers(marker_ring(case, seed))
        s["tangent"] = t
        return s
    s["lattice"] = make_lattice(case, nx, ny, seed)
    if case.get("markers"):
        s["lattice"].set_markers(marker_ring(case, seed))
        s["series"] = torch.zeros((case["steps"], 2), dtype=torch.float64).pin_memory()
    if kind == "series":
        s["series"] = torch.zeros((case["steps"], 3), dtype=torch.float64).pin_memory()
    s["rho"], s["u"] = torch.empty((ny, nx), device="cuda"), torch.empty((2, ny, nx), device="cuda")
    return s


def run(s):
    kind, steps = s["kind"], s["steps"]
    if kind == "ensemble":
        s["batch"].step(steps)
        for L, (rho, u) in zip(s["lattices"], s["views"]):
            L.moments(rho, u)
        return {"rho": s["rho"], "u": s["u"]}
    if kind == "adjoint":
        for p in (s["gamma"], s["omega"], s["force"]):
            p.grad = None
        J = lbmx_autograd.objective(s["gamma"], s["omega"], s["force"], s["adjoint"], steps)
        J.backward()
        return {"J": J.detach(), "gamma": s["gamma"].grad, "omega": s["omega"].grad, "force": s["force"].grad}
    if kind == "tangent":
        return {"series": s["tangent"].run(steps)}
    L = s["lattice"]
    if kind == "series":
        # the sums of every step, written by the steps into pinned memory
        L._check(L.lib.lbmx_step_sums(L.h, steps, lbmx.STEP_STORE_MOMENTS, s["series"].data_ptr()))
    elif "series" in s:
        L.step_forces(steps, flags=lbmx.STEP_STORE_MOMENTS, out=s["series"])
    else:
        L.step(steps)
    L.moments(s["rho"], s["u"])
    out = {"rho": s["rho"], "u": s["u"]}
    if "series" in s:
        out["series"] = s["series"]
    return out


# operations of one node's step: streaming costs none, the moments about 30,
# the collision as below
FLOPS = {"bgk": 130, "mrt": 140, "cm": 260, "cm_opt": 300}


def work(case):
    """The state and the call's inputs read once, the state and the outputs written once."""
    op, steps = case["op"], case["steps"]
    if case["kind"] == "ensemble":
        n = sum(k * k for k in sides_of(case, 0))
        return {"bytes": n * (18.0 * BYTES[case["storage"]] + 12), "flops": float(n) * steps * FLOPS[op]}
    n = float(case["nx"] * case["ny"])
    if case["kind"] == "adjoint":
        # rho, u, gamma and the weights in, the gradient out; the step, its recomputation and its reverse
        return {"bytes": n * 4 * (9 + 1 + 3 + 1), "flops": n * steps * 4 * FLOPS[op]}
    if case["kind"] == "tangent":
        return {"bytes": n * 4 * 36, "flops": n * steps * 3 * FLOPS[op]}
    return {"bytes": n * (18.0 * BYTES[case["storage"]] + 12), "flops": n * steps * FLOPS[op]}


# ---------------------------------------------------------------- 64 bits
# The model in plain torch: pull streaming of the post-collision populations,
# boundaries, moments with the Guo and Brinkman corrections, collision.
CX = (0, 1, 0, -1, 0, 1, -1, -1, 1)
CY = (0, 0, 1, 0, -1, 1, 1, -1, -1)
OPP = (0, 3, 4, 1, 2, 7, 8, 5, 6)
W = (4 / 9, 1 / 9, 1 / 9, 1 / 9, 1 / 9, 1 / 36, 1 / 36, 1 / 36, 1 / 36)
M_ROWS = ((1, 1, 1, 1, 1, 1, 1, 1, 1), (-4, -1, -1, -1, -1, 2, 2, 2, 2), (4, -2, -2, -2, -2, 1, 1, 1, 1),
          (0, 1, 0, -1, 0, 1, -1, -1, 1), (0, -2, 0, 2, 0, 1, -1, -1, 1), (0, 0, 1, 0, -1, 1, 1, -1, -1),
          (0, 0, -2, 0, 2, 1, 1, -1, -1), (0, 1, -1, 1, -1, 0, 0, 0, 0), (0, 0, 0, 0, 0, 1, -1, 1, -1))


def combine(row, v):
    out = None
    for k, x in zip(row, v):
        if k:
            out = k * x if out is None else out + k * x
    return out


def equilibrium(rho, ux, uy):
    uu = ux * ux + uy * uy
    out = []
    for q in range(9):
        cu = CX[q] * ux + CY[q] * uy
        out.append(W[q] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * uu))
    return out


class Flow64:
    def __init__(self, c, rho, u, gamma=None, omega=None, force=None, u_bc=None):
        dev = rho.device
        self.c, self.op, self.gamma = c, c["op"], gamma
        om32 = float(np.float32(c["omega"]))
        self.omega = om32 if omega is None else omega
        self.S = [self.omega if s == c["omega"] else float(np.float32(s)) for s in c["S"]]
        self.F = [float(np.float32(v)) for v in c["body"]] if force is None else force
        self.u_bc = float(np.float32(c["u_bc"])) if u_bc is None else u_bc
        wall = [float(np.float32(v)) for v in c["wall_u"]]
        ny, nx = rho.shape
        fl = torch.from_numpy(c["flags"]).to(dev)
        self.half = (fl == lbmx.HALFWAY_BB) | (fl == lbmx.MOVING_WALL_BB)
        moving = (fl == lbmx.MOVING_WALL_BB).double()
        x = torch.arange(nx, device=dev)[None, :].expand(ny, nx)
        y = torch.arange(ny, device=dev)[:, None].expand(ny, nx)
        px, py = c["periodic"]
        self.links = [None]
        self.bounce = []
        for q in range(1, 9):
            sx, sy = x - CX[q], y - CY[q]
            out = torch.zeros((ny, nx), dtype=torch.bool, device=dev)
            if not px:
                out |= (sx < 0) | (sx >= nx)
            if not py:
                out |= (sy < 0) | (sy >= ny)
            stale = out & ~self.half
            o = OPP[q]
            # a half-way node gets back what left it, less the wall's term
            term = 6.0 * W[o] * (CX[o] * wall[0] + CY[o] * wall[1])
            self.links.append((out & self.half if bool((out & self.half).any()) else None,
                               term * moving if term and bool(moving.any()) else None,
                               stale if bool(stale.any()) else None))
            ex, ey = x + CX[q], y + CY[q]
            b = (fl == lbmx.BOUNCE_BACK) & ((ex < 0) | (ex >= nx) | (ey < 0) | (ey >= ny))
            self.bounce.append(b if bool(b.any()) else None)
        self.inlet = fl == lbmx.ZOU_HE_PARABOLIC_LEFT
        self.outlet = fl == lbmx.ZOU_HE_PRESSURE_RIGHT
        self.has_in, self.has_out = bool(self.inlet.any()), bool(self.outlet.any())
        self.profile = 4.0 * y.double() * ((ny - 1) - y.double()) / float((ny - 1) ** 2)
        self.pc = equilibrium(rho, u[0], u[1])
        self.older = self.pc if any(l and l[2] is not None for l in self.links) else None
        self.markers = None

    def set_markers(self, xy, rounds=3):
        ny, nx = self.half.shape
        p = torch.from_numpy(xy.astype(np.float64)).to(self.half.device)
        base = torch.floor(p).long() - 1
        k = torch.arange(4, device=p.device)
        gx, gy = base[:, 0:1] + k, base[:, 1:2] + k

        def delta(r):
            a = r.abs()
            near = 0.125 * (3 - 2 * a + torch.sqrt((1 + 4 * a - 4 * a * a).clamp(min=0)))
            far = 0.125 * (5 - 2 * a - torch.sqrt((-7 + 12 * a - 4 * a * a).clamp(min=0)))
            return torch.where(a < 1, near, torch.where(a < 2, far, torch.zeros_like(a)))

        w = delta(p[:, 0:1] - gx)[:, :, None] * delta(p[:, 1:2] - gy)[:, None, :]
        self.markers = ((gy[:, None, :] * nx + gx[:, :, None]).reshape(len(xy), 16), w.reshape(len(xy), 16), rounds)

    def stream(self):
        ps = [self.pc[0]]
        for q in range(1, 9):
            v = torch.roll(self.pc[q], (CY[q], CX[q]), (0, 1))
            back, term, stale = self.links[q]
            if back is not None:
                r = self.pc[OPP[q]]
                v = torch.where(back, r if term is None else r - term, v)
            if stale is not None:
                v = torch.where(stale, self.older[q], v)
            ps.append(v)
        return ps

    def boundaries(self, f):
        for i in range(1, 9):
            if self.bounce[i - 1] is not None:
                f[OPP[i]] = torch.where(self.bounce[i - 1], f[i], f[OPP[i]])
        if self.has_in:
            ux = self.u_bc * self.profile
            rho = (f[0] + f[2] + f[4] + 2 * (f[3] + f[6] + f[7])) / (1 - ux)
            d = 0.5 * (f[2] - f[4])
            f[1] = torch.where(self.inlet, f[3] + (2 / 3) * rho * ux, f[1])
            f[5] = torch.where(self.inlet, f[7] - d + rho * ux / 6, f[5])
            f[8] = torch.where(self.inlet, f[6] + d + rho * ux / 6, f[8])
        if self.has_out:
            ux = -1 + (f[0] + f[2] + f[4] + 2 * (f[1] + f[5] + f[8]))
            d = 0.5 * (f[2] - f[4])
            f[3] = torch.where(self.outlet, f[1] - (2 / 3) * ux, f[3])
            f[7] = torch.where(self.outlet, f[5] + d - ux / 6, f[7])
            f[6] = torch.where(self.outlet, f[8] - d - ux / 6, f[6])
        return f

    def marker_forces(self, rho, ux, uy):
        idx, w, rounds = self.markers
        r = (w * rho.reshape(-1)[idx]).sum(1)
        fx, fy = torch.zeros_like(rho).reshape(-1), torch.zeros_like(rho).reshape(-1)
        ux, uy, half = ux.reshape(-1), uy.reshape(-1), 0.5 / rho.reshape(-1)
        drag = [0.0, 0.0]
        for _ in range(rounds):
            mx, my = -2 * r * (w * ux[idx]).sum(1), -2 * r * (w * uy[idx]).sum(1)
            gx = torch.zeros_like(ux).index_add(0, idx.reshape(-1), (w * mx[:, None]).reshape(-1))
            gy = torch.zeros_like(uy).index_add(0, idx.reshape(-1), (w * my[:, None]).reshape(-1))
            ux, uy, fx, fy = ux + gx * half, uy + gy * half, fx + gx, fy + gy
            drag = [drag[0] - mx.sum(), drag[1] - my.sum()]
        return fx.reshape(rho.shape), fy.reshape(rho.shape), drag

    def step(self):
        f = self.boundaries(self.stream())
        rho = sum(f[1:], f[0])
        jx = f[1] - f[3] + f[5] - f[6] - f[7] + f[8]
        jy = f[2] - f[4] + f[5] + f[6] - f[7] - f[8]
        Fx, Fy = self.F
        if self.markers is not None:
            gx, gy, self.drag = self.marker_forces(rho, jx / rho, jy / rho)
            Fx, Fy = Fx + gx, Fy + gy
        ux, uy = (jx + 0.5 * Fx) / rho, (jy + 0.5 * Fy) / rho
        if self.gamma is not None:
            ux, uy = ux / (1 + 0.5 * self.gamma), uy / (1 + 0.5 * self.gamma)
            Fx, Fy = Fx - self.gamma * rho * ux, Fy - self.gamma * rho * uy
        if self.op in ("cm", "cm_opt"):
            f = self.collide_cm(f, rho, ux, uy, Fx, Fy)
        elif self.op == "mrt":
            f = self.collide_mrt(f, rho, ux, uy, Fx, Fy)
        else:
            om = self.omega
            fe = equilibrium(rho, ux, uy)
            for q in range(9):
                cu = CX[q] * ux + CY[q] * uy
                g = (3 * (CX[q] - ux) + 9 * cu * CX[q]) * Fx + (3 * (CY[q] - uy) + 9 * cu * CY[q]) * Fy
                f[q] = f[q] + om * (fe[q] - f[q]) + W[q] * (1 - 0.5 * om) * g
        if self.older is not None:
            self.older = self.pc
        self.pc = f
        self.rho, self.u = rho, (ux, uy)

    def collide_mrt(self, f, rho, ux, uy, Fx, Fy):
        uu, fu = ux * ux + uy * uy, Fx * ux + Fy * uy
        eq = (rho, rho * (3 * uu - 2), rho * (1 - 3 * uu), rho * ux, -rho * ux, rho * uy, -rho * uy,
              rho * (ux * ux - uy * uy), rho * ux * uy)
        zero = torch.zeros_like(rho)
        G = (zero, 6 * fu, -6 * fu, Fx, -Fx, Fy, -Fy, 2 * (Fx * ux - Fy * uy), Fx * uy + Fy * ux)
        a = []
        for k in range(9):
            m = combine(M_ROWS[k], f)
            if k:
                m = m - self.S[k] * (m - eq[k]) + (1 - 0.5 * self.S[k]) * G[k]
            a.append(m / sum(v * v for v in M_ROWS[k]))
        return [combine([M_ROWS[k][q] for k in range(9)], a) for q in range(9)]

    def collide_cm(self, f, rho, ux, uy, Fx, Fy):
        k = {}
        for i in range(3):
            for j in range(3):
                k[i, j] = sum(f[q] * (CX[q] - ux) ** i * (CY[q] - uy) ** j for q in range(9))
        S = list(self.S)
        if self.op == "cm_opt":
            pxx, pyy = f[1] + f[3] + sum(f[5:]), f[2] + f[4] + sum(f[5:])
            pxy = f[5] - f[6] + f[7] - f[8]
            pi = torch.sqrt(pxx * pxx + 2 * pxy * pxy + pyy * pyy)
            j = rho * torch.sqrt(ux * ux + uy * uy)
            t = 0.0003 * rho / rho.mean() - 0.00775 * j / j.mean() + 0.00016 * pi / pi.mean() + 0.0087
            t = torch.where(t > 0, t, torch.full_like(t, 0.005)).clamp(max=1.5)
            S[6] = S[7] = S[8] = 1 / (3 * t + 0.5)
        z = torch.zeros_like(rho)
        c = {(0, 0): rho + z}
        c[1, 0] = (1 - S[1]) * k[1, 0] + (1 - 0.5 * S[1]) * Fx
        c[0, 1] = (1 - S[2]) * k[0, 1] + (1 - 0.5 * S[2]) * Fy
        ks, kd = k[2, 0] + k[0, 2], k[2, 0] - k[0, 2]
        t3, t4 = ks - S[3] * (ks - 2 * rho / 3), (1 - S[4]) * kd
        c[2, 0], c[0, 2], c[1, 1] = 0.5 * (t3 + t4), 0.5 * (t3 - t4), (1 - S[5]) * k[1, 1]
        c[2, 1] = (1 - S[6]) * k[2, 1] + (1 - 0.5 * S[6]) * Fy / 3
        c[1, 2] = (1 - S[7]) * k[1, 2] + (1 - 0.5 * S[7]) * Fx / 3
        c[2, 2] = k[2, 2] - S[8] * (k[2, 2] - rho / 9)
        px, py = (z + 1, ux, ux * ux), (z + 1, uy, uy * uy)
        r = {}
        for i in range(3):
            for j in range(3):
                r[i, j] = sum(math.comb(i, a) * math.comb(j, b) * px[i - a] * py[j - b] * c[a, b]
                              for a in range(i + 1) for b in range(j + 1))
        # a direction's share of the raw moments: the product of one-dimensional ones
        share = {0: ((0, 1), (2, -1)), 1: ((1, 0.5), (2, 0.5)), -1: ((1, -0.5), (2, 0.5))}
        return [sum(a * b * r[i, j] for i, a in share[CX[q]] for j, b in share[CY[q]]) for q in range(9)]


def flow64(case, nx, ny, seed, **kw):
    rho, u = fields(case, nx, ny, seed)
    return Flow64(setup(case, nx, ny), rho.double(), u.double(), **kw)


def exact(case, seed):
    kind, steps, nx, ny = case["kind"], case["steps"], case.get("nx"), case.get("ny")
    if kind == "adjoint":
        if nx * ny * steps > 48 << 20:
            return None
        c = setup(case, nx, ny)
        gamma = porous_field(case, seed).double().requires_grad_()
        omega = torch.tensor(float(np.float32(c["omega"])), dtype=torch.float64, device="cuda", requires_grad=True)
        force = torch.tensor([float(np.float32(v)) for v in c["body"]], dtype=torch.float64, device="cuda",
                             requires_grad=True)
        f = flow64(case, nx, ny, seed, gamma=gamma, omega=omega, force=force)
        w = flux_weights(case).double()
        J = torch.zeros((), dtype=torch.float64, device="cuda")
        for _ in range(steps):
            f.step()
            J = J + (w[1] * f.rho * f.u[0]).sum()
        J.backward()
        return {"J": J.detach(), "gamma": gamma.grad, "omega": omega.grad, "force": force.grad}
    with torch.no_grad():
        if kind == "tangent":
            h, out = 1e-5, []
            u0 = float(np.float32(0.05))
            for u_bc in (u0, u0 - h, u0 + h):
                f = flow64(case, nx, ny, seed, u_bc=u_bc)
                f.set_markers(marker_ring(case, seed))
                d = []
                for _ in range(steps):
                    f.step()
                    d.append(torch.stack(f.drag))
                out.append(torch.stack(d))
            return {"series": torch.cat([out[0], (out[2] - out[1]) / (2 * h)], 1)}
        if kind == "ensemble":
            rho, u = [], []
            for k, n in enumerate(sides_of(case, seed)):
                f = flow64(case, n, n, seed + 100 * k)
                for _ in range(steps):
                    f.step()
                rho.append(f.rho.reshape(-1))
                u += [f.u[0].reshape(-1), f.u[1].reshape(-1)]
            return {"rho": torch.cat(rho), "u": torch.cat(u)}
        f = flow64(case, nx, ny, seed)
        if case.get("markers"):
            f.set_markers(marker_ring(case, seed))
        series = []
        for _ in range(steps):
            f.step()
            if case.get("markers"):
                series.append(torch.stack(f.drag))
            elif kind == "series":
                series.append(torch.stack([f.rho.sum(), (f.rho * f.u[0]).sum(), (f.rho * f.u[1]).sum()]))
        out = {"rho": f.rho, "u": torch.stack(f.u)}
        if series:
            out["series"] = torch.stack(series)
        return out
