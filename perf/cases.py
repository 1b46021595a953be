"""Timed cases: the calls a user of the framework makes, at the sizes and with the options they are made in earnest.

Five kinds, all through the Python binding of the C ABI (``fluidprjct_b200.capi``):

``frame``   a caller's particles in, some steps, the particles back out: ``set_particles``, ``step(n)``, ``particles``
            (a frame of a host program that owns the particle state);
``scene``   an advancing scene whose state stays on the device: ``step(n)``, then the face velocities, the pressure
            and the labels copied into device buffers (what the training-data generator and a renderer read);
``pairs``   a scene stepped by the plain solver for training data: labels, right-hand side and pressure per step;
``unet``    the learned preconditioner's network: inference, loss and gradient, or a training step;
``csr``     the stand-alone solve of an upper-triangle CSR system in caller-owned device memory.

Scenes, time steps, particle counts, tolerances and weights are those of the benchmark, the tests and
``fluidprjct_b200.learned``.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.nn.functional as F

from fluidprjct_b200 import capi, scenes
from fluidprjct_b200.learned import DEFAULT_WEIGHTS

SOLID, FLUID, AIR = 0, 1, 2
CSR_TOL = 1e-12


def listed():
    return [
        # The 2D dam break of the configuration table: the smallest call, bound by latency and launches.
        dict(name="frame_2d_64", kind="frame", scene="dam2d", W=64, H=64, D=1, ppc=4, scheme="default",
             solver="pcg_mg", advection="rk2", dt=0.005, steps=10, tol=1e-6),
        # The reference's own 2D step on a wide, odd tank.
        dict(name="frame_ref2d_301x187", kind="frame", scene="dam2d", W=301, H=187, D=1, ppc=4, scheme="ref2d",
             solver="pcg_mg", advection="rk3ref", dt=0.002, steps=5, tol=1e-6),
        # The reference's shipped scale and defaults: a 50^3 grid, dx = 0.02, 4 particles per cell, RK3, plain PCG.
        dict(name="frame_3d_50_defaults", kind="frame", scene="box", W=50, H=50, D=50, ppc=4, scheme="default",
             solver="pcg", advection="rk3ref", dt=0.005, steps=2, tol=1e-6),
        # An odd, ragged box with the mixed-precision solver.
        dict(name="frame_3d_61x47x83_mixed", kind="frame", scene="box", W=61, H=47, D=83, ppc=8, scheme="default",
             solver="pcg_mixed", advection="rk2", dt=0.004, steps=2, tol=1e-6),
        # The headline dam break end to end: 3.83 M particles in from pinned memory, a step, and out again.
        dict(name="frame_dam128_e2e", kind="frame", scene="dam3d", W=128, H=128, D=128, ppc=8, scheme="default",
             solver="pcg_mg", advection="rk2", dt=0.002, steps=1, tol=1e-6),
        # The headline dam break advancing on the device.
        dict(name="scene_dam128", kind="scene", scene="dam3d", W=128, H=128, D=128, ppc=8, solver="pcg_mg",
             dt=0.002, steps=2, tol=1e-6),
        # ... with the learned guess and the mixed-precision refinement, the other half of the headline.
        dict(name="scene_dam128_learned_mixed", kind="scene", scene="dam3d", W=128, H=128, D=128, ppc=8,
             solver="pcg_learned_mixed", dt=0.002, steps=1, tol=1e-6),
        # The rigid-body drop: a 160^3 pool, two-way coupled sphere, SDF collision (dx not a power of two).
        dict(name="scene_pool160_sphere", kind="scene", scene="pool", W=160, H=160, D=160, ppc=8, solver="pcg_mg",
             dt=0.002, steps=2, tol=1e-6),
        # The large seabed scene with its moving paddle: the largest state.
        dict(name="scene_seabed_256x128x256", kind="scene", scene="seabed", W=256, H=128, D=256, ppc=8,
             solver="pcg_mg", dt=0.001, steps=1, tol=1e-6),
        # Training data: random boxes stepped with the plain FP64 solver to 1e-7.
        dict(name="pairs_boxes128_plain", kind="pairs", scene="boxes", W=128, H=128, D=128, ppc=4, solver="pcg",
             dt=0.002, steps=1, tol=1e-7),
        # One Adam step of the network at its training size.
        dict(name="unet_train_128", kind="unet", op="train", W=128, H=128, D=128),
        # The CSR solve without allocations, a Poisson system of 40^3 unknowns.
        dict(name="csr_poisson_40x40x40", kind="csr", W=40, H=40, D=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame2d", "frame3d", "frame3d", "scene", "scene", "pairs", "unet", "unet", "csr"])
    if kind == "frame2d":
        ref = rng.random() < 0.5
        return dict(kind="frame", scene="dam2d", W=_log(rng, 40, 400), H=_log(rng, 40, 300), D=1, ppc=4,
                    scheme="ref2d" if ref else "default", solver="pcg_mg" if ref else rng.choice(["pcg_mg", "pcg_mixed"]),
                    advection=rng.choice(["rk2", "rk3ref"]), dt=0.002, steps=5, tol=1e-6)
    if kind == "frame3d":
        return dict(kind="frame", scene="box", W=_log(rng, 20, 96), H=_log(rng, 20, 96), D=_log(rng, 20, 96),
                    ppc=rng.choice([4, 8]), scheme="default", solver=rng.choice(["pcg", "pcg_mixed", "pcg_mg"]),
                    advection=rng.choice(["rk2", "rk3ref"]), dt=0.004, steps=2, tol=1e-6)
    if kind == "scene":
        scene = rng.choice(["dam3d", "dam3d", "pool", "seabed"])
        solver = rng.choice(["pcg_mg", "pcg_mg", "pcg_learned", "pcg_learned_mixed"]) if scene == "dam3d" else "pcg_mg"
        n = _log(rng, 64, 160 if scene == "pool" else 144)
        W, H, D = (n, n, n) if scene == "pool" else (n, _log(rng, 48, 128), _log(rng, 64, 144))
        return dict(kind="scene", scene=scene, W=W, H=H, D=D, ppc=rng.choice([4, 8]), solver=solver, dt=0.002, steps=1,
                    tol=1e-6)
    if kind == "pairs":
        n = _log(rng, 48, 128)
        return dict(kind="pairs", scene="boxes", W=n, H=n, D=n, ppc=4, solver="pcg", dt=0.256 / n, steps=1, tol=1e-7)
    if kind == "unet":
        return dict(kind="unet", op=rng.choice(["forward", "loss_grad", "train"]), W=_log(rng, 24, 128),
                    H=_log(rng, 24, 128), D=_log(rng, 24, 128))
    return dict(kind="csr", W=_log(rng, 8, 60), H=_log(rng, 8, 60), D=_log(rng, 8, 60))


# ---------------------------------------------------------------- inputs

def _dx(c):
    """Unit height in 2D and in the boxes' longest axis; the large scenes keep 1/128 off a cube, as the seabed's."""
    if c["scene"] in ("dam2d", "box", "boxes", "pool"):
        return 1.0 / max(c["W"], c["H"], c["D"])
    return 1.0 / 128


def _labels(c, seed):
    W, H, D, dx = c["W"], c["H"], c["D"], _dx(c)
    if c["scene"] == "dam2d":
        return scenes.box_3d(W, H, 3, dx, 0.4 * W * dx, 0.5 * H * dx, 1e9)[1].copy()
    if c["scene"] == "box":
        return scenes.box_3d(W, H, D, dx, 0.55 * W * dx, 0.6 * H * dx, 0.7 * D * dx)
    if c["scene"] == "dam3d":
        return scenes.box_3d(W, H, D, dx, 0.4 * W * dx, 0.6 * H * dx, 1e9)
    if c["scene"] == "pool":
        return scenes.pool_3d(W, 0.35)
    return scenes.random_boxes(seed, n=W)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 11)
    return g


def _particles(lab, dx, ppc, seed):
    """ppc particles per FLUID cell at a random octant (quadrant) centre plus a jitter of U(-0.24, 0.24) dx, already
    moving: a smooth velocity field of up to 0.3 m/s, a state a few steps into a run."""
    two_d = lab.ndim == 2
    t = torch.from_numpy(np.ascontiguousarray(lab)).cuda()
    cells = (t == FLUID).nonzero()
    ax = [cells[:, 1], cells[:, 0]] if two_d else [cells[:, 2], cells[:, 1], cells[:, 0]]
    g = _gen(seed)
    pos = torch.zeros((len(cells) * ppc, 3), dtype=torch.float32, device="cuda")
    for a, i in enumerate(ax):
        i = i.repeat_interleave(ppc).double()
        side = torch.randint(0, 2, i.shape, device="cuda", generator=g).double() * 0.5 - 0.25
        jit = (torch.rand(i.shape, device="cuda", generator=g, dtype=torch.float64) - 0.5) * 0.48
        pos[:, a] = ((i + 0.5 + side + jit) * dx).float()
    vel = torch.zeros_like(pos)
    ph = torch.rand(3, device="cuda", generator=g) * 6.28
    for a in range(len(ax)):
        b = (a + 1) % len(ax)
        vel[:, a] = 0.3 * torch.sin(5.0 * pos[:, b] + ph[a]) * torch.cos(3.0 * pos[:, a] + ph[b])
    return pos, vel


def _solver(c, seed):
    W, H, D, dx = c["W"], c["H"], c["D"], _dx(c)
    two_d = D == 1
    kw = dict(dim=2 if two_d else 3, dx=dx, dt=c["dt"], pic_weight=0.05, solver=c["solver"], tol=c["tol"],
              advection=c.get("advection", "rk2"), output_format=capi.OUT_NONE)
    if two_d:
        kw["scheme"] = c["scheme"]
    if c["scene"] == "pool":
        kw.update(body_radius=0.12, body_density=0.5, body_pos=(0.5, 0.7, 0.5), active_body=1, collision="sdf")
    s = capi.Solver(**kw)
    if c["scene"] == "seabed":
        s.scene_seabed(W, H, D, level=0.45 * H * dx, bed_base=0.15 * H * dx, bed_amp=0.05, seed=4, water_xmin=0.1)
        s.set_paddle(0.1, 0.05, 1.0)
    else:
        s.set_labels(_labels(c, seed))
        if c["scene"] == "pool":
            s.load_sdf(None)
    if "learned" in c["solver"]:
        s.load_learned(DEFAULT_WEIGHTS)
    return s


def _pinned(t):
    return t.cpu().pin_memory().numpy()


def _unet_pair(c, seed):
    """Labels (walls, a water box, air), a smooth pressure on its FLUID cells and the right-hand side it solves."""
    W, H, D = c["W"], c["H"], c["D"]
    lab = torch.from_numpy(scenes.box_3d(W, H, D, 1.0 / max(W, H, D), 0.6 * W / max(W, H, D), 0.7 * H / max(W, H, D),
                                         2.0)).cuda()
    g = _gen(seed)
    low = torch.randn((1, 1, 6, 6, 6), device="cuda", generator=g, dtype=torch.float64)
    p = F.interpolate(low, size=(D, H, W), mode="trilinear", align_corners=True)[0, 0]
    p = (p * (lab == FLUID)).float()
    fl, diag = _operator(lab)
    return lab, _apply(p.double(), fl, diag).float(), p


def _csr_system(c, seed):
    """Upper triangle of the 7-point Dirichlet operator on a W x H x D box, and a right-hand side."""
    W, H, D = c["W"], c["H"], c["D"]
    n = W * H * D
    idx = np.arange(n).reshape(D, H, W)
    rows, cols = [idx.ravel()], [idx.ravel()]
    vals = [np.full(n, 6.0)]
    for lo, hi in ((idx[:, :, :-1], idx[:, :, 1:]), (idx[:, :-1], idx[:, 1:]), (idx[:-1], idx[1:])):
        rows.append(lo.ravel())
        cols.append(hi.ravel())
        vals.append(np.full(lo.size, -1.0))
    rows, cols, vals = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    order = np.lexsort((cols, rows))
    off = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=off[1:])
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=_gen(seed))
    return (torch.from_numpy(off).cuda(), torch.from_numpy(cols[order].astype(np.int32)).cuda(),
            torch.from_numpy(vals[order]).cuda(), b)


def prepare(case, seed):
    c = case
    if c["kind"] == "csr":
        off, cols, vals, b = _csr_system(c, seed)
        return dict(case=c, off=off, cols=cols, vals=vals, b=b, x=torch.zeros_like(b),
                    stream=torch.cuda.current_stream().cuda_stream)
    if c["kind"] == "unet":
        lab, rhs, p = _unet_pair(c, seed)
        net = capi.UNet(c["W"], c["H"], c["D"], train=c["op"] != "forward", seed=seed)
        if c["op"] == "forward":
            net.load(DEFAULT_WEIGHTS)
        return dict(case=c, net=net, lab=lab, rhs=rhs, p=p, x=torch.zeros_like(rhs))
    s = _solver(c, seed)
    st = dict(case=c, s=s)
    lab = s.labels()
    if c["D"] == 1:
        lab = lab[0]
    pos, vel = _particles(lab, _dx(c), c["ppc"], seed)
    st["pos"], st["vel"] = _pinned(pos), _pinned(vel)
    if c["kind"] == "frame":
        st["out_pos"], st["out_vel"] = _pinned(torch.zeros_like(pos)), _pinned(torch.zeros_like(vel))
        return st
    s.set_particles(st.pop("pos"), st.pop("vel"))
    cells = c["W"] * c["H"] * c["D"]
    st["lab"] = torch.zeros(cells, dtype=torch.uint8, device="cuda")
    which = dict(rhs=capi.GRID_RHS, p=capi.GRID_P) if c["kind"] == "pairs" else \
        dict(u=capi.GRID_U, v=capi.GRID_V, w=capi.GRID_W, p=capi.GRID_P)
    st["which"] = which
    st["grids"] = {k: torch.zeros(math.prod(s.grid_shape(w)), device="cuda") for k, w in which.items()}
    return st


def run(state):
    c = state["case"]
    if c["kind"] == "csr":
        capi.solve_csr_upper_noalloc(len(state["b"]), state["off"].data_ptr(), state["cols"].data_ptr(),
                                     state["vals"].data_ptr(), state["b"].data_ptr(), state["x"].data_ptr(),
                                     tol=CSR_TOL, max_iters=20000, stream=state["stream"])
        return state["x"]
    if c["kind"] == "unet":
        net, lab, rhs, p = state["net"], state["lab"], state["rhs"], state["p"]
        if c["op"] == "forward":
            net.forward(lab.data_ptr(), rhs.data_ptr(), state["x"].data_ptr())
            return state["x"]
        if c["op"] == "loss_grad":
            loss, grad = net.loss_grad(lab.data_ptr(), rhs.data_ptr(), p.data_ptr())
            return {"loss": loss, "grad": grad}
        loss = net.train_step(lab.data_ptr(), rhs.data_ptr(), p.data_ptr(), 5e-4, want_loss=True)
        return {"loss": loss, "weights": net.params()}
    s = state["s"]
    if c["kind"] == "frame":
        s.set_particles(state["pos"], state["vel"])
        s.step(c["steps"])
        if c["scheme"] == "ref2d":  # this scheme deletes particles: the arrays are as long as what is left
            pos, vel = s.particles()
        else:
            pos, vel = s.particles(out=(state["out_pos"], state["out_vel"]))
        return {"pos": pos, "vel": vel}
    s.step(c["steps"])
    for k, w in state["which"].items():
        s.grid_to_device(w, state["grids"][k].data_ptr(), state["grids"][k].numel())
    s.labels_to_device(state["lab"].data_ptr(), state["lab"].numel())
    return dict(state["grids"], labels=state["lab"])


# ---------------------------------------------------------------- what a pass cannot do without

def _fluid_fraction(c):
    return {"dam2d": 0.2, "box": 0.55 * 0.6 * 0.7, "dam3d": 0.24, "pool": 0.34, "seabed": 0.27, "boxes": 0.15}[c["scene"]]


def work(case):
    """Bytes: the inputs once and the outputs once (particles, or the state a step reads and writes; labels and grids).
    Flops: the network's convolutions; for a step the transfers of its particles and one application of the operator."""
    c = case
    nc = c["W"] * c["H"] * c["D"]
    if c["kind"] == "csr":
        nnz = 4 * nc
        return {"bytes": 12.0 * nnz + 4.0 * nc + 16.0 * nc, "flops": 2.0 * 7 * nc}
    if c["kind"] == "unet":
        net = [(16, 16, 1), (16, 16, 1), (16, 32, 8), (32, 32, 8), (32, 64, 64), (64, 64, 64), (96, 32, 8), (32, 32, 8),
               (48, 16, 1), (16, 16, 1)]
        fwd = sum(2.0 * 27 * i * o * nc / d for i, o, d in net)
        weights = 4.0 * 27 * sum(i * o for i, o, _ in net)
        if c["op"] == "forward":
            return {"bytes": 9.0 * nc + weights, "flops": fwd}
        return {"bytes": 9.0 * nc + 3 * weights, "flops": 3 * fwd}
    n = _fluid_fraction(c) * nc * c["ppc"]
    per_step = 400.0 * n + 20.0 * _fluid_fraction(c) * nc
    if c["kind"] == "frame":
        return {"bytes": 48.0 * n + nc, "flops": c["steps"] * per_step}
    out = 8.0 if c["kind"] == "pairs" else 16.0
    return {"bytes": 48.0 * n * c["steps"] + (out + 2.0) * nc, "flops": c["steps"] * per_step}


# ---------------------------------------------------------------- the same in 64 bits

def _sh(t, d, o):
    """t shifted by o along dimension d, zero outside: out[i] = t[i + o]."""
    out = torch.zeros_like(t)
    n = t.shape[d]
    out.narrow(d, max(0, -o), n - 1).copy_(t.narrow(d, max(0, o), n - 1))
    return out


def _operator(lab):
    """FLUID mask and diagonal: the FLUID or AIR neighbours inside the grid."""
    fl = lab == FLUID
    wet = ((lab == FLUID) | (lab == AIR)).double()
    diag = torch.zeros(lab.shape, dtype=torch.float64, device=lab.device)
    for d in range(lab.ndim):
        for o in (-1, 1):
            diag += _sh(wet, d, o)
    return fl, diag * fl


def _apply(p, fl, diag):
    s = diag * p
    for d in range(p.ndim):
        for o in (-1, 1):
            s -= _sh(p, d, o)
    return s * fl


def _cg(apply, b, inv, tol=1e-14, most=6000):
    x, r = torch.zeros_like(b), b.clone()
    z = r * inv
    p, rz, bb = z.clone(), (r * z).sum(), (b * b).sum()
    for it in range(most):
        q = apply(p)
        a = rz / (p * q).sum()
        x += a * p
        r -= a * q
        z = r * inv
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
        if it % 32 == 31 and not float((r * r).sum()) > tol * tol * float(bb):
            break
    return x


def _solve(lab, b):
    fl, diag = _operator(lab)
    inv = torch.where(diag > 0, 1.0 / diag.clamp(min=1.0), torch.zeros_like(diag))
    return _cg(lambda v: _apply(v, fl, diag), b * fl, inv)


class _Exact3:
    """The default step scheme without a body, in 64 bits (cells are those of the 32-bit positions)."""

    def __init__(self, c, lab):
        self.W, self.H, self.D = c["W"], c["H"], c["D"]
        self.dx, self.dt = float(np.float32(_dx(c))), float(np.float32(c["dt"]))
        self.alpha, self.C = float(np.float32(0.05)), float(np.float32(0.1))
        self.rk2 = c.get("advection", "rk2") == "rk2"
        self.base = torch.from_numpy(np.ascontiguousarray(lab)).cuda().reshape(self.D, self.H, self.W)
        self.shape = [(self.D, self.H, self.W + 1), (self.D, self.H + 1, self.W), (self.D + 1, self.H, self.W)]

    def label(self, pos):
        h = torch.tensor(self.dx, dtype=torch.float32, device="cuda")
        f = torch.floor(pos.float() / h).long()
        i, j, k = (f[:, a].clamp(0, n - 1) for a, n in enumerate((self.W, self.H, self.D)))
        lab = torch.where(self.base == SOLID, SOLID, AIR).to(torch.uint8).reshape(-1)
        cell = (k * self.H + j) * self.W + i
        hit = torch.zeros_like(lab, dtype=torch.bool)
        hit[cell] = True
        lab[hit & (lab != SOLID)] = FLUID
        self.lab = lab.reshape(self.D, self.H, self.W)

    def stencil(self, a, r, interp):
        """Base indices and fractions of component a at r = x / dx; interp clamps the base so that base + 1 exists."""
        n = [self.W, self.H, self.D]
        b, f = [], []
        for d in range(3):
            s = r[:, d] - (0.0 if d == a else 0.5)
            hi = (n[d] - 1 if d == a else max(n[d] - 2, 0)) if interp else (n[d] if d == a else n[d] - 1)
            i = torch.floor(s).clamp(0, hi)
            b.append(i.long())
            f.append((s - i).clamp(0, 1))
        return b, f

    def p2g(self, pos, vel):
        out = []
        r = pos / self.dx
        for a in range(3):
            sh = self.shape[a]
            num = torch.zeros(math.prod(sh), dtype=torch.float64, device="cuda")
            den = torch.zeros_like(num)
            b, f = self.stencil(a, r, False)
            for o in range(8):
                oo = (o & 1, o >> 1 & 1, o >> 2)
                w = torch.ones_like(f[0])
                ok = torch.ones_like(w, dtype=torch.bool)
                for d in range(3):
                    w = w * (f[d] if oo[d] else 1.0 - f[d])
                    ok &= b[d] + oo[d] < sh[2 - d]
                at = ((b[2] + oo[2]) * sh[1] + b[1] + oo[1]) * sh[2] + b[0] + oo[0]
                num.index_add_(0, at[ok], (w * vel[:, a])[ok])
                den.index_add_(0, at[ok], w[ok])
            out.append(torch.where(den > 1e-8, num / den.clamp(min=1e-30), torch.zeros_like(num)).reshape(sh))
        return out

    def sides(self, t, a, fill):
        """Values left and right of every face of component a."""
        d = 2 - a
        edge = list(t.shape)
        edge[d] = 1
        e = torch.full(edge, fill, dtype=t.dtype, device=t.device)
        return torch.cat([e, t], d), torch.cat([t, e], d)

    def pressure(self, U):
        scale = 1000.0 * self.dx / self.dt
        div = torch.zeros(self.lab.shape, dtype=torch.float64, device="cuda")
        for a in range(3):
            L, R = self.sides(self.lab, a, SOLID)
            u = torch.where((L == SOLID) | (R == SOLID), torch.zeros_like(U[a]), U[a])
            d, n = 2 - a, u.shape[2 - a] - 1
            div += u.narrow(d, 1, n) - u.narrow(d, 0, n)
        self.rhs = torch.where(self.lab == FLUID, -scale * div, torch.zeros_like(div))
        lab = self.lab if self.D > 1 else self.lab[0]
        return _solve(lab, self.rhs.reshape(lab.shape)).reshape(self.lab.shape)

    def project(self, U, p):
        k = self.dt / (1000.0 * self.dx)
        out = []
        for a in range(3):
            L, R = self.sides(self.lab, a, SOLID)
            pL, pR = self.sides(p, a, 0.0)
            out.append(torch.where((L == SOLID) | (R == SOLID), torch.zeros_like(U[a]), U[a] - k * (pR - pL)))
        return out

    def sample(self, grid, a, r):
        b, f = self.stencil(a, r, True)
        sh, g = self.shape[a], grid.reshape(-1)
        v = torch.zeros_like(f[0])
        for o in range(8):
            oo = (o & 1, o >> 1 & 1, o >> 2)
            w = torch.ones_like(v)
            for d in range(3):
                w = w * (f[d] if oo[d] else 1.0 - f[d])
            up = oo[2] if (self.D > 1 or a == 2) else 0
            v += w * g[((b[2] + up) * sh[1] + b[1] + oo[1]) * sh[2] + b[0] + oo[0]]
        return v

    def vel_at(self, U, x):
        r = x / self.dx
        return torch.stack([self.sample(U[a], a, r) for a in range(3)], 1)

    OFFSETS = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0), (1, -1, 0),
               (-1, -1, 0), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1), (0, 1, 1), (0, -1, 1), (0, 1, -1),
               (0, -1, -1), (1, 1, 1), (-1, 1, 1), (1, -1, 1), (1, 1, -1), (-1, -1, 1), (-1, 1, -1), (1, -1, -1),
               (-1, -1, -1), (-2, -1, 0), (0, -1, -2), (-2, -2, 0), (0, -2, -2), (-2, -2, -2), (-2, 0, -2), (2, -1, 0),
               (0, -1, 2)]

    def nudge(self, x):
        """Half a cell toward the nearest FLUID cell centre among the offsets; False where there is none."""
        n = torch.tensor([self.W, self.H, self.D], device="cuda")
        cell = torch.floor(x / self.dx).long()
        best = torch.full((len(x),), 1e10, dtype=torch.float64, device="cuda")
        move, found = torch.zeros_like(x), torch.zeros(len(x), dtype=torch.bool, device="cuda")
        for o in self.OFFSETS:
            off = torch.tensor(o, device="cuda")
            q = cell + off
            ok = ((q >= 0) & (q < n)).all(1)
            at = q.clamp(min=0).minimum(n - 1)
            ok &= self.lab[at[:, 2], at[:, 1], at[:, 0]] == FLUID
            d = (((q + 0.5) * self.dx - x) ** 2).sum(1)
            ok &= d < best
            best = torch.where(ok, d, best)
            move[ok] = off.double() * 0.5 * self.dx
            found |= ok
        return x + move, found

    def advect(self, U, x):
        top = torch.tensor([(n - 1) * self.dx for n in (self.W, self.H, self.D)], dtype=torch.float64, device="cuda")
        floor_speed = math.sqrt(5.0 * self.dx * float(np.float32(9.8)))
        x = x.clone()
        live = torch.arange(len(x), device="cuda")
        t = torch.zeros(len(x), dtype=torch.float64, device="cuda")
        for _ in range(1000):
            if not len(live):
                break
            p, s = x[live], t[live]
            k1 = self.vel_at(U, p)
            dT = self.C * self.dx / (k1.norm(dim=1) + floor_speed)
            last = s + dT >= self.dt
            dT = torch.where(last, self.dt - s, torch.where(s + 2 * dT >= self.dt, 0.5 * dT, dT))
            h = dT[:, None]
            k2 = self.vel_at(U, p + 0.5 * h * k1)
            if self.rk2:
                p = p + h * k2
            else:
                k3 = self.vel_at(U, p + 0.75 * h * k2)
                p = p + h * (2.0 / 9 * k1 + 3.0 / 9 * k2 + 4.0 / 9 * k3)
            p = p.clamp(min=0.0).minimum(top)
            c = torch.floor(p / self.dx).long()
            hit = (self.lab[c[:, 2], c[:, 1], c[:, 0]] == SOLID).nonzero()[:, 0]
            stop = last.clone()
            if len(hit):
                moved, found = self.nudge(p[hit])
                p[hit] = moved
                stop[hit[~found]] = True
            x[live], t[live] = p, s + dT
            live = live[~stop & (p >= 0).all(1)]
        return x

    def step(self, pos, vel):
        """One step; keeps lab, rhs, p and the projected U."""
        self.label(pos)
        saved = self.p2g(pos, vel)
        U = list(saved)
        U[1] = U[1] + self.dt * float(np.float32(-9.81))
        self.p = self.pressure(U)
        self.U = self.project(U, self.p)
        r = pos / self.dx
        pic = self.vel_at(self.U, pos)
        dlt = torch.stack([self.sample(self.U[a] - saved[a], a, r) for a in range(3)], 1)
        vel = self.alpha * pic + (1.0 - self.alpha) * (vel + dlt)
        return self.advect(self.U, pos), vel


def _exact_unet(c, seed):
    lab, rhs, p = _unet_pair(c, seed)
    net = capi.UNet(c["W"], c["H"], c["D"], train=False, seed=seed)
    if c["op"] == "forward":
        net.load(DEFAULT_WEIGHTS)
    w32 = torch.from_numpy(net.params()).cuda()
    net.close()
    w = w32.double().requires_grad_(True)
    spec = [(16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (96, 32), (32, 32), (48, 16), (16, 16)]
    fl = lab == FLUID
    s = rhs.double()[fl].square().mean().sqrt()
    pad = [(-n) % 4 for n in (c["W"], c["H"], c["D"])]
    pad = (0, pad[0], 0, pad[1], 0, pad[2])
    solid = ~fl & (lab != AIR)
    x = torch.stack([rhs.double() / s * fl, fl.double(), (lab == AIR).double(), solid.double()])
    x = torch.cat([F.pad(x[:3], pad), F.pad(x[3:], pad, value=1.0)], 0)
    x = torch.cat([x, torch.zeros((12, *x.shape[1:]), dtype=torch.float64, device="cuda")], 0)[None]
    at = 0
    ws = []
    for ci, co in spec:
        n = 27 * ci * co
        ws.append(w[at:at + n].reshape(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2).contiguous())
        at += n
    head = w[at:at + 16]

    def conv(v, l):
        return F.relu(F.conv3d(v, ws[l], padding=1))

    def up(v):
        return F.interpolate(v, scale_factor=2, mode="nearest")

    e0 = conv(conv(x, 0), 1)
    e1 = conv(conv(F.avg_pool3d(e0, 2), 2), 3)
    e2 = conv(conv(F.avg_pool3d(e1, 2), 4), 5)
    d1 = conv(conv(torch.cat([up(e2), e1], 1), 6), 7)
    d0 = conv(conv(torch.cat([up(d1), e0], 1), 8), 9)
    out = torch.einsum("c,czyx->zyx", head, d0[0])[:c["D"], :c["H"], :c["W"]]
    if c["op"] == "forward":
        return (out * s * fl).detach()
    t = p.double() / s
    loss = ((out - t)[fl].square().sum()) / t[fl].square().sum()
    loss.backward()
    g = w.grad
    if c["op"] == "loss_grad":
        return {"loss": float(loss.detach()), "grad": g}
    g = g * min(1.0, 1.0 / float(g.norm()))
    return {"loss": float(loss.detach()),
            "weights": w32.double() - float(np.float32(5e-4)) * g / (g.abs() + 1e-8)}


def exact(case, seed):
    """64-bit results by torch alone; None for the reference's 2D scheme, whose results are those of its 32-bit
    expressions in particle order, and for the scenes with a moving body."""
    c = case
    if c["kind"] == "csr":
        _, _, _, b = _csr_system(c, seed)
        b = b.reshape(c["D"], c["H"], c["W"])
        one = torch.ones(b.shape, dtype=torch.bool, device="cuda")
        six = torch.full(b.shape, 6.0, dtype=torch.float64, device="cuda")
        return _cg(lambda v: _apply(v, one, six), b, 1.0 / six).reshape(-1)
    if c["kind"] == "unet":
        return _exact_unet(c, seed)
    if c.get("scheme") == "ref2d" or c["scene"] in ("pool", "seabed"):
        return None
    lab = _labels(c, seed)
    e = _Exact3(c, lab)
    pos, vel = (t.double() for t in _particles(lab, _dx(c), c["ppc"], seed))
    for _ in range(c["steps"]):
        pos, vel = e.step(pos, vel)
    if c["kind"] == "frame":
        return {"pos": pos, "vel": vel}
    if c["kind"] == "pairs":
        return {"rhs": e.rhs.reshape(-1), "p": e.p.reshape(-1), "labels": None}
    return {"u": e.U[0].reshape(-1), "v": e.U[1].reshape(-1), "w": e.U[2].reshape(-1), "p": e.p.reshape(-1),
            "labels": None}
