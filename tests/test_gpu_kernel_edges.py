"""Kernels at the sizes where their tiling can go wrong, against plain numpy or torch results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd_upper(n, rng):
    """Upper triangle (CSR) of a symmetric matrix with diagonal in [4, 5] and four off-diagonals per row of sum at most
    2: eigenvalues in [2, 7], condition number at most 3.5.  Rows end with their longest reach, some are empty beyond
    the diagonal, and the diagonal is not the first entry of odd rows."""
    rows, cols, vals = [], [], []
    for off in (1, 7, 131):
        if n > off:
            i = np.arange(n - off)
            keep = rng.random(n - off) < 0.8
            rows.append(i[keep])
            cols.append(i[keep] + off)
            vals.append(rng.uniform(-1 / 3, 1 / 3, keep.sum()))
    i = np.arange(n)
    rows.append(i), cols.append(i), vals.append(rng.uniform(4, 5, n))
    rows, cols, vals = map(np.concatenate, (rows, cols, vals))
    order = np.lexsort((np.where(rows % 2, -cols, cols), rows))
    rows, cols, vals = rows[order], cols[order].astype(np.int32), vals[order]
    off = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(rows, minlength=n), out=off[1:])
    return off, cols, vals, rows


# one row; one CTA of 512 rows and its neighbours; one CTA per SM full and one row over; two rows a thread
@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 1025, 148 * 512, 148 * 512 + 1, 2 * 148 * 512 + 77, 1 << 18])
def test_csr_solve_sizes(n):
    """x of A x = b for b = A x_true.  CG stops at ||r|| <= tol ||b||, so ||x - x_true|| / ||x_true|| is at most
    cond tol = 3.5e-12, plus a few ulps of accumulated rounding."""
    import torch
    from fluidprjct_b200 import capi
    rng = np.random.default_rng(n)
    off, cols, vals, rows = _spd_upper(n, rng)
    xt = rng.standard_normal(n)
    b = np.zeros(n)
    np.add.at(b, rows, vals * xt[cols])
    up = rows != cols
    np.add.at(b, cols[up], (vals * xt[rows])[up])
    x, it, rr = capi.solve_csr_upper(off, cols, vals, b, tol=1e-12, max_iters=500)
    assert rr <= 1e-12 and np.linalg.norm(x - xt) <= 1e-11 * np.linalg.norm(xt)
    t = [torch.from_numpy(a).cuda() for a in (off, cols, vals, b)]
    y = torch.full_like(t[3], float("nan"))
    it2, rr2 = capi.solve_csr_upper_noalloc(n, *[a.data_ptr() for a in t], y.data_ptr(), tol=1e-12, max_iters=500)
    assert it2 == it and rr2 <= 1e-12 and np.linalg.norm(y.cpu().numpy() - xt) <= 1e-11 * np.linalg.norm(xt)
    # no iteration allowed: x = 0 and the relative residual 1
    it3, rr3 = capi.solve_csr_upper_noalloc(n, *[a.data_ptr() for a in t], y.data_ptr(), tol=1e-12, max_iters=0)
    assert it3 == 0 and rr3 == 1.0 and not y.any()


def test_csr_solve_leaves_x_alone_when_malformed():
    import torch
    from fluidprjct_b200 import capi
    n = 3000
    off = torch.arange(n + 1, dtype=torch.int32, device="cuda")
    cols = torch.arange(n, dtype=torch.int32, device="cuda")
    one = torch.ones(n, dtype=torch.float64, device="cuda")
    for what, at in (("off", 1500), ("cols", 2999)):
        o, c, x = off.clone(), cols.clone(), torch.full_like(one, 7.0)
        if what == "off":
            o[at] = at + 5  # decreases at the next row
        else:
            c[at] = n
        with pytest.raises(capi.FluidError) as e:
            capi.solve_csr_upper_noalloc(n, o.data_ptr(), c.data_ptr(), one.data_ptr(), one.data_ptr(), x.data_ptr())
        assert e.value.code == capi.FP_ERR_ARG and (x == 7.0).all()


def _cg64(fl, diag, b, tol=1e-13):
    """FP64 CG by torch of the unit operator over the FLUID mask fl (zero-padded by one cell)."""
    import torch

    def apply(v):
        s = diag * v
        for d in range(3):
            s = s - torch.roll(v, 1, d) - torch.roll(v, -1, d)
        return s * fl

    x, r = torch.zeros_like(b), b.clone()
    inv = torch.where(diag > 0, 1.0 / diag.clamp(min=1.0), torch.zeros_like(diag))
    z = r * inv
    p, rz, bb = z.clone(), (r * z).sum(), (b * b).sum()
    for it in range(20000):
        q = apply(p)
        a = rz / (p * q).sum()
        x, r = x + a * p, r - a * q
        z = r * inv
        new = (r * z).sum()
        p, rz = z + (new / rz) * p, new
        if it % 16 == 0 and float((r * r).sum()) <= tol * tol * float(bb):
            break
    return x


# One CTA with one cell per thread and with more (2D, 870 cells); several CTAs; 148 CTAs just below and above one
# cell per thread (71,944 and 78,336 cells); a share above the FP64 and one above the FP32 vectors' shared memory
@pytest.mark.parametrize("solver", ["pcg", "pcg_mixed"])
@pytest.mark.parametrize("shape", [(8, 8, 8), (32, 32, 1), (9, 31, 14), (48, 48, 36), (50, 50, 36), (112, 80, 96),
                                   (128, 96, 114)])
def test_pcg_sizes(solver, shape):
    """A box of water under one layer of air.  The solver stops at ||b - A x|| <= tol ||b|| with tol = 1e-9, so its
    relative error is at most cond(A) tol; the condition number of the operator on h layers of water under a free
    surface is at most 12 / (2 - 2 cos(pi / (2 h + 1))), below 1.3e5 at h = 127, and FP32 storage adds 6e-8."""
    import torch
    from fluidprjct_b200 import capi
    W, H, D = shape
    lab = np.full((D, H, W), 1, np.uint8)
    lab[:, 0], lab[:, -1], lab[:, :, 0], lab[:, :, -1] = 0, 0, 0, 0
    if D > 1:
        lab[0], lab[-1] = 0, 0
    lab[:, -2][lab[:, -2] == 1] = 2
    rng = np.random.default_rng(W * H + D)
    rhs = (rng.standard_normal(lab.shape) * (lab == 1)).astype(np.float32)
    s = capi.Solver(dim=3 if D > 1 else 2, dx=1.0 / W, dt=0.01, solver=solver, tol=1e-9, output_format=capi.OUT_NONE)
    s.set_labels(lab if D > 1 else lab[0])
    t = torch.nn.functional.pad(torch.from_numpy(lab).cuda().int(), (1, 1, 1, 1, 1, 1))
    wet = ((t == 1) | (t == 2)).double()
    fl = (t == 1).double()
    diag = sum(torch.roll(wet, o, d) for d in range(3) for o in (1, -1)) * fl
    want = _cg64(fl, diag, torch.nn.functional.pad(torch.from_numpy(rhs).cuda().double(), (1, 1, 1, 1, 1, 1)))
    want = want[1:-1, 1:-1, 1:-1]
    h = H - 3
    bound = 1e-9 * 12 / (2 - 2 * np.cos(np.pi / (2 * h + 1))) + 1e-7
    for _ in range(2):  # the second solve finds the work grids as the first left them
        x, it, rr, rc = s.pressure_solve(rhs)
        assert rc == 0 and rr <= 1e-9
        err = torch.from_numpy(x).cuda().double() - want
        assert float(err.norm() / want.norm()) <= bound
        assert not x[lab != 1].any()
    s.close()


def _ragged(shape, seed):
    """Labels: water with 3 % AIR and 8 % SOLID cells strewn in, SOLID where a piece of water touches no AIR."""
    from scipy.ndimage import binary_dilation, label
    rng = np.random.default_rng(seed)
    lab = rng.choice([0, 1, 2], size=shape, p=[0.08, 0.89, 0.03]).astype(np.uint8)
    part, n = label(lab == 1)
    open_ = np.unique(part[binary_dilation(lab == 2) & (lab == 1)])
    lab[(lab == 1) & ~np.isin(part, open_)] = 0
    if not (lab == 1).any():
        lab.flat[:2] = 1, 2
    return lab


# rows of one cell, of a quad with 1, 2 and 3 cells over, and of whole quads; one level only; the last grid-wide and the
# first block level; 2D; lists of up to one, two and more quads a thread
@pytest.mark.parametrize("shape", [(1, 5, 4), (4, 3, 2), (5, 5, 5), (6, 70, 1), (7, 33, 18), (31, 30, 29), (64, 64, 1),
                                   (129, 131, 1), (34, 61, 47), (66, 64, 70), (128, 128, 40), (157, 96, 83)])
def test_mg_quad_rows(shape):
    """The solve ends with ||b - A x|| <= 1e-9 ||b|| in FP64; rounding x to FP32 adds at most ||A|| 2^-24 ||x||, and
    ||A|| <= 12.  Twice the first term leaves room for the recurrence's drift."""
    import torch
    from fluidprjct_b200 import capi
    W, H, D = shape
    lab = _ragged((D, H, W), W * H + D)
    rng = np.random.default_rng(7)
    t = torch.nn.functional.pad(torch.from_numpy(lab).cuda().int(), (1, 1, 1, 1, 1, 1))
    fl = (t == 1).double()
    wet = ((t == 1) | (t == 2)).double()
    diag = sum(torch.roll(wet, o, d) for d in range(3) for o in (1, -1)) * fl
    s = capi.Solver(dim=3 if D > 1 else 2, dx=1.0 / 64, dt=0.01, solver="pcg_mg", tol=1e-9, output_format=capi.OUT_NONE)
    s.set_labels(lab if D > 1 else lab[0])
    for _ in range(2):  # the second solve finds the work grids as the first left them
        rhs = (rng.standard_normal(lab.shape) * (lab == 1)).astype(np.float32)
        x, it, rr, rc = s.pressure_solve(rhs)
        b = torch.nn.functional.pad(torch.from_numpy(rhs).cuda().double(), (1, 1, 1, 1, 1, 1))
        y = torch.nn.functional.pad(torch.from_numpy(x).cuda().double(), (1, 1, 1, 1, 1, 1))
        res = b - (diag * y - sum(torch.roll(y, o, d) for d in range(3) for o in (1, -1)) * fl)
        assert rc == 0 and not x[lab != 1].any()
        assert float(res.norm()) <= 2e-9 * float(b.norm()) + 12 * 2.0 ** -24 * float(y.norm())
    s.close()


def _faces_force(lab, p, dx, phi, com):
    """The face-fraction force and torque over every face of the grid, in FP64 (phi: SDF at given points)."""
    D, H, W = lab.shape
    P = np.pad(p.astype(np.float64), 1)
    L = np.pad(lab, 1)
    fa = (L == 1) | (L == 2)
    s, n = np.zeros_like(P), np.zeros_like(P)
    for d in range(3):
        for o in (1, -1):
            s += np.roll(np.where(fa, P, 0.0), o, d)
            n += np.roll(fa.astype(float), o, d)
    ext = np.where(L == 3, np.divide(s, n, out=np.zeros_like(s), where=n > 0), P)
    out = np.zeros(6)
    ax = [np.arange(m + 1, dtype=np.float32) for m in (W, H, D)]
    for a in range(3):
        x = [(c if a == b else c[:-1] + np.float32(0.5)) * np.float32(dx) for b, c in enumerate(ax)]
        X = np.stack(np.meshgrid(*x, indexing="ij")).astype(np.float32)  # 3, i, j, k
        th = np.clip(0.5 - phi(X) / dx, 0, 1)
        idx = np.stack(np.meshgrid(*[np.arange(len(c)) for c in x], indexing="ij"))
        hi = tuple(idx[2 - b] + 1 for b in range(3))
        lo = tuple(idx[2 - b] + (0 if 2 - b == a else 1) for b in range(3))
        ok = (th > 0) & (L[lo] != 0) & (L[hi] != 0)
        dF = np.where(ok, -th * (ext[hi] - ext[lo]) * dx * dx, 0.0)
        r = X.astype(np.float64) - np.asarray(com, np.float64)[:, None, None, None]
        f = np.zeros_like(r)
        f[a] = dF
        out[:3] += f.sum((1, 2, 3))
        out[3:] += np.stack([r[1] * f[2] - r[2] * f[1], r[2] * f[0] - r[0] * f[2], r[0] * f[1] - r[1] * f[0]]).sum((1, 2, 3))
    return out


# a sphere inside; over a corner of the grid; wholly outside it; larger than it; paddles inside and past both ends
@pytest.mark.parametrize("body", [("s", (0.5, 0.4, 0.5), 0.2), ("s", (0.02, 0.05, 0.9), 0.15), ("s", (2.0, 0.4, 0.5), 0.3),
                                  ("s", (0.5, 0.4, 0.5), 3.0), ("p", 0.31, 0), ("p", -0.4, 0), ("p", 1.7, 0)])
def test_body_force_box(body):
    """The force sums only the faces of the body's box.  Against every face of the grid in FP64: the kernel's theta is
    FP32 (rounding of phi / dx, about n 2^-24 for the n faces across the body), so 1e-5 of the sum of magnitudes."""
    from fluidprjct_b200 import capi, scenes
    n, dx = 24, np.float32(1 / 24)
    lab = scenes.box_3d(n, n + 5, n - 3, float(dx), 2.0, 0.8, 2.0)
    kw = dict(dx=float(dx), dt=0.002, solver="pcg_mg", output_format=capi.OUT_NONE, active_body=1)
    s = capi.Solver(**kw, **(dict(body_radius=body[2], body_pos=body[1], body_density=0.0, body_mass=0.0)
                             if body[0] == "s" else {}))
    s.set_labels(lab)
    if body[0] == "s":
        s.load_sdf(None)
        com = np.float32(body[1])
        phi = lambda X: np.sqrt(((X - com[:, None, None, None]) ** 2).sum(0)) - np.float32(body[2])
    else:
        s.set_paddle(body[1], 0.0, 1.0)
        com = np.float32([body[1], np.float32(0.5 * (n + 5) * float(dx)), np.float32(0.5 * (n - 3) * float(dx))])
        phi = lambda X: X[0] - com[0]
    lab = s.labels()
    p = np.random.default_rng(5).standard_normal(lab.shape).astype(np.float32)
    s.set_grid(capi.GRID_P, p)
    s.phase(capi.PHASE_BODY)
    st = s.stats()
    got = np.array(list(st["body_force"]) + list(st["body_torque"]))
    want = _faces_force(lab, p, float(dx), phi, com)
    scale = np.abs(p).sum() * float(dx) ** 2 * 6 if (lab == 3).any() else 1e-12
    assert np.abs(got - want).max() <= 1e-5 * scale
    if body in (("s", (2.0, 0.4, 0.5), 0.3), ("p", -0.4, 0)):
        assert not got.any()
    s.close()


@pytest.mark.parametrize("cells", [(120, 110), (128, 124), (330, 200)])
def test_ref2d_scan_sizes(cells):
    """The 2D step's scans below, at and above one pass of a block (16,384 bins or particles): P2G of one particle per
    cell at its centre gives each face its own cell's velocity, and no particle is lost or reordered."""
    from fluidprjct_b200 import capi
    W, H = cells
    lab = np.full((H, W), 2, np.uint8)
    lab[0], lab[-1], lab[:, 0], lab[:, -1] = 0, 0, 0, 0
    dx = 1.0 / 512
    s = capi.Solver(dim=2, dx=dx, dt=1e-4, pic_weight=0.0, solver="pcg_mg", scheme="ref2d", output_format=capi.OUT_NONE)
    s.set_labels(lab)
    jj, ii = np.meshgrid(np.arange(1, H - 1), np.arange(1, W - 1), indexing="ij")
    pos = np.stack([(ii.ravel() + 0.5) * dx, (jj.ravel() + 0.5) * dx, 0 * ii.ravel()], 1).astype(np.float32)
    vel = np.random.default_rng(1).uniform(-1, 1, pos.shape).astype(np.float32)
    vel[:, 2] = 0
    s.set_particles(pos, vel)
    s.phase(capi.PHASE_LABEL)
    s.phase(capi.PHASE_P2G)
    u, v = s.grid(capi.GRID_U)[0], s.grid(capi.GRID_V)[0]
    # neighbours' weights are hat(1 +- 2^-24 W), so at most W 2^-23 of their speed leaks in
    assert np.abs(u[1:-1, 1:-2] - vel[:, 0].reshape(H - 2, W - 2)).max() <= 8 * W * 2.0 ** -23
    assert np.abs(v[1:-2, 1:-1] - vel[:, 1].reshape(H - 2, W - 2)).max() <= 8 * W * 2.0 ** -23
    s.phase(capi.PHASE_CLEANUP)
    p2, v2 = s.particles()
    assert np.array_equal(p2, pos) and np.array_equal(v2, vel)
    s.close()


# one voxel on the coarsest level; whole 8 x 16 x 8 bricks; remainders in every axis; several bricks in z
@pytest.mark.parametrize("shape", [(4, 4, 4), (8, 16, 32), (12, 20, 36), (28, 36, 20), (40, 12, 72)])
def test_unet_gradient_tiles(shape):
    """Every layer's weight gradient against the oracle, which rounds to BF16 where the kernels do: only the order of
    FP32 sums and the BF16 flips it causes differ.  A flip is 2^-8 of one activation; 3e-2 and a cosine of 0.999 are
    the bounds that the network's other gradient test uses for them."""
    import torch
    from fluidprjct_b200 import capi
    from oracle import unet_oracle as U
    D, H, W = shape
    rng = np.random.default_rng(W + 10 * H + 100 * D)
    lab = np.where(rng.random(shape) < 0.8, 1, rng.integers(0, 4, shape)).astype(np.uint8)
    rhs, p = [np.where(lab == 1, rng.standard_normal(shape), 0).astype(np.float32) for _ in range(2)]
    th = U.init_params(D + H)
    net = capi.UNet(W, H, D, train=True)
    net.set_params(th)
    t = [torch.from_numpy(a).cuda() for a in (lab, rhs, p)]
    torch.cuda.synchronize()
    loss, g = net.loss_grad(*[a.data_ptr() for a in t])
    loss_ref, g_ref = U.loss_grad(th, lab, rhs, p, bf=True)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    at = np.cumsum([0] + U.layer_sizes() + [U.HEAD])
    for a, b in zip(at[:-1], at[1:]):
        x, y = g[a:b].astype(np.float64), g_ref[a:b].astype(np.float64)
        if not np.linalg.norm(y):
            assert not x.any()
            continue
        assert np.linalg.norm(x - y) <= 3e-2 * np.linalg.norm(y)
        assert x @ y >= 0.999 * np.linalg.norm(x) * np.linalg.norm(y)
    loss2, g2 = net.loss_grad(*[a.data_ptr() for a in t])
    assert loss2 == loss and np.array_equal(g2, g)


# grids smaller than a brick of 8 x 4 x 4, of whole bricks, with remainders in every axis, and flat
@pytest.mark.parametrize("shape", [(5, 3, 2), (8, 4, 4), (16, 8, 8), (17, 9, 5), (23, 6, 13), (33, 17, 1)])
def test_p2g_brick_edges(shape):
    """P2G against numpy in FP64, with empty cells, crowded ones (up to 40 particles) and particles on the far edges.
    Weights are products of three FP32 fractions (3 ulps each) and num and den sum at most 27 cells of at most 40
    particles: relative error of a face below (3 + 27 * 40) 2^-24 of its terms' magnitude, 7e-5; faces whose weights
    sum to less than 1e-3 are left out, since the fractions' absolute error (W 2^-24) is not small against them."""
    from fluidprjct_b200 import capi
    W, H, D = shape
    dx = np.float32(0.125)
    s = capi.Solver(dim=3 if D > 1 else 2, dx=float(dx), dt=0.01, output_format=capi.OUT_NONE)
    lab = np.full((D, H, W), 2, np.uint8)
    s.set_labels(lab if D > 1 else lab[0])
    rng = np.random.default_rng(W)
    n = W * H * D * 3
    pos = (rng.random((n, 3)) * np.array([W, H, D]) * dx).astype(np.float32)
    pos[: n // 6] = (rng.random((n // 6, 3)) * dx * 1.2).astype(np.float32)[:, :3]
    pos[-3:] = [[W * dx, 0, 0], [0, H * dx, 0], [0, 0, D * dx]]
    pos = np.minimum(pos, np.array([W, H, D], np.float32) * dx)
    if D == 1:
        pos[:, 2] = 0
    vel = rng.uniform(-1, 1, pos.shape).astype(np.float32)
    s.set_particles(pos, vel)
    for _ in range(2):  # the second transfer finds the pair array as the first left it
        s.phase(capi.PHASE_LABEL)
        s.phase(capi.PHASE_P2G)
    N = (W, H, D)
    r = pos.astype(np.float64) / float(dx)
    for a, which in enumerate((capi.GRID_U, capi.GRID_V, capi.GRID_W)):
        sh = tuple(N[d] + (d == a) for d in range(3))
        num, den = np.zeros(sh), np.zeros(sh)
        b, f = [], []
        for d in range(3):
            t = r[:, d] - (0.0 if d == a else 0.5)
            i = np.clip(np.floor(t), 0, N[d] if d == a else N[d] - 1)
            b.append(i.astype(int)), f.append(np.clip(t - i, 0, 1))
        for o in np.ndindex(2, 2, 2):
            w = np.prod([f[d] if o[d] else 1 - f[d] for d in range(3)], axis=0)
            q = [b[d] + o[d] for d in range(3)]
            ok = np.all([q[d] < sh[d] for d in range(3)], axis=0)
            np.add.at(num, tuple(c[ok] for c in q), (w * vel[:, a])[ok])
            np.add.at(den, tuple(c[ok] for c in q), w[ok])
        got = s.grid(which).transpose(2, 1, 0)
        far = den > 1e-3
        assert np.abs(got[far] - num[far] / den[far]).max() <= 1e-4
        assert not got[den == 0].any()
    s.close()


@pytest.mark.parametrize("dx", [1 / 160, 0.1, 0.02, 1 / 3, 0.0123, 1.9999999, 1.0000001, 0.99999994, 7.7, 0.25])
def test_cell_of_a_boundary_particle(dx):
    """Cells are floor(p / dx) of the FP32 quotient, exactly: one particle per row of cells, on a cell boundary or within
    three ulps of it, marks its cell FLUID and no other."""
    from fluidprjct_b200 import capi
    W, H, D = 64, 30, 30
    d = np.float32(dx)
    s = capi.Solver(dim=3, dx=float(d), dt=0.01, output_format=capi.OUT_NONE)
    s.set_labels(np.full((D, H, W), 2, np.uint8))
    rng = np.random.default_rng(3)
    j, k = np.meshgrid(np.arange(H), np.arange(D), indexing="ij")
    j, k = j.ravel(), k.ravel()
    x = (rng.integers(1, W, j.size).astype(np.float32) * d).view(np.int32) + rng.integers(-3, 4, j.size, dtype=np.int32)
    pos = np.stack([x.view(np.float32), (j + np.float32(0.5)) * d, (k + np.float32(0.5)) * d], 1).astype(np.float32)
    s.set_particles(pos)
    s.phase(capi.PHASE_LABEL)
    want = np.full((D, H, W), 2, np.uint8)
    want[k, j, np.floor(pos[:, 0] / d).astype(int)] = 1
    assert np.array_equal(s.labels(), want)
    s.close()


def test_p2g_of_a_velocity_that_is_not_finite():
    """A particle whose velocity has become infinite or NaN (here from faces set so) spoils the eight faces per component
    that it reaches and no other, not even those that other particles of its cell could reach.  The weights are exact
    (products of quarters), so the other faces are those of the finite particles, to the rounding of at most 18 terms,
    their sum and a quotient."""
    from fluidprjct_b200 import capi
    W, H, D, dx = 20, 14, 13, 0.125
    s = capi.Solver(dim=3, dx=dx, dt=0.01, output_format=capi.OUT_NONE)
    s.set_labels(np.full((D, H, W), 2, np.uint8))
    k, j, i = np.meshgrid(*[np.arange(m) for m in (D, H, W)], indexing="ij")
    cell = np.stack([i.ravel(), j.ravel(), k.ravel()], 1)
    rng = np.random.default_rng(4)
    s.set_particles(((cell + rng.choice([0.25, 0.75], cell.shape)) * dx).astype(np.float32))
    grids = (capi.GRID_U, capi.GRID_V, capi.GRID_W)
    for which in grids:
        g = rng.uniform(-1, 1, s.grid(which).shape).astype(np.float32)
        g[0, 0, 0], g[4, 3, 8], g[6, 8, 13] = np.inf, np.nan, -np.inf  # a corner, an edge of a brick, inside one
        s.set_grid(which, g)
    s.phase(capi.PHASE_G2P)
    s.phase(capi.PHASE_LABEL)
    s.phase(capi.PHASE_P2G)
    pos, vel = s.particles()
    r, vel = pos.astype(np.float64) / dx, vel.astype(np.float64)
    N = (W, H, D)
    for a, which in enumerate(grids):
        good = np.isfinite(vel[:, a])
        sh = tuple(N[d] + (d == a) for d in range(3))
        num, den, hit = np.zeros(sh), np.zeros(sh), np.zeros(sh, bool)
        t = r - 0.5 * (np.arange(3) != a)
        b = np.maximum(np.floor(t), 0).astype(int)
        f = np.clip(t - b, 0, 1)
        for o in np.ndindex(2, 2, 2):
            w = np.prod(np.where(o, f, 1 - f), axis=1)
            q = b + np.array(o)
            ok = (q < sh).all(1) & (w > 0)
            hit[tuple(q[ok & ~good].T)] = True
            np.add.at(num, tuple(q[ok & good].T), (w * np.where(good, vel[:, a], 0))[ok & good])
            np.add.at(den, tuple(q[ok & good].T), w[ok & good])
        got = s.grid(which).transpose(2, 1, 0)
        assert hit.any() and not np.isfinite(got[hit]).any()
        rest = ~hit & (den > 0)
        assert np.isfinite(got[rest]).all()
        assert np.abs(got[rest] - num[rest] / den[rest]).max() <= 24 * 2.0 ** -24
    s.close()


# dx no power of two; grids smaller than a brick, of whole bricks, with remainders in every axis, and flat
@pytest.mark.parametrize("shape, dx", [((5, 3, 2), 0.1), ((16, 8, 8), 1 / 3), ((17, 9, 5), 1 / 160), ((23, 6, 13), 7.7),
                                       ((33, 17, 1), 0.0123)])
def test_p2g_brick_edges_at_any_spacing(shape, dx):
    """P2G at a spacing whose quotients round, against numpy sums in FP64 of the same FP32 quotients: empty cells, cells
    of one to 70 particles side by side (lanes of a warp walk lists of different lengths), particles on and beyond the
    far edges.  The bound is that of weights of three FP32 factors (9 ulps with the fractions) and sums over at most 27
    cells of 70 particles, (9 + 27 * 70) 2^-24 = 1.2e-4 of the largest speed; faces of weight below 1e-3 are left out."""
    from fluidprjct_b200 import capi
    W, H, D = shape
    dx = np.float32(dx)
    s = capi.Solver(dim=3 if D > 1 else 2, dx=float(dx), dt=0.01, output_format=capi.OUT_NONE)
    lab = np.full((D, H, W), 2, np.uint8)
    s.set_labels(lab if D > 1 else lab[0])
    rng = np.random.default_rng(W + H)
    cell = np.stack(np.meshgrid(*[np.arange(m) for m in shape], indexing="ij"), -1).reshape(-1, 3)
    cell = np.repeat(cell, rng.choice([0, 1, 3, 70], len(cell), p=[0.3, 0.3, 0.35, 0.05]), axis=0)
    cell = rng.permutation(cell)
    far = np.array(shape)
    edge = np.concatenate([np.eye(3) * far, far[None], far + np.eye(3) * 0.75, [[0, 0, 0]]])  # on and beyond the far edges
    pos = (np.concatenate([cell + rng.random(cell.shape), edge]) * float(dx)).astype(np.float32)
    if D == 1:
        pos[:, 2] = 0
    vel = rng.uniform(-1, 1, pos.shape).astype(np.float32)
    s.set_particles(pos, vel)
    for _ in range(2):  # the second transfer finds the pair array as the first left it
        s.phase(capi.PHASE_LABEL)
        s.phase(capi.PHASE_P2G)
    r = (pos / dx).astype(np.float64)
    assert (pos / dx).dtype == np.float32
    for a, which in enumerate((capi.GRID_U, capi.GRID_V, capi.GRID_W)):
        sh = tuple(shape[d] + (d == a) for d in range(3))
        num, den = np.zeros(sh), np.zeros(sh)
        b, f = [], []
        for d in range(3):
            t = r[:, d] - (0.0 if d == a else 0.5)
            i = np.clip(np.floor(t), 0, shape[d] if d == a else shape[d] - 1)
            b.append(i.astype(int)), f.append(np.clip(t - i, 0, 1))
        for o in np.ndindex(2, 2, 2):
            w = np.prod([f[d] if o[d] else 1 - f[d] for d in range(3)], axis=0)
            q = [b[d] + o[d] for d in range(3)]
            ok = np.all([q[d] < sh[d] for d in range(3)], axis=0)
            np.add.at(num, tuple(c[ok] for c in q), (w * vel[:, a])[ok])
            np.add.at(den, tuple(c[ok] for c in q), w[ok])
        got = s.grid(which).transpose(2, 1, 0)
        heavy = den > 1e-3
        assert np.abs(got[heavy] - num[heavy] / den[heavy]).max() <= 1.2e-4
        assert not got[den == 0].any()
    s.close()


def _mg_residual(lab, seed, solves=2):
    """Solves by pcg_mg to 1e-9 with random right-hand sides and the bound of test_mg_quad_rows."""
    import torch
    from fluidprjct_b200 import capi
    D, H, W = lab.shape
    rng = np.random.default_rng(seed)
    t = torch.nn.functional.pad(torch.from_numpy(lab).cuda().int(), (1, 1, 1, 1, 1, 1))
    fl = (t == 1).double()
    wet = ((t == 1) | (t == 2)).double()
    diag = sum(torch.roll(wet, o, d) for d in range(3) for o in (1, -1)) * fl
    s = capi.Solver(dim=3 if D > 1 else 2, dx=1.0 / 64, dt=0.01, solver="pcg_mg", tol=1e-9, output_format=capi.OUT_NONE)
    s.set_labels(lab if D > 1 else lab[0])
    for _ in range(solves):  # the second solve finds the work grids as the first left them
        rhs = (rng.standard_normal(lab.shape) * (lab == 1)).astype(np.float32)
        x, it, rr, rc = s.pressure_solve(rhs)
        b = torch.nn.functional.pad(torch.from_numpy(rhs).cuda().double(), (1, 1, 1, 1, 1, 1))
        y = torch.nn.functional.pad(torch.from_numpy(x).cuda().double(), (1, 1, 1, 1, 1, 1))
        res = b - (diag * y - sum(torch.roll(y, o, d) for d in range(3) for o in (1, -1)) * fl)
        assert rc == 0 and it > 0 and not x[lab != 1].any()
        assert float(res.norm()) <= 2e-9 * float(b.norm()) + 12 * 2.0 ** -24 * float(y.norm())
    s.close()


# grids that no coarser one follows: level 0 is the whole hierarchy, swept by one block in global memory
@pytest.mark.parametrize("shape", [(2, 2, 2), (2, 1, 2), (2, 2, 1), (1, 2, 1)])
@pytest.mark.parametrize("air", [0, 1, -1])
def test_mg_one_level(shape, air):
    """A hierarchy of one level, all FLUID but one AIR cell (a red or a black one)."""
    lab = np.full(shape[::-1], 1, np.uint8)
    lab.flat[air] = 2
    _mg_residual(lab, 3)


# 938 and 1016 cells are left on the last of eight levels, in rows of one cell, which with their padding do not fit
@pytest.mark.parametrize("shape", [(3, 120000, 1), (4, 130000, 1), (2, 3, 120000)])
def test_mg_block_level_in_global_memory(shape):
    """Grids so long that not even the last level's copy fits in shared memory: block 0 solves it in global memory."""
    _mg_residual(_ragged(shape[::-1], shape[0]), 5)


def _face_terms(lab, p, dx, phi, com):
    """The face-fraction force's terms over every face of the grid, in FP64: (6, n) force and torque contributions, and
    each face's largest one (theta = 1).  phi gives the SDF at FP32 points and where it is in doubt."""
    P, L = np.pad(p.astype(np.float64), 1), np.pad(lab, 1)
    fa = (L == 1) | (L == 2)
    s, n = np.zeros_like(P), np.zeros_like(P)
    for d in range(3):
        for o in (1, -1):
            s += np.roll(np.where(fa, P, 0.0), o, d)
            n += np.roll(fa.astype(float), o, d)
    ext = np.where(L == 3, np.divide(s, n, out=np.zeros_like(s), where=n > 0), P)
    terms, doubt = [], []
    for a in range(3):
        c = [np.arange(m + (b == a), dtype=np.float32) for b, m in enumerate(lab.shape[::-1])]
        X = np.stack(np.meshgrid(*[(v if a == b else v + np.float32(0.5)) * np.float32(dx) for b, v in enumerate(c)],
                                 indexing="ij")).astype(np.float32).reshape(3, -1)
        i = np.stack(np.meshgrid(*[np.arange(len(v)) for v in c], indexing="ij")).reshape(3, -1)
        hi = tuple(i[2 - b] + 1 for b in range(3))
        lo = tuple(i[2 - b] + (2 - b != a) for b in range(3))
        f, unsure = phi(X)
        full = np.where((L[lo] != 0) & (L[hi] != 0), -(ext[hi] - ext[lo]) * dx * dx, 0.0)
        r = X.astype(np.float64) - np.asarray(com, np.float64)[:, None]

        def wrench(dF):
            F = np.zeros_like(r)
            F[a] = dF
            return np.concatenate([F, np.cross(r, F, axis=0)])
        terms.append(wrench(np.clip(0.5 - f / dx, 0, 1) * full))
        doubt.append(wrench(np.where(unsure, full, 0.0)))
    return np.concatenate(terms, 1), np.concatenate(doubt, 1)


# spheres inside, over a corner, outside and around the grid; paddles inside and past both ends; a voxel SDF turned about
# all axes: inside, over a corner, wholly outside
@pytest.mark.parametrize("body", [("s", (0.5, 0.4, 0.5), 0.2), ("s", (0.02, 0.05, 0.9), 0.15), ("s", (2.0, 0.4, 0.5), 0.3),
                                  ("s", (0.5, 0.4, 0.5), 3.0), ("p", 0.31, 0), ("p", -0.4, 0), ("p", 1.7, 0),
                                  ("v", (0.55, 0.5, 0.45), 0), ("v", (0.05, 0.1, 0.8), 0), ("v", (-3.0, 0.5, 0.5), 0)])
def test_body_force_of_every_face_in_the_box(body, tmp_path):
    """The force and torque of the body's box against all faces of the grid, to 1e-5 of the sum of the terms' magnitudes
    (FP32 theta: the rounding of phi / dx, about n 2^-24 for the n faces across).  A face at a voxel's side, where FP32
    may read the next voxel, may count as any theta from 0 to 1."""
    from fluidprjct_b200 import capi, scenes
    n, dx = 24, np.float32(1 / 24)
    lab = scenes.box_3d(n, n + 5, n - 3, float(dx), 2.0, 0.8, 2.0)
    kw = dict(dx=float(dx), dt=0.5, solver="pcg_mg", output_format=capi.OUT_NONE, active_body=1, body_mass=1e-3)
    if body[0] == "s":
        kw.update(body_radius=body[2], body_pos=body[1], body_density=0.0)
    elif body[0] == "v":
        kw.update(body_pos=body[1])
    s = capi.Solver(**kw)
    s.set_labels(lab)
    com = np.float32(body[1]) if body[0] != "p" else None
    weight = 1e-3
    if body[0] == "s":
        s.load_sdf(None)
        phi = lambda X: (np.sqrt(((X - com[:, None]) ** 2).sum(0)) - np.float32(body[2]), False)
    elif body[0] == "p":
        s.set_paddle(body[1], 0.0, 1.0)
        com = np.float32([body[1], np.float32(0.5 * (n + 5) * float(dx)), np.float32(0.5 * (n - 3) * float(dx))])
        phi = lambda X: (X[0] - com[0], False)
        weight = 0.0
    else:
        nv, org, cell = np.array([17, 11, 23]), np.float32([-0.1, 0.2, 0.05]), np.float32(0.03)
        val = np.random.default_rng(8).uniform(-1.0, 0.4, nv).astype(np.float32) * dx
        with open(tmp_path / "body.sdf", "w") as f:
            f.write(" ".join(map(str, nv)) + "\n" + " ".join("%.9g" % v for v in [*org, cell]) + "\n")
            f.write("\n".join("%.9g" % v for v in val.transpose(2, 1, 0).ravel()))
        s.load_sdf(tmp_path / "body.sdf")
        s.set_body_state(omega=(0.8, 1.1, -0.7))  # turned by the first integration, in the rotation from the second on
        for _ in range(2):
            s.phase(capi.PHASE_BODY)
            s.set_body_state(pos=body[1], vel=(0, 0, 0), omega=(0, 0, 0))
        th, ps, ph = s.stats()["body_angles"]
        ct, st, cp, sp, cf, sf = np.cos(th), np.sin(th), np.cos(ps), np.sin(ps), np.cos(ph), np.sin(ph)
        R = np.array([[ct * cp, st * sf - ct * cf * sp, cf * st + ct * sf * sp], [sp, cf * cp, -cp * sf],
                      [-cp * st, ct * sf + cf * st * sp, ct * cf - st * sf * sp]]).astype(np.float32)
        assert np.abs(R - np.eye(3)).max() > 0.3
        lc = org + (nv * cell).astype(np.float32) * np.float32(0.5)

        def phi(X):
            d = (X - com[:, None]).astype(np.float64)
            q = (R.astype(np.float64).T @ d + lc[:, None] - org[:, None]) / cell
            unsure = (np.abs(q - np.round(q)) < 2e-4).any(0) & ((q > -1) & (q < nv[:, None] + 1)).all(0)
            i = np.floor(q).astype(int)
            ins = ((i >= 0) & (i < nv[:, None])).all(0)
            i = np.where(ins, i, 0)
            return np.where(ins, val[tuple(i)], np.float32(1e30)), unsure
        s.phase(capi.PHASE_LABEL)
    lab = s.labels()
    p = np.random.default_rng(5).standard_normal(lab.shape).astype(np.float32)
    s.set_grid(capi.GRID_P, p)
    s.phase(capi.PHASE_BODY)
    st = s.stats()
    got = np.array(list(st["body_force"]) + list(st["body_torque"]))
    got[1] += float(np.float32(weight)) * float(np.float32(9.81))
    terms, doubt = _face_terms(lab, p, float(dx), phi, com)
    tol = 1e-5 * np.abs(terms).sum(1) + 1e-12
    assert (np.abs(got - terms.sum(1)) <= tol + np.abs(doubt).sum(1)).all(), (got, terms.sum(1), tol)
    # the bound sees a face: most of the body's carry more than it
    if np.abs(terms).sum() > 0:
        assert (np.median(np.abs(terms[:3][terms[:3] != 0])) > tol[:3]).all()
    else:
        assert not got[3:].any()
    s.close()


def test_csr_solve_of_two_million_rows():
    """As test_csr_solve_sizes, beyond the allocation-free call's range: 28 rows and more a thread."""
    from fluidprjct_b200 import capi
    n = (1 << 21) + 77
    rng = np.random.default_rng(3)
    off, cols, vals, rows = _spd_upper(n, rng)
    xt = rng.standard_normal(n)
    b = np.bincount(rows, vals * xt[cols], n)
    up = rows != cols
    b += np.bincount(cols[up], (vals * xt[rows])[up], n)
    x, it, rr = capi.solve_csr_upper(off, cols, vals, b, tol=1e-12, max_iters=500)
    assert rr <= 1e-12 and np.linalg.norm(x - xt) <= 1e-11 * np.linalg.norm(xt)
