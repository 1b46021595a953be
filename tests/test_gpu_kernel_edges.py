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
