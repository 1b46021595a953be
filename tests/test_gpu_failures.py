"""Failure paths of the step on the GPU, made to happen without any fault.

The persistent pressure solvers wait at grid barriers with a bounded number
of polls.  ``fp_set_wait_limit`` lowers that bound to a single poll, so a
block that is not the last to arrive gives up at once: the kernel records
DEV_TIMEOUT and every block returns at its next barrier.  Nothing waits on a
flag that no one sets, nothing traps, and every access stays in bounds.

Checked through the C ABI, for the solvers with a grid barrier:
  * the step returns FP_ERR_TIMEOUT;
  * the particles (positions and velocities) and the rigid body's state are
    those from before the step: the projection and G2P/advection kernels read
    the solve's status and skip, and the body is not integrated;
  * the next step with the default limit solves to tolerance and matches a
    fresh solver's first step from the same state (the host restored the
    solver's zero-state work grids after the timeout).
"""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _pool_with_sphere(O, solver, n=40):
    from fluidprjct_b200 import capi, scenes
    dx = 1.0 / n
    lab = scenes.box_3d(n, n, n, dx, 2.0, 0.6, 2.0)
    kw = dict(dx=dx, dt=0.002, pic_weight=0.05, solver=solver, tol=1e-7, body_radius=0.1, body_density=0.5,
              body_pos=(0.5, 0.55, 0.5), active_body=1, advection="rk2")
    s = capi.Solver(**kw)
    s.set_labels(lab)
    s.load_sdf(None)
    lab2 = lab.copy()
    lab2[s.labels() == capi.BODY] = capi.BODY
    pos = O.seed3d(lab2, dx, 8, 5)
    vel = np.random.default_rng(5).uniform(-0.3, 0.3, pos.shape).astype(np.float32)
    s.set_particles(pos, vel)
    return s, kw, lab, pos, vel


@pytest.mark.parametrize("solver", ["pcg_mg", "pcg", "pcg_mixed"])
def test_timed_out_solve_changes_nothing_and_the_next_step_recovers(O, solver):
    from fluidprjct_b200 import capi
    s, kw, lab, pos, vel = _pool_with_sphere(O, solver)
    body0 = {k: list(s.stats()[k]) for k in ("body_pos", "body_vel", "body_omega")}

    s.set_wait_limit(1)
    with pytest.raises(capi.FluidError) as e:
        s.step(1)
    assert e.value.code == capi.FP_ERR_TIMEOUT
    st = s.stats()
    assert st["solve_status"] == capi.FP_ERR_TIMEOUT
    p1, v1 = s.particles()
    assert np.array_equal(p1, pos) and np.array_equal(v1, vel), "a timed-out step moved particles"
    for k, v in body0.items():
        assert st[k] == v, f"a timed-out step changed the body's {k}"

    # default limit again: the step solves, and equals a fresh solver's step
    s.set_wait_limit(0)
    s.step(1)
    st = s.stats()
    assert st["solve_status"] == capi.FP_OK and st["residual"] <= 1e-7, st
    f = capi.Solver(**kw)
    f.set_labels(lab)
    f.load_sdf(None)
    f.set_particles(pos, vel)
    f.step(1)
    assert np.array_equal(s.labels(), f.labels())
    for g in (capi.GRID_P, capi.GRID_U, capi.GRID_V, capi.GRID_W):
        assert rel_l2(s.grid(g), f.grid(g)) < 1e-5, g
    pa, va = s.particles()
    pb, vb = f.particles()
    assert rel_l2(pa, pb) < 1e-6 and rel_l2(va, vb) < 1e-5
    assert np.allclose(s.stats()["body_pos"], f.stats()["body_pos"], atol=1e-9)
    f.close()
    s.close()


def test_wait_limit_rejects_negative_values():
    from fluidprjct_b200 import capi
    s = capi.Solver(dx=0.05, dt=0.002)
    with pytest.raises(capi.FluidError) as e:
        s.set_wait_limit(-1)
    assert e.value.code == capi.FP_ERR_ARG
    s.close()


def test_timed_out_csr_solve_is_no_answer():
    """The stand-alone CSR solve with a poll limit of 1 on 148 blocks, through the internal entry that takes the limit
    (fp_solve_csr_upper returns its status as it is): FP_ERR_TIMEOUT, with the caller's x, iteration count and residual
    untouched.  The same call with the default limit then solves."""
    import ctypes as C
    from fluidprjct_b200 import capi
    n = 148 * 512
    off, cols = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32)
    vals, b = np.random.default_rng(2).uniform(1, 2, n), np.ones(n)
    solve = capi.lib()._ZN2fp12csr_cg_solveEiPKiS1_PKdS3_PddiPiS4_P11CUstream_stj  # fp::csr_cg_solve
    solve.restype = C.c_int
    x, it, rr = np.full(n, 7.0), C.c_int(-3), C.c_double(-3.0)

    def call(polls):
        p = lambda a: C.c_void_p(a.ctypes.data)
        return solve(C.c_int(n), p(off), p(cols), p(vals), p(b), p(x), C.c_double(1e-12), C.c_int(10), C.byref(it),
                     C.byref(rr), C.c_void_p(None), C.c_uint(polls))

    assert call(1) == capi.FP_ERR_TIMEOUT
    assert (x == 7.0).all() and it.value == -3 and rr.value == -3.0
    assert call(1 << 27) == capi.FP_OK
    assert np.abs(x * vals - 1).max() <= 1e-12 and 0 < it.value <= 10 and 0 <= rr.value <= 1e-12


@pytest.mark.parametrize("solver", ["pcg_mg", "pcg", "pcg_mixed", "pcg_learned", "pcg_learned_mixed"])
def test_solve_times_of_a_call_that_fails_before_its_last_step(O, solver):
    """t_pcg and t_learned are those of the last solve, also when it is the one that failed and the call's last step was
    still to come.  A solve's time lies within its pressure phase."""
    from fluidprjct_b200 import capi
    from fluidprjct_b200.learned import DEFAULT_WEIGHTS
    s = _pool_with_sphere(O, solver)[0]
    learned = "learned" in solver
    if learned:
        s.load_learned(DEFAULT_WEIGHTS)
    s.step(2)
    st = s.stats()
    assert 0 < st["t_pcg"] <= st["t_pressure"] and (0 < st["t_learned"] < st["t_pcg"] if learned else st["t_learned"] == 0)
    s.set_wait_limit(1)
    with pytest.raises(capi.FluidError) as e:
        s.step(3)
    assert e.value.code == capi.FP_ERR_TIMEOUT
    st2 = s.stats()
    # a solve that gives up at its first barriers takes less time than one that ends
    assert 0 < st2["t_pcg"] - st2["t_learned"] < st["t_pcg"] - st["t_learned"]
    assert st2["t_learned"] > 0 if learned else st2["t_learned"] == 0
    s.close()


def test_ref2d_timers_of_a_call_that_fails_in_its_second_step():
    """The 2D scheme's phase timers are those of the last step that ended, also when a later step of the call fails.  A
    block of water falls freely (no divergence, nothing to solve) and reaches the floor in its second step; the grid
    spacing is so large that the right-hand side there is about 2e38 and the FP32 V-cycle overflows."""
    from fluidprjct_b200 import capi
    n, dx = 20, 1e34
    dt = float(np.sqrt(0.6 * dx / 9.81))  # a fall of 0.6 cells in the first step
    lab = np.full((n, n), capi.AIR, np.uint8)
    lab[0], lab[-1], lab[:, 0], lab[:, -1] = [capi.SOLID] * 4
    s = capi.Solver(dim=2, dx=dx, dt=dt, pic_weight=0.05, solver="pcg_mg", scheme="ref2d", output_format=capi.OUT_NONE)
    s.set_labels(lab)
    j, i = np.meshgrid(np.arange(2, 10), np.arange(4, 16), indexing="ij")
    pos = np.stack([(i.ravel() + 0.5) * dx, (j.ravel() + 0.5) * dx, 0.0 * i.ravel()], 1).astype(np.float32)
    names = ("t_label", "t_p2g", "t_pressure", "t_project", "t_advect", "t_total")

    def timers():
        st = s.stats()
        assert all(st[k] > 0 for k in names)
        assert abs(sum(st[k] for k in names[:-1]) - st["t_total"]) <= 1e-5 * st["t_total"]
        return [st[k] for k in names]

    s.set_particles(pos)
    s.step(1)
    first = timers()
    s.set_particles(pos)
    with pytest.raises(capi.FluidError) as e:
        s.step(3)
    assert e.value.code == capi.FP_ERR_SOLVER and s.stats()["step"] == 2
    assert timers() != first
    # no particles: no phase is left out
    s.set_particles(np.zeros((0, 3), np.float32))
    s.step(2)
    assert s.stats()["step"] == 4 and timers() != first
    s.close()


@pytest.mark.parametrize("solver", ["pcg_mg", "pcg", "pcg_mixed"])
def test_timed_out_solve_with_extrapolation_leaves_the_faces_of_p2g(O, solver):
    """The face grids after a step whose solve gave up hold that step's P2G output, also where velocities are
    extrapolated after the projection (P2G's sums may differ in their last bits)."""
    from fluidprjct_b200 import capi, scenes
    n, dx = 40, 1.0 / 40
    lab = scenes.box_3d(n, n, n, dx, 0.5, 0.5, 2.0)
    pos = O.seed3d(lab, dx, 8, 2)
    vel = np.random.default_rng(2).uniform(-0.5, 0.5, pos.shape).astype(np.float32)
    kw = dict(dx=dx, dt=0.002, solver=solver, output_format=capi.OUT_NONE)
    s, t = capi.Solver(extrapolate=3, **kw), capi.Solver(**kw)
    for a in (s, t):
        a.set_labels(lab)
        a.set_particles(pos, vel)
    s.set_wait_limit(1)
    with pytest.raises(capi.FluidError) as e:
        s.step(1)
    assert e.value.code == capi.FP_ERR_TIMEOUT
    for ph in (capi.PHASE_LABEL, capi.PHASE_P2G, capi.PHASE_SAVE, capi.PHASE_FORCES):
        t.phase(ph)
    for g in (capi.GRID_U, capi.GRID_V, capi.GRID_W):
        assert np.abs(s.grid(g) - t.grid(g)).max() <= 1e-5, g
    s.close()
    t.close()
