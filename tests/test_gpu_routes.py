"""Calls in orders and shapes that take another route through the host runtime
or the dispatch than the plain run of one case."""
import numpy as np
import pytest

import sddc_oracle as O
from helpers import case_channel, case_cylinder, case_periodic, rel_l2
from sddc_b200 import cases, ensemble, host, mesh
from sddc_b200.solver import NumericalFault, Solver

pytestmark = pytest.mark.gpu


def _records(ncell, n, ph, dt):
    edges = np.linspace(0, ncell, n + 1).astype(int)
    return [dict(first_cell=int(a), ncell=int(b - a), dt=dt, rinf=ph.rinf, pinf=ph.pinf, uinf=ph.uinf, vinf=ph.vinf,
                 bxinf=ph.bxinf, byinf=ph.byinf) for a, b in zip(edges[:-1], edges[1:])]


def test_sensor_of_a_batch_set_after_a_smaller_one():
    m, t, ph, Q = case_periodic(6, 3)
    dt = 0.1 * m.min_edge() / 3

    def sensor(s, n):
        s.set_cases(_records(t.ncell, n, ph, dt))
        s.set_state(Q)
        s.step_cases(2)
        return s.state(sm_ind=True)["sm_ind"]

    s = Solver(t, ph, precision="fp64")
    got = [sensor(s, n) for n in (2, 40, 3)]
    s.close()
    for n, g in zip((2, 40, 3), got):
        s = Solver(t, ph, precision="fp64")
        assert np.array_equal(sensor(s, n), g, equal_nan=True), n
        s.close()


@pytest.mark.parametrize("form", ["fp64_exact", "fp64", "mixed"])
def test_vjp_of_a_state_written_on_the_device(form):
    """The VJP is that of the state now in device memory, neighbours' traces
    included, also where a caller wrote it there."""
    import torch

    m, t, ph, Q = case_cylinder()
    Q2 = np.asfortranarray(Q * (1 + 0.01 * np.random.default_rng(3).uniform(-1, 1, Q.shape[::-1]).T))
    lam = np.asfortranarray(np.random.default_rng(4).standard_normal(Q.shape[::-1]).T)
    s = Solver(t, ph, precision=form)
    s.set_state(Q2, 0.0, 3.0, 1.0)
    want = s.vjp_resid(lam)
    s.set_state(Q, 0.0, 3.0, 1.0)
    owner = type("Q", (), {"__cuda_array_interface__": dict(shape=(Q.size,), typestr="<f8", version=2,
                                                            data=(s.device_state_ptr(), False))})()
    torch.as_tensor(owner, device="cuda").copy_(torch.from_numpy(Q2.ravel(order="K")))
    torch.cuda.synchronize()
    got = s.vjp_resid(lam)
    s.close()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("form", ["fp64_exact", "fp64", "mixed"])
def test_steps_of_a_diverged_mesh(form):
    """Every point faults: each call says so, at no more than a few times the
    cost of a sound one (the exact form's divisions of non-finite values are
    its slow ones), and the next sound call is sound."""
    import time

    m = mesh.periodic_box(64, 64)
    t = host.build_tables(m, 4)
    ph = cases.Physics(dxcycl=m.dxcycl, dycycl=m.dycycl)
    Q = cases.orszag_tang_state(t.xxsolu, 1e-8, 1)
    bad = Q.copy()
    bad[0] = -bad[0]
    dt = 0.1 * cases.cfl_dt(m, Q, 4)
    s = Solver(t, ph, precision=form)

    def run(q, faults):
        best = np.inf
        for _ in range(5):
            s.set_state(q)
            t0 = time.perf_counter()
            if faults:
                with pytest.raises(NumericalFault):
                    s.rk_s5p3(dt, 4)
            else:
                s.rk_s5p3(dt, 4)
            best = min(best, time.perf_counter() - t0)
        return best

    s.set_state(Q)
    s.rk_s5p3(dt, 3)
    sound, diverged, again = run(Q, False), run(bad, True), run(Q, False)
    s.set_state(bad)
    with pytest.raises(NumericalFault):
        s.compresid()
    s.set_state(Q)
    s.compresid()
    s.close()
    # (measured per stage 1.1 to 1.6 times; 100 to 130 with every warp's OR
    # across the host link)
    assert diverged < 10 * max(sound, again), (sound, diverged, again)


@pytest.mark.parametrize("form", ["fp64_exact", "fp64", "mixed"])
def test_steps_of_long_and_short_calls_are_the_same(form):
    """Eager steps, graphs of one step and of several: the same bits and time."""
    m, t, ph, Q = case_channel(9, 7, 4)
    dt = 0.1 * m.min_edge() / 4
    out = []
    for groups in ([1] * 50, [50], [20, 1, 29], [9] * 5 + [5]):
        s = Solver(t, ph, precision=form)
        s.set_state(Q)
        for n in groups:
            s.rk_s5p3(dt, n)
        out.append((s.state()["Q"].copy(), s.maxima()))
        s.close()
    for q, mx in out[1:]:
        assert np.array_equal(q, out[0][0]) and mx == out[0][1]


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("form", ["fp64_exact", "fp64", "mixed"])
@pytest.mark.parametrize("N,sizes", [(2, [(11, 9), (7, 3), (31, 33)]), (3, [(11, 9), (5, 7), (23, 21)]),
                                     (4, [(9, 9), (3, 5), (13, 11)]), (5, [(7, 9), (5, 5), (17, 13)]),
                                     (6, [(7, 5), (3, 3), (9, 11)])])
def test_batch_of_odd_cases_equals_separate_runs(N, sizes, form, persistent):
    """Cases of odd cell counts, so that tiles begin at odd cells: their state
    slices are no whole 16-byte units at odd N.  States, maxima and the
    residual, bit for bit those of each case in its own context."""
    cl = [cases.cylinder_case(a, b, N, ms=0.2 + 0.03 * k, ma=2.0, seed=k, noise=1e-4) for k, (a, b) in enumerate(sizes)]
    members = ensemble.build_members(cl)
    b = ensemble.Batch(members, precision=form, persistent=persistent)
    b.reset()
    b.step(2)
    b.solver.compresid()
    g = b.solver.state(resid=True)
    for k, m in enumerate(members):
        s = Solver(m.tables, m.case.physics, precision=form)
        s.set_state(m.Q0)
        s.rk_s5p3(m.dt, 2)
        s.compresid()
        w, mx = s.state(resid=True), s.maxima()
        s.close()
        assert np.array_equal(b.member_state(g["Q"], k), w["Q"]), k
        assert np.array_equal(b.member_state(g["resid"], k), w["resid"]), k
        assert b.solver.case_maxima(k) == (mx["eigvmax"], mx["umax"]), k
    b.close()


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("form", ["fp64_exact", "fp64"])
@pytest.mark.parametrize("N,count,a,b", [(3, 5, 45, 45), (5, 5, 35, 33), (5, 9, 45, 45), (6, 3, 33, 31)])
def test_batch_over_several_waves_equals_separate_runs(N, count, a, b, form, persistent):
    """More tiles than are resident at once, from odd cells on: the exact form
    by tiles and (N = 3; N = 5 in the larger batch) by lines."""
    members = ensemble.build_members([cases.cylinder_case(a, b, N, ms=0.25, ma=2.0, seed=1, noise=1e-4)] * count)
    one = members[0]
    bt = ensemble.Batch(members, precision=form, persistent=persistent)
    bt.reset()
    bt.step(2)
    g = bt.solver.state()["Q"]
    s = Solver(one.tables, one.case.physics, precision=form)
    s.set_state(one.Q0)
    s.rk_s5p3(one.dt, 2)
    w = s.state()["Q"]
    s.close()
    for k in range(count):
        assert np.array_equal(bt.member_state(g, k), w), k
    bt.close()


@pytest.mark.parametrize("N", [2, 3, 4, 5, 6])
def test_adjoint_of_every_form_is_the_exact_one(N):
    """The adjoint runs the exact form's stages whatever the context's form:
    by the same kernels, from metrics in another layout."""
    m, t, ph, Q = case_cylinder(9, 16, N)
    dt = 0.1 * cases.cfl_dt(m, Q, N)
    out = []
    for form in ("fp64_exact", "fp64", "mixed"):
        s = Solver(t, ph, precision=form)
        s.set_state(Q)
        r = s.adjoint_run(dt, 6, 2, 6, checkpoint_every=3)
        out.append((r["J"], r["Qbar0"], r["parbar"], s.state()["Q"].copy()))
        s.close()
    for r in out[1:]:
        assert r[0] == out[0][0] and all(np.array_equal(x, y) for x, y in zip(r[1:], out[0][1:]))


@pytest.mark.parametrize("N,nx,ny", [(2, 5, 3), (3, 33, 31), (4, 76, 75), (5, 9, 7), (5, 101, 69), (6, 41, 37)])
def test_five_stage_scheme_matches_oracle(N, nx, ny):
    """FiveStageRk on meshes of one wave (one kernel for all its stages) and of
    several (a kernel for each kind; at N = 4 in double without held states)."""
    m, t, ph, Q = case_channel(nx, ny, N)
    dt = 0.1 * m.min_edge() / N
    o = O.Oracle(t, ph)
    o.set_state(Q)
    o.five_stage_rk(dt, 2)
    ref = o.state()["Q"]
    for form, bar in (("fp64_exact", 0.0), ("fp64", 1e-12), ("mixed", 1e-6)):
        s = Solver(t, ph, precision=form, k_stage=5)
        s.set_state(Q)
        s.rk_s5p3(dt, 2)
        g = s.state()["Q"]
        s.close()
        assert np.array_equal(g, ref) if not bar else rel_l2(g, ref) <= bar, form
    s = Solver(t, ph, precision="fp64", k_stage=5)  # one case as a persistent batch
    s.set_cases(_records(t.ncell, 1, ph, dt))
    s.set_persistent(True)
    s.set_state(Q)
    s.step_cases(2)
    assert rel_l2(s.state()["Q"], ref) <= 1e-12
    s.close()


@pytest.mark.parametrize("N,nx,ny", [(2, 9, 7), (2, 141, 139), (3, 9, 7), (3, 97, 95), (5, 61, 59)])
def test_viscous_chain_matches_oracle_on_one_and_several_waves(N, nx, ny):
    """Below and above the CTAs resident at once: launches in order or begun
    early, and at N = 2 and 3 outside the exact form two kernels each."""
    import dataclasses

    m, t, ph, Q = case_channel(nx, ny, N, sides=("WALL", "OUTL", "SYMP", "INLE"))
    ph = dataclasses.replace(ph, mu=0.02, eta0=0.015)
    dt = min(0.02 * m.min_edge() / N, 0.02 * (m.min_edge() / N) ** 2 / ph.mu)
    o = O.Oracle(t, ph)
    o.set_state(Q)
    o.rk_s5p3(dt, 1)
    ref = o.state()["Q"]
    for form, bar in (("fp64_exact", 0.0), ("fp64", 1e-12), ("mixed", 1e-6)):
        s = Solver(t, ph, precision=form)
        s.set_state(Q)
        s.rk_s5p3(dt, 1)
        g = s.state()["Q"]
        s.close()
        assert np.array_equal(g, ref) if not bar else rel_l2(g, ref) <= bar, form
