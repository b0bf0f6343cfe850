"""The stage kernel that works by lines (csrc/line_kernel.cuh) at the edges of
its tiles, and the quotients its exact form takes from one reciprocal."""
import dataclasses
import os
import shutil
import subprocess

import numpy as np
import pytest

import sddc_oracle as O
from helpers import channel_physics, rel_l2, smooth_state
from sddc_b200 import cases, host, mesh
from sddc_b200.solver import Solver
from test_gpu_parity import _sensor_close

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
TILE = {2: 8, 3: 10, 4: 8, 5: 6, 6: 2}  # cells per CTA


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not available")
def test_quotients_round_as_division(tmp_path):
    exe = str(tmp_path / "quotients_check")
    subprocess.run([NVCC, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler",
                    "-ffp-contract=off", f"-I{os.path.join(os.path.dirname(HERE), 'sddc_b200', 'csrc')}",
                    os.path.join(HERE, "native", "quotients_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def _case(N, ncell):
    """A jittered channel with a boundary of another kind on each side."""
    m = mesh.channel_box(ncell, 1, sides=("WALL", "OUTL", "FREE", "INLE"), jitter=0.0, seed=N)
    if ncell % 2 == 0:
        m = mesh.channel_box(ncell // 2, 2, sides=("SYMP", "OUTL", "WALL", "INLE"), jitter=0.2, seed=N)
    t = host.build_tables(m, N)
    ph = channel_physics()
    return t, ph, smooth_state(t, ph, seed=ncell), 0.2 * m.min_edge() / N


def _by_lines(t, ph, dt, form, **kw):
    """A context whose stages run by lines in every form: a batch of one case."""
    s = Solver(t, ph, precision=form, **kw)
    s.set_cases([dict(first_cell=0, ncell=t.ncell, dt=dt, rinf=ph.rinf, pinf=ph.pinf, uinf=ph.uinf, vinf=ph.vinf,
                      bxinf=ph.bxinf, byinf=ph.byinf)])
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("N", sorted(TILE))
@pytest.mark.parametrize("k_stage", [3, 5])
def test_lines_match_oracle_at_tile_edges(N, k_stage):
    for ncell in sorted({1, 2, TILE[N] - 1, TILE[N], TILE[N] + 1, 3 * TILE[N] + 1}):
        if ncell < 1:
            continue
        t, ph, Q, dt = _case(N, ncell)
        o = O.Oracle(t, ph)
        o.set_state(Q)
        (o.rk_s5p3 if k_stage == 3 else o.five_stage_rk)(dt, 2)
        ref = o.state()["Q"]
        mo = o.maxima()
        # the bars of the parity tests: exact bit for bit, FP64 1e-12, mixed 1e-6
        for form, bar in (("fp64_exact", 0.0), ("fp64", 1e-12), ("mixed", 1e-6)):
            s = _by_lines(t, ph, dt, form, k_stage=k_stage)
            s.set_state(Q)
            s.step_cases(2)
            g = s.state()["Q"]
            if bar:
                assert rel_l2(g, ref) <= bar, (form, ncell)
            else:
                assert np.array_equal(g, ref), ncell
                assert s.case_maxima(0) == (mo["eigvmax"], mo["umax"])
            s.close()
            s = Solver(t, ph, precision=form, k_stage=k_stage)
            s.set_state(Q)
            s.rk_s5p3(dt, 2)
            assert np.array_equal(s.state()["Q"], g), (form, ncell)
            s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("N", sorted(TILE))
def test_viscous_lines_match_oracle_at_tile_edges(N):
    for ncell in sorted({1, 2, TILE[N] + 1, 2 * TILE[N]}):
        t, ph, Q, dt = _case(N, ncell)
        ph = dataclasses.replace(ph, mu=0.02, eta0=0.015)
        o = O.Oracle(t, ph)
        o.set_state(Q)
        o.rk_s5p3(0.2 * dt, 1)
        ref = o.state()["Q"]
        for form, bar in (("fp64_exact", 0.0), ("fp64", 1e-12), ("mixed", 1e-6)):
            s = Solver(t, ph, precision=form)
            s.set_state(Q)
            s.rk_s5p3(0.2 * dt, 1)
            g = s.state()["Q"]
            assert np.array_equal(g, ref) if not bar else rel_l2(g, ref) <= bar, (form, ncell)
            s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("N,nx,ny,mu", [(4, 76, 75, 0.0), (4, 64, 75, 0.02), (4, 64, 65, 0.0), (5, 101, 69, 0.0), (6, 37, 41, 0.0),
                                        (6, 15, 7, 0.0)])
def test_stages_match_oracle_over_several_waves(N, nx, ny, mu):
    """More tiles than CTAs are resident: at N = 4 in double 713 tiles take the
    kernel of three warps per scheduler, 520 the other one (the exact form by
    tiles).  The exact form runs by tiles of 6 cells at N = 5, at N = 6 of 8, and of
    6 on the smallest meshes."""
    m = mesh.channel_box(nx, ny, sides=("SYMP", "OUTL", "WALL", "INLE"), jitter=0.2, seed=N)
    t = host.build_tables(m, N)
    ph = channel_physics()
    ph = dataclasses.replace(ph, mu=mu, eta0=mu)
    Q, dt = smooth_state(t, ph, seed=nx), 0.2 * m.min_edge() / N * (0.2 if mu else 1.0)
    o = O.Oracle(t, ph)
    o.set_state(Q)
    o.rk_s5p3(dt, 1)
    ref = o.state()["Q"]
    for form, bar in (("fp64_exact", 0.0), ("fp64", 1e-12), ("mixed", 1e-6)):
        s = Solver(t, ph, precision=form)
        s.set_state(Q)
        s.rk_s5p3(dt, 1)
        g = s.state()["Q"]
        assert np.array_equal(g, ref) if not bar else rel_l2(g, ref) <= bar, form
        s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("N", sorted(TILE))
def test_vjp_lines_match_tangent_at_tile_edges(N):
    """<Qbar, V> = <Rbar, R'(Q) V>, the bar of the VJP tests (1e-11)."""
    for ncell in sorted({1, 2, TILE[N] - 1, TILE[N] + 1, 2 * TILE[N]}):
        t, ph, Q, _ = _case(N, ncell)
        rng = np.random.default_rng(ncell)
        lam, V = rng.standard_normal(Q.shape), rng.standard_normal(Q.shape)
        s = Solver(t, ph, precision="fp64_exact")
        s.set_state(Q, 0.0, 3.0, 1.0)
        Qbar, _ = s.vjp_resid(lam)
        s.close()
        T = O.Oracle(t, ph, tangent=True)
        T.set_state(Q + 1e-30j * V, 0.0, 3.0, 1.0)
        T.compresid()
        jv = T.state()["resid"].imag / 1e-30
        a, b = float(np.vdot(lam, jv)), float(np.vdot(Qbar, V))
        assert abs(a - b) <= 1e-11 * np.vdot(np.abs(lam), np.abs(jv)), (ncell, a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("N", [2, 3, 5, 6])
def test_reverse_steps_in_any_grouping_are_the_same(N):
    """A checkpoint at every step (each segment's first reverse stage takes its
    adjoint traces from the trace launch) and none (all from the VJP's end)."""
    c = cases.cylinder_case(5, 11, N, ms=0.5, noise=1e-3)
    t = host.build_tables(c.mesh, N)
    Q = c.initial_state(t)
    dt = cases.cfl_dt(c.mesh, Q, N)
    out = []
    for every in (1, 100):
        s = Solver(t, c.physics, precision="fp64_exact")
        s.set_state(Q)
        r = s.adjoint_run(dt, 4, 2, 4, checkpoint_every=every)
        out.append((r["J"], r["Qbar0"], r["parbar"], s.state()["Q"].copy()))
        s.rk_s5p3(dt, 1)  # the context goes on from the final state
        out[-1] += (s.state()["Q"].copy(),)
        s.close()
    assert out[0][0] == out[1][0] and all(np.array_equal(a, b) for a, b in zip(out[0][1:], out[1][1:]))
    s = Solver(t, c.physics, precision="fp64_exact")
    s.set_state(Q)
    s.rk_s5p3(dt, 5)
    assert np.array_equal(s.state()["Q"], out[0][4])
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["fp64_exact", "fp64", "mixed"])
def test_steps_in_any_grouping_are_the_same(form):
    """Single steps (eager, then a graph), a graph of several steps, and a dt
    that changes in between: the same states, maxima and time."""
    t, ph, Q, dt = _case(4, 40)
    out = []
    for groups in ([1] * 23, [23], [2, 11, 1, 9]):
        s = Solver(t, ph, precision=form)
        s.set_state(Q)
        for n in groups:
            s.rk_s5p3(dt, n)
        s.rk_s5p3(0.5 * dt, 1)
        s.rk_s5p3(0.5 * dt, 2)
        s.rk_s5p3(dt, 1)
        out.append((s.state()["Q"].copy(), s.maxima(), s.monitor()["mass"]))
        s.close()
    for q, mx, mass in out[1:]:
        assert np.array_equal(q, out[0][0]) and mx == out[0][1] and mass == out[0][2]


@pytest.mark.gpu
@pytest.mark.parametrize("N", [3, 5])
def test_both_exact_kernels_agree_with_zeros_and_fault(N):
    """A state with zero components (their quotients keep the zero), and the
    step at which the configured Mach number faults: by lines and by tiles
    the same bits."""
    c = cases.cylinder_case(8, 16, N, ms=1.5, ma=2.0, noise=0.0)
    t = host.build_tables(c.mesh, N)
    Q = c.initial_state(t)
    dt = cases.cfl_dt(c.mesh, Q, N)
    out = []
    for lines in (False, True):
        s = _by_lines(t, c.physics, dt, "fp64_exact") if lines else Solver(t, c.physics, precision="fp64_exact")
        s.set_state(Q)
        seen = []
        for _ in range(12):
            try:
                s.step_cases(1) if lines else s.rk_s5p3(dt, 1)
                fault = False
            except RuntimeError:
                fault = True
            seen.append((fault, s.state()["Q"].copy()))
        s.close()
        out.append(seen)
    for (fa, qa), (fb, qb) in zip(*out):
        assert fa == fb and np.array_equal(qa, qb, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("N", sorted(TILE))
def test_residual_lines_match_oracle_at_tile_edges(N):
    """The residual, all gradients and the sensor; two evaluations in a row, so
    that the second has c_h > 0."""
    for ncell in sorted({1, 2, TILE[N] - 1, TILE[N], TILE[N] + 1, 3 * TILE[N] + 1}):
        if ncell < 1:
            continue
        t, ph, Q, _ = _case(N, ncell)
        o = O.Oracle(t, ph)
        o.set_state(Q)
        o.compresid()
        o.compresid()
        ref, mo = o.state(), o.maxima()
        # the flux's rounding enters the residual magnified by |M| |F| / (J |resid|),
        # up to about 3e3 on these meshes: 3e3 eps (1.1e-16 and 6e-8)
        for form, bar in (("fp64_exact", 0.0), ("fp64", 4e-13), ("mixed", 2e-4)):
            s = Solver(t, ph, precision=form)
            s.set_state(Q)
            s.compresid()
            s.compresid()
            g = s.state(resid=True, nablaQs=True, sm_ind=True)
            if not bar:
                _sensor_close(g["sm_ind"], ref["sm_ind"])
            for k in ("resid", "nablaQs"):
                if bar:
                    assert rel_l2(g[k], ref[k]) <= bar, (form, ncell, k)
                else:
                    assert np.array_equal(g[k], ref[k]), (ncell, k)
            if not bar:
                mg = s.maxima()
                assert (mg["eigvmax"], mg["umax"]) == (mo["eigvmax"], mo["umax"])
            s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("N,nx,ny", [(5, 9, 7), (5, 100, 115), (4, 9, 7), (3, 31, 1)])
def test_caller_held_memory_at_any_eight_byte_address(N, nx, ny, form):
    """Arrays that no 16-byte copy can move (and, at 100x115 cells, traces packed
    into the scratch array) give the bits that aligned ones give."""
    import ctypes

    import torch
    import test_zz_no_alloc as Z

    torch.cuda.init()
    L = Z._bind()
    m = mesh.channel_box(nx, ny, sides=("WALL", "OUTL", "FREE", "INLE"), seed=N)
    t = host.build_tables(m, N)
    ph = channel_physics()
    Q = smooth_state(t, ph, seed=nx)
    met, faces = Z._packed(L, t)
    p, ops = Z._params(t, ph, form), [np.asfortranarray(x) for x in (t.Lmat, t.Mmat)]
    got = []
    for shift in (0, 1):
        def at(a):  # a copy on the device, `shift` doubles past an allocation's start
            d = torch.empty(a.size + shift, dtype=torch.float64, device="cuda")
            d[shift:] = torch.from_numpy(np.ravel(a, order="K"))
            return d[shift:]
        q, met_d, res, grad = at(Q), at(met), at(np.zeros(Q.size)), at(np.zeros(2 * Q.size))
        faces_d = torch.from_numpy(faces).cuda()
        out = np.zeros(2)
        torch.cuda.synchronize()
        rc = L.sddc_compresid_noalloc(ctypes.byref(p), *[Z._p(x) for x in ops], q.data_ptr(), met_d.data_ptr(),
                                      faces_d.data_ptr(), 3.0, 1.0, res.data_ptr(), grad.data_ptr(), Z._p(out), None)
        assert rc == 0, L.sddc_noalloc_last_error()
        got.append((res.cpu().numpy(), grad.cpu().numpy(), out))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    s = Solver(t, ph, precision=form)
    s.set_state(Q, 0.0, 3.0, 1.0)
    s.compresid()
    st = s.state(resid=True, nablaQs=True)
    s.close()
    for a, k in zip(got[0], ("resid", "nablaQs")):
        assert np.array_equal(a, np.ravel(st[k], order="K"))
