"""The work a user has this framework do, as cases that can be timed one by one.

Kinds (the ``kind`` of a case), each through the package's public calls:

* ``step``      time steps of a context whose state stays on the GPU
                (``Solver.rk_s5p3``), as the reference's time loop issues them;
* ``start``     a short run from a state on the host: ``set_state``, then steps;
* ``batch``     steps of an ensemble of cylinder cases in one context;
* ``residual``  one residual evaluation with all gradients into the caller's
                device memory (``sddc_compresid_noalloc`` of the C ABI);
* ``vjp``       the transposed Jacobian of the residual times a vector;
* ``adjoint``   drag of a run from a host state with its gradient by the
                discrete adjoint (``DragLiftProblem.run``).

Flows: ``cylinder`` is the O-grid of the configured cases (walls, inflow and
outflow), ``vortex`` the periodic Orszag-Tang case, ``wave`` an advected
density wave in a periodic box (smooth, so it can be stepped for any time).
"""
import ctypes
import functools
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from sddc_b200 import adjoint, cases, ensemble, host, mesh
from sddc_b200.solver import PRECISIONS, Params, Solver, lib

GAMMA = 5.0 / 3.0


def listed():
    return [
        # the smallest call: one step per call, nothing but launches and latency
        dict(name="wave_24x24_n4_mixed", kind="step", flow="wave", nx=24, ny=24, N=4, form="mixed", k=3, steps=1,
             tile=0, visc=0.0),
        # an odd little mesh at p = 2 with the other Runge-Kutta scheme
        dict(name="wave_47x33_n3_fp64_rk5", kind="step", flow="wave", nx=47, ny=33, N=3, form="fp64", k=5, steps=1,
             tile=0, visc=0.0),
        # the reference's own case from its initial state: the first 100 of its 500 steps
        dict(name="cylinder_32x64_n4_fp64", kind="start", flow="cylinder", nx=32, ny=64, N=4, form="fp64", k=3,
             steps=100, tile=0, visc=0.0),
        # p = 5 in the bit-exact form, a mesh that no tile divides
        dict(name="wave_121x87_n6_exact", kind="step", flow="wave", nx=121, ny=87, N=6, form="fp64_exact", k=3,
             steps=2, tile=0, visc=0.0),
        # viscous and resistive flow: two more kernels before every stage
        dict(name="vortex_128x128_n4_fp64_visc", kind="step", flow="vortex", nx=128, ny=128, N=4, form="fp64", k=3,
             steps=2, tile=0, visc=1e-3),
        # the benchmark's cylinder (p = 4, 3.3 million points) with the tile its tuner picks, mixed and FP64
        dict(name="cylinder_256x512_n5_mixed", kind="step", flow="cylinder", nx=256, ny=512, N=5, form="mixed", k=3,
             steps=2, tile=6, visc=0.0),
        dict(name="cylinder_256x512_n5_fp64", kind="step", flow="cylinder", nx=256, ny=512, N=5, form="fp64", k=3,
             steps=2, tile=6, visc=0.0),
        # Orszag-Tang, p = 3, with the default tile: the largest
        dict(name="vortex_512x512_n4_mixed", kind="step", flow="vortex", nx=512, ny=512, N=4, form="mixed", k=3,
             steps=2, tile=0, visc=0.0),
        # a parameter study: cases of uneven size in one context
        dict(name="batch_24_n4_mixed", kind="batch", count=24, N=4, form="mixed", steps=2, tile=6),
        # one residual for a caller that owns all device memory
        dict(name="residual_90x90_n5_fp64", kind="residual", flow="wave", nx=90, ny=90, N=5, form="fp64"),
        # backward: one vector through the residual, and a whole run with its gradient
        dict(name="vjp_64x128_n4", kind="vjp", flow="cylinder", nx=64, ny=128, N=4),
        dict(name="adjoint_64x128_n4", kind="adjoint", flow="cylinder", nx=64, ny=128, N=4, steps=40, every=20),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["start", "start", "batch", "residual", "vjp", "adjoint"])
    N = rng.choice([2, 3, 4, 4, 5, 5, 6])
    form = rng.choice(["mixed", "mixed", "fp64", "fp64_exact"])
    if kind == "step":
        flow = rng.choice(["wave", "wave", "vortex"])
        nx = _spread(rng, 8, 400)
        ny = max(8, min(400, int(round(nx * rng.uniform(0.5, 2.0)))))
        if flow == "vortex":  # large enough that the steps timed end before its shocks form
            nx, ny = max(nx, 300), max(ny, 300)
        return dict(kind=kind, flow=flow, nx=nx, ny=ny, N=N if flow == "wave" else 4, form=form,
                    k=rng.choice([3, 3, 3, 5]), steps=rng.choice([1, 2, 4]), tile=rng.choice([0, 0, 4, 6, 8, 16]),
                    visc=1e-3 if form != "mixed" and nx * ny < 20000 and rng.random() < 0.3 else 0.0)
    nr = _spread(rng, 12, 80)
    nt = max(20, int(round(nr * rng.uniform(1.5, 2.5))))
    if kind == "start":
        return dict(kind=kind, flow="cylinder", nx=nr, ny=nt, N=N, form=form, k=rng.choice([3, 3, 5]),
                    steps=rng.randint(1, 60), tile=rng.choice([0, 0, 4, 6, 8, 16]), visc=rng.choice([0.0, 0.0, 1e-3]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 24), N=rng.choice([3, 4, 4, 5]), form=form,
                    steps=rng.choice([1, 2, 4]), tile=rng.choice([0, 4, 6, 8]))
    if kind == "residual":
        nx = _spread(rng, 10, 90)
        return dict(kind=kind, flow="wave", nx=nx, ny=max(8, min(90, int(round(nx * rng.uniform(0.5, 1.5))))), N=N,
                    form=form)
    if kind == "vjp":
        return dict(kind=kind, flow="cylinder", nx=nr, ny=nt, N=N)
    return dict(kind=kind, flow="cylinder", nx=nr, ny=nt, N=rng.choice([3, 4, 4, 5]), steps=rng.randint(6, 40),
                every=rng.choice([5, 10, 20]))


# ---- inputs ----------------------------------------------------------------------


def _wave(xx, m, seed):
    """A density wave carried by a uniform magnetised flow, with seeded phases and noise."""
    rng = np.random.default_rng(seed)
    x, y = xx[0] * (2 * np.pi / m.dxcycl), xx[1] * (2 * np.pi / m.dycycl)
    rho = 1.0 + 0.05 * np.sin(x + rng.uniform(0, 6)) * np.cos(y + rng.uniform(0, 6))
    Q = np.asfortranarray(cases.conserved(rho, 0.8, 0.4, 0.1, 1.0, 0.3, 0.2, 0.1, 0.0))
    Q += rng.uniform(-1e-6, 1e-6, size=Q.shape[::-1]).T
    return Q


def _setup(case, seed):
    """(mesh tables, physics, initial state on the host, time step)."""
    nx, ny, N = case["nx"], case["ny"], case["N"]
    if case["flow"] == "cylinder":
        c = cases.cylinder_case(nx, ny, N, ms=0.5, ma=2.0, seed=seed)
        m, ph = c.mesh, c.physics
        t = host.build_tables(m, N)
        Q = c.initial_state(t)
    else:
        m = mesh.periodic_box(nx, ny)
        ph = cases.Physics(dxcycl=m.dxcycl, dycycl=m.dycycl)
        t = host.build_tables(m, N)
        Q = _wave(t.xxsolu, m, seed) if case["flow"] == "wave" else cases.orszag_tang_state(t.xxsolu, 1e-8, seed)
    ph.mu = ph.eta0 = case.get("visc", 0.0)
    dt = cases.cfl_dt(m, Q, N)
    if ph.mu:  # the diffusive limit, when it is the smaller one
        dt = min(dt, 0.02 * (m.min_edge() / N) ** 2 / ph.mu)
    return t, ph, Q, dt


class _DeviceArray:
    """A device pointer of the library for torch (no copy); the tensor keeps its owner alive."""

    def __init__(self, owner, address, n):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(address, False), version=2)


def _state_tensor(st, s):
    """The context's state (9,N,N,NCELL), variable fastest, where it lies on the GPU."""
    p = s.device_state_ptr()
    if st.get("ptr") != p:
        st["ptr"], st["view"] = p, torch.as_tensor(_DeviceArray(s, p, 9 * s.N * s.N * s.ncell), device="cuda")
    return st["view"]


def _batch_members(case, seed):
    """The ensemble's sizes belong to the case, its noise to the seed."""
    cs = ensemble.make_cases(case["count"], seed=case["count"], N=case["N"])
    for k, c in enumerate(cs):
        c.seed = seed * 1000 + k
    return ensemble.build_members(cs)


def _d(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _i(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))


def _noalloc(t, ph, form):
    """The C entry point with its packed tables on the GPU."""
    PD, PI, I, V, D = (ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int), ctypes.c_int, ctypes.c_void_p,
                       ctypes.c_double)
    L = lib()
    L.sddc_noalloc_pack_tables.argtypes = [I, I, PD, PD, PD, PI, I] + [PI, I] * 7 + [PD, PI]
    L.sddc_noalloc_packed_sizes.argtypes = [I, I] + [ctypes.POINTER(ctypes.c_size_t)] * 2
    L.sddc_compresid_noalloc.argtypes = [ctypes.POINTER(Params), PD, PD, V, V, V, D, D, V, V, PD, V]
    L.sddc_noalloc_last_error.restype = ctypes.c_char_p
    nm, nf = ctypes.c_size_t(), ctypes.c_size_t()
    L.sddc_noalloc_packed_sizes(t.N, t.ncell, ctypes.byref(nm), ctypes.byref(nf))
    met, faces = np.zeros(nm.value), np.zeros(nf.value, np.int32)
    args, keep = [], []
    for a in (t.ibfinter, t.ibfinl, t.ibfout, t.ibfwal, t.ibfsymp, t.ibfree, t.cyc2fpair):
        a = np.asfortranarray(a, dtype=np.int32)
        keep.append(a)
        args += [_i(a), len(a)]
    if L.sddc_noalloc_pack_tables(t.N, t.ncell, _d(t.S1), _d(t.S2), _d(t.Jac), _i(t.IF2C), t.nface, *args, _d(met),
                                  _i(faces)):
        raise RuntimeError(L.sddc_noalloc_last_error().decode())
    p = Params(N=t.N, ncell=t.ncell, ncellglob=t.ncell, vismode=ph.vismode, artiv=ph.artiv, k_stage=3,
               precision=PRECISIONS[form], dxcycl=ph.dxcycl, dycycl=ph.dycycl, rinf=ph.rinf, pinf=ph.pinf,
               uinf=ph.uinf, vinf=ph.vinf, bxinf=ph.bxinf, byinf=ph.byinf)
    return L, p, torch.from_numpy(met).cuda(), torch.from_numpy(faces).cuda()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = ensemble.Batch(_batch_members(case, seed), precision=case["form"], cells_per_cta=case["tile"])
        b.reset()
        return dict(kind=kind, batch=b, steps=case["steps"])
    t, ph, Q, dt = _setup(case, seed)
    st = dict(kind=kind, Q=Q, dt=dt, steps=case.get("steps", 0))
    if kind == "adjoint":
        n = case["steps"]
        st["problem"] = adjoint.DragLiftProblem(t, dt, n, n // 2, n, checkpoint_every=case["every"])
        st["fs"] = [getattr(ph, f) for f in adjoint.FREESTREAM]
        st["problem"].solver(st["fs"])
        return st
    if kind == "residual":
        L, p, met, faces = _noalloc(t, ph, case["form"])
        q = torch.from_numpy(Q.ravel(order="K")).cuda()
        st.update(L=L, p=p, met=met, faces=faces, q=q, resid=torch.empty_like(q), grad=q.new_empty(2 * q.numel()),
                  ops=(np.asfortranarray(t.Lmat), np.asfortranarray(t.Mmat)), out=np.zeros(2))
        return st
    s = Solver(t, ph, precision=case.get("form", "fp64_exact"), k_stage=case.get("k", 3),
               cells_per_cta=case.get("tile", 0))
    s.set_state(Q)
    st["solver"] = s
    if kind == "vjp":
        s.compresid()  # the state's own running maxima, so that c_h > 0
        st["Rbar"] = _weights(Q.shape, seed)
    return st


def _weights(shape, seed):
    return np.asfortranarray(np.random.default_rng(seed + 77).standard_normal(shape[::-1]).T)


def run(state):
    kind = state["kind"]
    if kind == "step":
        s = state["solver"]
        s.rk_s5p3(state["dt"], state["steps"])
        return _state_tensor(state, s)
    if kind == "start":
        s = state["solver"]
        s.set_state(state["Q"])
        s.rk_s5p3(state["dt"], state["steps"])
        return _state_tensor(state, s)
    if kind == "batch":
        b = state["batch"]
        b.step(state["steps"])
        return _state_tensor(state, b.solver)
    if kind == "vjp":
        qbar, par = state["solver"].vjp_resid(state["Rbar"])
        return dict(Qbar=qbar, parbar=par)
    if kind == "adjoint":
        r = state["problem"].run(state["Q"], state["fs"])
        return dict(J=r["J"], Qbar0=r["Qbar0"], parbar=r["parbar"])
    L, (Lm, Mm), out = state["L"], state["ops"], state["out"]
    rc = L.sddc_compresid_noalloc(ctypes.byref(state["p"]), _d(Lm), _d(Mm), state["q"].data_ptr(),
                                  state["met"].data_ptr(), state["faces"].data_ptr(), 3.0, 1.0,
                                  state["resid"].data_ptr(), state["grad"].data_ptr(), _d(out),
                                  torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(L.sddc_noalloc_last_error().decode())
    return dict(resid=state["resid"], nablaQs=state["grad"], maxima=out)


# ---- bytes and operations --------------------------------------------------------
# Per solution point and Runge-Kutta stage: 1406 operations at N = 4 and 1570
# at N = 5 (the reference's own arithmetic, counted), so about 1406 + 164 (N-4).


def _ops(N):
    return 1406.0 + 164.0 * (N - 4)


def _stage_bytes(N):
    """State in and out, Jac, and the four normal components at 2N(N+1) flux points, per solution point."""
    return 2 * 72.0 + 8.0 + 32.0 * (N + 1) / N


def work(case):
    N = case["N"]
    if case["kind"] == "batch":
        cells = sum(c.mesh.ncell for c in ensemble.make_cases(case["count"], seed=case["count"], N=N))
    else:
        cells = case["nx"] * case["ny"]
    dof = cells * N * N
    kind = case["kind"]
    if kind in ("step", "start", "batch"):
        n = 5 * case["steps"]
        # three of RK_S5P3's five stages read a register beside the state; the other scheme's read five in all
        byte = dof * n * (_stage_bytes(N) + (43.2 if case.get("k", 3) == 3 else 72.0))
        flops = dof * n * _ops(N)
        if case.get("visc"):
            flops += dof * n * 1500.0
        if kind == "start":
            byte += dof * 72.0
        return dict(bytes=byte, flops=flops)
    if kind == "residual":
        return dict(bytes=dof * (_stage_bytes(N) + 2 * 72.0), flops=dof * _ops(N))
    if kind == "vjp":
        return dict(bytes=dof * (_stage_bytes(N) + 72.0), flops=dof * 3.0 * _ops(N))
    n = 5 * case["steps"]
    # forward, recomputation and reverse sweep (about twice a residual's operations)
    return dict(bytes=dof * n * (2 * (_stage_bytes(N) + 43.2) + _stage_bytes(N) + 144.0), flops=dof * n * 4.0 * _ops(N))


# ---- the same in 64 bits, in torch -------------------------------------------------


class _Residual:
    """The spectral-difference residual of ideal or viscous GLM-MHD in torch (float64).

    Arrays: Q (cells, j, i, 9); flux points of the xi lines (cells, j, r, 9),
    of the eta lines (cells, i, r, 9); face points (cells, local face, point, 9).
    """

    def __init__(self, t, ph):
        N = self.N = t.N
        g = lambda a, ty=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=ty, device="cuda")  # noqa: E731
        self.L, self.M = g(t.Lmat), g(t.Mmat)
        self.nx = g(t.S1[0].transpose(3, 2, 1, 0))  # (c, j, r, 2)
        self.ny = g(t.S2[1].transpose(3, 1, 2, 0))  # (c, i, r, 2)
        self.J = g(t.Jac.transpose(2, 1, 0))[..., None]  # (c, j, i, 1)
        self.fs = [float(getattr(ph, f)) for f in ("rinf", "pinf", "uinf", "vinf", "bxinf", "byinf")]
        self.mu, self.eta0, self.vis = ph.mu, ph.eta0, ph.vismode
        F = t.IF2C.astype(np.int64)
        a, p1, p2 = F[t.ibfinter - 1], F[t.cyc2fpair[:, 0] - 1], F[t.cyc2fpair[:, 1] - 1]
        q = np.concatenate([np.stack([a[:, 0], a[:, 2], a[:, 1], a[:, 3]], 1),
                            np.stack([p1[:, 0], p1[:, 2], p2[:, 0], p2[:, 2]], 1)]) - 1
        self.pair = [g(q[:, k], torch.int64) for k in range(4)]
        self.bnd = {n: [g(F[f - 1, k] - 1, torch.int64) for k in (0, 2)]
                    for n, f in (("inl", t.ibfinl), ("out", t.ibfout), ("wal", t.ibfwal)) if len(f)}
        if len(t.ibfsymp) or len(t.ibfree):
            raise NotImplementedError
        self.lo = torch.tensor([-1.0, 1.0, 1.0, -1.0], dtype=torch.float64, device="cuda")  # end of the line a face is

    @staticmethod
    def faces(x, y):
        """Values at the flux points -> at the face points (c, 4, point, ...)."""
        return torch.stack([y[:, :, 0], x[:, :, -1], y[:, :, -1].flip(1), x[:, :, 0].flip(1)], 1)

    @staticmethod
    def ends(x, y, f):
        """Flux-point values with the faces' values f at the ends of the lines."""
        x = torch.cat([f[:, 3].flip(1)[:, :, None], x[:, :, 1:-1], f[:, 1][:, :, None]], 2)
        y = torch.cat([f[:, 0][:, :, None], y[:, :, 1:-1], f[:, 2].flip(1)[:, :, None]], 2)
        return x, y

    def lines(self, Q):
        return torch.einsum("cjik,ri->cjrk", Q, self.L), torch.einsum("cjik,rj->cirk", Q, self.L)

    def div(self, x, y):
        return torch.einsum("cjrk,ri->cjik", x, self.M) + torch.einsum("cirk,rj->cjik", y, self.M)

    @staticmethod
    def pressure(q):
        k = (q[..., 1] ** 2 + q[..., 2] ** 2 + q[..., 3] ** 2) / q[..., 0]
        b = q[..., 5] ** 2 + q[..., 6] ** 2 + q[..., 7] ** 2
        return (GAMMA - 1) * (q[..., 4] - 0.5 * k - 0.5 * b - 0.5 * q[..., 8] ** 2), b

    def flux(self, q, n, ch):
        """F n0 + G n1 of the ideal GLM system."""
        p, b2 = self.pressure(q)
        n0, n1 = n[..., 0], n[..., 1]
        u, v, w = q[..., 1] / q[..., 0], q[..., 2] / q[..., 0], q[..., 3] / q[..., 0]
        Bx, By, Bz, psi = q[..., 5], q[..., 6], q[..., 7], q[..., 8]
        un, bn, pt = u * n0 + v * n1, Bx * n0 + By * n1, p + 0.5 * b2
        f = [q[..., 0] * un, q[..., 1] * un + pt * n0 - Bx * bn, q[..., 2] * un + pt * n1 - By * bn,
             q[..., 3] * un - Bz * bn,
             un * (q[..., 4] - 0.5 * psi ** 2 + pt) - (u * Bx + v * By + w * Bz - ch * psi) * bn,
             Bx * un - u * bn + ch * psi * n0, By * un - v * bn + ch * psi * n1, Bz * un - w * bn, ch * bn]
        return torch.stack(f, -1), torch.stack([u, v, w], -1)

    def rusanov(self, ql, qr, n, sign, ch):
        """The left cell's face flux, the wave speeds and the averaged velocities."""
        mag = torch.sqrt((n ** 2).sum(-1))
        un = n / mag[..., None] * sign[..., None]
        fl, vl = self.flux(ql, un, ch)
        fr, vr = self.flux(qr, un, ch)
        B = 0.5 * (ql[..., 5:8] + qr[..., 5:8])
        r2 = 0.5 * (ql[..., 0] + qr[..., 0])
        ca = 0.5 * GAMMA * (self.pressure(ql)[0] + self.pressure(qr)[0]) / r2
        cd = (B ** 2).sum(-1) / r2
        cn = (B[..., 0] * un[..., 0] + B[..., 1] * un[..., 1]) ** 2 / r2
        cf = torch.sqrt(0.5 * (ca + cd + torch.sqrt((ca + cd) ** 2 - 4 * ca * cn)))
        va = 0.5 * (vl + vr)
        eig = (va[..., 0] * un[..., 0] + va[..., 1] * un[..., 1]).abs() + cf
        f = 0.5 * (fl + fr - eig[..., None] * (qr - ql))
        return f * (mag * sign)[..., None], eig, va.abs()

    def ghost(self, name, q, fs):
        rinf, pinf, uinf, vinf, bx, by = fs
        if name == "wal":  # no slip, the field reversed (vismode = 1)
            return q * q.new_tensor([1, -1, -1, -1, 1, -1, -1, -1, 1])
        z = torch.zeros_like(q[..., 0])
        if name == "inl":
            r, u, v, psi = z + rinf, z + uinf, z + vinf, q[..., 8]
        else:
            r, u, v, psi = q[..., 0], q[..., 1] / q[..., 0], q[..., 2] / q[..., 0], z
        e = pinf / (GAMMA - 1) + 0.5 * r * (u * u + v * v) + 0.5 * (bx * bx + by * by) + 0.5 * q[..., 8] ** 2
        return torch.stack([r, r * u, r * v, z, e, z + bx, z + by, z, psi], -1)

    def __call__(self, Q, ch, fs=None, grads=False):
        """(residual, largest wave speed, largest velocity[, gradients (c,j,i,2,9)], traces)."""
        fs = self.fs if fs is None else fs
        x, y = self.lines(Q)
        T, nf = self.faces(x, y), self.faces(self.nx, self.ny)
        Fx, vx = self.flux(x, self.nx, ch)
        Fy, vy = self.flux(y, self.ny, ch)
        cl, ll, cr, lr = self.pair
        ql, qr = T[cl, ll], T[cr, lr].flip(1)
        sl = self.lo[ll][:, None].expand(-1, self.N)
        f, e, va = self.rusanov(ql, qr, nf[cl, ll], sl, ch)
        sr = -self.lo[lr]
        slots = [(cl, ll, f, 0.5 * (ql + qr)), (cr, lr, (f * (sl * sr[:, None])[..., None]).flip(1),
                                                (0.5 * (ql + qr)).flip(1))]
        eig, um = [e.amax()], [va.amax(), vx[:, :, 1:-1].abs().amax(), vy[:, :, 1:-1].abs().amax()]
        for name, (c, lf) in self.bnd.items():
            q = T[c, lf]
            gh = self.ghost(name, q, fs)
            f, e, va = self.rusanov(q, gh, nf[c, lf], self.lo[lf][:, None].expand(-1, self.N), ch)
            slots.append((c, lf, f, 0.5 * (q + gh)))
            eig.append(e.amax())
            um.append(va.amax())
        ix = (torch.cat([s[0] for s in slots]), torch.cat([s[1] for s in slots]))
        FT = torch.zeros_like(T).index_put(ix, torch.cat([s[2] for s in slots]))
        VT = torch.zeros_like(T).index_put(ix, torch.cat([s[3] for s in slots]))
        Fx, Fy = self.ends(Fx, Fy, FT)
        R = -self.div(Fx, Fy)
        Vx, Vy = self.ends(x, y, VT)
        k = slice(None) if grads or self.mu else slice(5, 7)
        G = torch.stack([self.div(Vx[..., k] * self.nx[..., d:d + 1], Vy[..., k] * self.ny[..., d:d + 1]) / self.J
                         for d in (0, 1)], 3)
        divB = (G[..., 0, 0] + G[..., 1, 1] if k.start == 5 else G[..., 0, 5] + G[..., 1, 6])[..., None]
        if self.mu:
            R = R + self.div(*self.viscous(G, Vx, Vy))
        U = Q[..., 1:4] / Q[..., :1]
        B = Q[..., 5:8]
        src = torch.cat([torch.zeros_like(divB), B, (U * B).sum(-1, keepdim=True), U, torch.zeros_like(divB)], -1)
        damp = torch.zeros_like(Q)
        damp[..., 8] = 2.0
        R = R / self.J - divB * src - damp * Q
        return R, torch.stack(eig).amax(), torch.stack(um).amax(), G, T

    def viscous(self, G, Vx, Vy):
        """The viscous flux along the normals at the flux points (periodic meshes)."""
        G = G.flatten(-2)  # (c, j, i, 18)
        x, y = self.lines(G)
        T = self.faces(x, y)
        cl, ll, cr, lr = self.pair
        a = 0.5 * (T[cl, ll] + T[cr, lr].flip(1))
        x, y = self.ends(x, y, T.index_put((torch.cat([cl, cr]), torch.cat([ll, lr])), torch.cat([a, a.flip(1)])))
        return [self.vflux(q, g, n) for q, g, n in ((Vx, x, self.nx), (Vy, y, self.ny))]

    def vflux(self, q, g, n):
        rho, U, B, psi = q[..., :1], q[..., 1:4] / q[..., :1], q[..., 5:8], q[..., 8:9]
        U2 = (U ** 2).sum(-1, keepdim=True)
        inte = (q[..., 4:5] - 0.5 * U2 * rho - 0.5 * (B ** 2).sum(-1, keepdim=True) - 0.5 * psi ** 2) / rho
        D = []
        for d in (g[..., :9], g[..., 9:]):
            dr = d[..., :1]
            dU = (d[..., 1:4] - dr * U) / rho
            de = (d[..., 4:5] - 0.5 * U2 * dr - rho * (U * dU).sum(-1, keepdim=True)
                  - (B * d[..., 5:8]).sum(-1, keepdim=True) - dr * inte - psi * d[..., 8:9]) / rho
            D.append((dU, de[..., 0], d[..., 5:8]))
        (Ux, ex, Bx), (Uy, ey, By) = D
        mu, eta = self.mu, self.eta0
        tr = -2.0 / 3.0 * (Ux[..., 0] + Uy[..., 1])
        sh = mu * (Ux[..., 1] + Uy[..., 0])
        u, v, w = U[..., 0], U[..., 1], U[..., 2]
        z = torch.zeros_like(u)
        Jx, Jy, Jz = By[..., 2], -Bx[..., 2], Bx[..., 1] - By[..., 0]
        f1, f3, g2, g3 = mu * (2 * Ux[..., 0] + tr), mu * Ux[..., 2], mu * (2 * Uy[..., 1] + tr), mu * Uy[..., 2]
        kt = mu * GAMMA / 0.72
        F = [z, f1, sh, f3, u * f1 + v * sh + w * f3 + kt * ex + eta * (Jz * B[..., 1] - Jy * B[..., 2]), z, eta * Jz,
             -eta * Jy, z]
        Gf = [z, sh, g2, g3, sh * u + g2 * v + g3 * w + kt * ey + eta * (Jx * B[..., 2] - Jz * B[..., 0]), -eta * Jz,
              z, eta * Jx, z]
        return torch.stack(F, -1) * n[..., :1] + torch.stack(Gf, -1) * n[..., 1:]


def _ch(Lm, Um):
    s = Lm * (Lm - Um)
    return torch.where(s > 0, torch.sqrt(torch.where(s > 0, s, torch.ones_like(s))), torch.zeros_like(s))


_S3 = dict(a30=0.355909775063327, a32=0.644090224936674, a40=0.367933791638137, a43=0.632066208361863,
           a52=0.237593836598569, a54=0.762406163401431, b=(0.377268915331368, 0.377268915331368, 0.242995220537396,
                                                            0.238458932846290, 0.287632146308408))


def _step(res, Q0, Lm, Um, dt, k=3, fs=None):
    """One time step; the running maxima grow from stage to stage."""

    def rate(Q, Lm, Um):
        R, e, u, _, _ = res(Q, _ch(Lm, Um), fs)
        return R, torch.maximum(Lm, e), torch.maximum(Um, u)

    if k == 3:
        c, b = _S3, _S3["b"]
        R, Lm, Um = rate(Q0, Lm, Um)
        Q1 = Q0 + b[0] * dt * R
        R, Lm, Um = rate(Q1, Lm, Um)
        Q2 = Q1 + b[1] * dt * R
        R, Lm, Um = rate(Q2, Lm, Um)
        Q3 = c["a30"] * Q0 + c["a32"] * Q2 + b[2] * dt * R
        R, Lm, Um = rate(Q3, Lm, Um)
        Q4 = c["a40"] * Q0 + c["a43"] * Q3 + b[3] * dt * R
        R, Lm, Um = rate(Q4, Lm, Um)
        return c["a52"] * Q2 + c["a54"] * Q4 + b[4] * dt * R, Lm, Um
    R, Lm, Um = rate(Q0, Lm, Um)
    Q1 = Q0 + 0.39175222700392 * dt * R
    R, Lm, Um = rate(Q1, Lm, Um)
    Q2 = 0.44437049406734 * Q0 + 0.55562950593266 * Q1 + 0.36841059262959 * dt * R
    R, Lm, Um = rate(Q2, Lm, Um)
    Q3 = 0.6201018513854 * Q0 + 0.3798981486146 * Q2 + 0.25189177424738 * dt * R
    R3, Lm, Um = rate(Q3, Lm, Um)
    Q4 = 0.17807995410773 * Q0 + 0.82192004589227 * Q3 + 0.54497475021237 * dt * R3
    R, Lm, Um = rate(Q4, Lm, Um)
    return (0.00683325884039 * Q0 + 0.51723167208978 * Q2 + 0.12759831133288 * Q3 + 0.34833675773694 * Q4
            + 0.08460416338212 * dt * R3 + 0.22600748319395 * dt * R), Lm, Um


def _cells(Q):
    return torch.from_numpy(np.ascontiguousarray(Q.transpose(3, 2, 1, 0))).cuda()


def _host_layout(x):
    """(c, j, i, 9) -> a (9, i, j, c) array as the C ABI returns it."""
    return x.cpu().numpy().transpose(3, 2, 1, 0)


def _march(t, ph, Q, dt, n, k):
    res, q = _Residual(t, ph), _cells(Q)
    Lm = Um = q.new_zeros(())
    for _ in range(n):
        q, Lm, Um = _step(res, q, Lm, Um, dt, k)
    return q.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for m in _batch_members(case, seed):
            out.append(_march(m.tables, m.case.physics, m.Q0, m.dt, case["steps"], 3))
        return torch.cat(out)
    t, ph, Q, dt = _setup(case, seed)
    if case.get("visc") and case["flow"] == "cylinder":
        return None  # the reference's adiabatic-wall gradients are not restated here
    if kind in ("step", "start"):
        with torch.no_grad():
            return _march(t, ph, Q, dt, case["steps"], case["k"])
    res, q = _Residual(t, ph), _cells(Q)
    if kind == "residual":
        with torch.no_grad():
            R, e, u, G, _ = res(q, _ch(q.new_tensor(3.0), q.new_tensor(1.0)), grads=True)
        mx = np.array([max(3.0, e.item()), max(1.0, u.item())])
        return dict(resid=R.reshape(-1), nablaQs=G.reshape(-1), maxima=mx)
    fs = q.new_tensor(res.fs).requires_grad_()
    if kind == "vjp":
        with torch.no_grad():
            _, e, u, _, _ = res(q, q.new_zeros(()))
        ch = _ch(e, u).requires_grad_()
        q.requires_grad_()
        R = res(q, ch, fs)[0]
        gq, gc, gf = torch.autograd.grad(R, (q, ch, fs), _cells(_weights(Q.shape, seed)))
        return dict(Qbar=_host_layout(gq), parbar=torch.cat([gc[None], gf]).cpu().numpy())
    return _exact_adjoint(case, t, ph, res, q, dt, fs)


def _exact_adjoint(case, t, ph, res, q, dt, fs):
    N, n = case["N"], case["steps"]
    w = np.linalg.solve(np.vander(t.Xs, N, increasing=True).T, 1.0 / np.arange(1, N + 1))
    c, lf = res.bnd["wal"]
    # the weights at the face points: local faces 1 and 2 follow their lines, 3 and 4 run against them
    wf = torch.from_numpy(np.stack([w, w, w[::-1], w[::-1]])).cuda()[lf]
    norm = 2.0 / (ph.rinf * (ph.uinf ** 2 + ph.vinf ** 2))
    direction = np.array([ph.uinf, ph.vinf]) / math.hypot(ph.uinf, ph.vinf)

    def drag(Q):
        tr = _Residual.faces(*res.lines(Q))[c, lf]
        sign = res.lo[lf][:, None].expand(-1, N)
        f = res.rusanov(tr, res.ghost("wal", tr, fs), _Residual.faces(res.nx, res.ny)[c, lf], sign, 0.0)[0]
        F = (f[..., 1:3] * (wf * sign)[..., None]).sum((0, 1))
        return norm * (F[0] * direction[0] + F[1] * direction[1])

    step = functools.partial(_step, res, dt=dt, fs=fs)
    q.requires_grad_()
    x, Lm, Um, J = q, q.new_zeros(()), q.new_zeros(()), 0.0
    for m in range(n + 1):
        if m >= n // 2:
            J = J + drag(x) / (n - n // 2 + 1)
        if m < n:
            x, Lm, Um = checkpoint(step, x, Lm, Um, use_reentrant=False)
    gq, gf = torch.autograd.grad(J, (q, fs))
    return dict(J=float(J), Qbar0=_host_layout(gq), parbar=gf.cpu().numpy())
