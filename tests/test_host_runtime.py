"""The host runtime of the drop-in (csrc/context.cu, adjoint.cu, noalloc.cu,
line_launch.inc) against a stand-in of the CUDA runtime, tests/native/
fake_cudart.cpp: sizes of copies, order of work on streams, attributes of
launches, device memory, failing allocations.  Nothing is computed and no GPU
is used: the library is loaded in a child process in which the stand-in is
its libcudart."""
import os
import shutil
import subprocess
import sys
import textwrap

import pytest

from sddc_b200 import _native

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

pytestmark = pytest.mark.skipif(not os.path.exists(NVCC) or not os.path.exists(_native.GPU_LIB),
                                reason="nvcc or libsddc_b200.so not there (python -m sddc_b200.build)")

PRELUDE = """
import ctypes, sys
sys.path[:0] = [{root!r}, {here!r}]
import numpy as np
from helpers import *
from sddc_b200 import _native
from sddc_b200.solver import AdjointOpts, Params, Solver, SddcError, lib
F = ctypes.CDLL("libcudart.so.12")
F.fake_message.restype = ctypes.c_char_p
for f in ("fake_live", "fake_peak"):
    getattr(F, f).restype = ctypes.c_size_t
F.fake_launches.restype = ctypes.c_long
F.fake_fail_alloc.argtypes = [ctypes.c_long]

def clean():
    assert F.fake_violations() == 0, F.fake_message()

def launches(part):
    return F.fake_launches(part.encode())
"""


@pytest.fixture(scope="module")
def runtime(tmp_path_factory):
    """A directory with the stand-in as libcudart.so.12."""
    d = tmp_path_factory.mktemp("cudart")
    (d / "versions.map").write_text("libcudart.so.12 { global: *; };\n")
    subprocess.run([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC",
                    "-shared", "-cudart", "none", f"-I{os.path.join(ROOT, 'sddc_b200', 'csrc')}",
                    os.path.join(HERE, "native", "fake_cudart.cpp"), os.path.join(HERE, "native", "fake_args.cu"),
                    "-o", str(d / "libcudart.so.12"), "-Xlinker", f"--version-script={d / 'versions.map'}", "-Xlinker",
                    "-soname=libcudart.so.12"], check=True, capture_output=True)
    return str(d)


def _run(runtime, body):
    code = PRELUDE.format(root=ROOT, here=HERE) + textwrap.dedent(body)
    env = dict(os.environ, LD_LIBRARY_PATH=runtime)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env=env, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_sensor_read_after_a_larger_batch_is_set(runtime):
    """The copy of the running maxima that a sensor read takes has the size of
    the batch now set, not of the one at the first read."""
    _run(runtime, """
        m, t, ph, Q = case_periodic(6, 3)

        def set_cases(s, n):
            edges = np.linspace(0, t.ncell, n + 1).astype(int)
            s.set_cases([dict(first_cell=int(a), ncell=int(b - a), dt=1e-3, rinf=1., pinf=1., uinf=.1, vinf=0., bxinf=0.,
                              byinf=0.) for a, b in zip(edges[:-1], edges[1:])])
            s.set_state(Q)
            s.step_cases(2)

        s = Solver(t, ph, precision="fp64")
        s.set_state(Q)
        s.rk_s5p3(1e-3, 1)
        s.state(sm_ind=True)
        for n in (2, 12, 3, 40):
            set_cases(s, n)
            s.state(sm_ind=True)
        clean()
        """)


def test_an_error_of_a_launch_is_reported_once(runtime):
    """A stage launch that failed is its own call's error, not also the next
    call's."""
    _run(runtime, """
        m, t, ph, Q = case_cylinder()
        for kernel, call in ((b"line_kernel", lambda s: s.rk_s5p3(1e-3, 1)), (b"resid_kernel", lambda s: s.compresid())):
            s = Solver(t, ph, precision="fp64")
            s.set_state(Q)
            F.fake_fail(kernel)
            try:
                call(s)
                assert False
            except SddcError as e:
                assert e.code == -2
            F.fake_fail(b"")
            s.set_state(Q)
            call(s)
            s.close()
        clean()
        """)


NOALLOC = """
        import test_zz_no_alloc as Z
        L = Z._bind()
        m, t, ph, Q = case_cylinder()
        met, faces = Z._packed(L, t)

        def device(a):
            p = ctypes.c_void_p()
            assert F.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(a.nbytes)) == 0
            return p

        def stream():
            p = ctypes.c_void_p()
            assert F.cudaStreamCreateWithFlags(ctypes.byref(p), 1) == 0
            return p

        p, ops, out = Z._params(t, ph, 1), [np.asfortranarray(x) for x in (t.Lmat, t.Mmat)], np.zeros(2)
        dev = [device(a) for a in (Q, met, faces, Q, np.zeros(2 * Q.size))]

        def call(st):
            return L.sddc_compresid_noalloc(ctypes.byref(p), *[Z._p(x) for x in ops], *dev[:3], 0.0, 0.0, *dev[3:],
                                            Z._p(out), st)
"""


def test_allocation_free_call_after_a_fault_on_another_stream(runtime):
    """A fault belongs to the call that found it: nothing orders the next
    call's stream after what that one left in its own."""
    _run(runtime, NOALLOC + """
        a, b = stream(), stream()
        for good in (b, a, b):
            F.fake_fault(b"resid_kernel")
            assert call(a) == -4
            F.fake_fault(b"")
            assert call(good) == 0, L.sddc_noalloc_last_error()
        clean()
        """)


def test_allocation_free_call_after_one_that_broke_off(runtime):
    """A call that could not launch its residual leaves no flag behind."""
    _run(runtime, NOALLOC + """
        a, b = stream(), stream()
        F.fake_fault(b"trace_kernel")
        F.fake_fail(b"resid_kernel")
        assert call(a) == -2
        F.fake_fault(b"")
        F.fake_fail(b"")
        assert call(b) == 0, L.sddc_noalloc_last_error()
        clean()
        """)


def test_every_kernel_has_its_attributes_on_every_gpu(runtime):
    """Kernels ask for more shared memory than a device gives without being
    told: on each GPU of a process, in every form and at every N."""
    _run(runtime, """
        for device in (0, 1, 0, 2):
            F.cudaSetDevice(device)
            for N in (2, 3, 4, 5, 6):
                m, t, ph, Q = case_cylinder(3, 8, N)
                big = case_cylinder(24, 32, N)
                for form in ("fp64_exact", "fp64", "mixed"):
                    s = Solver(t, ph, precision=form)
                    s.set_state(Q)
                    s.compresid()
                    s.rk_s5p3(1e-3, 2)
                    s.vjp_resid(Q)
                    s.adjoint_run(1e-3, 2, 1, 2)
                    for k in (False, True):
                        s.set_cases([dict(first_cell=0, ncell=t.ncell, dt=1e-3, rinf=1., pinf=1., uinf=.1, vinf=0.,
                                          bxinf=0., byinf=0.)])
                        s.set_persistent(k)
                        s.set_state(Q)
                        s.step_cases(1)
                    s.close()
                    s = Solver(big[1], big[2], precision=form, k_stage=5)
                    s.set_state(big[3])
                    s.rk_s5p3(1e-3, 1)
                    s.close()
                    ph.mu = 0.01
                    s = Solver(t, ph, precision=form)
                    ph.mu = 0.0
                    s.set_state(Q)
                    s.rk_s5p3(1e-3, 1)
                    s.close()
        clean()
        """)


def test_calls_after_a_failed_allocation(runtime):
    """Whichever allocation of a call fails: the call says so, and what follows
    finds the context as it was or whole, never half of what was to be made."""
    _run(runtime, """
        m, t, ph, Q = case_periodic(6, 3)
        def records(n):
            edges = np.linspace(0, t.ncell, n + 1).astype(int)
            return [dict(first_cell=int(a), ncell=int(b - a), dt=1e-3, rinf=1., pinf=1., uinf=.1, vinf=0., bxinf=0.,
                         byinf=0.) for a, b in zip(edges[:-1], edges[1:])]

        def fails(call, k):
            F.fake_fail_alloc(k)
            try:
                call()
                return False
            except SddcError as e:
                assert e.code == -5, e
                return True
            finally:
                F.fake_fail_alloc(-1)

        # the VJP's work space and the residual's arrays
        for call in (lambda s: s.vjp_resid(Q), lambda s: s.compresid()):
            k = 0
            while True:
                s = Solver(t, ph, precision="fp64")
                s.set_state(Q)
                failed = fails(lambda: call(s), k)
                call(s)
                s.compresid()
                s.state(resid=True, nablaQs=True)
                s.close()
                if not failed:
                    break
                k += 1
            assert k > 1, k
        # a batch: the one that was set, or none, stays in force
        for before in (0, 3):
            for k in range(5):
                s = Solver(t, ph, precision="fp64")
                if before:
                    s.set_cases(records(before))
                s.set_state(Q)
                step = (lambda: s.step_cases(1)) if before else (lambda: s.rk_s5p3(1e-3, 1))
                step()
                assert fails(lambda: s.set_cases(records(20)), k)
                step()
                s.compresid()
                s.monitor()
                s.state(sm_ind=True)
                if before:
                    assert fails(lambda: s.set_persistent(True), k % 2)
                    n = launches("persistent")
                    step()
                    assert launches("persistent") == n
                s.set_cases(records(20))
                s.set_state(Q)
                s.step_cases(1)
                s.monitor()
                s.close()
        clean()
        """)


def test_graphs_are_captured_where_their_steps_pay(runtime):
    """A dt that changes from call to call (an adaptive step) pays for no more
    captures than its steps win back; a constant dt gets its graphs."""
    _run(runtime, """
        m, t, ph, Q = case_cylinder()
        s = Solver(t, ph, precision="fp64")
        s.set_state(Q)

        def graphs(calls):
            a, b = launches("graph instantiation"), launches("graph launch")
            for dt, n in calls:
                s.rk_s5p3(dt, n)
            return launches("graph instantiation") - a, launches("graph launch") - b

        # ten steps with a dt each: the graph of a single step, no longer one
        assert graphs([(1e-3 * (1 + 1e-6 * k), 10) for k in range(1, 6)]) == (5, 45)
        # a dt for two single steps each: none
        assert graphs([(2e-3 * (1 + 1e-6 * (k // 2)), 1) for k in range(10)]) == (0, 0)
        # one dt: a graph after some single steps; the longer one in a long call
        # and, from many calls, after as many steps
        assert graphs([(3e-3, 1)] * 20) == (1, 12)
        assert graphs([(3e-3, 8)]) == (0, 8)
        assert graphs([(3e-3, 8)] * 2) == (1, 2)
        assert graphs([(4e-3, 41)]) == (1, 5)
        clean()
        """)


def test_device_memory_of_an_adjoint_run(runtime):
    """What include/sddc.h says a run holds, and no state more: the checkpoints,
    two stores of stage states and traces, six adjoint registers."""
    _run(runtime, """
        m, t, ph, Q = case_cylinder(8, 16, 4)
        s = Solver(t, ph, precision="fp64_exact")
        s.set_state(Q)
        s.vjp_resid(Q)  # the work space is there
        state, traces, tiles = Q.size * 8, t.ncell * 4 * 36 * 8, t.ncell // 8
        for steps, every, stores in ((4, 4, 1), (4, 2, 2), (6, 2, 2)):
            live = F.fake_live()
            F.fake_reset_peak()
            s.adjoint_run(1e-3, steps, 1, steps, checkpoint_every=every)
            run = F.fake_peak() - live
            assert F.fake_live() == live
            want = (steps // every + 6) * state + stores * ((5 * every + 1) * (state + traces) + 5 * every * 2 * tiles * 8)
            assert want <= run < want + state // 2, (steps, every, run, want)
        clean()
        """)


def test_exact_stages_take_the_kernel_that_the_waves_favour(runtime):
    """148 SMs: sizes at which a sweep put one kernel at least 5% ahead, single
    and in batches (the launches recorded, not run)."""
    _run(runtime, """
        def route(s, step):
            a, b = launches("stage_kernel"), launches("line_kernel")
            step(s)
            a, b = launches("stage_kernel") - a, launches("line_kernel") - b
            assert sorted((a, b)) == [0, 5], (a, b)
            return "tiles" if a else "lines"

        def single(N, nx, ny):
            m = mesh.periodic_box(nx, ny)
            t = host.build_tables(m, N)
            s = Solver(t, channel_physics(), precision="fp64_exact")
            s.set_state(np.ones((9, N, N, t.ncell), order="F"))
            r = route(s, lambda s: s.rk_s5p3(1e-3, 1))
            s.close()
            return r

        def batch(N, nx, ny, count, persistent=False):
            m = mesh.periodic_box(nx, ny * count)
            t = host.build_tables(m, N)
            s = Solver(t, channel_physics(), precision="fp64_exact")
            s.set_cases([dict(first_cell=k * nx * ny, ncell=nx * ny, dt=1e-3, rinf=1., pinf=1., uinf=.1, vinf=0.,
                              bxinf=0., byinf=0.) for k in range(count)])
            s.set_persistent(persistent)
            s.set_state(np.ones((9, N, N, t.ncell), order="F"))
            r = route(s, lambda s: s.step_cases(1))
            s.close()
            return r

        for N, nx, ny, want in ((2, 8, 8, "tiles"), (2, 64, 64, "tiles"), (2, 100, 100, "lines"), (2, 180, 180, "lines"),
                                (3, 8, 8, "tiles"), (3, 67, 67, "tiles"), (3, 74, 74, "lines"), (3, 90, 90, "lines"),
                                (3, 97, 97, "tiles"), (3, 127, 127, "lines"), (4, 8, 8, "tiles"), (4, 67, 67, "tiles"),
                                (4, 80, 80, "lines"), (4, 90, 90, "tiles"), (4, 120, 120, "tiles"), (4, 220, 220, "lines"),
                                (5, 8, 8, "tiles"), (5, 120, 120, "tiles"), (6, 90, 90, "tiles")):
            assert single(N, nx, ny) == want, (N, nx, ny)
        for N, nx, ny, count, want in ((3, 8, 8, 8, "tiles"), (3, 22, 23, 16, "lines"), (4, 8, 8, 8, "tiles"),
                                       (4, 22, 23, 16, "tiles"), (5, 22, 23, 8, "tiles"), (5, 22, 23, 16, "tiles"),
                                       (5, 45, 45, 16, "lines"), (6, 22, 23, 16, "tiles")):
            assert batch(N, nx, ny, count) == want, (N, nx, ny, count)
        assert batch(4, 22, 23, 16, True) == "lines" and batch(4, 8, 8, 8, True) == "tiles"
        clean()
        """)
