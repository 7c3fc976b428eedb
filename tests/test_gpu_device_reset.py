"""cudaDeviceReset as an ordinary event of a driver (the reference's main.cu calls
it at its end): the library's addresses of the old context are not used in the
new one.  Each case is a process of its own, as the reset ends what every other
user of the device in the process holds."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import ctypes as C, glob, os, sys
import numpy as np
import nvidia.cuda_runtime as rt
from multicomponent_color_gradient_b200 import Solver, _lib, derive
cudart = C.CDLL(glob.glob(os.path.join(list(rt.__path__)[0], "lib", "libcudart.so.*"))[0])
def call(name, *args):
    rc = getattr(cudart, name)(*args)
    assert rc == 0, (name, rc)
def case(n=30):
    return derive(dict(NX=n, NY=20, NZ=18, bubble_radius=5.0, tau=0.7, sigma=0.01, beta_recolor=0.7,
                       boundary="periodic", NSTATS_START_STEP=10 ** 9))
"""


def run(body):
    env = dict(os.environ, PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", PRELUDE + body], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr


def test_static_sums_after_a_reset():
    """mcg_conservation_sums_static looks its scratch up again: the context after
    the reset has the pointer of the one before, but another id."""
    run("""
def sums():
    with Solver(case()) as S:
        S.init_bubble()
        S.step(3)
        want = S.conservation_sums()
        pops = S.get_populations()
    bufs = []
    for a in (*pops, np.zeros(5)):
        p = C.c_void_p()
        call("cudaMalloc", C.byref(p), C.c_size_t(a.nbytes))
        call("cudaMemcpy", p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1)
        bufs.append(p)
    lib = _lib.load()
    assert lib.mcg_conservation_sums_static(bufs[0], bufs[1], 30, 20, 18, bufs[2], None) == 0
    got = np.zeros(5)
    call("cudaMemcpy", got.ctypes.data_as(C.c_void_p), bufs[2], C.c_size_t(40), 2)
    np.testing.assert_allclose(got, want, rtol=1e-12, atol=1e-9)
sums()
# another place for the library's module in the next context
for _ in range(2):
    call("cudaDeviceReset")
    p = C.c_void_p()
    call("cudaMalloc", C.byref(p), C.c_size_t(64 << 20))
    sums()
""")


def test_adjoint_runs_and_late_close_after_a_reset():
    """A handle that is open at the reset leaves nothing to the next one: runs of
    the new context take new memory, and the old handle's close, though late,
    frees nothing of it."""
    run("""
def start(n=30):
    S = Solver(case(n))
    S.init_bubble()
    return S
target = np.linspace(-1, 1, 30 * 20 * 18).astype(np.float32)
old = start()
want = old.adjoint_run(target, 8, 3, tape=4)
call("cudaDeviceReset")
new = start()
got = new.adjoint_run(target, 8, 3, tape=4)
np.testing.assert_array_equal(got["dJ_du0"], want["dJ_du0"])
new.step(2)
fields = new.get_fields()
with start() as S:
    S.step(2)
    plain = S.get_fields()
new.close()
new = start()
old.close()
new.step(2)
after = new.get_fields()
for k in plain:
    np.testing.assert_array_equal(fields[k], plain[k])
    np.testing.assert_array_equal(after[k], plain[k])
np.testing.assert_allclose(got["J"], want["J"], rtol=1e-9)
new.close()
""")
