"""The integrator's queue of vector operations (csrc/nv_queue.h) on the CPU,
over a stand-in for the CUDA runtime (fake_cudart.cpp) that records and
refuses launches: what a launch hands back is its own request, never a device
word of one before it."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "pihm-cuda_gb300")
LIB = os.path.join(PKG, "lib", "libpihm_gpu.so")

SETUP = f"""
import ctypes, os, sys
sys.path[:0] = [{PKG!r}, {HERE!r}]
import numpy as np
import pihm_gpu.watershed as W
from pihm_gpu import nvector, solver
fake = ctypes.CDLL(os.environ["LD_PRELOAD"])
fake.fake_flushes.restype = ctypes.c_long
VP = ctypes.c_void_p
lib = solver._bind(nvector.load())
t = ctypes.c_double(0.0)

def integrator(y, rhs, user_data, deferred=-1):
    m = lib.pihm_bdf_create()
    assert lib.pihm_bdf_init(m, rhs, 0.0, y) == 0
    assert lib.pihm_bdf_ss_tolerances(m, 1e-4, 1e-4) == 0
    assert lib.pihm_bdf_set_user_data(m, user_data) == 0
    assert lib.pihm_bdf_set_deferred_scalars(m, deferred) == 0
    return m
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(LIB):
        pytest.skip("g++ or the library not found")
    so = str(tmp_path_factory.mktemp("fake") / "libfakecudart.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", os.path.join(PKG, "csrc"), "-I",
                    os.path.join(os.path.dirname(PKG), "include"), os.path.join(HERE, "fake_cudart.cpp"), "-o", so], check=True)
    return so


def _child(fake, code):
    r = subprocess.run([sys.executable, "-c", SETUP + code], env=dict(os.environ, LD_PRELOAD=fake),
                       capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]


def test_no_launch_reads_the_word_of_a_destroyed_context(fake):
    _child(fake, """
from pihm_gpu.single import GpuWatershed
ws = W.generate(60, 4, seed=1)
z = np.zeros(1)

def words():
    out = (ctypes.c_uint64 * 100000)()
    n = fake.fake_words(out, 100000)
    assert 0 < n <= 100000
    return [out[k] for k in range(n)]

a, b = (GpuWatershed(ws, W.relax_state(ws), z, z, z) for _ in range(2))
lib.pihm_gpu_error_word.restype = VP
lib.pihm_gpu_error_word.argtypes = [VP]
word = lib.pihm_gpu_error_word(a.g.h)
fake.fake_reset()
m = integrator(a.y, a.rhs, a.user_data)
lib.pihm_bdf_solve(m, 60.0, a.y, ctypes.byref(t))
assert word in words()
a.close()
fake.fake_reset()
assert lib.pihm_bdf_set_user_data(m, b.user_data) == 0
assert lib.pihm_bdf_init(m, b.rhs, 0.0, b.y) == 0
lib.pihm_bdf_solve(m, 60.0, b.y, ctypes.byref(t))
assert word not in words()
lib.pihm_bdf_free(m)
""")


@pytest.mark.parametrize("deferred", [0, 1])
def test_a_lost_launch_ends_the_call_in_an_error(fake, deferred):
    """Every launch of queued operations whose value nobody waits for, refused
    in turn: the call that lost it returns an error, and the integrator
    initialised again is usable."""
    _child(fake, f"""
RHS = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_double, VP, VP, VP)
cb = RHS(lambda t, y, ydot, ud: 0)
y = lib.N_VNew_PihmGpu(40, None)
m = integrator(y, ctypes.cast(cb, VP), None, {deferred})
solve = lambda: lib.pihm_bdf_solve(m, 1.0, y, ctypes.byref(t))
fake.fake_reset()
assert solve() == 0
flushes = fake.fake_flushes()
assert flushes > 2
for k in range(flushes):
    assert lib.pihm_bdf_init(m, ctypes.cast(cb, VP), 0.0, y) == 0
    fake.fake_reset()
    fake.fake_refuse(k)
    rc = solve()
    assert fake.fake_flushes() > k and rc < 0, (k, rc)
    fake.fake_refuse(-1)
    assert lib.pihm_bdf_init(m, ctypes.cast(cb, VP), 0.0, y) == 0
    assert solve() == 0
lib.pihm_bdf_free(m)
lib.N_VDestroy_PihmGpu(y)
""")
