"""The library's host code on the CPU: its own objects, linked against a CUDA
runtime without a device (fake_cudart.c).  A test is a script run in a
process of its own, as the package loads one library per process; it finds
``ip`` (the package), ``np``, ``C`` (ctypes), ``L`` (the loaded library with
the runtime's fake_* controls) and the helpers below in scope.
"""
import os
import subprocess
import sys

from ipole_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = """
import ctypes as C
import numpy as np
import ipole_b200 as ip
L = ip.lib()
L.fake_log.restype = C.c_char_p
L.fake_inflight.argtypes = [C.c_void_p]

def grid(n1, n2, n3):
    g = ip.Grid()
    g.n1, g.n2, g.n3 = n1, n2, n3
    return g

def fields(g):
    return [np.ones((g.n1 + 2) * (g.n2 + 2) * (g.n3 + 2)) for _ in range(10)]

def camera(**kw):
    c = ip.Camera()
    c.nx = c.ny = 64
    c.maxnstep, c.emission_type, c.target_nturns, c.eps = 100, 4, -1, 0.01
    for k, v in kw.items():
        setattr(c, k, v)
    return c

def code(f, *a):
    try:
        f(*a)
    except ip.IpgError as e:
        return e.code
    return 0

def kernels():
    return L.fake_log().decode().split()
"""

# an adjoint of more rays than one launch gives eight lanes each
ADJOINT = """
g = grid(2, 2, 2)
ij = np.zeros((6000, 2), np.int32)
c.upload_arrays(g, fields(g))
def call():
    return code(c.adjoint, camera(), ij, np.zeros((len(ij), 4)), 64)
"""
# a level of a batch: one camera, n geodesics with two instances each
BATCH = """
g = grid(2, 2, 2)
prims = (C.POINTER(C.c_double) * 9)(*[f.ctypes.data_as(C.POINTER(C.c_double)) for f in (fields(g) * 2)[:9]])
cam, el, slot = camera(), (C.c_double * 8)(), (C.c_int * 2)(0, 0)
class Items(C.Structure):
    _fields_ = [("n_geo", C.c_size_t), ("geo_ij", C.c_void_p), ("geo_grp", C.c_void_p), ("geo_mask", C.c_void_p),
                ("n_xf", C.c_size_t), ("xf_geo", C.c_void_p), ("xf_slot", C.c_void_p), ("xf_out", C.c_void_p),
                ("xf_order", C.c_void_p), ("geo_order", C.c_void_p), ("n_long", C.c_size_t),
                ("long_steps", C.c_double), ("pred_steps", C.c_double)]
buf = np.zeros(1 << 20, np.int32)
def call(n=6000):
    it = Items(n, *[buf.ctypes.data] * 3, 2 * n, *[buf.ctypes.data] * 5, 0, 0., 0.)
    return L.ipg__batch_trace(c._h, C.byref(it), None)
def begin():
    assert L.ipg_upload_iharm_batch(c._h, C.byref(g), prims, C.c_double(4 / 3), C.c_double(4 / 3),
                                    C.c_double(5 / 3)) == 0
    assert L.ipg__batch_begin(c._h, C.byref(cam), 1, slot, 2, el, 1, 0) == 0
begin()
"""


def library(tmp):
    """Builds the library over the fake runtime into the folder tmp."""
    build.build()
    src = os.path.join(HERE, "fake_cudart.c")
    obj, lib = os.path.join(tmp, "fake_cudart.o"), os.path.join(tmp, "libipole_fake.so")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc())))
    objs = [os.path.join(build.BUILD, f[:f.rindex(".")] + ".o")
            for f in ["ipg_kernels.cu", *build.CU_EXTRA, *build.HOST_SRC]]
    subprocess.run(["gcc", "-w", "-O1", "-fPIC", "-I", os.path.join(cuda, "include"), "-c", src, "-o", obj], check=True)
    subprocess.run(["g++", "-shared", "-fopenmp", "-o", lib, obj, *objs, "-lz", "-lm", "-Wl,-z,defs"], check=True)
    return lib


def run(lib, script):
    env = dict(os.environ, IPOLE_B200_LIB=lib, PYTHONPATH=os.path.dirname(HERE))
    r = subprocess.run([sys.executable, "-c", PRELUDE + script], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
