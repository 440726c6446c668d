"""Failing CUDA calls in the library's host code, on the CPU over a fake CUDA
runtime: what a call leaves behind when one of its steps fails."""
import pytest

from tests import fake_cuda
from tests.fake_cuda import ADJOINT, BATCH


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_cuda.library(str(tmp_path_factory.mktemp("fake")))


@pytest.mark.parametrize("fn", ["cudaMalloc", "cudaMemcpyAsync"])
@pytest.mark.parametrize("nth", [1, 2])
def test_failed_upload_leaves_no_model(lib, fn, nth):
    """A second upload, of a smaller dump, that fails: the next trace either
    has the first dump whole or is refused; never the first dump's grid over
    an array of the second's size."""
    fake_cuda.run(lib, f"""
for first in (grid(8, 8, 8), None):
    with ip.Context(0, 8 << 20) as c:
        if first is not None:
            c.upload_arrays(first, fields(first))
        small = grid(2, 2, 2)
        L.fake_reset()
        L.fake_fail(b"{fn}", {nth})
        rc = code(c.upload_arrays, small, fields(small))
        L.fake_reset()
        if rc == 0:
            continue # fewer calls than that
        ij = np.zeros((1, 2), np.int32)
        assert code(c.trace, camera(), ij) == ip.IPG_E_STATE, (first, rc)
        c.upload_arrays(small, fields(small)) # and the context goes on
        assert code(c.trace, camera(), ij) == 0
""")


@pytest.mark.parametrize("fn,nth", [("cudaMemcpyAsync", 3), ("cudaMemcpy", 1)])
def test_failed_batch_upload_leaves_no_model(lib, fn, nth):
    """the same for a batch's primitives"""
    fake_cuda.run(lib, f"""
g = grid(4, 4, 4)
prims = (C.POINTER(C.c_double) * 9)(*[f.ctypes.data_as(C.POINTER(C.c_double)) for f in (fields(g) * 2)[:9]])
up = lambda: L.ipg_upload_iharm_batch(c._h, C.byref(g), prims, C.c_double(4 / 3), C.c_double(4 / 3), C.c_double(5 / 3))
cam, el, slot = camera(), (C.c_double * 8)(), (C.c_int * 1)(0)
begin = lambda: L.ipg__batch_begin(c._h, C.byref(cam), 1, slot, 1, el, 1, 0)
with ip.Context(0, 8 << 20) as c:
    assert up() == 0 and begin() == 0
    L.fake_reset()
    L.fake_fail(b"{fn}", {nth})
    assert up() != 0
    L.fake_reset()
    assert begin() == ip.IPG_E_STATE
    assert up() == 0 and begin() == 0
""")


@pytest.mark.parametrize("call", ["c.upload_arrays(big, fields(big))", "c.trace(camera(), np.zeros((9, 2), np.int32))",
                                  "c.thermal_coefficients(np.ones((7, 5)))"])
def test_recovers_after_out_of_memory(lib, call):
    """a call that finds no memory fails by itself: the next upload, trace and
    fits, which have what they need, are not refused for it"""
    fake_cuda.run(lib, f"""
with ip.Context(0, 8 << 20) as c:
    g, big = grid(2, 2, 2), grid(3, 3, 3)
    c.upload_arrays(g, fields(g))
    def failing():
        {call}
    L.fake_fail(b"cudaMalloc", 1)
    assert code(failing) == ip.IPG_E_CUDA
    assert code(c.upload_arrays, g, fields(g)) == 0
    assert code(c.trace, camera(), np.zeros((9, 2), np.int32)) == 0
    assert code(c.thermal_coefficients, np.ones((7, 5))) == 0
""")


@pytest.mark.parametrize("call", ["c.upload_arrays(g, fields(g))",
                                  "c.thermal_coefficients(np.ones(((1 << 18) + 9, 5)))"])
@pytest.mark.parametrize("fn", ["cudaGetLastError", "cudaMemcpyAsync"])
def test_failed_call_waits_for_its_copies(lib, call, fn):
    """a call that fails between its copies returns after the ones in flight,
    which use the caller's arrays, are done"""
    fake_cuda.run(lib, f"""
with ip.Context(0, 8 << 20) as c:
    g = grid(2, 2, 2)
    def failing():
        {call}
    failing()
    L.fake_reset()
    L.fake_fail(b"{fn}", 2)
    assert code(failing) == ip.IPG_E_CUDA
    assert L.fake_inflight(None) == 0
""")


@pytest.mark.parametrize("what", [ADJOINT, BATCH], ids=["adjoint", "batch"])
@pytest.mark.parametrize("fn", ["cudaGetLastError", "cudaEventRecord", "cudaStreamWaitEvent", "cudaFuncSetAttribute"])
def test_failed_wave_leaves_no_second_stream_running(lib, what, fn):
    """The heads of the adjoint's and the batches' waves run on a stream of
    their own.  Wherever a wave fails, what that stream still does to the pool
    and the result must be over when the call returns: the next call is
    ordered after the context's stream only."""
    fake_cuda.run(lib, f"""
c = ip.Context(0, 8 << 20)
{what}
assert call() == 0
forked = 0
for nth in range(1, 200):
    L.fake_reset()
    L.fake_fail(b"{fn}", nth)
    rc = call()
    forked += any("coop" in k for k in kernels())
    assert L.fake_inflight(c.stream()) == 0, nth
    if rc == 0:
        break
assert nth > 1 and forked > 0
""")
