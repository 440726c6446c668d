"""What calls launch, on the CPU: the kernels that a fake CUDA runtime was
asked for."""
import pytest

from tests import fake_cuda
from tests.fake_cuda import ADJOINT, BATCH

TRACE = """
g = grid(2, 2, 2)
c.upload_arrays(g, fields(g))
def call(n=6000):
    return code(c.trace, camera(), np.zeros((n, 2), np.int32))
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_cuda.library(str(tmp_path_factory.mktemp("fake")))


@pytest.mark.parametrize("what,call,least", [(TRACE, "call()", 5), (TRACE, "call(100)", 3), (ADJOINT, "call()", 13),
                                             (BATCH, "call()", 5), (BATCH, "call(100)", 3), (BATCH, "call(70000)", 5)],
                         ids=["trace", "trace100", "adjoint", "batch", "batch100", "batch70000"])
def test_launches_are_counted(lib, what, call, least):
    """stats()["launches"]: every launch of a ray kernel counts, the heads that
    waves run on a stream of their own among them"""
    fake_cuda.run(lib, f"""
c = ip.Context(0, 8 << 20)
{what}
L.fake_reset()
assert {call} == 0
rays = [k for k in kernels() if any(n in k for n in ("k_geodesic", "k_len_", "k_coef", "k_walk", "k_transfer",
                                                     "k_xfer_batch", "k_adj_"))]
assert len(rays) >= {least}, rays
assert c.stats()["launches"] == len(rays), (c.stats()["launches"], rays)
""")


def test_batch_launches_do_not_depend_on_earlier_calls(lib):
    """a large batch after two small ones of the same shape, and after two of
    its own size, launches what it launches first of all, however long the
    earlier calls' kernels took"""
    fake_cuda.run(lib, f"""
ms = [1.]
times = C.CFUNCTYPE(C.c_float)(lambda: ms[0])
L.fake_elapsed(times)
seen = set()
for sizes in ([70000], [100, 100, 70000], [70000, 70000, 70000]):
    for order in (1, -1): # the later call the slower one, or the faster
        c = ip.Context(0, 8 << 20)
        {BATCH.replace(chr(10), chr(10) + "        ")}
        for k, n in enumerate(sizes):
            if k:
                begin()
            ms[0] = 10. * 2. ** (order * k)
            L.fake_reset()
            assert call(n) == 0
        seen.add(tuple(kernels()))
        c.close()
assert len(seen) == 1, seen
""")


@pytest.mark.parametrize("side,large", [(270, False), (290, True), (300, True), (320, False), (345, False), (370, False),
                                        (400, True)])
def test_longest_class_of_large_images(lib, side, large):
    """3.45% of the rays 3 times the mean long or longer and 0.4% 5 times, as in
    images of the synthetic dumps: the longest class starts at 2.5 times the
    mean where that holds at most 22 rays per SM or more than 34 (148 SMs),
    else, and in smaller images, at 4 times"""
    fake_cuda.run(lib, f"""
n = {side} ** 2
geo = []
def kernel(name, args):
    at = lambda k, t: C.cast(args[k], C.POINTER(t))[0]
    if b"k_len_hist" in name:
        hist = C.cast(at(3, C.c_void_p), C.POINTER(C.c_int))
        hist[40], hist[24], hist[7] = int(.004 * n), int(.0305 * n), n - int(.004 * n) - int(.0305 * n)
    elif b"k_geodesic" in name and b"count" not in name:
        geo.append(at(2, C.c_int))
cb = C.CFUNCTYPE(None, C.c_char_p, C.POINTER(C.c_void_p))(kernel)
L.fake_on_launch(cb)
c = ip.Context(0, 8 << 30)
g = grid(2, 2, 2)
c.upload_arrays(g, fields(g))
assert code(c.trace, camera(nx={side}, ny={side}), np.zeros((n, 2), np.int32)) == 0
assert sum(geo) == n and geo[0] == int(.004 * n) + ({large} and int(.0305 * n)), geo
""")
