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
