"""stats()["launches"] against the kernels that a fake CUDA runtime was asked
to launch, on the CPU: every launch of a ray kernel counts, the heads that
waves run on a stream of their own among them."""
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
