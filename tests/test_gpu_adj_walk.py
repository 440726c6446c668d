"""The adjoint walk's lanes per ray (k_adj_walk: 32, 16, 8 or 4 by the number
of rays, as k_walk).

The loss is linear in the pixels, so the gradient of a list is the sum of the
gradients of its parts, which the parts' sizes make other launches walk: the
counts straddle the edges at which the lanes change and leave partly filled
warps and blocks of records.  The two differ by the order in which a cell's
contributions are added only.
"""
import numpy as np
import pytest

import ipole_b200 as ip
from tests import common

pytestmark = pytest.mark.gpu

RESIDENT = 148 * 8


@pytest.mark.parametrize("extra", [[], ["--target_nturns=1"]], ids=["all", "subring"])
@pytest.mark.parametrize("n", [2, RESIDENT + 1, 2 * RESIDENT + 1, 4 * RESIDENT + 3])
def test_gradient_is_the_sum_of_its_parts(n, extra, dumps):
    meta, _ = common.load_golden("c1_bright_32")
    args = [f"--dump={dumps.get(meta)}", "--freqcgs=230e9", "--thetacam=163", "--rotcam=20", "--MBH=6.5e9",
            "--dsource=16.8e6", "--fov=160", "--M_unit=3e27", "--trat_small=1", "--trat_large=20", "--nx=160",
            "--ny=160", *extra]
    p = ip.Params.from_args(args)
    m = ip.Model.load(p)
    cam = ip.camera_for(p, m.grid)
    r = np.random.default_rng(n)
    at = r.choice(160 * 160, size=n, replace=False)
    ij = np.stack([at // 160, at % 160], axis=1).astype(np.int32)
    dL = r.standard_normal((n, 4))
    ncell = m.field(0).size
    with ip.Context(0, 12 << 30) as c:
        c.upload(m)
        whole, out = c.adjoint(cam, ij, dL, ncell)
        parts = [np.zeros(ncell) for _ in whole]
        for lo in range(0, n, max(1, RESIDENT // 2)):
            s = slice(lo, min(n, lo + max(1, RESIDENT // 2)))
            g, o = c.adjoint(cam, ij[s], dL[s], ncell)
            assert o.tobytes() == out[s].tobytes()
            parts = [a + np.ravel(b) for a, b in zip(parts, g)]
    for a, b in zip(parts, whole):
        b = np.ravel(b)
        assert np.isfinite(b).all()
        # (pixels with no emission in the sub-ring have no gradient)
        assert (b != 0).any() == any((out[k] != 0).any() for k in "IQUV")
        # a cell adds at most ~1e5 contributions of at most the largest
        # gradient's size: their rounding stays far below 1e-10 of it
        assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
