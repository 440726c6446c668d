"""The geodesic with eight lanes per ray (k_geodesic_coop, launches of up to
32 rays per SM) against the geodesic with one lane per ray (k_geodesic,
larger launches; IPG_NO_SPLIT keeps them in one launch).

The finite-difference connection amplifies every rounding, so the eight-lane
form must leave the same records: every output of a pixel traced in a small
list must be the bits of the same pixel traced in a large one.  The counts
are the smallest, a partly filled warp, and both sides of the largest launch
that takes eight lanes.
"""
import numpy as np
import pytest

import ipole_b200 as ip
from tests import common

pytestmark = pytest.mark.gpu

COOP_MAX = 148 * 32


@pytest.mark.parametrize("extra", [[], ["-unpol"], ["--target_nturns=1"], ["--thetacam=17", "--rotcam=30"],
                                   ["--maxnstep=800"]],
                         ids=["pol", "unpol", "subring", "incl17", "maxnstep"])
@pytest.mark.parametrize("rec", [ip.IPG_RECORDS_FP64, ip.IPG_RECORDS_MIXED])
def test_geodesic_bit_identical(extra, rec, dumps, monkeypatch):
    monkeypatch.setenv("IPG_NO_SPLIT", "1")
    meta, _ = common.load_golden("c1_bright_32")
    args = [f"--dump={dumps.get(meta)}", "--freqcgs=230e9", "--thetacam=163", "--phicam=0", "--MBH=6.5e9",
            "--dsource=16.8e6", "--fov=160", "--M_unit=3e27", "--trat_small=1", "--trat_large=20", "--nx=120",
            "--ny=120", *extra]
    p = ip.Params.from_args(args)
    m = ip.Model.load(p)
    cam = ip.camera_for(p, m.grid)
    ij = np.array([(i, j) for i in range(120) for j in range(120)], np.int32)
    with ip.Context(0, 12 << 30) as c:
        c.upload(m)
        c.set_record_precision(rec)
        ref = c.trace(cam, ij, allow_maxnstep=True)
        for n in (1, 3, 33, COOP_MAX, COOP_MAX + 1):
            at = np.random.default_rng(n).choice(len(ij), size=n, replace=False)
            got = c.trace(cam, ij[at], allow_maxnstep=True)
            assert got.tobytes() == ref[at].tobytes(), (extra, rec, n)


def test_geodesic_waves_bit_identical(dumps):
    """a pool too small for the list: rays deferred at their first and at
    later chunks"""
    meta, _ = common.load_golden("c1_bright_32")
    p = common.params_for(meta, dumps.get(meta))
    m = ip.Model.load(p)
    out = []
    for pool in (0, 64 << 20):
        with ip.Context(0, pool) as c:
            c.upload(m)
            out.append(c.render(p, m))
            waves = c.stats()["waves"]
    assert waves > 1
    assert out[0].pol.tobytes() == out[1].pol.tobytes() and np.array_equal(out[0].nstep, out[1].nstep)


@pytest.mark.parametrize("extra", [[], ["-unpol"], ["--target_nturns=1"]], ids=["pol", "unpol", "subring"])
@pytest.mark.parametrize("rec", [ip.IPG_RECORDS_FP64, ip.IPG_RECORDS_MIXED])
@pytest.mark.parametrize("n", [68, 70])
def test_batch_wave_head_bit_identical(n, extra, rec, dumps):
    """a batch's wave: all rays with eight lanes (68 x 68 items), or its
    longest rays beside the others with one (70 x 70)"""
    meta, _ = common.load_golden("c1_bright_32")
    args = [f"--dump={dumps.get(meta)}", "--freqcgs=230e9", "--thetacam=163", "--phicam=0", "--MBH=6.5e9",
            "--dsource=16.8e6", "--fov=160", "--trat_small=1", "--trat_large=20", f"--nx={n}", f"--ny={n}", *extra]
    ps = [ip.Params.from_args([*args, f"--M_unit={mu}"]) for mu in (3e27, 6e27)]
    with ip.Context(0, 8 << 30) as c:
        models = [ip.Model.load(p) for p in ps]
        c.set_record_precision(rec)
        c.upload_batch(models[0])
        imgs = c.render_batch(ps, models[0])
        for p, m, im in zip(ps, models, imgs):
            c.upload(m)
            ref = c.render(p, m)
            for k in ("unpol", "tau", "nstep"):
                assert np.asarray(getattr(ref, k)).tobytes() == np.asarray(getattr(im, k)).tobytes(), k
            if ref.pol is not None:
                assert ref.pol.tobytes() == im.pol.tobytes()
