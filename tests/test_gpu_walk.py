"""The transfer walk with several lanes per ray (k_walk, the default) against
the walk with one lane per ray (k_transfer, IPG_XFER_STAGE=0).

Both spell out the roundings of the transfer's sums and products, so their
outputs must agree in every bit.  The ray counts straddle the edges at which
the launch changes its lanes per ray (32, 16, 8, 4: one, two and four times
eight rays per SM) and leave partly filled warps; the rays' step counts leave
partly filled blocks of records.
"""
import os

import numpy as np
import pytest

import ipole_b200 as ip
from tests import common

pytestmark = pytest.mark.gpu

RESIDENT = 148 * 8
FORMS = [(ip.IPG_RECORDS_FP64, ip.IPG_STEP_FP64), (ip.IPG_RECORDS_MIXED, ip.IPG_STEP_FP64),
         (ip.IPG_RECORDS_FP64, ip.IPG_STEP_FP32), (ip.IPG_RECORDS_MIXED, ip.IPG_STEP_FP32)]


def _trace(model, cam, ij, stage, rec, step):
    old = os.environ.pop("IPG_XFER_STAGE", None)
    if stage is not None:
        os.environ["IPG_XFER_STAGE"] = stage
    try:
        with ip.Context(0, 8 << 30) as c:  # the setting is read when a context is created
            c.upload(model)
            c.set_record_precision(rec)
            c.set_step_precision(step)
            return c.trace(cam, ij)
    finally:
        os.environ.pop("IPG_XFER_STAGE", None)
        if old is not None:
            os.environ["IPG_XFER_STAGE"] = old


def _case(dumps, extra=()):
    meta, _ = common.load_golden("c1_bright_32")
    dump = dumps.get(meta)
    args = [f"--dump={dump}", "--freqcgs=230e9", "--thetacam=163", "--phicam=0", "--MBH=6.5e9", "--dsource=16.8e6",
            "--fov=160", "--M_unit=3e27", "--trat_small=1", "--trat_large=20", "--nx=160", "--ny=160", *extra]
    p = ip.Params.from_args(args)
    m = ip.Model.load(p)
    return m, ip.camera_for(p, m.grid)


@pytest.mark.parametrize("n", [1, 3, RESIDENT, RESIDENT + 1, 2 * RESIDENT + 1, 4 * RESIDENT + 3])
def test_walk_bit_identical(n, dumps):
    m, cam = _case(dumps, ["--rotcam=20"])
    at = np.random.default_rng(n).choice(160 * 160, size=n, replace=False)
    ij = np.stack([at // 160, at % 160], axis=1).astype(np.int32)
    for rec, step in FORMS:
        a, b = _trace(m, cam, ij, "0", rec, step), _trace(m, cam, ij, None, rec, step)
        assert a.tobytes() == b.tobytes(), (n, rec, step)


@pytest.mark.parametrize("extra", [["-unpol"], ["--stokes_floors=1"], ["--target_nturns=1"], ["--emission_type=1"]],
                         ids=["unpol", "floors", "subring", "pandya"])
def test_walk_options_bit_identical(extra, dumps):
    m, cam = _case(dumps, extra)
    at = np.arange(0, 160 * 160, 97)
    ij = np.stack([at // 160, at % 160], axis=1).astype(np.int32)
    for rec, step in FORMS:
        a, b = _trace(m, cam, ij, "0", rec, step), _trace(m, cam, ij, None, rec, step)
        assert a.tobytes() == b.tobytes(), (extra, rec, step)


@pytest.mark.parametrize("n,extra", [(3, []), (25, ["--target_nturns=1"]), (40, ["--stokes_floors=1"]), (50, ["-unpol"]),
                                     (50, [])])
def test_batch_walk_bit_identical(n, extra, dumps):
    """the batches' walk (the instances' coefficients from their own blocks)
    with 32, 16, 8 and 4 lanes per item against each instance's own render,
    in every form"""
    meta, _ = common.load_golden("c1_bright_32")
    args = [f"--dump={dumps.get(meta)}", "--freqcgs=230e9", "--thetacam=163", "--phicam=0", "--MBH=6.5e9",
            "--dsource=16.8e6", "--fov=160", "--trat_small=1", "--trat_large=20", f"--nx={n}", f"--ny={n}", *extra]
    ps = [ip.Params.from_args([*args, f"--M_unit={mu}"]) for mu in (3e27, 6e27)]
    models = [ip.Model.load(p) for p in ps]
    for rec, step in FORMS:
        with ip.Context(0, 4 << 30) as c:
            c.set_record_precision(rec)
            c.set_step_precision(step)
            c.upload_batch(models[0])
            imgs = c.render_batch(ps, models[0])
            for p, m, im in zip(ps, models, imgs):
                c.upload(m)
                ref = c.render(p, m)
                for k in ("unpol", "tau", "nstep", "pol"):
                    a, b = getattr(ref, k), getattr(im, k)
                    assert (a is None) == (b is None) and (a is None or a.tobytes() == b.tobytes()), (n, rec, step, k)
