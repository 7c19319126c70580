"""The static fields lc2_set_images computes (box sums in rows of 128 columns
and segments of 16 lines, weighting factors, static bins) at grid sizes around
those limits, through LC2 against the FP64 oracle; a refused image leaves the
context as it was."""
import numpy as np
import pytest

from lc2registration_gb300 import capi, synth
from lc2registration_gb300.geometry import Geometry, affine2d, affine3d
from tests.helpers import make_context, oracle_eval

pytestmark = pytest.mark.gpu


def _case(dim, r, hr_moving, seed=3):
    rng = np.random.default_rng(seed)
    nd = 2 if dim[2] == 1 else 3
    g = Geometry(dim, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    mr, noise = rng.random((2, dim[2], dim[1], dim[0]))
    us = 0.2 + 0.6 * mr + 0.3 * noise
    us[:, :2, -9:] = 0.0  # invalid patches in a corner of the ultrasound
    imgs = [us.astype(np.float32), mr.astype(np.float32)]
    if not hr_moving:
        imgs.reverse()
    c = g.center()
    mat = (affine2d(0.5, [0.2, -0.1], center=c[:2]) if nd == 2 else
           affine3d([1.0, -2.0, 1.5], [0.3, -0.2, 0.6], center=c))
    return synth.Case("2D" if nd == 2 else "3D", g, imgs[0], g, imgs[1], [1.0] * nd, r, hr_moving,
                      {}, mat)


@pytest.mark.parametrize("hr_moving", [True, False])
@pytest.mark.parametrize("dim,r", [((129, 33, 1), 12), ((128, 16, 1), 1), ((257, 47, 1), 5),
                                   ((130, 17, 16), 2), ((127, 16, 15), 4), ((20, 33, 17), 6)])
def test_static_fields(dim, r, hr_moving):
    case = _case(dim, r, hr_moving)
    ctx = make_context(case)
    got = ctx.evaluate(case.true_mat)
    want = oracle_eval(case, case.true_mat, use_boxsum=False)
    assert want > 0 and abs(got / want - 1.0) < 1e-5
    ctx.close()


def test_refused_image_leaves_the_context():
    case = _case((40, 32, 24), 2, True)
    ctx = make_context(case)
    ref = ctx.evaluate(case.true_mat)
    for which in (0, 1):
        bad = [case.fixed.copy(), case.moving.copy()]
        bad[which][3, 4, 5] = np.nan
        with pytest.raises(capi.LC2Error, match=f"NaN/Inf at {(3 * 32 + 4) * 40 + 5}"):
            ctx.set_images(*bad)
        assert ctx.evaluate(case.true_mat) == ref
    ctx.close()
