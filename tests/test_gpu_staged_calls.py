"""The staged calls after an evaluation: lc2_evaluate_batch leaves its transforms
staged and its values fetchable, whichever way the batch went (up to 128
transforms through pinned host memory, one of them read from there), and new
images leave the staged transforms as they are."""
import numpy as np
import pytest

from lc2registration_gb300 import capi, synth
from tests.helpers import make_context, perturbed

pytestmark = pytest.mark.gpu


def _case(mode, r):
    return (synth.case_2d(seed=5, size=48, r=r) if mode == "2D" else
            synth.case_3d(seed=6, mr_size=32, us_size=24, r=r, blobs=5))


@pytest.mark.parametrize("count", [1, 2, 128, 129])
@pytest.mark.parametrize("mode,r", [("2D", 3), ("3D", 2), ("3D", 0)])
def test_fetch_and_launch_after_an_evaluation(mode, r, count):
    case = _case(mode, r)
    mats = perturbed(case, np.random.default_rng(1), count)
    others = perturbed(case, np.random.default_rng(2), 130)
    ctx = make_context(case)
    got = ctx.evaluate_batch(mats)               # the first call after new images
    np.testing.assert_array_equal(ctx.fetch(count), got)
    ctx.launch(count)
    np.testing.assert_array_equal(ctx.fetch(count), got)
    # over an older staged launch's transforms and values
    ctx.stage(others)
    ctx.launch(130)
    assert not np.array_equal(ctx.fetch(130)[:count], got)
    np.testing.assert_array_equal(ctx.evaluate_batch(mats), got)
    np.testing.assert_array_equal(ctx.fetch(count), got)
    ctx.launch(count)
    np.testing.assert_array_equal(ctx.fetch(count), got)
    # a refused batch and new images leave the staged transforms
    bad = others[:2].copy()
    bad[1, 0, 0] = np.nan
    with pytest.raises(capi.LC2Error, match="NaN"):
        ctx.evaluate_batch(bad)
    ctx.set_images(case.fixed, case.moving)
    ctx.launch(count)
    np.testing.assert_array_equal(ctx.fetch(count), got)
    with pytest.raises(capi.LC2Error, match="staged"):
        ctx.launch(count + 1)
    ctx.close()
