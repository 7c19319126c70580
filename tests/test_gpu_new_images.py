"""New images in a context that has already evaluated (and captured its CUDA
graphs): the values are those of a fresh context."""
import numpy as np
import pytest

from lc2registration_gb300 import synth
from tests.helpers import make_context, perturbed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["2D", "3D"])
def test_new_images_in_a_used_context(mode):
    case = (synth.case_2d(seed=5, size=64, r=3) if mode == "2D" else
            synth.case_3d(seed=6, mr_size=40, us_size=32, r=2, blobs=5))
    mats = perturbed(case, np.random.default_rng(1), 4)
    ctx = make_context(case)
    ctx.evaluate_batch(mats)
    # other value ranges: other fixed-point scales
    ctx.set_images(2.0 * case.fixed, 0.3 * case.moving)
    got = ctx.evaluate_batch(mats)
    case.fixed, case.moving = 2.0 * case.fixed, 0.3 * case.moving
    fresh = make_context(case)
    np.testing.assert_array_equal(got, fresh.evaluate_batch(mats))
    ctx.close()
    fresh.close()
