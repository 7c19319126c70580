"""lc2_evaluate_batch returns small batches through pinned host memory (at most
128 values, and a single transform is read from there too): the same values as
the staged calls on both sides of the limits, in any order of sizes."""
import numpy as np
import pytest

from lc2registration_gb300 import synth
from tests.helpers import make_context, perturbed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,r", [("2D", 3), ("3D", 2), ("3D", 0)])
def test_small_calls_equal_staged_calls(mode, r):
    case = (synth.case_2d(seed=5, size=48, r=r) if mode == "2D" else
            synth.case_3d(seed=6, mr_size=32, us_size=24, r=r, blobs=5))
    mats = perturbed(case, np.random.default_rng(1), 130)
    ctx = make_context(case)
    for count in (1, 2, 1, 127, 128, 129, 130, 1, 64):
        got = ctx.evaluate_batch(mats[:count])
        ctx.stage(mats[:count])
        ctx.launch(count)
        np.testing.assert_array_equal(got, ctx.fetch(count))
    np.testing.assert_array_equal([ctx.evaluate(m) for m in mats[:5]], got[:5])
    ctx.close()
