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


@pytest.mark.parametrize("mode,r", [("2D", 3), ("3D", 2), ("3D", 0)])
def test_sums_between_batches_of_any_size(mode, r):
    """Staged launches and evaluations in any order of sizes, past the buffers'
    first 64 transforms, with kernel timing and without graphs: the sums each
    starts from are those the one before left."""
    case = _case(mode, r)
    mats = perturbed(case, np.random.default_rng(3), 150)
    ctx = make_context(case)
    ref = [ctx.evaluate(m) for m in mats]
    for k, count in enumerate((3, 64, 150, 1, 149, 65, 150)):
        ctx.stage(mats[:count])
        for _ in range(2):
            ctx.launch(count)
        ctx.launch(count // 2)
        np.testing.assert_array_equal(ctx.fetch(count), ref[:count])
        ctx.set_option(capi.OPTION_GRAPHS, k % 2)
        ctx.enable_kernel_timing(k % 3 == 0)
        np.testing.assert_array_equal(ctx.evaluate_batch(mats[:count]), ref[:count])
        if r:
            ctx.weighting_map(mats[0])
    ctx.close()


def test_staged_launch_does_not_pay_for_larger_batches():
    """One transform of mutual information after a batch of 4096 (1 GiB of
    histograms): no slower than before it but for the noise of the host's
    clock; clearing them all takes 150 us or more."""
    import time

    case = _case("3D", 0)
    mats = perturbed(case, np.random.default_rng(1), 1).repeat(4096, axis=0)
    ctx = make_context(case)

    def one():
        best = 1e9
        for _ in range(50):
            t0 = time.perf_counter()
            ctx.stage(mats[:1])
            ctx.launch(1)
            ctx.fetch(1)
            best = min(best, time.perf_counter() - t0)
        return best

    one()
    before = one()
    ctx.evaluate_batch(mats)
    assert one() < before + 60e-6
    ctx.close()


def test_staging_ahead_of_a_running_launch():
    """Transforms staged while an earlier launch runs: the copy of the ones
    before them has read them by then."""
    case = synth.case_3d(seed=6, mr_size=64, us_size=64, r=3, blobs=5)
    a, b, c = (perturbed(case, np.random.default_rng(s), 200) for s in (1, 2, 3))
    ctx = make_context(case)
    want = ctx.evaluate_batch(b)
    for _ in range(5):
        ctx.stage(a)
        for _ in range(4):
            ctx.launch(200)
        ctx.stage(b)
        ctx.launch(200)
        ctx.stage(c)
        np.testing.assert_array_equal(ctx.fetch(200), want)
    ctx.close()
