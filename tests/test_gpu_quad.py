"""The moments pass in column quads (k_fused_quad, the default for 3D contexts
of a resampled MR/CT at radius 1-4) against the 16-row kernel it shares no
moments code with: the same bits at the edges of its tiles, quads, z chunks and
padded images, on both branches of its solve, and per voxel."""
import numpy as np
import pytest

from lc2registration_gb300 import capi, synth
from lc2registration_gb300.geometry import Geometry, affine3d
from tests.helpers import make_context, oracle_eval

pytestmark = pytest.mark.gpu


def _case(dim, r, seed=7):
    """Grid of (x, y, z) = dim inside a slightly larger moving image whose
    slices hold, in turn, noise, an exponential (M and its Sobel magnitude
    collinear), a ramp (constant Sobel magnitude) and a constant."""
    rng = np.random.default_rng(seed)
    md = tuple(d + 6 for d in dim)
    mov = 0.3 + 0.2 * rng.random((md[2], md[1], md[0])).astype(np.float32)
    x = np.arange(md[0], dtype=np.float32)
    q = max(1, md[2] // 4)
    mov[q:2 * q] = 0.2 * np.float32(1.03) ** x
    mov[2 * q:3 * q] = 0.1 + 0.01 * x
    mov[3 * q:] = 0.4
    us = (0.1 + rng.random((dim[2], dim[1], dim[0]))).astype(np.float32)
    mg = Geometry(md, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    ug = Geometry(dim, (1.0, 1.0, 1.0), (3.0, 3.0, 3.0))
    c = ug.center()
    mats = np.stack([affine3d([0, 0, 0], [0, 0, 0], center=c),
                     affine3d([3.0, -2.0, 4.0], [1.5, -2.25, 0.75], [1.02, 0.97, 1.0],
                              [0.02, 0.0, -0.01], c),
                     affine3d([0, 0, 0], [0.6 * dim[0], 0, 0], center=c)])
    return synth.Case("3D", ug, us, mg, mov, [1.0, 1.0, 1.0], r, True, {}, mats[0]), mats


@pytest.mark.parametrize("dim,r", [((32, 24, 12), 4), ((33, 25, 9), 4), ((31, 40, 11), 4),
                                   ((64, 41, 10), 3), ((37, 23, 7), 3), ((65, 17, 16), 2),
                                   ((5, 5, 5), 2), ((96, 50, 3), 1), ((1, 64, 33), 1)])
def test_quad_kernel_equals_16_row_kernel(dim, r):
    case, mats = _case(dim, r)
    ctx = make_context(case, "f32")
    ctx.set_option(capi.OPTION_TILE_ROWS, 16)
    ref = ctx.evaluate_batch(mats)
    fields = [ctx.weighting_map(m)[1] for m in mats]
    ctx.set_option(capi.OPTION_TILE_ROWS, 0)
    for zc in (0, 1, 5):
        ctx.set_option(capi.OPTION_ZCHUNK, zc)
        np.testing.assert_array_equal(ctx.evaluate_batch(mats), ref)
    ctx.set_option(capi.OPTION_ZCHUNK, 0)
    for m, f in zip(mats, fields):
        np.testing.assert_array_equal(ctx.weighting_map(m)[1], f)
    # the padded presample buffer again after the other kernel used an unpadded one
    ctx.set_option(capi.OPTION_TILE_ROWS, 8)
    np.testing.assert_array_equal(ctx.evaluate_batch(mats), ref)
    ctx.set_option(capi.OPTION_TILE_ROWS, 0)
    np.testing.assert_array_equal(ctx.evaluate_batch(mats), ref)
    # twice the images: the quantised ultrasound and weighting factors follow
    ctx.set_images(2.0 * case.fixed, case.moving)
    got = ctx.evaluate_batch(mats)
    ctx.set_option(capi.OPTION_TILE_ROWS, 16)
    np.testing.assert_array_equal(ctx.evaluate_batch(mats), got)
    ctx.close()


@pytest.mark.parametrize("dim,r", [((32, 24, 12), 4), ((33, 25, 9), 4), ((31, 40, 11), 4),
                                   ((64, 41, 10), 3), ((37, 23, 7), 3), ((65, 17, 16), 2),
                                   ((5, 5, 5), 2), ((96, 50, 3), 1), ((1, 64, 33), 1)])
def test_fixed_quad_kernel_equals_16_row_kernel(dim, r):
    """HighResolutionModality: Fixed: the structured volume is the static image,
    the ultrasound (with zeros, which invalidate their patches) is resampled."""
    case, mats = _case(dim, r)
    us = case.fixed.copy()
    us[:, : us.shape[1] // 5] = 0.0
    fixed = np.ascontiguousarray(case.moving[3:-3, 3:-3, 3:-3])
    case = synth.Case("3D", case.fixed_geom, fixed, case.fixed_geom, us, [1.0, 1.0, 1.0], r, False,
                      {}, mats[0])
    ctx = make_context(case, "f32")
    ctx.set_option(capi.OPTION_TILE_ROWS, 16)
    ref = ctx.evaluate_batch(mats)
    ctx.set_option(capi.OPTION_TILE_ROWS, 0)
    for zc in (0, 1, 5):
        ctx.set_option(capi.OPTION_ZCHUNK, zc)
        np.testing.assert_array_equal(ctx.evaluate_batch(mats), ref)
    want = oracle_eval(case, mats[0], use_boxsum=False)
    assert abs(ref[0] - want) <= 1e-5 * abs(want)
    ctx.close()


@pytest.mark.parametrize("hr_moving", [True, False])
@pytest.mark.parametrize("dim,r", [((64, 40, 20), 2), ((33, 27, 20), 3), ((65, 56, 12), 4)])
def test_batches_of_two_overlapping_launches(dim, r, hr_moving):
    """Batches that fill the device run the rows 24-row tiles leave over in a
    launch of their own that overlaps the first: same bits as the 16-row kernel,
    from graphs and without, in groups and after another batch's buffers."""
    case, mats = _case(dim, r)
    if not hr_moving:
        fixed = np.ascontiguousarray(case.moving[3:-3, 3:-3, 3:-3])
        case = synth.Case("3D", case.fixed_geom, fixed, case.fixed_geom, case.fixed, [1.0, 1.0, 1.0],
                          r, False, {}, mats[0])
    rng = np.random.default_rng(1)
    c = case.fixed_geom.center()
    mats = np.stack([affine3d(rng.uniform(-4, 4, 3), rng.uniform(-3, 3, 3), center=c)
                     for _ in range(100)])
    ctx = make_context(case, "f32")
    ctx.set_option(capi.OPTION_TILE_ROWS, 16)
    ref = ctx.evaluate_batch(mats)
    ctx.set_option(capi.OPTION_TILE_ROWS, 0)
    for graphs in (1, 0):
        ctx.set_option(capi.OPTION_GRAPHS, graphs)
        for zc in (0, 5):
            ctx.set_option(capi.OPTION_ZCHUNK, zc)
            for n in (60, 100, 60):
                np.testing.assert_array_equal(ctx.evaluate_batch(mats[:n]), ref[:n])
    ctx.close()
