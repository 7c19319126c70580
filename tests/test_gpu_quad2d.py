"""2D windows in column quads (k_quad2d, and the stacks' work-list kernel built
on the same tile): 16- and 32-row tiles and the work list give the same bits at
the edges of tiles, quads and images and on both branches of the solve, and the
values match the FP64 oracle."""
import numpy as np
import pytest

from lc2registration_gb300 import capi, synth
from lc2registration_gb300.geometry import Geometry, affine2d
from tests.helpers import make_context, oracle_eval

pytestmark = pytest.mark.gpu

SIZES = [(32, 32, 3), (31, 33, 1), (33, 31, 2), (64, 17, 4), (70, 49, 5), (45, 65, 6), (5, 5, 2),
         (1, 40, 1), (97, 3, 3)]


def _images(nx, ny, structured, seed=5):
    """(ultrasound, moving image of nx + 6 by ny + 6). structured: bands of
    noise, an exponential (the image and its Sobel magnitude collinear), a ramp
    (constant Sobel magnitude) and a constant."""
    rng = np.random.default_rng(seed)
    mov = 0.2 + 0.6 * rng.random((1, ny + 6, nx + 6))
    if structured:
        x = np.arange(nx + 6)
        q = max(1, (ny + 6) // 4)
        mov[0, q:2 * q] = 0.2 * 1.03 ** (x % 64)
        mov[0, 2 * q:3 * q] = 0.1 + 0.01 * x
        mov[0, 3 * q:] = 0.4
    us = 0.1 + 0.6 * mov[:, 3:-3, 3:-3] + 0.3 * rng.random((1, ny, nx))
    us[:, : ny // 6] = 0.0  # invalid patches
    return us.astype(np.float32), mov.astype(np.float32)


@pytest.mark.parametrize("nx,ny,r", SIZES)
def test_tile_heights_and_oracle_2d(nx, ny, r):
    ug = Geometry((nx, ny, 1), (1.0, 1.0, 1.0), (3.0, 3.0, 0.0))
    mg = Geometry((nx + 6, ny + 6, 1), (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    c = ug.center()[:2]
    mats = np.stack([affine2d(0.0, [0.0, 0.0], center=c), affine2d(2.0, [0.7, -1.2], center=c),
                     affine2d(0.0, [0.6 * nx, 0.0], center=c)])
    for structured in (True, False):
        us, mov = _images(nx, ny, structured)
        case = synth.Case("2D", ug, us, mg, mov, [1.0, 1.0], r, True, {}, mats[0])
        ctx = make_context(case)
        got = {}
        for rows in (16, 32):
            ctx.set_option(capi.OPTION_TILE_ROWS, rows)
            got[rows] = ctx.evaluate_batch(mats), [ctx.weighting_map(m)[1] for m in mats]
        np.testing.assert_array_equal(got[16][0], got[32][0])
        np.testing.assert_array_equal(got[16][1], got[32][1])
        if not structured:
            for m, g in zip(mats[:2], got[16][0]):
                want = oracle_eval(case, m, use_boxsum=False)
                assert abs(g - want) <= 1e-5 * abs(want)
        ctx.close()


@pytest.mark.parametrize("r", [1, 4, 6])
def test_work_list_equals_contexts(r):
    sizes = [(32, 32), (31, 33), (70, 49), (20, 65)]
    mr = synth.mr_phantom((48, 48, 48), 8, 1.5, seed=11)
    mg = Geometry((48, 48, 48), (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    frames = []
    for i, (nx, ny) in enumerate(sizes):
        fg = Geometry((nx, ny, 1), (0.5, 0.5, 1.0), (6.0, 6.0, 12.0 + 6 * i))
        us, _ = _images(nx, ny, False, seed=i)
        frames.append(synth.Case("2DTo3D", fg, us, mg, mr, [0.5, 0.5], r, True, {}, np.eye(4)))
    st = capi.Stack(mg, r, "f32")
    st.set_moving(mr)
    for i, f in enumerate(frames):
        assert st.add_frame(f.fixed_geom, f.virt_spacing, f.fixed) == i
    ids = np.repeat(np.arange(len(frames)), 3)
    mats = np.stack([np.eye(4, dtype=np.float32)] * len(ids))
    mats[1::3, 2, 3] = 2.25
    mats[2::3, 0, 1] = 0.125
    got = st.evaluate(ids, mats)
    ctxs = [make_context(f) for f in frames]
    np.testing.assert_array_equal(got, [ctxs[i].evaluate(m) for i, m in zip(ids, mats)])
