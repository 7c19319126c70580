"""Moving images so long that a coordinate near the far end has few fraction
bits in float32 (600000 voxels: steps of 1/16): the samples 1/64 voxel beyond
the last one are outside, whichever way a tile is resampled."""
import numpy as np
import pytest

from lc2registration_gb300 import capi, synth
from lc2registration_gb300.geometry import Geometry
from oracle import oracle as O
from tests.helpers import make_context

pytestmark = pytest.mark.gpu

END = 599999  # last voxel along x


def _case(nd, r, hr_moving, vx, last):
    """Grid column `last` of vx falls on END + 1/64; exact in float32."""
    rng = np.random.default_rng(7)
    mdim = (END + 1, 48, 1) if nd == 2 else (END + 1, 16, 4)
    vdim = (vx, 40, 1) if nd == 2 else (vx, 16, 4)
    mov = np.empty(mdim[::-1], dtype=np.float32)
    rng.random(out=mov, dtype=np.float32)
    first = END - last
    us = 0.2 + 0.5 * mov[:vdim[2], :vdim[1], first:first + vx]
    us = np.concatenate([us, np.full(vdim[2:0:-1] + (vx - us.shape[2],), 0.4)], axis=2)
    us = (us + 0.2 * rng.random(us.shape)).astype(np.float32)
    # the moving image's origin puts voxel `first` on grid column 0
    mg = Geometry(mdim, (1.0, 1.0, 1.0), (-float(first), 0.0, 0.0))
    vg = Geometry(vdim, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    mat = np.eye(3 if nd == 2 else 4, dtype=np.float32)
    mat[0, -1] = 1.0 / 64
    mat[1, -1] = 2.0 if nd == 2 else 0.0
    return synth.Case("2D" if nd == 2 else "3D", vg, us, mg, mov, [1.0] * nd, r, hr_moving, {}, mat)


@pytest.mark.parametrize("nd,hr_moving", [(2, True), (2, False), (3, True), (3, False)])
def test_samples_beyond_the_end_are_outside(nd, hr_moving):
    r = 2
    # the last column of a tile's resampled region (2D) or of a tile (3D)
    case = _case(nd, r, hr_moving, 100, 64 + r if nd == 2 else 63)
    mats = case.true_mat[None].repeat(2, axis=0)
    ctx = make_context(case)
    got = ctx.evaluate_batch(mats)
    _, f = ctx.evaluate_fields(mats[0])
    warped = f["M"] if hr_moving else f["U"]
    last = 64 + r if nd == 2 else 63
    assert (warped[..., last] == 0.0).all() and (warped[..., last - 1] > 0.0).any()
    ctx.set_option(capi.OPTION_GENERIC, 1)
    np.testing.assert_allclose(got, ctx.evaluate_batch(mats), rtol=1e-6, atol=0)
    ctx.close()


def test_mutual_information_beyond_the_end():
    case = _case(3, 1, True, 100, 63)
    mi = capi.Context("3D", case.fixed_geom, case.moving_geom, case.virt_spacing, 0, True, "f32")
    mi.set_images(case.fixed, case.moving)
    lc = make_context(case)
    _, f = lc.evaluate_fields(case.true_mat)
    assert abs(mi.evaluate(case.true_mat) - O.nmi(f["U"], f["M"])) <= 1e-12
