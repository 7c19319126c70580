"""The resampling's tile classes -- inside, across the border, outside, and
transforms too coarse for its integer floors -- give the values of the plain
sampling: transforms whose sample positions are exact in float32, so that both
sample at the same positions."""
import numpy as np
import pytest

from lc2registration_gb300 import capi, synth
from lc2registration_gb300.geometry import Geometry
from oracle import oracle as O
from tests.helpers import make_context

pytestmark = pytest.mark.gpu

DIM = (75, 41, 27)


def _case(r, hr_moving=True):
    rng = np.random.default_rng(2)
    g = Geometry(DIM, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    mov = (0.2 + 0.6 * rng.random(DIM[::-1])).astype(np.float32)
    us = (0.1 + 0.5 * mov + 0.3 * rng.random(DIM[::-1])).astype(np.float32)
    return synth.Case("3D", g, us, g, mov, [1.0, 1.0, 1.0], r, hr_moving, {}, np.eye(4))


def _mats():
    """Scalings about (32, 16, 8), shifts by halves and a reflection; scales of
    2^17 and more leave the integer floors' range inside a tile."""
    out = []
    c = np.array([32.0, 16.0, 8.0])
    for s in ([1, 1, 1], [0.5, 0.5, 2], [4, 1, 0.25], [64, 64, 64], [-1, 1, 1], [2.0 ** -10] * 3,
              [2.0 ** 17, 1, 1], [2.0 ** 20] * 3):
        m = np.eye(4)
        m[:3, :3] = np.diag(s)
        m[:3, 3] = c - np.array(s) * c
        out.append(m)
    for t in ([0.5, 0, 0], [40, -20.5, 3], [-74, 0, 0], [74.5, 0, 0], [500, 0, 0], [0, 0, 1e6],
              [0, -40.5, 26]):
        m = np.eye(4)
        m[:3, 3] = t
        out.append(m)
    return np.stack(out).astype(np.float32)


@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("hr_moving", [True, False])
def test_presampled_equals_sampled_in_the_kernel(storage, hr_moving):
    case = _case(2, hr_moving)
    ctx = make_context(case, storage)
    # without the scale of 2^-10, which leaves every patch nearly constant: its
    # columns lie at the degeneracy threshold, where the two paths' Sobel
    # magnitudes, not their samples, decide
    mats = np.delete(_mats(), 5, axis=0)
    got = ctx.evaluate_batch(mats)
    assert (got > 0.0).sum() >= 6
    ctx.set_option(capi.OPTION_GENERIC, 1)
    np.testing.assert_allclose(got, ctx.evaluate_batch(mats), rtol=1e-6, atol=0)
    ctx.close()


def test_mutual_information_samples():
    case = _case(2)
    mi = capi.Context("3D", case.fixed_geom, case.moving_geom, case.virt_spacing, 0, True, "f32")
    mi.set_images(case.fixed, case.moving)
    lc = make_context(case)
    for m, v in zip(_mats(), mi.evaluate_batch(_mats())):
        _, f = lc.evaluate_fields(m)
        assert abs(v - O.nmi(f["U"], f["M"])) <= 1e-12


@pytest.mark.parametrize("hr_moving", [True, False])
def test_mutual_information_of_a_crowded_bin(hr_moving):
    """Constant images with a few other voxels: one joint bin holds nearly the
    whole grid, many times what a 16-bit half of the shared histogram can."""
    dim = (130, 100, 70)
    g = Geometry(dim, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    us, mov = np.full((2,) + dim[::-1], 0.5, dtype=np.float32)
    rng = np.random.default_rng(4)
    for img in (us, mov):
        img[rng.integers(0, dim[2], 900), rng.integers(0, dim[1], 900),
            rng.integers(0, dim[0], 900)] = rng.random(900).astype(np.float32)
    case = synth.Case("3D", g, us, g, mov, [1.0, 1.0, 1.0], 2, hr_moving, {}, np.eye(4))
    mi = capi.Context("3D", g, g, [1.0, 1.0, 1.0], 0, hr_moving, "f32")
    mi.set_images(us, mov)
    mats = np.stack([np.eye(4, dtype=np.float32)] * 4)
    mats[1:, 0, 3] = [0.5, 1.0, 3.0]
    lc = make_context(case)
    for m, v in zip(mats, mi.evaluate_batch(mats)):
        _, f = lc.evaluate_fields(m)
        ref = O.nmi(f["U"], f["M"])
        assert abs(v - ref) <= 1e-12 * ref
        assert mi.evaluate(m) == v
