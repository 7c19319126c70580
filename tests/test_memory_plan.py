"""lc2_context_bytes (host only): what a context holds and lc2_set_images takes
on top stays within what such a request has been admitted with -- the buffers
of the images, the static fields and 64 presampled images or 2 GiB of them, and
one image on its way in."""
import numpy as np
import pytest

from lc2registration_gb300 import capi
from lc2registration_gb300.geometry import Geometry

GIB = 1 << 30


def _admitted(mode, fdim, mdim, vdim, r, hr_moving, storage, max_batch=0):
    """(held, peak - held) of a context without padded fields."""
    nd = 3 if mode == "3D" else 2
    nv, nf, nm = (int(np.prod(d)) for d in (vdim, fdim, mdim))
    es = 4 if storage == "f32" else 2
    mi = r == 0
    slots = max(1, min(max_batch or 1, 1024, 65535 // vdim[2]))
    held = nv * 4 * (2 if hr_moving else 1) * slots + nm * es + nv * (es if hr_moving else 4)
    held += 0 if hr_moving else nv * 4
    if not mi:
        held += nv * 8 if hr_moving else nv * (16 + 24 + 16)
    else:
        held += nv + 64 * (4 * (65536 + 2) + 8 * 2 * 32)
    held += 64 * (96 + 16 + 8)
    if nd == 3 and not mi:
        held += 4 * nv * max(1, min(64, 2 * GIB // (4 * nv)))
    extra = 4 * max(nm, nf)
    if not hr_moving and not mi:
        extra = max(extra, 12 * nv)
    return held, extra


def _configs(n, seed):
    rng = np.random.default_rng(seed)
    for _ in range(n):
        mode = ["2D", "3D", "2DTo3D"][rng.integers(3)]
        nd = 2 if mode == "2D" else 3
        size = lambda: int(np.exp(rng.uniform(0, np.log(400))))
        fdim = [size() for _ in range(3)]
        mdim = [size() for _ in range(3)]
        if mode != "3D":
            fdim[2] = 1
        if mode == "2D":
            mdim[2] = 1
        sp = float(rng.choice([0.5, 1.0, 2.0]))
        vs = [sp] * nd
        if mode == "2DTo3D":
            vs[2] = 1.0
        vdim = [int(np.ceil(np.float32(d) / np.float32(s))) for d, s in zip(fdim, vs)]
        vdim += [1] * (3 - len(vdim))
        r = int(rng.integers(0 if mode == "3D" else 1, 7 if mode == "3D" else 13))
        yield (mode, tuple(fdim), tuple(mdim), tuple(vdim), vs, r, bool(rng.integers(2)),
               ["f32", "f16", "bf16"][rng.integers(3)])


def _bytes(mode, fdim, mdim, vs, r, hr, storage):
    g = lambda d: Geometry(d, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    return capi.context_bytes(capi.make_config(mode, g(fdim), g(mdim), vs, r, hr, storage))


def test_set_images_takes_no_more_than_one_image():
    for mode, fdim, mdim, vdim, vs, r, hr, storage in _configs(400, 1):
        held, peak = _bytes(mode, fdim, mdim, vs, r, hr, storage)
        _, extra = _admitted(mode, fdim, mdim, vdim, r, hr, storage)
        assert peak - held <= extra, (mode, fdim, mdim, vs, r, hr, storage)


def test_a_context_holds_no_more_than_it_was_admitted_with():
    """But for 32 MiB of presampled images of small grids, the error flag's 4
    bytes, and grids whose static fields and one presampled image alone are more:
    beyond 500^3, or of a few voxels along an axis."""
    more = 0
    for mode, fdim, mdim, vdim, vs, r, hr, storage in _configs(600, 2):
        held, _ = _bytes(mode, fdim, mdim, vs, r, hr, storage)
        want, _ = _admitted(mode, fdim, mdim, vdim, r, hr, storage)
        nv = int(np.prod(vdim))
        quad = mode == "3D" and 1 <= r <= 4
        if quad and (nv > 100_000_000 or min(vdim) < 8):
            continue
        assert held <= want + 4 + (32 << 20 if quad and 256 * nv < 32 << 20 else 0), (
            mode, fdim, mdim, vs, r, hr, storage, held, want)
        more += held > want + 4
    assert more < 60


@pytest.mark.parametrize("dim,r", [((96, 96, 96), 3), ((256, 256, 256), 4), ((160, 160, 160), 3),
                                   ((200, 200, 8), 4), ((512, 512, 16), 4)])
@pytest.mark.parametrize("hr_moving", [True, False])
def test_padded_grids_fit_what_was_admitted(dim, r, hr_moving):
    held, _ = _bytes("3D", dim, dim, [1.0] * 3, r, hr_moving, "f32")
    assert held <= _admitted("3D", dim, dim, dim, r, hr_moving, "f32")[0] + 4


def test_server_takes_every_request_that_fits_without_padded_fields():
    """Small, thin and very large grids whose padded fields pass the budget run
    without them; one byte less is refused."""
    reg = dict(initial=[0, 0, 0, 0, 0, 0, 1, 1, 1, 0, 0, 0], lower=[-1] * 6 + [0.9] * 3 + [-0.1] * 3,
               upper=[1] * 6 + [1.1] * 3 + [0.1] * 3, center=(8.0, 8.0, 8.0),
               rounds=[(["translation"], 1e-2)])
    geo = lambda d: Geometry(d, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    for dim, r in (((16, 16, 16), 2), ((24, 20, 1), 4), ((2, 218, 474), 4), ((600, 500, 700), 4)):
        for hr in (True, False):
            cfg = capi.make_config("3D", geo(dim), geo(dim), [1.0] * 3, r, hr)
            held, extra = _admitted("3D", dim, dim, dim, r, hr, "f32")
            lean = held + 4 + (4 * int(np.prod(dim)) if hr else 8 * int(np.prod(dim)))
            assert capi.context_bytes(cfg)[1] > lean
            srv = capi.Server(budget_bytes=lean, max_active=1)
            t = srv.submit(cfg, lc2_of_matrices=lambda m: np.ones(len(m)), **reg)
            assert srv.poll(t)["status"] == 0
            assert srv.stats()["peak_bytes"] == lean <= held + 4 + extra
            srv.close()
            srv = capi.Server(budget_bytes=lean - 1, max_active=1)
            with pytest.raises(capi.LC2Error, match="OUT_OF_MEMORY"):
                srv.submit(cfg, lc2_of_matrices=lambda m: np.ones(len(m)), **reg)
            srv.close()
