"""Device memory while lc2_set_images and batches run, watched from a second
thread, stays within lc2_context_bytes' peak; new images between batches too."""
import ctypes
import threading

import numpy as np
import pytest

from lc2registration_gb300 import capi
from lc2registration_gb300.geometry import Geometry, affine2d, affine3d

pytestmark = pytest.mark.gpu


class Watch:
    """Largest live device memory of the library while it is entered."""

    def __enter__(self):
        self.lib, self.stop, self.top = capi.load(), threading.Event(), 0
        self.thread = threading.Thread(target=self.run)
        self.thread.start()
        return self

    def run(self):
        b, n = ctypes.c_size_t(), ctypes.c_longlong()
        while not self.stop.is_set():
            self.lib.lc2_debug_device_bytes(ctypes.byref(b), ctypes.byref(n))
            self.top = max(self.top, b.value)

    def __exit__(self, *a):
        self.stop.set()
        self.thread.join()


@pytest.mark.parametrize("hr_moving", [True, False])
@pytest.mark.parametrize("dim,r", [((1600, 1200, 1), 4), ((160, 150, 140), 3), ((150, 140, 130), 5),
                                   ((140, 130, 120), 0), ((300, 300, 6), 4)])
def test_peak_is_not_exceeded(dim, r, hr_moving):
    nd = 2 if dim[2] == 1 else 3
    rng = np.random.default_rng(1)
    fixed, moving = rng.random((2,) + dim[::-1], dtype=np.float32)
    g = Geometry(dim, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    cfg = capi.make_config("2D" if nd == 2 else "3D", g, g, [1.0] * nd, r, hr_moving)
    held, peak = capi.context_bytes(cfg)
    mat = affine2d(1.0, [0.5, 0.2]) if nd == 2 else affine3d([1, 2, 1], [0.5, 0.2, 0.1])
    ctx = capi.Context("2D" if nd == 2 else "3D", g, g, [1.0] * nd, r, hr_moving, "f32")
    with Watch() as w:
        for _ in range(2):
            ctx.set_images(fixed, moving)
            ctx.evaluate_batch(np.stack([mat] * 64))
    ctx.close()
    assert held / 2 < w.top <= peak


@pytest.mark.parametrize("r", [2, 3, 4])
@pytest.mark.parametrize("hr_moving", [True, False])
def test_request_without_padded_fields_equals_alone(hr_moving, r):
    """A budget that holds a request's context only without its padded fields:
    the same registration as with them."""
    from lc2registration_gb300 import synth
    from tests.helpers import make_context
    from tests.test_memory_plan import _admitted

    case = synth.case_3d(seed=14, mr_size=32, us_size=24, r=r, blobs=6)
    if not hr_moving:
        case = synth.Case("3D", case.moving_geom, case.moving, case.fixed_geom, case.fixed,
                          list(case.moving_geom.spacing), r, hr_moving=False, true_params={}, true_mat=None)
    c = case.fixed_geom.center()
    reg = dict(initial=[0, 0, 0, 0, 0, 0, 1, 1, 1, 0, 0, 0],
               lower=[-8, -8, -8, -6, -6, -6] + [0.9] * 3 + [-0.05] * 3,
               upper=[8, 8, 8, 6, 6, 6] + [1.1] * 3 + [0.05] * 3, center=c,
               direct_entries=["translation"], direct_maxeval=40, rounds=[(["translation", "rotation"], 1e-3)])
    ctx = make_context(case)
    alone = capi.register(ctx, **reg)
    held, extra = _admitted("3D", case.fixed_geom.dim, case.moving_geom.dim, ctx.virtual_dims(), r,
                            hr_moving, "f32")
    ctx.close()
    cfg = capi.make_config("3D", case.fixed_geom, case.moving_geom, case.virt_spacing, r, hr_moving)
    budget = held + 4 + extra
    assert capi.context_bytes(cfg)[1] > budget
    srv = capi.Server(budget_bytes=budget, max_active=2)
    with Watch() as w:
        got = srv.poll(srv.submit(cfg, case.fixed, case.moving, **reg))
    srv.close()
    assert got["status"] == 0, got["message"]
    np.testing.assert_array_equal(got["params"][:12], alone["params"])
    assert got["lc2"] == alone["lc2"] and got["evaluations"] == alone["evaluations"]
    assert w.top <= budget


def test_failed_upload_has_waited_for_the_images():
    """An allocation that fails between the two uploads: the first image, in
    pinned memory, is no longer being read when the call returns."""
    import torch

    dim = (300, 300, 300)
    g = Geometry(dim, (1.0, 1.0, 1.0), (0.0, 0.0, 0.0))
    imgs = [torch.rand(dim[::-1]).pin_memory() for _ in range(2)]
    ctx = capi.Context("3D", g, g, [1.0] * 3, 2, True, "f16")
    lib = capi.load()
    for k in (1, 2):
        lib.lc2_debug_fail_allocation(k)
        with pytest.raises(capi.LC2Error, match="OUT_OF_MEMORY"):
            ctx.set_images(imgs[0].numpy(), imgs[1].numpy())
        lib.lc2_debug_fail_allocation(0)
        assert torch.cuda.ExternalStream(ctx.stream()).query()
    ctx.set_images(imgs[0].numpy(), imgs[1].numpy())
    assert ctx.evaluate(np.eye(4, dtype=np.float32)) > 0.0
    ctx.close()
