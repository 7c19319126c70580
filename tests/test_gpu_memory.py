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
