"""A step leaves nothing behind for the next: the projection backward clears the
gradient records it read, so a gradient-only step repeated on the same
parameters, also after a step from other cameras, gives the same gradient
rows.  Two runs of one step differ by the order of float atomics: a few
roundings (2^-24 each) of a sum's terms, 1e-5 of the norm with room for
cancellation in single rows.  Sizes around the groups of 32 views, the CTAs'
128 splats and the sort tiles; the compensation records too."""
import ctypes as C

import numpy as np
import pytest

from nanotracer_b200 import CameraUniform, GpuSplatBuffer, TrainConfig, Trainer
from nanotracer_b200._lib import SC_BWD_EXACT, check, lib
from nanotracer_b200.raster import cameras_array
from nanotracer_b200.scene import FOV_Y, orbit_pose, random_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact", [True, False])
@pytest.mark.parametrize("compensated", [False, True])
@pytest.mark.parametrize("n,V", [(1, 1), (127, 1), (129, 3), (4097, 2), (300, 32), (300, 33)])
def test_repeated_gradient_steps_agree(ctx, n, V, compensated, exact):
    W, H = 70, 45
    g = GpuSplatBuffer.upload(ctx, random_scene(n, n))
    tr = Trainer(ctx, TrainConfig(n_views=V, width=W, height=H, depth_max=8.0, compensated_sums=compensated,
                                  exact_backward=exact))
    y, x = np.mgrid[0:H, 0:W]
    tgt = np.broadcast_to((0.5 + 0.3 * np.sin(0.2 * x + 0.1 * y))[None, ..., None], (V, H, W, 3))
    tr.set_targets(ctx.storage_buffer("t", np.ascontiguousarray(tgt, np.float32)))
    shard = (n + 63) // 64 * 64
    rows = ctx.storage_buffer_zeroed("rows", 59 * shard * 4)

    def step(angle):
        cams = [CameraUniform.from_pose(*orbit_pose(angle + 11.0 * v), FOV_Y, W, H, n) for v in range(V)]
        loss = C.c_double()
        check(lib().sc_trainer_step_grads(tr.handle, g.handle, cameras_array(cams), 1.0 / V, 1, shard, rows.cptr,
                                          C.byref(loss)), ctx.handle)
        return rows.readback(np.float32, 59 * shard).reshape(59, shard).astype(np.float64)

    first = step(0.0)
    assert not first[:, n:].any() and np.linalg.norm(first) > 0
    for k in range(3):
        if k == 1:
            step(140.0)
        again = step(0.0)
        assert np.linalg.norm(again - first) <= 1e-5 * np.linalg.norm(first)
