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


def _grad_stepper(ctx, g, V, W, H, **kw):
    n = g.n
    tr = Trainer(ctx, TrainConfig(n_views=V, width=W, height=H, depth_max=8.0, **kw))
    y, x = np.mgrid[0:H, 0:W]
    tgt = np.broadcast_to((0.5 + 0.3 * np.sin(0.2 * x + 0.1 * y))[None, ..., None], (V, H, W, 3))
    tr.set_targets(ctx.storage_buffer("t", np.ascontiguousarray(tgt, np.float32)))
    shard = (n + 63) // 64 * 64
    rows = ctx.storage_buffer_zeroed("rows", 59 * shard * 4)

    def step(cams):
        loss = C.c_double()
        check(lib().sc_trainer_step_grads(tr.handle, g.handle, cameras_array(cams), 1.0 / V, 1, shard, rows.cptr,
                                          C.byref(loss)), ctx.handle)
        return rows.readback(np.float32, 59 * shard).reshape(59, shard).astype(np.float64), tr.images(), loss.value
    return tr, step


@pytest.mark.parametrize("form", [dict(), dict(sort_mode=1), dict(ssim_lambda=0.2), dict(compensated_sums=True),
                                  dict(exact_backward=False)], ids=str)
def test_replayed_steps_of_moving_cameras_equal_eager_ones(ctx, form):
    """From the second step on the trainer replays a captured graph, whose cameras
    come from the call: images bit for bit, gradients to the atomics' rounding."""
    V, W, H, n = 2, 90, 61, 3000
    g = GpuSplatBuffer.upload(ctx, random_scene(n, 3))
    _, replayed = _grad_stepper(ctx, g, V, W, H, **form)
    _, eager = _grad_stepper(ctx, g, V, W, H, use_graph=False, **form)
    for k in range(5):
        cams = [CameraUniform.from_pose(*orbit_pose(40.0 * k + 100.0 * v), FOV_Y, W, H, n) for v in range(V)]
        (ga, ia, la), (gb, ib, lb) = replayed(cams), eager(cams)
        assert np.array_equal(ia, ib) and abs(la - lb) <= 1e-9 * abs(lb)
        assert np.linalg.norm(gb) > 0 and np.linalg.norm(ga - gb) <= 1e-5 * np.linalg.norm(gb)


@pytest.mark.parametrize("sort_mode", [0, 1])
def test_a_replayed_step_that_outgrows_its_lists_runs_again(ctx, sort_mode):
    """Cameras that look away from the scene, replayed, then ones that see 200000
    splats: the lists do not fit, the step grows them and runs again, and equals
    a fresh trainer's."""
    W, H, n = 512, 384, 200_000
    g = GpuSplatBuffer.upload(ctx, random_scene(n, 8))
    eye, tgt, up = (np.asarray(a, np.float64) for a in orbit_pose(15.0))
    near = CameraUniform.from_pose(eye, tgt, up, FOV_Y, W, H, n)
    away = CameraUniform.from_pose(eye, 2 * eye - tgt, up, FOV_Y, W, H, n)
    tr, step = _grad_stepper(ctx, g, 1, W, H, sort_mode=sort_mode)
    for _ in range(4):
        step([away])
    assert tr.stats()["pairs"] < 1000
    kernels, launched = tr.stats()["kernels_per_step"], ctx.launch_count
    ga, ia, la = step([near])
    assert tr.stats()["pairs"] > 100_000
    assert ctx.launch_count - launched >= 2 * kernels - 2
    gb, ib, lb = _grad_stepper(ctx, g, 1, W, H, sort_mode=sort_mode)[1]([near])
    assert np.array_equal(ia, ib) and abs(la - lb) <= 1e-9 * abs(lb)
    assert np.linalg.norm(ga - gb) <= 1e-5 * np.linalg.norm(gb)
    gc, ic, _ = step([near])
    assert np.array_equal(ic, ib) and np.linalg.norm(gc - gb) <= 1e-5 * np.linalg.norm(gb)
