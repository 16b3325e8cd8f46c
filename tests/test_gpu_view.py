"""The headless viewer frame (view.py, nano-view/src/lib.rs:762-795):
project -> bin (REF32 keys, depth_max = max(4 d, 50)) -> composite -> tonemap,
against the oracle's forward on the same projected records."""
import math

import numpy as np
import pytest

from nanotracer_b200.scene import random_scene
from nanotracer_b200.view import HeadlessView, OrbitCamera


def _tonemap(img):
    def srgb(c):
        c = np.clip(c, 0, 1)
        return np.where(c > 0.0031308, 1.055 * c ** (1 / 2.4) - 0.055, c * 12.92)
    rgb = img[..., :3] / (1 + np.maximum(img[..., :3], 0))
    return np.concatenate([np.round(np.clip(srgb(rgb), 0, 1) * 255), np.round(np.clip(img[..., 3:], 0, 1) * 255)], -1)


def test_orbit_camera_position():
    o = OrbitCamera(target=np.array([1, 2, 3], np.float32), distance=2.0, azimuth=0.0, elevation=math.pi / 2)
    assert np.allclose(o.position(), [1, 4, 3], atol=1e-6)
    o = OrbitCamera(distance=3.0, azimuth=math.pi / 2, elevation=0.0)
    assert np.allclose(o.position(), [0, 0, 3], atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("azimuth,elevation", [(0.3, 0.2), (2.0, -0.4)])
def test_frame_matches_oracle_forward(ctx, oracle, azimuth, elevation):
    W, H = 320, 200
    scene = random_scene(4000, 17)
    view = HeadlessView(ctx, scene, W, H)
    orbit = OrbitCamera(distance=4.0, azimuth=azimuth, elevation=elevation)
    px = view.frame(orbit)
    hdr = view.hdr()
    assert px.shape == (H, W, 4) and px.dtype == np.uint8
    assert np.abs(px.astype(int) - _tonemap(hdr).astype(int)).max() <= 1
    # the oracle composites the device's projected records with its own REF32 binning
    rec = view.projected.readback(np.float32).reshape(-1, 12)[: len(scene)]
    tl = oracle.tiling(W, H, 16, 16, max(4.0 * 4.0, 50.0))
    _, pay, ranges = oracle.bin_ref(rec, tl)
    want, _, _ = oracle.composite(rec, pay, ranges, tl)
    assert np.mean(np.abs(hdr - want) <= 1e-4) > 0.999
    assert (hdr[..., 3] > 0).mean() > 0.05  # something was drawn


@pytest.mark.gpu
@pytest.mark.parametrize("n,size,distance", [(1, (16, 16), 4.0), (300, (33, 17), 1.5), (20000, (333, 211), 2.2),
                                             (20000, (64, 800), 30.0)])
def test_frame_equals_the_stage_calls_bit_for_bit(ctx, n, size, distance):
    """The one-call frame blends the splats of sc_bin's REF32 lists in their
    order: the image before and after tonemapping, and the records, are those of
    project -> bin -> composite -> tonemap, from one frame to the next (the
    item buffers grow on the way) and with the store's FP64 determinant option."""
    from nanotracer_b200 import CameraUniform, TilingParams
    from tests.util import GpuPipe
    W, H = size
    scene = random_scene(n, n + 3)
    view = HeadlessView(ctx, scene, W, H)
    try:
        for k, (az, el) in enumerate([(0.3, 0.2), (2.5, -0.5), (4.0, 0.9)]):
            ctx.set_fp64_det(k == 2)
            orbit = OrbitCamera(distance=distance, azimuth=az, elevation=el)
            px = view.frame(orbit)
            cam = CameraUniform.from_pose(orbit.position(), orbit.target, (0.0, 1.0, 0.0), orbit.fov_y, W, H, n)
            pipe = GpuPipe(ctx, scene, cam, TilingParams(W, H, 16, max(4.0 * distance, 50.0)))
            rec = pipe.project()[0]
            pipe.bin()
            img, _ = pipe.composite()
            assert np.array_equal(view.hdr(), img[0])
            assert np.array_equal(view.projected.readback(np.float32).reshape(-1, 12)[:n], rec)
            out = ctx.storage_buffer_zeroed("rgba8", 4 * W * H)
            pipe.r.tonemap(pipe.img, W, H, out)
            assert np.array_equal(px, out.readback(np.uint8).reshape(H, W, 4))
    finally:
        ctx.set_fp64_det(False)


@pytest.mark.gpu
def test_frame_shows_a_splat_of_nan_opacity_as_the_stage_calls_do(ctx):
    """A NaN alpha is clamped to 0.99 by the blend: such a splat covers its
    rectangle's pixels in the stage calls, and so it does in the frame."""
    from nanotracer_b200 import CameraUniform, TilingParams
    from tests.util import GpuPipe
    W, H, n = 120, 75, 40
    scene = random_scene(n, 5)
    scene.opacities[::9] = np.nan
    view = HeadlessView(ctx, scene, W, H)
    orbit = OrbitCamera(distance=3.0, azimuth=0.7, elevation=0.1)
    view.frame(orbit)
    cam = CameraUniform.from_pose(orbit.position(), orbit.target, (0.0, 1.0, 0.0), orbit.fov_y, W, H, n)
    pipe = GpuPipe(ctx, scene, cam, TilingParams(W, H, 16, 50.0))
    rec = pipe.project()[0]
    pipe.bin()
    img, _ = pipe.composite()
    assert (np.isnan(rec[:, 11]) & (rec[:, 7] != 0)).any()
    assert np.array_equal(view.hdr(), img[0])
