"""Headless forward path of the viewer: the compute pass of nano-view's frame
(crates/nano-view/src/lib.rs:762-795) — CameraUniform from the orbit pose,
project, bin with 16x16 tiles and depth_max = max(4 * orbit distance, 50),
composite, tonemap — into an RGBA8 device buffer instead of a swapchain
texture.  There is no window here; frame() returns the pixels."""
from __future__ import annotations

import ctypes as C
import math
from dataclasses import dataclass, field

import numpy as np

from ._lib import check, lib, ptr
from .gpu import CudaCtx
from .raster import CameraUniform, Rasterizer
from .splat_gpu import GpuSplatBuffer
from .splat_store import SplatBuffer
from .tile_binner import TilingParams


@dataclass
class OrbitCamera:
    """nano-view's OrbitCamera (lib.rs:152-169): spherical pose around a target."""

    target: np.ndarray = field(default_factory=lambda: np.zeros(3, np.float32))
    distance: float = 4.0
    azimuth: float = 0.0
    elevation: float = 0.0
    fov_y: float = math.radians(50.0)

    def position(self) -> np.ndarray:
        # lib.rs:161-168, in f32
        ce = np.float32(math.cos(np.float32(self.elevation)))
        d = np.float32(self.distance)
        t = np.asarray(self.target, np.float32)
        return np.array([t[0] + d * ce * np.float32(math.cos(np.float32(self.azimuth))),
                         t[1] + d * np.float32(math.sin(np.float32(self.elevation))),
                         t[2] + d * ce * np.float32(math.sin(np.float32(self.azimuth)))], np.float32)


class HeadlessView:
    """One viewport: the device splat store plus the per-frame buffers."""

    TILE = 16

    def __init__(self, ctx: CudaCtx, splats: SplatBuffer | GpuSplatBuffer, width: int, height: int):
        self.ctx = ctx
        self.splats = splats if isinstance(splats, GpuSplatBuffer) else GpuSplatBuffer.upload(ctx, splats)
        self.width, self.height = int(width), int(height)
        self.rasterizer = Rasterizer(ctx)
        self.projected = ctx.storage_buffer_zeroed("projected", 48 * lib().sc_view_records(self.splats.handle))
        self.image = self.rasterizer.alloc_image(self.width, self.height, 1)
        self.rgba8 = ctx.storage_buffer_zeroed("rgba8", 4 * self.width * self.height)
        self._view = None
        t, h = self._params(0.0).struct(), C.c_void_p()
        check(lib().sc_view_create(ctx.handle, C.byref(t), C.byref(h)), ctx.handle)
        self._view = h  # the library's working arrays, kept from frame to frame

    def _params(self, depth_max: float) -> TilingParams:
        return TilingParams(self.width, self.height, self.TILE, depth_max)

    def tiling(self, orbit: OrbitCamera) -> TilingParams:
        return self._params(max(orbit.distance * 4.0, 50.0))

    def frame(self, orbit: OrbitCamera) -> np.ndarray:
        """Render one frame; returns (height, width, 4) uint8 (sRGB, alpha = coverage)."""
        n = self.splats.n
        cam = CameraUniform.from_pose(orbit.position(), np.asarray(orbit.target, np.float32), (0.0, 1.0, 0.0),
                                      orbit.fov_y, self.width, self.height, n)
        params = self.tiling(orbit)
        out = np.empty((self.height, self.width, 4), np.uint8)
        check(lib().sc_view_frame(self._view, self.splats.handle, C.byref(cam.c), float(params.depth_max),
                                  self.projected.cptr, self.image.cptr, self.rgba8.cptr, ptr(out)), self.ctx.handle)
        return out

    def hdr(self) -> np.ndarray:
        """The last frame before tonemapping: (height, width, 4) float32 (rgb, 1 - T)."""
        return self.image.readback(np.float32).reshape(self.height, self.width, 4)

    def __del__(self):
        try:
            if self._view and self.ctx.handle:
                lib().sc_view_free(self.ctx.handle, self._view)
                self._view = None
        except Exception:
            pass
