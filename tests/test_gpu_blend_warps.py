"""The blends at the sizes where a warp's own walk can go wrong: tile shapes
that split into 8 x 8 blocks, whole rows or single pixels per thread, images
that cut tiles, lists shorter than a stage, of a whole number of stages and
much longer, and warps that take more entries than the trainer first has room
for.

The trainer's backward walks the entries that its forward wrote down, the
stage calls' backward walks the lists; both form the same terms (the same
instructions) and add them in float in another order, so their projected
gradients agree to float rounding: a sum of m terms differs by at most
m 2^-24 of the terms' magnitudes, and sqrt(m) of that in the mean — 1e-5 of the
norm for the few thousand terms here.  The stage calls themselves are held to
the oracle as in the other parity tests."""
import ctypes as C

import numpy as np
import pytest

from nanotracer_b200 import (AdamMomentBuffers, CameraUniform, GpuSplatBuffer, GradSplatBuffers, Rasterizer, TileBinner,
                             TilingParams)
from nanotracer_b200._lib import SC_BWD_EXACT, SC_BWD_REF, SC_KEYS_REF32, check, lib
from nanotracer_b200.raster import cameras_array
from nanotracer_b200.scene import FOV_Y, orbit_pose, random_scene
from nanotracer_b200.train import TrainConfig, Trainer
from tests.util import GpuPipe, check_pg_explained, margins

pytestmark = pytest.mark.gpu

# (tile_w, tile_h): 8 x 8 blocks; a warp of whole rows; a tile width that is no
# multiple of 8; one pixel per thread (odd height)
TILES = [(16, 16), (8, 8), (32, 8), (32, 2), (4, 16), (32, 3)]


def _scene(n, opaque=True):
    s = random_scene(n, 7 * n + 1)
    if not opaque:  # wide and faint: every pixel takes nearly every splat
        s.scales[:] = np.log(0.6)
        s.opacities[:] = -4.0
    return s


def _targets(W, H):
    y, x = np.mgrid[0:H, 0:W]
    return np.stack([0.5 + 0.4 * np.sin(0.1 * x), 0.5 + 0.4 * np.cos(0.07 * y), 0.3 + 0.002 * (x + y) % 0.5],
                    -1).astype(np.float32)[None]


def _stage_grads(ctx, scene, cam, tl, tgt, W, H):
    """Parameter gradient rows (59, n) and the image through the stage calls (exact mode)."""
    pipe = GpuPipe(ctx, scene, cam, tl)
    pipe.project(), pipe.bin()
    img, _ = pipe.composite()
    pipe.backward((np.concatenate([img[..., :3] - tgt, np.zeros_like(img[..., :1])], -1) *
                   np.float32(2.0 / (3.0 * W * H))).astype(np.float32), SC_BWD_EXACT)
    grads = GradSplatBuffers(ctx, pipe.g.capacity)
    pipe.r.project_backward(pipe.g, pipe.pg, cam, grads)
    return grads.readback(len(scene)).flat().T, img[0]


def _trainer_grads(ctx, scene, cam, cfg, tgt):
    n = len(scene)
    g = GpuSplatBuffer.upload(ctx, scene)
    tr = Trainer(ctx, cfg)
    tr.set_targets(ctx.storage_buffer("t", tgt))
    shard = (n + 63) // 64 * 64
    out = ctx.storage_buffer_zeroed("grads", 59 * shard * 4)
    loss = C.c_double()
    for _ in range(2):  # the sizing step, then the captured one
        check(lib().sc_trainer_step_grads(tr.handle, g.handle, cameras_array([cam]), 1.0, 1, shard, out.cptr,
                                          C.byref(loss)), ctx.handle)
    return out.readback(np.float32, 59 * shard).reshape(59, shard)[:, :n], tr.images()[0]


@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("n,opaque,size", [(1, True, (33, 17)), (31, False, (40, 24)), (32, False, (40, 24)),
                                           (33, False, (61, 35)), (700, False, (50, 30)), (4000, True, (203, 117))])
def test_trainer_backward_over_the_takers_equals_the_list_backward(ctx, tile, n, opaque, size):
    W, H = size
    scene = _scene(n, opaque)
    cam = CameraUniform.from_pose(*orbit_pose(20.0), FOV_Y, W, H, n)
    tl = TilingParams(W, H, tile[0], 8.0, tile_h_override=tile[1])
    tgt = _targets(W, H)
    want, img = _stage_grads(ctx, scene, cam, tl, tgt, W, H)
    cfg = TrainConfig(n_views=1, width=W, height=H, tile_w=tile[0], tile_h=tile[1], depth_max=8.0, tile_cull=False)
    got, timg = _trainer_grads(ctx, scene, cam, cfg, tgt)
    assert np.array_equal(img, timg)
    for lo, hi in [(0, 3), (3, 7), (7, 10), (10, 11), (11, 14), (14, 59)]:
        d = np.linalg.norm((got[lo:hi] - want[lo:hi]).astype(np.float64))
        assert d <= 1e-5 * np.linalg.norm(want[lo:hi].astype(np.float64)) + 1e-30, (lo, d)


def _faint(n):
    """Wide and so faint that no pixel saturates: a warp takes a quarter of them
    or more, over 40 chunks of 32 where a new trainer has room for some 70 in
    a pool of one tile's warps."""
    s = _scene(n)
    s.scales[:] = np.log(0.6)
    s.opacities[:] = -5.0
    return s


@pytest.mark.parametrize("tile", [(16, 16), (8, 8), (32, 3)])
def test_a_step_that_takes_more_entries_than_there_is_room_for_runs_again(ctx, tile):
    """The forward runs out of chunks: the step's backward and Adam are skipped,
    the pools grow to the counted need and the step runs again.  Its gradients
    are the list backward's, and a training step's parameters and moments those
    of a trainer that had the room already (its second step; moments and
    parameters start from the same values)."""
    n, W, H = 8000, 64, 48
    scene = _faint(n)
    cam = CameraUniform.from_pose(*orbit_pose(20.0), FOV_Y, W, H, n)
    tl = TilingParams(W, H, tile[0], 8.0, tile_h_override=tile[1])
    tgt = _targets(W, H)
    want, img = _stage_grads(ctx, scene, cam, tl, tgt, W, H)
    cfg = TrainConfig(n_views=1, width=W, height=H, tile_w=tile[0], tile_h=tile[1], depth_max=8.0, tile_cull=False)
    g = GpuSplatBuffer.upload(ctx, scene)
    tr = Trainer(ctx, cfg)
    tr.set_targets(ctx.storage_buffer("t", tgt))
    shard = (n + 63) // 64 * 64
    out = ctx.storage_buffer_zeroed("grads", 59 * shard * 4)
    loss = C.c_double()

    def grad_step():
        before = ctx.launch_count
        check(lib().sc_trainer_step_grads(tr.handle, g.handle, cameras_array([cam]), 1.0, 1, shard, out.cptr,
                                          C.byref(loss)), ctx.handle)
        return ctx.launch_count - before

    runs = [grad_step() for _ in range(3)]
    kernels = tr.stats()["kernels_per_step"]
    assert runs[0] == 2 * kernels and runs[1:] == [kernels, kernels], (runs, kernels)
    got = out.readback(np.float32, 59 * shard).reshape(59, shard)[:, :n]
    assert np.array_equal(img, tr.images()[0])
    for lo, hi in [(0, 3), (3, 7), (7, 10), (10, 11), (11, 14), (14, 59)]:
        d = np.linalg.norm((got[lo:hi] - want[lo:hi]).astype(np.float64))
        assert d <= 1e-5 * np.linalg.norm(want[lo:hi].astype(np.float64)), (lo, d)

    def train_step(trainer):
        gs = GpuSplatBuffer.upload(ctx, scene)
        mo = AdamMomentBuffers(ctx, gs.capacity)
        acc = ctx.storage_buffer_zeroed("acc", 4 * gs.capacity)
        before = ctx.launch_count
        ls = trainer.step(gs, mo, acc, [cam], 1)
        m, v = mo.download(n)
        return ctx.launch_count - before, ls, gs.readback().flat(), m.flat().astype(np.float64), v.flat(), \
            acc.readback(np.float32, n)

    fresh = Trainer(ctx, cfg)
    fresh.set_targets(ctx.storage_buffer("t", tgt))
    la, lossa, pa, ma, va, aa = train_step(fresh)
    lb, lossb, pb, mb, vb, ab = train_step(fresh)
    assert la >= 2 * lb - 2 and abs(lossa - lossb) <= 1e-9 * lossb
    assert np.linalg.norm(ma - mb) <= 1e-5 * np.linalg.norm(mb)
    assert np.linalg.norm((va - vb).astype(np.float64)) <= 2e-5 * np.linalg.norm(vb.astype(np.float64))
    assert np.allclose(aa, ab, rtol=1e-3, atol=1e-5 * ab.max())
    # the first Adam step moves a parameter by lr times its gradient's sign: where
    # the gradient stands above its rounding, both moved alike
    clear = np.abs(mb) > 1e-3 * np.abs(mb).max(axis=0)
    assert np.allclose(pa[clear], pb[clear], rtol=1e-6, atol=1e-7) and clear.mean() > 0.3


@pytest.mark.parametrize("mode", [SC_BWD_EXACT, SC_BWD_REF])
@pytest.mark.parametrize("tile", TILES)
def test_list_backward_against_the_oracle_for_every_warp_layout(ctx, oracle, tile, mode):
    n, W, H = 1500, 101, 67
    cam = CameraUniform.from_pose(*orbit_pose(35.0), FOV_Y, W, H, n)
    tl = TilingParams(W, H, tile[0], 8.0, tile_h_override=tile[1])
    pipe = GpuPipe(ctx, _scene(n), cam, tl)
    rec = pipe.project()[0]
    _, payloads, ranges = pipe.bin()
    img, aux = pipe.composite()
    rng = np.random.default_rng(5)
    dl = np.zeros((H, W, 4), np.float32)
    dl[..., :3] = rng.normal(0, 1e-3, (H, W, 3))
    pg = pipe.backward(dl[None], mode)[0]
    otl = oracle.tiling(W, H, tile[0], tile[1], 8.0)
    _, flags, _ = margins(oracle, rec, payloads, ranges, otl, mode)
    tfin = np.ascontiguousarray(aux[0, ..., 0]).view(np.float32)
    want, absum = oracle.composite_backward(rec, payloads, ranges.reshape(-1), otl, img[0].reshape(-1, 4),
                                            dl.reshape(-1, 4), mode, np.ascontiguousarray(aux[0, ..., 1]).reshape(-1),
                                            tfin.reshape(-1), want_abs=True)
    check_pg_explained(pg, want, absum, flags, label=f"tile {tile} mode {mode}")


@pytest.mark.parametrize("n,size", [(1200, (480, 320)), (2500, (640, 480))])
def test_trainer_backward_starts_heavy_tiles_first(ctx, n, size):
    """Images of more tiles than start at once, whose silhouette tiles take a
    few hundred faint splats and fall into the lists that the backward starts with:
    every tile is still walked exactly once."""
    W, H = size
    scene = _scene(n)
    scene.scales[:] = np.log(0.25)
    scene.opacities[:] = -3.0
    cam = CameraUniform.from_pose(*orbit_pose(20.0), FOV_Y, W, H, n)
    tl = TilingParams(W, H, 8, 8.0)
    tgt = _targets(W, H)
    want, img = _stage_grads(ctx, scene, cam, tl, tgt, W, H)
    cfg = TrainConfig(n_views=1, width=W, height=H, tile_w=8, tile_h=8, depth_max=8.0, tile_cull=False)
    got, timg = _trainer_grads(ctx, scene, cam, cfg, tgt)
    assert np.array_equal(img, timg)
    for lo, hi in [(0, 3), (3, 7), (7, 10), (10, 11), (11, 14), (14, 59)]:
        d = np.linalg.norm((got[lo:hi] - want[lo:hi]).astype(np.float64))
        assert d <= 1e-5 * np.linalg.norm(want[lo:hi].astype(np.float64)), (lo, d)


@pytest.mark.parametrize("mode", [SC_BWD_EXACT, SC_BWD_REF])
def test_a_splat_at_the_alpha_threshold_is_blended_at_its_centre(ctx, oracle, mode):
    """The blend takes alpha >= 1/255; a splat of exactly that opacity reaches
    it at a pixel on its centre (g = 1), one float below it nowhere."""
    W, H = 33, 19
    at = np.float32(1.0) / np.float32(255.0)
    rec = np.zeros((2, 12), np.float32)
    for k, (x, op) in enumerate([(8.5, at), (24.5, np.nextafter(at, np.float32(0)))]):
        rec[k] = [x, 9.5, 1.0, 6.0, 0.4, 0.1, 0.3, 1.0, 0.9, 0.5, 0.2, op]
    tl = TilingParams(W, H, 16, 8.0)
    r, binner = Rasterizer(ctx), TileBinner(ctx)
    proj = ctx.storage_buffer("rec", rec)
    bins = binner.bin(proj, 2, tl, stride=2, n_views=1, key_mode=SC_KEYS_REF32)
    img, aux = r.alloc_image(W, H), r.alloc_aux(W, H)
    r.composite(proj, bins, img, tl, 2, 1, aux=aux)
    got = img.readback(np.float32).reshape(H, W, 4)
    otl = oracle.tiling(W, H, 16, 16, 8.0)
    _, pay, ranges = oracle.bin_ref(rec, otl)
    want, _, _ = oracle.composite(rec, pay, ranges, otl)
    want = np.asarray(want).reshape(H, W, 4)
    assert want[9, 8, 3] > 0 and (want[..., 3] > 0).sum() == 1
    assert np.allclose(got, want, rtol=0, atol=1e-7)
    dl = np.full((H, W, 4), 0.5, np.float32)
    pg = ctx.storage_buffer_zeroed("pg", rec.nbytes)
    r.composite_backward(proj, bins, img, ctx.storage_buffer("dl", dl), pg, tl, 2, 1, mode=mode, aux=aux)
    g = pg.readback(np.float32).reshape(2, 12)
    # one pixel at T = 1, dx = dy = 0: dcolor = alpha dL/dC, dopacity = dL/dC . colour
    assert np.allclose(g[0, 8:11], 0.5 * at, rtol=1e-6) and abs(g[0, 2] - 0.5 * 1.6) <= 1e-5
    assert not g[1].any()


@pytest.mark.parametrize("mode", [SC_BWD_EXACT, SC_BWD_REF])
@pytest.mark.parametrize("tile", TILES)
def test_a_gradient_that_is_not_finite_reaches_the_splats_of_its_pixel_only(ctx, tile, mode):
    """A pixel skips a splat by adding nothing to it: with dL/dC of NaN or
    infinity at two pixels, the projected gradients that are not finite are those
    of the splats that these pixels take, and the others are what they are with
    zeros there.  A splat whose record is NaN, which no pixel takes, gets zeros."""
    n, W, H = 900, 61, 45
    cam = CameraUniform.from_pose(*orbit_pose(35.0), FOV_Y, W, H, n)
    pipe = GpuPipe(ctx, _scene(n), cam, TilingParams(W, H, tile[0], 8.0, tile_h_override=tile[1]))
    rec = pipe.project()[0].copy()
    broken = np.arange(n) % 100 == 0
    rec[broken, :4] = np.nan, 20.0, 3.0, 40.0  # listed in tile column 0
    rec[broken, 7] = 1.0
    pipe.proj.upload(rec)
    _, pay, _ = pipe.bin()
    assert np.isin(np.flatnonzero(broken), pay).all()
    img, aux = pipe.composite()
    assert np.isfinite(img).all()
    dl = np.zeros((1, H, W, 4), np.float32)
    dl[..., :3] = np.random.default_rng(3).normal(0, 1e-3, (1, H, W, 3))
    spots = [(20, 30), (33, 17)]
    only = np.zeros_like(dl)
    for y, x in spots:
        dl[0, y, x, :3] = 0.0
        only[0, y, x, :3] = 1.0
    base = pipe.backward(dl, mode)[0]
    taken = pipe.backward(only, mode)[0][:, 8:11].any(axis=1)  # dcolor = sum T alpha dL/dC
    assert 0 < taken.sum() < n // 2
    for (y, x), bad in zip(spots, (np.nan, np.inf)):
        dl[0, y, x, :3] = bad
    got = pipe.backward(dl, mode)[0]
    assert not got[broken].any()
    assert not np.isfinite(got[taken]).all(axis=1).any()
    # the atomics' order differs between the runs
    scale = np.abs(base).max(axis=0)
    assert np.allclose(got[~taken], base[~taken], rtol=1e-4, atol=1e-6 * scale.max())
