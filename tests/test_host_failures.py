"""Host paths that a GPU test must not bring about: allocations that fail in
the middle of a step, and the sizes of arrays that kernels read.  The library's
own objects are linked with a CUDA runtime whose device memory is host memory
(fake_cudart.cpp) and run in a child process; no kernel runs."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PRELUDE = """
import numpy as np
from nanotracer_b200 import AdamMomentBuffers, CameraUniform, CudaCtx, GpuSplatBuffer, TilingParams
from nanotracer_b200._lib import SplatCudaError, lib
from nanotracer_b200.scene import FOV_Y, orbit_pose, random_scene
from nanotracer_b200.train import TrainConfig, Trainer
import ctypes as C
L = lib()
for f in (L.fake_bad, L.fake_composites, L.fake_replays, L.fake_pool_cap, L.fake_live):
    f.restype = C.c_uint64
L.fake_step.argtypes = [C.c_uint64, C.c_uint64, C.c_uint32, C.c_uint32]
L.fake_scan_total.argtypes = [C.c_uint64]
CAPACITY, TAKERS = 2, 4
ctx = CudaCtx(0)
scene = random_scene(300, 1)
W, H = 64, 48
cam = CameraUniform.from_pose(*orbit_pose(10.0), FOV_Y, W, H, 300)

def trainer(**kw):
    cfg = TrainConfig(n_views=1, width=W, height=H, depth_max=8.0, **kw)
    g = GpuSplatBuffer.upload(ctx, scene)
    mo = AdamMomentBuffers(ctx, g.capacity)
    acc = ctx.storage_buffer_zeroed("acc", 4 * g.capacity)
    tr = Trainer(ctx, cfg)
    tr.set_targets(ctx.storage_buffer_zeroed("targets", 12 * W * H))
    n = [0]
    def step():
        n[0] += 1
        return tr.step(g, mo, acc, [cam], n[0])
    return tr, step
"""


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    from nanotracer_b200 import build
    build.build()
    out = tmp_path_factory.mktemp("fake") / "libsplatcuda_fake.so"
    cuda = Path(build._nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I", str(cuda),
                    str(Path(__file__).with_name("fake_cudart.cpp")), *map(str, sorted(build.BUILD.glob("*.o"))),
                    "-o", str(out)], check=True)
    return out


def run(fake_lib, body):
    r = subprocess.run([sys.executable, "-c", PRELUDE + body], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "SPLATCUDA_LIB": str(fake_lib), "PYTHONPATH": str(ROOT)})
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("sort_mode", [0, 1])
@pytest.mark.parametrize("nth", [1, 2])
def test_a_step_after_a_failed_growth_of_the_takers_runs_on_live_chunks(fake_lib, sort_mode, nth):
    """A step draws more chunks than there are, and the larger arrays cannot be
    had (the first or the second of them): the call fails, and the next steps
    blend into chunks that are there and grow them as soon as they can."""
    run(fake_lib, f"""
tr, step = trainer(sort_mode={sort_mode})
step(), step()
L.fake_step(0, 0, TAKERS, 5000)
L.fake_fail({nth})
try:
    step()
    raise SystemExit("the failed allocation was not reported")
except SplatCudaError as e:
    assert e.status == 2, e
step()
assert L.fake_bad() == 0, "a blend ran without its chunks"
L.fake_step(0, 0, TAKERS, 5000)
step()
assert L.fake_bad() == 0 and L.fake_pool_cap() >= 5000
""")


@pytest.mark.parametrize("sort_mode", [0, 1])
def test_list_arrays_end_on_a_whole_group_of_four_words_in_the_trainer(fake_lib, sort_mode):
    """The blends read their lists in 16-byte groups, the last of which may reach
    beyond the list: into the array's own bytes, whatever count sized it."""
    run(fake_lib, f"""
tr, step = trainer(sort_mode={sort_mode})
step()
for n in (65537, 200002, 700003):
    L.fake_step(n, n, CAPACITY, 0)  # sizes the arrays for n + n / 4 + 65536 words
    step()
assert L.fake_composites() >= 4 and L.fake_bad() == 0
""")


def test_list_arrays_end_on_a_whole_group_of_four_words_in_the_binner(fake_lib):
    run(fake_lib, """
from nanotracer_b200 import Rasterizer, TileBinner
g = GpuSplatBuffer.upload(ctx, scene)
r, tl = Rasterizer(ctx), TilingParams(W, H, 16, 8.0)
proj, img = r.alloc_projected(g), r.alloc_image(W, H)
for n in (1, 101, 4002, 70003):
    L.fake_scan_total(n)  # sizes the arrays for n + n / 8 + 1024 words
    bins = TileBinner(ctx).bin(proj, 300, tl, stride=g.capacity)
    r.composite(proj, bins, img, tl, g.capacity)
assert L.fake_composites() == 4 and L.fake_bad() == 0
""")


@pytest.mark.parametrize("sort_mode", [0, 1])
def test_steps_of_the_same_inputs_replay_a_graph_and_others_do_not(fake_lib, sort_mode):
    """The first step sizes the arrays, the second is captured, and the graph is
    launched from then on; a store that takes a freed one's place in memory with
    another capacity, and stores taken in turn, are launched afresh."""
    run(fake_lib, f"""
tr, step = trainer(sort_mode={sort_mode})
for k in range(5):
    step()
    assert L.fake_replays() == k, (k, L.fake_replays())
def arrays(capacity):
    g = GpuSplatBuffer.upload(ctx, scene, capacity=capacity)
    mo = AdamMomentBuffers(ctx, 4096)
    return g, mo
acc, far = ctx.storage_buffer_zeroed("acc", 4 * 4096), arrays(2048)
g, mo = arrays(512)
r0 = L.fake_replays()
for t in (1, 2):
    tr.step(g, mo, acc, [cam], t)
assert L.fake_replays() == r0 + 1
g.free()
again = GpuSplatBuffer.upload(ctx, scene, capacity=1024)
tr.step(again, mo, acc, [cam], 3)
assert L.fake_replays() == r0 + 1, "a graph of another capacity was replayed"
for t in range(4, 8):
    tr.step(*((again, mo) if t % 2 else far), acc, [cam], t)
assert L.fake_replays() == r0 + 1
# an overflow in a replayed step: the arrays grow, and the step runs again
tr.step(*far, acc, [cam], 8), tr.step(*far, acc, [cam], 9)
r1, c1 = L.fake_replays(), L.fake_composites()
L.fake_step(300001, 300001, CAPACITY, 0)
L.fake_step(300001, 300001, TAKERS, 3000)
L.fake_step(300001, 300001, 0, 3000)
tr.step(*far, acc, [cam], 10)
assert (L.fake_replays() - r1, L.fake_composites() - c1) == (3, 3) and L.fake_pool_cap() >= 3000
assert L.fake_bad() == 0
""")


def test_many_scenes_replay_a_graph(fake_lib):
    run(fake_lib, """
from nanotracer_b200.scenes import Scene, ScenesTrainer
tr = ScenesTrainer(ctx, 2, W, H)
for i in range(2):
    g = GpuSplatBuffer.upload(ctx, scene)
    tr.set_scene(i, Scene(g, AdamMomentBuffers(ctx, g.capacity), ctx.storage_buffer_zeroed("a", 4 * g.capacity),
                          W, H, ctx.storage_buffer_zeroed("t", 12 * W * H)))
for t in range(1, 6):
    tr.step([cam, cam], t)
assert L.fake_replays() == 4 and L.fake_bad() == 0
""")


def test_trainers_and_views_share_the_contexts_page_locked_slots(fake_lib):
    """More of them than there are slots, taken and given back in any order, and
    the context closed while one lives: each reads its own results, and all
    memory comes back."""
    run(fake_lib, """
import gc
from nanotracer_b200.view import HeadlessView, OrbitCamera
base = L.fake_live()
trainers = [trainer() for _ in range(20)]
for k, (tr, step) in enumerate(trainers):
    L.fake_step(100 + k, 0, 0, 0)
    step()
assert [tr.stats()["pairs"] for tr, _ in trainers] == [100 + k for k in range(20)]
views = [HeadlessView(ctx, scene, W, H) for _ in range(3)]
del trainers[::2], tr, step
gc.collect()
views += [HeadlessView(ctx, scene, W, H) for _ in range(12)]
for v in views:
    v.frame(OrbitCamera())
for k, (tr, step) in enumerate(trainers):
    step()
assert L.fake_bad() == 0
del views, v, trainers, tr, step
gc.collect()
assert L.fake_live() == base, (L.fake_live(), base)
tr, _ = trainer()
handle, ctx2 = tr.handle, ctx.handle
tr.handle = None
gc.collect()
lib().sc_ctx_destroy(ctx2)
ctx.handle = None
lib().sc_trainer_free(None, handle)
""")
