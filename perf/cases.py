"""Performance cases: the work a user of the framework has it do, through its
public entry points.

Four kinds of call are covered:

  train    one iteration of the batched trainer (Trainer.step), from a small
           scene on a small image, where launches and latency count, to the
           1M-splat, 8-view 1080p iteration and a 3M-splat one; both storage
           forms, the MSE and the SSIM loss, plain and compensated sums, the
           three tile shapes
  scenes   one iteration over many scenes of uneven sizes (ScenesTrainer.step)
  frame    one viewer frame to host RGBA8 (HeadlessView.frame)
  stages   one iteration driven stage by stage through the rasteriser, binner
           and optimiser objects, as the reference's own host loop does it

Scenes have the synthetic benchmark's distributions (scene.py): means uniform
in [-1, 1]^3, quaternions and opacity logits normal, order-3 SH.  `log_sigma`
is the mean log-scale (0.03 for the benchmark scene; smaller splats are a scene
late in its training), `radius` the orbit's (4: the scene in the middle of the
image; 1.6: the scene fills it).  Targets are smooth synthetic photographs, so
that they depend on the seed alone.

Every state is a run under way: moments hold values, and the learning rates
are those of the end of a schedule (a thousandth of the first ones), so that a
scene, and with it the work, stays what it was from pass to pass.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import nanotracer_b200 as nt
from nanotracer_b200 import lib
from nanotracer_b200._lib import SC_BWD_EXACT, SC_BWD_REF, SC_KEYS_NATIVE64, SC_KEYS_REF32, check
from nanotracer_b200.scenes import Scene, ScenesTrainer
from nanotracer_b200.train import BENCH_LRS
from nanotracer_b200.view import HeadlessView, OrbitCamera

ROWS = 59
FOV_Y = math.radians(50.0)
LRS = tuple(1e-3 * x for x in BENCH_LRS)
BETA1, BETA2, EPS = 0.9, 0.999, 1e-15
T0 = 2000        # optimiser steps behind the state
MOMENT = 1e-7    # scale of the first moments (gradients of a mean over an image are this small)
DEPTH_MAX = 8.0


# ---------------------------------------------------------------- the cases
def _train(n, views, width, height, *, bf16=False, ssim=0.0, comp=False, tile_w=16, tile_h=16, sigma=0.03,
           radius=4.0):
    return {"kind": "train", "n": n, "views": views, "width": width, "height": height, "bf16": bf16, "ssim": ssim,
            "comp": comp, "tile_w": tile_w, "tile_h": tile_h, "sigma": sigma, "radius": radius}


def listed():
    return [
        # the configuration of a first try and of unit tests: one small image, latency counts
        dict(_train(5_000, 1, 256, 256), name="train_5k_256"),
        # an ordinary single-view iteration, the reference's train() shape
        dict(_train(200_000, 1, 1024, 1024), name="train_200k_1024"),
        # the plain form of the benchmark: one 1080p view per iteration, fp32
        dict(_train(1_000_000, 1, 1920, 1080), name="train_1m_1080p"),
        # the benchmark itself: 8 views of 1080p per iteration, bf16 storage
        dict(_train(1_000_000, 8, 1920, 1080, bf16=True), name="train_1m_1080p_8v_bf16"),
        # the precision form: 3M splats, 4 views, bf16 storage, compensated sums
        dict(_train(3_000_000, 4, 1920, 1080, bf16=True, comp=True), name="train_3m_1080p_4v_comp"),
        # the SSIM loss on photographs of an odd size (a scene that fills the image, small splats)
        dict(_train(333_333, 2, 1237, 822, ssim=0.2, sigma=0.012, radius=1.6), name="train_ssim_333k_1237x822_2v"),
        # uneven scenes, 10k-500k splats and three image sizes, in one step
        {"kind": "scenes", "name": "scenes_16", "scenes": 16, "lo": 10_000, "hi": 500_000, "sigma": 0.03},
        # the viewer: a frame of a finished scene on a 1080p window
        {"kind": "frame", "name": "frame_1m_1080p", "n": 1_000_000, "width": 1920, "height": 1080, "sigma": 0.015,
         "radius": 2.2},
        # a frame of a small scene in a small window
        {"kind": "frame", "name": "frame_20k_640x360", "n": 20_000, "width": 640, "height": 360, "sigma": 0.03,
         "radius": 4.0},
        # a host loop over the stage objects, one view, exact backward
        {"kind": "stages", "name": "stages_100k_800x600", "n": 100_000, "views": 1, "width": 800, "height": 600,
         "exact_bwd": True, "keys64": False, "sigma": 0.02, "radius": 3.0},
        # the same with the reference's backward and 64-bit keys, odd sizes, several views
        {"kind": "stages", "name": "stages_ref_61k_1013x571_3v", "n": 61_111, "views": 3, "width": 1013,
         "height": 571, "exact_bwd": False, "keys64": True, "sigma": 0.03, "radius": 4.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["train", "scenes", "frame", "stages"], [6, 1, 2, 3])[0]
    sigma = math.exp(rng.uniform(math.log(0.01), math.log(0.03)))
    radius = rng.choice([1.6, 2.2, 3.0, 4.0])
    width, height = _log_int(rng, 160, 1920), _log_int(rng, 120, 1080)
    if kind == "train":
        views = rng.choice([1, 1, 1, 2, 3, 4, 8])
        n = _log_int(rng, 3_000, min(1_000_000, 3_000_000 // views))
        tile_w, tile_h = rng.choice([(16, 16), (16, 16), (16, 16), (8, 8), (32, 8)])
        return _train(n, views, width, height, bf16=rng.random() < 0.5, ssim=rng.choice([0.0, 0.0, 0.2]),
                      comp=rng.random() < 0.15, tile_w=tile_w, tile_h=tile_h, sigma=sigma, radius=radius)
    if kind == "scenes":
        lo = _log_int(rng, 3_000, 30_000)
        return {"kind": "scenes", "scenes": rng.randint(2, 12), "lo": lo, "hi": lo * rng.randint(2, 10),
                "sigma": sigma}
    if kind == "frame":
        return {"kind": "frame", "n": _log_int(rng, 5_000, 1_000_000), "width": width, "height": height,
                "sigma": sigma, "radius": rng.choice([2.2, 3.0, 4.0])}
    return {"kind": "stages", "n": _log_int(rng, 3_000, 150_000), "views": rng.randint(1, 3),
            "width": min(width, 1100), "height": min(height, 700), "exact_bwd": rng.random() < 0.6,
            "keys64": rng.random() < 0.5, "sigma": sigma, "radius": max(radius, 2.2)}


# ---------------------------------------------------------------- what they cannot do without
def _param_bytes(bf16):
    return 14 * 4 + 45 * (2 if bf16 else 4)


def work(case):
    """Bytes: parameters and moments read and written once, targets read,
    images written.  Flops: about 400 per projected splat and view and its
    adjoint, and per pixel the blend of some 60 splats (17 operations forward,
    29 backward) where the path has them."""
    kind = case["kind"]
    if kind == "train":
        px = case["views"] * case["width"] * case["height"]
        state = 2 * _param_bytes(case["bf16"]) + 4 * ROWS * (2 if case["bf16"] else 4) + 8
        return {"bytes": case["n"] * (state + 4 * ROWS) + px * (16 + 12),
                "flops": case["n"] * (case["views"] * 1200 + ROWS * 12) + px * 60 * 46}
    if kind == "scenes":
        sizes = _scene_sizes(case)
        n = sum(s[0] for s in sizes)
        px = sum(s[1] * s[2] for s in sizes)
        return {"bytes": n * (2 * 236 + 4 * 236 + 8 + 4 * ROWS) + px * 28, "flops": n * (1200 + ROWS * 12) + px * 60 * 46}
    px = case["width"] * case["height"]
    if kind == "frame":
        return {"bytes": case["n"] * 236 + px * 4, "flops": case["n"] * 400 + px * 60 * 17}
    v = case["views"]
    return {"bytes": case["n"] * (2 * 236 + 4 * 236 + 8 + 12 * ROWS + v * 48) + v * px * (16 + 12 + 16),
            "flops": case["n"] * (v * 1200 + ROWS * 12) + v * px * 60 * 46}


# ---------------------------------------------------------------- inputs
_CTX = None


def _ctx():
    """One context per program."""
    global _CTX
    if _CTX is None:
        _CTX = nt.CudaCtx(0)
    return _CTX


class _Window:
    """A device buffer of the library seen as a tensor; the owners live as long as it does."""

    def __init__(self, ptr, shape, typestr, owners):
        self.owners = owners
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": typestr,
                                         "version": 3}


def _tensor(ptr, shape, *owners, typestr="<f4"):
    return torch.as_tensor(_Window(ptr, shape, typestr, owners), device="cuda")


def _gen(seed, stream):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1000 + stream)


def _rows(n, sigma, seed, stream=0):
    """Parameter rows (59, n): position, quaternion, log-scale, opacity logit, SH DC, SH rest."""
    g = _gen(seed, stream)
    p = torch.randn(ROWS, n, generator=g, device="cuda")
    p[0:3] = torch.rand(3, n, generator=g, device="cuda") * 2.0 - 1.0
    p[3:7] /= p[3:7].norm(dim=0, keepdim=True).clamp_min(1e-12)
    p[7:10] = p[7:10] * 0.3 + math.log(sigma)
    p[11:14] *= 0.3
    p[14:59] *= 0.05
    return p


def _splats(p):
    a = p.T.contiguous().cpu().numpy()
    return nt.SplatBuffer(a[:, 0:3], a[:, 3:7], a[:, 7:10], a[:, 10], a[:, 11:14], a[:, 14:59])


def _moment_rows(n, seed, stream=0):
    """First and second moments (2, 59, n)."""
    g = _gen(seed, 100 + stream)
    m = torch.randn(2, ROWS, n, generator=g, device="cuda") * MOMENT
    m[1] = m[1].square() * 0.25 + (0.5 * MOMENT) ** 2
    return m


def _moments(ctx, capacity, n, bf16, seed, stream=0):
    mo = nt.AdamMomentBuffers(ctx, capacity, bf16=bf16)
    rows = _moment_rows(n, seed, stream)
    torch.cuda.synchronize()
    check(lib().sc_moments_unpack_shards(ctx.handle, mo.handle, n, C.c_void_p(rows.data_ptr()), 1, n), ctx.handle)
    ctx.synchronize()
    return mo


def _photos(views, height, width, seed, stream=0):
    """Smooth images (views, height, width, 3) with values in [0, 1]."""
    g = _gen(seed, 200 + stream)
    out = torch.zeros(views, 3, height, width, device="cuda")
    for cells, weight in ((4, 0.5), (17, 0.3), (61, 0.2)):
        coarse = torch.rand(views, 3, cells, cells, generator=g, device="cuda")
        out += weight * torch.nn.functional.interpolate(coarse, size=(height, width), mode="bilinear",
                                                        align_corners=False)
    return out.permute(0, 2, 3, 1).contiguous()


def _device_copy(ctx, label, t):
    b = ctx.storage_buffer_zeroed(label, t.numel() * t.element_size())
    ctx.synchronize()
    _tensor(b.ptr, (t.numel(),), b).copy_(t.reshape(-1))
    torch.cuda.synchronize()
    return b


def _eye(v, views, radius):
    """Views spread around the orbit with a few degrees of elevation."""
    a, e = 2.0 * math.pi * v / views + 0.3, math.radians(10.0) * math.sin(1.7 * v + 0.5)
    return radius * math.cos(e) * math.sin(a), radius * math.sin(e), radius * math.cos(e) * math.cos(a)


def _cams(n, views, width, height, radius):
    return [nt.CameraUniform.from_pose(_eye(v, views, radius), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), FOV_Y, width, height,
                                       n) for v in range(views)]


def _scene_sizes(case):
    """(splats, width, height) of each scene: counts log-uniform over [lo, hi] by a fixed low-discrepancy sequence."""
    images = ((512, 512), (1024, 768), (1920, 1080))
    out = []
    for i in range(case["scenes"]):
        u = (0.5 + 0.6180339887498949 * i) % 1.0
        n = int(round(math.exp(math.log(case["lo"]) + u * math.log(case["hi"] / case["lo"]))))
        out.append((n,) + images[(i * 5 + 1) % 3])
    return out


# ---------------------------------------------------------------- train
def _prepare_train(case, seed):
    ctx = _ctx()
    n, v, w, h = case["n"], case["views"], case["width"], case["height"]
    g = nt.GpuSplatBuffer.upload(ctx, _splats(_rows(n, case["sigma"], seed)), bf16_rest=case["bf16"])
    mo = _moments(ctx, g.capacity, n, case["bf16"], seed)
    acc = ctx.storage_buffer_zeroed("grad_acc", 4 * g.capacity)
    cfg = nt.TrainConfig(n_views=v, width=w, height=h, tile_w=case["tile_w"], tile_h=case["tile_h"],
                         depth_max=DEPTH_MAX, lrs=LRS, bf16=case["bf16"], ssim_lambda=case["ssim"],
                         compensated_sums=case["comp"])
    tr = nt.Trainer(ctx, cfg)
    targets = _device_copy(ctx, "targets", _photos(v, h, w, seed))
    tr.set_targets(targets)
    packed = ctx.storage_buffer_zeroed("params", 4 * ROWS * n)
    ctx.synchronize()
    return {"kind": "train", "ctx": ctx, "tr": tr, "g": g, "mo": mo, "acc": acc, "targets": targets, "packed": packed,
            "cams": _cams(n, v, w, h, case["radius"]), "n": n, "shape": (v, h, w, 4), "t": T0}


def _pack_params(ctx, g, n, out):
    check(lib().sc_splats_pack_range(ctx.handle, g.handle, 0, n, n, out.cptr), ctx.handle)


def _run_train(s):
    s["t"] += 1
    loss = s["tr"].step(s["g"], s["mo"], s["acc"], s["cams"], s["t"])
    _pack_params(s["ctx"], s["g"], s["n"], s["packed"])
    return {"loss": np.float32(loss),  # a mean over f32 images
            "images": _tensor(s["tr"].images_ptr(), s["shape"], s["tr"], s["targets"]),
            "params": _tensor(s["packed"].ptr, (ROWS, s["n"]), s["packed"]),
            "grad_acc": _tensor(s["acc"].ptr, (s["n"],), s["acc"])}


# ---------------------------------------------------------------- scenes
def _prepare_scenes(case, seed):
    ctx = _ctx()
    sizes = _scene_sizes(case)
    st = ScenesTrainer(ctx, len(sizes), max(s[1] for s in sizes), max(s[2] for s in sizes), lrs=LRS,
                       depth_max=DEPTH_MAX)
    cams, packed = [], []
    for i, (n, w, h) in enumerate(sizes):
        g = nt.GpuSplatBuffer.upload(ctx, _splats(_rows(n, case["sigma"], seed, i)))
        mo = _moments(ctx, g.capacity, n, False, seed, i)
        acc = ctx.storage_buffer_zeroed("grad_acc", 4 * g.capacity)
        target = _device_copy(ctx, "target", _photos(1, h, w, seed, i))
        st.set_scene(i, Scene(g, mo, acc, w, h, target))
        cams += [nt.CameraUniform.from_pose(_eye(i, len(sizes), 4.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), FOV_Y, w, h,
                                            n)]
        packed.append(ctx.storage_buffer_zeroed("params", 4 * ROWS * n))
    ctx.synchronize()
    return {"kind": "scenes", "ctx": ctx, "st": st, "cams": cams, "packed": packed, "sizes": sizes, "t": T0}


def _run_scenes(s):
    s["t"] += 1
    st = s["st"]
    losses = st.step(s["cams"], s["t"])
    p = C.c_void_p()
    check(lib().sc_scenes_trainer_images(st.handle, C.byref(p)), s["ctx"].handle)
    images = _tensor(p.value, (st.n, st.max_height, st.max_width, 4), st)
    out = {"losses": losses.astype(np.float32), "images": [], "params": [], "grad_acc": []}
    for i, (n, w, h) in enumerate(s["sizes"]):
        sc = st.scenes[i]
        _pack_params(s["ctx"], sc.splats, n, s["packed"][i])
        out["images"].append(images[i, :h, :w])
        out["params"].append(_tensor(s["packed"][i].ptr, (ROWS, n), s["packed"][i]))
        out["grad_acc"].append(_tensor(sc.grad_acc.ptr, (n,), sc.grad_acc))
    return out


# ---------------------------------------------------------------- frame
def _prepare_frame(case, seed):
    ctx = _ctx()
    view = HeadlessView(ctx, _splats(_rows(case["n"], case["sigma"], seed)), case["width"], case["height"])
    orbit = OrbitCamera(distance=case["radius"], azimuth=0.1 + 0.37 * (seed % 17), elevation=0.2)
    ctx.synchronize()
    return {"kind": "frame", "view": view, "orbit": orbit, "image": view.image,
            "shape": (case["height"], case["width"], 4)}


def _run_frame(s):
    rgba8 = s["view"].frame(s["orbit"])
    return {"rgba8": rgba8, "hdr": _tensor(s["image"].ptr, s["shape"], s["image"])}


# ---------------------------------------------------------------- stages
def _prepare_stages(case, seed):
    ctx = _ctx()
    n, v, w, h = case["n"], case["views"], case["width"], case["height"]
    g = nt.GpuSplatBuffer.upload(ctx, _splats(_rows(n, case["sigma"], seed)))
    r = nt.Rasterizer(ctx)
    s = {"kind": "stages", "ctx": ctx, "g": g, "mo": _moments(ctx, g.capacity, n, False, seed),
         "grads": nt.GradSplatBuffers(ctx, g.capacity), "acc": ctx.storage_buffer_zeroed("grad_acc", 4 * g.capacity),
         "adam": nt.AdamGpu(ctx), "r": r, "binner": nt.TileBinner(ctx), "tl": nt.TilingParams(w, h, 16, DEPTH_MAX),
         "cams": _cams(n, v, w, h, case["radius"]), "proj": r.alloc_projected(g, v), "img": r.alloc_image(w, h, v),
         "aux": r.alloc_aux(w, h, v), "dl": ctx.storage_buffer_zeroed("dl_dc", v * w * h * 16),
         "pg": r.alloc_projected_grad(g, v), "targets": _device_copy(ctx, "targets", _photos(v, h, w, seed)),
         "packed": ctx.storage_buffer_zeroed("params", 4 * ROWS * n),
         "packed_mo": ctx.storage_buffer_zeroed("moments", 8 * ROWS * n),
         "mode": SC_BWD_EXACT if case["exact_bwd"] else SC_BWD_REF,
         "keys": SC_KEYS_NATIVE64 if case["keys64"] else SC_KEYS_REF32, "n": n, "v": v, "w": w, "h": h, "t": T0}
    ctx.synchronize()
    return s


def _run_stages(s):
    s["t"] += 1
    ctx, g, r, tl, n, v, w, h = (s[k] for k in ("ctx", "g", "r", "tl", "n", "v", "w", "h"))
    stride = g.capacity
    r.project(g, s["cams"], s["proj"])
    bins = s["binner"].bin(s["proj"], n, tl, stride=stride, n_views=v, key_mode=s["keys"])
    r.composite(s["proj"], bins, s["img"], tl, stride, v, aux=s["aux"])
    loss = r.mse_loss_grad(s["img"], s["targets"], tl, s["dl"], n_views=v, scale=1.0 / v)
    r.zero_projected_grad(s["pg"])
    r.composite_backward(s["proj"], bins, s["img"], s["dl"], s["pg"], tl, stride, v, mode=s["mode"], aux=s["aux"])
    for k in range(v):
        r.project_backward(g, s["pg"], s["cams"][k], s["grads"], accumulate=k > 0, view_offset=k * stride * 48)
    s["adam"].accumulate_grad(s["grads"], s["acc"], n)
    s["adam"].step_all(g, s["grads"], s["mo"], s["t"], nt.AdamConfig(beta1=BETA1, beta2=BETA2, eps=EPS), lrs=LRS)
    s["adam"].apply_constraints(g)
    _pack_params(ctx, g, n, s["packed"])
    check(lib().sc_moments_pack_range(ctx.handle, s["mo"].handle, 0, n, n, s["packed_mo"].cptr), ctx.handle)
    return {"loss": loss.astype(np.float32), "pairs": bins.total_pairs,
            "images": _tensor(s["img"].ptr, (v, h, w, 4), s["img"]),
            "dl_dc": _tensor(s["dl"].ptr, (v, h, w, 4), s["dl"]),
            "projected_grad": _tensor(s["pg"].ptr, (v, stride, 12), s["pg"])[:, :n],
            "moments": _tensor(s["packed_mo"].ptr, (2, ROWS, n), s["packed_mo"]),
            "params": _tensor(s["packed"].ptr, (ROWS, n), s["packed"]),
            "grad_acc": _tensor(s["acc"].ptr, (n,), s["acc"])}


# ---------------------------------------------------------------- entry points
def prepare(case, seed):
    return {"train": _prepare_train, "scenes": _prepare_scenes, "frame": _prepare_frame,
            "stages": _prepare_stages}[case["kind"]](case, seed)


def run(state):
    return {"train": _run_train, "scenes": _run_scenes, "frame": _run_frame,
            "stages": _run_stages}[state["kind"]](state)


# ---------------------------------------------------------------- in 64 bits
SH1 = 0.488602
SH2 = (1.0925485, -1.0925485, 0.31539157, -1.0925485, 0.54627424)
SH3 = (-0.5900436, 2.8906114, -0.4570458, 0.37317634, -0.4570458, 1.4453057, -0.5900436)
SH0 = 0.2820948


def _camera64(eye, target, height):
    """World-to-camera rotation rows (right, up, backward), translation and focal length, rounded to f32 as stored."""
    f32 = np.float32
    unit = lambda a: a / np.sqrt((a * a).sum(dtype=f32), dtype=f32)  # noqa: E731
    e, t = np.array(eye, f32), np.array(target, f32)
    f = unit(t - e)
    s = unit(np.cross(f, np.array([0, 1, 0], f32)).astype(f32))
    u = np.cross(s, f).astype(f32)
    rot = np.stack([s, u, -f]).astype(f32)
    tr = np.array([-(e * s).sum(dtype=f32), -(e * u).sum(dtype=f32), (e * f).sum(dtype=f32)], f32)
    focal = f32(height) / (f32(2.0) * np.tan(f32(FOV_Y) * f32(0.5), dtype=f32))
    d = lambda a: torch.tensor(np.asarray(a, np.float64), device="cuda")  # noqa: E731
    return d(rot), d(tr), float(focal), d(e)


def _project64(p, cam, width, height):
    """Projected splats of parameter rows p (59, n) in f64, differentiable the
    way the adjoint is defined: the covariance does not depend on the position,
    the view direction is a constant, and the colour's clamp passes gradients."""
    rot, tr, focal, eye = cam
    pos, q, ls = p[0:3], p[3:7], p[7:10]
    c = rot @ pos + tr[:, None]
    depth = -c[2]
    mx = width * 0.5 + focal * c[0] / depth
    my = height * 0.5 - focal * c[1] / depth
    cd = c.detach()
    w, x, y, z = q
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]).reshape(3, 3, -1)
    iz = -1.0 / cd[2]
    j0 = torch.stack([focal * iz, torch.zeros_like(iz), -focal * cd[0] * iz * iz])
    j1 = torch.stack([torch.zeros_like(iz), -focal * iz, focal * cd[1] * iz * iz])
    # the adjoint's sign convention for the depth axis: its rows act on (x, y, z) of the camera frame
    m0, m1 = torch.einsum("an,ab->bn", j0, rot), torch.einsum("an,ab->bn", j1, rot)
    sig = ls.exp()
    b0 = torch.einsum("bn,bcn->cn", m0, R) * sig
    b1 = torch.einsum("bn,bcn->cn", m1, R) * sig
    s00, s01, s11 = (b0 * b0).sum(0) + 0.3, (b0 * b1).sum(0), (b1 * b1).sum(0) + 0.3
    det = s00 * s11 - s01 * s01
    conic = torch.stack([s11 / det, -s01 / det, s00 / det])
    mid = (0.5 * (s00 + s11)).detach()
    radius = torch.ceil(3.0 * (mid + (mid * mid - det.detach()).clamp_min(0.0).sqrt()).sqrt())
    dvec = eye[:, None] - pos.detach()
    x, y, z = dvec / dvec.norm(dim=0, keepdim=True)
    xx, yy, zz = x * x, y * y, z * z
    basis = torch.stack([-SH1 * y, SH1 * z, -SH1 * x, SH2[0] * x * y, SH2[1] * y * z, SH2[2] * (2 * zz - xx - yy),
                         SH2[3] * x * z, SH2[4] * (xx - yy), SH3[0] * y * (3 * xx - yy), SH3[1] * x * y * z,
                         SH3[2] * y * (4 * zz - xx - yy), SH3[3] * z * (2 * zz - 3 * xx - 3 * yy),
                         SH3[4] * x * (4 * zz - xx - yy), SH3[5] * z * (xx - yy), SH3[6] * x * (xx - 3 * yy)])
    raw = SH0 * p[11:14] + (p[14:59].reshape(3, 15, -1) * basis).sum(1) + 0.5
    color = raw + (raw.clamp_min(0.0) - raw).detach()
    opacity = torch.sigmoid(p[10])
    big = max(width, height) + radius
    visible = ((depth >= 0.01) & (det > 0) & (mx >= -radius) & (mx < width + radius) & (my >= -radius) &
               (my < height + radius) & (radius < big))
    return mx, my, depth, radius, conic, color, opacity, visible.detach()


def _pairs64(mx, my, depth, radius, visible, width, height, keys64):
    """(tile, splat) pairs in the blend's order: by tile, then depth key, then splat."""
    tx, ty = -(-width // 16), -(-height // 16)
    x0 = ((mx - radius) / 16).floor().clamp_min(0).long()
    x1 = ((mx + radius) / 16).floor().clamp_max(tx - 1).long()
    y0 = ((my - radius) / 16).floor().clamp_min(0).long()
    y1 = ((my + radius) / 16).floor().clamp_max(ty - 1).long()
    nx, ny = (x1 - x0 + 1).clamp_min(0), (y1 - y0 + 1).clamp_min(0)
    cnt = torch.where(visible, nx * ny, torch.zeros_like(nx))
    key = depth.float().double() if keys64 else ((depth.float() / DEPTH_MAX).clamp(0, 1) * 65535.0).floor().double()
    order = torch.argsort(key, stable=True)
    order = order[cnt[order] > 0]
    c = cnt[order]
    ids = torch.repeat_interleave(order, c)
    k = torch.arange(ids.numel(), device=ids.device) - torch.repeat_interleave(c.cumsum(0) - c, c)
    tile = (y0[ids] + k // nx[ids]) * tx + x0[ids] + k % nx[ids]
    tile, at = torch.sort(tile, stable=True)
    counts = torch.bincount(tile, minlength=tx * ty)
    return ids[at], counts, counts.cumsum(0) - counts, tx


def _blend64(splat, ids, counts, starts, tx, width, height, dl_of=None):
    """The image (height, width, 4) and, with dl_of(image) -> dL/dC, the
    gradients of the splat tensor (9, n): mean, opacity, conic, colour."""
    dev = ids.device
    image = torch.zeros(height, width, 4, dtype=torch.float64, device=dev)
    grad = torch.zeros_like(splat)
    tiles = torch.argsort(counts)
    tiles = tiles[counts[tiles] > 0]
    lens = counts[tiles].tolist()
    px = torch.arange(256, device=dev)

    def groups():
        i = 0
        while i < len(lens):
            j = i + 1
            while j < len(lens) and (j + 1 - i) * lens[j] <= 60_000:
                j += 1
            yield tiles[i:j], lens[j - 1]
            i = j

    def forward(t, length, sp):
        slot = torch.arange(length, device=dev)
        have = slot[None] < counts[t][:, None]
        idx = ids[(starts[t][:, None] + slot[None]).clamp_max(ids.numel() - 1)]
        e = sp[:, idx]                                            # (9, tiles, length)
        gx = (t % tx * 16)[:, None] + px[None] % 16
        gy = (t // tx * 16)[:, None] + px[None] // 16
        dx = gx[:, None].double() + 0.5 - e[0][..., None]
        dy = gy[:, None].double() + 0.5 - e[1][..., None]
        quad = e[3][..., None] * dx * dx + 2 * e[4][..., None] * dx * dy + e[5][..., None] * dy * dy
        a = (e[2][..., None] * torch.exp(-0.5 * quad)).clamp_max(0.99)
        a = torch.where(have[..., None] & (quad >= 0) & (a >= 1.0 / 255.0), a, torch.zeros_like(a))
        logs = torch.log1p(-a)
        before = torch.exp(logs.cumsum(1) - logs)
        keep = before.detach() >= 1e-4                             # a pixel stops once its T is below
        wgt = torch.where(keep, a * before, torch.zeros_like(a))
        col = torch.einsum("tlp,ctl->tpc", wgt, e[6:9])
        left = torch.exp(torch.where(keep, logs, torch.zeros_like(logs)).sum(1))
        inside = (gx < width) & (gy < height)
        return col, left, gx, gy, inside

    image_groups = list(groups())
    with torch.no_grad():
        for t, length in image_groups:
            col, left, gx, gy, ok = forward(t, length, splat)
            image[gy[ok], gx[ok]] = torch.cat([col, (1.0 - left)[..., None]], -1)[ok]
    if dl_of is None:
        return image, None
    dl = dl_of(image)
    for t, length in image_groups:
        sp = splat.detach().requires_grad_(True)
        col, _, gx, gy, ok = forward(t, length, sp)
        (col[ok] * dl[gy[ok], gx[ok]]).sum().backward()
        grad += sp.grad
    return image, grad


def exact(case, seed):
    kind = case["kind"]
    if kind != "stages":
        return None  # whole iterations; a frame's floats are covered by the stages
    n, views, w, h = case["n"], case["views"], case["width"], case["height"]
    p = _rows(n, case["sigma"], seed).double()
    targets = _photos(views, h, w, seed).double()
    images, dls, pgs, losses, pairs = [], [], [], [], 0
    total = torch.zeros_like(p)
    for v in range(views):
        cam = _camera64(_eye(v, views, case["radius"]), (0.0, 0.0, 0.0), h)
        pv = p.detach().requires_grad_(True)
        mx, my, depth, radius, conic, color, opacity, visible = _project64(pv, cam, w, h)
        ids, counts, starts, tx = _pairs64(mx.detach(), my.detach(), depth.detach(), radius, visible, w, h,
                                           case["keys64"])
        pairs += ids.numel()
        splat = torch.cat([mx[None], my[None], opacity[None], conic, color])
        dl_of = lambda img: (img[..., :3] - targets[v]) * (2.0 / (3.0 * w * h) / views)  # noqa: B023,E731
        img, gs = _blend64(splat.detach(), ids, counts, starts, tx, w, h, dl_of if case["exact_bwd"] else None)
        images.append(img)
        dls.append(dl_of(img))
        losses.append(float((img[..., :3] - targets[v]).square().sum() / (3.0 * w * h)))
        if gs is None:
            continue
        pad = torch.zeros(1, n, dtype=torch.float64, device="cuda")
        pgs.append(torch.cat([gs[0:3], pad, gs[3:6], pad, gs[6:9], pad]).T)
        shown = torch.where(visible[None], splat, torch.zeros_like(splat))
        (shown * torch.where(visible[None], gs, torch.zeros_like(gs))).sum().backward()
        total += pv.grad
    out = {"loss": np.array(losses, np.float64), "pairs": None, "images": torch.stack(images), "dl_dc": torch.nn.functional.pad(torch.stack(dls), (0, 1)),
           "projected_grad": None, "moments": None, "params": None, "grad_acc": None}
    if not case["exact_bwd"]:
        return out  # the reference's walk past a pixel's stop has no value of its own in 64 bits
    mom = _moment_rows(n, seed).double()
    m = BETA1 * mom[0] + (1 - BETA1) * total
    u = BETA2 * mom[1] + (1 - BETA2) * total.square()
    lr = torch.tensor(LRS, dtype=torch.float64, device="cuda").repeat_interleave(
        torch.tensor([3, 4, 3, 1, 3, 45], device="cuda"))[:, None]
    t = T0 + 1
    q = p - lr * (m / (1 - BETA1 ** t)) / ((u / (1 - BETA2 ** t)).sqrt() + EPS)
    q[3:7] = q[3:7] / q[3:7].norm(dim=0, keepdim=True).clamp_min(1e-8)
    q[7:10] = q[7:10].clamp(-10.0, 5.0)
    q[10] = q[10].clamp(-10.0, 10.0)
    out.update(projected_grad=torch.stack(pgs), moments=torch.stack([m, u]), params=q,
               grad_acc=total[0:3].abs().sum(0))
    return out
