"""Packing and unpacking of parameters and moments move values unchanged, at
counts around a CTA's 2048 elements, odd offsets and odd pitches: checked
against the stores' own host copies, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from nanotracer_b200 import AdamMomentBuffers, GpuSplatBuffer, SplatBuffer
from nanotracer_b200._lib import check, lib

pytestmark = pytest.mark.gpu
ROWS = 59


def _bf16(a):
    """f32 values that bf16 holds exactly."""
    return (np.ascontiguousarray(a, np.float32).view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n,lo,count,shard", [(1, 0, 1, 1), (7, 3, 4, 5), (2048, 0, 2048, 2048), (2049, 0, 2049, 2049),
                                              (5001, 2, 4097, 4099), (6000, 1024, 2047, 2112)])
def test_pack_range_and_unpack_are_exact(ctx, n, lo, count, shard, bf16):
    rng = np.random.default_rng(n + lo)
    p = _bf16(rng.normal(0, 1, (n, ROWS)))
    m, v = _bf16(rng.normal(0, 1, (n, ROWS))), _bf16(rng.normal(0, 1, (n, ROWS)))
    g = GpuSplatBuffer.upload(ctx, SplatBuffer.from_flat(p), bf16_rest=bf16)
    mo = AdamMomentBuffers.upload_from_cpu(ctx, SplatBuffer.from_flat(m), SplatBuffer.from_flat(v), bf16=bf16)
    out = ctx.storage_buffer_zeroed("out", 2 * ROWS * shard * 4)
    check(lib().sc_splats_pack_range(ctx.handle, g.handle, lo, count, shard, out.cptr), ctx.handle)
    got = out.readback(np.float32, ROWS * shard).reshape(ROWS, shard)
    assert np.array_equal(got[:, :count], p[lo:lo + count].T) and not got[:, count:].any()
    check(lib().sc_moments_pack_range(ctx.handle, mo.handle, lo, count, shard, out.cptr), ctx.handle)
    got = out.readback(np.float32).reshape(2, ROWS, shard)
    assert np.array_equal(got[0, :, :count], m[lo:lo + count].T)
    assert np.array_equal(got[1, :, :count], v[lo:lo + count].T)
    # back from chunks of `shard` splats that cover all n
    k = -(-n // shard)
    pad = np.zeros((k * shard, ROWS), np.float32)
    pad[:n] = p[::-1]
    chunks = ctx.storage_buffer("in", np.ascontiguousarray(pad.reshape(k, shard, ROWS).transpose(0, 2, 1)))
    check(lib().sc_splats_unpack_shards(ctx.handle, g.handle, chunks.cptr, k, shard), ctx.handle)
    assert np.array_equal(g.readback().flat(), p[::-1])
    padm = np.zeros((2, k * shard, ROWS), np.float32)
    padm[0, :n], padm[1, :n] = v, m
    chunks = ctx.storage_buffer("in", np.ascontiguousarray(padm.reshape(2, k, shard, ROWS).transpose(1, 0, 3, 2)))
    check(lib().sc_moments_unpack_shards(ctx.handle, mo.handle, n, chunks.cptr, k, shard), ctx.handle)
    gm, gv = mo.download(n)
    assert np.array_equal(gm.flat(), v) and np.array_equal(gv.flat(), m)
