"""A download lays out what is asked for in pieces of the workspace that is
there: the device memory of a context does not grow with the cloud that it
hands out."""
import ctypes as C

import numpy as np
import pytest

from helpers import converter, gpu_cloud
from nicp_b200 import _lib as L
from nicp_b200 import api, synth

pytestmark = pytest.mark.gpu


def _big(ctx, n):
    rng = np.random.default_rng(n)
    p = np.concatenate([rng.random((n, 3), np.float32), np.ones((n, 1), np.float32)], 1)
    m = np.concatenate([rng.random((n, 3), np.float32), np.zeros((n, 1), np.float32)], 1)
    k = rng.random(n, np.float32)
    o = rng.random((2, n, 3, 3), np.float32)
    o = o + o.transpose(0, 1, 3, 2)
    c = api.Cloud(ctx)
    c.upload(p, m, k, o[0], o[1])
    return c, dict(points=p, normals=m, curvature=k, omega_p=o[0], omega_n=o[1])


def _same(got, want):
    return all(np.array_equal(got[k], want[k]) for k in want)


def test_memory_stays(built):
    ctx = api.Context(0)
    d1, _, _, cam = synth.render_pair(47, "320x240")
    _, conv = converter(cam, ctx)
    gpu_cloud(ctx, conv, d1)
    c, want = _big(ctx, 1000003)  # 36 MB of points, normals, curvature; 108 MB in all
    before = ctx.device_bytes()
    n = 1000003
    p, m, k = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32), np.zeros(n, np.float32)
    ctx.check(ctx.lib.nicp_cloud_download(c.h, L.fptr(p), L.fptr(m), L.fptr(k), None, None, None, None))
    assert _same(dict(points=p, normals=m, curvature=k), {x: want[x] for x in ("points", "normals", "curvature")})
    assert ctx.device_bytes() == before
    assert _same(c.download(), want) and ctx.device_bytes() == before
    del c
    ctx.close()


def test_context_without_a_workspace(built):
    """The first download of a context takes a piece's room, whatever the cloud."""
    ctx = api.Context(0)
    c, want = _big(ctx, 700001)
    before = ctx.device_bytes()
    assert _same(c.download(), want)
    assert 0 < ctx.device_bytes() - before <= 24 << 20
    # nothing asked for: nothing taken
    ctx.check(ctx.lib.nicp_cloud_download(c.h, *[None] * 7))
    del c
    ctx.close()


def test_stats_in_pieces(built):
    ctx = api.Context(0)
    d1, _, _, cam = synth.render_pair(48, "640x480")
    _, conv = converter(cam, ctx, keep_stats=True)
    scene, _ = gpu_cloud(ctx, conv, d1)
    want = scene.download(stats=True)
    n = len(want["points"])
    for s in range(3):  # seven times the frame: 330 MB in all
        other = api.Cloud(ctx)
        conv.compute(other, d1)
        for _ in range(s):
            again = api.Cloud(ctx)
            conv.compute(again, d1)
            other.add(again)
        scene.add(other)
    total = scene.size()
    assert total == 7 * n
    before = ctx.device_bytes()
    got = scene.download(stats=True)
    assert ctx.device_bytes() == before
    for key, w in want.items():
        for s in range(7):
            assert np.array_equal(got[key][s * n:(s + 1) * n], w), (key, s)
    del scene, other, again
    ctx.close()
