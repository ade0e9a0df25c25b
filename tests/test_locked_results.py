"""Results into page-locked buffers, as a capture program holds them: the same
bytes as into ordinary memory, in one transfer per array; a destination that is
not host memory is refused."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import converter, gpu_cloud
from nicp_b200 import _lib as L
from nicp_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", ["160x120", "640x480"])
def test_page_locked_destinations(ctx, size):
    d1, _, _, cam = synth.render_pair(43, size)
    proj, conv = converter(cam, ctx, keep_stats=True)
    cloud, _ = gpu_cloud(ctx, conv, d1, keep_index=False)
    want = cloud.download(stats=True)
    n, P = len(want["points"]), cam["rows"] * cam["cols"]
    keys = ("points", "normals", "curvature", "omega_p", "omega_n", "eigenvalues", "eigenvectors")
    held = [torch.full(want[k].shape, 7.0, pin_memory=True) for k in keys]
    ptr = [C.cast(t.data_ptr(), L.f32p) for t in held]
    ctx.check(ctx.lib.nicp_cloud_download(cloud.h, *ptr))
    for k, t in zip(keys, held):
        assert np.array_equal(t.numpy(), want[k]), k
    # one array page-locked, the other not
    cam_s, T = proj.camera(), np.eye(4, dtype=np.float32)
    index, depth = proj.project(cloud)
    li = torch.zeros(P, dtype=torch.int32, pin_memory=True)
    pd = np.zeros(P, np.float32)
    ctx.check(ctx.lib.nicp_project(ctx.h, cloud.h, C.byref(cam_s), L.fptr(L.f16(T)), C.cast(li.data_ptr(), L.i32p),
                                   L.fptr(pd)))
    assert np.array_equal(li.numpy(), index.reshape(-1)) and np.array_equal(pd, depth.reshape(-1))
    # a few points of a small cloud: below the size of the small pinned buffer
    small = api.Cloud(ctx)
    small.upload(want["points"][:5], want["normals"][:5], want["curvature"][:5])
    lp = torch.zeros(5, 4, pin_memory=True)
    ctx.check(ctx.lib.nicp_cloud_download(small.h, C.cast(lp.data_ptr(), L.f32p), None, None, None, None, None, None))
    assert np.array_equal(lp.numpy(), want["points"][:5])


def test_device_destination_is_refused(ctx):
    for n in (5, 5000):
        p = np.concatenate([np.random.default_rng(n).normal(size=(n, 3)), np.ones((n, 1))], 1).astype(np.float32)
        c = api.Cloud(ctx)
        c.upload(p, np.zeros((n, 4), np.float32), np.zeros(n, np.float32))
        dev = torch.zeros(n, 4, device="cuda")
        assert ctx.lib.nicp_cloud_download(c.h, C.cast(dev.data_ptr(), L.f32p), None, None, None, None, None,
                                           None) == L.NICP_ECUDA
        assert np.array_equal(c.download()["points"], p)
