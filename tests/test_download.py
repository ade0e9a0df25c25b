"""What was uploaded comes back: the export kernel's last CTA, and copies below
and above the size at which worker threads share them."""
import numpy as np
import pytest

from nicp_b200 import _lib as L
from nicp_b200 import api

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 255, 256, 257, 5000, 77673, 300001])
def test_round_trip(ctx, n):
    rng = np.random.default_rng(n)
    p = np.concatenate([rng.normal(size=(n, 3)), np.ones((n, 1))], 1).astype(np.float32)
    m = np.concatenate([rng.normal(size=(n, 3)), np.zeros((n, 1))], 1).astype(np.float32)
    k = rng.random(n).astype(np.float32)
    sym = rng.normal(size=(2, n, 3, 3)).astype(np.float32)
    sym = sym + sym.transpose(0, 1, 3, 2)
    c = api.Cloud(ctx)
    c.upload(p, m, k, sym[0], sym[1])
    d = c.download()
    assert np.array_equal(d["points"], p) and np.array_equal(d["normals"], m) and np.array_equal(d["curvature"], k)
    assert np.array_equal(d["omega_p"], sym[0]) and np.array_equal(d["omega_n"], sym[1])
    # any output may be left out
    only = np.zeros((n, 9), np.float32)
    ctx.check(ctx.lib.nicp_cloud_download(c.h, None, None, None, None, L.fptr(only), None, None))
    assert np.array_equal(only.reshape(n, 3, 3), sym[1])
