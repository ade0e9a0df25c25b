"""The grid search of the nearest-neighbour association over the forms where it
can go wrong -- clouds of one point to many, ties, clouds with empty space
between them (the wide search), queries outside the grid, small and unlimited
radii, points and normals that are not finite -- against the REF32 oracle's
exhaustive scan: the same list, bit for bit."""
import numpy as np
import pytest

from nicp_b200 import api
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def _cloud(rng, n, spread, kind):
    p = rng.uniform(-1, 1, (n, 3)) * spread
    if kind == "plane":
        p[:, 2] = 0.5
    elif kind == "line":
        p[:, 1:] = 0.25
    elif kind == "clusters":  # a few distant groups
        p = p * 0.02 + rng.integers(-3, 4, (n, 1)) * np.array([0.9, 0.2, -0.4])
    elif kind == "grid":      # many equal distances
        p = np.round(p * 8) / 8
    m = rng.normal(size=(n, 3))
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    if kind in ("plane", "grid"):
        m = np.tile([0.0, 0.0, -1.0], (n, 1))
    m[rng.random(n) < 0.3] = 0.0
    return p.astype(np.float32), m.astype(np.float32)


def _upload(ctx, p, m):
    c = api.Cloud(ctx)
    n = len(p)
    c.upload(np.concatenate([p, np.ones((n, 1), np.float32)], 1), np.concatenate([m, np.zeros((n, 1), np.float32)], 1),
             np.zeros(n, np.float32))
    z = np.zeros((n, 9))
    o = O.Cloud.from_arrays(O.REF32, np.concatenate([p, np.ones((n, 1))], 1).astype(np.float64),
                            np.concatenate([m, np.zeros((n, 1))], 1).astype(np.float64), np.zeros(n), z, z)
    return c, o


def _check(ctx, ref, cur, T, scaling, demoted, radius):
    (gr, orf), (gc, oc) = _upload(ctx, *ref), _upload(ctx, *cur)
    cf = api.CorrespondenceFinderNN(ctx)
    cf.setNormalScaling(scaling)
    cf.setDemotedToGICP(demoted)
    cf.setInlierDistanceThreshold(radius)
    got = cf.compute(gr, gc, T)
    prm = O.align_params(corr_demoted_to_gicp=1 if demoted else 0, inlier_distance_threshold=radius)
    want = O.correspond_nn(O.REF32, orf, oc, np.asarray(T, np.float32).astype(np.float64), scaling, prm)
    assert np.array_equal(got, want)
    return len(got)


@pytest.mark.parametrize("kind", ["volume", "plane", "line", "clusters", "grid"])
@pytest.mark.parametrize("nr,nc", [(1, 1), (31, 1), (33, 2), (127, 129), (129, 640), (1500, 2000)])
@pytest.mark.parametrize("scaling,demoted,radius", [(1.0, False, 1.0), (0.2, True, 0.05), (0.05, True, 1000.0)])
def test_search_equals_exhaustive_scan(ctx, kind, nr, nc, scaling, demoted, radius):
    rng = np.random.default_rng(nr * 131 + nc)
    cur = _cloud(rng, nc, 1.0, kind)
    ref = _cloud(rng, nr, 1.3, kind)  # beyond the current cloud's box too
    T = np.eye(4, dtype=np.float32)
    T[:3, 3] = [0.01, -0.02, 0.005]
    _check(ctx, ref, cur, T, scaling, demoted, radius)


def test_search_with_values_that_are_not_finite(ctx):
    rng = np.random.default_rng(5)
    cur, ref = _cloud(rng, 400, 1.0, "plane"), _cloud(rng, 300, 1.0, "plane")
    for p, m in (cur, ref):
        p[3], p[17, 1], m[40, 2], m[41] = np.nan, np.inf, np.nan, np.inf
    assert _check(ctx, ref, cur, np.eye(4, dtype=np.float32), 1.0, False, 1.0) > 50


def test_search_far_from_everything(ctx):
    rng = np.random.default_rng(6)
    cur, ref = _cloud(rng, 200, 0.5, "volume"), _cloud(rng, 100, 0.5, "volume")
    T = np.eye(4, dtype=np.float32)
    T[:3, 3] = [2e5, -3e6, 1e4]
    assert _check(ctx, ref, cur, T, 1.0, False, 1.0) == 0
    assert _check(ctx, ref, cur, T, 1.0, True, 1e7) >= 0
