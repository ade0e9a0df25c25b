"""A pair whose image has few tiles is aligned by another fused kernel (one CTA
per tile, chained launches) than a batch: both form the same sums in the same
order, so the results are the same bits.  And the sum of the tile partials,
over tile counts around its group and batch sizes."""
import numpy as np
import pytest

from helpers import converter, gpu_cloud
from nicp_b200 import _lib as L
from nicp_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = api.Context(0)
    yield c
    c.close()


def _camera(rows, cols):
    f = 525.0 * max(cols, 64) / 640.0
    return dict(rows=rows, cols=cols, fx=f, fy=f, cx=(cols - 1) / 2.0, cy=(rows - 1) / 2.0, min_distance=0.01,
                max_distance=6.0)


def _pair(ctx, rows, cols, seed):
    cam = _camera(rows, cols)
    rng = np.random.default_rng(seed)
    scene, P = synth.make_scene(seed), synth.base_pose(rng)
    Q = P @ synth.random_offset(rng, 1.0, 1.0, 0.02, 0.02)
    args = (cam["fx"], cam["fy"], cam["cx"], cam["cy"], rows, cols)
    d = [synth.render(scene, X, *args, noise_seed=seed + k) for k, X in enumerate((P, Q))]
    proj, conv = converter(cam, ctx)
    conv.statsCalculator().setMinImageRadius(2)
    conv.statsCalculator().setMinPoints(4)
    return proj, [gpu_cloud(ctx, conv, x, keep_index=False)[0] for x in d]


# one tile exactly, one pixel less and more, a few, a ragged image, three CTAs per SM nearly full
SIZES = [(32, 32), (31, 33), (41, 25), (60, 80), (337, 451), (480, 640)]
VARIANTS = [dict(), dict(inner=2, stats=True), dict(demoted=True, z_scaling=True), dict(robust=False, max_chi2=0.5)]


@pytest.mark.parametrize("rows,cols", SIZES)
@pytest.mark.parametrize("variant", range(len(VARIANTS)))
def test_alone_equals_in_a_large_batch(ctx, rows, cols, variant):
    v = VARIANTS[variant]
    proj, (ref, cur) = _pair(ctx, rows, cols, 3 + rows)
    corr, lin, prm = api.CorrespondenceFinderProjective(ctx).params(), api.Linearizer(ctx).params(), L.AlignParams()
    ctx.lib.nicp_default_align_params(prm)
    prm.outer_iterations, prm.inner_iterations = 4, v.get("inner", 1)
    prm.compute_statistics = 1 if v.get("stats") else 0
    corr.demoted_to_gicp = lin.demoted_to_gicp = 1 if v.get("demoted") else 0
    lin.z_scaling = 1 if v.get("z_scaling") else 0
    lin.robust_kernel = 0 if v.get("robust") is False else 1
    lin.inlier_max_chi2 = v.get("max_chi2", lin.inlier_max_chi2)
    cam = proj.camera()
    tiles = (rows * cols + 1023) // 1024
    n = 3 * 160 // tiles + 2  # beyond three tiles per SM
    alone = api.align_batch(ctx, [ref], [cur], [cam], None, corr, lin, prm)[0]
    many = api.align_batch(ctx, [ref] * n, [cur] * n, [cam] * n, None, corr, lin, prm)
    assert alone.num_correspondences > 0
    for r in (many[0], many[n - 1]):
        assert np.array_equal(np.array(alone.T), np.array(r.T), equal_nan=True)
        assert np.float32(alone.error).tobytes() == np.float32(r.error).tobytes()
        assert (alone.inliers, alone.num_correspondences) == (r.inliers, r.num_correspondences)
        assert np.array_equal(np.array(alone.omega), np.array(r.omega), equal_nan=True)


@pytest.mark.parametrize("tiles", [1, 15, 16, 17, 127, 128, 129, 300])
def test_tile_partials_add_up(ctx, tiles):
    """H and b of a list are the sums of H and b of its 1024-entry tiles: FP64
    sums of at most 300 partials, 300 half ulps relative to their magnitudes."""
    _, (ref, cur) = _pair(ctx, 60, 80, 5)
    m = min(ref.size(), cur.size())
    tile = np.stack([np.arange(1024) % m, (np.arange(1024) * 7) % m], 1).astype(np.int32)
    lists = [np.roll(tile, k, axis=0) if k % 3 else (tile + k) % m for k in range(tiles)]
    lin = api.Linearizer(ctx)
    lin.update(ref, cur, np.concatenate(lists), 1)
    H, b, inliers = lin.H(), lin.b(), lin.inliers()
    Hs, bs, mags, magb, count = np.zeros((6, 6)), np.zeros(6), np.zeros((6, 6)), np.zeros(6), 0
    for t in lists:
        lin.update(ref, cur, t, 1)
        Hs, bs, count = Hs + lin.H(), bs + lin.b(), count + lin.inliers()
        mags, magb = mags + np.abs(lin.H()), magb + np.abs(lin.b())
    assert inliers == count
    eps = 300 * 2.0 ** -53
    assert np.all(np.abs(H - Hs) <= 2 * eps * mags) and np.all(np.abs(b - bs) <= 2 * eps * magb)


@pytest.mark.parametrize("n", [2, 3, 4, 5, 9])
def test_parts_of_a_batch(ctx, n):
    """A batch's loop runs in one to four parts, cut by tiles: each pair's
    result is what it is alone, wherever the cuts fall."""
    corr, lin, prm = api.CorrespondenceFinderProjective(ctx).params(), api.Linearizer(ctx).params(), L.AlignParams()
    ctx.lib.nicp_default_align_params(prm)
    prm.outer_iterations = 4
    pairs = [_pair(ctx, rows, cols, 11 + rows) for rows, cols in ((480, 640), (60, 80), (337, 451))]
    order = [0] * n + [1, 2]  # n of 300 tiles, then 5 and 149
    order = order[n // 2:] + order[:n // 2]
    alone = [api.align_batch(ctx, [c[0]], [c[1]], [p.camera()], None, corr, lin, prm)[0] for p, c in pairs]
    many = api.align_batch(ctx, [pairs[k][1][0] for k in order], [pairs[k][1][1] for k in order],
                           [pairs[k][0].camera() for k in order], None, corr, lin, prm)
    for k, r in zip(order, many):
        assert np.array_equal(np.array(alone[k].T), np.array(r.T), equal_nan=True)
        assert np.float32(alone[k].error).tobytes() == np.float32(r.error).tobytes()
        assert (alone[k].inliers, alone[k].num_correspondences) == (r.inliers, r.num_correspondences)
