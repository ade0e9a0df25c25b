"""No outer iteration, with the solution's statistics: the pose is the guess,
and the statistics are those of an empty correspondence list -- whatever
earlier calls left in the workspace's index images and lists."""
import numpy as np
import pytest

from helpers import cams, converter, gpu_cloud, oracle_cloud_from_gpu, perturb
from nicp_b200 import _lib as L
from nicp_b200 import api, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pair(ctx):
    d1, d2, _, cam = synth.render_pair(41, "160x120", deg=1.0, meters=0.02)
    proj, conv = converter(cam, ctx)
    return proj, cam, [gpu_cloud(ctx, conv, d, keep_index=False)[0] for d in (d1, d2)]


def _same(r, o):
    assert np.array_equal(np.array(r.T).reshape(4, 4), o["T"])
    assert (r.error, r.inliers, r.num_correspondences, r.outer_iterations_run) == (0, 0, 0, 0)
    assert (r.translational_ratio, r.rotational_ratio) == (o["translational_ratio"], o["rotational_ratio"])
    assert r.solution_valid == o["solution_valid"] == 0
    assert not np.any(r.omega) and not np.any(r.mean)


# alone (one CTA per tile), a batch beyond that, and the list kernels
@pytest.mark.parametrize("n,threads", [(1, 1), (40, 1), (1, 4)])
def test_projective(ctx, pair, n, threads):
    proj, cam, (ref, cur) = pair
    corr, lin, prm = api.CorrespondenceFinderProjective(ctx).params(), api.Linearizer(ctx).params(), L.AlignParams()
    ctx.lib.nicp_default_align_params(prm)
    corr.parity_threads = threads
    guess = perturb(3).astype(np.float32)
    args = ([ref] * n, [cur] * n, [proj.camera()] * n, [guess] * n, corr, lin, prm)
    assert api.align_batch(ctx, *args)[0].num_correspondences > 100
    prm.outer_iterations = 0
    got = api.align_batch(ctx, *args)
    o = O.align(O.F64, oracle_cloud_from_gpu(O.F64, ref.download()), oracle_cloud_from_gpu(O.F64, cur.download()),
                cams(cam)[1], guess=guess.astype(np.float64), prm=O.align_params(outer_iterations=0), statistics=True)
    for r in (got[0], got[-1]):
        _same(r, o)


def test_nearest_neighbour(ctx, pair):
    _, _, (ref, cur) = pair
    al = api.AlignerNN(None, api.Linearizer(ctx), api.CorrespondenceFinderNN(ctx), ctx)
    al.computeStatistics = True
    al.setReferenceCloud(ref)
    al.setCurrentCloud(cur)
    al.align()
    assert al.inliers() > 100
    al.setOuterIterations(0)
    T = al.align()
    o = O.align_nn(O.F64, oracle_cloud_from_gpu(O.F64, ref.download()), oracle_cloud_from_gpu(O.F64, cur.download()),
                   prm=O.align_params(outer_iterations=0), statistics=True)
    assert np.array_equal(T, o["T"]) and al.inliers() == 0 and al.error() == 0
    assert not al.solutionValid() and not np.any(al.omega())
