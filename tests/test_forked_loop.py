"""A batch whose loop runs in parts on branches of a captured graph: the
autotuner times that form, and pairs that leave early do so by themselves."""
import numpy as np
import pytest

from helpers import converter, gpu_cloud
from nicp_b200 import _lib as L
from nicp_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def batch(built):
    own = api.Context(0)
    refs, curs, cams = [], [], []
    for k, size in enumerate(["640x480", "320x240", "640x480", "160x120", "640x480", "320x240"]):
        d1, d2, _, cam = synth.render_pair(71 + k, size, deg=0.2 + k, meters=0.005 * (1 + k))
        proj, conv = converter(cam, own)
        refs.append(gpu_cloud(own, conv, d1, keep_index=False)[0])
        curs.append(gpu_cloud(own, conv, d2, keep_index=False)[0])
        cams.append(proj.camera())
    yield own, refs, curs, cams
    del refs, curs
    own.close()


def _align(b, pick, eps=0.0):
    own, refs, curs, cams = b
    prm = L.AlignParams()
    own.lib.nicp_default_align_params(prm)
    prm.outer_iterations, prm.early_exit_eps = 20, eps
    corr, lin = api.CorrespondenceFinderProjective(own).params(), api.Linearizer(own).params()
    return api.align_batch(own, [refs[k] for k in pick], [curs[k] for k in pick], [cams[k] for k in pick], None, corr,
                           lin, prm)


def _same(a, b):
    return (np.array_equal(np.array(a.T), np.array(b.T)) and a.inliers == b.inliers
            and a.outer_iterations_run == b.outer_iterations_run and np.array_equal(np.array(a.omega), np.array(b.omega)))


def test_early_exit_in_parts(batch):
    """1069 tiles in three parts, with pairs that stop before the last iteration."""
    alone = [_align(batch, [k], 1e-4)[0] for k in range(6)]
    assert min(r.outer_iterations_run for r in alone) < 20
    for order in ([0, 1, 2, 3, 4, 5], [5, 4, 3, 2, 1, 0], [3, 0, 2, 1, 4]):
        for k, r in zip(order, _align(batch, order, 1e-4)):
            assert _same(r, alone[k]), (order, k)


def test_the_form_that_runs_is_tuned(batch):
    own, everyone = batch[0], list(range(6))
    base = _align(batch, everyone)
    own.set_autotune(True)
    try:
        launches = []
        for _ in range(2):
            before = own.kernel_launches()
            tuned = _align(batch, everyone)
            launches.append(own.kernel_launches() - before)
    finally:
        own.set_autotune(False)
    # a warm-up, the default, three other projections, two other fused passes
    # -- then the loop itself, all with the forked loop's launches
    assert launches[0] == 8 * launches[1]
    assert all(_same(a, b) for a, b in zip(base, tuned))
