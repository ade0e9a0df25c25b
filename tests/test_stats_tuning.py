"""The autotuner's choice for the stats kernel belongs to the form that it
timed: builds with and without Stats tune each their own."""
import pytest

from helpers import converter, gpu_cloud
from nicp_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [True, False])
def test_each_form_is_tuned(built, first):
    d1, _, _, cam = synth.render_pair(59, "160x120")
    ctx = api.Context(0)
    ctx.set_autotune(True)
    launches = {}
    for stats in (first, not first, first, not first):
        _, conv = converter(cam, ctx, keep_stats=stats)
        before = ctx.kernel_launches()
        c, _ = gpu_cloud(ctx, conv, d1, keep_index=False)
        launches.setdefault(stats, []).append(ctx.kernel_launches() - before)
        del c
    # a tuned build times every shape twice
    assert all(a > b for a, b in launches.values()), launches
    ctx.close()
