"""The context's page-locked staging block (pinned_block.hpp) over a stand-in
for the CUDA runtime, no GPU: an allocation that fails, growth.  And on the GPU:
loops captured before a move."""
import os
import subprocess

import numpy as np
import pytest

from helpers import converter
from nicp_b200 import _lib as L
from nicp_b200 import api, synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdio>
#include "pinned_block.hpp"

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
  nicp::PinnedBlock b;
  CHECK(b.reserve(1000) == cudaSuccess && b.p && b.cap >= 1000);
  char *first = b.p;
  CHECK(b.reserve(b.cap) == cudaSuccess && b.p == first);
  // a larger block cannot be had: the error, and nothing is handed out as if it could
  fake.lock_fails = true;
  CHECK(b.reserve((size_t)64 << 20) != cudaSuccess);
  CHECK(b.reserve(1000) != cudaSuccess && !b.p);
  fake.lock_fails = false;
  CHECK(b.reserve(1000) == cudaSuccess && b.p && fake.is_locked(b.p) && fake.is_locked(b.p + 999));
  b.release();
  CHECK(fake.allocated == fake.freed && !b.p && !b.cap);
  return 0;
}
"""


GROWTH = r"""
#include <cstdio>
#include "pinned_block.hpp"

// moves of a block over calls that ask for `step` bytes more each, up to `most`
static int moves(size_t step, size_t most) {
  nicp::PinnedBlock b;
  char *at = nullptr;
  int n = 0;
  for (size_t bytes = step; bytes <= most; bytes += step) {
    if (b.reserve(bytes) != cudaSuccess || b.cap < bytes) return -1;
    n += at && b.p != at;
    at = b.p;
  }
  b.release();
  return n;
}

int main() {
  std::printf("%d %d\n", moves(1408, 700 * 1408), moves(10000, (size_t)64 << 20));
  return 0;
}
"""


def _run(tmp_path, probe):
    src, exe = tmp_path / "block.cpp", tmp_path / "block"
    src.write_text(probe)
    subprocess.run([os.environ.get("NICP_CXX", "g++"), "-std=c++17", "-O1",
                    "-I", os.path.join(ROOT, "tests", "cpp", "fake_cuda"), "-I", os.path.join(ROOT, "nicp_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    return subprocess.run([str(exe)], capture_output=True, text=True)


def test_growth_moves_the_block_seldom(tmp_path):
    """Captured loops are dropped when the block moves: not at all up to the
    results of 700 pairs, once per doubling beyond 1 MB (64 MB: six)."""
    r = _run(tmp_path, GROWTH)
    assert [int(x) for x in r.stdout.split()] == [0, 6]


def test_a_failed_growth_leaves_no_block(tmp_path):
    r = _run(tmp_path, PROBE)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_captured_loops_across_a_move(ctx):
    """A geometry that was captured gives the same result after a batch whose
    results do not fit the first block."""
    d1, d2, _, cam = synth.render_pair(53, "160x120", deg=1.0, meters=0.02)
    corr, lin, prm = api.CorrespondenceFinderProjective(ctx).params(), api.Linearizer(ctx).params(), L.AlignParams()
    ctx.lib.nicp_default_align_params(prm)
    prm.outer_iterations = 3
    own = api.Context(0)  # (its blocks are as small as they start)
    ref, cur = api.Cloud(own), api.Cloud(own)
    proj, conv = converter(cam, own)
    conv.compute(ref, d1)
    conv.compute(cur, d2)
    results = []
    for n in (1, 2, 900, 1, 2, 900):
        r = api.align_batch(own, [ref] * n, [cur] * n, [proj.camera()] * n, None, corr, lin, prm)
        results += [np.array(r[0].T), np.array(r[n - 1].T)]
    assert all(np.array_equal(results[0], r) for r in results)
    del ref, cur
    own.close()
