"""The context's page-locked staging block (pinned_block.hpp) over a stand-in
for the CUDA runtime, no GPU: an allocation that fails, growth."""
import os
import subprocess

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


def test_a_failed_growth_leaves_no_block(tmp_path):
    src, exe = tmp_path / "block.cpp", tmp_path / "block"
    src.write_text(PROBE)
    subprocess.run([os.environ.get("NICP_CXX", "g++"), "-std=c++17", "-O1",
                    "-I", os.path.join(ROOT, "tests", "cpp", "fake_cuda"), "-I", os.path.join(ROOT, "nicp_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
