"""What a captured alignment loop is made from (host arithmetic, no GPU).

A captured loop is replayed for a call with the same key, so the key has to
fix every offset that the loop holds.  Batches whose images differ in a few
rows or columns can share their count, tiles, parts and z-buffer bytes and
still lay the tile -> pair table elsewhere: over a neighbourhood of sizes, plans
with one key have one set of offsets.

A loop whose fused pass is one CTA per tile of all pairs has one part, whatever
its tiles: the parts would each process all pairs, at the same time."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROBE = r"""
#include <cstdio>
#include <map>
#include <set>
#include "pair_plan.hpp"
using namespace nicp;

static PairPlan plan(std::vector<int> pixels, bool keep_ref) {
  PairPlan pl;
  pl.n = (int)pixels.size();
  pl.keep_ref = keep_ref;
  pl.structured = true;
  pl.P = pixels;
  lay_out_pairs(pl, {320, 1408, 256, 1024, 1024}, std::vector<int>(pixels.size(), 300000), 0);
  plan_parts(pl);
  return pl;
}
static std::string key(const PairPlan &pl) {
  std::string k;
  pl.put(k);
  return k;
}

int main() {
  const PairPlan a = plan({470 * 630, 470 * 634}, true), b = plan({471 * 630, 472 * 630}, true);
  std::printf("%d %d %d %d ", a.zbuf_bytes == b.zbuf_bytes, a.total_tiles == b.total_tiles,
              a.o_tile_pair != b.o_tile_pair, key(a) != key(b));
  // every two images of one set of sizes, and a third one small
  std::set<int> sizes;
  for (int r = 470; r < 490; r++)
    for (int c = 630; c < 650; c += 3) sizes.insert(r * c);
  std::map<std::string, std::vector<size_t>> seen;
  long plans = 0, ambiguous = 0;
  for (int keep = 0; keep < 2; keep++)
    for (int p : sizes)
      for (int q : sizes)
        for (int third = 0; third < 2; third++) {
          std::vector<int> pixels = {p, q};
          if (third) pixels.push_back(1000 + p % 50);
          const PairPlan pl = plan(pixels, keep != 0);
          const std::vector<size_t> at = {pl.o_pairs, pl.o_states, pl.o_krt, pl.o_zbuf, pl.zbuf_bytes, pl.o_tile_pair};
          plans++;
          ambiguous += seen.emplace(key(pl), at).first->second != at;
        }
  // parts of eight pairs of 900 tiles, forked or with one CTA per tile
  PairPlan few = plan(std::vector<int>(8, 720 * 1280), true);
  std::printf("%ld %ld %d ", plans, ambiguous, (int)few.part_pair.size() - 1);
  const std::string forked = key(few);
  few.few = true;
  plan_parts(few);
  std::printf("%d %d\n", (int)few.part_pair.size() - 1, key(few) != forked);
}
"""


def test_equal_keys_have_equal_offsets(tmp_path):
    src, exe = tmp_path / "keys.cpp", tmp_path / "keys"
    src.write_text(PROBE)
    subprocess.run([os.environ.get("NICP_CXX", "g++"), "-std=c++17", "-O1", "-I", os.path.join(ROOT, "nicp_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    same_zbuf, same_tiles, moved, told_apart, plans, ambiguous, parts, few_parts, few_told = map(
        int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert (same_zbuf, same_tiles, moved) == (1, 1, 1)  # the sizes at which the table moves alone
    assert told_apart and plans > 10000 and ambiguous == 0
    assert parts == 4 and few_parts == 1 and few_told
