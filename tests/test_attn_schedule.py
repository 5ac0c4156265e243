"""The attention kernel's queue of work items, run on the host from the kernel's own source: every (head, query group) is in
exactly one entry, whatever the numbers of heads, groups and SMs."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pbs_attn_b200", "csrc")
SOURCE = r"""
#include <vector>
#include "pbs_schedule.h"
using namespace pbs;
// 0: every item once, nothing past the end; else a code of what is wrong
extern "C" int check(int BH, int G, int sms) {
  const Schedule w = make_schedule(BH, G, sms);
  if (w.n_items != BH * G || w.ctas < 1 || w.ctas > sms || w.ctas > w.n_items) return 1;
  if (w.pairs < 0 || 2 * w.pairs > w.n_items || entries(w) < w.ctas) return 2;
  std::vector<int> seen(BH * G, 0);
  int last = G + 1;
  for (int q = 0; q < entries(w); ++q)
    for (int j = 0; j < (q < w.pairs ? 2 : 1); ++j) {
      int bh = -1, g = -1;
      if (!queue_item(w, q, j, bh, g)) return 3;
      if (bh < 0 || bh >= BH || g < 0 || g >= G) return 4;
      if (seen[bh * G + g]++) return 5;
      if (q >= w.pairs) {                                  // single groups: the longest first
        if (g > last) return 6;
        last = g;
      }
    }
  for (int n : seen) if (n != 1) return 7;
  int bh, g;
  for (int q = entries(w); q < entries(w) + 2 * sms; ++q)
    if (queue_item(w, q, 0, bh, g)) return 8;
  for (int q = w.pairs; q < entries(w); ++q)
    if (queue_item(w, q, 1, bh, g)) return 9;
  return 0;
}
"""


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    d = tmp_path_factory.mktemp("schedule")
    src, lib = d / "check.cpp", d / "check.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    return ctypes.CDLL(str(lib)).check


# few SMs reach whole waves, rests and partly taken heads at small sizes
@pytest.mark.parametrize("sms", [1, 2, 3, 7, 12, 148])
def test_every_item_is_in_exactly_one_entry(check, sms):
    sizes = [(bh, g) for bh in range(1, 41) for g in range(1, 34)]
    sizes += [(32, 512), (4, 512), (28, 128), (128, 8), (37, 8), (8, 74), (70, 9), (1, 2048)]
    bad = [(bh, g, rc) for bh, g in sizes if (rc := check(bh, g, sms))]
    assert not bad, bad[:5]
