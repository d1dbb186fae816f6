"""The FP64 quadrature's split, compiled for the host: every range of points
that a grid's screening can leave fits the workspace sized for the whole grid,
and tiles and chunks cover the triangle and the range exactly once."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'napmo_b200',
                    'csrc')

PROGRAM = r'''
#include <cstdio>
#include <cstdlib>
#include <set>
#include <utility>
#include "quad_plan.h"
using namespace napmo;

static void fail(const char *what, int n, int full, int npad) {
  std::printf("%s: n %d, grid %d, range %d\n", what, n, full, npad);
  std::exit(1);
}

// partial sums (tiles or chunks) of a plan, after checking that they cover it
static long slots_of(int n, int full, int npad, const QuadPlan &p) {
  const int classes = n <= kSmallN ? 1 : 4;
  long used = 0;
  for (int c = 0; c < classes; ++c) {
    if (p.ntile[c] == 0) continue;
    if (p.chunk[c] <= 0 || p.chunk[c] % kQuadStage) fail("chunk length", n, full, npad);
    if ((long)p.nch[c] * p.chunk[c] < npad || (long)(p.nch[c] - 1) * p.chunk[c] >= npad)
      fail("range not covered once", n, full, npad);
    if (n > kSmallN && p.first[c + 1] - p.first[c] != p.nch[c] * p.ntile[c])
      fail("CTA numbers", n, full, npad);
    used += (long)p.nch[c] * p.ntile[c];
  }
  if (used != (n <= kSmallN ? p.nch[0] : p.first[4])) fail("slots", n, full, npad);
  return used;
}

static void check(int n, int full, int step) {
  const int slots = quad_default_slots(n);
  long bound = 0;
  quad_plan_slots(n, full, slots, &bound);
  for (int npad = kQuadStage; npad <= full; npad += step)
    if (slots_of(n, full, npad, quad_plan_slots(n, npad, slots)) > bound)
      fail("beyond the workspace", n, full, npad);
}

int main() {
  const int sizes[] = {1,   15,  16,  17,  25,  32,  33,  48,  49,  60,  64,  65,  80,  96,
                       112, 113, 127, 128, 129, 144, 200, 210, 255, 256, 257, 300, 310, 384,
                       385, 510, 512, 513, 1000, 1920};
  for (int n : sizes) {
    for (int full = 128; full <= 12800; full += 128) check(n, full, kQuadStage);
    for (int full : {16512, 40064, 100096, 785280, 1147648, 1872512})
      check(n, full, full < 50000 ? kQuadStage : 11 * kQuadStage);
    // a fixed workspace: the plan stays within the slots it is given
    const int nblk = (n + kQuadTile - 1) / kQuadTile, tiles = nblk * (nblk + 1) / 2;
    for (int slots : {tiles, tiles + 1, 2 * tiles + 3, 128})
      for (int npad = 128; npad <= 6400; npad += 128)
        if (slots >= tiles && slots_of(n, npad, npad, quad_plan_slots(n, npad, slots)) > slots)
          fail("beyond the given slots", n, slots, npad);
    if (n <= kSmallN) continue;
    const QuadPlan p = quad_plan_slots(n, 4096, quad_default_slots(n));
    std::set<std::pair<int, int>> seen;
    int all = 0;
    for (int c = 0; c < 4; ++c)
      for (int t = 0; t < p.ntile[c]; ++t, ++all) {
        int mb, nb;
        quad_tile(c, t, nblk, mb, nb);
        if (mb < 0 || mb > nb || nb >= nblk) fail("tile", n, c, t);
        seen.insert({mb, nb});
      }
    if (all != tiles || (int)seen.size() != tiles) fail("triangle", n, all, tiles);
  }
  return 0;
}
'''


@pytest.mark.skipif(shutil.which('g++') is None, reason='needs a host compiler')
def test_every_range_fits_the_workspace(tmp_path):
    src, exe = tmp_path / 'plan.cpp', tmp_path / 'plan'
    src.write_text(PROGRAM)
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-I', CSRC, str(src), '-o', str(exe)])
    done = subprocess.run([str(exe)], stdout=subprocess.PIPE, universal_newlines=True)
    assert done.returncode == 0, done.stdout
