"""The attention kernel's walk over key tiles, compiled for the host from the kernel's own source: what it visits is what the mask lets the queries see, and
its closed-form counts are what it visits, on every rank of every layout (the GPU tests run one rank)."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_DRIVER = r"""
#include <algorithm>
#include <cstdio>
#include <set>
#include <utility>
#define __device__
using std::max; using std::min;
constexpr int kTQ = 128, kTK = 128;
struct DeviceContext { int rank, world; };
struct RingArgs { DeviceContext ctx; int S, causal, zigzag; };
@SOURCE@
// first position of 128-token tile t of rank r's block, in the whole sequence
static long pos(int r, int W, int S, int t, bool zigzag) {
  const long i = (long)t * 128;
  if (!zigzag) return (long)r * S + i;
  return i < S / 2 ? (long)r * (S / 2) + i : (long)(2 * W - 1 - r) * (S / 2) + (i - S / 2);
}
template <bool kByKeys> int check(int W, int r, int S, bool causal, bool zigzag, Item it) {
  RingArgs a{{r, W}, S, causal, zigzag};
  const int T = (S + 127) / 128;
  std::set<std::pair<int, int>> want, got;
  int n[2] = {0, 0};
  for (int o = 0; o < W; ++o)
    for (int t = 0; t < T; ++t) {
      bool any = false;
      for (int i = 0; i < it.n_q; ++i) {
        const bool sees = !causal || pos(r, W, S, it.qt[i], zigzag) >= pos(o, W, S, t, zigzag);
        n[i] += sees; any |= sees;
      }
      if (any) want.insert({o, t});
    }
  int w[2] = {0, 0}, steps = 0, c0, c1, all;
  for (TileWalk<kByKeys> k(a, it); k.next(); ++steps) {
    if (!got.insert({k.origin, k.t}).second) return 1;
    w[0] += k.needs(0); w[1] += k.needs(1);
  }
  TileWalk<kByKeys>(a, it).count(c0, c1, all);
  if (got != want || all != steps) return 2;
  if (!kByKeys && (c0 != w[0] || c1 != w[1] || w[0] != n[0] || w[1] != n[1])) return 3;
  return 0;
}
int main() {
  long forms = 0;
  for (int W : {1, 2, 3, 4, 8})
    for (int S : {1, 100, 128, 129, 256, 384, 512, 768, 1000, 1280, 2048})
      for (int causal = 0; causal < 2; ++causal)
        for (int zigzag = 0; zigzag < 2; ++zigzag) {
          if ((S % 128 && W > 1) || (zigzag && S % 256)) continue;
          const int T = (S + 127) / 128;
          for (int r = 0; r < W; ++r)
            for (int q = 0; q < T; ++q) {
              int e = check<false>(W, r, S, causal, zigzag, Item{{q, q}, {0, 1}, 0, 2});           // two heads of one tile
              if (!e) e = check<true>(W, r, S, causal, zigzag, Item{{q, q}, {0, 0}, 0, 2});         // one tile, by keys
              if (!e && q % 2 == 0) e = check<false>(W, r, S, causal, zigzag, Item{{q, q + 1}, {0, 0}, 0, q + 1 < T ? 2 : 1});
              if (e) { printf("W %d r %d S %d causal %d zigzag %d q %d: %d\n", W, r, S, causal, zigzag, q, e); return 1; }
              forms += 3;
            }
        }
  printf("%ld forms agree\n", forms);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host C++ compiler")
def test_tile_walk_visits_what_the_mask_allows_and_counts_it(tmp_path):
    with open(os.path.join(ROOT, "csrc", "kernels", "ring_attention_tc.cu")) as f:
        text = f.read()
    parts = [re.search(r"^struct Item \{.*?^\};", text, re.S | re.M), re.search(r"^template <bool kByKeys>\nstruct TileWalk \{.*?^\};", text, re.S | re.M)]
    src = tmp_path / "walk.cpp"
    src.write_text(_DRIVER.replace("@SOURCE@", "\n".join(p.group(0) for p in parts)))
    build = subprocess.run(["g++", "-O1", "-std=c++17", "-Wno-unknown-pragmas", str(src), "-o", str(tmp_path / "walk")], capture_output=True, text=True, timeout=120)
    assert build.returncode == 0, build.stderr[-3000:]
    run = subprocess.run([str(tmp_path / "walk")], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and "forms agree" in run.stdout, run.stdout
