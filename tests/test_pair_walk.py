"""How CTA pairs share out the tiles of a product (xotorch_b200/csrc/prefill_tc.cuh, PairWalk): the header's own rule and walk, compiled for the host, over pair
counts, K blocks and tile counts — every K block of every tile exactly once, one finisher a tile, one slot a piece, and the finisher's list of slots is the
tile's earlier pieces in the order of K."""
import shutil
import subprocess
from pathlib import Path

import pytest

SRC = Path(__file__).resolve().parent.parent / "xotorch_b200" / "csrc" / "prefill_tc.cuh"
MAIN = r"""
int main() {
  long bad = 0, cut = 0;
  for (int pairs : {1, 2, 3, 7, 66, 74})
    for (int nkb = 1; nkb <= 420; nkb += nkb < 20 ? 1 : 13)
      for (int total = 1; total <= 4 * pairs + 3; ++total) {
        const PairSplit sp = pair_split(total, pairs, nkb);
        const int np = pair_count(total, pairs, sp);
        bad += np > pairs || np < 1;
        cut += sp.n[0] > 0;
        struct Piece { int pair, t, k0, k1, slot, step, front; };
        std::vector<Piece> left, finish;
        std::vector<int> blocks(total, 0), used(pair_slots(pairs), 0);
        std::vector<std::vector<std::pair<int, int>>> cover(total);
        for (int p = 0; p < np; ++p) {
          const PairWalk w(total, nkb, np, p, sp);
          for (int i = 0, t, k0, k1, slot = -1, step = 0; w.get(i, t, k0, k1, slot, step); ++i) {
            if (t < 0 || t >= total || k0 < 0 || k0 >= k1 || k1 > nkb || i > total) { ++bad; break; }
            cover[t].push_back({k0, k1});
            const bool part = k1 < nkb;
            const int front = k0 == 0 && !part ? 0 : w.before(t);
            bad += (k0 > 0) != (front > 0);
            if (part) {
              const int id = slot + front * step;
              if (id < 0 || id >= (int)used.size()) ++bad; else ++used[id];
              left.push_back({p, t, k0, k1, slot, step, front});
            } else {
              finish.push_back({p, t, k0, k1, slot, step, front});
            }
          }
        }
        for (auto& c : cover) {
          std::sort(c.begin(), c.end());
          int at = 0;
          for (auto& x : c) { bad += x.first != at; at = x.second; }
          bad += at != nkb;
        }
        for (int u : used) bad += u > 1;
        bad += (int)finish.size() != total;
        for (auto& f : finish) {
          std::vector<std::pair<int, int>> mine;
          for (auto& l : left) if (l.t == f.t) mine.push_back({l.k0, l.slot + l.front * l.step});
          std::sort(mine.begin(), mine.end());
          bad += (int)mine.size() != f.front;
          for (size_t i = 0; i < mine.size() && (int)i < f.front; ++i) bad += mine[i].second != f.slot + (int)i * f.step;
        }
      }
  printf("%ld %ld\n", bad, cut);
}
"""


def test_every_block_once(tmp_path):
  if not shutil.which("g++"):
    pytest.skip("no host compiler")
  text = SRC.read_text()
  struct = text[text.index("struct PairSplit {"):]
  struct = struct[:struct.index("};") + 2]
  walk = text[text.index("constexpr int PAIR_SLOT"):text.index("// 16 columns (piece c of 8)")]
  (tmp_path / "walk.cpp").write_text("#include <algorithm>\n#include <cstdio>\n#include <vector>\n#define __device__\n#define __host__\n#define __forceinline__ inline\n" + struct + "\n" + walk + MAIN)
  subprocess.check_call(["g++", "-O1", "-std=c++17", "-o", str(tmp_path / "walk"), str(tmp_path / "walk.cpp")])
  bad, cut = map(int, subprocess.check_output([str(tmp_path / "walk")], text=True).split())
  assert bad == 0 and cut > 1000
