"""The kernels' own work splits (tk_split.h, compiled here for the host): every unit,
tile, row and job exactly once, as one front through the batch; the batch kernels'
TMA ring under that split, with the loop left after a short tile; and the three tile
kinds of the matrix-vector kernel, six-row boxes included."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "tensorkyber_b200", "csrc")

DRIVER = r"""
#include <stdio.h>
#include <stdlib.h>
#include <algorithm>
#include <vector>
#include "tk_split.h"
using namespace tk;

#define CHECK(c) do { if (!(c)) { printf("FAIL line %d: %s\n", __LINE__, #c); exit(1); } } while (0)

// k_ntt_mma with S slots on nunits units and G CTAs
template <int W, bool kDown>
static void batch(int nunits, int G, int S, bool short_tiles) {
  std::vector<char> seen(nunits);
  std::vector<int> lo, hi;                       // extent of tile k over the launch
  int least = 1 << 30, most = 0;
  for (int c = 0; c < G; c++) {
    const FrontTiles<W, kDown> T(nunits, G, c);
    const int n = T.tiles();
    std::vector<int> slot(S, -1), uses(S, 0);    // tile loaded; completed phases
    auto load = [&](int k, int s) { CHECK(slot[s] == -1); slot[s] = k; uses[s]++; };
    for (int t = 0; t < S - 1; t++) if (t < n) load(t, t);
    int s = 0, phase = 0, units = 0, k = 0;
    for (; k < n; k++) {
      CHECK(slot[s] == k && ((uses[s] - 1) & 1) == phase);    // the wait's tile and parity
      if (k + S - 1 < n) load(k + S - 1, (s + S - 1) % S);
      const int u0 = T.unit0(k), nu = T.units(k);
      CHECK(nu > 0 && nu <= W && u0 >= 0 && u0 + nu <= nunits);
      for (int u = u0; u < u0 + nu; u++) { CHECK(!seen[u]); seen[u] = 1; }
      units += nu;
      if ((int)lo.size() <= k) { lo.push_back(u0); hi.push_back(u0 + nu); }
      lo[k] = std::min(lo[k], u0);
      hi[k] = std::max(hi[k], u0 + nu);
      slot[s] = -1;
      if (short_tiles && nu <= 3 * W / 4) { CHECK(k == n - 1); k++; break; }
      if (++s == S) { s = 0; phase ^= 1; }
    }
    CHECK(k == n);
    for (int t : slot) CHECK(t == -1);           // no load in flight when the CTA ends
    least = std::min(least, units);
    most = std::max(most, units);
  }
  for (char x : seen) CHECK(x);
  CHECK(most - least <= 1);
  for (size_t k = 1; k < lo.size(); k++) CHECK(kDown ? hi[k] <= lo[k - 1] : lo[k] >= hi[k - 1]);
}

static void tc(int ntiles, int G, bool down) {
  std::vector<char> seen(ntiles);
  for (int c = 0; c < G; c++)
    for (int k = 0, n = front_tile_count(ntiles, G, c); k < n; k++) {
      const int t = front_tile(ntiles, G, c, k, down);
      CHECK(t >= 0 && t < ntiles && !seen[t]);
      CHECK((down ? ntiles - 1 - t : t) / G == k);
      seen[t] = 1;
    }
  for (char x : seen) CHECK(x);
}

// one batch of the matrix-vector kernel in tiles of kind `units`
static void matvec(int k, int units, int njobs) {
  const int nvec = njobs * k, tj = tile_jobs(k, units), box = tile_box_rows(k, units);
  CHECK(tj * k == tile_rows(k, units) && tile_units(k, units) <= (units == 1 ? 1 : 4));
  std::vector<char> rows(nvec), jobs(njobs);
  for (int t = 0; t < (njobs + tj - 1) / tj; t++) {
    const int row0 = t * tile_rows(k, units);
    for (int w = 0; w < tile_units(k, units); w++)   // box w: rows of the batch
      for (int r = row0 + 8 * w; r < std::min(row0 + 8 * w + box, nvec); r++) {
        CHECK(!rows[r]);
        rows[r] = 1;
      }
    for (int j = 0; j < tj && t * tj + j < njobs; j++) {
      CHECK(!jobs[t * tj + j]);
      jobs[t * tj + j] = 1;
      for (int i = 0; i < k; i++) {                  // the job's rows: in the tile, in a box
        const int at = j * k + i;
        CHECK(row0 + at == (t * tj + j) * k + i && at < tile_rows(k, units));
        CHECK(at / 8 < tile_units(k, units) && at % 8 < box);
      }
    }
  }
  for (char x : rows) CHECK(x);
  for (char x : jobs) CHECK(x);
}

int main() {
  const int sizes[] = {1, 2, 3, 4, 5, 7, 8, 37, 443, 444, 445, 888, 1332, 1776, 1777, 2051, 12501,
                       32768, 131073};
  const int grids[] = {1, 3, 148, 296, 444, 592};
  for (int n : sizes)
    for (int g : grids) {
      const int G = std::min(g, n);
      for (int S = 2; S <= 3; S++) {
        batch<4, false>(n, G, S, true);
        batch<4, true>(n, G, S, true);
        batch<8, false>(n, G, S, true);
        batch<8, true>(n, G, S, true);
        batch<4, false>(n, G, S, false);             // several segments, addend
        batch<4, true>(n, G, S, false);
      }
      tc(n, std::min(n, 148), false);
      tc(n, std::min(n, 148), true);
    }
  for (int k = 2; k <= 4; k++)
    for (int units : {1, 2, 4})
      for (int n = 1; n <= 70; n++) matvec(k, units, n);
  printf("ok\n");
  return 0;
}
"""


def test_splits_of_the_kernels(tmp_path):
    src, exe = tmp_path / "split.cpp", tmp_path / "split"
    src.write_text(DRIVER)
    p = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", f"-I{CSRC}", str(src),
                        "-o", str(exe)], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout


@pytest.mark.parametrize("was,now", [("(k * G + cta) * W", "(k * G + cta) * W + 1"),
                                     ("left0 = (int)((long long)cta", "left0 = (int)((long long)(cta + 1)"),
                                     ("k == 3 && units == 1 ? 6 : 8", "8")])
def test_a_wrong_split_is_seen(tmp_path, was, now):
    src, exe = tmp_path / "split.cpp", tmp_path / "split"
    src.write_text(DRIVER)
    with open(os.path.join(CSRC, "tk_split.h")) as f:
        text = f.read()
    assert was in text
    (tmp_path / "tk_split.h").write_text(text.replace(was, now))
    subprocess.run(["g++", "-std=c++17", "-O2", f"-I{tmp_path}", str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 1 and "FAIL" in r.stdout
