"""The split of the tensor-core search over thread blocks, on the CPU: every pair of
query block and database tile belongs to exactly one part, the parts of a block of
queries have places 0 .. count - 1 once each, and the places fit the slots."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-orb_b200", "csrc")
SOURCE = r"""
#define __host__
#define __device__
#include "orbx_match_plan.cuh"
#include <cstdio>
#include <cstdlib>
#include <vector>
using namespace orbx;
static int check(int nq, int ndb, int slots, int grid) {
  const MPlan p = m_plan(nq, ndb, slots, grid);
  const int qt = (nq + 255) / 256, dt = ndb > 240 ? (ndb + 239) / 240 : 1;
  if (p.qtiles != qt || p.dbtiles != dt || (nq > 0) != (p.grid > 0) || p.grid > grid) return 1;
  if (!nq) return 0;
  std::vector<char> seen((size_t)qt * dt, 0);
  std::vector<int> count(qt, -1);
  std::vector<std::vector<char>> place(qt);
  long long longest = 0;
  for (int b = 0; b < p.grid; b++) {
    const long long end = m_start(p, slots, b + 1);
    if (m_start(p, slots, b) >= end) return 2;
    if (end - m_start(p, slots, b) > longest) longest = end - m_start(p, slots, b);
    for (long long x = m_start(p, slots, b); x < end;) {
      const MPart r = m_part(p, x, end);
      if (r.qb < 0 || r.qb >= qt || r.t0 < 0 || r.t1 <= r.t0 || r.t1 > dt) return 3;
      for (int t = r.t0; t < r.t1; t++)
        if (seen[(size_t)r.qb * dt + t]++) return 4;
      int n, slot;
      m_slot(p, slots, r.qb, r.t0, b, &n, &slot);
      if (count[r.qb] < 0) { count[r.qb] = n; place[r.qb].assign(n, 0); }
      if (n != count[r.qb] || slot < 0 || slot >= n || place[r.qb][slot]++) return 5;
      if (slots <= 2 ? n != 1 : n > slots) return 6;
      x += r.t1 - r.t0;
    }
  }
  for (char c : seen) if (c != 1) return 7;
  for (auto& v : place) for (char c : v) if (c != 1) return 8;
  if (slots > 2 && longest > p.total / p.grid + 1) return 9;
  return 0;
}
int main(int, char** v) {
  const int grid = atoi(v[1]);
  for (int slots : {1, 2, 3, 5, 17, 64, 152})
    for (int nq : {0, 1, 256, 257, 600, 2048, 2049, 5000, 37888, 65536, 70001})
      for (int ndb : {0, 1, 240, 241, 480, 4801, 30720, 262144, 737280, 800000, 1100001}) {
        const int bad = check(nq, ndb, slots, grid);
        if (bad) { printf("%d: nq %d ndb %d slots %d\n", bad, nq, ndb, slots); return 1; }
      }
  return 0;
}
"""


@pytest.mark.parametrize("grid", [1, 2, 147, 148])
def test_every_pair_once_and_slots_fit(tmp_path, grid):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-x", "c++", "-I", CSRC, str(src), "-o", str(exe)])
    out = subprocess.run([str(exe), str(grid)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
