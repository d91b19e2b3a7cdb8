"""The merge scratch of the tensor-core search, on the CPU: sized for a capacity, it gives
every smaller search the slots that its parts on all SMs need, whatever it was sized for,
and does not grow with slots times queries."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-orb_b200", "csrc")
SOURCE = r"""
#define __host__
#define __device__
#include "orbx_match_plan.cuh"
#include <cstdio>
#include <initializer_list>
using namespace orbx;
int main() {
  for (int cap : {1, 128, 256, 300, 2048, 2049, 10000, 32768, 70001})
    for (int ndb_cap : {0, 240, 30720, 131072, 737280, 1100001, (1 << 22) - 1}) {
      const long long rows = m_part_rows(cap, ndb_cap);
      // no more than 32 slots of every query, or what every SM's part of 256 needs
      if (rows > 32ll * cap + 256 * 168) { printf("cap %d ndb %d: %lld rows\n", cap, ndb_cap, rows); return 1; }
      for (int nq : {1, 100, 256, 257, 512, 1500, 2048, 2049, 5000, 10000, 32768, 70001})
        for (int ndb : {0, 1, 241, 4801, 131072, 262144, 737280, 800000, 1100001, (1 << 22) - 1}) {
          if (nq > cap || ndb > ndb_cap) continue;
          const int slots = m_slots(rows, nq);
          const MPlan p = m_plan(nq, ndb, slots, kPlanGrid), best = m_plan(nq, ndb, 1 << 20, kPlanGrid);
          if (p.grid != best.grid || p.panels != best.panels) {
            printf("cap %d: %d in %d: %d of %d blocks\n", cap, nq, ndb, p.grid, best.grid);
            return 1;
          }
          if ((long long)slots * nq > rows) { printf("cap %d: %d slots of %d\n", cap, slots, nq); return 1; }
          for (int qb = 0; qb < p.qtiles; qb++) {
            int n, slot;
            m_slot(p, slots, qb, 0, m_block(p, slots, (long long)qb * m_panel_tiles(p, 0)), &n, &slot);
            if (n > slots) { printf("cap %d: %d in %d: %d parts, %d slots\n", cap, nq, ndb, n, slots); return 1; }
          }
        }
    }
  return 0;
}
"""


def test_scratch_fits_every_smaller_search(tmp_path):
    src, exe = tmp_path / "scratch.cpp", tmp_path / "scratch"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-x", "c++", "-I", CSRC, str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
