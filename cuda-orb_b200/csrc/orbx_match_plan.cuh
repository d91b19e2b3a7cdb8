// The split of a tensor-core search over thread blocks (orbx_match_imma.cu): plain
// arithmetic, the same on the host, which sizes the grid and the scratch, and in
// every block.
#pragma once

namespace orbx {

// How the blocks share a search.  The pairs (256 queries, database tile) lie in one
// line, a block of queries' tiles in a row, and each block takes an equal length of
// it: at most one start and one end inside a block of queries, so few scans begin
// anew (a scan's first columns nearly all enter the top two), and no block waits for
// a last wave.  A database larger than the L2 goes by panels, all queries against
// one before the next, so that the blocks read the same tiles at about the same time.
// Blocks of queries whose tiles lie with several thread blocks merge their results
// through `slots` slots of MatchWork::part.
constexpr int kPlanQueries = 256;   // queries of a block of queries
constexpr int kPlanRows = 240;      // database rows of a tile
constexpr int kMPanel = 2048;       // tiles of a panel: 63 MB of expanded rows
constexpr int kMPanelFrom = 3072;   // tiles from which a database goes by panels
constexpr int kMPanelQueries = 8;   // blocks of queries up to which it never does
struct MPlan {
  int qtiles, dbtiles, panels, grid;
  long long total;
};
struct MPart {
  int qb, t0, t1;  // database tiles [t0, t1)
};
__host__ __device__ inline MPlan m_plan(int nq, int ndb, int slots, int grid) {
  MPlan p;
  p.qtiles = (nq + kPlanQueries - 1) / kPlanQueries;
  p.dbtiles = ndb > kPlanRows ? (ndb + kPlanRows - 1) / kPlanRows : 1;  // an empty database: one tile without rows
  p.panels = p.dbtiles < kMPanelFrom || p.qtiles <= kMPanelQueries ? 1 : (p.dbtiles + kMPanel - 1) / kMPanel;
  p.total = (long long)p.qtiles * p.dbtiles;
  // a block of queries has at most grid / qtiles + 2 * panels parts
  if (slots <= 2 * p.panels) p.panels = 1;
  long long g = slots > 2 ? (long long)(slots - 2 * p.panels) * p.qtiles : p.qtiles;
  g = g < p.total ? g : p.total;
  p.grid = (int)(g < grid ? g : grid);
  // few blocks of queries: no thread block has two of them, where that idles at most
  // a sixteenth (1500 x 262144: 144 blocks instead of 148)
  if (slots > 2 && p.qtiles && p.qtiles < p.grid && p.grid % p.qtiles * 16 <= p.grid) p.grid -= p.grid % p.qtiles;
  return p;
}
// First pair of block b (whole blocks of queries when there are no slots to merge).
__host__ __device__ inline long long m_start(const MPlan& p, int slots, int b) {
  return slots > 2 ? p.total * b / p.grid : (long long)p.qtiles * b / p.grid * p.dbtiles;
}
// The block whose pairs hold pair x.
__host__ __device__ inline int m_block(const MPlan& p, int slots, long long x) {
  return slots > 2 ? (int)(((x + 1) * p.grid - 1) / p.total)
                   : (int)(((x / p.dbtiles + 1) * p.grid - 1) / p.qtiles);
}
__host__ __device__ inline int m_panel_tiles(const MPlan& p, int panel) {
  return panel == p.panels - 1 ? p.dbtiles - panel * kMPanel : kMPanel;
}
// The part of the pairs [x, end) that lies in one block of queries and one panel.
__host__ __device__ inline MPart m_part(const MPlan& p, long long x, long long end) {
  MPart r;
  int panel = 0;
  if (p.panels > 1) {
    panel = (int)(x / ((long long)p.qtiles * kMPanel));
    panel = panel < p.panels - 1 ? panel : p.panels - 1;
  }
  const int tiles = m_panel_tiles(p, panel);
  const long long y = x - (long long)p.qtiles * kMPanel * panel;
  r.qb = (int)(y / tiles);
  const int t = (int)(y - (long long)r.qb * tiles);
  const long long n = end - x < tiles - t ? end - x : tiles - t;
  r.t0 = panel * kMPanel + t;
  r.t1 = r.t0 + (int)n;
  return r;
}
// Parts that block of queries qb has, and the place among them of the one that
// block b makes of database tile t.
__host__ __device__ inline void m_slot(const MPlan& p, int slots, int qb, int t, int b, int* count, int* slot) {
  int n = 0;
  *slot = 0;
  for (int panel = 0; panel < p.panels; panel++) {
    const int tiles = m_panel_tiles(p, panel);
    const long long x = (long long)p.qtiles * kMPanel * panel + (long long)qb * tiles;
    const int b0 = m_block(p, slots, x), b1 = m_block(p, slots, x + tiles - 1);
    if (t >= panel * kMPanel && t < panel * kMPanel + tiles) *slot = n + b - b0;
    n += b1 - b0 + 1;
  }
  *count = n;
}

// Merge scratch of searches of up to nq queries in up to ndb rows, in rows of one query's
// best two.  A search of n queries takes `slots` of them each, by the count it finds on
// the device, so few queries have as many slots as their parts on all SMs need, whatever
// the scratch was sized for: 148 / qtiles + 1 + 2 * panels (m_plan) for each of n <= 256 *
// qtiles.  32768 queries in 131072 rows: 1.1 MB (20 MB as 77 slots for every query).
constexpr int kPlanGrid = 148;      // blocks of a launch: one per SM
constexpr int kPlanMaxSlots = 152;  // every SM has a part of one block of queries
__host__ __device__ inline long long m_part_rows(int nq, int ndb) {
  const MPlan p = m_plan(nq, ndb, 1 << 20, kPlanGrid);
  return (long long)kPlanQueries * (kPlanGrid + (long long)p.qtiles * (1 + 2 * p.panels));
}
__host__ __device__ inline int m_slots(long long part_rows, int nq) {
  // (the kernel's part_rows has 32 bits, and so has its division)
  const long long s = nq <= 0 ? 0 : part_rows >> 32 ? part_rows / nq : (long long)((unsigned)part_rows / (unsigned)nq);
  return s < 1 ? 1 : s > kPlanMaxSlots ? kPlanMaxSlots : (int)s;
}

// Of n uses that went round a ring of k entries, those of entry i.  A block does not
// exit before the last commit to each of its barriers has arrived: the arrival is a
// write to its shared memory, which may belong to another block by then.
__host__ __device__ inline unsigned m_ring_uses(unsigned n, unsigned k, unsigned i) { return (n + k - 1 - i) / k; }

}  // namespace orbx
