// Brute-force k = 2 Hamming matching, XOR + popcount form, for sm_100a.
//
// gHammingMatch (orbd.cu:1471-1559) gives each query a 32-thread block that
// re-reads the whole train set.  Here a block owns 128 queries, one per thread
// and row group, held in registers, and streams a slice of the train set through
// shared memory, so each train row is read once per 128 queries.  When there are
// few queries the train set is split across blocks; the last block to finish a
// query tile merges the partial results.  The running top-2 is kept as two
// 32-bit keys (distance << 22 | index), which orders by distance, then index.
//
// What bounds it: at thousands of queries the integer units (hamming256: 16
// logic operations and 4 population counts per pair; 8 of each before), below
// that the chain of dependent global accesses around a short scan.  Four row
// groups of 128 threads per block shorten that scan and the merge fourfold.
// 5000 x 4801: 53.3 -> 39.8 us; 16384 x 32768: 1021 -> 695 us (the ALU is full: 48
// cycles per warp and row); 1100 x 1300 with counts on the device: 9.5 -> 8.4 us.
// Two queries per thread, which halves the shared-memory reads, was slower (870
// us): each check then covers fewer rows and passes more often.
#include <algorithm>

#include "orbx_stages.cuh"

namespace orbx {

constexpr int kMThreads = kMQ * kMGroups;
constexpr int kMResident = 2;  // blocks per SM

__global__ void __launch_bounds__(kMThreads, kMResident) k_match_popc(MatchArgs a, MatchWork w) {
  __shared__ MatchSmem<kMGroups> sm;
  chain_wait();
  match_popc_block<kMGroups, false>(a, w, blockIdx.x, gridDim.x, sm);
}

__global__ void __launch_bounds__(kMThreads, kMResident) k_match_popc_batch(const MatchJob* jobs) {
  __shared__ MatchSmem<kMGroups> sm;
  chain_wait();
  const MatchJob& J = jobs[blockIdx.y];
  match_popc_block<kMGroups, false>(J.args, J.work, blockIdx.x, gridDim.x, sm);
}

// Grid of one search: full waves of resident blocks where the query count is
// known.  Of the splits that give 1 to 4 waves the cheapest is taken; a wave costs
// a split's rows plus about 50 rows' worth of fixed latencies per block (5000 x
// 4801: 39.8 us, 44.6 us with as many splits as blocks would allow).  Counts on the
// device: two waves at the default blocks_per_sm of 8 (of 256 threads), spread by
// the kernel; blocks without work exit.
static int match_popc_blocks(int nq_cap, int ndb, int splits_cap, bool counted, int blocks_per_sm) {
  const int tiles = (nq_cap + kMQ - 1) / kMQ;
  const int resident = 148 * kMResident;
  if (counted) {
    const int most = std::min(splits_cap, std::max(1, (ndb + 63) / 64));
    int best = 1;
    double best_cost = 1e300;
    for (int s = 1; s <= most; s++) {
      const long long waves = ((long long)tiles * s + resident - 1) / resident;
      const double cost = (double)waves * ((double)ndb / s + 50.0);
      if (cost < best_cost) {
        best_cost = cost;
        best = s;
      }
    }
    return tiles * best;
  }
  const long long target = (long long)(blocks_per_sm > 0 ? blocks_per_sm : 8) * 148 / 2;
  long long blocks = (long long)tiles * splits_cap;
  if (blocks > target) blocks = target;
  if (blocks < tiles) blocks = tiles;
  return (int)blocks;
}

cudaError_t launch_match_popc(const MatchArgs& a, const MatchWork& w, cudaStream_t s, int blocks_per_sm) {
  if (w.nq_cap <= 0) return cudaSuccess;
  const bool counted = !a.d_nq && !a.d_ndb;
  const int nq = counted ? std::min(a.nq, w.nq_cap) : w.nq_cap;
  if (nq <= 0) return cudaSuccess;
  return launch_chained(k_match_popc, match_popc_blocks(nq, a.ndb, w.splits_cap, counted, blocks_per_sm), kMThreads, s, a,
                        w);
}

cudaError_t launch_match_popc_batch(const MatchJob* d_jobs, int n_jobs, int blocks_per_job, cudaStream_t s) {
  if (n_jobs <= 0 || blocks_per_job <= 0) return cudaSuccess;
  return launch_chained(k_match_popc_batch, dim3(blocks_per_job, n_jobs), kMThreads, s, d_jobs);
}

}  // namespace orbx
