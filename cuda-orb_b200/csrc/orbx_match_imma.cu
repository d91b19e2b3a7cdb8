// Brute-force k = 2 Hamming matching on the 5th-generation tensor cores.
//
// A 256-bit descriptor b is expanded to 256 values s_k = 2*b_k - 1 (+-1), so for
// two descriptors dot(s, t) = 256 - 2 * Hamming(s, t).  The values are 4-bit floats
// (e2m1, where +-1 is exact) with block scales of 1, multiplied by tcgen05.mma
// kind::mxf4 into fp32: every partial sum is a whole number of at most 256, so the
// dot product is exact.  One block owns up to 256 queries, as two query tiles of
// 128 (the MMA's M) that stay in shared memory, and walks 240-row database tiles
// (the MMA's N) with K = 256 = four K=64 MMA steps per database and query tile:
//   warp 0     TMA producer: the query tiles once, database tiles through a
//              4-stage shared-memory ring (128-byte swizzle, no multicast);
//   warp 1     MMA issuer: one elected thread issues the four MMAs of a step
//              into one of two TMEM accumulators (240 columns; the scales take
//              16 of the others) and commits them to the ring's "empty" (after a
//              database tile's last step) and the accumulator's "full" barriers;
//   warps 2-17 epilogue, two sets of eight: set s takes every second step, i.e.
//              accumulator s.  A warp reads its 32 TMEM lanes (queries) over half
//              the columns, 60 at a time, and keeps a running best / second-best
//              key per query.
// Steps alternate between the two query tiles of a database tile, so set s holds
// query tile s; with at most 128 queries there is one query tile, the steps
// alternate between database tiles, and the sets' results are merged.
// The block's result per query is the top-2 by (distance, index), the same
// keys as the XOR-popc kernel (orbx_match.cu), so both forms agree bit for bit.
// Every barrier wait is bounded by a clock deadline; on expiry the block
// records kErrImmaTimeout, drains its in-flight copies, frees TMEM and exits.
//
// What bounds it: the epilogue.  With int8 values (kind::i8, half the rate and twice
// the bytes) 65536 x 65536 took 785 us, 660 of them the tensor pipe's; now the MMAs
// alone need 336 us, with the loads of their results 357, with the maximum test of
// every chunk 445.  The rest are the chunks that pass it: a warp that examines one
// keeps its accumulator, so the others wait for it.  They are kept few by long scans
// (orbx_match_plan.cuh: 616 -> 532 us) and by bounds shared between column parts, sets
// and blocks, and cheap by tournaments over column groups.  A chunk is what the
// registers hold: each costs a round trip to TMEM (40 columns: 563 us).  More, shorter
// accumulators or more epilogue warps were slower (3 x 160 columns 685 against 646 us,
// 24 warps 767: each step costs every warp about 700 cycles).  From int8 values to
// this form: 65536 x 65536 785 -> 532 us, 1500 x 262144 95 -> 73 us.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <utility>

#include "orbx_device.cuh"
#include "orbx_internal.cuh"
#include "orbx_match_plan.cuh"

namespace orbx {

constexpr int kIBM = 128;  // queries per query tile (MMA M)
constexpr int kIBQ = kPlanQueries;  // queries per block of k_match_imma
static_assert(kIBQ == 2 * kIBM, "two query tiles");
constexpr int kMBN = kPlanRows;  // database rows per tile of k_match_imma: two accumulators leave TMEM columns for the scales
constexpr int kMChunk = 60;           // columns an epilogue warp examines at a time,
constexpr int kMGroups = 4;           // in so many groups
constexpr int kMParts = 2;            // epilogue warps per set and 32 TMEM lanes
constexpr int kMChunks = kMBN / (kMChunk * kMParts);  // chunks of one of them per step
constexpr int kMEpiWarps = 2 * 4 * kMParts;
constexpr int kMThreads = (2 + kMEpiWarps) * 32;
constexpr int kMStages = 4;
constexpr int kIEpiWarps = 8;  // of k_rerank_imma
constexpr uint32_t kMATile = kIBM * kPm1RowBytes;  // one 128-byte swizzle row per descriptor
constexpr uint32_t kMBTile = kMBN * kPm1RowBytes;
static_assert(kPm1RowBytes == 128 && kMBTile % 1024 == 0, "whole swizzle atoms");
constexpr uint32_t kMNumBars = 2 * 2 + 2 * kMStages + 2 * 2 + 1;  // full and empty: query tiles, ring, accumulators; the epilogue's own
// accumulator a starts at TMEM column 256 * a; the scales (all 1) lie between them
constexpr uint32_t kMAcc = 256;
constexpr uint32_t kMScaleCol = kMBN, kMScaleCols = 16;
// 1024 bytes of alignment slack, two pairs of query tiles, the ring, the merge scratch
// (best two per set, column part and row), the barriers, TMEM base + abort flag
constexpr uint32_t kIMergeBytes = 2 * kMParts * kIBM * 8;
constexpr uint32_t kISmemBytes = 1024 + 4 * kMATile + kMStages * kMBTile + kIMergeBytes + 8 * kMNumBars + 16;
// dynamic tiles + the static s_last and per-row bounds
static_assert(kISmemBytes + 16 + 2 * kMParts * kIBM * 4 <= 232448, "exceeds the 227 KB shared-memory opt-in");
constexpr uint32_t kITmemCols = 512;
constexpr long long kIDeadlineCycles = 4000000000ll;  // ~2 s at 2 GHz

// instruction descriptor for kind::mxf4: E2M1 x E2M1, UE8M0 scales, both K-major, N = 240, M = 128, K = 64
constexpr uint32_t kMDesc = (1u << 7) | (1u << 10) | ((uint32_t)(kMBN >> 3) << 17) | (1u << 23) |
                            ((uint32_t)(kIBM >> 7) << 27);

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1u << 16) | ((uint64_t)(1024u >> 4) << 32) |
         ((uint64_t)1u << 46) | ((uint64_t)2u << 61);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// A waiting thread is suspended by the barrier unit (woken when the phase
// completes, or after this many nanoseconds) instead of spinning on the
// ALU pipe that the epilogue warps need.
constexpr uint32_t kTryWaitSuspendNs = 20000;
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(kTryWaitSuspendNs)
      : "memory");
  return ok != 0;
}

// Bounded wait: false once the block's deadline has passed or another role aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long deadline,
                                          volatile int* abort_flag) {
  while (!mbar_try(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() > deadline) return false;
  }
  return true;
}

// The last of a barrier's `uses` phases, each of one commit, is over (bounded).
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t uses) {
  if (!uses) return;
  const long long deadline = clock64() + kIDeadlineCycles;
  while (!mbar_try(bar, (uses - 1) & 1u) && clock64() < deadline) {
  }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          dst),
      "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// One K = 64 step on 4-bit floats with one scale per 32 values (all 1, at sfa and sfb).
__device__ __forceinline__ void umma_f4(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t sfa,
                                        uint32_t sfb, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%5], p;\n\t}" ::"r"(
          tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(sfa), "r"(sfb), "r"(acc)
      : "memory");
}

// Scales of 1 (UE8M0 127) in this warp's 32 lanes of 16 TMEM columns.
__device__ __forceinline__ void tmem_store_unit_scales(uint32_t taddr) {
  const uint32_t one = 0x7F7F7F7Fu;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
      "%1};" ::"r"(taddr),
      "r"(one)
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- reading and comparing the fp32 accumulators -----------------------------
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]),
        "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]),
        "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),
        "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(taddr));
}
// N values of the lane's row, loaded and waited for; as operands of the statements
// after the wait they cannot be read before it.
template <int N>
__device__ __forceinline__ void tmem_read(uint32_t taddr, float* v) {
  static_assert(N % 4 == 0 && N < 64, "loads of 32, 16, 8 and 4");
  if constexpr (N & 32) tmem_ld32(taddr, v);
  if constexpr (N & 16) tmem_ld16(taddr + (N & 32), v + (N & 32));
  if constexpr (N & 8) tmem_ld8(taddr + (N & 48), v + (N & 48));
  if constexpr (N & 4) tmem_ld4(taddr + (N & 56), v + (N & 56));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; i += 4)
    asm volatile("" : "+f"(v[i]), "+f"(v[i + 1]), "+f"(v[i + 2]), "+f"(v[i + 3])::"memory");
}
// Value given to columns that hold no database row (below every dot product).
constexpr float kMaskedDotF = -400.f;

__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// Conversions of small whole numbers by the add whose rounding leaves them in the low
// mantissa bits: two operations, where a convert instruction makes the chain wait.
__device__ __forceinline__ int whole_to_int(float u) { return __float_as_int(u + 12582912.f) - 0x4B400000; }
__device__ __forceinline__ float int_to_whole(int i) { return __int_as_float(i + 0x4B400000) - 12582912.f; }

// The maximum of N values, by three-input maxima.
template <int N>
__device__ __forceinline__ float max_of(const float* v) {
  float m[N];
#pragma unroll
  for (int i = 0; i < N; i++) m[i] = v[i];
  int n = N;
#pragma unroll
  for (int round = 0; round < 4; round++) {
    int o = 0;
#pragma unroll
    for (int i = 0; i < N; i += 3) {
      if (i + 2 < n) m[o++] = fmax3(m[i], m[i + 1], m[i + 2]);
      else if (i + 1 < n) m[o++] = fmaxf(m[i], m[i + 1]);
      else if (i < n) m[o++] = m[i];
    }
    n = o;
  }
  return m[0];
}
// The best two of columns B .. E-1 of a chunk, merged into the running best two
// keys (distance << 22 | index): local keys u = column - 64 * dot, whole numbers
// below 2^15 and exact in fp32, go through a tournament of minima (its depth, not
// its 23 operations for ten columns, is what a warp waits for), so ties keep the
// lower column.  base is the key of a zero dot product at the chunk's column 0, and
// a value of one takes 1 << SH off.  Masked columns carry no key.
template <int B, int E, int SH>
__device__ __forceinline__ void push_best2(const float* vc, uint32_t base, uint32_t& k1, uint32_t& k2) {
  constexpr int n = E - B, h = n / 2;
  float a1[h], a2[h];
#pragma unroll
  for (int i = 0; i < h; i++) {
    const float x = fmaf(vc[B + 2 * i], -64.f, (float)(B + 2 * i)),
                y = fmaf(vc[B + 2 * i + 1], -64.f, (float)(B + 2 * i + 1));
    a1[i] = fminf(x, y);
    a2[i] = fmaxf(x, y);
  }
#pragma unroll
  for (int d = 1; d < h; d *= 2)
#pragma unroll
    for (int i = 0; i + d < h; i += 2 * d) {
      a2[i] = fmin3(fmaxf(a1[i], a1[i + d]), a2[i], a2[i + d]);
      a1[i] = fminf(a1[i], a1[i + d]);
    }
  float u1 = a1[0], u2 = a2[0];
  if constexpr (n & 1) {
    const float x = fmaf(vc[E - 1], -64.f, (float)(E - 1));
    u2 = fminf(u2, fmaxf(u1, x));
    u1 = fminf(u1, x);
  }
  auto key = [&](float u) {
    const int i = whole_to_int(u);
    return u >= -64.f * kMaskedDotF ? kNoKeyShared : base + ((uint32_t)(i >> 6) << SH) + (uint32_t)(i & 63);
  };
  const uint32_t p1 = key(u1), p2 = key(u2);
  k2 = __vimin3_u32(max(k1, p1), k2, p2);
  k1 = min(k1, p1);
}

// Expands 256-bit descriptors to rows of 256 e2m1 values (+1: 2, -1: 10), rows at
// or past the count to zeros: the query set, whose rows' shared bounds it also
// clears, and the database set (either may have no rows) in one launch.  Four bytes
// of bits to one 16-byte store; the values of a descriptor come in the order of its
// bits, least first.
struct ExpandSet {
  const uint8_t* bits;
  int n;
  const int* d_n;  // optional count on the device
  int rows;
  uint8_t* out;
};
__global__ void __launch_bounds__(256) k_expand_pm1(ExpandSet q, ExpandSet db, uint32_t* bound, int bounds) {
  __shared__ uint32_t lut[256];
  {
    uint32_t v = 0;
    for (int j = 0; j < 8; j++) v |= (((threadIdx.x >> j) & 1u) ? 0x2u : 0xAu) << (4 * j);
    lut[threadIdx.x] = v;
  }
  __syncthreads();
  chain_wait();
  const int nq = q.rows ? (q.d_n ? min(*q.d_n, q.rows) : min(q.n, q.rows)) : 0;
  const int nd = db.rows ? (db.d_n ? min(*db.d_n, db.rows) : min(db.n, db.rows)) : 0;
  constexpr int kPer = kPm1RowBytes / 16;  // stores per row
  const long long tq = (long long)q.rows * kPer, total = tq + (long long)db.rows * kPer;
  const long long i0 = (long long)blockIdx.x * blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  for (long long i = i0; i < bounds; i += step) bound[i] = kNoKeyShared;
  for (long long i = i0; i < total; i += step) {
    const bool is_q = i < tq;
    const ExpandSet& e = is_q ? q : db;
    const long long k = is_q ? i : i - tq;
    uint4 v{};
    if (k / kPer < (is_q ? nq : nd)) {
      const uint8_t* b = e.bits + 4 * k;  // descriptors may start on any byte
      v = make_uint4(lut[b[0]], lut[b[1]], lut[b[2]], lut[b[3]]);
    }
    reinterpret_cast<uint4*>(e.out)[k] = v;
  }
}

// A warp's wait: every lane tries once (no broadcast when the phase is over, the
// common case); after that lane 0 polls and the result is broadcast.
// Bounded waits of k_match_imma: false when a wait takes longer than
// kIDeadlineCycles or another role has given up.
__device__ __forceinline__ bool im_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try(bar, parity)) return true;
  return mbar_wait(bar, parity, clock64() + kIDeadlineCycles, abort_flag);
}
__device__ __forceinline__ bool im_warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
  int ok = 0;
  if ((threadIdx.x & 31) == 0) ok = im_wait(bar, parity, abort_flag) ? 1 : 0;
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

template <int SIZE, int SH, int... G>
__device__ __forceinline__ void push_groups(const float* vc, const bool* hit, uint32_t base, uint32_t& k1, uint32_t& k2,
                                            std::integer_sequence<int, G...>) {
  ((hit[G] ? push_best2<SIZE * G, SIZE * (G + 1), SH>(vc, base, k1, k2) : (void)0), ...);
}

__device__ __forceinline__ uint32_t lds_volatile(uint32_t a) {
  uint32_t v;
  asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts_volatile(uint32_t a, uint32_t v) {
  asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// One warp's part of a scan: its 32 queries over its columns of every accumulator of
// its set.  A function of its own, so that the registers around it are not the loop's.
struct ScanArgs {
  uint32_t* gq;       // the lane's query's bound, shared with the blocks that have its other parts, or null
  uint32_t k2_mine;   // shared memory: this warp's second-best key of the lane's row,
  uint32_t k2_set;    // that of the other column part,
  uint32_t k2_other;  // and those of the other set, kIBM apart, or 0 when it has other queries
  uint32_t tcol, full, empty, phase;
  int steps, col, stride, ndb;  // first column of the first step, columns from step to step
  volatile int* abort_flag;
};
__device__ __noinline__ bool m_scan(const ScanArgs sa, uint2* best) {
  static_assert(kMParts == 2, "one other column part");
  const int lane = threadIdx.x & 31;
  uint32_t k1 = kNoKeyShared, k2 = kNoKeyShared;  // best and second-best key of this row
  uint32_t told = kNoKeyShared, asked = kNoKeyShared, heard = kNoKeyShared;  // published, being read, read
  float thr_gb = kMaskedDotF;  // a dot at or below this cannot reach the row's final top two
  // (no key yet: far below every dot)
  auto next_thr = [&]() { return fmaxf(thr_gb, int_to_whole(256 - 2 * (int)(k2 >> kIdxBitsShared))); };
  float thr = kMaskedDotF;
  // columns arrive in increasing index order, so only a strictly larger dot
  // than the own second best can enter the top two.  Most chunks end at the
  // maximum test; one that passes looks at the column groups with a value above
  // the threshold.  These are few (a lane's top two change a few times per scan)
  // but they were half of the kernel's time when each group was a serial chain
  // with its own test.
  auto examine = [&](const float* vc, int gc) {
    constexpr int kSize = kMChunk / kMGroups;
    float gm[kMGroups];
#pragma unroll
    for (int g = 0; g < kMGroups; g++) gm[g] = max_of<kSize>(vc + kSize * g);
    if (!__any_sync(0xffffffffu, max_of<kMGroups>(gm) > thr)) return;
    bool hit[kMGroups];
#pragma unroll
    for (int g = 0; g < kMGroups; g++) hit[g] = __any_sync(0xffffffffu, gm[g] > thr);
    // distance << 22 = (256 - dot) << 21
    const uint32_t base = (256u << (kIdxBitsShared - 1)) + (uint32_t)gc;
    push_groups<kSize, kIdxBitsShared - 1>(vc, hit, base, k1, k2, std::make_integer_sequence<int, kMGroups>());
    thr = next_thr();
  };
  int c0 = sa.col;  // first column of the step
  for (int n = 0; n < sa.steps; n++, c0 += sa.stride) {
    // bounds from the others of this block that scan the row's query (every step,
    // while the accumulator is not full yet) and from its other parts (read in the
    // first steps and then every fourth, used one step later): a column can reach the
    // row's final top two only below their distance, or at it if its index can be the
    // lower one.
    {
      heard = min(heard, asked);
      if (sa.gq && (n < 8 || (n & 3) == 0)) asked = __ldcg(sa.gq);
      uint32_t gb = heard;
      gb = min(gb, lds_volatile(sa.k2_set));
      if (sa.k2_other)
        gb = min(gb, min(lds_volatile(sa.k2_other), lds_volatile(sa.k2_other + 4u * kIBM)));
      thr_gb = fmaxf(thr_gb, int_to_whole(256 - 2 * (int)(gb >> kIdxBitsShared) - ((int)(gb & kIdxMaskShared) >= c0)));
      thr = fmaxf(thr, thr_gb);
    }
    if (!im_warp_wait(sa.full, (sa.phase + (uint32_t)n) & 1u, sa.abort_flag)) return false;
    tc_fence_after();
#pragma unroll 1
    for (int c = 0; c < kMChunks; c++) {
      float v[kMChunk];
      tmem_read<kMChunk>(sa.tcol + (uint32_t)(kMChunk * c), v);
      if (c == kMChunks - 1) {
        // every column of this part is in registers: hand the accumulator back
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(sa.empty);
      }
      const int gc = c0 + kMChunk * c;
      if (gc + kMChunk > sa.ndb) {
#pragma unroll
        for (int j = 0; j < kMChunk; j++)
          if (gc + j >= sa.ndb) v[j] = kMaskedDotF;
      }
      examine(v, gc);
    }
    if (k2 < told) {
      told = k2;
      sts_volatile(sa.k2_mine, k2);
      // two distinct rows at or below k2: the query's final second best is no worse
      if (sa.gq) atomicMin(sa.gq, k2);
    }
  }
  *best = make_uint2(k1, k2);
  return true;
}

__global__ void __launch_bounds__(kMThreads, 1)
    k_match_imma(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmD, MatchArgs a,
                 MatchWork w, unsigned part_rows, int* err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  uint8_t* sA = smem;
  uint8_t* sB = sA + 4 * kMATile;
  uint2* s_merge = reinterpret_cast<uint2*>(sB + kMStages * kMBTile);
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(s_merge) + kIMergeBytes);
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(bars + kMNumBars);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
  __shared__ unsigned int s_last;
  // current second-best key per query row of each set and column part: two keys at
  // or below it exist, so it bounds what the others that scan the same query keep
  // for that row
  __shared__ uint32_t s_k2[2 * kMParts][kIBM];

  // the split, for the roles: in registers to the end it cost the scan spills (1500 x
  // 262144: 78.0 against 72.8 us)
  __shared__ MPlan plan;
  __shared__ int slots;
  __shared__ long long x_beg, x_end;

  chain_wait();
  const int nq = min(a.d_nq ? *a.d_nq : a.nq, w.nq_cap);
  const int ndb = a.d_ndb ? *a.d_ndb : a.ndb;
  {
    const int sl = m_slots(part_rows, nq);
    const MPlan p = m_plan(nq, ndb, sl, (int)gridDim.x);
    if ((int)blockIdx.x >= p.grid) return;  // uniform over the block: before any barrier or TMEM use
    if (threadIdx.x == 0) {
      plan = p;
      slots = sl;
    }
    if ((threadIdx.x & ~32u) == 0)
      *(threadIdx.x ? &x_end : &x_beg) = m_start(p, sl, blockIdx.x + (threadIdx.x ? 1 : 0));
  }

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t bar0 = smem_u32(bars);
#define BAR_AFULL(s) (bar0 + 8u * (s))
#define BAR_AEMPTY(s) (bar0 + 8u * (2 + (s)))
#define BAR_BFULL(s) (bar0 + 8u * (4 + (s)))
#define BAR_BEMPTY(s) (bar0 + 8u * (4 + kMStages + (s)))
#define BAR_ACCFULL(s) (bar0 + 8u * (4 + 2 * kMStages + (s)))
#define BAR_ACCEMPTY(s) (bar0 + 8u * (6 + 2 * kMStages + (s)))
#define BAR_EPI (bar0 + 8u * (8 + 2 * kMStages))

  for (int i = threadIdx.x; i < 2 * kMParts * kIBM; i += blockDim.x) (&s_k2[0][0])[i] = kNoKeyShared;
  if (threadIdx.x == 0) {
    mbar_init(BAR_EPI, kMEpiWarps);
    for (int s = 0; s < kMStages; s++) {
      mbar_init(BAR_BFULL(s), 1);
      mbar_init(BAR_BEMPTY(s), 1);
    }
    for (int s = 0; s < 2; s++) {
      mbar_init(BAR_AFULL(s), 1);
      mbar_init(BAR_AEMPTY(s), 1);
      mbar_init(BAR_ACCFULL(s), 1);
      mbar_init(BAR_ACCEMPTY(s), kMEpiWarps / 2);
    }
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)),
                 "r"(kITmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;
  // the scales of both operands, before the first MMA: four warps, one per 32 lanes
  if (warp >= 2 && warp < 6)
    tmem_store_unit_scales(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + kMScaleCol);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == 0) {
    if (lane == 0) {
      // TMA producer
      int issued[kMStages];
      for (int s = 0; s < kMStages; s++) issued[s] = 0;
      int parts = 0, tg = 0, a_loads = 0;  // parts, database tiles and query loads so far
      bool ok = true;
      for (long long x = x_beg; ok && x < x_end; parts++) {
        const MPart r = m_part(plan, x, x_end);
        x += r.t1 - r.t0;
        const int ab = parts & 1;
        if (parts >= 2 && !im_wait(BAR_AEMPTY(ab), (uint32_t)((parts >> 1) - 1) & 1u, s_abort)) {
          ok = false;
          break;
        }
        const bool two = nq - r.qb * kIBQ > kIBM;  // two query tiles
        a_loads++;
        mbar_expect_tx(BAR_AFULL(ab), two ? 2 * kMATile : kMATile);
        for (int m = 0; m < (two ? 2 : 1); m++)
          tma_load_2d(smem_u32(sA + (2 * ab + m) * kMATile), &tmQ, 0, r.qb * kIBQ + m * kIBM, BAR_AFULL(ab));
        for (int t = r.t0; t < r.t1; t++, tg++) {
          const int s = tg % kMStages;
          const int use = tg / kMStages;
          if (use > 0 && !im_wait(BAR_BEMPTY(s), (use - 1) & 1, s_abort)) {
            ok = false;
            break;
          }
          mbar_expect_tx(BAR_BFULL(s), kMBTile);
          tma_load_2d(smem_u32(sB + s * kMBTile), &tmD, 0, t * kMBN, BAR_BFULL(s));
          issued[s]++;
        }
      }
      if (!ok) {
        *s_abort = 1;
        atomicOr(err, kErrImmaTimeout);
      }
      // Drain before the block may exit: every issued copy has landed and every
      // MMA that read a stage has completed (its commit arrived on "empty").
      long long dl;
      for (int ab = 0; ab < 2; ab++) {
        const int loads = (a_loads + 1 - ab) >> 1;
        if (loads == 0) continue;
        dl = clock64() + kIDeadlineCycles;
        while (!mbar_try(BAR_AFULL(ab), (uint32_t)(loads - 1) & 1u) && clock64() < dl) {
        }
      }
      for (int s = 0; s < kMStages; s++) {
        if (issued[s] == 0) continue;
        const uint32_t par = (uint32_t)(issued[s] - 1) & 1u;
        dl = clock64() + kIDeadlineCycles;
        while (!mbar_try(BAR_BFULL(s), par) && clock64() < dl) {
        }
        dl = clock64() + kIDeadlineCycles;
        while (!mbar_try(BAR_BEMPTY(s), par) && clock64() < dl) {
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // MMA issuer: four K=64 MMAs per step into accumulator (step & 1)
      bool ok = true;
      int parts = 0, tg = 0, g = 0;  // parts, database tiles and steps so far
      const uint32_t sfa = tmem_base + kMScaleCol, sfb = sfa + kMScaleCols / 2;
      for (long long x = x_beg; ok && x < x_end; parts++) {
        const MPart r = m_part(plan, x, x_end);
        x += r.t1 - r.t0;
        const int ab = parts & 1;
        const int per = nq - r.qb * kIBQ > kIBM ? 2 : 1;
        const uint64_t da0 = sw128_desc(smem_u32(sA + 2 * ab * kMATile));
        ok = im_wait(BAR_AFULL(ab), (uint32_t)(parts >> 1) & 1u, s_abort);
        for (int t = r.t0; ok && t < r.t1; t++, tg++) {
          const int s = tg % kMStages;
          ok = im_wait(BAR_BFULL(s), (uint32_t)(tg / kMStages) & 1u, s_abort);
          const uint64_t db = sw128_desc(smem_u32(sB + s * kMBTile));
          for (int qt = 0; ok && qt < per; qt++, g++) {
            const int acc = g & 1;
            if (g >= 2 && !im_wait(BAR_ACCEMPTY(acc), (uint32_t)((g - 2) >> 1) & 1u, s_abort)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t d = tmem_base + (uint32_t)acc * kMAcc;
            const uint64_t da = da0 + (uint64_t)(qt * (kMATile >> 4));
#pragma unroll
            for (int k = 0; k < 4; k++)  // 64 values are 32 bytes of a row: two descriptor units
              umma_f4(d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), kMDesc, sfa, sfb, k > 0 ? 1u : 0u);
            if (qt == per - 1) umma_commit(BAR_BEMPTY(s));  // the database tile's last step
            umma_commit(BAR_ACCFULL(acc));
          }
        }
        if (!ok) break;
        umma_commit(BAR_AEMPTY(ab));
      }
      if (!ok) {
        *s_abort = 1;
        atomicOr(err, kErrImmaTimeout);
      }
      // the producer drains the ring's "empty" barriers, this thread its other commits
      for (uint32_t i = 0; i < 2; i++) {
        mbar_drain(BAR_AEMPTY(i), m_ring_uses((uint32_t)parts, 2, i));
        mbar_drain(BAR_ACCFULL(i), m_ring_uses((uint32_t)g, 2, i));
      }
    }
  } else {
    // epilogue: steps of this warp's set, TMEM lanes 32 * (warp & 3) .. (one
    // query per lane), columns [kMChunks * kMChunk * part, + kMChunks * kMChunk)
    const int set = (warp - 2) / (4 * kMParts);
    const int part = ((warp - 2) >> 2) % kMParts;
    const int me = kMParts * set + part;
    const int row = (warp & 3) * 32 + lane;
    const int e = threadIdx.x - 64;  // of the epilogue's threads
    bool ok = true;
    int g0 = 0;            // steps before this part
    uint32_t sync_phase = 0;
    // all epilogue warps: false on a timeout
    auto epi_sync = [&]() {
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_EPI);
      const bool done = im_warp_wait(BAR_EPI, sync_phase++ & 1u, s_abort);
      __syncwarp();
      return done;
    };
    long long x = x_beg, uncounted = x_beg;  // pairs before which all parts have been counted in tile_done
    while (x < x_end) {
    const MPart r = m_part(plan, x, x_end);
    x += r.t1 - r.t0;
    const bool two = nq - r.qb * kIBQ > kIBM;
    const int nsteps = (two ? 2 : 1) * (r.t1 - r.t0);
    int n_parts, slot;
    m_slot(plan, slots, r.qb, r.t0, blockIdx.x, &n_parts, &slot);
    const int first = set ^ (g0 & 1);  // this set's first step and, of two, its query tile
    const int q = r.qb * kIBQ + (two ? first * kIBM : 0) + row;
    // second-best bound shared by the blocks that have the query's other parts
    ScanArgs sa;
    sa.gq = (w.bound && n_parts > 1 && q < nq) ? w.bound + q : nullptr;
    sa.k2_mine = smem_u32(&s_k2[me][row]);
    sa.k2_set = smem_u32(&s_k2[kMParts * set + (part + 1) % kMParts][row]);
    sa.k2_other = two ? 0u : smem_u32(&s_k2[kMParts * (set ^ 1)][row]);
    sa.tcol = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)set * kMAcc + (uint32_t)(part * kMChunks * kMChunk);
    sa.full = BAR_ACCFULL(set);
    sa.empty = BAR_ACCEMPTY(set);
    sa.phase = (uint32_t)((g0 + first) >> 1);
    sa.steps = (nsteps - first + 1) >> 1;
    sa.col = (r.t0 + (two ? 0 : first)) * kMBN + part * kMChunks * kMChunk;
    sa.stride = two ? kMBN : 2 * kMBN;
    sa.ndb = ndb;
    sa.abort_flag = s_abort;
    uint2 best;
    ok = m_scan(sa, &best);
    if (!ok) break;
    g0 += nsteps;
    // the best two of each query over the block's sets and column parts
    s_merge[(kMParts * first + part) * kIBM + row] = best;
    ok = epi_sync();
    if (!ok) break;
    s_k2[me][row] = kNoKeyShared;  // for the next part
    const int rows = two ? kIBQ : kIBM;
    const bool mine = e < rows && r.qb * kIBQ + e < nq;
    if (mine) {
      uint32_t m1 = kNoKeyShared, m2 = kNoKeyShared;
      for (int g = 0; g < (two ? kMParts : 2 * kMParts); g++) {
        const uint2 pk = s_merge[(two ? kMParts * (e / kIBM) + g : g) * kIBM + e % kIBM];
        top2_push_shared(m1, m2, pk.x);
        top2_push_shared(m1, m2, pk.y);
      }
      if (n_parts == 1)
        finish_query_shared(a, r.qb * kIBQ + e, m1, m2);
      else
        reinterpret_cast<uint2*>(w.part)[(size_t)slot * nq + r.qb * kIBQ + e] = make_uint2(m1, m2);
    }
    if (n_parts > 1) {
      // the block that finishes the last part of these queries merges all parts
      __threadfence();
      ok = epi_sync();
      if (!ok) break;
      if (e == 0) s_last = (atomicAdd(&w.tile_done[r.qb], 1u) == (unsigned)(n_parts - 1)) ? 1u : 0u;
      uncounted = x;
      ok = epi_sync();
      if (!ok) break;
      if (s_last) {
        __threadfence();
        if (e == 0) w.tile_done[r.qb] = 0u;
        const int per = two ? kMParts : 2 * kMParts;
        if (e < rows * per) {
          const int qr = r.qb * kIBQ + e % rows;
          uint32_t m1 = kNoKeyShared, m2 = kNoKeyShared;
          if (qr < nq) {
            const uint2* pt = reinterpret_cast<const uint2*>(w.part) + qr;
#pragma unroll 8
            for (int s2 = e / rows; s2 < n_parts; s2 += per) {
              const uint2 pk = __ldcg(pt + (size_t)s2 * nq);
              top2_push_shared(m1, m2, pk.x);
              top2_push_shared(m1, m2, pk.y);
            }
          }
          s_merge[e] = make_uint2(m1, m2);
        }
        ok = epi_sync();
        if (!ok) break;
        if (mine) {
          uint32_t m1 = kNoKeyShared, m2 = kNoKeyShared;
          for (int g = 0; g < per; g++) {
            const uint2 pk = s_merge[g * rows + e];
            top2_push_shared(m1, m2, pk.x);
            top2_push_shared(m1, m2, pk.y);
          }
          finish_query_shared(a, r.qb * kIBQ + e, m1, m2);
        }
      }
    }
    uncounted = x;
    ok = epi_sync();  // s_merge and s_last are free
    if (!ok) break;
    }
    if (!ok) {
      *s_abort = 1;
      if (lane == 0) atomicOr(err, kErrImmaTimeout);
      // the counters of the parts not finished return to zero all the same
      if (e == 0)
        for (long long y = uncounted; y < x_end;) {
          const MPart r = m_part(plan, y, x_end);
          y += r.t1 - r.t0;
          int n_parts, slot;
          m_slot(plan, slots, r.qb, r.t0, blockIdx.x, &n_parts, &slot);
          if (n_parts > 1 && atomicAdd(&w.tile_done[r.qb], 1u) == (unsigned)(n_parts - 1)) w.tile_done[r.qb] = 0u;
        }
    }
  }
#undef BAR_AFULL
#undef BAR_AEMPTY
#undef BAR_BFULL
#undef BAR_BEMPTY
#undef BAR_ACCFULL
#undef BAR_ACCEMPTY
#undef BAR_EPI

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kITmemCols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------
// Probe rerank of the learned proposal on the tensor cores
//
// A work item is one cluster c with up to 128 of the query slots that probe it
// (list[probe_offsets[c] ..], grouped by cluster; slot = query * 8 + probe).
// The cluster's rows are kept packed (32 bytes each, padded per cluster to
// 240-row tiles) and expanded in shared memory, so HBM carries a quarter of
// the bytes expanded rows would.  The blocks are persistent and claim items
// from a global counter (items differ widely in size); the producer thread
// claims them and passes them to the other roles through a small queue:
//   warp 0      producer: each tile's packed rows by cp.async.bulk
//               into a 4-stage ring;
//   warp 1      MMA issuer, as in k_match_imma, into two 240-column
//               accumulators; commits release the expanded stage, the
//               accumulator and, after an item's last tile, its query tile;
//   warps 2-9   expanders: at an item's start they gather its slots' queries
//               as signed rows (two threads per row) into one of two query tiles,
//               then expand each packed tile to masked rows into a ring of four
//               database tiles, one row per thread, in the 128-byte swizzled
//               K-major layout the TMA writes (rr_db_chunk);
//   warps 10-17 epilogue: warp w reads TMEM lanes 32 * (w % 4) and 120 columns,
//               keeps the top-2 keys (distance << 22 | database index) of each
//               slot over the item's tiles (distance = popcount(query) - dot')
//               and writes them to partial[slot * 2 + column group].
// Each cluster's list is in increasing database index, so column order is
// index order and ties resolve as in the other matchers.  Every wait is bounded (kIDeadlineCycles per
// wait); on expiry the block records kErrImmaTimeout, drains its copies and
// exits.
//
// What bounds it: the ALU (expansion and the epilogue's tests).  32768 queries, 8
// probes in 512 lists of about 2048 rows: 372 us with one candidate after another,
// 306 us with the tournament updates, 245 us with the expansion by masks to int8 and
// the query's shared bound read one tile ahead, 206 us with 4-bit floats, which halve
// the expansion's stores, 203 us with 8 epilogue warps that hold 60 columns each
// instead of 16 with 32 (and half the results to merge: 12.3 -> 8.6 us there).
// ---------------------------------------------------------------------------
constexpr int kRrExpWarps = 8;
constexpr int kRrThreads = (2 + kRrExpWarps + kIEpiWarps) * 32;
constexpr uint32_t kRrPStages = 4;
constexpr uint32_t kRrXStages = 4;  // expanded database tiles
constexpr uint32_t kRrPTile = kMBN * 32;  // packed rows of one tile
constexpr uint32_t kRrQueue = 8;  // claimed items in flight between the producer and the other roles
constexpr uint32_t kRrNumBars = 2 + 2 + 2 * kRrPStages + 2 * kRrXStages + 2 + 2 + 2 * kRrQueue;
// the item queue's consumers: the MMA thread, the expander and the epilogue warps
constexpr uint32_t kRrQueueReaders = 1 + kRrExpWarps + kIEpiWarps;
constexpr uint32_t kRrSmemBytes =
    1024 + 2 * kMATile + kRrXStages * kMBTile + kRrPStages * kRrPTile + 8 * kRrNumBars + 4 * kRrQueue + 16;
static_assert(kRrSmemBytes + 16 <= 232448, "exceeds the 227 KB shared-memory opt-in");
static_assert(kRrExpWarps * 32 >= kMBN && kRrExpWarps * 32 == 2 * kIBM, "one expander thread per row, two per query");
constexpr int kRrCols = kMBN / kRrGroups;  // columns of an epilogue warp
constexpr int kRrChunk = 60;               // examined at a time

struct RrItem {
  int c;      // cluster
  int e0;     // first slot in list
  int rows;   // slots in this item (1..128)
  int nrow;   // the cluster's database rows
  int pbase;  // first padded row of the cluster
  int tiles;  // 240-row tiles
};

__device__ __forceinline__ RrItem rr_item(const RerankImmaArgs& a, int it) {
  int lo = 0, hi = a.n_clusters;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(a.item_offsets + mid) <= it) lo = mid;
    else hi = mid;
  }
  RrItem r;
  r.c = lo;
  r.e0 = __ldg(a.probe_offsets + lo) + (it - __ldg(a.item_offsets + lo)) * kIBM;
  r.rows = min(kIBM, __ldg(a.probe_offsets + lo + 1) - r.e0);
  r.nrow = __ldg(a.ivf_offsets + lo + 1) - __ldg(a.ivf_offsets + lo);
  r.pbase = __ldg(a.pad_offsets + lo);
  r.tiles = (r.nrow + kMBN - 1) / kMBN;
  return r;
}

// Bounded wait with a fresh deadline: false on expiry or when another role aborted.
__device__ __forceinline__ bool rr_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return mbar_wait(bar, parity, clock64() + kIDeadlineCycles, abort_flag);
}
__device__ __forceinline__ bool rr_warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
  int ok = 0;
  if ((threadIdx.x & 31) == 0) ok = rr_wait(bar, parity, abort_flag) ? 1 : 0;
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// The order of the 256 products of a dot product is free, and so is how a weight
// is shared between its factors; both are chosen so that a database row's packed
// words expand by masking alone.  Output word k (k = 0 .. 3) of a packed word holds
// its bits k, 4 + k, 8 + k .. in place, i.e. nibbles of 0 or 1 << k: 0.5, 1 or 2 as
// e2m1 (bit 3, the sign, is shifted down to 0.5).  The query's values are +-2, +-1,
// +-0.5 and +-2: every product is the query's sign where the row has a one, the
// accumulator is dot' and Hamming(q, row) = popcount(q) - dot'.  40 operations and
// eight stores per row.
__device__ __forceinline__ uint4 rr_db_chunk(uint32_t w) {
  return make_uint4(w & 0x11111111u, w & 0x22222222u, w & 0x44444444u, (w >> 3) & 0x11111111u);
}
__device__ __forceinline__ uint32_t rr_query_word(uint32_t w, int k, uint32_t code) {
  return (code * 0x11111111u) | ((~(w >> k) & 0x11111111u) << 3);
}
__device__ __forceinline__ uint4 rr_query_chunk(uint32_t w) {
  return make_uint4(rr_query_word(w, 0, 4u), rr_query_word(w, 1, 2u), rr_query_word(w, 2, 1u), rr_query_word(w, 3, 4u));
}

// Swizzled address of 16-byte chunk cc of row r in a K-major tile of 128-byte rows.
__device__ __forceinline__ uint8_t* sw128_chunk(uint8_t* tile, int r, int cc) {
  return tile + r * 128 + ((cc ^ (r & 7)) << 4);
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// The next claimed item of the queue (-1 when none is left), for a whole warp;
// one arrival per warp frees the entry.  False on a timeout.
__device__ __forceinline__ bool rr_next_item(uint32_t qfull, uint32_t qempty, volatile int* s_queue, uint32_t qs,
                                             uint32_t parity, volatile int* abort_flag, int* it) {
  if (!rr_warp_wait(qfull, parity, abort_flag)) return false;
  *it = s_queue[qs];
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(qempty);
  return true;
}

// A chunk of N columns, rows col0 .. of the cluster's nrow, against a lane's best two
// keys (distance = pc - dot').  The columns arrive in list order, so only a strictly
// larger dot' than the current second best's can enter, and no column farther than
// the second best that another item of the same query holds (equal distances stay,
// their index decides).
template <int N>
__device__ __forceinline__ void rr_examine(float* v, int col0, int nrow, int pc, float thr_gb, uint32_t& k1,
                                           uint32_t& k2) {
  constexpr int kGroups = 4, kSize = N / kGroups;
  if (nrow - col0 < N) {
#pragma unroll
    for (int j = 0; j < N; j++)
      if (j >= nrow - col0) v[j] = kMaskedDotF;
  }
  // (no key yet: below every dot')
  const float thr = fmaxf(int_to_whole(pc - (int)(k2 >> kIdxBitsShared)), thr_gb);
  float gm[kGroups];
#pragma unroll
  for (int g = 0; g < kGroups; g++) gm[g] = max_of<kSize>(v + kSize * g);
  if (!__any_sync(0xffffffffu, max_of<kGroups>(gm) > thr)) return;
  bool hit[kGroups];
#pragma unroll
  for (int g = 0; g < kGroups; g++) hit[g] = __any_sync(0xffffffffu, gm[g] > thr);
  push_groups<kSize, kIdxBitsShared>(v, hit, ((uint32_t)pc << kIdxBitsShared) + (uint32_t)col0, k1, k2,
                                     std::make_integer_sequence<int, kGroups>());
}

__global__ void __launch_bounds__(kRrThreads, 1) k_rerank_imma(RerankImmaArgs a) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw & 1023u)) & 1023u);
  uint8_t* sA = smem;               // two query tiles
  uint8_t* sX = sA + 2 * kMATile;   // ring of expanded database tiles
  uint8_t* sP = sX + kRrXStages * kMBTile;   // ring of packed database tiles
  uint64_t* bars = reinterpret_cast<uint64_t*>(sP + kRrPStages * kRrPTile);
  volatile int* s_queue = reinterpret_cast<volatile int*>(bars + kRrNumBars);
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(const_cast<int*>(s_queue) + kRrQueue);
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);

  chain_wait();
  const int n_items = __ldg(a.item_offsets + a.n_clusters);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t bar0 = smem_u32(bars);
#define RR_AFULL(b) (bar0 + 8u * (b))
#define RR_AEMPTY(b) (bar0 + 8u * (2 + (b)))
#define RR_PFULL(s) (bar0 + 8u * (4 + (s)))
#define RR_PEMPTY(s) (bar0 + 8u * (4 + kRrPStages + (s)))
#define RR_XFULL(x) (bar0 + 8u * (4 + 2 * kRrPStages + (x)))
#define RR_XEMPTY(x) (bar0 + 8u * (4 + 2 * kRrPStages + kRrXStages + (x)))
#define RR_REST (4 + 2 * kRrPStages + 2 * kRrXStages)
#define RR_ACCFULL(x) (bar0 + 8u * (RR_REST + (x)))
#define RR_ACCEMPTY(x) (bar0 + 8u * (RR_REST + 2 + (x)))
#define RR_QFULL(k) (bar0 + 8u * (RR_REST + 4 + (k)))
#define RR_QEMPTY(k) (bar0 + 8u * (RR_REST + 4 + kRrQueue + (k)))

  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; b++) {
      mbar_init(RR_AFULL(b), kRrExpWarps);
      mbar_init(RR_AEMPTY(b), 1);
      mbar_init(RR_ACCFULL(b), 1);
      mbar_init(RR_ACCEMPTY(b), kIEpiWarps);
    }
    for (uint32_t x = 0; x < kRrXStages; x++) {
      mbar_init(RR_XFULL(x), kRrExpWarps);
      mbar_init(RR_XEMPTY(x), 1);
    }
    for (uint32_t st = 0; st < kRrPStages; st++) {
      mbar_init(RR_PFULL(st), 1);
      mbar_init(RR_PEMPTY(st), kRrExpWarps);
    }
    for (uint32_t k = 0; k < kRrQueue; k++) {
      mbar_init(RR_QFULL(k), 1);
      mbar_init(RR_QEMPTY(k), kRrQueueReaders);
    }
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)),
                 "r"(kITmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *s_tmem;
  // the scales of both operands, before the first MMA: four warps, one per 32 lanes
  if (warp >= 2 + kRrExpWarps && warp < 6 + kRrExpWarps)
    tmem_store_unit_scales(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + kMScaleCol);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == 0) {
    if (lane == 0) {
      // producer: the packed rows of every tile of every item of this block, in order
      uint32_t issued[kRrPStages];
      for (uint32_t st = 0; st < kRrPStages; st++) issued[st] = 0u;
      uint32_t g = 0, k = 0;
      bool ok = true;
      while (ok) {
        // claim the next item and hand it to the other roles (-1: none left)
        const uint32_t qs = k % kRrQueue;
        if (k >= kRrQueue && !rr_wait(RR_QEMPTY(qs), ((k / kRrQueue) - 1) & 1u, s_abort)) {
          ok = false;
          break;
        }
        int it = atomicAdd(a.item_counter, 1);
        if (it >= n_items) it = -1;
        s_queue[qs] = it;
        mbar_arrive(RR_QFULL(qs));
        k++;
        if (it < 0) break;
        const RrItem r = rr_item(a, it);
        for (int t = 0; t < r.tiles; t++, g++) {
          const uint32_t st = g % kRrPStages;
          if (g >= kRrPStages && !rr_wait(RR_PEMPTY(st), ((g / kRrPStages) - 1) & 1u, s_abort)) {
            ok = false;
            break;
          }
          mbar_expect_tx(RR_PFULL(st), kRrPTile);
          bulk_load(smem_u32(sP + st * kRrPTile), a.pad_desc + (size_t)(r.pbase + t * kMBN) * 32, kRrPTile,
                    RR_PFULL(st));
          issued[st]++;
        }
      }
      if (!ok) {
        *s_abort = 1;
        atomicOr(a.err, kErrImmaTimeout);
      }
      // drain: every issued copy has landed and been read
      for (uint32_t st = 0; st < kRrPStages; st++) {
        if (issued[st] == 0) continue;
        const uint32_t par = (issued[st] - 1) & 1u;
        long long dl = clock64() + kIDeadlineCycles;
        while (!mbar_try(RR_PFULL(st), par) && clock64() < dl) {
        }
        dl = clock64() + kIDeadlineCycles;
        while (!mbar_try(RR_PEMPTY(st), par) && clock64() < dl && !*s_abort) {
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // MMA issuer
      uint32_t g = 0, na = 0, k = 0;
      bool ok = true;
      while (ok) {
        const uint32_t qs = k % kRrQueue;
        if (!rr_wait(RR_QFULL(qs), (k / kRrQueue) & 1u, s_abort)) {
          ok = false;
          break;
        }
        const int it = s_queue[qs];
        mbar_arrive(RR_QEMPTY(qs));
        k++;
        if (it < 0) break;
        const RrItem r = rr_item(a, it);
        if (r.tiles == 0) continue;
        const uint32_t b = na & 1u;
        if (!rr_wait(RR_AFULL(b), (na >> 1) & 1u, s_abort)) {
          ok = false;
          break;
        }
        const uint64_t da = sw128_desc(smem_u32(sA + b * kMATile));
        const uint32_t sfa = tmem_base + kMScaleCol, sfb = sfa + kMScaleCols / 2;
        for (int t = 0; t < r.tiles; t++, g++) {
          const uint32_t x = g % kRrXStages, acc = g & 1u;
          if (!rr_wait(RR_XFULL(x), (g / kRrXStages) & 1u, s_abort) ||
              (g >= 2 && !rr_wait(RR_ACCEMPTY(acc), ((g >> 1) - 1) & 1u, s_abort))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem_base + acc * kMAcc;
          const uint64_t db = sw128_desc(smem_u32(sX + x * kMBTile));
#pragma unroll
          for (int k = 0; k < 4; k++)
            umma_f4(d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), kMDesc, sfa, sfb, k > 0 ? 1u : 0u);
          umma_commit(RR_XEMPTY(x));
          umma_commit(RR_ACCFULL(acc));
        }
        if (!ok) break;
        umma_commit(RR_AEMPTY(b));
        na++;
      }
      if (!ok) {
        *s_abort = 1;
        atomicOr(a.err, kErrImmaTimeout);
      }
      // every commit has arrived (m_ring_uses)
      for (uint32_t i = 0; i < 2; i++) {
        mbar_drain(RR_AEMPTY(i), m_ring_uses(na, 2, i));
        mbar_drain(RR_ACCFULL(i), m_ring_uses(g, 2, i));
      }
      for (uint32_t i = 0; i < kRrXStages; i++) mbar_drain(RR_XEMPTY(i), m_ring_uses(g, kRrXStages, i));
    }
  } else if (warp < 2 + kRrExpWarps) {
    // expanders: thread e (0..255)
    const int e = threadIdx.x - 64;
    uint32_t na = 0, g = 0, k = 0;
    bool ok = true;
    while (ok) {
      int it;
      const uint32_t qs = k % kRrQueue;
      if (!rr_next_item(RR_QFULL(qs), RR_QEMPTY(qs), s_queue, qs, (k / kRrQueue) & 1u, s_abort, &it)) {
        ok = false;
        break;
      }
      k++;
      if (it < 0) break;
      const RrItem ri = rr_item(a, it);
      if (ri.tiles == 0) continue;
      // the item's queries: row e >> 1, K half e & 1
      const uint32_t b = na & 1u;
      if (na >= 2 && !rr_warp_wait(RR_AEMPTY(b), ((na >> 1) - 1) & 1u, s_abort)) {
        ok = false;
        break;
      }
      {
        const int r = e >> 1, half = e & 1;
        uint4 w = make_uint4(0u, 0u, 0u, 0u);
        if (r < ri.rows) {
          const int q = __ldca(a.list + ri.e0 + r) >> 3;
          w = __ldg(reinterpret_cast<const uint4*>(a.q_bits) + 2 * (size_t)q + half);
        }
        const uint32_t wd[4] = {w.x, w.y, w.z, w.w};
        uint8_t* tile = sA + b * kMATile;
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint4 v = (r < ri.rows) ? rr_query_chunk(wd[j]) : make_uint4(0u, 0u, 0u, 0u);
          *reinterpret_cast<uint4*>(sw128_chunk(tile, r, 4 * half + j)) = v;
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(RR_AFULL(b));
      na++;
      // the item's database tiles: row e of each
      for (int t = 0; t < ri.tiles; t++, g++) {
        const uint32_t st = g % kRrPStages, x = g % kRrXStages;
        if (!rr_warp_wait(RR_PFULL(st), (g / kRrPStages) & 1u, s_abort) ||
            (g >= kRrXStages && !rr_warp_wait(RR_XEMPTY(x), (g / kRrXStages - 1) & 1u, s_abort))) {
          ok = false;
          break;
        }
        if (e < kMBN) {
          const uint4* src = reinterpret_cast<const uint4*>(sP + st * kRrPTile) + 2 * e;
          const uint4 w0 = src[0], w1 = src[1];
          const uint32_t wd[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
          uint8_t* tile = sX + x * kMBTile;
#pragma unroll
          for (int cc = 0; cc < 8; cc++) *reinterpret_cast<uint4*>(sw128_chunk(tile, e, cc)) = rr_db_chunk(wd[cc]);
        }
        // The packed stage is released here, not right after its loads: the stores
        // and the fence have waited for them, and a copy (async proxy) issued before
        // they were complete replaced words still to be read (one tile in about
        // 50000, in one of 25 searches of 32768 queries).
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(RR_XFULL(x));
          mbar_arrive(RR_PEMPTY(st));
        }
      }
    }
    if (!ok) {
      *s_abort = 1;
      if (lane == 0) atomicOr(a.err, kErrImmaTimeout);
    }
  } else {
    // epilogue
    const int ew = warp - 2 - kRrExpWarps;
    const int quarter = warp & 3;
    const int colgrp = ew >> 2;
    const int row = quarter * 32 + lane;
    uint32_t g = 0, k = 0;
    bool ok = true;
    while (ok) {
      int it;
      const uint32_t qs = k % kRrQueue;
      if (!rr_next_item(RR_QFULL(qs), RR_QEMPTY(qs), s_queue, qs, (k / kRrQueue) & 1u, s_abort, &it)) {
        ok = false;
        break;
      }
      k++;
      if (it < 0) break;
      const RrItem ri = rr_item(a, it);
      // this lane's slot and its query's popcount
      int slot = -1, pc = 0;
      if (row < ri.rows) {
        slot = __ldca(a.list + ri.e0 + row);
        const uint4* qp = reinterpret_cast<const uint4*>(a.q_bits) + 2 * (size_t)(slot >> 3);
        const uint4 w0 = __ldg(qp), w1 = __ldg(qp + 1);
        pc = __popc(w0.x) + __popc(w0.y) + __popc(w0.z) + __popc(w0.w) + __popc(w1.x) + __popc(w1.y) +
             __popc(w1.z) + __popc(w1.w);
      }
      // best two keys of this row over the item, distance << 22 | row within the
      // cluster: the cluster's list is in increasing database index, so they order
      // like keys of database indices, into which they are turned at the end
      uint32_t k1 = kNoKeyShared, k2 = kNoKeyShared;
      uint32_t asked = slot >= 0 ? __ldcg(a.q_bound + (slot >> 3)) : kNoKeyShared;
      float thr_gb = kMaskedDotF;
      for (int t = 0; t < ri.tiles; t++, g++) {
        const uint32_t acc = g & 1u;
        if (!rr_warp_wait(RR_ACCFULL(acc), (g >> 1) & 1u, s_abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        // the query's bound from its other items so far (any stale value is a valid,
        // looser bound): read while the tile before was examined
        if (asked != kNoKeyShared) thr_gb = fmaxf(thr_gb, int_to_whole(pc - (int)(asked >> kIdxBitsShared) - 1));
        if (slot >= 0) asked = __ldcg(a.q_bound + (slot >> 3));
        const uint32_t taddr =
            tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * kMAcc + (uint32_t)(colgrp * kRrCols);
        const int col0 = t * kMBN + colgrp * kRrCols;  // first column's row within the cluster
        static_assert(kRrCols == 2 * kRrChunk, "two chunks");
        float v[kRrChunk];
        tmem_read<kRrChunk>(taddr, v);
        rr_examine<kRrChunk>(v, col0, ri.nrow, pc, thr_gb, k1, k2);
        tmem_read<kRrChunk>(taddr + (uint32_t)kRrChunk, v);
        // every column of this group is in registers: hand the accumulator back
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(RR_ACCEMPTY(acc));
        rr_examine<kRrChunk>(v, col0 + kRrChunk, ri.nrow, pc, thr_gb, k1, k2);
      }
      if (!ok) break;
      if (slot >= 0) {
        auto member = [&](uint32_t key) {
          return key == kNoKeyShared
                     ? key
                     : (key & ~kIdxMaskShared) | (uint32_t)__ldg(a.pad_members + ri.pbase + (key & kIdxMaskShared));
        };
        a.partial[(size_t)slot * kRrGroups + colgrp] = make_uint2(member(k1), member(k2));
        // two distinct rows at or below k2: the query's final second best is no worse
        if (k2 != kNoKeyShared) atomicMin(a.q_bound + (slot >> 3), k2);
      }
    }
    if (!ok) {
      *s_abort = 1;
      if (lane == 0) atomicOr(a.err, kErrImmaTimeout);
    }
  }
#undef RR_AFULL
#undef RR_AEMPTY
#undef RR_PFULL
#undef RR_PEMPTY
#undef RR_XFULL
#undef RR_XEMPTY
#undef RR_ACCFULL
#undef RR_REST
#undef RR_ACCEMPTY
#undef RR_QFULL
#undef RR_QEMPTY

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kITmemCols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

static bool make_rows_map(CUtensorMap* m, const void* base, uint64_t rows, uint32_t box_rows) {
  // one box is whole rows: 128 bytes, the swizzle's span
  auto enc = tensor_map_encoder();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)kPm1RowBytes, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)kPm1RowBytes};
  cuuint32_t box[2] = {(cuuint32_t)kPm1RowBytes, box_rows};
  cuuint32_t es[2] = {1u, 1u};
  const CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

int imma_rows_q(int n) { return (n + kIBM - 1) / kIBM * kIBM; }
int imma_rows_db(int n) { return (n + kMBN - 1) / kMBN * kMBN; }

cudaError_t launch_expand_pm1(const uint8_t* bits, int n, const int* d_n, int rows, uint8_t* out, cudaStream_t s) {
  return launch_chained(k_expand_pm1, 4 * 148, 256, s, ExpandSet{bits, n, d_n, rows, out}, ExpandSet{},
                        static_cast<uint32_t*>(nullptr), 0);
}

cudaError_t launch_match_imma(const ImmaLaunch& L, cudaStream_t s) {
  if (L.nq_cap <= 0) return cudaSuccess;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(k_match_imma, cudaFuncAttributeMaxDynamicSharedMemorySize, kISmemBytes);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  const int qrows = imma_rows_q(L.nq_cap);
  const int dbrows = imma_rows_db(L.ndb_cap > 0 ? L.ndb_cap : 1);
  {
    ExpandSet q{}, db{};
    if (!L.q_ready) q = ExpandSet{L.args.q, L.args.nq, L.args.d_nq, qrows, L.q_pm1};
    if (L.ndb_cap > 0 && !L.db_ready) db = ExpandSet{L.args.db, L.args.ndb, L.args.d_ndb, dbrows, L.db_pm1};
    const int bounds = L.work.bound ? std::min(L.work.nq_cap, L.nq_cap) : 0;
    if (q.rows || db.rows || bounds) {
      const cudaError_t e = launch_chained(k_expand_pm1, 4 * 148, 256, s, q, db, L.work.bound, bounds);
      if (e != cudaSuccess) return e;
    }
  }
  CUtensorMap tq, td;
  if (!make_rows_map(&tq, L.q_pm1, (uint64_t)qrows, kIBM)) return cudaErrorInvalidValue;
  if (!make_rows_map(&td, L.db_pm1, (uint64_t)dbrows, kMBN)) return cudaErrorInvalidValue;
  const unsigned part_rows =
      L.work.part && L.work.tile_done ? (unsigned)std::min<long long>(L.part_rows, 0xFFFFFFFFll) : 0u;
  const MPlan plan = m_plan(L.nq_cap, std::max(L.ndb_cap, 0), m_slots(part_rows, L.nq_cap), kPlanGrid);
  // counts on the device may be smaller than the capacities and spread over more blocks
  const int grid = L.args.d_nq || L.args.d_ndb ? (int)std::min<long long>(plan.total, kPlanGrid) : plan.grid;
  return launch_chained_smem(k_match_imma, grid, kMThreads, kISmemBytes, s, tq, td, L.args, L.work, part_rows, L.err);
}

cudaError_t launch_rerank_imma(const RerankImmaArgs& a, int max_items, cudaStream_t s) {
  if (max_items <= 0) return cudaSuccess;
  if (!a.pad_desc || (reinterpret_cast<uintptr_t>(a.pad_desc) & 15u)) return cudaErrorInvalidValue;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(k_rerank_imma, cudaFuncAttributeMaxDynamicSharedMemorySize, kRrSmemBytes);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return cudaErrorInvalidValue;
  const int blocks = max_items < sms ? max_items : sms;  // persistent: one block per SM
  return launch_chained_smem(k_rerank_imma, blocks, kRrThreads, kRrSmemBytes, s, a);
}

}  // namespace orbx
