// OpenCV-compatible mode (include/orbx.h, orbx_ocv_*): cv::ORB's published
// algorithm on the GPU, for callers who want OpenCV-like keypoints rather than
// the reference's.  The reference exposes retain_topn but never uses it
// (orb.cpp:41); this mode is where a Harris top-N retain lives.
//
//   pyramid   level 0 = the image; level l = level l-1 resized by 1/scale_factor
//             (bilinear, pixel centres aligned), one launch per level
//   tiles     every level in 64 x 26 tiles, one launch: separable 7x7 Gaussian
//             (sigma 2, reflect-101 border), FAST 9-arc segment test and score,
//             and the 3x3 strict maxima of the score outside edge_threshold,
//             appended as unique 64-bit keys (score, ~position)
//   retain    per level, the best 2 * budget keys by FAST score, then (Harris
//             mode) the best budget keys by Harris score; the keys are unique,
//             so ties cannot split the sets
//   describe  one warp per kept key: its rank among the level's keys (which
//             decides whether it is kept and where it goes, so the output order
//             is deterministic), intensity-centroid angle on the level, rBRIEF
//             with the rotated pattern on the blurred level
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "orb_pattern31.h"
#include "orbx_device.cuh"
#include "orbx_fast.cuh"
#include "orbx_internal.cuh"
#include "orbx_ocv_stage.cuh"

namespace orbx {

constexpr int kOcvMaxLevels = 16;
constexpr int kOcvCandCap = 1 << 17;  // NMS survivors kept per level
constexpr int kOcvSelCap = 8192;      // keys per level after the first retain
constexpr int kOcvHarrisBlock = 7;    // Harris window (blockSize)

constexpr int kOcvTW = 64, kOcvTH = 26;  // tile of the blur + detect kernel
constexpr int kOcvTieCap = 6144;  // equal-score keys kept in shared memory by the first retain

struct OcvLevel {
  int w, h, pitch, n_keep;
  long long off;       // byte offset of the level in the level buffers
  const uint8_t* img;  // the level's pixels: in the level buffer, or the caller's image
  int img_pitch;
  int whole;           // columns that are staged by 16-byte loads: past it single pixels
  float fx, fy;        // size of the level below over this one's
  int tile0, tiles_x;  // first tile of the level, tiles per row
  int key0;            // first of the level's key slots over all levels, in blocks of 8
  float scale;         // scale_factor^level
};

struct OcvArgs {
  int L, edge, fast_thr, harris, patch;
  OcvLevel lv[kOcvMaxLevels];
  float g[7];  // Gaussian taps
  float harris_s4;
  uint8_t* img;
  uint8_t* blr;
  unsigned long long* cand;  // [L][kOcvCandCap]
  int* ncand;
  unsigned long long* sel;   // [L][kOcvSelCap]: after the FAST retain, in no order
  int* nsel;
  unsigned long long* hkey;  // [L][kOcvSelCap]: Harris keys of sel
  const int* umax;
  const int8_t* pattern;
  orbx_ocv_keypoint* out;
  uint8_t* desc;
  int* count;
  int cap;
};

struct OcvWork {
  size_t level_bytes = 0;
  uint8_t *img = nullptr, *blr = nullptr;
  unsigned long long *cand = nullptr, *sel = nullptr, *hkey = nullptr;
  int* counts = nullptr;  // ncand, nsel: 2 * kOcvMaxLevels
  int* umax = nullptr;
  int8_t* pattern = nullptr;
};

void ocv_free(OcvWork* w) {
  if (!w) return;
  cudaFree(w->img);
  cudaFree(w->blr);
  cudaFree(w->cand);
  cudaFree(w->sel);
  cudaFree(w->hkey);
  cudaFree(w->counts);
  cudaFree(w->umax);
  cudaFree(w->pattern);
  delete w;
}

namespace {

// The level whose range [first(l), first(l + 1)) holds i.
template <class First>
__device__ __forceinline__ int ocv_level_of(const OcvArgs& a, int i, First first) {
  int l = 0;
  while (l + 1 < a.L && i >= first(a.lv[l + 1])) l++;
  return l;
}

// Order-preserving image of a float in 32 bits.
__device__ __forceinline__ uint32_t ocv_order(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ocv_unorder(uint32_t o) {
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}

// Blocks of the copy and resize kernels: 64 x 4 threads, 256 columns by 4 rows.  A
// level may have more rows than a grid's second dimension has blocks; the third
// carries on.
constexpr unsigned kOcvGridRows = 65535;
dim3 ocv_grid(const OcvLevel& V) {
  const unsigned rows = (V.h + 3) / 4;
  return dim3((V.w + 255) / 256, std::min(rows, kOcvGridRows), (rows + kOcvGridRows - 1) / kOcvGridRows);
}
__device__ __forceinline__ int ocv_row() { return (blockIdx.z * kOcvGridRows + blockIdx.y) * 4 + threadIdx.y; }

// The first launch of a call clears its counters.
__device__ __forceinline__ void ocv_clear(const OcvArgs& a) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && threadIdx.y == 0 && threadIdx.x < 2 * kOcvMaxLevels)
    a.ncand[threadIdx.x] = 0;  // ncand, then nsel
}

// Level 0 into the level buffer, for images whose rows do not start on 16 bytes.
__global__ void __launch_bounds__(256) k_ocv_copy0(const __grid_constant__ OcvArgs a, const uint8_t* src,
                                                   int src_pitch) {
  chain_wait();
  ocv_clear(a);
  const OcvLevel& V = a.lv[0];
  const int x = 4 * (blockIdx.x * 64 + threadIdx.x), y = ocv_row();
  if (x >= V.w || y >= V.h) return;
  uint32_t v = 0u;
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (x + j < V.w) v |= (uint32_t)src[(long long)y * src_pitch + x + j] << (8 * j);
  *reinterpret_cast<uint32_t*>(a.img + V.off + (long long)y * V.pitch + x) = v;
}

// Level l from level l - 1, bilinear with pixel centres aligned; 4 columns per
// thread, no division.  The launches of one call depend on each other, so what
// counts is the latency of each, and the gap before it (launch_chained).
__global__ void __launch_bounds__(256) k_ocv_resize(const __grid_constant__ OcvArgs a, int l, int clear) {
  const OcvLevel& D = a.lv[l];
  const OcvLevel& S = a.lv[l - 1];
  const int xw = 4 * (blockIdx.x * 64 + threadIdx.x), y = ocv_row();
  const float sy = fmaxf((y + 0.5f) * D.fy - 0.5f, 0.f);
  int y0 = (int)sy;
  const float fy = sy - (float)y0;
  y0 = min(y0, S.h - 1);
  const int y1 = min(y0 + 1, S.h - 1);
  chain_wait();
  if (clear) ocv_clear(a);
  if (xw >= D.w || y >= D.h) return;
  const uint8_t* r0 = S.img + (long long)y0 * S.img_pitch;
  const uint8_t* r1 = S.img + (long long)y1 * S.img_pitch;
  int b00[4], b01[4], b10[4], b11[4];
  float fx4[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int x = min(xw + j, D.w - 1);
    const float sx = fmaxf((x + 0.5f) * D.fx - 0.5f, 0.f);
    int x0 = (int)sx;
    fx4[j] = sx - (float)x0;
    x0 = min(x0, S.w - 1);
    const int x1 = min(x0 + 1, S.w - 1);
    b00[j] = r0[x0], b01[j] = r0[x1];
    b10[j] = r1[x0], b11[j] = r1[x1];
  }
  uint32_t word = 0u;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const float fx = fx4[j];
    const float p00 = (float)b00[j], p01 = (float)b01[j], p10 = (float)b10[j], p11 = (float)b11[j];
    const float v = (1.f - fy) * ((1.f - fx) * p00 + fx * p01) + fy * ((1.f - fx) * p10 + fx * p11);
    word |= (uint32_t)min(max(__float2int_rn(v), 0), 255) << (8 * j);
  }
  // a row's last word may reach into its padding, which nothing reads as pixels
  *reinterpret_cast<uint32_t*>(a.img + D.off + (long long)y * D.pitch + xw) = word;
}

// Blur, FAST and non-maximum suppression of one tile of a level.  The tile is
// staged with a 4-pixel halo (16-byte loads: one per thread) and everything after
// that works in shared memory, where the separate kernels it replaces went
// through global memory pixel by pixel (49 taps per blurred pixel, a full
// 9-arc test per pixel).  The blur filters two columns per packed FP32
// instruction (column k of the tile's left half with column k of its right
// half) and each sum runs in the order of the 49-tap form: rows left to right,
// then top to bottom, one fused multiply-add each.  The four-cardinal pre-test
// leaves a few percent of the pixels for the 9-arc test and the score.
// 1920x1080, 8 levels (6.4 Mpixel): 219 us for the three kernels, 33 us for this
// one (both from a cold cache); bound by instruction issue.
constexpr int kOcvStageSW = kOcvTW + 32;   // bytes per staged row: columns -16 .. 79
constexpr int kOcvStageRows = kOcvTH + 8;  // rows -4 .. kOcvTH + 3
constexpr int kOcvBlurRows = kOcvTH + 6;
constexpr int kOcvScoreSW = kOcvTW + 16;   // score rows: columns -4 .. 75
constexpr int kOcvScoreRows = kOcvTH + 2;  // rows -1 .. kOcvTH
constexpr int kOcvWords = kOcvTW / 4 + 2;  // words tested per row: columns -4 .. kOcvTW + 3
struct OcvTileSmem {
  __align__(16) uint8_t stage[kOcvStageRows * kOcvStageSW];
  __align__(16) float4 row[kOcvBlurRows * kOcvTW / 4];
  __align__(16) uint8_t score[kOcvScoreRows * kOcvScoreSW];
  uint16_t cand[kOcvScoreRows * kOcvWords * 4];
  unsigned long long key[kOcvTH * kOcvTW / 4 + 64];  // strict 3x3 maxima: at most one in four pixels (and edges)
  int n_cand, n_key, base;
};

// bit 7 of each byte of a word of four centres that pass the cardinal pre-test
// of FAST-9 (every run of 9 ring pixels holds two neighbouring cardinal points)
__device__ __forceinline__ uint32_t ocv_pretest4(const uint8_t* w, uint32_t k1) {
  constexpr int sw = kOcvStageSW;
  const uint32_t c = *reinterpret_cast<const uint32_t*>(w);
  const uint32_t cl = *reinterpret_cast<const uint32_t*>(w - 4);
  const uint32_t cr = *reinterpret_cast<const uint32_t*>(w + 4);
  const uint32_t p0 = *reinterpret_cast<const uint32_t*>(w + 3 * sw);
  const uint32_t p8 = *reinterpret_cast<const uint32_t*>(w - 3 * sw);
  return fast9_pretest4(c, p0, __byte_perm(c, cr, 0x6543), p8, __byte_perm(cl, c, 0x4321), k1);
}

__global__ void __launch_bounds__(256) k_ocv_tiles(const __grid_constant__ OcvArgs a) {
  __shared__ OcvTileSmem sm;
  const int t = threadIdx.x;
  const int l = ocv_level_of(a, blockIdx.x, [](const OcvLevel& v) { return v.tile0; });
  const OcvLevel& V = a.lv[l];
  const int lt = blockIdx.x - V.tile0;
  const int ty = lt / V.tiles_x;
  const int x0 = (lt - ty * V.tiles_x) * kOcvTW, y0 = ty * kOcvTH;
  const int w = V.w, h = V.h;
  for (int i = t; i < kOcvScoreRows * kOcvScoreSW / 16; i += 256) reinterpret_cast<uint4*>(sm.score)[i] = uint4{};
  if (t == 0) sm.n_cand = sm.n_key = 0;
  chain_wait();
  // staged rows are reflected at the level's top and bottom; loads past a row's
  // last column or before its start are left out (rows start on 16 bytes)
  static_assert(kOcvStageRows * 6 <= 256, "one staging load per thread");
  if (t < kOcvStageRows * 6) {
    const int r = t / 6, c = t - 6 * r;
    const int x = x0 - 16 + 16 * c, y = reflect101(y0 - 4 + r, h);
    const uint8_t* q = V.img + (long long)y * V.img_pitch + x;
    uint8_t* d = sm.stage + r * kOcvStageSW + 16 * c;
    uint4 v{};
    const bool whole = x >= 0 && x < V.whole;
    if (whole) v = __ldca(reinterpret_cast<const uint4*>(q));
    *reinterpret_cast<uint4*>(d) = v;
    if (!whole) {
#pragma unroll 1
      for (int i = 0, n = ocv_stage_bytes(x, y, w, h); i < n; i++) d[i] = __ldca(q + i);
    }
  }
  __syncthreads();
  // columns -3 .. -1 and w .. w + 2 reflected (for the blur)
  if (x0 == 0 || x0 + kOcvTW + 3 > w) {
    if (t < kOcvStageRows * 6) {
      const int r = t / 6, e = t - 6 * r;
      const int x = e < 3 ? e - 3 : w + e - 3;
      if (x < 0 ? x0 == 0 : x < x0 + kOcvTW + 3) {
        const int sx = reflect101(x, w) - x0 + 16;
        // a level narrower than the reach clamps to columns that may lie outside the stage; nothing reads those outputs
        if (sx >= 0 && sx < kOcvStageSW) sm.stage[r * kOcvStageSW + x - x0 + 16] = sm.stage[r * kOcvStageSW + sx];
      }
    }
    __syncthreads();
  }

  // blur, rows: thread (row, gc) filters columns 4 gc .. 4 gc + 3 of both halves
  float2 g[7];
#pragma unroll
  for (int i = 0; i < 7; i++) g[i] = make_float2(a.g[i], a.g[i]);
  {
    static_assert(kOcvBlurRows * 8 == 256, "one row item per thread");
    const int r = t >> 3, gc = t & 7;
    const uint8_t* s = sm.stage + (r + 1) * kOcvStageSW + 16 + 4 * gc;
    uint32_t wl[3], wr[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      wl[i] = *reinterpret_cast<const uint32_t*>(s - 4 + 4 * i);
      wr[i] = *reinterpret_cast<const uint32_t*>(s - 4 + 4 * i + kOcvTW / 2);
    }
    float2 p[10];
#pragma unroll
    for (int j = 0; j < 10; j++) {
      const uint32_t sel = 0x7540u + ((j + 1) & 3);
      p[j] = __fadd2_rn(make_float2(__uint_as_float(__byte_perm(wl[(j + 1) >> 2], 0x4B000000u, sel)),
                                    __uint_as_float(__byte_perm(wr[(j + 1) >> 2], 0x4B000000u, sel))),
                        make_float2(-8388608.f, -8388608.f));
    }
    float2 q[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      q[j] = __fmul2_rn(g[0], p[j]);
#pragma unroll
      for (int d = 1; d < 7; d++) q[j] = __ffma2_rn(g[d], p[j + d], q[j]);
    }
    // the 16-byte slots of a row in two planes: lanes write consecutive slots
    float4* out = sm.row + r * (kOcvTW / 4) + gc;
    out[0] = make_float4(q[0].x, q[0].y, q[1].x, q[1].y);
    out[8] = make_float4(q[2].x, q[2].y, q[3].x, q[3].y);
  }

  // pre-test of the words of the tile and its 1-pixel ring, where a score can count
  const int xs0 = max(a.edge - 1, x0 - 1), xs1 = min(w - a.edge + 1, x0 + kOcvTW + 1);  // columns [xs0, xs1)
  const int ys0 = max(a.edge - 1, y0 - 1), ys1 = min(h - a.edge + 1, y0 + kOcvTH + 1);
  const uint32_t k1 = (0x7FFFu - (uint32_t)a.fast_thr) * 0x00010001u;
  if (xs0 < xs1 && ys0 < ys1) {
    for (int i = t; i < kOcvScoreRows * kOcvWords; i += 256) {
      const int r = i / kOcvWords, c = i - r * kOcvWords;
      const int x = x0 - 4 + 4 * c, y = y0 - 1 + r;
      if (y < ys0 || y >= ys1 || x + 4 <= xs0 || x >= xs1) continue;
      uint32_t m = ocv_pretest4(sm.stage + (r + 3) * kOcvStageSW + 12 + 4 * c, k1);
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (x + j < xs0 || x + j >= xs1) m &= ~(0x80u << (8 * j));
      if (m) {
        int pos = atomicAdd(&sm.n_cand, __popc(m));
        while (m) {
          const int j = (__ffs(m) >> 3) - 1;
          m &= m - 1u;
          sm.cand[pos++] = (uint16_t)(r * kOcvScoreSW + 4 * c + j);
        }
      }
    }
  }
  __syncthreads();

  // blur, columns: thread (row, gc)
  if (t < kOcvTH * 8) {
    const int r = t >> 3, gc = t & 7, y = y0 + r;
    if (y < h) {
      float2 acc[4];
#pragma unroll
      for (int d = 0; d < 7; d++) {
        const float4 v0 = sm.row[(r + d) * (kOcvTW / 4) + gc], v1 = sm.row[(r + d) * (kOcvTW / 4) + gc + 8];
        const float2 hv[4] = {make_float2(v0.x, v0.y), make_float2(v0.z, v0.w), make_float2(v1.x, v1.y),
                              make_float2(v1.z, v1.w)};
#pragma unroll
        for (int j = 0; j < 4; j++) acc[j] = d == 0 ? __fmul2_rn(g[0], hv[j]) : __ffma2_rn(g[d], hv[j], acc[j]);
      }
      // rounded to nearest even by adding 1.5 * 2^23; 0 <= acc < 255.5
      uint32_t bl = 0u, br = 0u;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float2 v = __fadd2_rn(acc[j], make_float2(12582912.f, 12582912.f));
        bl |= (__float_as_uint(v.x) & 0xFFu) << (8 * j);
        br |= (__float_as_uint(v.y) & 0xFFu) << (8 * j);
      }
      uint8_t* q = a.blr + V.off + (long long)y * V.pitch + x0 + 4 * gc;  // the pitch covers the tile
      *reinterpret_cast<uint32_t*>(q) = bl;
      *reinterpret_cast<uint32_t*>(q + kOcvTW / 2) = br;
    }
  }

  // 9-arc test and score of the candidates
  const int nc = sm.n_cand;
  for (int i = t; i < nc; i += 256) {
    const int at = sm.cand[i];
    const int r = at / kOcvScoreSW, c = at - r * kOcvScoreSW;
    const uint8_t* p = sm.stage + (r + 3) * kOcvStageSW + 12 + c;
    const int v = p[0];
    if (fast9_full(p, kOcvStageSW, v - a.fast_thr, v + a.fast_thr)) {
      int d[25];
#pragma unroll
      for (int k = 0; k < 25; k++) d[k] = (int)(short)(v - p[ring_dy(k) * kOcvStageSW + ring_dx(k)]);
      sm.score[at] = (uint8_t)min(max((int)fast_score(d, a.fast_thr), 1), 255);
    }
  }
  __syncthreads();
  // strict maxima among the tile's own pixels outside the edge band
  for (int i = t; i < nc; i += 256) {
    const int at = sm.cand[i];
    const int c = sm.score[at];
    const int r = at / kOcvScoreSW, x = x0 - 4 + at - r * kOcvScoreSW, y = y0 - 1 + r;
    if (!c || x < max(a.edge, x0) || x >= min(w - a.edge, x0 + kOcvTW) || y < max(a.edge, y0) ||
        y >= min(h - a.edge, y0 + kOcvTH))
      continue;
    const uint8_t* s = sm.score + at;
    constexpr int p = kOcvScoreSW;
    if (c <= s[-p - 1] || c <= s[-p] || c <= s[-p + 1] || c <= s[-1] || c <= s[1] || c <= s[p - 1] || c <= s[p] ||
        c <= s[p + 1])
      continue;
    const int pos = atomicAdd(&sm.n_key, 1);
    sm.key[pos] = ((unsigned long long)c << 32) | (0xFFFFFFFFu - (uint32_t)((long long)y * w + x));
  }
  __syncthreads();
  const int nk = sm.n_key;
  if (nk == 0) return;
  if (t == 0) sm.base = atomicAdd(&a.ncand[l], nk);
  __syncthreads();
  for (int i = t; i < nk; i += 256)
    if (sm.base + i < kOcvCandCap) a.cand[(size_t)l * kOcvCandCap + sm.base + i] = sm.key[i];
}

// Of 256 bins, counted from the top, the one where the running count reaches
// `want`; *above gets the count of the bins above it.  Every thread of the block
// (at least 256) calls it; s_warp holds 8 ints.
__device__ __forceinline__ int ocv_top_bin(const int* s_hist, int want, int* s_warp, int* s_bin, int* s_above) {
  const int t = threadIdx.x, lane = t & 31;
  int v = 0, incl = 0;
  if (t < 256) {
    v = s_hist[255 - t];
    incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += n;
    }
    if (lane == 31) s_warp[t >> 5] = incl;
  }
  __syncthreads();
  if (t < 256) {
    for (int k = 0; k < (t >> 5); k++) incl += s_warp[k];
    if (incl >= want && incl - v < want) {
      *s_bin = 255 - t;
      *s_above = incl - v;
    }
  }
  __syncthreads();
  return *s_bin;
}

// Per level (one block of 1024 threads): the min(n, k) keys with the best FAST
// scores, and of the keys with the last score taken those earliest in raster
// order.  A histogram of the 8-bit scores gives that last score, one pass takes
// the keys above it and collects the ones at it, and four 8-bit passes over
// these find the position up to which they are taken: 15.5 -> 5.2 us for 5000
// features, against eight passes over all keys and a sort.
__global__ void __launch_bounds__(1024) k_ocv_select(const __grid_constant__ OcvArgs a, int mult) {
  __shared__ int s_hist[256];
  __shared__ uint32_t s_tie[kOcvTieCap];
  __shared__ int s_warp[8], s_bin, s_above, s_cnt, s_ntie;
  const int l = blockIdx.x, t = threadIdx.x, lane = t & 31;
  const int k = min(a.lv[l].n_keep * mult, kOcvSelCap);
  const unsigned long long* in = a.cand + (size_t)l * kOcvCandCap;
  unsigned long long* dst = a.sel + (size_t)l * kOcvSelCap;
  if (t < 256) s_hist[t] = 0;
  if (t == 0) s_cnt = s_ntie = 0;
  chain_wait();
  const int n = min(a.ncand[l], kOcvCandCap);
  if (n <= k) {
    for (int j = t; j < n; j += 1024) dst[j] = in[j];
    if (t == 0) a.nsel[l] = n;
    return;
  }
  if (k == 0) return;  // nsel was cleared
  __syncthreads();
  for (int j = t; j < n; j += 1024) atomicAdd(&s_hist[(int)(in[j] >> 32)], 1);
  __syncthreads();
  const int last = ocv_top_bin(s_hist, k, s_warp, &s_bin, &s_above);
  const int need = k - s_above;  // keys to take among those scored `last`
  for (int j0 = 0; j0 < n; j0 += 1024) {
    const int j = j0 + t;
    const unsigned long long key = j < n ? in[j] : 0ull;
    const int sc = (int)(key >> 32);  // 0 past the end: no key scores 0
    const unsigned up = __ballot_sync(0xffffffffu, sc > last), eq = __ballot_sync(0xffffffffu, sc == last);
    int bu = 0, be = 0;
    if (lane == 0) {
      if (up) bu = atomicAdd(&s_cnt, __popc(up));
      if (eq) be = atomicAdd(&s_ntie, __popc(eq));
    }
    bu = __shfl_sync(0xffffffffu, bu, 0) + __popc(up & ((1u << lane) - 1u));
    be = __shfl_sync(0xffffffffu, be, 0) + __popc(eq & ((1u << lane) - 1u));
    if (sc > last) dst[bu] = key;
    if (sc == last && be < kOcvTieCap) s_tie[be] = (uint32_t)key;
  }
  __syncthreads();
  const int m = s_ntie;
  const bool held = m <= kOcvTieCap;  // else the passes read the keys again
  const int nt = held ? m : n;
  auto tie = [&](int j, uint32_t* low) {
    if (held) {
      *low = s_tie[j];
      return true;
    }
    const unsigned long long key = in[j];
    *low = (uint32_t)key;
    return (int)(key >> 32) == last;
  };
  uint32_t prefix = 0u, mask = 0u;
  int want = need;
  for (int sh = 24; sh >= 0 && m > need; sh -= 8) {
    if (t < 256) s_hist[t] = 0;
    __syncthreads();
    for (int j = t; j < nt; j += 1024) {
      uint32_t low;
      if (tie(j, &low) && (low & mask) == prefix) atomicAdd(&s_hist[(low >> sh) & 0xFFu], 1);
    }
    __syncthreads();
    const int bin = ocv_top_bin(s_hist, want, s_warp, &s_bin, &s_above);
    want -= s_above;
    prefix |= (uint32_t)bin << sh;
    mask |= 0xFFu << sh;
    __syncthreads();
  }
  for (int j = t; j < nt; j += 1024) {
    uint32_t low;
    if (tie(j, &low) && low >= prefix) {
      const int pos = atomicAdd(&s_cnt, 1);
      if (pos < kOcvSelCap) dst[pos] = ((unsigned long long)last << 32) | low;
    }
  }
  if (t == 0) a.nsel[l] = k;
}

// Harris score (blockSize 7, k = 0.04, derivatives of the 3x3 Sobel form) of
// the keys kept by the FAST retain; the Harris key keeps the position bits.
// Eight lanes per key, one window row each (the integer sums are exact in any
// order): 23.6 -> 7.7 us for 5000 features (cold), one thread per key before.
__global__ void __launch_bounds__(64) k_ocv_harris(const __grid_constant__ OcvArgs a) {
  const int l = ocv_level_of(a, blockIdx.x, [](const OcvLevel& v) { return v.key0; });
  const OcvLevel& V = a.lv[l];
  const int j = 8 * (blockIdx.x - V.key0) + (threadIdx.x >> 3), sub = threadIdx.x & 7;
  chain_wait();
  const bool on = j < a.nsel[l];
  const unsigned long long key = on ? a.sel[(size_t)l * kOcvSelCap + j] : 0ull;
  const uint32_t low = (uint32_t)key;
  int sa = 0, sb = 0, sc = 0;
  if (on && sub < 7) {
    const uint32_t idx = 0xFFFFFFFFu - low;
    const int y = (int)(idx / (uint32_t)V.w), x = (int)(idx - (uint32_t)y * (uint32_t)V.w);
    const int p = V.img_pitch;
    const uint8_t* r = V.img + (long long)(y + sub - 3) * p + x;
    int s1[9], d1[9];  // column sums (1 2 1) and differences of the three rows
#pragma unroll
    for (int i = 0; i < 9; i++) {
      const int u = r[i - 4 - p], m = r[i - 4], d = r[i - 4 + p];
      s1[i] = u + 2 * m + d;
      d1[i] = d - u;
    }
#pragma unroll
    for (int i = 0; i < 7; i++) {
      const int ix = s1[i + 2] - s1[i], iy = d1[i] + 2 * d1[i + 1] + d1[i + 2];
      sa += ix * ix;
      sb += iy * iy;
      sc += ix * iy;
    }
  }
#pragma unroll
  for (int d = 4; d >= 1; d >>= 1) {
    sa += __shfl_xor_sync(0xffffffffu, sa, d);
    sb += __shfl_xor_sync(0xffffffffu, sb, d);
    sc += __shfl_xor_sync(0xffffffffu, sc, d);
  }
  if (!on || sub) return;
  const float fa = (float)sa, fb = (float)sb, fc = (float)sc;
  const float r = (fa * fb - fc * fc - 0.04f * (fa + fb) * (fa + fb)) * a.harris_s4;
  a.hkey[(size_t)l * kOcvSelCap + j] = ((unsigned long long)ocv_order(r) << 32) | low;
}

// One warp per key: its rank among the level's n keys (n - 1 comparisons spread
// over the block: each thread compares the keys it loads with the block's
// eight), then, when the rank is inside the level's budget, angle, descriptor
// and output entry.  The rank replaces a radix select and a bitonic sort by one
// block per level, 34 us for 5000 features, at 3 us more in this kernel (18.7 ->
// 21.8 us, cold).
__global__ void __launch_bounds__(256) k_ocv_describe(const __grid_constant__ OcvArgs a) {
  __shared__ unsigned long long s_key[8];
  __shared__ int s_rank[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int l = ocv_level_of(a, blockIdx.x, [](const OcvLevel& v) { return v.key0; });
  const int j0 = 8 * (blockIdx.x - a.lv[l].key0);
  const unsigned long long* keys = (a.harris ? a.hkey : a.sel) + (size_t)l * kOcvSelCap;
  chain_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    int tot = 0;
    for (int m = 0; m < a.L; m++) tot += min(a.nsel[m], a.lv[m].n_keep);
    *a.count = min(tot, a.cap);
  }
  const int n = a.nsel[l];
  if (j0 >= n) return;
  if (threadIdx.x < 8) {
    s_key[threadIdx.x] = j0 + (int)threadIdx.x < n ? keys[j0 + threadIdx.x] : ~0ull;
    s_rank[threadIdx.x] = 0;
  }
  __syncthreads();
  {
    unsigned long long mine[8];
    int above[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      mine[i] = s_key[i];
      above[i] = 0;
    }
    for (int j = threadIdx.x; j < n; j += 256) {
      const unsigned long long key = keys[j];
#pragma unroll
      for (int i = 0; i < 8; i++) above[i] += key > mine[i];
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int c = (int)__reduce_add_sync(0xffffffffu, (unsigned)above[i]);
      if (lane == 0 && c) atomicAdd(&s_rank[i], c);
    }
  }
  __syncthreads();
  const int rank = s_rank[warp];
  if (j0 + warp >= n || rank >= a.lv[l].n_keep) return;
  int base = 0;
  for (int m = 0; m < l; m++) base += min(a.nsel[m], a.lv[m].n_keep);
  const int o = base + rank;
  if (o >= a.cap) return;
  const OcvLevel& V = a.lv[l];
  const unsigned long long key = s_key[warp];
  const uint32_t idx = 0xFFFFFFFFu - (uint32_t)key;
  const int y = (int)(idx / (uint32_t)V.w), x = (int)(idx - (uint32_t)y * (uint32_t)V.w);
  int p = V.img_pitch;
  // intensity centroid over the disc of radius patch / 2
  const int half = a.patch / 2;
  const uint8_t* c = V.img + (long long)y * p + x;
  int m10 = 0, m01 = 0;
  const int u = lane - half;
  if (lane <= 2 * half) {
    m10 = u * (int)c[u];
    for (int v = 1; v <= half; v++) {
      const int d = a.umax[v];
      if (u >= -d && u <= d) {
        const int vp = c[u + v * p], vm = c[u - v * p];
        m10 += u * (vp + vm);
        m01 += v * (vp - vm);
      }
    }
  }
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    m10 += __shfl_xor_sync(0xffffffffu, m10, s);
    m01 += __shfl_xor_sync(0xffffffffu, m01, s);
  }
  float ang = atan2f((float)m01, (float)m10) * (180.f / 3.14159265358979f);
  if (ang < 0.f) ang += 360.f;
  // rBRIEF on the blurred level: lane t computes byte t from 8 point pairs
  const float th = ang * (3.14159265358979f / 180.f);
  const float ca = cosf(th), sa = sinf(th);
  p = V.pitch;
  const uint8_t* b = a.blr + V.off + (long long)y * p + x;
  uint32_t byte = 0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int t = 8 * lane + k;
    const float x0 = a.pattern[4 * t], y0 = a.pattern[4 * t + 1];
    const float x1 = a.pattern[4 * t + 2], y1 = a.pattern[4 * t + 3];
    const int i0 = b[__float2int_rn(x0 * sa + y0 * ca) * p + __float2int_rn(x0 * ca - y0 * sa)];
    const int i1 = b[__float2int_rn(x1 * sa + y1 * ca) * p + __float2int_rn(x1 * ca - y1 * sa)];
    byte |= (uint32_t)(i0 < i1) << k;
  }
  a.desc[(size_t)o * 32 + lane] = (uint8_t)byte;
  if (lane == 0) {
    orbx_ocv_keypoint kp;
    kp.x = (float)x * V.scale;
    kp.y = (float)y * V.scale;
    kp.size = (float)a.patch * V.scale;
    kp.angle = ang;
    kp.response = a.harris ? ocv_unorder((uint32_t)(key >> 32)) : (float)(uint32_t)(key >> 32);
    kp.octave = l;
    a.out[o] = kp;
  }
}

}  // namespace
}  // namespace orbx

using namespace orbx;

namespace {
struct OGuard {
  int prev = -1;
  explicit OGuard(int d) {
    if (cudaGetDevice(&prev) == cudaSuccess && prev != d)
      cudaSetDevice(d);
    else
      prev = -1;
  }
  ~OGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};
#define OCHK(x)                                                             \
  do {                                                                      \
    cudaError_t _e = (x);                                                   \
    if (_e != cudaSuccess) {                                                \
      (void)cudaGetLastError();                                             \
      return _e == cudaErrorMemoryAllocation ? ORBX_ERR_NOMEM : ORBX_ERR_CUDA; \
    }                                                                       \
  } while (0)
}  // namespace

ORBX_API int orbx_ocv_default_params(orbx_ocv_params* p) {
  if (!p) return ORBX_ERR_ARG;
  // cv::ORB defaults except the budget (500 there)
  p->nfeatures = 5000;
  p->scale_factor = 1.2f;
  p->nlevels = 8;
  p->edge_threshold = 31;
  p->score_type = 0;
  p->patch_size = 31;
  p->fast_threshold = 20;
  return ORBX_OK;
}

ORBX_API int orbx_ocv_detect_and_compute(orbx_ctx* ctx, const orbx_ocv_params* p, const uint8_t* d_image, int w, int h,
                                         int pitch, orbx_ocv_keypoint* d_keypoints, uint8_t* d_desc, int* d_n,
                                         int cap) {
  if (!ctx || !p || !d_image || !d_keypoints || !d_desc || !d_n || cap < 0 || w < 16 || h < 16 || pitch < w)
    return ORBX_ERR_ARG;
  if (p->nfeatures < 1 || p->nfeatures > 16000 || !(p->scale_factor > 1.f && p->scale_factor <= 2.f) ||
      p->nlevels < 1 || p->nlevels > kOcvMaxLevels || p->edge_threshold < 19 || p->patch_size != 31 ||
      p->fast_threshold < 0 || p->fast_threshold > 255 || (p->score_type != 0 && p->score_type != 1))
    return ORBX_ERR_ARG;
  if ((long long)w * h >= (1ll << 31)) return ORBX_ERR_SIZE;
  OGuard g(ctx_device(ctx));
  cudaStream_t s = ctx_stream(ctx);
  OcvArgs a{};
  a.L = p->nlevels;
  a.edge = p->edge_threshold;
  a.fast_thr = p->fast_threshold;
  a.harris = p->score_type == 0 ? 1 : 0;
  a.patch = p->patch_size;
  int n_tiles = 0, n_key_blocks = 0;
  // levels: sizes rounded from the previous scale, budgets geometric in 1 / scale
  {
    const double f = 1.0 / p->scale_factor;
    double per = p->nfeatures * (1.0 - f) / (1.0 - std::pow(f, (double)p->nlevels));
    const int mult = a.harris ? 2 : 1;
    int used = 0, tiles = 0, key_blocks = 0;
    long long off = 0;
    for (int l = 0; l < a.L; l++) {
      const double sc = std::pow((double)p->scale_factor, (double)l);
      OcvLevel& V = a.lv[l];
      V.w = std::max(1, (int)std::lround(w / sc));
      V.h = std::max(1, (int)std::lround(h / sc));
      V.pitch = (V.w + 127) / 128 * 128;
      V.off = off;
      V.scale = (float)sc;
      if (l < a.L - 1) {
        V.n_keep = (int)std::lround(per);
        used += V.n_keep;
        per *= f;
      } else {
        V.n_keep = std::max(p->nfeatures - used, 0);
      }
      if (V.n_keep * (a.harris ? 2 : 1) > kOcvSelCap) return ORBX_ERR_SIZE;
      off += (long long)V.pitch * (V.h + 1);
      V.img_pitch = V.whole = V.pitch;
      if (l > 0) {
        V.fx = (float)a.lv[l - 1].w / (float)V.w;
        V.fy = (float)a.lv[l - 1].h / (float)V.h;
      }
      V.tile0 = tiles;
      V.tiles_x = (V.w + kOcvTW - 1) / kOcvTW;
      tiles += V.tiles_x * ((V.h + kOcvTH - 1) / kOcvTH);
      V.key0 = key_blocks;
      key_blocks += (V.n_keep * mult + 7) / 8;
    }
    n_tiles = tiles;
    n_key_blocks = key_blocks;
    // Gaussian taps for sigma 2
    double gs[7], sum = 0.0;
    for (int i = 0; i < 7; i++) {
      gs[i] = std::exp(-(double)((i - 3) * (i - 3)) / (2.0 * 4.0));
      sum += gs[i];
    }
    for (int i = 0; i < 7; i++) a.g[i] = (float)(gs[i] / sum);
    const double hs = 1.0 / (4.0 * kOcvHarrisBlock * 255.0);
    a.harris_s4 = (float)(hs * hs * hs * hs);
    // workspace
    OcvWork*& W = ctx_ocv(ctx);
    if (!W) W = new OcvWork();
    const size_t lb = (size_t)off;
    if (W->level_bytes < lb) {
      cudaFree(W->img);
      cudaFree(W->blr);
      W->img = W->blr = nullptr;
      W->level_bytes = 0;
      OCHK(cudaMalloc(&W->img, lb));
      OCHK(cudaMalloc(&W->blr, lb));
      W->level_bytes = lb;
    }
    if (!W->cand) {
      OCHK(cudaMalloc(&W->cand, sizeof(unsigned long long) * (size_t)kOcvMaxLevels * kOcvCandCap));
      OCHK(cudaMalloc(&W->sel, sizeof(unsigned long long) * (size_t)kOcvMaxLevels * kOcvSelCap));
      OCHK(cudaMalloc(&W->hkey, sizeof(unsigned long long) * (size_t)kOcvMaxLevels * kOcvSelCap));
      OCHK(cudaMalloc(&W->counts, sizeof(int) * 2 * kOcvMaxLevels));
      int umax[64] = {0};
      umax_table(p->patch_size, umax);
      OCHK(cudaMalloc(&W->umax, sizeof(umax)));
      OCHK(cudaMemcpy(W->umax, umax, sizeof(umax), cudaMemcpyHostToDevice));
      OCHK(cudaMalloc(&W->pattern, sizeof(kOrbPattern31)));
      OCHK(cudaMemcpy(W->pattern, kOrbPattern31, sizeof(kOrbPattern31), cudaMemcpyHostToDevice));
    }
    a.img = W->img;
    a.blr = W->blr;
    a.cand = W->cand;
    a.sel = W->sel;
    a.hkey = W->hkey;
    a.ncand = W->counts;
    a.nsel = W->counts + kOcvMaxLevels;
    a.umax = W->umax;
    a.pattern = W->pattern;
  }
  a.out = d_keypoints;
  a.desc = d_desc;
  a.count = d_n;
  a.cap = cap;
  // level 0 is the caller's image in place when its rows start on 16 bytes
  const bool copy = ((reinterpret_cast<uintptr_t>(d_image) | (uintptr_t)pitch) & 15u) != 0;
  for (int l = 0; l < a.L; l++) a.lv[l].img = a.img + a.lv[l].off;
  if (!copy) {
    a.lv[0].img = d_image;
    a.lv[0].img_pitch = pitch;
    a.lv[0].whole = w / 16 * 16;
  }
  const dim3 block(64, 4);
  if (copy)
    OCHK(launch_chained(k_ocv_copy0, ocv_grid(a.lv[0]), block, s, a, d_image, pitch));
  else if (a.L == 1)
    OCHK(cudaMemsetAsync(a.ncand, 0, sizeof(int) * 2 * kOcvMaxLevels, s));
  for (int l = 1; l < a.L; l++)
    OCHK(launch_chained(k_ocv_resize, ocv_grid(a.lv[l]), block, s, a, l, (int)(l == 1 && !copy)));
  OCHK(launch_chained(k_ocv_tiles, n_tiles, 256, s, a));
  OCHK(launch_chained(k_ocv_select, a.L, 1024, s, a, a.harris ? 2 : 1));
  if (a.harris && n_key_blocks > 0) OCHK(launch_chained(k_ocv_harris, n_key_blocks, 64, s, a));
  OCHK(launch_chained(k_ocv_describe, std::max(n_key_blocks, 1), 256, s, a));
  return ORBX_OK;
}
