// Stage bodies of the sm_100a ORB pipeline as device functions: pyramid +
// blur tiles, FAST-9 + score tiles and NMS strips.  Each kernel of the
// five-launch form (orbx_detect.cu) runs one of them per block, and the
// persistent batch kernel (orbx_persist.cu) runs them per claimed work item.
#pragma once
#include "orbx_device.cuh"
#include "orbx_internal.cuh"
#include "orbx_fast.cuh"

namespace orbx {

// Loads of data a stage reads: plain (coherent) cached loads, not the read-only
// path.  In the persistent kernel an earlier stage wrote it in the same launch, and a
// chained kernel has started before the kernel that wrote it ended (chain_wait).
template <bool P, class T>
__device__ __forceinline__ T ldx(const T* p) {
  return __ldca(p);
}

// The frame table of a launch: from the launch parameters (INL, batches of up
// to kInlineFrames frames, constant-bank reads) or from global memory.
template <bool INL>
__device__ __forceinline__ const Frame& batch_frame(const Batch& b, int f) {
  if constexpr (INL)
    return b.inl[f];
  else
    return b.frames[f];
}
// Index of the frame whose range [base[f], base[f+1]) holds t (base in the
// launch parameters when INL).
template <bool INL>
__device__ __forceinline__ int find_frame_in(const int* base, int n, int t) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    int v;
    if constexpr (INL)
      v = base[mid];
    else
      v = __ldg(base + mid);
    if (v <= t)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------------------
// Pyramid + blur
//
// Octave o is the nearest-neighbour decimation img[y<<o][x<<o] of level 0
// (gDownSampleUnroll4, orbd.cu:514-535; octave 0 is a copy, orbd.cu:1584).
// The blurred pyramid is the separable 7-tap sigma-2 filter of each octave with
// reflect-101 borders (gConv2dUnroll, orbd.cu:1273-1338), computed here out of
// place, so it has no dependence on block scheduling.  With pyr_src set the
// octaves are read from an existing pyramid instead (hGassianBlur on a
// caller's buffer, orbd.cu:1732-1773).
//
// What bounds it: instruction issue (a pixel needs 14 FP32 operations and 1.9
// bytes of traffic), and on one frame the latency of a block's two passes.  A
// block takes kPyrTW columns and TH rows.  First, 8 threads per source row (TH +
// 6 of them) each read the words of 8 columns of the tile's left half and of 8
// of its right half straight from global memory, store the raw bytes, and filter
// the row: the two halves sit in the two halves of packed FP32 registers, so one
// instruction filters two pixels, and 8 columns share 14 byte-to-float
// conversions.  Only the filtered rows go through shared memory.  Then each
// thread takes 4 columns of both halves and 4 consecutive rows, for which it
// reads 10 filtered rows.  The code that one block runs through is kept short
// (few unrolled copies, one word-load form per octave): on a frame of one wave
// of blocks its instruction fetch is part of the time.  For a 1920x1080 pair the
// form before, which staged bytes and floats of a 128 x 30 tile in shared memory
// and filtered every row by itself, took 9.09 M warp instructions; this one
// takes 7.09 M with the pair's 26-row tiles (5.6 M with 58 rows).  24 mixed pairs
// (147 Mpixel, 58 rows): 558 -> 305 us.
// ---------------------------------------------------------------------------

// Exact small-integer <-> float conversions on the full-rate pipes: a float
// whose exponent field is 2^23 holds the integer in its mantissa.  byte_bits:
// the byte of `word` that selector `sel` (0x754j, j = 0..3) picks, in the low
// mantissa byte of 2^23, i.e. the float bits of 2^23 + byte.
__device__ __forceinline__ float byte_bits(uint32_t word, uint32_t sel) {
  return __uint_as_float(__byte_perm(word, 0x4B000000u, sel));
}
// Low bytes of four 32-bit words packed into one word (a | b << 8 | c << 16 | d << 24).
__device__ __forceinline__ uint32_t pack_low_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}
__device__ __forceinline__ float2 pair2(float v) { return make_float2(v, v); }
// gauss_dot4 on both lanes of a pair: the same operations in the same order,
// each lane rounded as the scalar form (one packed sm_100 FP32 instruction per step).
__device__ __forceinline__ float2 gauss_dot4x2(const float2* k, float2 t0, float2 t1, float2 t2, float2 t3) {
  float2 acc = __ffma2_rn(k[0], t0, __fmul2_rn(k[1], t1));
  acc = __ffma2_rn(k[2], t2, acc);
  return __ffma2_rn(k[3], t3, acc);
}

// Source of one octave's rows.
struct PyrSrc {
  const uint8_t* base;
  long long pitch;  // bytes between octave rows
  int sh;           // log2 of the bytes between octave pixels
  int ow;
  Span span;
  BoundsRec* rec;
};
// How four neighbouring pixels of an octave row load as one word.
enum : int {
  kPyrWord = 0,    // octave 0 (or a caller's pyramid): an aligned word
  kPyrEvery2 = 1,  // octave 1: every second byte of 8 aligned bytes
  kPyrEvery4 = 2,  // octave 2: every fourth byte of 16 aligned bytes
  kPyrBytes = 3    // octaves 3, 4 and images whose base or pitch is not aligned: four byte loads
};
// Octave columns 4 w .. 4 w + 3 of a row (w inside the octave; columns past its
// last one hold anything).  An aligned word of a row's last pixel ends inside
// the row's pitch at octave 0, and at octaves 1 and 2 at worst in the image row
// below, which exists since octave rows are 2 or 4 image rows apart; byte loads
// stop at the last pixel.
template <bool PL, int KIND>
__device__ __forceinline__ uint32_t pyr_word(const PyrSrc& p, const uint8_t* row, int w) {
  if constexpr (KIND != kPyrBytes) {
    const uint8_t* q = row + ((4 << KIND) * w);
    if (!ORBX_IN(p.rec, kSitePyrLoad, p.span, q, 4 << KIND)) return 0u;
    if constexpr (KIND == kPyrWord) {
      return ldx<PL>(reinterpret_cast<const uint32_t*>(q));
    } else if constexpr (KIND == kPyrEvery2) {
      const uint2 v = ldx<PL>(reinterpret_cast<const uint2*>(q));
      return __byte_perm(v.x, v.y, 0x6420);
    } else {
      const uint4 v = ldx<PL>(reinterpret_cast<const uint4*>(q));
      return pack_low_bytes(v.x, v.y, v.z, v.w);
    }
  } else {
    uint32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint8_t* q = row + (min(4 * w + j, p.ow - 1) << p.sh);
      v[j] = ORBX_IN(p.rec, kSitePyrLoad, p.span, q, 1) ? ldx<PL>(q) : 0u;
    }
    return pack_low_bytes(v[0], v[1], v[2], v[3]);
  }
}

// The words of columns x - 4 .. x + 11 of a row (x a multiple of 8), columns
// outside the octave reflected (reflect-101).  The four words are loaded with
// their indices clamped to the octave; a reflected column that an output needs
// (at most 3 past an edge) lies in one of them, and with n = ow - x columns left
// from x on, byte selectors put it in place: column n + e is column n - 2 - e.
// out[1] takes bytes of words (0, 1), out[2] of (n <= 4 ? 0 : 2, 1), out[3] of
// (n <= 8 ? 1 : 3, 2), in that order; n >= 12 is the identity.
__device__ __constant__ uint16_t kPyrSel[13][3] = {
    {0x0000, 0x0000, 0x0000}, {0x1234, 0x0000, 0x0000}, {0x3454, 0x0002, 0x0000},
    {0x5654, 0x0034, 0x0000}, {0x7654, 0x0456, 0x0000}, {0x7654, 0x5670, 0x0000},
    {0x7654, 0x7010, 0x0002}, {0x7654, 0x1210, 0x0034}, {0x7654, 0x3210, 0x0456},
    {0x7654, 0x3210, 0x5670}, {0x7654, 0x3210, 0x7010}, {0x7654, 0x3210, 0x1210},
    {0x7654, 0x3210, 0x3210}};
template <bool PL, int KIND>
__device__ __forceinline__ void pyr_words_edge(const PyrSrc& p, const uint8_t* row, int x, uint32_t out[4]) {
  const int n = min(max(p.ow - x, 0), 12);
  const int w = x >> 2, last = (p.ow - 1) >> 2;
  uint32_t v[4];
#pragma unroll
  for (int i = 0; i < 4; i++) v[i] = pyr_word<PL, KIND>(p, row, min(max(w - 1 + i, 0), last));
  out[0] = x == 0 ? __byte_perm(v[1], 0u, 0x1230) : v[0];  // columns -3, -2, -1 are columns 3, 2, 1
  out[1] = __byte_perm(v[0], v[1], kPyrSel[n][0]);
  out[2] = __byte_perm(n <= 4 ? v[0] : v[2], v[1], kPyrSel[n][1]);
  out[3] = __byte_perm(n <= 8 ? v[1] : v[3], v[2], kPyrSel[n][2]);
}
// The same for a thread's columns of both halves of a tile; inside: the tile's
// words all lie in the octave.
template <bool PL, int KIND>
__device__ __forceinline__ void pyr_words(const PyrSrc& p, const uint8_t* row, int x, bool inside, uint32_t wl[4],
                                          uint32_t wr[4]) {
  constexpr int kHalf = kPyrTW / 2;
  if (inside) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      wl[i] = pyr_word<PL, KIND>(p, row, (x >> 2) - 1 + i);
      wr[i] = pyr_word<PL, KIND>(p, row, (x >> 2) - 1 + i + kHalf / 4);
    }
  } else {
    pyr_words_edge<PL, KIND>(p, row, x, wl);
    pyr_words_edge<PL, KIND>(p, row, x + kHalf, wr);
  }
}

// Position of pyramid tile t (tile index over the batch) of TH rows.
struct PyrTile {
  int f;       // frame
  int o;       // octave
  int lt;      // tile index within the octave
  int x0, y0;  // octave-pixel origin
};
template <bool INL, int TH>
__device__ __forceinline__ PyrTile pyr_tile_at(const Batch& b, int t) {
  const int* base = INL ? b.inl_pyr_base : b.pyr_base;
  PyrTile g;
  g.f = find_frame_in<INL>(base, b.n_frames, t);
  const Frame& F = batch_frame<INL>(b, g.f);
  int lt = t - (INL ? base[g.f] : __ldg(base + g.f));
  int o = 0;
  while (o + 1 < F.n_oct && lt >= F.pyr_tile_base[o + 1]) o++;
  lt -= F.pyr_tile_base[o];
  const int tiles_x = F.pyr_tiles_x[o];
  g.o = o;
  g.lt = lt;
  const int ty = lt / tiles_x;
  g.x0 = (lt - ty * tiles_x) * kPyrTW;
  g.y0 = ty * TH;
  return g;
}

// The horizontally filtered rows of a tile.  Column k of the left half and
// column k of the right half form pair k; two pairs are a 16-byte slot, and
// slot 4 g + m of a row lies at m * 8 + (g + 4 (m >> 1)) % 8, so that the 8
// threads that write a row and the 16 that read it touch distinct banks.
constexpr int kPyrRowSlots = kPyrTW / 4;
__device__ __forceinline__ int pyr_slot(int g, int m) { return m * 8 + ((g + 4 * (m >> 1)) & 7); }
template <int TH>
struct PyrSmem {
  float4 row[(TH + 6) * kPyrRowSlots];
};

// Four columns x .. x + 3 of octave row y as stored: columns past the row carry
// the caller's padding (the reference copies h * pitch0 bytes, orbd.cu:1584) or
// zeros.  x is below the octave's pitch.
template <bool PL>
__device__ __forceinline__ uint32_t pyr_padded(const PyrSrc& p, bool copy_pad, int x, int y, uint32_t v) {
  const int n = p.ow - x;
  if (n >= 4) return v;
  const uint32_t mask = n <= 0 ? 0u : (1u << (8 * n)) - 1u;
  uint32_t pad = 0u;
  if (copy_pad) {
    const uint8_t* q = p.base + y * p.pitch + x;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t v1 = ORBX_IN(p.rec, kSitePyrPadLoad, p.span, q + j, 1) ? ldx<PL>(q + j) : 0u;
      pad |= v1 << (8 * j);
    }
  }
  return (v & mask) | (pad & ~mask);
}

// One pyramid tile (tile index t over the batch).  PL: the level-0 image is
// copied in during the same launch (coherent loads instead of the read-only path).
template <bool PL, int TH, bool INL = false>
__device__ __forceinline__ void pyr_tile(const Batch& b, int t, PyrSmem<TH>& sm) {
  static_assert(kPyrTW == 128 && kPyrThreads == 256 && (TH + 6) % 16 == 0, "thread layout of the two passes");
  constexpr int kHalf = kPyrTW / 2;
  const PyrTile g = pyr_tile_at<INL, TH>(b, t);
  const Frame& F = batch_frame<INL>(b, g.f);
  if (g.o == 0 && g.lt == 0) {
    for (int i = threadIdx.x; i < F.nms_strips; i += blockDim.x)
      if (ORBX_IN_ROWS(b.bounds, kSiteFrameState, i, F.nms_strips)) F.nms_status[i] = 0ull;
    if (threadIdx.x == 0) {
      *F.count = 0;
      if (F.total) *F.total = 0;
    }
  }
  if (t == 0 && threadIdx.x == 0) *b.nms_ticket = 0u;
  const int o = g.o, oh = F.oh[o];
  PyrSrc src;
  src.rec = b.bounds;
  src.ow = F.ow[o];
  if (F.pyr_src) {
    src.base = F.pyr_src + F.ooff[o];
    src.pitch = F.op[o];
    src.sh = 0;
    src.span = Span{F.pyr_src, F.ooff[F.n_oct]};
  } else {
    src.base = F.img;
    src.pitch = (long long)F.pitch_in << o;
    src.sh = o;
    src.span = img_span(F);
  }
  const bool aligned = ((reinterpret_cast<uintptr_t>(src.base) | (uintptr_t)src.pitch) & ((4u << src.sh) - 1u)) == 0;
  const int kind = src.sh <= 2 && aligned ? src.sh : kPyrBytes;
  const bool copy_pad = F.pyr_src || (o == 0 && F.pitch_in == F.op[0]);
  const bool full = g.x0 + kPyrTW <= src.ow;
  const bool inside = g.x0 > 0 && g.x0 + kPyrTW + 4 <= src.ow;

  float2 k[4];
#pragma unroll
  for (int i = 0; i < 4; i++) k[i] = pair2(b.gauss[i]);
  // rows: thread (row, gc) filters columns 8 gc .. 8 gc + 7 of both halves
  {
    const float2 m23 = pair2(-8388608.0f);
    const int gc = threadIdx.x & 7;
    const int xl = g.x0 + 8 * gc, xr = xl + kHalf;
#pragma unroll 1
    for (int r = threadIdx.x >> 3; r < TH + 6; r += 32) {
      const int yy = g.y0 - 3 + r;
      if (yy >= oh + 3) break;  // rows below the octave's halo reach no output
      const uint8_t* row = src.base + reflect101(yy, oh) * src.pitch;
      uint32_t wl[4], wr[4];  // columns x - 4 .. x + 11
      int x = xl;
      asm volatile("" : "+r"(x));  // offsets and selectors formed per row: kept across rows they would spill
      switch (kind) {
        case kPyrWord: pyr_words<PL, kPyrWord>(src, row, x, inside, wl, wr); break;
        case kPyrEvery2: pyr_words<PL, kPyrEvery2>(src, row, x, inside, wl, wr); break;
        case kPyrEvery4: pyr_words<PL, kPyrEvery4>(src, row, x, inside, wl, wr); break;
        default: pyr_words<PL, kPyrBytes>(src, row, x, inside, wl, wr);
      }
      if (r >= 3 && r < TH + 3 && yy < oh) {
        uint32_t c[4] = {wl[1], wl[2], wr[1], wr[2]};
        if (!full) {
#pragma unroll
          for (int i = 0; i < 4; i++)
            c[i] = pyr_padded<PL>(src, copy_pad, (i < 2 ? xl : xr) + 4 * (i & 1), yy, c[i]);
        }
        uint8_t* q = F.pyr + F.ooff[o] + (long long)yy * F.op[o] + xl;
        if (ORBX_IN(b.bounds, kSitePyrStore, octave_span(F.pyr, F, o), q, kHalf + 8)) {
          *reinterpret_cast<uint2*>(q) = make_uint2(c[0], c[1]);
          *reinterpret_cast<uint2*>(q + kHalf) = make_uint2(c[2], c[3]);
        }
      }
      // pair j: column x - 3 + j of both halves as floats (2^23 + byte, minus
      // 2^23); integer tap sums are exact in float, so they are summed as floats
      float2 p[14];
#pragma unroll
      for (int j = 0; j < 14; j++) {
        const uint32_t sel = 0x7540u + ((j + 1) & 3);
        p[j] = __fadd2_rn(make_float2(byte_bits(wl[(j + 1) >> 2], sel), byte_bits(wr[(j + 1) >> 2], sel)), m23);
      }
      float4* out = sm.row + r * kPyrRowSlots;
#pragma unroll
      for (int m = 0; m < 4; m++) {
        float2 q[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          const int j = 2 * m + e;
          q[e] = gauss_dot4x2(k, p[j + 3], __fadd2_rn(p[j + 2], p[j + 4]), __fadd2_rn(p[j + 1], p[j + 5]),
                              __fadd2_rn(p[j], p[j + 6]));
        }
        out[pyr_slot(gc, m)] = make_float4(q[0].x, q[0].y, q[1].x, q[1].y);
      }
    }
  }
  __syncthreads();

  // columns: thread (run, cg) filters rows 4 run .. 4 run + 3 of column pairs
  // 4 cg .. 4 cg + 3
  const int cg = threadIdx.x & 15;
  const int s0 = pyr_slot(cg >> 1, 2 * (cg & 1)), s1 = pyr_slot(cg >> 1, 2 * (cg & 1) + 1);
  const int xl = g.x0 + 4 * cg, xr = xl + kHalf;
  // rounded to the nearest integer, ties to even, by adding 1.5 * 2^23: the
  // result's low byte is the blurred pixel (0 <= v <= 255)
  const float2 rne = pair2(12582912.0f);
#pragma unroll 1
  for (int r0 = 4 * (threadIdx.x >> 4); r0 < TH; r0 += 64) {
    if (g.y0 + r0 >= oh) break;
    uint32_t ul[4] = {}, ur[4] = {};  // four blurred columns of each row, per half
#pragma unroll 1
    for (int c = 0; c < 2; c++) {  // two column pairs at a time: 40 registers of filtered rows
      float2 h[10][2];
#pragma unroll
      for (int i = 0; i < 10; i++) {
        const float4 v = sm.row[min(r0 + i, TH + 5) * kPyrRowSlots + (c ? s1 : s0)];
        h[i][0] = make_float2(v.x, v.y);
        h[i][1] = make_float2(v.z, v.w);
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float2 v[2];
#pragma unroll
        for (int j = 0; j < 2; j++)
          v[j] = __fadd2_rn(gauss_dot4x2(k, h[i + 3][j], __fadd2_rn(h[i + 2][j], h[i + 4][j]),
                                         __fadd2_rn(h[i + 1][j], h[i + 5][j]), __fadd2_rn(h[i][j], h[i + 6][j])),
                            rne);
        const uint32_t l = __byte_perm(__float_as_uint(v[0].x), __float_as_uint(v[1].x), 0x0040);
        const uint32_t r = __byte_perm(__float_as_uint(v[0].y), __float_as_uint(v[1].y), 0x0040);
        ul[i] = __byte_perm(ul[i], l, 0x5432);
        ur[i] = __byte_perm(ur[i], r, 0x5432);
      }
    }
    uint8_t* q = F.blr + F.ooff[o] + (long long)(g.y0 + r0) * F.op[o] + xl;
#pragma unroll
    for (int i = 0; i < 4; i++, q += F.op[o]) {
      const int y = g.y0 + r0 + i;
      if (r0 + i >= TH || y >= oh) break;
      if (!full) {
        ul[i] = pyr_padded<PL>(src, copy_pad, xl, y, ul[i]);
        ur[i] = pyr_padded<PL>(src, copy_pad, xr, y, ur[i]);
      }
      if (!ORBX_IN(b.bounds, kSitePyrStore, octave_span(F.blr, F, o), q, kHalf + 4)) continue;
      *reinterpret_cast<uint32_t*>(q) = ul[i];
      *reinterpret_cast<uint32_t*>(q + kHalf) = ur[i];
    }
  }
}

// ---------------------------------------------------------------------------
// FAST-9 + score -> level-0 keyed score map
//
// gCalcExtramaMap (orbd.cu:672-756) run for octaves 0..n-1 in order
// (orbd.cu:1616-1634): a pixel is a corner when 9 contiguous ring pixels are
// all darker than v - t or all brighter than v + t (the reference's LUT pre-test
// and arc loop decide exactly this).  Its score lands at level-0 position
// (x << o, y << o) if strictly greater than what a lower octave put there.
// One block owns a kDetTW x kDetTH level-0 tile and all octave pixels that map
// into it; it stages each octave's pixels with a 4-pixel halo (the Harris
// window with its Sobel reach) in shared memory using the pyramid's linear
// addressing, so reads past an octave edge return the same neighbouring bytes
// as in the reference, merges the octaves in shared memory, and writes the
// tile's occupancy bits densely and its scores sparsely (no clearing pass).
//
// What bounds it: instruction issue (ALU pipe 50%, issue 60% of active cycles)
// and, on one frame, the latency of its five phases.  Staging is one 16-byte load
// per thread for octave 0 and one for the others together; the pre-test compares
// two centres per instruction in 16-bit lanes; a Harris lane shares the column
// sums and differences of its three rows between its seven columns.  A
// 1920x1080 pair takes 9.44 M warp instructions (11.9 M with 4-byte staging,
// byte-compare pre-test and per-column derivatives), 24 mixed pairs 442 us (541).
// ---------------------------------------------------------------------------
constexpr int kHalo = 4;  // rows above and below, and the least columns to the sides
// The stage of octave o: rows of det_sw(o) bytes, the tile's first column
// det_left(o) bytes in.  The column halos are as wide as the widest aligned load
// that divides the tile's start: 16 bytes for octaves 0 to 2, then 8 and 4.
__host__ __device__ constexpr int det_left(int o) { return o <= 2 ? 16 : o == 3 ? 8 : 4; }
__host__ __device__ constexpr int det_sw(int o) { return (kDetTW >> o) + 2 * det_left(o); }
__host__ __device__ constexpr int det_rows(int o) { return (kDetTH >> o) + 2 * kHalo; }
__host__ __device__ constexpr int det_stage_off(int octave) {
  int s = 0;
  for (int o = 0; o < octave; o++) s += (det_sw(o) * det_rows(o) + 15) / 16 * 16;
  return s;
}
__host__ __device__ constexpr int det_stage_bytes() { return det_stage_off(kMaxOctaves); }
// The same for an octave known only at run time: stride, and offset of octave
// pixel (0, 0) of the tile.
__device__ __forceinline__ int det_sw_at(int o) {
  return o <= 2 ? (kDetTW >> o) + 32 : o == 3 ? det_sw(3) : det_sw(4);
}
__device__ __forceinline__ int det_origin_at(int o) {
  constexpr int at[kMaxOctaves] = {det_stage_off(0) + kHalo * det_sw(0) + det_left(0),
                                   det_stage_off(1) + kHalo * det_sw(1) + det_left(1),
                                   det_stage_off(2) + kHalo * det_sw(2) + det_left(2),
                                   det_stage_off(3) + kHalo * det_sw(3) + det_left(3),
                                   det_stage_off(4) + kHalo * det_sw(4) + det_left(4)};
  return o == 0 ? at[0] : o == 1 ? at[1] : o == 2 ? at[2] : o == 3 ? at[3] : at[4];
}

// The pre-test of the four centres in the aligned word at w of a staged tile
// (row stride sw bytes, a multiple of 4).
__device__ __forceinline__ uint32_t fast9_pretest_word(const uint8_t* w, int sw, uint32_t k1) {
  const uint32_t c = *reinterpret_cast<const uint32_t*>(w);
  const uint32_t cl = *reinterpret_cast<const uint32_t*>(w - 4);
  const uint32_t cr = *reinterpret_cast<const uint32_t*>(w + 4);
  const uint32_t p0 = *reinterpret_cast<const uint32_t*>(w + 3 * sw);   // ring 0: (x, y + 3)
  const uint32_t p8 = *reinterpret_cast<const uint32_t*>(w - 3 * sw);   // ring 8: (x, y - 3)
  const uint32_t p4 = __byte_perm(c, cr, 0x6543);                       // ring 4: (x + 3, y)
  const uint32_t p12 = __byte_perm(cl, c, 0x4321);                      // ring 12: (x - 3, y)
  return fast9_pretest4(c, p0, p4, p8, p12, k1);
}

__device__ __forceinline__ float corner_fast_score(const Batch& b, const uint8_t* c, int sw) {
  const int v = c[0];
  int d[25];
#pragma unroll
  for (int k = 0; k < 25; k++) d[k] = (int)(short)(v - c[ring_dy(k) * sw + ring_dx(k)]);
  return fast_score(d, b.fast_thr);
}

// Tile-level candidate lists hold (octave, row, column) of the octave tile as
// o << 11 | ly << 6 | lx; a tile has at most 2048 + 512 + 128 + 32 + 8 pixels.
constexpr int kDetMaxCand = 2728;
__device__ __forceinline__ uint16_t det_item(int o, int ly, int lx) { return (uint16_t)((o << 11) | (ly << 6) | lx); }

// Merge key of a level-0 position: the larger score wins and, between equal
// scores, the lower octave (the reference visits octaves in increasing order
// and replaces only on a strictly larger score).  Only scores > 0 are stored.
__device__ __forceinline__ unsigned long long det_key(float score, int o) {
  return ((unsigned long long)__float_as_uint(score) << 32) | (unsigned)(7 - o);
}

struct DetSmem {
  __align__(16) uint8_t stage[det_stage_bytes()];
  __align__(16) unsigned long long key[kDetTH * kDetTW];
  uint16_t cand[kDetMaxCand];
  uint16_t corner[kDetMaxCand];
  int n[2];
  uint32_t occ[kDetTH * kDetTW / 32];
  int ow[kMaxOctaves], oh[kMaxOctaves];
};

// Load i of octave O's stage of a detect tile: det_rows(O) rows of det_sw(O)
// bytes, in the pyramid's linear addressing, 16, 8 or 4 bytes per load (octave
// offsets and pitches are multiples of 128).
template <int O, bool P>
__device__ __forceinline__ void stage_octave(const Frame& F, const uint8_t* pyr, int X0, int Y0, uint8_t* s_stage, int i,
                                             BoundsRec* rec) {
  constexpr int B = det_left(O);
  constexpr int per_row = det_sw(O) / B;
  const int r = i / per_row, c = i - r * per_row;
  const uint8_t* sp =
      pyr + F.ooff[O] + (long long)((Y0 >> O) - kHalo + r) * F.op[O] + ((X0 >> O) - det_left(O) + B * c);
  uint8_t* dp = s_stage + det_stage_off(O) + r * det_sw(O) + B * c;
  const bool in = ORBX_IN(rec, kSiteDetLoad, guarded_span(pyr, F), sp, B);
  if constexpr (B == 16)
    *reinterpret_cast<uint4*>(dp) = in ? ldx<P>(reinterpret_cast<const uint4*>(sp)) : uint4{};
  else if constexpr (B == 8)
    *reinterpret_cast<uint2*>(dp) = in ? ldx<P>(reinterpret_cast<const uint2*>(sp)) : uint2{};
  else
    *reinterpret_cast<uint32_t*>(dp) = in ? ldx<P>(reinterpret_cast<const uint32_t*>(sp)) : 0u;
}
template <int O>
__host__ __device__ constexpr int det_loads() { return det_rows(O) * (det_sw(O) / det_left(O)); }

// Pre-test of word w (four centres) of octave O of a detect tile: octave O
// has (32 >> O) rows of (16 >> O) words.  A warp takes rows r and r + 2 of octave
// 0, whose words are in distinct banks.  Centres that pass are appended to the
// tile's candidate list.
template <int O>
__device__ __forceinline__ void pretest_word(int w, int X0, int Y0, const uint8_t* s_stage, int ow, int oh,
                                             uint32_t k1, int* s_n, uint16_t* s_cand) {
  static_assert(kDetTW == 64 && kDetTH == 32, "word layout assumes 64 x 32 detect tiles");
  constexpr int nwl = 4 - O;  // log2 words per row
  constexpr int sw = det_sw(O);
  constexpr int origin = det_stage_off(O) + kHalo * sw + det_left(O);
  int ly = w >> nwl;
  if constexpr (O == 0) ly = (ly & ~3) | ((ly & 1) << 1) | ((ly >> 1) & 1);
  const int lx = (w & ((1 << nwl) - 1)) << 2;
  const int x = (X0 >> O) + lx, y = (Y0 >> O) + ly;
  uint32_t m = 0u;
  if (y >= 3 && y < oh - 3 && x < ow - 3) {
    m = fast9_pretest_word(s_stage + origin + ly * sw + lx, sw, k1);
    if (x < 3 || x + 3 >= ow - 3) {  // border word: keep the centres with 3 <= x + k < ow - 3
      uint32_t vm = 0u;
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (x + k >= 3 && x + k < ow - 3) vm |= 0xFFu << (8 * k);
      m &= vm;
    }
  }
  if (m) {
    int pos = atomicAdd(&s_n[0], __popc(m));
    while (m) {
      const int k = (__ffs(m) >> 3) - 1;
      m &= m - 1u;
      s_cand[pos++] = det_item(O, ly, lx + k);
    }
  }
}

// One detect tile (tile index t over the batch).  P: the raw pyramid was
// written earlier in the same launch (coherent loads instead of the read-only path).
template <bool P, bool INL = false>
__device__ __forceinline__ void det_tile(const Batch& b, int t, DetSmem& sm) {
  uint8_t* s_stage = sm.stage;
  unsigned long long* s_key = sm.key;
  uint16_t* s_cand = sm.cand;
  uint16_t* s_corner = sm.corner;
  int* s_n = sm.n;
  uint32_t* s_occ = sm.occ;
  int* s_ow = sm.ow;
  int* s_oh = sm.oh;
  const int* base = INL ? b.inl_det_base : b.det_base;
  const int f = find_frame_in<INL>(base, b.n_frames, t);
  const Frame& F = batch_frame<INL>(b, f);
  const int lt = t - (INL ? base[f] : __ldg(base + f));
  const int X0 = (lt % F.det_tiles_x) * kDetTW;
  const int Y0 = (lt / F.det_tiles_x) * kDetTH;
  const int n_oct = F.n_oct;
  const uint8_t* pyr = F.pyr;
  const int warp = threadIdx.x >> 5;
  const int thr = b.fast_thr;

  for (int i = threadIdx.x; i < kDetTH * kDetTW / 2; i += blockDim.x)
    reinterpret_cast<ulonglong2*>(s_key)[i] = make_ulonglong2(0ull, 0ull);
  if (threadIdx.x < kDetTH * kDetTW / 32) s_occ[threadIdx.x] = 0u;
  if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
  if (threadIdx.x < kMaxOctaves) {
    s_ow[threadIdx.x] = threadIdx.x < n_oct ? F.ow[threadIdx.x] : 0;
    s_oh[threadIdx.x] = threadIdx.x < n_oct ? F.oh[threadIdx.x] : 0;
  }
  // stage every octave's tile with its halo: one load per thread for octave 0,
  // one for the other octaves together
  {
    const int t = threadIdx.x;
    constexpr int n1 = det_loads<1>(), n2 = n1 + det_loads<2>(), n3 = n2 + det_loads<3>(), n4 = n3 + det_loads<4>();
    static_assert(det_loads<0>() <= 256 && n4 <= 256, "two staging loads per thread");
    if (t < det_loads<0>()) stage_octave<0, P>(F, pyr, X0, Y0, s_stage, t, b.bounds);
    if (t < n1) {
      if (n_oct > 1) stage_octave<1, P>(F, pyr, X0, Y0, s_stage, t, b.bounds);
    } else if (t < n2) {
      if (n_oct > 2) stage_octave<2, P>(F, pyr, X0, Y0, s_stage, t - n1, b.bounds);
    } else if (t < n3) {
      if (n_oct > 3) stage_octave<3, P>(F, pyr, X0, Y0, s_stage, t - n2, b.bounds);
    } else if (t < n4) {
      if (n_oct > 4) stage_octave<4, P>(F, pyr, X0, Y0, s_stage, t - n3, b.bounds);
    }
  }
  __syncthreads();

  // 1. cardinal pre-test, four centres per word: the 512 words of octave 0 take
  //    two passes of the block, the 128 + 32 + 8 + 2 words of octaves 1..4 one
  {
    const uint32_t k1 = (0x7FFFu - (uint32_t)min(max(thr, 0), 255)) * 0x00010001u;
    const int t = threadIdx.x;
    pretest_word<0>(t, X0, Y0, s_stage, s_ow[0], s_oh[0], k1, s_n, s_cand);
    pretest_word<0>(t + 256, X0, Y0, s_stage, s_ow[0], s_oh[0], k1, s_n, s_cand);
    if (t < 128) {
      if (n_oct > 1) pretest_word<1>(t, X0, Y0, s_stage, s_ow[1], s_oh[1], k1, s_n, s_cand);
    } else if (t < 160) {
      if (n_oct > 2) pretest_word<2>(t - 128, X0, Y0, s_stage, s_ow[2], s_oh[2], k1, s_n, s_cand);
    } else if (t < 168) {
      if (n_oct > 3) pretest_word<3>(t - 160, X0, Y0, s_stage, s_ow[3], s_oh[3], k1, s_n, s_cand);
    } else if (t < 170) {
      if (n_oct > 4) pretest_word<4>(t - 168, X0, Y0, s_stage, s_ow[4], s_oh[4], k1, s_n, s_cand);
    }
  }
  __syncthreads();

  // 2. full 9-arc segment test of the candidates
  {
    const int n1 = s_n[0];
    for (int j = threadIdx.x; j < n1; j += blockDim.x) {
      const int e = s_cand[j];
      const int o = e >> 11, ly = (e >> 6) & 31, lx = e & 63;
      const int sw = det_sw_at(o);
      const uint8_t* c = s_stage + det_origin_at(o) + ly * sw + lx;
      const int v = c[0];
      if (fast9_full(c, sw, v - thr, v + thr)) s_corner[atomicAdd(&s_n[1], 1)] = (uint16_t)e;
    }
  }
  __syncthreads();

  // 3. scores of the corners, merged into the level-0 map
  {
    const int n2 = s_n[1];
    if (b.harris) {
      // 32 groups of 8 lanes, one corner per group; lanes 0..6 of a group take
      // one row each of the 7x7 Harris window (the 32-bit sums wrap, so their
      // order is free)
      const int gid = threadIdx.x >> 3, sub = threadIdx.x & 7;
      for (int j0 = 0; j0 < n2; j0 += 32) {
        if (j0 + 4 * warp >= n2) break;  // this warp's four groups have no corner (warp-uniform)
        const int j = j0 + gid;
        int dxx = 0, dyy = 0, dxy = 0;
        int e = 0;
        if (j < n2) {
          e = s_corner[j];
          const int o = e >> 11, ly = (e >> 6) & 31, lx = e & 63;
          const int sw = det_sw_at(o);
          const uint8_t* c = s_stage + det_origin_at(o) + ly * sw + lx;
          if (sub < 7) {  // lane `sub` of the group takes window row sub - 3, its 7 columns unrolled
            const uint8_t* r = c + (sub - 3) * sw;
            const uint8_t* ru = r - sw;
            const uint8_t* rd = r + sw;
            int s1[9], d1[9];  // column sums (1 2 1) and differences of the three rows, columns -4 .. 4
#pragma unroll
            for (int i = 0; i < 9; i++) {
              const int u = ru[i - 4], m = r[i - 4], d = rd[i - 4];
              s1[i] = u + 2 * m + d;
              d1[i] = d - u;
            }
#pragma unroll
            for (int i = 0; i < 7; i++) {
              const int dx = s1[i + 2] - s1[i];
              const int dy = d1[i] + 2 * d1[i + 1] + d1[i + 2];
              dxx += dx * dx;
              dyy += dy * dy;
              dxy += dx * dy;
            }
          }
        }
#pragma unroll
        for (int d = 4; d >= 1; d >>= 1) {
          dxx += __shfl_xor_sync(0xffffffffu, dxx, d);
          dyy += __shfl_xor_sync(0xffffffffu, dyy, d);
          dxy += __shfl_xor_sync(0xffffffffu, dxy, d);
        }
        if (j < n2 && sub == 0) {
          const int o = e >> 11, ly = (e >> 6) & 31, lx = e & 63;
          const float score = harris_combine(dxx, dyy, dxy, b.harris_scale4);
          if (score > 0.f) {
            const int m = (ly << o) * kDetTW + (lx << o);
            if (atomicMax(&s_key[m], det_key(score, o)) == 0ull) atomicOr(&s_occ[m >> 5], 1u << (m & 31));
          }
        }
      }
    } else {
      for (int j = threadIdx.x; j < n2; j += blockDim.x) {
        const int e = s_corner[j];
        const int o = e >> 11, ly = (e >> 6) & 31, lx = e & 63;
        const int sw = det_sw_at(o);
        const float score = corner_fast_score(b, s_stage + det_origin_at(o) + ly * sw + lx, sw);
        if (score > 0.f) {
          const int m = (ly << o) * kDetTW + (lx << o);
          if (atomicMax(&s_key[m], det_key(score, o)) == 0ull) atomicOr(&s_occ[m >> 5], 1u << (m & 31));
        }
      }
    }
  }
  __syncthreads();

  // Output: the tile's occupancy words (every word written, so no clearing
  // pass), then score and octave only where a bit is set.  The tile's 64
  // columns are two aligned 32-bit words of each row (pitch0 is a multiple of 128).
  if (threadIdx.x < kDetTH * kDetTW / 32) {
    const int r = threadIdx.x >> 1, half = threadIdx.x & 1;
    const int Y = Y0 + r;
    if (Y < F.h) {
      uint32_t m = s_occ[threadIdx.x];
      const size_t a0 = (size_t)Y * F.op[0] + X0 + 32 * half;
      if (ORBX_IN_ROWS(b.bounds, kSiteDetStore, (long long)(a0 >> 5), map_px(F) >> 5)) F.occ[a0 >> 5] = m;
      while (m) {
        const int k = __ffs(m) - 1;
        m &= m - 1u;
        const unsigned long long key = s_key[r * kDetTW + 32 * half + k];
        if (!ORBX_IN_ROWS(b.bounds, kSiteDetStore, (long long)(a0 + k), map_px(F))) continue;
        F.vmap[a0 + k] = __uint_as_float((uint32_t)(key >> 32));
        F.oct8[a0 + k] = (uint8_t)(7 - (int)(key & 0xFFu));
      }
    }
  }
}

// ---------------------------------------------------------------------------
// NMS + ordered compaction
//
// gNmsUnroll4 (orbd.cu:919-983): a level-0 position with score v > 0 from
// octave o survives unless a neighbour in the square of radius 2^o has a larger
// score, or an equal one at dx <= 0 && dy <= 0.  The reference appends
// survivors with atomicInc (order and, past max_pts, the kept subset depend on
// scheduling).  Here each block takes a full-width strip of F.nms_rows rows in
// ticket order, ranks its survivors with warp ballots, and chains strip totals
// with a decoupled look-back, so keypoints come out in raster order and the cap
// keeps the first max_pts of them.
// ---------------------------------------------------------------------------
constexpr unsigned long long kFlagAgg = 1ull << 32;
constexpr unsigned long long kFlagPre = 2ull << 32;
constexpr int kLookPerLane = 8;  // look-back words read per lane and round: 256 predecessors

// Warp 0 of a strip's block resolves the strip's exclusive prefix.  In each
// round lane l reads the look-back words of predecessors j - l - 32u, u = 0..7
// (each of the eight loads is 32 consecutive words, so a round touches 64
// sectors), and the warp stops at the nearest predecessor that already carries
// an inclusive prefix.  A look-back word holds its flag and its count together
// and nothing else is read on its strength, so plain relaxed loads and stores
// suffice (a release store would wait for a fence).  A published word only ever
// changes from an aggregate to an inclusive prefix of the same strip, and
// summing aggregates back to any prefix gives the same total, so words already
// seen published are kept and only the pending ones are read again, after a
// back-off that doubles from 32 ns to 256 ns: the words of a frame share a few
// L2 sectors, and a store to them completes only after the reads queued there.
// The wait is bounded by wait_cycles of clock64(); on expiry it sets
// kErrLookbackTimeout and returns the prefix found so far.
__device__ __forceinline__ int nms_lookback(unsigned long long* st, int s, int lane, int* err,
                                            long long wait_cycles) {
  int excl = 0;
  int j = s - 1;
  const long long t0 = clock64();
  while (j >= 0) {
    unsigned long long wv[kLookPerLane];
#pragma unroll
    for (int u = 0; u < kLookPerLane; u++) {
      const int idx = j - lane - 32 * u;
      wv[u] = (idx >= 0) ? ld_relaxed_u64(&st[idx]) : kFlagPre;
    }
    unsigned sleep_ns = 32;
    bool timed_out = false;
    for (;;) {
      // the nearest inclusive prefix: smallest distance lane + 32u
      int first_u = kLookPerLane, first_lane = 32;
#pragma unroll
      for (int u = kLookPerLane - 1; u >= 0; u--) {
        const unsigned pre = __ballot_sync(0xffffffffu, (wv[u] & (3ull << 32)) == kFlagPre);
        if (pre) {
          first_u = u;
          first_lane = __ffs(pre) - 1;
        }
      }
      // words up to and including that prefix must all be published
      bool notready = false;
#pragma unroll
      for (int u = 0; u < kLookPerLane; u++) {
        const bool need = u < first_u || (u == first_u && lane <= first_lane);
        if (need && (wv[u] & (3ull << 32)) == 0ull) notready = true;
      }
      if (!__any_sync(0xffffffffu, notready)) {
        int v = 0;
#pragma unroll
        for (int u = 0; u < kLookPerLane; u++) {
          const bool need = u < first_u || (u == first_u && lane <= first_lane);
          if (need) v += (int)(unsigned)wv[u];
        }
#pragma unroll
        for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        excl += v;
        j = (first_u < kLookPerLane) ? -1 : j - 32 * kLookPerLane;
        break;
      }
      if (__any_sync(0xffffffffu, clock64() - t0 > wait_cycles)) {  // warp-uniform decision
        timed_out = true;
        break;
      }
      __nanosleep(sleep_ns);
      if (sleep_ns < 256) sleep_ns <<= 1;
#pragma unroll
      for (int u = 0; u < kLookPerLane; u++) {
        const int idx = j - lane - 32 * u;
        if (idx >= 0 && (wv[u] & (3ull << 32)) == 0ull) wv[u] = ld_relaxed_u64(&st[idx]);
      }
    }
    if (timed_out) {
      if (lane == 0) atomicOr(err, kErrLookbackTimeout);
      break;
    }
  }
  return excl;
}

// Neighbour rule of gNmsUnroll4 (orbd.cu:938-956) for the centre at linear
// index idx (score v, octave o), checked by a group of kNmsGroup lanes: lane
// `sub` of the group takes window rows dy = sub - r, sub + kNmsGroup - r, ...;
// each row is at most two occupancy words, and scores are read only where a
// bit is set.  Returns whether this lane's rows hold a suppressing position.
// Positions are linear like the reference's (a column past the edge is the
// adjacent row's entry); positions outside the map, reachable only with an
// edge threshold below 2^o, are empty.  Occ(wi) gives occupancy word wi and
// Score(wi, word, bit) the score of a set bit.
constexpr int kNmsGroup = 8;
constexpr int kNmsChunkWords = 128;  // occupancy words compacted per round: at most 4096 centres

template <class Occ, class Score>
__device__ __forceinline__ bool nms_window_suppressed(long long idx, float v, int o, int p0, long long npx, int sub,
                                                      Occ occ, Score score) {
  const int r = 1 << o;
  for (int dyi = sub; dyi <= 2 * r; dyi += kNmsGroup) {
    const int dy = dyi - r;
    const long long rc = idx + (long long)dy * p0;
    long long lo = rc - r, hi = rc + r;
    if (hi < 0 || lo >= npx) continue;
    if (lo < 0) lo = 0;
    if (hi >= npx) hi = npx - 1;
    for (long long wi = lo >> 5; wi <= (hi >> 5); wi++) {
      const long long base = wi << 5;
      const uint32_t word = occ(wi);
      uint32_t m = word;
      if (base < lo) m &= ~0u << (int)(lo - base);
      if (hi - base < 31) m &= (2u << (int)(hi - base)) - 1u;
      while (m) {
        const int bb = __ffs(m) - 1;
        m &= m - 1u;
        const long long li = base + bb;
        if (li == idx) continue;
        const int dx = (int)(li - rc);
        const float u = score(wi, word, bb);
        if (u > v || (u == v && dx <= 0 && dy <= 0)) return true;
      }
    }
  }
  return false;
}

// Staged form of a strip (kNmsStageWords occupancy words: the strip's rows with
// a halo of R + 1 rows on each side; kNmsStageBits set bits with their scores
// and octaves gathered next to them).
constexpr int kNmsStageWords = 2048;
constexpr int kNmsStageBits = 2048;

struct NmsSmem {
  uint32_t sur[kNmsMaxWords];
  int pref[kNmsMaxWords];
  union {
    struct {  // rounds over the maps in global memory
      uint16_t cand[kNmsChunkWords * 32];
      float cv[kNmsChunkWords * 32];
      uint8_t co[kNmsChunkWords * 32];
    } g;
    struct {  // staged strip
      uint32_t occ[kNmsStageWords];
      float score[kNmsStageBits];
      uint16_t pfx[kNmsStageWords + 1];  // set bits before each staged word
      uint16_t idx[kNmsStageBits];       // bit offset of each set bit from the first staged word
      uint8_t oct[kNmsStageBits];
    } w;
  } u;
  int ncand[2];
  int warp_tot[8];
  int base;
};

// Exclusive scan over the block (256 threads) of one count per thread; *total
// gets the sum.  Every thread must call it.
__device__ __forceinline__ int block_scan_excl(int local, int* s_warp_tot, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = local;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int n = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += n;
  }
  if (lane == 31) s_warp_tot[warp] = incl;
  __syncthreads();
  int warp_off = 0, tot = 0;
#pragma unroll
  for (int w2 = 0; w2 < 8; w2++) {
    const int t = s_warp_tot[w2];
    if (w2 < warp) warp_off += t;
    tot += t;
  }
  __syncthreads();
  total = tot;
  return warp_off + incl - local;
}

// One NMS strip; `ticket` is the strip's index over the batch, and strips must
// start in ticket order (the look-back waits only on smaller tickets).  P: the
// score map was written earlier in the same launch.
template <bool P, bool INL = false>
__device__ __forceinline__ void nms_strip(const Batch& b, int ticket, NmsSmem& sm) {
  uint32_t* s_sur = sm.sur;
  int* s_pref = sm.pref;
  int* s_ncand = sm.ncand;
  int* s_warp_tot = sm.warp_tot;
  int& s_base = sm.base;
  const int* strip_base = INL ? b.inl_nms_base : b.nms_base;
  const int f = find_frame_in<INL>(strip_base, b.n_frames, ticket);
  const Frame& F = batch_frame<INL>(b, f);
  const int s = ticket - (INL ? strip_base[f] : __ldg(strip_base + f));
  const int border = F.border;
  const int row0 = border + s * F.nms_rows;
  const int row1 = min(row0 + F.nms_rows, F.h - border);
  const int xlo = border, xhi = F.w - border;  // columns [xlo, xhi)
  const int wlo = xlo >> 5, whi = (xhi - 1) >> 5;
  const int nw = whi - wlo + 1;
  const int nwords = (row1 - row0) * nw;
  const int p0 = F.op[0];  // a multiple of 128
  const int wpr = p0 >> 5;  // occupancy words per row
  const long long npx = (long long)F.h * p0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gid = warp * (32 / kNmsGroup) + (lane / kNmsGroup), sub = lane % kNmsGroup;
  const uint32_t gmask = ((1u << kNmsGroup) - 1u) << (lane & ~(kNmsGroup - 1));
  const uint32_t* occ_map = F.occ;
  const float* score_map = F.vmap;
  [[maybe_unused]] BoundsRec* rec = b.bounds;
  auto g_occ = [=](long long wi) {
    return ORBX_IN_ROWS(rec, kSiteNmsOcc, wi, npx >> 5) ? ldx<P>(occ_map + wi) : 0u;
  };
  auto g_score = [=](long long wi, uint32_t, int bb) {
    return ORBX_IN_ROWS(rec, kSiteNmsScore, (wi << 5) + bb, npx) ? ldx<P>(score_map + ((wi << 5) + bb)) : 0.f;
  };

  for (int k = threadIdx.x; k < nwords; k += blockDim.x) s_sur[k] = 0u;

  // Staged pass 1.  The halo R is the largest window radius present (2^(n_oct-1)),
  // halved until the strip fits the staging buffer; centres of octaves with a
  // larger radius read their windows from global memory.
  int R = 1 << (F.n_oct - 1);
  while (R >= 1 && (min(F.h, row1 + R + 1) - max(0, row0 - R - 1)) * wpr > kNmsStageWords) R >>= 1;
  const int srow0 = max(0, row0 - R - 1), srow1 = min(F.h, row1 + R + 1);
  const int ns = (srow1 - srow0) * wpr;
  const long long W0 = (long long)srow0 * wpr;  // first staged word
  bool staged = R >= 1;
  uint32_t* s_occ = sm.u.w.occ;
  uint16_t* s_pfx = sm.u.w.pfx;
  uint16_t* s_idx = sm.u.w.idx;
  float* s_score = sm.u.w.score;
  uint8_t* s_oct = sm.u.w.oct;
  // a staged word, or the global one for a word outside the stage (not reached
  // for radii up to R; kept so that no index leaves the buffers)
  auto w_occ = [=](long long wi) {
    const long long sw = wi - W0;
    return (sw >= 0 && sw < ns) ? s_occ[sw] : g_occ(wi);
  };
  auto w_score = [=](long long wi, uint32_t word, int bb) {
    const long long sw = wi - W0;
    return (sw >= 0 && sw < ns) ? s_score[s_pfx[sw] + __popc(word & ((1u << bb) - 1u))]
                                : g_score(wi, word, bb);
  };
  if (staged) {
    for (int i = threadIdx.x; i < ns; i += blockDim.x) s_occ[i] = g_occ(W0 + i);
    __syncthreads();
    // set bits before each word (contiguous runs of words per thread), and the
    // list of set bits in raster order
    const int per = (ns + 255) >> 8;
    const int beg = min((int)threadIdx.x * per, ns), end = min(beg + per, ns);
    int local = 0;
    for (int i = beg; i < end; i++) local += __popc(s_occ[i]);
    int total;
    int run = block_scan_excl(local, s_warp_tot, total);
    if (total <= kNmsStageBits) {
      for (int i = beg; i < end; i++) {
        s_pfx[i] = (uint16_t)run;
        uint32_t m = s_occ[i];
        while (m) {
          const int bb = __ffs(m) - 1;
          m &= m - 1u;
          s_idx[run++] = (uint16_t)((i << 5) | bb);
        }
      }
      if (threadIdx.x == 0) s_pfx[ns] = (uint16_t)total;
      __syncthreads();
      // scores and octaves of the set bits, four loads in flight per thread
      for (int r0 = threadIdx.x; r0 < total; r0 += 4 * blockDim.x) {
        long long li[4];
        bool ok[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int r = r0 + q * blockDim.x;
          ok[q] = r < total;
          li[q] = (W0 << 5) + (ok[q] ? s_idx[r] : 0);
        }
        float v[4];
        uint8_t o[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const bool in = ok[q] && ORBX_IN_ROWS(rec, kSiteNmsScore, li[q], npx);
          v[q] = in ? ldx<P>(F.vmap + li[q]) : 0.f;
          o[q] = in ? ldx<P>(F.oct8 + li[q]) : (uint8_t)0;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) {
          if (ok[q]) {
            s_score[r0 + q * blockDim.x] = v[q];
            s_oct[r0 + q * blockDim.x] = o[q];
          }
        }
      }
      __syncthreads();
      // the centres are the set bits of the strip's own rows (ranks c_lo ..
      // c_hi - 1) in columns [xlo, xhi), checked by 32 groups of 8 lanes
      const int c_lo = s_pfx[(row0 - srow0) * wpr], c_hi = s_pfx[(row1 - srow0) * wpr];
      for (int j0 = c_lo; j0 < c_hi; j0 += 32 * 8 / kNmsGroup) {
        const int j = j0 + gid;
        bool sup = false;
        int kk = -1, bit = 0;
        if (j < c_hi) {
          const int rel = s_idx[j];
          const int rr = rel / p0, c = rel - rr * p0;
          if (c >= xlo && c < xhi) {
            const int row = srow0 + rr;
            const long long idx = (long long)row * p0 + c;
            const int o = s_oct[j];
            sup = (1 << o) <= R ? nms_window_suppressed(idx, s_score[j], o, p0, npx, sub, w_occ, w_score)
                                : nms_window_suppressed(idx, s_score[j], o, p0, npx, sub, g_occ, g_score);
            kk = (row - row0) * nw + ((c >> 5) - wlo);
            bit = c & 31;
          }
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, sup);
        if (kk >= 0 && sub == 0 && !(bal & gmask)) atomicOr(&s_sur[kk], 1u << bit);
      }
    } else {
      staged = false;
    }
  }

  if (!staged) {
    // pass 1 over global memory, in rounds of kNmsChunkWords words: the centres
    // of the round (with their scores) are compacted into shared memory, then
    // checked by 32 groups of 8 lanes, so a textured patch of the strip spreads
    // over every warp
    uint16_t* s_cand = sm.u.g.cand;
    float* s_cv = sm.u.g.cv;
    uint8_t* s_co = sm.u.g.co;
    if (threadIdx.x == 0) s_ncand[0] = 0;
    for (int c0 = 0, round = 0; c0 < nwords; c0 += kNmsChunkWords, round++) {
      int* cnt = &s_ncand[round & 1];
      __syncthreads();  // the previous round's checks are done; its counter is free
      if (threadIdx.x == 0) s_ncand[(round + 1) & 1] = 0;
      const int k = c0 + (int)threadIdx.x;
      if (threadIdx.x < kNmsChunkWords && k < nwords) {
        const int row = row0 + k / nw;
        const int wj = wlo + k % nw;
        const int cbase = wj << 5;
        uint32_t m = g_occ((long long)row * wpr + wj);
        if (cbase < xlo) m &= ~0u << (xlo - cbase);
        if (xhi - cbase < 32) m &= (xhi - cbase <= 0) ? 0u : ((xhi - cbase == 32) ? ~0u : ((1u << (xhi - cbase)) - 1u));
        if (m) {
          int pos = atomicAdd(cnt, __popc(m));
          while (m) {
            const int bit = __ffs(m) - 1;
            m &= m - 1u;
            const long long idx = (long long)row * p0 + cbase + bit;
            s_cand[pos] = (uint16_t)(((k - c0) << 5) | bit);
            const bool in = ORBX_IN_ROWS(rec, kSiteNmsScore, idx, npx);
            s_cv[pos] = in ? ldx<P>(F.vmap + idx) : 0.f;
            s_co[pos] = in ? ldx<P>(F.oct8 + idx) : (uint8_t)0;
            pos++;
          }
        }
      }
      __syncthreads();
      const int nc = *cnt;
      for (int j0 = 0; j0 < nc; j0 += 32 * 8 / kNmsGroup) {
        const int j = j0 + gid;
        bool sup = false;
        int kk = 0, bit = 0;
        if (j < nc) {
          const int e = s_cand[j];
          kk = c0 + (e >> 5);
          bit = e & 31;
          const int row = row0 + kk / nw;
          const int cbase = (wlo + kk % nw) << 5;
          sup = nms_window_suppressed((long long)row * p0 + cbase + bit, s_cv[j], s_co[j], p0, npx, sub, g_occ,
                                      g_score);
        }
        const uint32_t bal = __ballot_sync(0xffffffffu, sup);
        if (j < nc && sub == 0 && !(bal & gmask)) atomicOr(&s_sur[kk], 1u << bit);
      }
    }
  }
  __syncthreads();

  // exclusive scan of the survivor counts, in word order
  const int per = (nwords + 255) >> 8;
  const int beg = min((int)threadIdx.x * per, nwords), end = min(beg + per, nwords);
  int local = 0;
  for (int i = beg; i < end; i++) local += __popc(s_sur[i]);
  int strip_total;
  int run = block_scan_excl(local, s_warp_tot, strip_total);
  for (int i = beg; i < end; i++) {
    s_pref[i] = run;
    run += __popc(s_sur[i]);
  }

  // decoupled look-back over the frame's strips (warp 0)
  if (warp == 0 && ORBX_IN_ROWS(rec, kSiteFrameState, s, F.nms_strips)) {
    unsigned long long* st = F.nms_status;
    int excl = 0;
    if (s == 0) {
      if (lane == 0) st_relaxed_u64(&st[0], kFlagPre | (unsigned)strip_total);
    } else {
      if (lane == 0) st_relaxed_u64(&st[s], kFlagAgg | (unsigned)strip_total);
      __syncwarp();
      excl = nms_lookback(st, s, lane, b.err, b.wait_cycles);
      if (lane == 0) st_relaxed_u64(&st[s], kFlagPre | (unsigned)(excl + strip_total));
    }
    if (lane == 0) {
      s_base = excl;
      if (s == F.nms_strips - 1) {
        const int tot = excl + strip_total;
        *F.count = min(tot, F.max_pts);
        if (F.total) *F.total = tot;
      }
    }
  }
  __syncthreads();
  const int base = s_base;
  if (base >= F.max_pts) return;

  // pass 2: write the survivors (score and octave from the stage when staged)
  for (int k = threadIdx.x; k < nwords; k += blockDim.x) {
    uint32_t m = s_sur[k];
    if (!m) continue;
    const int row = row0 + k / nw;
    const int cbase = (wlo + k % nw) << 5;
    const long long wi = ((long long)row * p0 + cbase) >> 5;
    int rank = base + s_pref[k];
    while (m) {
      const int bit = __ffs(m) - 1;
      m &= m - 1u;
      if (rank >= F.max_pts) break;
      const long long idx = (long long)row * p0 + cbase + bit;
      orbx_point q;
      q.x = cbase + bit;
      q.y = row;
      if (staged) {
        const int sw = (int)(wi - W0);
        const int sr = s_pfx[sw] + __popc(s_occ[sw] & ((1u << bit) - 1u));
        q.octave = s_oct[sr];
        q.score = s_score[sr];
      } else {
        const bool in = ORBX_IN_ROWS(rec, kSiteNmsScore, idx, npx);
        q.octave = in ? F.oct8[idx] : 0;
        q.score = in ? F.vmap[idx] : 0.f;
      }
      q.angle = 0.f;
      q.match = 0;
      q.distance = 0;
      if (ORBX_IN_ROWS(rec, kSiteNmsPts, rank, F.max_pts)) F.pts[rank] = q;
      rank++;
    }
  }
}

// ---------------------------------------------------------------------------
// Orientation and rBRIEF (orbx_describe.cu and the persistent kernel)
// ---------------------------------------------------------------------------
// Plain loads of data written earlier in the same launch (PL) or by earlier
// launches; PL uses the coherent cached path explicitly.
template <bool PL, class T>
__device__ __forceinline__ T ldc(const T* p) {
  if constexpr (PL)
    return __ldca(p);
  else
    return *p;
}

constexpr int kDescWarps = 8;

// getValue (orbd.cu:1341-1348): the rotated point is
// (rint(x*c - y*s), rint(x*s + y*c)), evaluated by the reference build as
// fma(x, c, -(y*s)) and fma(x, s, y*c).
template <bool PL>
__device__ __forceinline__ int sample_at(const uint8_t* center, int pitch, float x, float y, float s, float c,
                                         BoundsRec* rec, Span blr) {
  const int ix = __float2int_rn(__fmaf_rn(x, c, -__fmul_rn(y, s)));
  const int iy = __float2int_rn(__fmaf_rn(x, s, __fmul_rn(y, c)));
  const uint8_t* p = center + (ptrdiff_t)iy * pitch + ix;
  return ORBX_IN(rec, kSiteDescSample, blr, p, 1) ? ldc<PL>(p) : 0;
}

template <int WTA, bool PL>
__device__ __forceinline__ uint8_t describe_byte(const uint8_t* center, int pitch, const float* px, const float* py,
                                                 float s, float c, BoundsRec* rec, Span blr) {
#define G(j) sample_at<PL>(center, pitch, px[j], py[j], s, c, rec, blr)
  uint8_t val = 0;
  if (WTA == 2) {  // feature2 (orbd.cu:1351-1361)
#pragma unroll
    for (int j = 0; j < 8; j++) val |= (uint8_t)((G(2 * j) < G(2 * j + 1)) << j);
  } else if (WTA == 3) {  // feature3 (orbd.cu:1364-1388), including its index reuse of 8 and skip of 10
    const int idx[4][3] = {{0, 1, 2}, {3, 4, 5}, {6, 7, 8}, {8, 9, 11}};
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const int t0 = G(idx[g][0]), t1 = G(idx[g][1]), t2 = G(idx[g][2]);
      const int v = t2 > t1 ? (t2 > t0 ? 2 : 0) : (t1 > t0);
      val |= (uint8_t)(v << (2 * g));
    }
  } else {  // feature4 (orbd.cu:1391-1434)
#pragma unroll
    for (int g = 0; g < 4; g++) {
      int t0 = G(4 * g), t1 = G(4 * g + 1), t2 = G(4 * g + 2), t3 = G(4 * g + 3);
      int u = 0, v = 2;
      if (t1 > t0) t0 = t1, u = 1;
      if (t3 > t2) t2 = t3, v = 3;
      val |= (uint8_t)((t0 > t2 ? u : v) << (2 * g));
    }
  }
#undef G
  return val;
}

// This lane's pattern points of descriptor byte `lane` (setPattern,
// orbd.cu:95-410): PSTEP (x, y) int8 pairs, contiguous per lane, fetched as
// raw words (load_pattern_raw) so that the loads can be in flight with other
// work, then converted (pattern_points).
template <int WTA>
struct PatternRaw {
  static constexpr int PSTEP = (WTA == 3) ? 12 : 16;
  static constexpr int WORDS = PSTEP / 2;  // 2 * PSTEP bytes
  uint32_t w[WORDS];
};
template <int WTA>
__device__ __forceinline__ PatternRaw<WTA> load_pattern_raw(const Batch& b, int lane) {
  PatternRaw<WTA> r;
  constexpr int W = PatternRaw<WTA>::WORDS;
  // 2 * PSTEP * lane bytes in: a multiple of 8 (WTA 3) or 16, and the table is 16-byte aligned
  const uint32_t* src = reinterpret_cast<const uint32_t*>(b.pattern) + W * lane;
  if constexpr (W % 4 == 0) {
#pragma unroll
    for (int i = 0; i < W / 4; i++) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(src) + i);
      r.w[4 * i] = v.x, r.w[4 * i + 1] = v.y, r.w[4 * i + 2] = v.z, r.w[4 * i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < W / 2; i++) {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(src) + i);
      r.w[2 * i] = v.x, r.w[2 * i + 1] = v.y;
    }
  }
  return r;
}
template <int WTA>
__device__ __forceinline__ void pattern_points(const PatternRaw<WTA>& r, float* px, float* py) {
#pragma unroll
  for (int j = 0; j < PatternRaw<WTA>::PSTEP; j++) {
    const uint32_t word = r.w[j >> 1];
    const int sh = 16 * (j & 1);
    px[j] = (float)(int)(int8_t)((word >> sh) & 0xFFu);
    py[j] = (float)(int)(int8_t)((word >> (sh + 8)) & 0xFFu);
  }
}
template <int WTA>
__device__ __forceinline__ void load_pattern(const Batch& b, int lane, float* px, float* py) {
  pattern_points<WTA>(load_pattern_raw<WTA>(b, lane), px, py);
}

template <int WTA, bool PL>
__device__ __forceinline__ void describe_keypoint(const Batch& b, const Frame& F, int k, const float* px,
                                                  const float* py, const int* s_umax, int lane) {
  const int half_k = b.half_k;
  if (!ORBX_IN_ROWS(b.bounds, kSiteDescPts, k, F.max_pts)) return;
  orbx_point* P = F.pts + k;
  const int x = ldc<PL>(&P->x), y = ldc<PL>(&P->y), o = ldc<PL>(&P->octave);
  const int pitch = F.op[o];
  const long long coff = F.ooff[o] + (long long)(y >> o) * pitch + (x >> o);

  float angle;
  if (b.describe_mode != kDescribeDescOnly) {
    // intensity centroid on the raw octave: lane v + half_k owns disc row v
    // and reads it as nine aligned words at once (octave pitches are multiples
    // of 128, so every row has the same alignment); the integer sums are exact
    // in any order
    const uint8_t* center = F.pyr + coff;
    int m10 = 0, m01 = 0;
    if (lane <= 2 * half_k) {
      const int v = lane - half_k;
      const int um = s_umax[v < 0 ? -v : v];
      const uintptr_t ra = reinterpret_cast<uintptr_t>(center + (ptrdiff_t)v * pitch - half_k);  // column -half_k
      const uint32_t* wp = reinterpret_cast<const uint32_t*>(ra & ~(uintptr_t)3);
      const unsigned sh = 8u * (unsigned)(ra & 3);
      uint32_t w[9];
      const bool in = ORBX_IN(b.bounds, kSiteDescMoment, guarded_span(F.pyr, F), wp, 36);
#pragma unroll
      for (int i = 0; i < 9; i++) w[i] = in ? ldc<PL>(wp + i) : 0u;
      int sum = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t r = __funnelshift_r(w[i], w[i + 1], sh);  // columns 4i - half_k .. 4i + 3 - half_k
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int uu = 4 * i + k - half_k;
          if ((unsigned)(uu + um) <= (unsigned)(2 * um)) {  // |uu| <= um
            const int val = (int)((r >> (8 * k)) & 0xFFu);
            m10 += uu * val;
            sum += val;
          }
        }
      }
      m01 = v * sum;
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
      m10 += __shfl_xor_sync(0xffffffffu, m10, d);
      m01 += __shfl_xor_sync(0xffffffffu, m01, d);
    }
    angle = fast_atan2(__int2float_rn(m01), __int2float_rn(m10));
    if (lane == 0) P->angle = angle;
    if (b.describe_mode == kDescribeAngleOnly) return;
  } else {
    angle = ldc<PL>(&P->angle);
  }

  // rBRIEF on the blurred octave
  const float sn = __sinf(angle);
  const float cs = __cosf(angle);
  const uint8_t byte = describe_byte<WTA, PL>(F.blr + coff, pitch, px, py, sn, cs, b.bounds, guarded_span(F.blr, F));
  F.desc[(size_t)k * 32 + lane] = byte;
}

// ---------------------------------------------------------------------------
// k = 2 XOR-popcount matching (orbx_match.cu and the persistent kernel)
// ---------------------------------------------------------------------------
constexpr int kMQ = 128;      // queries per block
constexpr int kMGroups = 4;   // row groups per block of the launched matchers
constexpr int kMChunk = 512;  // train rows per shared-memory chunk (16 KB)
constexpr int kIdxBits = kIdxBitsShared;
constexpr uint32_t kNoKey = kNoKeyShared;

__device__ __forceinline__ void top2_push(uint32_t& k1, uint32_t& k2, uint32_t key) { top2_push_shared(k1, k2, key); }
__device__ __forceinline__ void finish_query(const MatchArgs& a, int q, uint32_t k1, uint32_t k2) {
  finish_query_shared(a, q, k1, k2);
}

// Hamming distance of a query (q) and a train row (t0, t1).  Four carry-save
// adders turn the eight XORed words into one word of ones, one left over, one of
// twos and one of fours, so four population counts do instead of eight: that
// unit takes 8 cycles per warp where the ALU takes 2 for each of the adders'
// eight three-input operations.
__device__ __forceinline__ uint32_t csa_carry(uint32_t a, uint32_t b, uint32_t c) { return (a & b) | (c & (a | b)); }
__device__ __forceinline__ uint32_t hamming256(const uint32_t* q, const uint4& t0, const uint4& t1) {
  const uint32_t x0 = q[0] ^ t0.x, x1 = q[1] ^ t0.y, x2 = q[2] ^ t0.z, x3 = q[3] ^ t0.w;
  const uint32_t x4 = q[4] ^ t1.x, x5 = q[5] ^ t1.y, x6 = q[6] ^ t1.z, x7 = q[7] ^ t1.w;
  const uint32_t s1 = x0 ^ x1 ^ x2, c1 = csa_carry(x0, x1, x2);
  const uint32_t s2 = x3 ^ x4 ^ x5, c2 = csa_carry(x3, x4, x5);
  const uint32_t s3 = s1 ^ s2 ^ x6, c3 = csa_carry(s1, s2, x6);
  const uint32_t twos = c1 ^ c2 ^ c3, fours = csa_carry(c1, c2, c3);
  return __popc(s3) + __popc(x7) + 2 * __popc(twos) + 4 * __popc(fours);
}

template <int RG>
struct MatchSmem {
  uint4 db[kMChunk * 2];
  uint2 part[(RG - 1) * kMQ];  // the other row groups' best two, per query
  unsigned int last;
};

// Merges the row groups' best two of each query; the threads of group 0 get them.
template <int RG>
__device__ __forceinline__ void match_merge_groups(MatchSmem<RG>& sm, int rg, int ql, uint32_t& k1, uint32_t& k2) {
  if (rg) sm.part[(rg - 1) * kMQ + ql] = make_uint2(k1, k2);
  __syncthreads();
  if (rg) return;
#pragma unroll
  for (int g = 0; g < RG - 1; g++) {
    const uint2 o = sm.part[g * kMQ + ql];
    top2_push(k1, k2, o.x);
    top2_push(k1, k2, o.y);
  }
}

// One block's share of a k = 2 search: kMQ queries, one per thread, and RG groups
// of threads with a share of the train rows each (kMQ * RG threads).  Per query
// the row groups' and the splits' results are merged as keys, so the outcome does
// not depend on how the rows are shared out.  bid / nblk replace blockIdx.x /
// gridDim.x so that a batch launch or a work item of the persistent kernel can run
// one search each.  P: the descriptors and counts were written earlier in the
// same launch.
template <int RG, bool P>
__device__ __forceinline__ void match_popc_block(const MatchArgs& a, const MatchWork& w, int bid, int nblk,
                                                 MatchSmem<RG>& sm) {
  const int ql = threadIdx.x % kMQ, rg = threadIdx.x / kMQ;
  const int nq = min(a.d_nq ? ldx<P>(a.d_nq) : a.nq, w.nq_cap);
  const int ndb = a.d_ndb ? ldx<P>(a.d_ndb) : a.ndb;
  // Spread (query tile, train split) pairs over the launched blocks using the
  // actual counts, which may be far below the capacities the grid was sized for.
  const int tiles = (nq + kMQ - 1) / kMQ;
  if (tiles == 0) return;
  int splits = nblk / tiles;
  splits = min(splits, w.splits_cap);
  splits = min(splits, max(1, (ndb + 63) / 64));
  splits = max(splits, 1);
  const int tile = bid / splits;
  const int split = bid - tile * splits;
  if (tile >= tiles) return;
  const int q = tile * kMQ + ql;
  const bool active = q < nq;

  uint32_t qw[8];
  {
    const uint4* qp = reinterpret_cast<const uint4*>(a.q) + 2 * (size_t)(active ? q : 0);
    const bool in = ORBX_IN_ROWS(a.bounds, kSiteMatchQ, active ? q : 0, a.q_cap);
    const uint4 v0 = in ? ldx<P>(qp) : uint4{}, v1 = in ? ldx<P>(qp + 1) : uint4{};
    qw[0] = v0.x; qw[1] = v0.y; qw[2] = v0.z; qw[3] = v0.w;
    qw[4] = v1.x; qw[5] = v1.y; qw[6] = v1.z; qw[7] = v1.w;
  }

  const int r_beg = (int)((long long)ndb * split / splits);
  const int r_end = (int)((long long)ndb * (split + 1) / splits);
  uint32_t k1 = kNoKey, k2 = kNoKey;
  uint32_t second = kNoKey >> kIdxBits;  // distance of k2
  const uint4* db4 = reinterpret_cast<const uint4*>(a.db);
  for (int r0 = r_beg; r0 < r_end; r0 += kMChunk) {
    const int rows = min(kMChunk, r_end - r0);
    __syncthreads();
    for (int i = threadIdx.x; i < rows * 2; i += kMQ * RG)
      sm.db[i] = ORBX_IN_ROWS(a.bounds, kSiteMatchDb, r0 + (i >> 1), a.db_cap) ? ldx<P>(db4 + 2 * (size_t)r0 + i)
                                                                              : uint4{};
    __syncthreads();
    const int j_end = rows * (rg + 1) / RG;
    int j = rows * rg / RG;
    // four rows at a time: rows come in increasing index order, so only a
    // distance below the second best can enter the top two
    for (; j + 4 <= j_end; j += 4) {
      uint32_t d[4];
#pragma unroll
      for (int i = 0; i < 4; i++) d[i] = hamming256(qw, sm.db[2 * (j + i)], sm.db[2 * (j + i) + 1]);
      if (__vimin3_u32(d[0], d[1], min(d[2], d[3])) < second) {
#pragma unroll
        for (int i = 0; i < 4; i++) top2_push(k1, k2, (d[i] << kIdxBits) | (uint32_t)(r0 + j + i));
        second = k2 >> kIdxBits;
      }
    }
    for (; j < j_end; j++)
      top2_push(k1, k2, (hamming256(qw, sm.db[2 * j], sm.db[2 * j + 1]) << kIdxBits) | (uint32_t)(r0 + j));
    second = k2 >> kIdxBits;
  }

  match_merge_groups<RG>(sm, rg, ql, k1, k2);
  if (splits == 1) {
    if (active && rg == 0) finish_query(a, q, k1, k2);
    return;
  }
  // publish this split's partial top-2; the last split to finish the tile merges
  if (active && rg == 0) {
    uint2* part = reinterpret_cast<uint2*>(w.part);
    part[(size_t)split * w.nq_cap + q] = make_uint2(k1, k2);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) sm.last = (atomicAdd(&w.tile_done[tile], 1u) == (unsigned)(splits - 1)) ? 1u : 0u;
  __syncthreads();
  if (!sm.last) return;
  __threadfence();
  if (threadIdx.x == 0) w.tile_done[tile] = 0u;  // ready for the next launch
  const uint2* part = reinterpret_cast<const uint2*>(w.part) + q;
  k1 = k2 = kNoKey;
  if (active) {
#pragma unroll 4
    for (int sp = rg; sp < splits; sp += RG) {
      const uint2 pk = __ldcg(part + (size_t)sp * w.nq_cap);
      top2_push(k1, k2, pk.x);
      top2_push(k1, k2, pk.y);
    }
  }
  match_merge_groups<RG>(sm, rg, ql, k1, k2);
  if (active && rg == 0) finish_query(a, q, k1, k2);
}

}  // namespace orbx
