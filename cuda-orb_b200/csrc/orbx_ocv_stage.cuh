// Which bytes of a level's rows the tile kernel of the OpenCV-compatible mode reads
// (orbx_ocv.cu): plain arithmetic, the same on the host.
#pragma once

namespace orbx {

// Of the 16 bytes from column x (a multiple of 16) of row y of a w x h level, how many
// are read.  Level 0 may be the caller's image, of which only the pixels are known to
// be there: it may be a view that ends with its allocation.
__host__ __device__ inline int ocv_stage_bytes(int x, int y, int w, int h) {
  if (x < 0 || x >= w || y < 0 || y >= h) return 0;
  return x + 16 <= w ? 16 : w - x;
}

}  // namespace orbx
