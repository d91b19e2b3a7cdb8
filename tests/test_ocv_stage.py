"""The bytes that the tile kernel of the OpenCV-compatible mode reads of an image, on
the CPU: every pixel the tiles need, and none past the image's last pixel."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-orb_b200", "csrc")
SOURCE = r"""
#define __host__
#define __device__
#include "orbx_ocv_stage.cuh"
#include <cstdio>
#include <vector>
using namespace orbx;
// tiles of 64 x 26, staged with 16 columns and 4 rows around them
static int check(int w, int h, int pitch) {
  const long long end = (long long)(h - 1) * pitch + w;  // one past the last pixel
  std::vector<char> seen((size_t)end, 0);
  for (int y0 = 0; y0 < h; y0 += 26)
    for (int x0 = 0; x0 < w; x0 += 64)
      for (int r = 0; r < 34; r++)
        for (int c = 0; c < 6; c++) {
          const int x = x0 - 16 + 16 * c;
          int y = y0 - 4 + r;
          if (y < 0) y = -y;
          if (y >= h) y = 2 * h - 2 - y;
          y = y < 0 ? 0 : y >= h ? h - 1 : y;
          const int n = ocv_stage_bytes(x, y, w, h);
          if (n < 0 || n > 16) return 1;
          if (n && (x < 0 || (long long)y * pitch + x + n > end)) return 2;
          for (int i = 0; i < n; i++) seen[(size_t)y * pitch + x + i] = 1;
          for (int i = n; i < 16; i++)
            if (x + i >= 0 && x + i < w) return 3;
        }
  for (int y = 0; y < h; y++)
    for (int x = 0; x < w; x++)
      if (!seen[(size_t)y * pitch + x]) return 4;
  return 0;
}
int main() {
  for (int w : {16, 17, 31, 32, 63, 64, 65, 79, 80, 81, 127, 128, 129, 311, 320, 960})
    for (int h : {16, 25, 26, 27, 53, 131})
      for (int more : {0, 16, 64, 960}) {
        const int pitch = (w + 15) / 16 * 16 + more;
        const int bad = check(w, h, pitch);
        if (bad) { printf("%d: w %d h %d pitch %d\n", bad, w, h, pitch); return 1; }
      }
  return 0;
}
"""


def test_reads_end_with_the_image(tmp_path):
    src, exe = tmp_path / "stage.cpp", tmp_path / "stage"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-x", "c++", "-I", CSRC, str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
