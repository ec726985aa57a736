/*
 * Host check of the line passes' index arithmetic
 * (itk-rs_gb300/csrc/line_window.hpp, the header that conv_lines.cu compiles):
 * for every small geometry of an axis -- image, request inside it, radius,
 * warps per block -- every position that the passes along y / z and along x
 * load lies inside the smallest source that holds the request's taps, and
 * every requested output takes its taps from the positions that clamp-to-edge
 * names.
 * Build: g++ -std=c++17 -O2 -I itk-rs_gb300/csrc line_window.cpp
 */
#include <algorithm>
#include <cstdio>

#include "line_window.hpp"

using namespace itkg;

static long outside = 0, wrong = 0, geometries = 0;

static void check(int64_t lo, int64_t hi, int64_t at, int64_t n, int R) {
  ++geometries;
  // the source: what the requested outputs reach, clipped to the image
  const int64_t s0 = std::max(lo, at - R) - lo, s1 = std::min(hi, at + n - 1 + R) - lo;
  auto in = [&](int64_t p) { if (p < s0 || p > s1) ++outside; };
  auto tap = [&](int64_t o, int k) { return std::min(std::max(o + k - R, lo), hi) - lo; };
  const int64_t runs = (n + kLineRun - 1) / kLineRun;
  // along y and z: a run per thread, the pointer stepped from entry to entry
  for (int64_t run = 0; run < runs; ++run) {
    const int64_t o0 = at + run * kLineRun;
    const int nv = (int)std::min<int64_t>(kLineRun, n - run * kLineRun);
    const LineWindow w = line_window(o0, nv, R, lo, hi);
    int64_t p = line_at(w, 0);
    for (int j = 0; j < 2 * R + kLineRun; ++j) {
      in(p);
      if (p != line_at(w, j)) ++wrong;
      for (int m = std::max(0, j - 2 * R); m <= std::min(nv - 1, j); ++m)
        if (p != tap(o0 + m, j - m)) ++wrong;
      p += line_steps(w, j) ? 1 : 0;
    }
  }
  // along x: a block of nw runs stages its window, 128 entries at a time
  for (int nw = 1; nw <= 8; ++nw)
    for (int64_t x = 0; x < n; x += nw * kLineRun) {
      const int64_t span = std::min<int64_t>(nw * kLineRun, n - x);
      const LineWindow w = line_window(at + x, span, R, lo, hi);
      const int width = nw * kLineRun + 2 * R;
      for (int i = 0; i < (width + 127) / 128 * 128; ++i) in(line_at(w, i));
      for (int m = 0; m < span; ++m)
        for (int k = 0; k <= 2 * R; ++k)
          if (line_at(w, m + k) != tap(at + x + m, k)) ++wrong;
    }
}

int main() {
  const int radii[] = {8, 9, 13, 24, 65};
  for (int R : radii)
    for (int64_t lo : {int64_t(0), int64_t(-7), int64_t(1) << 40})
      for (int64_t size : {1, 2, 15, 16, 17, 33, 64, 97, 150})
        for (int64_t a = 0; a < size; a += a < 3 || a > size - 4 ? 1 : 5)
          for (int64_t n = 1; a + n <= size; n += n < 18 || a + n > size - 3 ? 1 : 7)
            check(lo, lo + size - 1, lo + a, n, R);
  std::printf("%ld geometries: %ld loads outside the source, %ld wrong taps\n", geometries, outside, wrong);
  return outside || wrong ? 1 : 0;
}
