// Index arithmetic of the line passes (conv_lines.cu), apart from the kernels
// so that a host program can walk it over every geometry (tests/cpp/line_window.cpp).
//
// Positions along the pass axis are counted from the image's first one (`lo`).
// A pass's source holds the positions its requested outputs reach and no more
// (an intermediate image, or a caller's buffer that covers exactly the input
// region of a request), while the kernels load whole windows: 2R + kLineRun
// positions for a run of kLineRun outputs, of which the last run of a request
// may hold fewer.  So a window ends at the last tap of its last requested
// output, not at the image's end; the positions after it repeat that one, and
// only outputs outside the request take them.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define ITKG_LINE_HD __host__ __device__ __forceinline__
#else
#define ITKG_LINE_HD inline
#endif

namespace itkg {

constexpr int kLineRun = 16;  // outputs per thread

struct LineWindow {
  int first;  // position of window entry 0; negative before the image's first position
  int last;   // the largest position that may be loaded
};

// Window of the outputs at .. at + n - 1 (absolute indices, n >= 1) of an axis
// whose image spans [lo, hi].
ITKG_LINE_HD LineWindow line_window(int64_t at, int64_t n, int radius, int64_t lo, int64_t hi) {
  const int64_t end = at + n - 1 + radius;
  LineWindow w;
  w.first = (int)(at - radius - lo);
  w.last = (int)((end < hi ? end : hi) - lo);
  return w;
}

// The position that window entry i is loaded from.
ITKG_LINE_HD int line_at(const LineWindow& w, int i) {
  const int p = w.first + i;
  return p < 0 ? 0 : (p > w.last ? w.last : p);
}

// Whether entry i + 1 lies one position after entry i (else at the same one):
// line_at(w, i + 1) == line_at(w, i) + line_steps(w, i).
ITKG_LINE_HD bool line_steps(const LineWindow& w, int i) { return (unsigned)(w.first + i) < (unsigned)w.last; }

}  // namespace itkg
