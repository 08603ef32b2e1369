// gg_band.h -- bands of the near-far shortest-path searches (plain C++).
#pragma once

#include <limits>

namespace gg {

// `want` as a distance of type T: at least one positive value of the type, at most a
// quarter of its largest finite one (threshold plus width stays in range).  Clamped before it is
// converted: outside the type's range the conversion is undefined (x86 gives INT_MIN, Arm
// saturates).
template <typename T>
inline T band_width(double want) {
  const double top = static_cast<double>(std::numeric_limits<T>::max()) / 4;
  if (!(want > 0.0)) want = 1.0;
  if (want > top) want = top;
  const T width = static_cast<T>(want);
  return width > T(0) ? width : T(1);
}

// Empty bands in a row (each twice as wide as the one before) that a search takes before it
// gives up: more than the doublings from the smallest Float64 to the largest.  A gap between
// two distances takes about log2(gap / width) of them, which no count of vertices bounds
// (1400 short paths 2^52 apart take some 45000), so they do not count as steps.
static const int kEmptyBandRun = 2200;

}  // namespace gg
