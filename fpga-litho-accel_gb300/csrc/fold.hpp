// Four-row folding of the FP32 transforms (imaging_fold.cu).  With the centred row coordinate
// y' = Y + (Fy-Ly)/2 - Fy/2 and h = Fy/2, the rows y' = b, -b, h - b, -(h - b) of a base row
// 0 <= b <= h/2 share their cos and sin up to signs:
//   cos(2 pi v (h - b)/Fy) = (-1)^v cos(2 pi v b/Fy),  sin(2 pi v (h - b)/Fy) = -(-1)^v sin(2 pi v b/Fy),
// so one row of coefficients serves four mask or image rows.  Plain C++ (host and device), so
// the folding is also checked on the CPU.
#pragma once
#include "fi_mirror.hpp"

namespace litho {

// base rows of a geometry: those b that fold at least one row of it
LITHO_FO_HD inline int fold_nbase(int Ly, int Fy) {
  const int nb = fo_nbase(Ly, Fy), q = Fy / 4 + 1;
  return nb < q ? nb : q;
}

// row of base row b, k = 0..3 (y' = b, -b, h - b, -(h - b)), or -1 where that row is not in the
// geometry or is another k's row (b = 0; 2b = h)
LITHO_FO_HD inline int fold_row(int b, int k, int Ly, int Fy) {
  const int h = Fy / 2;
  if (k < 2) return fo_row(b, k, Ly, Fy);
  return 2 * b == h ? -1 : fo_row(h - b, k - 2, Ly, Fy);
}

// the same as ranges: row k of base row b is in the geometry for lo <= b < lo + n, at y' = +-b + off
struct FoldRange {
  int lo, n;
};
LITHO_FO_HD inline FoldRange fold_range(int k, int Ly, int Fy) {
  const int h = Fy / 2, oy = fo_oy(Ly, Fy), top = Ly - 1 + oy, half = (h - 1) / 2;  // 2b < h: b <= half
  int lo, hi;
  if (k == 0) {
    lo = 0;
    hi = top;
  } else if (k == 1) {
    lo = 1;
    hi = -oy;
  } else {
    lo = h - (k == 2 ? top : -oy);
    hi = half;
    if (lo < 0) lo = 0;
  }
  const int q = h / 2;  // base rows go up to h/2
  if (hi > q) hi = q;
  return FoldRange{lo, hi >= lo ? hi - lo + 1 : 0};
}
// row Y of (b, k), in the geometry or not
LITHO_FO_HD inline int fold_y(int b, int k, int Ly, int Fy) {
  const int oy = fo_oy(Ly, Fy), yp = k < 2 ? b : Fy / 2 - b;
  return ((k & 1) ? -yp : yp) - oy;
}

}  // namespace litho
