// lbx_march.h — columns and segments of the single-pass step k_cg_march
// (lbx_fluid.cu).  Plain C++.
#pragma once
#include <algorithm>
#include <cmath>

namespace lbx {

// Columns of w x h cells, kx of them along x and `cols` in all (cut at the
// box's ends), marched in segments of zlen planes.
struct MarchPlan {
  int w, h, zlen, kx, cols;
};

// Limits of a CTA computing in type C: its threads (at least w h, and at least
// one per ring cell), its window planes of ROWS x PITCH cells and its ring.
template <typename C>
struct March {
  static constexpr int NT = 256, PITCH = sizeof(C) == 4 ? 40 : 34, ROWS = sizeof(C) == 4 ? 16 : 10;
  static constexpr int WMAX = PITCH - 2, HMAX = ROWS - 2, RING = 2 * (PITCH + HMAX);
  static constexpr int LEN = 16;  // planes of a segment: more leave the end of a step to a few CTAs
  static_assert(RING <= NT, "a ring cell per thread");
};

// The shape and segment length with the smallest estimate of the step's time
// on `resident` CTAs.  A segment costs its planes and 0.4 for the two planes it
// only sums; the whole segments go to the resident CTAs in turn, then the cut
// ones at the end of z; a plane costs more with its ring, with short rows, and,
// with FP32 pairs (`fp32`) and enough planes that memory bounds the step, where
// rows do not fill 256-byte lines.  Shapes: 32 cells wide, and the widths that
// split x evenly.  The weights are fitted: against every shape and length
// measured (40 boxes of 16^3 to 300 x 200 x 100, five pairs of model and
// storage, a new droplet and a noise field) the choice is 1.1 % slower than the
// best on average and 11 % at worst; columns of 32 x 8 in waves of equal
// segments, which it replaces, were 15 % and 79 %.
template <typename C>
MarchPlan march_plan(int nx, int ny, int nz, int resident, bool fp32) {
  using M = March<C>;
  const double extra = 0.4;
  MarchPlan best{0, 0, 0, 0, 0};
  double least = 0;
  long ctas = 0;  // of the best; the fewest of equal estimates
  auto width = [&](int w) {
    const int hmax = std::min(M::HMAX, M::NT / w), rows = (ny + hmax - 1) / hmax;
    for (int ky = rows; ky <= std::min(rows + 1, ny); ++ky) {
      const int h = (ny + ky - 1) / ky, kx = (nx + w - 1) / w;
      const long cols = long(kx) * ((ny + h - 1) / h);
      const bool lines = fp32 && cols * nz > 4L * resident;
      const double plane = 1.0 + 1.5 * (2 * (w + h) + 4) / M::NT + 0.1 * std::max(0, 32 - w) / 16 +
                           (w % 16 ? 0.03 : 0.0) + (lines && w % 32 ? 0.15 : 0.0);
      for (int len = 1; len <= std::min(nz, M::LEN); ++len) {
        const int segs = (nz + len - 1) / len;
        const double job = len + extra, cut = nz - (segs - 1) * len + extra;
        const long whole = cols * (segs - 1);
        double t = job;
        if (whole + cols > resident) {
          const long turns = whole / resident, late = whole % resident, idle = resident - late;
          const long fit = late ? long(std::ceil(job / cut)) : cols, rounds = (cols + idle - 1) / idle;
          if (rounds <= fit) t = std::max((turns + (late ? 1 : 0)) * job, turns * job + rounds * cut);
          else t = turns * job + (fit + (cols - idle * fit + resident - 1) / resident) * cut;
        }
        t *= plane;
        const long n = whole + cols;
        if (!best.w || t < least * (1 - 1e-9) || (t < least * (1 + 1e-9) && n < ctas)) {
          least = t;
          ctas = n;
          best = MarchPlan{w, h, len, kx, int(cols)};
        }
      }
    }
  };
  if (nx > 32) width(32);
  for (int kx = (nx + M::WMAX - 1) / M::WMAX, last = 0; kx <= nx; ++kx) {
    const int w = (nx + kx - 1) / kx;
    if (last && w < 16) break;  // narrower columns are mostly ring
    if (w != last) width(w);
    last = w;
  }
  return best;
}

}  // namespace lbx
