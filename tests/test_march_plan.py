"""Columns and segments of the single-pass step (lbx_march.h), on the host.

Every column has a thread per cell and per ring cell, fits the shared window, and together they cover the box once.
On boxes that columns of 32 x 8 do not divide, at least three quarters of the columns' cells lie in the box (of 32 x 8
columns 43 % did at 33 x 33 and 60 % at 65 x 57, where the step took up to 1.3 times as long as two passes).
"""
import subprocess

SOURCE = r"""
#include "lbx_march.h"
#include <cstdio>
template <typename C> int check(int nx, int ny, int nz, int resident, bool fp32 = false) {
  using M = lbx::March<C>;
  const lbx::MarchPlan p = lbx::march_plan<C>(nx, ny, nz, resident, fp32);
  const int ky = p.kx > 0 ? p.cols / p.kx : 0;
  const int ring = 2 * (p.w + 2) + 2 * p.h;
  bool ok = p.w >= 1 && p.h >= 1 && p.zlen >= 1 && p.zlen <= nz && p.w * p.h <= M::NT && ring <= M::RING &&
            p.w + 2 <= M::PITCH && p.h + 2 <= M::ROWS && p.kx * ky == p.cols;
  // the columns cover the box, none lies outside it
  ok = ok && (p.kx - 1) * p.w < nx && p.kx * p.w >= nx && (ky - 1) * p.h < ny && ky * p.h >= ny;
  if (!ok) std::printf("%d x %d x %d: w %d h %d zlen %d kx %d cols %d\n", nx, ny, nz, p.w, p.h, p.zlen, p.kx, p.cols);
  return !ok;
}
int main() {
  int bad = 0;
  for (int nx = 3; nx <= 140; nx += nx < 45 ? 1 : 3)
    for (int ny = 3; ny <= 140; ny += (nx * 7) % 11 + 1)
      for (int nz : {3, 17, 64}) bad += check<float>(nx, ny, nz, 296, nx % 2) + check<double>(nx, ny, nz, 148);
  for (int n : {200, 257, 1000, 4099})
    for (int m : {3, 33}) bad += check<float>(n, m, 5, 296) + check<float>(m, n, 5, 1) + check<double>(n, m, 40, 148);
  const int awkward[][3] = {{33, 33, 33}, {40, 40, 40}, {65, 57, 49}, {100, 64, 64}, {100, 100, 100}, {20, 200, 50}};
  for (auto& d : awkward) {
    const lbx::MarchPlan p = lbx::march_plan<float>(d[0], d[1], d[2], 296, true);
    const double share = double(d[0]) * d[1] / (double(p.cols) * p.w * p.h);
    if (share < 0.75) {
      std::printf("%d x %d x %d: %.2f of the columns in the box\n", d[0], d[1], d[2], share);
      ++bad;
    }
  }
  return bad != 0;
}
"""


def test_columns_fit_the_kernel_and_cover_the_box(tmp_path):
    from lbcuda_b200 import build as B
    src = tmp_path / "plan.cpp"
    src.write_text(SOURCE)
    exe = str(tmp_path / "plan")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", B.CSRC, str(src), "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stdout[:2000]
