"""The index arithmetic of the candidate list's cell ranges, compiled for the host."""

import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pgm_jax_b200", "csrc")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>
#include "pgm_device.cuh"

// number of violations for one type: cells outside the axis, cells named twice, and, for ordinary arguments, cells
// that an atom of the range of the search can be in and that are not named
template <typename T>
int check() {
  std::mt19937 gen(5);
  auto uniform = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); };
  const T inf = std::numeric_limits<T>::infinity(), nan = std::numeric_limits<T>::quiet_NaN(), big = std::numeric_limits<T>::max();
  const T odd[] = {nan, inf, -inf, big, -big, T(3e9), T(-3e9), T(0), T(-0.0), T(1), T(-1)};
  int bad = 0;
  for (int trial = 0; trial < 200000; ++trial) {
    const int n = 1 + gen() % 64, ci = gen() % n;
    T f = T(uniform(-0.01, 1.01)), z = T(uniform(0, 1.2 * n));
    bool ordinary = true;
    if (trial % 4 == 0) { f = odd[gen() % 11]; ordinary = false; }
    if (trial % 8 < 2) { z = odd[gen() % 11]; ordinary = false; }
    int lo, hi, seen[64] = {0};
    pgm::cells_within<T>(f, z, ci, n, lo, hi);
    const pgm::CellRange r = pgm::wrapped_cells(lo, hi, n);
    if (r.lo < 0 || r.hi >= n || r.lo > r.hi || r.hi2 < -1 || r.hi2 >= n) { ++bad; continue; }
    for (int c = r.lo; c <= r.hi; ++c) ++seen[c];
    for (int c = 0; c <= r.hi2; ++c) ++seen[c];
    for (int c = 0; c < n; ++c) bad += seen[c] > 1;
    if (!ordinary) continue;
    for (int k = 0; k < 20; ++k) {  // points at most z cell widths away, on any image
      const double x = ci + double(f) + uniform(-1, 1) * double(z);
      const int c = ((int)std::floor(x) % n + n) % n;
      bad += !seen[c];
    }
  }
  // the ranges of the general path: ci - R .. ci + R with 2 R + 1 < n
  for (int n = 2; n <= 64; ++n)
    for (int ci = 0; ci < n; ++ci)
      for (int R = 0; 2 * R + 1 < n; ++R) {
        const pgm::CellRange r = pgm::wrapped_cells(ci - R, ci + R, n);
        int seen[64] = {0}, total = 0;
        for (int c = r.lo; c <= r.hi; ++c) ++seen[c];
        for (int c = 0; c <= r.hi2; ++c) ++seen[c];
        for (int c = 0; c < n; ++c) total += seen[c];
        for (int d = -R; d <= R; ++d) bad += seen[((ci + d) % n + n) % n] != 1;
        bad += total != 2 * R + 1;
      }
  return bad;
}

int main() {
  const int a = check<float>(), b = check<double>();
  std::printf("%d %d\n", a, b);
  return a || b;
}
"""


def test_cell_ranges_stay_on_the_axis_and_cover_the_search(tmp_path):
    """Every range names each cell at most once and none outside its axis, whatever the position, box and width
    (NaN, infinities, the largest numbers); for ordinary ones it holds every cell within reach."""
    from pgm_jax_b200.build import NVCC

    src, exe = tmp_path / "ranges.cu", tmp_path / "ranges"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
