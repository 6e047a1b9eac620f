"""The interleaved gradient stencil (Layout::build_ell) holds every entry of
the CSR rows in order, also for stencils of more than 65,535 entries, and
places beyond 2^31 are counted exactly; compiled for the host from the
layout's own source."""
import subprocess

from fvs2d_gb300 import _build

SRC = r"""
#include <cstdio>
#include "fvs_layout.hpp"
using namespace fvs;
// stencils of the given lengths: entry j of cell ic names cell (7 ic + j) % nc, with coefficients (ic, j)
static bool check(const std::vector<int>& len) {
  Layout<float> L;
  L.nc = (int)len.size();
  for (int ic = 0; ic < L.nc; ic++) {
    for (int j = 0; j < len[ic]; j++) {
      L.st_cell.push_back((7 * ic + j) % L.nc);
      L.st_coef.push_back(float(ic));
      L.st_coef.push_back(float(j));
    }
    L.st_ptr.push_back((int)L.st_cell.size());
  }
  L.build_ell();
  size_t rows = 0;
  for (int g = 0; g < L.nc; g += 32) rows += *std::max_element(len.begin() + g, len.begin() + std::min(g + 32, L.nc));
  if (L.ell_cell.size() != 32 * rows || L.ell_coef.size() != 64 * rows) return false;
  std::vector<char> seen(L.ell_cell.size(), 0);
  for (int ic = 0; ic < L.nc; ic++) {
    if (L.ell_n[ic] != len[ic]) return false;
    for (int j = 0; j < len[ic]; j++) {
      const size_t at = L.ell_place(ic, j);
      if (at >= seen.size() || seen[at]++ || L.ell_cell[at] != (7 * ic + j) % L.nc || L.ell_coef[2 * at] != float(ic) ||
          L.ell_coef[2 * at + 1] != float(j))
        return false;
    }
  }
  return true;
}
int main() {
  std::printf("%d", check({3, 0, 18, 12, 1}));
  std::vector<int> v(65, 3);
  v[31] = 9; v[32] = 1; v[64] = 70000;
  std::printf(" %d", check(v));
  // two groups whose longest stencils have 70 million entries
  Layout<float> L;
  L.nc = 64;
  for (int ic = 0; ic < 64; ic++) L.st_ptr.push_back(L.st_ptr.back() + (ic % 32 ? 2 : 70000000));
  L.build_ell_rows();
  std::printf(" %zu %zu\n", L.ell_place(32, 0), L.ell_place(63, 1));
}
"""


def test_rows(tmp_path):
    f, exe = tmp_path / "t.cu", str(tmp_path / "t")
    f.write_text(SRC)
    subprocess.run([_build.nvcc(), "-O1", "-std=c++17", *_build.ARCH, "-I", _build.INCLUDE, "-I", _build.CSRC, str(f),
                    "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["1", "1", str(32 * 70_000_000), str(32 * 70_000_001 + 31)]
