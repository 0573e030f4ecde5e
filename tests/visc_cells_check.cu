// Host-side walk over the cells that a launch of k_visc_lsq covers
// (ucg::visc_lsq_cell in ucns3d_b200/csrc/engine/recon2.cuh, the function by
// which the kernel picks its cell), compiled with nvcc as host code and run by
// tests/test_visc_cells.py.  stdin: "n ntile nugrp", the tiles' cells
// [ntile][128], the groups with cells that are not in a tile [nugrp], per cell
// whether it is in a tile [n]; stdout: how often each cell is written by the
// launch with tiles, then by the one without.
#include <cstdio>
#include <vector>

#include "../ucns3d_b200/csrc/engine/recon2.cuh"

int main() {
  long n, ntile, nugrp;
  if (std::scanf("%ld %ld %ld", &n, &ntile, &nugrp) != 3) return 1;
  std::vector<int32_t> tcell(ntile * ucg::SET_TILE), ugrp(nugrp);
  std::vector<int8_t> tiled(n);
  int x;
  for (auto& t : tcell) std::scanf("%d", &t);
  for (auto& g : ugrp) std::scanf("%d", &g);
  for (auto& t : tiled) {
    if (std::scanf("%d", &x) != 1) return 1;
    t = (int8_t)x;
  }
  ucg::Problem p{};
  p.n = n;
  p.ntile = ntile;
  p.nugrp = nugrp;
  p.tcell = tcell.data();
  p.ugrp = ugrp.data();
  p.tiled = nugrp ? tiled.data() : nullptr;  // as the engine: no list where every cell is in a tile
  std::vector<int> set(n, 0), own(n, 0);
  for (int64_t b = 0; b < ucg::visc_lsq_own(p) + ntile; ++b)
    for (int t = 0; t < 128; ++t) {
      const int64_t c = ucg::visc_lsq_cell<true>(p, b, t);
      if (c >= 0) ++set.at(c);
    }
  for (int64_t b = 0; b < (n + 127) / 128; ++b)
    for (int t = 0; t < 128; ++t) {
      const int64_t c = ucg::visc_lsq_cell<false>(p, b, t);
      if (c >= 0) ++own.at(c);
    }
  for (int c : set) std::printf("%d ", c);
  for (int c : own) std::printf("%d ", c);
  return 0;
}
