// Lock-free union-find over a parent array (p[x] <= x, roots have p[x] == x):
// the larger root goes under the smaller, so a tree's root is its minimum id.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gb {

__device__ __forceinline__ uint32_t find_root(uint32_t* p, uint32_t x) {
  uint32_t px = p[x];
  while (px != x) {
    const uint32_t ppx = p[px];
    if (ppx != px) p[x] = ppx;  // path halving (benign race: ancestors only)
    x = px;
    px = ppx;
  }
  return x;
}

// Link the trees of a and b: larger root goes under the smaller (ECL-CC style).
__device__ __forceinline__ void link(uint32_t* p, uint32_t a, uint32_t b) {
  uint32_t ra = find_root(p, a), rb = find_root(p, b);
  for (int guard = 0; ra != rb && guard < (1 << 20); ++guard) {
    if (ra < rb) {
      const uint32_t ret = atomicCAS(&p[rb], rb, ra);
      if (ret == rb) break;
      rb = find_root(p, ret);
    } else {
      const uint32_t ret = atomicCAS(&p[ra], ra, rb);
      if (ret == ra) break;
      ra = find_root(p, ret);
    }
  }
}

}  // namespace gb
