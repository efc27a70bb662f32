// The launch of the g(r) histogram (action_kernels.cu), free of CUDA so that its
// limits can be checked on the host.
#pragma once

#include <algorithm>

#ifdef __CUDACC__
#define PIMC_HD __host__ __device__ __forceinline__
#else
#define PIMC_HD inline
#endif

namespace pimc {

struct GofrShape {
  int tile;         // particles a tile: 64, or 32 where that would leave the SMs short of blocks
  long long items;  // tile pairs x slices
  int blocks;
};

// slices: the S - 1 that are counted.  One resident wave of four blocks an SM, and
// more only where a block's items could wrap its 32-bit bins (every pair of an
// item can fall in one bin: 2^20 - 1 items of 64 x 64).
inline GofrShape gofr_shape(long long n, long long slices, int sm_count) {
  auto count = [&](int tile) {
    const long long nt = (n + tile - 1) / tile;
    return nt * (nt + 1) / 2 * slices;
  };
  GofrShape g;
  g.tile = count(64) >= 4ll * sm_count ? 64 : 32;
  g.items = count(g.tile);
  const long long most = 0xffffffffll / (g.tile * g.tile);
  g.blocks = (int)std::max(std::min(g.items, 4ll * sm_count), (g.items + most - 1) / most);
  return g;
}

// Block b's items are [gofr_first(b), gofr_first(b + 1)): equal shares to one.
PIMC_HD long long gofr_first(long long items, long long blocks, long long b) {
  const long long per = items / blocks, rem = items - per * blocks;
  return per * b + (b < rem ? b : rem);
}

}  // namespace pimc
