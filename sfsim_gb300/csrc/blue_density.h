// blue_density.h -- launch shape of k_blue_density (k_noise.cu), host code.
#pragma once

#include <algorithm>
#include <cstddef>

namespace sfsim {

// A block's shared memory: the Gauss weights and the list of the set pixels.
inline size_t blue_density_smem(int m) {
  const size_t h = (size_t)(m / 2 + 1);
  return 8 * h * h + 2 * (((size_t)m * m + 1) / 2);
}

constexpr int kDensityWarps = 16;  // of a block at most

// Warps of a block: one while all blocks are on the SMs at once, so that the
// pixels' chains of additions spread over them; where the shared memory leaves
// room for few blocks, as many as put every block on an SM in one wave (a
// second wave repeats the whole chain).  One warp a block throughout took 137,
// 160 and 349 ms for whole tables of 192, 200 and 256 pixels a side, so 131, 146
// and 303 (4, 9 and 14 warps).
inline int blue_density_warps(int m, int sms) {
  const long long room = 227 * 1024, block = (long long)blue_density_smem(m) + 1024;
  const long long resident = sms * std::min<long long>(32, std::max<long long>(1, room / block));
  const long long warps = ((long long)m * m + 31) / 32;
  return (int)std::min<long long>(kDensityWarps, (warps + resident - 1) / resident);
}

}  // namespace sfsim
