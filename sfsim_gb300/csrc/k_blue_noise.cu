// k_blue_noise.cu -- the void-and-cluster steps of the blue-noise table
// (src/clj/sfsim/bluenoise.clj:112-169), one CTA per chain of steps.
//
// A step sets or clears one pixel, adds its Gauss weight to the density of
// every pixel and finds the next largest or least density.  The steps form one
// chain, so a step's latency is the cost.  Two things keep it short:
//
// * An FP64 addition of a weight below half a unit in the last place of the
//   density changes nothing.  The pixels go in tiles of 8x4, one lane each; a
//   tile whose smallest density has an exponent 56 above that of the weight at
//   its nearest pixel is left out, and so are its extrema, which the tile
//   keeps.  All other tiles take the full FP64 addition, so the densities and
//   with them the ranks are those of updating every pixel.
// * Where every step only clears pixels (their densities fall) or only sets
//   them (the others rise), the second extremum is the next step's if the
//   first's weight there is such a lost one, as no other pixel can overtake
//   it; likewise the third and fourth.  They go in one step.
// * Extrema are found with warp-wide integer maxima of order-preserving keys;
//   the first warp takes those of the warps' candidates.
//
// What bounds it: one SM's instruction issue (56 % of the cycles; 4400
// instructions a pixel, 24 tiles' additions and maxima) and the latency of a
// step's chain (tile test, additions, maxima, two barriers).  64x64, sigma 1.5:
// phase 3's 2048 pixels go in 816 steps, 1.93 ms, where updating every pixel on
// a cluster of 8 CTAs took 4.36 (its FP64 additions are a sixth, but every step
// waits for the exchange of candidates); the whole table 10.2 -> 4.5 ms,
// 16x16 0.67 -> 0.45, 128x128 45 -> 21.  One pixel a step was 5.1 ms, 16 warps
// 5.1; the final choice by every warp for itself (one barrier) 5.9.
#include <stdint.h>

#include "kernels.h"

namespace sfsim {

namespace {

constexpr int kTileW = 8, kTileH = 4;
constexpr int kTileWarps = 32;
constexpr int kTogether = 4;  // pixels of a step at most

// An extremum: order-preserving key, and the pixel as (y << 16 | x) + 1, 0 for
// none.  Larger keys win, of equal keys the larger pixel (max-key / min-key
// keep the last of equal elements); searches for the least complement the key.
struct Extremum {
  unsigned hi, lo, at;
};
__device__ __forceinline__ bool above(const Extremum& a, const Extremum& b) {
  const unsigned long long ka = (unsigned long long)a.hi << 32 | a.lo, kb = (unsigned long long)b.hi << 32 | b.lo;
  return (ka > kb) | ((ka == kb) & (a.at > b.at));
}

__device__ __forceinline__ Extremum warp_best(Extremum e) {
  Extremum r;
  r.hi = __reduce_max_sync(0xffffffffu, e.hi);
  r.lo = __reduce_max_sync(0xffffffffu, e.hi == r.hi ? e.lo : 0u);
  r.at = __reduce_max_sync(0xffffffffu, e.hi == r.hi && e.lo == r.lo ? e.at : 0u);
  return r;
}

// The keys of a density (never NaN or -0.0) for the largest or the least.
// POSITIVE: it has no sign.
template <bool POSITIVE>
__device__ __forceinline__ Extremum key(double d, bool least, unsigned at) {
  unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned flip = POSITIVE || !(hi >> 31) ? 0u : 0xffffffffu;
  hi = (hi ^ flip) | (flip ? 0u : 0x80000000u), lo ^= flip;
  return least ? Extremum{~hi, ~lo, at} : Extremum{hi, lo, at};
}

__device__ __forceinline__ int exponent(double d) { return (__double2hiint(d) >> 20) & 0x7ff; }

// Distance on a circle of m pixels.
__device__ __forceinline__ int around(int d, int m) {
  d = abs(d);
  return min(d, m - d);
}
__device__ __forceinline__ int around(int c, int lo, int hi, int m) {  // of c from [lo, hi]
  return c >= lo && c <= hi ? 0 : min(around(c - lo, m), around(c - hi, m));
}
__device__ __forceinline__ int px(unsigned at) { return (int)((at - 1) & 0xffffu); }
__device__ __forceinline__ int py(unsigned at) { return (int)((at - 1) >> 16); }

// Tiles across and down, and the pitch of their numbers: those of a window of
// tiles that share neither row nor column then fall to different warps.
__host__ __device__ inline int tiles_across(int m) { return (m + kTileW - 1) / kTileW; }
__host__ __device__ inline int tiles_down(int m) { return (m + kTileH - 1) / kTileH; }
__host__ __device__ inline int tile_pitch(int m) {
  int w = tiles_across(m) | 1;
  while (w % kTileWarps < 3 || w % kTileWarps > kTileWarps - 3) w += 2;
  return w;
}

// Shared memory: the Gauss weights, the densities tile by tile, then by tile
// number its extrema (with the high key of the tile's next best pixel; two of
// them where both kinds are searched), mask and least exponent.
size_t tile_smem(int m, bool both) {
  const size_t h = (size_t)(m / 2 + 1), numbers = (size_t)tile_pitch(m) * tiles_down(m);
  return (((sizeof(double) * (h * h + 32 * (size_t)tiles_across(m) * tiles_down(m))) + 15) & ~size_t(15)) +
         numbers * (both ? 3 : 2) * sizeof(uint4);
}

struct TileShared {
  uint4 best[kTileWarps];  // the warps' candidates: an Extremum, and the high key of the warp's next best pixel
  unsigned chosen[kTogether];
  int count;
};

// The pixels of one chain of steps.  Warp w owns the tiles numbered
// w + i kTileWarps.  CLUSTER: the largest density of the set pixels is
// searched; VOID: the least of the others.
template <bool CLUSTER, bool VOID>
struct Tiles {
  static constexpr bool several = CLUSTER != VOID;  // pixels a step
  int m, h, lane, warp, across, pitch, owned;
  double* table;
  double* density;
  uint4* ext;   // [CLUSTER + VOID][numbers]
  uint4* info;  // mask, least exponent, first pixel (y << 16 | x), first density; a number without tile: -, 0x7ff
  TileShared* sh;
  int numbers;
  bool stale;  // the warp's candidate is to be found again

  __device__ Tiles(int m_, const double* g_table, unsigned char* smem, TileShared* sh_)
      : m(m_), h((m_ >> 1) + 1), lane(threadIdx.x & 31), warp(threadIdx.x >> 5), sh(sh_) {
    across = tiles_across(m), pitch = tile_pitch(m);
    numbers = pitch * tiles_down(m);
    stale = true;
    owned = (numbers - warp + kTileWarps - 1) / kTileWarps;
    table = reinterpret_cast<double*>(smem);
    density = table + h * h;
    ext = reinterpret_cast<uint4*>(smem + (((sizeof(double) * (h * h + 32 * across * tiles_down(m))) + 15) & ~15));
    info = ext + numbers * (CLUSTER + VOID);
    for (int t = threadIdx.x; t < h * h; t += blockDim.x) table[t] = g_table[t];
    __syncthreads();
  }

  // N tiles at once (their chains of maxima overlap): the densities changed by
  // the chosen pixels of by[], then mask, least exponent and extrema renewed.
  template <int N>
  __device__ __forceinline__ void process(const int (&t)[N], const unsigned (&by)[N], bool add) {
    double d[N];
    bool set[N], valid[N];
    unsigned at[N];
#pragma unroll
    for (int n = 0; n < N; n++) {
      const uint4 tile = info[t[n]];
      const unsigned x = (tile.z & 0xffffu) + (lane & (kTileW - 1)), y = (tile.z >> 16) + lane / kTileW;
      double* cell = density + tile.w + lane;
      valid[n] = x < m && y < m;
      at[n] = (y << 16 | x) + 1;
      d[n] = *cell;
      set[n] = tile.x >> lane & 1u;
      for (unsigned rest = by[n]; rest; rest &= rest - 1) {
        const unsigned c = sh->chosen[__ffs(rest) - 1];
        const double f = valid[n] ? table[around((int)y - py(c), m) * h + around((int)x - px(c), m)] : 0.0;
        d[n] = add ? __dadd_rn(d[n], f) : __dsub_rn(d[n], f);
      }
      *cell = d[n];
    }
    renew(t, d, set, valid, at);
  }
  template <int N>
  __device__ __forceinline__ void renew(const int (&t)[N], const double (&d)[N], const bool (&set)[N],
                                        const bool (&valid)[N], const unsigned (&at)[N]) {
    int least[N];
    Extremum k[2][N], b[2][N];
    unsigned next[2][N];
#pragma unroll
    for (int n = 0; n < N; n++) {
      k[0][n] = valid[n] && set[n] == CLUSTER ? key<several>(d[n], !CLUSTER, at[n]) : Extremum{0, 0, 0};
      if (!several) k[1][n] = valid[n] && !set[n] ? key<several>(d[n], true, at[n]) : Extremum{0, 0, 0};
      if (!several) least[n] = __reduce_min_sync(0xffffffffu, valid[n] ? exponent(d[n]) : 0x7ff);
    }
#pragma unroll
    for (int e = 0; e < CLUSTER + VOID; e++) {
#pragma unroll
      for (int n = 0; n < N; n++) b[e][n].hi = __reduce_max_sync(0xffffffffu, k[e][n].hi);
#pragma unroll
      for (int n = 0; n < N; n++)
        b[e][n].lo = __reduce_max_sync(0xffffffffu, k[e][n].hi == b[e][n].hi ? k[e][n].lo : 0u);
#pragma unroll
      for (int n = 0; n < N; n++)
        b[e][n].at = __reduce_max_sync(0xffffffffu,
                                       k[e][n].hi == b[e][n].hi && k[e][n].lo == b[e][n].lo ? k[e][n].at : 0u);
#pragma unroll
      for (int n = 0; n < N; n++)
        next[e][n] = several ? __reduce_max_sync(0xffffffffu, k[e][n].at == b[e][n].at ? 0u : k[e][n].hi) : 0u;
    }
    if (lane == 0) {
#pragma unroll
      for (int n = 0; n < N; n++) {
        // Only the pixels that are searched matter where none comes back among
        // them: the least of the voids' densities is their extremum, and the
        // set pixels' hold their own weight, 1, up to rounding.
        if (several)
          least[n] = b[0][n].at == 0 ? 0x7ff : CLUSTER ? 1022 : (int)(~b[0][n].hi >> 20 & 0x7ff);
        info[t[n]].y = (unsigned)least[n];
#pragma unroll
        for (int e = 0; e < CLUSTER + VOID; e++)
          ext[e * numbers + t[n]] = make_uint4(b[e][n].hi, b[e][n].lo, b[e][n].at, next[e][n]);
      }
    }
    __syncwarp();
  }

  __device__ void load(const double* g_density, const unsigned char* g_mask) {
    for (int i = 0; i < owned; i++) {
      const int t[1] = {warp + i * kTileWarps}, ty = t[0] / pitch, tx = t[0] - ty * pitch;
      const int x = tx * kTileW + (lane & (kTileW - 1)), y = ty * kTileH + lane / kTileW;
      const bool valid[1] = {x < m && y < m};
      const double d[1] = {valid[0] ? g_density[y * m + x] : 0.0};
      const bool set[1] = {valid[0] && g_mask[y * m + x]};
      const unsigned at[1] = {((unsigned)y << 16 | (unsigned)x) + 1};
      const unsigned first = tx < across ? (ty * across + tx) * 32 : 0;
      if (tx < across) density[first + lane] = d[0];
      const unsigned bits = __ballot_sync(0xffffffffu, set[0]);
      if (lane == 0) info[t[0]] = make_uint4(bits, 0, (unsigned)(ty * kTileH) << 16 | (unsigned)(tx * kTileW), first);
      renew(t, d, set, valid, at);
    }
  }
  // the mask back to memory, inverted on request
  __device__ void store(unsigned char* g_mask, bool invert) const {
    for (int i = 0; i < owned; i++) {
      const int t = warp + i * kTileWarps, ty = t / pitch, tx = t - ty * pitch;
      const int x = tx * kTileW + (lane & (kTileW - 1)), y = ty * kTileH + lane / kTileW;
      if (x < m && y < m) g_mask[y * m + x] = ((info[t].x >> lane & 1u) != 0) != invert;
    }
  }

  // The pixels of the next step, at most `limit`, into sh->chosen until the next
  // call; their number, the same for every thread.
  __device__ int choose(bool want_void, int limit) {
    if (!several || stale) {
      const uint4* mine = ext + (!several && want_void ? numbers : 0);
      Extremum e{0, 0, 0};
      unsigned after = 0;  // the high key of the lane's best pixel but e
      for (int i = lane; i < owned; i += 32) {
        const uint4 q = mine[warp + i * kTileWarps];
        const Extremum k{q.x, q.y, q.z};
        if (above(k, e)) {
          after = max(e.hi, q.w);
          e = k;
        } else {
          after = max(after, k.hi);
        }
      }
      const Extremum w = warp_best(e);
      if (several) after = __reduce_max_sync(0xffffffffu, e.at == w.at ? after : e.hi);
      if (lane == 0) sh->best[warp] = make_uint4(w.hi, w.lo, w.at, after);
      stale = false;
    }
    __syncthreads();
    if (warp == 0) select(min(limit, several ? kTogether : 1), want_void);
    __syncthreads();
    return sh->count;
  }

  // The first warp: the best candidate, and those after it that the steps
  // before them leave the best.
  __device__ __forceinline__ void select(int limit, bool want_void) {
    static_assert(kTileWarps <= 32 && kTogether == 4, "a lane a candidate; six pairs");
    uint4 q = make_uint4(0, 0, 0, 0);
    if (lane < kTileWarps) q = sh->best[lane];
    unsigned hi[kTogether], at[kTogether], after[kTogether];
#pragma unroll
    for (int j = 0; j < (several ? kTogether : 1); j++) {
      const Extremum b = warp_best(Extremum{q.x, q.y, q.z});
      hi[j] = b.hi, at[j] = b.at;
      const bool mine = q.z == b.at;
      after[j] = several ? __reduce_max_sync(0xffffffffu, mine ? q.w : 0u) : 0u;
      if (mine) q = make_uint4(0, 0, 0, 0);
    }
    int count = at[0] != 0 && limit > 0;
    if (several) {
      // lane p < 6: the pair (early, late) = (0,1) (0,2) (1,2) (0,3) (1,3) (2,3); is the weight of early lost in late?
      const int late = lane < 1 ? 1 : lane < 3 ? 2 : 3;
      const int early = lane - late * (late - 1) / 2;
      const unsigned a0 = early == 0 ? at[0] : early == 1 ? at[1] : at[2];
      const unsigned a1 = late == 1 ? at[1] : late == 2 ? at[2] : at[3];
      const unsigned h1 = late == 1 ? hi[1] : late == 2 ? hi[2] : hi[3];
      const unsigned high = VOID ? ~h1 : h1;  // of the key of the largest
      bool lost = false;
      if (lane < 6 && a0 && a1 && high >> 31)
        lost = exponent(table[around(py(a1) - py(a0), m) * h + around(px(a1) - px(a0), m)]) + 56 <=
               (int)(high >> 20 & 0x7ff);
      const unsigned ok = __ballot_sync(0xffffffffu, lost);
      unsigned passed = 0;  // the high key of the best pixel that is no candidate
#pragma unroll
      for (int j = 1; j < kTogether; j++) {
        passed = max(passed, after[j - 1]);
        const unsigned need = ((1u << j) - 1) << (j * (j - 1) / 2);
        if (count == j && j < limit && at[j] && hi[j] > passed && (ok & need) == need) count = j + 1;
      }
    }
    if (lane == 0) {
#pragma unroll
      for (int j = 0; j < (several ? kTogether : 1); j++) sh->chosen[j] = at[j];
      sh->count = count;
    }
  }

  // Sets or clears the chosen pixels, in order, and adds their weights to, or
  // takes them from, the densities.
  __device__ void change(int count, bool add, bool set_c) {
    const int j = lane & 3;
    const unsigned c = sh->chosen[j];
    if (lane < count) {  // its mask bit; chosen pixels are in different tiles
      const int t = py(c) / kTileH * pitch + px(c) / kTileW;
      if (t % kTileWarps == warp) {
        const unsigned bit = 1u << ((py(c) % kTileH) * kTileW + px(c) % kTileW);
        info[t].x = set_c ? info[t].x | bit : info[t].x & ~bit;
      }
    }
    __syncwarp();
    for (int i0 = 0; i0 < owned; i0 += 8) {
      // lane: tile i0 + lane / 4, chosen pixel lane % 4; is its weight lost in the whole tile?
      const int i = i0 + (lane >> 2);
      bool near = false;
      if (i < owned && j < count) {
        const uint4 tile = info[warp + i * kTileWarps];
        if (tile.y < 0x7ff) {
          const int x0 = (int)(tile.z & 0xffffu), y0 = (int)(tile.z >> 16);
          const double f = table[around(py(c), y0, min(y0 + kTileH, m) - 1, m) * h +
                                 around(px(c), x0, min(x0 + kTileW, m) - 1, m)];  // the tile's largest
          near = exponent(f) + 56 > (int)tile.y;
        }
      }
      unsigned todo = __ballot_sync(0xffffffffu, near);
      stale = stale || todo;
      while (todo) {
        const int a = (__ffs(todo) - 1) >> 2;
        const unsigned by_a = todo >> (4 * a) & 15u;
        todo &= ~(15u << (4 * a));
        const int ta = warp + (i0 + a) * kTileWarps;
        if (todo) {
          const int b = (__ffs(todo) - 1) >> 2;
          const unsigned by_b = todo >> (4 * b) & 15u;
          todo &= ~(15u << (4 * b));
          const int t[2] = {ta, warp + (i0 + b) * kTileWarps};
          const unsigned by[2] = {by_a, by_b};
          process<2>(t, by, add);
        } else {
          const int t[1] = {ta};
          const unsigned by[1] = {by_a};
          process<1>(t, by, add);
        }
      }
    }
  }
  __device__ int index(unsigned at) const { return py(at) * m + px(at); }
};

}  // namespace

// seed-pattern (bluenoise.clj:112-124): remove the tightest cluster, add the
// largest void, until they coincide; the pattern is left in `mask`.
__global__ void __launch_bounds__(32 * kTileWarps, 1)
    k_blue_tiles_seed(int m, const double* table, const double* density, unsigned char* mask) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ TileShared sh;
  Tiles<true, true> t(m, table, smem, &sh);
  t.load(density, mask);
  int count = t.choose(false, 1);
  for (int it = 0; it < m * m * 4 && count; it++) {  // the pattern settles long before this bound
    const unsigned c = sh.chosen[0];
    t.change(1, false, false);
    if (!t.choose(true, 1)) break;  // cannot happen for 1 <= n <= m*m/2
    const unsigned v = sh.chosen[0];
    t.change(1, true, true);
    if (v == c) break;
    count = t.choose(false, 1);
  }
  t.store(mask, false);
}

// dither-phase1 and dither-phase2 (bluenoise.clj:127-154), both from the seed
// pattern and its density, a CTA each: ranks n-1 .. 0 for the removed
// clusters, n .. m*m/2 - 1 for the filled voids.  The second leaves the
// complement of the half-filled pattern in `work` for phase 3.
__global__ void __launch_bounds__(32 * kTileWarps, 1)
    k_blue_tiles_phases(int m, int n, const double* table, const double* density, const unsigned char* mask,
                        unsigned char* work, int* dither) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ TileShared sh;
  if (blockIdx.x == 0) {
    Tiles<true, false> t(m, table, smem, &sh);
    t.load(density, mask);
    for (int r = n; r > 0;) {
      const int count = t.choose(false, r);
      if (!count) break;
      if ((int)threadIdx.x < count) dither[t.index(sh.chosen[threadIdx.x])] = r - 1 - (int)threadIdx.x;
      t.change(count, false, false);
      r -= count;
    }
  } else {
    Tiles<false, true> t(m, table, smem, &sh);
    t.load(density, mask);
    for (int r = n; r < m * m / 2;) {
      const int count = t.choose(true, m * m / 2 - r);
      if (!count) break;
      if ((int)threadIdx.x < count) dither[t.index(sh.chosen[threadIdx.x])] = r + (int)threadIdx.x;
      t.change(count, true, true);
      r += count;
    }
    t.store(work, true);
  }
}

// dither-phase3 (bluenoise.clj:157-169) on the complement `work` with its
// density: ranks m*m/2 .. m*m - 1 for the removed clusters.
__global__ void __launch_bounds__(32 * kTileWarps, 1)
    k_blue_tiles_phase3(int m, const double* table, const double* density, const unsigned char* work, int* dither) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ TileShared sh;
  Tiles<true, false> t(m, table, smem, &sh);
  t.load(density, work);
  for (int r = m * m / 2; r < m * m;) {
    const int count = t.choose(false, m * m - r);
    if (!count) break;
    if ((int)threadIdx.x < count) dither[t.index(sh.chosen[threadIdx.x])] = r + (int)threadIdx.x;
    t.change(count, false, false);
    r += count;
  }
}

// The tiles serve where their state fits in shared memory (to 136x136) and a
// pixel's weights reach few of them, or no cluster takes the table.  Measured,
// tiles / cluster: 64x64, sigma 2.5 (79 tiles in reach) 7.8 / 10.0 ms, 2.85
// (100) 9.1 / 9.9, 3 (110) 9.6 / 10.0, 6 (all 128) 13.2 / 9.8; 96x96, 2.5 16.4 /
// 25.5, 4 (186) 30.1 / 24.5; 128x128, 2.5 29.5 / 44.0, 6 (all 512) 91 / 43.
// Against one CTA that updates every pixel: 45x45, 1.5 2.6 / 6.2, 30 5.0 / 6.2;
// 91x91, 6 44 / 52; 135x135, 20 144 / 213.
bool blue_tiles_serve(int m, double sigma) {
  if (tile_smem(m, true) > 220 * 1024) return false;
  // pixels within this distance take weights above 2^-57 of their centre's
  const double reach = 8.9 * sigma;
  const double across = (2 * reach + kTileW) / kTileW, down = (2 * reach + kTileH) / kTileH;
  return across * down <= 100 || tiles_across(m) * tiles_down(m) <= 100 || blue_noise_cluster_size(m) == 0;
}

int launch_blue_tiles(int stage, int m, int n, const double* table, double* density, double* density0,
                      unsigned char* mask, unsigned char* work, int* dither, cudaStream_t st) {
  const size_t smem = tile_smem(m, stage == 0);
  auto fits = [&](auto kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess;
  };
  const int threads = 32 * kTileWarps;
  if (stage == 0) {
    if (!fits(k_blue_tiles_seed)) return -1;
    k_blue_tiles_seed<<<1, threads, smem, st>>>(m, table, density, mask);
  } else if (stage == 1) {
    if (!fits(k_blue_tiles_phases)) return -1;
    k_blue_tiles_phases<<<2, threads, smem, st>>>(m, n, table, density0, mask, work, dither);
  } else {
    if (!fits(k_blue_tiles_phase3)) return -1;
    k_blue_tiles_phase3<<<1, threads, smem, st>>>(m, table, density, work, dither);
  }
  return 0;
}

}  // namespace sfsim
