// hv_spatial.cuh -- the spatial order of a source catalogue: sort words, and
// the order of a small catalogue by counting.
#pragma once

#include "hv_internal.cuh"

namespace hv {

// Key: Morton code (16 bits per axis) of the octahedral projection of the
// unit vector.
__device__ __forceinline__ uint32_t spread16(uint32_t a) {
  a = (a | (a << 8)) & 0x00FF00FFu;
  a = (a | (a << 4)) & 0x0F0F0F0Fu;
  a = (a | (a << 2)) & 0x33333333u;
  a = (a | (a << 1)) & 0x55555555u;
  return a;
}

// Sort word of source i: (Morton key << 32) | i, or all ones for padding.
__device__ __forceinline__ unsigned long long sort_word(const float* __restrict__ crd_eq,
                                                        int nsrc, int i) {
  unsigned long long v = ~0ull;
  {
    if (i < nsrc) {
      const float x = crd_eq[i], y = crd_eq[(size_t)nsrc + i], z = crd_eq[2 * (size_t)nsrc + i];
      const float n = fabsf(x) + fabsf(y) + fabsf(z);
      float u = n > 0.f ? x / n : 0.f, w = n > 0.f ? y / n : 0.f;
      if (z < 0.f) {
        const float uu = (1.f - fabsf(w)) * (u < 0.f ? -1.f : 1.f);
        const float ww = (1.f - fabsf(u)) * (w < 0.f ? -1.f : 1.f);
        u = uu;
        w = ww;
      }
      // NaN-safe quantisation to [0, 65535]
      const float qu = fminf(fmaxf((u + 1.f) * 32767.5f, 0.f), 65535.f);
      const float qw = fminf(fmaxf((w + 1.f) * 32767.5f, 0.f), 65535.f);
      const uint32_t key = spread16((uint32_t)qu) | (spread16((uint32_t)qw) << 1);
      v = ((unsigned long long)key << 32) | (uint32_t)i;
    }
  }
  return v;
}

// Catalogues of up to this many sources are ordered by counting.
constexpr int kRankSort = 8192;
constexpr int kRankThreads = 256;                       // a block's threads
constexpr int kRankSources = kRankThreads / 32 * 4;     // and sources

// Sources [kRankSources b, +kRankSources) of a catalogue of n <= kRankSort to
// their places in the order of the sort words: the number of words before
// each.  Every block forms all keys in shared memory (as uint4, n rounded up
// to 4), and a warp counts for 4 neighbouring sources at once, 4 keys a lane
// and step, so that a key read from shared memory serves 4 comparisons.
// Quadratic in n, but without a barrier after the keys, and on as many SMs as
// there are blocks: 11.6 us under ncu for 3072 sources with the rest of the
// setup beside them, and 32 antennas x 5000 sources x 6 slices (twelve
// launches of the radix sort before) 138 -> 71 us a call.
__device__ __forceinline__ void rank_sort_block(const float* __restrict__ crd_eq,
                                                const float* __restrict__ I, int n,
                                                float* __restrict__ crd_s,
                                                float* __restrict__ I_s, int b, uint32_t* key) {
  const int ng = ceil_div(n, 4);
  for (int i = threadIdx.x; i < 4 * ng; i += kRankThreads)
    key[i] = (uint32_t)(sort_word(crd_eq, n, i) >> 32);
  __syncthreads();
  const int lane = threadIdx.x & 31, own = b * (kRankSources / 4) + (threadIdx.x >> 5);
  if (own >= ng) return;
  const uint4* key4 = reinterpret_cast<const uint4*>(key);
  const uint4 k0 = key4[own];
  const uint32_t mine[4] = {k0.x, k0.y, k0.z, k0.w};
  int c[4] = {0, 0, 0, 0};
  // equal keys before the sources at hand come before them
  int g = lane;
#pragma unroll 4
  for (; g < own; g += 32) {
    const uint4 k = key4[g];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      c[e] += (k.x <= mine[e]) + (k.y <= mine[e]) + (k.z <= mine[e]) + (k.w <= mine[e]);
  }
  if (g == own) g += 32;
  // those after them do not (nor does the padding, all ones)
#pragma unroll 4
  for (; g < ng; g += 32) {
    const uint4 k = key4[g];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      c[e] += (k.x < mine[e]) + (k.y < mine[e]) + (k.z < mine[e]) + (k.w < mine[e]);
  }
  int at = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    c[e] = __reduce_add_sync(0xffffffffu, c[e]);
#pragma unroll
    for (int q = 0; q < 4; ++q) c[e] += q < e ? mine[q] <= mine[e] : mine[q] < mine[e];
    at = lane == e ? c[e] : at;
  }
  const int i = 4 * own + lane;
  if (lane < 4 && i < n) {
    crd_s[at] = crd_eq[i];
    crd_s[(size_t)n + at] = crd_eq[(size_t)n + i];
    crd_s[2 * (size_t)n + at] = crd_eq[2 * (size_t)n + i];
    I_s[at] = I[i];
  }
}

}  // namespace hv
