// hv_median.cu -- the 2-D median filter of hera_gpu (MedianFilter).
//
// The reference (hera_gpu/median_filter.py:8-365) zero-pads every image by
// half the window on each side (median_filter.py:318), and for each pixel of
// the original image takes the element of rank floor(k0 * k1 / 2) of its
// k0 x k1 window (rows x columns; median_filter.py:223-257, FloydWirth_kth on
// a per-thread copy of the window), one image per stream.
//
// Here one launch covers every image of the call, with a kernel by window:
//  * 3 x 3 (median3x3_kernel), the other odd windows with sides up to 9, and
//    one-dimensional ones up to 11 (median_merge_kernel<H, W>): a warp slides
//    down a strip of columns with everything in registers, neighbouring
//    columns by shuffles;
//  * any other window of up to 81 elements (median_filter_kernel<K>): a block
//    of 8 x 32 output pixels stages its window tile -- (8 + k0 - 1) x (32 + k1
//    - 1) values, the zero padding included -- in shared memory, and each
//    thread keeps the k + 1 smallest keys sorted in registers, each window key
//    pushed through them by min/max pairs (2 (k + 1) integer ops per key);
//  * larger windows (K = 0): a most-significant-bit-first radix select, 32
//    counting passes over the keys in shared memory.
// Values are compared as order-preserving 32-bit keys, so the result is
// exactly the window's element of that rank (a selection, no arithmetic),
// NaN and signed zeros included.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>

#include "heravis.h"
#include "hv_kernels.h"

namespace {

constexpr int kMfCols = 32;  // output columns per block (a warp's lanes)
constexpr int kMfRows = 8;   // output rows per block
constexpr int kMfSmemLimit = 200 * 1024;

// Keys that order like the floats: negative values have every bit flipped,
// the others the sign bit set.
__device__ __forceinline__ uint32_t mf_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float mf_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// grid (ceil(cols / 32), ceil(rows / 8), nimg), block (32, 8); dynamic shared
// memory (8 + k0 - 1) * (32 + k1 - 1) keys.  K > 0: windows of at most 2 K - 1
// elements select with K registers; K == 0: radix select.
template <int K>
__global__ void __launch_bounds__(kMfCols * kMfRows)
median_filter_kernel(const float* __restrict__ in, float* __restrict__ out, int rows, int cols,
                     int k0, int k1) {
  extern __shared__ uint32_t tile[];
  const int tw = kMfCols + k1 - 1, th = kMfRows + k0 - 1;
  // tile origin in image coordinates (the window of pixel (r, c) starts at
  // (r - k0 / 2, c - k1 / 2), as the reference's padded image)
  const int r0 = (int)blockIdx.y * kMfRows - k0 / 2;
  const int c0 = (int)blockIdx.x * kMfCols - k1 / 2;
  const size_t plane = (size_t)rows * cols;
  const float* img = in + (size_t)blockIdx.z * plane;
  for (int i = (int)(threadIdx.y * kMfCols + threadIdx.x); i < tw * th; i += kMfCols * kMfRows) {
    const int r = r0 + i / tw, c = c0 + i % tw;
    const float v = (r >= 0 && r < rows && c >= 0 && c < cols) ? img[(size_t)r * cols + c] : 0.f;
    tile[i] = mf_key(v);
  }
  __syncthreads();
  const int r = (int)(blockIdx.y * kMfRows + threadIdx.y), c = (int)(blockIdx.x * kMfCols + threadIdx.x);
  if (r >= rows || c >= cols) return;
  const uint32_t* win = tile + threadIdx.y * tw + threadIdx.x;
  const int rank = (k0 * k1) / 2;
  if (K > 0) {
    // s[0..K) holds the smallest keys seen so far, ascending; a new key
    // sinks to its place and the largest falls out
    uint32_t sm[K > 0 ? K : 1];
#pragma unroll
    for (int q = 0; q < K; ++q) sm[q] = 0xffffffffu;
    for (int i = 0; i < k0; ++i) {
      const uint32_t* row = win + i * tw;
      for (int j = 0; j < k1; ++j) {
        uint32_t v = row[j];
#pragma unroll
        for (int q = 0; q < K; ++q) {
          const uint32_t lo = min(sm[q], v);
          v = max(sm[q], v);
          sm[q] = lo;
        }
      }
    }
    // rank <= K - 1: pick sm[rank] without dynamic indexing
    uint32_t key = sm[0];
#pragma unroll
    for (int q = 1; q < K; ++q) key = q == rank ? sm[q] : key;
    out[(size_t)blockIdx.z * plane + (size_t)r * cols + c] = mf_value(key);
    return;
  }
  // radix select of the rank-k key, most significant bit first: at bit b
  // the candidates share `prefix` above b; count those with bit b clear
  int left = rank;
  uint32_t prefix = 0;
#pragma unroll 1
  for (int b = 31; b >= 0; --b) {
    const uint32_t bit = 1u << b;
    const uint32_t mask = ~(bit - 1u);  // bits b..31
    int cnt = 0;
#pragma unroll 1
    for (int i = 0; i < k0; ++i) {
      const uint32_t* row = win + i * tw;
#pragma unroll 4
      for (int j = 0; j < k1; ++j) cnt += (row[j] & mask) == prefix;
    }
    if (left >= cnt) {
      left -= cnt;
      prefix |= bit;
    }
  }
  out[(size_t)blockIdx.z * plane + (size_t)r * cols + c] = mf_value(prefix);
}

// ------------------------------------------------------- strip kernels ----
// Signed keys that order like the floats (a negative value has its other bits
// flipped); the map is its own inverse, and 0.0f, the padding, is key 0.
__device__ __forceinline__ int sm_key(float x) {
  const int u = __float_as_int(x);
  return u ^ ((u >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float sm_value(int k) {
  return __int_as_float(k ^ ((k >> 31) & 0x7fffffff));
}
__device__ __forceinline__ int med3(int a, int b, int c) {
  return max(min(a, b), min(max(a, b), c));
}

constexpr int kStripWarps = 4;  // warps a block, each with its own strip or rows
// Output rows a warp takes, at most (8 and 32 were slower for one window or
// another at full size); fewer, down to 2, while that leaves fewer warps than
// kStripFill: an image of 100 x 100 is bound by its warps' serial rows.
constexpr int kStripRows = 16, kStripFill = 152 * 8;

// The strip of a warp: warps of consecutive index take consecutive strips of
// the same rows.
__device__ __forceinline__ bool strip_of_warp(int nstrips, int rows, int take, int& strip,
                                              int& row0) {
  const long long w = (long long)blockIdx.x * kStripWarps + (threadIdx.x >> 5);
  strip = (int)(w % nstrips);
  const long long r = w / nstrips * take;
  row0 = (int)r;
  return r < rows;
}

// The 3 x 3 window (the reference's default): with each window column sorted
// into (lo, mid, hi), the median of the nine is med3(max of the three lo, med3
// of the three mid, min of the three hi), an exact selection.  A lane holds 4
// columns (one 128-bit load a row, the next pair of rows loaded before the
// present one is worked on) and gets the columns beside them from its
// neighbours; rows go in pairs, sorted once for the two output rows that share
// them: about 19 min/max a pixel.  Bound by those and HBM (8 B a pixel).
// Measured on GB300, 7000 x 7000: 0.188 ms with blocks that staged a tile in
// shared memory and synchronised, 0.094 ms now (4.2 TB/s, 0.61 of the copy
// rate; the min/max issue rate is the other bound).
// vec: rows start 16-byte aligned in both images (cols % 4 == 0 and aligned
// bases).
struct Row4 {
  float4 v;
  float edge;  // lane 0: the column to the left; lane 31: to the right
};
template <bool kVec>
__device__ __forceinline__ Row4 load_row4(const float* __restrict__ img, int r, int rows, int cols,
                                          int c, int lane) {
  Row4 x{make_float4(0.f, 0.f, 0.f, 0.f), 0.f};
  if (r < 0 || r >= rows) return x;
  const float* p = img + (size_t)r * cols + c;
  if (kVec) {
    if (c < cols) x.v = *reinterpret_cast<const float4*>(p);
  } else {
    if (c < cols) x.v.x = p[0];
    if (c + 1 < cols) x.v.y = p[1];
    if (c + 2 < cols) x.v.z = p[2];
    if (c + 3 < cols) x.v.w = p[3];
  }
  if (lane == 0 && c > 0) x.edge = p[-1];
  if (lane == 31 && c + 4 < cols) x.edge = p[4];
  return x;
}
__device__ __forceinline__ void expand_row4(const Row4& x, int lane, int (&k)[6]) {
  k[1] = sm_key(x.v.x);
  k[2] = sm_key(x.v.y);
  k[3] = sm_key(x.v.z);
  k[4] = sm_key(x.v.w);
  k[0] = __shfl_up_sync(0xffffffffu, k[4], 1);
  k[5] = __shfl_down_sync(0xffffffffu, k[1], 1);
  const int e = sm_key(x.edge);
  if (lane == 0) k[0] = e;
  if (lane == 31) k[5] = e;
}

template <bool kVec>
__global__ void __launch_bounds__(kStripWarps * 32)
median3x3_kernel(const float* __restrict__ in, float* __restrict__ out, int rows, int cols,
                 int nstrips, int take) {
  int strip, row0;
  if (!strip_of_warp(nstrips, rows, take, strip, row0)) return;
  const int lane = threadIdx.x & 31, c = strip * 128 + 4 * lane;
  const size_t plane = (size_t)rows * cols;
  const float* img = in + (size_t)blockIdx.y * plane;
  float* dst = out + (size_t)blockIdx.y * plane;
  const int row1 = min(rows, row0 + take);
  int ka[6], kb[6];
  expand_row4(load_row4<kVec>(img, row0 - 1, rows, cols, c, lane), lane, ka);
  expand_row4(load_row4<kVec>(img, row0, rows, cols, c, lane), lane, kb);
  Row4 n0 = load_row4<kVec>(img, row0 + 1, rows, cols, c, lane);
  Row4 n1 = load_row4<kVec>(img, row0 + 2, rows, cols, c, lane);
  for (int r = row0; r < row1; r += 2) {
    int kc[6], kd[6];
    expand_row4(n0, lane, kc);
    expand_row4(n1, lane, kd);
    if (r + 2 < row1) {
      n0 = load_row4<kVec>(img, r + 3, rows, cols, c, lane);
      n1 = load_row4<kVec>(img, r + 4, rows, cols, c, lane);
    }
    // output rows r (input rows a b c) and r + 1 (b c d)
    int lo[2][6], md[2][6], hi[2][6];
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const int p = min(kb[j], kc[j]), q = max(kb[j], kc[j]);
#pragma unroll
      for (int o = 0; o < 2; ++o) {
        const int x = o ? kd[j] : ka[j];
        lo[o][j] = min(p, x);
        hi[o][j] = max(q, x);
        md[o][j] = max(p, min(q, x));
      }
      ka[j] = kc[j];
      kb[j] = kd[j];
    }
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      float v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int mx = max(max(lo[o][q], lo[o][q + 1]), lo[o][q + 2]);
        const int mn = min(min(hi[o][q], hi[o][q + 1]), hi[o][q + 2]);
        v[q] = sm_value(med3(mx, med3(md[o][q], md[o][q + 1], md[o][q + 2]), mn));
      }
      if (r + o < row1) {
        float* d = dst + (size_t)(r + o) * cols + c;
        if (kVec) {
          if (c < cols) *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (c + q < cols) d[q] = v[q];
        }
      }
    }
  }
}

// Sorted lists in registers.  merge() is Batcher's odd-even merge for lists of
// any two lengths (Knuth, The Art of Computer Programming 3, 5.3.4); every
// comparator is a separate min and max, so the compiler drops those that lead
// only to elements nobody reads.
template <int N>
struct List {
  int x[N > 0 ? N : 1];
};
template <int NA, int NB>
__device__ __forceinline__ List<NA + NB> merge(const List<NA>& a, const List<NB>& b) {
  List<NA + NB> o;
  if constexpr (NA == 0 || NB == 0) {
#pragma unroll
    for (int i = 0; i < NA; ++i) o.x[i] = a.x[i];
#pragma unroll
    for (int i = 0; i < NB; ++i) o.x[i] = b.x[i];
  } else if constexpr (NA == 1 && NB == 1) {
    o.x[0] = min(a.x[0], b.x[0]);
    o.x[1] = max(a.x[0], b.x[0]);
  } else {
    List<(NA + 1) / 2> ao;
    List<NA / 2> ae;
    List<(NB + 1) / 2> bo;
    List<NB / 2> be;
#pragma unroll
    for (int i = 0; i < NA; ++i) (i & 1 ? ae.x[i / 2] : ao.x[i / 2]) = a.x[i];
#pragma unroll
    for (int i = 0; i < NB; ++i) (i & 1 ? be.x[i / 2] : bo.x[i / 2]) = b.x[i];
    const auto v = merge(ao, bo);
    const auto w = merge(ae, be);
    constexpr int NV = (NA + 1) / 2 + (NB + 1) / 2, NW = NA / 2 + NB / 2;
    o.x[0] = v.x[0];
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      if (i + 1 < NV) {
        o.x[2 * i + 1] = min(w.x[i], v.x[i + 1]);
        o.x[2 * i + 2] = max(w.x[i], v.x[i + 1]);
      } else {
        o.x[2 * i + 1] = w.x[i];
      }
    }
    if constexpr (NV == NW + 2) o.x[NA + NB - 1] = v.x[NV - 1];
  }
  return o;
}
template <int N>
__device__ __forceinline__ List<N> sort(const int* a) {
  List<N> o;
  if constexpr (N == 1) {
    o.x[0] = a[0];
  } else {
    o = merge(sort<N / 2>(a), sort<N - N / 2>(a + N / 2));
  }
  return o;
}
template <int N>
__device__ __forceinline__ List<N> shift_down(const List<N>& a, int lanes) {
  List<N> o;
#pragma unroll
  for (int i = 0; i < N; ++i) o.x[i] = __shfl_down_sync(0xffffffffu, a.x[i], lanes);
  return o;
}

// Element of rank H of the union of a sorted middle list m (H + 1 elements)
// and a sorted column c (H): the smallest, over the splits of H + 1 elements
// between the lists, of the larger of the two last ones taken.
template <int H>
__device__ __forceinline__ int select_with(const List<H + 1>& m, const List<H>& c) {
  int best = m.x[H];
#pragma unroll
  for (int i = 1; i <= H; ++i) best = min(best, max(m.x[i - 1], c.x[H - i]));
  return best;
}

// Elements [kFirst, kFirst + N) of a sorted list.
template <int N, int kFirst, int NA>
__device__ __forceinline__ List<N> middle(const List<NA>& a) {
  List<N> o;
#pragma unroll
  for (int i = 0; i < N; ++i) o.x[i] = a.x[kFirst + i];
  return o;
}

// H x W windows, W odd: the two windows of a pair of neighbouring pixels share
// W - 1 columns, of whose sorted elements only H + 1, around the median's
// rank, can be a median once the H of the remaining column are known.  A lane
// sorts 2 columns and merges them; the W - 1 shared columns are (W - 1) / 2
// such pairs, its own and those of the lanes above it, merged in a tree whose
// inner nodes serve two lanes each.  Lane t, 1 <= t <= kPairs, then selects for
// its two pixels with one more column each, from the lanes t - 1 and t + (W -
// 1) / 2.  Bound by the min/max issue rate.  Measured on GB300 (before: a
// selection from scratch a pixel, n^2 / 2 min/max): two images of 2003 x 1501,
// 5 x 5, 131 us and 33 us; three of 1698 x 2276, 9 x 9, 2034 us and 180 us.
// W = 1 has no shared columns: a pixel's column alone.
template <int H, int W>
__global__ void __launch_bounds__(kStripWarps * 32, 4)
median_merge_kernel(const float* __restrict__ in, float* __restrict__ out, int rows, int cols,
                    int nstrips, int take) {
  static_assert(H % 2 == 1 && W % 2 == 1 && W <= 11, "odd windows");
  constexpr int kHalf = (W - 1) / 2;
  constexpr int kPairs = 31 - kHalf;
  constexpr int kLow = H * W / 2 - H;  // of the shared elements, ranks kLow .. kLow + H
  int strip, row0;
  if (!strip_of_warp(nstrips, rows, take, strip, row0)) return;
  const int lane = threadIdx.x & 31;
  const size_t plane = (size_t)rows * cols;
  const float* img = in + (size_t)blockIdx.y * plane;
  float* dst = out + (size_t)blockIdx.y * plane;
  // pixel pair of lane t: columns c, c + 1; the lane's window columns are
  // c - W / 2 + 1 and + 2
  const int c = strip * (2 * kPairs) + 2 * (lane - 1);
  const int x0 = c - W / 2 + 1;
  const bool in0 = x0 >= 0 && x0 < cols, in1 = x0 + 1 >= 0 && x0 + 1 < cols;
  const bool mine = lane >= 1 && lane <= kPairs;
  const int row1 = min(rows, row0 + take);
  int a[H], b[H];
  auto load = [&](int r, float& u, float& v) {
    u = v = 0.f;
    if (r < 0 || r >= rows) return;
    const float* p = img + (size_t)r * cols + x0;
    if (in0) u = p[0];
    if (in1) v = p[1];
  };
#pragma unroll
  for (int i = 0; i < H - 1; ++i) {
    float u, v;
    load(row0 - H / 2 + i, u, v);
    a[i + 1] = sm_key(u);
    b[i + 1] = sm_key(v);
  }
  float nu, nv;
  load(row0 - H / 2 + H - 1, nu, nv);
#pragma unroll 1
  for (int r = row0; r < row1; ++r) {
#pragma unroll
    for (int i = 0; i < H - 1; ++i) {
      a[i] = a[i + 1];
      b[i] = b[i + 1];
    }
    a[H - 1] = sm_key(nu);
    b[H - 1] = sm_key(nv);
    if (r + 1 < row1) load(r + 1 - H / 2 + H - 1, nu, nv);
    const List<H> sa = sort<H>(a), sb = sort<H>(b);
    int k0, k1;
    if constexpr (W == 1) {
      k0 = __shfl_up_sync(0xffffffffu, sb.x[H / 2], 1);
      k1 = sa.x[H / 2];
    } else {
      const auto p = merge(sa, sb);
      List<H + 1> m;
      if constexpr (W == 3) {
        m = middle<H + 1, kLow>(p);
      } else {
        const auto q = merge(p, shift_down(p, 1));
        if constexpr (W == 5) m = middle<H + 1, kLow>(q);
        else if constexpr (W == 7) m = middle<H + 1, kLow>(merge(q, shift_down(p, 2)));
        else if constexpr (W == 9) m = middle<H + 1, kLow>(merge(q, shift_down(q, 2)));
        else m = middle<H + 1, kLow>(merge(merge(q, shift_down(q, 2)), shift_down(p, 4)));
      }
      List<H> left;
#pragma unroll
      for (int i = 0; i < H; ++i) left.x[i] = __shfl_up_sync(0xffffffffu, sb.x[i], 1);
      k0 = select_with<H>(m, left);
      k1 = select_with<H>(m, shift_down(sa, kHalf));
    }
    const float v0 = sm_value(k0), v1 = sm_value(k1);
    if (mine) {
      float* d = dst + (size_t)r * cols + c;
      if (c < cols) d[0] = v0;
      if (c + 1 < cols) d[1] = v1;
    }
  }
}

// Rows a warp takes and the grid of a strip launch.
int strip_grid(int nstrips, int rows, int nimg, dim3* grid) {
  auto warps = [&](int take) { return (long long)nstrips * ((rows + take - 1) / take); };
  int take = kStripRows;
  while (take > 2 && warps(take) * nimg < kStripFill) take /= 2;
  *grid = dim3((unsigned)((warps(take) + kStripWarps - 1) / kStripWarps), nimg);
  return take;
}
template <int H, int W>
bool launch_merge(const float* d_in, float* d_out, int nimg, int rows, int cols, cudaStream_t st) {
  constexpr int kOut = 2 * (31 - (W - 1) / 2);
  const int nstrips = (cols + kOut - 1) / kOut;
  dim3 grid;
  const int take = strip_grid(nstrips, rows, nimg, &grid);
  median_merge_kernel<H, W><<<grid, kStripWarps * 32, 0, st>>>(d_in, d_out, rows, cols, nstrips,
                                                               take);
  return true;
}
template <int H>
bool launch_merge_w(const float* d_in, float* d_out, int nimg, int rows, int cols, int k1,
                    cudaStream_t st) {
  switch (k1) {
    case 1: return launch_merge<H, 1>(d_in, d_out, nimg, rows, cols, st);
    case 3: return launch_merge<H, 3>(d_in, d_out, nimg, rows, cols, st);
    case 5: return launch_merge<H, 5>(d_in, d_out, nimg, rows, cols, st);
    case 7: return launch_merge<H, 7>(d_in, d_out, nimg, rows, cols, st);
    case 9: return launch_merge<H, 9>(d_in, d_out, nimg, rows, cols, st);
    default: return false;
  }
}
// A strip kernel for the window, if it has one.
bool launch_strips(const float* d_in, float* d_out, int nimg, int rows, int cols, int k0, int k1,
                   cudaStream_t st) {
  if (k0 == 3 && k1 == 3) {
    const int nstrips = (cols + 127) / 128;
    dim3 grid;
    const int take = strip_grid(nstrips, rows, nimg, &grid);
    if ((cols & 3) == 0 &&
        ((reinterpret_cast<uintptr_t>(d_in) | reinterpret_cast<uintptr_t>(d_out)) & 15) == 0)
      median3x3_kernel<true><<<grid, kStripWarps * 32, 0, st>>>(d_in, d_out, rows, cols, nstrips,
                                                                take);
    else
      median3x3_kernel<false><<<grid, kStripWarps * 32, 0, st>>>(d_in, d_out, rows, cols, nstrips,
                                                                take);
    return true;
  }
  switch (k0) {
    case 1:
      if (k1 == 11) return launch_merge<1, 11>(d_in, d_out, nimg, rows, cols, st);
      return launch_merge_w<1>(d_in, d_out, nimg, rows, cols, k1, st);
    case 3: return launch_merge_w<3>(d_in, d_out, nimg, rows, cols, k1, st);
    case 5: return launch_merge_w<5>(d_in, d_out, nimg, rows, cols, k1, st);
    case 7: return launch_merge_w<7>(d_in, d_out, nimg, rows, cols, k1, st);
    case 9: return launch_merge_w<9>(d_in, d_out, nimg, rows, cols, k1, st);
    case 11: return k1 == 1 && launch_merge<11, 1>(d_in, d_out, nimg, rows, cols, st);
    default: return false;
  }
}

int check_args(hv_context* ctx, int nimg, int rows, int cols, int k0, int k1, size_t* smem) {
  char msg[256];
  if (nimg < 0 || rows < 0 || cols < 0 || k0 < 1 || k1 < 1 || nimg > 65535 ||
      (long long)rows > 65535LL * kMfRows) {
    snprintf(msg, sizeof msg, "median filter: bad sizes (images %d, %d x %d, window %d x %d)",
             nimg, rows, cols, k0, k1);
    if (ctx) hv_context_set_error(ctx, msg);
    return HV_ERR_ARG;
  }
  *smem = sizeof(uint32_t) * (size_t)(kMfRows + k0 - 1) * (kMfCols + k1 - 1);
  if (*smem > (size_t)kMfSmemLimit) {
    snprintf(msg, sizeof msg, "median filter: a %d x %d window needs %zu bytes of shared memory "
             "per block (at most %d)", k0, k1, *smem, kMfSmemLimit);
    if (ctx) hv_context_set_error(ctx, msg);
    return HV_ERR_ARG;
  }
  return HV_OK;
}

int launch(hv_context* ctx, const float* d_in, float* d_out, int nimg, int rows, int cols, int k0,
           int k1, cudaStream_t st) {
  size_t smem = 0;
  int r = check_args(ctx, nimg, rows, cols, k0, k1, &smem);
  if (r != HV_OK) return r;
  if ((size_t)nimg * rows * cols == 0) return HV_OK;
  static bool configured = false;
  if (!configured) {
    for (const void* k : {reinterpret_cast<const void*>(median_filter_kernel<0>),
                          reinterpret_cast<const void*>(median_filter_kernel<5>),
                          reinterpret_cast<const void*>(median_filter_kernel<13>),
                          reinterpret_cast<const void*>(median_filter_kernel<25>),
                          reinterpret_cast<const void*>(median_filter_kernel<41>)})
      if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMfSmemLimit) !=
          cudaSuccess)
        return HV_ERR_CUDA;
    configured = true;
  }
  const dim3 grid((cols + kMfCols - 1) / kMfCols, (rows + kMfRows - 1) / kMfRows, nimg);
  const dim3 block(kMfCols, kMfRows);
  const int n = k0 * k1;  // the register form needs n / 2 + 1 <= K
  if (launch_strips(d_in, d_out, nimg, rows, cols, k0, k1, st)) {
  } else if (n <= 9) median_filter_kernel<5><<<grid, block, smem, st>>>(d_in, d_out, rows, cols, k0, k1);
  else if (n <= 25) median_filter_kernel<13><<<grid, block, smem, st>>>(d_in, d_out, rows, cols, k0, k1);
  else if (n <= 49) median_filter_kernel<25><<<grid, block, smem, st>>>(d_in, d_out, rows, cols, k0, k1);
  else if (n <= 81) median_filter_kernel<41><<<grid, block, smem, st>>>(d_in, d_out, rows, cols, k0, k1);
  else median_filter_kernel<0><<<grid, block, smem, st>>>(d_in, d_out, rows, cols, k0, k1);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    if (ctx) hv_context_set_error(ctx, cudaGetErrorString(e));
    return HV_ERR_CUDA;
  }
  hv_context_add_launches(ctx, 1);
  return HV_OK;
}

}  // namespace

extern "C" {

int hv_median_filter_device(hv_context* ctx, const float* d_in, float* d_out, int nimg, int rows,
                            int cols, int k0, int k1, void* stream) {
  const bool empty = nimg <= 0 || rows <= 0 || cols <= 0;
  if (!ctx || (!empty && (!d_in || !d_out))) return HV_ERR_ARG;
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : hv_context_stream(ctx);
  return launch(ctx, d_in, d_out, nimg, rows, cols, k0, k1, st);
}

int hv_median_filter(hv_context* ctx, const float* in, float* out, int nimg, int rows, int cols,
                     int k0, int k1) {
  if (!ctx) return HV_ERR_ARG;
  size_t smem = 0;
  int r = check_args(ctx, nimg, rows, cols, k0, k1, &smem);
  if (r != HV_OK) return r;
  const size_t bytes = sizeof(float) * (size_t)nimg * rows * cols;
  if (bytes == 0) return HV_OK;
  if (!in || !out) return HV_ERR_ARG;
  cudaStream_t st = hv_context_stream(ctx);
  void *d_in = nullptr, *d_out = nullptr;
  if (hv_context_malloc(ctx, &d_in, bytes, st) != cudaSuccess ||
      hv_context_malloc(ctx, &d_out, bytes, st) != cudaSuccess) {
    cudaGetLastError();
    if (d_in) cudaFreeAsync(d_in, st);
    hv_context_set_error(ctx, "median filter: device allocation failed");
    return HV_ERR_OOM;
  }
  r = HV_OK;
  if (cudaMemcpyAsync(d_in, in, bytes, cudaMemcpyHostToDevice, st) != cudaSuccess) r = HV_ERR_CUDA;
  if (r == HV_OK)
    r = launch(ctx, static_cast<const float*>(d_in), static_cast<float*>(d_out), nimg, rows,
               cols, k0, k1, st);
  if (r == HV_OK &&
      cudaMemcpyAsync(out, d_out, bytes, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    r = HV_ERR_CUDA;
  cudaFreeAsync(d_in, st);
  cudaFreeAsync(d_out, st);
  if (cudaStreamSynchronize(st) != cudaSuccess && r == HV_OK) r = HV_ERR_CUDA;
  return r;
}

}  // extern "C"
