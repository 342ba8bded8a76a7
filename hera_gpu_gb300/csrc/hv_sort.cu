// hv_sort.cu -- spatial ordering of the source catalogue for the fused path.
//
// The visibility sum is over sources, so their order is free.  Putting
// sources that are close on the sky next to each other makes the 32 sources
// of a pipeline stage fall on the same few beam pixels: the beam gathers of a
// stage hit L1, and the phase of a source can be taken relative to a nearby
// reference source.  Rotation to topocentric is an isometry, so an order
// that is local on the equatorial sphere stays local at every time.
//
// Sort: by the words (key << 32 | index) of hv_spatial.cuh -- a total order, so
// the permutation (and every result downstream) is deterministic -- with a
// radix sort for one catalogue (one of at most kRankSort sources is ordered by
// counting, among the call's setup) and a segmented bitonic network for a
// batch.
#include <algorithm>
#include <utility>

#include "hv_internal.cuh"
#include "hv_kernels.h"
#include "hv_spatial.cuh"

namespace hv {

// -------------------------------------------------------- single call ----
// Least-significant-digit radix sort of the words by key, four stable passes
// of 8 bits, so that equal keys keep their index order: the order of the
// (key, index) words.  It is bound by launches and latency (a 1M-source
// catalogue is 8 MB).  Measured on GB300 under ncu, gather included: 139 us
// at 1M sources (12 launches), 71 us at 100k.  A bitonic network of the words
// took 444 us (57 launches) and 138 us.
constexpr int kRadixTile = 2048;   // words a block, 8 a thread
constexpr int kRadixThreads = 256;

// Stable ranks within a warp's row of 32 digits: the lanes of the same digit
// (match) take consecutive ranks from the warp's counter of that digit.
__device__ __forceinline__ int radix_rank(int* cnt, int digit, bool valid) {
  const unsigned peers = __match_any_sync(0xffffffffu, valid ? digit : -1);
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  int base = 0;
  if (valid && lane == leader) {
    base = cnt[digit];
    cnt[digit] = base + __popc(peers);
  }
  __syncwarp();
  return __shfl_sync(0xffffffffu, base, leader) + __popc(peers & ((1u << lane) - 1u));
}

// Exclusive prefix over the first 256 threads' values (every thread of the
// block calls; ws: 8 ints of shared memory).
__device__ __forceinline__ int prefix256(int v, int* ws) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (warp < 8 && lane == 31) ws[warp] = incl;
  __syncthreads();
  int base = 0;
  for (int w = 0; w < 8; ++w) base += w < warp ? ws[w] : 0;
  return base + incl - v;
}

// Counts of one digit per block: table[digit][block].  The first pass makes
// the words.
template <bool kFirst>
__global__ void __launch_bounds__(kRadixThreads)
radix_count_kernel(const float* __restrict__ crd_eq, int n, unsigned long long* __restrict__ kv,
                   int shift, int* __restrict__ table) {
  __shared__ int h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * kRadixTile;
#pragma unroll
  for (int q = 0; q < kRadixTile / kRadixThreads; ++q) {
    const long long i = base + q * kRadixThreads + threadIdx.x;
    if (i < n) {
      unsigned long long w;
      if (kFirst) {
        w = sort_word(crd_eq, n, (int)i);
        kv[i] = w;
      } else {
        w = kv[i];
      }
      atomicAdd(&h[(int)(w >> shift) & 255], 1);
    }
  }
  __syncthreads();
  table[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

// Row d of the table to its exclusive prefix over the blocks, its sum to
// totals[d] (one block a digit).
__global__ void __launch_bounds__(256)
radix_scan_kernel(int* __restrict__ table, int nblk, int* __restrict__ totals) {
  __shared__ int ws[8];
  __shared__ int carry;
  int* row = table + (size_t)blockIdx.x * nblk;
  if (threadIdx.x == 0) carry = 0;
  for (int b0 = 0; b0 < nblk; b0 += 256) {
    const int b = b0 + threadIdx.x;
    const int v = b < nblk ? row[b] : 0;
    __syncthreads();  // ws and carry of the last round
    const int c = carry;
    const int pre = prefix256(v, ws);
    if (b < nblk) row[b] = c + pre;
    __syncthreads();
    if (threadIdx.x == 255) carry = c + pre + v;
  }
  __syncthreads();
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// The words of a block to their places; the last pass gathers the catalogue
// there instead.
template <bool kLast>
__global__ void __launch_bounds__(kRadixThreads)
radix_scatter_kernel(const unsigned long long* __restrict__ src, int n, int shift,
                     const int* __restrict__ table, const int* __restrict__ totals,
                     unsigned long long* __restrict__ dst, const float* __restrict__ crd_eq,
                     const float* __restrict__ I, float* __restrict__ crd_s,
                     float* __restrict__ I_s) {
  constexpr int W = kRadixThreads / 32, R = kRadixTile / kRadixThreads;
  __shared__ int cnt[W][256];
  __shared__ int ws[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int w = 0; w < W; ++w) cnt[w][threadIdx.x] = 0;
  const int at = prefix256(totals[threadIdx.x], ws) +
                 table[(size_t)threadIdx.x * gridDim.x + blockIdx.x];
  __syncthreads();
  const long long base = (long long)blockIdx.x * kRadixTile + warp * (32 * R) + lane;
  unsigned long long w[R];
  int rank[R];
#pragma unroll
  for (int r = 0; r < R; ++r) w[r] = base + r * 32 < n ? src[base + r * 32] : 0ull;
#pragma unroll
  for (int r = 0; r < R; ++r)
    rank[r] = radix_rank(cnt[warp], (int)(w[r] >> shift) & 255, base + r * 32 < n);
  __syncthreads();
  {
    int run = at;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const int c = cnt[k][threadIdx.x];
      cnt[k][threadIdx.x] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (base + r * 32 >= n) continue;
    const int pos = cnt[warp][(int)(w[r] >> shift) & 255] + rank[r];
    if (kLast) {
      const uint32_t i = (uint32_t)w[r];
      crd_s[pos] = crd_eq[i];
      crd_s[(size_t)n + pos] = crd_eq[(size_t)n + i];
      crd_s[2 * (size_t)n + pos] = crd_eq[2 * (size_t)n + i];
      I_s[pos] = I[i];
    } else {
      dst[pos] = w[r];
    }
  }
}

size_t sort_table_bytes(int nsrc) {
  return nsrc <= kRankSort ? 0
                            : sizeof(int) * 256 * ((size_t)ceil_div(nsrc, kRadixTile) + 1);
}

cudaError_t launch_sort_sources(const float* crd_eq, const float* I_sky, int nsrc, void* kv_buf,
                                void* table_buf, float* crd_sorted, float* I_sorted,
                                int* launches, cudaStream_t st) {
  // the words go back and forth between crd_sorted (12 bytes a source, not
  // written as such before the last pass, which reads kv) and kv
  auto* a = reinterpret_cast<unsigned long long*>(crd_sorted);
  auto* b = static_cast<unsigned long long*>(kv_buf);
  const int nblk = ceil_div(nsrc, kRadixTile);
  int* table = static_cast<int*>(table_buf);
  int* totals = table + (size_t)256 * nblk;
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 32 + 8 * pass;
    if (pass == 0)
      radix_count_kernel<true><<<nblk, kRadixThreads, 0, st>>>(crd_eq, nsrc, a, shift, table);
    else
      radix_count_kernel<false><<<nblk, kRadixThreads, 0, st>>>(crd_eq, nsrc, a, shift, table);
    radix_scan_kernel<<<256, 256, 0, st>>>(table, nblk, totals);
    if (pass < 3)
      radix_scatter_kernel<false><<<nblk, kRadixThreads, 0, st>>>(
          a, nsrc, shift, table, totals, b, nullptr, nullptr, nullptr, nullptr);
    else
      radix_scatter_kernel<true><<<nblk, kRadixThreads, 0, st>>>(
          a, nsrc, shift, table, totals, nullptr, crd_eq, I_sky, crd_sorted, I_sorted);
    std::swap(a, b);
  }
  if (launches) *launches = 12;
  return cudaGetLastError();
}

// ------------------------------------------------------------ batches ----
constexpr int kSortTile = 2048;  // elements sorted in shared memory per block

// Every simulation of a batch sorted in one set of launches: simulation s
// owns a segment of sort_pad(S_s) words (its own kv buffer), and each pass
// of a bitonic network runs within every segment long enough for it, so a
// simulation's order is exactly the one it gets alone.
__global__ void sort_keys_batch_kernel(const PrepSim* __restrict__ sims, int nsims,
                                       const long long* __restrict__ pre, long long total) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int si = find_segment(pre, nsims, e);
    const PrepSim& sm = sims[si];
    const int l = (int)(e - __ldg(pre + si));
    sm.kv[l] = sort_word(sm.crd_eq, sm.S, l);
  }
}

__global__ void bitonic_global_batch_kernel(const PrepSim* __restrict__ sims, int nsims,
                                            const long long* __restrict__ pre, long long total,
                                            int j, int k) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int si = find_segment(pre, nsims, e);
    const long long n = 2 * (__ldg(pre + si + 1) - __ldg(pre + si));
    if ((long long)k > n) continue;  // this segment is sorted already
    unsigned long long* kv = sims[si].kv;
    const int i = (int)(e - __ldg(pre + si));
    const int lo = ((i / j) * 2 * j) + (i % j);
    const int hi = lo + j;
    const bool up = (lo & k) == 0;
    const unsigned long long a = kv[lo], b = kv[hi];
    if ((a > b) == up) {
      kv[lo] = b;
      kv[hi] = a;
    }
  }
}

__global__ void __launch_bounds__(1024)
bitonic_shared_batch_kernel(const PrepSim* __restrict__ sims, int nsims,
                            const long long* __restrict__ pre, int k0, int k1) {
  __shared__ unsigned long long s[kSortTile];
  const int si = find_segment(pre, nsims, blockIdx.x);
  const long long n = (long long)kSortTile * (__ldg(pre + si + 1) - __ldg(pre + si));
  if ((long long)k0 > n) return;  // the whole block: one segment
  unsigned long long* kv = sims[si].kv;
  const size_t base = (size_t)(blockIdx.x - __ldg(pre + si)) * kSortTile;
  s[threadIdx.x] = kv[base + threadIdx.x];
  s[threadIdx.x + 1024] = kv[base + threadIdx.x + 1024];
  __syncthreads();
  const int kmax = (int)min((long long)k1, n);
  for (int k = k0; k <= kmax; k <<= 1) {
    for (int j = min(k / 2, kSortTile / 2); j > 0; j >>= 1) {
      const int t = threadIdx.x;
      const int lo = ((t / j) * 2 * j) + (t % j);
      const int hi = lo + j;
      const bool up = ((base + lo) & (size_t)k) == 0;
      const unsigned long long a = s[lo], b = s[hi];
      if ((a > b) == up) {
        s[lo] = b;
        s[hi] = a;
      }
      __syncthreads();
    }
  }
  kv[base + threadIdx.x] = s[threadIdx.x];
  kv[base + threadIdx.x + 1024] = s[threadIdx.x + 1024];
}

__global__ void gather_sorted_batch_kernel(const PrepSim* __restrict__ sims, int nsims,
                                           const long long* __restrict__ pre, long long total) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int si = find_segment(pre, nsims, e);
    const PrepSim& sm = sims[si];
    const int i = (int)(e - __ldg(pre + si));
    if (i >= sm.S) continue;
    const uint32_t src = (uint32_t)(sm.kv[i] & 0xffffffffu);
    const size_t S = (size_t)sm.S;
    sm.crd_s[i] = sm.crd_eq[src];
    sm.crd_s[S + i] = sm.crd_eq[S + src];
    sm.crd_s[2 * S + i] = sm.crd_eq[2 * S + src];
    sm.I_s[i] = sm.I_sky[src];
  }
}

cudaError_t launch_sort_batch(const PrepSim* sims, int nsims, const PrepPre& pre,
                              const PrepTotals& tot, int* launches, cudaStream_t st) {
  int nl = 0;
  const int gk = (int)std::min<long long>((tot.key + 255) / 256, 152 * 16);
  const int gp = (int)std::min<long long>((tot.pair + 255) / 256, 152 * 16);
  sort_keys_batch_kernel<<<gk, 256, 0, st>>>(sims, nsims, pre.key, tot.key);
  ++nl;
  bitonic_shared_batch_kernel<<<(unsigned)tot.tile, 1024, 0, st>>>(sims, nsims, pre.tile, 2,
                                                                    kSortTile);
  ++nl;
  for (int k = 2 * kSortTile; k <= tot.max_key; k <<= 1) {
    for (int j = k / 2; j >= kSortTile; j >>= 1) {
      bitonic_global_batch_kernel<<<gp, 256, 0, st>>>(sims, nsims, pre.pair, tot.pair, j, k);
      ++nl;
    }
    bitonic_shared_batch_kernel<<<(unsigned)tot.tile, 1024, 0, st>>>(sims, nsims, pre.tile, k, k);
    ++nl;
  }
  gather_sorted_batch_kernel<<<gk, 256, 0, st>>>(sims, nsims, pre.key, tot.key);
  ++nl;
  if (launches) *launches = nl;
  return cudaGetLastError();
}

int sort_pad(int nsrc) {
  int n = kSortTile;
  while (n < nsrc) n <<= 1;
  return n;
}

}  // namespace hv
