// hv_plain.cu -- the plain form of the hot path: the reference's method
// (hera_gpu/vis.py:224-250) with its bugs removed.
//
//   gen_phasors : v[s][a] = A_a(l_s, m_s) sqrt(I_s) exp(2 pi i U_a . s)
//                 (InterpolateBeam + MeasEq, vis.py:46-110) written to HBM.
//   herk_plain  : V[a][b] = sum_s v[a,s] conj(v[b,s]) on the upper triangle
//                 only, FP32 (precision 1) or FP64 (precision 2, where the
//                 tensor-core product of hv_f64.cu does not apply) FMA on the
//                 CUDA cores; the reference runs a full CGEMM/ZGEMM
//                 (vis.py:246-249).  Sources are split into chunks of
//                 kPlainChunk; each chunk's partial sum is stored.
//   reduce      : sums the chunk partials in a fixed order (compensated in
//                 FP32) and writes the full Hermitian matrix, replacing the
//                 host-side sum over chunks of vis.py:258.
#include <algorithm>

#include "hv_internal.cuh"
#include "hv_kernels.h"

namespace hv {

// ------------------------------------------------------------ phasors ----
__device__ __forceinline__ float2 make_phasor(const SrcRec32& r, const Ucoef32& u, float A) {
  return phasor32(r, u, A);
}
__device__ __forceinline__ double2 make_phasor(const SrcRec64& r, const Ucoef64& u, double A) {
  return phasor64(r, u, A);
}

// A warp generates `span` sources for 32 antennas, whose coefficients stay in
// its registers.  Slice z of the launch: time z / nf, frequency z % nf.
template <typename R>
__global__ void __launch_bounds__(256)
gen_phasors_kernel(const PlainDims d, int span, const typename Traits<R>::Rec* __restrict__ rec,
                   const typename Traits<R>::U* __restrict__ U, const R* __restrict__ beamT,
                   int PP, int dx, int dy, typename Traits<R>::C* __restrict__ v) {
  using C = typename Traits<R>::C;
  const int z = blockIdx.y, tl = z / d.nf, f = z % d.nf;
  const int n = d.counts[tl];
  const int groups = d.Np / 32;
  const long long job = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const long long s0 = job / groups * span;
  if (s0 >= n) return;
  const int a = (int)(job % groups) * 32 + (threadIdx.x & 31);
  const typename Traits<R>::U u = U[((size_t)tl * d.u_nf + f) * d.Np + a];
  const R* beam = beamT + (size_t)f * PP * d.Np;
  rec += (size_t)tl * d.rec_stride;
  v += (size_t)z * d.v_stride + a;
  const int s1 = (int)min((long long)n, s0 + span);
#pragma unroll 2
  for (int s = (int)s0; s < s1; ++s) {
    C val;
    val.x = R(0); val.y = R(0);
    if (a < d.nant) {
      const typename Traits<R>::Rec r = rec[s];
      val = make_phasor(r, u, beam_bilinear<R>(beam, d.Np, a, r, dx, dy));
    }
    v[(size_t)s * d.Np] = val;
  }
}

// Sources a warp takes at most; fewer while that leaves fewer warps than fill the
// GPU twice (half the sources are above the horizon; groups of padding hardly
// count), since they come one after the other: 4 antennas x 100 sources 66 us at
// 64, 5 at one; 350 x 20000 47 us at 64, 21 at 8, more again at 4.
constexpr int kGenSpan = 64, kGenFill = 2 * 152 * 64;

template <typename R>
cudaError_t launch_gen_phasors(const PlainDims& d, int nz, const void* rec, int nsrc_max,
                               const void* U, const R* beamT, int P, void* v, cudaStream_t st) {
  const int dx = P > 1 ? 1 : 0, dy = P > 1 ? P : 0;
  const int nsrc = std::max(nsrc_max, 1);
  auto jobs = [&](int span) { return (long long)ceil_div(nsrc, span) * (d.Np / 32); };
  int span = kGenSpan;
  while (span > 1 && (long long)ceil_div(nsrc, span) * ceil_div(d.nant, 32) * nz < kGenFill)
    span /= 2;
  gen_phasors_kernel<R><<<dim3((unsigned)((jobs(span) + 7) / 8), nz), 256, 0, st>>>(
      d, span, reinterpret_cast<const typename Traits<R>::Rec*>(rec),
      reinterpret_cast<const typename Traits<R>::U*>(U), beamT, P * P, dx, dy,
      reinterpret_cast<typename Traits<R>::C*>(v));
  return cudaGetLastError();
}

// ---------------------------------------------------------- SIMT herk ----
constexpr int kHT = 64;   // output tile (antennas) per CTA edge
constexpr int kHK = 16;   // sources per smem stage

__device__ __forceinline__ void decode_upper(int t, int nb, int& I, int& J) {
  I = 0;
  while (t >= nb - I) { t -= nb - I; ++I; }
  J = I + t;
}

// One tile of a chunk, 4 x 4 outputs a thread.  FP64: bound by the FP64 pipe (2 FMA
// a clock and SM).  FP32: each stage of 16 sources is summed from zero, as in
// herk_plain_kernel, whose bits it gives; for launches of few blocks.
template <typename R>
__device__ __forceinline__ void herk_tile(const typename Traits<R>::C* __restrict__ v, int n,
                                          int Np, R* __restrict__ partial) {
  using C = typename Traits<R>::C;
  constexpr bool kTwoLevel = sizeof(R) == 4;
  const int s0 = blockIdx.y * kPlainChunk;
  if (s0 >= n) return;
  const int s1 = min(s0 + kPlainChunk, n);
  int I, J;
  decode_upper(blockIdx.x, Np / kHT, I, J);

  __shared__ __align__(16) C As[kHK][kHT];
  __shared__ __align__(16) C Bs[kHK][kHT];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  R acc_re[4][4], acc_im[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc_re[i][j] = acc_im[i][j] = R(0);

  const C* vA = v + (size_t)I * kHT;
  const C* vB = v + (size_t)J * kHT;
  C ra[4], rb[4];
  auto gload = [&](int s) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = threadIdx.x + q * 256;
      const int k = idx >> 6, c = idx & 63;
      const bool ok = s + k < s1;
      C z; z.x = R(0); z.y = R(0);
      ra[q] = ok ? vA[(size_t)(s + k) * Np + c] : z;
      rb[q] = ok ? vB[(size_t)(s + k) * Np + c] : z;
    }
  };
  gload(s0);
  for (int s = s0; s < s1; s += kHK) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int idx = threadIdx.x + q * 256;
      As[idx >> 6][idx & 63] = ra[q];
      Bs[idx >> 6][idx & 63] = rb[q];
    }
    __syncthreads();
    if (s + kHK < s1) gload(s + kHK);
    R st_re[4][4], st_im[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        st_re[i][j] = kTwoLevel ? R(0) : acc_re[i][j];
        st_im[i][j] = kTwoLevel ? R(0) : acc_im[i][j];
      }
#pragma unroll
    for (int k = 0; k < kHK; ++k) {
      C a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // v_a conj(v_b) = (ar br + ai bi) + i (ai br - ar bi)
          st_re[i][j] = fma(a[i].x, b[j].x, fma(a[i].y, b[j].y, st_re[i][j]));
          st_im[i][j] = fma(a[i].y, b[j].x, fma(-a[i].x, b[j].y, st_im[i][j]));
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc_re[i][j] = kTwoLevel ? acc_re[i][j] + st_re[i][j] : st_re[i][j];
        acc_im[i][j] = kTwoLevel ? acc_im[i][j] + st_im[i][j] : st_im[i][j];
      }
    __syncthreads();
  }
  R* pre = partial + (size_t)blockIdx.y * 2 * Np * Np;
  R* pim = pre + (size_t)Np * Np;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int b = J * kHT + tx * 4 + j;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int a = I * kHT + ty * 4 + i;
      pre[(size_t)b * Np + a] = acc_re[i][j];
      pim[(size_t)b * Np + a] = acc_im[i][j];
    }
  }
}

// Pairs of FP32 values in one 64-bit register, combined by the packed FMA
// (two of them a lane and instruction, each rounded as a scalar one).
using F2 = unsigned long long;
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 pack2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float half2(F2 v, int h) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
  return h ? hi : lo;
}

// FP32: a 64 x 64 tile of a chunk, 4 (rows a) x 4 (columns b) outputs a thread.
// Bound by the FMA pipe and by the shared-memory reads that feed it.  The
// columns' values are kept as separate real and imaginary arrays, read as
// pairs without bank conflicts; the rows' values doubled (ar ar ai ai), so that
// a packed FMA takes them as they come (a warp reads only two distinct ones at
// a time, a broadcast).  Two buffers, one barrier a stage of 16 sources.  Each
// stage is summed from zero and added to the running total, so the total's
// rounding walks over kPlainChunk / 16 additions instead of kPlainChunk (about
// 4x less error at the same chunk).  Measured on GB300, 350 antennas x 50k
// sources (ncu): scalar FMAs on interleaved complex values, whose column reads
// had two-way bank conflicts, 872 us a slice; now 792 us (43 TFLOP/s issued;
// scalar FMAs on this layout 930 us).
__global__ void __launch_bounds__(256, 2)
herk_plain_kernel(const PlainDims d, const float2* __restrict__ v_base,
                  float* __restrict__ partial) {
  const int z = blockIdx.z;
  const int n = d.counts[z / d.nf], Np = d.Np;
  const int s0 = blockIdx.y * kPlainChunk;
  if (s0 >= n) return;
  const int s1 = min(s0 + kPlainChunk, n);
  int I, J;
  decode_upper(blockIdx.x, Np / kHT, I, J);
  const float2* v = v_base + (size_t)z * d.v_stride;
  __shared__ __align__(16) float4 As[2][kHK][kHT];
  __shared__ __align__(16) float Br[2][kHK][kHT], Bi[2][kHK][kHT];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  F2 acc_re[4][2] = {}, acc_im[4][2] = {};
  const float2* vA = v + (size_t)I * kHT;
  const float2* vB = v + (size_t)J * kHT;
  const int c = threadIdx.x & 63, k0 = threadIdx.x >> 6;  // this thread loads sources k0 + 4 q
  float2 ra[4], rb[4];
  auto gload = [&](int s) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = s + k0 + 4 * q;
      const bool ok = k < s1;
      ra[q] = ok ? vA[(size_t)k * Np + c] : make_float2(0.f, 0.f);
      rb[q] = ok ? vB[(size_t)k * Np + c] : make_float2(0.f, 0.f);
    }
  };
  gload(s0);
  int buf = 0;
  const F2 minus = pack2(-1.f, -1.f);
  for (int s = s0; s < s1; s += kHK, buf ^= 1) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      As[buf][k0 + 4 * q][c] = make_float4(ra[q].x, ra[q].x, ra[q].y, ra[q].y);
      Br[buf][k0 + 4 * q][c] = rb[q].x;
      Bi[buf][k0 + 4 * q][c] = rb[q].y;
    }
    __syncthreads();  // (the other buffer's readers are past it before the next)
    if (s + kHK < s1) gload(s + kHK);
    F2 st_re[4][2] = {}, st_im[4][2] = {};
#pragma unroll
    for (int k = 0; k < kHK; ++k) {
      const ulonglong2 br = *reinterpret_cast<const ulonglong2*>(&Br[buf][k][tx * 4]);
      const ulonglong2 bi = *reinterpret_cast<const ulonglong2*>(&Bi[buf][k][tx * 4]);
      const F2 b_re[2] = {br.x, br.y}, b_im[2] = {bi.x, bi.y};
      const F2 b_ni[2] = {fma2(bi.x, minus, 0ull), fma2(bi.y, minus, 0ull)};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(&As[buf][k][ty * 4 + i]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          // v_a conj(v_b) = (ar br + ai bi) + i (ai br - ar bi)
          st_re[i][j] = fma2(a.x, b_re[j], fma2(a.y, b_im[j], st_re[i][j]));
          st_im[i][j] = fma2(a.y, b_re[j], fma2(a.x, b_ni[j], st_im[i][j]));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        acc_re[i][j] = add2(acc_re[i][j], st_re[i][j]);
        acc_im[i][j] = add2(acc_im[i][j], st_im[i][j]);
      }
  }
  float* pre = partial + (size_t)z * d.p_stride + (size_t)blockIdx.y * 2 * Np * Np +
               (size_t)(J * kHT + tx * 4) * Np + I * kHT + ty * 4;
  float* pim = pre + (size_t)Np * Np;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    *reinterpret_cast<float4*>(pre + (size_t)j * Np) =
        make_float4(half2(acc_re[0][j >> 1], j & 1), half2(acc_re[1][j >> 1], j & 1),
                    half2(acc_re[2][j >> 1], j & 1), half2(acc_re[3][j >> 1], j & 1));
    *reinterpret_cast<float4*>(pim + (size_t)j * Np) =
        make_float4(half2(acc_im[0][j >> 1], j & 1), half2(acc_im[1][j >> 1], j & 1),
                    half2(acc_im[2][j >> 1], j & 1), half2(acc_im[3][j >> 1], j & 1));
  }
}

template <typename R>
__global__ void __launch_bounds__(256)
herk_tile_kernel(const PlainDims d, const typename Traits<R>::C* __restrict__ v,
                 R* __restrict__ partial) {
  const int z = blockIdx.z;
  herk_tile<R>(v + (size_t)z * d.v_stride, d.counts[z / d.nf], d.Np,
               partial + (size_t)z * d.p_stride);
}

__global__ void __launch_bounds__(256)
herk_flagged_kernel(const F64Dims d, const double2* __restrict__ v,
                    const int* __restrict__ flags, double* __restrict__ partial,
                    size_t partial_stride) {
  const int z = blockIdx.z;
  if (!flags[z]) return;
  const int n = max(0, min(d.counts[z / d.nf] - d.s0, d.S));
  herk_tile<double>(v + (size_t)z * d.v_stride, n, d.Np, partial + (size_t)z * partial_stride);
}

cudaError_t launch_herk_flagged(const F64Dims& d, int nz, const void* v, const int* flags,
                                double* partial, size_t partial_stride, cudaStream_t st) {
  const int nb = d.Np / kHT;
  const dim3 grid(nb * (nb + 1) / 2, ceil_div(d.S, kPlainChunk), nz);
  herk_flagged_kernel<<<grid, 256, 0, st>>>(d, static_cast<const double2*>(v), flags, partial,
                                            partial_stride);
  return cudaGetLastError();
}

// FP32 launches whose blocks with sources (about half of the catalogue's chunks)
// are on the SMs at once, two each, take herk_tile, and launches of one or two
// slices that fill the SMs about twice: a packed block alone on its SM, or one of
// two, ends later (350 antennas x 20k sources x 4 slices 1058 us a call, packed,
// and 963; 512 x 8000 x 8 1050 and 964; 350 x 100k x 2 2024 and 1908), while a
// last wave that is half empty costs it less (700 x 5000 x 5 950 and 1104), and
// launches of more waves are even or faster packed.
constexpr int kHerkWave = 2 * 152;
bool herk_few(int tiles, int nsrc_max, int nz) {
  const long long blocks = (long long)tiles * ceil_div((nsrc_max + 1) / 2, kPlainChunk) * nz;
  return blocks <= kHerkWave ||
         (nz <= 2 && blocks > kHerkWave * 17 / 10 && blocks <= 2 * kHerkWave);
}

template <typename R>
cudaError_t launch_herk_plain(const PlainDims& d, int nz, const void* v, int nsrc_max, R* partial,
                              cudaStream_t st) {
  const int nb = d.Np / kHT;
  const dim3 grid(nb * (nb + 1) / 2, ceil_div(std::max(nsrc_max, 1), kPlainChunk), nz);
  if constexpr (sizeof(R) == 4) {
    if (!herk_few(grid.x, nsrc_max, nz)) {
      herk_plain_kernel<<<grid, 256, 0, st>>>(d, static_cast<const float2*>(v), partial);
      return cudaGetLastError();
    }
  }
  herk_tile_kernel<R><<<grid, 256, 0, st>>>(d, static_cast<const typename Traits<R>::C*>(v),
                                            partial);
  return cudaGetLastError();
}

// ------------------------------------------------------------- reduce ----
struct KahanF {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
};
struct SumD {
  double s = 0.0;
  __device__ __forceinline__ void add(double x) { s += x; }
};
template <typename R> struct Acc;
template <> struct Acc<float> { using type = KahanF; };
template <> struct Acc<double> { using type = SumD; };

// A slice's upper triangle is reduced in 32 x 32 tiles (row tile A <= column
// tile B) by blocks of 256 threads: block `part` of a tile takes kCols of its
// columns b and every row, kCols / 8 elements a thread.  An element is a
// serial compensated sum over the slice's chunks, so the kernel is bound by
// memory latency until enough loads are in flight: a thread loads
// kReduceAhead chunks (both planes) before it adds any of them.  With many
// chunks (single calls: tens to hundreds) a block takes a quarter of a tile,
// which spreads small arrays (one to a few tiles a slice) over the SMs; with
// few chunks a block takes a whole tile, since finding its place costs more
// than its loads.  Measured on GB300: 30 antennas x 25 slices x 204 chunks
// 437 us before (whole tiles, one chunk at a time), 29 us now; 350 antennas x
// 60 slices x 34 chunks 325 us and 176 us (1 GB of partial sums: 5.7 TB/s).
constexpr int kReduceAhead = 8;
// Chunks from which a tile is split over four blocks (at 512 antennas x 10
// slices x 2 chunks splitting it costs 10 us; from 34 chunks on it pays).
constexpr int kReduceSplitChunks = 8;
//
// kAntisym (the fused kernel's partial sums): in the diagonal pairs of its
// antenna blocks (block_rows antennas each) the imaginary plane holds M with Im V = M - M^T, so their blocks sum
// M's transposed part as well (read along its rows, handed over through TM).
template <typename R, int kCols, bool kAntisym>
__device__ __forceinline__ void reduce_part(const R* __restrict__ partial_base,
                                            size_t slice_stride, const int* __restrict__ counts,
                                            int nf, int t0, int ntimes_out, int chunk, int Np,
                                            int nant,
                                            typename Traits<R>::C* __restrict__ out_base,
                                            int block_rows, int tile, int part, int sl,
                                            typename Traits<R>::C (*T)[33], R (*TM)[33]) {
  using C = typename Traits<R>::C;
  const int nbt = ceil_div(nant, 32);
  int A, B;
  decode_upper(tile, nbt, A, B);
  const int b0 = B * 32 + part * kCols;
  if (b0 >= nant) return;
  const int tl = sl / nf, f = sl % nf;
  const R* partial = partial_base + (size_t)sl * slice_stride;
  C* out = out_base + ((size_t)f * ntimes_out + t0 + tl) * (size_t)nant * nant;
  const int n = counts[tl];
  const int nk = n > 0 ? ceil_div(n, chunk) : 0;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const size_t plane = (size_t)Np * Np;
  const int a = A * 32 + tx;
  const bool antisym = kAntisym && A / (block_rows / 32) == B / (block_rows / 32);
  if (antisym) {
#pragma unroll 1
    for (int i = threadIdx.x; i < 32 * kCols; i += 256) {
      const int aa = i / kCols, bb = i % kCols;
      const R* p = partial + plane + (size_t)(A * 32 + aa) * Np + b0 + bb;
      typename Acc<R>::type m;
      int k = 0;
      for (; k + kReduceAhead <= nk; k += kReduceAhead) {
        R x[kReduceAhead];
#pragma unroll
        for (int q = 0; q < kReduceAhead; ++q) x[q] = p[(size_t)(k + q) * 2 * plane];
#pragma unroll
        for (int q = 0; q < kReduceAhead; ++q) m.add(x[q]);
      }
      for (; k < nk; ++k) m.add(p[(size_t)k * 2 * plane]);
      TM[bb][aa] = m.s;
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int bb = ty; bb < kCols; bb += 8) {
    const int b = b0 + bb;
    typename Acc<R>::type re, im;
    // rows and columns past nant lie in the padding (Np is a multiple of
    // 128), so every lane loads and the loop's conditions are uniform
    const R* p = partial + (size_t)b * Np + a;
    int k = 0;
    for (; k + kReduceAhead <= nk; k += kReduceAhead) {
      R x[kReduceAhead], y[kReduceAhead];
#pragma unroll
      for (int q = 0; q < kReduceAhead; ++q) {
        x[q] = p[(size_t)(k + q) * 2 * plane];
        y[q] = p[(size_t)(k + q) * 2 * plane + plane];
      }
#pragma unroll
      for (int q = 0; q < kReduceAhead; ++q) {
        re.add(x[q]);
        im.add(y[q]);
      }
    }
    for (; k < nk; ++k) {
      re.add(p[(size_t)k * 2 * plane]);
      im.add(p[(size_t)k * 2 * plane + plane]);
    }
    C val;
    val.x = re.s;
    val.y = a == b ? R(0) : antisym ? im.s - TM[bb][tx] : im.s;
    T[bb][tx] = val;
    if (a <= b && b < nant) {
      // below the diagonal: out[b][a] = conj(V[a][b]), a contiguous
      val.y = a == b ? R(0) : -val.y;
      out[(size_t)b * nant + a] = val;
    }
  }
  __syncthreads();
  // above the diagonal: out[a][b], kCols consecutive b a row
#pragma unroll
  for (int i = threadIdx.x; i < 32 * kCols; i += 256) {
    const int aa = i / kCols, bb = i % kCols;
    const int ao = A * 32 + aa, bo = b0 + bb;
    if (ao < bo && bo < nant) out[(size_t)ao * nant + bo] = T[bb][aa];
  }
}

template <typename R, int kCols, bool kAntisym>
__global__ void __launch_bounds__(256)
reduce_kernel(const R* __restrict__ partial_base, size_t slice_stride,
              const int* __restrict__ counts, int nf, int t0, int ntimes_out, int chunk, int Np,
              int nant, typename Traits<R>::C* __restrict__ out_base, int block_rows) {
  __shared__ typename Traits<R>::C T[kCols][33];
  __shared__ R TM[kAntisym ? kCols : 1][33];
  constexpr int kParts = 32 / kCols;
  reduce_part<R, kCols, kAntisym>(partial_base, slice_stride, counts, nf, t0, ntimes_out, chunk,
                                  Np, nant, out_base, block_rows, blockIdx.x / kParts,
                                  blockIdx.x % kParts, blockIdx.y, T, TM);
}

// Every simulation of a batch: its split-K chunks reduced into its output.
__global__ void __launch_bounds__(256)
reduce_batch_kernel(const PrepSim* __restrict__ sims, int nsims,
                    const long long* __restrict__ pre) {
  __shared__ float2 T[32][33];
  __shared__ float TM[32][33];
  const int si = find_segment(pre, nsims, blockIdx.x);
  const PrepSim& sm = sims[si];
  const int nbt = ceil_div(sm.nant, 32);
  const int tiles = nbt * (nbt + 1) / 2;
  const int local = (int)(blockIdx.x - __ldg(pre + si));
  const size_t slice = (size_t)ceil_div(sm.S > 0 ? sm.S : 1, sm.chunk) * 2 * sm.Np * sm.Np;
  reduce_part<float, 32, true>(sm.partial, slice, sm.counts, sm.F, 0, sm.T, sm.chunk, sm.Np,
                               sm.nant, static_cast<float2*>(sm.out), sm.block_rows, local % tiles, 0,
                               local / tiles, T, TM);
}

cudaError_t launch_reduce_batch(const PrepSim* sims, int nsims, const PrepPre& pre,
                                const PrepTotals& tot, cudaStream_t st) {
  if (tot.red <= 0) return cudaSuccess;
  reduce_batch_kernel<<<(unsigned)tot.red, 256, 0, st>>>(sims, nsims, pre.red);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_reduce(const R* partial, size_t slice_stride, const int* counts, int nt,
                          int nf, int t0, int ntimes_out, int chunk, int max_chunks, int Np,
                          int nant, int block_rows, void* out, cudaStream_t st) {
  using C = typename Traits<R>::C;
  const int nbt = ceil_div(nant, 32);
  const bool split = max_chunks >= kReduceSplitChunks;
  const dim3 grid(nbt * (nbt + 1) / 2 * (split ? 4 : 1), nt * nf);
  auto* kernel = split ? (block_rows ? reduce_kernel<R, 8, true> : reduce_kernel<R, 8, false>)
                       : (block_rows ? reduce_kernel<R, 32, true> : reduce_kernel<R, 32, false>);
  kernel<<<grid, 256, 0, st>>>(partial, slice_stride, counts, nf, t0, ntimes_out, chunk, Np, nant,
                               reinterpret_cast<C*>(out), block_rows);
  return cudaGetLastError();
}

template cudaError_t launch_gen_phasors<float>(const PlainDims&, int, const void*, int, const void*, const float*, int, void*, cudaStream_t);
template cudaError_t launch_gen_phasors<double>(const PlainDims&, int, const void*, int, const void*, const double*, int, void*, cudaStream_t);
template cudaError_t launch_herk_plain<float>(const PlainDims&, int, const void*, int, float*, cudaStream_t);
template cudaError_t launch_herk_plain<double>(const PlainDims&, int, const void*, int, double*, cudaStream_t);
template cudaError_t launch_reduce<float>(const float*, size_t, const int*, int, int, int, int, int, int, int, int, int, void*, cudaStream_t);
template cudaError_t launch_reduce<double>(const double*, size_t, const int*, int, int, int, int, int, int, int, int, int, void*, cudaStream_t);

}  // namespace hv
