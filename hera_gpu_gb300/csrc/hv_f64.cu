// hv_f64.cu -- the FP64 Hermitian product on the tensor cores (precision 2).
//
// GB300 issues about 2 FP64 FMAs a clock and SM (1.25 TFLOP/s), so a SIMT
// product of FP64 phasors is bound by that pipe: 32.8 ms for 350 antennas x
// 50k sources.  Here the product is formed exactly from small integers on the
// FP8 tensor cores, after Ootomo, Ozaki and Yokota ("DGEMM on integer matrix
// multiplication unit", 2024) and Ozaki, Ogita, Oishi and Rump ("Error-free
// transformations of matrix multiplication ...", Numer. Algorithms 59, 2012):
//   * per (slice, antenna) the phasors are scaled by a power of two (from the
//     antenna's largest component over the sources at hand) and rounded once
//     to 59-bit integers X -- 6 bits finer than the largest component's own
//     FP64 spacing;
//   * X is written in 12 balanced base-32 digits d_0 .. d_11 (|d| <= 16, exact
//     in E4M3), most significant first;
//   * sum_s X_a X_b is a sum of digit products of weight 32^(22 - i - j).  The
//     classes c = i + j <= 11 are kept (78 of 144 digit pairs; those dropped
//     are below 2^-56 of the largest product); a class sum over at most 5461
//     sources and 6 digit pairs stays below 2^24, where the FP32
//     accumulation of kind::f8f6f4 is exact;
//   * class sums go to 64-bit integers in global memory (two neighbouring
//     classes a word, added with integer reductions: exact and independent of
//     order), and are converted once, smallest class first, in FP64.
// The result is deterministic.  What the rounding to 59 bits and the dropped
// classes lose is relative to the two antennas' largest components, M_a M_b:
// about 2^-59 sqrt(n) M_a M_b over n sources.  An FP64 sum loses 2^-53 of its
// partial sums instead, which are small where two antennas are bright on
// different sources.  So the two amplitudes' overlap is formed along with the
// class sums, and a slice with a pair of antennas whose overlap is too small for
// the digits to be at least as exact as the FP64 sum takes the SIMT product
// (kOverlapMin).  Elsewhere the distance from an exact evaluation is set by the
// rounding of U (the phases themselves are formed in integers): relative
// Frobenius errors against 113-bit arithmetic of 3.6e-15 at 16
// antennas x 1000 sources (SIMT product 4.0e-15), 5.5e-15 at 40 x 2000
// (6.9e-15), and 2.2e-16 on a 2.5 m array, where the phases are exact enough to
// show the product (1.1e-15).
//
// Measured on GB300, one slice of 350 antennas x 50k sources above the horizon
// (ncu): phasors 0.33 ms, digits 0.26 ms, class sums and overlaps 0.74 ms,
// conversion 0.02 ms; with SIMT 1.30 ms and 32.8 ms.  A call of 3 such slices
// 102.6 -> 3.87 ms (3.73 without the overlaps).
//
// Slices whose phasors are not finite, whose antenna scales leave
// [2^-400, 2^400], or with a pair of antennas of too little overlap are flagged
// on the device and take the SIMT product of hv_plain.cu from the same phasors.
//
//   gen64      phasors in FP64 to HBM, and the largest component per antenna
//   digits64   phasors -> digit tiles, in the layout the MMAs read
//   mma64      class sums and overlaps (TMA bulk copies, tcgen05, integer
//              reductions)
//   overlap64  flags the slices with a pair of too little overlap
//   final64    class sums (or the SIMT chunks of a flagged slice) -> output
#include <algorithm>

#include "hv_internal.cuh"
#include "hv_kernels.h"
#include "hv_ptx.cuh"

namespace hv {

namespace {

constexpr int kDig = 12;                   // base-32 digits of a component
constexpr int kPlanes = 2 * kDig;          // (digit, re / im)
constexpr int kGroups = kDig / 2;          // words: classes 2 g and 2 g + 1
constexpr int kTile = 4096;                // 128 antennas x 32 sources of one plane
constexpr int kTable = 1024;               // sin / cos table: multiples of 1/1024 cycle
constexpr int kGenSrc = 64;                // sources a warp generates for its 32 antennas
constexpr int kGenWarps = 8;

// Sources of slice z above the horizon that belong to the window of sources
// at hand (at most F64Dims::S from s0 on).
__device__ __forceinline__ int window_count(const F64Dims& d, int z) {
  return max(0, min(d.counts[z / d.nf] - d.s0, d.S));
}

// --------------------------------------------------------------- gen64 ----
constexpr long long kTwoPi = 7244019458077122842ll;  // 2 pi 2^60

// cos and sin of the multiples of 1/1024 cycle, in units of 2^-62 and within a
// few of them: Taylor series up to pi / 4 in integers, and symmetry.
__global__ void sincos_table_kernel(longlong2* __restrict__ tab) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= kTable) return;
  static_assert(kTable == 1024, "quadrants of 256");
  const int m = k & 255, j = m > 128 ? 256 - m : m;
  auto mul = [](long long a, long long b) { return (long long)((__int128)a * b >> 62); };
  const long long th = (long long)((__int128)kTwoPi * j >> 8);  // 2 pi j / 1024
  const long long t2 = mul(th, th);
  long long c = 1ll << 62, s = th, tc = c, ts = th;
  for (int i = 1; i <= 10; ++i) {
    tc = -mul(tc, t2) / ((2 * i - 1) * (2 * i));
    ts = -mul(ts, t2) / (2 * i * (2 * i + 1));
    c += tc;
    s += ts;
  }
  const long long x = m > 128 ? s : c, y = m > 128 ? c : s;  // first quadrant
  const int q = k >> 8;
  tab[k] = q == 0   ? make_longlong2(x, y)
           : q == 1 ? make_longlong2(-y, x)
           : q == 2 ? make_longlong2(-x, -y)
                    : make_longlong2(y, -x);
}

// Smallest E >= 0 with every |component| < 2^E (above 1000 if one is not
// finite), and a component in units of 2^(E - 62).
__device__ __forceinline__ int fixed_exponent(double x, double y, double z) {
  const int m = max(__double2hiint(x) & 0x7fffffff,
                    max(__double2hiint(y) & 0x7fffffff, __double2hiint(z) & 0x7fffffff));
  return max(0, (m >> 20) - 1022);
}
__device__ __forceinline__ long long to_fixed(double x, int E) {
  return __double2ll_rn(x * __hiloint2double((1023 + 62 - E) << 20, 0));
}

// cos and sin, in units of 2^-62, of a phase in units of 2^-64 cycle: its
// nearest multiple of 1/1024 cycle from the table, the rest r (|r| <= 2^-11
// cycles) by the Taylor series in theta = 2 pi r up to theta^5, whose first
// dropped terms are below 2e-18, and the addition theorem.  Every product
// keeps an error below 2^-58.
__device__ __forceinline__ void sincos_fixed(unsigned long long ph,
                                             const longlong2* __restrict__ tab, long long& cs,
                                             long long& sn) {
  const uint32_t k = (uint32_t)((ph + (1ull << 53)) >> 54);  // mod 1024
  const long long r = (long long)(ph - ((unsigned long long)k << 54));
  const longlong2 t = tab[k];
  const long long th = __mul64hi(r << 9, kTwoPi);               // theta 2^69
  const unsigned long long h = (unsigned long long)__mul64hi(th, th);  // theta^2 2^74
  const uint32_t hq = (uint32_t)(h >> 26);                      // theta^2 2^48
  const uint32_t q4 = __umulhi(hq, hq);                         // theta^4 2^64
  // theta^2 / 6 - theta^4 / 120, 2^50
  const int w = (int)(__umulhi(hq, 2863311531u) - __umulhi(q4, 2185u));
  // sin theta 2^64 and (1 - cos theta) 2^64 (in this sign: nvcc 13.0 makes
  // -2^32 of the difference 0 - 0 the other way round)
  const long long sr = (th >> 5) - (((long long)(int)(th >> 30) * w) >> 25);
  const long long cr = (long long)((h >> 11) - __umulhi(q4, 178956971u));
  const long long s7 = sr << 7, c16 = cr << 16;
  cs = t.x - (__mul64hi(t.x, c16) >> 16) - (__mul64hi(t.y, s7) >> 7);
  sn = t.y - (__mul64hi(t.y, c16) >> 16) + (__mul64hi(t.x, s7) >> 7);
}
// x 2^-62, rounded once.
__device__ __forceinline__ double from_fixed62(long long x) {
  const double d = (double)x;
  const int hi = __double2hiint(d);
  return __hiloint2double(x == 0 ? 0 : hi - (62 << 20), __double2loint(d));
}

// One source of a warp's batch, as its 32 antennas read it.
struct GenSrc {
  long long sx, sy, sz;       // direction, units of 2^(e - 62)
  double w00, w01, w10, w11;  // bilinear weights times sqrt(I)
  long long pix;
  int e;
};

// A warp generates kGenSrc sources for 32 antennas: U stays in registers, a
// source's weights are formed once per warp.
//
// The phase and its sine and cosine are formed in 64-bit integers: the FP64
// pipe takes 16 clocks for an instruction of a warp, as long as some 40
// integer ones.  U and the direction are rounded to 62 bits below a power of
// two each, their products summed exactly in 128 bits, of which the 64 below
// one cycle are kept: the phase is off by at most 2^-60 of the largest |U| times
// |s|, where an FP64 sum is by about 2^-53 of it.  8 FP64 instructions
// remain a phasor (4 beam and amplitude, 2 conversions, 2 products).  350
// antennas x 50k sources: 0.33 ms, against 0.80 with 22 FP64 instructions (the
// phase, its reduction and the series in FP64) and 1.30 with sincospi.
// Phases of 2^56 cycles and more, and those that are not finite, take the FP64
// sum and the library functions.
__global__ void __launch_bounds__(kGenWarps * 32)
gen64_kernel(const F64Dims d, const SrcRec64* __restrict__ rec, size_t rec_stride,
             const Ucoef64* __restrict__ U, const double* __restrict__ beamT, int PP, int dx,
             int dy, const longlong2* __restrict__ table, double2* __restrict__ v,
             uint32_t* __restrict__ rowmax) {
  __shared__ longlong2 tab[kTable];
  __shared__ GenSrc src[kGenWarps][32];
  const int z = blockIdx.z, n = window_count(d, z);
  const int ng = ceil_div(d.nant, 32);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long job0 = (long long)blockIdx.x * kGenWarps;
  if (job0 / ng * kGenSrc >= n) return;
  for (int i = threadIdx.x; i < kTable; i += kGenWarps * 32) tab[i] = table[i];
  __syncthreads();
  const long long job = job0 + warp;
  const int a = (int)(job % ng) * 32 + lane;
  const long long sbeg = job / ng * kGenSrc;
  if (sbeg >= n) return;
  const int tl = z / d.nf, f = z % d.nf;
  rec += (size_t)tl * rec_stride + d.s0;
  // padded antennas (a < Np) have U = 0 and a zero beam; they are not stored
  U += ((size_t)tl * d.u_nf + f) * d.Np + a;
  long long ux, uy, uz;
  int ue;
  {
    const Ucoef64 u = *U;
    ue = fixed_exponent(u.x, u.y, u.z);
    ux = to_fixed(u.x, ue);
    uy = to_fixed(u.y, ue);
    uz = to_fixed(u.z, ue);
  }
  const double* beam = beamT + (size_t)f * PP * d.Np + a;
  double2* out = v + (size_t)z * d.v_stride + a;
  uint32_t top = 0, low = 0;
  for (int b = 0; b < kGenSrc; b += 32) {
    const int s0 = (int)sbeg + b, m = min(32, n - s0);
    if (m <= 0) break;
    __syncwarp();
    if (lane < m) {
      const SrcRec64 r = rec[s0 + lane];
      GenSrc g;
      g.e = fixed_exponent(r.sx, r.sy, r.sz);
      g.sx = to_fixed(r.sx, g.e);
      g.sy = to_fixed(r.sy, g.e);
      g.sz = to_fixed(r.sz, g.e);
      const double y1 = r.amp * r.fy, y0 = fma(-r.amp, r.fy, r.amp);
      g.w01 = y0 * r.fx;
      g.w00 = fma(-y0, r.fx, y0);
      g.w11 = y1 * r.fx;
      g.w10 = fma(-y1, r.fx, y1);
      g.pix = (long long)r.pix * d.Np;
      src[warp][lane] = g;
    }
    __syncwarp();
#pragma unroll 2
    for (int s = 0; s < m; ++s) {
      const GenSrc& g = src[warp][s];
      const double* bp = beam + g.pix;
      const double b00 = __ldg(bp), b01 = __ldg(bp + (size_t)dx * d.Np),
                   b10 = __ldg(bp + (size_t)dy * d.Np), b11 = __ldg(bp + (size_t)(dx + dy) * d.Np);
      const double A = fma(g.w11, b11, fma(g.w10, b10, fma(g.w01, b01, g.w00 * b00)));
      double sn, cs;
      // the sum is in units of 2^(ue + e - 124) cycles, below 3 x 2^124
      const int sh = 60 - ue - g.e;
      if (sh >= 4) {
        const __int128 p = (__int128)ux * g.sx + (__int128)uy * g.sy + (__int128)uz * g.sz;
        long long ci, si;
        sincos_fixed((unsigned long long)(p >> sh), tab, ci, si);
        cs = from_fixed62(ci);
        sn = from_fixed62(si);
      } else {
        const Ucoef64 u = *U;
        const SrcRec64 r = rec[s0 + s];
        const double ph = fma(u.x, r.sx, fma(u.y, r.sy, u.z * r.sz));
        sincospi(2.0 * (ph - rint(ph)), &sn, &cs);
      }
      const double re = A * cs, im = A * sn;
      if (a < d.nant) out[(size_t)(s0 + s) * d.Np] = make_double2(re, im);
      top = max(top, max(__double2hiint(re) & 0x7fffffffu, __double2hiint(im) & 0x7fffffffu));
      low |= (uint32_t)__double2loint(re) | (uint32_t)__double2loint(im);
    }
  }
  // the high word of the largest component (its exponent gives the scale);
  // 1 marks components that are not zero but have a zero high word
  if (top == 0 && low != 0) top = 1;
  if (a < d.nant && top) atomicMax(rowmax + (size_t)z * d.Np + a, top);
}

// ------------------------------------------------------------ digits64 ----
// Exponent field of an antenna's largest component: 0 for an antenna of
// zeros; fields outside [623, 1423] (2^-400 .. 2^400, infinities and NaN) are
// not scaled: their slice is flagged.
__device__ __forceinline__ bool row_field(uint32_t rowmax, int& field) {
  field = (int)(rowmax >> 20);
  return rowmax == 0 || (field >= 623 && field <= 1423);
}

// Largest component below 2^(field - 1022): v as a 59-bit integer, rounded to
// nearest (half away from zero).
__device__ __forceinline__ long long scaled_int(double v, int field) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  int ex = (int)(b >> 52) & 0x7ff;
  unsigned long long m = b & 0xfffffffffffffull;
  if (ex) m |= 1ull << 52;
  else ex = 1;
  const int sh = ex - field + 6;  // <= 6
  unsigned long long x;
  if (sh >= 0) x = m << sh;
  else if (sh > -60) x = (m + (1ull << (-sh - 1))) >> -sh;
  else x = 0;
  return (b >> 63) ? -(long long)x : (long long)x;
}

// Overlap of antennas a and b over the sources of a window: sum_s w_a w_b with
// the weights w = 256 (m / 2^E)^2, m the larger component of the phasor and 2^E
// the power of two above the antenna's largest, rounded down to 4 significant
// bits (exact in E4M3).  It is 2^16 P^2 for the FP64 sum's typical partial sum P
// in units of 2^(E_a + E_b), where that sum rounds by about 2^-54.3 P sqrt(min(n,
// kPlainChunk)) and the digits by 2^-59.4 sqrt(n) (root mean squares of rounding
// errors spread evenly): the digits are the more exact from 2^5.8 = 56 on for n up
// to kPlainChunk, and in proportion to n beyond.  Arrays of Airy or random beams
// over 150 to 100k sources lie at 5 to 600 times this limit.
constexpr int kOverlapMin = 64;
// Sums are capped here to fit in 32 bits.  They are exact in FP32 up to 2^24, and
// the limit never exceeds 1024.
constexpr float kOverlapCap = 1073741824.f;

// Where a slice's weights start in its digits.
__device__ __forceinline__ size_t weight_tiles(const F64Dims& d) {
  return (size_t)(d.Np / 128) * d.nks * (kPlanes * kTile);
}
// A component (its high word) in units of 2^-15 of the scale, rounded down.
__device__ __forceinline__ uint32_t top15(int hi, int field) {
  const int ex = (hi >> 20) & 0x7ff;
  return ex > field - 16 ? (uint32_t)((hi & 0xfffff) | 0x100000) >> (6 + field - ex) : 0u;
}
// E4M3 code of the weight of m units.
__device__ __forceinline__ uint32_t weight_code(uint32_t m) {
  const uint32_t w = m * m >> 22;
  const int e = 31 - __clz(w | 1u);
  return w ? (uint32_t)((e + 7) << 3) | ((w << 3 >> e) & 7u) : 0u;
}

// Digit tiles: [slice][antenna block][source step of 32][plane][4096], a plane
// tile in the K-major core-matrix layout the MMAs read without a swizzle (8
// antennas x 16 sources a 128-byte core matrix; the two along the sources
// adjacent, then the next 8 antennas), so that every group of planes of a
// step is one contiguous bulk copy.  One block makes a step: thread (antenna,
// half of the step, component) 16 sources, and the weights of 8 of them, whose
// tiles lie behind the digits, [antenna block][source step][4096].  Bound by HBM
// (16 B read, 25 B written a phasor).
__global__ void __launch_bounds__(512)
digits64_kernel(const F64Dims d, const double2* __restrict__ v,
                const uint32_t* __restrict__ rowmax, uint8_t* __restrict__ dig,
                int* __restrict__ flags) {
  __shared__ uint8_t lut[33];  // E4M3 codes of -16 .. 16
  const int ks = blockIdx.x, blk = blockIdx.y, z = blockIdx.z;
  const int n = window_count(d, z);
  if (ks * 32 >= n) return;
  if (threadIdx.x < 33) {
    const int x = (int)threadIdx.x - 16, m = abs(x);
    uint32_t code = 0;
    if (m) {
      const int e = 31 - __clz(m);
      code = (uint32_t)((e + 7) << 3) | (uint32_t)(((m << 3) >> e) & 7);
    }
    lut[threadIdx.x] = (uint8_t)(code | (x < 0 ? 0x80u : 0u));
  }
  __syncthreads();
  const int row = threadIdx.x & 127, half = (threadIdx.x >> 7) & 1, ri = threadIdx.x >> 8;
  const int a = blk * 128 + row;
  const uint32_t rm = a < d.nant ? rowmax[(size_t)z * d.Np + a] : 0u;
  int field;
  const bool ok = row_field(rm, field);
  if (!ok && ks == 0 && half == 0 && ri == 0) atomicOr(flags + z, 1);
  uint32_t w[kDig][4];
  const double* src = reinterpret_cast<const double*>(v + (size_t)z * d.v_stride) + 2 * (size_t)a + ri;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int k = 0; k < kDig; ++k) w[k][q] = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int s = ks * 32 + half * 16 + q * 4 + e;
      long long x = 0;
      if (rm != 0 && ok && s < n) x = scaled_int(src[2 * (size_t)s * d.Np], field);
      // balanced digits: adding 16 at every place but the top one makes each
      // lower digit its 5 bits minus 16
      unsigned long long y = (unsigned long long)x;
#pragma unroll
      for (int k = 0; k < kDig - 1; ++k) y += 16ull << (5 * k);
#pragma unroll
      for (int k = 0; k < kDig; ++k) {
        // digit of weight 32^k is plane digit kDig - 1 - k
        const int idx = k == kDig - 1 ? (int)((long long)y >> (5 * k)) + 16
                                      : (int)(y >> (5 * k)) & 31;
        w[kDig - 1 - k][q] |= (uint32_t)lut[idx] << (8 * e);
      }
    }
  }
  const size_t tile = (size_t)blk * d.nks + ks;
  const int at = (row >> 3) * 256 + half * 128 + (row & 7) * 16;
  uint8_t* zd = dig + (size_t)z * d.dig_stride;
  uint8_t* out = zd + tile * (kPlanes * kTile) + ri * kTile + at;
#pragma unroll
  for (int k = 0; k < kDig; ++k)
    *reinterpret_cast<uint4*>(out + (size_t)k * 2 * kTile) =
        make_uint4(w[k][0], w[k][1], w[k][2], w[k][3]);
  // the weights of the thread's half of the 16 sources, from both components
  // (their high words, read again: with them the loop above took 83 registers,
  // one block an SM instead of two)
  uint32_t wt[2] = {0, 0};
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int s = ks * 32 + half * 16 + ri * 8 + e;
    if (rm != 0 && ok && s < n) {
      const int4 h = *reinterpret_cast<const int4*>(src - ri + 2 * (size_t)s * d.Np);
      wt[e >> 2] |= weight_code(max(top15(h.y, field), top15(h.w, field))) << (8 * (e & 3));
    }
  }
  *reinterpret_cast<uint2*>(zd + weight_tiles(d) + tile * kTile + at + 8 * ri) =
      make_uint2(wt[0], wt[1]);
}

// --------------------------------------------------------------- mma64 ----
// A work item: a pair of antenna blocks, a chunk of source steps and a unit,
// which fills the 512 TMEM columns with the real and imaginary sums of two
// accumulators.  Units in order of falling cost (digit pairs).
//
// Two different blocks: two neighbouring classes, 2 g and 2 g + 1, over a range
// of A digits i0 .. i1 (at most 6, so that two stages of the planes they need
// fit in shared memory), added to word g as 32 x the one + the other.
//
// A block with itself: the sum S over the digit pairs (i, j) of a class is
// Hermitian, the pairs (i, j) and (j, i) each other's adjoint.  So the units 0-5
// take the pairs i < j only, with twice the weight, others the pairs (i, i) of
// two digits 2 k and 2 k + 1 (the even classes 4 k and 4 k + 2, words 2 k and
// 2 k + 1), and the conversion takes (S + S^H) / 2: 42 digit pairs instead
// of 78, and the digits are read once.  Three blocks: 0.93 -> 0.86 ms a slice.
//
// The last unit of a pair of blocks sums the overlaps, one product of the weights
// a step, over the whole window (the first chunk's item, plain stores); its stages
// take as many steps as fit.
constexpr int kDigUnits = 9, kUnits = kDigUnits + 1;
__constant__ int8_t kUnit[kDigUnits][3] = {{5, 0, 5}, {5, 6, 11}, {2, 0, 5}, {4, 0, 4}, {4, 5, 9},
                                        {3, 0, 3}, {3, 4, 7},  {1, 0, 3}, {0, 0, 1}};
// {g, 0} or {k, 1} of a block with itself
__constant__ int8_t kOwnUnit[kDigUnits][2] = {{5, 0}, {4, 0}, {3, 0}, {2, 0}, {1, 0},
                                           {0, 1}, {1, 1}, {2, 1}, {0, 0}};
constexpr int kMaxA = 6, kMaxB = 7;        // digits a unit needs of A and of B
constexpr int kOverSteps = 2 * kMaxA;      // steps of weights a stage holds
constexpr int kStageBytes = (kMaxA + kMaxB) * 2 * kTile;
constexpr int kStages = 2;
constexpr int kMmaSmem = kStages * kStageBytes + 128;
constexpr int kMmaThreads = 256;
// Source steps an accumulation may span: 6 pairs x 2 products x 256 x 32
// sources x 128 steps < 2^24.
constexpr int kMaxChunkSteps = 128;

// Descriptor of a K-major operand without swizzle: core matrices along K 128
// bytes apart (leading offset), groups of 8 rows 256 bytes (stride offset).
constexpr uint32_t kPlainDescHi = (256u >> 4) | (1u << 14);
__device__ __forceinline__ uint32_t plain_desc_lo(uint32_t saddr) {
  return ((saddr & 0x3FFFFu) >> 4) | ((128u >> 4) << 16);
}

__device__ __forceinline__ void mma64(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo,
                                      uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %5, 0;\n"
      " mov.b64 da, {%1, %3};\n mov.b64 db, {%2, %3};\n"
      " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], da, db, %4, p;\n}\n" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(kPlainDescHi), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes,
                                          uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void add_word(unsigned long long* w, long long x) {
  asm volatile("red.global.add.u64 [%0], %1;" ::"l"(w), "l"((unsigned long long)x) : "memory");
}

__global__ void __launch_bounds__(kMmaThreads, 1)
mma64_kernel(const F64Dims d, const uint8_t* __restrict__ dig, const int* __restrict__ flags,
             long long* __restrict__ W, int npairs, int nchunks, int chunk_steps, int* err,
             unsigned long long wait_ns) {
  extern __shared__ __align__(1024) uint8_t smem[];
  // all pairs and units of a chunk together: they read the same digits, 14 MB
  // a chunk of 46 steps and 3 blocks, from L2 (a sweep of all chunks a unit
  // read 5 GB from HBM a slice, 0.86 -> 0.79 ms at one)
  const int pair = blockIdx.x % npairs, unit = blockIdx.x / npairs % kUnits;
  const int cz = blockIdx.x / (npairs * kUnits), chunk = cz % nchunks, z = cz / nchunks;
  const int steps = ceil_div(window_count(d, z), 32);
  const bool over = unit == kDigUnits;
  const int k0 = chunk * chunk_steps, k1 = over ? steps : min(steps, k0 + chunk_steps);
  if (k0 >= k1 || flags[z] || (over && chunk)) return;
  int I = 0, J = pair;
  for (const int nb = d.Np / 128; J >= nb - I; ++I) J -= nb - I;
  J += I;
  // digits of A and of B
  const int du = over ? 0 : unit;
  const bool own = I == J, same = own && (over || kOwnUnit[du][1]);
  const int g = own ? kOwnUnit[du][0] : kUnit[du][0];
  const int i0 = same ? 2 * g : own ? 0 : kUnit[du][1];
  const int i1 = same ? 2 * g + 1 : own ? g : kUnit[du][2];
  const int j0 = same ? i0 : own ? g + 1 : max(0, 2 * g - i1);
  const int j1 = same ? i1 : 2 * g + 1 - i0;
  const uint32_t base = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStages * kStageBytes);
  const uint32_t bar0 = smem_u32(bars);
  auto full = [&](int s) { return bar0 + 8u * s; };
  auto empty = [&](int s) { return bar0 + 8u * (kStages + s); };
  const uint32_t done = bar0 + 8u * (2 * kStages);
  uint32_t* holder = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(holder + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(holder)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *holder;
  // pipeline steps: one source step, or kOverSteps of them
  const int nsteps = over ? ceil_div(k1 - k0, kOverSteps) : k1 - k0;
  if (warp == 0 && lane == 0) {
    // producer: the unit's A planes and B planes of each step, contiguous
    const size_t step_bytes = (size_t)(over ? kOverSteps : kPlanes) * kTile;
    const uint8_t* zd = dig + (size_t)z * d.dig_stride + (over ? weight_tiles(d) : 0);
    const size_t block = (size_t)d.nks * (over ? 1 : kPlanes) * kTile;
    const size_t first = (size_t)k0 * (over ? 1 : kPlanes) * kTile;
    const uint8_t* pa = zd + I * block + first + (over ? 0 : i0 * 2 * kTile);
    const uint8_t* pb = zd + J * block + first + (over ? 0 : j0 * 2 * kTile);
    uint32_t na = (uint32_t)(i1 - i0 + 1) * 2 * kTile, nb = (uint32_t)(j1 - j0 + 1) * 2 * kTile;
    int k = 0;
    for (; k < nsteps; ++k, pa += step_bytes, pb += step_bytes) {
      const int s = k % kStages;
      if (!wait1(empty(s), ((k / kStages) & 1) ^ 1, abort_flag, err, wait_ns)) break;
      const uint32_t st = base + (uint32_t)s * kStageBytes;
      if (over) na = nb = (uint32_t)min(kOverSteps, k1 - k0 - k * kOverSteps) * kTile;
      mbar_expect_tx(full(s), same ? na : na + nb);
      bulk_load(st, pa, na, full(s));
      if (!same) bulk_load(st + kMaxA * 2 * kTile, pb, nb, full(s));
    }
    // copies still in flight land before the CTA can exit
    for (int q = max(0, k - kStages); q < k; ++q)
      wait_drain(full(q % kStages), (q / kStages) & 1, err, wait_ns);
  } else if (warp == 1 && lane == 0) {
    const uint32_t idp = idesc_mma(128, false, 0u), idn = idesc_mma(128, true, 0u);
    for (int k = 0; k < nsteps; ++k) {
      const int s = k % kStages;
      if (!wait1(full(s), (k / kStages) & 1, abort_flag, err, wait_ns)) break;
      tc_fence_after();
      const uint32_t st = base + (uint32_t)s * kStageBytes;
      const uint32_t a0 = plain_desc_lo(st);
      const uint32_t b0 = same ? a0 : plain_desc_lo(st + kMaxA * 2 * kTile);
      constexpr uint32_t kP = kTile >> 4;  // descriptor units of a plane
      if (over)
        for (int t = 0; t < min(kOverSteps, k1 - k0 - k * kOverSteps); ++t)
          mma64(tmem, a0 + t * kP, b0 + t * kP, idp, k > 0 || t > 0);
#pragma unroll 1
      for (int q = 0; q < (over ? 0 : 2); ++q) {
        const uint32_t dre = tmem + 256u * q, dim = dre + 128u;
        uint32_t acc = k > 0;
        for (int i = i0; i <= i1; ++i) {
          const int j = same ? i : 2 * g + q - i;
          if (j < j0 || j > j1 || (same && i != i0 + q)) continue;
          const uint32_t a = a0 + (uint32_t)(i - i0) * 2 * kP, b = b0 + (uint32_t)(j - j0) * 2 * kP;
          mma64(dre, a, b, idp, acc);           // Re Re
          mma64(dim, a + kP, b, idp, acc);      // Im Re
          mma64(dre, a + kP, b + kP, idp, 1u);  // Im Im
          mma64(dim, a, b + kP, idn, 1u);       // -Re Im
          acc = 1u;
        }
      }
      mma_commit(empty(s));
    }
    // the accumulators are complete, and no MMA is in flight after this
    mma_commit(done);
    wait_drain(done, 0, err, wait_ns);
  }
  __syncwarp();
  // the sums, exact integers, added to the slice's words (W[g][re / im][b][a],
  // a contiguous across a warp)
  const bool ok = wait_warp(done, 0, abort_flag, err, wait_ns) && !*abort_flag;
  tc_fence_after();
  if (ok) {
    const int q = warp & 3, ri = warp >> 2;
    const int a = I * 128 + q * 32 + lane;
    const size_t plane = (size_t)d.Np * d.Np;
    unsigned long long* w = reinterpret_cast<unsigned long long*>(W) + (size_t)z * d.w_stride +
                            (size_t)(2 * (same ? 2 * g : g) + ri) * plane +
                            (size_t)J * 128 * d.Np + a;
    uint32_t* wo = reinterpret_cast<uint32_t*>(W + (size_t)z * d.w_stride + 2 * kGroups * plane) +
                   (size_t)J * 128 * d.Np + a;
    const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)ri * 128u;
    const long long weight = own ? 2 : 1;
    const bool no_hi = own && !same && g == 0;  // (no pair i < j in class 0)
#pragma unroll 1
    for (int c = 0; c < (over ? ri ? 0 : 128 : 0); c += 32) {
      float x[32];
      tmem_ld32(tq + c, x);
#pragma unroll
      for (int k = 0; k < 32; ++k)
        wo[(size_t)(c + k) * d.Np] = (uint32_t)fminf(x[k], kOverlapCap);
    }
#pragma unroll 1
    for (int c = over ? 128 : 0; c < 128; c += 32) {
      float hi[32], lo[32];
      tmem_ld32(tq + c, hi);
      tmem_ld32(tq + 256u + c, lo);
#pragma unroll
      for (int x = 0; x < 32; ++x) {
        if (no_hi) hi[x] = 0.f;
        unsigned long long* wx = w + (size_t)(c + x) * d.Np;
        if (same) {
          add_word(wx, 32ll * __float2int_rn(hi[x]));
          add_word(wx + 2 * plane, 32ll * __float2int_rn(lo[x]));
        } else {
          add_word(wx, weight * (32ll * __float2int_rn(hi[x]) + __float2int_rn(lo[x])));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512)
                 : "memory");
  }
}

// ----------------------------------------------------------- overlap64 ----
// Flags the slices with a pair of antennas, neither of zeros, whose overlap is
// below the limit.
__global__ void __launch_bounds__(256)
overlap64_kernel(const F64Dims d, const long long* __restrict__ W,
                 const uint32_t* __restrict__ rowmax, int* __restrict__ flags) {
  const int z = blockIdx.y, n = window_count(d, z);
  const unsigned long long limit = (unsigned long long)kOverlapMin * max(n, kPlainChunk);
  const uint32_t* rm = rowmax + (size_t)z * d.Np;
  const uint32_t* o = reinterpret_cast<const uint32_t*>(W + (size_t)z * d.w_stride +
                                                        (size_t)2 * kGroups * d.Np * d.Np);
  const int b = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (n == 0 || b >= d.nant || rm[b] == 0) return;
  bool low = false;
#pragma unroll 4
  for (int a = threadIdx.x & 31; a <= b; a += 32) {
    const unsigned long long x = o[(size_t)b * d.Np + a];
    low |= rm[a] != 0 & x * kPlainChunk < limit;
  }
  if (low) atomicOr(flags + z, 1);
}

// ------------------------------------------------------------- final64 ----
// V = 2^(E_a + E_b - 13) sum_g W_g 2^(-10 g) of a window of sources, smallest
// words first, stored (the first window) or added to the output, both
// triangles; a flagged slice sums its SIMT chunks in order instead.
__global__ void __launch_bounds__(256)
final64_kernel(const F64Dims d, const long long* __restrict__ W,
               const uint32_t* __restrict__ rowmax, const int* __restrict__ flags,
               const double* __restrict__ partial, size_t partial_stride, int t0, int f0,
               int ntimes, double2* __restrict__ out_base) {
  __shared__ double2 T[32][33];
  const int z = blockIdx.y;
  const int n = window_count(d, z);
  const bool first = d.s0 == 0;
  if (n == 0 && !first) return;
  const int nbt = ceil_div(d.nant, 32);
  int A = 0, B = blockIdx.x;
  for (; B >= nbt - A; ++A) B -= nbt - A;
  B += A;
  double2* out = out_base + ((size_t)(f0 + z % d.nf) * ntimes + t0 + z / d.nf) *
                                (size_t)d.nant * d.nant;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const size_t plane = (size_t)d.Np * d.Np;
  const bool simt = flags[z] != 0;
  const bool own = A / 4 == B / 4;  // a block of 128 with itself
  const int a = A * 32 + tx;
  int fa = 0;
  if (a < d.nant) row_field(rowmax[(size_t)z * d.Np + a], fa);
#pragma unroll 1
  for (int bb = ty; bb < 32; bb += 8) {
    const int b = B * 32 + bb;
    double2 val = make_double2(0.0, 0.0);
    if (a <= b && b < d.nant) {
      const size_t at = (size_t)b * d.Np + a;
      if (simt) {
        const double* p = partial + (size_t)z * partial_stride + at;
        for (int k = 0; k * kPlainChunk < n; ++k, p += 2 * plane) {
          val.x += p[0];
          val.y += p[plane];
        }
      } else if (n > 0) {
        const long long* w = W + (size_t)z * d.w_stride + at;
        long long x[kGroups], y[kGroups];
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
          x[g] = w[(size_t)(2 * g) * plane];
          y[g] = w[(size_t)(2 * g + 1) * plane];
        }
        if (own) {  // S + S^H, exact
          const long long* wt = W + (size_t)z * d.w_stride + (size_t)a * d.Np + b;
#pragma unroll
          for (int g = 0; g < kGroups; ++g) {
            x[g] += wt[(size_t)(2 * g) * plane];
            y[g] -= wt[(size_t)(2 * g + 1) * plane];
          }
        }
#pragma unroll
        for (int g = kGroups - 1; g >= 0; --g) {
          val.x = fma(val.x, 0x1p-10, (double)x[g]);
          val.y = fma(val.y, 0x1p-10, (double)y[g]);
        }
        int fb;
        row_field(rowmax[(size_t)z * d.Np + b], fb);
        const int e = fa + fb - 2 * 1022 - 13 - (own ? 1 : 0);
        val.x = scalbn(val.x, e);
        val.y = scalbn(val.y, e);
      }
      if (!first) {
        const double2 o = out[(size_t)a * d.nant + b];
        val.x += o.x;
        val.y += o.y;
      }
      if (a == b) val.y = 0.0;
      T[bb][tx] = val;
    }
  }
  // every read of the output above the diagonal is done before the writes
  __syncthreads();
#pragma unroll 1
  for (int bb = ty; bb < 32; bb += 8) {
    // below the diagonal: out[b][a] = conj(V[a][b]), a contiguous
    const int b = B * 32 + bb;
    if (a <= b && b < d.nant) {
      double2 val = T[bb][tx];
      val.y = a == b ? 0.0 : -val.y;
      out[(size_t)b * d.nant + a] = val;
    }
    // above it: out[a][b], b contiguous
    const int ao = A * 32 + bb, bo = B * 32 + tx;
    if (ao < bo && bo < d.nant) out[(size_t)ao * d.nant + bo] = T[tx][bb];
  }
}

}  // namespace

size_t f64_digit_bytes(int Np, int S) {
  // a flagged slice keeps its SIMT chunk sums here
  const size_t dig = (size_t)(kPlanes + 1) * (Np / 128) * (size_t)ceil_div(S, 32) * kTile;
  const size_t part = sizeof(double) * 2 * (size_t)Np * Np * ceil_div(S, kPlainChunk);
  return std::max(dig, part);
}
size_t f64_word_bytes(int Np) {
  return (sizeof(long long) * 2 * kGroups + sizeof(uint32_t)) * (size_t)Np * Np;
}
size_t f64_table_bytes() { return sizeof(longlong2) * kTable; }

cudaError_t launch_f64_table(void* table, cudaStream_t st) {
  sincos_table_kernel<<<kTable / 256, 256, 0, st>>>(static_cast<longlong2*>(table));
  return cudaGetLastError();
}

cudaError_t launch_f64_phasors(const F64Dims& d, int nz, const void* rec, size_t rec_stride,
                               const void* U, const double* beamT, int P, const void* table,
                               void* v, uint32_t* rowmax, cudaStream_t st) {
  const long long jobs = (long long)ceil_div(d.S, kGenSrc) * ceil_div(d.nant, 32);
  const dim3 grid((unsigned)((jobs + kGenWarps - 1) / kGenWarps), 1, nz);
  gen64_kernel<<<grid, kGenWarps * 32, 0, st>>>(
      d, static_cast<const SrcRec64*>(rec), rec_stride, static_cast<const Ucoef64*>(U), beamT,
      P * P, P > 1 ? 1 : 0, P > 1 ? P : 0, static_cast<const longlong2*>(table),
      static_cast<double2*>(v), rowmax);
  return cudaGetLastError();
}

cudaError_t launch_f64_product(const F64Dims& d, int nz, const void* v, const uint32_t* rowmax,
                               void* dig, int* flags, long long* W, int num_sms, int* err,
                               unsigned long long wait_ns, cudaStream_t st) {
  const int nb = d.Np / 128, npairs = nb * (nb + 1) / 2;
  digits64_kernel<<<dim3(d.nks, nb, nz), 512, 0, st>>>(
      d, static_cast<const double2*>(v), rowmax, static_cast<uint8_t*>(dig), flags);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(mma64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMmaSmem);
  if (e != cudaSuccess) return e;
  // about 4 items an SM over the window (half of it above the horizon): an
  // item's start and its reductions take as long as some 20 steps (200
  // antennas x 50k sources 550 us a call at 12 items an SM, 499 at 4, 500 at
  // 3); at least 8 steps
  const long long units = (long long)kDigUnits * npairs * nz;
  const long long per_sm = (units * std::max(1, d.nks / 2) + num_sms - 1) / num_sms;
  const int steps = (int)std::min<long long>(kMaxChunkSteps, std::max<long long>(8, per_sm / 4));
  const int nchunks = ceil_div(d.nks, steps);
  const unsigned items = (unsigned)((long long)nchunks * npairs * nz * kUnits);
  mma64_kernel<<<items, kMmaThreads, kMmaSmem, st>>>(
      d, static_cast<const uint8_t*>(dig), flags, W, npairs, nchunks, steps, err,
      wait_ns ? wait_ns : 10000000000ull);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  overlap64_kernel<<<dim3(ceil_div(d.nant, 8), nz), 256, 0, st>>>(d, W, rowmax, flags);
  return cudaGetLastError();
}

cudaError_t launch_f64_final(const F64Dims& d, int nz, const long long* W,
                             const uint32_t* rowmax, const int* flags, const void* partial,
                             int t0, int f0, int ntimes, void* out, cudaStream_t st) {
  const int nbt = ceil_div(d.nant, 32);
  final64_kernel<<<dim3(nbt * (nbt + 1) / 2, nz), 256, 0, st>>>(
      d, W, rowmax, flags, static_cast<const double*>(partial), d.dig_stride / sizeof(double), t0,
      f0, ntimes, static_cast<double2*>(out));
  return cudaGetLastError();
}

}  // namespace hv
