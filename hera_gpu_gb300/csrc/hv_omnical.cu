// hv_omnical.cu -- hera_gpu's omnical redundant-calibration solver.
//
// Each problem ("pixel") p solves data[p, b] ~ g[i_b] conj(g[j_b]) u[k_b] for
// the gains g (nants) and unique baselines u (nubls) by the Omnical
// iteration of hera_gpu/redcal.py:358-743:
//   dwgts_b = |dmdl_b|^2 w_b and the weights gwgt / uwgt (their sums over
//   the baselines of each antenna / unique baseline) every check_every
//   iterations (redcal.py:590-604, kernels :117-132, :171-196);
//   gbuf / ubuf = sums of d_b = data_b conj(dmdl_b) dwgts_b / |dmdl_b|^2
//   (conjugated where the antenna is j_b; :199-236);
//   x *= (1 - gain) + gain buf / wgt (:239-280, the gain a float32 and
//   1 - gain formed in float32, redcal.py:625,630);
//   every check_every iterations (from check_after on, and at maxiter) the
//   stepped solution is checked: conv = sqrt(sum |new - old|^2 / sum |new|^2)
//   below conv_crit, or a chi^2 above the last, ends the problem keeping the
//   old solution; otherwise chisq and iters are updated (:283-354, host
//   :644-702).
//
// The reference launches a dozen kernels per iteration over 64 problems at
// a time and scatters with global atomics.  Here one launch solves every
// problem: one CTA per problem (a persistent grid that takes problems from
// a counter), every iteration inside the kernel, the solution and the
// per-baseline values in shared memory (a panel of baselines at a time when
// they do not all fit), the model recomputed from the solution where it is
// needed.  The sums over each antenna's and each unique baseline's
// baselines are gathers over a fixed incidence list (CSR), each segment
// summed by a fixed group of lanes in a fixed order, so the result does not
// depend on scheduling and repeats bit for bit.  In float32, most arrays
// of 31 to 256 antennas whose baselines are distinct antenna pairs take a kernel
// of their own (omnical_dense_kernel).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <numeric>
#include <vector>

#include "heravis.h"
#include "hv_kernels.h"

namespace {

template <typename R> struct Cx;
template <> struct Cx<float> { using T = float2; };
template <> struct Cx<double> { using T = double2; };

// Launch and loop shape, as measured best on GB300 (float32 / float64):
//   OM_UNROLL_*  baselines a thread takes per pass of the per-baseline loops
//   OM_GATHER_*  incidence entries a lane loads ahead in the segment gathers
//   OM_MINB      CTAs of 512 threads an SM (2: 64 registers a thread)
//   OM_WANT_*    CTAs of 512 threads an SM the panels of baselines are sized for
#ifndef OM_UNROLL_F
#define OM_UNROLL_F 1
#define OM_UNROLL_D 1
#define OM_GATHER_F 4
#define OM_GATHER_D 2
#endif
#ifndef OM_MINB
#define OM_MINB 2
#endif
#ifndef OM_WANT_F
#define OM_WANT_F 2
#define OM_WANT_D 2
#endif
constexpr int kOmMaxThreads = 512;
constexpr int kOmSmemLimit = 226 * 1024;  // dynamic shared memory, below the 227 KB per CTA
constexpr int kOmThreadsPerSm = 1024 * (OM_MINB > 2 ? 2 : OM_MINB) / 2;  // register limit

template <typename R>
struct OmParams {
  int ndata, nants, nubls, nbls;
  int panel, npanels;     // baselines per panel (the last may be shorter), panels
  const uint2* bl;        // [nbls] (i | j << 16, k)
  const int* seg_off;     // [npanels][nants + nubls + 1] into seg_ent
  const uint32_t* seg_ent;// baseline within its panel | (conjugate << 31)
  const int* seg_ord;     // float64: [npanels][nants + nubls] segments, longest first
  const typename Cx<R>::T* data;  // [ndata][nbls]
  const R* wgts;                  // [ndata][nbls]
  typename Cx<R>::T* gains;       // [ndata][nants], in/out
  typename Cx<R>::T* ubls;        // [ndata][nubls], in/out
  R* chisq;
  R* conv;
  uint32_t* iters;
  R conv_crit;
  float gstep;
  int maxiter, check_every, check_after;
  int group;       // lanes per segment in the gathers (1, 2, 4, 8, 16 or 32)
  int sum_threads; // threads whose order the sums over the block follow (>= blockDim.x)
  int* counter;    // next problem
};

template <typename C>
__device__ __forceinline__ C cmul(C a, C b) {
  C r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
template <typename C>
__device__ __forceinline__ C conjc(C a) {
  a.y = -a.y;
  return a;
}
template <typename C>
__device__ __forceinline__ auto mag2(C a) -> decltype(a.x) {
  return a.x * a.x + a.y * a.y;
}

// g[i] conj(g[j]) u[k] (gen_dmdl, redcal.py:70-94); sol = g | u
template <typename C>
__device__ __forceinline__ C model(const C* sol, int nants, uint2 e) {
  return cmul(cmul(sol[e.x & 0xffffu], conjc(sol[e.x >> 16])), sol[nants + e.y]);
}

// Sum of three values over the block, in a fixed order; every thread gets
// the sums.  red: 3 * 32 values of shared memory.
template <typename R>
__device__ void block_sum3(R& a, R& b, R& c, R* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  __syncthreads();  // red may still be read from the last call
  if (lane == 0) {
    red[warp] = a;
    red[32 + warp] = b;
    red[64 + warp] = c;
  }
  __syncthreads();
  a = red[0];
  b = red[32];
  c = red[64];
  for (int w = 1; w < nw; ++w) {
    a += red[w];
    b += red[32 + w];
    c += red[64 + w];
  }
}

// The same for the values that part(v, a, b, c) gives for each of nv threads (a
// multiple of 32, at least blockDim.x): a CTA of fewer threads takes several
// each, in the order in which nv threads would be added.
template <typename R, typename Part>
__device__ __forceinline__ void block_sum3_of(int nv, Part part, R& a, R& b, R& c, R* red) {
  __syncthreads();  // red may still be read from the last call
  for (int v = threadIdx.x; v < nv; v += blockDim.x) {
    a = b = c = 0;
    part(v, a, b, c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
      c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if ((v & 31) == 0) {
      red[v >> 5] = a;
      red[32 + (v >> 5)] = b;
      red[64 + (v >> 5)] = c;
    }
  }
  __syncthreads();
  a = red[0];
  b = red[32];
  c = red[64];
  for (int w = 1; w < nv >> 5; ++w) {
    a += red[w];
    b += red[32 + w];
    c += red[64 + w];
  }
}

// For every segment s of the incidence list: a group of G lanes sums
// val(entry) over the segment's entries (lane l takes entries l, l + G, ...,
// kGU at a time, added in that order; then a butterfly over the group) and
// lane 0 of the group calls out(s, sum).  With kOrd (float64) the groups take
// the segments in the order ord, by falling length, so that those of a warp are
// about as long; in float32 the look-up cost 5% and gained nothing.  The loop
// over segments is uniform across the block, so every lane takes part in every
// shuffle.
template <bool kOrd, int kGU, typename V, typename Val, typename Out>
__device__ __forceinline__ void seg_gather(const int* __restrict__ off,
                                           const uint32_t* __restrict__ ent,
                                           const int* __restrict__ ord, int nseg, int G, Val val,
                                           Out out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per_warp = 32 / G, ngroups = (blockDim.x >> 5) * per_warp;
  const int gid = warp * per_warp + lane / G, gl = lane & (G - 1);
  for (int base = 0; base < nseg; base += ngroups) {
    const bool has = base + gid < nseg;
    const int s = kOrd && has ? __ldg(ord + base + gid) : base + gid;
    V acc = V{};
    if (has) {
      const int e1 = __ldg(off + s + 1);
      int e = __ldg(off + s) + gl;
      for (; e + (kGU - 1) * G < e1; e += kGU * G) {
        uint32_t x[kGU];
#pragma unroll
        for (int q = 0; q < kGU; ++q) x[q] = __ldg(ent + e + q * G);
#pragma unroll
        for (int q = 0; q < kGU; ++q) acc = acc + val(x[q]);
      }
      for (; e < e1; e += G) acc = acc + val(__ldg(ent + e));
    }
    for (int o = G >> 1; o > 0; o >>= 1) acc = acc + V::shfl_xor(acc, o);
    if (gl == 0 && has) out(s, acc);
  }
}

// Values summed by seg_gather.
template <typename R>
struct RealV {
  R v;
  __device__ RealV operator+(RealV o) const { return RealV{v + o.v}; }
  __device__ static RealV shfl_xor(RealV a, int o) {
    return RealV{__shfl_xor_sync(0xffffffffu, a.v, o)};
  }
};
template <typename R>
struct CplxV {
  R x, y;
  __device__ CplxV operator+(CplxV o) const { return CplxV{x + o.x, y + o.y}; }
  __device__ static CplxV shfl_xor(CplxV a, int o) {
    return CplxV{__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o)};
  }
};

// Baselines per thread per pass of the per-baseline loops, their loads
// issued before any of their stores.
template <typename R> struct Unroll {
  static constexpr int n = sizeof(R) == 4 ? OM_UNROLL_F : OM_UNROLL_D;
  static constexpr int gather = sizeof(R) == 4 ? OM_GATHER_F : OM_GATHER_D;  // seg_gather
};

// sum_b |data_b - model_b|^2 w_b over the baselines of thread tid of nt
// (calc_chisq, redcal.py:97-114)
template <typename R, typename C>
__device__ __forceinline__ R chisq_part(const C* sol, int nants, const uint2* __restrict__ bl,
                                        const C* data, const R* wgt, int nbls, int tid, int nt) {
  constexpr int U = Unroll<R>::n;
  R acc = 0;
  for (int b0 = tid; b0 < nbls; b0 += U * nt) {
    uint2 e[U];
    C x[U];
    R w[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const int b = b0 + q * nt;
      if (b < nbls) {
        e[q] = bl[b];
        x[q] = data[b];
        w[q] = wgt[b];
      }
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      if (b0 + q * nt < nbls) {
        const C m = model(sol, nants, e[q]);
        const R dx = x[q].x - m.x, dy = x[q].y - m.y;
        acc += (dx * dx + dy * dy) * w[q];
      }
    }
  }
  return acc;
}

// One CTA per problem.  Shared memory, per segment (antennas, then unique
// baselines): the solution and the stepped solution (complex, swapped after
// each accepted step; the stepped one also holds the partial sums of the
// panels before the last), the weights gwgt | uwgt, the magnitudes when they
// were formed and their ratios to the current ones; reduction scratch; d for
// one panel of baselines (complex; also the weights dwgts while they are
// formed); with one panel, data and w too (kDataShared), else they are read
// from global memory (the L2 keeps a problem's rows across its iterations).
//
// The baselines are taken a panel at a time: the per-baseline values of a
// panel, then its gathers, the panel sums added in panel order.  Panels keep
// the shared memory of a CTA small enough for two CTAs an SM.
//
// dwgts_b / |dmdl_b|^2 of calc_gu_buf (redcal.py:219) is
// w_b |m0_b|^2 / |m_b|^2 with m0 the model when the weights were formed;
// |m_b|^2 = |g_i|^2 |g_j|^2 |u_k|^2, so the factor is taken as
// w_b ra_i ra_j ru_k with ra = |g0|^2 / |g|^2 per antenna and ru per unique
// baseline: nants + nubls divisions an iteration instead of nbls.
//
// kFactored (float64, which is bound by the FP64 pipe): the ratios are kept
// multiplied into the factors, p_a = conj(g_a) ra_a and c_k = conj(u_k) ru_k,
// so that d_b = data_b w_b p_i conj(p_j) c_k takes 14 operations instead of 17,
// and 12 where data w is kept in shared memory (chi^2 reads the data again);
// the weights come from the factors' magnitudes (3 instead of 11), and gain /
// weight is divided when the weights are formed.  12 iterations of 1000 problems
// of 54 antennas: 1.72 ms without, 1.52 with data and w kept apart and the
// segments gathered in their own order, 1.35 now; 200 of 180 antennas 5.05, 4.42
// and 4.07 ms.  It takes 8 bytes more of shared memory a segment; problems that
// only fit without it go without.
template <typename R, bool kDataShared, bool kFactored>
__global__ void __launch_bounds__(kOmMaxThreads, OM_MINB) omnical_kernel(const OmParams<R> p) {
  using C = typename Cx<R>::T;
  constexpr int U = Unroll<R>::n;
  extern __shared__ __align__(16) unsigned char smem[];
  const int nants = p.nants, nubls = p.nubls, nbls = p.nbls, nseg = nants + nubls;
  const int PB = p.panel, np = p.npanels;
  C* const solA = reinterpret_cast<C*>(smem);
  C* const solB = solA + nseg;
  R* const gw = reinterpret_cast<R*>(solB + nseg);  // gwgt | uwgt
  R* const mg0 = gw + nseg;                         // |g0|^2 | |u0|^2
  R* const ra = mg0 + nseg;                         // ratios
  R* const red = ra + (kFactored ? 2 : 1) * nseg;   // 96 values
  C* const pc = reinterpret_cast<C*>(ra);           // kFactored: p | c instead of the ratios
  unsigned char* next = reinterpret_cast<unsigned char*>(red + 96);
  next = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(next) + 15) & ~uintptr_t(15));
  C* const d = reinterpret_cast<C*>(next);
  R* const dw = reinterpret_cast<R*>(d);
  C* const sdata = d + PB;
  R* const sw = reinterpret_cast<R*>(sdata + nbls);
  __shared__ int s_prob;

  const int tid = threadIdx.x, nt = blockDim.x, nv = p.sum_threads;
  const R one_m = (R)(1.0f - p.gstep);  // formed in float, as the reference
  const R gs = (R)p.gstep;
  const uint2* __restrict__ bl = p.bl;

  for (;;) {
    __syncthreads();  // the last problem's reads of s_prob and shared arrays are done
    if (tid == 0) s_prob = atomicAdd(p.counter, 1);
    __syncthreads();
    const int prob = s_prob;
    if (prob >= p.ndata) return;
    const C* const gdata = p.data + (size_t)prob * nbls;
    const R* const gwgt = p.wgts + (size_t)prob * nbls;
    for (int a = tid; a < nants; a += nt) solA[a] = p.gains[(size_t)prob * nants + a];
    for (int k = tid; k < nubls; k += nt) solA[nants + k] = p.ubls[(size_t)prob * nubls + k];
    if (kDataShared) {
      for (int b = tid; b < nbls; b += nt) {
        C x = __ldg(gdata + b);
        const R w = __ldg(gwgt + b);
        if (kFactored) {  // data w: what an iteration needs
          x.x *= w;
          x.y *= w;
        }
        sdata[b] = x;
        sw[b] = w;
      }
    }
    const C* const data = kDataShared ? sdata : gdata;
    const C* const cdata = kDataShared && !kFactored ? sdata : gdata;  // for chi^2
    const R* const wgt = kDataShared ? sw : gwgt;
    __syncthreads();
    C *sol = solA, *nsol = solB;

    // chi^2 of the starting solution (redcal.py:566-577)
    R chisq, z1, z2;
    block_sum3_of<R>(nv, [&](int v, R& x, R&, R&) {
      x = chisq_part<R>(sol, nants, bl, cdata, wgt, nbls, v, nv);
    }, chisq, z1, z2, red);
    R conv = 0;
    uint32_t iters = 0;

    for (int it = 1; it <= p.maxiter; ++it) {
      if (it % p.check_every == 1) {
        // weights from the current model (calc_dwgts, calc_gu_wgt)
        for (int s = tid; s < nseg; s += nt) {
          mg0[s] = mag2(sol[s]);
          if constexpr (kFactored) pc[s] = conjc(sol[s]);
          else ra[s] = 1;
        }
        if (kFactored) __syncthreads();  // the magnitudes are read below
        for (int pn = 0; pn < np; ++pn) {
          const int b0 = pn * PB, nb = min(PB, nbls - b0);
          for (int b = tid; b < nb; b += nt) {
            const uint2 e = bl[b0 + b];
            if constexpr (kFactored)
              dw[b] = mg0[e.x & 0xffffu] * mg0[e.x >> 16] * (mg0[nants + e.y] * wgt[b0 + b]);
            else
              dw[b] = mag2(model(sol, nants, e)) * wgt[b0 + b];
          }
          __syncthreads();
          seg_gather<sizeof(R) == 8, Unroll<R>::gather, RealV<R>>(
              p.seg_off + (size_t)pn * (nseg + 1), p.seg_ent,
              p.seg_ord + (size_t)pn * nseg, nseg, p.group,
              [&](uint32_t e) { return RealV<R>{dw[e & 0x7fffffffu]}; },
              [&](int s, RealV<R> v) {
                const R x = pn ? gw[s] + v.v : v.v;
                gw[s] = kFactored && pn == np - 1 ? gs / x : x;
              });
          __syncthreads();  // dw is overwritten below
        }
      } else {
        for (int s = tid; s < nseg; s += nt) {
          const R q = mg0[s] / mag2(sol[s]);
          if constexpr (kFactored) {
            C c = conjc(sol[s]);
            c.x *= q;
            c.y *= q;
            pc[s] = c;
          } else {
            ra[s] = q;
          }
        }
        __syncthreads();
      }
      // d_b = data_b conj(m_b) dwgts_b / |m_b|^2 (calc_gu_buf), summed per
      // antenna and unique baseline, then the step (update_gains/_ubls)
      for (int pn = 0; pn < np; ++pn) {
        const int b0 = pn * PB, nb = min(PB, nbls - b0);
        for (int c0 = tid; c0 < nb; c0 += U * nt) {
          uint2 e[U];
          C x[U];
          R w[U];
#pragma unroll
          for (int q = 0; q < U; ++q)
            if (c0 + q * nt < nb) {
              e[q] = bl[b0 + c0 + q * nt];
              x[q] = data[b0 + c0 + q * nt];
              if (!(kFactored && kDataShared)) w[q] = wgt[b0 + c0 + q * nt];
            }
#pragma unroll
          for (int q = 0; q < U; ++q)
            if (c0 + q * nt < nb) {
              const int i = e[q].x & 0xffffu, j = e[q].x >> 16;
              C z;
              if constexpr (kFactored) {
                if constexpr (!kDataShared) {
                  x[q].x *= w[q];
                  x[q].y *= w[q];
                }
                z = cmul(cmul(x[q], cmul(pc[i], conjc(pc[j]))), pc[nants + e[q].y]);
              } else {
                const C m = model(sol, nants, e[q]);
                const R t = w[q] * ra[i] * ra[j] * ra[nants + e[q].y];
                z = cmul(x[q], conjc(m));
                z.x *= t;
                z.y *= t;
              }
              d[c0 + q * nt] = z;
            }
        }
        __syncthreads();
        const bool last = pn == np - 1;
        seg_gather<sizeof(R) == 8, Unroll<R>::gather, CplxV<R>>(
            p.seg_off + (size_t)pn * (nseg + 1), p.seg_ent,
            p.seg_ord + (size_t)pn * nseg, nseg, p.group,
            [&](uint32_t e) {
              const C z = d[e & 0x7fffffffu];
              return CplxV<R>{z.x, (e >> 31) ? -z.y : z.y};
            },
            [&](int s, CplxV<R> v) {
              if (pn) {
                v.x = nsol[s].x + v.x;
                v.y = nsol[s].y + v.y;
              }
              C f;
              if (!last) {
                f.x = v.x;
                f.y = v.y;
                nsol[s] = f;  // partial sum
                return;
              }
              if constexpr (kFactored) {
                const R q = gw[s];  // gain / weight
                f.x = one_m + q * v.x;
                f.y = q * v.y;
              } else {
                f.x = one_m + gs * v.x / gw[s];
                f.y = gs * v.y / gw[s];
              }
              nsol[s] = cmul(sol[s], f);
            });
        __syncthreads();
      }
      const bool check = !(it < p.maxiter && (it < p.check_after || it % p.check_every != 0));
      if (!check) {
        C* t = sol; sol = nsol; nsol = t;
        continue;
      }
      // convergence and chi^2 of the stepped solution (calc_conv,
      // calc_chisq, update_active)
      R nchisq, csum, cwgt;
      block_sum3_of<R>(nv, [&](int v, R& x2, R& cs, R& cw) {
        x2 = chisq_part<R>(nsol, nants, bl, cdata, wgt, nbls, v, nv);
        for (int s = v; s < nseg; s += nv) {
          const C x = nsol[s], y = sol[s];
          const R dx = x.x - y.x, dy = x.y - y.y;
          cs += dx * dx + dy * dy;
          cw += mag2(x);
        }
      }, nchisq, csum, cwgt, red);
      conv = sqrt(csum / cwgt);
      if (conv < p.conv_crit || nchisq > chisq) break;
      chisq = nchisq;
      iters = (uint32_t)it;
      C* t = sol; sol = nsol; nsol = t;
    }
    __syncthreads();
    for (int a = tid; a < nants; a += nt) p.gains[(size_t)prob * nants + a] = sol[a];
    for (int k = tid; k < nubls; k += nt) p.ubls[(size_t)prob * nubls + k] = sol[nants + k];
    if (tid == 0) {
      p.chisq[prob] = chisq;
      p.conv[prob] = conv;
      p.iters[prob] = iters;
    }
  }
}

// ------------------------------------------------------- dense kernel ----
// Arrays whose baselines are antenna pairs, each pair at most once (the usual
// case), seen as the lower triangle of the antenna matrix: a group of GL lanes
// takes a row r, lane l its columns l, l + GL, ... below r, the same ones in
// every row.  The column antennas' sums so stay in registers, the row antenna's
// factor is one broadcast, its sum a register until the row's butterfly, and a
// baseline costs the column antenna's factor (read again in every row, consecutive
// lanes at consecutive places), one gather (its unique baseline's factor) and one
// read-modify-write (its sum) in shared memory.  The general kernel above gathers
// six solution values, stores d and reads it back three times through incidence
// lists, a panel of baselines at a time.
//
// Sums of unique baselines: every group has two private copies (one for pairs
// stored as (row, column), one for (column, row)), added up in a fixed order
// after the pass; the plan makes sure that no unique baseline occurs twice
// among the lanes that write a copy at the same time.  So the result does not
// depend on scheduling.
//
// With p_a = conj(g_a) |g0_a|^2 / |g_a|^2 and c_k likewise for u_k,
//   d_b = data_b w_b p_i conj(p_j) c_k
// (see the general kernel); for a pair stored as (column, row) the conjugate
// is formed, from the conjugates of data and c_k.
//
// float32 only: float64 is bound by the FP64 pipe, where adding up the private
// copies costs more than the gathers (54 antennas, 1000 problems, 12
// iterations: 2.1 ms, general kernel 1.7 ms).
//
// Bound by issue slots (68% busy at 180 antennas) and the shared-memory pipe
// (79%: gathers and updates at the unique baselines' scattered places).
// Measured on GB300, 12 iterations of 2000 problems, general kernel and this
// one: 180 antennas 3.70 and 2.48 ms, 128 antennas 2.84 and 1.64 ms, 54
// antennas 0.44 and 0.36 ms.
//
// It is taken where it is not slower than the general kernel, be the problems few
// or many: their number must not decide, since a problem gives the same result
// alone or among others.  Measured over 10 to 2000 problems (time over the
// general kernel's, few and many problems):
//  * smaller arrays stay with the general kernel (4000 problems of 20 antennas
//    148 and 165 us, 28 antennas 237 and 237, 31 antennas 335 and 292), and so do
//    arrays of 65 to 87, whose few warps a problem are slower while a call has few
//    problems (70 antennas 1.11 and 0.97, 80 1.02 and 0.91, 84 1.18 and 0.95; 88
//    0.96 and 0.81);
//  * the two copies of the unique baselines' sums a group are cleared and added
//    up in every iteration, which counts for arrays of up to 64 antennas: they may
//    have kDenseCopies sums for a pair of antennas, a full hexagon has 1.9 to 2.8
//    (54 antennas: 3.3 sums 0.98 and 0.84, 4.4 1.15 and 0.96; 62: 2.9 sums 0.93
//    and 0.85, 3.8 1.06 and 0.86);
//  * the copies also fill the shared memory.  One CTA an SM is enough for 108 to
//    128 antennas, whose general kernel takes long rows (128 antennas, 723 unique
//    baselines: 0.74 and 0.78), and from 225 on (225: 0.68 and 1.02), elsewhere
//    two are needed (96 antennas: 277 unique baselines, two CTAs, 0.85 and 0.79;
//    370, one, 0.71 and 1.05; 150: 568, two, 0.93 and 0.87; 852, one, 0.75 and
//    1.22).
constexpr int kDenseMinAnts = 31, kDenseMaxAnts = 256;
constexpr int kDenseGap0 = 65, kDenseGap1 = 87;
constexpr double kDenseCopies = 3.5;
constexpr int kDenseThreads = 256;
constexpr uint32_t kNoPair = 0x7fffu;  // slot without a baseline (256 antennas: < 32640 pairs)

struct DenseParams {
  int ndata, nants, nubls, nbls;
  const int* row_off;    // [nants] first slot of each row
  const uint32_t* slots; // baseline | (column, row) order << 15 | unique baseline << 16
  const float2* data;
  const float* wgts;
  float2* gains;
  float2* ubls;
  float* chisq;
  float* conv;
  uint32_t* iters;
  float conv_crit;
  float gstep;
  int maxiter, check_every, check_after;
  int* counter;
};

size_t dense_smem(int nants, int nubls, int groups) {
  const size_t nseg = (size_t)nants + nubls;
  return sizeof(float2) * (3 * nseg + 2 * (size_t)groups * nubls + (size_t)groups * nants + nants) +
         sizeof(float) * (2 * nseg + 96) + 16;
}

// Sum of the n partial sums part(i), each cleared after it was read (clear(i)):
// four running sums, added pairwise at the end, since one running sum's error
// grows with its 16 or 32 additions (gains of 53 antennas after 12 iterations
// 9.7e-8 from 64 bits, 7.8e-8 this way and in the general kernel).
template <typename V, typename Part, typename Clear>
__device__ __forceinline__ V sum_parts(int n, Part part, Clear clear) {
  V a[4] = {V{}, V{}, V{}, V{}};
  int i = 0;
#pragma unroll 1
  for (; i + 4 <= n; i += 4) {
    V x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = part(i + q);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      clear(i + q);
      a[q] = a[q] + x[q];
    }
  }
#pragma unroll 1
  for (; i < n; ++i) {
    a[0] = a[0] + part(i);
    clear(i);
  }
  return (a[0] + a[1]) + (a[2] + a[3]);
}

template <int GL, int NB>
__global__ void __launch_bounds__(kDenseThreads, NB <= 6 ? 3 : 2)
omnical_dense_kernel(const DenseParams p) {
  using R = float;
  using C = float2;
  constexpr int GW = 32 / GL;  // groups a warp
  extern __shared__ __align__(16) unsigned char smem[];
  const int nants = p.nants, nubls = p.nubls, nbls = p.nbls, nseg = nants + nubls;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarps = blockDim.x >> 5, ngroups = nwarps * GW;
  const int grp = warp * GW + lane / GL, gl = lane & (GL - 1);
  const int tid = threadIdx.x, nt = blockDim.x;
  C* const solA = reinterpret_cast<C*>(smem);
  C* const solB = solA + nseg;
  C* const pc = solB + nseg;                  // p | c
  C* const ucopy = pc + nseg;                 // [group][order][nubls]
  C* const colsum = ucopy + 2 * ngroups * nubls;  // [group][nants]
  C* const rowsum = colsum + ngroups * nants;     // [nants]
  R* const gw = reinterpret_cast<R*>(rowsum + nants);  // gwgt | uwgt
  R* const mg0 = gw + nseg;                   // |g0|^2 | |u0|^2
  R* const red = mg0 + nseg;                  // 96 values
  __shared__ int s_prob;
  const R one_m = (R)(1.0f - p.gstep);  // formed in float, as the reference
  const R gs = (R)p.gstep;

  for (;;) {
    __syncthreads();
    if (tid == 0) s_prob = atomicAdd(p.counter, 1);
    __syncthreads();
    const int prob = s_prob;
    if (prob >= p.ndata) return;
    const C* const __restrict__ data = p.data + (size_t)prob * nbls;
    const R* const __restrict__ wgt = p.wgts + (size_t)prob * nbls;
    for (int s = tid; s < nseg; s += nt) {
      const C x = s < nants ? p.gains[(size_t)prob * nants + s]
                            : p.ubls[(size_t)prob * nubls + (s - nants)];
      solA[s] = x;
      pc[s] = conjc(x);
      mg0[s] = mag2(x);
    }
    for (int i = tid; i < 2 * ngroups * nubls; i += nt) ucopy[i] = C{};
    if (tid == 0) rowsum[0] = C{};
    __syncthreads();
    C *sol = solA, *nsol = solB;

    // Every pair of this group, a row at a time: the data and weights of the
    // whole row are loaded together (its slots were while the row before was
    // worked on), then row_begin(row), pair(chunk, valid, swapped, unique
    // baseline, data, weight) for each chunk (converged: the chunk loop is
    // uniform across the warp) and row_end(row).  A chunk's column antenna is
    // chunk * GL + gl (past nants where the pair is not valid: a read within
    // the shared arrays, unused).
    auto rows = [&](auto&& row_begin, auto&& pair, auto&& row_end) {
      auto load_slots = [&](int rw, uint32_t (&e)[NB]) {
        const uint32_t* slot = p.slots + __ldg(p.row_off + max(rw - lane / GL, 0)) + gl;
#pragma unroll
        for (int cb = 0; cb < NB; ++cb) e[cb] = cb * GL < rw ? __ldg(slot + cb * GL) : kNoPair;
      };
      uint32_t e[NB];
      int rw = nants - 1 - warp * GW;
      load_slots(rw, e);
#pragma unroll 1
      for (; rw >= 1; rw -= ngroups) {
        C d[NB];
        R w[NB];
        uint32_t en[NB];
#pragma unroll
        for (int cb = 0; cb < NB; ++cb) {
          const uint32_t b = e[cb] & kNoPair;
          d[cb] = b != kNoPair ? __ldg(data + b) : C{};
          w[cb] = b != kNoPair ? __ldg(wgt + b) : R(0);
        }
        load_slots(rw - ngroups, en);
        const int r = max(rw - lane / GL, 0);
        row_begin(r);
#pragma unroll
        for (int cb = 0; cb < NB; ++cb)
          if (cb * GL < rw)
            pair(cb, (e[cb] & kNoPair) != kNoPair, (int)((e[cb] >> 15) & 1u), (int)(e[cb] >> 16),
                 d[cb], w[cb]);
        row_end(r);
#pragma unroll
        for (int cb = 0; cb < NB; ++cb) e[cb] = en[cb];
      }
    };
    auto group_sum = [&](R v) {
#pragma unroll
      for (int o = GL / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      return v;
    };
    C* const my_u = ucopy + 2 * grp * nubls;
    // sum |data - model|^2 w of a solution over this thread's pairs
    auto chisq_part = [&](const C* x) {
      R acc = 0;
      C gr{};
      rows([&](int r) { gr = x[r]; },
           [&](int cb, bool ok, int sw, int k, C d, R w) {
             if (!ok) return;
             C u = x[nants + k];
             if (sw) {
               u = conjc(u);
               d = conjc(d);
             }
             const C m = cmul(cmul(gr, conjc(x[cb * GL + gl])), u);
             const R dx = d.x - m.x, dy = d.y - m.y;
             acc += (dx * dx + dy * dy) * w;
           },
           [&](int) {});
      return acc;
    };

    // chi^2 of the starting solution (redcal.py:566-577)
    R chisq = chisq_part(sol), z1 = 0, z2 = 0;
    block_sum3(chisq, z1, z2, red);
    R conv = 0;
    uint32_t iters = 0;

    for (int it = 1; it <= p.maxiter; ++it) {
      if (it % p.check_every == 1) {
        // weights from the current model (calc_dwgts, calc_gu_wgt): |m|^2 w
        R col[NB];
#pragma unroll
        for (int cb = 0; cb < NB; ++cb) col[cb] = 0;
        C gr{};
        R row = 0;
        rows([&](int r) {
               row = 0;
               gr = sol[r];
             },
             [&](int cb, bool ok, int sw, int k, C, R w) {
               R dw = 0;
               if (ok) {
                 const C u = sol[nants + k];
                 dw = mag2(cmul(cmul(gr, conjc(sol[cb * GL + gl])), sw ? conjc(u) : u)) * w;
                 my_u[sw * nubls + k].x += dw;
               }
               row += dw;
               col[cb] += dw;
               __syncwarp();
             },
             [&](int r) {
               const R v = group_sum(row);
               if (gl == 0) rowsum[r].x = v;
             });
#pragma unroll
        for (int cb = 0; cb < NB; ++cb)
          if (cb * GL + gl < nants) colsum[grp * nants + cb * GL + gl].x = col[cb];
        __syncthreads();
        for (int s = tid; s < nseg; s += nt) {
          R v;
          if (s < nants) {
            v = sum_parts<RealV<R>>(
                    ngroups, [&](int g) { return RealV<R>{colsum[g * nants + s].x}; },
                    [](int) {}).v;
            if (s) v += rowsum[s].x;
          } else {
            C* const u = ucopy + (s - nants);
            v = sum_parts<RealV<R>>(
                    2 * ngroups, [&](int c) { return RealV<R>{u[c * nubls].x}; },
                    [&](int c) { u[c * nubls].x = 0; }).v;
          }
          gw[s] = v;
        }
        __syncthreads();
      }
      // d_b of every pair (calc_gu_buf), summed per antenna and unique
      // baseline, then the step (update_gains/_ubls)
      {
        C col[NB];
#pragma unroll
        for (int cb = 0; cb < NB; ++cb) col[cb] = C{};
        C gr{}, row{};
        rows([&](int r) {
               row = C{};
               gr = pc[r];
             },
             [&](int cb, bool ok, int sw, int k, C d, R w) {
               if (ok) {
                 C c = pc[nants + k];
                 if (sw) {
                   c = conjc(c);
                   d = conjc(d);
                 }
                 d.x *= w;
                 d.y *= w;
                 const C z = cmul(cmul(d, cmul(gr, conjc(pc[cb * GL + gl]))), c);
                 row.x += z.x;
                 row.y += z.y;
                 col[cb].x += z.x;
                 col[cb].y -= z.y;
                 C& u = my_u[sw * nubls + k];
                 C t = u;
                 t.x += z.x;
                 t.y += sw ? -z.y : z.y;
                 u = t;
               }
               __syncwarp();
             },
             [&](int r) {
               const R x = group_sum(row.x), y = group_sum(row.y);
               if (gl == 0) {
                 C t;
                 t.x = x;
                 t.y = y;
                 rowsum[r] = t;
               }
             });
#pragma unroll
        for (int cb = 0; cb < NB; ++cb)
          if (cb * GL + gl < nants) colsum[grp * nants + cb * GL + gl] = col[cb];
      }
      __syncthreads();
      const bool rebase = (it + 1) % p.check_every == 1;
      for (int s = tid; s < nseg; s += nt) {
        CplxV<R> v;
        if (s < nants) {
          v = sum_parts<CplxV<R>>(
              ngroups,
              [&](int g) {
                const C t = colsum[g * nants + s];
                return CplxV<R>{t.x, t.y};
              },
              [](int) {});
          if (s) v = v + CplxV<R>{rowsum[s].x, rowsum[s].y};
        } else {
          C* const u = ucopy + (s - nants);
          v = sum_parts<CplxV<R>>(
              2 * ngroups,
              [&](int c) {
                const C t = u[c * nubls];
                return CplxV<R>{t.x, t.y};
              },
              [&](int c) { u[c * nubls] = C{}; });
        }
        C f;
        f.x = one_m + gs * v.x / gw[s];
        f.y = gs * v.y / gw[s];
        const C x = cmul(sol[s], f);
        nsol[s] = x;
        // the next iteration's factor: its weights are formed anew from x, or
        // those at hand go on
        C c = conjc(x);
        if (rebase) {
          mg0[s] = mag2(x);
        } else {
          const R q = mg0[s] / mag2(x);
          c.x *= q;
          c.y *= q;
        }
        pc[s] = c;
      }
      __syncthreads();
      const bool check = !(it < p.maxiter && (it < p.check_after || it % p.check_every != 0));
      if (check) {
        // convergence and chi^2 of the stepped solution (calc_conv,
        // calc_chisq, update_active)
        R nchisq = chisq_part(nsol), csum = 0, cwgt = 0;
        for (int s = tid; s < nseg; s += nt) {
          const C x = nsol[s], y = sol[s];
          const R dx = x.x - y.x, dy = x.y - y.y;
          csum += dx * dx + dy * dy;
          cwgt += mag2(x);
        }
        block_sum3(nchisq, csum, cwgt, red);
        conv = sqrt(csum / cwgt);
        if (conv < p.conv_crit || nchisq > chisq) break;
        chisq = nchisq;
        iters = (uint32_t)it;
      }
      C* t = sol; sol = nsol; nsol = t;
    }
    __syncthreads();
    for (int s = tid; s < nseg; s += nt) {
      if (s < nants) p.gains[(size_t)prob * nants + s] = sol[s];
      else p.ubls[(size_t)prob * nubls + (s - nants)] = sol[s];
    }
    if (tid == 0) {
      p.chisq[prob] = chisq;
      p.conv[prob] = conv;
      p.iters[prob] = iters;
    }
  }
}

// Launch shape of the dense kernel: lanes a row, chunks of columns a lane, and
// the table of pairs by row.
struct DensePlan {
  int gl = 0, nb = 0, threads = 0;
  std::vector<int> row_off;
  std::vector<uint32_t> slots;
};

// Rows of up to 128 antennas take half a warp: fewer idle lanes at the row's
// end (54 antennas: 77% busy, 61% with whole warps).
bool make_dense_plan(const uint32_t* ggu, int nbls, int nants, int nubls, DensePlan* pl) {
  if (nants < kDenseMinAnts || nants > kDenseMaxAnts ||
      (nants >= kDenseGap0 && nants <= kDenseGap1) || nbls < 1 || nubls < 1 || nubls > 65535 ||
      nbls > nants * (nants - 1) / 2)
    return false;
  pl->gl = nants <= 128 ? 16 : 32;
  const int need = (nants + pl->gl - 1) / pl->gl;
  pl->nb = pl->gl == 32 ? (need <= 6 ? 6 : 8) : need <= 2 ? 2 : need <= 4 ? 4 : need <= 6 ? 6 : 8;
  // a few rows a group: small arrays take few warps, so that more problems
  // share an SM
  const int gw = 32 / pl->gl;
  const int warps = std::max(1, std::min(kDenseThreads / 32, (nants + 3 * gw - 1) / (3 * gw)));
  pl->threads = 32 * warps;
  const size_t smem = dense_smem(nants, nubls, warps * gw);
  if (smem > (size_t)kOmSmemLimit) return false;
  if (nants <= 64 ? 2.0 * warps * gw * nubls > kDenseCopies * (nants * (nants - 1) / 2)
                  : (nants < 108 || (nants > 128 && nants < 225)) &&
                        2 * (smem + 1024) > (size_t)(228 * 1024))
    return false;
  // rows padded to whole chunks of the longest row of their warp's groups
  pl->row_off.resize(nants);
  int n = 0;
  for (int r = 0; r < nants; ++r) {
    pl->row_off[r] = n;
    n += (r + gw - 1 + pl->gl - 1) / pl->gl * pl->gl + (r + gw - 1 == 0 ? pl->gl : 0);
  }
  pl->slots.assign(n, kNoPair);
  for (int b = 0; b < nbls; ++b) {
    const uint32_t i = ggu[3 * b], j = ggu[3 * b + 1], k = ggu[3 * b + 2];
    if (i == j) return false;
    const uint32_t r = std::max(i, j), c = std::min(i, j);
    uint32_t& s = pl->slots[pl->row_off[r] + c];
    if (s != kNoPair) return false;  // the pair again
    s = (uint32_t)b | (i == r ? 0u : 0x8000u) | (k << 16);
  }
  // no unique baseline twice among the lanes that add to one copy at a time
  std::vector<int> seen(2 * (size_t)nubls, -1);
  int stamp = 0;
  for (int r = 1; r < nants; ++r)
    for (int c0 = 0; c0 < r; c0 += pl->gl, ++stamp)
      for (int c = c0; c < std::min(r, c0 + pl->gl); ++c) {
        const uint32_t s = pl->slots[pl->row_off[r] + c];
        if ((s & kNoPair) == kNoPair) continue;
        int& q = seen[(size_t)((s >> 15) & 1u) * nubls + (s >> 16)];
        if (q == stamp) return false;
        q = stamp;
      }
  return true;
}

using DenseFn = void (*)(DenseParams);
DenseFn dense_kernel(int gl, int nb) {
  if (gl == 32) return nb == 6 ? omnical_dense_kernel<32, 6> : omnical_dense_kernel<32, 8>;
  return nb == 2   ? omnical_dense_kernel<16, 2>
         : nb == 4 ? omnical_dense_kernel<16, 4>
         : nb == 6 ? omnical_dense_kernel<16, 6>
                   : omnical_dense_kernel<16, 8>;
}

struct Plan {
  int threads = 64, sum_threads = 64, group = 1, blocks_per_sm = 1, panel = 0, npanels = 1;
  bool data_shared = false, factored = false;
  size_t smem = 0;
};

// Launch shape: threads = about half the baselines (64 .. max_threads); everything
// in shared memory when that leaves 16 warps an SM, else panels of
// baselines sized for two CTAs (or the thread limit) an SM.
template <typename R>
int make_plan(int nants, int nubls, int nbls, bool factored, int max_threads, Plan* out) {
  using C = typename Cx<R>::T;
  Plan pl;
  const int t = ((nbls / 2 + 31) / 32) * 32;
  pl.threads = std::max(64, std::min(max_threads, t));
  const size_t nseg = (size_t)nants + nubls;
  pl.factored = factored;
  const size_t fixed =
      (2 * sizeof(C) + (factored ? 4 : 3) * sizeof(R)) * nseg + 96 * sizeof(R) + 16;
  auto per_sm = [&](size_t s) {
    return std::min(32, std::min(kOmThreadsPerSm / pl.threads, (int)((228 * 1024) / (s + 1024))));
  };
  const size_t all = fixed + (2 * sizeof(C) + sizeof(R)) * (size_t)nbls;
  if (all <= (size_t)kOmSmemLimit && per_sm(all) * pl.threads >= 512) {
    pl.data_shared = true;
    pl.panel = std::max(nbls, 1);
    pl.npanels = 1;
    pl.smem = all;
  } else {
    const int want = std::max(1, (sizeof(R) == 4 ? OM_WANT_F : OM_WANT_D) * 512 / pl.threads);
    const size_t target = std::min((size_t)kOmSmemLimit, (size_t)(228 * 1024) / want - 1024);
    if (fixed + 32 * sizeof(C) > target) return HV_ERR_ARG;
    const size_t pb = std::min((size_t)std::max(nbls, 1), (target - fixed) / sizeof(C));
    pl.npanels = (int)((nbls + pb - 1) / pb);
    pl.npanels = std::max(pl.npanels, 1);
    pl.panel = (nbls + pl.npanels - 1) / pl.npanels;
    pl.smem = fixed + sizeof(C) * (size_t)pl.panel;
  }
  pl.blocks_per_sm = std::max(1, per_sm(pl.smem));
  pl.sum_threads = pl.threads;
  // lanes per segment, a power of two <= 32, from the mean segment length
  // of a panel: float32 (latency-bound) about its square root; float64
  // (bound by the FP64 pipe, where each level of the butterfly over the
  // lanes costs adds) 2 from a length of 22 on (26 where data and weights are
  // in shared memory), 4 from four times that.  Measured, one and two lanes: 54
  // antennas (28.2, 256 threads) 1.38 and 1.27 ms, 45 (23.0) 1.29 and 1.36, 180
  // (22.8, panels) 4.36 and 4.08; two and four lanes: 61 (32.5) 1.32 and 1.44,
  // 135 (34.2, panels) 2.22 and 2.39.
  const double mean = nseg ? 3.0 * pl.panel / nseg : 1.0;
  int g = 1;
  if (sizeof(R) == 4)
    while (g < 32 && 4.0 * g * g <= mean) g *= 2;
  else
    while (g < 32 && (pl.data_shared ? 26.0 : 22.0) * g * g <= mean) g *= 2;
  pl.group = g;
  *out = pl;
  return HV_OK;
}

// The plan of a call.  Float64 problems whose data and weights are in shared
// memory take CTAs of 256 threads where a call has more than two problems an
// SM: more of them share it, and their barriers and serial sums overlap (54
// antennas, 1000 problems of 12 iterations: 1.43 and 1.35 ms; 37 antennas, 1500:
// 1.15 and 1.02), while few problems end sooner with 512 threads each (77
// antennas, 15 problems: 0.50 and 0.40 ms of 256 and 512).  Both
// sum in the same order, so that a problem gives the same result alone or among
// others.
template <typename R>
int choose_plan(int nants, int nubls, int nbls, bool factored, int ndata, int num_sms, Plan* out) {
  const int r = make_plan<R>(nants, nubls, nbls, factored, kOmMaxThreads, out);
  Plan few;
  if (sizeof(R) == 8 && r == HV_OK && out->data_shared && ndata > 2 * num_sms &&
      make_plan<R>(nants, nubls, nbls, factored, 256, &few) == HV_OK && few.data_shared) {
    few.sum_threads = out->threads;
    *out = few;
  }
  return r;
}

int fail(hv_context* ctx, int code, const char* msg) {
  if (ctx) hv_context_set_error(ctx, msg);
  return code;
}

int check_indices(hv_context* ctx, const uint32_t* ggu, int nbls, int nants, int nubls) {
  char msg[200];
  for (int b = 0; b < nbls; ++b) {
    const uint32_t i = ggu[3 * b], j = ggu[3 * b + 1], k = ggu[3 * b + 2];
    if (i >= (uint32_t)nants || j >= (uint32_t)nants || k >= (uint32_t)nubls) {
      snprintf(msg, sizeof msg, "omnical: baseline %d indexes (%u, %u, %u) out of range "
               "(%d antennas, %d unique baselines)", b, i, j, k, nants, nubls);
      return fail(ctx, HV_ERR_ARG, msg);
    }
  }
  return HV_OK;
}

// Incidence lists of the baselines, one per panel of `panel` baselines: for
// antenna a, the panel's baselines with i == a (as is) and j == a
// (conjugated); for unique baseline k, those with k; entries hold the
// baseline's index within its panel.
void build_csr(const uint32_t* ggu, int nbls, int nants, int nubls, int panel, int npanels, bool order,
               std::vector<uint2>& bl, std::vector<int>& off, std::vector<uint32_t>& ent) {
  const int nseg = nants + nubls;
  bl.resize(nbls);
  // the panels' offsets, then (order) each panel's segments by falling length
  off.assign((size_t)npanels * ((order ? 2 : 1) * nseg + 1), 0);
  ent.resize((size_t)3 * nbls);
  size_t base = 0;
  for (int pn = 0; pn < npanels; ++pn) {
    const int b0 = pn * panel, b1 = std::min(nbls, b0 + panel);
    int* o = off.data() + (size_t)pn * (nseg + 1);
    std::vector<int> cnt(nseg + 1, 0);
    for (int b = b0; b < b1; ++b) {
      cnt[ggu[3 * b] + 1]++;
      cnt[ggu[3 * b + 1] + 1]++;
      cnt[nants + ggu[3 * b + 2] + 1]++;
    }
    o[0] = (int)base;
    for (int s = 0; s < nseg; ++s) o[s + 1] = o[s] + cnt[s + 1];
    if (order) {
      int* ord = off.data() + (size_t)npanels * (nseg + 1) + (size_t)pn * nseg;
      std::iota(ord, ord + nseg, 0);
      std::stable_sort(ord, ord + nseg, [&](int x, int y) { return cnt[x + 1] > cnt[y + 1]; });
    }
    std::vector<int> pos(o, o + nseg);
    for (int b = b0; b < b1; ++b) {
      const uint32_t i = ggu[3 * b], j = ggu[3 * b + 1], k = ggu[3 * b + 2];
      bl[b] = make_uint2(i | (j << 16), k);
      ent[pos[i]++] = (uint32_t)(b - b0);
      ent[pos[j]++] = (uint32_t)(b - b0) | 0x80000000u;
      ent[pos[nants + k]++] = (uint32_t)(b - b0);
    }
    base = (size_t)o[nseg];
  }
}

int check_sizes(hv_context* ctx, int precision, int nbls, int nants, int nubls, int ndata,
                int maxiter, int check_every) {
  char msg[200];
  if ((precision != 1 && precision != 2) || nbls < 0 || nants < 0 || nubls < 0 || ndata < 0 ||
      maxiter < 0 || check_every <= 1 || nants > 65535 || nbls > 0x7fffffff / 3) {
    snprintf(msg, sizeof msg, "omnical: bad arguments (precision %d, %d baselines, %d antennas, "
             "%d unique baselines, %d problems, maxiter %d, check_every %d)", precision, nbls,
             nants, nubls, ndata, maxiter, check_every);
    return fail(ctx, HV_ERR_ARG, msg);
  }
  return HV_OK;
}

int run_dense(hv_context* ctx, const DensePlan& dp, int nbls, void* d_gains, int nants,
              void* d_ubls, int nubls, const void* d_data, const void* d_wgts, int ndata,
              double conv_crit, int maxiter, int check_every, int check_after, double gain,
              void* d_chisq, uint32_t* d_iters, void* d_conv, cudaStream_t st) {
  const DenseFn fn = dense_kernel(dp.gl, dp.nb);
  const size_t smem = dense_smem(nants, nubls, dp.threads / dp.gl);
  int per_sm = 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kOmSmemLimit) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, dp.threads, smem) != cudaSuccess)
    return HV_ERR_CUDA;
  const int grid = std::min(ndata, std::max(1, per_sm) * std::max(1, hv_context_num_sms(ctx)));
  const size_t n_off = sizeof(int) * dp.row_off.size(), n_slot = sizeof(uint32_t) * dp.slots.size();
  const size_t o_slot = (n_off + 255) & ~size_t(255), o_cnt = (o_slot + n_slot + 255) & ~size_t(255);
  void* buf = nullptr;
  if (hv_context_malloc(ctx, &buf, o_cnt + 256, st) != cudaSuccess) {
    cudaGetLastError();
    return fail(ctx, HV_ERR_OOM, "omnical: device allocation failed");
  }
  char* b8 = static_cast<char*>(buf);
  int r = HV_OK;
  if (cudaMemcpyAsync(b8, dp.row_off.data(), n_off, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(b8 + o_slot, dp.slots.data(), n_slot, cudaMemcpyHostToDevice, st) !=
          cudaSuccess ||
      cudaMemsetAsync(b8 + o_cnt, 0, sizeof(int), st) != cudaSuccess)
    r = HV_ERR_CUDA;
  if (r == HV_OK) {
    DenseParams p;
    p.ndata = ndata;
    p.nants = nants;
    p.nubls = nubls;
    p.nbls = nbls;
    p.row_off = reinterpret_cast<const int*>(b8);
    p.slots = reinterpret_cast<const uint32_t*>(b8 + o_slot);
    p.data = static_cast<const float2*>(d_data);
    p.wgts = static_cast<const float*>(d_wgts);
    p.gains = static_cast<float2*>(d_gains);
    p.ubls = static_cast<float2*>(d_ubls);
    p.chisq = static_cast<float*>(d_chisq);
    p.conv = static_cast<float*>(d_conv);
    p.iters = d_iters;
    p.conv_crit = (float)conv_crit;
    p.gstep = (float)gain;
    p.maxiter = maxiter;
    p.check_every = check_every;
    p.check_after = check_after;
    p.counter = reinterpret_cast<int*>(b8 + o_cnt);
    fn<<<grid, dp.threads, smem, st>>>(p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      hv_context_set_error(ctx, cudaGetErrorString(e));
      r = HV_ERR_CUDA;
    } else {
      hv_context_add_launches(ctx, 1);
    }
  }
  cudaFreeAsync(buf, st);
  return r;
}

template <typename R>
int run_typed(hv_context* ctx, const uint32_t* ggu, int nbls, void* d_gains, int nants,
              void* d_ubls, int nubls, const void* d_data, const void* d_wgts, int ndata,
              double conv_crit, int maxiter, int check_every, int check_after, double gain,
              void* d_chisq, uint32_t* d_iters, void* d_conv, cudaStream_t st) {
  int r = check_indices(ctx, ggu, nbls, nants, nubls);
  if (r != HV_OK) return r;
  if (ndata == 0) return HV_OK;
  if (sizeof(R) == 4) {
    DensePlan dp;
    if (make_dense_plan(ggu, nbls, nants, nubls, &dp))
      return run_dense(ctx, dp, nbls, d_gains, nants, d_ubls, nubls, d_data, d_wgts, ndata,
                       conv_crit, maxiter, check_every, check_after, gain, d_chisq, d_iters,
                       d_conv, st);
  }
  Plan pl;
  const int nsm = std::max(1, hv_context_num_sms(ctx));
  if ((sizeof(R) == 4 || choose_plan<R>(nants, nubls, nbls, true, ndata, nsm, &pl) != HV_OK) &&
      choose_plan<R>(nants, nubls, nbls, false, ndata, nsm, &pl) != HV_OK)
    return fail(ctx, HV_ERR_ARG, "omnical: too many antennas and unique baselines for one CTA");
  std::vector<uint2> bl;
  std::vector<int> off;
  std::vector<uint32_t> ent;
  build_csr(ggu, nbls, nants, nubls, pl.panel, pl.npanels, sizeof(R) == 8, bl, off, ent);
  const int grid = std::max(1, std::min(ndata, pl.blocks_per_sm * nsm));
  const size_t n_bl = sizeof(uint2) * bl.size(), n_off = sizeof(int) * off.size(),
               n_ent = sizeof(uint32_t) * ent.size();
  const size_t o_off = (n_bl + 255) & ~size_t(255);
  const size_t o_ent = (o_off + n_off + 255) & ~size_t(255);
  const size_t o_cnt = (o_ent + n_ent + 255) & ~size_t(255);
  const size_t total = o_cnt + 256;
  void* buf = nullptr;
  if (hv_context_malloc(ctx, &buf, total, st) != cudaSuccess) {
    cudaGetLastError();
    return fail(ctx, HV_ERR_OOM, "omnical: device allocation failed");
  }
  char* b8 = static_cast<char*>(buf);
  r = HV_OK;
  if ((n_bl && cudaMemcpyAsync(b8, bl.data(), n_bl, cudaMemcpyHostToDevice, st) != cudaSuccess) ||
      cudaMemcpyAsync(b8 + o_off, off.data(), n_off, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      (n_ent && cudaMemcpyAsync(b8 + o_ent, ent.data(), n_ent, cudaMemcpyHostToDevice, st) !=
                    cudaSuccess) ||
      cudaMemsetAsync(b8 + o_cnt, 0, sizeof(int), st) != cudaSuccess)
    r = HV_ERR_CUDA;
  if (r == HV_OK) {
    static bool configured[2] = {false, false};
    if (!configured[sizeof(R) == 8]) {
      constexpr bool kF = sizeof(R) == 8;
      for (const void* k : {reinterpret_cast<const void*>(omnical_kernel<R, false, false>),
                            reinterpret_cast<const void*>(omnical_kernel<R, true, false>),
                            reinterpret_cast<const void*>(omnical_kernel<R, false, kF>),
                            reinterpret_cast<const void*>(omnical_kernel<R, true, kF>)})
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kOmSmemLimit) !=
            cudaSuccess)
          r = HV_ERR_CUDA;
      if (r == HV_OK) configured[sizeof(R) == 8] = true;
    }
  }
  if (r == HV_OK) {
    using C = typename Cx<R>::T;
    OmParams<R> p;
    p.ndata = ndata;
    p.nants = nants;
    p.nubls = nubls;
    p.nbls = nbls;
    p.panel = pl.panel;
    p.npanels = pl.npanels;
    p.bl = reinterpret_cast<const uint2*>(b8);
    p.seg_off = reinterpret_cast<const int*>(b8 + o_off);
    p.seg_ord = p.seg_off + (size_t)pl.npanels * (nants + nubls + 1);
    p.seg_ent = reinterpret_cast<const uint32_t*>(b8 + o_ent);
    p.data = static_cast<const C*>(d_data);
    p.wgts = static_cast<const R*>(d_wgts);
    p.gains = static_cast<C*>(d_gains);
    p.ubls = static_cast<C*>(d_ubls);
    p.chisq = static_cast<R*>(d_chisq);
    p.conv = static_cast<R*>(d_conv);
    p.iters = d_iters;
    p.conv_crit = (R)conv_crit;
    p.gstep = (float)gain;
    p.maxiter = maxiter;
    p.check_every = check_every;
    p.check_after = check_after;
    p.group = pl.group;
    p.sum_threads = pl.sum_threads;
    p.counter = reinterpret_cast<int*>(b8 + o_cnt);
    constexpr bool kF = sizeof(R) == 8;
    if (pl.factored)
      (pl.data_shared ? omnical_kernel<R, true, kF>
                      : omnical_kernel<R, false, kF>)<<<grid, pl.threads, pl.smem, st>>>(p);
    else
      (pl.data_shared ? omnical_kernel<R, true, false>
                      : omnical_kernel<R, false, false>)<<<grid, pl.threads, pl.smem, st>>>(p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      hv_context_set_error(ctx, cudaGetErrorString(e));
      r = HV_ERR_CUDA;
    } else {
      hv_context_add_launches(ctx, 1);
    }
  }
  cudaFreeAsync(buf, st);
  return r;
}

int run_device(hv_context* ctx, int precision, const uint32_t* ggu, int nbls, void* d_gains,
               int nants, void* d_ubls, int nubls, const void* d_data, const void* d_wgts,
               int ndata, double conv_crit, int maxiter, int check_every, int check_after,
               double gain, void* d_chisq, uint32_t* d_iters, void* d_conv, cudaStream_t st) {
  if (precision == 1)
    return run_typed<float>(ctx, ggu, nbls, d_gains, nants, d_ubls, nubls, d_data, d_wgts,
                            ndata, conv_crit, maxiter, check_every, check_after, gain, d_chisq,
                            d_iters, d_conv, st);
  return run_typed<double>(ctx, ggu, nbls, d_gains, nants, d_ubls, nubls, d_data, d_wgts, ndata,
                           conv_crit, maxiter, check_every, check_after, gain, d_chisq, d_iters,
                           d_conv, st);
}

}  // namespace

extern "C" {

int hv_omnical_device(hv_context* ctx, int precision, const uint32_t* ggu, int nbls,
                      void* d_gains, int nants, void* d_ubls, int nubls, const void* d_data,
                      const void* d_wgts, int ndata, double conv_crit, int maxiter,
                      int check_every, int check_after, double gain, void* d_chisq,
                      uint32_t* d_iters, void* d_conv, void* stream) {
  if (!ctx) return HV_ERR_ARG;
  int r = check_sizes(ctx, precision, nbls, nants, nubls, ndata, maxiter, check_every);
  if (r != HV_OK) return r;
  if (ndata > 0 && (!d_gains || !d_chisq || !d_iters || !d_conv || (nbls > 0 && (!ggu || !d_data || !d_wgts)) ||
                    (nubls > 0 && !d_ubls)))
    return fail(ctx, HV_ERR_ARG, "omnical: null buffer");
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : hv_context_stream(ctx);
  return run_device(ctx, precision, ggu, nbls, d_gains, nants, d_ubls, nubls, d_data, d_wgts,
                    ndata, conv_crit, maxiter, check_every, check_after, gain, d_chisq, d_iters,
                    d_conv, st);
}

int hv_omnical(hv_context* ctx, int precision, const uint32_t* ggu, int nbls, void* gains,
               int nants, void* ubls, int nubls, const void* data, const void* wgts, int ndata,
               double conv_crit, int maxiter, int check_every, int check_after, double gain,
               void* chisq, uint32_t* iters, void* conv) {
  if (!ctx) return HV_ERR_ARG;
  int r = check_sizes(ctx, precision, nbls, nants, nubls, ndata, maxiter, check_every);
  if (r != HV_OK) return r;
  if (ndata == 0) return (nbls > 0 && !ggu) ? HV_ERR_ARG : check_indices(ctx, ggu, nbls, nants, nubls);
  if (!gains || !chisq || !iters || !conv || (nbls > 0 && (!ggu || !data || !wgts)) ||
      (nubls > 0 && !ubls))
    return fail(ctx, HV_ERR_ARG, "omnical: null buffer");
  const size_t rs = precision == 1 ? 4 : 8;
  const size_t n_g = 2 * rs * (size_t)ndata * nants, n_u = 2 * rs * (size_t)ndata * nubls;
  const size_t n_d = 2 * rs * (size_t)ndata * nbls, n_w = rs * (size_t)ndata * nbls;
  const size_t n_c = rs * (size_t)ndata, n_i = sizeof(uint32_t) * (size_t)ndata;
  size_t o[7], tot = 0;
  const size_t sz[7] = {n_g, n_u, n_d, n_w, n_c, n_c, n_i};
  for (int i = 0; i < 7; ++i) {
    o[i] = tot;
    tot += (sz[i] + 255) & ~size_t(255);
  }
  cudaStream_t st = hv_context_stream(ctx);
  void* buf = nullptr;
  if (hv_context_malloc(ctx, &buf, tot, st) != cudaSuccess) {
    cudaGetLastError();
    return fail(ctx, HV_ERR_OOM, "omnical: device allocation failed");
  }
  char* b = static_cast<char*>(buf);
  r = HV_OK;
  const void* src[4] = {gains, ubls, data, wgts};
  for (int i = 0; i < 4 && r == HV_OK; ++i)
    if (sz[i] && cudaMemcpyAsync(b + o[i], src[i], sz[i], cudaMemcpyHostToDevice, st) !=
                     cudaSuccess)
      r = HV_ERR_CUDA;
  if (r == HV_OK)
    r = run_device(ctx, precision, ggu, nbls, b + o[0], nants, b + o[1], nubls, b + o[2],
                   b + o[3], ndata, conv_crit, maxiter, check_every, check_after, gain, b + o[4],
                   reinterpret_cast<uint32_t*>(b + o[6]), b + o[5], st);
  void* dst[7] = {gains, ubls, nullptr, nullptr, chisq, conv, iters};
  for (int i : {0, 1, 4, 5, 6})
    if (r == HV_OK && sz[i] &&
        cudaMemcpyAsync(dst[i], b + o[i], sz[i], cudaMemcpyDeviceToHost, st) != cudaSuccess)
      r = HV_ERR_CUDA;
  cudaFreeAsync(buf, st);
  const cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess && r == HV_OK) {
    hv_context_set_error(ctx, cudaGetErrorString(e));
    r = HV_ERR_CUDA;
  }
  return r;
}

}  // extern "C"
