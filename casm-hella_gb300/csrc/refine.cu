// refine.cu -- differentiable candidate refinement (include/hella_refine.h).
//
// Per channel a warp accumulates
//   S0 = sum r^2,  S1 = sum r e,  S2 = sum r e u,  S3 = sum r e u^2
// (r = d - m, e = exp(-u^2/2)), every element's model value recomputed from
// theta (a Gaussian at the channel's fractional delay), from which the
// adjoint of chi2 follows:
//   d chi2/d amp   = -2 sum_c s_c S1        (s_c = (f_c/f0)^index)
//   d chi2/d index = -2 sum_c amp s_c ln(f_c/f0) S1
//   d chi2/d t0    = -2 sum_c amp s_c S2 / sigma
//   d chi2/d dm    = -2 sum_c tab_c amp s_c S2 / sigma
//   d chi2/d width = -2 sum_c amp s_c S3 / sigma * dsigma/dwidth
// The sums over channels have one fixed order: two channels a slot, eight
// slots a 16-channel group, the groups in order (deterministic results, the
// same from every kernel here).
//
// Support.  In fp32 e is exactly 0 beyond |u| = 14.5 (2^(-0.7213 u^2) is
// under half the smallest denormal), so an element outside [mu - 14.75
// sigma, mu + 14.75 sigma] has r = d and adds exactly 0 to S1, S2 and S3:
// only S0 needs it (and a non-finite d, whose r e is NaN).  k_refine (the
// forward and adjoint calls: one read of the cutouts, HBM-bound) evaluates
// the model on the support only; k_refine_fit reads, in all passes but the
// last, the support only.
#include "hella_refine.h"
#include "hg_internal.h"
#include "hg_plan.h"

#include <cmath>
#include <cstdint>
#include <new>
#include <vector>

namespace {

constexpr int kWarps = 8;
constexpr int kChPerWarp = 2;
constexpr int kChPerBlock = kWarps * kChPerWarp;  // channels of a group
constexpr int kNp = 6;     // chi2 + 5 gradient partials
constexpr unsigned kAll = 0xffffffffu;

struct RefineArgs {
  const float *cut;     // [n][nchan][nsamp]
  const float *dm_ref;  // [n]
  const float *theta;   // [n][5]
  const float *tab;     // [nchan] delay per unit DM, samples
  const float *lnf;     // [nchan] ln(f_c / f0)
  int nchan, nsamp, nblk;
  float c_w;            // sigma (samples) per ms of FWHM
  float *part;          // [2][n][nblk][kNp]
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(kAll, v, o));
  return v;
}

// The model of one channel at one theta, and its support.
struct Chan {
  float tb, lnf, s, sc, b;  // delay per DM, ln(f/f0), s_c, amp s_c, -mu / sigma
  int qa, qb;               // float4 groups [qa, qb) hold every element with e != 0
};

__device__ __forceinline__ Chan channel(const RefineArgs &a, int c, float dmr, const float *th,
                                        float sigma, float inv) {
  Chan m;
  m.tb = a.tab[c];
  m.lnf = a.lnf[c];
  const int off = (int)__fadd_rn(__fmul_rn(dmr, m.tb), 0.5f);  // the plan's integer delay
  // mu = t0 + dm*tab - off, formed without cancelling two large delays:
  // (dm - dm_ref)*tab is small, and dm_ref*tab - off is rounded once
  const float res = __fmaf_rn(dmr, m.tb, -(float)off);
  const float mu = __fadd_rn(__fmaf_rn(__fsub_rn(th[0], dmr), m.tb, th[1]), res);
  m.s = expf(__fmul_rn(th[4], m.lnf));
  m.sc = __fmul_rn(th[3], m.s);
  m.b = __fmul_rn(-mu, inv);
  // 14.75 sigma, two samples, and the rounding of mu / sigma; every element where a parameter
  // is not finite or sigma is 0 (u and e are then not those of a Gaussian)
  const int nq = a.nsamp / 4;
  const float half = 14.75f * fabsf(sigma) + 2.f + 2.4e-7f * fabsf(mu);
  const float lo = mu - half, hi = mu + half;
  if (fabsf(sigma) > 1e-18f && fabsf(sigma) < 1e18f && fabsf(mu) < 1e18f && fabsf(m.sc) < 3.0e38f) {
    m.qa = lo > 0.f ? (int)fminf(lo * 0.25f, (float)nq) : 0;
    m.qb = hi < 0.f ? 0 : min(nq, (int)fminf(hi * 0.25f, (float)nq) + 1);
  } else {
    m.qa = 0;
    m.qb = nq;
  }
  return m;
}

struct Sums {
  float s0, s1, s2, s3;
};

// One element: data d at sample t.
template <bool CHI, bool GRAD>
__device__ __forceinline__ void element(float d, float t, const Chan &m, float inv, Sums &a) {
  const float u = __fmaf_rn(t, inv, m.b);
  const float e = exp2f(__fmul_rn(-0.72134752f, __fmul_rn(u, u)));  // exp(-u^2/2)
  const float r = __fsub_rn(d, __fmul_rn(m.sc, e));
  if (CHI) a.s0 = __fmaf_rn(r, r, a.s0);
  if (GRAD) {
    const float re = __fmul_rn(r, e);
    a.s1 = __fadd_rn(a.s1, re);
    a.s2 = __fmaf_rn(re, u, a.s2);
    a.s3 = __fmaf_rn(__fmul_rn(re, u), u, a.s3);
  }
}

// Every element of one channel by one warp (lane l: float4 groups l, l + 32,
// ... in order): kLoads 16-byte loads in flight per lane; a round's groups
// outside the support add d^2 only.  Returns the warp's totals.  nan_chi: a
// non-finite element makes s0 NaN too.
template <bool GRAD, int kLoads>
__device__ __forceinline__ Sums whole_row(const float4 *__restrict__ row, int nq, int lane, const Chan &m, float inv,
                                          bool nan_chi) {
  Sums a{0.f, 0.f, 0.f, 0.f};
  float nz = 0.f;  // 0, or NaN once an element outside the support is not finite
  for (int q0 = 0; q0 < nq; q0 += 32 * kLoads) {
    float4 d4[kLoads];
#pragma unroll
    for (int l = 0; l < kLoads; ++l)
      d4[l] = q0 + 32 * l + lane < nq ? __ldcs(row + q0 + 32 * l + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int l = 0; l < kLoads; ++l) {
      const int qw = q0 + 32 * l, q = qw + lane;
      if (qw >= m.qb || qw + 32 <= m.qa) {  // the whole warp's group (lanes past nq hold zeros)
        const float dv[4] = {d4[l].x, d4[l].y, d4[l].z, d4[l].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          a.s0 = __fmaf_rn(dv[k], dv[k], a.s0);
          if (GRAD) nz = __fmaf_rn(dv[k], 0.f, nz);
        }
      } else if (q < nq) {
        const float dv[4] = {d4[l].x, d4[l].y, d4[l].z, d4[l].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) element<true, GRAD>(dv[k], __fadd_rn((float)(4 * q), (float)k), m, inv, a);
      }
    }
  }
  if (GRAD) {
    a.s1 = __fadd_rn(a.s1, nz);
    a.s2 = __fadd_rn(a.s2, nz);
    a.s3 = __fadd_rn(a.s3, nz);
    if (nan_chi) a.s0 = __fadd_rn(a.s0, nz);
  }
  a.s0 = warp_sum(a.s0);
  if (GRAD) {
    a.s1 = warp_sum(a.s1);
    a.s2 = warp_sum(a.s2);
    a.s3 = warp_sum(a.s3);
  }
  return a;
}

// A channel's totals into its slot's partials (chi2, then the gradient in
// the order of theta: dm, t0, width, amp, index).
template <bool GRAD>
__device__ __forceinline__ void add_channel(float (&acc)[kNp], const Sums &t, const Chan &m, float inv, float c_w) {
  acc[0] = __fadd_rn(acc[0], t.s0);
  if (GRAD) {
    const float gmu = __fmul_rn(__fmul_rn(-2.f, m.sc), __fmul_rn(inv, t.s2));
    acc[1] = __fmaf_rn(m.tb, gmu, acc[1]);
    acc[2] = __fadd_rn(acc[2], gmu);
    acc[3] = __fadd_rn(acc[3], __fmul_rn(__fmul_rn(-2.f, m.sc), __fmul_rn(__fmul_rn(inv, c_w), t.s3)));
    acc[4] = __fadd_rn(acc[4], __fmul_rn(__fmul_rn(-2.f, m.s), t.s1));
    acc[5] = __fadd_rn(acc[5], __fmul_rn(__fmul_rn(-2.f, __fmul_rn(m.sc, m.lnf)), t.s1));
  }
}

// Sum over the groups, in order, of partial k = threadIdx.x of one cutout
// (part [nblk][kNp]; 0 for threads without a partial).  All threads of a
// 256-thread block call it; buf holds 256 floats x kNp.
constexpr int kSumChunk = 256;
__device__ __forceinline__ float group_sum(const float *part, int nblk, float *buf) {
  float s = 0.f;
  for (int b0 = 0; b0 < nblk; b0 += kSumChunk) {
    const int nb = min(kSumChunk, nblk - b0);
    __syncthreads();
    for (int i = threadIdx.x; i < nb * kNp; i += blockDim.x) buf[i] = __ldcg(part + (size_t)b0 * kNp + i);
    __syncthreads();
    if (threadIdx.x < kNp) {
#pragma unroll 8
      for (int b = 0; b < nb; ++b) s = __fadd_rn(s, buf[b * kNp + threadIdx.x]);
    }
  }
  return s;
}

// Forward (GRAD = false: chi2) or adjoint (gtheta = gchi2 * gradient).  A
// block per (16-channel group, cutout), two channels a warp; the block that
// finishes a cutout last (counter `done`, which wraps to 0 at nblk by itself:
// calls that a caller let overlap spoil their own results only) adds the groups'
// partials.  Bound by its one read of the cutouts: the two calls on 64 cutouts x
// 1024 x 2048 (2 x 537 MB) take 173 us, 93 % of the measured 6689 GB/s; 208 us
// with every element's exponential evaluated and the groups added by a second
// kernel of one thread a cutout (6 and 18 us of them).
template <bool GRAD>
__global__ void __launch_bounds__(kWarps * 32) k_refine(RefineArgs a, unsigned *done, const float *gchi2,
                                                          float *out) {
  __shared__ float red[kWarps][kNp];
  __shared__ float buf[kSumChunk * kNp];
  __shared__ int last_s;
  const int i = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float th[HELLA_REFINE_NPAR];
#pragma unroll
  for (int k = 0; k < HELLA_REFINE_NPAR; ++k) th[k] = a.theta[(size_t)i * HELLA_REFINE_NPAR + k];
  const float sigma = __fmul_rn(th[2], a.c_w), inv = __frcp_rn(sigma), dmr = a.dm_ref[i];
  float acc[kNp] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int j = 0; j < kChPerWarp; ++j) {
    const int c = blockIdx.x * kChPerBlock + warp * kChPerWarp + j;
    const Chan m = channel(a, c, dmr, th, sigma, inv);
    const float4 *row = reinterpret_cast<const float4 *>(a.cut + ((size_t)i * a.nchan + c) * a.nsamp);
    add_channel<GRAD>(acc, whole_row<GRAD, 8>(row, a.nsamp / 4, lane, m, inv, false), m, inv, a.c_w);
  }
  if (lane == 0)
    for (int k = 0; k < kNp; ++k) red[warp][k] = acc[k];
  __syncthreads();
  float *part = a.part + (size_t)i * a.nblk * kNp;
  if (tid < kNp) {
    float v = 0.f;
    for (int w = 0; w < kWarps; ++w) v = __fadd_rn(v, red[w][tid]);
    __stcg(part + (size_t)blockIdx.x * kNp + tid, v);
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) last_s = atomicInc(done + i, a.nblk - 1) == a.nblk - 1;
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  const float s = group_sum(part, a.nblk, buf);
  if (!GRAD && tid == 0) out[i] = s;
  if (GRAD && tid >= 1 && tid < kNp) out[(size_t)i * HELLA_REFINE_NPAR + tid - 1] = __fmul_rn(gchi2[i], s);
}

// The S1..S3 of a group's 16 channels over their supports, four channels at a
// time with eight lanes each: lane l of a channel takes the float4 groups that
// are l mod 8, in order.  The totals are whole_row's: its lanes l, l + 8, l + 16
// and l + 24 are the four sets of sums x[] a lane keeps here (a lane's groups
// go through the sets in turn), added in its tree's order.  Lane j < 16 gets
// channel j's sums (mine: channel j's model in lanes j and j + 16; iters: the
// longest support in eights).  Eight lanes rather than a warp a channel: a
// support is 3 to 60 groups long, so a warp would evaluate up to 32 for 3, or
// 64 for 33 (50 steps on 64 cutouts: 973 us, a warp a channel 1052 us).
__device__ __forceinline__ Sums support_group(const float4 *__restrict__ base, int nq, int lane, const Chan &mine,
                                              float inv, int iters) {
  constexpr int W = 8, N = 32 / W;
  const int l = lane & (W - 1);
  Sums t{0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
  for (int j0 = 0; j0 < kChPerBlock; j0 += N) {
    const int j = j0 + lane / W;
    Chan m;
    m.sc = __shfl_sync(kAll, mine.sc, j);
    m.b = __shfl_sync(kAll, mine.b, j);
    const int qa = __shfl_sync(kAll, mine.qa, j), qb = __shfl_sync(kAll, mine.qb, j);
    const float4 *row = base + (size_t)j * nq;
    Sums x[4] = {};
    int q = qa + ((l - qa) & (W - 1));
    for (int it = 0; it < iters; it += 4, q += 4 * W) {
      float4 d[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        d[u] = q + u * W < qb ? __ldg(row + q + u * W) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (it + u >= iters) break;  // the same in every lane
        // past the support: d = 0 and amplitude 0 add 0
        Chan mu = m;
        mu.sc = q + u * W < qb ? m.sc : 0.f;
        const float f = (float)(4 * (q + u * W));
        element<false, true>(d[u].x, f, mu, inv, x[u]);
        element<false, true>(d[u].y, __fadd_rn(f, 1.f), mu, inv, x[u]);
        element<false, true>(d[u].z, __fadd_rn(f, 2.f), mu, inv, x[u]);
        element<false, true>(d[u].w, __fadd_rn(f, 3.f), mu, inv, x[u]);
      }
    }
    const float a1 = __fadd_rn(__fadd_rn(x[0].s1, x[2].s1), __fadd_rn(x[1].s1, x[3].s1));
    const float a2 = __fadd_rn(__fadd_rn(x[0].s2, x[2].s2), __fadd_rn(x[1].s2, x[3].s2));
    const float a3 = __fadd_rn(__fadd_rn(x[0].s3, x[2].s3), __fadd_rn(x[1].s3, x[3].s3));
    // the tree over lane offsets 4, 2, 1, three sums at once: the upper half of the lanes takes
    // over S2 at the first offset, the second and fourth quarters S3 at the next
    const bool hi = l & 4, sec = l & 2;
    float v = __fadd_rn(hi ? a2 : a1, __shfl_xor_sync(kAll, hi ? a1 : a2, 4));
    const float s3 = __fadd_rn(a3, __shfl_xor_sync(kAll, a3, 4));
    v = __fadd_rn(sec ? s3 : v, __shfl_xor_sync(kAll, sec ? v : s3, 2));
    v = __fadd_rn(v, __shfl_xor_sync(kAll, v, 1));
    const int src = (lane & (N - 1)) * W;  // lanes j0 .. j0 + N - 1 take channel lane - j0's
    const float s1 = __shfl_sync(kAll, v, src), w3 = __shfl_sync(kAll, v, src + 2), s2 = __shfl_sync(kAll, v, src + 4);
    if (lane / N == j0 / N) {
      t.s1 = s1;
      t.s2 = s2;
      t.s3 = w3;
    }
  }
  return t;
}

struct Rates {
  float lr[HELLA_REFINE_NPAR];
};

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// All steps of one cutout's fit by one cluster of blocks, a warp per
// 16-channel group: every step but the last reads only the bursts' supports
// (about 30 sigma of each channel: a few percent of a cutout, which stays in
// L2 from step to step), the last one everything, for chi2 and for elements
// that are not finite.  Each block keeps theta and the Adam moments (thread
// 1 + k: parameter k) and adds the groups' partials itself, so that a step
// costs one cluster barrier; the partials alternate between two buffers,
// which a block reaches again only after the barrier of the step between.
// 50 steps on 64 cutouts x 1024 x 2048: 973 us (0.88-1.05 ms with the widths
// drawn), against 6050 us for a read of every element a step and two launches.
// Of those, 80 us are the last step's read (115 us on 64 cutouts).  The other
// steps are bound by the latency of their loads from L2 (a step of all cutouts:
// 5.0 us for one, 7.4 for 16, 8.9 for 32, 11.0 for 50) as long as all clusters
// are resident, which eight blocks a cutout are up to about 52 cutouts; past
// that the last ones run after the first ones' steps (14 to 17 us for 54 to 64,
// 26 for 128).  Three blocks an SM (80 registers): with four (64, some spilled)
// a step of one cutout, where residency does not matter, takes 9.7 us instead
// of 7.
constexpr int kFitCluster = 8;
__global__ void __launch_bounds__(kWarps * 32, 3) k_refine_fit(RefineArgs a, int n, int csize, int steps, Rates ad,
                                                             float *theta, float *chi2) {
  __shared__ float buf[kSumChunk * kNp];
  __shared__ float th_s[HELLA_REFINE_NPAR];
  __shared__ float red[kWarps][kWarps][kNp];
  const int i = blockIdx.x / csize, rank = blockIdx.x % csize;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, par = tid - 1, nq = a.nsamp / 4;
  if (tid < HELLA_REFINE_NPAR) th_s[tid] = theta[(size_t)i * HELLA_REFINE_NPAR + tid];
  __syncthreads();
  float mom = 0.f, var = 0.f, chi = 0.f;
  double b1 = 1.0, b2 = 1.0;  // beta^t
  const float dmr = a.dm_ref[i];
  for (int t = 0; t < steps; ++t) {
    const bool whole = t + 1 == steps;
    const float sigma = __fmul_rn(th_s[2], a.c_w), inv = __frcp_rn(sigma);
    float *part = a.part + ((size_t)(t & 1) * n + i) * a.nblk * kNp;
    for (int g = rank * kWarps + warp; g < a.nblk; g += csize * kWarps) {
      const int c = g * kChPerBlock + (lane & (kChPerBlock - 1));
      const Chan mine = channel(a, c, dmr, th_s, sigma, inv);
      const float4 *base = reinterpret_cast<const float4 *>(a.cut + ((size_t)i * a.nchan + (size_t)g * kChPerBlock) * a.nsamp);
      Sums sum{0.f, 0.f, 0.f, 0.f};
      if (whole) {
        for (int j = 0; j < kChPerBlock; ++j) {
          Chan m;
          m.sc = __shfl_sync(kAll, mine.sc, j);
          m.b = __shfl_sync(kAll, mine.b, j);
          m.qa = __shfl_sync(kAll, mine.qa, j);
          m.qb = __shfl_sync(kAll, mine.qb, j);
          const Sums r = whole_row<true, 8>(base + (size_t)j * nq, nq, lane, m, inv, t > 0);
          if (lane == j) sum = r;
        }
      } else {
        const int len = (int)__reduce_max_sync(kAll, (unsigned)max(0, mine.qb - mine.qa));
        sum = support_group(base, nq, lane, mine, inv, (len + 7) / 8);
      }
      // slot w of the group: channels 2w, then 2w + 1, whose sums and model move to lane 2w
      float acc[kNp] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      add_channel<true>(acc, sum, mine, inv, a.c_w);
      const Sums sum1{__shfl_down_sync(kAll, sum.s0, 1), __shfl_down_sync(kAll, sum.s1, 1),
                      __shfl_down_sync(kAll, sum.s2, 1), __shfl_down_sync(kAll, sum.s3, 1)};
      Chan m1 = mine;
      m1.tb = __shfl_down_sync(kAll, mine.tb, 1);
      m1.lnf = __shfl_down_sync(kAll, mine.lnf, 1);
      m1.s = __shfl_down_sync(kAll, mine.s, 1);
      m1.sc = __shfl_down_sync(kAll, mine.sc, 1);
      add_channel<true>(acc, sum1, m1, inv, a.c_w);
      if (lane < kChPerBlock && !(lane & 1))
#pragma unroll
        for (int k = 0; k < kNp; ++k) red[warp][lane >> 1][k] = acc[k];
      __syncwarp();
      if (lane < kNp) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) v = __fadd_rn(v, red[warp][w][lane]);
        __stcg(part + (size_t)g * kNp + lane, v);
      }
      __syncwarp();
    }
    cluster_sync();
    const float s = group_sum(part, a.nblk, buf);
    if (tid == 0) chi = s;
    if (par >= 0 && par < HELLA_REFINE_NPAR) {
      b1 *= 0.9;
      b2 *= 0.999;
      const float bc1 = (float)(1.0 - b1), bc2 = (float)(1.0 - b2);
      mom = __fmaf_rn(0.9f, mom, __fmul_rn(0.1f, s));
      var = __fmaf_rn(0.999f, var, __fmul_rn(0.001f, __fmul_rn(s, s)));
      const float step = __fdiv_rn(__fmul_rn(ad.lr[par], __fdiv_rn(mom, bc1)),
                                   __fadd_rn(__fsqrt_rn(__fdiv_rn(var, bc2)), 1e-8f));
      float v = __fsub_rn(th_s[par], step);
      if (par == 0) v = fmaxf(v, 0.f);    // dm
      if (par == 2) v = fmaxf(v, 0.05f);  // width, ms
      th_s[par] = v;
    }
    __syncthreads();
  }
  if (rank == 0) {
    if (tid < HELLA_REFINE_NPAR) theta[(size_t)i * HELLA_REFINE_NPAR + tid] = th_s[tid];
    if (tid == 0 && chi2) chi2[i] = chi;
  }
}

}  // namespace

struct hella_refine {
  hella_refine_params p{};
  cudaStream_t stream = nullptr;
  int nblk = 0;
  std::vector<float> tab;
  float *d_tab = nullptr, *d_part = nullptr;
  float *d_lnf = nullptr;  // in d_tab's allocation, as
  unsigned *d_done = nullptr;  // [ncut] groups of a cutout done; 0 between calls
  float c_w = 0.f;
};

namespace {

hella_status check_ptrs(const hella_refine *r, int n, const float *cut, const float *dm_ref, const float *theta) {
  if (!r || !cut || !dm_ref || !theta || n < 1 || n > r->p.ncut) return HELLA_ERR_INVALID_ARG;
  if (reinterpret_cast<uintptr_t>(cut) % 16) return HELLA_ERR_INVALID_ARG;  // float4 rows
  return HELLA_OK;
}

RefineArgs args(hella_refine *r, const float *cut, const float *dm_ref, const float *theta) {
  RefineArgs a{};
  a.cut = cut;
  a.dm_ref = dm_ref;
  a.theta = theta;
  a.tab = r->d_tab;
  a.lnf = r->d_lnf;
  a.nchan = r->p.nchan;
  a.nsamp = r->p.nsamp;
  a.nblk = r->nblk;
  a.c_w = r->c_w;
  a.part = r->d_part;
  return a;
}

}  // namespace

extern "C" {

void hella_refine_destroy(hella_refine *r) {
  if (!r) return;
  cudaSetDevice(r->p.device);
  cudaStreamSynchronize(r->stream);
  cudaFree(r->d_tab);
  cudaFree(r->d_part);
  delete r;
}

hella_status hella_refine_create(hella_refine **out, const hella_refine_params *p) {
  if (!out || !p) return HELLA_ERR_INVALID_ARG;
  *out = nullptr;
  if (p->ncut < 1 || p->nchan < 16 || p->nchan % kChPerBlock || p->nsamp < 128 || p->nsamp % 128 ||
      !(p->tsamp > 0) || !(p->f0_mhz > 0) || !(p->df_mhz != 0) ||
      p->f0_mhz - p->nchan * std::fabs(p->df_mhz) <= 0)
    return HELLA_ERR_INVALID_ARG;
  if (cudaSetDevice(p->device) != cudaSuccess) {
    cudaGetLastError();
    return HELLA_ERR_CUDA;
  }
  hella_refine *r = new (std::nothrow) hella_refine;
  if (!r) return HELLA_ERR_ALLOC;
  r->p = *p;
  r->nblk = p->nchan / kChPerBlock;
  r->c_w = (float)(1.0 / (2.0 * std::sqrt(2.0 * std::log(2.0)) * p->tsamp * 1e3));
  r->tab = hg::delay_table(p->nchan, p->tsamp, p->f0_mhz, p->df_mhz);
  // one buffer and one copy: tab | lnf | done (zeros)
  std::vector<float> up((size_t)2 * p->nchan + p->ncut, 0.f);
  for (int c = 0; c < p->nchan; ++c) {
    up[c] = r->tab[c];
    up[p->nchan + c] = (float)std::log((p->f0_mhz - c * std::fabs(p->df_mhz)) / p->f0_mhz);
  }
  if (cudaMalloc(&r->d_tab, up.size() * 4) != cudaSuccess ||
      cudaMalloc(&r->d_part, (size_t)2 * p->ncut * r->nblk * kNp * 4) != cudaSuccess) {
    cudaGetLastError();
    hella_refine_destroy(r);
    return HELLA_ERR_ALLOC;
  }
  r->d_lnf = r->d_tab + p->nchan;
  r->d_done = reinterpret_cast<unsigned *>(r->d_lnf + p->nchan);
  if (cudaMemcpy(r->d_tab, up.data(), up.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess) {
    cudaGetLastError();
    hella_refine_destroy(r);
    return HELLA_ERR_CUDA;
  }
  *out = r;
  return HELLA_OK;
}

hella_status hella_refine_set_stream(hella_refine *r, void *stream) {
  if (!r) return HELLA_ERR_INVALID_ARG;
  r->stream = (cudaStream_t)stream;
  return HELLA_OK;
}

hella_status hella_refine_delay_table(const hella_refine *r, float *tab) {
  if (!r || !tab) return HELLA_ERR_INVALID_ARG;
  for (int c = 0; c < r->p.nchan; ++c) tab[c] = r->tab[c];
  return HELLA_OK;
}

hella_status hella_refine_forward(hella_refine *r, int n, const float *cut, const float *dm_ref,
                                  const float *theta, float *chi2) {
  hella_status s = check_ptrs(r, n, cut, dm_ref, theta);
  if (s != HELLA_OK || !chi2) return s != HELLA_OK ? s : HELLA_ERR_INVALID_ARG;
  if (cudaSetDevice(r->p.device) != cudaSuccess) return HELLA_ERR_CUDA;
  k_refine<false><<<dim3(r->nblk, n), kWarps * 32, 0, r->stream>>>(args(r, cut, dm_ref, theta), r->d_done, nullptr,
                                                                  chi2);
  hg::count_launches(1);
  return cudaGetLastError() == cudaSuccess ? HELLA_OK : HELLA_ERR_CUDA;
}

hella_status hella_refine_adjoint(hella_refine *r, int n, const float *cut, const float *dm_ref,
                                  const float *theta, const float *gchi2, float *gtheta) {
  hella_status s = check_ptrs(r, n, cut, dm_ref, theta);
  if (s != HELLA_OK || !gchi2 || !gtheta) return s != HELLA_OK ? s : HELLA_ERR_INVALID_ARG;
  if (cudaSetDevice(r->p.device) != cudaSuccess) return HELLA_ERR_CUDA;
  k_refine<true><<<dim3(r->nblk, n), kWarps * 32, 0, r->stream>>>(args(r, cut, dm_ref, theta), r->d_done, gchi2,
                                                                 gtheta);
  hg::count_launches(1);
  return cudaGetLastError() == cudaSuccess ? HELLA_OK : HELLA_ERR_CUDA;
}

hella_status hella_refine_fit(hella_refine *r, int n, const float *cut, const float *dm_ref, float *theta,
                              int steps, const float *lr, float *chi2) {
  hella_status s = check_ptrs(r, n, cut, dm_ref, theta);
  if (s != HELLA_OK || !lr || steps < 0) return s != HELLA_OK ? s : HELLA_ERR_INVALID_ARG;
  if (cudaSetDevice(r->p.device) != cudaSuccess) return HELLA_ERR_CUDA;
  if (steps == 0) return HELLA_OK;
  Rates rt;
  for (int k = 0; k < HELLA_REFINE_NPAR; ++k) rt.lr[k] = lr[k];
  int csize = 1;  // blocks per cutout: a group a warp, up to the portable cluster size
  while (csize < kFitCluster && csize * kWarps < r->nblk) csize *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)n * csize);
  cfg.blockDim = dim3(kWarps * 32);
  cfg.stream = r->stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = csize;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_refine_fit, args(r, cut, dm_ref, theta), n, csize, steps, rt, theta,
                                           chi2);
  hg::count_launches(1);
  if (e != cudaSuccess) cudaGetLastError();
  return e == cudaSuccess ? HELLA_OK : HELLA_ERR_CUDA;
}

}  // extern "C"
