// flagger.cu -- casm-hella's spectral RFI flagger and normaliser on GB300.
//
// Reference: src/hella/src/flagger.cu:345-411 (fast_flagger) with the
// default configuration (no SCRUNCH lines): bandpass_flag (:216-242), then
// apply_scrunch(8, 8, 100, flag=0, ts=1) (:385-401), then transpose_output
// (transpose.cu:48-76).
//
// Design.  The reference materialises an fp16 copy of the gulp and rewrites
// it ~14 times.  Here the fp16 plane is never stored: up to the time-series
// correction every value depends only on its channel and its u8 input level,
// so each stage publishes a 256-entry lookup table per channel and every
// reduction pass re-reads the u8 gulp (1 byte per sample) and maps it
// through the table.  The per-time division and the final normalisation are
// applied on the fly.  Each reduction reproduces the reference's order:
//   calc_bandpass_new  (flagger.cu:86-112)   32 lane partials in time order,
//                                            warp shuffle tree, / width
//   computeRowMeans    (normalization.cu:19-69) 256 strided partials, warp
//   computeRowVariances(normalization.cu:72-122) trees, 8-warp sum, / width
//   calculate_stddev host loops (normalization.cu:138-153) sequential over
//                                            channels, done by one thread
//   measure_ts         (timeseries.cu:19-36)  fp16 running sum over channels
// so the output bytes equal the reference's on the same gulp.
#include "hg_internal.h"
#include "hella_search.h"
#include "hg_ptx.h"

#include <algorithm>
#include <cmath>

namespace hg {
namespace {


__device__ __forceinline__ __half hzero() { return __float2half_rn(0.f); }
__device__ __forceinline__ __half hone() { return __float2half_rn(1.f); }

// Value of u8 level v of a channel after flagger stage `stage`:
//  1 bandpass_correct   divide_by_bp (flagger.cu:180-194)
//  2 normalize_data     (x + half(-mean)) * half(1/std) (flagger.cu:198-214)
//  3 spectral flag      1, or x + 1 (replace_data_and_add_bandpass :146-158)
//  4 bandpass_correct   of the final scrunch
struct ChanState {
  float bp1, bp3;
  bool flag2;
  __half add, mul;
};
__device__ __half chain_value(int stage, int v, const ChanState &ch) {
  __half x = __float2half_rn((float)v);
  if (stage >= 1) x = ch.bp1 > 0.f ? __hdiv(x, __float2half_rn(ch.bp1)) : hzero();
  if (stage >= 2) x = __hmul(__hadd(x, ch.add), ch.mul);
  if (stage >= 3) x = ch.flag2 ? hone() : __hadd(x, hone());
  if (stage >= 4) x = ch.bp3 > 0.f ? __hdiv(x, __float2half_rn(ch.bp3)) : hzero();
  return x;
}

// The tables lie in slices of kLutSl channels, [level][channel]: a level's row
// is whole words of channel pairs, and blocks stage rows or parts of them as
// they are.  The last slice of a beam may be part empty.
__device__ __forceinline__ __half *lut_row(__half *lut, int nchan, int b, int c, int level) {
  return lut + (((size_t)b * ((nchan + kLutSl - 1) / kLutSl) + c / kLutSl) * 256 + level) * kLutSl + c % kLutSl;
}

// Warp tree over the 32 lane partials of a channel, / w (flagger.cu:103-111);
// lane 0 has the result.
__device__ __forceinline__ float lane_total(const float *part, int gulp) {
  float v = part[threadIdx.x & 31];
  for (int off = 16; off > 0; off /= 2) v = __fadd_rn(v, __shfl_down_sync(0xffffffffu, v, off));
  return __fdiv_rn(v, (float)gulp);
}
// Where that total goes.  mode 0: bp1, 1: bp2 + spectral flag, 2: bp3, 3: bpx.
__device__ __forceinline__ void put_bandpass(const FlagState &st, int mode, int bc, float bp) {
  if (mode == 0) st.bp1[bc] = bp;
  if (mode == 1) {
    st.bp2[bc] = bp;
    st.flag2[bc] = (bp < st.spec_min || bp > st.spec_max) ? 1 : 0;
  }
  if (mode == 2) st.bp3[bc] = bp;
  if (mode == 3) st.bpx[bc] = bp;
}

// The tables of `stage`.  With fin >= 0 the lane partials of the pass before are
// first brought to that mode's bandpass (a pass of its own would cost a launch,
// 3 us, for 128 bytes a channel): every block does so for its own 32 channels, the
// first of a column of blocks for all readers to come, and the values of its own
// blocks come from shared memory.
constexpr int kLutC = 32;  // channels a block
__global__ void __launch_bounds__(256) k_build_lut(FlagState st, int stage, int fin, int rows) {
  __shared__ float bp_s[kLutC];
  const int cl = threadIdx.x % kLutC, c0 = blockIdx.x * kLutC, b = blockIdx.z, wi = threadIdx.x / 32;
  const int bc0 = b * st.nchan + c0;
  if (fin >= 0) {
#pragma unroll
    for (int i = wi; i < kLutC; i += 8) {
      const float bp = lane_total(st.part + (size_t)(bc0 + i) * 32, st.gulp);
      if (cl == 0) {
        bp_s[i] = bp;
        if (blockIdx.y == 0) put_bandpass(st, fin, bc0 + i, bp);
      }
    }
    __syncthreads();
  }
  const int bc = bc0 + cl;
  ChanState ch{};
  if (stage >= 1) ch.bp1 = fin == 0 ? bp_s[cl] : st.bp1[bc];
  if (stage >= 3) {
    ch.flag2 = fin == 1 ? bp_s[cl] < st.spec_min || bp_s[cl] > st.spec_max : st.flag2[bc] != 0;
  }
  if (stage >= 4) ch.bp3 = fin == 2 ? bp_s[cl] : st.bp3[bc];
  if (stage >= 2) {
    ch.add = st.hsc[b * 8 + 0];
    ch.mul = st.hsc[b * 8 + 1];
  }
  __half *row = lut_row(st.lut, st.nchan, b, c0 + cl, 0);
#pragma unroll 4
  for (int v = wi; v < rows; v += 8) row[(blockIdx.y * rows + v) * kLutSl] = chain_value(stage, blockIdx.y * rows + v, ch);
}
// 8 levels a block, 32 where that still leaves two blocks an SM (1024 channels x 8 beams:
// 9.2 us, 17.9 us with 8).
void launch_lut(const FlagState &st, int stage, int fin, cudaStream_t s) {
  const int rows = st.nchan / kLutC * st.nbeam * 8 >= 2 * 152 ? 32 : 8;
  k_build_lut<<<dim3(st.nchan / kLutC, 256 / rows, st.nbeam), 256, 0, s>>>(st, stage, fin, rows);
}

// a / b for half-precision a, b with r = 1 / b rounded: one correction step
// after a first product (P. Markstein, IBM J. Res. Dev. 34, 1990) gives the
// float quotient, whose rounding to half is the half quotient (24 bits are twice
// 11 and two more).  Not for zero, infinite or NaN b, nor for such a quotient: the
// correction then makes NaN or infinity of them, which callers look for and
// leave to __hdiv.  (A zero of the other sign may come out for -0 / b.)
__device__ __forceinline__ float div_step(float a, float b, float r) {
  const float q = __fmul_rn(a, r);
  return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
}

// The sums over time.  MOD = 32, calc_bandpass_new: lane l of channel c sums
// samples l, l + 32, ... (below 32 floor(w / 32)) in time order.  MOD = 256,
// computeRowMeans / computeRowVariances: column j sums samples j, j + 256, ...
// below 256 floor(w / 256).  RAW: the levels themselves; else their table values.
// TS: values divided by half(ts[t]) (divide_by_ts, timeseries.cu:38-55).  VAR:
// (x - mean)^2 with the fused multiply-add the reference's compiler emits.
//
// A warp takes 32 CH channels of one sum after another (`per` of them), a lane CH
// neighbouring ones: one load a row feeds CH sums.  The block's table slice is in
// shared memory as it lies in global memory, [level][pair]; with CH = 4 the upper
// 16 lanes take their channel pairs in the other order, so that a lookup of a
// warp never hits a bank twice, and one byte permute makes the address from level
// and lane.  Each warp's rows (and their divisors) arrive by asynchronous copies,
// ROWS a stage, AHEAD stages on their way, without block-wide waits.  Raw levels
// are added two to a word, a stage at a time: whole numbers below 2^24, the same
// in any order (kRawMax).  Bound by instruction issue and the lookups (shared
// memory): 8 beams x 32,768 samples x 1024 channels 65 us (94 us with a
// half-precision lookup on two banks and eight rows in flight a thread), divided
// by ts 104 us (146 us), lane sums 58 us (117 us), of levels 41 us.
constexpr int kSumWarps = 8;
constexpr int kLutBytes = kLutSl * 256 * (int)sizeof(__half);
constexpr int kRawMax = (1 << 24) / 255;  // levels that a float adds up exactly
constexpr int sum_stage(int rows, int ch, bool ts) { return rows * (32 * ch + (ts ? 8 : 0)); }  // bytes
template <int N>
__device__ __forceinline__ void copy_async(void *d, const void *src) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(d);
  if (N == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(src) : "memory");
}
template <int MOD, bool VAR, bool TS, bool RAW, int CH, int ROWS, int AHEAD>
__global__ void __launch_bounds__(32 * kSumWarps, 2) k_sums(const uint8_t *__restrict__ gulp, FlagState st, int which,
                                                            int per) {
  extern __shared__ __align__(16) uint8_t sum_s[];
  constexpr int kRowB = 32 * CH, kPieces = kRowB / 16, kStep = 32 / kPieces;  // bytes and 16-byte pieces of a row; rows a copy
  constexpr int kDepth = AHEAD + 1, kStage = ROWS * (kRowB + (TS ? 8 : 0));
  const int b = blockIdx.z, c0 = blockIdx.x * kLutSl, nchan = st.nchan, w = st.gulp;
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  constexpr int kParts = 4 / CH;  // warps side by side on the slice
  const int part = wi % kParts, cw = c0 + part * kRowB, nw = (blockDim.x >> 5) / kParts;
  if (!RAW) {
    const uint8_t *src = reinterpret_cast<const uint8_t *>(lut_row(st.lut, nchan, b, c0, 0));
#pragma unroll 4
    for (int i = threadIdx.x * 16; i < kLutBytes; i += blockDim.x * 16) copy_async<16>(sum_s + i, src + i);
  }
  uint8_t *ring = sum_s + (RAW ? 0 : kLutBytes) + wi * kDepth * kStage;
  const int nk = w / MOD, nst = (nk + ROWS - 1) / ROWS;
  const int j0 = blockIdx.y * per * nw + wi / kParts, total = per * nst;
  // the copies: this lane's place in a stage, the row it reads next and its sum
  const int pr = lane / kPieces, pk = lane % kPieces;
  const size_t step = (size_t)MOD * nchan;
  const bool piece = cw + 16 * pk < nchan;
  const uint8_t *const first_row = gulp + (size_t)b * w * nchan + cw + 16 * pk + pr * step;
  const uint8_t *src = first_row + (size_t)j0 * nchan;
  const float2 *tsrc = TS ? st.tdiv + (size_t)b * w + j0 + lane * MOD : nullptr;
  int lj = j0, lk = 0, lslot = 0, left = total;
  auto load = [&]() {
    if (left > 0) {
      uint8_t *d = ring + lslot + pr * kRowB + 16 * pk;
#pragma unroll
      for (int u = 0; u < ROWS; u += kStep)
        if (piece && lk + u + pr < nk) copy_async<16>(d + u * kRowB, src + u * step);
      if (TS && lane < ROWS && lk + lane < nk) copy_async<8>(ring + lslot + ROWS * kRowB + lane * 8, tsrc);
      --left;
      lslot = lslot == AHEAD * kStage ? 0 : lslot + kStage;
      lk += ROWS;
      src += ROWS * step;
      if (TS) tsrc += ROWS * MOD;
      if (lk >= nk) {
        lk = 0;
        lj += nw;
        src = first_row + (size_t)lj * nchan;
        if (TS) tsrc = st.tdiv + (size_t)b * w + lj + lane * MOD;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const float mean = VAR ? st.scal[b * 8 + 2 * which] : 0.f;
#pragma unroll 1
  for (int i = 0; i < AHEAD; ++i) load();
  const bool hi = CH == 4 && lane >= 16;
  // addresses of channels 0, 1 and (CH = 4) 2, 3 as taken, without the level
  const uint32_t first = 128u * part + 2u * CH * lane + (hi ? 4u : 0u);
  const uint32_t second = 8u * lane + (hi ? 0u : 4u);
  const bool exact = RAW && nk <= kRawMax;
  float acc[CH];
  uint32_t total_s[CH];
#pragma unroll
  for (int q = 0; q < CH; ++q) acc[q] = 0.f, total_s[q] = 0u;
  if (!RAW) {  // the whole table, from all threads
    asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD - 1) : "memory");
    __syncthreads();
  }
  // one row; `fast`: quotients by div_step, else by __hdiv
  auto row = [&](const uint8_t *d, int r, bool fast) {
    uint32_t x;
    if (CH == 4) {
      x = *reinterpret_cast<const uint32_t *>(d + r * kRowB + 4 * lane);
      x = __byte_perm(x, x, hi ? 0x1032 : 0x3210);
    } else {
      x = *reinterpret_cast<const uint16_t *>(d + r * kRowB + 2 * lane);
    }
    float f[CH];
    if (RAW) {
#pragma unroll
      for (int q = 0; q < CH; ++q)
        f[q] = __fsub_rn(__uint_as_float(__byte_perm(x, 0x4b000000u, 0x7440 + q)), 8388608.f);  // 2^23 + level - 2^23
    } else {
      __half h[CH];
#pragma unroll
      for (int q = 0; q < CH; ++q)
        h[q] = *reinterpret_cast<const __half *>(sum_s + __byte_perm(x, q < 2 ? first : second, 0x7704 + 16 * q) +
                                                 2 * (q & 1));
#pragma unroll
      for (int q = 0; q < CH; ++q) f[q] = __half2float(h[q]);
      if (TS) {
        const float2 t = *reinterpret_cast<const float2 *>(d + ROWS * kRowB + r * 8);
        if (fast) {
#pragma unroll
          for (int q = 0; q < CH; q += 2) {
            const __half2 p = __floats2half2_rn(div_step(f[q], t.x, t.y), div_step(f[q + 1], t.x, t.y));
            f[q] = __low2float(p);
            f[q + 1] = __high2float(p);
          }
        } else {
          const __half th = __float2half_rn(t.x);
#pragma unroll
          for (int q = 0; q < CH; ++q) f[q] = __half2float(__hdiv(h[q], th));
        }
      }
    }
#pragma unroll
    for (int q = 0; q < CH; ++q) {
      if (VAR) {
        const float e = __fsub_rn(f[q], mean);
        acc[q] = __fmaf_rn(e, e, acc[q]);
      } else {
        acc[q] = __fadd_rn(acc[q], f[q]);
      }
    }
  };
  int slot = 0, k0 = 0, j = j0;
#pragma unroll 1
  for (int i = 0; i < total; ++i) {
    load();  // its slot was read in the iteration before, behind __syncwarp
    asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD) : "memory");
    __syncwarp();
    const uint8_t *d = ring + slot;
    slot = slot == AHEAD * kStage ? 0 : slot + kStage;
    const int n = min(ROWS, nk - k0);
    if (RAW && exact) {
      uint32_t even = 0u, odd = 0u;  // sums of bytes 0, 2 and 1, 3: at most 255 ROWS each
      static_assert(ROWS <= 256, "16 bits a sum");
#pragma unroll 8
      for (int r = 0; r < n; ++r) {
        const uint32_t x = *reinterpret_cast<const uint32_t *>(d + r * kRowB + 4 * lane);
        even += x & 0x00ff00ffu;
        odd += (x >> 8) & 0x00ff00ffu;
      }
      total_s[0] += even & 0xffffu;
      total_s[1] += odd & 0xffffu;
      total_s[CH - 2] += even >> 16;
      total_s[CH - 1] += odd >> 16;
    } else {
      float before[CH];
#pragma unroll
      for (int q = 0; q < CH; ++q) before[q] = acc[q];
      if (n == ROWS) {
#pragma unroll 8
        for (int r = 0; r < ROWS; ++r) row(d, r, true);
      } else {
#pragma unroll 1
        for (int r = 0; r < n; ++r) row(d, r, true);
      }
      if (TS) {  // a quotient that div_step does not give leaves its sum infinite or NaN
        bool finite = true;
#pragma unroll
        for (int q = 0; q < CH; ++q) finite = finite && fabsf(acc[q]) <= 3.0e38f;
        if (!finite) {
#pragma unroll
          for (int q = 0; q < CH; ++q) acc[q] = before[q];
#pragma unroll 1
          for (int r = 0; r < n; ++r) row(d, r, false);
        }
      }
    }
    k0 += ROWS;
    if (k0 >= nk) {
      const int c = cw + CH * lane;
      float *pp = st.part + ((size_t)b * nchan + c) * MOD + j;
      if (c < nchan)
#pragma unroll
        for (int q = 0; q < CH; ++q)
          if (RAW && exact)
            pp[q * MOD] = (float)total_s[q];
          else
            pp[(hi ? q ^ 2 : q) * MOD] = acc[q];
#pragma unroll
      for (int q = 0; q < CH; ++q) acc[q] = 0.f, total_s[q] = 0u;
      k0 = 0;
      j += nw;
    }
    __syncwarp();
  }
}

// lane_total by itself, one warp per (beam, channel).
__global__ void k_lane_finish(FlagState st, int mode) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (gw >= st.nbeam * st.nchan) return;
  const float bp = lane_total(st.part + (size_t)gw * 32, st.gulp);
  if ((threadIdx.x & 31) == 0) put_bandpass(st, mode, gw, bp);
}

// Thread 0 of the reference's 256-thread block: each warp's shuffle tree,
// then warp totals 1..7 added in order, / nw.  One warp per channel, a block's
// channels of one beam (nchan % 32 == 0).  The last block of a beam then runs
// calculate_stddev's host loop (normalization.cu:138-153): sequential sum over
// channels, / nchan; the variance pass also forms the half-precision
// normalisation constants of normalize_data (flagger.cu:205-206).  (A launch of
// its own for that cost 3 to 9 us.)
constexpr int kBeamT = 256, kMaxChan = 8192;  // the largest nchan accepted
template <bool VAR>
__global__ void __launch_bounds__(kBeamT) k_row_finish(FlagState st, int which) {
  const int c = blockIdx.x * (kBeamT / 32) + (threadIdx.x >> 5), b = blockIdx.y, lane = threadIdx.x & 31;
  const float *p = st.part + ((size_t)b * st.nchan + c) * 256;
  float v[8];
#pragma unroll
  for (int wi = 0; wi < 8; ++wi) v[wi] = p[wi * 32 + lane];
#pragma unroll
  for (int wi = 0; wi < 8; ++wi)
    for (int off = 16; off > 0; off /= 2) v[wi] = __fadd_rn(v[wi], __shfl_down_sync(0xffffffffu, v[wi], off));
  float tot = v[0];
#pragma unroll
  for (int wi = 1; wi < 8; ++wi) tot = __fadd_rn(tot, v[wi]);
  float *rv = st.rowval + (size_t)b * st.nchan;
  if (lane == 0) rv[c] = __fdiv_rn(tot, (float)(256 * (st.gulp / 256)));
  if (!last_block(st.done + b, gridDim.x)) return;
  float s = block_seq_sum(rv, st.nchan);
  if (threadIdx.x != 0) return;
  s = __fdiv_rn(s, (float)st.nchan);
  if (!VAR) {
    st.scal[b * 8 + 2 * which] = s;
  } else {
    const float sd = __fsqrt_rn(s), mean = st.scal[b * 8 + 2 * which];
    st.scal[b * 8 + 2 * which + 1] = sd;
    st.hsc[b * 8 + 2 * which] = __float2half_rn(-mean);
    st.hsc[b * 8 + 2 * which + 1] = __float2half_rn(__fdiv_rn(1.f, sd));
  }
}

// med_filter_bandpass (median_filter.cpp:85-107, median_filter :36-77) with
// a window of win (odd) channels: channel i in [h, nchan - h) takes the
// middle element of its sorted window (h = win / 2), the first h channels
// take channel h's value and the last h channel nchan - h - 1's.  Any sort
// leaves the same middle element, so the values are the reference's.  One
// block per beam, in place: the row is staged in shared memory first.
__global__ void __launch_bounds__(kBeamT) k_bp_median(float *__restrict__ bp, int nchan, int win) {
  __shared__ float row[kMaxChan];
  float *r = bp + (size_t)blockIdx.x * nchan;
  for (int c = threadIdx.x; c < nchan; c += blockDim.x) row[c] = r[c];
  __syncthreads();
  const int h = win / 2;
  for (int c = threadIdx.x; c < nchan; c += blockDim.x) {
    const int i = min(max(c, h), nchan - h - 1);
    float w[kMaxBpMedian];
    for (int k = 0; k < win; ++k) {  // insertion sort of the window
      const float v = row[i - h + k];
      int j = k - 1;
      while (j >= 0 && w[j] > v) {
        w[j + 1] = w[j];
        --j;
      }
      w[j + 1] = v;
    }
    r[c] = w[h];
  }
}

// k_lane_finish for mode, then the bandpass median filter where the
// reference's bandpass_correct applies it (modes 0, 2 and 3: every bandpass
// that data are divided by; not the spectral-flag bandpass of mode 1).
unsigned lane_finish(const FlagState &st, int mode, int fin_blocks, cudaStream_t s) {
  k_lane_finish<<<fin_blocks, 256, 0, s>>>(st, mode);
  if (mode == 1 || st.bp_median <= 1) return 1;
  float *bp = mode == 0 ? st.bp1 : mode == 2 ? st.bp3 : st.bpx;
  k_bp_median<<<st.nbeam, kBeamT, 0, s>>>(bp, st.nchan, st.bp_median);
  return 2;
}

// measure_ts: per sample, fp16 running sum over channels in channel order,
// then ts = float(sum) / nchan.  A lane holds a sample; lane l is l channel
// pairs behind lane 0, so the 32 lanes of a warp look up 32 different pairs,
// and with the table as [level][pair] every lookup of a warp hits 32 different
// banks whatever the levels are (with all lanes on one channel the levels fall
// on random banks, three to four passes a lookup).  An iteration takes two
// pairs of every lane; the first and last 16 leave out what lies outside.
// The table (kTsSlots chunks of kTsC channels, two 64 KB halves of 64 pairs: a
// byte permute puts level, pair and half into an address) and each warp's 32
// gulp rows (kTsRows chunks) are rings that asynchronous copies fill one chunk
// ahead.  Bound by the lookups (shared memory): 65,536 samples x 2048 channels
// 48 us, 147 us with the lanes on one channel.
constexpr int kTsC = 64, kTsSlots = 4, kTsRows = 3;
constexpr int kTsLut = kTsSlots * kTsC * 256 * (int)sizeof(__half);  // bytes of the table ring
constexpr int kTsPitch = kTsRows * kTsC;                            // bytes of a ring row: even lanes' words and
                                                                    // odd lanes' fall on different banks
constexpr int kTsWarps = 16;                                        // most sums a block (warps)
__host__ __device__ constexpr int ts_smem(int nw) { return kTsLut + nw * 32 * kTsPitch; }
__global__ void __launch_bounds__(32 * kTsWarps) k_ts(const uint8_t *__restrict__ gulp, FlagState st, int nw) {
  extern __shared__ __align__(16) uint8_t ts_s[];
  const int b = blockIdx.y, nchan = st.nchan, w = st.gulp;
  const int tid = threadIdx.x, lane = tid & 31, wi = tid >> 5;
  const int t0 = (blockIdx.x * nw + wi) * 32;
  const bool live = wi < nw && t0 < w;  // the other warps only copy (w % 32 == 0: whole warps)
  uint8_t *rows = ts_s + kTsLut + wi * 32 * kTsPitch;
  const uint8_t *g = gulp + ((size_t)b * w + t0) * nchan;
  const int nchunk = (nchan + kTsC - 1) / kTsC;
  auto copy16 = [](void *d, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(d)), "l"(src)
                 : "memory");
  };
  // a thread's part of each chunk: table rows lv, lv + lstep, .., channels 8 lk .. + 7; gulp rows rr,
  // rr + 8, .., bytes 16 rk .. + 15
  constexpr int kLk = kTsC / 8, kRk = kTsC / 16;
  const int lk = tid % kLk, lv = tid / kLk, lstep = blockDim.x / kLk, rk = lane % kRk, rr = lane / kRk;
  auto load = [&](int m) {  // chunk m of the table and the rows
    if (m < nchunk) {
      uint8_t *d = ts_s + (m & 2) * (kTsLut / 4) + (m & 1) * (kTsC * 2) + lv * 256 + lk * 16;
      const __half *src = lut_row(st.lut, nchan, b, m * kTsC, lv) + 8 * lk;
#pragma unroll 4
      for (int v = lv; v < 256; v += lstep, d += lstep * 256, src += lstep * kLutSl) copy16(d, src);
      if (live && m * kTsC + rk * 16 < nchan) {
        uint8_t *e = rows + rr * kTsPitch + m % kTsRows * kTsC + rk * 16;
        const uint8_t *q = g + (size_t)rr * nchan + m * kTsC + rk * 16;
#pragma unroll
        for (int r = 0; r < 32; r += 32 / kRk) copy16(e + r * kTsPitch, q + (size_t)r * nchan);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int nq = nchan / 4, np = nchan / 2;
  const uint32_t sel = lane & 1 ? 0x5432u : 0x7654u;  // odd lanes start in the middle of a word of four channels
  uint32_t y = (4u * (128u - lane)) & 0x1ffu;         // 4 x pair, modulo the table ring
  uint32_t rq = (kTsPitch - 4 * (lane / 2)) % kTsPitch;  // byte in the ring row
  uint32_t prev = 0;
  __half s = hzero();
  const uint8_t *rl = rows + lane * kTsPitch;
  auto iterate = [&](int i, bool edge) {
    const uint32_t cur = *reinterpret_cast<const uint32_t *>(rl + rq);
    const uint32_t x = __byte_perm(prev, cur, sel), y1 = (y + 4u) & 0x1ffu;
    prev = cur;
    __half v[4];
    v[0] = *reinterpret_cast<const __half *>(ts_s + __byte_perm(x, y, 0x7504));
    v[1] = *reinterpret_cast<const __half *>(ts_s + __byte_perm(x, y, 0x7514) + 2);
    v[2] = *reinterpret_cast<const __half *>(ts_s + __byte_perm(x, y1, 0x7524));
    v[3] = *reinterpret_cast<const __half *>(ts_s + __byte_perm(x, y1, 0x7534) + 2);
    if (edge) {  // adding +0 changes no sum: it starts at +0 and is never -0
      const int p = 2 * i - lane;
      if (p < 0 || p >= np) v[0] = v[1] = hzero();
      if (p + 1 < 0 || p + 1 >= np) v[2] = v[3] = hzero();
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) s = __hadd(s, v[k]);
    y = (y + 8u) & 0x1ffu;
    rq = min(rq + 4u, rq + 4u - (uint32_t)kTsPitch);
  };
  constexpr int kIt = kTsC / 4;  // iterations a chunk; 16 more after the last channel
  load(0);
  for (int m = 0; m * kIt < nq + 16; ++m) {
    load(m + 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (live) {
      const int i0 = m * kIt, i1 = min(i0 + kIt, nq + 16);
      if (i0 >= 16 && i1 <= nq) {
#pragma unroll 8
        for (int i = i0; i < i1; ++i) iterate(i, false);
      } else {
#pragma unroll 1
        for (int i = i0; i < i1; ++i) iterate(i, true);
      }
    }
    __syncthreads();  // chunk m - 1 is overwritten next
  }
  if (live) {
    const float ts = __fdiv_rn(__half2float(s), (float)nchan);
    st.ts[(size_t)b * w + t0 + lane] = ts;
    const __half h = __float2half_rn(ts);
    st.hts[(size_t)b * w + t0 + lane] = h;
    st.tdiv[(size_t)b * w + t0 + lane] = make_float2(__half2float(h), __frcp_rn(__half2float(h)));
  }
}

// The launchers below with a null gulp only allow their kernel the most dynamic
// shared memory that any gulp takes, the same for all (flag_prepare).

// Launches k_sums.  Lane sums have 32 chains a channel: with fewer than four
// warps an SM in all, a lane takes two channels (twice the warps; levels are added
// two to a word anyway), blocks are as small as spreads them over the SMs and
// 32-row stages keep their fixed cost down (512 channels x 16,384 samples: 10.7 us,
// levels 9.1 us, 16 us with one chain a thread and 64 loads in flight); else, and for the row sums, 8 warps
// a block, two blocks an SM.
template <int MOD, bool VAR, bool TS, bool RAW, int CH, int ROWS, int AHEAD>
cudaError_t launch_sums(const FlagState &st, const uint8_t *gulp, int which, int nw, int per, cudaStream_t s) {
  const auto k = k_sums<MOD, VAR, TS, RAW, CH, ROWS, AHEAD>;
  auto smem = [](int warps) { return (RAW ? 0 : kLutBytes) + warps * (AHEAD + 1) * sum_stage(ROWS, CH, TS); };
  if (!gulp) return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem(kSumWarps));
  k<<<dim3(lut_slices(st.nchan), MOD / (nw * CH / 4 * per), st.nbeam), 32 * nw, smem(nw), s>>>(gulp, st, which, per);
  return cudaSuccess;
}
template <bool RAW>
cudaError_t launch_lanes(const FlagState &st, const uint8_t *gulp, cudaStream_t s) {
  const long warps = 32L * lut_slices(st.nchan) * st.nbeam;
  if (warps > 4 * 152) return launch_sums<32, false, false, RAW, 4, 16, 2>(st, gulp, 0, kSumWarps, 1, s);
  constexpr int kCh = RAW ? 4 : 2;
  const int lanes = warps > 2 * 152 ? 4 : warps > 152 ? 2 : 1;  // a block
  return launch_sums<32, false, false, RAW, kCh, 32, RAW ? 4 : 3>(st, gulp, 0, lanes * 4 / kCh, 1, s);
}
template <bool VAR, bool TS>
cudaError_t launch_rows(const FlagState &st, const uint8_t *gulp, int which, cudaStream_t s) {
  // several sums a warp where that leaves three blocks for each that fits: the table is staged less often
  const long blocks = 256L / kSumWarps * lut_slices(st.nchan) * st.nbeam;
  const int per = blocks >= 4 * 3 * 304 ? 4 : blocks >= 2 * 3 * 304 ? 2 : 1;
  return launch_sums<256, VAR, TS, false, 4, 8, 4>(st, gulp, which, kSumWarps, per, s);
}

// Launches k_ts with as many warps a block as fill whole rounds of one block
// an SM (the table ring leaves no room for two), and four at least to copy.
cudaError_t launch_ts(const FlagState &st, const uint8_t *gulp, cudaStream_t s) {
  if (!gulp) return cudaFuncSetAttribute(k_ts, cudaFuncAttributeMaxDynamicSharedMemorySize, ts_smem(kTsWarps));
  const long per = st.gulp / 32, warps = per * st.nbeam;
  const long rounds = (warps + 152 * kTsWarps - 1) / (152 * kTsWarps);
  const int nw = (int)((warps + 152 * rounds - 1) / (152 * rounds));
  k_ts<<<dim3((unsigned)((per + nw - 1) / nw), st.nbeam), 32 * std::max(nw, 4), ts_smem(std::max(nw, 4)), s>>>(gulp, st,
                                                                                                          nw);
  return cudaSuccess;
}

// transpose_output (transpose.cu:321-331): u8 = trunc(clamp(255/14 (x+4))).
constexpr float kRequant = 255.f / 14.f;
__device__ __forceinline__ uint8_t requant(__half h) {
  float v = __fmul_rn(kRequant, __fadd_rn(__half2float(h), 4.f));
  if (v < 0.f) v = 0.f;
  if (v > 255.f) v = 255.f;
  return (uint8_t)v;
}
// The same bytes as the lowest of lo and hi: x is held in [-4, 10 + 1/128], whose
// ends give 0 and 255 (NaN gives 0), and 2^23 plus the product, rounded toward zero
// once, ends in its whole part (k_fp16_selftest compares every half on the device).
__device__ __forceinline__ void requant2(__half2 x, uint32_t &lo, uint32_t &hi) {
  x = __hmin2(__hmax2(x, __float2half2_rn(-4.f)), __float2half2_rn(10.0078125f));
  lo = __float_as_uint(__fmaf_rz(kRequant, __fadd_rn(__low2float(x), 4.f), 8388608.f));
  hi = __float_as_uint(__fmaf_rz(kRequant, __fadd_rn(__high2float(x), 4.f), 8388608.f));
}

// Final stage: divide_by_ts, normalize_data, requantise, and write the
// channel-major ring.  A block takes a slice of 128 channels, its table in
// shared memory for all of its `run` tiles of kOutT samples.  Warps hold samples,
// lanes four channels, looked up as in k_sums; a lane's four samples of four
// channels become four words of four samples by byte permutes, go through a
// shared tile ([channel within lane][lane], an odd number of words a row:
// conflict-free both ways) and leave as 128 bytes of one channel a warp.  The
// next tile's words are loaded before the current one's are mapped.  The ring
// position of a gulp (and R) are multiples of 32, so no word straddles the
// ring's end.  Bound by instruction issue (about 20 a sample): 8 beams x 32,768 samples
// x 1024 channels 198 us, 424 us with one channel a lane and half-precision
// division.
constexpr int kOutT = 128, kOutRows = kOutT / 8;  // samples a tile, a warp
constexpr int kOutPitch = kOutT / 4 + 1;          // words a tile row
constexpr int kOutTile = 4 * 32 * kOutPitch * 4, kOutTd = 2 * kOutT * (int)sizeof(float2);
constexpr int kOutSmem = kLutBytes + kOutTile + kOutTd;
__global__ void __launch_bounds__(256, 2) k_flag_out(const uint8_t *__restrict__ gulp, FlagState st,
                                                     uint8_t *__restrict__ plain, long R, long wpos,
                                                     const GulpPos *dpos, int run) {
  if (dpos) wpos = dpos->wpos;
  extern __shared__ __align__(16) uint8_t out_s[];
  uint32_t *tile = reinterpret_cast<uint32_t *>(out_s + kLutBytes);
  const int b = blockIdx.z, c0 = blockIdx.x * kLutSl, nchan = st.nchan, w = st.gulp;
  const int tid = threadIdx.x, lane = tid & 31, wi = tid >> 5;
  const int tile0 = blockIdx.y * run, ntile = min(run, (w + kOutT - 1) / kOutT - tile0);
  const uint8_t *lsrc = reinterpret_cast<const uint8_t *>(lut_row(st.lut, nchan, b, c0, 0));
#pragma unroll 4
  for (int i = tid * 16; i < kLutBytes; i += 256 * 16) copy_async<16>(out_s + i, lsrc + i);
  // this warp's samples of a tile: kOutRows from wi * kOutRows on; their words and divisors
  float2 *td = reinterpret_cast<float2 *>(out_s + kLutBytes + kOutTile) + wi * kOutRows;
  const bool mine = c0 + 4 * lane < nchan;
  const uint8_t *g = gulp + ((size_t)b * w + tile0 * kOutT + wi * kOutRows) * nchan + c0 + 4 * lane;
  uint32_t x[kOutRows] = {};
  auto load = [&](int k) {
    const int t = (tile0 + k) * kOutT + wi * kOutRows;
    if (k < ntile && t < w) {  // w % 32 == 0: all of the warp's samples or none
      if (mine)
#pragma unroll
        for (int r = 0; r < kOutRows; ++r) x[r] = *reinterpret_cast<const uint32_t *>(g + (size_t)r * nchan);
      if (lane < kOutRows) copy_async<8>(td + (k & 1) * kOutT + lane, st.tdiv + (size_t)b * w + t + lane);
      g += (size_t)kOutT * nchan;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(0);
  const __half2 a2 = __half2half2(st.hsc[b * 8 + 2]), m2 = __half2half2(st.hsc[b * 8 + 3]);
  const bool hi = lane >= 16;  // channels 2, 3 of its four first
  const uint32_t first = 8u * lane + (hi ? 4u : 0u), second = 8u * lane + (hi ? 0u : 4u);
  uint8_t *pb = plain + ((size_t)b * nchan + c0) * R;
  for (int k = 0; k < ntile; ++k) {
    uint32_t cur[kOutRows];
#pragma unroll
    for (int r = 0; r < kOutRows; ++r) cur[r] = __byte_perm(x[r], x[r], hi ? 0x1032 : 0x3210);
    load(k + 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // the table; the divisors; the tile's readers are done
    const float2 *tdk = td + (k & 1) * kOutT;
#pragma unroll
    for (int r0 = 0; r0 < kOutRows; r0 += 4) {
      uint32_t o[4][4];  // [sample][channel as taken]
      auto map = [&](bool fast) {
        __half2 sum = __half2half2(hzero());
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float2 t = tdk[r0 + r];
          __half h[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            h[q] = *reinterpret_cast<const __half *>(
                out_s + __byte_perm(cur[r0 + r], q < 2 ? first : second, 0x7704 + 16 * q) + 2 * (q & 1));
#pragma unroll
          for (int q = 0; q < 4; q += 2) {
            __half2 p;
            if (fast) {
              p = __floats2half2_rn(div_step(__half2float(h[q]), t.x, t.y), div_step(__half2float(h[q + 1]), t.x, t.y));
              sum = __hadd2(sum, p);
            } else {
              const __half th = __float2half_rn(t.x);
              p = __halves2half2(__hdiv(h[q], th), __hdiv(h[q + 1], th));
            }
            requant2(__hmul2(__hadd2(p, a2), m2), o[r][q], o[r][q + 1]);
          }
        }
        return __half2float(__low2half(sum)) + __half2float(__high2half(sum));
      };
      // a quotient that div_step does not give leaves the sum infinite or NaN
      if (!(fabsf(map(true)) <= 1e30f)) map(false);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t lo = __byte_perm(o[0][q], o[1][q], 0x0040), hi2 = __byte_perm(o[2][q], o[3][q], 0x0040);
        tile[((hi ? q ^ 2 : q) * 32 + lane) * kOutPitch + (wi * kOutRows + r0) / 4] = __byte_perm(lo, hi2, 0x5410);
      }
    }
    __syncthreads();
    const int t = (tile0 + k) * kOutT, nq = min(kOutT, w - t) / 4;  // w % 32 == 0
    long pos = wpos + t + 4 * lane;
    if (pos >= R) pos -= R;
    if (lane < nq) {
      uint8_t *d = pb + (size_t)wi * R + pos;
      const uint32_t *row = tile + ((wi & 3) * 32 + (wi >> 2)) * kOutPitch + lane;  // channel wi; wi + 8 is two lanes on
      const int nc = min(kLutSl, nchan - c0);
#pragma unroll 4
      for (int c = wi; c < nc; c += 8, d += 8 * R, row += 2 * kOutPitch) *reinterpret_cast<uint32_t *>(d) = *row;
    }
  }
}
static_assert(kOutT / 4 == 32, "a lane a word of a tile's row");

// Launches k_flag_out with runs that leave four blocks an SM (two fit) where the
// gulp has as many tiles.
cudaError_t launch_out(const FlagState &st, const uint8_t *gulp, uint8_t *plain, long R, long wpos,
                       const GulpPos *dpos, cudaStream_t s) {
  if (!gulp) return cudaFuncSetAttribute(k_flag_out, cudaFuncAttributeMaxDynamicSharedMemorySize, kOutSmem);
  const int tiles = (st.gulp + kOutT - 1) / kOutT;
  const long all = (long)tiles * lut_slices(st.nchan) * st.nbeam;
  const int run = (int)std::max(1L, std::max(all / (4 * 152), (tiles + 65534L) / 65535));
  k_flag_out<<<dim3(lut_slices(st.nchan), (tiles + run - 1) / run, st.nbeam), 256, kOutSmem, s>>>(gulp, st, plain, R,
                                                                                              wpos, dpos, run);
  return cudaSuccess;
}

}  // namespace

namespace {
// ------------------------------------------------ SCRUNCH entries (planes)
// Kernels of the plane path, each the counterpart of a reference kernel run
// on the fp16 copy of the gulp; index `i` runs over [nbeam][nchan][gulp].

// The data after bandpass_flag (table stage 3) as a channel-major plane.
__global__ void k_plane_init(const uint8_t *__restrict__ gulp, FlagState st) {
  __shared__ uint8_t tile[32][33];
  const int b = blockIdx.z, c0 = blockIdx.x * 32, t0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y, nchan = st.nchan, w = st.gulp;
  const uint8_t *g = gulp + (size_t)b * w * nchan;
#pragma unroll
  for (int j = 0; j < 32; j += 8) tile[ty + j][tx] = g[(size_t)(t0 + ty + j) * nchan + c0 + tx];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    const int c = c0 + ty + j;
    st.P[((size_t)b * nchan + c) * w + t0 + tx] = *lut_row(st.lut, nchan, b, c, tile[tx][ty + j]);
  }
}

// A map over the plane, row by row: eight neighbouring halves a thread, op(half,
// channel row, sample); the gulp is a multiple of 32 samples.  (One element a
// thread with a 64-bit division for its row took 10 to 12 us for 512 x 8192, 4.4 to 5.4 us.)
constexpr int kMapT = 256;
template <class Op>
__device__ __forceinline__ void plane_map(const FlagState &st, const __half *in, __half *out, Op op) {
  const int t = 8 * (blockIdx.x * kMapT + threadIdx.x);
  if (t >= st.gulp) return;
  const size_t row = (size_t)blockIdx.z * st.nchan + blockIdx.y, i = row * st.gulp + t;
  uint4 q = *reinterpret_cast<const uint4 *>(in + i);
  __half *h = reinterpret_cast<__half *>(&q);
#pragma unroll
  for (int k = 0; k < 8; ++k) h[k] = op(h[k], row, t + k);
  *reinterpret_cast<uint4 *>(out + i) = q;
}
dim3 map_grid(const FlagState &st) { return dim3((st.gulp / 8 + kMapT - 1) / kMapT, st.nchan, st.nbeam); }
constexpr int kPlaneB = 64;  // loads in flight a thread in the plane's sums, whose chains are few (512 x 8192: lane
                             // sums 11.2 -> 7.3 us, time series 36 -> 12 us; the launch bounds give them registers)

// calc_bandpass_new partials of the plane (lane l: samples l, l+32, ...).
// One warp per (beam, channel).
__global__ void __launch_bounds__(256, 2) k_plane_lanes(FlagState st) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (gw >= st.nbeam * st.nchan) return;
  const __half *p = st.P + (size_t)gw * st.gulp + lane;
  const int np = st.gulp / 32;
  float s = 0.f;
  int i = 0;
  for (; i + kPlaneB <= np; i += kPlaneB) {  // loads in flight, then the sums in order
    __half v[kPlaneB];
#pragma unroll
    for (int u = 0; u < kPlaneB; ++u) v[u] = p[(size_t)(i + u) * 32];
#pragma unroll
    for (int u = 0; u < kPlaneB; ++u) s = __fadd_rn(s, __half2float(v[u]));
  }
  for (; i < np; ++i) s = __fadd_rn(s, __half2float(p[(size_t)i * 32]));
  st.part[(size_t)gw * 32 + lane] = s;
}

// divide_by_bp (flagger.cu:180-194) with bandpass bp [nbeam][nchan].
__global__ void __launch_bounds__(kMapT) k_plane_div(FlagState st, const float *bp) {
  const float v = bp[(size_t)blockIdx.z * st.nchan + blockIdx.y];
  const __half d = __float2half_rn(v);
  plane_map(st, st.P, st.P, [=](__half x, size_t, int) { return v > 0.f ? __hdiv(x, d) : hzero(); });
}

// computeRowMeans / computeRowVariances partials of the plane.
template <bool VAR>
__global__ void __launch_bounds__(256) k_plane_rows(FlagState st, int which) {
  const int c = blockIdx.x, b = blockIdx.y, j = threadIdx.x, w = st.gulp;
  const __half *p = st.P + ((size_t)b * st.nchan + c) * w + j;
  const float mean = VAR ? st.scal[b * 8 + 2 * which] : 0.f;
  float s = 0.f;
#pragma unroll 8
  for (int k = 0; k < w / 256; ++k) {
    const float f = __half2float(p[(size_t)k * 256]);
    if (VAR) {
      const float d = __fsub_rn(f, mean);
      s = __fmaf_rn(d, d, s);
    } else {
      s = __fadd_rn(s, f);
    }
  }
  st.part[((size_t)b * st.nchan + c) * 256 + j] = s;
}

// normalize_data (flagger.cu:198-214) with the constants of slot `which`.
__global__ void __launch_bounds__(kMapT) k_plane_norm(FlagState st, int which) {
  const __half a = st.hsc[blockIdx.z * 8 + 2 * which], m = st.hsc[blockIdx.z * 8 + 2 * which + 1];
  plane_map(st, st.P, st.P, [=](__half x, size_t, int) { return __hmul(__hadd(x, a), m); });
}

// npp_convolve_handler (convolution.cu:20-55): an xw (time) x yw (channel)
// box of equal taps k, anchor (xw/2, yw/2), replicate border, fp32 sum of
// fp16 input, fp16 output.  Tap (j, i) multiplies input (c + ay - j,
// t + ax - i); the sum runs j outer, i inner, one fmaf per tap.  A block
// computes 64 samples x 16 channels from a staged halo tile.
constexpr int kBoxT = 64, kBoxC = 16;
__global__ void __launch_bounds__(256) k_box(const __half *__restrict__ in, __half *__restrict__ out,
                                             int nchan, int w, int xw, int yw, float k) {
  extern __shared__ float tile[];
  const int b = blockIdx.z, t0 = blockIdx.x * kBoxT, c0 = blockIdx.y * kBoxC, tid = threadIdx.x;
  const int ax = xw / 2, ay = yw / 2;
  const int tw = kBoxT + xw - 1, th = kBoxC + yw - 1;
  const int cb = c0 + ay - (yw - 1), tb = t0 + ax - (xw - 1);  // tile origin (before clamping)
  const __half *src = in + (size_t)b * nchan * w;
  for (int q = tid; q < tw * th; q += 256) {
    const int r = q / tw, col = q - r * tw;
    const int cc = min(max(cb + r, 0), nchan - 1), tt = min(max(tb + col, 0), w - 1);
    tile[q] = __half2float(src[(size_t)cc * w + tt]);
  }
  __syncthreads();
  const int tl = tid & (kBoxT - 1);
  for (int cl = tid >> 6; cl < kBoxC; cl += 256 / kBoxT) {
    const int c = c0 + cl, t = t0 + tl;
    float acc = 0.f;
    for (int j = 0; j < yw; ++j) {
      const float *row = tile + (size_t)(cl + yw - 1 - j) * tw + tl + xw - 1;
      for (int i = 0; i < xw; ++i) acc = __fmaf_rn(k, row[-i], acc);
    }
    if (c < nchan && t < w) out[((size_t)b * nchan + c) * w + t] = __float2half_rn(acc);
  }
}

// threshold_data (flagger.cu:162-176): mask 1 where the smoothed value
// exceeds +-half(thr).
__global__ void __launch_bounds__(kMapT) k_plane_thresh(FlagState st, __half hp, __half hn) {
  const float p = __half2float(hp), m = __half2float(hn);
  plane_map(st, st.S, st.M, [=](__half x, size_t, int) {
    const float v = __half2float(x);
    return (v > p || v < m) ? hone() : hzero();
  });
}

// replace_data (flagger.cu:128-144) with FLAG1/FLAG2, then add_number 1.
__global__ void __launch_bounds__(kMapT) k_plane_replace(FlagState st) {
  const int c = blockIdx.y;
  const bool band = c >= st.flag_lo && c < st.flag_hi;
  const __half *S = st.S;
  const size_t w = st.gulp;
  plane_map(st, st.P, st.P, [=](__half x, size_t row, int t) {
    return __hadd(band || __half2float(S[row * w + t]) > 0.f ? hzero() : x, hone());
  });
}

// calc_bandpass (flagger.cu:50-81) of the grown mask: thread t sums its
// contiguous floor(w/256) samples in fp16, / half(256 floor(w/256)), then an
// fp16 tree.  Block = (channel, beam).
__global__ void __launch_bounds__(256) k_plane_bp16(FlagState st) {
  __shared__ __half ps[256];
  const int c = blockIdx.x, b = blockIdx.y, t = threadIdx.x, np = st.gulp / 256;
  const __half *p = st.S + ((size_t)b * st.nchan + c) * st.gulp + (size_t)t * np;
  __half s = hzero();
  for (int i = 0; i < np; ++i) s = __hadd(s, p[i]);
  ps[t] = __hdiv(s, __float2half_rn((float)(256 * np)));
  __syncthreads();
  for (int h = 128; h >= 1; h /= 2) {
    if (t < h) ps[t] = __hadd(ps[t], ps[t + h]);
    __syncthreads();
  }
  if (t == 0) st.fsb[(size_t)b * st.nchan + c] = __half2float(ps[0]);
}

// replace_data_and_add_bandpass (flagger.cu:146-158): flagged channels 1,
// the others x + 1.
__global__ void __launch_bounds__(kMapT) k_plane_spec(FlagState st) {
  const bool flagged = st.flag2[(size_t)blockIdx.z * st.nchan + blockIdx.y];
  plane_map(st, st.P, st.P, [=](__half x, size_t, int) { return flagged ? hone() : __hadd(x, hone()); });
}

// add_bandpass into d_flagSpec (flagger.cu:333-334), beams in order.
__global__ void k_flagspec_add(FlagState st) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= st.nchan) return;
  float f = st.flagspec[c];
  for (int b = 0; b < st.nbeam; ++b) f = __fadd_rn(f, st.fsb[(size_t)b * st.nchan + c]);
  st.flagspec[c] = f;
}

// measure_ts + divide_by_ts (timeseries.cu:19-55) on the plane.
__global__ void __launch_bounds__(64, 8) k_plane_ts(FlagState st) {
  const int b = blockIdx.y, t = blockIdx.x * blockDim.x + threadIdx.x, w = st.gulp;
  if (t >= w) return;
  const __half *p = st.P + (size_t)b * st.nchan * w + t;
  __half s = hzero();
  int c = 0;
  for (; c + kPlaneB <= st.nchan; c += kPlaneB) {
    __half v[kPlaneB];
#pragma unroll
    for (int u = 0; u < kPlaneB; ++u) v[u] = p[(size_t)(c + u) * w];
#pragma unroll
    for (int u = 0; u < kPlaneB; ++u) s = __hadd(s, v[u]);
  }
  for (; c < st.nchan; ++c) s = __hadd(s, p[(size_t)c * w]);
  const float ts = __fdiv_rn(__half2float(s), (float)st.nchan);
  st.ts[(size_t)b * w + t] = ts;
  st.hts[(size_t)b * w + t] = __float2half_rn(ts);
}

__global__ void __launch_bounds__(kMapT) k_plane_tsdiv(FlagState st) {
  const __half *hts = st.hts + (size_t)blockIdx.z * st.gulp;
  plane_map(st, st.P, st.P, [=](__half x, size_t, int t) { return __hdiv(x, hts[t]); });
}

// transpose_output of the plane into the channel-major ring.
__global__ void k_plane_out(FlagState st, uint8_t *__restrict__ plain, long R, long wpos, const GulpPos *dpos) {
  if (dpos) wpos = dpos->wpos;
  const int b = blockIdx.z, c = blockIdx.y, w = st.gulp;
  const __half *p = st.P + ((size_t)b * st.nchan + c) * w;
  uint8_t *row = plain + ((size_t)b * st.nchan + c) * R;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < w; t += gridDim.x * blockDim.x) {
    long pos = wpos + t;
    if (pos >= R) pos -= R;
    row[pos] = requant(p[t]);
  }
}

}  // namespace

namespace {

// SCRUNCH entries and the final scrunch on fp16 planes (flagger.cu:365-401),
// from the data after bandpass_flag.
cudaError_t scrunch_planes(const FlagState &st, const void *gulp, uint8_t *plain, long R, long wpos,
                           const GulpPos *dpos, cudaStream_t s) {
  const int fin_blocks = (st.nbeam * st.nchan * 32 + 255) / 256;
  const dim3 fing(st.nchan / (kBeamT / 32), st.nbeam);
  const size_t n = (size_t)st.nbeam * st.nchan * st.gulp;
  const dim3 chg(st.nchan, st.nbeam);
  unsigned launches = 0;
  auto normalize = [&](int which) {
    k_plane_rows<false><<<chg, 256, 0, s>>>(st, which);
    k_row_finish<false><<<fing, kBeamT, 0, s>>>(st, which);
    k_plane_rows<true><<<chg, 256, 0, s>>>(st, which);
    k_row_finish<true><<<fing, kBeamT, 0, s>>>(st, which);
    k_plane_norm<<<map_grid(st), kMapT, 0, s>>>(st, which);
    launches += 5;
  };
  auto bandpass_correct = [&](int mode, const float *bp) {
    k_plane_lanes<<<fin_blocks, 256, 0, s>>>(st);
    launches += lane_finish(st, mode, fin_blocks, s);
    k_plane_div<<<map_grid(st), kMapT, 0, s>>>(st, bp);
    launches += 2;
  };
  if (st.f16_input) {
    // the DADA path (transpose.cu:87-90): the gulp is the fp16 plane; bandpass_flag on it
    cudaError_t e = cudaMemcpyAsync(st.P, gulp, n * sizeof(__half), cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    bandpass_correct(0, st.bp1);
    normalize(0);
    k_plane_lanes<<<fin_blocks, 256, 0, s>>>(st);
    k_lane_finish<<<fin_blocks, 256, 0, s>>>(st, 1);
    k_plane_spec<<<map_grid(st), kMapT, 0, s>>>(st);
    launches += 3;
  } else {
    k_plane_init<<<dim3(st.nchan / 32, st.gulp / 32, st.nbeam), dim3(32, 8), 0, s>>>(
        static_cast<const uint8_t *>(gulp), st);
    launches += 1;
  }
  for (int e = 0; e < st.nscrunch; ++e) {
    const int xw = st.sc_t[e], yw = st.sc_f[e];
    bandpass_correct(3, st.bpx);
    normalize(2);
    const float k = (float)(1. / xw / yw);
    const float thr = (float)(st.sc_thresh[e] / std::sqrt(1. * xw * yw));
    const __half hp = __float2half_rn(thr), hn = __float2half_rn((float)(-1. * thr));
    const dim3 bg((st.gulp + kBoxT - 1) / kBoxT, (st.nchan + kBoxC - 1) / kBoxC, st.nbeam);
    const size_t smem = sizeof(float) * (size_t)(kBoxT + xw - 1) * (kBoxC + yw - 1);
    k_box<<<bg, 256, smem, s>>>(st.P, st.S, st.nchan, st.gulp, xw, yw, k);
    k_plane_thresh<<<map_grid(st), kMapT, 0, s>>>(st, hp, hn);
    k_box<<<bg, 256, smem, s>>>(st.M, st.S, st.nchan, st.gulp, xw, yw, k);
    k_plane_replace<<<map_grid(st), kMapT, 0, s>>>(st);
    launches += 4;
    if (st.flagspec) {
      k_plane_bp16<<<chg, 256, 0, s>>>(st);
      k_flagspec_add<<<(st.nchan + 255) / 256, 256, 0, s>>>(st);
      launches += 2;
    }
  }
  // apply_scrunch(8, 8, 100, flag=0, ts=1)
  bandpass_correct(2, st.bp3);
  k_plane_ts<<<dim3((st.gulp + 63) / 64, st.nbeam), 64, 0, s>>>(st);
  k_plane_tsdiv<<<map_grid(st), kMapT, 0, s>>>(st);
  normalize(1);
  k_plane_out<<<dim3((st.gulp + 1023) / 1024, st.nchan, st.nbeam), 256, 0, s>>>(st, plain, R, wpos, dpos);
  launches += 3;
  count_launches(launches);
  return cudaGetLastError();
}

cudaError_t flag_impl(const FlagState &st, const void *gulp_in, uint8_t *plain, long R, long wpos,
                      const GulpPos *dpos, cudaStream_t s) {
  if (st.f16_input) return scrunch_planes(st, gulp_in, plain, R, wpos, dpos, s);
  const uint8_t *gulp = static_cast<const uint8_t *>(gulp_in);
  const int fin_blocks = (st.nbeam * st.nchan * 32 + 255) / 256;
  const dim3 fing(st.nchan / (kBeamT / 32), st.nbeam);

  cudaError_t e = cudaSuccess;
  unsigned launches = 0;
  // lane sums, the bandpass of `mode` and the tables of `stage` made with it (through
  // the median filter where bandpass_correct applies it)
  auto bandpass = [&](bool raw, int mode, int stage) {
    if (e == cudaSuccess) e = raw ? launch_lanes<true>(st, gulp, s) : launch_lanes<false>(st, gulp, s);
    ++launches;
    const bool median = mode != 1 && st.bp_median > 1;
    if (median) launches += lane_finish(st, mode, fin_blocks, s);
    launch_lut(st, stage, median ? -1 : mode, s);
    ++launches;
  };
  auto normalize = [&](int which) {  // calculate_stddev: mean pass, variance pass
    if (e == cudaSuccess) e = which ? launch_rows<false, true>(st, gulp, which, s) : launch_rows<false, false>(st, gulp, which, s);
    k_row_finish<false><<<fing, kBeamT, 0, s>>>(st, which);
    if (e == cudaSuccess) e = which ? launch_rows<true, true>(st, gulp, which, s) : launch_rows<true, false>(st, gulp, which, s);
    k_row_finish<true><<<fing, kBeamT, 0, s>>>(st, which);
    launches += 4;
  };
  // bandpass_flag: bandpass_correct (calc_bandpass_new, divide_by_bp), normalize_data
  bandpass(true, 0, 1);
  normalize(0);
  // calc_bandpass_new of the normalised data -> spectral flag
  launch_lut(st, 2, -1, s);
  bandpass(false, 1, 3);
  if (e != cudaSuccess) return e;
  if (st.nscrunch > 0) {
    count_launches(launches + 1);
    return scrunch_planes(st, gulp, plain, R, wpos, dpos, s);
  }
  // apply_scrunch(8,8,100,flag=0,ts=1): bandpass_correct, ts_correct, normalize_data
  bandpass(false, 2, 4);
  if (e == cudaSuccess) e = launch_ts(st, gulp, s);
  normalize(1);
  if (e != cudaSuccess) return e;
  // transpose_output into the ring
  if ((e = launch_out(st, gulp, plain, R, wpos, dpos, s)) != cudaSuccess) return e;
  count_launches(launches + 3);
  return cudaGetLastError();
}
}  // namespace

cudaError_t flag_prepare(const FlagState &st) {
  cudaError_t e = launch_lanes<true>(st, nullptr, nullptr);
  if (e == cudaSuccess) e = launch_lanes<false>(st, nullptr, nullptr);
  if (e == cudaSuccess) e = launch_rows<false, false>(st, nullptr, 0, nullptr);
  if (e == cudaSuccess) e = launch_rows<true, false>(st, nullptr, 0, nullptr);
  if (e == cudaSuccess) e = launch_rows<false, true>(st, nullptr, 1, nullptr);
  if (e == cudaSuccess) e = launch_rows<true, true>(st, nullptr, 1, nullptr);
  if (e == cudaSuccess) e = launch_ts(st, nullptr, nullptr);
  if (e == cudaSuccess) e = launch_out(st, nullptr, nullptr, 0, 0, nullptr, nullptr);
  return e;
}

// The ring writers store 4-byte words: the ring length and every write
// position (gulp starts) are multiples of 32 samples.
cudaError_t flag_gulp(const FlagState &st, const void *gulp, uint8_t *plain, long R, long wpos,
                      cudaStream_t s) {
  if (R % 32 != 0 || wpos % 32 != 0 || st.gulp % 32 != 0) return cudaErrorInvalidValue;
  return flag_impl(st, gulp, plain, R, wpos, nullptr, s);
}

cudaError_t flag_gulp_dev(const FlagState &st, const void *gulp, uint8_t *plain, long R,
                          const GulpPos *pos, cudaStream_t s) {
  if (R % 32 != 0 || st.gulp % 32 != 0) return cudaErrorInvalidValue;
  return flag_impl(st, gulp, plain, R, 0, pos, s);
}

// ----------------------------------------------------------- self-check
namespace {

__global__ void k_fp16_selftest(unsigned long long *bad, unsigned int *first) {
  auto check = [&](bool mismatch, unsigned int a, unsigned int b) {
    if (mismatch) {
      atomicAdd(bad, 1ull);
      atomicCAS(first, 0xffffffffu, (a << 16) | b);
    }
  };
  auto quotient = [](__half a, __half b) {  // as k_sums and k_flag_out form it
    return div_step(__half2float(a), __half2float(b), __frcp_rn(__half2float(b)));
  };
  const unsigned long long n = 31744ull * 31743ull;  // a in [0, 0x7c00), b in [1, 0x7c00)
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned short ab = (unsigned short)(i / 31743ull);
    const unsigned short bb = (unsigned short)(i % 31743ull + 1);
    const __half a = __ushort_as_half(ab), b = __ushort_as_half(bb);
    const float fa = __half2float(a), fb = __half2float(b);
    bool mismatch = __half_as_ushort(__hdiv(a, b)) != __half_as_ushort(__float2half_rn(__fdiv_rn(fa, fb)));
    if ((i & 63) == 0) {
      mismatch |= __half_as_ushort(__hadd(a, b)) != __half_as_ushort(__float2half_rn(__fadd_rn(fa, fb)));
      mismatch |= __half_as_ushort(__hmul(a, b)) != __half_as_ushort(__float2half_rn(__fmul_rn(fa, fb)));
    }
#pragma unroll
    for (int sg = 0; sg < 4; ++sg) {  // signs; of a zero quotient the sign may differ
      const __half sa = sg & 1 ? __hneg(a) : a, sb = sg & 2 ? __hneg(b) : b;
      const unsigned short q = __half_as_ushort(__float2half_rn(quotient(sa, sb))), h = __half_as_ushort(__hdiv(sa, sb));
      mismatch |= q != h && ((q | h) & 0x7fffu) != 0;
    }
    check(mismatch, ab, bb);
  }
  // zero, infinite or NaN divisors and dividends: what div_step gives is not finite (zero by infinity too);
  // every half requantised, as either of a pair
  const unsigned int h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h < 65536u) {
    const __half x = __ushort_as_half((unsigned short)h);
    const unsigned short odd[] = {0x0000, 0x8000, 0x7c00, 0xfc00, 0x7e00, 0xfe01};
    bool mismatch = false;
    for (int k = 0; k < 6; ++k) {
      mismatch |= fabsf(quotient(x, __ushort_as_half(odd[k]))) <= 3.0e38f;
      if (k > 1) mismatch |= fabsf(quotient(__ushort_as_half(odd[k]), x)) <= 3.0e38f;
    }
    const __half y = __ushort_as_half((unsigned short)(h ^ 0x5a5au));
    uint32_t lo, hi;
    requant2(__halves2half2(x, y), lo, hi);
    mismatch |= (lo & 0xffu) != requant(x) || (hi & 0xffu) != requant(y);
    check(mismatch, h, h);
  }
}

}  // namespace
}  // namespace hg

extern "C" hella_status hella_fp16_selftest(int device, unsigned long long *mismatches,
                                            uint32_t *first_bad) {
  if (!mismatches || !first_bad) return HELLA_ERR_INVALID_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return HELLA_ERR_CUDA;
  unsigned long long *d_bad = nullptr;
  unsigned int *d_first = nullptr;
  hella_status st = HELLA_OK;
  if (cudaMalloc(&d_bad, 8) != cudaSuccess || cudaMalloc(&d_first, 4) != cudaSuccess) {
    st = HELLA_ERR_ALLOC;
  } else if (cudaMemset(d_bad, 0, 8) != cudaSuccess || cudaMemset(d_first, 0xff, 4) != cudaSuccess) {
    st = HELLA_ERR_CUDA;
  } else {
    hg::k_fp16_selftest<<<152 * 8, 256>>>(d_bad, d_first);
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(mismatches, d_bad, 8, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(first_bad, d_first, 4, cudaMemcpyDeviceToHost) != cudaSuccess)
      st = HELLA_ERR_CUDA;
  }
  cudaFree(d_bad);
  cudaFree(d_first);
  cudaGetLastError();
  return st;
}
