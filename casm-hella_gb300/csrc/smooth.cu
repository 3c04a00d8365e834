// smooth.cu -- casm-hella's smoothing, per-width normalisation and peak
// finding on GB300.
//
// Reference: src/hella/src/smooth.cpp:21-127 and src/hella/src/peaks.cu:
// 31-117.  For every width sm = wmin*2^k < wmax the reference filters the
// dedispersed plane with a 3 x (2sm+1) kernel (DM weights 0.3/1/0.3 times
// time taps v(u)^2, normalised to sum 1), crops rows 1..ndms-2 and columns
// wmax/2 .. wmax/2+gulp, and standardises each width with
// calculate_stddev (normalization.cu:125-162).  find_peaks takes sigma of
// the standardised width-0 plane, gates the beam on 0.1 < sigma < 5 and
// emits every sample above snr*sigma in (width, DM row, time) order.
//
// Arithmetic (the oracle follows it operation for operation):
//   y[x]   = fmaf(0.3f, dd[r][x] + dd[r+2][x], dd[r+1][x])  (exact sum)
//   out[j] = fmaf chain over k = 0..2sm of tap[k] * y[clamp(x0 + k)]
// i.e. the DM weights factored out of the 2-D kernel, whose middle row
// supplies the time taps.  Borders replicate (NPP_BORDER_REPLICATE).
//
// Kernels.  k_firS filters a row with every width up to 32 from a register
// window (a block per row), k_firL with one larger width and a sliding window
// (a block per row and width).  Both form the
// row-mean partials of the reference's order (thread j sums columns j, j+256,
// ...) as they go; the plane is written once and read once more for the
// variance.  Row maxima let the peak pass skip rows that cannot hold
// a candidate.
#include "hg_internal.h"
#include "hg_ptx.h"

#include <algorithm>

namespace hg {
namespace {

constexpr int kT = 256;  // threads per row block of the statistics passes

__device__ __forceinline__ float block256_tree(const float *p) {
  // p: 256 partials in shared memory; called by one whole warp, returns in
  // its lane 0 the total the reference's thread 0 forms (normalization.cu:
  // 41-68: each warp's shuffle tree, then the warp totals in order).
  const int lane = threadIdx.x & 31;
  float tot = 0.f;
  for (int wi = 0; wi < 8; ++wi) {
    float v = p[wi * 32 + lane];
    for (int off = 16; off > 0; off /= 2) v = __fadd_rn(v, __shfl_down_sync(0xffffffffu, v, off));
    tot = wi == 0 ? v : __fadd_rn(tot, v);
  }
  return tot;
}

__device__ __forceinline__ float normv(float x, const float *st) {
  // smooth.cpp:105-123: skipped when std <= 0; else AddC(-mean), MulC(1/std)
  return st[1] > 0.f ? __fmul_rn(__fadd_rn(x, st[2]), st[3]) : x;
}

// Beam and beam-local row of global row `gr` of a launch.
__device__ __forceinline__ const SmoothBeam &row_beam(const SmoothArgs &a, int gr, int *r) {
  const SmoothBeam &B = a.beams[a.row_beam[gr]];
  *r = gr - B.row0;
  return B;
}

// 32 bytes to global memory in one store (a whole sector a lane).
__device__ __forceinline__ void store8(float *p, const float *v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The three dedispersed rows a smoothed row is made of, and its y values.
struct YRows {
  const float *a, *b, *c;
  int n;       // columns
  bool vec;    // 16-byte loads of columns 4k are aligned
  __device__ __forceinline__ YRows(const SmoothBeam &B, int r, int ntime_dd)
      : a(B.dd + (size_t)r * B.dd_stride), b(a + B.dd_stride), c(b + B.dd_stride), n(ntime_dd),
        vec((reinterpret_cast<uintptr_t>(B.dd) & 15) == 0 && B.dd_stride % 4 == 0) {}
  static __device__ __forceinline__ float y(float a, float b, float c) { return __fmaf_rn(0.3f, __fadd_rn(a, c), b); }
  __device__ __forceinline__ float at(int col) const {  // borders replicate
    col = col < 0 ? 0 : (col >= n ? n - 1 : col);
    return y(a[col], b[col], c[col]);
  }
};

// Row total of 256 partials p and maximum mx (every lane's), by one warp.
__device__ __forceinline__ void row_finish(const SmoothBeam &B, int b, int r, const float *p, float mx, int nwcol) {
  const float tot = block256_tree(p);
  for (int o = 16; o > 0; o /= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) {
    B.rowmean[(size_t)b * B.h + r] = __fdiv_rn(tot, (float)nwcol);
    B.rowmax[(size_t)b * B.h + r] = mx;
  }
}

// k_firS: the widths 1, 2, 4 .. 32 (wmin 1) of a launch, a block of four warps
// per row.  An iteration makes 1024 outputs of every width, a warp 256 of
// them, lane t outputs 8t .. 8t + 7 from the 72 y values they read, kept in
// registers, so that a tap is eight multiply-adds on registers and a constant:
// the taps are kernel arguments.  The y values sit in shared memory as groups
// of 8 at a pitch of 12 words (conflict-free 16-byte reads at a lane stride of
// one group), in two buffers: the 64 values two iterations share are copied to
// the front of the other one.  The three rows are copied an iteration ahead
// (cp.async, each thread the columns it reads back; in 4-byte pieces at the
// row's ends and where rows are not 16-byte aligned).  The outputs also go to
// shared memory, where thread i keeps the row-mean partials of columns 4i ..
// 4i + 3 (mod 256) of half of the widths and adds the warps' chunks in order:
// two block barriers an iteration.  Bound by issue (about 1330 instructions for
// a warp's 256 outputs, 1056 of them multiply-adds, issued 70 % of the cycles).
// 8923 rows x 32768 x 6 widths: 1.92 ms, with rows staged by plain loads, taps
// in shared memory and a barrier-separated transpose of 2048 outputs 3.1 ms;
// 493 rows x 16384: 85 us against 103.  Three blocks an SM (132 registers)
// rather than four (124): 1.92 against 2.05 ms; a warp a row with the partials
// in registers 1.81 ms, but 105 us on the 493 rows, one warp's walk being long.
constexpr int kSO = 8;                   // outputs per lane
constexpr int kSWarps = 4;               // warps per block
constexpr int kST = 32 * kSWarps;        // threads per block
constexpr int kSC = kST * kSO;           // outputs per iteration
constexpr int kSSpan = 64;               // span of width 32
constexpr int kSW = 6;                   // widths 1, 2, 4, 8, 16, 32
constexpr int kSWin = kSO + kSSpan;      // y values a lane reads (72)
constexpr int kSPitch = 12;              // words from one group of 8 to the next
constexpr int kSY = (kSC + kSSpan) / 8 * kSPitch;
constexpr int kSRaw = 3 * kSC;           // words of an iteration's staged rows
constexpr size_t kSSmem = sizeof(float) * (2 * kSY + kSRaw + kSW * kSC);
__host__ __device__ constexpr int small_tap(int b) { return 2 * ((1 << b) - 1) + b; }  // first tap of width 2^b
struct SmallTaps {
  float t[small_tap(kSW)];
};
// Word of 16-byte slot s: the two slots of a lane's 8 values trade places in every other eight, so
// that lanes reading or writing slots 2t (or 2t + 1) meet no bank conflict.
__device__ __forceinline__ int slot_word(int s) { return 4 * (s ^ ((s >> 3) & 1)); }

// One width (2 SM + 1 taps) of a lane's 8 outputs from its register window.
template <int SM, int ANCHOR>
__device__ __forceinline__ void firS_width(const float (&win)[kSWin], const float *tp, float (&acc)[kSO]) {
  constexpr int NT = 2 * SM + 1, OFF = ANCHOR ? kSSpan - 2 * SM : 0;
#pragma unroll
  for (int i = 0; i < kSO; ++i) acc[i] = 0.f;
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < kSO; ++i) acc[i] = __fmaf_rn(tp[n], win[OFF + i + n], acc[i]);
}

template <int ANCHOR>
__global__ void __launch_bounds__(kST, 3) k_firS(SmoothArgs a, const __grid_constant__ SmallTaps taps, int b0, int b1) {
  extern __shared__ __align__(16) float sm[];
  int r;
  const SmoothBeam &B = row_beam(a, blockIdx.x, &r);
  if (!*B.active) return;
  float *Y = sm, *const raw = sm + 2 * kSY, *const out_s = raw + kSRaw;  // Y: two buffers, this iteration's
  const int tid = threadIdx.x, warp = tid >> 5, nout = a.ntime_out;
  const YRows rows(B, r, a.ntime_dd);
  const int org = a.wmax / 2 - (ANCHOR ? kSSpan : 0);
  const bool vec = rows.vec && org % 4 == 0;
  float mx[kSW], part[kSW / 2][4];
#pragma unroll
  for (int b = 0; b < kSW; ++b) mx[b] = -INFINITY;
#pragma unroll
  for (int b = 0; b < kSW / 2; ++b)
#pragma unroll
    for (int i = 0; i < 4; ++i) part[b][i] = 0.f;
  const uint32_t raw0 = (uint32_t)__cvta_generic_to_shared(raw);
  const int sl0 = slot_word(2 * tid), sl1 = slot_word(2 * tid + 1);
  auto load = [&](int cs) {  // this thread's 8 columns of the rows that enter with the outputs from cs
    if (cs < nout) {
      const int w0 = cs + org + kSSpan, c0 = w0 + kSO * tid;
      const float *src[3] = {rows.a, rows.b, rows.c};
      if (vec && w0 >= 0 && w0 + kSC <= rows.n) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          cp_async16(raw0 + 4u * (k * kSC + sl0), src[k] + c0);
          cp_async16(raw0 + 4u * (k * kSC + sl1), src[k] + c0 + 4);
        }
      } else {
        for (int i = 0; i < kSO; ++i) {
          const int col = min(max(c0 + i, 0), rows.n - 1), w = (i < 4 ? sl0 : sl1) + (i & 3);
          for (int k = 0; k < 3; ++k) cp_async4(raw0 + 4u * (k * kSC + w), src[k] + col);
        }
      }
    }
    cp_async_commit();
  };
  load(0);
  if (tid < kSSpan) Y[kSPitch * (tid / 8) + tid % 8] = rows.at(org + tid);
  const int pb = 3 * (tid >> 6), pq = tid & 63;  // partials: widths pb .. pb + 2, slot pq of each chunk
#pragma unroll 1
  for (int cs = 0, buf = 0; cs < nout; cs += kSC, buf ^= 1) {
    Y = sm + buf * kSY;
    cp_async_wait<0>();  // the rows this thread copied
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float *x = raw + (h ? sl1 : sl0);
      const float4 u = *reinterpret_cast<const float4 *>(x), v = *reinterpret_cast<const float4 *>(x + kSC),
                   w = *reinterpret_cast<const float4 *>(x + 2 * kSC);
      *reinterpret_cast<float4 *>(Y + kSPitch * (kSSpan / 8 + tid) + 4 * h) =
          make_float4(YRows::y(u.x, v.x, w.x), YRows::y(u.y, v.y, w.y), YRows::y(u.z, v.z, w.z),
                      YRows::y(u.w, v.w, w.w));
    }
    load(cs + kSC);
    __syncthreads();
    float win[kSWin];
#pragma unroll
    for (int q = 0; q < kSWin / 4; ++q) {
      const float4 v = *reinterpret_cast<const float4 *>(Y + kSPitch * (tid + q / 2) + 4 * (q & 1));
      win[4 * q] = v.x;
      win[4 * q + 1] = v.y;
      win[4 * q + 2] = v.z;
      win[4 * q + 3] = v.w;
    }
    if (tid < kSSpan / 4) {  // the next iteration's first 64 values
      const int o = kSPitch * (tid / 2) + 4 * (tid & 1);
      *reinterpret_cast<float4 *>(sm + (buf ^ 1) * kSY + o) = *reinterpret_cast<const float4 *>(Y + o + kSPitch * (kSC / 8));
    }
    const bool valid = cs + kSO * tid < nout;  // nout % 8 == 0
    float acc[kSO];
    auto emit = [&](int b) {
      if (valid) {
        store8(B.boxes + ((size_t)(b - a.w0) * B.h + r) * nout + cs + kSO * tid, acc);
#pragma unroll
        for (int i = 0; i < kSO; i += 2) mx[b] = max3(mx[b], acc[i], acc[i + 1]);
      }
      *reinterpret_cast<float4 *>(out_s + b * kSC + sl0) = make_float4(acc[0], acc[1], acc[2], acc[3]);
      *reinterpret_cast<float4 *>(out_s + b * kSC + sl1) = make_float4(acc[4], acc[5], acc[6], acc[7]);
    };
    if (b0 <= 5 && 5 < b1) { firS_width<32, ANCHOR>(win, taps.t + small_tap(5), acc); emit(5); }
    if (b0 <= 4 && 4 < b1) { firS_width<16, ANCHOR>(win, taps.t + small_tap(4), acc); emit(4); }
    if (b0 <= 3 && 3 < b1) { firS_width<8, ANCHOR>(win, taps.t + small_tap(3), acc); emit(3); }
    if (b0 <= 2 && 2 < b1) { firS_width<4, ANCHOR>(win, taps.t + small_tap(2), acc); emit(2); }
    if (b0 <= 1 && 1 < b1) { firS_width<2, ANCHOR>(win, taps.t + small_tap(1), acc); emit(1); }
    if (b0 <= 0 && 0 < b1) { firS_width<1, ANCHOR>(win, taps.t + small_tap(0), acc); emit(0); }
    __syncthreads();
    const int nm = min(kSWarps, (nout - cs) / 256);  // whole chunks: their columns count for the row mean
#pragma unroll
    for (int j = 0; j < kSW / 2; ++j)
      if (b0 <= pb + j && pb + j < b1) {
#pragma unroll
        for (int m = 0; m < kSWarps; ++m)
          if (m < nm) {
            const float4 v = *reinterpret_cast<const float4 *>(out_s + (pb + j) * kSC + slot_word(64 * m + pq));
            part[j][0] = __fadd_rn(part[j][0], v.x);
            part[j][1] = __fadd_rn(part[j][1], v.y);
            part[j][2] = __fadd_rn(part[j][2], v.z);
            part[j][3] = __fadd_rn(part[j][3], v.w);
          }
      }
  }
  // row totals: partials and the warps' maxima through shared memory, a warp a width
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSW / 2; ++j)
    *reinterpret_cast<float4 *>(out_s + (pb + j) * 256 + 4 * pq) =
        make_float4(part[j][0], part[j][1], part[j][2], part[j][3]);
#pragma unroll
  for (int b = 0; b < kSW; ++b) sm[b * kST + tid] = mx[b];
  __syncthreads();
  const int nwcol = 256 * (nout / 256);
  for (int b = b0 + warp; b < b1; b += kSWarps) {
    float m = -INFINITY;
#pragma unroll
    for (int i = 0; i < kSWarps; ++i) m = fmaxf(m, sm[b * kST + 32 * i + (tid & 31)]);
    row_finish(B, b, r, out_s + b * 256, m, nwcol);
  }
}

// k_firL: one width of any size, a block of four warps per (row, width), the
// widest width's blocks first so that the short ones fill the last wave.  An
// iteration makes 2048 outputs, thread t outputs 16t .. 16t + 15 with a
// sliding window of 16 y values in registers: four taps are 64 multiply-adds,
// one 16-byte read of the y values that enter the window and one of the taps
// (both a group of four ahead).  The iteration's y values and the span before
// them sit in shared memory as rows of 16 at a pitch of 20 words: window
// element n of thread t is word 20 (t + n / 16) + n % 16, a constant offset
// from one base, conflict-free at a lane stride of one row.  The outputs also
// go to shared memory (16-byte slots permuted, conflict-free), where thread i
// adds those of columns 2i and 2i + 1 (mod 256) to its row-mean partials in
// order; three block barriers an iteration.  Bound by multiply-add issue: 79 %
// of the cycles issue, the rest are mostly dispatch stalls of warps that are
// ready.  2499 rows x 65536 x widths 64, 128, 256: 5.09 ms = 1.47e11 multiply-
// adds at 72 % of the FP32 rate (with width 1-32's k_firS 6.14 ms; one kernel
// for all nine widths with a barrier pair per width and 2048 outputs 7.50 ms).
// A warp a row walks too long where rows are few: 394 rows x 10016, 190 us
// against 143.  Six blocks an SM (85 registers) 5.09 ms, five 5.17.
constexpr int kLO = 16;          // outputs per thread
constexpr int kLT = 128;         // threads per block
constexpr int kLC = kLT * kLO;   // outputs per iteration
constexpr int kLPitch = 20;      // words from one row of 16 y values to the next
__host__ __device__ constexpr int firL_taps(int smw) { return (2 * smw + 1 + 15) / 16 * 16 + 8; }
// rows of 16: the threads', the taps' blocks, one block read ahead
__host__ __device__ constexpr int firL_rows(int smw) { return kLT + 2 + (2 * smw + 1) / 16; }

__device__ __forceinline__ int firL_word(int x) { return kLPitch * (x / 16) + x % 16; }

__global__ void __launch_bounds__(kLT, 6) k_firL(SmoothArgs a, int bend) {
  extern __shared__ __align__(16) float sm[];
  const int b = bend - 1 - blockIdx.y, smw = a.wmin << b, ntap = 2 * smw + 1, tid = threadIdx.x;
  int r;
  const SmoothBeam &B = row_beam(a, blockIdx.x, &r);
  if (!*B.active) return;
  float *const out_s = sm, *const taps = sm + kLC, *const Y = taps + firL_taps(smw);
  for (int i = tid; i < firL_taps(smw); i += kLT) taps[i] = i < a.tap_n[b] ? a.taps[a.tap_off[b] + i] : 0.f;
  const YRows rows(B, r, a.ntime_dd);
  const int H = 2 * smw, org = a.wmax / 2 - (a.anchor ? H : 0), nout = a.ntime_out;
  const bool vec = rows.vec && (org + H) % 4 == 0 && H % 4 == 0;
  float *const dst = B.boxes + ((size_t)(b - a.w0) * B.h + r) * nout;
  float part0 = 0.f, part1 = 0.f, mx = -INFINITY;
  for (int x = tid; x < H; x += kLT) Y[firL_word(x)] = rows.at(org + x);
  const float *base = Y + kLPitch * tid;
  const int nblk = ntap / 16, tail = ntap % 16, key = (tid >> 1) & 3;
  const float *pcol;  // column 2 tid of the iteration's first 256 in out_s
  {
    const int t = tid / 8, q = (tid % 8) / 2;
    pcol = out_s + 16 * t + 4 * (q ^ ((t >> 1) & 3)) + 2 * (tid & 1);
  }
#pragma unroll 1
  for (int cs = 0; cs < nout; cs += kLC) {
    const int c0 = cs + org + H;  // columns c0 .. c0 + 2047 enter as y values H .. H + 2047
    if (vec && c0 >= 0 && c0 + kLC <= rows.n) {
      float4 x[4], y[4], z[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = c0 + 4 * tid + 4 * kLT * k;
        x[k] = *reinterpret_cast<const float4 *>(rows.a + c);
        y[k] = *reinterpret_cast<const float4 *>(rows.b + c);
        z[k] = *reinterpret_cast<const float4 *>(rows.c + c);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        *reinterpret_cast<float4 *>(Y + firL_word(H + 4 * tid + 4 * kLT * k)) =
            make_float4(YRows::y(x[k].x, y[k].x, z[k].x), YRows::y(x[k].y, y[k].y, z[k].y),
                        YRows::y(x[k].z, y[k].z, z[k].z), YRows::y(x[k].w, y[k].w, z[k].w));
    } else {
#pragma unroll 4
      for (int k = 0; k < kLC / kLT; ++k) Y[firL_word(H + tid + kLT * k)] = rows.at(c0 + tid + kLT * k);
    }
    __syncthreads();
    // win[(i + kk) % 16] holds y at window element 16 kq + kk + i of output i; slot kk is refilled
    // after step kk of block kq
    float acc[kLO], win[kLO];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 v = *reinterpret_cast<const float4 *>(base + 4 * q);
      win[4 * q] = v.x, win[4 * q + 1] = v.y, win[4 * q + 2] = v.z, win[4 * q + 3] = v.w;
    }
#pragma unroll
    for (int i = 0; i < kLO; ++i) acc[i] = 0.f;
    float4 cn = *reinterpret_cast<const float4 *>(taps), yn = *reinterpret_cast<const float4 *>(base + kLPitch);
    const float *yp = base + kLPitch, *tp = taps;
#pragma unroll 1
    for (int kq = 0; kq < nblk; ++kq, yp += kLPitch, tp += 16) {
#pragma unroll
      for (int k4 = 0; k4 < 16; k4 += 4) {
        const float cf[4] = {cn.x, cn.y, cn.z, cn.w}, yv[4] = {yn.x, yn.y, yn.z, yn.w};
        cn = *reinterpret_cast<const float4 *>(tp + k4 + 4);
        yn = *reinterpret_cast<const float4 *>(yp + (k4 == 12 ? kLPitch : k4 + 4));
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
          for (int i = 0; i < kLO; ++i) acc[i] = __fmaf_rn(cf[jj], win[(i + k4 + jj) % 16], acc[i]);
          win[k4 + jj] = yv[jj];
        }
      }
    }
#pragma unroll
    for (int k4 = 0; k4 < 16; k4 += 4) {  // the last `tail` taps (no zero taps are issued)
      if (k4 >= tail) break;
      const float cf[4] = {cn.x, cn.y, cn.z, cn.w}, yv[4] = {yn.x, yn.y, yn.z, yn.w};
      if (k4 + 4 < tail) {
        cn = *reinterpret_cast<const float4 *>(tp + k4 + 4);
        yn = *reinterpret_cast<const float4 *>(yp + k4 + 4);
      }
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        if (k4 + jj >= tail) break;
#pragma unroll
        for (int i = 0; i < kLO; ++i) acc[i] = __fmaf_rn(cf[jj], win[(i + k4 + jj) % 16], acc[i]);
        win[k4 + jj] = yv[jj];
      }
    }
    if (cs + kLO * tid < nout) {  // nout % 16 == 0
      store8(dst + cs + kLO * tid, acc);
      store8(dst + cs + kLO * tid + 8, acc + 8);
#pragma unroll
      for (int i = 0; i < kLO; i += 2) mx = max3(mx, acc[i], acc[i + 1]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<float4 *>(out_s + kLO * tid + 4 * (q ^ key)) =
          make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
    __syncthreads();
    const int nm = min(kLC / 256, (nout - cs) / 256);  // whole 256s: their columns count for the row mean
#pragma unroll
    for (int m = 0; m < kLC / 256; ++m)
      if (m < nm) {
        const float2 v = *reinterpret_cast<const float2 *>(pcol + 256 * m);
        part0 = __fadd_rn(part0, v.x);
        part1 = __fadd_rn(part1, v.y);
      }
    if (cs + kLC < nout) {  // the last H y values move to the front, at most 2048 between barriers
      for (int x0 = 0; x0 < H; x0 += kLC) {
        const int n = min(kLC, H - x0);
        if (H % 4 == 0) {
          for (int x = x0 + 4 * tid; x < x0 + n; x += 4 * kLT)
            *reinterpret_cast<float4 *>(Y + firL_word(x)) = *reinterpret_cast<const float4 *>(Y + firL_word(x + kLC));
        } else {
          for (int x = x0 + tid; x < x0 + n; x += kLT) Y[firL_word(x)] = Y[firL_word(x + kLC)];
        }
        __syncthreads();
      }
    }
  }
  __syncthreads();
  for (int o = 16; o > 0; o /= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  out_s[2 * tid] = part0;
  out_s[2 * tid + 1] = part1;
  if ((tid & 31) == 0) out_s[256 + (tid >> 5)] = mx;
  __syncthreads();
  if (tid < 32) row_finish(B, b, r, out_s, out_s[256 + (tid & 3)], 256 * (nout / 256));
}

constexpr int kFin = 256;

// Host loop of calculate_stddev (normalization.cu:138-142): sequential over
// rows, / height.  Block = (beam, width of the launch).
__global__ void __launch_bounds__(kFin) k_mean_finish(SmoothArgs a) {
  const SmoothBeam &B = a.beams[blockIdx.x];
  const int j = blockIdx.y;
  if (!*B.active) return;
  const int b = a.w0 + j, h = B.h;
  const float s = block_seq_sum(B.rowmean + (size_t)b * h, h);
  if (threadIdx.x == 0) B.stats[b * 4 + 0] = __fdiv_rn(s, (float)h);
}

// The host loop over rows for one (beam, width b): variance -> std and the
// normalisation constants.  NORM0: the gate statistics of the normalised
// width-0 plane.  By a whole block.
template <bool NORM0, bool VAR>
__device__ __forceinline__ void stat_finish(const SmoothArgs &a, const SmoothBeam &B, int b) {
  float m = block_seq_sum(B.rowvar + (size_t)b * B.h, B.h);
  if (threadIdx.x != 0) return;
  m = __fdiv_rn(m, (float)B.h);
  if (NORM0) {
    if (!VAR) {
      B.gate[0] = m;
    } else {
      const float sig = __fsqrt_rn(m);
      B.gate[1] = sig;
      B.gate[2] = __fmul_rn(a.snr, sig);
      B.gate[3] = (a.nogate || (sig < 5 && (double)sig > 0.1)) ? 1.f : 0.f;  // definitions.h:66,71-72
    }
  } else {
    const float sd = __fsqrt_rn(m), mu = B.stats[b * 4 + 0];
    B.stats[b * 4 + 1] = sd;
    B.stats[b * 4 + 2] = -1.0f * mu;
    B.stats[b * 4 + 3] = __fdiv_rn(1.0f, sd);
  }
}

// stat_finish by itself.  Block = (beam, width of the launch).
template <bool NORM0, bool VAR>
__global__ void __launch_bounds__(kFin) k_stat_finish(SmoothArgs a) {
  const SmoothBeam &B = a.beams[blockIdx.x];
  if (*B.active) stat_finish<NORM0, VAR>(a, B, NORM0 ? 0 : a.w0 + (int)blockIdx.y);
}

// computeRowVariances over one row of one width plane.  NORM0: the
// normalised width-0 plane (find_peaks' sigma, peaks.cu:171-178), which
// needs width 0 in the launch (w0 == 0).  FIN: the last row's block of a (beam,
// width) runs stat_finish.  Bound by the memory: 2499 rows x 65,536 x 9 widths 840 us
// (6.9 TB/s).
template <bool NORM0, bool VAR, bool FIN>
__global__ void __launch_bounds__(kT, !NORM0 && !FIN ? 8 : 6) k_row_stat(SmoothArgs a) {
  __shared__ float p_s[kT];
  int r;
  const SmoothBeam &B = row_beam(a, blockIdx.x, &r);
  if (!*B.active) return;
  const int j = NORM0 ? 0 : blockIdx.y, b = a.w0 + j, h = B.h, tid = threadIdx.x;
  const float *x = B.boxes + ((size_t)j * h + r) * a.ntime_out;
  const int nwcol = 256 * (a.ntime_out / 256);
  const float *st = B.stats + b * 4;
  const float mean = NORM0 ? B.gate[0] : st[0];
  const float norm[4] = {0.f, NORM0 ? st[1] : 0.f, NORM0 ? st[2] : 0.f, NORM0 ? st[3] : 0.f};  // normv's, read once
  float s = 0.f;
  auto add = [&](float v) {
    if (NORM0) v = normv(v, norm);
    if (VAR) {
      const float d = __fsub_rn(v, mean);
      s = __fmaf_rn(d, d, s);
    } else {
      s = __fadd_rn(s, v);
    }
  };
  // sixteen loads in flight per thread, then the sums in column order
  constexpr int kB = 16;
  int col = tid;
  for (; col + (kB - 1) * kT < nwcol; col += kB * kT) {
    float v[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) v[u] = x[col + u * kT];
#pragma unroll
    for (int u = 0; u < kB; ++u) add(v[u]);
  }
  for (; col < nwcol; col += kT) add(x[col]);
  p_s[tid] = s;
  __syncthreads();
  if (tid < 32) {
    const float tot = block256_tree(p_s);
    if (tid == 0) B.rowvar[(size_t)b * h + r] = __fdiv_rn(tot, (float)nwcol);
  }
  if (FIN && last_block(B.done + b, (unsigned)h)) stat_finish<NORM0, VAR>(a, B, b);
}

// A pass and the loop over its rows: one launch where the rows are few (512
// channels x 16,384 samples, 3300 row blocks: 39 us for the two launches, 37 us for one), two
// where waiting for the count of rows done holds blocks back more than a launch
// costs (16 beams x 8192 samples: 508 + 10 us, 540 us).
template <bool NORM0, bool VAR>
unsigned row_stat(const SmoothArgs &a, int nw, cudaStream_t s) {
  if ((long)a.nrows * nw <= 4096) {
    k_row_stat<NORM0, VAR, true><<<dim3(a.nrows, nw), kT, 0, s>>>(a);
    return 1;
  }
  k_row_stat<NORM0, VAR, false><<<dim3(a.nrows, nw), kT, 0, s>>>(a);
  k_stat_finish<NORM0, VAR><<<dim3(a.nbeam, nw), kFin, 0, s>>>(a);
  return 2;
}

// Unnormalised planes (hella_smooth(ctx, 0)): stats zero for the widths.
__global__ void k_stat_zero(SmoothArgs a) {
  const SmoothBeam &B = a.beams[blockIdx.x];
  const int j = threadIdx.x;
  if (j >= a.nw || !*B.active) return;
  for (int q = 0; q < 4; ++q) B.stats[(a.w0 + j) * 4 + q] = 0.f;
}

__global__ void __launch_bounds__(kT) k_count(SmoothArgs a) {
  __shared__ int c_s[kT / 32];
  int r;
  const SmoothBeam &B = row_beam(a, blockIdx.x, &r);
  const int j = blockIdx.y, b = a.w0 + j, h = B.h, tid = threadIdx.x;
  const size_t row = (size_t)b * h + r;
  const float st[4] = {0.f, B.stats[b * 4 + 1], B.stats[b * 4 + 2], B.stats[b * 4 + 3]};  // normv's, read once
  const float thr = B.gate[2];
  // normalisation is monotonic, so the row maximum decides the whole row
  if (!*B.active || B.gate[3] == 0.f || !(normv(B.rowmax[row], st) > thr)) {
    if (tid == 0) B.counts[row] = 0;
    return;
  }
  const float *x = B.boxes + ((size_t)j * h + r) * a.ntime_out;
  int n = 0;
  constexpr int kB = 16;  // loads in flight per thread
  int col = tid;
  for (; col + (kB - 1) * kT < a.ntime_out; col += kB * kT) {
    float v[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u) v[u] = x[col + u * kT];
#pragma unroll
    for (int u = 0; u < kB; ++u) n += normv(v[u], st) > thr;
  }
  for (; col < a.ntime_out; col += kT) n += normv(x[col], st) > thr;
  for (int off = 16; off > 0; off /= 2) n += __shfl_xor_sync(0xffffffffu, n, off);
  if ((tid & 31) == 0) c_s[tid >> 5] = n;
  __syncthreads();
  if (tid == 0) {
    int t = 0;
    for (int i = 0; i < kT / 32; ++i) t += c_s[i];
    B.counts[row] = t;
  }
}

// Per beam: exclusive scan of the row counts of the launch's widths in
// (width, row) order, after the candidates of earlier widths; the beam's
// total is capped at its cap.  1024 rows at a time, neighbouring ones in
// neighbouring threads, warp sums by shuffles.
__global__ void __launch_bounds__(1024) k_scan(SmoothArgs a) {
  __shared__ int w_s[32];
  const SmoothBeam &B = a.beams[blockIdx.x];
  if (!*B.active) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nrows = a.nw * B.h;
  const int *counts = B.counts + (size_t)a.w0 * B.h;
  int *offsets = B.offsets + (size_t)a.w0 * B.h;
  int base = B.total[0];
  int next = tid < nrows ? counts[tid] : 0;
  for (int i0 = 0; i0 < nrows; i0 += 1024) {
    const int i = i0 + tid, c = next;
    next = i + 1024 < nrows ? counts[i + 1024] : 0;
    int v = c;
    for (int off = 1; off < 32; off *= 2) {
      const int u = __shfl_up_sync(0xffffffffu, v, off);
      if (lane >= off) v += u;
    }
    __syncthreads();  // the sums of the round before have been read
    if (lane == 31) w_s[warp] = v;
    __syncthreads();
    int t = w_s[lane];
    for (int off = 1; off < 32; off *= 2) {
      const int u = __shfl_up_sync(0xffffffffu, t, off);
      if (lane >= off) t += u;
    }
    const int before = __shfl_sync(0xffffffffu, t, (warp + 31) & 31);
    if (i < nrows) offsets[i] = base + v - c + (warp ? before : 0);
    base += __shfl_sync(0xffffffffu, t, 31);
  }
  if (tid == 0) B.total[0] = min(base, B.cap);
}

// Ordered compaction of one row's candidates, kWCols columns a round: a warp
// takes a contiguous eighth of them, kWN values a thread loaded at once, the warps'
// hits are published once a round, and a hit is written at the row's offset + the
// hits of earlier rounds, warps, 32-column groups and lanes.  Bound by the loads'
// latency on the few rows that have hits (16 or 32 values a thread leave too few
// blocks an SM for the many rows that have none): 512 channels x 16,384 samples 15 us,
// 47 us with 1024 columns and two barriers a round.
constexpr int kWN = 8, kWCols = kWN * kT;
__global__ void __launch_bounds__(kT, 8) k_write(SmoothArgs a) {
  __shared__ int w_s[2][kT / 32];
  int r;
  const SmoothBeam &B = row_beam(a, blockIdx.x, &r);
  const int j = blockIdx.y, b = a.w0 + j, h = B.h, tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const size_t row = (size_t)b * h + r;
  if (!*B.active || B.counts[row] == 0 || B.offsets[row] >= B.cap) return;
  const float st[4] = {0.f, B.stats[b * 4 + 1], B.stats[b * 4 + 2], B.stats[b * 4 + 3]};  // normv's, read once
  const float thr = B.gate[2];
  const float *x = B.boxes + ((size_t)j * h + r) * a.ntime_out;
  int base = B.offsets[row];  // the same in every thread
  for (int c0 = 0, k = 0; c0 < a.ntime_out && base < B.cap; c0 += kWCols, k ^= 1) {
    const int w0 = c0 + warp * (kWCols / (kT / 32));
    float v[kWN];
#pragma unroll
    for (int m = 0; m < kWN; ++m) v[m] = w0 + m * 32 + lane < a.ntime_out ? x[w0 + m * 32 + lane] : 0.f;
    int n = 0;
#pragma unroll
    for (int m = 0; m < kWN; ++m) {
      v[m] = normv(v[m], st);
      n += __popc(__ballot_sync(0xffffffffu, w0 + m * 32 + lane < a.ntime_out && v[m] > thr));
    }
    if (lane == 0) w_s[k][warp] = n;
    __syncthreads();  // the other buffer's readers passed the barrier before
    int pos0 = base, round = 0;
#pragma unroll
    for (int i = 0; i < kT / 32; ++i) {
      if (i < warp) pos0 += w_s[k][i];
      round += w_s[k][i];
    }
    if (n)
#pragma unroll
      for (int m = 0; m < kWN; ++m) {
        const int col = w0 + m * 32 + lane;
        const unsigned bal = __ballot_sync(0xffffffffu, col < a.ntime_out && v[m] > thr);
        const int pos = pos0 + __popc(bal & ((1u << lane) - 1u));
        if (((bal >> lane) & 1u) && pos < B.cap) {
          B.cand_i[pos] = make_int4(B.beam_id, r + 1, b, col);
          B.cand_v[pos] = v[m];
        }
        pos0 += __popc(bal);
      }
    base += round;
  }
}

// Normalised copy of beam 0's planes of the launch's widths (inspection).
__global__ void k_normalise_copy(SmoothArgs a, float *dst) {
  const SmoothBeam &B = a.beams[0];
  const size_t plane = (size_t)B.h * a.ntime_out;
  const size_t n = plane * a.nw;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    dst[i] = normv(B.boxes[i], B.stats + (a.w0 + i / plane) * 4);
}

}  // namespace

cudaError_t smooth_planes(const SmoothArgs &a, cudaStream_t s) {
  if (a.nrows <= 0 || a.nw <= 0) return cudaSuccess;
  if (a.ntime_out % kLO != 0) return cudaErrorInvalidValue;
  const int bend = a.w0 + a.nw;
  // widths 1 .. 32 of a list that starts at 1 go through k_firS, which reads and stages a row once
  // for all of them; every other width through k_firL
  const int bs = a.wmin == 1 ? std::max(a.w0, std::min(bend, kSW)) : a.w0;
  if (bs < bend) {
    const int smw = a.wmin << (bend - 1);
    const size_t smem = sizeof(float) * ((size_t)kLC + firL_taps(smw) + (size_t)firL_rows(smw) * kLPitch);
    cudaError_t e = cudaFuncSetAttribute(k_firL, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost);
    if (e != cudaSuccess) return e;
    k_firL<<<dim3(a.nrows, bend - bs), kLT, smem, s>>>(a, bend);
    count_launches(1);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (a.w0 < bs) {
    SmallTaps t{};
    for (int b = 0, off = 0; b < std::min(a.nbox, kSW); ++b) {  // padded to multiples of 16 in taps_host
      const int n = 2 * (1 << b) + 1;
      std::copy(a.taps_host + off, a.taps_host + off + n, t.t + small_tap(b));
      off += (n + 15) / 16 * 16;
    }
    auto kern = a.anchor ? k_firS<1> : k_firS<0>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSSmem);
    if (e != cudaSuccess) return e;
    kern<<<a.nrows, kST, kSSmem, s>>>(a, t, a.w0, bs);
    count_launches(1);
    return cudaGetLastError();
  }
  return cudaSuccess;
}

cudaError_t smooth_stats(const SmoothArgs &a, cudaStream_t s, int scale) {
  if (a.nrows <= 0 || a.nw <= 0) return cudaSuccess;
  unsigned n = 0;
  if (scale) {
    k_mean_finish<<<dim3(a.nbeam, a.nw), kFin, 0, s>>>(a);
    n += 1 + row_stat<false, true>(a, a.nw, s);
  } else {
    k_stat_zero<<<a.nbeam, 32, 0, s>>>(a);
    n += 1;
  }
  if (a.w0 == 0) {  // the gate statistics of the normalised width-0 plane
    n += row_stat<true, false>(a, 1, s);
    n += row_stat<true, true>(a, 1, s);
  }
  count_launches(n);
  return cudaGetLastError();
}

cudaError_t find_peaks(const SmoothArgs &a, cudaStream_t s) {
  if (a.nrows <= 0 || a.nw <= 0) return cudaSuccess;
  k_count<<<dim3(a.nrows, a.nw), kT, 0, s>>>(a);
  k_scan<<<a.nbeam, 1024, 0, s>>>(a);
  k_write<<<dim3(a.nrows, a.nw), kT, 0, s>>>(a);
  count_launches(3);
  return cudaGetLastError();
}

cudaError_t normalise_copy(const SmoothArgs &a, float *dst, cudaStream_t s) {
  k_normalise_copy<<<1024, 256, 0, s>>>(a, dst);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace hg
