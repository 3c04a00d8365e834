// pairs.cu -- add modes 5 and 6 of the dedispersion: rows of channel
// groups, pairs (g = 2) or quads (g = 4) (hg_internal.h).
//
// Same exact integer sums as k_dedisp (out[d][t] = sum over active channels
// c of x[c][t + delay(c, d)], the operation casm-hella obtains from
// dedisp_execute_adv, src/hella/src/dedisperse.cpp:17-48), computed in two
// launches per window:
//
// k_pair_build: one block per (group, 4096 window positions for pairs, 2048
//   for quads).  The group's channels' packed words of the chunk (for channel
//   i widened by the group's range of relative delays r_i) are bulk-copied
//   from the ring into shared memory as they are, then one warp per row
//   writes every row of the group from them: a packed word holds bytes p,
//   p + 256, p + 512 and p + 768 of a channel, so one read of each channel
//   gives two words of row(r)[p] = x[c0][p] + sum_i x[c_i][p + r_i], that of
//   p (bytes 0 and 2) and that of p + 256 (bytes 1 and 3); the next row's
//   metadata is loaded while a row is written.  Reads are the ring once per
//   group; writes the rows, coalesced, with streaming stores.  A row keeps,
//   tile by tile, only the words its trials read where those span less than
//   a 1024-sample tile.  Bound by the row writes: quads of 2048 channels, DM
//   0-2000 (14.9 GB) 2.49 ms = 6.0 TB/s, 2.75 ms with the samples split into
//   16-bit lanes as they were staged (four shared reads a word written, 25
//   instructions a word against 19); eight beams of 1024 channels 3.28
//   against 3.91 ms.  Walking positions and keeping the sums over the first
//   channels from row to row costs more: most blocks of 256 positions are
//   cut by a row's tile windows (4.88 ms).
//
// k_pair_sum: the persistent staging pipeline of k_dedisp (work item =
//   16-trial tile x 1024 output samples, stages issued warp by warp with
//   cp.async.bulk onto full/empty mbarriers, every wait bounded) over stage
//   records instead of channels.  A stage stages the windows of the rows
//   its groups use (lane i copies row i) and the record's trial offsets;
//   thread j then reads, per group and trial, the words j and j + 256 of
//   the trial's window: four output samples (j, j+256, j+512, j+768) in two
//   SWAR registers of 16-bit lanes, two groups per three-input add.  The
//   lanes are widened into 32-bit totals, held in tensor memory, every
//   pair_lanecap(g) groups.
//
// Per group and trial the inner loop is two shared loads and one add for
// 4g channel-samples, against two loads, four byte permutes and two adds
// per eight in k_dedisp; shared-memory traffic is 2/g bytes per
// channel-sample, so the sums are bound by shared-memory bandwidth (reads
// and staged rows at 80 to 93 % of its cycles), quads by the rows' latency as
// well (with nothing staged 5.8 of 7.4 ms), and the build by its row writes
// (g = 4: about three times the rows of g = 2).
#include "hg_internal.h"
#include "hg_ptx.h"

#include <algorithm>
#include <array>
#include <cstring>

namespace hg {
namespace {

constexpr int S = kPackS;
constexpr int kTileSamples = 4 * S;
// window positions per build block: 4096 for pairs, 2048 for quads (whose
// four channel windows would otherwise leave three blocks per SM)
__host__ __device__ constexpr int build_chunk(int g) { return g <= 2 ? 4096 : 2048; }
constexpr int kTmemAt = 440;              // the block's tensor memory address, in the first unit's header
constexpr int kBarHdr = 448;              // full[4] | empty[4] | per-warp staging cursors
constexpr int kBuildMost = 200 * 1024;    // bytes of a build block's chunk and ranges, without the windows' alignment
constexpr int kMaxBuf = 4;

// Shared memory of one unit of the sum (half a block): barriers and cursors, staging buffers.
__host__ __device__ constexpr size_t unit_smem(int bufbytes, int nbuf) { return kBarHdr + (size_t)nbuf * bufbytes; }

// Words of a copy that only outputs past the last one would read: the last time tile's `rem`
// outputs need the words j < rem alone when they are at most 512 (word j + 256 holds outputs
// j + 256 and j + 768).
__host__ __device__ constexpr int words_cut(int rem) { return rem < 2 * S ? 2 * S - (rem + 3) / 4 * 4 : 0; }

__host__ __device__ constexpr int stage_hdr_bytes(int cc) { return 16 + cc * kPairDPT * 4; }

// Window positions a row spans from its first position: all its words for
// a single run, (ntt - 1) tiles of 1024 and one stride for tiled rows.
__device__ __forceinline__ long row_positions(const DedispArgs &a, int r) {
  const int stride = a.pair_rtile[r];
  return stride == kTileSamples ? (long)a.pair_rwords[r] : (long)(a.ntt - 1) * kTileSamples + stride;
}

// A row's metadata, all of it loaded together (one wait per row).
struct BuildRow {
  int w, z1, z2, z3, stride, words;
  long long off;
};

__device__ __forceinline__ BuildRow build_row(const DedispArgs &a, int r, bool quad) {
  const int4 in = a.pair_rinfo[r];
  const int4 in2 = quad ? a.pair_rinfo2[r] : make_int4(-1, -1, 0, 0);
  return BuildRow{in.w, in.z, in2.z, in2.w, a.pair_rtile[r], a.pair_rwords[r], a.pair_roff[r]};
}

// Words of a staged channel window: kBuildCH positions and the channel's range of relative delays,
// with up to 3 words before (copies start 16-byte aligned) and rounded to whole 16 bytes.
__host__ __device__ constexpr int build_window(int ch, int span) { return (ch + span + 6) / 4 * 4; }

// Where channel i's window starts in shared memory (i = g: the words of all g).  Channel 0 is what the
// delays are relative to and has no range of its own.
__host__ __device__ constexpr int build_at(int i, int ch, int span) {
  return i ? build_window(ch, 0) + (i - 1) * build_window(ch, span) : 0;
}

// One run of up to 256 packed words of a row: output word i takes bytes 0 and 2 of the packed
// words x[c_i][i], output word i + 256 (i < n2) bytes 1 and 3, for lo <= i < hi.  NC: the group's
// channels.  With both, the odd bytes are split off and added; the sum of the whole words, in which
// they sit 8 bits up, less that leaves the even bytes' sums.
template <int NC, bool BOTH, bool FULL>
__device__ __forceinline__ void build_run(uint32_t *dst, const uint32_t *sm, const int (&x)[kPairGMax], int lo, int hi,
                                          int n2) {
  constexpr int U = 2;  // words of each channel in flight per lane
#pragma unroll(FULL ? 4 : 1)
  for (int i0 = (FULL ? 0 : lo) + (threadIdx.x & 31); i0 < (FULL ? 256 : hi); i0 += 32 * U) {
    uint32_t w[U][NC];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || FULL || i0 + 32 * u < hi)
#pragma unroll
        for (int c = 0; c < NC; ++c) w[u][c] = sm[x[c] + i0 + 32 * u];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + 32 * u;
      const bool in = u == 0 || FULL || i < hi;
      // rows are read back by other blocks much later: streaming stores
      if (BOTH) {
        uint32_t t = w[u][0], o = __byte_perm(w[u][0], 0u, 0x4341);
#pragma unroll
        for (int c = 1; c < NC; ++c) t += w[u][c], o += __byte_perm(w[u][c], 0u, 0x4341);
        if (in) __stcs(dst + i, t - 256u * o);
        if (FULL || (in && i < n2)) __stcs(dst + 256 + i, o);
      } else {
        uint32_t e = w[u][0] & 0x00ff00ffu;
#pragma unroll
        for (int c = 1; c < NC; ++c) e += w[u][c] & 0x00ff00ffu;
        if (in) __stcs(dst + i, e);
      }
    }
  }
}

template <int G>
__global__ void __launch_bounds__(256, G == 4 ? 4 : 5) k_pair_build(DedispArgs a) {
  extern __shared__ __align__(128) uint32_t sm[];
  __shared__ __align__(8) unsigned long long bar_s;
  __shared__ int off_s[kPairGMax];
  constexpr int kBuildCH = build_chunk(G);
  const int k = blockIdx.y, z = blockIdx.z;  // group, beam of the launch
  const long P0 = (long)blockIdx.x * kBuildCH;
  const DedispBeam bm = a.beams ? a.beams[z] : a.one;
  const int r0 = a.pair_prow[k];
  const int r1 = a.pair_rend ? a.pair_rend[(size_t)z * a.pair_npair + k] : a.pair_prow[k + 1];
  int any = 0;  // does a row of the group cover a position of this chunk?
  for (int r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
    const int w = a.pair_rinfo[r].w;
    any |= P0 < (long)w + row_positions(a, r) && P0 + kBuildCH > (long)w;
  }
  if (!__syncthreads_or(any)) return;
  // channel i's packed words for positions [P0 + rmin_i, P0 + kBuildCH + rmax_i), window position p
  // at ring word (win0 + p) mod R and at sm[off_s[i] + p - P0 + r] for relative delay r: one bulk
  // copy by lane i, more where the ring wraps
  const int4 i0 = a.pair_rinfo[r0], j0 = a.pair_rinfo2[r0];
  const int nc = i0.y < 0 ? 1 : G == 2 || j0.x < 0 ? 2 : j0.y < 0 ? 3 : 4;  // channels of the group
  const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&bar_s);
  if (threadIdx.x == 0) {
    mbar_init(bar, kPairGMax);
    mbar_fence_init();
  }
  __syncthreads();
  if (threadIdx.x < kPairGMax) {
    const int i = threadIdx.x;
    if (i < nc) {
      const int c = i == 0 ? i0.x : i == 1 ? i0.y : i == 2 ? j0.x : j0.y;
      const int2 rr = i > 0 ? a.pair_prange[k * (kPairGMax - 1) + i - 1] : make_int2(0, 0);
      const long R = a.R;  // a multiple of 4, as the copies' ends
      long pos = (bm.win0 + P0 + rr.x) % R;
      if (pos < 0) pos += R;
      const int sh = (int)(pos & 3), len = (sh + kBuildCH + rr.y - rr.x + 3) / 4 * 4;
      const int at = build_at(i, kBuildCH, a.pair_span);
      off_s[i] = at + sh - rr.x;
      pos -= sh;
      mbar_arrive_tx(bar, 4u * (uint32_t)len);
      const uint32_t s0 = (uint32_t)__cvta_generic_to_shared(sm);
      for (int done = 0; done < len;) {
        const int n = (int)min((long)(len - done), R - pos);
        bulk_g2s(s0 + 4u * (uint32_t)(at + done), bm.packed + (size_t)c * R + pos, 4u * (uint32_t)n, bar);
        done += n;
        pos = 0;
      }
    } else {
      off_s[i] = 0;
      mbar_arrive(bar);
    }
  }
  __syncthreads();  // off_s
  if (!mbar_wait(bar, 0)) {
    if (threadIdx.x == 0 && a.err) atomicOr(a.err, 1);
    mbar_wait(bar, 0);  // the copies in flight land before the block ends
    return;
  }
  const int of0 = off_s[0], of1 = off_s[1], of2 = off_s[2], of3 = off_s[3];
  const int cut = words_cut(a.nout - (a.ntt - 1) * kTileSamples);  // words of the last tile nobody reads
  // one warp per row: the row's metadata is loaded once, the next row's while this one is written.
  // Position first + 512 h + i (i < 256) gives words i and i + 256 of the row's h-th half tile: of
  // the words of tile h / 2 from 512 (h % 2) on, or of a single run from 512 h on.
  const int nwarp = blockDim.x >> 5;
  int r = r0 + (threadIdx.x >> 5);
  BuildRow nx{};
  if (r < r1) nx = build_row(a, r, G == 4);
  for (; r < r1; r += nwarp) {
    const BuildRow in = nx;
    if (r + nwarp < r1) nx = build_row(a, r + nwarp, G == 4);
    const bool run = in.stride == kTileSamples;
    const int total = in.words - cut, nh = run ? (total + 511) / 512 : 2 * a.ntt;
    const int rel = (int)(P0 - in.w);  // chunk start relative to the row's first position
    const int h0 = max(0, (rel - 255 + 511) >> 9), h1 = min(nh, (rel + kBuildCH + 511) >> 9);
    uint32_t *dst = a.pair_rows + (size_t)z * a.pair_rows_stride + in.off;
    const int s0 = of0, s1 = of1 + in.z1, s2 = of2 + in.z2, s3 = of3 + in.z3;
    for (int h = h0; h < h1; ++h) {
      const int q = 512 * h - rel;  // chunk offset of the half tile's first position
      const int left = run ? total - 512 * h : in.stride - 512 * (h & 1) - (h >> 1 == a.ntt - 1 ? cut : 0);
      if (left <= 0) continue;
      uint32_t *d = dst + (run ? 512 * h : (h >> 1) * in.stride + 512 * (h & 1));
      const int lo = max(0, -q), n2 = min(256, left - 256), hi = min(min(256, left), kBuildCH - q);
      const int x[kPairGMax] = {s0 + q, s1 + q, s2 + q, s3 + q};
      const bool full = lo == 0 && hi == 256 && n2 == 256;
      if (nc == G) {
        if (full) build_run<G, true, true>(d, sm, x, lo, hi, n2);
        else if (n2 > lo) build_run<G, true, false>(d, sm, x, lo, hi, n2);
        else build_run<G, false, false>(d, sm, x, lo, hi, n2);
      } else if (G == 4 && nc == 3) {  // the last group
        build_run<3, true, false>(d, sm, x, lo, hi, n2);
      } else if (G == 4 && nc == 2) {
        build_run<2, true, false>(d, sm, x, lo, hi, n2);
      } else {
        build_run<1, true, false>(d, sm, x, lo, hi, n2);
      }
    }
  }
}

// Tile and time tile of item l of a beam's, over its first `ntt` time tiles: `group` DM tiles a time
// tile together.
__device__ __forceinline__ void pair_item(const DedispArgs &a, int ntiles, int ntt, int l, int *tile, int *tt) {
  const int per_group = a.group * ntt;
  const int g = l / per_group, r = l - g * per_group;
  const int gsz = min(a.group, ntiles - g * a.group);
  *tt = r / gsz;
  *tile = g * a.group + (r - *tt * gsz);
}

// A block is two units of 256 threads (one where work or shared memory is for
// one), each with staging buffers, barriers and work items of its own: one
// block an SM, because the totals live in tensor memory and blocks that hold
// some do not share an SM (two 256-thread blocks ran one after the other).
// The 64 totals a thread would otherwise keep in registers are touched once
// in 64 quads; without them the shared reads of several trials are in flight
// at once.  Eight beams of 1024 channels (quads): 7.45 ms against 7.89 with
// the totals in registers (7.75 once a stage's record is prefetched), 16
// beams' short gulps (pairs) 6.18 against 6.30, 2048 channels to DM 2000 the
// same 6.9 ms; lanes added into the output plane instead (red.add every 57
// quads) 9.5 ms there.  Tiles of 32 trials, two units summing 16 each from the
// same staged rows, stage 30 % less and are slower (7.74, 6.37, 7.08 ms).
// MULTI: the launch serves several beams (a.beams, batched context): each
// item looks up its beam; else the one beam's record stays in registers.
template <int CC, bool MULTI>
__global__ void __launch_bounds__(2 * kDedispThreads, 1) k_pair_sum(DedispArgs a, int bufbytes, int nbuf) {
  extern __shared__ __align__(128) uint32_t smem[];
  constexpr int DPT = kPairDPT;
  constexpr int NWARP = kDedispThreads / 32;
  constexpr int HB = stage_hdr_bytes(CC);
  constexpr uint32_t kTotCols = 256;  // four warps' 64 totals a lane
  const int REC = pair_rec_int4(CC);
  const int half = threadIdx.x / kDedispThreads, unit = blockIdx.x * (blockDim.x / kDedispThreads) + half;
  const int units = gridDim.x * (blockDim.x / kDedispThreads);
  char *const mine = reinterpret_cast<char *>(smem) + (size_t)half * unit_smem(bufbytes, nbuf);
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(mine);
  auto full_of = [&](int b) { return sbase + 8u * b; };
  auto empty_of = [&](int b) { return sbase + 32u + 8u * b; };
  auto buf_of = [&](int b) { return sbase + kBarHdr + (uint32_t)b * (uint32_t)bufbytes; };
  const int tid = threadIdx.x % kDedispThreads, lane = tid & 31, warp = tid >> 5;
  // the stage a warp stages next: stage st of the nst stages of block-local item k
  struct Cursor {
    int k, st, s0, nst, t0, z;  // z: beam of the item in the launch
  };
  static_assert(64 + NWARP * sizeof(Cursor) <= kTmemAt, "staging cursors");
  Cursor *cur = reinterpret_cast<Cursor *>(mine + 64) + warp;
  if (tid == 0) {
    for (int b = 0; b < nbuf; ++b) {
      mbar_init(full_of(b), 32);      // every lane of the staging warp arrives once per fill
      mbar_init(empty_of(b), NWARP);  // one arrival per warp once it is done reading
    }
    mbar_fence_init();
  }
  if (threadIdx.x < 32) tmem_alloc((uint32_t)__cvta_generic_to_shared(smem) + kTmemAt, kTotCols);
  __syncthreads();
  // this thread's 64 totals: columns 4 m + k (trial m, sample j + 256 k)
  const uint32_t tmem = smem[kTmemAt / 4];
  const uint32_t totals = tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)(threadIdx.x >> 7) * 64u;

  // Beam z of launch item `item` and the item's tile and time tile.  A last
  // time tile that only needs part of its words (words_cut; outputs past a
  // gulp of whole tiles are the smoothing's few) makes a short item: those of
  // all tiles and beams come last and fill the last round, which whole items
  // would mostly leave empty (16 beams x 8256 outputs 6.23 -> 5.95 ms).  Beam z's tiles are the launch's from (beams[z].
  // item0 - beams[0].item0) / ntt on; a beam without trials has none.
  const DedispBeam b0 = MULTI ? a.one : (a.beams ? a.beams[0] : a.one);
  const int nlong = words_cut(a.nout - (a.ntt - 1) * kTileSamples) > 0 && a.ntt > 1 ? a.ntt - 1 : a.ntt;
  const int shorts = a.nitems / a.ntt * nlong;  // first short item
  auto locate = [&](int item, int *z, int *tile, int *tt) -> DedispBeam {
    const bool tail = item >= shorts;
    const int per = tail ? 1 : nlong;  // items of a tile
    if (tail) item -= shorts;
    int zz = 0;
    DedispBeam bz = b0;
    if (MULTI) {
      const int i0 = a.beams[0].item0;
      while (zz + 1 < a.nbeam && (a.beams[zz + 1].item0 - i0) / a.ntt * per <= item) ++zz;
      bz = a.beams[zz];
      item -= (bz.item0 - i0) / a.ntt * per;
    }
    *z = zz;
    pair_item(a, (bz.dm_count + DPT - 1) / DPT, per, item, tile, tt);
    if (tail) *tt = a.ntt - 1;
    return bz;
  };
  auto load_item = [&](int k) -> bool {  // lane 0
    const int item = unit + k * units;
    if (item >= a.nitems) return false;
    int z, tile, tt;
    locate(item, &z, &tile, &tt);
    const int s0 = a.pair_tile_st[tile];
    *cur = Cursor{k, 0, s0, a.pair_tile_st[tile + 1] - s0, tt * kTileSamples, z};
    return true;
  };
  auto advance = [&](int n) -> bool {  // lane 0
    int st = cur->st + n;
    while (st >= cur->nst) {
      st -= cur->nst;
      if (!load_item(cur->k + 1)) return false;
    }
    cur->st = st;
    return true;
  };
  unsigned g_next = (unsigned)warp;  // next stage this warp stages
  bool p_done;                       // no stage left for this warp
  {
    int more = 0;
    if (lane == 0) more = load_item(0) && advance(warp);
    p_done = !__shfl_sync(0xffffffffu, more, 0);
    __syncwarp();
  }
  // the record of the warp's next stage on its way to L1: the staging warp would otherwise sit out
  // two loads from L2 or DRAM, and the unit with it
  auto prefetch = [&]() {
    const int4 *r = a.pair_rec + (size_t)(cur->s0 + cur->st) * REC;
    prefetch_l1(lane == 31 ? r : r + 1 + CC * DPT / 4 + lane);
  };
  if (!p_done) prefetch();
  auto issue = [&](bool block, bool *timed_out) -> bool {
    const unsigned g = g_next;
    const int b = (int)(g % (unsigned)nbuf);
    if (g >= (unsigned)nbuf) {
      const uint32_t par = ((g / nbuf) - 1u) & 1u;
      if (block) {
        if (!mbar_wait(empty_of(b), par)) {
          *timed_out = true;
          return false;
        }
      } else if (!mbar_test(empty_of(b), par)) {
        return false;
      }
    }
    const int4 *r = a.pair_rec + (size_t)(cur->s0 + cur->st) * REC;
    const int tt = cur->t0 / kTileSamples;
    const int nrows = __ldg(&r->y);
    const uint32_t bar = full_of(b);
    fence_proxy_async();
    if (lane < nrows) {
      // {first word (low, high), words | byte slot / 16 << 16, the row's words per time tile}
      const int4 rw = __ldg(r + 1 + CC * DPT / 4 + lane);
      const long start = (long)(((unsigned long long)(unsigned)rw.y << 32) | (unsigned)rw.x);
      const uint32_t nb = (((uint32_t)rw.z & 0xffffu) - (uint32_t)words_cut(a.nout - cur->t0)) * 4u,
                     slot = ((uint32_t)rw.z >> 16) * 16u;
      mbar_arrive_tx(bar, nb + (lane == 0 ? (uint32_t)HB : 0u));
      const uint32_t *rows = MULTI ? a.pair_rows + (size_t)cur->z * a.pair_rows_stride : a.pair_rows;
      bulk_g2s(buf_of(b) + HB + slot, rows + start + (long)tt * rw.w, nb, bar);
      if (lane == 0) bulk_g2s(buf_of(b), r, HB, bar);
    } else {
      mbar_arrive(bar);
    }
    __syncwarp();
    g_next += NWARP;
    int more = 0;
    if (lane == 0) more = advance(NWARP);
    p_done = !__shfl_sync(0xffffffffu, more, 0);
    __syncwarp();
    if (!p_done) prefetch();
    return true;
  };
  // After a wait ran out: record it, let this warp's copies land, end.
  auto fail = [&](unsigned gs_c) {
    if (lane == 0 && a.err) atomicOr(a.err, 1);
    for (unsigned g = gs_c; g < g_next; ++g)
      if (g % NWARP == (unsigned)warp) mbar_wait(full_of((int)(g % nbuf)), (g / nbuf) & 1u);
  };

  unsigned gs_c = 0;  // stages consumed
  bool ok = true;     // no wait of this warp ran out
  for (int item = unit; ok && item < a.nitems; item += units) {
    int z, tile, tt;
    const DedispBeam bm = locate(item, &z, &tile, &tt);
    // what of the warp's outputs there is in the last time tile: words j (any), words j + 256
    const int rem = a.nout - tt * kTileSamples - 32 * warp;
    const bool any = rem > 0, both = rem > S;
    const int nstage = a.pair_tile_st[tile + 1] - a.pair_tile_st[tile];
    uint32_t acc_a[DPT], acc_b[DPT];  // acc_a: samples j, j+512; acc_b: j+256, j+768
#pragma unroll
    for (int m = 0; m < DPT; ++m) acc_a[m] = acc_b[m] = 0u;
    bool stored = false;  // the totals hold the lanes of earlier stages
    auto widen = [&](uint32_t (&v)[4 * DPT]) {
      if (stored) {
        tmem_ld64(totals, v);
      } else {
#pragma unroll
        for (int i = 0; i < 4 * DPT; ++i) v[i] = 0u;
      }
#pragma unroll
      for (int m = 0; m < DPT; ++m) {
        v[4 * m] += acc_a[m] & 0xffffu;
        v[4 * m + 1] += acc_b[m] & 0xffffu;
        v[4 * m + 2] += acc_a[m] >> 16;
        v[4 * m + 3] += acc_b[m] >> 16;
      }
    };
    int npairs = 0;  // groups in the 16-bit lanes
    for (int st = 0; st < nstage; ++st) {
      {
        bool to = false;
        while (!p_done && g_next < gs_c + nbuf)
          if (!issue(g_next <= gs_c, &to)) break;
        const int b = (int)(gs_c % (unsigned)nbuf);
        if (to || !mbar_wait(full_of(b), (gs_c / nbuf) & 1u)) {
          fail(gs_c);
          ok = false;
          break;
        }
      }
      const int b = (int)(gs_c % (unsigned)nbuf);
      const uint32_t hb = buf_of(b), ob = hb + 16u, rb = hb + (uint32_t)HB + (uint32_t)tid * 4u;
      const int ng = (int)lds32(hb);
      auto add2 = [&](int i) {  // pairs i and i + 1
#pragma unroll
        for (int q = 0; q < DPT / 4; ++q) {
          const int4 x1 = lds128(ob + (uint32_t)(i * DPT + 4 * q) * 4u);
          const int4 x2 = lds128(ob + (uint32_t)((i + 1) * DPT + 4 * q) * 4u);
          const int o1[4] = {x1.x, x1.y, x1.z, x1.w}, o2[4] = {x2.x, x2.y, x2.z, x2.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int m = 4 * q + j;
            const uint32_t p1 = rb + (uint32_t)o1[j], p2 = rb + (uint32_t)o2[j];
            acc_a[m] += lds32(p1) + lds32(p2);
            acc_b[m] += lds32(p1 + 4u * S) + lds32(p2 + 4u * S);
          }
        }
      };
      auto add1 = [&](int i) {
#pragma unroll
        for (int q = 0; q < DPT / 4; ++q) {
          const int4 x1 = lds128(ob + (uint32_t)(i * DPT + 4 * q) * 4u);
          const int o1[4] = {x1.x, x1.y, x1.z, x1.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int m = 4 * q + j;
            const uint32_t p1 = rb + (uint32_t)o1[j];
            acc_a[m] += lds32(p1);
            acc_b[m] += lds32(p1 + 4u * S);
          }
        }
      };
      if (both) {
        int i = 0;
        for (; i + 1 < ng; i += 2) add2(i);
        if (i < ng) add1(i);
      } else if (any) {
        for (int i = 0; i < ng; ++i)
#pragma unroll
          for (int q = 0; q < DPT / 4; ++q) {
            const int4 x1 = lds128(ob + (uint32_t)(i * DPT + 4 * q) * 4u);
            acc_a[4 * q] += lds32(rb + (uint32_t)x1.x);
            acc_a[4 * q + 1] += lds32(rb + (uint32_t)x1.y);
            acc_a[4 * q + 2] += lds32(rb + (uint32_t)x1.z);
            acc_a[4 * q + 3] += lds32(rb + (uint32_t)x1.w);
          }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty_of(b));  // this warp is done with buffer b
      ++gs_c;
      npairs += ng;
      if (npairs + CC > a.pair_lanecap) {
        uint32_t v[4 * DPT];
        widen(v);
        tmem_st64(totals, v);
        stored = true;
#pragma unroll
        for (int m = 0; m < DPT; ++m) acc_a[m] = acc_b[m] = 0u;
        npairs = 0;
      }
    }
    if (!ok) break;
    uint32_t v[4 * DPT];
    widen(v);
    const int t0 = tt * kTileSamples;
#pragma unroll
    for (int m = 0; m < DPT; ++m) {
      const int i = tile * DPT + m;
      if (i >= bm.dm_count) break;
      float *o = bm.out + (size_t)i * a.out_stride;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int t = t0 + tid + k * S;
        if (t < a.nout) o[t] = (float)v[4 * m + k];
      }
    }
  }
  tmem_wait_st();
  __syncthreads();
  if (threadIdx.x < 32) tmem_free(tmem, kTotCols);
}

template <int CC, bool MULTI>
cudaError_t launch_sum(const DedispArgs &a, cudaStream_t s) {
  const int bufbytes = stage_hdr_bytes(CC) + a.pair_stage;
  // the pipeline asked for, else the deepest that leaves room for two units; two buffers at least
  const size_t share = kSmemMost / 2 / 16 * 16;  // one block an SM
  int nbuf = a.nbuf;
  if (!nbuf) {
    nbuf = kMaxBuf;
    while (nbuf > 2 && unit_smem(bufbytes, nbuf) > share) --nbuf;
  }
  if (nbuf < 2 || nbuf > kMaxBuf) return cudaErrorInvalidValue;
  const size_t one = unit_smem(bufbytes, nbuf);
  if (one > kSmemMost) return cudaErrorInvalidValue;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  // units per block: two where they fit, unless each item can have an SM of its own
  const int halves = one <= share && a.nitems > sms ? 2 : 1;
  auto kern = k_pair_sum<CC, MULTI>;
  if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost)) != cudaSuccess)
    return e;
  const int grid = std::max(1, std::min((a.nitems + halves - 1) / halves, sms));
  kern<<<grid, halves * kDedispThreads, halves * one, s>>>(a, bufbytes, nbuf);
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace

PairTables dedisp_pair_tables(const int *delays, int nchan, const int *chans, int nact, int dm_first,
                              int dm_count, int cc, int ntt, int g) {
  PairTables t;
  t.g = g;
  t.cc = cc;
  t.ntt = ntt;
  t.dm_count = dm_count;
  t.ntiles = (dm_count + kPairDPT - 1) / kPairDPT;
  t.npair = (nact + g - 1) / g;
  const int stage_max = pair_stage_budget(cc);
  auto dl = [&](int d, int c) { return delays[(size_t)(dm_first + d) * nchan + c]; };
  // rows: per group, one per distinct pattern (r_1, r_2, r_3) of relative
  // delays, in increasing (lexicographic) order
  using Pat = std::array<int, kPairGMax - 1>;
  std::vector<Pat> rel(dm_count), u;
  t.row_of.assign((size_t)dm_count * t.npair, 0);
  t.prow.assign(t.npair + 1, 0);
  t.prange.assign((size_t)t.npair * (kPairGMax - 1), make_int2(0, 0));
  for (int k = 0; k < t.npair; ++k) {
    int c[kPairGMax];
    for (int i = 0; i < kPairGMax; ++i) c[i] = i < g && g * k + i < nact ? chans[g * k + i] : -1;
    for (int d = 0; d < dm_count; ++d)
      for (int i = 1; i < kPairGMax; ++i) rel[d][i - 1] = c[i] >= 0 ? dl(d, c[i]) - dl(d, c[0]) : 0;
    u = rel;
    std::sort(u.begin(), u.end());
    u.erase(std::unique(u.begin(), u.end()), u.end());
    const int base = (int)t.rinfo.size();
    for (const Pat &v : u) {
      t.rinfo.push_back(make_int4(c[0], c[1], v[0], 1 << 30));
      t.rinfo2.push_back(make_int4(c[2], c[3], v[1], v[2]));
    }
    for (int d = 0; d < dm_count; ++d) {
      const int id = base + (int)(std::lower_bound(u.begin(), u.end(), rel[d]) - u.begin());
      t.row_of[(size_t)d * t.npair + k] = id;
      t.rinfo[id].w = std::min(t.rinfo[id].w, dl(d, c[0]));
    }
    for (int i = 1; i < kPairGMax; ++i) {
      int lo = 0, hi = 0;
      for (size_t j = 0; j < u.size(); ++j) {
        lo = j ? std::min(lo, u[j][i - 1]) : u[j][i - 1];
        hi = j ? std::max(hi, u[j][i - 1]) : u[j][i - 1];
      }
      t.prange[(size_t)k * (kPairGMax - 1) + i - 1] = make_int2(lo, hi);
      t.max_span = std::max(t.max_span, hi - lo);
    }
    t.prow[k + 1] = (int)t.rinfo.size();
  }
  t.nrows = (int)t.rinfo.size();
  // per row, the union of its copies' windows within a time tile: [lo, hi) words from its first position
  std::vector<long long> lo(t.nrows, 1LL << 60), hi(t.nrows, 0);
  int max_nw = 0;
  // stage records
  const int REC = pair_rec_int4(cc);
  const int offs0 = 4, rows0 = 4 + cc * kPairDPT;  // int positions in a record
  std::vector<int> rec(REC * 4);
  struct Fix {
    size_t rec_int;  // int index of the row entry in t.rec
    int row, bal;
  };
  std::vector<Fix> fixes;
  std::vector<Fix> pending;
  int ng = 0, nr = 0, bytes = 0;
  auto flush = [&]() {
    const size_t at = t.rec.size() * 4;
    for (Fix f : pending) fixes.push_back(Fix{at + f.rec_int, f.row, f.bal});
    pending.clear();
    rec[0] = ng;
    rec[1] = nr;
    const size_t n0 = t.rec.size();
    t.rec.resize(n0 + REC);
    std::memcpy(&t.rec[n0], rec.data(), rec.size() * sizeof(int));
    t.max_stage = std::max(t.max_stage, bytes);
    std::fill(rec.begin(), rec.end(), 0);
    ng = nr = bytes = 0;
  };
  int ids[kPairDPT], av[kPairDPT];
  t.tile_st.push_back(0);
  for (int i = 0; i < t.ntiles; ++i) {
    const int d0 = i * kPairDPT, nt = std::min(kPairDPT, dm_count - d0);
    for (int k = 0; k < t.npair; ++k) {
      const int c0 = chans[g * k];
      int uid[kPairDPT], ub[kPairDPT], us[kPairDPT], nu = 0;
      for (int m = 0; m < nt; ++m) {
        ids[m] = t.row_of[(size_t)(d0 + m) * t.npair + k];
        av[m] = dl(d0 + m, c0) - t.rinfo[ids[m]].w;
        int j = 0;
        while (j < nu && uid[j] != ids[m]) ++j;
        if (j == nu) {
          uid[nu] = ids[m];
          ub[nu] = us[nu] = av[m];
          ++nu;
        } else {
          ub[j] = std::min(ub[j], av[m]);
          us[j] = std::max(us[j], av[m]);
        }
      }
      int add = 0, bal[kPairDPT], nw[kPairDPT];
      for (int j = 0; j < nu; ++j) {
        const int sh = ub[j] & 3;
        bal[j] = ub[j] - sh;
        nw[j] = (2 * S + (us[j] - ub[j]) + sh + 3) / 4 * 4;
        add += nw[j] * 4;
      }
      if (ng > 0 && (ng == cc || nr + nu > kPairRowsMax || bytes + add > stage_max)) flush();
      for (int j = 0; j < nu; ++j) {
        const int slot = bytes;
        for (int m = 0; m < nt; ++m)
          if (ids[m] == uid[j]) rec[offs0 + ng * kPairDPT + m] = slot + (av[m] - bal[j]) * 4;
        int *rw = &rec[rows0 + 4 * nr];
        rw[2] = (nw[j] & 0xffff) | (slot / 16) << 16;  // words (< 2^16) | byte slot / 16
        max_nw = std::max(max_nw, nw[j]);
        pending.push_back(Fix{(size_t)(rows0 + 4 * nr), uid[j], bal[j]});
        lo[uid[j]] = std::min(lo[uid[j]], (long long)bal[j]);
        hi[uid[j]] = std::max(hi[uid[j]], (long long)bal[j] + nw[j]);
        ++nr;
        bytes += nw[j] * 4;
      }
      ++ng;
    }
    if (ng > 0) flush();
    t.tile_st.push_back((int)(t.rec.size() / REC));
  }
  // Row layout.  A row keeps, for each time tile tt, the words its copies read: [tt * 1024 + lo,
  // tt * 1024 + hi) of its positions.  When hi - lo < 1024 the tiles' windows do not meet and are
  // stored one after another (tile stride hi - lo words); else the row is one run from lo (stride
  // 1024: the tiles' windows overlap).  Word i then holds position
  //   first + (i / stride) * 1024 + i % stride,   first = (smallest delay of its trials) + lo,
  // and a copy of tile tt starts at word tt * stride + (bal - lo).  Offsets and lengths stay
  // multiples of 4 words, so every copy starts 16-byte aligned.
  t.roff.resize(t.nrows);
  t.rwords.resize(t.nrows);
  t.rtile.resize(t.nrows);
  long long off = 0;
  for (int r = 0; r < t.nrows; ++r) {
    const long long span = hi[r] - lo[r];  // multiple of 4: lo and hi are
    const int stride = span < kTileSamples ? (int)span : kTileSamples;
    const long long w = (long long)(ntt - 1) * stride + span;
    t.rinfo[r].w += (int)lo[r];
    t.roff[r] = off;
    t.rwords[r] = (int)w;
    t.rtile[r] = stride;
    off += w;
    t.npos = std::max(t.npos, (long)t.rinfo[r].w + (long)(ntt - 1) * kTileSamples + (long)span);
  }
  t.words = (long)off;
  if (max_nw > 0xffff) t.max_stage = 1 << 30;  // a copy longer than its 16-bit field: no launch takes these
  int *ri = reinterpret_cast<int *>(t.rec.data());
  for (const Fix &f : fixes) {
    const unsigned long long start = (unsigned long long)(t.roff[f.row] + f.bal - lo[f.row]);
    ri[f.rec_int] = (int)(unsigned)(start & 0xffffffffull);
    ri[f.rec_int + 1] = (int)(unsigned)(start >> 32);
    ri[f.rec_int + 3] = t.rtile[f.row];
  }
  return t;
}

void pair_row_ends(const PairTables &t, int count, int *ends) {
  for (int k = 0; k < t.npair; ++k) {
    int e = t.prow[k];
    for (int d = 0; d < std::min(count, t.dm_count); ++d) e = std::max(e, t.row_of[(size_t)d * t.npair + k] + 1);
    ends[k] = e;
  }
}

cudaError_t dedisperse_pairs(const DedispArgs &a, cudaStream_t s) {
  const int g = a.pair_g;
  if ((a.beams && (a.nbeam < 1 || a.nbeam > kPairMaxBeams || (a.nbeam > 1 && a.pair_rows_stride <= 0))) ||
      a.dpt != kPairDPT || (a.mode != 5 && a.mode != 6) || (g != 2 && g != 4) ||
      !a.pair_rows || !a.pair_rec || !a.pair_tile_st || !a.pair_rinfo || !a.pair_rinfo2 || !a.pair_roff ||
      !a.pair_rwords || !a.pair_rtile || !a.pair_prow || !a.pair_prange || a.pair_npair <= 0 ||
      a.pair_npair > 65535 ||
      a.pair_stage <= 0 || a.pair_stage % 16 != 0 || a.pair_span < 0 || a.pair_lanecap < 1 ||
      a.pair_lanecap > pair_lanecap(g))
    return cudaErrorInvalidValue;
  if (a.R <= 0 || (!a.beams && a.one.win0 < 0)) return cudaErrorInvalidValue;
  // the group's channel windows: ch words for c0, ch + its r range for the others, up to 200 KB of
  // them (ranges of 43,008 samples for pairs, 14,336 for quads); the windows' alignment comes on top
  const int ch = build_chunk(g);
  if (((size_t)g * ch + (size_t)(g - 1) * a.pair_span) * 4 > kBuildMost) return cudaErrorInvalidValue;
  const size_t bsmem = (size_t)build_at(g, ch, a.pair_span) * 4;
  auto kern = g == 4 ? k_pair_build<4> : k_pair_build<2>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kBuildMost + 1024);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((a.pair_npos + ch - 1) / ch), (unsigned)a.pair_npair, (unsigned)(a.beams ? a.nbeam : 1));
  kern<<<grid, 256, bsmem, s>>>(a);
  count_launches(1);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  const bool multi = a.beams && a.nbeam > 1;
  switch (a.cc * 2 + (multi ? 1 : 0)) {
    case 8: return launch_sum<4, false>(a, s);
    case 9: return launch_sum<4, true>(a, s);
    case 16: return launch_sum<8, false>(a, s);
    case 17: return launch_sum<8, true>(a, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace hg
