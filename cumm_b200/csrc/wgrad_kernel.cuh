// Weight-gradient kernel of the mask-based sparse convolution (and the gather-gather
// "ShuffleAB" GEMM) for sm_100a.
//
//   dW[k, f, c] = alpha * sum_r dout[o_r, k] * X[idx[f, o_r], c] + beta * dW_prev[k, f, c]
//
// The reduction runs over (sorted) rows, so both tcgen05 operands are gathered rows held
// "MN-major": a gathered row is 128-byte-swizzled along its channels and the 128 rows of a
// tile are the K dimension of the MMA.  Work is cut into units (filter offset f, range of
// row tiles); a unit accumulates in TMEM, leaves one fp32 partial [128 x BLOCK_N] in the
// workspace and counts itself in; the unit that completes an offset sets the offset's ready flag.
// The partials of an offset are summed in unit order (the result does not depend on timing)
// by CTAs that have finished their own units and wait, bounded, for that flag: an offset with few
// units by one CTA (the offsets are dealt out over the grid); an offset with many units (the
// centre of a submanifold convolution has one per CTA) by all CTAs, each taking a fixed share
// of the tile's positions.  One launch, no atomics on data.  The wait
// is the only place where a CTA depends on others: like every wait in this library it gives up
// after a second and reports through the status word, and the launcher keeps the grid within
// the number of SMs so that all CTAs run at once (the reference serialises split-K slices through
// an unbounded spinning semaphore, cumm/conv/kernel.py:960-1083).
//
// Semantics follow cumm/gemm/blockmma/mma.py:608-648,722-740 (a row takes part for
// offset f iff the reduced-mask word covering it has bit f), cumm/conv/sparse_iters.py
// :284-316 (A = dout[mask_argsort[r]], B = X[indices[f, mask_argsort[r]]], -1 -> zeros)
// and cumm/conv/kernel.py:890-897 (offsets outside mask_filter are left untouched).
#pragma once
#include "ptx.cuh"
#include "rowconv_kernel.cuh"

namespace cb2 {

enum : int { kWgradMaskConv = 0, kWgradPairList = 1 };
// Row-gather implementations: 16-byte cp.async per chunk, or TMA tile::gather4, four rows per
// request (a row coordinate of -1 is out of bounds and reads as zeros).
enum : int { kGatherCpAsync = 0, kGatherTma4 = 2 };

struct WgradParams {
  const void *dout;        // A rows [*, m_total]  (fp16)
  const void *x;           // B rows [*, n_total]  (fp16)
  const int32_t *indices;  // [kv, n_rows]
  const uint32_t *rmask;   // reduced masks: `words` words (32 filter offsets each) per mask_width sorted rows
  const int32_t *argsort;  // [n_rows]
  const int32_t *a_inds;   // pair-list mode
  const int32_t *b_inds;   //   "
  float *partials;         // workspace: [unit][m_tile][n_tile][128 x BLOCK_N] fp32
  int *ctl;                // workspace, zero between calls but for [1]: [0] CTAs that have left; [1] what the plan
                           // is (kWgradPlanTiles, kWgradPlanRows); [9 + 8 by, 13 + 8 by) bit masks of the ready offsets of output tile by; from kWgradCtlBase on, per
                           // (f, by) at a pitch of four ints: units arrived
  int *sched;              // workspace header: [0,128) number of row tiles carrying offset f
  const int *lists;        // workspace: per offset, the ordered list of those tiles
  int list_stride;         // ints between two offsets' lists
  int *row_head;           // workspace or null, for plans with row lists: [0,128) first entry of offset f's row
                           // list, -1 = walked by tiles; [128,256) its entries
  const int *rows;         // workspace: the row lists
  int *status;
  void *out;               // dW
  const void *src;         // source for beta (dW itself unless the caller gave another)
  long long ldo;           // elements between consecutive m rows of out
  long long f_stride;      // elements between consecutive f slices
  float alpha, beta;
  int out_f32;
  long long ld_dout, ld_x;
  int n_rows;
  int a_rows, b_rows;
  int m_total, n_total;
  int kv;
  int mask_width;
  int words;               // mask words per chunk of mask_width rows: ceil(kv / 32)
  int rmask_words;         // chunks the reduced-mask array holds
  uint32_t mask_filter;
  int mode;
  int plan_fixed;          // the plan is an earlier call's
};

// A_ATOMS: 64-channel column blocks of dout a tile loads.  With up to 64 output channels one is
// enough: the MMA still has 128 rows, the upper 64 read whatever follows the stage's first block and
// their sums are never stored.  The stages are as many as 192 KB hold, so that narrow layers have as
// many bytes in flight as wide ones.
template <int BLOCK_N, int A_ATOMS, int GATHER> struct WgradCfg {
  static constexpr int A_BYTES = 128 * 128 * A_ATOMS;       // 128 rows x 64 channels per block
  static constexpr int B_BYTES = 128 * 2 * BLOCK_N;         // 128 rows x BLOCK_N fp16
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SA = GATHER == kGatherCpAsync ? 3 : 192 * 1024 / STAGE_BYTES;  // 3, 4 or 6
  static constexpr int M_ROWS = 64 * A_ATOMS;               // rows of a partial sum that are kept
  static constexpr int TMEM_COLS = 2 * BLOCK_N;
  // Epilogue (4 warps), MMA issuer, twelve warps that gather: four per stage, or two where there are
  // more than three stages (issuing a stage's requests takes a warp longer than an MMA step: with one
  // warp per stage the 128-channel layer took 45 instead of 35 us).
  static constexpr int GW = SA == 3 ? 4 : 2;
  static constexpr int THREADS = 544;
  static constexpr int FULL_COUNT = GATHER == kGatherCpAsync ? 128 : 1;
  static constexpr int OFF_STAGES = 0;
  static constexpr int OFF_ROWIDX = SA * STAGE_BYTES;       // 3 x 2 buffers x 2 operands x 128 ints
  static constexpr int OFF_SCHED = OFF_ROWIDX + 3 * 2 * 2 * 128 * 4;  // this CTA's units, then units per offset
  static constexpr int TILE_CAP = 2048;                      // tiles of one CTA staged in shared memory
  static constexpr int OFF_TILES = OFF_SCHED + 1280 * 4;
  static constexpr int OFF_BARS = OFF_TILES + TILE_CAP * 4;
  static constexpr int BAR_ACC_FULL = 2 * SA, BAR_ACC_EMPTY = BAR_ACC_FULL + 2, BAR_FINAL = BAR_ACC_EMPTY + 2;
  static constexpr int OFF_MISC = OFF_BARS + (BAR_FINAL + 2) / 2 * 2 * 8;
  static constexpr int SMEM_BYTES = OFF_MISC + 64 + 1024;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget of one CTA exceeded");
  static_assert(A_ATOMS == 2 || GATHER == kGatherTma4, "the cp.async path loads both column blocks");
};

// Does row tile `tile` (sorted rows [128*tile, 128*tile + 128)) carry filter offset f?  OR of the
// reduced-mask words of offset f's group of 32 over the chunks that cover the tile.
__device__ __forceinline__ bool wgrad_tile_has(const WgradParams &p, int tile, int f) {
  if (p.mode != kWgradMaskConv)
    return true;
  if (!((p.mask_filter >> (f & 31)) & 1u))
    return false;
  const uint32_t *col = p.rmask + (f >> 5);
  if (p.mask_width == 128)  // the usual case: one chunk per tile
    return tile < p.rmask_words && ((__ldg(col + (long long)tile * p.words) >> (f & 31)) & 1u);
  const int r0 = tile * 128;
  int r1 = r0 + 127;
  if (r1 >= p.n_rows)
    r1 = p.n_rows - 1;
  int w0 = r0 / p.mask_width, w1 = r1 / p.mask_width;
  uint32_t v = 0;
  for (int w = w0; w <= w1; ++w)
    if (w < p.rmask_words)
      v |= __ldg(col + (long long)w * p.words);
  return (v >> (f & 31)) & 1u;
}

// ---------------------------------------------------------------- schedule
// The work is the sequence of all (filter offset f, row tile carrying f) pairs, offsets in
// ascending order, tiles in ascending order inside an offset: T steps in all, with what an offset's
// units cost charged in steps.  CTA c of G takes the steps [c*T/G, (c+1)*T/G) -- every CTA the same
// number, whatever the offsets' shares -- and each maximal run of one offset inside a CTA's range is a UNIT: it accumulates in TMEM
// and leaves one fp32 partial.  The units of an offset are consecutive in this numbering, and
// there are at most G + kv - 1 of them.
//
// A small planning kernel (one block per offset) writes, per offset, the count and the ordered
// list of its tiles, and clears the control words; the main kernel derives
// everything else from the kv counts.  The plan depends only on the reduced masks, the row
// count and the mask filter, so a caller that runs the same layer again (the next training
// step) may keep it: see `reuse_plan` in the C ABI.
//   sched[f]                      tiles carrying offset f
//   lists[f * list_stride + k]    the k-th of them

// Which kind a plan is stands in a control word, not in what the caller says: a plan may be used again
// through an argument record of another workspace size or with other flags than it was made with.
enum : int { kWgradPlanTiles = 0, kWgradPlanRows = 1 };
__device__ __forceinline__ int wgrad_ctl_start(int i, int plan) { return i == 1 ? plan : 0; }

// One warp plans for up to 128 offsets: lane l owns offsets 4l .. 4l+3.
constexpr int kWgradMaxOffsets = 128;
// Exclusive prefix sum, in offset order, of four values per lane; `total` = the sum of all.
__device__ __forceinline__ void wgrad_scan4(const int (&v)[4], int (&excl)[4], int &total) {
  const int lane = (int)lane_id();
  const int mine = v[0] + v[1] + v[2] + v[3];
  int incl = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d)
      incl += t;
  }
  total = __shfl_sync(0xffffffffu, incl, 31);
  int run = incl - mine;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    excl[j] = run;
    run += v[j];
  }
}
// A unit costs its CTA about as much as kWgradUnitSteps steps (a partial sum stored, counted in, and
// read again by whoever sums): every offset is charged that many steps before its own, or the CTAs that
// get a dozen offsets of one or two steps each are the last to finish.  The cuts are made in charged steps.
// (Over 247 shapes of 1500 to 490 000 rows two and three steps are the same in the mean, and three moves the cuts
// by luck, us: 150 000 uniform rows at 128 channels 27.7 and 26.5, 80 000 20.6 and 21.2, 10 000 scanned ones 20.3
// and 20.9; 104 to 72 channels, stride 2 from 150 000 uniform rows 58 and 64, 150 000 scanned ones 73.4 and 76.0.)
constexpr int kWgradUnitSteps = 2;
// Given the step counts of this lane's offsets: P = charged steps before the offset's first own step,
// T = all charged steps, c_first = CTA holding the offset's first step, S = units of the offset, U = units
// before it.
__device__ __forceinline__ void wgrad_plan_warp(const int (&cnt)[4], int G, int (&P)[4], int &T, int (&c_first)[4],
                                                int (&S)[4], int (&U)[4]) {
  int charged[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
    charged[j] = cnt[j] > 0 ? cnt[j] + kWgradUnitSteps : 0;
  wgrad_scan4(charged, P, T);
#pragma unroll
  for (int j = 0; j < 4; ++j)
    P[j] += kWgradUnitSteps;
  // the CTA holding step x is the largest c with c*T/G <= x, i.e. ceil((x+1)*G/T) - 1
  auto chunk_of = [&](int x) -> int {
    const int c = (int)((((long long)x + 1) * G + T - 1) / T) - 1;
    return c < G - 1 ? c : G - 1;
  };
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    c_first[j] = 0;
    S[j] = 0;
    if (cnt[j] > 0) {
      c_first[j] = chunk_of(P[j]);
      S[j] = chunk_of(P[j] + cnt[j] - 1) - c_first[j] + 1;
    }
  }
  int total_units;
  wgrad_scan4(S, U, total_units);
}

// One block per filter offset: count and list the tiles that carry it.  Warp w owns a
// contiguous span of tiles, so the list comes out in ascending order with one block-wide
// synchronisation per batch of 1024 * K tiles.
__global__ void __launch_bounds__(1024) wgrad_plan_kernel(const WgradParams p, int *lists, int list_stride, int n_ctl) {
  constexpr int K = 4;  // 4096 tiles per batch
  __shared__ int s_w[32];
  const int f = blockIdx.x;
  // the control words start from zero (every later call leaves them at zero again)
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_ctl; i += gridDim.x * blockDim.x)
    p.ctl[i] = wgrad_ctl_start(i, kWgradPlanTiles);
  const int ntiles = (p.n_rows + 127) / 128;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  grid_dep_launch();  // the main kernel may set itself up meanwhile; it waits before reading the lists
  int *list = lists + (long long)f * list_stride;
  int running = 0;
  for (int base = 0; base < ntiles; base += 1024 * K) {
    bool on[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int t = base + (wid * K + k) * 32 + lane;
      on[k] = t < ntiles && wgrad_tile_has(p, t, f);
    }
    int mine = 0;
#pragma unroll
    for (int k = 0; k < K; ++k)
      mine += __popc(__ballot_sync(0xffffffffu, on[k]));
    __syncthreads();  // s_w of the previous batch has been read
    if (lane == 0)
      s_w[wid] = mine;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
      const int v = s_w[w];
      all += v;
      if (w < wid)
        before += v;
    }
    int pos = running + before;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const uint32_t bal = __ballot_sync(0xffffffffu, on[k]);
      if (on[k])
        list[pos + __popc(bal & ((1u << lane) - 1u))] = base + (wid * K + k) * 32 + lane;
      pos += __popc(bal);
    }
    running += all;
  }
  if (threadIdx.x == 0)
    p.sched[f] = running;
}

// ---------------------------------------------------------------- plan with row lists
// A tile of 128 sorted rows carries every offset that any of its rows has, so away from the centre
// most of a tile's rows are empty for most of its offsets: on a scanned scene every second row, with
// 125 offsets four of five.  Where that is so the reduction does not run over tiles but over the rows
// themselves: a step takes the next 128 rows that have a neighbour at the offset, and an offset has
// ceil(pairs / 128) steps.  Two kernels make the lists: one marks, per (offset, tile), the rows that take
// part (a 128-bit word) and counts them per chunk of tiles, the other turns counts into places and
// writes the lists in sorted order, so the sums have one fixed order.  Offsets whose tiles are at least
// four fifths full, and lists that find no room, are walked by tiles.  (The kernel by tiles and by rows, and
// what planning adds: 100 003 rows of a scanned scene, 64 channels, 8234 and 4030 steps, 75 and 40 us, 3.5 and
// 19 us; 34 000 rows, 125 offsets, 270 and 35 us, 5 and 32 us; 150 000 uniform rows, 128 channels, 34.0 and
// 32.4 us, 3.6 and 13 us; 960 000 such rows, 105 us either way, 7 and 25 us -- there lists do not pay.  At four
// fifths the shorter walk is worth the table read that makes it.)
constexpr int kWgradPlanThreads = 1024;  // a warp per tile of a group of 32
constexpr int kWgradMaxChunks = 64;
// tiles per chunk: whole groups of 32
__host__ __device__ inline int wgrad_chunk_tiles(int ntiles) {
  return 32 * ((ntiles + 32 * kWgradMaxChunks - 1) / (32 * kWgradMaxChunks));
}

// Rows of tile t, which carries offset f, that take part there, 32 per word (warp-collective); o = the
// output rows.
__device__ __forceinline__ uint4 wgrad_tile_rows(const WgradParams &p, int t, int f, int (&o)[4]) {
  const int lane = (int)lane_id();
  uint32_t w[4];
  bool on[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int r = t * 128 + q * 32 + lane;
    o[q] = r < p.n_rows ? __ldg(p.argsort + r) : -1;
    on[q] = o[q] >= 0;
    if (p.mask_width < 128 && on[q])
      on[q] = (__ldg(p.rmask + (long long)(r / p.mask_width) * p.words + (f >> 5)) >> (f & 31)) & 1u;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    w[q] = __ballot_sync(0xffffffffu, on[q] && __ldg(p.indices + (long long)f * p.n_rows + o[q]) >= 0);
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ bool wgrad_listed(long long rows, long long tiles) {
  return 512 * tiles > 5 * rows;  // tiles less than four fifths full
}

// Few tiles: both in one launch, a block per offset, every list with room for all rows (so that no offset
// has to know the others' counts).  A block takes 32 tiles at a time, one round after the other, so the line lies
// low for as many offsets as blocks of two launches fill the chip with, and higher for more (planning and the
// kernel in one and in two launches, scanned scenes: 27 offsets, 51 tiles 22.4 and 24.0 us, 79 tiles 25.8 and
// 25.1, 219 tiles 35.3 and 29.2; 125 offsets, 51 tiles 24.6 and 28.0, 235 tiles 53.6 and 61.2; a uniform one
// of 469 tiles 53.9 and 41.5).
constexpr int kWgradRoomyTiles = 256;  // up to here the lists have room for all rows whichever way they are made
__host__ __device__ inline bool wgrad_one_block(long long ntiles, int kv) { return ntiles <= (kv <= 32 ? 64 : kWgradRoomyTiles); }
__global__ void __launch_bounds__(kWgradPlanThreads) wgrad_plan_rows_kernel(const WgradParams p, int *lists, int *rows,
                                                                            int n_ctl) {
  __shared__ int s_n[32];
  const int f = blockIdx.x;
  for (int i = f * blockDim.x + threadIdx.x; i < n_ctl; i += gridDim.x * blockDim.x)
    p.ctl[i] = wgrad_ctl_start(i, kWgradPlanRows);
  grid_dep_launch();  // the main kernel may set itself up meanwhile; it waits before reading the plan
  const int ntiles = (p.n_rows + 127) / 128;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long long base = (long long)f * ((p.n_rows + 127) / 128 * 128);
  int all_rows = 0, all_tiles = 0;
  for (int t0 = 0; t0 < ntiles; t0 += 32) {
    const int t = t0 + wid;
    int o[4];
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (t < ntiles && wgrad_tile_has(p, t, f))
      v = wgrad_tile_rows(p, t, f, o);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    const int n = __popc(w[0]) + __popc(w[1]) + __popc(w[2]) + __popc(w[3]);
    __syncthreads();  // s_n of the previous round has been read
    if (lane == 0)
      s_n[wid] = n;
    __syncthreads();
    const int c = s_n[lane];
    const unsigned any = __ballot_sync(0xffffffffu, c > 0);
    const int round_rows = __reduce_add_sync(0xffffffffu, c);
    int at = all_rows + __reduce_add_sync(0xffffffffu, lane < wid ? c : 0);
    if (lane == 0 && n > 0)
      lists[(long long)f * p.list_stride + all_tiles + __popc(any & ((1u << wid) - 1u))] = t;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if ((w[q] >> lane) & 1u)
        rows[base + at + __popc(w[q] & ((1u << lane) - 1u))] = o[q];
      at += __popc(w[q]);
    }
    all_rows += round_rows;
    all_tiles += __popc(any);
  }
  if (threadIdx.x == 0) {
    const bool listed = wgrad_listed(all_rows, all_tiles);
    p.sched[f] = listed ? (all_rows + 127) / 128 : all_tiles;
    p.row_head[f] = listed ? (int)base : -1;
    p.row_head[kWgradMaxOffsets + f] = all_rows;
  }
}

// grid (chunks, offsets); bits[f][tile][4], counts[f][chunk] = {rows, tiles with any}
__global__ void __launch_bounds__(kWgradPlanThreads) wgrad_mark_rows_kernel(const WgradParams p, uint4 *bits, int2 *counts,
                                                                            int n_ctl) {
  __shared__ int2 s_sum[kWgradPlanThreads / 32];
  const int f = blockIdx.y, chunk = blockIdx.x;
  grid_dep_launch();  // the next kernel waits before it reads what this one writes
  for (int i = (f * gridDim.x + chunk) * blockDim.x + threadIdx.x; i < n_ctl; i += gridDim.x * gridDim.y * blockDim.x)
    p.ctl[i] = wgrad_ctl_start(i, kWgradPlanRows);
  const int ntiles = (p.n_rows + 127) / 128;
  const int per = wgrad_chunk_tiles(ntiles), run = per / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int t0 = chunk * per + wid * run, t1 = min(t0 + run, ntiles);
  uint4 *mine = bits + (long long)f * p.list_stride;
  int rows = 0, tiles = 0;
  for (int first = t0; first < t1; first += 32) {
    // the mask words of the warp's tiles in one load: away from the centre most have nothing to do
    const bool has = first + lane < t1 && wgrad_tile_has(p, first + lane, f);
    if (first + lane < t1 && !has)
      mine[first + lane] = make_uint4(0u, 0u, 0u, 0u);
    for (unsigned left = __ballot_sync(0xffffffffu, has); left; left &= left - 1) {
      const int t = first + __ffs(left) - 1;
      int o[4];
      const uint4 v = wgrad_tile_rows(p, t, f, o);
      const int n = __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
      rows += n;
      tiles += n > 0;
      if (lane == 0)
        mine[t] = v;
    }
  }
  if (lane == 0)
    s_sum[wid] = make_int2(rows, tiles);
  __syncthreads();
  if (threadIdx.x == 0) {
    int2 all = make_int2(0, 0);
    for (int w = 0; w < kWgradPlanThreads / 32; ++w)
      all.x += s_sum[w].x, all.y += s_sum[w].y;
    counts[f * gridDim.x + chunk] = all;
  }
}

// A block of the second kernel whose chunk has none of the offset's rows is gone at once; the others add up the
// counts with all warps, a warp per offset, their loads in flight together (with a thread per offset, one load
// after the other, planning and the kernel took 163 instead of 130 us for 960 000 uniform rows, 54.5 instead
// of 45.6 for 150 000, 123 instead of 118 for 300 000 scanned ones).  Warp w takes a contiguous run of the
// chunk's tiles.
__global__ void __launch_bounds__(kWgradPlanThreads) wgrad_list_rows_kernel(const WgradParams p, const uint4 *bits,
                                                                            const int2 *counts, int *lists, int *rows,
                                                                            long long capacity) {
  __shared__ int s_rows[kWgradMaxOffsets], s_tiles[kWgradMaxOffsets];
  __shared__ int s_base, s_before[2];
  __shared__ int2 s_n[32];
  const int f = blockIdx.y, chunk = blockIdx.x, n_chunks = gridDim.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  grid_dep_launch();  // the main kernel may set itself up meanwhile; it waits before reading the plan
  grid_dep_wait();
  if (chunk > 0 && __ldg(counts + f * n_chunks + chunk).x == 0)
    return;
#pragma unroll
  for (int j = 0; j < kWgradMaxOffsets / 32; ++j) {
    const int g = 32 * j + wid;
    int2 all = make_int2(0, 0), before = make_int2(0, 0);
    if (g < p.kv) {
#pragma unroll
      for (int i = 0; i < kWgradMaxChunks / 32; ++i) {
        const int c = 32 * i + lane;
        const int2 v = c < n_chunks ? __ldg(counts + g * n_chunks + c) : make_int2(0, 0);
        all.x += v.x, all.y += v.y;
        if (c < chunk)
          before.x += v.x, before.y += v.y;
      }
    }
    all.x = __reduce_add_sync(0xffffffffu, all.x), all.y = __reduce_add_sync(0xffffffffu, all.y);
    if (lane == 0)
      s_rows[g] = all.x, s_tiles[g] = all.y;
    if (g == f) {
      before.x = __reduce_add_sync(0xffffffffu, before.x), before.y = __reduce_add_sync(0xffffffffu, before.y);
      if (lane == 0)
        s_before[0] = before.x, s_before[1] = before.y;
    }
  }
  const int ntiles = (p.n_rows + 127) / 128;
  const int per = wgrad_chunk_tiles(ntiles), run = per / 32;
  const int t0 = chunk * per + wid * run, t1 = min(min(t0 + run, (chunk + 1) * per), ntiles);
  const uint4 *mine = bits + (long long)f * p.list_stride;
  int2 n = make_int2(0, 0);
  for (int t = t0 + lane; t < t1; t += 32) {
    const uint4 w = __ldg(mine + t);
    const int c = __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
    n.x += c, n.y += c > 0;
  }
  n.x = __reduce_add_sync(0xffffffffu, n.x), n.y = __reduce_add_sync(0xffffffffu, n.y);
  if (lane == 0)
    s_n[wid] = n;
  __syncthreads();
  if (wid == 0) {
    int size[4], first[4], total;
    bool listed[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int g = 4 * lane + j;
      listed[j] = wgrad_listed(s_rows[g], s_tiles[g]);
      size[j] = listed[j] ? (s_rows[g] + 127) / 128 : 0;  // in steps
    }
    wgrad_scan4(size, first, total);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (4 * lane + j == f) {
        const int base = listed[j] && 128ll * (first[j] + size[j]) <= capacity ? 128 * first[j] : -1;
        s_base = base;
        if (chunk == 0) {
          p.sched[f] = base >= 0 ? size[j] : s_tiles[f];
          p.row_head[f] = base;
          p.row_head[kWgradMaxOffsets + f] = s_rows[f];
        }
      }
  }
  const int2 others = s_n[lane];
  int at = s_before[0] + __reduce_add_sync(0xffffffffu, lane < wid ? others.x : 0);
  int at_tile = s_before[1] + __reduce_add_sync(0xffffffffu, lane < wid ? others.y : 0);
  __syncthreads();
  const int base = s_base;
  for (int t = t0; t < t1; ++t) {
    const uint4 v = __ldg(mine + t);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    if ((v.x | v.y | v.z | v.w) == 0)
      continue;
    if (base < 0) {
      if (lane == 0)
        lists[(long long)f * p.list_stride + at_tile] = t;
      ++at_tile;
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if ((w[q] >> lane) & 1u)
          rows[base + at + __popc(w[q] & ((1u << lane) - 1u))] = __ldg(p.argsort + t * 128 + q * 32 + lane);
        at += __popc(w[q]);
      }
    }
  }
}

// Per CTA, in shared memory: s_plan[0] = number of units of this CTA, s_plan[1], s_plan[2] = whether its tiles are in
// shared memory and whether the plan lists rows, then, from 8 on, seven ints per unit
// {f, first step of the offset, one past the last, unit number, offset of its tiles in s_tiles, first
// entry of the offset's row list or -1, its entries};
// s_tiles = the CTA's tiles in step order (when they fit; otherwise the walk reads the lists); a step
// of a row list stands there as its own number.
// The unit number is global: the units of an offset are consecutive.  After the unit records:
// s_plan[kWgradPlanUnits + f] = units of offset f over all CTAs, s_plan[kWgradPlanFirst + f] = the
// first of them.
constexpr int kWgradPlanUnits = 8 + 7 * kWgradMaxOffsets;
constexpr int kWgradPlanFirst = kWgradPlanUnits + kWgradMaxOffsets;
constexpr int kWgradPlanInts = kWgradPlanFirst + kWgradMaxOffsets;
static_assert(kWgradPlanInts <= 1280, "room reserved in shared memory");
constexpr int kWgradMaxOutTiles = 128; // (m, n) tiles of the weight gradient a launch can have
constexpr int kWgradCtlBase = 8 + 8 * kWgradMaxOutTiles;  // first per-(offset, tile) control word
constexpr int kWgradSharedSumUnits = 16;  // offsets with more units than this are summed by all CTAs together
template <int TILE_CAP>
__device__ __forceinline__ void wgrad_load_plan(const WgradParams &p, const int *lists, int list_stride, int *s_plan,
                                                int *s_tiles) {
  const int G = gridDim.x, c = blockIdx.x;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int cnt[4], P[4], c_first[4], S[4], U[4], T;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int f = 4 * lane + j;
      cnt[j] = (f < p.kv) ? __ldcg(p.sched + f) : 0;
    }
    wgrad_plan_warp(cnt, G, P, T, c_first, S, U);
    const int b0 = (int)(((long long)c * T) / G), b1 = (int)(((long long)(c + 1) * T) / G);
    const bool lists_rows = p.row_head && __ldcg(p.ctl + 1) == kWgradPlanRows;
    int has[4], k0[4], k1[4], len[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int f = 4 * lane + j;
      s_plan[kWgradPlanUnits + f] = S[j];
      s_plan[kWgradPlanFirst + f] = U[j];
      has[j] = (cnt[j] > 0 && c >= c_first[j] && c < c_first[j] + S[j]) ? 1 : 0;
      k0[j] = k1[j] = 0;
      if (has[j]) {
        k0[j] = max(b0, P[j]) - P[j];
        k1[j] = min(b1, P[j] + cnt[j]) - P[j];
        if (k1[j] < k0[j])
          k1[j] = k0[j];
      }
      len[j] = k1[j] - k0[j];
    }
    int slot[4], toff[4], n_units, total_len;
    wgrad_scan4(has, slot, n_units);
    wgrad_scan4(len, toff, total_len);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (has[j]) {
        int *e = s_plan + 8 + 7 * slot[j];
        e[0] = 4 * lane + j;
        e[5] = lists_rows ? __ldcg(p.row_head + 4 * lane + j) : -1;
        e[6] = lists_rows ? __ldcg(p.row_head + kWgradMaxOffsets + 4 * lane + j) : 0;
        e[1] = k0[j];
        e[2] = k1[j];
        e[3] = U[j] + (c - c_first[j]);
        e[4] = toff[j];
      }
    if (lane == 0) {
      s_plan[0] = n_units;
      s_plan[1] = total_len <= TILE_CAP ? 1 : 0;  // tiles are staged in shared memory
      s_plan[2] = lists_rows;
    }
  }
  __syncthreads();
  if (s_plan[1]) {
    const int n = s_plan[0];
    for (int j = 0; j < n; ++j) {
      const int *e = s_plan + 8 + 7 * j;
      const int *src = lists + (long long)e[0] * list_stride + e[1];
      for (int i = threadIdx.x; i < e[2] - e[1]; i += blockDim.x)
        s_tiles[e[4] + i] = e[5] >= 0 ? e[1] + i : __ldcg(src + i);
    }
  }
  __syncthreads();
}

// Rows of step `tile` of the unit e.
__device__ __forceinline__ int wgrad_step_rows(const WgradParams &p, const int *e, int tile) {
  return (e[5] >= 0 ? e[6] : p.n_rows) - tile * 128;
}

// Walk this CTA's units.  on_tile(tile, e, first_of_unit) for each step of the unit with record e,
// on_unit_end(u, f, n_tiles).  Every role runs the identical walk.
template <class TileFn, class EndFn>
__device__ __forceinline__ void wgrad_walk(const int *lists, int list_stride, const int *s_plan, const int *s_tiles,
                                           TileFn on_tile, EndFn on_unit_end) {
  const int n = s_plan[0];
  const bool staged = s_plan[1] != 0;
  for (int j = 0; j < n; ++j) {
    const int *e = s_plan + 8 + 7 * j;
    const int f = e[0], k0 = e[1], k1 = e[2], u = e[3], toff = e[4];
    const int *src = lists + (long long)f * list_stride + k0;
    for (int i = 0; i < k1 - k0; ++i) {
      const int tile = staged ? s_tiles[toff + i] : e[5] >= 0 ? k0 + i : __ldg(src + i);
      if (!on_tile(tile, e, i == 0))
        return;
    }
    if (!on_unit_end(u, f, k1 - k0))
      return;
  }
}

template <int BLOCK_N, int A_ATOMS, int GATHER>
__global__ void __launch_bounds__(WgradCfg<BLOCK_N, A_ATOMS, GATHER>::THREADS, 1)
wgrad_kernel(const __grid_constant__ CUtensorMap tmap_dout, const __grid_constant__ CUtensorMap tmap_x,
             const WgradParams p) {
  using Cfg = WgradCfg<BLOCK_N, A_ATOMS, GATHER>;
  extern __shared__ uint8_t smem_raw[];
  if (threadIdx.x == 0)
    CB2_TRACE_CTA(0, 0);
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
  uint8_t *smem = smem_raw + pad;
  const uint32_t sbase = raw_addr + pad;
  int *rowidx = reinterpret_cast<int *>(smem + Cfg::OFF_ROWIDX);
  int *s_plan = reinterpret_cast<int *>(smem + Cfg::OFF_SCHED);
  int *s_tiles = reinterpret_cast<int *>(smem + Cfg::OFF_TILES);
  volatile int *misc = reinterpret_cast<volatile int *>(smem + Cfg::OFF_MISC);
  volatile int *abort_flag = misc + 1;
  const uint32_t bars = sbase + Cfg::OFF_BARS;
  auto full_s = [&](int s) { return bars + 8u * s; };
  auto empty_s = [&](int s) { return bars + 8u * (Cfg::SA + s); };
  auto acc_full = [&](int s) { return bars + 8u * (Cfg::BAR_ACC_FULL + s); };
  auto acc_empty = [&](int s) { return bars + 8u * (Cfg::BAR_ACC_EMPTY + s); };
  const uint32_t final_bar = bars + 8u * Cfg::BAR_FINAL;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_tiles_n = (p.n_total + BLOCK_N - 1) / BLOCK_N;
  const int mt = blockIdx.y / n_tiles_n, nt = blockIdx.y % n_tiles_n;
  const int m0 = mt * 128, n0 = nt * BLOCK_N;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::SA; ++s) {
      mbar_init(full_s(s), Cfg::FULL_COUNT);
      mbar_init(empty_s(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(acc_full(s), 1);
      mbar_init(acc_empty(s), 128);
    }
    mbar_init(final_bar, 1);
    mbar_init_fence();
    misc[1] = 0;
    misc[2] = 1;
#ifndef CB2_TRACE_WGRAD_CTA
#define CB2_TRACE_WGRAD_CTA 0
#endif
    CB2_TRACE_SELECT(blockIdx.x == CB2_TRACE_WGRAD_CTA);
  }
  if (warp == 4) {
    tmem_alloc(sbase + Cfg::OFF_MISC, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  if (threadIdx.x == 0)
    CB2_TRACE_EVENT(5, 10, 0);
  // A plan that an earlier call made is read while the predecessor still runs, and so are the tables where it lists rows,
  // which says that they are as they were, too.  Whoever touches rows, partial sums, control words or the result waits
  // first; the next kernel may begin once this one's predecessor has ended.  (One call back to back, plan and tables read
  // behind the wait and before it, us: 2000 rows of a crop at 64 channels 15.0 and 14.2, scanned scenes of 9000 at 128 20.1
  // and 17.6, 100 003 at 64 30.5 and 28.3, 60 000 at 256 90 and 85, 150 000 uniform rows at 128 28.3 and 26.6, 960 000 106
  // and 102; forward, input and weight gradient of 20 000 uniform ones at 64 35.8 and 32.5.)
  if (!p.plan_fixed)
    grid_dep_wait();  // counts and lists come from the planning kernel
  wgrad_load_plan<Cfg::TILE_CAP>(p, p.lists, p.list_stride, s_plan, s_tiles);  // contains __syncthreads
  if (threadIdx.x == 0)
    CB2_TRACE_EVENT(5, 11, 0);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = static_cast<uint32_t>(misc[0]);

  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.status)
      atomicCAS(p.status, 0, code);
  };
  const int gy = gridDim.y;

  // ---- shared by the epilogue warps and the summing phase at the end
  const int *s_units = s_plan + kWgradPlanUnits;
  const int *s_first = s_plan + kWgradPlanFirst;
  constexpr int ROWS = Cfg::M_ROWS;
  constexpr int kTileF4 = ROWS * BLOCK_N / 4;  // float4 per [ROWS x BLOCK_N] tile
  // partial layout: float4 (col/4, row) at index (col/4) * ROWS + row, so that the 32 rows of a
  // warp touch 512 contiguous bytes
  auto partial_of = [&](int u) {
    return reinterpret_cast<float4 *>(p.partials) + ((long long)u * gy + blockIdx.y) * kTileF4;
  };
  auto ctl_of = [&](int f) { return p.ctl + kWgradCtlBase + 4 * ((long long)f * gy + blockIdx.y); };
  // dW[m0 + row, f, n0 + 4 * q .. + 3] from four sums
  auto write_out = [&](int f, int row, int q, float4 v) {
    const int m = m0 + row, n = n0 + 4 * q;
    if (m >= p.m_total || n >= p.n_total)
      return;
    const long long off = (long long)m * p.ldo + (long long)f * p.f_stride + n;
    float r[4] = {v.x, v.y, v.z, v.w};
    if (p.out_f32) {
      float *o = reinterpret_cast<float *>(p.out);
      const float *sp = reinterpret_cast<const float *>(p.src);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        o[off + j] = (p.beta != 0.f) ? __fmaf_rn(p.alpha, r[j], __fmul_rn(p.beta, sp[off + j])) : __fmul_rn(p.alpha, r[j]);
    } else {
      __half *o = reinterpret_cast<__half *>(p.out);
      const __half *sp = reinterpret_cast<const __half *>(p.src);
      __half h[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float t = (p.beta != 0.f) ? __fmaf_rn(p.alpha, r[j], __fmul_rn(p.beta, __half2float(sp[off + j])))
                                        : __fmul_rn(p.alpha, r[j]);
        h[j] = __float2half_rn(t);
      }
      *reinterpret_cast<uint2 *>(o + off) = *reinterpret_cast<const uint2 *>(h);
    }
  };
  if (warp < 4) {
    // ======================= epilogue: one fp32 partial per unit; the unit that completes an
    // offset marks it ready for the summing phase
    const int et = threadIdx.x;
    grid_dep_wait();
    grid_dep_launch();
    // Offsets inside the filter that no row tile carries get alpha * 0 + beta * source; CTA c
    // takes those with f = c (mod G).
    for (int f = blockIdx.x; f < p.kv; f += gridDim.x)
      if ((p.mode != kWgradMaskConv || ((p.mask_filter >> (f & 31)) & 1u)) && s_units[f] == 0)
        for (int q = 0; q < BLOCK_N / 4; ++q)
          write_out(f, et, q, make_float4(0.f, 0.f, 0.f, 0.f));  // rows past m_total are left out there
    int acc_use = 0;
    wgrad_walk(
        p.lists, p.list_stride, s_plan, s_tiles,
        [&](int, const int *, bool) -> bool { return true; },
        [&](int u, int f, int active) -> bool {
          float4 *dst = partial_of(u) + et;
          if (active == 0) {
            // a unit without tiles (fewer steps than CTAs) still owns a partial: all zeros
            for (int q = 0; q < BLOCK_N / 4 && et < ROWS; ++q)
              dst[q * ROWS] = make_float4(0.f, 0.f, 0.f, 0.f);
          } else {
            const int buf = acc_use & 1;
            if (et == 0) {
              CB2_TRACE_EVENT(4, 7, u);
              bool ok = mbar_wait(acc_full(buf), (acc_use >> 1) & 1, abort_flag);
              CB2_TRACE_EVENT(4, 8, u);  // accumulator complete
              misc[2] = ok ? 1 : 0;
              if (!ok)
                fail(kStatusWaitTimeout);
            }
            named_bar_sync(1, 128);
            if (misc[2] == 0)
              return false;
            tc_fence_after();
            const uint32_t trow = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) +
                                  static_cast<uint32_t>(buf * BLOCK_N);
#pragma unroll 1
            for (int round = 0; round < BLOCK_N / 32 && warp * 32 < ROWS; ++round) {
              uint32_t v[32];
              tmem_ld32(trow + round * 32, v);
              tmem_ld_wait();
#pragma unroll
              for (int q = 0; q < 8; ++q)
                reinterpret_cast<uint4 *>(dst)[(round * 8 + q) * ROWS] = make_uint4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
            }
            tc_fence_before();
            mbar_arrive(acc_empty(buf));
            ++acc_use;
          }
          // count the unit in; the one that completes the offset marks it ready
          __threadfence();  // this thread's part of the partial is visible before the unit counts
          named_bar_sync(1, 128);
          if (et == 0) {
            if (atomicAdd(ctl_of(f), 1) == s_units[f] - 1) {
              __threadfence();
              atomicOr(p.ctl + 9 + 8 * blockIdx.y + (f >> 5), 1 << (f & 31));  // ready: every partial of f is in place
            }
            CB2_TRACE_EVENT(4, 9, u);  // partial written
          }
          return true;
        });
  } else if (warp == 4) {
    // ======================= MMA issuer
    constexpr uint32_t idesc = make_idesc(0, true, true, 128, BLOCK_N);
    int stage = 0, acc_use = 0;
    uint32_t phase = 0;
    bool ok_all = true;
    grid_dep_wait();  // no operand comes before
    // The lane that issues.  Elected, the descriptors stay in uniform registers and a step costs the issuer a third:
    // 100 003 scanned rows at 64 channels 40.2 -> 35.3 us, 30 011 rows of 125 offsets 31.7 -> 27.4.  At the widest
    // tiles, three stages, it makes no difference but on the largest scenes, which it slows down (128 channels, lane 0
    // and elected: 20 000 scanned rows 23.9 and 23.5, 60 000 37.8 and 37.1, 100 003 50.8 and 50.7, 150 000 uniform ones
    // 30.9 and 31.0, 400 000 55.9 and 56.2, 960 000 104.5 and 106.6).
    auto issuer = [&]() { return Cfg::SA > 3 ? elect_one() : lane == 0; };
    const uint64_t adesc_base = make_smem_desc(sbase + Cfg::OFF_STAGES, 128 * 128, 1024);
    const uint64_t bdesc_base = make_smem_desc(sbase + Cfg::OFF_STAGES + Cfg::A_BYTES, 128 * 128, 1024);
    wgrad_walk(
        p.lists, p.list_stride, s_plan, s_tiles,
        [&](int tile, const int *e, bool first) -> bool {
          const int buf = acc_use & 1;
          // the warp walks together, its state the same in every lane; one lane issues
          bool ok = true;
          if (first)
            ok = mbar_wait(acc_empty(buf), ((acc_use >> 1) & 1) ^ 1, abort_flag);
          ok = ok && mbar_wait(full_s(stage), phase, abort_flag);
          if (!__all_sync(0xffffffffu, ok)) {
            if (lane == 0)
              fail(kStatusWaitTimeout);
            ok_all = false;
            return false;
          }
          if constexpr (GATHER == kGatherCpAsync)
            fence_proxy_async_smem();
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * BLOCK_N);
          // descriptors differ from the first stage's only in the start address (units of 16 bytes)
          const uint64_t adesc = adesc_base + static_cast<uint64_t>((stage * Cfg::STAGE_BYTES) >> 4);
          const uint64_t bdesc = bdesc_base + static_cast<uint64_t>((stage * Cfg::STAGE_BYTES) >> 4);
          const int rows = __shfl_sync(0xffffffffu, wgrad_step_rows(p, e, tile), 0);
          if (issuer()) {
            if (rows >= 128) {
#pragma unroll
              for (int ks = 0; ks < 8; ++ks)
                tc_mma<0>(d_tmem, adesc + ks * (2048 >> 4), bdesc + ks * (2048 >> 4), idesc, (first && ks == 0) ? 0u : 1u);
            } else {
              for (int ks = 0; ks < (rows + 15) / 16; ++ks)
                tc_mma<0>(d_tmem, adesc + ks * (2048 >> 4), bdesc + ks * (2048 >> 4), idesc, (first && ks == 0) ? 0u : 1u);
            }
            tc_commit(empty_s(stage));
            CB2_TRACE_EVENT(3, 6, tile);  // MMAs issued
          }
          __syncwarp();
          if (++stage == Cfg::SA) {
            stage = 0;
            phase ^= 1u;
          }
          return true;
        },
        [&](int, int, int active) -> bool {
          if (active > 0) {
            if (issuer())
              tc_commit(acc_full(acc_use & 1));
            __syncwarp();
            ++acc_use;
          }
          return true;
        });
    if (issuer()) {
      tc_commit(final_bar);  // every MMA has retired before the stages are used anew and TMEM is released
      if (!mbar_drain(final_bar, 0, kWaitLimitNs))
        fail(kStatusWaitTimeout);
    }
    __syncwarp();
  } else if constexpr (GATHER == kGatherTma4) {
    // ======================= gather both operands: the GW warps of group g own stage g, steps g,
    // g + SA, ... of this CTA.  A lane fetches a quad of four tile rows, one request per column block and
    // operand; a missing row is asked for out of bounds and reads as zeros.  The row numbers run ahead of the copies:
    // while the group waits for its stage, the neighbour indices of its next step and the sort order of
    // the one after are on their way.
    const int g = (warp - 5) / Cfg::GW;
    const int quad = (warp - 5) % Cfg::GW * (32 / Cfg::GW) + lane;
    const bool has_quad = lane < 32 / Cfg::GW;
    const bool first_lane = (warp - 5) % Cfg::GW == 0 && lane == 0;
    if (g < Cfg::SA) {
      const int n_units = s_plan[0];
      const bool staged = s_plan[1] != 0;
      bool dep_waited = s_plan[2] == 0;
      if (dep_waited)
        grid_dep_wait();  // the predecessor may have written the tables
      struct Step {
        int tile, f, list, rows;
      };
      int unit = 0, seen = 0;  // the unit `next_step` stands in, and the CTA's steps before it
      int at = g;              // the step `next_step` returns next
      auto next_step = [&]() -> Step {
        Step r = {-1, 0, -1, 0};
        while (unit < n_units) {
          const int *e = s_plan + 8 + 7 * unit;
          const int len = e[2] - e[1];
          if (at < seen + len) {
            const int k = at - seen;
            r.f = e[0];
            r.list = e[5];
            r.rows = e[6];
            r.tile = staged ? s_tiles[e[4] + k] : e[5] >= 0 ? e[1] + k : __ldg(p.lists + (long long)e[0] * p.list_stride + e[1] + k);
            break;
          }
          seen += len;
          ++unit;
        }
        at += Cfg::SA;
        return r;
      };
      struct Rows {
        int v[4];
      };
      const bool wide_order = (reinterpret_cast<uintptr_t>(p.mode == kWgradMaskConv ? p.argsort : p.a_inds) & 15u) == 0;
      // rows of dout (pair lists: of both operands) that lane's tile rows stand for
      auto load_order = [&](const Step &st, Rows &a) {
        const int r0 = st.tile * 128 + 4 * quad;
        const int *order = p.mode != kWgradMaskConv ? p.a_inds : st.list >= 0 ? p.rows + st.list : p.argsort;
        const int n = st.list >= 0 ? st.rows : p.n_rows;
        if (st.tile >= 0 && has_quad && (wide_order || st.list >= 0) && r0 + 4 <= n) {
          const int4 o = __ldg(reinterpret_cast<const int4 *>(order + r0));
          a.v[0] = o.x, a.v[1] = o.y, a.v[2] = o.z, a.v[3] = o.w;
          return;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          a.v[j] = -1;
          if (st.tile >= 0 && has_quad && r0 + j < n)
            a.v[j] = __ldg(order + r0 + j);
        }
      };
      auto load_rows = [&](const Step &st, const Rows &a, Rows &b) {
        const int r0 = st.tile * 128 + 4 * quad;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          b.v[j] = -1;
          if (st.tile >= 0 && has_quad && r0 + j < (st.list >= 0 ? st.rows : p.n_rows)) {
            if (p.mode == kWgradMaskConv) {
              // a chunk of at least a tile carries the offset, or the tile would not be in the list
              const bool on = st.list >= 0 || p.mask_width >= 128 ||
                              ((__ldg(p.rmask + (long long)((r0 + j) / p.mask_width) * p.words + (st.f >> 5)) >> (st.f & 31)) & 1u);
              if (on && a.v[j] >= 0)
                b.v[j] = __ldg(p.indices + (long long)st.f * p.n_rows + a.v[j]);
            } else {
              b.v[j] = __ldg(p.b_inds + r0 + j);
            }
          }
        }
      };
      const uint32_t a_quad = sbase + Cfg::OFF_STAGES + g * Cfg::STAGE_BYTES + quad * (4 * 128);
      const uint32_t b_quad = a_quad + Cfg::A_BYTES;
      Step cur = next_step(), nxt = next_step();
      Rows ca, cb, na, nb;
      load_order(cur, ca);
      load_order(nxt, na);
      load_rows(cur, ca, cb);
      uint32_t phase = 1;
      for (; cur.tile >= 0; phase ^= 1u) {
        const Step after = next_step();
        Rows fa;
        load_rows(nxt, na, nb);
        load_order(after, fa);
        int ia[4], ib[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          ib[j] = cb.v[j];
          ia[j] = (p.mode != kWgradMaskConv || ib[j] >= 0) ? ca.v[j] : -1;  // a zero B row makes the A row irrelevant
          if (ia[j] >= p.a_rows || ib[j] >= p.b_rows) {
            fail(kStatusBadIndex);
            ia[j] = ib[j] = -1;
          }
          ia[j] = row_or_zeros(ia[j], 4 * quad + j);
          ib[j] = row_or_zeros(ib[j], 4 * quad + j);
        }
        if (first_lane)
          CB2_TRACE_EVENT(g, 1, cur.tile + (ib[0] == 0x7fffffff));  // indices loaded
        if (!mbar_wait_warp(empty_s(g), phase, abort_flag)) {
          if (lane == 0)
            fail(kStatusWaitTimeout);
          break;
        }
        if (!dep_waited) {
          grid_dep_wait();
          dep_waited = true;
        }
        if (first_lane) {
          CB2_TRACE_EVENT(g, 2, cur.tile);  // stage free
          mbar_arrive_expect_tx(full_s(g), Cfg::STAGE_BYTES);
        }
        if (has_quad) {
#pragma unroll
          for (int ka = 0; ka < A_ATOMS; ++ka)
            tma_gather4(a_quad + ka * (128 * 128), &tmap_dout, full_s(g), m0 + ka * 64, ia[0], ia[1], ia[2], ia[3]);
#pragma unroll
          for (int kb = 0; kb < BLOCK_N / 64; ++kb)
            tma_gather4(b_quad + kb * (128 * 128), &tmap_x, full_s(g), n0 + kb * 64, ib[0], ib[1], ib[2], ib[3]);
        }
        if (first_lane)
          CB2_TRACE_EVENT(g, 3, cur.tile);  // copies issued
        cur = nxt, nxt = after;
        ca = na, cb = nb, na = fa;
      }
      mbar_drain(full_s(g), phase);  // the group's last copies
    }
  } else {
    // ======================= the same with 16-byte cp.async: group g of 128 threads owns stage g
    grid_dep_wait();
    const int g = (warp - 5) >> 2;
    const int gt = threadIdx.x - (5 * 32 + g * 128);
    int *group_rowidx = rowidx + g * 512;
    volatile int *my_flag = misc + 8 + 2 * g;  // per row buffer: a thread that runs ahead writes the other one
    int step = 0;
    const uint8_t *a_bytes = reinterpret_cast<const uint8_t *>(p.dout);
    const uint8_t *b_bytes = reinterpret_cast<const uint8_t *>(p.x);
    constexpr int CPR_B = BLOCK_N / 8;  // 16-byte chunks per B row (fp16)
    wgrad_walk(
        p.lists, p.list_stride, s_plan, s_tiles,
        [&](int tile, const int *e, bool) -> bool {
          const int f = e[0];
          const bool mine = (step % Cfg::SA) == g;
          const int use = step / Cfg::SA;
          ++step;
          if (!mine)
            return true;
          const int r = tile * 128 + gt;
          int ia = -1, ib = -1;
          if (e[5] >= 0) {
            if (r < e[6]) {
              ia = __ldg(p.rows + e[5] + r);
              ib = __ldg(p.indices + (long long)f * p.n_rows + ia);
            }
          } else if (r < p.n_rows) {
            if (p.mode == kWgradMaskConv) {
              const uint32_t word = __ldg(p.rmask + (long long)(r / p.mask_width) * p.words + (f >> 5));
              const int o = __ldg(p.argsort + r);  // independent of `word`: both loads are in flight together
              if ((word >> (f & 31)) & 1u) {
                ib = __ldg(p.indices + (long long)f * p.n_rows + o);
                ia = (ib >= 0) ? o : -1;  // a zero B row makes the A row irrelevant
              }
            } else {
              ia = __ldg(p.a_inds + r);
              ib = __ldg(p.b_inds + r);
            }
          }
          if (ia >= p.a_rows || ib >= p.b_rows) {
            fail(kStatusBadIndex);
            ia = ib = -1;
          }
          const uint32_t a_stage = sbase + Cfg::OFF_STAGES + g * Cfg::STAGE_BYTES;
          const uint32_t b_stage = a_stage + Cfg::A_BYTES;
          if (gt == 0) {
            CB2_TRACE_EVENT(g, 1, step - 1 + (ib == 0x7fffffff));  // indices loaded
            bool ok = mbar_wait(empty_s(g), (use & 1) ^ 1, abort_flag);
            CB2_TRACE_EVENT(g, 2, step - 1);             // stage free
            my_flag[use & 1] = ok ? 1 : 0;
            if (!ok)
              fail(kStatusWaitTimeout);
          }
          int *ridx_a = group_rowidx + (use & 1) * 256;
          int *ridx_b = ridx_a + 128;
          ridx_a[gt] = ia;
          ridx_b[gt] = ib;
          named_bar_sync(2 + g, 128);
          if (my_flag[use & 1] == 0)
            return false;
          {
            // A rows: 256 B (128 channels of dout starting at m0), 16 chunks per row
            const int c = gt & 15, row0 = gt >> 4;
            const bool col_ok = (m0 + c * 8) < p.m_total;
            const uint32_t dst_c = a_stage + (c >> 3) * (128 * 128);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int row = row0 + i * 8;
              const int ridx = ridx_a[row];
              const uint32_t dst = dst_c + (row >> 3) * 1024 + (row & 7) * 128 + (((c & 7) ^ (row & 7)) << 4);
              const bool valid = col_ok && ridx >= 0;
              const uint8_t *srcp = valid ? a_bytes + ((long long)ridx * p.ld_dout + m0 + c * 8) * 2 : a_bytes;
              cp_async_16(dst, srcp, valid ? 16u : 0u);
            }
          }
          {
            const int c = gt % CPR_B, row0 = gt / CPR_B;
            constexpr int RSTEP = 128 / CPR_B;
            const bool col_ok = (n0 + c * 8) < p.n_total;
            const uint32_t dst_c = b_stage + (c >> 3) * (128 * 128);
#pragma unroll
            for (int i = 0; i < CPR_B; ++i) {
              const int row = row0 + i * RSTEP;
              const int ridx = ridx_b[row];
              const uint32_t dst = dst_c + (row >> 3) * 1024 + (row & 7) * 128 + (((c & 7) ^ (row & 7)) << 4);
              const bool valid = col_ok && ridx >= 0;
              const uint8_t *srcp = valid ? b_bytes + ((long long)ridx * p.ld_x + n0 + c * 8) * 2 : b_bytes;
              cp_async_16(dst, srcp, valid ? 16u : 0u);
            }
          }
          // async arrive when this thread's copies land; the consumer fences (see rowconv kernel)
          cp_async_mbar_arrive_noinc(full_s(g));
          if (gt == 0)
            CB2_TRACE_EVENT(g, 3, step - 1);  // copies issued
          return true;
        },
        [&](int, int, int) -> bool { return true; });
    cp_async_wait_all();
  }

  // ---------------------------------------------------------------- summing
  // Every role has finished its walk; the whole CTA now sums partials.  Each output element is
  // summed by one thread in unit order -- for the offsets with many units: by sixteen warps, each
  // over every sixteenth unit, whose sums are combined in warp order.
  tc_fence_before();
  __syncthreads();
  grid_dep_wait();  // long over; the warps without a part in the above have not waited yet
  if (threadIdx.x == 0)
    CB2_TRACE_CTA(2, global_timer_ns());  // roles done
  if (*abort_flag == 0) {
    const int tid = threadIdx.x;
    float4 *s_part = reinterpret_cast<float4 *>(smem + Cfg::OFF_STAGES);  // the operand stages are idle now
    const long long ustride = (long long)gy * kTileF4;
    // this CTA's share of the offsets with many units: positions [c, c + 1) * kTileF4 / G in runs of 32
    const int q_begin = (int)(((long long)blockIdx.x * kTileF4) / gridDim.x) & ~31;
    const int q_end = blockIdx.x + 1 == gridDim.x ? kTileF4 : ((int)(((long long)(blockIdx.x + 1) * kTileF4) / gridDim.x) & ~31);
    // Which offsets this CTA helps to sum, and which positions of each: worked out once, by one
    // thread per offset, and packed in offset order (a CTA takes part in two or three offsets; a loop
    // over all of them, with its divisions run by every thread, cost more than the sums themselves).
    int *s_take = reinterpret_cast<int *>(smem + Cfg::OFF_ROWIDX);  // the row-index buffers are idle now
    {
      bool take = false;
      int lo = 0, hi = 0;
      unsigned ballot = 0;
      if (tid < 128) {
        const int f = tid;
        if (f < p.kv && s_units[f] > 0) {
          if (s_units[f] > kWgradSharedSumUnits) {
            lo = q_begin, hi = q_end;
            take = q_begin < q_end;
          } else {
            // an offset with few units belongs to a small group of neighbouring CTAs (the groups are
            // dealt out evenly over the grid), each summing an equal run of positions
            const int group = max(1, (int)gridDim.x / p.kv);
            const int member = (int)blockIdx.x - (f * (int)gridDim.x) / p.kv;
            take = member >= 0 && member < group;
            lo = ((member * kTileF4) / group) & ~1;
            hi = member + 1 == group ? kTileF4 : (((member + 1) * kTileF4) / group) & ~1;
          }
        }
        ballot = __ballot_sync(0xffffffffu, take);
        if (lane == 0)
          s_take[384 + warp] = static_cast<int>(ballot);
      }
      __syncthreads();
      if (tid < 128 && take) {
        int rank = __popc(ballot & ((1u << lane) - 1u));
        for (int w = 0; w < warp; ++w)
          rank += __popc(static_cast<uint32_t>(s_take[384 + w]));
        s_take[rank] = tid;
        s_take[128 + rank] = lo;
        s_take[256 + rank] = hi;
      }
      __syncthreads();
    }
    const int n_take = __popc(static_cast<uint32_t>(s_take[384])) + __popc(static_cast<uint32_t>(s_take[385])) +
                       __popc(static_cast<uint32_t>(s_take[386])) + __popc(static_cast<uint32_t>(s_take[387]));
    for (int i = 0; i < n_take; ++i) {
      const int f = s_take[i], lo = s_take[128 + i], hi = s_take[256 + i];
      const int S = s_units[f];
      const bool shared_sum = S > kWgradSharedSumUnits;
      if (tid == 0) {
        // bounded wait for the last unit of f
        const int *flag = p.ctl + 9 + 8 * blockIdx.y + (f >> 5);
        int ok = 1;
        unsigned long long t0 = 0;
        for (unsigned spin = 0; !((static_cast<uint32_t>(ld_acquire_gpu(flag)) >> (f & 31)) & 1u); ++spin) {
          __nanosleep(100);
          if ((spin & 63u) == 63u) {
            const unsigned long long now = global_timer_ns();
            if (t0 == 0)
              t0 = now;
            else if (now - t0 > kWaitLimitNs) {
              ok = 0;
              break;
            }
          }
        }
        if (!ok)
          fail(kStatusWaitTimeout);
        misc[6] = ok;
        CB2_TRACE_EVENT(6, 20, f);  // offset ready
      }
      __syncthreads();
      const bool ok = misc[6] != 0;
      __syncthreads();  // everybody has read the result before thread 0 writes the next one
      if (!ok)
        break;
      const float4 *src = partial_of(s_first[f]);
      if (!shared_sum) {
        // two positions per thread at a time, all units' loads of both in flight together
        for (int q0 = lo + 2 * tid; q0 < hi; q0 += 2 * Cfg::THREADS) {
          float4 acc[2];
#pragma unroll
          for (int g = 0; g < 2; ++g)
            acc[g] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
          for (int j = 0; j < S; ++j) {
            const float4 *sp = src + j * ustride + q0;
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              const float4 v = __ldcg(sp + g);
              acc[g].x += v.x;
              acc[g].y += v.y;
              acc[g].z += v.z;
              acc[g].w += v.w;
            }
          }
#pragma unroll
          for (int g = 0; g < 2; ++g)
            write_out(f, (q0 + g) % ROWS, (q0 + g) / ROWS, acc[g]);
        }
      } else {
        for (int q0 = lo; q0 < hi; q0 += 32) {
          if (warp < 16) {
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 *sp = src + q0 + lane;
#pragma unroll 8
            for (int j = warp; j < S; j += 16) {
              const float4 v = __ldcg(sp + j * ustride);
              acc.x += v.x;
              acc.y += v.y;
              acc.z += v.z;
              acc.w += v.w;
            }
            s_part[warp * 32 + lane] = acc;
          }
          __syncthreads();
          if (warp == 0) {
            float4 acc = s_part[lane];
#pragma unroll
            for (int w = 1; w < 16; ++w) {
              const float4 v = s_part[w * 32 + lane];
              acc.x += v.x;
              acc.y += v.y;
              acc.z += v.z;
              acc.w += v.w;
            }
            const int q = q0 + lane;
            write_out(f, q % ROWS, q / ROWS, acc);
          }
          __syncthreads();
        }
      }
      if (tid == 0)
        CB2_TRACE_EVENT(6, 21, f);  // summed
    }
  }
  // the last CTA to leave puts every control word back to zero for the next call
  if (threadIdx.x == 0) {
    __threadfence();
    misc[6] = atomicAdd(p.ctl, 1) == (int)(gridDim.x * gridDim.y) - 1 ? 1 : 0;
  }
  __syncthreads();
  if (misc[6]) {
    const int n_ctl = kWgradCtlBase + 4 * p.kv * gy;
    for (int i = threadIdx.x; i < n_ctl; i += Cfg::THREADS)
      if (i != 1)
        p.ctl[i] = 0;
    __threadfence();
  }
  if (threadIdx.x == 0)
    CB2_TRACE_CTA(1, 0);
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

} // namespace cb2
