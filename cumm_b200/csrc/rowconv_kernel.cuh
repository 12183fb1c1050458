// Row-gather implicit-GEMM kernel for sm_100a: forward and input-gradient of the
// mask-based sparse convolution, and the gather-GEMM-scatter GEMM (one filter offset with
// explicit row lists).  One persistent CTA per SM takes 128-row tiles of the (sorted)
// output rows from a scheduler warp (global ticket counter, ring of tiles in shared memory);
// for every filter offset present in the tile's OR-ed neighbour mask it gathers the 128
// operand rows into a 128-byte-swizzled shared-memory tile (TMA tile::gather4, a warp per 128-byte
// column block of a stage, or 16-byte cp.async; missing neighbours read as zeros), brings the
// matching weight slice in by TMA, and one thread issues tcgen05.mma into a TMEM accumulator.
// Eight (fp16) or sixteen (int8) epilogue warps read the accumulator back, apply
// alpha/beta/bias/activation (or the int8 requantisation) and write the rows to their scattered
// destinations, whole 32-byte sectors at a time.  No atomics on data: every
// output row is owned by exactly one tile.
//
// What it computes follows the reference kernel's control flow
// (cumm/conv/kernel.py:825-920, cumm/conv/sparse_iters.py:317-356,
// cumm/gemm/mask_iters.py:971-988, cumm/gemm/out_iters.py:541-553); how it computes it
// does not: the reference stages everything through registers and mma.sync.
#pragma once
#include "ptx.cuh"
#include <cuda.h>
#include <cuda_fp16.h>

namespace cb2 {

enum : int { kModeMaskConv = 0, kModeGatherGemm = 1 };
enum : int { kSrcNone = 0, kSrcRows = 1, kSrcVector = 2 };
enum : int { kStatusOk = 0, kStatusWaitTimeout = 1, kStatusBadIndex = 2 };

struct RowConvParams {
  const void *a;      // operand rows to gather  [a_rows, red]
  void *out;          // destination rows        [*, nn]
  const void *src;    // source rows for beta (same indexing as out) or a length-nn vector
  const float *scale; // int8 requantisation, per output channel
  const float *bias;  //   "
  const int32_t *indices;  // [kv, n_rows] (mask-conv mode)
  const uint32_t *mask;    // [n_rows, mask_words] sorted order
  const int32_t *argsort;  // [n_rows]
  uint32_t *mask_out;      // [tiles, mask_words] or null
  const int32_t *a_inds;   // gather-GEMM mode (null = identity)
  const int32_t *c_inds;   //   "
  int *status;             // device status word (0 = ok)
  int *tickets;            // two zero-initialised ints (next ticket, finished CTAs) or null = static round-robin
  long long lda, ldo, lds; // row strides in elements
  int n_rows;              // rows to produce (sorted positions, or m)
  int a_rows;              // rows available in `a`
  int red;                 // reduction width per filter offset
  int nn;                  // output width
  int kv;
  int n_parts;             // column parts of BLOCK_N that a row tile is computed in, each an item of its own
  int mask_words;          // 32-bit words per row mask: ceil(kv / 32), word w covers offsets 32w .. 32w+31
  int mode;
  int src_mode;
  int split;               // CTAs of a cluster that share an item's offsets (kernels with SPLIT)
  int tables_fixed;        // indices, mask and argsort are as an earlier call on this stream found them
  int skip_empty_tiles;    // input-gradient: a tile whose mask is 0 is left untouched
  int reverse_mask;
  uint32_t mask_filter;
  float alpha, beta, act_alpha;
  int act_type;
  uint32_t b_lbo, b_sbo;   // weight-tile descriptor offsets (bytes)
};

#ifndef CB2_ROWCONV_GROUP_THREADS
#define CB2_ROWCONV_GROUP_THREADS 128
#endif
#ifndef CB2_ROWCONV_RING
#define CB2_ROWCONV_RING 12
#endif
#ifndef CB2_ROWCONV_TICKET_BATCH
#define CB2_ROWCONV_TICKET_BATCH 4
#endif
#ifndef CB2_ROWCONV_NARROW_STAGES
#define CB2_ROWCONV_NARROW_STAGES 7
#endif
#ifndef CB2_ROWCONV_WIDE_STAGES
#define CB2_ROWCONV_WIDE_STAGES 4
#endif
#ifndef CB2_ROWCONV_EPI_PARTS
#define CB2_ROWCONV_EPI_PARTS 4
#endif

// TMA_GATHER: operand rows are fetched by the TMA unit (tile::gather4, four rows per request, a warp per
// 128-byte column block of a stage) instead of 16-byte cp.async issued by 128 threads per group (see run_rowconv for
// which).  The copy engine path keeps the load/store queues of the SM free for
// the other roles and leaves the kernel of wide rows at 19 warps instead of 23.  (Rows of 256 bytes, cp.async
// and gather4, forward: 150 000 uniform rows 28.3 and 26.3 us, 960 000 93.3 and 87.5, 60 000 scanned rows at
// 256 channels 124 and 112.)
// MASK_WORDS: mask words per row the ring slots have room for (1: kernel volumes up to 32; 4: up
// to 128, the reference's "dynamic mask" kernels, cumm/gemm/blockmma/mma.py:78-270).
template <int KIND, int NATOM_K, int BLOCK_N, bool B_MN, bool TMA_GATHER, int MASK_WORDS = 1> struct RowConvCfg {
  static constexpr int ES = KIND == 0 ? 2 : 1;            // operand element bytes
  static constexpr int OES = KIND == 0 ? 2 : 1;           // output element bytes
  static constexpr int ATOM_ELEMS = 128 / ES;             // elements per 128-byte swizzle row
  static constexpr int UMMA_K = 32 / ES;
  static constexpr int KRED = NATOM_K * ATOM_ELEMS;       // reduction elements per stage
  static constexpr int TILE_M = 128;
  // What bounds a step is not the bytes of a stage but how many steps are on their way, so narrow fp16 rows
  // have seven stages (forward of 100 003 scanned rows at 64 channels: seven 24.1, eight 24.4, nine 24.9 us; 125 offsets,
  // 30 011 rows: 44.7, 43.5, 43.5; 20 000 uniform rows 8.5, 8.4, 8.4) and wide fp16 rows
  // four, which is what the shared memory holds.  int8 keeps five beside sixteen epilogue warps: its stages
  // hold the weights too.
  static constexpr int SA =
      TMA_GATHER && NATOM_K == 1 ? (KIND == 1 ? (BLOCK_N >= 128 ? 5 : 6) : CB2_ROWCONV_NARROW_STAGES)
                                 : (KIND == 0 ? CB2_ROWCONV_WIDE_STAGES : 3);
  // Groups that gather: one per stage with the copy engine.  Groups of four warps (cp.async) are three, whatever
  // the stages, and take the steps in turn: their copies are asynchronous, so a group fills a stage while its
  // last is on the way.
  static constexpr int GROUPS = TMA_GATHER ? SA : 3;
  static constexpr int A_STAGE_BYTES = TILE_M * 128 * NATOM_K;
  static constexpr int ROWIDX_BYTES = TMA_GATHER ? 0 : GROUPS * 2 * 128 * 4;  // row numbers pass through registers
  static constexpr int B_SLOT_BYTES = BLOCK_N * 128 * NATOM_K;
  static constexpr int MW = MASK_WORDS;
  // Outputs wider than BLOCK_N: column parts drawn with the tiles (fp16), or one grid row per part
  // (int8, whose sixteen epilogue warps have no register to spare for a part that changes).
  static constexpr bool PARTS = KIND == 0;
  // tile ring slots (four mask words beside wide rows: what is left)
  static constexpr int RING = MASK_WORDS == 1 ? CB2_ROWCONV_RING
                              : KIND == 0 && NATOM_K == 2 ? CB2_ROWCONV_RING / 2 - 1 : CB2_ROWCONV_RING / 2;
  // fp16: each epilogue warp turns its 32 rows of 64 bytes around in 2 KB of its own before they are stored
  // (600 000 uniform rows, forward: 50.5 -> 44.5 us at 64 channels, 74.5 -> 71.4 at 128).  int8 rows are half
  // as long and their registers all taken: each thread stores its own 32 bytes.
  static constexpr int EPI_WARP_BYTES = KIND == 0 ? 32 * 64 : 0;
  static constexpr int EPI_BYTES = 8 * EPI_WARP_BYTES;
  static constexpr bool DEALT = KIND == 0;  // a CTA's first ticket is its own number
  // steps a CTA may hold (drawn, not issued) and still draw: what a ticket, the tile's words, its indices and its first
  // rows take.  (6, 8, 12, 16: 100 003 scanned rows at 64 channels 33.6, 30.4, 27.6, 27.7 us, 150 000 at 128 65.9,
  // 64.5, 64.5, 64.7, 150 000 uniform ones 22.0, 21.7, 22.0, 22.4.)
  static constexpr int STEP_BUDGET = NATOM_K == 1 ? 12 : 8;
  static constexpr int RING_SLOT_INTS = 136 + 128 * MASK_WORDS;  // header; 128 gather rows; 128 output rows / row masks
  // int8 rows of up to 128 bytes: a stage holds the step's weight tile beside its rows, under the same pair
  // of barriers -- one wait and one commit per step for the issuer (46.7 -> 43.7 us for the stride-2
  // layer; the weights of a run of tiles with the same offset come from L2 each time).  fp16 keeps slots
  // of their own: there it lost (135 -> 144 us for the scanned scene's step).
  static constexpr bool JOINT = KIND == 1 && TMA_GATHER && NATOM_K == 1;
  // mbarriers: operand stages, accumulators, the final one, weight slots, tile ring
  static constexpr int BAR_EMPTY_A = SA, BAR_ACC_FULL = 2 * SA, BAR_ACC_EMPTY = BAR_ACC_FULL + 2,
                       BAR_FINAL = BAR_ACC_EMPTY + 2, BAR_FULL_B = BAR_FINAL + 1, BAR_EMPTY_B = BAR_FULL_B + 6,
                       BAR_RING = (BAR_EMPTY_B + 6 + 1) / 2 * 2;
  // Weight slots: as many as fit (2 to 6).  A tile whose mask carries many offsets needs a new
  // weight tile every step, and with two slots the L2 latency of that load bounds the step.
  static constexpr int FIXED_BYTES = SA * A_STAGE_BYTES + ROWIDX_BYTES + EPI_BYTES +
                                     2 * BLOCK_N * 4 + RING * RING_SLOT_INTS * 4 + (BAR_RING + 3 * RING) * 8 + 64 + 1024;
  static constexpr int SB_FIT = (232448 - FIXED_BYTES) / B_SLOT_BYTES;
  static constexpr int SB = JOINT ? SA : SB_FIT < 2 ? 2 : (SB_FIT > 6 ? 6 : SB_FIT);
  static constexpr int NUM_ACC = 2;                       // TMEM accumulators: one fills while one drains
  static constexpr int TMEM_COLS = NUM_ACC * BLOCK_N;     // 128 or 256: power of two >= 32
  // Epilogue: several threads per tile row, each converting its share of the columns.  The
  // conversion is a chain of dependent fixed-latency instructions, so its rate is set by how
  // many warps each SM sub-partition can switch between, not by arithmetic throughput.
  static constexpr int EPI_HALVES = (KIND == 1 && BLOCK_N >= 128) ? CB2_ROWCONV_EPI_PARTS : 2;
  static constexpr int EPI_THREADS = 128 * EPI_HALVES;
  // Groups of epilogue warps that take turns at the tiles: a requantised tile is a long chain per warp
  // (read, convert, scale, convert, pack, store), and two tiles on their way at once fill its gaps
  // (stride-2 int8 layer, 3839 tiles: 43.7 -> 42.1 us).  Each group owns one accumulator: it waits for and
  // gives back every use of that one, in order, so that a barrier's parity never lies two uses back.
  static constexpr int EPI_GROUPS = (KIND == 1 && BLOCK_N >= 128) ? 2 : 1;
  static_assert(EPI_GROUPS == 1 || EPI_GROUPS == NUM_ACC, "an accumulator belongs to one group");
  static_assert(EPI_BYTES == EPI_WARP_BYTES * EPI_THREADS / 32 || KIND == 1, "every epilogue warp has its bytes");
  static constexpr int GROUP_THREADS = TMA_GATHER ? 32 * NATOM_K : CB2_ROWCONV_GROUP_THREADS;
  static constexpr int FULL_A_COUNT = JOINT ? 2 : TMA_GATHER ? NATOM_K : GROUP_THREADS;
  static constexpr int MMA_WARP = EPI_THREADS / 32;
  static constexpr int TMA_WARP = MMA_WARP + 1;
  static constexpr int FIRST_GATHER_WARP = TMA_WARP + 1;
  static constexpr int SCHED_WARP = FIRST_GATHER_WARP + GROUPS * GROUP_THREADS / 32;  // the last warp hands out tiles
  static constexpr int THREADS = (SCHED_WARP + 1) * 32;
  static constexpr int RING_CONSUMER_WARPS = SCHED_WARP;   // every warp but the scheduler
  static constexpr int CLEARED_THREADS = EPI_THREADS + GROUPS * GROUP_THREADS;  // SPLIT: stages cleared, sums may come
  // shared memory map (offsets from a 1024-byte aligned base)
  static constexpr int OFF_A = 0;
  static constexpr int OFF_B = OFF_A + SA * A_STAGE_BYTES;
  static constexpr int OFF_EPI = OFF_B + SB * B_SLOT_BYTES;          // EPI_WARP_BYTES per epilogue warp
  static constexpr int OFF_ROWIDX = OFF_EPI + EPI_BYTES;             // ROWIDX_BYTES
  static constexpr int OFF_SCALE = OFF_ROWIDX + ROWIDX_BYTES;  // 2 * BLOCK_N floats
  static constexpr int OFF_RING = OFF_SCALE + 2 * BLOCK_N * 4;       // RING slots
  static constexpr int OFF_BARS = OFF_RING + RING * RING_SLOT_INTS * 4;  // BAR_RING + 3 * RING mbarriers
  static constexpr int OFF_MISC = OFF_BARS + (BAR_RING + 3 * RING) * 8;  // tmem ptr, abort, flags
  static constexpr int SMEM_BYTES = OFF_MISC + 64 + 1024;            // + alignment slack
  static_assert(SMEM_BYTES <= 232448, "shared memory budget of one CTA exceeded");
  static_assert(SB <= 6, "the barrier table holds six weight slots");
  static_assert(NUM_ACC == 2, "the barrier table holds two accumulators");
};

__device__ __forceinline__ float apply_act(float x, int act_type, float act_alpha) {
  switch (act_type) {
  case 1:
    return fmaxf(x, 0.f);
  case 2:
    return 1.f / (1.f + expf(-x));
  case 3:
    return x >= 0.f ? x : x * act_alpha;
  default:
    return x;
  }
}

// Four floats -> four int8 in one word, round-to-nearest-even, saturating, NaN -> 0 (what
// cvt.rni.sat.s8.f32 returns for each): to int32 first (NaN -> 0, saturating at the int32 range),
// then two saturating packs of two values each -- the reference's packed converter
// (include/tensorview/gemm/math/numeric_convert.h:1107-1138).  Six instructions per four values;
// a clamp-and-magic-add form in the arithmetic pipes took eleven and measured 4 % slower on the
// stride-2 int8 convolution: the kernel is bound by instruction issue, not by a pipe.
__device__ __forceinline__ uint32_t cvt_pack4_s8(float a, float b, float c, float d) {
  int ia, ib, ic, id;
  asm("cvt.rni.s32.f32 %0, %1;" : "=r"(ia) : "f"(a));
  asm("cvt.rni.s32.f32 %0, %1;" : "=r"(ib) : "f"(b));
  asm("cvt.rni.s32.f32 %0, %1;" : "=r"(ic) : "f"(c));
  asm("cvt.rni.s32.f32 %0, %1;" : "=r"(id) : "f"(d));
  uint32_t hi, out;
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, 0;" : "=r"(hi) : "r"(id), "r"(ic));       // bytes {c, d}
  asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(out) : "r"(ib), "r"(ia), "r"(hi));  // {a, b, c, d}
  return out;
}

// Tiles are handed out by one scheduler warp per CTA through a small shared-memory ring.
// A slot holds {tile, OR-ed neighbour mask of the tile, first output column, the 128 rows the
// gather starts from, the 128 destination rows}.  Outputs wider than BLOCK_N are cut into column
// parts; an item is one part of one tile, and the parts of a tile are drawn one after the other, by
// different CTAs at about the same time, so that the operand rows are fetched from memory once.  With `tickets` the scheduler draws tiles from a global counter
// (dynamic scheduling: a tile whose mask carries many offsets costs many steps, and a static
// split leaves the CTAs that own such tiles running long after the others), last tiles of
// the sorted order first because those carry the most offsets.
struct RingView {
  int *slots;
  uint32_t full0, empty0;  // addresses of the first "published" / "released" barrier
  uint32_t landed0;        // first "copies landed" barrier (scheduler only)
  int ring, slot_ints;
  volatile int *abort_flag;
  __device__ __forceinline__ int *slot(int i) const { return slots + i * slot_ints; }
};

// OR of the neighbour masks of a tile's rows, word by word, from the raw mask words of its ring
// slot (warp-collective); returns the number of filter offsets present.
template <int MW>
__device__ __forceinline__ int ring_tile_masks(const RowConvParams &p, const int *sl, int tile, uint32_t (&km)[MW]) {
#pragma unroll
  for (int w = 0; w < MW; ++w)
    km[w] = 0u;
  if (tile < 0 || p.mode != kModeMaskConv) {
    km[0] = 1u;
    return 1;
  }
  const int lane = (int)lane_id();
  int count = 0;
#pragma unroll
  for (int w = 0; w < MW; ++w) {
    if (w < p.mask_words) {
      uint32_t m = 0;
      if constexpr (MW == 1) {
        const int4 m4 = *reinterpret_cast<const int4 *>(sl + 136 + 4 * lane);  // four rows' words in one load
        m = static_cast<uint32_t>(m4.x | m4.y | m4.z | m4.w);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          m |= static_cast<uint32_t>(sl[136 + (i * 32 + lane) * MW + w]);
      }
      m = __reduce_or_sync(0xffffffffu, m) & p.mask_filter;
      const int left = p.kv - 32 * w;  // offsets this word covers
      if (left < 32)
        m &= left > 0 ? (1u << left) - 1u : 0u;
      km[w] = m;
      count += __popc(m);
    }
  }
  return count;
}

// Walks the tiles the scheduler publishes; every consumer warp of the CTA has one and runs the
// identical walk, so their step counters agree.  next() reads a tile's header into registers, the same
// in every lane, lets the role read its rows and gives the slot back at once; the role loops over the
// tile's (filter offset, reduction pass) steps itself.  (With slots held until a tile has been issued
// the look-ahead was too short for tiles with many offsets: 148 instead of 135 us for a training step of
// a scanned scene at 64 channels.)  Every lane polls for itself: with one lane polling and a shuffle the
// forward pass of 960 000 uniform rows took 121 instead of 104 us.
template <int MW> struct TileCursor {
  static_assert(MW == 1 || MW == 4, "one mask word, or four");
  int slot = 0;
  uint32_t phase = 0;
  int tile, n0;
  int offsets;  // filter offsets present
  // the offsets still to be taken, bit i = weight offset i (reverse_mask has been applied)
  uint32_t m;
  unsigned long long lo, hi;  // four words
  // Returns 1 on a tile, 0 at the end, -1 when the wait gave up.  read(slot) runs before the slot is
  // given back.  ALONE: one thread walks for its warp (the MMA issuer).  UNDER: the role walks before the predecessor's
  // end, and the scheduler may wait for that.
  template <bool ALONE = false, bool UNDER = false, class ReadFn>
  __device__ __forceinline__ int next(const RowConvParams &p, const RingView &rv, ReadFn read) {
    const bool ok = mbar_wait<UNDER>(rv.full0 + 8u * slot, phase, rv.abort_flag);
    auto same = [](auto v) {
      if constexpr (ALONE)
        return v;
      else
        return __shfl_sync(0xffffffffu, v, 0);
    };
    if (ALONE ? !ok : !__all_sync(0xffffffffu, ok))
      return -1;
    const int *sl = rv.slot(slot);
    const int4 head = *reinterpret_cast<const int4 *>(sl);
    tile = same(head.x);
    n0 = same(head.w);
    if constexpr (MW == 1) {
      m = same(static_cast<uint32_t>(head.y));
      if (p.reverse_mask)
        m = __brev(m) >> (32 - p.kv);
      offsets = __popc(m);
    } else {
      const int4 w = *reinterpret_cast<const int4 *>(sl + 4);
      auto join = [](int a, int b) {
        return (static_cast<unsigned long long>(static_cast<uint32_t>(b)) << 32) | static_cast<uint32_t>(a);
      };
      lo = same(join(w.x, w.y));
      hi = same(join(w.z, w.w));
      if (p.reverse_mask) {  // 128 bits reversed, then shifted down by 128 - kv
        const unsigned long long rl = __brevll(hi), rh = __brevll(lo);
        const int s = 128 - p.kv;
        lo = s >= 64 ? rh >> (s - 64) : (s == 0 ? rl : (rl >> s) | (rh << (64 - s)));
        hi = s >= 64 ? 0ull : rh >> s;
      }
      offsets = __popcll(lo) + __popcll(hi);
    }
    read(sl);
    if constexpr (!ALONE)
      __syncwarp();
    if (ALONE || lane_id() == 0)
      mbar_arrive(rv.empty0 + 8u * slot);
    if (++slot == rv.ring) {
      slot = 0;
      phase ^= 1u;
    }
    return tile >= 0 ? 1 : 0;
  }
  __device__ __forceinline__ int first_offset() const {
    if constexpr (MW == 1)
      return __ffs(m) - 1;
    else
      return lo ? __ffsll(lo) - 1 : 63 + __ffsll(hi);
  }
  __device__ __forceinline__ int last_offset() const {
    if constexpr (MW == 1)
      return 31 - __clz(m);
    else
      return hi ? 127 - __clzll(hi) : 63 - __clzll(lo);
  }
  __device__ __forceinline__ int take() {
    const int f = first_offset();
    if constexpr (MW == 1)
      m &= m - 1;
    else if (lo)
      lo &= lo - 1;
    else
      hi &= hi - 1;
    return f;
  }
};

// The scheduler warp: draws tiles and fetches their mask words and row numbers straight into
// a ring slot with 4-byte cp.async.  The slot's "landed" barrier is completed by the copies
// themselves (one asynchronous arrival per lane), so any number of tiles can be in flight and
// each is published -- its OR-ed mask computed once, here -- as soon as ITS words are there.
// Slot layout (ints): [0] tile (-1 = no more tiles), [3] first output column, [1] OR-ed mask (with several mask words per
// row: the OR of all of them, and the OR-ed words themselves at [4, 4 + MW)), [2] steps charged
// for the tile (scheduler only), [8,136) rows the gather starts from, from 136 on the destination
// rows in gather-GEMM mode / the rows' raw mask words (MW per row) in conv mode (in conv mode the
// destination rows are the gather rows).
__device__ __forceinline__ void cp_async_4(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// An L2 prefetch of the first tile's words runs while the CTA sets up its barriers and tensor memory.
// `progress` (shared memory): steps that the MMA issuer has issued, tiles without an offset counted as one.
// `first`, `dealt`: see below.  WAIT_FIRST: a convolution's tables are read behind the predecessor's end, unless the caller
// knows them to be as they were.  SPLIT: the CTA's cluster has one item, and this CTA every split-th of its offsets.  `split_state` (shared memory)
// becomes what that makes of the CTA; it stays kSplitUnknown in one that gives up before its item is known.
// (Items of up to 0, 3 and 7 offsets kept, forward, before launches overlapped, us: 1900 and 4000 uniform rows at 64 channels 8.4, 6.9, 6.9 and 9.1, 7.7,
// 7.7; 8 offsets, 3800 rows at 64 and 128 9.6, 9.6, 9.2 and 10.9, 10.9, 11.4.)
constexpr int kSplitSoloOffsets = 3;
enum SplitState {
  kSplitUnknown = 0,
  kSplitSolo,     // the item has so few offsets that the first CTA keeps them all: the exchange would cost more than they do
  kSplitNothing,  // shared, none of the offsets is this CTA's
  kSplitSums      // shared, the epilogue warps leave this CTA's sums in shared memory and count themselves
};
template <int MW, bool SPLIT, int STEP_BUDGET, bool WAIT_FIRST>
__device__ __forceinline__ void scheduler_run(const RowConvParams &p, const RingView &rv, int ntiles, int block_n,
                                              int kpasses, int first, int dealt, volatile int *progress,
                                              volatile int *split_state) {
  const int nitems = ntiles * p.n_parts;
  const int lane = (int)lane_id();
  const bool dynamic = !SPLIT && p.tickets != nullptr && gridDim.y == 1;
  const bool conv = p.mode == kModeMaskConv;
  int drawn = 0;
  // `first` is the CTA's first ticket, the others come from the counter, which begins behind the `dealt` ones that
  // every CTA has as its own number.  Where tiles are light they come
  // in batches and the next batch is requested before the current one is used up: the counter's round trip through
  // L2 would otherwise be paid per tile.  Batches shrink to one ticket as the counter nears the end so the tail stays
  // balanced.  A ticket that is on its way is a tile nobody else can take, so that heavy tiles are asked for
  // one at a time and not before the CTA is about to need one.  (Ahead of time for tiles of up to 2, 4, 6 and 12 steps:
  // 100 003 scanned rows at 64 channels 27.8, 28.2, 30.4, 30.2 us, 60 000, 104 to 72, 39.9, 39.9, 42.3, 45.7.)
  constexpr int MAX_BATCH = CB2_ROWCONV_TICKET_BATCH;
  int cur_base = first, cur_left = 1, next_base = 0, next_cnt = 0;
  auto request = [&](int seen, int last_steps) {
    // (the first tiles carry the most offsets: four of those in one hand set the length of a launch)
    int b = last_steps > 2 ? 1 : (nitems - seen) / ((int)gridDim.x * 4);
    next_cnt = b < 1 ? 1 : (b > MAX_BATCH ? MAX_BATCH : b);
    if (lane == 0)
      next_base = dealt + atomicAdd(p.tickets, next_cnt);
  };
  auto draw = [&](int last_steps) -> int {
    int t;
    if (dynamic) {
      if (cur_left == 0) {
        if (next_cnt == 0)
          request(cur_base, last_steps);
        cur_base = __shfl_sync(0xffffffffu, next_base, 0);
        cur_left = next_cnt;
        next_cnt = 0;
        if (cur_base < nitems && last_steps <= 2)
          request(cur_base, last_steps);
      }
      t = cur_base++;
      --cur_left;
    } else if (SPLIT) {
      t = drawn == 0 ? (int)blockIdx.x / p.split : nitems;
    } else {
      t = blockIdx.x + drawn * gridDim.x;
    }
    ++drawn;
    return t;
  };
  const uint32_t slots_addr = smem_u32(rv.slots);
  // Tiles a CTA has drawn cannot be taken over by an idle CTA, so the look-ahead is bounded by
  // WORK, not by tiles: a CTA draws while the steps it holds (one per offset in a tile's mask, until
  // they have been issued) are within STEP_BUDGET.  Until a tile's mask has landed it is
  // charged what the previous tiles cost, half-way back to it where the last was lighter, and the very first one is
  // charged the whole budget: a CTA learns what its first tile weighs before it takes a second.  (Forward, us, tiles held
  // until every role had read them, then until issued, then with charges that remember heavier tiles: 60 000 scanned
  // rows, 104 to 72 channels, 48.1, 48.6, 39.4, 150 000 at 128 70.1, 74.1, 64.5, 100 003 at 64 30.5, 31.2, 27.8; 125 offsets,
  // 30 011 rows 59.7, 52.6, 52.4.)
  int issued = 0, accounted = 0, released = 0, drawn_steps = 0;
  int item_tile = -1;  // SPLIT: the tile whose mask words this CTA reports, and those words
  uint32_t item_mask[MW] = {};
  int guess = (conv && dynamic) ? STEP_BUDGET + 1 : 1;
  // The scheduler's own instructions are what paces a CTA whose tiles carry one offset each: every
  // poll here is made by all lanes at once (a vote instead of a test by one lane and a shuffle), and releases are only looked at when the
  // CTA could not draw otherwise.
  auto account = [&]() {
    while (accounted < issued &&
           __any_sync(0xffffffffu, mbar_poll(rv.landed0 + 8u * (accounted % rv.ring), (accounted / rv.ring) & 1))) {
      int *sl = rv.slot(accounted % rv.ring);
      uint32_t km[MW];
      int offsets = ring_tile_masks<MW>(p, sl, sl[0], km);
      if constexpr (SPLIT) {
        if (sl[0] >= 0) {
          const int rank = (int)cluster_rank();
          item_tile = rank == 0 && p.mask_out && sl[3] == 0 ? sl[0] : -1;
#pragma unroll
          for (int w = 0; w < MW; ++w)
            item_mask[w] = km[w];  // forward: not reversed
          const bool alone = offsets <= kSplitSoloOffsets;
          int before = 0, kept = 0;
#pragma unroll
          for (int w = 0; w < MW; ++w) {  // lane l has bit l
            const int at = before + __popc(km[w] & ((1u << lane) - 1u));
            const bool mine = ((km[w] >> lane) & 1u) && (alone ? rank == 0 : at % p.split == rank);
            before += __popc(km[w]);
            km[w] = __ballot_sync(0xffffffffu, mine);
            kept += __popc(km[w]);
          }
          offsets = kept;
          if (lane == 0)
            *split_state = alone ? kSplitSolo : kept ? kSplitSums : kSplitNothing;
        }
      }
      const int nsteps = (sl[0] >= 0) ? max(1, offsets * kpasses) : 1;
      drawn_steps += nsteps - sl[2];
      __syncwarp();
      if (lane == 0) {
        uint32_t any = 0;
#pragma unroll
        for (int w = 0; w < MW; ++w) {
          any |= km[w];
          if (MW > 1)
            sl[4 + w] = static_cast<int>(km[w]);
        }
        sl[1] = static_cast<int>(any);
        CB2_TRACE_EVENT(6, 14, sl[0]);  // tile published
        mbar_arrive(rv.full0 + 8u * (accounted % rv.ring));
      }
      __syncwarp();
      guess = accounted == 0 ? nsteps : max(nsteps, (guess + nsteps) / 2);
      ++accounted;
    }
  };
  auto account_released = [&]() {
    while (released < accounted &&
           __any_sync(0xffffffffu, mbar_poll(rv.empty0 + 8u * (released % rv.ring), (released / rv.ring) & 1))) {
      ++released;
    }
  };
  auto within_budget = [&]() { return SPLIT || __any_sync(0xffffffffu, drawn_steps - *progress <= STEP_BUDGET); };
  auto can_draw = [&]() { return issued - released < rv.ring && within_budget(); };
  // tables whose tiles can be fetched with two 16-byte copies per lane
  const bool wide_copies = conv && MW == 1 && p.mask_words == 1 &&
                           ((reinterpret_cast<uintptr_t>(p.argsort) | reinterpret_cast<uintptr_t>(p.mask)) & 15u) == 0;
  if (WAIT_FIRST && conv && !p.tables_fixed)
    grid_dep_wait();  // the predecessor may have written the tables; who gathers learns its rows from here
  bool ended = false;
  for (;;) {
    account();
    bool may_draw = can_draw();
    if (!may_draw) {
      account_released();
      may_draw = can_draw();
    }
    if (!may_draw) {
      // first learn what the tiles in flight weigh, then wait for the oldest one to be read or for steps to be issued
      bool ok = true;
      if (accounted < issued)
        ok = mbar_wait_warp(rv.landed0 + 8u * (accounted % rv.ring), (accounted / rv.ring) & 1, rv.abort_flag);
      else if (issued - released >= rv.ring)
        ok = mbar_wait_warp<true>(rv.empty0 + 8u * (released % rv.ring), (released / rv.ring) & 1, rv.abort_flag);
      else if constexpr (!SPLIT)
        ok = wait_for([&]() { return within_budget(); }, rv.abort_flag);
      if (!ok)
        break;  // gave up
      continue;
    }
    const int si = issued % rv.ring;
    const int ticket = draw(guess);
#ifndef CB2_TRACE_TICKET
#define CB2_TRACE_TICKET 0  // 0: follow the CTA that got the heaviest tile
#endif
    if (ticket == CB2_TRACE_TICKET && lane == 0)
      CB2_TRACE_SELECT(1);
    int tile = -1, part = 0;
    if (ticket < nitems) {
      tile = ticket;
      if (p.n_parts > 1) {
        tile = ticket / p.n_parts;
        part = ticket - tile * p.n_parts;
      }
      if (conv)
        tile = ntiles - 1 - tile;  // the last tiles of the sorted order carry the most offsets
    }
    int *sl = rv.slot(si);
    const uint32_t sa = slots_addr + static_cast<uint32_t>(si * rv.slot_ints) * 4u;
    if (lane == 0) {
      sl[0] = tile;
      sl[2] = guess;
      sl[3] = part * block_n;
    }
    drawn_steps += guess;
    if (wide_copies && tile >= 0 && (tile + 1) * 128 <= p.n_rows) {
      cp_async_16(sa + (8 + 4 * lane) * 4, p.argsort + tile * 128 + 4 * lane, 16u);
      cp_async_16(sa + (136 + 4 * lane) * 4, p.mask + tile * 128 + 4 * lane, 16u);
    } else
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int j = i * 32 + lane;
      const int r = tile * 128 + j;
      if (tile >= 0 && r < p.n_rows) {
        if (conv) {
          cp_async_4(sa + (8 + j) * 4, p.argsort + r);
#pragma unroll
          for (int w = 0; w < MW; ++w)
            if (w < p.mask_words)
              cp_async_4(sa + (136 + j * MW + w) * 4, p.mask + (long long)r * p.mask_words + w);
        } else {
          sl[8 + j] = r;
          if (p.c_inds)
            cp_async_4(sa + (136 + j) * 4, p.c_inds + r);
          else
            sl[136 + j] = r;
        }
      } else {
        sl[8 + j] = -1;
#pragma unroll
        for (int w = 0; w < MW; ++w)
          sl[136 + j * MW + w] = conv ? 0 : -1;
      }
    }
    cp_async_mbar_arrive_noinc(rv.landed0 + 8u * si);  // arrives when this lane's copies have landed
    __syncwarp();  // the plain stores above are read by other lanes when the slot is published
    if (lane == 0)
      CB2_TRACE_EVENT(6, 16, tile);  // tile drawn, fetch issued
    ++issued;
    if (tile < 0) {
      ended = true;
      break;
    }
  }
  // publish what is still in flight (the end marker at the latest)
  while (ended && accounted < issued) {
    ended = mbar_wait_warp(rv.landed0 + 8u * (accounted % rv.ring), (accounted / rv.ring) & 1, rv.abort_flag);
    if (ended)
      account();
  }
  // The predecessor may still read or write the tile masks where the tables were read ahead of its end.
  if constexpr (SPLIT) {
    if (item_tile >= 0) {
      grid_dep_wait();
#pragma unroll
      for (int w = 0; w < MW; ++w)
        if (lane == 0 && w < p.mask_words)
          p.mask_out[(long long)item_tile * p.mask_words + w] = item_mask[w];
    }
  }
  // the last CTA to run out of tiles, or to give up, puts the two counters back to zero for the next launch
  if (dynamic && lane == 0) {
    if (next_cnt != 0)  // an outstanding request must have been served before the counters may be reset
      asm volatile("" ::"r"(next_base) : "memory");
    __threadfence();
    const int done = atomicAdd(p.tickets + 1, 1);
    if (done == (int)(gridDim.x * gridDim.y) - 1) {
      p.tickets[0] = 0;
      p.tickets[1] = 0;
      __threadfence();
    }
  }
  cp_async_wait_all();
}

// Eight columns of an output row from their sums, as the epilogue of whole tiles makes them.
__device__ __forceinline__ uint4 rowconv_finish8(const RowConvParams &p, const float (&v)[8], int o, int ncol) {
  float t[8];
  if (p.src_mode != kSrcNone && p.beta != 0.f) {
    const __half *sp = reinterpret_cast<const __half *>(p.src) + (p.src_mode == kSrcRows ? (long long)o * p.lds : 0ll) + ncol;
    __align__(16) __half h[8];
    if (p.src_mode == kSrcRows) {
      *reinterpret_cast<uint4 *>(h) = __ldg(reinterpret_cast<const uint4 *>(sp));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        h[i] = __ldg(sp + i);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      t[i] = __fmaf_rn(p.alpha, v[i], __fmul_rn(p.beta, __half2float(h[i])));
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      t[i] = __fmul_rn(p.alpha, v[i]);
  }
  uint32_t packed[4];
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    const __half2 h2 = __floats2half2_rn(apply_act(t[i], p.act_type, p.act_alpha), apply_act(t[i + 1], p.act_type, p.act_alpha));
    packed[i / 2] = *reinterpret_cast<const uint32_t *>(&h2);
  }
  return make_uint4(packed[0], packed[1], packed[2], packed[3]);
}

// SPLIT: a launch with so few items that most SMs would be idle.  What such a launch takes is one tile's offsets,
// one after the other, so a cluster of `split` CTAs shares an item's offsets: each sums its own in tensor memory and
// leaves the sums, fp32, in its shared memory; then each makes the output rows of its share of the tile from the
// sums of all, in the order of the CTAs, through distributed shared memory.  (Figures: cluster_split.  Clusters of
// two, for up to half as many items as SMs, gained 8 % on 9000 scanned rows and lost 6 % on uniform ones, most of
// whose tiles have one offset.)
template <int KIND, int NATOM_K, int BLOCK_N, bool B_MN, bool TMA_GATHER, int MASK_WORDS = 1, bool SPLIT = false>
__global__ void __launch_bounds__(RowConvCfg<KIND, NATOM_K, BLOCK_N, B_MN, TMA_GATHER, MASK_WORDS>::THREADS, 1)
rowconv_kernel(const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ CUtensorMap tmap_a,
               const RowConvParams p) {
  using Cfg = RowConvCfg<KIND, NATOM_K, BLOCK_N, B_MN, TMA_GATHER, MASK_WORDS>;
  constexpr int MW = MASK_WORDS;
  static_assert(!SPLIT || (KIND == 0 && TMA_GATHER && Cfg::OFF_EPI >= 128 * BLOCK_N * 4), "sums fit the operand stages");
  extern __shared__ uint8_t smem_raw[];
  if (threadIdx.x == 0)
    CB2_TRACE_CTA(0, 0);
  // Programmatic dependent launch: the next kernel on the stream may be scheduled onto SMs as
  // they free up, and this one may itself have started before its predecessor finished.  What runs
  // ahead is the set-up and, but for fp16 convolutions, the scheduler's tickets, row lists and mask words, the first
  // row-index loads and int8's scale and bias: a predecessor that writes those must not let its dependents start early
  // (see launch_after).  In an fp16 convolution the scheduler waits before it reads a table, so that it may follow
  // whatever made its tables, at the price of its first lookups' overlap -- but not where the
  // caller has said that an earlier call found the tables as they are.  Every role calls
  // grid_dep_wait() before it first touches operand rows, weights, the output or the tile masks.  The weight warp lets the
  // next kernel begin.
  // 1024-byte alignment: required by the 128-byte swizzle atoms of TMA and tcgen05.
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
  uint8_t *smem = smem_raw + pad;
  const uint32_t sbase = raw_addr + pad;

  int *rowidx = reinterpret_cast<int *>(smem + Cfg::OFF_ROWIDX);
  float *s_scale = reinterpret_cast<float *>(smem + Cfg::OFF_SCALE);
  float *s_bias = s_scale + BLOCK_N;
  volatile int *misc = reinterpret_cast<volatile int *>(smem + Cfg::OFF_MISC);
  // misc[0] tmem base, misc[1] abort flag, misc[15] steps issued, misc[2] SPLIT: a SplitState, misc[3] SPLIT: epilogue warps whose sums are
  // in this CTA's shared memory, misc[4 + 2 g, 6 + 2 g) what gather group g's waits returned, one for each of its
  // row buffers
  volatile int *abort_flag = misc + 1;

  const uint32_t bars = sbase + Cfg::OFF_BARS;
  auto full_a = [&](int s) { return bars + 8u * s; };
  auto empty_a = [&](int s) { return bars + 8u * (Cfg::BAR_EMPTY_A + s); };
  auto acc_full = [&](int s) { return bars + 8u * (Cfg::BAR_ACC_FULL + s); };
  auto acc_empty = [&](int s) { return bars + 8u * (Cfg::BAR_ACC_EMPTY + s); };
  const uint32_t final_bar = bars + 8u * Cfg::BAR_FINAL;
  auto full_b = [&](int s) { return bars + 8u * (Cfg::BAR_FULL_B + s); };
  auto empty_b = [&](int s) { return bars + 8u * (Cfg::BAR_EMPTY_B + s); };
  RingView rv;
  rv.slots = reinterpret_cast<int *>(smem + Cfg::OFF_RING);
  rv.full0 = bars + 8u * Cfg::BAR_RING;
  rv.empty0 = rv.full0 + 8u * Cfg::RING;
  rv.landed0 = rv.empty0 + 8u * Cfg::RING;
  rv.ring = Cfg::RING;
  rv.slot_ints = Cfg::RING_SLOT_INTS;
  rv.abort_flag = abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int ntiles = (p.n_rows + 127) / 128;
  const int kpasses = (p.red + Cfg::KRED - 1) / Cfg::KRED;

  // Scheduler warp: the first ticket.  (int8 asks the counter: its tiles in the order in which the CTAs arrive.  Stride 2
  // from 150 000 uniform rows, 39.6 us, and 41.6 by the CTAs' numbers, whose first rows arrive later.)
  int first_ticket = blockIdx.x;
  if (!SPLIT && !Cfg::DEALT && warp == Cfg::SCHED_WARP && p.tickets != nullptr && gridDim.y == 1 && lane == 0)
    first_ticket = atomicAdd(p.tickets, 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::SA; ++s) {
      mbar_init(full_a(s), Cfg::FULL_A_COUNT);
      mbar_init(empty_a(s), 1);
    }
    for (int s = 0; s < Cfg::SB; ++s) {
      mbar_init(full_b(s), 1);
      mbar_init(empty_b(s), 1);
    }
    for (int s = 0; s < Cfg::NUM_ACC; ++s) {
      mbar_init(acc_full(s), 1);
      mbar_init(acc_empty(s), Cfg::EPI_THREADS / 32 / Cfg::EPI_GROUPS);
    }
    mbar_init(final_bar, 1);
    for (int s = 0; s < Cfg::RING; ++s) {
      mbar_init(rv.full0 + 8u * s, 1);
      mbar_init(rv.landed0 + 8u * s, 32);  // one copy-completion arrival per scheduler lane
      mbar_init(rv.empty0 + 8u * s, Cfg::RING_CONSUMER_WARPS);
    }
    mbar_init_fence();
    misc[1] = 0;
    misc[2] = 0;
    misc[3] = 0;
    misc[15] = 0;
    CB2_TRACE_SELECT(0);
  }
  if (KIND == 1) {
    for (int i = threadIdx.x; i < BLOCK_N; i += blockDim.x) {
      int n = blockIdx.y * BLOCK_N + i;
      s_scale[i] = (n < p.nn && p.scale) ? p.scale[n] : 0.f;
      s_bias[i] = (n < p.nn && p.bias) ? p.bias[n] : 0.f;
    }
  }
  if (warp == Cfg::MMA_WARP) {
    tmem_alloc(sbase + Cfg::OFF_MISC, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == Cfg::SCHED_WARP)
    first_ticket = __shfl_sync(0xffffffffu, first_ticket, 0);
  if (!SPLIT && warp == Cfg::SCHED_WARP && p.mode == kModeMaskConv) {
    // the first tile's sort order and masks: 128 ints each, four 128-byte lines each
    const int tile = ntiles - 1 - first_ticket / p.n_parts;
    if (tile >= 0 && lane < 8) {
      const int r = tile * 128 + (lane & 3) * 32;
      if (r < p.n_rows) {
        const void *line = (lane < 4) ? static_cast<const void *>(p.argsort + r) : static_cast<const void *>(p.mask + (long long)r * p.mask_words);
        asm volatile("prefetch.global.L2 [%0];" ::"l"(line));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = static_cast<uint32_t>(misc[0]);
  if (threadIdx.x == 0)
    CB2_TRACE_EVENT(5, 11, 0);  // set-up done

  auto fail = [&](int code) {
    *abort_flag = 1;
    if (p.status)
      atomicCAS(p.status, 0, code);
  };

  if (warp < Cfg::MMA_WARP) {
    // ======================= epilogue: TMEM -> registers -> scattered rows.  A thread holds 32
    // consecutive columns of one row.  int8 stores them itself, 32 bytes at a time (whole sectors); an fp16
    // warp passes its 32 rows through 2 KB of shared memory of its own, so that four lanes store 64 bytes
    // side by side.  Either way every warp runs at its own pace and the accumulator is free again as soon
    // as the last column has been read.  (Staging the whole tile put two barriers of all epilogue warps
    // into every tile; storing 32 bytes a thread made 32 requests of every store of a warp.)
    const int et = threadIdx.x;
    const int erow = et & 127;   // the tile row this thread reads from TMEM (lane quarter = warp & 3)
    constexpr int HALVES = Cfg::EPI_HALVES / Cfg::EPI_GROUPS;
    const int half = (et >> 7) % HALVES;   // which share of the columns
    const int group = (et >> 7) / HALVES;  // which accumulator is this thread's (with several groups)
    constexpr int COLS_PER_HALF = BLOCK_N / HALVES;
    const bool sectors = ((reinterpret_cast<uintptr_t>(p.out) | static_cast<uintptr_t>(p.ldo * Cfg::OES)) & 31u) == 0;
    int buf = 0;
    uint32_t acc_phase = 0;
    auto next_acc = [&]() {
      if (++buf == Cfg::NUM_ACC) {
        buf = 0;
        acc_phase ^= 1u;
      }
    };
    // The sums will lie where the gather warps clear their stages, and a warp without a step of its own has nothing
    // else that orders its clearing before them.
    if constexpr (SPLIT)
      named_bar_sync(1, Cfg::CLEARED_THREADS);
    grid_dep_wait();
    CB2_PROF_BEGIN();
    TileCursor<MW> tc;
    int o = -1;  // destination row of this thread's tile row
    for (int more; (more = tc.next(p, rv, [&](const int *sl) {
                      o = (p.mode == kModeMaskConv) ? sl[8 + erow] : sl[136 + erow];
                    })) > 0;) {
          const int tile = tc.tile;
          const bool has_work = tc.offsets != 0;
          if (!has_work && (p.skip_empty_tiles || (SPLIT && (cluster_rank() != 0 || misc[2] != kSplitSolo))))
            continue;
          // A tile without work uses no accumulator and passes none on: whoever is next in turn stores it.
          if (Cfg::EPI_GROUPS > 1 && buf != group) {
            if (has_work)
              next_acc();
            continue;
          }
          const int n0 = Cfg::PARTS ? tc.n0 : static_cast<int>(blockIdx.y) * BLOCK_N;
          CB2_PROF_MARK(0);  // walk
          if (!SPLIT && erow == 0 && half == 0 && p.mask_out && n0 == 0) {
            if constexpr (MW == 1) {
              p.mask_out[tile] = tc.m;  // forward: not reversed
            } else {
#pragma unroll
              for (int w = 0; w < MW; ++w)
                if (w < p.mask_words)
                  p.mask_out[(long long)tile * p.mask_words + w] = static_cast<uint32_t>((w < 2 ? tc.lo : tc.hi) >> (32 * (w & 1)));
            }
          }
          if (has_work) {
            if (et == 0)
              CB2_TRACE_EVENT(4, 7, tile);
            const bool ok = mbar_wait(acc_full(buf), acc_phase, abort_flag);
            if (et == 0)
              CB2_TRACE_EVENT(4, 8, tile);  // accumulator complete
            if (!__all_sync(0xffffffffu, ok)) {
              if (lane == 0)
                fail(kStatusWaitTimeout);
              break;
            }
            tc_fence_after();
          }
          CB2_PROF_MARK(1);  // accumulator complete
          const uint32_t trow = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) +
                                static_cast<uint32_t>(buf * BLOCK_N);
          if constexpr (SPLIT) {
            if (misc[2] != kSplitSolo) {
              // The operand stages are idle: every MMA of the CTA has completed, and every stage was cleared before
              // this warp began.  Four columns of row r at [column / 4][r], so that a warp's rows lie side by side
#pragma unroll 1
              for (int round = 0; round < COLS_PER_HALF / 32; ++round) {
                uint32_t v[32];
                const int col0 = half * COLS_PER_HALF + round * 32;
                tmem_ld32(trow + col0, v);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 8; ++q)
                  st_shared_16(sbase + ((col0 / 4 + q) * 128 + erow) * 16, &v[4 * q]);
              }
              __syncwarp();
              if (lane == 0)
                atomicAdd(const_cast<int *>(misc + 3), 1);
              next_acc();
              continue;
            }
          }
          const bool use_src = (p.src_mode != kSrcNone) && (p.beta != 0.f);
          // fast path: out = cvt(acc); everything else goes through the general epilogue
          const bool plain = !use_src && p.act_type == 0 && p.alpha == 1.f;
          constexpr int ROUNDS = COLS_PER_HALF / 32;
          // 16-byte pieces of this thread's row; the columns past nn are not stored
          auto store = [&](int ncol, const auto &packed) {
            constexpr int N = sizeof(packed) / 16, PIECE = 16 / Cfg::OES;
            if constexpr (Cfg::EPI_WARP_BYTES > 0) {
              // four lanes store 64 bytes of a row side by side (the exclusive or keeps a quarter warp's
              // pieces in different banks)
              const uint32_t buf_w = sbase + Cfg::OFF_EPI + warp * Cfg::EPI_WARP_BYTES;
#pragma unroll
              for (int q = 0; q < N; ++q)
                st_shared_16(buf_w + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4), &packed[4 * q]);
              __syncwarp();
              const int q = lane & 3;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int r = i * 8 + (lane >> 2);
                const int to = __shfl_sync(0xffffffffu, o, r);
                const uint4 piece = ld_shared_16(buf_w + r * 64 + ((q ^ ((r >> 1) & 3)) << 4));
                if (to >= 0 && ncol + q * PIECE < p.nn)
                  *reinterpret_cast<uint4 *>(reinterpret_cast<uint8_t *>(p.out) +
                                             ((long long)to * p.ldo + ncol + q * PIECE) * Cfg::OES) = piece;
              }
              __syncwarp();
              return;
            }
            if (o < 0)
              return;
            uint8_t *dst = reinterpret_cast<uint8_t *>(p.out) + ((long long)o * p.ldo + ncol) * Cfg::OES;
            if (sectors && ncol + N * PIECE <= p.nn) {
#pragma unroll
              for (int q = 0; q < N; q += 2)
                st_global_32(dst + 16 * q, &packed[4 * q]);
            } else {
#pragma unroll
              for (int q = 0; q < N; ++q)
                if (ncol + q * PIECE < p.nn)
                  *reinterpret_cast<uint4 *>(dst + 16 * q) =
                      make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
            }
          };
#pragma unroll 1
          for (int round = 0; round < ROUNDS; ++round) {
            uint32_t v[32];
            const int col0 = half * COLS_PER_HALF + round * 32;
            if (has_work) {
              tmem_ld32(trow + col0, v);
              tmem_ld_wait();
              if (round == ROUNDS - 1) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                  mbar_arrive(acc_empty(buf));
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                v[i] = 0u;
            }
            const int ncol0 = n0 + col0;
            if constexpr (KIND == 0) {
              uint32_t packed[16];
              if (plain) {
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                  __half2 h2 = __floats2half2_rn(__uint_as_float(v[i]), __uint_as_float(v[i + 1]));
                  packed[i / 2] = *reinterpret_cast<uint32_t *>(&h2);
                }
              } else {
                float t[32];
                if (use_src) {
                  if (p.src_mode == kSrcRows) {
                    uint4 srcv[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                      srcv[q] = make_uint4(0, 0, 0, 0);
                    if (o >= 0) {
                      const uint4 *sp = reinterpret_cast<const uint4 *>(
                          reinterpret_cast<const __half *>(p.src) + (long long)o * p.lds + ncol0);
#pragma unroll
                      for (int q = 0; q < 4; ++q)
                        if (ncol0 + q * 8 < p.nn)
                          srcv[q] = __ldg(sp + q);
                    }
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                      const __half2 h = reinterpret_cast<const __half2 *>(srcv)[i / 2];
                      t[i] = __fmaf_rn(p.alpha, __uint_as_float(v[i]), __fmul_rn(p.beta, __low2float(h)));
                      t[i + 1] = __fmaf_rn(p.alpha, __uint_as_float(v[i + 1]), __fmul_rn(p.beta, __high2float(h)));
                    }
                  } else {
                    const __half *bv = reinterpret_cast<const __half *>(p.src);
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                      const float sv = (ncol0 + i < p.nn) ? __half2float(__ldg(bv + ncol0 + i)) : 0.f;
                      t[i] = __fmaf_rn(p.alpha, __uint_as_float(v[i]), __fmul_rn(p.beta, sv));
                    }
                  }
                } else {
#pragma unroll
                  for (int i = 0; i < 32; ++i)
                    t[i] = __fmul_rn(p.alpha, __uint_as_float(v[i]));
                }
                if (p.act_type == 1) {
#pragma unroll
                  for (int i = 0; i < 32; ++i)
                    t[i] = fmaxf(t[i], 0.f);
                } else if (p.act_type != 0) {
#pragma unroll
                  for (int i = 0; i < 32; ++i)
                    t[i] = apply_act(t[i], p.act_type, p.act_alpha);
                }
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                  __half2 h2 = __floats2half2_rn(t[i], t[i + 1]);
                  packed[i / 2] = *reinterpret_cast<uint32_t *>(&h2);
                }
              }
              store(ncol0, packed);
            } else {
              uint32_t packed[8];
              float t[32];
              {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  t[i] = __int2float_rn(static_cast<int>(v[i]));
                const float4 *sc4 = reinterpret_cast<const float4 *>(s_scale + col0);
                const float4 *bi4 = reinterpret_cast<const float4 *>(s_bias + col0);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                  const float4 sc = sc4[q], bi = bi4[q];
                  t[4 * q + 0] = __fmaf_rn(sc.x, t[4 * q + 0], bi.x);
                  t[4 * q + 1] = __fmaf_rn(sc.y, t[4 * q + 1], bi.y);
                  t[4 * q + 2] = __fmaf_rn(sc.z, t[4 * q + 2], bi.z);
                  t[4 * q + 3] = __fmaf_rn(sc.w, t[4 * q + 3], bi.w);
                }
              }
              if (use_src) {
                uint4 srcv[2];
                srcv[0] = srcv[1] = make_uint4(0, 0, 0, 0);
                if (o >= 0) {
                  const uint4 *sp = reinterpret_cast<const uint4 *>(
                      reinterpret_cast<const int8_t *>(p.src) + (long long)o * p.lds + ncol0);
#pragma unroll
                  for (int q = 0; q < 2; ++q)
                    if (ncol0 + q * 16 < p.nn)
                      srcv[q] = __ldg(sp + q);
                }
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  t[i] = __fmaf_rn(p.beta, static_cast<float>(reinterpret_cast<const int8_t *>(srcv)[i]), t[i]);
              }
              if (p.act_type == 1) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  t[i] = fmaxf(t[i], 0.f);
              } else if (p.act_type != 0) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  t[i] = apply_act(t[i], p.act_type, p.act_alpha);
              }
#pragma unroll
              for (int i = 0; i < 32; i += 4)
                packed[i / 4] = cvt_pack4_s8(t[i], t[i + 1], t[i + 2], t[i + 3]);
              store(ncol0, packed);
            }
          }
          CB2_PROF_MARK(3);  // TMEM -> rows
          if (has_work)
            next_acc();
          if (et == 0)
            CB2_TRACE_EVENT(4, 9, tile);  // rows stored
    }
    if (et == 0)
      CB2_PROF_END2();
  } else if (warp == Cfg::MMA_WARP) {
    // ======================= MMA issuer: one thread, from the walk to the commits.  It paces tiles with
    // several offsets.  Elected, so that the compiler keeps descriptors in uniform registers: with lane 0
    // chosen by its number four MMAs took 310 cycles of a step's 1000, elected 100; a thread that walks by itself
    // needs no votes between them.  A step of 64 channels takes it 560 cycles: 80 to see its operands there, 95 for four
    // MMAs, 215 for two commits, 170 to look at the next step's barriers.  (Warp that walks together, lane 0 by number /
    // the same, elected to issue / one thread, before the gathers were sped up: 30 011 rows of 125 offsets 87 / 79 / 77.8 us,
    // 100 003 scanned rows at 64 channels 42.5 / 39.5 / 39.8, after: - / 73 / 60.6 and - / 35.7 / 34.1.)  Whoever is waited
    // for next is looked at as soon as a step is committed.
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc(KIND, false, B_MN, 128, BLOCK_N);
      constexpr int KSTEPS_FULL = NATOM_K * 4;
      const uint64_t adesc_base = make_smem_desc(sbase + Cfg::OFF_A, 16, 1024);
      const uint64_t bdesc_base = B_MN ? make_smem_desc(sbase + Cfg::OFF_B, p.b_lbo, p.b_sbo)
                                       : make_smem_desc(sbase + Cfg::OFF_B, 16, 1024);
      const int ksteps_last = (p.red - (kpasses - 1) * Cfg::KRED + Cfg::UMMA_K - 1) / Cfg::UMMA_K;
      TileCursor<MW> tc;
      int stage = 0, bslot = Cfg::SB - 1, buf = 0, last_key = -1, steps = 0;
      uint32_t a_phase = 0, b_phase = 1, acc_phase = 1;
      bool ok = true;
      volatile int *const progress = misc + 15;
      grid_dep_wait();  // no operand comes before
      CB2_PROF_BEGIN();
      for (int more; ok && (more = tc.template next<true>(p, rv, [](const int *) {})) != 0;) {
        CB2_PROF_MARK(0);  // next tile
        if (more < 0) {
          ok = false;
          break;
        }
        if (tc.offsets == 0) {
          ++steps;  // what the scheduler charged
          if constexpr (!SPLIT)
            *progress = steps;
          continue;
        }
        // consecutive steps of a tile never share a weight tile; consecutive tiles may (kpasses and n0
        // are in the key: weights have as many columns)
        const bool new_b = (tc.first_offset() * kpasses) * p.nn + tc.n0 != last_key;
        auto next_b = [&]() {
          if (++bslot == Cfg::SB) {
            bslot = 0;
            b_phase ^= 1u;
          }
        };
        if (!Cfg::JOINT && new_b) {
          if (last_key >= 0)
            tc_commit(empty_b(bslot));
          next_b();
        }
        ok = mbar_wait(acc_empty(buf), acc_phase, abort_flag);
        CB2_PROF_MARK(1);  // accumulator free
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * BLOCK_N);
        const int total = tc.offsets * kpasses;
        int kp = 0;
        bool a_there = mbar_test(full_a(stage), a_phase), b_there = Cfg::JOINT || mbar_test(full_b(bslot), b_phase);
        for (int s = 0; s < total; ++s) {
          if constexpr (Cfg::JOINT)
            bslot = stage;
          if (!b_there)
            ok = ok && mbar_wait(full_b(bslot), b_phase, abort_flag);
          CB2_PROF_MARK(2);  // weight tile present
          if (!a_there)
            ok = ok && mbar_wait(full_a(stage), a_phase, abort_flag);
          CB2_PROF_MARK(3);  // rows present
          if (!ok)
            break;
          if constexpr (!TMA_GATHER)
            fence_proxy_async_smem();  // gathered rows were written through the generic proxy
          tc_fence_after();
          // descriptors differ from the stage's / slot's base descriptor only in the start address field
          // (bits 0-13, units of 16 bytes)
          const uint64_t adesc0 = adesc_base + static_cast<uint64_t>((stage * Cfg::A_STAGE_BYTES) >> 4);
          const uint64_t bdesc0 = bdesc_base + static_cast<uint64_t>((bslot * Cfg::B_SLOT_BYTES) >> 4);
          auto issue = [&](int ks, uint32_t acc) {
            const int ka = ks >> 2, kk = ks & 3;
            const uint64_t adesc = adesc0 + static_cast<uint64_t>((ka * (Cfg::TILE_M * 128) + kk * 32) >> 4);
            const uint64_t bdesc = bdesc0 + static_cast<uint64_t>(B_MN ? (((ka * 4 + kk) * (Cfg::UMMA_K * 128)) >> 4)
                                                                       : ((ka * (BLOCK_N * 128) + kk * 32) >> 4));
            tc_mma<KIND>(d_tmem, adesc, bdesc, idesc, acc);
          };
          const bool last_pass = ++kp == kpasses;
          // unrolled either way: addresses worked out in a loop cost more than the MMAs
          if (!last_pass || ksteps_last == KSTEPS_FULL) {
#pragma unroll
            for (int ks = 0; ks < KSTEPS_FULL; ++ks)
              issue(ks, (s == 0 && ks == 0) ? 0u : 1u);
          } else {
#pragma unroll
            for (int ks = 0; ks < KSTEPS_FULL - 1; ++ks)
              if (ks < ksteps_last)
                issue(ks, (s == 0 && ks == 0) ? 0u : 1u);
          }
          CB2_PROF_MARK(5);  // MMAs issued
          tc_commit(empty_a(stage));
          if (last_pass)
            kp = 0;
          if (++stage == Cfg::SA) {
            stage = 0;
            a_phase ^= 1u;
          }
          ++steps;
          if constexpr (!SPLIT)
            *progress = steps;
          if (s == total - 1) {
            tc_commit(acc_full(buf));
          } else {
            if (!Cfg::JOINT) {
              tc_commit(empty_b(bslot));
              next_b();
              b_there = mbar_test(full_b(bslot), b_phase);
            }
            a_there = mbar_test(full_a(stage), a_phase);
          }
          CB2_PROF_MARK(6);  // commits
        }
        last_key = (tc.last_offset() * kpasses + kpasses - 1) * p.nn + tc.n0;
        if (++buf == Cfg::NUM_ACC) {
          buf = 0;
          acc_phase ^= 1u;
        }
      }
      CB2_TRACE_CTA(2, (unsigned long long)steps);
      CB2_PROF_END();
      if (!ok)
        fail(kStatusWaitTimeout);
      tc_commit(final_bar);  // every MMA has retired before TMEM is released
      if (!mbar_drain(final_bar, 0, kWaitLimitNs))
        fail(kStatusWaitTimeout);
    }
    __syncwarp();
  } else if (warp == Cfg::TMA_WARP) {
    // ======================= weight tiles by TMA (lane 0 issues)
    TileCursor<MW> tc;
    int bslot = 0, last_key = -1;
    uint32_t b_phase = 1;
    bool ok = true;
    if (lane == 0)
      tma_prefetch_desc(&tmap_b);
    grid_dep_wait();
    // Only now: the next launch may begin while this one runs, but not while this one's predecessor does.  A record has
    // two pairs of ticket counters, and three launches of it in flight would have two that draw from one.
    grid_dep_launch();
    for (int more; ok && (more = tc.next(p, rv, [](const int *) {})) != 0;) {
      ok = more > 0;
      for (int left = ok ? tc.offsets : 0; ok && left > 0; --left) {
        const int f = tc.take();
        for (int kp = 0; ok && kp < kpasses; ++kp) {
          const int key = (f * kpasses + kp) * p.nn + tc.n0;
          if (!Cfg::JOINT && key == last_key)
            continue;
          last_key = key;
          const uint32_t full = Cfg::JOINT ? full_a(bslot) : full_b(bslot);
          ok = __all_sync(0xffffffffu, mbar_wait(Cfg::JOINT ? empty_a(bslot) : empty_b(bslot), b_phase, abort_flag));
          if (ok && lane == 0) {
            const int n0 = Cfg::PARTS ? tc.n0 : static_cast<int>(blockIdx.y) * BLOCK_N;
            const uint32_t dst = sbase + Cfg::OFF_B + bslot * Cfg::B_SLOT_BYTES;
            mbar_arrive_expect_tx(full, Cfg::B_SLOT_BYTES);
            if constexpr (!B_MN) {
              // [BLOCK_N rows x 128 B] per reduction atom; rows = output channels
#pragma unroll
              for (int ka = 0; ka < NATOM_K; ++ka)
                tma_load_3d(dst + ka * (BLOCK_N * 128), &tmap_b, full, kp * Cfg::KRED + ka * Cfg::ATOM_ELEMS, f, n0);
            } else {
              // [KRED rows x 128 B] per block of ATOM_ELEMS output channels; rows = reduction
#pragma unroll
              for (int na = 0; na < BLOCK_N / Cfg::ATOM_ELEMS; ++na)
                tma_load_3d(dst + na * (Cfg::KRED * 128), &tmap_b, full, n0 + na * Cfg::ATOM_ELEMS, f, kp * Cfg::KRED);
            }
          }
          __syncwarp();
          if (++bslot == Cfg::SB) {
            bslot = 0;
            b_phase ^= 1u;
          }
        }
      }
    }
    if (!ok && lane == 0)
      fail(kStatusWaitTimeout);
    for (int s = 0; s < Cfg::SB; ++s)  // slots before bslot were last filled in this round, the others in the one before
      mbar_drain(Cfg::JOINT ? full_a(s) : full_b(s), s < bslot ? b_phase ^ 1u : b_phase);
    __syncwarp();
  } else if (warp == Cfg::SCHED_WARP) {
    // ======================= scheduler: draws tiles, publishes their masks and row numbers
    scheduler_run<MW, SPLIT, Cfg::STEP_BUDGET, KIND == 0>(p, rv, ntiles, BLOCK_N, kpasses, first_ticket,
                                                          Cfg::DEALT ? (int)gridDim.x : 0, misc + 15, misc + 2);
  } else {
    // ======================= operand-row gather: group g owns stage g
    if constexpr (TMA_GATHER) {
      // One warp per group and 128-byte column block; lane L fetches tile rows 4L .. 4L+3 ("its quad") with
      // one request.  A quad none of whose rows has a neighbour at this offset is
      // not requested at all -- for the offsets away from the centre that is most quads, and the
      // copy engine's request rate is what bounds such steps.  The stage therefore keeps the
      // invariant "a quad that was not requested holds zeros": it is cleared once here, and a
      // quad that was filled in the previous use and is not needed now is requested with no row at all (fp16)
      // or cleared by stores again (int8).  (Scanned rows, forward, us, requested and cleared: fp16, 100 003 at 64 channels
      // 36.0 and 36.5, 40 to 72 channels 40 000 28.2 and 31.1, 80 000 53.2 and 48.4, 150 000 64.5 and 70.3; int8, 112 to 32,
      // 40 000 24.5 and 23.9, 80 000 34.2 and 30.6, 150 000 at 32 to 96 50.3 and 46.9, at 128 44.0 and 44.0.)
      // The neighbour indices of the group's next step in the tile are on their way while it waits for its stage
      // (the same scene: 39.8 -> 36.4 us; 125 offsets, 30 011 rows: 77 -> 61).
      const int g = (warp - Cfg::FIRST_GATHER_WARP) / NATOM_K;
      const int part = (warp - Cfg::FIRST_GATHER_WARP) % NATOM_K;
      if (lane == 0)
        tma_prefetch_desc(&tmap_a);
      const uint32_t first_quad = sbase + Cfg::OFF_A + g * Cfg::A_STAGE_BYTES + part * (Cfg::TILE_M * 128);
      const uint32_t my_quad = first_quad + lane * (4 * 128);
      for (int q = 0; q < 32; ++q)
        st_shared_zero16(first_quad + q * (4 * 128) + lane * 16);
      fence_proxy_async_smem();  // generic-proxy stores, read by the tensor core
      if constexpr (SPLIT)
        named_bar_arrive(1, Cfg::CLEARED_THREADS);
      __syncwarp();
      uint32_t dirty = 0;  // quads of this stage that hold gathered rows
      bool dep_waited = false, ok = true;
      int stage = 0;         // stage of the CTA's next tile's first step
      uint32_t phase = 1;    // of this group's own stage
      TileCursor<MW> tc;
      int4 o = make_int4(-1, -1, -1, -1);
      for (int more; ok && (more = tc.template next<false, true>(p, rv, [&](const int *sl) {
                             o = *reinterpret_cast<const int4 *>(sl + 8 + lane * 4);
                           })) != 0;) {
        ok = more > 0;
        const int total = ok ? tc.offsets * kpasses : 0;
        int f = -1, upto = 0;  // the offset taken last, and the first step that needs the next one
        auto look_up = [&](int step, int (&idx)[4], int &kp) {
          while (step >= upto) {
            f = tc.take();
            upto += kpasses;
          }
          kp = step - (upto - kpasses);
          const int row[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            idx[r] = -1;
            if (row[r] >= 0) {
              if (p.mode == kModeMaskConv)
                idx[r] = __ldg(p.indices + (long long)f * p.n_rows + row[r]);
              else
                idx[r] = p.a_inds ? __ldg(p.a_inds + row[r]) : row[r];
            }
          }
        };
        int ahead[4], ahead_kp = 0;
        int step = g - stage + (g < stage ? Cfg::SA : 0);
        stage = (stage + total) % Cfg::SA;
        if (step < total)
          look_up(step, ahead, ahead_kp);
        for (; step < total; step += Cfg::SA) {
          int idx[4];
          const int kp = ahead_kp;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            idx[r] = ahead[r];
            if (idx[r] >= p.a_rows) {  // reported; the copy engine would read such a row as zeros
              fail(kStatusBadIndex);
              idx[r] = -1;
            }
          }
          if (step + Cfg::SA < total)
            look_up(step + Cfg::SA, ahead, ahead_kp);
          if (lane == 0)
            CB2_TRACE_EVENT(g, 1, f + (idx[0] == 0x7fffffff));  // index loaded
          ok = mbar_wait_warp(empty_a(g), phase, abort_flag);
          if (!ok)
            break;
          phase ^= 1u;
          if (!dep_waited) {
            grid_dep_wait();
            dep_waited = true;
          }
          const bool wanted = (idx[0] & idx[1] & idx[2] & idx[3]) >= 0;  // some row index is not -1
          const uint32_t need = __ballot_sync(0xffffffffu, wanted);
          const uint32_t ask = KIND == 1 ? need : need | dirty;
          if (KIND == 1 && (dirty & ~need)) {
            for (uint32_t q = dirty & ~need; q; q &= q - 1)
              st_shared_zero16(first_quad + (__ffs(q) - 1) * (4 * 128) + lane * 16);
            fence_proxy_async_smem();  // as at the start
            __syncwarp();              // before lane 0 arrives
          }
          if (lane == 0) {
            CB2_TRACE_EVENT(g, 2, f);  // stage free
            mbar_arrive_expect_tx(full_a(g), static_cast<uint32_t>(__popc(ask)) * 512);
          }
          __syncwarp();
          if ((ask >> lane) & 1u)
            tma_gather4(my_quad, &tmap_a, full_a(g), kp * Cfg::KRED + part * Cfg::ATOM_ELEMS,
                        row_or_zeros(idx[0], 4 * lane), row_or_zeros(idx[1], 4 * lane + 1),
                        row_or_zeros(idx[2], 4 * lane + 2), row_or_zeros(idx[3], 4 * lane + 3));
          dirty = need;
          if (lane == 0)
            CB2_TRACE_EVENT(g, 3, f);  // copies issued
        }
      }
      if (!ok && lane == 0)
        fail(kStatusWaitTimeout);
      mbar_drain(full_a(g), phase);  // the group's last copies
    } else {
      constexpr int GT = Cfg::GROUP_THREADS;
      constexpr int RPT = (128 + GT - 1) / GT;                  // tile rows whose index each thread fetches
      const int g = (warp - Cfg::FIRST_GATHER_WARP) / (GT / 32);
      const int gt = threadIdx.x - (Cfg::FIRST_GATHER_WARP * 32 + g * GT);
      constexpr int CPR = NATOM_K * 8;                  // 16-byte chunks per operand row
      constexpr int RSTEP = GT / CPR;
      const int c = gt % CPR;
      const int row0 = gt / CPR;
      int *group_rowidx = rowidx + g * 256;  // two buffers, alternating per step of the group
      volatile int *my_flag = misc + 4 + 2 * g;
      bool dep_waited = false, ok = true;
      uint32_t steps = 0;  // the CTA's steps before this tile; step n fills stage n % SA and is group n % GROUPS'
      uint32_t use = 0;    // steps this group has taken
      int o[RPT];
#pragma unroll
      for (int r = 0; r < RPT; ++r)
        o[r] = -1;
      const uint8_t *a_bytes = reinterpret_cast<const uint8_t *>(p.a);
      TileCursor<MW> tc;
      for (int more; ok && (more = tc.template next<false, true>(p, rv, [&](const int *sl) {
                             // the rows this thread's gathers start from (sort index, or the row itself)
#pragma unroll
                             for (int r = 0; r < RPT; ++r)
                               o[r] = (gt + r * GT < 128) ? sl[8 + gt + r * GT] : -1;
                           })) > 0;) {
        const int total = tc.offsets * kpasses;
        int f = -1, upto = 0;  // the offset taken last, and the first step that needs the next one
        auto look_up = [&](int step, int (&idx)[RPT]) {
          while (step >= upto) {
            f = tc.take();
            upto += kpasses;
          }
#pragma unroll
          for (int r = 0; r < RPT; ++r) {
            idx[r] = -1;
            if (o[r] >= 0) {
              if (p.mode == kModeMaskConv)
                idx[r] = __ldg(p.indices + (long long)f * p.n_rows + o[r]);
              else
                idx[r] = p.a_inds ? __ldg(p.a_inds + o[r]) : o[r];
            }
          }
        };
        // The neighbour indices of the group's next step in the tile are on their way while it waits for the
        // stage and copies (100 000 scanned rows at 128 channels, forward: 66.5 -> 60.2 us).
        int ahead[RPT];
        const int turn = static_cast<int>(steps % Cfg::GROUPS);
        int step = g - turn + (g < turn ? Cfg::GROUPS : 0);
        if (step < total)
          look_up(step, ahead);
        for (; step < total; step += Cfg::GROUPS) {
          const uint32_t n = steps + step;
          const int st = static_cast<int>(n % Cfg::SA);
          const uint32_t st_phase = ((n / Cfg::SA) & 1u) ^ 1u;
          const int kp = step - (upto - kpasses);  // the step's offset is the one taken last
          int idx[RPT];
#pragma unroll
          for (int r = 0; r < RPT; ++r) {
            idx[r] = ahead[r];
            if (idx[r] >= p.a_rows) {  // never dereference a row the caller did not provide
              fail(kStatusBadIndex);
              idx[r] = -1;
            }
          }
          if (step + Cfg::GROUPS < total)
            look_up(step + Cfg::GROUPS, ahead);
          if (gt == 0) {
            CB2_TRACE_EVENT(g, 1, f + (idx[0] == 0x7fffffff));  // index loaded
            const bool free = mbar_wait(empty_a(st), st_phase, abort_flag);
            CB2_TRACE_EVENT(g, 2, f);  // stage free
            my_flag[use & 1] = free ? 1 : 0;
            if (!free)
              fail(kStatusWaitTimeout);
          }
          // Double-buffered, as the flag is: a thread that runs ahead writes the other buffer than the one
          // slower threads of the group may still be reading for the previous step.
          int *my_rowidx = group_rowidx + (use & 1) * 128;
#pragma unroll
          for (int r = 0; r < RPT; ++r)
            if (gt + r * GT < 128)
              my_rowidx[gt + r * GT] = idx[r];
          named_bar_sync(2 + g, Cfg::GROUP_THREADS);
          ++use;
          if (my_flag[(use - 1) & 1] == 0) {
            ok = false;
            break;
          }
          if (!dep_waited) {
            grid_dep_wait();
            dep_waited = true;
          }
          const uint32_t a_stage = sbase + Cfg::OFF_A + st * Cfg::A_STAGE_BYTES;
          const int byte_off = kp * Cfg::KRED * Cfg::ES + c * 16;
          const bool col_ok = byte_off < p.red * Cfg::ES;
          const uint32_t dst_c = a_stage + (c >> 3) * (Cfg::TILE_M * 128);
#pragma unroll
          for (int i = 0; i < (128 + RSTEP - 1) / RSTEP; ++i) {
            const int row = row0 + i * RSTEP;
            if ((128 % RSTEP) != 0 && row >= 128)
              break;
            const int ridx = my_rowidx[row];
            const uint32_t dst = dst_c + (row >> 3) * 1024 + (row & 7) * 128 + (((c & 7) ^ (row & 7)) << 4);
            const bool valid = col_ok && ridx >= 0;
            const uint8_t *srcp = valid ? a_bytes + ((long long)ridx * p.lda) * Cfg::ES + byte_off : a_bytes;
            cp_async_16(dst, srcp, valid ? 16u : 0u);
          }
          // The barrier is signalled by the copy engine when this thread's copies have landed;
          // the thread itself runs on to its next step.  The consumer makes the data visible
          // to the tensor core with a proxy fence after its wait.
          cp_async_mbar_arrive_noinc(full_a(st));
          if (gt == 0)
            CB2_TRACE_EVENT(g, 3, f);  // copies issued
        }
        steps += total;
      }
      cp_async_wait_all();
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if constexpr (SPLIT) {
    // Every CTA of the cluster passes both barriers, whatever became of its waits: none leaves while another may read
    // its shared memory.  Rows are made only where every CTA has what its state promises; where one gave up (the status
    // word says so) the item's rows stay as they were, and the slot its rows would be read from may not even be filled.
    cluster_sync();
    if (misc[2] != kSplitSolo) {
      int state = kSplitNothing, warps = 0;  // of the CTA whose rank is this lane's number
      if (lane < p.split)
        ld_cluster_2ints(cluster_map(sbase + Cfg::OFF_MISC + 8, lane), state, warps);
      const bool sums = state == kSplitSums && warps == Cfg::EPI_THREADS / 32;
      const unsigned have = __ballot_sync(0xffffffffu, sums);
      const bool whole = __all_sync(0xffffffffu, sums || state == kSplitNothing);
      grid_dep_wait();
      const int rows = 128 / p.split, first = (int)cluster_rank() * rows;
      const int *sl = rv.slot(0);  // the item's: the ring's first, and never used again
      const int n0 = sl[3];
      if (whole && (have != 0 || !p.skip_empty_tiles))
        for (int i = threadIdx.x; i < rows * (BLOCK_N / 8); i += Cfg::THREADS) {
          const int row = first + i % rows, col = i / rows * 8;
          const int to = sl[8 + row];
          if (to < 0 || n0 + col >= p.nn)
            continue;
          float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
          for (int c = 0; c < p.split; ++c)
            if ((have >> c) & 1u) {
              const uint32_t at = cluster_map(sbase + (col / 4 * 128 + row) * 16, c);
              const float4 a = ld_cluster_16(at), b = ld_cluster_16(at + 128 * 16);
              v[0] += a.x, v[1] += a.y, v[2] += a.z, v[3] += a.w;
              v[4] += b.x, v[5] += b.y, v[6] += b.z, v[7] += b.w;
            }
          *reinterpret_cast<uint4 *>(reinterpret_cast<__half *>(p.out) + (long long)to * p.ldo + n0 + col) =
              rowconv_finish8(p, v, to, n0 + col);
        }
      __syncwarp();
    }
    cluster_sync();
  }
  if (threadIdx.x == 0)
    CB2_TRACE_CTA(1, 0);
  if (warp == Cfg::MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

} // namespace cb2
