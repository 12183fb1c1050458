// Neighbour tables of a sparse convolution, built on the GPU: input-voxel hash table, active
// output voxels of a strided convolution, indices[f, o], neighbour masks, the stable sort of the
// outputs by mask, and the same for the backward direction.
//
// This is the step BEFORE the convolution kernels.  It is not part of cumm itself (its callers
// build these tables with cumm's hash headers, include/tensorview/hash/hash.cu.h:43-263 and
// include/tensorview/hash/ops.h:24-150); the table convention is the one the convolution kernels
// read (include/tensorview/gemm/core/nvrtc_params.h:38-65): indices [kv, N_out] in original row
// order with -1 for a missing neighbour, filter offsets in (z, y, x) row-major order, bit f of a
// row's mask set iff it has a neighbour at offset f, rows sorted by mask value with a STABLE
// sort, active outputs of a strided convolution ordered by their linearised (batch, z, y, x).
// Everything is integer work on HBM-resident arrays: coalesced passes, no tensor cores.
// All loops are bounded: a probe sequence visits at most `capacity` slots and reports a full
// table through the status word instead of spinning.
// None of these kernels triggers programmatic dependent launch (griddepcontrol.launch_dependents):
// the convolution kernels read masks, sort orders and index rows BEFORE their own
// griddepcontrol.wait, which is only sound while whatever wrote those tables has completed in
// the ordinary stream order.  Keep it that way.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cb2pg {

constexpr unsigned long long kEmptyKey = ~0ULL;
enum : int { kStatusTableFull = 3, kStatusBadCoord = 4 };

struct Geometry {
  int grid[3];    // input grid (z, y, x)
  int ogrid[3];   // output grid
  int ksize[3], stride[3], pad[3], dil[3];
  int kv;
  int batch_size;
};

__device__ __forceinline__ uint32_t mix64(unsigned long long k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdULL;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ULL;
  k ^= k >> 33;
  return static_cast<uint32_t>(k);
}

__device__ __forceinline__ unsigned long long linear_key(int b, int z, int y, int x, const int (&g)[3]) {
  return ((static_cast<unsigned long long>(b) * g[0] + z) * g[1] + y) * g[2] + x;
}

// ---------------------------------------------------------------- hash table: voxel -> smallest row
// One 8-byte word per slot, (tag << 32) | row, all ones = empty: a lookup is one load where a key
// array and a row array took two dependent ones.  While the grid has fewer than 2^32 cells the tag
// IS the linearised voxel (`exact`); above, it is 32 bits of another hash of it and a match is
// confirmed against the row's coordinates.
struct HashView {
  unsigned long long *slots;
  uint32_t cap_mask;
  int exact;
  const int32_t *coords;
};

__device__ __forceinline__ uint32_t hash_tag(const HashView &h, unsigned long long key) {
  return h.exact ? static_cast<uint32_t>(key) : static_cast<uint32_t>((key * 0x9e3779b97f4a7c15ULL) >> 32);
}
__device__ __forceinline__ bool hash_match(const HashView &h, unsigned long long entry, uint32_t tag, int b, int z,
                                           int y, int x) {
  if (static_cast<uint32_t>(entry >> 32) != tag)
    return false;
  if (h.exact)
    return true;
  const int4 c = __ldg(reinterpret_cast<const int4 *>(h.coords) + static_cast<uint32_t>(entry));
  return c.x == b && c.y == z && c.z == y && c.w == x;
}

__global__ void __launch_bounds__(256) hash_insert_kernel(const int32_t *__restrict__ coords, int n, Geometry g,
                                                          HashView h, int *status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const int4 c = reinterpret_cast<const int4 *>(coords)[i];
  if (c.x < 0 || c.x >= g.batch_size || c.y < 0 || c.y >= g.grid[0] || c.z < 0 || c.z >= g.grid[1] || c.w < 0 ||
      c.w >= g.grid[2]) {
    atomicCAS(status, 0, kStatusBadCoord);
    return;
  }
  const unsigned long long key = linear_key(c.x, c.y, c.z, c.w, g.grid);
  const uint32_t tag = hash_tag(h, key);
  const unsigned long long entry = (static_cast<unsigned long long>(tag) << 32) | static_cast<uint32_t>(i);
  uint32_t slot = mix64(key) & h.cap_mask;
  for (uint32_t probe = 0; probe <= h.cap_mask; ++probe) {
    const unsigned long long prev = atomicCAS(h.slots + slot, kEmptyKey, entry);
    if (prev == kEmptyKey)
      return;
    if (hash_match(h, prev, tag, c.x, c.y, c.z, c.w)) {
      atomicMin(h.slots + slot, entry);  // duplicates resolve to the first row, as a stable sort + search does
      return;
    }
    slot = (slot + 1) & h.cap_mask;
  }
  atomicCAS(status, 0, kStatusTableFull);
}

// ---------------------------------------------------------------- active outputs of a strided conv
// One thread per input voxel: the output positions that read it, one per filter offset whose
// (in + pad - r * dil) is a multiple of the stride on every axis (for stride 2 that is 8 of the
// 27 offsets; the loops prune whole planes and rows of offsets at once).  New positions are
// appended (unordered) to `list`, one counter update per group of lanes that found one together.
__global__ void __launch_bounds__(256) out_candidates_kernel(const int32_t *__restrict__ coords, int n, Geometry g,
                                                             unsigned long long *set_keys, uint32_t cap_mask,
                                                             unsigned long long *list, int list_cap, int *counter,
                                                             int *status) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const int4 c = reinterpret_cast<const int4 *>(coords)[i];
  if (c.x < 0 || c.x >= g.batch_size)
    return;  // reported by the insert kernel
  const int lane = threadIdx.x & 31;
  for (int rz = 0; rz < g.ksize[0]; ++rz) {
    const int nz = c.y + g.pad[0] - rz * g.dil[0];
    if (nz < 0 || nz % g.stride[0] != 0 || nz / g.stride[0] >= g.ogrid[0])
      continue;
    for (int ry = 0; ry < g.ksize[1]; ++ry) {
      const int ny = c.z + g.pad[1] - ry * g.dil[1];
      if (ny < 0 || ny % g.stride[1] != 0 || ny / g.stride[1] >= g.ogrid[1])
        continue;
      for (int rx = 0; rx < g.ksize[2]; ++rx) {
        const int nx = c.w + g.pad[2] - rx * g.dil[2];
        if (nx < 0 || nx % g.stride[2] != 0 || nx / g.stride[2] >= g.ogrid[2])
          continue;
        const unsigned long long key =
            linear_key(c.x, nz / g.stride[0], ny / g.stride[1], nx / g.stride[2], g.ogrid);
        uint32_t slot = mix64(key) & cap_mask;
        bool done = false, fresh = false;
        for (uint32_t probe = 0; probe <= cap_mask && !done; ++probe) {
          const unsigned long long prev = atomicCAS(set_keys + slot, kEmptyKey, key);
          if (prev == key)
            done = true;
          else if (prev == kEmptyKey)
            done = fresh = true;
          else
            slot = (slot + 1) & cap_mask;
        }
        if (!done)
          atomicCAS(status, 0, kStatusTableFull);
        if (fresh) {
          // the lanes that got here together share one counter update
          const unsigned together = __activemask();
          const int leader = __ffs(together) - 1;
          int base = 0;
          if (lane == leader)
            base = atomicAdd(counter, __popc(together));
          base = __shfl_sync(together, base, leader);
          const int at = base + __popc(together & ((1u << lane) - 1u));
          if (at < list_cap)
            list[at] = key;
          else
            atomicCAS(status, 0, kStatusTableFull);
        }
      }
    }
  }
}

__global__ void __launch_bounds__(256) decode_out_coords_kernel(const unsigned long long *__restrict__ keys, int n,
                                                                Geometry g, int32_t *out_coords) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n)
    return;
  unsigned long long k = keys[o];
  const int x = static_cast<int>(k % g.ogrid[2]);
  k /= g.ogrid[2];
  const int y = static_cast<int>(k % g.ogrid[1]);
  k /= g.ogrid[1];
  const int z = static_cast<int>(k % g.ogrid[0]);
  k /= g.ogrid[0];
  reinterpret_cast<int4 *>(out_coords)[o] = make_int4(static_cast<int>(k), z, y, x);
}

// ---------------------------------------------------------------- the sort of rows by mask: shapes
// Rows are sorted by their neighbour masks with a stable LSD radix sort on the kv mask bits, taken as
// one integer whose last word is the most significant, in digits of up to nine bits (three passes
// for the 27 offsets of a 3x3x3 kernel).  The rows are cut into at most kSortChunks equal chunks, one
// CTA each.  hist[pass][chunk][digit] counts the digits of the chunk's rows as they stand BEFORE that
// pass: the kernel that makes the masks fills pass 0, every pass fills the next one's counts while it
// scatters, so a pass is one launch (it was three: count, scan, scatter).
constexpr int kSortDigitBits = 9;
constexpr int kSortBins = 1 << kSortDigitBits;
constexpr int kSortChunks = 74;     // two sides (forward and backward tables) fill 148 SMs
constexpr int kSortThreads = kSortBins;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;       // rows per thread and round
constexpr int kProbeThreads = 256;  // chunks are whole multiples of this

struct SortShape {
  int bits, words, passes, width;  // mask bits; words per mask; passes; bits per digit (the last may be narrower)
};
inline SortShape sort_shape(int kv) {
  SortShape s;
  s.bits = kv;
  s.words = (kv + 31) / 32;
  s.passes = (kv + kSortDigitBits - 1) / kSortDigitBits;
  s.width = (kv + s.passes - 1) / s.passes;
  return s;
}
inline int sort_chunk(long long n) {  // rows per chunk
  const long long least = (n + kSortChunks - 1) / kSortChunks;
  const long long c = (least + kProbeThreads - 1) / kProbeThreads * kProbeThreads;
  return static_cast<int>(c < 2048 ? 2048 : c);
}
inline size_t sort_hist_ints(const SortShape &s, long long n_max) {  // room for any n up to n_max
  const long long chunks = (n_max + 2047) / 2048;
  return static_cast<size_t>(s.passes) * (chunks < kSortChunks ? chunks : kSortChunks) * kSortBins;
}

// Counts the first digit of one row per thread into the block's chunk (all threads of a block of
// kProbeThreads take part; the block's rows lie in one chunk).
__device__ __forceinline__ void count_first_digit(int *s_hist, bool valid, uint32_t low_word, int width, int *hist,
                                                  int chunk_index) {
  for (int d = threadIdx.x; d < kSortBins; d += blockDim.x)
    s_hist[d] = 0;
  __syncthreads();
  const uint32_t digit = valid ? (low_word & ((1u << width) - 1u)) : 0xffffffffu;
  const unsigned peers = __match_any_sync(0xffffffffu, digit);  // most rows of a sparse scene share one mask
  if (valid && static_cast<int>(threadIdx.x & 31) == __ffs(peers) - 1)
    atomicAdd(&s_hist[digit], __popc(peers));
  __syncthreads();
  for (int d = threadIdx.x; d < kSortBins; d += blockDim.x)
    if (s_hist[d])
      atomicAdd(hist + static_cast<long long>(chunk_index) * kSortBins + d, s_hist[d]);
  __syncthreads();
}

// One side of a table set (forward or backward) as the kernels that finish its masks see it.
struct MaskSide {
  int32_t *indices;   // [kv, n]
  uint32_t *rows;     // [n, words] unsorted masks
  int *hist;          // counts of the first pass
  int n, chunk;
};

// ---------------------------------------------------------------- indices[f, o] and masks
// One thread per output voxel; consecutive threads write consecutive columns of every row of the
// table.  Lookups are issued nine at a time: their first loads are in flight together, so a thread
// waits for ceil(kv / 9) memory round trips instead of kv.
// `mirror` (submanifold convolutions whose offsets are symmetric): o' is o's neighbour at offset f
// exactly if o is o's neighbour at offset kv - 1 - f, so the backward table is the forward one with
// the offsets reversed and is written by the same thread.  A row that repeats another row's voxel
// has no backward neighbours (nothing points at it).
template <int NW>
__global__ void __launch_bounds__(kProbeThreads, 4) probe_kernel(const int32_t *__restrict__ out_coords, Geometry g,
                                                              const HashView h, const MaskSide side,
                                                              const MaskSide mirror, int words, int width) {
  constexpr int B = 9;
  __shared__ int s_hist[kSortBins];
  const int o = blockIdx.x * kProbeThreads + threadIdx.x;
  const bool valid = o < side.n;
  const bool has_mirror = mirror.indices != nullptr;
  uint32_t m[NW], mb[NW];
#pragma unroll
  for (int w = 0; w < NW; ++w)
    m[w] = mb[w] = 0u;
  if (valid) {
    const int4 c = __ldg(reinterpret_cast<const int4 *>(out_coords) + o);
    const int z0 = c.y * g.stride[0] - g.pad[0], y0 = c.z * g.stride[1] - g.pad[1], x0 = c.w * g.stride[2] - g.pad[2];
    int rz = 0, ry = 0, rx = 0;
    bool repeats = false;
    for (int f0 = 0; f0 < g.kv; f0 += B) {
      unsigned long long entry[B];
      uint32_t slot[B], tag[B];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        entry[j] = kEmptyKey;
        slot[j] = tag[j] = 0u;
        const int z = z0 + rz * g.dil[0], y = y0 + ry * g.dil[1], x = x0 + rx * g.dil[2];
        if (f0 + j < g.kv && z >= 0 && z < g.grid[0] && y >= 0 && y < g.grid[1] && x >= 0 && x < g.grid[2]) {
          const unsigned long long key = linear_key(c.x, z, y, x, g.grid);
          slot[j] = mix64(key) & h.cap_mask;
          tag[j] = hash_tag(h, key);
          entry[j] = __ldg(h.slots + slot[j]);
        }
        if (++rx == g.ksize[2]) {
          rx = 0;
          if (++ry == g.ksize[1]) {
            ry = 0;
            ++rz;
          }
        }
      }
#pragma unroll
      for (int j = 0; j < B; ++j) {
        const int f = f0 + j;
        if (f < g.kv) {
          int idx = -1;
          unsigned long long e = entry[j];
          uint32_t s = slot[j];
          for (uint32_t probe = 0; probe <= h.cap_mask && e != kEmptyKey; ++probe) {
            const int xy = g.ksize[1] * g.ksize[2];
            if (hash_match(h, e, tag[j], c.x, z0 + f / xy * g.dil[0], y0 + f % xy / g.ksize[2] * g.dil[1],
                           x0 + f % g.ksize[2] * g.dil[2])) {
              idx = static_cast<int>(static_cast<uint32_t>(e));
              break;
            }
            s = (s + 1) & h.cap_mask;
            e = __ldg(h.slots + s);
          }
          side.indices[static_cast<long long>(f) * side.n + o] = idx;
#pragma unroll
          for (int w = 0; w < NW; ++w)
            if (idx >= 0 && (NW == 1 || (f >> 5) == w))
              m[w] |= 1u << (f & 31);
          if (has_mirror) {
            const int fb = g.kv - 1 - f;
            mirror.indices[static_cast<long long>(fb) * mirror.n + o] = idx;
#pragma unroll
            for (int w = 0; w < NW; ++w)
              if (idx >= 0 && (NW == 1 || (fb >> 5) == w))
                mb[w] |= 1u << (fb & 31);
            if (f == fb)
              repeats = idx != o;
          }
        }
      }
    }
    if (has_mirror && repeats) {
      for (int f = 0; f < g.kv; ++f)
        mirror.indices[static_cast<long long>(f) * mirror.n + o] = -1;
#pragma unroll
      for (int w = 0; w < NW; ++w)
        mb[w] = 0u;
    }
#pragma unroll
    for (int w = 0; w < NW; ++w)
      if (w < words) {
        side.rows[static_cast<long long>(o) * words + w] = m[w];
        if (has_mirror)
          mirror.rows[static_cast<long long>(o) * words + w] = mb[w];
      }
  }
  count_first_digit(s_hist, valid, m[0], width, side.hist, blockIdx.x * kProbeThreads / side.chunk);
  if (has_mirror)
    count_first_digit(s_hist, valid, mb[0], width, mirror.hist, blockIdx.x * kProbeThreads / mirror.chunk);
}

// indices_bwd[f, i] = o for every indices[f, o] = i (the table the input gradient walks)
__global__ void __launch_bounds__(256) invert_table_kernel(const int32_t *__restrict__ indices, int n_out, int kv,
                                                           int n_in, int32_t *indices_bwd) {
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= static_cast<long long>(n_out) * kv)
    return;
  const int f = static_cast<int>(t / n_out), o = static_cast<int>(t % n_out);
  const int i = indices[t];
  if (i >= 0 && i < n_in)
    indices_bwd[static_cast<long long>(f) * n_in + i] = o;
}

// the unsorted masks of a finished table
__global__ void __launch_bounds__(kProbeThreads) masks_from_table_kernel(const MaskSide side, int kv, int words, int width) {
  __shared__ int s_hist[kSortBins];
  const int j = blockIdx.x * kProbeThreads + threadIdx.x;
  const bool valid = j < side.n;
  uint32_t low = 0;
  if (valid)
    for (int w = 0; w < words; ++w) {
      uint32_t m = 0;
#pragma unroll 8
      for (int b = 0; b < 32; ++b)
        if (32 * w + b < kv && side.indices[static_cast<long long>(32 * w + b) * side.n + j] >= 0)
          m |= 1u << b;
      side.rows[static_cast<long long>(j) * words + w] = m;
      if (w == 0)
        low = m;
    }
  count_first_digit(s_hist, valid, low, width, side.hist, blockIdx.x * kProbeThreads / side.chunk);
}

// ---------------------------------------------------------------- strided convolutions through a bitmap of outputs
// One bit per cell of the output grid.  Active outputs are ordered by their linearised position, so
// an output's row number is the number of set bits before its own: no set of keys, no sort of keys, and
// both tables follow from the input voxels alone (the rows an input feeds are looked up by counting)
// instead of kv hash lookups per output.  With 32 cells per word, rank(cell) =
// block_first[cell / kBitmapBlockCells] + word_first[cell / 32] + popcount(bits below).
constexpr int kBitmapThreads = 512;
constexpr int kBitmapWordsPerThread = 8;
constexpr int kBitmapBlockWords = kBitmapThreads * kBitmapWordsPerThread;
struct Bitmap {
  uint32_t *words;
  int *word_first;   // set bits before the word, inside its block
  int *block_first;  // set bits before the block
  int n_words, n_blocks;
};

// fills several ranges of 32-bit words in one launch
struct FillRanges {
  uint32_t *ptr[6];
  long long words[6];
  uint32_t value[6];
  int count;
};
__global__ void __launch_bounds__(256) fill_kernel(const FillRanges r) {
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long first = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (int k = 0; k < r.count; ++k) {
    const uint32_t v = r.value[k];
    const long long head = min(r.words[k], static_cast<long long>((16u - (reinterpret_cast<uintptr_t>(r.ptr[k]) & 15u)) & 15u) / 4);
    const long long n4 = (r.words[k] - head) / 4, tail = r.words[k] - head - 4 * n4;
    uint4 *p4 = reinterpret_cast<uint4 *>(r.ptr[k] + head);
    for (long long i = first; i < n4; i += step)
      p4[i] = make_uint4(v, v, v, v);
    if (first < head)
      r.ptr[k][first] = v;
    if (first < tail)
      r.ptr[k][head + 4 * n4 + first] = v;
  }
}

// Output positions that read input coordinate `at` along one axis through offset r: at + pad - r * dil
// divided by the stride, or -1.
__device__ __forceinline__ int out_position(const Geometry &g, int axis, int at, int r) {
  const int num = at + g.pad[axis] - r * g.dil[axis];
  if (num < 0 || num % g.stride[axis] != 0)
    return -1;
  const int p = num / g.stride[axis];
  return p < g.ogrid[axis] ? p : -1;
}

// One thread per (input voxel, rz, ry); bits of one word set together.
__global__ void __launch_bounds__(256) bitmap_mark_kernel(const int32_t *__restrict__ coords, int n, Geometry g,
                                                          uint32_t *words) {
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int planes = g.ksize[0] * g.ksize[1];
  const int i = static_cast<int>(t / planes), zy = static_cast<int>(t % planes);
  if (i >= n)
    return;
  const int4 c = __ldg(reinterpret_cast<const int4 *>(coords) + i);
  if (c.x < 0 || c.x >= g.batch_size)
    return;  // reported with the other bad coordinates when the tables are filled
  const int oz = out_position(g, 0, c.y, zy / g.ksize[1]), oy = out_position(g, 1, c.z, zy % g.ksize[1]);
  if (oz < 0 || oy < 0)
    return;
  const uint32_t line = static_cast<uint32_t>(linear_key(c.x, oz, oy, 0, g.ogrid));
  uint32_t word = 0, bits = 0;
  for (int rx = 0; rx < g.ksize[2]; ++rx) {
    const int ox = out_position(g, 2, c.w, rx);
    if (ox < 0)
      continue;
    const uint32_t cell = line + ox;
    if (bits && (cell >> 5) != word) {
      atomicOr(words + word, bits);
      bits = 0;
    }
    word = cell >> 5;
    bits |= 1u << (cell & 31);
  }
  if (bits)
    atomicOr(words + word, bits);
}

// Exclusive scan over a block of kBitmapThreads values; returns the scan, `total` = the sum.
__device__ __forceinline__ int block_scan_512(int v, int *s_warp, int &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d)
      incl += t;
  }
  __syncthreads();  // s_warp of an earlier call has been read
  if (lane == 31)
    s_warp[warp] = incl;
  __syncthreads();
  int before = 0;
  total = 0;
#pragma unroll
  for (int w = 0; w < 16; ++w) {
    const int x = s_warp[w];
    total += x;
    before += w < warp ? x : 0;
  }
  return before + incl - v;
}

// counters[0] = all set bits, counters[1] = blocks that have counted (zero before the launch).  The
// block that counts last scans the block sums: nobody waits for anybody.
__global__ void __launch_bounds__(kBitmapThreads) bitmap_rank_kernel(const Bitmap bm, int *counters) {
  __shared__ int s_warp[16];
  __shared__ int s_last;
  const int w0 = blockIdx.x * kBitmapBlockWords + threadIdx.x * kBitmapWordsPerThread;
  int pc[kBitmapWordsPerThread], sum = 0;
#pragma unroll
  for (int q = 0; q < kBitmapWordsPerThread; q += 4) {  // the word array is padded to whole blocks
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(bm.words + w0 + q));
    pc[q] = __popc(v.x), pc[q + 1] = __popc(v.y), pc[q + 2] = __popc(v.z), pc[q + 3] = __popc(v.w);
    sum += pc[q] + pc[q + 1] + pc[q + 2] + pc[q + 3];
  }
  int total;
  int run = block_scan_512(sum, s_warp, total);
#pragma unroll
  for (int q = 0; q < kBitmapWordsPerThread; q += 4) {
    int4 f;
    f.x = run, f.y = f.x + pc[q], f.z = f.y + pc[q + 1], f.w = f.z + pc[q + 2];
    run = f.w + pc[q + 3];
    *reinterpret_cast<int4 *>(bm.word_first + w0 + q) = f;
  }
  if (threadIdx.x == 0) {
    bm.block_first[blockIdx.x] = total;
    __threadfence();
    s_last = atomicAdd(counters + 1, 1) == bm.n_blocks - 1;
  }
  __syncthreads();
  if (!s_last)
    return;
  __threadfence();
  int base = 0;
  for (int b0 = 0; b0 < bm.n_blocks; b0 += kBitmapThreads) {
    const int b = b0 + threadIdx.x;
    const int v = b < bm.n_blocks ? __ldcg(bm.block_first + b) : 0;
    const int before = block_scan_512(v, s_warp, total);
    if (b < bm.n_blocks)
      bm.block_first[b] = base + before;
    base += total;
  }
  if (threadIdx.x == 0)
    counters[0] = base;
}

__device__ __forceinline__ int bitmap_rank(const Bitmap &bm, uint32_t cell) {
  const uint32_t w = cell >> 5;
  return __ldg(bm.block_first + w / kBitmapBlockWords) + __ldg(bm.word_first + w) +
         __popc(__ldg(bm.words + w) & ((1u << (cell & 31)) - 1u));
}

// coordinates of the active outputs, in row order; one thread per word
__global__ void __launch_bounds__(256) bitmap_coords_kernel(const Bitmap bm, int n_out, Geometry g, int32_t *out_coords) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= bm.n_words)
    return;
  uint32_t bits = __ldg(bm.words + w);
  if (!bits)
    return;
  int o = bm.block_first[w / kBitmapBlockWords] + bm.word_first[w];
  for (; bits && o < n_out; bits &= bits - 1, ++o) {
    uint32_t k = static_cast<uint32_t>(w) * 32u + (__ffs(bits) - 1);
    const int x = static_cast<int>(k % g.ogrid[2]);
    k /= g.ogrid[2];
    const int y = static_cast<int>(k % g.ogrid[1]);
    k /= g.ogrid[1];
    const int z = static_cast<int>(k % g.ogrid[0]);
    k /= g.ogrid[0];
    reinterpret_cast<int4 *>(out_coords)[o] = make_int4(static_cast<int>(k), z, y, x);
  }
}

// indices[f, o] = i and bit f of row o's mask for every output o that reads input i through f.  The table
// and the masks start as -1 and 0; of several rows with one voxel the smallest wins.
__global__ void __launch_bounds__(256) bitmap_scatter_kernel(const int32_t *__restrict__ coords, int n, Geometry g,
                                                             const Bitmap bm, const MaskSide out, int words, int *status) {
  const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int planes = g.ksize[0] * g.ksize[1];
  const int i = static_cast<int>(t / planes), zy = static_cast<int>(t % planes);
  if (i >= n)
    return;
  const int4 c = __ldg(reinterpret_cast<const int4 *>(coords) + i);
  if (c.x < 0 || c.x >= g.batch_size || c.y < 0 || c.y >= g.grid[0] || c.z < 0 || c.z >= g.grid[1] || c.w < 0 ||
      c.w >= g.grid[2]) {
    atomicCAS(status, 0, kStatusBadCoord);
    return;
  }
  const int oz = out_position(g, 0, c.y, zy / g.ksize[1]), oy = out_position(g, 1, c.z, zy % g.ksize[1]);
  if (oz < 0 || oy < 0)
    return;
  const uint32_t line = static_cast<uint32_t>(linear_key(c.x, oz, oy, 0, g.ogrid));
  for (int rx = 0; rx < g.ksize[2]; ++rx) {
    const int ox = out_position(g, 2, c.w, rx);
    if (ox < 0)
      continue;
    const int o = bitmap_rank(bm, line + ox);
    if (o >= out.n)
      continue;
    const int f = zy * g.ksize[2] + rx;
    atomicMin(reinterpret_cast<uint32_t *>(out.indices) + static_cast<long long>(f) * out.n + o, static_cast<uint32_t>(i));
    atomicOr(out.rows + static_cast<long long>(o) * words + (f >> 5), 1u << (f & 31));
  }
}

// Blocks below `bwd_blocks`: the backward table, indices_bwd[f, i] = o where indices[f, o] = i, and its
// masks.  The other blocks: first-digit counts of the forward masks that the scatter finished.
template <int NW>
__global__ void __launch_bounds__(kProbeThreads) bitmap_backward_kernel(const int32_t *__restrict__ coords, Geometry g,
                                                                        const Bitmap bm, const MaskSide out,
                                                                        const MaskSide in, int bwd_blocks, int words,
                                                                        int width) {
  __shared__ int s_hist[kSortBins];
  if (static_cast<int>(blockIdx.x) >= bwd_blocks) {
    const int block = blockIdx.x - bwd_blocks;
    const int o = block * kProbeThreads + threadIdx.x;
    const bool valid = o < out.n;
    count_first_digit(s_hist, valid, valid ? out.rows[static_cast<long long>(o) * words] : 0u, width, out.hist,
                      block * kProbeThreads / out.chunk);
    return;
  }
  const int i = blockIdx.x * kProbeThreads + threadIdx.x;
  const bool valid = i < in.n;
  uint32_t m[NW];
#pragma unroll
  for (int w = 0; w < NW; ++w)
    m[w] = 0u;
  if (valid) {
    const int4 c = __ldg(reinterpret_cast<const int4 *>(coords) + i);
    const bool ok = c.x >= 0 && c.x < g.batch_size && c.y >= 0 && c.y < g.grid[0] && c.z >= 0 && c.z < g.grid[1] &&
                    c.w >= 0 && c.w < g.grid[2];
    int f = 0;
    for (int rz = 0; rz < g.ksize[0]; ++rz) {
      const int oz = ok ? out_position(g, 0, c.y, rz) : -1;
      for (int ry = 0; ry < g.ksize[1]; ++ry) {
        const int oy = oz >= 0 ? out_position(g, 1, c.z, ry) : -1;
        for (int rx = 0; rx < g.ksize[2]; ++rx, ++f) {
          const int ox = oy >= 0 ? out_position(g, 2, c.w, rx) : -1;
          int found = -1;
          if (ox >= 0) {
            const int o = bitmap_rank(bm, static_cast<uint32_t>(linear_key(c.x, oz, oy, ox, g.ogrid)));
            if (o < out.n && __ldg(out.indices + static_cast<long long>(f) * out.n + o) == i)
              found = o;
          }
          in.indices[static_cast<long long>(f) * in.n + i] = found;
#pragma unroll
          for (int w = 0; w < NW; ++w)
            if (found >= 0 && (NW == 1 || (f >> 5) == w))
              m[w] |= 1u << (f & 31);
        }
      }
    }
#pragma unroll
    for (int w = 0; w < NW; ++w)
      if (w < words)
        in.rows[static_cast<long long>(i) * words + w] = m[w];
  }
  count_first_digit(s_hist, valid, m[0], width, in.hist, blockIdx.x * kProbeThreads / in.chunk);
}

// ---------------------------------------------------------------- one pass of the sort of rows by mask
struct SortSide {
  const uint32_t *rows;  // [n, words] unsorted masks
  const uint32_t *kin;   // one word per mask: the masks in the order of the previous pass; else null
  const int *vin;        // rows in the order of the previous pass; null = 0, 1, 2, ...
  uint32_t *kout;        // one word per mask: the masks in the new order; several: sorted masks, last pass only
  int *vout;
  const int *hist;       // counts of this pass
  int *hist_next;        // counts of the next pass, or null
  uint32_t *tile_masks;  // last pass: OR of the masks of each run of 128 sorted rows (zero before); or null
  int n, chunk, n_chunks;
};
struct SortSides {
  SortSide side[2];
};
template <bool WIDE>
__global__ void __launch_bounds__(kSortThreads) sort_pass_kernel(const SortSides sides, int pass, const SortShape shape) {
  const SortSide &s = sides.side[blockIdx.y];
  __shared__ int s_cnt[kSortWarps][kSortBins];
  __shared__ int s_base[kSortBins];
  __shared__ int s_warp[16];
  const int me = blockIdx.x;
  if (me >= s.n_chunks)
    return;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  // where this chunk's rows of digit t go: rows with smaller digits, then those of earlier chunks
  int before = 0, all = 0;
#pragma unroll 16
  for (int c = 0; c < s.n_chunks; ++c) {
    const int v = __ldg(s.hist + c * kSortBins + t);
    all += v;
    before += c < me ? v : 0;
  }
  int total;
  s_base[t] = block_scan_512(all, s_warp, total) + before;
  const int begin = me * s.chunk, end = min(begin + s.chunk, s.n);
  const int bit0 = pass * shape.width;
  const uint32_t digit_mask = (1u << min(shape.width, shape.bits - bit0)) - 1u;
  const int bit1 = bit0 + shape.width;
  const bool last = bit1 >= shape.bits;
  const uint32_t next_mask = last ? 0u : (1u << min(shape.width, shape.bits - bit1)) - 1u;
  auto wide_digit = [&](int row, int bit, uint32_t mask) -> uint32_t {
    const uint32_t *r = s.rows + static_cast<long long>(row) * shape.words + (bit >> 5);
    const uint32_t lo = __ldg(r);
    const uint32_t hi = (bit & 31) + kSortDigitBits > 32 && (bit >> 5) + 1 < shape.words ? __ldg(r + 1) : 0u;
    return __funnelshift_r(lo, hi, bit & 31) & mask;
  };
  for (int tile = begin; tile < end; tile += kSortThreads * kSortItems) {
    for (int w = 0; w < kSortWarps; ++w)
      s_cnt[w][t] = 0;
    uint32_t key[kSortItems], digit[kSortItems];
    int val[kSortItems], rank[kSortItems];
    const int base = tile + warp * 32 * kSortItems + lane;
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
      const int idx = base + it * 32;
      val[it] = -1;
      key[it] = 0u;
      if (idx < end) {
        val[it] = s.vin ? __ldg(s.vin + idx) : idx;
        if (!WIDE)
          key[it] = __ldg(s.kin + idx);
      }
    }
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
      digit[it] = 0xffffffffu;
      if (val[it] >= 0)
        digit[it] = WIDE ? wide_digit(val[it], bit0, digit_mask) : ((key[it] >> bit0) & digit_mask);
    }
    __syncthreads();
    // rank inside the warp's 32 * kSortItems consecutive rows, in their order
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
      const unsigned peers = __match_any_sync(0xffffffffu, digit[it]);
      rank[it] = 0;
      if (val[it] >= 0)
        rank[it] = s_cnt[warp][digit[it]] + __popc(peers & ((1u << lane) - 1u));
      __syncwarp();
      if (val[it] >= 0 && lane == __ffs(peers) - 1)
        s_cnt[warp][digit[it]] += __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    int run = s_base[t];
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const int c = s_cnt[w][t];
      s_cnt[w][t] = run;
      run += c;
    }
    s_base[t] = run;
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kSortItems; ++it) {
      const bool valid = val[it] >= 0;
      const int pos = valid ? s_cnt[warp][digit[it]] + rank[it] : 0;
      if (valid) {
        s.vout[pos] = val[it];
        if (!WIDE)
          s.kout[pos] = key[it];
      }
      if (!last) {
        uint32_t where = 0xffffffffu;
        if (valid) {
          const uint32_t next = WIDE ? wide_digit(val[it], bit1, next_mask) : ((key[it] >> bit1) & next_mask);
          where = static_cast<uint32_t>(pos / s.chunk) * kSortBins + next;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, where);
        if (valid && lane == __ffs(peers) - 1)
          atomicAdd(s.hist_next + where, __popc(peers));
      } else if (valid) {
        if (WIDE) {
          for (int w = 0; w < shape.words; ++w) {
            const uint32_t m = __ldg(s.rows + static_cast<long long>(val[it]) * shape.words + w);
            s.kout[static_cast<long long>(pos) * shape.words + w] = m;
            if (s.tile_masks)
              atomicOr(s.tile_masks + static_cast<long long>(pos >> 7) * shape.words + w, m);
          }
        } else if (s.tile_masks) {
          atomicOr(s.tile_masks + (pos >> 7), key[it]);
        }
      }
    }
    __syncthreads();
  }
}

// A sequence of gather-GEMM-scatter calls (one per filter offset, each with its own pair lists)
// turned into the neighbour table of ONE convolution: table[f, c_inds_f[i]] = a_inds_f[i].
// One thread per pair; `first[f]` = pairs before call f.
constexpr int kSeqMaxCalls = 32;
struct SeqPairLists {
  const int32_t *a_inds[kSeqMaxCalls];  // null = the pair's own position
  const int32_t *c_inds[kSeqMaxCalls];
  long long first[kSeqMaxCalls + 1];
  int count;
};
__global__ void __launch_bounds__(256) seq_scatter_kernel(SeqPairLists L, int n_out, int a_rows, int32_t *__restrict__ table,
                                                          int *status) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= L.first[L.count])
    return;
  int f = 0;
  while (f + 1 < L.count && t >= L.first[f + 1])
    ++f;
  const long long i = t - L.first[f];
  const int o = L.c_inds[f][i];
  const int a = L.a_inds[f] ? L.a_inds[f][i] : (int)i;
  if (o < 0 || o >= n_out || a < 0 || a >= a_rows) {
    atomicCAS(status, 0, 2);  // row index out of range: reported, not dereferenced
    return;
  }
  table[(long long)f * n_out + o] = a;
}

// Neighbour tables of a DENSE convolution (every grid position is a row, channels last): the
// coordinate rule of the reference's dense iterators, in = out * stride - pad + r * dilation per
// axis (cumm/conv/input_iters.py:2666,2684), written in the layout the row-gather kernels read.
// With them a dense convolution runs through the same kernels as a sparse one whose voxels fill
// the grid.  One thread per (row, filter offset); rows are (batch, z, y, x) row-major.
struct DenseGeometry {
  int batch;
  int in_dims[3], out_dims[3];
  int ksize[3], stride[3], pad[3], dil[3];
  int kv;
};
// forward: indices[f, o] = input row feeding output row o through offset f, or -1
__global__ void __launch_bounds__(256) dense_table_fwd_kernel(DenseGeometry g, long long n_out, int32_t *__restrict__ indices) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_out * g.kv)
    return;
  const int f = (int)(t / n_out);
  const long long o = t % n_out;
  long long rem = o;
  int oc[3];
  for (int a = 2; a >= 0; --a) {
    oc[a] = (int)(rem % g.out_dims[a]);
    rem /= g.out_dims[a];
  }
  const long long b = rem;
  int r[3], fr = f;
  for (int a = 2; a >= 0; --a) {
    r[a] = fr % g.ksize[a];
    fr /= g.ksize[a];
  }
  long long row = b;
  bool ok = true;
  for (int a = 0; a < 3; ++a) {
    const int ic = oc[a] * g.stride[a] - g.pad[a] + r[a] * g.dil[a];
    ok = ok && ic >= 0 && ic < g.in_dims[a];
    row = row * g.in_dims[a] + ic;
  }
  indices[t] = ok ? (int32_t)row : -1;
}
// backward: indices[f, i] = output row that input row i feeds through offset f, or -1
__global__ void __launch_bounds__(256) dense_table_bwd_kernel(DenseGeometry g, long long n_in, int32_t *__restrict__ indices) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_in * g.kv)
    return;
  const int f = (int)(t / n_in);
  const long long i = t % n_in;
  long long rem = i;
  int ic[3];
  for (int a = 2; a >= 0; --a) {
    ic[a] = (int)(rem % g.in_dims[a]);
    rem /= g.in_dims[a];
  }
  const long long b = rem;
  int r[3], fr = f;
  for (int a = 2; a >= 0; --a) {
    r[a] = fr % g.ksize[a];
    fr /= g.ksize[a];
  }
  long long row = b;
  bool ok = true;
  for (int a = 0; a < 3; ++a) {
    const int num = ic[a] + g.pad[a] - r[a] * g.dil[a];
    const int oc = num / g.stride[a];
    ok = ok && num >= 0 && num % g.stride[a] == 0 && oc < g.out_dims[a];
    row = row * g.out_dims[a] + oc;
  }
  indices[t] = ok ? (int32_t)row : -1;
}
// every row carries every offset (the table says which neighbours exist); rows keep their order
__global__ void __launch_bounds__(256) dense_masks_kernel(long long n, int kv, int words, uint32_t *__restrict__ mask,
                                                          int32_t *__restrict__ argsort) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n)
    return;
  argsort[t] = (int32_t)t;
  for (int w = 0; w < words; ++w) {
    const int left = kv - 32 * w;
    mask[t * words + w] = left >= 32 ? 0xffffffffu : (1u << left) - 1u;
  }
}

// ---------------------------------------------------------------- ascending sort of output keys
// Output grids too large for the bitmap: the keys of the active outputs, 8 bits per pass, three
// kernels per pass -- per-tile digit histograms, one exclusive scan over the (digit, tile) matrix, and a
// scatter in which the warps of a block take turns (in element order) to claim their digits' positions.
constexpr int kKeySortThreads = 256;
constexpr int kKeySortItems = 8;
constexpr int kKeySortTile = kKeySortThreads * kKeySortItems;

__global__ void __launch_bounds__(kKeySortThreads) key_hist_kernel(const unsigned long long *__restrict__ keys, int n,
                                                                   int shift, int *hist, int ntiles) {
  __shared__ int h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int base = blockIdx.x * kKeySortTile;
#pragma unroll
  for (int it = 0; it < kKeySortItems; ++it) {
    const int idx = base + it * kKeySortThreads + threadIdx.x;
    if (idx < n)
      atomicAdd(&h[static_cast<int>((keys[idx] >> shift) & 0xff)], 1);
  }
  __syncthreads();
  hist[threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan, in place, of the (digit, tile) count matrix in digit-major order (all tiles of
// digit 0, then digit 1, ...), `total4` int4 in all (the tail beyond 256 * ntiles is padding whose
// values nobody reads).  One block; every thread owns a contiguous run of int4 that it reads
// twice with several loads in flight: the kernel is a handful of memory latencies long.
__global__ void __launch_bounds__(1024) key_scan_kernel(int4 *data, int total4) {
  __shared__ int s_sum[1024];
  const int per = (total4 + 1023) / 1024;
  const int lo = min(threadIdx.x * per, total4), hi = min(lo + per, total4);
  int sum = 0;
#pragma unroll 8
  for (int i = lo; i < hi; ++i) {
    const int4 v = data[i];
    sum += v.x + v.y + v.z + v.w;
  }
  // block-wide exclusive scan of the 1024 sums: warp scans, then a scan of the 32 warp totals
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d)
      incl += t;
  }
  if (lane == 31)
    s_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const int w = s_sum[lane];
    int wi = w;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wi, d);
      if (lane >= d)
        wi += t;
    }
    s_sum[lane] = wi - w;
  }
  __syncthreads();
  int run = s_sum[warp] + incl - sum;
#pragma unroll 8
  for (int i = lo; i < hi; ++i) {
    const int4 v = data[i];
    int4 o;
    o.x = run;
    o.y = run + v.x;
    o.z = o.y + v.y;
    o.w = o.z + v.z;
    run = o.w + v.w;
    data[i] = o;
  }
}

__global__ void __launch_bounds__(kKeySortThreads) key_scatter_kernel(const unsigned long long *__restrict__ kin,
                                                                      unsigned long long *kout, int n, int shift,
                                                                      const int *__restrict__ offsets, int ntiles) {
  __shared__ int cnt[256];
  cnt[threadIdx.x] = offsets[threadIdx.x * ntiles + blockIdx.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int base = blockIdx.x * kKeySortTile;
  for (int it = 0; it < kKeySortItems; ++it) {
    const int idx = base + it * kKeySortThreads + threadIdx.x;
    const bool valid = idx < n;
    const unsigned long long key = valid ? kin[idx] : 0;
    const unsigned digit = valid ? static_cast<unsigned>((key >> shift) & 0xff) : 0x100u + lane;  // invalid: unique
    const unsigned peers = __match_any_sync(0xffffffffu, digit);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    const int leader = __ffs(peers) - 1;
    int claimed = 0;
    for (int w = 0; w < kKeySortThreads / 32; ++w) {
      __syncthreads();
      if (warp == w && valid && rank == 0) {
        claimed = cnt[digit];
        cnt[digit] = claimed + __popc(peers);
      }
    }
    claimed = __shfl_sync(0xffffffffu, claimed, leader);
    if (valid)
      kout[claimed + rank] = key;
  }
}

} // namespace cb2pg
