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
#include <type_traits>

namespace cb2pg {

constexpr unsigned long long kEmptyKey = ~0ULL;
enum : int { kStatusTableFull = 3, kStatusBadCoord = 4 };

struct Geometry {
  int grid[3];    // input grid (z, y, x)
  int ogrid[3];   // output grid
  int ksize[3], stride[3], pad[3], dil[3];
  int period[3];  // stride / gcd(stride, dil): the offsets through which a cell feeds outputs are this far apart
  int drop[3];    // dil / gcd(stride, dil): and those outputs this far
  int kv;
  int batch_size;
};

// Integer mixers: the 64- and (HashKey<true>::bucket) 32-bit finalisers of MurmurHash3 (Austin Appleby, public domain).
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
// One 8-byte word per slot, (tag << 32) | row, all ones = empty; four slots of one 32-byte sector make
// a bucket and are read together.  Four consecutive cells share a bucket, so that the three neighbours
// of one (z, y) line are found in one sector or two.  A full bucket runs over into the next.  While the
// grid has fewer than 2^32 cells the tag IS the linearised voxel (EXACT, all in 32 bits); above, it is
// 32 bits of a hash of it and a match is confirmed against the row's coordinates.
constexpr int kBucket = 4;
struct HashView {
  unsigned long long *slots;
  uint32_t bucket_mask;  // buckets - 1
  const int32_t *coords;
};
template <bool EXACT> struct HashKey;
template <> struct HashKey<true> {
  using Key = uint32_t;
  static __device__ __forceinline__ uint32_t bucket(const HashView &h, Key key) {
    uint32_t k = key >> 2;
    k = (k ^ (k >> 16)) * 0x85ebca6bu;
    k = (k ^ (k >> 13)) * 0xc2b2ae35u;
    return (k ^ (k >> 16)) & h.bucket_mask;
  }
  static __device__ __forceinline__ uint32_t tag(Key key) { return key; }
};
template <> struct HashKey<false> {
  using Key = unsigned long long;
  static __device__ __forceinline__ uint32_t bucket(const HashView &h, Key key) { return mix64(key >> 2) & h.bucket_mask; }
  static __device__ __forceinline__ uint32_t tag(Key key) { return static_cast<uint32_t>((key * 0x9e3779b97f4a7c15ULL) >> 32); }
};
template <bool EXACT>
__device__ __forceinline__ bool hash_match(const HashView &h, unsigned long long entry, uint32_t tag, int b, int z,
                                           int y, int x) {
  if (entry == kEmptyKey || static_cast<uint32_t>(entry >> 32) != tag)
    return false;
  if (EXACT)
    return true;
  const int4 c = __ldg(reinterpret_cast<const int4 *>(h.coords) + static_cast<uint32_t>(entry));
  return c.x == b && c.y == z && c.z == y && c.w == x;
}
struct BucketWords {
  ulonglong2 lo, hi;
};
__device__ __forceinline__ BucketWords load_bucket(const HashView &h, uint32_t bucket) {
  const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(h.slots + static_cast<size_t>(bucket) * kBucket);
  return {__ldg(p), __ldg(p + 1)};
}
// row of the voxel among a bucket's entries, -1 = not there, -2 = the bucket is full: look in the next
template <bool EXACT>
__device__ __forceinline__ int find_in_bucket(const HashView &h, const BucketWords &w, uint32_t tag, int b, int z, int y,
                                              int x) {
  const unsigned long long e[kBucket] = {w.lo.x, w.lo.y, w.hi.x, w.hi.y};
#pragma unroll
  for (int i = 0; i < kBucket; ++i)
    if (hash_match<EXACT>(h, e[i], tag, b, z, y, x))
      return static_cast<int>(static_cast<uint32_t>(e[i]));
  return e[kBucket - 1] == kEmptyKey ? -1 : -2;
}

template <bool EXACT>
__global__ void __launch_bounds__(256) hash_insert_kernel(const int32_t *__restrict__ coords, int n, Geometry g,
                                                          HashView h, int *status) {
  cb2::grid_dep_wait();
  using HK = HashKey<EXACT>;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const int4 c = reinterpret_cast<const int4 *>(coords)[i];
  if (c.x < 0 || c.x >= g.batch_size || c.y < 0 || c.y >= g.grid[0] || c.z < 0 || c.z >= g.grid[1] || c.w < 0 ||
      c.w >= g.grid[2]) {
    atomicCAS(status, 0, kStatusBadCoord);
    return;
  }
  const typename HK::Key key = static_cast<typename HK::Key>(linear_key(c.x, c.y, c.z, c.w, g.grid));
  const uint32_t tag = HK::tag(key);
  const unsigned long long entry = (static_cast<unsigned long long>(tag) << 32) | static_cast<uint32_t>(i);
  uint32_t bucket = HK::bucket(h, key);
  for (uint32_t probe = 0; probe <= h.bucket_mask; ++probe) {
    unsigned long long *slot = h.slots + static_cast<size_t>(bucket) * kBucket;
    for (int q = 0; q < kBucket; ++q, ++slot) {
      const unsigned long long prev = atomicCAS(slot, kEmptyKey, entry);
      if (prev == kEmptyKey)
        return;
      if (hash_match<EXACT>(h, prev, tag, c.x, c.y, c.z, c.w)) {
        atomicMin(slot, entry);  // duplicates resolve to the first row, as a stable sort + search does
        return;
      }
    }
    bucket = (bucket + 1) & h.bucket_mask;
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
// scatters, so a pass is one launch (it was three: count, scan, scatter).  Chunks lie 2 KB apart: with a
// digit's counts side by side the updates of all CTAs met in the same few lines (45 instead of 28 us).
constexpr int kSortDigitBits = 9;
constexpr int kSortBins = 1 << kSortDigitBits;
// Two sides (forward and backward tables) of one size fill the 148 SMs of this part (tables of 960 000 rows:
// 364 us; 410 with 37 chunks, 371 with 148; a stride-2 table of 491 000 outputs 198, 230 and 208).
constexpr int kSortChunks = 74;
constexpr size_t kSortHistInts = static_cast<size_t>(kSortBins) * kSortChunks;  // of a pass
constexpr int kSortThreads = kSortBins;
constexpr int kSortWarps = kSortThreads / 32;
// Rows per thread and round: as many as a chunk needs, up to eight.  (Table sets of chunks of 2048 rows, eight and four, us:
// 150 000 uniform rows 75.9 and 71.7, scanned ones 107.4 and 104.8, 125 offsets, 30 011 rows, 419 and 379; of chunks of 6656, stride 2
// from 150 000 rows, 164.8 and 172.1.)
constexpr int kSortItems = 8, kSortItemsSmall = 4;
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
// The lanes that hold the same digit (of `width` bits; lanes outside `valid` are nobody's peers): a vote
// per bit, which is faster than match.any.
__device__ __forceinline__ unsigned digit_peers(uint32_t digit, int width, unsigned valid) {
  unsigned peers = valid;
  for (int b = 0; b < width; ++b) {
    const bool bit = (digit >> b) & 1u;
    const unsigned v = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? v : ~v;
  }
  return peers;
}

// Counts the first digit of one row per thread into the block's chunk (all threads of a block of
// kProbeThreads take part; the block's rows lie in one chunk).
__device__ __forceinline__ void count_first_digit(int *s_hist, bool valid, uint32_t low_word, int width, int *hist,
                                                  int chunk_index) {
  for (int d = threadIdx.x; d < kSortBins; d += blockDim.x)
    s_hist[d] = 0;
  __syncthreads();
  const uint32_t digit = low_word & ((1u << width) - 1u);
  // most rows of a sparse scene share one mask
  const unsigned peers = digit_peers(digit, width, __ballot_sync(0xffffffffu, valid));
  if (valid && static_cast<int>(threadIdx.x & 31) == __ffs(peers) - 1)
    atomicAdd(&s_hist[digit], __popc(peers));
  __syncthreads();
  for (int d = threadIdx.x; d < kSortBins; d += blockDim.x)
    if (s_hist[d])
      atomicAdd(hist + chunk_index * kSortBins + d, s_hist[d]);
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
// table.  Lookups are issued three at a time, so that their loads are in flight together.
// `mirror` (submanifold convolutions whose offsets are symmetric): o' is o's neighbour at offset f
// exactly if o is o's neighbour at offset kv - 1 - f, so the backward table is the forward one with
// the offsets reversed and is written by the same thread.  A row that repeats another row's voxel
// has no backward neighbours (nothing points at it).
template <int NW, bool EXACT>
__global__ void __launch_bounds__(kProbeThreads, 4) probe_kernel(const int32_t *__restrict__ out_coords, Geometry g,
                                                              const HashView h, const MaskSide side,
                                                              const MaskSide mirror, int words, int width) {
  cb2::grid_dep_wait();
  constexpr int B = 3;
  using HK = HashKey<EXACT>;
  using Key = typename HK::Key;
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
    // linear index of offset 0's cell; modulo the word where that cell lies outside, which is never looked up
    const Key line = (static_cast<Key>(c.x) * g.grid[0] + z0) * g.grid[1] + y0;
    int rz = 0, ry = 0, rx = 0;
    bool repeats = false;
    for (int f0 = 0; f0 < g.kv; f0 += B) {
      BucketWords found[B];
      uint32_t bucket[B], tag[B];
      bool in[B];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        const int z = z0 + rz * g.dil[0], y = y0 + ry * g.dil[1], x = x0 + rx * g.dil[2];
        in[j] = f0 + j < g.kv && z >= 0 && z < g.grid[0] && y >= 0 && y < g.grid[1] && x >= 0 && x < g.grid[2];
        const Key key = (line + static_cast<Key>(rz * g.dil[0]) * g.grid[1] + ry * g.dil[1]) * g.grid[2] + x;
        bucket[j] = in[j] ? HK::bucket(h, key) : 0u;
        tag[j] = HK::tag(key);
        if (j > 0 && bucket[j] == bucket[j - 1])
          found[j] = found[j - 1];
        else
          found[j] = load_bucket(h, bucket[j]);
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
          if (in[j]) {
            int z = 0, y = 0, x = 0;
            if (!EXACT) {
              const int xy = g.ksize[1] * g.ksize[2];
              z = z0 + f / xy * g.dil[0], y = y0 + f % xy / g.ksize[2] * g.dil[1], x = x0 + f % g.ksize[2] * g.dil[2];
            }
            idx = find_in_bucket<EXACT>(h, found[j], tag[j], c.x, z, y, x);
            for (uint32_t probe = 0; idx == -2 && probe < h.bucket_mask; ++probe) {
              bucket[j] = (bucket[j] + 1) & h.bucket_mask;
              idx = find_in_bucket<EXACT>(h, load_bucket(h, bucket[j]), tag[j], c.x, z, y, x);
            }
            idx = max(idx, -1);
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
__global__ void __launch_bounds__(256) fill_kernel(const __grid_constant__ FillRanges r) {  // one grid row per range
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long first = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  uint32_t *ptr = r.ptr[blockIdx.y];
  const long long words = r.words[blockIdx.y];
  const uint32_t v = r.value[blockIdx.y];
  const long long head = min(words, static_cast<long long>((16u - (reinterpret_cast<uintptr_t>(ptr) & 15u)) & 15u) / 4);
  const long long n4 = (words - head) / 4, tail = words - head - 4 * n4;
  uint4 *p4 = reinterpret_cast<uint4 *>(ptr + head);
#pragma unroll 4
  for (long long i = first; i < n4; i += step)
    p4[i] = make_uint4(v, v, v, v);
  if (first < head)
    ptr[first] = v;
  if (first < tail)
    ptr[head + 4 * n4 + first] = v;
}

// The outputs that read a cell, one axis: through offsets r, r + period, ... at positions p, p - drop, ...
// Every lane walks its own offsets (two or fewer per axis for a 3x3x3 kernel of stride 2), where a loop
// over all offsets would run each of them for the whole warp.
struct AxisWalk {
  int r, p;
};
__device__ __forceinline__ AxisWalk first_output(const Geometry &g, int axis, int at) {
  AxisWalk w = {0, 0};
  for (; w.r < g.period[axis]; ++w.r) {
    const int num = at + g.pad[axis] - w.r * g.dil[axis];
    w.p = num / g.stride[axis];
    if (w.p * g.stride[axis] == num)
      return w;
  }
  w.r = g.ksize[axis];  // none
  return w;
}
// fn(f, cell) for every output cell the voxel feeds and the offset it feeds it through
template <class Fn> __device__ __forceinline__ void for_each_output(const Geometry &g, const int4 &c, Fn fn) {
  const AxisWalk wz = first_output(g, 0, c.y), wy = first_output(g, 1, c.z), wx = first_output(g, 2, c.w);
  for (int rz = wz.r, oz = wz.p; rz < g.ksize[0]; rz += g.period[0], oz -= g.drop[0]) {
    if (oz < 0 || oz >= g.ogrid[0])
      continue;
    for (int ry = wy.r, oy = wy.p; ry < g.ksize[1]; ry += g.period[1], oy -= g.drop[1]) {
      if (oy < 0 || oy >= g.ogrid[1])
        continue;
      const uint32_t line = static_cast<uint32_t>((c.x * g.ogrid[0] + oz) * g.ogrid[1] + oy) * g.ogrid[2];
      for (int rx = wx.r, ox = wx.p; rx < g.ksize[2]; rx += g.period[2], ox -= g.drop[2])
        if (ox >= 0 && ox < g.ogrid[2])
          fn((rz * g.ksize[1] + ry) * g.ksize[2] + rx, line + ox);
    }
  }
}
__device__ __forceinline__ bool inside(const Geometry &g, const int4 &c) {
  return c.x >= 0 && c.x < g.batch_size && c.y >= 0 && c.y < g.grid[0] && c.z >= 0 && c.z < g.grid[1] && c.w >= 0 &&
         c.w < g.grid[2];
}

// One thread per input voxel; bits of one word set together.
__global__ void __launch_bounds__(128) bitmap_mark_kernel(const int32_t *__restrict__ coords, int n, Geometry g,
                                                          uint32_t *words) {
  cb2::grid_dep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const int4 c = __ldg(reinterpret_cast<const int4 *>(coords) + i);
  if (c.x < 0 || c.x >= g.batch_size)
    return;  // reported with the other bad coordinates when the tables are filled
  uint32_t word = 0, bits = 0;
  for_each_output(g, c, [&](int, uint32_t cell) {
    if (bits && (cell >> 5) != word) {
      atomicOr(words + word, bits);
      bits = 0;
    }
    word = cell >> 5;
    bits |= 1u << (cell & 31);
  });
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
  cb2::grid_dep_wait();
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
  cb2::grid_dep_wait();
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
__global__ void __launch_bounds__(128) bitmap_scatter_kernel(const int32_t *__restrict__ coords, int n, Geometry g,
                                                             const Bitmap bm, const MaskSide out, int words, int *status) {
  cb2::grid_dep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  const int4 c = __ldg(reinterpret_cast<const int4 *>(coords) + i);
  if (!inside(g, c)) {
    atomicCAS(status, 0, kStatusBadCoord);
    return;
  }
  for_each_output(g, c, [&](int f, uint32_t cell) {
    const int o = bitmap_rank(bm, cell);
    if (o < out.n) {
      atomicMin(reinterpret_cast<uint32_t *>(out.indices) + static_cast<long long>(f) * out.n + o, static_cast<uint32_t>(i));
      atomicOr(out.rows + static_cast<long long>(o) * words + (f >> 5), 1u << (f & 31));
    }
  });
}

// Blocks below `bwd_blocks`: the backward table, indices_bwd[f, i] = o where indices[f, o] = i (-1
// before), and its masks.  The other blocks: first-digit counts of the forward masks that the scatter
// finished.
template <int NW>
__global__ void __launch_bounds__(kProbeThreads) bitmap_backward_kernel(const int32_t *__restrict__ coords, Geometry g,
                                                                        const Bitmap bm, const MaskSide out,
                                                                        const MaskSide in, int bwd_blocks, int words,
                                                                        int width) {
  cb2::grid_dep_wait();
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
    if (inside(g, c))
      for_each_output(g, c, [&](int f, uint32_t cell) {
        const int o = bitmap_rank(bm, cell);
        if (o < out.n && __ldg(out.indices + static_cast<long long>(f) * out.n + o) == i) {
          in.indices[static_cast<long long>(f) * in.n + i] = o;
#pragma unroll
          for (int w = 0; w < NW; ++w)
            if (NW == 1 || (f >> 5) == w)
              m[w] |= 1u << (f & 31);
        }
      });
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
// FEW: chunks of kSortItemsSmall rows per thread.
template <bool WIDE, bool FEW>
__global__ void __launch_bounds__(kSortThreads) sort_pass_kernel(const __grid_constant__ SortSides sides, int pass,
                                                                 const SortShape shape) {
  cb2::grid_dep_wait();
  constexpr int kItems = FEW ? kSortItemsSmall : kSortItems;
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
  // All loads in flight together: one after the other they were most of a pass, three times 25 of them still 3 us of a set of
  // 150 000 rows (78.9 -> 75.9); for few chunks the 74 cost as much as they save (20 000 rows 57.2 -> 60.7).
  auto count = [&](auto many, int c0) {
    constexpr int N = decltype(many)::value;
    int v[N];
#pragma unroll
    for (int i = 0; i < N; ++i)
      v[i] = c0 + i < s.n_chunks ? __ldg(s.hist + (c0 + i) * kSortBins + t) : 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      all += v[i];
      before += c0 + i < me ? v[i] : 0;
    }
  };
  // Never more chunks than kSortChunks.  Written as a loop of that one round all the same where a thread has four rows
  // (72 us, straight 78), straight where it has eight (164 us, as a loop 174, stride 2): what the compiler makes of it.
  if (s.n_chunks <= 25)
    count(std::integral_constant<int, 25>(), 0);
  else if constexpr (FEW)
    for (int c0 = 0; c0 < s.n_chunks; c0 += kSortChunks)
      count(std::integral_constant<int, kSortChunks>(), c0);
  else
    count(std::integral_constant<int, kSortChunks>(), 0);
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
  for (int tile = begin; tile < end; tile += kSortThreads * kItems) {
    for (int w = 0; w < kSortWarps; ++w)
      s_cnt[w][t] = 0;
    uint32_t key[kItems], digit[kItems];
    int val[kItems], rank[kItems];
    const int base = tile + warp * 32 * kItems + lane;
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
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
    for (int it = 0; it < kItems; ++it) {
      digit[it] = 0u;
      if (val[it] >= 0)
        digit[it] = WIDE ? wide_digit(val[it], bit0, digit_mask) : ((key[it] >> bit0) & digit_mask);
    }
    __syncthreads();
    // rank inside the warp's 32 * kItems consecutive rows, in their order
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
      const unsigned peers = digit_peers(digit[it], shape.width, __ballot_sync(0xffffffffu, val[it] >= 0));
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
    for (int it = 0; it < kItems; ++it) {
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
        // Most rows of a sparse scene share one mask and stay together: the lanes that agree with the
        // first one are counted in one update.
        const uint32_t where0 = __shfl_sync(0xffffffffu, where, 0);
        const unsigned agree = __ballot_sync(0xffffffffu, where == where0);
        if (lane == 0 && valid)
          atomicAdd(s.hist_next + where, __popc(agree));
        else if (valid && where != where0)
          atomicAdd(s.hist_next + where, 1);
      } else {
        const int run = valid ? pos >> 7 : -1;  // the same for tile masks
        const int run0 = __shfl_sync(0xffffffffu, run, 0);
        const bool agrees = valid && run == run0;
        for (int w = 0; w < (WIDE ? shape.words : 1); ++w) {
          uint32_t m = key[it];
          if (WIDE && valid) {
            m = __ldg(s.rows + static_cast<long long>(val[it]) * shape.words + w);
            s.kout[static_cast<long long>(pos) * shape.words + w] = m;
          }
          if (s.tile_masks) {
            const uint32_t any = __reduce_or_sync(0xffffffffu, agrees ? m : 0u);
            if (valid && (lane == 0 || !agrees))
              atomicOr(s.tile_masks + static_cast<long long>(run) * shape.words + w, lane == 0 ? any : m);
          }
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
