// C ABI of the library: argument validation (the checks of the reference's host
// prologues, cumm/gemm/nvrtc_code.py:34-146 and cumm/conv/nvrtc_code.py:20-260), kernel
// selection, TMA descriptor set-up and launches.  No CPU compute path exists here: when
// no kernel fits the descriptor the call fails with CB2_ERR_UNSUPPORTED.
#include "../../include/cumm_b200.h"
#include "rowconv_kernel.cuh"
#include "wgrad_kernel.cuh"
#include "pairgen_kernels.cuh"
#include "peer_reduce_kernel.cuh"

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>

#ifndef CB2_DEFAULT_GATHER
#define CB2_DEFAULT_GATHER 2
#endif

namespace {

using namespace cb2;

thread_local std::string g_err;
std::atomic<uint64_t> g_launches{0};
struct LaunchInfo {
  int num_regs = 0, num_threads = 0, smem_bytes = 0, cluster = 1;
};
thread_local LaunchInfo g_last_launch;
template <class Kern> int kernel_regs(Kern kern) {
  cudaFuncAttributes attr;
  return cudaFuncGetAttributes(&attr, kern) == cudaSuccess ? attr.numRegs : 0;
}

int set_err(int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

#define CB2_CHECK_ARG(cond, ...)                                                                   \
  do {                                                                                             \
    if (!(cond))                                                                                   \
      return set_err(CB2_ERR_INVALID_ARG, __VA_ARGS__);                                            \
  } while (0)
#define CB2_CHECK_RT(cond, ...)                                                                    \
  do {                                                                                             \
    if (!(cond))                                                                                   \
      return set_err(CB2_ERR_RUNTIME, __VA_ARGS__);                                                \
  } while (0)
#define CB2_CUDA(expr)                                                                             \
  do {                                                                                             \
    cudaError_t e__ = (expr);                                                                      \
    if (e__ != cudaSuccess)                                                                        \
      return set_err(CB2_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e__));               \
  } while (0)

constexpr int kMaxDevices = 64;
constexpr int kTicketSlots = 256;
constexpr size_t kStatusBytes = (16 + 2 * kTicketSlots) * sizeof(int);

struct DeviceState {
  bool ready = false;
  int num_sms = 0;
  int *status = nullptr;
};
DeviceState g_dev[kMaxDevices];
std::mutex g_mu;

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;

int get_device(DeviceState **out) {
  int dev = 0;
  CB2_CUDA(cudaGetDevice(&dev));
  CB2_CHECK_RT(dev >= 0 && dev < kMaxDevices, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_mu);
  DeviceState &st = g_dev[dev];
  if (!st.ready) {
    cudaDeviceProp prop;
    CB2_CUDA(cudaGetDeviceProperties(&prop, dev));
    CB2_CHECK_RT(prop.major == 10, "cumm_b200 kernels are built for sm_100a only; device %d is sm_%d%d",
                 dev, prop.major, prop.minor);
    st.num_sms = prop.multiProcessorCount;
    // word 0: kernel status; from word 16 on: kTicketSlots pairs of scheduling counters
    CB2_CUDA(cudaMalloc(&st.status, kStatusBytes));
    CB2_CUDA(cudaMemset(st.status, 0, kStatusBytes));
    st.ready = true;
  }
  if (!g_encode) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    CB2_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
    CB2_CHECK_RT(fn != nullptr && q == cudaDriverEntryPointSuccess, "cuTensorMapEncodeTiled not available");
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  *out = &st;
  return CB2_OK;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// 3-D tensor map over a weight-like tensor [outer, mid, inner] (inner contiguous).
int make_weight_map(CUtensorMap *map, const void *ptr, int es, uint64_t inner, uint64_t mid, uint64_t outer,
                    uint64_t mid_stride_elems, uint64_t outer_stride_elems, uint32_t box_inner,
                    uint32_t box_outer) {
  cuuint64_t dims[3] = {inner, mid, outer};
  cuuint64_t strides[2] = {mid_stride_elems * es, outer_stride_elems * es};
  cuuint32_t box[3] = {box_inner, 1, box_outer};
  cuuint32_t estr[3] = {1, 1, 1};
  CB2_CHECK_ARG(aligned16(ptr), "weight pointer must be 16-byte aligned");
  CB2_CHECK_ARG(strides[0] % 16 == 0 && strides[1] % 16 == 0, "weight strides must be multiples of 16 bytes");
  CUresult r = g_encode(map, es == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3,
                        const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  CB2_CHECK_RT(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  return CB2_OK;
}

// 2-D tensor map over gathered operand rows [rows, width] (row stride ld elements); the box is
// one row of 128 bytes, so a gather is one request per (row, column block).
int make_rows_map(CUtensorMap *map, const void *ptr, int es, uint64_t width, uint64_t rows, uint64_t ld) {
  cuuint64_t dims[2] = {width, rows > 0 ? rows : 1};
  cuuint64_t strides[1] = {ld * es};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / es), 1};
  cuuint32_t estr[2] = {1, 1};
  CB2_CHECK_ARG(aligned16(ptr), "operand pointer must be 16-byte aligned");
  CB2_CHECK_ARG(strides[0] % 16 == 0, "operand row stride must be a multiple of 16 bytes");
  CUresult r = g_encode(map, es == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2,
                        const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  CB2_CHECK_RT(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled (rows) failed with code %d", (int)r);
  return CB2_OK;
}

// Which row-gather implementation the kernels use: 0 cp.async, otherwise TMA gather4.
int gather_mode() {
  static int mode = -1;
  if (mode < 0) {
    int m = CB2_DEFAULT_GATHER;
    if (const char *v = getenv("CUMM_B200_GATHER"))
      m = atoi(v);
    mode = (m >= 0 && m <= 2) ? m : CB2_DEFAULT_GATHER;
  }
  return mode;
}

// Launch with programmatic stream serialisation: the kernel may be scheduled while its
// predecessor on the stream is still running and synchronises with it through
// griddepcontrol.wait in its own code.  CUMM_B200_PDL=0 launches everything the ordinary way.
// The planning kernels of the weight gradient do not take part: their blocks would wait beside the row kernel before them (a
// training step with 125 offsets 155.8 -> 177.7 us).
// The kernels of table generation take part too, but none triggers its dependent: a dependent's launch overlaps the
// predecessor's end and no more (150 000 uniform rows, us: ordinary launches 85.4 and, stride 2, 186; so 76.5 and 170;
// triggered as soon as a kernel starts 91.5 and 199, its successor's waiting blocks hold the SMs).
// int8 convolutions and gather-GEMM-scatter calls read their tables and row lists before their own wait (if they waited:
// int8, stride 2 from 150 000 rows, 40.9 -> 42.4 us).  PTX asks a dependent to wait where its prerequisite
// issues launch_dependents; the kernels that make tables here do not, so their blocks have all ended by then.
template <class Kern, class... Args>
cudaError_t launch_after(int cluster, Kern kern, dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                         Args... args) {
  static const bool pdl = [] {
    const char *v = getenv("CUMM_B200_PDL");
    return !v || atoi(v) > 0;
  }();
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (pdl) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = cluster;
    attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// How many CTAs share an item's filter offsets in a launch whose items leave most SMs idle: 4 or 8 where the clusters
// fit the CTAs the launch may have and are all resident at once (each has one item; 148 SMs hold 33 clusters of four and
// 15 of eight), else 1, and the ordinary kernel runs.  Four from two offsets a CTA on, eight from
// eight: with ordinary launches both sides were even there (8 offsets, 2000 and 3800 rows at 64 channels, us, one CTA and
// four: 8.8 and 8.8, 9.6 and 9.6).  Overlap with the predecessor has since done more for one CTA than for four, which pay from 16
// offsets on now, at 128 channels from 12; the line has not followed.  (One forward after the other over fixed tables, us, one CTA
// and four.  8 offsets: crops of 1000, 1900 and 3800 rows at 64 channels 4.8 and 6.2, 5.0 and 6.3,
// 5.6 and 9.2, 1900 at 128 7.8 and 7.7; 12: 5.8 and 6.3, 6.5 and 6.7, 6.8 and 9.4, at 128 10.2 and 8.5; 18: 7.7 and 7.0, 8.3 and 7.3, 8.5
// and 10.0, 13.4 and 9.4; 27: 10.0 and 7.5, 10.7 and 7.9, 11.1 and 10.8, 18.2 and 10.5, scanned scenes of 2000 rows 9.5 and 7.1, uniform
// ones, whose tiles stay with one CTA of the cluster, 3.9 and 4.5.  125 offsets at 32 channels, one CTA, four and eight: crops of 1900
// rows 45.4, 15.5 and 16.2; four and eight: of 1000 rows 14.1 and 11.7, scanned scenes of 1000 rows 12.0 and 8.9.)
// `resident`: per device, clusters of 4 and 8 CTAs of this kernel that it holds, plus one (0 = not known yet: not
// asked, or without an answer).
using ResidentClusters = std::atomic<int>[kMaxDevices][2];
template <class Kern>
int cluster_split(Kern kern, ResidentClusters &resident, int threads, int smem, int max_ctas, long long items, int kv) {
  int dev = 0;
  if (4 * items > max_ctas || kv < 8 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return 1;
  for (int e = 1; e >= 0; --e) {
    const int split = 4 << e;
    if (items * split > max_ctas || kv < (e ? 64 : 8))
      continue;
    int n = resident[dev][e].load();
    if (n == 0) {
      cudaLaunchConfig_t cfg;
      memset(&cfg, 0, sizeof(cfg));
      cfg.gridDim = dim3(split);
      cfg.blockDim = dim3(threads);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = split;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int found = 0;
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&found, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 1;
      }
      n = found + 1;
      resident[dev][e].store(n);
    }
    if (items <= n - 1)
      return split;
  }
  return 1;
}

template <int KIND, int NATOM_K, int BLOCK_N, bool B_MN, bool TMA_GATHER, int MW = 1, bool SPLIT = false>
int launch_rowconv_inst(const CUtensorMap &map, const CUtensorMap &map_a, const RowConvParams &p, int gx, int gy,
                        int max_ctas, cudaStream_t stream) {
  using Cfg = RowConvCfg<KIND, NATOM_K, BLOCK_N, B_MN, TMA_GATHER, MW>;
  auto kern = rowconv_kernel<KIND, NATOM_K, BLOCK_N, B_MN, TMA_GATHER, MW, SPLIT>;
  if constexpr (!SPLIT && KIND == 0 && TMA_GATHER) {
    static ResidentClusters resident;
    const long long items = (p.n_rows + 127) / 128 * static_cast<long long>(p.n_parts);
    RowConvParams shared = p;
    shared.split = p.mode != kModeMaskConv ? 1
                                           : cluster_split(rowconv_kernel<KIND, NATOM_K, BLOCK_N, B_MN, TMA_GATHER, MW, true>,
                                                           resident, Cfg::THREADS, Cfg::SMEM_BYTES, max_ctas, items, p.kv);
    if (shared.split > 1)
      return launch_rowconv_inst<KIND, NATOM_K, BLOCK_N, B_MN, TMA_GATHER, MW, true>(map, map_a, shared, gx, gy, max_ctas,
                                                                                     stream);
  }
  static std::atomic<uint64_t> configured{0};  // bit per device
  static std::atomic<int> regs{0};
  int dev = 0;
  CB2_CUDA(cudaGetDevice(&dev));
  if (!(configured.load() & (1ull << dev))) {
    CB2_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    regs.store(kernel_regs(kern));
    configured.fetch_or(1ull << dev);
  }
  const int cluster = SPLIT ? p.split : 1;
  g_last_launch.num_regs = regs.load();
  g_last_launch.num_threads = Cfg::THREADS;
  g_last_launch.smem_bytes = Cfg::SMEM_BYTES;
  g_last_launch.cluster = cluster;
  // Every row kernel's launch and set-up overlaps its predecessor's end.  It nearly halves a run of gather-GEMM-scatter
  // calls; int8 convolutions gain 4 %; fp16 ones, which wait before they read a table: one forward after the other, us,
  // 58 787 uniform rows, 40 to 56, 14.7 -> 11.5, 42 077 at 128 18.3 -> 15.9, 60 000 scanned ones at 256 102.4 -> 99.0, training steps
  // that plan each time 1 to 13 % less.  With tables that an earlier call found as they are, tickets, masks and indices are
  // read under the predecessor's end, too.  (Forward, input and weight gradient in turn, ordinary launches and
  // overlapped: 150 000 uniform rows at 128 channels 84.0 and 77.8, 100 003 scanned ones at 64 100.1 and 94.2, stride 2 from
  // 40 009, 32 to 64, 46.6 and 41.0, 9000 at 128 62.0 and 56.1, 125 offsets, 30 011 rows, 136.2 and 127.5.)
  CB2_CUDA(launch_after(cluster, kern, dim3(gx * cluster, gy), dim3(Cfg::THREADS), Cfg::SMEM_BYTES, stream, map, map_a, p));
  g_launches.fetch_add(1);
  return CB2_OK;
}

struct RowConvPlan {
  int kind;     // 0 f16, 1 s8
  int natom_k;  // 1 or 2
  int block_n;  // 64 or 128
  bool b_mn;
};

// tile_n / tile_k: GemmAlgoDesp::tile_shape[1] / [2] of the caller's descriptor (0 = choose from the
// problem: the narrowest tile that covers the output width / the reduction width).
int plan_rowconv(int kind, int red, int nn, bool b_mn, int tile_n, int tile_k, RowConvPlan *plan) {
  plan->kind = kind;
  plan->b_mn = b_mn;
  const int atom = kind == 0 ? 64 : 128;
  if (tile_n != 0 && tile_n != 64 && tile_n != 128)
    return set_err(CB2_ERR_UNSUPPORTED, "can't find any suitable algo: tile_shape[1] = %d (kernels exist for 64 and 128)",
                   tile_n);
  if (tile_k != 0 && tile_k != atom && !(kind == 0 && tile_k == 2 * atom))
    return set_err(CB2_ERR_UNSUPPORTED, "can't find any suitable algo: tile_shape[2] = %d (kernels exist for %d%s)",
                   tile_k, atom, kind == 0 ? " and 128" : "");
  plan->natom_k = tile_k ? tile_k / atom : ((kind == 0 && red > atom) ? 2 : 1);
  plan->block_n = tile_n ? tile_n : (nn <= 64 ? 64 : 128);
  if (kind == 1 && b_mn)
    return set_err(CB2_ERR_UNSUPPORTED, "int8 is supported for forward only (the reference skips 1-byte "
                                        "dtypes for backward ops)");
  return CB2_OK;
}

int launch_rowconv(const RowConvPlan &pl, const CUtensorMap &map, const CUtensorMap &map_a, bool tma_gather,
                   const RowConvParams &p, int gx, int gy, int max_ctas, cudaStream_t s) {
  // Kernel volumes above 32 (several mask words per row): no cp.async variant for rows of up to 128
  // bytes.
#define CB2_INST(K, A, N, M)                                                                      \
  if (pl.kind == K && pl.natom_k == A && pl.block_n == N && pl.b_mn == M) {                        \
    if (p.mask_words > 1)                                                                          \
      return tma_gather ? launch_rowconv_inst<K, A, N, M, true, 4>(map, map_a, p, gx, gy, max_ctas, s)       \
                        : launch_rowconv_inst<K, A, N, M, A == 1, 4>(map, map_a, p, gx, gy, max_ctas, s);    \
    return tma_gather ? launch_rowconv_inst<K, A, N, M, true>(map, map_a, p, gx, gy, max_ctas, s)            \
                      : launch_rowconv_inst<K, A, N, M, false>(map, map_a, p, gx, gy, max_ctas, s);          \
  }
  CB2_INST(0, 1, 64, false)
  CB2_INST(0, 1, 128, false)
  CB2_INST(0, 2, 64, false)
  CB2_INST(0, 2, 128, false)
  CB2_INST(0, 1, 64, true)
  CB2_INST(0, 1, 128, true)
  CB2_INST(0, 2, 64, true)
  CB2_INST(0, 2, 128, true)
  CB2_INST(1, 1, 64, false)
  CB2_INST(1, 1, 128, false)
#undef CB2_INST
  return set_err(CB2_ERR_UNSUPPORTED, "no row-conv kernel for kind=%d natom=%d block_n=%d b_mn=%d", pl.kind,
                 pl.natom_k, pl.block_n, (int)pl.b_mn);
}

// Common tail of the row-gather launches (forward, backward input, ShuffleAC GEMM).
int run_rowconv(DeviceState *dev, RowConvParams &p, int kind, bool b_mn, int tile_n, int tile_k, void *sched_scratch,
                int max_ctas, const void *w_ptr, uint64_t w_inner, uint64_t w_mid, uint64_t w_outer,
                uint64_t w_mid_stride, uint64_t w_outer_stride, cudaStream_t stream) {
  RowConvPlan pl;
  int rc = plan_rowconv(kind, p.red, p.nn, b_mn, tile_n, tile_k, &pl);
  if (rc)
    return rc;
  const int es = kind == 0 ? 2 : 1;
  const int atom = 128 / es;
  const int kred = pl.natom_k * atom;
  CB2_CHECK_ARG(p.n_rows >= 0, "negative row count");
  if (p.n_rows == 0)
    return CB2_OK;
  CB2_CHECK_ARG((p.red * es) % 16 == 0, "reduction width %d is not a multiple of 16 bytes", p.red);
  CB2_CHECK_ARG((p.nn * es) % 16 == 0, "output width %d is not a multiple of 16 bytes", p.nn);
  CB2_CHECK_ARG((p.lda * es) % 16 == 0 && (p.ldo * es) % 16 == 0, "row strides must be multiples of 16 bytes");
  CB2_CHECK_ARG(aligned16(p.a) && aligned16(p.out), "operand pointers must be 16-byte aligned");
  if (p.src_mode == kSrcRows)
    CB2_CHECK_ARG(aligned16(p.src) && (p.lds * es) % 16 == 0, "source rows must be 16-byte aligned");
  CUtensorMap map;
  rc = make_weight_map(&map, w_ptr, es, w_inner, w_mid, w_outer, w_mid_stride, w_outer_stride, atom,
                       b_mn ? kred : pl.block_n);
  if (rc)
    return rc;
  // Operand rows go through the copy engine (tile::gather4 requests of four rows and 128 bytes), but rows of
  // more than 128 bytes whose column blocks cross 128-byte lines by 16-byte cp.async.  (60 000 scanned rows,
  // forward to 128 channels, us, gather4 and cp.async: 72 channels 44.0 and 37.5, 88 53.6 and 46.1, 104 51.4 and 44.9, 112 36.9
  // and 35.3, 120 44.5 and 40.4, 128 31.6 and 34.8, 136 67.2 and 60.6, 160 54.1 and 55.5, 192 50.9 and 56.7, 200 70.7 and 65.0, 224 56.0
  // and 57.7, 248 71.3 and 66.9, 256 52.6 and 58.4, 320 72.9 and 82.3, 512 97.7 and 109.1; 150 000 uniform rows 104 20.5 and 22.7, 128
  // 20.3 and 22.0, 136 30.0 and 26.5, 192 24.9 and 25.4, 256 25.8 and 25.9; of one column block: 40 38.2 and 33.3, uniform 18.3 and
  // 22.0, 64 21.3 and 25.6, uniform 18.4 and 21.3; int8 128, stride 2, 40 and 44.)  Wide rows that overlap, or are all one (a stride below the width), are no
  // tensor that a map describes: cp.async takes them.  CUMM_B200_GATHER forces one path.
  const bool in_lines = (reinterpret_cast<uintptr_t>(p.a) | static_cast<uintptr_t>(p.lda * es)) % 128 == 0 && p.lda >= p.red;
  const bool tma_gather = (p.mask_words > 1 && pl.natom_k == 1) ||
                          (getenv("CUMM_B200_GATHER") ? gather_mode() != 0 : (pl.natom_k == 1 || in_lines));
  CUtensorMap map_a;
  memset(&map_a, 0, sizeof(map_a));
  if (tma_gather) {
    rc = make_rows_map(&map_a, p.a, es, p.red, p.a_rows, p.lda);
    if (rc)
      return rc;
  }
  p.b_lbo = static_cast<uint32_t>(kred * 128);
  p.b_sbo = 1024;
  p.status = dev->status;
  // Dynamic tile scheduling draws from a pair of device counters that the kernel itself
  // returns to zero: the caller's (one pair per argument record, so a captured launch never
  // shares with anybody), else one from the device's pool taken round-robin, so that eager
  // launches that overlap on different streams use different pairs unless more than
  // kTicketSlots are in flight.
  static std::atomic<unsigned> next_slot{0};
  CB2_CHECK_ARG((reinterpret_cast<uintptr_t>(sched_scratch) & 15u) == 0, "sched_scratch must be 16-byte aligned");
  CB2_CHECK_ARG(max_ctas >= 0, "max_ctas must not be negative");
  static const bool static_tiles = getenv("CUMM_B200_STATIC_TILES") != nullptr;
  p.tickets = static_tiles    ? nullptr
              : sched_scratch ? reinterpret_cast<int *>(sched_scratch)
                              : dev->status + 16 + 2 * (next_slot.fetch_add(1) % kTicketSlots);
  const int ntiles = (p.n_rows + 127) / 128;
  const int parts = (p.nn + pl.block_n - 1) / pl.block_n;
  const int gy = kind == 0 ? 1 : parts;  // RowConvCfg::PARTS
  p.n_parts = kind == 0 ? parts : 1;
  const long long items = static_cast<long long>(ntiles) * p.n_parts;
  CB2_CHECK_RT(items < (1ll << 30), "too many output tiles (%lld)", items);
  const int sms = (max_ctas > 0 && max_ctas < dev->num_sms) ? max_ctas : dev->num_sms;
  const int gx = static_cast<int>(std::min<long long>(std::max(sms / gy, 1), items));
  return launch_rowconv(pl, map, map_a, tma_gather, p, gx, gy, sms, stream);
}

// ---------------------------------------------------------------- weight gradient
struct WgradLayout {
  int block_n, gy, G, slots, list_stride, n_ctl;
  size_t off_ctl, off_partials, off_lists, total;
  // with row lists (see wgrad_mark_rows_kernel): their part comes after `total`
  int n_chunks;
  long long row_capacity;
  size_t off_head, off_counts, off_bits, off_rows, total_lists;
};

// Workspace of the weight gradient: 512-byte header (tile counts per offset), the control words,
// fp32 partials (one per unit: at most G + kv - 1), and per offset the list of the
// row tiles that carry it.  G = CTAs per (m, n) tile of the launch.
void wgrad_layout(int num_sms, int max_ctas, int m_total, int n_total, long long n_rows, int kv, int tile_n,
                  WgradLayout *L) {
  L->block_n = (tile_n == 64 || tile_n == 128) ? tile_n : (n_total <= 64 ? 64 : 128);
  const int mt = (m_total + 127) / 128, nt = (n_total + L->block_n - 1) / L->block_n;
  L->gy = mt * nt;
  const int sms = (max_ctas > 0 && max_ctas < num_sms) ? max_ctas : num_sms;
  L->G = sms / L->gy;
  if (L->G < 1)
    L->G = 1;
  L->slots = L->G + (kv > 32 ? kv : 32);
  const int kvs = kv > 0 ? kv : 1;
  L->n_ctl = kWgradCtlBase + 4 * kvs * L->gy;
  L->off_ctl = 512;
  L->off_partials = L->off_ctl + ((size_t)L->n_ctl * 4 + 255) / 256 * 256;
  L->off_lists = L->off_partials + (size_t)L->slots * L->gy * 128 * L->block_n * 4;
  const long long ntiles = (n_rows + 127) / 128;
  L->list_stride = (int)((ntiles + 63) / 64 * 64);
  L->total = L->off_lists + (size_t)kvs * L->list_stride * 4;
  // Room for 8 + kv / 8 listed rows per row (11 of 27 offsets, 23 of 125): scanned scenes have five and
  // thirteen neighbours per row, the centre, which every row has, is not listed.
  const int per = wgrad_chunk_tiles((int)ntiles);
  L->n_chunks = per > 0 ? (int)((ntiles + per - 1) / per) : 0;
  L->row_capacity = (n_rows * std::min(kvs, 8 + kvs / 8) + 127) / 128 * 128;
  if (ntiles <= kWgradRoomyTiles)
    L->row_capacity = ntiles * 128 * kvs;
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  L->off_head = up(L->total);
  L->off_counts = L->off_head + 2 * kWgradMaxOffsets * 4;
  L->off_bits = up(L->off_counts + (size_t)kvs * L->n_chunks * 8);
  L->off_rows = L->off_bits + (size_t)kvs * L->list_stride * 16;
  L->total_lists = L->off_rows + (size_t)L->row_capacity * 4;
}

template <int BLOCK_N, int A_ATOMS, int GATHER>
int launch_wgrad_inst(const CUtensorMap &ma, const CUtensorMap &mb, const WgradParams &p, int gx, int gy,
                      cudaStream_t stream) {
  using Cfg = WgradCfg<BLOCK_N, A_ATOMS, GATHER>;
  auto kern = wgrad_kernel<BLOCK_N, A_ATOMS, GATHER>;
  static std::atomic<uint64_t> configured{0};
  static std::atomic<int> regs{0};
  int dev = 0;
  CB2_CUDA(cudaGetDevice(&dev));
  if (!(configured.load() & (1ull << dev))) {
    CB2_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    regs.store(kernel_regs(kern));
    configured.fetch_or(1ull << dev);
  }
  g_last_launch.num_regs = regs.load();
  g_last_launch.num_threads = Cfg::THREADS;
  g_last_launch.smem_bytes = Cfg::SMEM_BYTES;
  g_last_launch.cluster = 1;
  CB2_CUDA(launch_after(1, kern, dim3(gx, gy), dim3(Cfg::THREADS), Cfg::SMEM_BYTES, stream, ma, mb, p));
  g_launches.fetch_add(1);
  return CB2_OK;
}

int run_wgrad(DeviceState *dev, WgradParams &p, int tile_n, int max_ctas, int plan_flags, void *workspace,
              size_t workspace_bytes, cudaStream_t stream) {
  const bool reuse_plan = (plan_flags & ~CB2_PLAN_ROW_LISTS) != 0;
  CB2_CHECK_RT(tile_n == 0 || tile_n == 64 || tile_n == 128,
               "can't find any suitable algo: tile_shape[1] = %d (kernels exist for 64 and 128)", tile_n);
  CB2_CHECK_ARG(max_ctas >= 0, "max_ctas must not be negative");
  WgradLayout L;
  wgrad_layout(dev->num_sms, max_ctas, p.m_total, p.n_total, p.n_rows, p.kv, tile_n, &L);
  CB2_CHECK_RT(workspace != nullptr && workspace_bytes >= L.total, "workspace at least %zu bytes.", L.total);
  CB2_CHECK_ARG(reinterpret_cast<uintptr_t>(workspace) % 256 == 0, "workspace must be 256-byte aligned");
  CB2_CHECK_RT(L.gy <= kWgradMaxOutTiles, "the weight gradient has %d output tiles of 128 x %d; at most %d are supported",
               L.gy, L.block_n, kWgradMaxOutTiles);
  CB2_CHECK_ARG(p.m_total % 8 == 0 && p.n_total % 8 == 0, "channel counts must be multiples of 8");
  CB2_CHECK_ARG((p.ld_dout * 2) % 16 == 0 && (p.ld_x * 2) % 16 == 0, "row strides must be multiples of 16 bytes");
  CB2_CHECK_ARG(aligned16(p.dout) && aligned16(p.x), "operand pointers must be 16-byte aligned");
  CB2_CHECK_ARG((reinterpret_cast<uintptr_t>(p.out) & 7u) == 0 && (reinterpret_cast<uintptr_t>(p.src) & 7u) == 0 &&
                    p.ldo % 4 == 0 && p.f_stride % 4 == 0,
                "the weight gradient and its row / offset strides must be 8-byte aligned");
  uint8_t *ws = reinterpret_cast<uint8_t *>(workspace);
  p.sched = reinterpret_cast<int *>(ws);
  p.ctl = reinterpret_cast<int *>(ws + L.off_ctl);
  p.partials = reinterpret_cast<float *>(ws + L.off_partials);
  p.lists = reinterpret_cast<const int *>(ws + L.off_lists);
  p.list_stride = L.list_stride;
  p.plan_fixed = reuse_plan ? 1 : 0;
  p.status = dev->status;
  // Row lists where the caller allows them and the workspace has room, tiles otherwise.  A plan that is
  // there already says for itself which of the two it is, whatever this call's flags and size are.
  const bool possible = p.mode == kWgradMaskConv && p.n_rows > 0 && L.row_capacity < (1ll << 31);
  const bool row_lists = possible && workspace_bytes >= L.total_lists && (plan_flags & CB2_PLAN_ROW_LISTS);
  if (possible && (reuse_plan || row_lists)) {
    p.row_head = reinterpret_cast<int *>(ws + L.off_head);
    p.rows = reinterpret_cast<const int *>(ws + L.off_rows);
  }
  if (!reuse_plan && row_lists && wgrad_one_block((p.n_rows + 127) / 128, p.kv)) {
    wgrad_plan_rows_kernel<<<p.kv, kWgradPlanThreads, 0, stream>>>(p, reinterpret_cast<int *>(ws + L.off_lists),
                                                                   reinterpret_cast<int *>(ws + L.off_rows), L.n_ctl);
    CB2_CUDA(cudaGetLastError());
    g_launches.fetch_add(1);
  } else if (!reuse_plan && row_lists) {
    const dim3 grid(L.n_chunks, p.kv);
    uint4 *bits = reinterpret_cast<uint4 *>(ws + L.off_bits);
    int2 *counts = reinterpret_cast<int2 *>(ws + L.off_counts);
    wgrad_mark_rows_kernel<<<grid, kWgradPlanThreads, 0, stream>>>(p, bits, counts, L.n_ctl);
    CB2_CUDA(cudaGetLastError());
    CB2_CUDA(launch_after(1, wgrad_list_rows_kernel, grid, dim3(kWgradPlanThreads), 0, stream, p, bits, counts,
                          reinterpret_cast<int *>(ws + L.off_lists), reinterpret_cast<int *>(ws + L.off_rows),
                          L.row_capacity));
    g_launches.fetch_add(2);
  } else if (!reuse_plan) {
    // counts and lists of the row tiles per offset; control words to zero
    wgrad_plan_kernel<<<p.kv, 1024, 0, stream>>>(p, reinterpret_cast<int *>(ws + L.off_lists), L.list_stride, L.n_ctl);
    CB2_CUDA(cudaGetLastError());
    g_launches.fetch_add(1);
  }
  CUtensorMap ma, mb;
  int rc = make_rows_map(&ma, p.dout, 2, p.m_total, p.a_rows, p.ld_dout);
  if (rc)
    return rc;
  rc = make_rows_map(&mb, p.x, 2, p.n_total, p.b_rows, p.ld_x);
  if (rc)
    return rc;
  const bool tma = gather_mode() != 0;
#define CB2_INST(N, A)                                                                              \
  if (tma && L.block_n == N && (p.m_total <= 64 ? 1 : 2) == A)                                      \
    return launch_wgrad_inst<N, A, kGatherTma4>(ma, mb, p, L.G, L.gy, stream);
  CB2_INST(64, 1)
  CB2_INST(64, 2)
  CB2_INST(128, 1)
  CB2_INST(128, 2)
#undef CB2_INST
  return L.block_n == 64 ? launch_wgrad_inst<64, 2, kGatherCpAsync>(ma, mb, p, L.G, L.gy, stream)
                         : launch_wgrad_inst<128, 2, kGatherCpAsync>(ma, mb, p, L.G, L.gy, stream);
}

// ---------------------------------------------------------------- allocation-free variant
// Scratch for cb2_conv_backward_weight_static: lives in the library image, one copy per GPU
// that loads it, for the life of the process.  In host code this name is only a handle for
// cudaGetSymbolAddress, never a pointer a kernel may be given.
constexpr size_t kStaticScratchBytes = 16u << 20;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
static __device__ int g_static_status[16];

struct StaticState {
  bool ready = false;
  DeviceState dev;  // num_sms, and `status` pointing at g_static_status on that device
  void *scratch = nullptr;
};
StaticState g_static[kMaxDevices];

// Per-device set-up of the allocation-free path, with that device current: resolves the
// device addresses of the two static arrays.  Nothing here allocates.
int get_device_static(StaticState **out) {
  int dev = 0;
  CB2_CUDA(cudaGetDevice(&dev));
  CB2_CHECK_RT(dev >= 0 && dev < kMaxDevices, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_mu);
  StaticState &st = g_static[dev];
  if (!st.ready) {
    cudaDeviceProp prop;
    CB2_CUDA(cudaGetDeviceProperties(&prop, dev));
    CB2_CHECK_RT(prop.major == 10, "cumm_b200 kernels are built for sm_100a only; device %d is sm_%d%d", dev,
                 prop.major, prop.minor);
    st.dev.num_sms = prop.multiProcessorCount;
    void *scratch = nullptr, *status = nullptr;
    CB2_CUDA(cudaGetSymbolAddress(&scratch, g_static_scratch));
    CB2_CUDA(cudaGetSymbolAddress(&status, g_static_status));
    CB2_CHECK_RT(scratch != nullptr && status != nullptr, "could not resolve the static scratch on device %d", dev);
    st.scratch = scratch;
    st.dev.status = reinterpret_cast<int *>(status);
    st.dev.ready = true;
    st.ready = true;
  }
  if (!g_encode) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    CB2_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
    CB2_CHECK_RT(fn != nullptr && q == cudaDriverEntryPointSuccess, "cuTensorMapEncodeTiled not available");
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  *out = &st;
  return CB2_OK;
}

int kind_of(int da, int db, int dc, int is_int8, bool allow_f32_out) {
  if (da == CB2_DTYPE_F16 && db == CB2_DTYPE_F16 &&
      (dc == CB2_DTYPE_F16 || (allow_f32_out && dc == CB2_DTYPE_F32)) && !is_int8)
    return 0;
  if (da == CB2_DTYPE_I8 && db == CB2_DTYPE_I8 && dc == CB2_DTYPE_I8 && is_int8)
    return 1;
  return -1;
}

} // namespace

extern "C" {

#ifdef CB2_TRACE
// Debug builds only: copy the device trace buffer to the host and reset it.
int cb2_debug_read_trace(void *host_dst, size_t bytes) {
  if (bytes != sizeof(cb2::TraceBuf))
    return set_err(CB2_ERR_INVALID_ARG, "trace buffer is %zu bytes", sizeof(cb2::TraceBuf));
  CB2_CUDA(cudaDeviceSynchronize());
  CB2_CUDA(cudaMemcpyFromSymbol(host_dst, cb2::g_trace, bytes));
  static cb2::TraceBuf zero;
  CB2_CUDA(cudaMemcpyToSymbol(cb2::g_trace, &zero, bytes));
  return CB2_OK;
}
#endif

} // extern "C" (reopened below, after the helpers of the table builder)

// ---------------------------------------------------------------- neighbour tables on the GPU
namespace {

struct PairgenLayout {
  cb2pg::Geometry g;
  cb2pg::SortShape shape;
  uint32_t cap_in, cap_set;  // hash capacities (powers of two); 0 = not used
  bool exact;                // a voxel's linear index fits the hash table's 32-bit tag
  bool mirror;               // the backward table is the forward one with the offsets reversed
  bool bitmap;               // active outputs of a strided conv through a bitmap of the output grid
  long long bitmap_words;    // whole blocks
  long long list_cap;        // active outputs a strided conv can have at most
  long long nmax;            // rows the mask sorts may have to hold
  int key_bits;
  size_t hist_ints;          // of one side
  size_t off_counters, off_hash, off_bits, off_word_first, off_block_first, off_set_keys, off_list_a, off_list_b,
      off_key_hist, off_hist, total;
  size_t off_rows[2], off_m[2], off_v[2];  // per side: unsorted masks (several words), mask and row scratch
};

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

uint32_t pow2_at_least(unsigned long long v) {
  uint32_t c = 64;
  while (c < v && c < (1u << 31))
    c <<= 1;
  return c;
}

int pairgen_layout(const cb2_pairgen_args *a, PairgenLayout *L) {
  CB2_CHECK_ARG(a != nullptr, "null arguments");
  CB2_CHECK_ARG(a->n_in >= 0 && a->batch_size >= 1, "bad n_in / batch_size (%d, %d)", a->n_in, a->batch_size);
  long long kv = 1, cells = a->batch_size;
  for (int i = 0; i < 3; ++i) {
    CB2_CHECK_ARG(a->grid[i] >= 1 && a->ksize[i] >= 1 && a->stride[i] >= 1 && a->dil[i] >= 1 && a->pad[i] >= 0,
                  "bad geometry on axis %d", i);
    L->g.grid[i] = a->grid[i];
    L->g.ksize[i] = a->ksize[i];
    L->g.stride[i] = a->stride[i];
    L->g.pad[i] = a->pad[i];
    L->g.dil[i] = a->dil[i];
    const int span = a->grid[i] + 2 * a->pad[i] - a->dil[i] * (a->ksize[i] - 1) - 1;
    L->g.ogrid[i] = a->subm ? a->grid[i] : (span >= 0 ? span / a->stride[i] + 1 : 0);
    CB2_CHECK_ARG(L->g.ogrid[i] >= 1, "the kernel does not fit the grid on axis %d", i);
    kv *= a->ksize[i];
    cells *= L->g.ogrid[i];
  }
  CB2_CHECK_RT(kv <= 128, "kernel volume %lld is not supported (masks hold up to 128 offsets)", kv);
  if (a->subm)
    for (int i = 0; i < 3; ++i)
      CB2_CHECK_ARG(a->stride[i] == 1, "a submanifold convolution has stride 1");
  L->g.kv = static_cast<int>(kv);
  L->shape = cb2pg::sort_shape(L->g.kv);
  L->g.batch_size = a->batch_size;
  const long long n_in = a->n_in;
  unsigned __int128 in_cells = a->batch_size;
  L->mirror = a->subm;
  for (int i = 0; i < 3; ++i) {
    in_cells *= static_cast<unsigned>(a->grid[i]);
    L->mirror = L->mirror && a->ksize[i] % 2 == 1 && 2ll * a->pad[i] == static_cast<long long>(a->ksize[i] - 1) * a->dil[i];
  }
  L->exact = in_cells < 0xffffffffull;
  // outputs an input can feed: per axis, the offsets r with (in + pad - r * dil) divisible by the stride
  long long per_input = 1;
  for (int i = 0; i < 3; ++i) {
    int gcd = a->stride[i], b = a->dil[i];
    while (b) {
      const int t = gcd % b;
      gcd = b;
      b = t;
    }
    const int period = a->stride[i] / gcd;  // r takes every period-th value
    L->g.period[i] = period;
    L->g.drop[i] = a->dil[i] / gcd;
    per_input *= std::min(a->ksize[i], (a->ksize[i] + period - 1) / period);
  }
  L->list_cap = a->subm ? 0 : std::min<long long>(n_in * per_input, cells);
  CB2_CHECK_RT(L->list_cap < (1ll << 30), "too many candidate outputs (%lld)", L->list_cap);
  // The bitmap is cleared, counted and read once each whatever the scene, so it has to be small
  // beside the scene or small altogether: up to 64 bytes per input voxel, or 4 MiB.
  L->bitmap = !a->subm && cells < (1ll << 31) - 64 && cells / 8 <= std::max<long long>(4 << 20, 64 * n_in);
  const long long block_words = cb2pg::kBitmapBlockWords;
  L->bitmap_words = L->bitmap ? ((cells + 31) / 32 + block_words - 1) / block_words * block_words : 0;
  L->cap_in = L->bitmap ? 0 : pow2_at_least(2ull * static_cast<unsigned long long>(n_in));
  L->cap_set = (a->subm || L->bitmap) ? 0 : pow2_at_least(2ull * static_cast<unsigned long long>(L->list_cap));
  const long long keys_cap = L->cap_set ? L->list_cap : 0;
  L->nmax = std::max<long long>(a->subm ? n_in : L->list_cap, n_in);
  L->key_bits = 1;
  while (L->key_bits < 63 && (1ll << L->key_bits) < cells)
    ++L->key_bits;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align256(off + bytes);
    return at;
  };
  L->off_counters = take(256);
  L->off_hash = take(static_cast<size_t>(L->cap_in) * 8);
  L->off_bits = take(static_cast<size_t>(L->bitmap_words) * 4);
  L->off_word_first = take(static_cast<size_t>(L->bitmap_words) * 4);
  L->off_block_first = take(static_cast<size_t>(L->bitmap_words / block_words) * 4);
  L->off_set_keys = take(static_cast<size_t>(L->cap_set) * 8);
  L->off_list_a = take(static_cast<size_t>(keys_cap) * 8);
  L->off_list_b = take(static_cast<size_t>(keys_cap) * 8);
  L->off_key_hist = take(keys_cap ? static_cast<size_t>(256) * ((keys_cap + cb2pg::kKeySortTile - 1) / cb2pg::kKeySortTile + 1) * 4 : 0);
  L->hist_ints = cb2pg::kSortHistInts * L->shape.passes;
  L->off_hist = take(2 * L->hist_ints * 4);
  for (int side = 0; side < 2; ++side) {
    const size_t n = static_cast<size_t>(side == 0 ? L->nmax : n_in);
    L->off_rows[side] = take(L->shape.words > 1 ? n * L->shape.words * 4 : 0);
    L->off_m[side] = take(L->shape.words > 1 ? 0 : n * 4);
    L->off_v[side] = take(n * 4);
  }
  L->total = off;
  return CB2_OK;
}

// Ascending sort of n output keys on `bits` low bits, 8 per pass, ping-ponging between the result
// buffer and the scratch buffer.  The unsorted input has to be where key_sort_source() says -- the
// scratch buffer for an odd number of passes, the result buffer for an even number.
inline int key_sort_passes(int bits) { return bits <= 8 ? 1 : (bits + 7) / 8; }
unsigned long long *key_sort_source(unsigned long long *result, unsigned long long *scratch, int bits) {
  return key_sort_passes(bits) % 2 ? scratch : result;
}
int key_sort(unsigned long long *result, unsigned long long *scratch, int n, int bits, int *hist, cudaStream_t s) {
  if (n <= 0)
    return CB2_OK;
  const int ntiles = (n + cb2pg::kKeySortTile - 1) / cb2pg::kKeySortTile;
  unsigned long long *ks = key_sort_source(result, scratch, bits), *kd = (ks == result) ? scratch : result;
  for (int p = 0; p < key_sort_passes(bits); ++p) {
    cb2pg::key_hist_kernel<<<ntiles, cb2pg::kKeySortThreads, 0, s>>>(ks, n, 8 * p, hist, ntiles);
    cb2pg::key_scan_kernel<<<1, 1024, 0, s>>>(reinterpret_cast<int4 *>(hist), (256 * ntiles + 3) / 4);
    cb2pg::key_scatter_kernel<<<ntiles, cb2pg::kKeySortThreads, 0, s>>>(ks, kd, n, 8 * p, hist, ntiles);
    CB2_CUDA(cudaGetLastError());
    g_launches.fetch_add(3);
    std::swap(ks, kd);
  }
  return CB2_OK;
}

// One side's masks on their way to being sorted: where the unsorted masks are built, and what the
// sort needs and leaves.
struct MaskSort {
  cb2pg::MaskSide side;
  uint32_t *m_tmp;
  int *v_tmp;
  uint32_t *mask;  // results
  int *argsort;
  uint32_t *tile_masks;
};
// `rows`: room for unsorted masks of several words; one-word masks are sorted between `mask` and `m_tmp`
// and start in whichever lets the last pass end in `mask`.
MaskSort make_mask_sort(const cb2pg::SortShape &shape, int32_t *indices, int n, uint32_t *rows, uint32_t *m_tmp,
                        int *v_tmp, int *hist, uint32_t *mask, int *argsort, uint32_t *tile_masks) {
  MaskSort j;
  j.side.indices = indices;
  j.side.rows = shape.words > 1 ? rows : (shape.passes % 2 ? m_tmp : mask);
  j.side.hist = hist;
  j.side.n = n;
  j.side.chunk = cb2pg::sort_chunk(n);
  j.m_tmp = m_tmp;
  j.v_tmp = v_tmp;
  j.mask = mask;
  j.argsort = argsort;
  j.tile_masks = tile_masks;
  return j;
}

// All passes, both sides of a table set in the same launches.  Counts of the first pass and the
// unsorted masks are there, the other counts and the tile masks are zero.
int sort_masks(const MaskSort *jobs, int count, const cb2pg::SortShape &shape, cudaStream_t s) {
  int max_chunks = 1;
  for (int p = 0; p < shape.passes; ++p) {
    cb2pg::SortSides sides;
    memset(&sides, 0, sizeof(sides));
    const int to_go = shape.passes - 1 - p;
    bool few = true;
    for (int q = 0; q < count; ++q) {
      const MaskSort &j = jobs[q];
      few = few && j.side.chunk <= cb2pg::kSortThreads * cb2pg::kSortItemsSmall;
      cb2pg::SortSide &o = sides.side[q];
      o.n = j.side.n;
      o.chunk = j.side.chunk;
      o.n_chunks = (j.side.n + j.side.chunk - 1) / j.side.chunk;
      max_chunks = std::max(max_chunks, o.n_chunks);
      o.hist = j.side.hist + p * cb2pg::kSortHistInts;
      o.hist_next = to_go ? j.side.hist + (p + 1) * cb2pg::kSortHistInts : nullptr;
      o.rows = j.side.rows;
      // results of the last pass in the result arrays, of the one before it in scratch, and so on
      o.vout = to_go % 2 ? j.v_tmp : j.argsort;
      o.vin = p == 0 ? nullptr : (to_go % 2 ? j.argsort : j.v_tmp);
      o.kout = shape.words > 1 ? j.mask : (to_go % 2 ? j.m_tmp : j.mask);
      o.kin = shape.words > 1 ? nullptr : (to_go % 2 ? j.mask : j.m_tmp);
      o.tile_masks = to_go ? nullptr : j.tile_masks;
    }
    const dim3 grid(max_chunks, count);
    auto kern = few ? (shape.words > 1 ? cb2pg::sort_pass_kernel<true, true> : cb2pg::sort_pass_kernel<false, true>)
                    : (shape.words > 1 ? cb2pg::sort_pass_kernel<true, false> : cb2pg::sort_pass_kernel<false, false>);
    CB2_CUDA(launch_after(1, kern, grid, dim3(cb2pg::kSortThreads), 0, s, sides, p, shape));
    g_launches.fetch_add(1);
  }
  return CB2_OK;
}

struct Fill {
  cb2pg::FillRanges r;
  long long most = 0;
  Fill() { r.count = 0; }
  void add(void *ptr, size_t bytes, uint32_t value) {
    if (!ptr || !bytes)
      return;
    r.ptr[r.count] = reinterpret_cast<uint32_t *>(ptr);
    r.words[r.count] = static_cast<long long>(bytes / 4);
    r.value[r.count++] = value;
    most = std::max<long long>(most, static_cast<long long>(bytes / 4));
  }
  void run(const DeviceState *dev, cudaStream_t s) const {
    const long long blocks = std::min<long long>((most / 4 + 1023) / 1024 + 1, 8ll * dev->num_sms);
    cb2pg::fill_kernel<<<dim3(static_cast<unsigned>(blocks), r.count), 256, 0, s>>>(r);
    g_launches.fetch_add(1);
  }
};

cb2pg::Bitmap pairgen_bitmap(const PairgenLayout &L, uint8_t *ws) {
  cb2pg::Bitmap bm;
  bm.words = reinterpret_cast<uint32_t *>(ws + L.off_bits);
  bm.word_first = reinterpret_cast<int *>(ws + L.off_word_first);
  bm.block_first = reinterpret_cast<int *>(ws + L.off_block_first);
  bm.n_words = static_cast<int>(L.bitmap_words);
  bm.n_blocks = static_cast<int>(L.bitmap_words / cb2pg::kBitmapBlockWords);
  return bm;
}

int pairgen_common(const cb2_pairgen_args *a, PairgenLayout *L, DeviceState **dev) {
  int rc = get_device(dev);
  if (rc)
    return rc;
  rc = pairgen_layout(a, L);
  if (rc)
    return rc;
  CB2_CHECK_RT(a->in_coords != nullptr || a->n_in == 0, "in_coords must not empty");
  CB2_CHECK_ARG(aligned16(a->in_coords), "in_coords must be 16-byte aligned");
  CB2_CHECK_RT(a->workspace != nullptr && a->workspace_bytes >= L->total, "workspace at least %zu bytes.", L->total);
  CB2_CHECK_ARG(reinterpret_cast<uintptr_t>(a->workspace) % 256 == 0, "workspace must be 256-byte aligned");
  return CB2_OK;
}

} // namespace

extern "C" {

size_t cb2_pairgen_workspace_size(const cb2_pairgen_args *a) {
  PairgenLayout L;
  if (pairgen_layout(a, &L))
    return 0;
  return L.total;
}

int cb2_pairgen_count_outputs(const cb2_pairgen_args *a, int *n_out, void *stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  PairgenLayout L;
  DeviceState *dev;
  int rc = pairgen_common(a, &L, &dev);
  if (rc)
    return rc;
  CB2_CHECK_ARG(n_out != nullptr, "n_out must not be null");
  if (a->subm || a->n_in == 0) {
    *n_out = a->n_in;
    return CB2_OK;
  }
  uint8_t *ws = reinterpret_cast<uint8_t *>(a->workspace);
  int *counter = reinterpret_cast<int *>(ws + L.off_counters);
  Fill fill;
  fill.add(counter, 256, 0u);
  unsigned long long *set_keys = reinterpret_cast<unsigned long long *>(ws + L.off_set_keys);
  unsigned long long *list_a = reinterpret_cast<unsigned long long *>(ws + L.off_list_a);
  unsigned long long *list_b = reinterpret_cast<unsigned long long *>(ws + L.off_list_b);
  if (L.bitmap) {
    const cb2pg::Bitmap bm = pairgen_bitmap(L, ws);
    fill.add(bm.words, static_cast<size_t>(L.bitmap_words) * 4, 0u);
    fill.run(dev, stream);
    CB2_CUDA(launch_after(1, cb2pg::bitmap_mark_kernel, dim3((a->n_in + 127) / 128), dim3(128), 0, stream, a->in_coords,
                          a->n_in, L.g, bm.words));
    CB2_CUDA(launch_after(1, cb2pg::bitmap_rank_kernel, dim3(bm.n_blocks), dim3(cb2pg::kBitmapThreads), 0, stream, bm,
                          counter));
    g_launches.fetch_add(2);
  } else {
    fill.add(set_keys, static_cast<size_t>(L.cap_set) * 8, 0xffffffffu);
    fill.run(dev, stream);
    cb2pg::out_candidates_kernel<<<(a->n_in + 255) / 256, 256, 0, stream>>>(
        a->in_coords, a->n_in, L.g, set_keys, L.cap_set - 1, key_sort_source(list_a, list_b, L.key_bits),
        static_cast<int>(L.list_cap), counter, dev->status);
    g_launches.fetch_add(1);
  }
  CB2_CUDA(cudaGetLastError());
  int count = 0;
  CB2_CUDA(cudaMemcpyAsync(&count, counter, sizeof(int), cudaMemcpyDeviceToHost, stream));
  CB2_CUDA(cudaStreamSynchronize(stream));
  CB2_CHECK_RT(count >= 0 && count <= L.list_cap, "active-output count %d out of range", count);
  if (!L.bitmap) {
    rc = key_sort(list_a, list_b, count, L.key_bits, reinterpret_cast<int *>(ws + L.off_key_hist), stream);
    if (rc)
      return rc;
  }
  *n_out = count;
  return CB2_OK;
}

int cb2_pairgen_run(const cb2_pairgen_args *a, void *stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  PairgenLayout L;
  DeviceState *dev;
  int rc = pairgen_common(a, &L, &dev);
  if (rc)
    return rc;
  const int n_in = a->n_in;
  const int n_out = a->subm ? n_in : a->n_out;
  CB2_CHECK_ARG(n_out >= 0 && n_out <= L.nmax, "n_out %d out of range", n_out);
  if (n_out == 0)
    return CB2_OK;
  CB2_CHECK_RT(a->indices && a->mask && a->mask_argsort, "error: indices, mask or mask_argsort empty");
  CB2_CHECK_RT(a->subm || a->out_coords, "out_coords must not empty");
  CB2_CHECK_ARG(a->subm || aligned16(a->out_coords), "out_coords must be 16-byte aligned");
  const bool bwd = a->indices_bwd != nullptr;
  CB2_CHECK_RT(!bwd || (a->mask_bwd && a->mask_argsort_bwd), "error: backward mask or mask_argsort empty");
  uint8_t *ws = reinterpret_cast<uint8_t *>(a->workspace);
  const cb2pg::SortShape &shape = L.shape;
  const int words = shape.words;
  auto at32 = [&](size_t off) { return reinterpret_cast<uint32_t *>(ws + off); };
  auto at_int = [&](size_t off) { return reinterpret_cast<int *>(ws + off); };
  MaskSort jobs[2];
  jobs[0] = make_mask_sort(shape, a->indices, n_out, at32(L.off_rows[0]), at32(L.off_m[0]), at_int(L.off_v[0]),
                           at_int(L.off_hist), a->mask, a->mask_argsort, a->tile_masks);
  jobs[1] = make_mask_sort(shape, a->indices_bwd, n_in, at32(L.off_rows[1]), at32(L.off_m[1]), at_int(L.off_v[1]),
                           at_int(L.off_hist) + L.hist_ints, a->mask_bwd, a->mask_argsort_bwd, nullptr);
  const cb2pg::MaskSide none = {nullptr, nullptr, nullptr, 0, 1};
  const auto blocks = [](long long n) { return static_cast<unsigned>((n + 255) / 256); };
  Fill fill;
  fill.add(at_int(L.off_hist), 2 * L.hist_ints * 4, 0u);
  fill.add(a->tile_masks, static_cast<size_t>((n_out + 127) / 128) * words * 4, 0u);
  if (L.bitmap) {
    const cb2pg::Bitmap bm = pairgen_bitmap(L, ws);
    fill.add(a->indices, static_cast<size_t>(L.g.kv) * n_out * 4, 0xffffffffu);
    fill.add(jobs[0].side.rows, static_cast<size_t>(n_out) * words * 4, 0u);
    if (bwd)
      fill.add(a->indices_bwd, static_cast<size_t>(L.g.kv) * n_in * 4, 0xffffffffu);
    fill.run(dev, stream);
    CB2_CUDA(launch_after(1, cb2pg::bitmap_coords_kernel, dim3(blocks(bm.n_words)), dim3(256), 0, stream, bm, n_out, L.g,
                          a->out_coords));
    CB2_CUDA(launch_after(1, cb2pg::bitmap_scatter_kernel, dim3((n_in + 127) / 128), dim3(128), 0, stream, a->in_coords,
                          n_in, L.g, bm, jobs[0].side, words, dev->status));
    const int bwd_blocks = bwd ? static_cast<int>(blocks(n_in)) : 0;
    auto kern = words > 1 ? cb2pg::bitmap_backward_kernel<4> : cb2pg::bitmap_backward_kernel<1>;
    CB2_CUDA(launch_after(1, kern, dim3(bwd_blocks + blocks(n_out)), dim3(cb2pg::kProbeThreads), 0, stream, a->in_coords,
                          L.g, bm, jobs[0].side, jobs[1].side, bwd_blocks, words, shape.width));
    CB2_CUDA(cudaGetLastError());
    g_launches.fetch_add(3);
  } else {
    cb2pg::HashView h;
    h.slots = reinterpret_cast<unsigned long long *>(ws + L.off_hash);
    h.bucket_mask = L.cap_in / cb2pg::kBucket - 1;
    h.coords = a->in_coords;
    const bool mirror = bwd && L.mirror;
    fill.add(h.slots, static_cast<size_t>(L.cap_in) * 8, 0xffffffffu);
    if (bwd && !mirror)
      fill.add(a->indices_bwd, static_cast<size_t>(L.g.kv) * n_in * 4, 0xffffffffu);
    fill.run(dev, stream);
    auto insert = L.exact ? cb2pg::hash_insert_kernel<true> : cb2pg::hash_insert_kernel<false>;
    CB2_CUDA(launch_after(1, insert, dim3(blocks(n_in)), dim3(256), 0, stream, a->in_coords, n_in, L.g, h, dev->status));
    const int32_t *out_coords = a->in_coords;
    if (!a->subm) {
      cb2pg::decode_out_coords_kernel<<<blocks(n_out), 256, 0, stream>>>(
          reinterpret_cast<const unsigned long long *>(ws + L.off_list_a), n_out, L.g, a->out_coords);
      out_coords = a->out_coords;
      g_launches.fetch_add(1);
    }
    auto kern = L.exact ? (words > 1 ? cb2pg::probe_kernel<4, true> : cb2pg::probe_kernel<1, true>)
                        : (words > 1 ? cb2pg::probe_kernel<4, false> : cb2pg::probe_kernel<1, false>);
    CB2_CUDA(launch_after(1, kern, dim3(blocks(n_out)), dim3(cb2pg::kProbeThreads), 0, stream, out_coords, L.g, h,
                          jobs[0].side, mirror ? jobs[1].side : none, words, shape.width));
    g_launches.fetch_add(2);
    if (bwd && !mirror) {
      cb2pg::invert_table_kernel<<<blocks(static_cast<long long>(n_out) * L.g.kv), 256, 0, stream>>>(
          a->indices, n_out, L.g.kv, n_in, a->indices_bwd);
      cb2pg::masks_from_table_kernel<<<blocks(n_in), cb2pg::kProbeThreads, 0, stream>>>(jobs[1].side, L.g.kv, words,
                                                                                       shape.width);
      g_launches.fetch_add(2);
    }
    CB2_CUDA(cudaGetLastError());
  }
  return sort_masks(jobs, bwd ? 2 : 1, shape, stream);
}

// ---------------------------------------------------------------- a layer's ShuffleAC calls in one launch
struct SeqLayout {
  size_t off_table, off_mask, off_argsort, off_m, off_v, off_hist, off_tickets, total;
};
static void seq_layout(int count, long long n, SeqLayout *L) {
  const cb2pg::SortShape shape = cb2pg::sort_shape(count);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align256(off + bytes);
    return at;
  };
  L->off_tickets = take(256);
  L->off_table = take(static_cast<size_t>(count) * n * 4);
  L->off_mask = take(static_cast<size_t>(n) * 4);
  L->off_argsort = take(static_cast<size_t>(n) * 4);
  L->off_m = take(static_cast<size_t>(n) * 4);
  L->off_v = take(static_cast<size_t>(n) * 4);
  L->off_hist = take(cb2pg::kSortHistInts * shape.passes * 4);
  L->total = off;
}

size_t cb2_gemm_sequence_workspace_size(const cb2_gemm_sequence_args *a) {
  if (!a || a->count < 1 || a->count > cb2pg::kSeqMaxCalls || a->n_out_rows < 0)
    return 0;
  SeqLayout L;
  seq_layout(a->count, a->n_out_rows, &L);
  return L.total;
}

int cb2_gemm_sequence_run(const cb2_gemm_sequence_args *a, void *stream_v) {
  CB2_CHECK_ARG(a != nullptr && a->calls != nullptr, "null arguments");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  DeviceState *dev;
  int rc = get_device(&dev);
  if (rc)
    return rc;
  CB2_CHECK_ARG(a->count >= 1 && a->count <= cb2pg::kSeqMaxCalls, "a sequence holds 1 to %d calls", cb2pg::kSeqMaxCalls);
  CB2_CHECK_ARG(a->n_out_rows >= 0, "negative row count");
  const cb2_gemm_args &c0 = a->calls[0];
  CB2_CHECK_RT(c0.ptr_A && c0.ptr_B && c0.ptr_C, "a,b,c must not empty");
  CB2_CHECK_RT(kind_of(c0.dtype_a, c0.dtype_b, c0.dtype_c, 0, false) == 0,
               "can't find any suitable algo for dtypes (%d,%d,%d): only f16,f16,f16 is built", c0.dtype_a, c0.dtype_b,
               c0.dtype_c);
  CB2_CHECK_ARG(c0.k % 8 == 0 && c0.n % 8 == 0, "this m, n, k isn't supported due to misaligned contiguous dim.");
  // what makes the calls one layer
  const long long b_step = a->count > 1 ? (reinterpret_cast<const char *>(a->calls[1].ptr_B) -
                                           reinterpret_cast<const char *>(c0.ptr_B))
                                        : 0;
  cb2pg::SeqPairLists lists;
  memset(&lists, 0, sizeof(lists));
  lists.count = a->count;
  for (int f = 0; f < a->count; ++f) {
    const cb2_gemm_args &c = a->calls[f];
    const bool same = c.shuffle_type == CB2_SHUFFLE_AC && !c.trans_a && !c.trans_c && c.trans_b == c0.trans_b &&
                      c.ptr_A == c0.ptr_A && c.stride_A == c0.stride_A && c.rows_A == c0.rows_A && c.ptr_C == c0.ptr_C &&
                      c.stride_C == c0.stride_C && (c.ptr_D == nullptr || c.ptr_D == c.ptr_C) && !c.d_is_vector &&
                      c.n == c0.n && c.k == c0.k && c.stride_B == c0.stride_B && c.alpha == 1.f && c.beta == 1.f &&
                      c.act_type == CB2_ACT_NONE && c.dtype_a == c0.dtype_a && c.dtype_b == c0.dtype_b &&
                      c.dtype_c == c0.dtype_c && c.m >= 0 && c.indiceBorC != nullptr &&
                      reinterpret_cast<const char *>(c.ptr_B) - reinterpret_cast<const char *>(c0.ptr_B) == f * b_step;
    if (!same)
      return set_err(CB2_ERR_UNSUPPORTED,
                     "call %d of the sequence does not fit the layer form (ShuffleAC, shared A and C, alpha = beta = 1, "
                     "no activation, equally spaced B): run the calls one by one",
                     f);
    lists.a_inds[f] = c.indiceA;
    lists.c_inds[f] = c.indiceBorC;
    lists.first[f + 1] = lists.first[f] + c.m;
  }
  CB2_CHECK_RT(b_step % 2 == 0 && b_step >= 0, "B matrices must be ascending slices of one tensor");
  const int n = a->n_out_rows;
  if (n == 0)
    return CB2_OK;
  SeqLayout L;
  seq_layout(a->count, n, &L);
  CB2_CHECK_RT(a->workspace != nullptr && a->workspace_bytes >= L.total, "workspace at least %zu bytes.", L.total);
  CB2_CHECK_ARG(reinterpret_cast<uintptr_t>(a->workspace) % 256 == 0, "workspace must be 256-byte aligned");
  uint8_t *ws = reinterpret_cast<uint8_t *>(a->workspace);
  int32_t *table = reinterpret_cast<int32_t *>(ws + L.off_table);
  uint32_t *mask = reinterpret_cast<uint32_t *>(ws + L.off_mask);
  int32_t *argsort = reinterpret_cast<int32_t *>(ws + L.off_argsort);
  if (!a->reuse_tables) {
    const cb2pg::SortShape shape = cb2pg::sort_shape(a->count);
    const MaskSort job = make_mask_sort(shape, table, n, nullptr, reinterpret_cast<uint32_t *>(ws + L.off_m),
                                        reinterpret_cast<int *>(ws + L.off_v), reinterpret_cast<int *>(ws + L.off_hist), mask,
                                        argsort, nullptr);
    Fill fill;
    fill.add(ws + L.off_tickets, 256, 0u);
    fill.add(table, static_cast<size_t>(a->count) * n * 4, 0xffffffffu);
    fill.add(ws + L.off_hist, cb2pg::kSortHistInts * shape.passes * 4, 0u);
    fill.run(dev, stream);
    const long long pairs = lists.first[a->count];
    if (pairs > 0) {
      cb2pg::seq_scatter_kernel<<<static_cast<unsigned>((pairs + 255) / 256), 256, 0, stream>>>(lists, n, c0.rows_A, table,
                                                                                              dev->status);
      g_launches.fetch_add(1);
    }
    cb2pg::masks_from_table_kernel<<<(n + cb2pg::kProbeThreads - 1) / cb2pg::kProbeThreads, cb2pg::kProbeThreads, 0, stream>>>(
        job.side, a->count, 1, shape.width);
    CB2_CUDA(cudaGetLastError());
    g_launches.fetch_add(1);
    rc = sort_masks(&job, 1, shape, stream);
    if (rc)
      return rc;
  }
  RowConvParams p;
  memset(&p, 0, sizeof(p));
  p.a = c0.ptr_A;
  p.out = c0.ptr_C;
  p.indices = table;
  p.mask = mask;
  p.argsort = argsort;
  p.n_rows = n;
  p.a_rows = c0.rows_A;
  p.red = c0.k;
  p.nn = c0.n;
  p.lda = c0.stride_A;
  p.ldo = c0.stride_C;
  p.kv = a->count;
  p.mask_words = 1;
  p.mode = kModeMaskConv;
  p.mask_filter = 0xffffffffu;
  p.alpha = 1.f;
  p.beta = 1.f;
  p.src = c0.ptr_C;
  p.src_mode = kSrcRows;
  p.lds = c0.stride_C;
  // the weight tensor as [outer, f, inner]: B_f is [n, k] (trans_b) or [k, n]
  const bool b_mn = !c0.trans_b;
  const uint64_t inner = b_mn ? c0.n : c0.k, outer = b_mn ? c0.k : c0.n;
  const uint64_t f_stride = a->count > 1 ? static_cast<uint64_t>(b_step / 2) : inner;
  return run_rowconv(dev, p, 0, b_mn, c0.tile_n, c0.tile_k, ws + L.off_tickets, c0.max_ctas, c0.ptr_B, inner, a->count, outer,
                     f_stride, c0.stride_B, stream);
}

// ---------------------------------------------------------------- tables of a dense convolution
int cb2_exchange_capture_mode(int *mode) {
  CB2_CHECK_ARG(mode != nullptr, "null arguments");
  cudaStreamCaptureMode m = static_cast<cudaStreamCaptureMode>(*mode);
  CB2_CUDA(cudaThreadExchangeStreamCaptureMode(&m));
  *mode = m;
  return CB2_OK;
}

int cb2_dense_tables_run(const cb2_dense_tables_args *a, void *stream_v) {
  CB2_CHECK_ARG(a != nullptr, "null arguments");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  DeviceState *dev;
  int rc = get_device(&dev);
  if (rc)
    return rc;
  cb2pg::DenseGeometry g;
  g.batch = a->batch;
  long long n_in = a->batch, n_out = a->batch, kv = 1;
  CB2_CHECK_ARG(a->batch >= 1, "bad batch %d", a->batch);
  for (int i = 0; i < 3; ++i) {
    CB2_CHECK_ARG(a->in_dims[i] >= 1 && a->out_dims[i] >= 1 && a->ksize[i] >= 1 && a->stride[i] >= 1 &&
                      a->dil[i] >= 1 && a->pad[i] >= 0,
                  "bad geometry on axis %d", i);
    const int span = a->in_dims[i] + 2 * a->pad[i] - a->dil[i] * (a->ksize[i] - 1) - 1;
    CB2_CHECK_ARG(span >= 0 && a->out_dims[i] == span / a->stride[i] + 1,
                  "output extent %d on axis %d does not match input %d, kernel %d, stride %d, padding %d, dilation %d",
                  a->out_dims[i], i, a->in_dims[i], a->ksize[i], a->stride[i], a->pad[i], a->dil[i]);
    g.in_dims[i] = a->in_dims[i];
    g.out_dims[i] = a->out_dims[i];
    g.ksize[i] = a->ksize[i];
    g.stride[i] = a->stride[i];
    g.pad[i] = a->pad[i];
    g.dil[i] = a->dil[i];
    n_in *= a->in_dims[i];
    n_out *= a->out_dims[i];
    kv *= a->ksize[i];
  }
  CB2_CHECK_RT(kv <= 128, "kernel volume %lld: the kernels handle up to 128 filter offsets", kv);
  CB2_CHECK_RT(n_in < (1ll << 31) && n_out < (1ll << 31), "too many rows for 32-bit row indices");
  CB2_CHECK_RT(a->indices_fwd != nullptr, "error: indices empty");
  g.kv = (int)kv;
  const int words = ((int)kv + 31) / 32;
  auto blocks = [](long long n) { return (unsigned)((n + 255) / 256); };
  cb2pg::dense_table_fwd_kernel<<<blocks(n_out * kv), 256, 0, stream>>>(g, n_out, a->indices_fwd);
  g_launches.fetch_add(1);
  if (a->indices_bwd) {
    cb2pg::dense_table_bwd_kernel<<<blocks(n_in * kv), 256, 0, stream>>>(g, n_in, a->indices_bwd);
    g_launches.fetch_add(1);
  }
  if (a->mask_fwd && a->argsort_fwd) {
    cb2pg::dense_masks_kernel<<<blocks(n_out), 256, 0, stream>>>(n_out, (int)kv, words, a->mask_fwd, a->argsort_fwd);
    g_launches.fetch_add(1);
  }
  if (a->mask_bwd && a->argsort_bwd) {
    cb2pg::dense_masks_kernel<<<blocks(n_in), 256, 0, stream>>>(n_in, (int)kv, words, a->mask_bwd, a->argsort_bwd);
    g_launches.fetch_add(1);
  }
  CB2_CUDA(cudaGetLastError());
  return CB2_OK;
}

// ---------------------------------------------------------------- sum over GPUs through peer memory
struct PeerLayout {
  long long shard_f4, shard_bytes, result_bytes;
  size_t total;
};
static void peer_layout(long long numel, int world, PeerLayout *L) {
  const long long n4 = numel / 4;
  L->shard_f4 = (n4 + world - 1) / world;
  // a float4 travels as two 16-byte lines: two floats and two copies of the call number each
  L->shard_bytes = static_cast<long long>(align256(static_cast<size_t>(L->shard_f4) * cb2::kPeerLineBytesPerF4));
  L->result_bytes = static_cast<long long>(align256(static_cast<size_t>(n4) * cb2::kPeerLineBytesPerF4));
  L->total = cb2::kPeerControlBytes + 2 * static_cast<size_t>(world) * L->shard_bytes + 2 * static_cast<size_t>(L->result_bytes);
}

size_t cb2_peer_allreduce_buffer_size(long long numel, int world) {
  if (numel <= 0 || numel % 4 || numel / 4 > 0x3fffffff || world < 1 || world > cb2::kPeerMaxWorld)
    return 0;
  PeerLayout L;
  peer_layout(numel, world, &L);
  return L.total;
}

int cb2_peer_allreduce(const cb2_peer_allreduce_args *a, void *stream_v) {
  CB2_CHECK_ARG(a != nullptr, "null arguments");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  DeviceState *dev;
  int rc = get_device(&dev);
  if (rc)
    return rc;
  CB2_CHECK_ARG(a->world >= 1 && a->world <= cb2::kPeerMaxWorld && a->rank >= 0 && a->rank < a->world,
                "bad rank / world (%d, %d)", a->rank, a->world);
  CB2_CHECK_ARG(a->numel > 0 && a->numel % 4 == 0 && a->numel / 4 <= 0x3fffffff, "numel must be a positive multiple of 4 below 2^32");
  CB2_CHECK_RT(a->peer_buffers && a->src && (a->out_f32 || a->out_f16), "buffers, source and an output must not empty");
  CB2_CHECK_ARG(aligned16(a->src) && aligned16(a->out_f32) && (reinterpret_cast<uintptr_t>(a->out_f16) & 7u) == 0,
                "source and outputs must be 16-byte (fp16: 8-byte) aligned");
  cb2::PeerReduceParams p;
  memset(&p, 0, sizeof(p));
  for (int r = 0; r < a->world; ++r) {
    CB2_CHECK_RT(a->peer_buffers[r] != nullptr && reinterpret_cast<uintptr_t>(a->peer_buffers[r]) % 256 == 0,
                 "peer buffer %d is null or not 256-byte aligned", r);
    p.peer[r] = reinterpret_cast<unsigned char *>(a->peer_buffers[r]);
  }
  PeerLayout L;
  peer_layout(a->numel, a->world, &L);
  p.src = a->src;
  p.out32 = a->out_f32;
  p.out16 = reinterpret_cast<__half *>(a->out_f16);
  p.n4 = static_cast<int>(a->numel / 4);
  p.shard_f4 = static_cast<int>(L.shard_f4);
  p.shard_bytes = L.shard_bytes;
  p.result_bytes = L.result_bytes;
  p.rank = a->rank;
  p.world = a->world;
  p.timeout_ns = a->timeout_ns ? a->timeout_ns : 1000000000ull;
  p.status = dev->status;
  // every CTA waits for data that other GPUs send only after they have seen this grid's whole
  // scatter: the whole grid must be resident at once, beside whatever else runs (small CTAs)
  static const int max_grid = [] {
    const char *v = getenv("CUMM_B200_PEER_GRID");
    const int g = v ? atoi(v) : 96;
    return g >= 1 ? g : 96;
  }();
  int grid = static_cast<int>(std::min<long long>((a->numel / 4 + cb2::kPeerThreads - 1) / cb2::kPeerThreads, max_grid));
  grid = std::max(1, std::min(grid, dev->num_sms));
  CB2_CHECK_ARG(a->own_sm_smem_bytes >= 0 && a->own_sm_smem_bytes <= 48 * 1024, "own_sm_smem_bytes must be 0 .. 48 KiB");
  cb2::peer_reduce_kernel<<<grid, cb2::kPeerThreads, static_cast<size_t>(a->own_sm_smem_bytes), stream>>>(p);
  CB2_CUDA(cudaGetLastError());
  g_launches.fetch_add(1);
  return CB2_OK;
}

// ---------------------------------------------------------------- the kernel table
static cb2_kernel_desp make_desp(int op_type, int shuffle, bool int8, bool ta, bool tb, int tn, int tk) {
  cb2_kernel_desp d;
  memset(&d, 0, sizeof(d));
  d.op_type = op_type;
  d.shuffle_type = shuffle;
  d.dtype_a = d.dtype_b = d.dtype_c = int8 ? CB2_DTYPE_I8 : CB2_DTYPE_F16;
  d.dacc = int8 ? CB2_DTYPE_I32 : CB2_DTYPE_F32;
  d.dcomp = CB2_DTYPE_F32;
  d.trans_a = ta;
  d.trans_b = tb;
  d.trans_c = 0;
  const int shape[3] = {128, tn, tk};
  for (int i = 0; i < 3; ++i)
    d.tile_shape[i] = d.warp_tile_shape[i] = shape[i];
  d.tensorop[0] = 128;
  d.tensorop[1] = tn;
  d.tensorop[2] = int8 ? 32 : 16;
  d.num_stage = 3;
  d.element_per_access = int8 ? 16 : 8;
  d.split_k_serial = (op_type == CB2_CONV_BACKWARD_WEIGHT || shuffle == CB2_SHUFFLE_AB) ? 1 : 0;
  d.mask_sparse = op_type >= 0 ? 1 : 0;
  d.increment_k_first = op_type >= 0 ? 1 : 0;
  d.is_int8_inference = int8 ? 1 : 0;
  d.min_arch_major = 10;
  d.min_arch_minor = 0;
  return d;
}

static int emit(const cb2_kernel_desp &d, cb2_kernel_desp *out, int capacity, int n) {
  if (out && n < capacity)
    out[n] = d;
  return n + 1;
}

// The variants launch_rowconv and run_wgrad can dispatch to (the CB2_INST list above).
int cb2_enumerate_gemm_desps(cb2_kernel_desp *out, int capacity) {
  int n = 0;
  const int shuffles[2] = {CB2_SHUFFLE_NONE, CB2_SHUFFLE_AC};
  for (int s = 0; s < 2; ++s)
    for (int tb = 1; tb >= 0; --tb)
      for (int tn = 64; tn <= 128; tn += 64)
        for (int tk = 64; tk <= 128; tk += 64)
          n = emit(make_desp(-1, shuffles[s], false, false, tb != 0, tn, tk), out, capacity, n);
  for (int tn = 64; tn <= 128; tn += 64)
    n = emit(make_desp(-1, CB2_SHUFFLE_AB, false, true, false, tn, 128), out, capacity, n);
  return n;
}

int cb2_enumerate_conv_desps(cb2_kernel_desp *out, int capacity) {
  int n = 0;
  // every variant twice: for kernel volumes up to 32, and (dynamic_mask) up to 128
  for (int dyn = 0; dyn <= 1; ++dyn) {
    auto add = [&](cb2_kernel_desp d) {
      d.dynamic_mask = dyn;
      n = emit(d, out, capacity, n);
    };
    // (trans_a, trans_b) per op: cumm/conv/params.py:61-69
    for (int op = CB2_CONV_FORWARD; op <= CB2_CONV_BACKWARD_INPUT; ++op)
      for (int tn = 64; tn <= 128; tn += 64)
        for (int tk = 64; tk <= 128; tk += 64)
          add(make_desp(op, CB2_SHUFFLE_NONE, false, false, op == CB2_CONV_FORWARD, tn, tk));
    for (int tn = 64; tn <= 128; tn += 64) {
      add(make_desp(CB2_CONV_BACKWARD_WEIGHT, CB2_SHUFFLE_NONE, false, true, false, tn, 128));
      add(make_desp(CB2_CONV_FORWARD, CB2_SHUFFLE_NONE, true, false, true, tn, 128));
    }
  }
  return n;
}

const char *cb2_last_error(void) { return g_err.c_str(); }

int cb2_tile_m(void) { return 128; }

uint64_t cb2_launch_count(void) { return g_launches.load(); }

int cb2_last_launch_info(int *num_regs, int *num_threads, int *smem_bytes) {
  if (num_regs)
    *num_regs = g_last_launch.num_regs;
  if (num_threads)
    *num_threads = g_last_launch.num_threads;
  if (smem_bytes)
    *smem_bytes = g_last_launch.smem_bytes;
  return CB2_OK;
}

int cb2_last_launch_cluster(void) { return g_last_launch.cluster; }

int cb2_device_status(int *status) {
  DeviceState *dev;
  int rc = get_device(&dev);
  if (rc)
    return rc;
  CB2_CUDA(cudaDeviceSynchronize());
  int v = 0;
  CB2_CUDA(cudaMemcpy(&v, dev->status, sizeof(int), cudaMemcpyDeviceToHost));
  if (v != 0)  // a kernel that gave up may have left its scheduling counters non-zero: clear everything
    CB2_CUDA(cudaMemset(dev->status, 0, kStatusBytes));
  if (status)
    *status = v;
  return CB2_OK;
}

size_t cb2_gemm_workspace_size(const cb2_gemm_args *a) {
  if (!a || a->shuffle_type != CB2_SHUFFLE_AB)
    return 0;
  DeviceState *dev;
  if (get_device(&dev))
    return 0;
  WgradLayout L;
  wgrad_layout(dev->num_sms, a->max_ctas, a->m, a->n, a->k, 1, a->tile_n, &L);
  return L.total;
}

size_t cb2_conv_workspace_size(const cb2_conv_args *a) {
  if (!a || a->op_type != CB2_CONV_BACKWARD_WEIGHT)
    return 0;
  DeviceState *dev;
  if (get_device(&dev))
    return 0;
  WgradLayout L;
  wgrad_layout(dev->num_sms, a->max_ctas, a->K, a->C, a->N, a->kernel_volume, a->tile_n, &L);
  return L.total;
}

size_t cb2_conv_workspace_size_lists(const cb2_conv_args *a) {
  if (!a || a->op_type != CB2_CONV_BACKWARD_WEIGHT)
    return 0;
  DeviceState *dev;
  if (get_device(&dev))
    return 0;
  WgradLayout L;
  wgrad_layout(dev->num_sms, a->max_ctas, a->K, a->C, a->N, a->kernel_volume, a->tile_n, &L);
  return L.total_lists;
}

size_t cb2_static_scratch_bytes(void) { return kStaticScratchBytes; }

int cb2_conv_backward_weight_static(const cb2_conv_args *a, void *stream_v) {
  CB2_CHECK_ARG(a != nullptr, "null arguments");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  StaticState *st;
  int rc = get_device_static(&st);
  if (rc)
    return rc;
  CB2_CHECK_RT(a->op_type == CB2_CONV_BACKWARD_WEIGHT, "the static-scratch entry point computes the weight gradient only");
  CB2_CHECK_RT(a->ptr_A && a->ptr_B && a->ptr_C, "input, weight, output must not empty");
  CB2_CHECK_RT(a->indice_ptr && a->mask_ptr && a->mask_argsort_ptr, "error: indices, mask or mask_argsort empty");
  CB2_CHECK_RT(a->kernel_volume >= 1 && a->kernel_volume <= 32, "kernel volume %d is not supported", a->kernel_volume);
  CB2_CHECK_ARG(a->N >= 0 && a->C > 0 && a->K > 0, "bad N,C,K (%d,%d,%d)", a->N, a->C, a->K);
  CB2_CHECK_RT(kind_of(a->dtype_a, a->dtype_b, a->dtype_c, a->is_int8_inference, true) == 0,
               "can't find any suitable algo for dtypes (%d,%d,%d)", a->dtype_a, a->dtype_b, a->dtype_c);
  CB2_CHECK_ARG(a->C % 8 == 0 && a->K % 8 == 0, "fp16 channel counts must be multiples of 8");
  CB2_CHECK_RT(a->mask_width > 0 && (a->mask_width % 128 == 0 || 128 % a->mask_width == 0),
               "error: mask_width must be positive and divide or be a multiple of %d", 128);
  const int need_words = (a->N + a->mask_width - 1) / a->mask_width;
  CB2_CHECK_RT(a->mask_words >= need_words, "reduced mask has %d words, %d needed", a->mask_words, need_words);
  WgradLayout L;
  wgrad_layout(st->dev.num_sms, a->max_ctas, a->K, a->C, a->N, a->kernel_volume, a->tile_n, &L);
  CB2_CHECK_RT(L.total <= kStaticScratchBytes,
               "this problem (K=%d, C=%d, N=%d) needs %zu bytes of scratch; the static scratch holds %zu. Use "
               "cb2_conv_run with a caller-provided workspace instead.",
               a->K, a->C, a->N, L.total, kStaticScratchBytes);
  WgradParams p;
  memset(&p, 0, sizeof(p));
  p.dout = a->ptr_A;
  p.x = a->ptr_B;
  p.indices = a->indice_ptr;
  p.rmask = a->mask_ptr;
  p.argsort = a->mask_argsort_ptr;
  p.ld_dout = a->K;
  p.ld_x = a->C;
  p.n_rows = a->N;
  p.a_rows = a->rows_A;
  p.b_rows = a->rows_B;
  p.m_total = a->K;
  p.n_total = a->C;
  p.kv = a->kernel_volume;
  p.mask_width = a->mask_width;
  p.words = 1;
  p.rmask_words = a->mask_words;
  p.mask_filter = a->mask_filter;
  p.mode = kWgradMaskConv;
  p.out = a->ptr_C;
  p.src = a->ptr_D ? a->ptr_D : a->ptr_C;
  p.ldo = (long long)a->kernel_volume * a->C;
  p.f_stride = a->C;
  p.alpha = a->alpha;
  p.beta = a->beta;
  p.out_f32 = a->dtype_c == CB2_DTYPE_F32 ? 1 : 0;
  // the planning kernel of every call clears the control words the main kernel uses and the main
  // kernel rewrites every partial it later reads, so whatever an earlier call (of any size) left
  // in the scratch does not matter
  return run_wgrad(&st->dev, p, a->tile_n, a->max_ctas, 0, st->scratch, kStaticScratchBytes, stream);
}

int cb2_static_status(int *status) {
  StaticState *st;
  int rc = get_device_static(&st);
  if (rc)
    return rc;
  CB2_CUDA(cudaDeviceSynchronize());
  int v = 0;
  CB2_CUDA(cudaMemcpy(&v, st->dev.status, sizeof(int), cudaMemcpyDeviceToHost));
  if (v != 0)
    CB2_CUDA(cudaMemset(st->dev.status, 0, sizeof(int)));
  if (status)
    *status = v;
  return CB2_OK;
}

int cb2_gemm_run(const cb2_gemm_args *a, void *stream_v) {
  CB2_CHECK_ARG(a != nullptr, "null arguments");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  DeviceState *dev;
  int rc = get_device(&dev);
  if (rc)
    return rc;
  CB2_CHECK_RT(a->ptr_A && a->ptr_B && a->ptr_C, "a,b,c must not empty");
  CB2_CHECK_RT(!a->trans_c, "trans_c is not supported by the sm_100a kernels");
  const int kind = kind_of(a->dtype_a, a->dtype_b, a->dtype_c, 0, false);
  CB2_CHECK_RT(kind == 0, "can't find any suitable algo for dtypes (%d,%d,%d): only f16,f16,f16 is built",
               a->dtype_a, a->dtype_b, a->dtype_c);
  CB2_CHECK_ARG(a->m >= 0 && a->n > 0 && a->k >= 0, "bad m,n,k (%d,%d,%d)", a->m, a->n, a->k);
  if (a->shuffle_type == CB2_SHUFFLE_AB) {
    CB2_CHECK_RT(a->trans_a && !a->trans_b, "shuffle AB must be nt, i.e. backward weight");
    CB2_CHECK_RT(a->indiceA && a->indiceBorC, "a_inds,b_inds tensor must not empty");
    CB2_CHECK_ARG(a->m % 8 == 0 && a->n % 8 == 0,
                  "this m, n, k isn't supported due to misaligned contiguous dim.");
    WgradParams p;
    memset(&p, 0, sizeof(p));
    p.dout = a->ptr_A;
    p.x = a->ptr_B;
    p.a_inds = a->indiceA;
    p.b_inds = a->indiceBorC;
    p.ld_dout = a->stride_A;
    p.ld_x = a->stride_B;
    p.n_rows = a->k;
    p.a_rows = a->rows_A;
    p.b_rows = a->rows_B;
    p.m_total = a->m;
    p.n_total = a->n;
    p.kv = 1;
    p.mask_width = 128;
    p.words = 1;
    p.mask_filter = 0xffffffffu;
    p.mode = kWgradPairList;
    p.out = a->ptr_C;
    p.src = a->ptr_D ? a->ptr_D : a->ptr_C;
    p.ldo = a->stride_C;
    p.f_stride = 0;
    p.alpha = a->alpha;
    p.beta = a->beta;
    p.out_f32 = 0;
    return run_wgrad(dev, p, a->tile_n, a->max_ctas, a->reuse_plan, a->workspace, a->workspace_bytes, stream);
  }
  CB2_CHECK_RT(a->shuffle_type == CB2_SHUFFLE_AC || a->shuffle_type == CB2_SHUFFLE_NONE, "unknown shuffle type %d",
               a->shuffle_type);
  CB2_CHECK_RT(!a->trans_a, "a of shuffle AB must be row major");
  if (a->shuffle_type == CB2_SHUFFLE_AC)
    CB2_CHECK_RT(a->indiceBorC != nullptr, "a_inds,c_inds tensor must not empty");
  CB2_CHECK_ARG(a->k % 8 == 0 && a->n % 8 == 0, "this m, n, k isn't supported due to misaligned contiguous dim.");
  RowConvParams p;
  memset(&p, 0, sizeof(p));
  p.a = a->ptr_A;
  p.out = a->ptr_C;
  p.a_inds = a->indiceA;
  p.c_inds = a->indiceBorC;
  p.lda = a->stride_A;
  p.ldo = a->stride_C;
  p.n_rows = a->m;
  p.a_rows = a->rows_A;
  p.red = a->k;
  p.nn = a->n;
  p.kv = 1;
  p.mask_words = 1;
  p.mode = kModeGatherGemm;
  p.mask_filter = 0xffffffffu;
  p.alpha = a->alpha;
  p.beta = a->beta;
  p.act_alpha = a->act_alpha;
  p.act_type = a->act_type;
  if (a->beta != 0.f) {
    p.src = a->ptr_D ? a->ptr_D : a->ptr_C;
    p.src_mode = a->d_is_vector ? kSrcVector : kSrcRows;
    p.lds = a->ptr_D ? a->stride_D : a->stride_C;
    if (a->d_is_vector)
      CB2_CHECK_RT(a->ptr_D != nullptr, "d must be a valid bias");
  }
  // B: [n, k] (trans_b) is K-major for the tensor core, [k, n] is MN-major.
  const bool b_mn = !a->trans_b;
  const uint64_t inner = b_mn ? a->n : a->k;
  const uint64_t outer = b_mn ? a->k : a->n;
  return run_rowconv(dev, p, 0, b_mn, a->tile_n, a->tile_k, a->sched_scratch, a->max_ctas, a->ptr_B, inner, 1, outer,
                     a->stride_B, a->stride_B, stream);
}

int cb2_conv_run(const cb2_conv_args *a, void *stream_v) {
  CB2_CHECK_ARG(a != nullptr, "null arguments");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  DeviceState *dev;
  int rc = get_device(&dev);
  if (rc)
    return rc;
  CB2_CHECK_RT(a->ptr_A && a->ptr_B && a->ptr_C, "input, weight, output must not empty");
  CB2_CHECK_RT(a->indice_ptr != nullptr, "error: indices empty");
  CB2_CHECK_RT(a->mask_ptr != nullptr, "error: mask empty");
  CB2_CHECK_RT(a->mask_argsort_ptr != nullptr, "error: mask_argsort empty");
  CB2_CHECK_RT(a->kernel_volume >= 1 && a->kernel_volume <= 128,
               "kernel volume %d: the kernels handle up to 128 filter offsets (four mask words per row)",
               a->kernel_volume);
  CB2_CHECK_RT(a->groups == 1 || a->groups == 0, "groups must be 1");
  CB2_CHECK_ARG(a->N >= 0 && a->C > 0 && a->K > 0, "bad N,C,K (%d,%d,%d)", a->N, a->C, a->K);
  const bool wgrad = a->op_type == CB2_CONV_BACKWARD_WEIGHT;
  const int kind = kind_of(a->dtype_a, a->dtype_b, a->dtype_c, a->is_int8_inference, wgrad);
  CB2_CHECK_RT(kind >= 0, "can't find any suitable algo for dtypes (%d,%d,%d) int8_inference=%d", a->dtype_a,
               a->dtype_b, a->dtype_c, a->is_int8_inference);
  if (kind == 1) {
    CB2_CHECK_RT(a->op_type == CB2_CONV_FORWARD, "int8 inference is forward only");
    CB2_CHECK_RT(a->bias_pointer && a->scale_pointer, "int8 inference must have both scale and bias");
    CB2_CHECK_ARG(a->C % 16 == 0 && a->K % 16 == 0, "int8 channel counts must be multiples of 16");
  } else {
    CB2_CHECK_ARG(a->C % 8 == 0 && a->K % 8 == 0, "fp16 channel counts must be multiples of 8");
  }
  if (wgrad) {
    CB2_CHECK_RT(a->mask_width > 0 && (a->mask_width % 128 == 0 || 128 % a->mask_width == 0),
                 "error: mask_width must be positive and divide or be a multiple of %d", 128);
    const int need_words = (a->N + a->mask_width - 1) / a->mask_width * ((a->kernel_volume + 31) / 32);
    CB2_CHECK_RT(a->mask_words >= need_words, "reduced mask has %d words, %d needed", a->mask_words, need_words);
    WgradParams p;
    memset(&p, 0, sizeof(p));
    p.dout = a->ptr_A;
    p.x = a->ptr_B;
    p.indices = a->indice_ptr;
    p.rmask = a->mask_ptr;
    p.argsort = a->mask_argsort_ptr;
    p.ld_dout = a->K;
    p.ld_x = a->C;
    p.n_rows = a->N;
    p.a_rows = a->rows_A;
    p.b_rows = a->rows_B;
    p.m_total = a->K;
    p.n_total = a->C;
    p.kv = a->kernel_volume;
    p.mask_width = a->mask_width;
    p.words = (a->kernel_volume + 31) / 32;
    p.rmask_words = a->mask_words / p.words;
    p.mask_filter = a->mask_filter;
    p.mode = kWgradMaskConv;
    p.out = a->ptr_C;
    p.src = a->ptr_D ? a->ptr_D : a->ptr_C;
    p.ldo = (long long)a->kernel_volume * a->C;
    p.f_stride = a->C;
    p.alpha = a->alpha;
    p.beta = a->beta;
    p.out_f32 = a->dtype_c == CB2_DTYPE_F32 ? 1 : 0;
    return run_wgrad(dev, p, a->tile_n, a->max_ctas, a->reuse_plan, a->workspace, a->workspace_bytes, stream);
  }
  const bool dgrad = a->op_type == CB2_CONV_BACKWARD_INPUT;
  CB2_CHECK_RT(dgrad || a->op_type == CB2_CONV_FORWARD, "unknown op type %d", a->op_type);
  RowConvParams p;
  memset(&p, 0, sizeof(p));
  p.a = a->ptr_A;
  p.out = a->ptr_C;
  p.indices = a->indice_ptr;
  p.mask = a->mask_ptr;
  p.argsort = a->mask_argsort_ptr;
  p.mask_out = dgrad ? nullptr : a->mask_out_ptr;
  p.n_rows = a->N;
  p.a_rows = a->rows_A;
  p.red = dgrad ? a->K : a->C;
  p.nn = dgrad ? a->C : a->K;
  p.lda = p.red;
  p.ldo = p.nn;
  p.kv = a->kernel_volume;
  p.mask_words = (a->kernel_volume + 31) / 32;
  p.mode = kModeMaskConv;
  p.tables_fixed = a->reuse_plan & 1;
  p.skip_empty_tiles = dgrad ? 1 : 0;
  p.reverse_mask = (dgrad && a->reverse_mask) ? 1 : 0;
  p.mask_filter = a->mask_filter;
  p.alpha = a->alpha;
  p.beta = a->beta;
  p.act_alpha = a->act_alpha;
  p.act_type = a->act_type;
  if (kind == 1) {
    p.scale = reinterpret_cast<const float *>(a->scale_pointer);
    p.bias = reinterpret_cast<const float *>(a->bias_pointer);
    if (a->beta != 0.f) {
      p.src = a->ptr_D ? a->ptr_D : a->ptr_C;
      p.src_mode = kSrcRows;
      p.lds = p.nn;
    }
  } else if (a->beta != 0.f) {
    p.src = a->ptr_D ? a->ptr_D : a->ptr_C;
    p.src_mode = a->d_is_bias ? kSrcVector : kSrcRows;
    p.lds = p.nn;
  }
  // weight [K, kv, C]: forward reduces over C (K-major B), backward input over K (MN-major B)
  return run_rowconv(dev, p, kind, dgrad, a->tile_n, a->tile_k, a->sched_scratch, a->max_ctas, a->ptr_B, a->C,
                     a->kernel_volume, a->K, a->C, (uint64_t)a->kernel_volume * a->C, stream);
}

} // extern "C"
