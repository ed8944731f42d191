// C-ABI entry points of libb200gmm (declared in include/b200gmm.h): argument
// checks, TMA tensor-map construction and kernel launches.  No torch types, no
// exceptions, no allocation: scratch comes from the caller.
#include "../../include/b200gmm.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <mutex>
#include <vector>

#include "ep_exchange.cuh"
#include "gmm_kernel.cuh"

namespace {

using namespace b200gmm;

std::atomic<int64_t> g_launches{0};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

typedef CUresult (*CtxGetCurrentFn)(CUcontext*);

CtxGetCurrentFn ctx_get_current_fn() {
  static CtxGetCurrentFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<CtxGetCurrentFn>(p);
  }();
  return fn;
}

// cuTensorMapEncodeTiled is a driver call and fails with "invalid context" on a
// thread that has a CUDA device selected but no context bound yet (e.g. an
// autograd worker whose allocations all came from a cache).  Binding the
// device's primary context to the calling thread is what cudaSetDevice does.
int ensure_context(int dev) {
  CtxGetCurrentFn get = ctx_get_current_fn();
  CUcontext ctx = nullptr;
  if (get != nullptr && get(&ctx) == CUDA_SUCCESS && ctx != nullptr) return B200GMM_OK;
  if (cudaSetDevice(dev) != cudaSuccess) return B200GMM_ECUDA;
  if (get != nullptr && (get(&ctx) != CUDA_SUCCESS || ctx == nullptr)) return B200GMM_ECUDA;
  return B200GMM_OK;
}

struct DeviceInfo {
  int sm_count = 0;
  int cc_major = 0;
  int pair_ctas = 0;  // CTAs a launch of the 2-CTA-cluster variant may use (even, <= sm_count)
  bool attrs_set = false;
};

// Everything one launch of gmm_kernel needs, whatever the variant.
struct LaunchArgs {
  int grid = 0;
  cudaStream_t stream = nullptr;
  CUtensorMap map_a, map_b, map_b2, map_c, map_a2;
  __nv_bfloat16* c = nullptr;
  const int64_t* batch_sizes = nullptr;  // device
  Problem p;
  uint32_t* status = nullptr;
  CUtensorMap* slots = nullptr;
  uint32_t* sched_counter = nullptr;      // zeroed on the stream before the launch (unused: single_wave)
  InlineSizes inline_sizes;               // batch_sizes == nullptr: these
  bool overlap = false;                   // the prologue may overlap the kernel before it in the stream
  const int64_t* row_dest = nullptr;      // scatter / combine epilogue
  const float* row_scale = nullptr;
  int reduce_add = 0;
  const int32_t* a_rows = nullptr;        // gather variant
  const __nv_bfloat16* a_src = nullptr;
  int64_t a_src_rows = 0;
  int64_t dest_lo = 0, dest_hi = 0;       // window every row_dest entry must fall into (0, 0: unchecked)
  const __nv_bfloat16* gate_grad = nullptr;  // gated product: output gradient, selects the backward epilogue
  PushArgs push = {};                     // rows to move while the product runs (src == nullptr: none)
};

template <int MODE, int CTAS, bool GATHER, bool SWIGLU, bool PUSH = false, bool PAIR_SWAP = false>
cudaError_t launch_gmm(const LaunchArgs& a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.grid);
  cfg.blockDim = dim3(GATHER ? GatherWarps<CTAS>::kBlockThreads : (PUSH ? kGemmPushThreads : kThreads));
  cfg.dynamicSmemBytes = PUSH ? kSmemBytesPush : kSmemBytes;
  cfg.stream = a.stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CTAS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = a.overlap ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, gmm_kernel<MODE, CTAS, GATHER, SWIGLU, PUSH, PAIR_SWAP>, a.map_a, a.map_b, a.map_b2, a.map_c, a.map_a2, a.c,
                            a.batch_sizes, a.p, a.status, a.slots, a.sched_counter, a.row_dest, a.a_rows, a.a_src, a.a_src_rows,
                            a.row_scale, a.reduce_add, a.dest_lo, a.dest_hi, a.gate_grad, a.push, a.inline_sizes);
}

// The tile counter's zeros, as a kernel that overlaps its neighbours (gmm_kernel.cuh).
cudaError_t zero_counter(uint32_t* sched_counter, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(32);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, zero_counter_kernel, sched_counter);
}

// The two gradients of a small product (gmm_kernel.cuh: gmm_gradients_kernel), as two launches prepared
// them.
template <int MODE>
cudaError_t launch_gradients(const LaunchArgs& d, const LaunchArgs& w) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(d.grid + w.grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = d.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto args = [](const LaunchArgs& a) { return ProductArgs{a.map_a, a.map_b, a.map_c, a.c, a.p, a.grid}; };
  return cudaLaunchKernelEx(&cfg, gmm_gradients_kernel<MODE>, args(d), args(w), d.batch_sizes, d.status, d.slots, d.inline_sizes);
}

// The plain forward / dgrad kernels with push warps (a.push.src != nullptr).
cudaError_t launch_with_push(const LaunchArgs& a, int ctas) {
  if (a.p.mode == kNN)
    return ctas == 2 ? launch_gmm<kNN, 2, false, false, true>(a) : launch_gmm<kNN, 1, false, false, true>(a);
  if (a.p.mode == kNT)
    return ctas == 2 ? launch_gmm<kNT, 2, false, false, true>(a) : launch_gmm<kNT, 1, false, false, true>(a);
  return cudaErrorInvalidValue;
}

// The layout (a.p.mode) picks the last template argument; the gated product has no wgrad form.
template <int CTAS, bool GATHER, bool SWIGLU>
cudaError_t launch_layout(const LaunchArgs& a) {
  if (a.p.mode == kNN) return launch_gmm<kNN, CTAS, GATHER, SWIGLU>(a);
  if (a.p.mode == kNT) return launch_gmm<kNT, CTAS, GATHER, SWIGLU>(a);
  if constexpr (!SWIGLU) return launch_gmm<kTN, CTAS, GATHER, false>(a);
  return cudaErrorInvalidValue;
}

template <bool GATHER, bool SWIGLU>
cudaError_t launch_variant(const LaunchArgs& a, int ctas) {
  if constexpr (!GATHER) {
    if (ctas == 2 && a.p.swap_rows > 0)
      return a.p.mode == kNN ? launch_gmm<kNN, 2, false, SWIGLU, false, true>(a) : launch_gmm<kNT, 2, false, SWIGLU, false, true>(a);
  }
  return ctas == 2 ? launch_layout<2, GATHER, SWIGLU>(a) : launch_layout<1, GATHER, SWIGLU>(a);
}

template <int MODE, int CTAS, bool GATHER = false, bool SWIGLU = false, bool PUSH = false, bool PAIR_SWAP = false>
cudaError_t set_smem_attr() {
  return cudaFuncSetAttribute(gmm_kernel<MODE, CTAS, GATHER, SWIGLU, PUSH, PAIR_SWAP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(PUSH ? kSmemBytesPush : kSmemBytes));
}

// Per-device facts, looked up once.  Index = CUDA device ordinal.
int device_info(DeviceInfo** out) {
  static std::mutex mu;
  static DeviceInfo infos[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return B200GMM_ECUDA;
  if (ensure_context(dev) != B200GMM_OK) return B200GMM_ECUDA;
  std::lock_guard<std::mutex> lock(mu);
  DeviceInfo& d = infos[dev];
  if (d.sm_count == 0) {
    if (cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&d.cc_major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess)
      return B200GMM_ECUDA;
  }
  if (d.cc_major != 10) return B200GMM_EDEVICE;
  if (!d.attrs_set) {
    if (set_smem_attr<kNN, 1>() != cudaSuccess || set_smem_attr<kNT, 1>() != cudaSuccess ||
        set_smem_attr<kTN, 1>() != cudaSuccess || set_smem_attr<kNN, 2>() != cudaSuccess ||
        set_smem_attr<kNT, 2>() != cudaSuccess || set_smem_attr<kTN, 2>() != cudaSuccess ||
        set_smem_attr<kNN, 1, true>() != cudaSuccess || set_smem_attr<kNT, 1, true>() != cudaSuccess ||
        set_smem_attr<kNN, 2, true>() != cudaSuccess || set_smem_attr<kNT, 2, true>() != cudaSuccess ||
        set_smem_attr<kTN, 1, true>() != cudaSuccess || set_smem_attr<kTN, 2, true>() != cudaSuccess ||
        set_smem_attr<kNN, 1, false, true>() != cudaSuccess || set_smem_attr<kNT, 1, false, true>() != cudaSuccess ||
        set_smem_attr<kNN, 2, false, true>() != cudaSuccess || set_smem_attr<kNT, 2, false, true>() != cudaSuccess ||
        set_smem_attr<kNN, 1, false, false, true>() != cudaSuccess || set_smem_attr<kNT, 1, false, false, true>() != cudaSuccess ||
        set_smem_attr<kNN, 2, false, false, true>() != cudaSuccess || set_smem_attr<kNT, 2, false, false, true>() != cudaSuccess ||
        set_smem_attr<kNN, 2, false, false, false, true>() != cudaSuccess ||
        set_smem_attr<kNT, 2, false, false, false, true>() != cudaSuccess ||
        set_smem_attr<kNN, 2, false, true, false, true>() != cudaSuccess || set_smem_attr<kNT, 2, false, true, false, true>() != cudaSuccess)
      return B200GMM_ECUDA;
    if (cudaFuncSetAttribute(gmm_gradients_kernel<kNN>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemBytes)) != cudaSuccess ||
        cudaFuncSetAttribute(gmm_gradients_kernel<kNT>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemBytes)) != cudaSuccess)
      return B200GMM_ECUDA;
    // How many 2-CTA clusters of this kernel the device can hold at once (a GPC
    // with an odd number of free SMs leaves one out).
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(d.sm_count & ~1);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, gmm_kernel<kNN, 2>, &cfg) != cudaSuccess || clusters <= 0) {
      (void)cudaGetLastError();
      clusters = 0;
    }
    d.pair_ctas = 2 * clusters;
    if (d.pair_ctas > (d.sm_count & ~1)) d.pair_ctas = d.sm_count & ~1;
    d.attrs_set = true;
  }
  *out = &d;
  return B200GMM_OK;
}

int env_int(const char* name, int fallback) {
  const char* v = std::getenv(name);
  return (v != nullptr && *v != '\0') ? std::atoi(v) : fallback;
}

int64_t env_int64(const char* name, int64_t fallback) {
  const char* v = std::getenv(name);
  return (v != nullptr && *v != '\0') ? std::atoll(v) : fallback;
}

// bf16 tensor map (128-byte swizzle unless told otherwise); dims/box innermost first,
// strides in bytes for dimensions 1 .. rank-1 (nullptr: packed).
int encode_map(CUtensorMap* map, const void* base, int rank, const uint64_t* dims,
               const uint32_t* box, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B,
               const uint64_t* strides = nullptr) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return B200GMM_ECUDA;
  cuuint64_t gdim[4];
  cuuint64_t gstride[3];
  cuuint32_t gbox[4];
  cuuint32_t estride[4] = {1, 1, 1, 1};
  uint64_t stride = 2;
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    gbox[i] = box[i];
    stride *= dims[i];
    if (i + 1 < rank) gstride[i] = strides != nullptr ? strides[i] : stride;
  }
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, static_cast<cuuint32_t>(rank),
                        const_cast<void*>(base), gdim, gstride, gbox, estride,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS && env_int("B200GMM_DEBUG", 0) != 0) {
    std::fprintf(stderr, "b200gmm: cuTensorMapEncodeTiled -> %d: base %p rank %d dims {%llu,%llu,%llu} box {%u,%u,%u}\n",
                 static_cast<int>(r), base, rank, (unsigned long long)gdim[0], (unsigned long long)gdim[1],
                 (unsigned long long)(rank > 2 ? gdim[2] : 0), gbox[0], gbox[1], rank > 2 ? gbox[2] : 0u);
  }
  return r == CUDA_SUCCESS ? B200GMM_OK : B200GMM_ETENSORMAP;
}

// A row-major [.., rows, cols] operand whose tiles are staged as boxes of 64 columns
// (MN-major for the tensor core): seen as {64, rows, cols / 64 (, experts)}, one TMA
// load brings `boxes` neighbouring 64-column boxes, which land one after the other
// in shared memory exactly as separate loads would put them.  cols % 64 == 0.
int encode_blocked(CUtensorMap* map, const void* base, uint64_t cols, uint64_t rows, uint64_t experts,
                   uint32_t box_rows, uint32_t boxes) {
  const uint64_t dims[4] = {64, rows, cols / 64, experts};
  const uint64_t strides[3] = {cols * 2, 128, rows * cols * 2};
  const uint32_t box[4] = {64, box_rows, boxes, 1};
  return encode_map(map, base, experts > 0 ? 4 : 3, dims, box, CU_TENSOR_MAP_SWIZZLE_128B, strides);
}

// Whether rows of an operand start at any 16 bytes: a k-block of such a row is five sectors in two
// lines of L2 instead of four in one.  (b's rows are d1 long in the NT layout.)
bool ragged_rows(int64_t d1, int64_t n, int trans_b) { return d1 % 16 != 0 || (!trans_b && n % 16 != 0); }

// Which kernel features a plain, gathered or gated launch uses (schedule.cuh: Problem).
struct Features {
  bool gather = false;
  bool swiglu = false;
  bool gated_backward = false;
  bool scatter = false;  // row_dest: rows of the result go where a table says
};

constexpr int kNeverWide = 1000;  // Problem::wide_cost: every tile one accumulator wide

// Problem::wide_cost, what two rounds of narrow tiles cost as a round of wide ones, in percent.
// Rows that start at any 16 bytes are bound by the bytes that enter an SM, of which a
// wide tile has three quarters (7 experts, 3001 rows, 1000 x 2504: 26.4 / 23.0 us); others by power,
// and by little else.  The gated backward's epilogue, which reads a gradient and writes two, leaves
// nothing to gain (16 experts of 1024 rows, 2048 x 4096: wide 561 us, narrow 540).  A gathered product
// copies its rows 16 bytes at a time, which a wide tile does half as often (67 experts of 206 rows, 13024 x
// 280: 260 / 211; 18 experts, 34044 rows, 3592 x 552: 250 / 213).  Scattered rows leave in 64-byte
// copies: while an accumulator's are sent the other one has to wait, unless the contraction is long
// (16384 rows, 8 experts, 4096 x 14336: 1573 / 1660; 14336 x 4096, 8192 rows: 892 / 855).
int wide_cost(const Features& f, int64_t d1, bool trans_a, bool ragged) {
  if (f.scatter && d1 < 8192) return kNeverWide;
  if (trans_a) return 97;
  if (f.gather) return 70;
  return ragged ? 80 : (f.gated_backward ? 100 : 97);
}

// Which variant a problem runs on.  Only shapes known on the host may decide
// (batch_sizes can live on the device).  B200GMM_CTAS=1|2 overrides.
//
// A one-CTA tile and a pair's narrow one are as much work for an SM, 128 x 256 outputs, so the rounds of tiles
// that the grid makes compare them, for experts of even size, half a row tile of each idle.  What
// a pair's round costs less for is bytes: per k-block an SM loads 48 KiB for 128 x 256 outputs (one CTA), 32 (a
// pair's narrow tile) or 24 (wide).  What is saved by that depends on how busy memory and the
// power supply are.
//   512 rows an expert and more: pairs, 0.76 to 1 of the time of one-CTA tiles (19 experts, 54879 rows,
//     9736 x 96: 371 us one-CTA, 284; 2 of 33358, 2248 x 1120: 410 / 339), unless one-CTA tiles make far fewer
//     rounds than the fewest a pair's can (one of 1084, 552 x 1936, gated: 11.2 / 18.7; but 6 of 1002, 2016 x 264,
//     gated, which fit one round of either: 24.2 / 21.8).
//   128 to 511 rows: pairs for rows that start at any 16 bytes, which are two lines of L2 where they
//     could be one (64 experts of 128 rows, 4088 x 8184: 1351 / 933; 7 of 428, dgrad 2504 -> 1000: 29.7 / 25.0), where
//     they make a tenth less by this reckoning, and not where one-CTA tiles are one round of fewer
//     than 384 rows each.  Others where the contraction is 1536 and more and one-CTA tiles make eight
//     rounds and more: repeated for a third of a second, under the power cap, one-CTA / pairs (64 experts of 256
//     rows, 2048 x 4096: 386 / 344, dgrad 402 / 346; 32 of 256, 4096 x 4096: 367 / 323; 128 of 128, Zipf, 4096 x 2048: 480 /
//     433; 96 of 384, 3072 x 3072: 801 / 769, gated 1527 / 1486; 64 of 384, 1536 x 4096: 379 / 340; 256 of 256, Zipf, 7168 x
//     2048: 2436 / 2382, dgrad 2322 / 2159); in bursts of 10 ms the two are even.  Short ones lose (200 of 150, Zipf,
//     512 x 512: 37.9 / 46.1, gated 59.8 / 80.6).  So do the gathered product (146 of 126, 6712 x 2496: 1185 / 1487),
//     scattered rows (64 of 116, 1864 x 2872: 199 / 204) and the gated backward (16 of 386, 1416 x 11392: 547 / 584).
//   A short contraction leaves an accumulator little time to be read out while the other one
//     fills, which a pair's wide tile does not have: one CTA below 416 (any 16 bytes) and 512 (49 experts,
//     98681 rows, 72 x 2000: 101 / 159; 81, 68558, 432 x 2608: 223 / 240; 173, 110139, 128 x 856: 77 / 113).
// wgrad loads its operands for as many k-blocks as an expert has rows, and writes as much in
// either form: the line lies at 512 rows (0.9 at 256 and 1.02 at 512; 18 experts, 34044 rows, 3592 x 552:
// 273 / 214; 7, 3001, 1000 x 2504: 34.2 / 35.2).
int choose_ctas(int z, int64_t tokens, int64_t d1, int64_t n, int trans_a, int trans_b, const Features& f = Features(),
                const DeviceInfo* dev = nullptr) {
  const int forced = env_int("B200GMM_CTAS", 0);
  if (forced == 1 || forced == 2) return forced;
  if (z <= 0 || tokens <= 0 || d1 <= 0 || n <= 0 || std::max(tokens, n) > (int64_t(1) << 32)) return 1;  // (refused later)
  const auto rows_from = [&](int64_t mean) { return tokens >= mean * int64_t(z); };
  if (trans_a) return rows_from(512) && d1 >= 256 ? 2 : 1;
  const bool ragged = ragged_rows(d1, f.swiglu ? n / 2 : n, trans_b);
  if (d1 < (ragged ? 416 : 512)) return 1;
  if (!rows_from(512) && (!rows_from(128) || f.gather || f.scatter || f.gated_backward)) return 1;
  const int64_t sms = dev != nullptr ? dev->sm_count : 148, pairs = std::max<int64_t>(dev != nullptr ? dev->pair_ctas / 2 : 74, 1);
  const auto fewest = [&](int64_t rows) { return (tokens + rows - 1) / rows; };
  const auto row_tiles = [&](int64_t rows) {  // of experts of even size, half a tile of each idle
    return z == 1 ? fewest(rows) : tokens / rows + std::min<int64_t>(z, tokens) / 2;
  };
  const int64_t nt = (n + kBlockN - 1) / kBlockN, one_tiles = row_tiles(kBlockM) * nt;
  const int64_t pair_rows = rows_from(512) ? fewest(2 * kBlockM) : row_tiles(2 * kBlockM);
  if (one_tiles <= sms && !rows_from(384)) return 1;
  if (!rows_from(512) && !ragged) return d1 >= 1536 && one_tiles >= 8 * sms ? 2 : 1;
  const int64_t one = 125 * rounds_narrow(one_tiles, sms);
  const int64_t pair = std::min(100 * rounds_narrow(pair_rows * nt, pairs),
                                wide_cost(f, d1, false, ragged) * rounds_wide(pair_rows * ((nt + 1) / 2), pairs));
  return rows_from(512) ? (112 * one < 100 * pair ? 1 : 2) : (100 * pair < 90 * one ? 2 : 1);
}

// Which launches run their tiles of few rows with swapped operands (schedule.cuh), and up
// to how many rows a tile.  What the form saves is tensor work on rows that do not exist,
// that is, power: launches that stream weights for long run into the power cap, and the
// clock follows.  What it costs is an epilogue that transposes.  Measured over 1 to 256
// experts, k = 64 .. 7168, uniform and Zipf routing, both forms in turn, 40 ms each; time
// without / with (under the power cap a figure moves by a tenth from run to run):
//   rows an expert (mean)  plain products and scattered rows: 1.00 to 1.25 up to 64 (256
//     experts, k = 7168, n = 2048, Zipf: 1128 / 908 us at 8 rows, 1457 / 1183 at 32, 1571 / 1339 at
//     64), even from 80 to 128, 0.81 to 1.02 from 144 on, where remainders share their weights
//     with whole tiles (192 rows each: 2172 / 2669 us).  Gated product: 1.04 up to 48 on
//     average (same experts, 32 rows, Zipf: 3060 / 2361 us), 0.98 at 64, 0.79 to 1.0 from 96 on.
//   contraction  scattered rows and the gated product gain most where it is short and the
//     epilogue counts (64 experts of 8 rows, n = 4096, k = 64: 30.8 / 20.6 and 39.2 / 24.6 us).  A
//     plain product's whole boxes leave as TMA stores in either form: 0.92 to 1.10 at k =
//     64 and 128, even at 256 and 384; it takes the form from 512 on.
//   tiles  where most SMs have none, one SM's pipeline is the bound, not HBM and not power:
//     1 expert of 16 rows, k = 4096: plain 0.92 with 16 tiles, 0.97 with 48, 1.01 with 64;
//     scattered 0.97, 1.02, 1.05; gated 0.84, 0.89, 0.92, and 1.06 with 100.
// Not the gathered product (0.95 to 1.0 nearly everywhere: its copies are the bound, and
// the rows that do not exist are not copied in either form), and not the gated backward,
// which reads its gradient row by row there (104 and 222 us at 40 rows, k = 512).
// A pair's tiles of up to 192 of 256 rows: the last row tile of an expert, and all of a small
// expert.  Time without / with:
//   256 experts of 256 rows on average, Zipf, 7168 x 2048: 2480 / 2244 us, dgrad 2486 / 2152; 64 experts of 64
//     rows, 4088 x 8184: 942 / 815; below 512 rows, over drawn sizes: forward and gated 1.02, dgrad 1.06.
//   large experts (8 of 1024 rows, 4096 x 14336): gated product 1676 / 1599 us, scattered rows 887 / 867,
//     forward 815 / 822 (1.04 in another run), dgrad 812 / 844; of 4096: forward 2910 / 2877, dgrad 2934 / 3055.
//     Drawn sizes: forward and gated 1.01 to 1.02 from 512 to 2048 rows, 0.98 to 1.0 above; dgrad even.  So NN up
//     to 2048 rows and NT up to 512.
//   few tiles: one pair's pipeline is the bound, as above (322 rows, one expert, 5976 x 4736: 37 us with
//     one-CTA tiles, 63 with this): a tile for every SM.
int swap_rows(const Problem& p, const Features& f, int ctas, int sm_count) {
  constexpr int64_t kMeanRows = 64, kMeanRowsGated = 48, kPlainMinK = 512;
  if (p.mode == kTN || f.gather || f.gated_backward) return 0;
  if (ctas == 2) {
    const int64_t pair_tiles = (2 * p.tokens / p.tile_m + std::min<int64_t>(p.z, p.tokens)) * p.nt / 2;
    return pair_tiles >= sm_count && p.tokens < (p.mode == kNN ? 2048 : 512) * int64_t(p.z) ? 3 * kBlockM / 2 : 0;
  }
  const int64_t tiles = int64_t(p.nt) * std::min<int64_t>(p.z, p.tokens);  // experts with rows have one row tile, mostly
  if (f.swiglu) return p.tokens <= kMeanRowsGated * p.z && 3 * tiles >= 2 * sm_count ? kBlockM / 2 : 0;
  if (!f.scatter && p.d1 < kPlainMinK) return 0;
  return p.tokens <= kMeanRows * p.z && 2 * tiles >= sm_count ? kBlockM / 2 : 0;
}

int check_problem(int z, int64_t tokens, int64_t d1, int64_t n, int trans_a, int trans_b, int ctas,
                  Problem* p, const Features& f = Features()) {
  if (trans_a && trans_b) return B200GMM_EINVAL;
  if (z < 0 || tokens < 0 || d1 < 0 || n < 0) return B200GMM_EINVAL;
  if (z > kMaxExperts) return B200GMM_ELIMIT;
  if ((d1 % 8) != 0 || (n % 8) != 0) return B200GMM_EALIGN;
  if (tokens >= (int64_t(1) << 31) - 256 || d1 >= (int64_t(1) << 31) - 256 ||
      n >= (int64_t(1) << 31) - 256)
    return B200GMM_ELIMIT;
  p->mode = trans_a ? kTN : (trans_b ? kNT : kNN);
  p->z = z;
  p->tokens = tokens;
  p->d1 = d1;
  p->n = n;
  if (ctas != 1 && ctas != 2) return B200GMM_EINVAL;
  p->tile_m = kBlockM * ctas;
  p->tile_n = kBlockN * ctas;
  derive(p);
  p->wide_a = 0;
  p->wide_b = 0;
  // Row tiles swept together: with 16 the tiles in flight are 16 x 5 (a pair: 256 x 512 each),
  // about a square of the output, and an expert of up to 4096 rows reads its weights from
  // HBM once.  (Pairs, 32768 rows, 8 experts of 4096 x 14336, 8 against 16: 3007 / 2964, dgrad
  // 2978 / 2950, wgrad 2945 / 2899 us; with 4 1 to 3 % slower than with 8.)
  p->group_m = env_int("B200GMM_GROUP_M", 16);
  if (p->group_m < 1) p->group_m = 1;
  // Tiles are drawn from a global counter.  For wgrad, where a tile's duration is
  // its expert's row count, the experts are taken largest first, so that the
  // CTAs that finish early find short tiles left.
  p->order = (z > 1 && p->mode == kTN) ? 1 : 0;
  // Transposed tiles for experts of at most 64 rows: off unless asked for.  They
  // take 4x fewer tensor-core cycles on such experts, but those experts are bound
  // by streaming their weights from HBM either way, and measured end to end the
  // launch was not faster with them (B200GMM_LIGHT=1 switches them on).
  p->light = (p->mode != kTN && ctas == 1 && !f.gather && !f.swiglu) ? env_int("B200GMM_LIGHT", 0) : 0;
  // A pair's tiles two accumulators wide or one (narrow_tiles).  wgrad's are as long as their expert has
  // rows: with few a CTA and experts of 2048 rows and more the long ones end the launch (11 experts,
  // 126529 rows, 4144 x 576: 712 us with tiles of 256 columns, 872 with 512).
  p->narrow_rounds = trans_a && tokens >= 2048 * int64_t(z) ? 16 : 0;
  p->wide_cost = wide_cost(f, d1, trans_a != 0, ragged_rows(d1, f.swiglu ? n / 2 : n, trans_b));
  p->swap_units = 1;
  p->swap_rows = 0;  // decided where the device is known (settle)
  p->dest_indexed = 0;
  p->dest_rows = 0;
  p->pair_sum = 0;
  p->zero_rest = 0;
  p->single_wave = 0;  // decided where the grid is (settle)
  const int64_t wait_ns = env_int64("B200GMM_WAIT_LIMIT_NS", static_cast<int64_t>(ptx::kWaitLimitNs));
  p->wait_ns = wait_ns > 0 ? wait_ns : static_cast<int64_t>(ptx::kWaitLimitNs);
  // Upper bound on the tile count must fit the kernel's 32-bit tile index (twice:
  // positions drawn past the end still have to fit).
  const int64_t nt = (n + kBlockN - 1) / kBlockN;
  const int64_t row_tiles = trans_a ? int64_t(z) * ((d1 + p->tile_m - 1) / p->tile_m)
                                    : (tokens / p->tile_m + 3 * int64_t(z));  // + transposed tiles, half as wide
  if (row_tiles * nt >= (int64_t(1) << 30)) return B200GMM_ELIMIT;
  return B200GMM_OK;
}

// The CTAs of a launch that fills the device.
int grid_ctas(int ctas, int sm_count, int pair_ctas) { return std::min(ctas == 2 ? pair_ctas : sm_count, kMaxCtas); }

// What check_problem leaves to where the device is known.
void settle(Problem* p, const Features& f, int ctas, int sm_count, int pair_ctas) {
  p->swap_rows = swap_rows(*p, f, ctas, sm_count);
  p->swap_units = f.swiglu ? ctas : 1;
  // A launch whose every possible tile is the first of some cluster draws no positions:
  // no counter to zero, and no more CTAs than tiles (run_impl).  Together with the inline
  // batch_sizes there this leaves a small call with one operation on the stream instead
  // of two or three; its kernel can then also start while the one before it ends.
  // A training step of 512 rows (4 experts, 128 x 128, host batch_sizes): 108.9 -> 99.3 us,
  // host-bound before and after; token generation, where the overlap counts (64 rows, 8
  // experts of 4096 x 14336): 135.9 -> 129.4 us.
  p->single_wave = !p->light && max_tiles(*p) * ctas <= grid_ctas(ctas, sm_count, pair_ctas) ? 1 : 0;
}

// Argument checks alone (no launch): what run_impl would refuse for these sizes.
int check_args_only(int z, int64_t tokens, int64_t d1, int64_t n, int trans_b) {
  Problem p;
  return check_problem(z, tokens, d1, n, 0, trans_b, 1, &p);
}

size_t round128(size_t x) { return (x + 127) & ~size_t(127); }

// ---- scratch for b200gmm_run_static ------------------------------------------
// Same layout as a caller-provided workspace, sized for the entry point's own
// expert limit.  Lives in every CUDA context that loads this library, from load
// until exit.
constexpr size_t kStaticScratchBytes =
    ((size_t(B200GMM_STATIC_MAX_EXPERTS) * sizeof(int64_t) + 16 + 127) & ~size_t(127)) +
    size_t(kMaxCtas) * kMapSlots * 2 * sizeof(CUtensorMap);
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// Device address of g_static_scratch on the current device.  In host code the
// symbol's name is only a handle; the address a kernel can use has to be asked
// for, per device, with that device current.
int static_scratch_address(void** out) {
  // One lookup per device; afterwards a plain atomic load, no lock.
  static std::atomic<void*> addr[64];
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return B200GMM_ECUDA;
  void* p = addr[dev].load(std::memory_order_acquire);
  if (p == nullptr) {
    std::lock_guard<std::mutex> lock(mu);
    p = addr[dev].load(std::memory_order_relaxed);
    if (p == nullptr) {
      if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || p == nullptr) {
        (void)cudaGetLastError();
        return B200GMM_ECUDA;
      }
      addr[dev].store(p, std::memory_order_release);
    }
  }
  *out = p;
  return B200GMM_OK;
}

// Workspace layout: [0, 8z) device copy of batch_sizes; then, 128-byte aligned,
// kMaxCtas x kMapSlots x {a, b} tensor maps edited by the wgrad kernel.
size_t maps_offset(int z) { return round128(size_t(z) * sizeof(int64_t) + 16); }
size_t maps_bytes() { return size_t(kMaxCtas) * kMapSlots * 2 * sizeof(CUtensorMap); }

// Whether a copy from this host array reads it before the copy call returns.  A pinned
// (or managed) array is read when the stream gets to the copy, and earlier work of the
// stream may be what fills it.
bool pageable(const void* host) {
  cudaPointerAttributes attr;
  if (cudaPointerGetAttributes(&attr, host) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return attr.type == cudaMemoryTypeUnregistered;
}

}  // namespace

extern "C" {

int b200gmm_workspace_bytes(int z, size_t* out_bytes) {
  if (out_bytes == nullptr || z < 0) return B200GMM_EINVAL;
  if (z > kMaxExperts) return B200GMM_ELIMIT;
  *out_bytes = maps_offset(z) + maps_bytes();
  return B200GMM_OK;
}

}  // extern "C"

namespace {

// The kernels' build_schedule, replayed: clamped row prefix sums, the order of
// the experts, tile prefix sums in that order.
struct HostSchedule {
  std::vector<int> row_start, perm, tile_start;
  HostSchedule(const Problem& p, const int64_t* sizes)
      : row_start(size_t(p.z) + 1), perm(static_cast<size_t>(p.z)), tile_start(size_t(p.z) + 1) {
    int64_t start = 0;
    for (int e = 0; e < p.z; ++e) {
      row_start[e] = static_cast<int>(start < p.tokens ? start : p.tokens);
      start += sizes[e] < 0 ? 0 : sizes[e];
    }
    row_start[p.z] = static_cast<int>(start < p.tokens ? start : p.tokens);
    for (int e = 0; e < p.z; ++e) perm[e] = e;
    if (p.order)
      std::stable_sort(perm.begin(), perm.end(), [&](int x, int y) {
        return row_start[x + 1] - row_start[x] > row_start[y + 1] - row_start[y];
      });
    for (int i = 0; i < p.z; ++i)
      tile_start[i + 1] = tile_start[i] + expert_tiles(p, row_start[perm[i] + 1] - row_start[perm[i]]);
  }
  // The kernels' TileWalker: positions come in increasing order, *pos is the cursor over the experts.
  TileOrder order(const Problem& p, int clusters) const {
    if (p.tile_n > kBlockN) return tile_order(p, tile_start.back(), clusters);
    return TileOrder{TileGrid{p.nt, kBlockN, p.group_m}, tile_start.back(), tile_start.back()};
  }
  void decode(const Problem& p, const TileOrder& o, int position, int* pos, Tile* out) const {
    int half;
    const int t = tile_of_position(o, position, &half), nt = p.tile_n > kBlockN ? o.grid.nt : 1;
    while (t >= tile_start[*pos + 1] * nt) ++*pos;
    const int e = perm[*pos];
    *out = make_tile(p, o.grid, e, t - tile_start[*pos] * nt, row_start[e], row_start[e + 1]);
    take_half(out, half);
  }
};

// Shared body of b200gmm_run and b200gmm_run_scatter.  row_dest == nullptr: rows
// go to c.  Otherwise (non-transposed a only) row i of the result goes to the
// address row_dest[i] and c is not touched.
int run_impl(const void* a, const void* b, void* c, const int64_t* batch_sizes,
             int batch_sizes_on_device, int z, int64_t tokens, int64_t dim_a1, int64_t n,
             int trans_a, int trans_b, void* workspace, size_t workspace_bytes,
             uint32_t* device_status, void* cuda_stream, const int64_t* row_dest,
             const int32_t* a_rows = nullptr, int64_t a_source_rows = 0, const void* b2 = nullptr,
             const float* row_scale = nullptr, int reduce_add = 0, const void* dest_base = nullptr,
             int64_t dest_bytes = 0, const void* gate_grad = nullptr, const PushArgs* push = nullptr,
             bool* push_launched = nullptr, bool pair_sum = false, bool zero_rest = false,
             int64_t dest_rows = -1, LaunchArgs* prepared = nullptr) {
  // prepared != nullptr: the launch is described there and left to the caller (plain products of one
  // wave of tiles).
  // dest_rows >= 0: row_dest holds rows of the [dest_rows, n] destination at
  // dest_base instead of addresses.
  // pair_sum: a is [2, tokens, dim_a1], c = a[0] x b + a[1] x b2 (b2 is then no gate).
  // zero_rest (with gate_grad): also the rows of c that belong to no expert are written.
  // push != nullptr: rows to move inside the same launch (plain forward / dgrad
  // kernels only); *push_launched tells the caller whether a launch took them.
  // gate_grad != nullptr: backward epilogue of the gated product; c is [2, tokens, n].
  if (gate_grad != nullptr && (b2 == nullptr || row_dest != nullptr || (reinterpret_cast<uintptr_t>(gate_grad) & 15)))
    return B200GMM_EINVAL;
  if (dest_base != nullptr && (row_dest == nullptr || dest_bytes < 0)) return B200GMM_EINVAL;
  if ((row_scale != nullptr || reduce_add) && row_dest == nullptr) return B200GMM_EINVAL;
  if (a_rows != nullptr && (dim_a1 == 0 || a_source_rows <= 0 || (trans_a && row_dest != nullptr)))
    return B200GMM_EINVAL;
  // b2 != nullptr: gated product silu(a @ b) * (a @ b2); n counts the columns of
  // each of b, b2 and c, the schedule runs over 2n virtual columns.
  const bool swiglu = (b2 != nullptr) && !pair_sum;
  if (swiglu && (trans_a || a_rows != nullptr)) return B200GMM_EINVAL;
  if (pair_sum && (trans_a || a_rows != nullptr || row_dest != nullptr)) return B200GMM_EINVAL;
  if (b2 != nullptr && (reinterpret_cast<uintptr_t>(b2) & 15)) return B200GMM_EALIGN;
  if (swiglu && (n % 8) != 0) return B200GMM_EALIGN;
  const int64_t n_out = n;
  if (swiglu) n = 2 * n;
  if (row_dest != nullptr) {
    if (trans_a || dim_a1 == 0) return B200GMM_EINVAL;
    if (c == nullptr) c = const_cast<void*>(a);  // never written; keeps the argument checks below uniform
  }
  Problem p;
  Features feat;
  feat.gather = (a_rows != nullptr);
  feat.swiglu = swiglu;
  feat.gated_backward = gate_grad != nullptr;
  feat.scatter = row_dest != nullptr;
  // (a call that does nothing needs no device)
  DeviceInfo* dev = nullptr;
  const int dev_rc = z > 0 && tokens > 0 && dim_a1 > 0 && n > 0 ? device_info(&dev) : B200GMM_OK;
  int ctas = prepared != nullptr ? 1 : choose_ctas(z, tokens, dim_a1, n, trans_a, trans_b, feat, dev);
  int rc = check_problem(z, tokens, dim_a1, n, trans_a, trans_b, ctas, &p, feat);
  if (rc != B200GMM_OK) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  if (z == 0) return B200GMM_OK;
  if (batch_sizes == nullptr) return B200GMM_EINVAL;

  // Degenerate shapes: nothing to multiply.  Only wgrad has output to define
  // (zeros), and only when that output is non-empty.
  if (p.mode == kTN) {
    if (dim_a1 == 0 || n == 0) return B200GMM_OK;
    if (c == nullptr) return B200GMM_EINVAL;
    if (tokens == 0) {
      if (cudaMemsetAsync(c, 0, size_t(z) * size_t(dim_a1) * size_t(n) * 2, stream) != cudaSuccess)
        return B200GMM_ECUDA;
      return B200GMM_OK;
    }
  } else {
    if (tokens == 0 || n == 0) return B200GMM_OK;
    if (c == nullptr) return B200GMM_EINVAL;
    if (dim_a1 == 0) {
      // k == 0: every product is an empty sum.
      if (cudaMemsetAsync(c, 0, size_t(tokens) * size_t(n_out) * 2, stream) != cudaSuccess)
        return B200GMM_ECUDA;
      return B200GMM_OK;
    }
  }
  if (a == nullptr || b == nullptr) return B200GMM_EINVAL;
  if (pair_sum) {
    if (b2 == nullptr) return B200GMM_EINVAL;
    // rows of a's second part and the length of both parts of the contraction, each
    // rounded up to a k-block, are 32-bit numbers in the kernel (schedule.cuh: make_tile)
    if (2 * tokens + 2 * kBlockM >= (int64_t(1) << 31) || 2 * (dim_a1 + kBlockK) >= (int64_t(1) << 31)) return B200GMM_ELIMIT;
  }
  if ((reinterpret_cast<uintptr_t>(a) & 15) || (reinterpret_cast<uintptr_t>(b) & 15) ||
      (reinterpret_cast<uintptr_t>(c) & 15))
    return B200GMM_EALIGN;

  if (dev_rc != B200GMM_OK) return dev_rc;

  if (ctas == 2 && dev->pair_ctas < 2) {
    ctas = 1;
    if ((rc = check_problem(z, tokens, dim_a1, n, trans_a, trans_b, ctas, &p, feat)) != B200GMM_OK) return rc;
  }

  const bool with_push = push != nullptr && push->src != nullptr && push->n_items > 0 && !feat.gather && !swiglu && p.mode != kTN;
  p.dest_indexed = dest_rows >= 0 ? 1 : 0;
  p.dest_rows = dest_rows;
  p.pair_sum = pair_sum ? 1 : 0;
  p.zero_rest = zero_rest ? 1 : 0;
  if (pair_sum) {
    p.light = 0;  // (transposed tiles know no second part)
  }
  settle(&p, feat, ctas, dev->sm_count, dev->pair_ctas);
  if (with_push && ctas == 2) p.swap_rows = 0;  // (no such kernels)

  size_t need = 0;
  b200gmm_workspace_bytes(z, &need);
  if (workspace == nullptr || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) & 127))
    return B200GMM_EWORKSPACE;
  CUtensorMap* slots = reinterpret_cast<CUtensorMap*>(static_cast<char*>(workspace) + maps_offset(z));
  // The tile counter of the kernel's scheduler sits in the 16 bytes after the
  // batch_sizes copy and starts every launch at zero.
  uint32_t* sched_counter = reinterpret_cast<uint32_t*>(static_cast<char*>(workspace) + size_t(z) * sizeof(int64_t));
  const int max_ctas = grid_ctas(ctas, dev->sm_count, dev->pair_ctas);
  const bool single_wave = p.single_wave != 0;

  // A capturing stream keeps the copy of host batch_sizes (a replay reads them again)
  // and full dependencies between its kernels.
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) return B200GMM_ECUDA;
  const bool capturing = capture != cudaStreamCaptureStatusNone;
  if (!single_wave && (capturing ? cudaMemsetAsync(sched_counter, 0, 16, stream) : zero_counter(sched_counter, stream)) != cudaSuccess) {
    (void)cudaGetLastError();
    return B200GMM_ECUDA;
  }
  LaunchArgs la;
  la.overlap = !capturing;
  const int64_t* bs_dev = batch_sizes;
  if (!batch_sizes_on_device && z <= kInlineExperts && !capturing && pageable(batch_sizes)) {
    for (int e = 0; e < z; ++e)
      la.inline_sizes.v[e] = static_cast<int32_t>(std::max<int64_t>(-1, std::min<int64_t>(batch_sizes[e], tokens + 1)));
    bs_dev = nullptr;
  } else if (!batch_sizes_on_device) {
    if (cudaMemcpyAsync(workspace, batch_sizes, size_t(z) * sizeof(int64_t), cudaMemcpyHostToDevice,
                        stream) != cudaSuccess)
      return B200GMM_ECUDA;
    bs_dev = static_cast<const int64_t*>(workspace);
  }

  CUtensorMap map_a, map_b, map_b2, map_a2;
  bool have_b2 = (b2 != nullptr);
  // N: columns of b (and of b2, and of c); the Problem's n is twice that for the gated product.
  const uint64_t T = uint64_t(tokens), D1 = uint64_t(dim_a1), N = uint64_t(n_out), Z = uint64_t(z);
  const bool gather = (a_rows != nullptr);  // a is then fetched row by row, without a tensor map
  const bool swap_maps = p.swap_rows > 0 || p.light;
  if (p.mode == kNN) {
    const uint64_t da[2] = {D1, pair_sum ? 2 * T : T};
    const uint32_t ba[2] = {kBlockK, uint32_t(kBlockM)};
    const uint64_t db[3] = {N, D1, Z};
    const uint32_t bb[3] = {64, kBlockK, 1};
    // (One load per 64-column box: a single load of all the boxes of a stage through
    // a {64, k, n / 64, z} view of b measured 10-15 % slower in this layout.)
    if ((rc = encode_map(&map_b, b, 3, db, bb)) != 0) return rc;
    if (b2 != nullptr && (rc = encode_map(&map_b2, b2, 3, db, bb)) != 0) return rc;
    if (gather) map_a = map_b;
    else if ((rc = encode_map(&map_a, a, 2, da, ba)) != 0) return rc;
    if (swap_maps) {  // swapped and transposed tiles fetch their few rows of a in boxes of 32
      const uint32_t bl[2] = {kBlockK, 32};
      if ((rc = encode_map(&map_a2, a, 2, da, bl)) != 0) return rc;
    }
  } else if (p.mode == kNT) {
    const uint64_t da[2] = {D1, pair_sum ? 2 * T : T};
    const uint32_t ba[2] = {kBlockK, uint32_t(kBlockM)};
    const uint64_t db[3] = {D1, N, Z};
    // rows of b per box: a CTA's share of the tile; for the gated product half a tile from each of b, b2
    const uint32_t bb[3] = {kBlockK, uint32_t(swiglu ? kBlockN / 2 : kBlockN / ctas), 1};
    if ((rc = encode_map(&map_b, b, 3, db, bb)) != 0) return rc;
    if (b2 != nullptr && (rc = encode_map(&map_b2, b2, 3, db, bb)) != 0) return rc;
    if (gather) map_a = map_b;
    else if ((rc = encode_map(&map_a, a, 2, da, ba)) != 0) return rc;
    if (swap_maps) {
      const uint32_t bl[2] = {kBlockK, 32};
      if ((rc = encode_map(&map_a2, a, 2, da, bl)) != 0) return rc;
    }
    if (p.light) {  // transposed tiles: 128 rows of b[i] as the M operand
      const uint32_t bw[3] = {kBlockK, uint32_t(kLightCols), 1};
      if ((rc = encode_map(&map_b2, b, 3, db, bw)) != 0) return rc;
      have_b2 = true;
    }
  } else {
    const uint64_t da[2] = {D1, T};
    const uint64_t db[2] = {N, T};
    const uint32_t bx[2] = {64, kBlockK};
    // wgrad: both operands are staged as 64-column boxes; where the column count
    // allows, one load brings all boxes of a stage (half the TMA instructions).
    p.wide_b = (N % 64 == 0) ? 1 : 0;
    p.wide_a = (D1 % 64 == 0 && !gather) ? 1 : 0;
    if (p.wide_b) rc = encode_blocked(&map_b, b, N, T, 0, kBlockK, kBlockN / ctas / 64);
    else rc = encode_map(&map_b, b, 2, db, bx);
    if (rc != 0) return rc;
    if (gather) map_a = map_b;
    else if ((rc = p.wide_a ? encode_blocked(&map_a, a, D1, T, 0, kBlockK, kBlockM / 64)
                            : encode_map(&map_a, a, 2, da, bx)) != 0) return rc;
  }

  if (!have_b2) map_b2 = map_b;  // unused by the kernel, but a valid map
  if (!swap_maps) map_a2 = map_a;

  // Output map for the epilogue's TMA stores: 32 x 32 boxes, 64-byte swizzle; for
  // plain wgrad (c[z, m, n] is addressed as z*m rows) 64 x 32 boxes with 128-byte
  // swizzle.  Unused (left zeroed) when the rows are scattered through row_dest.
  CUtensorMap map_c = {};
  if (row_dest == nullptr) {
    const uint64_t dc[2] = {N, p.mode == kTN ? Z * D1 : (gate_grad != nullptr ? 2 * T : T)};
    const bool wide = p.mode == kTN && !gather && ctas == 1;  // Geometry::kWideOut
    const uint32_t bc[2] = {wide ? 64u : 32u, 32};
    if (dc[1] >= (uint64_t(1) << 31)) return B200GMM_ELIMIT;
    if ((rc = encode_map(&map_c, c, 2, dc, bc, wide ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B)) != 0)
      return rc;
  }

  // A launch that carries a row transfer keeps every CTA, however few its tiles: the
  // items are dealt over the grid.  (6 rows in 4 experts, k = 64, n = 72, beside 4000 rows of
  // 21504 bytes: 6466 us on the tiles' four CTAs, 196 us on all.)
  la.grid = single_wave && !with_push ? static_cast<int>(max_tiles(p)) * ctas : max_ctas;
  la.stream = stream;
  la.map_a = map_a;
  la.map_b = map_b;
  la.map_b2 = map_b2;
  la.map_c = map_c;
  la.map_a2 = map_a2;
  la.sched_counter = sched_counter;
  la.c = static_cast<__nv_bfloat16*>(c);
  la.batch_sizes = bs_dev;
  la.p = p;
  la.status = device_status;
  la.slots = slots;
  la.row_dest = row_dest;
  la.row_scale = row_scale;
  la.reduce_add = reduce_add;
  la.gate_grad = static_cast<const __nv_bfloat16*>(gate_grad);
  if (dest_base != nullptr) {
    la.dest_lo = static_cast<int64_t>(reinterpret_cast<uintptr_t>(dest_base));
    la.dest_hi = la.dest_lo + dest_bytes;
    if (la.dest_hi == 0) la.dest_hi = 1;  // an empty window at address 0 still rejects every row
  }
  if (gather) {
    la.a_rows = a_rows;
    la.a_src = static_cast<const __nv_bfloat16*>(a);
    la.a_src_rows = a_source_rows;
  }
  if (with_push) {
    la.push = *push;
    la.push.via_tma = env_int("B200GMM_PUSH_TMA", 1) ? 1 : 0;  // bulk copies measured faster than the register path
    // Optional pacing: spread the transfer over a share (B200GMM_PUSH_SPREAD percent; default
    // 0, as fast as it goes, which measured best) of the time the product is expected to
    // take at 1 PFLOP/s.
    const int spread = env_int("B200GMM_PUSH_SPREAD", 0);
    const double product_ns = 2.0 * double(tokens) * double(dim_a1) * double(n) / 1.0e6;
    const int64_t warps = int64_t(la.grid) * kPushWarps;
    const int64_t items_per_warp = (push->n_items + warps - 1) / warps;
    la.push.interval_ns = (spread > 0 && items_per_warp > 0)
                              ? static_cast<int64_t>(product_ns * (spread > 100 ? 100 : spread) / 100.0 / double(items_per_warp))
                              : 0;
    // (the pacing is a wait like any other: all of it stays inside the wait limit)
    if (la.push.interval_ns * items_per_warp > p.wait_ns) la.push.interval_ns = p.wait_ns / items_per_warp;
  }
  if (prepared != nullptr) {
    *prepared = la;
    return B200GMM_OK;
  }
  const cudaError_t err = gather      ? launch_variant<true, false>(la, ctas)
                          : swiglu    ? launch_variant<false, true>(la, ctas)
                          : with_push ? launch_with_push(la, ctas)
                                      : launch_variant<false, false>(la, ctas);
  if (err != cudaSuccess) {
    (void)cudaGetLastError();
    return B200GMM_ECUDA;
  }
  if (with_push && push_launched != nullptr) *push_launched = true;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return B200GMM_OK;
}

int swiglu_backward(const void* a, const void* b_gate, const void* b_up, const void* grad_out,
                    void* grad_products, const int64_t* batch_sizes, int batch_sizes_on_device, int z,
                    int64_t tokens, int64_t dim_a1, int64_t n, int trans_b, void* workspace,
                    size_t workspace_bytes, uint32_t* device_status, void* cuda_stream, bool zero_rest) {
  if (grad_products == nullptr || (grad_out == nullptr && tokens > 0 && n > 0)) return B200GMM_EINVAL;
  if (b_up == nullptr && tokens > 0 && n > 0 && dim_a1 > 0 && z > 0) return B200GMM_EINVAL;
  if (dim_a1 == 0 || tokens == 0 || n == 0 || z == 0) {
    // g = u = 0 everywhere: dg = dh * 0 * silu'(0) = 0 and du = dh * silu(0) = 0
    if (tokens > 0 && n > 0 && z > 0 &&
        cudaMemsetAsync(grad_products, 0, size_t(2) * size_t(tokens) * size_t(n) * 2,
                        static_cast<cudaStream_t>(cuda_stream)) != cudaSuccess)
      return B200GMM_ECUDA;
    return check_args_only(z, tokens, dim_a1, n, trans_b);
  }
  return run_impl(a, b_gate, grad_products, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, 0, trans_b,
                  workspace, workspace_bytes, device_status, cuda_stream, nullptr, nullptr, 0, b_up, nullptr, 0, nullptr, 0,
                  grad_out, nullptr, nullptr, false, zero_rest);
}

}  // namespace

extern "C" {

int b200gmm_run(const void* a, const void* b, void* c, const int64_t* batch_sizes,
                int batch_sizes_on_device, int z, int64_t tokens, int64_t dim_a1, int64_t n,
                int trans_a, int trans_b, void* workspace, size_t workspace_bytes,
                uint32_t* device_status, void* cuda_stream) {
  return run_impl(a, b, c, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, trans_a, trans_b,
                  workspace, workspace_bytes, device_status, cuda_stream, nullptr);
}

int b200gmm_run_gradients(const void* a, const void* b, const void* grad, void* a_grad, void* b_grad,
                          const int64_t* batch_sizes, int batch_sizes_on_device, int z, int64_t tokens, int64_t dim_a1,
                          int64_t n, int trans_b, void* workspace, size_t workspace_bytes, uint32_t* device_status,
                          void* cuda_stream) {
  const void *lhs = trans_b ? grad : a, *rhs = trans_b ? a : grad;
  const int64_t lhs_cols = trans_b ? n : dim_a1, rhs_cols = trans_b ? dim_a1 : n;
  // One launch of one-CTA tiles where all tiles of both products fit the SMs at once and the input
  // gradient's are plain.  Side by side they take the time of the longer; two launches
  // of a few microseconds each cost the host about as much as all of their preparation.
  bool together = z > 0 && tokens > 0 && dim_a1 > 0 && n > 0 && env_int("B200GMM_CTAS", 1) == 1;
  DeviceInfo* dev = nullptr;
  Problem d, w;
  together = together && check_problem(z, tokens, n, dim_a1, 0, !trans_b, 1, &d) == B200GMM_OK &&
             check_problem(z, tokens, lhs_cols, rhs_cols, 1, 0, 1, &w) == B200GMM_OK && !d.light &&
             device_info(&dev) == B200GMM_OK && max_tiles(d) + max_tiles(w) <= std::min(dev->sm_count, kMaxCtas) &&
             swap_rows(d, Features(), 1, dev->sm_count) == 0;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (together && cudaStreamIsCapturing(static_cast<cudaStream_t>(cuda_stream), &capture) != cudaSuccess) return B200GMM_ECUDA;
  together = together && capture == cudaStreamCaptureStatusNone;  // (a captured product keeps its own full dependencies)
  LaunchArgs ld, lw;
  int rc = run_impl(grad, b, a_grad, batch_sizes, batch_sizes_on_device, z, tokens, n, dim_a1, 0, !trans_b, workspace,
                    workspace_bytes, device_status, cuda_stream, nullptr, nullptr, 0, nullptr, nullptr, 0, nullptr, 0, nullptr,
                    nullptr, nullptr, false, false, -1, together ? &ld : nullptr);
  if (rc != B200GMM_OK) return rc;
  rc = run_impl(lhs, rhs, b_grad, batch_sizes, batch_sizes_on_device, z, tokens, lhs_cols, rhs_cols, 1, 0, workspace,
                workspace_bytes, device_status, cuda_stream, nullptr, nullptr, 0, nullptr, nullptr, 0, nullptr, 0, nullptr,
                nullptr, nullptr, false, false, -1, together ? &lw : nullptr);
  if (rc != B200GMM_OK || !together) return rc;
  if ((trans_b ? launch_gradients<kNN>(ld, lw) : launch_gradients<kNT>(ld, lw)) != cudaSuccess) {
    (void)cudaGetLastError();
    return B200GMM_ECUDA;
  }
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return B200GMM_OK;
}

int b200gmm_run_scatter(const void* a, const void* b, const int64_t* row_dest, const void* dest_base,
                        int64_t dest_bytes, const int64_t* batch_sizes,
                        int batch_sizes_on_device, int z, int64_t tokens, int64_t dim_a1, int64_t n,
                        int trans_b, void* workspace, size_t workspace_bytes, uint32_t* device_status,
                        void* cuda_stream) {
  if (row_dest == nullptr) return B200GMM_EINVAL;
  return run_impl(a, b, nullptr, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, 0, trans_b,
                  workspace, workspace_bytes, device_status, cuda_stream, row_dest, nullptr, 0, nullptr, nullptr, 0,
                  dest_base, dest_bytes);
}

int b200gmm_run_scatter_push(const void* a, const void* b, const int64_t* row_dest, const void* dest_base,
                             int64_t dest_bytes, const int64_t* batch_sizes, int batch_sizes_on_device, int z,
                             int64_t tokens, int64_t dim_a1, int64_t n, int trans_b, const void* push_src,
                             int64_t push_row_bytes, int64_t push_items, const int32_t* push_src_row,
                             const int32_t* push_dst_rank, const int64_t* push_dst_row,
                             const void* const* push_peer_base, void* workspace, size_t workspace_bytes,
                             uint32_t* device_status, void* cuda_stream) {
  if (row_dest == nullptr) return B200GMM_EINVAL;
  if (push_row_bytes <= 0 || (push_row_bytes % 16) != 0 || push_items < 0) return B200GMM_EINVAL;
  if (push_items > 0) {
    if (push_src == nullptr || push_dst_rank == nullptr || push_dst_row == nullptr || push_peer_base == nullptr)
      return B200GMM_EINVAL;
    if (reinterpret_cast<uintptr_t>(push_src) & 15) return B200GMM_EALIGN;
  }
  PushArgs push = {};
  push.src = static_cast<const uint4*>(push_src);
  push.row_vecs = push_row_bytes / 16;
  push.n_items = push_items;
  push.src_row = push_src_row;
  push.dst_rank = push_dst_rank;
  push.dst_row = push_dst_row;
  push.peer_base = const_cast<void* const*>(push_peer_base);
  push.interval_ns = 0;
  push.via_tma = 0;
  bool pushed = false;
  const int rc = run_impl(a, b, nullptr, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, 0, trans_b,
                          workspace, workspace_bytes, device_status, cuda_stream, row_dest, nullptr, 0, nullptr,
                          nullptr, 0, dest_base, dest_bytes, nullptr, &push, &pushed);
  if (rc != B200GMM_OK || pushed || push_items == 0) return rc;
  // The product was empty and launched nothing: the rows still have to move.
  return b200gmm_push_rows(push_src, push_row_bytes, push_items, push_src_row, push_dst_rank, push_dst_row,
                           push_peer_base, 0, cuda_stream);
}

int b200gmm_run_combine(const void* a, const void* b, const int64_t* row_dest, const void* dest_base,
                        int64_t dest_bytes, const float* row_weight,
                        int accumulate, const int64_t* batch_sizes, int batch_sizes_on_device, int z,
                        int64_t tokens, int64_t dim_a1, int64_t n, int trans_b, void* workspace,
                        size_t workspace_bytes, uint32_t* device_status, void* cuda_stream) {
  if (row_dest == nullptr) return B200GMM_EINVAL;
  if (row_weight != nullptr && (reinterpret_cast<uintptr_t>(row_weight) & 3)) return B200GMM_EALIGN;
  // k == 0 would take the zero-fill shortcut of the shared body, which writes c;
  // a combine has no c, and adding zeros changes nothing.
  if (dim_a1 == 0) return accumulate ? B200GMM_OK : B200GMM_EINVAL;
  return run_impl(a, b, nullptr, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, 0, trans_b,
                  workspace, workspace_bytes, device_status, cuda_stream, row_dest, nullptr, 0, nullptr,
                  row_weight, accumulate ? 1 : 0, dest_base, dest_bytes);
}

int b200gmm_run_combine_rows(const void* a, const void* b, const int64_t* row_index, void* out, int64_t out_rows,
                             const float* row_weight, int accumulate, const int64_t* batch_sizes,
                             int batch_sizes_on_device, int z, int64_t tokens, int64_t dim_a1, int64_t n, int trans_b,
                             void* workspace, size_t workspace_bytes, uint32_t* device_status, void* cuda_stream) {
  if (row_index == nullptr || out_rows < 0 || (out == nullptr && out_rows > 0)) return B200GMM_EINVAL;
  if (row_weight != nullptr && (reinterpret_cast<uintptr_t>(row_weight) & 3)) return B200GMM_EALIGN;
  if (dim_a1 == 0) return accumulate ? B200GMM_OK : B200GMM_EINVAL;  // as b200gmm_run_combine
  return run_impl(a, b, nullptr, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, 0, trans_b,
                  workspace, workspace_bytes, device_status, cuda_stream, row_index, nullptr, 0, nullptr,
                  row_weight, accumulate ? 1 : 0, out, out_rows * n * 2, nullptr, nullptr, nullptr, false, false, out_rows);
}

int b200gmm_run_gather(const void* x, int64_t x_rows, const int32_t* row_index, const void* b, void* c,
                       const int64_t* row_dest, const void* dest_base, int64_t dest_bytes,
                       const int64_t* batch_sizes, int batch_sizes_on_device,
                       int z, int64_t tokens, int64_t dim_a1, int64_t n, int trans_b, void* workspace,
                       size_t workspace_bytes, uint32_t* device_status, void* cuda_stream) {
  if (row_index == nullptr || x_rows <= 0 || x_rows >= (int64_t(1) << 31)) return B200GMM_EINVAL;
  if (c == nullptr && row_dest == nullptr) return B200GMM_EINVAL;
  return run_impl(x, b, c, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, 0, trans_b, workspace,
                  workspace_bytes, device_status, cuda_stream, row_dest, row_index, x_rows, nullptr, nullptr, 0,
                  dest_base, dest_bytes);
}

int b200gmm_run_gather_wgrad(const void* x, int64_t x_rows, const int32_t* row_index, const void* grad, void* c,
                             const int64_t* batch_sizes, int batch_sizes_on_device, int z, int64_t tokens,
                             int64_t dim_x1, int64_t n, void* workspace, size_t workspace_bytes,
                             uint32_t* device_status, void* cuda_stream) {
  if (row_index == nullptr || x_rows <= 0 || x_rows >= (int64_t(1) << 31)) return B200GMM_EINVAL;
  return run_impl(x, grad, c, batch_sizes, batch_sizes_on_device, z, tokens, dim_x1, n, 1, 0, workspace,
                  workspace_bytes, device_status, cuda_stream, nullptr, row_index, x_rows);
}

int b200gmm_run_swiglu(const void* a, const void* b_gate, const void* b_up, void* c, const int64_t* row_dest,
                       const void* dest_base, int64_t dest_bytes, const int64_t* batch_sizes, int batch_sizes_on_device, int z, int64_t tokens,
                       int64_t dim_a1, int64_t n, int trans_b, void* workspace, size_t workspace_bytes,
                       uint32_t* device_status, void* cuda_stream) {
  if (c == nullptr && row_dest == nullptr) return B200GMM_EINVAL;
  if (b_up == nullptr && tokens > 0 && n > 0 && dim_a1 > 0 && z > 0) return B200GMM_EINVAL;
  if (b_up == nullptr || dim_a1 == 0)  // nothing to multiply: silu(0) * 0 = 0, the plain path's zeros
    return run_impl(a, b_gate, c, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, 0, trans_b, workspace,
                    workspace_bytes, device_status, cuda_stream, row_dest, nullptr, 0, nullptr, nullptr, 0, dest_base,
                    dest_bytes);
  return run_impl(a, b_gate, c, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, 0, trans_b, workspace,
                  workspace_bytes, device_status, cuda_stream, row_dest, nullptr, 0, b_up, nullptr, 0, dest_base,
                  dest_bytes);
}

int b200gmm_run_swiglu_backward(const void* a, const void* b_gate, const void* b_up, const void* grad_out,
                                void* grad_products, const int64_t* batch_sizes, int batch_sizes_on_device, int z,
                                int64_t tokens, int64_t dim_a1, int64_t n, int trans_b, void* workspace,
                                size_t workspace_bytes, uint32_t* device_status, void* cuda_stream) {
  return swiglu_backward(a, b_gate, b_up, grad_out, grad_products, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1,
                         n, trans_b, workspace, workspace_bytes, device_status, cuda_stream, false);
}

int b200gmm_run_swiglu_backward_full(const void* a, const void* b_gate, const void* b_up, const void* grad_out,
                                     void* grad_products, const int64_t* batch_sizes, int batch_sizes_on_device, int z,
                                     int64_t tokens, int64_t dim_a1, int64_t n, int trans_b, void* workspace,
                                     size_t workspace_bytes, uint32_t* device_status, void* cuda_stream) {
  return swiglu_backward(a, b_gate, b_up, grad_out, grad_products, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1,
                         n, trans_b, workspace, workspace_bytes, device_status, cuda_stream, true);
}

int b200gmm_run_pair_sum(const void* a_pair, const void* b0, const void* b1, void* c, const int64_t* batch_sizes,
                         int batch_sizes_on_device, int z, int64_t tokens, int64_t dim_a1, int64_t n, int trans_b,
                         void* workspace, size_t workspace_bytes, uint32_t* device_status, void* cuda_stream) {
  if (b1 == nullptr && tokens > 0 && n > 0 && dim_a1 > 0 && z > 0) return B200GMM_EINVAL;
  return run_impl(a_pair, b0, c, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, 0, trans_b, workspace,
                  workspace_bytes, device_status, cuda_stream, nullptr, nullptr, 0, b1, nullptr, 0, nullptr, 0, nullptr,
                  nullptr, nullptr, true);
}

int b200gmm_run_static(const void* a, const void* b, void* c, const int64_t* batch_sizes,
                       int batch_sizes_on_device, int z, int64_t tokens, int64_t dim_a1, int64_t n,
                       int trans_a, int trans_b, uint32_t* device_status, void* cuda_stream) {
  if (z > B200GMM_STATIC_MAX_EXPERTS) return B200GMM_ELIMIT;
  void* scratch = nullptr;
  const int rc = static_scratch_address(&scratch);
  if (rc != B200GMM_OK) return rc;
  return b200gmm_run(a, b, c, batch_sizes, batch_sizes_on_device, z, tokens, dim_a1, n, trans_a,
                     trans_b, scratch, kStaticScratchBytes, device_status, cuda_stream);
}

int b200gmm_push_rows(const void* src, int64_t row_bytes, int64_t n_items, const int32_t* src_row,
                      const int32_t* dst_rank, const int64_t* dst_row, const void* const* peer_base,
                      int max_ctas, void* cuda_stream) {
  if (row_bytes <= 0 || (row_bytes % 16) != 0 || n_items < 0) return B200GMM_EINVAL;
  if (n_items == 0) return B200GMM_OK;
  if (src == nullptr || dst_rank == nullptr || dst_row == nullptr || peer_base == nullptr)
    return B200GMM_EINVAL;
  if (reinterpret_cast<uintptr_t>(src) & 15) return B200GMM_EALIGN;
  DeviceInfo* dev = nullptr;
  const int rc = device_info(&dev);
  if (rc != B200GMM_OK) return rc;
  // Rows are handed out grid-stride to 4 CTAs per SM: enough loads in flight to
  // fill NVLink and HBM.  max_ctas > 0 caps the grid for a transfer that should
  // leave memory bandwidth to other work.
  int64_t grid = int64_t(dev->sm_count) * 4;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  if (grid > n_items) grid = n_items;
  push_rows_kernel<<<static_cast<unsigned>(grid), kPushThreads, 0, static_cast<cudaStream_t>(cuda_stream)>>>(
      static_cast<const uint4*>(src), row_bytes / 16, n_items, src_row, dst_rank, dst_row,
      const_cast<void* const*>(peer_base));
  if (cudaGetLastError() != cudaSuccess) return B200GMM_ECUDA;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return B200GMM_OK;
}

int b200gmm_sum_slots(const void* slots, void* out, int64_t tokens, int top_k, int64_t cols, void* cuda_stream) {
  if (tokens < 0 || cols < 0 || top_k < 1 || top_k > kSumMaxTopK || (cols % 8) != 0) return B200GMM_EINVAL;
  if (tokens == 0 || cols == 0) return B200GMM_OK;
  if (slots == nullptr || out == nullptr) return B200GMM_EINVAL;
  if ((reinterpret_cast<uintptr_t>(slots) | reinterpret_cast<uintptr_t>(out)) & 15) return B200GMM_EALIGN;
  DeviceInfo* dev = nullptr;
  const int rc = device_info(&dev);
  if (rc != B200GMM_OK) return rc;
  const int64_t total = tokens * (cols / 8);
  int64_t grid = (total + kSumThreads - 1) / kSumThreads;
  const int64_t cap = int64_t(dev->sm_count) * 16;
  if (grid > cap) grid = cap;
  sum_slots_kernel<<<static_cast<unsigned>(grid), kSumThreads, 0, static_cast<cudaStream_t>(cuda_stream)>>>(
      static_cast<const uint4*>(slots), static_cast<uint4*>(out), tokens, top_k, cols / 8);
  if (cudaGetLastError() != cudaSuccess) return B200GMM_ECUDA;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return B200GMM_OK;
}

int b200gmm_fill_offsets(const int64_t* batch_sizes_device, int z, int64_t dim_a1, int64_t n,
                         int trans_a, int trans_b, int64_t* out_device, void* cuda_stream) {
  if (trans_a && trans_b) return B200GMM_EINVAL;
  if (z < 0 || dim_a1 < 0 || n < 0) return B200GMM_EINVAL;
  if (z > kMaxExperts) return B200GMM_ELIMIT;
  if (z == 0) return B200GMM_OK;
  if (batch_sizes_device == nullptr || out_device == nullptr) return B200GMM_EINVAL;
  Problem p = {};
  p.mode = trans_a ? kTN : (trans_b ? kNT : kNN);
  p.z = z;
  p.d1 = dim_a1;
  p.n = n;
  p.tile_m = kBlockM;
  p.tile_n = kBlockN;
  p.group_m = 1;
  derive(&p);
  fill_offsets_kernel<<<1, 32, 0, static_cast<cudaStream_t>(cuda_stream)>>>(batch_sizes_device, p,
                                                                            out_device);
  if (cudaGetLastError() != cudaSuccess) return B200GMM_ECUDA;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return B200GMM_OK;
}

int b200gmm_schedule_host(const int64_t* batch_sizes_host, int z, int64_t tokens, int64_t dim_a1,
                          int64_t n, int trans_a, int trans_b, int cluster_ctas, int64_t* out,
                          int64_t max_tiles, int64_t* n_tiles) {
  Problem p;
  if (cluster_ctas == 0) cluster_ctas = choose_ctas(z, tokens, dim_a1, n, trans_a, trans_b);
  const int rc = check_problem(z, tokens, dim_a1, n, trans_a, trans_b, cluster_ctas, &p);
  if (rc != B200GMM_OK) return rc;
  if (n_tiles == nullptr || (z > 0 && batch_sizes_host == nullptr)) return B200GMM_EINVAL;
  const HostSchedule h(p, batch_sizes_host);
  Tile tile;
  int64_t count = 0;  // accumulators: a wide tile is two
  int expert_pos = 0;
  const TileOrder order = h.order(p, 0);
  for (int t = 0; t < order.total; ++t) {
    h.decode(p, order, t, &expert_pos, &tile);
    for (int unit = 0; unit < tile.units; ++unit, ++count) {
      if (out == nullptr || count >= max_tiles) continue;
      int64_t* o = out + count * B200GMM_SCHEDULE_FIELDS;
      o[0] = tile.expert;
      o[1] = tile.row0;
      o[2] = tile.col0 + unit * kBlockN;
      o[3] = tile.valid_rows;
      o[4] = tile_stages(tile);
      o[5] = tile.kind;
    }
  }
  *n_tiles = count;
  return B200GMM_OK;
}

int b200gmm_launch_forms(const int64_t* batch_sizes_host, int z, int64_t tokens, int64_t dim_a1, int64_t n, int trans_a,
                         int trans_b, int features, int sm_count, int pair_ctas, int64_t* forms, int64_t* positions,
                         int64_t max_positions) {
  if (forms == nullptr || sm_count <= 0 || pair_ctas < 0 || (features & ~0xf) != 0) return B200GMM_EINVAL;
  for (int i = 0; i < B200GMM_FORM_FIELDS; ++i) forms[i] = 0;
  Features f;
  f.gather = (features & B200GMM_FORM_GATHER) != 0;
  f.gated_backward = (features & B200GMM_FORM_GATED_BACKWARD) != 0;
  f.swiglu = f.gated_backward || (features & B200GMM_FORM_GATED) != 0;
  f.scatter = (features & B200GMM_FORM_SCATTER) != 0;
  if (n < 0 || (f.swiglu && (trans_a || f.gather)) || (f.scatter && trans_a)) return B200GMM_EINVAL;
  if (f.swiglu) n *= 2;
  DeviceInfo dev;
  dev.sm_count = sm_count;
  dev.pair_ctas = pair_ctas;
  int ctas = choose_ctas(z, tokens, dim_a1, n, trans_a, trans_b, f, &dev);
  if (pair_ctas < 2) ctas = 1;
  Problem p;
  const int rc = check_problem(z, tokens, dim_a1, n, trans_a, trans_b, ctas, &p, f);
  if (rc != B200GMM_OK) return rc;
  if (z > 0 && batch_sizes_host == nullptr) return B200GMM_EINVAL;
  forms[0] = ctas;
  if (z == 0 || tokens == 0 || dim_a1 == 0 || n == 0) return B200GMM_OK;
  settle(&p, f, ctas, sm_count, pair_ctas);
  const HostSchedule h(p, batch_sizes_host);
  const int clusters = ctas == 2 ? grid_ctas(2, sm_count, pair_ctas) / 2 : 0;
  const TileOrder order = h.order(p, clusters);
  Tile tile;
  int expert_pos = 0;
  for (int i = 0; i < order.total; ++i) {
    h.decode(p, order, i, &expert_pos, &tile);
    if (positions != nullptr && i < max_positions) {
      int64_t* o = positions + int64_t(i) * B200GMM_POSITION_FIELDS;
      o[0] = tile.expert;
      o[1] = tile.row0;
      o[2] = tile.col0;
      o[3] = tile.valid_rows;
      o[4] = tile.units;
    }
    ++forms[tile.units == 2 ? 1 : tile.units == 1 ? 2 : 3];
    if (tile.units > 0 && p.mode != kTN && swapped_rows(p, tile) != 0) ++forms[4];
  }
  forms[5] = ctas == 2 && order.grid.tile_n == kBlockN ? 1 : 0;
  forms[6] = p.single_wave;
  return B200GMM_OK;
}

int b200gmm_schedule_device(const int64_t* batch_sizes_device, int z, int64_t tokens, int64_t dim_a1,
                            int64_t n, int trans_a, int trans_b, int cluster_ctas, int32_t* out_device,
                            int64_t max_tiles, int32_t* n_tiles_device, uint32_t* device_status,
                            void* cuda_stream) {
  Problem p;
  if (cluster_ctas == 0) cluster_ctas = choose_ctas(z, tokens, dim_a1, n, trans_a, trans_b);
  const int rc = check_problem(z, tokens, dim_a1, n, trans_a, trans_b, cluster_ctas, &p);
  if (rc != B200GMM_OK) return rc;
  if (n_tiles_device == nullptr || (z > 0 && batch_sizes_device == nullptr) || max_tiles < 0 ||
      max_tiles >= (int64_t(1) << 31) || (max_tiles > 0 && out_device == nullptr))
    return B200GMM_EINVAL;
  schedule_dump_kernel<<<1, kThreads, 0, static_cast<cudaStream_t>(cuda_stream)>>>(
      batch_sizes_device, p, out_device, static_cast<int>(max_tiles), n_tiles_device, device_status);
  if (cudaGetLastError() != cudaSuccess) return B200GMM_ECUDA;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return B200GMM_OK;
}

int b200gmm_selftest_wait_timeout(int64_t limit_ns, uint32_t* device_status, void* cuda_stream) {
  // A limit beyond a tenth of a second would only hold the GPU for nothing.
  if (limit_ns <= 0 || limit_ns > 100000000 || device_status == nullptr) return B200GMM_EINVAL;
  wait_timeout_kernel<<<1, 32, 0, static_cast<cudaStream_t>(cuda_stream)>>>(static_cast<uint64_t>(limit_ns),
                                                                           device_status);
  if (cudaGetLastError() != cudaSuccess) return B200GMM_ECUDA;
  g_launches.fetch_add(1, std::memory_order_relaxed);
  return B200GMM_OK;
}

int b200gmm_tile_shape(int cluster_ctas, int* out3) {
  if (out3 == nullptr || (cluster_ctas != 1 && cluster_ctas != 2)) return B200GMM_EINVAL;
  out3[0] = kBlockM * cluster_ctas;
  out3[1] = kBlockN;
  out3[2] = kBlockK;
  return B200GMM_OK;
}

int64_t b200gmm_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

const char* b200gmm_strerror(int code) {
  switch (code) {
    case B200GMM_OK: return "ok";
    case B200GMM_EINVAL: return "invalid argument (null pointer, negative size, or trans_a and trans_b both set)";
    case B200GMM_EALIGN: return "row lengths must be multiples of 8 bf16 elements and pointers 16-byte aligned";
    case B200GMM_ELIMIT: return "too many experts (max 1024), too many tiles, or a dimension >= 2^31";
    case B200GMM_EWORKSPACE: return "workspace missing, smaller than b200gmm_workspace_bytes(z), or not 128-byte aligned";
    case B200GMM_ECUDA: return "a CUDA runtime or driver call failed";
    case B200GMM_ETENSORMAP: return "cuTensorMapEncodeTiled rejected a tensor (address, stride or extent)";
    case B200GMM_EDEVICE: return "current device is not compute capability 10.x (B200, sm_100a)";
    case B200GMM_ETIMEOUT: return "a bounded wait inside the kernel gave up (device status word)";
    default: return "unknown b200gmm error code";
  }
}

}  // extern "C"
