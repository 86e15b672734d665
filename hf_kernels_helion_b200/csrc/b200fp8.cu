// C ABI of the block-FP8 hot path (declarations and contracts: include/b200fp8.h).
// Host side only validates, builds TMA descriptors and launches; nothing here
// allocates, frees or synchronises.
#include "../../include/b200fp8.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstring>
#include <mutex>

#include "gemm_streamk.cuh"
#include "gemm_tile.cuh"
#include "quant.cuh"

namespace {

using namespace b200fp8;

constexpr int kMaxDevices = 64;

// What the choice of a form depends on besides the shape.
struct Limits {
  int sm_count = 0;
  int pair_clusters = 0;   // CTA pairs of the pair kernels that can be resident at once
  int clusters[kClusterMax + 1] = {};   // clusters of c CTAs of gemm_cluster_kernel that can be resident at once
};

struct DeviceInfo : Limits {
  std::atomic<int> ready{0};
  int cc_major = 0;
};
DeviceInfo g_dev[kMaxDevices];
std::mutex g_mutex;

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
std::atomic<EncodeTiledFn> g_encode{nullptr};

// Per-device facts, read once; also opts every kernel into its dynamic shared memory size.
int device_info(const DeviceInfo** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return B200FP8_ERR_ARCH;
  DeviceInfo& d = g_dev[dev];
  if (!d.ready.load(std::memory_order_acquire)) {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!d.ready.load(std::memory_order_relaxed)) {
      if (cudaDeviceGetAttribute(&d.cc_major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
          cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return B200FP8_ERR_ARCH;
      if (d.cc_major != 10) return B200FP8_ERR_ARCH;
      bool ok = true;
      auto opt_in = [&ok](const void* fn, int bytes) {
        ok = ok && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
      };
      // setmaxnreg.inc blocks until registers are free: refuse to run a kernel whose compiled
      // register count (what the launch allocates) cannot cover its own re-balancing plan
      auto regs_ok = [&ok](const void* fn, int threads, int regs_needed_total) {
        cudaFuncAttributes attr;
        ok = ok && cudaFuncGetAttributes(&attr, fn) == cudaSuccess && attr.numRegs * threads >= regs_needed_total;
      };
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_kernel<256, 0>), TileCfg<256>::THREADS,
              128 * TileCfg<256>::REGS_CONTROL + 256 * TileCfg<256>::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_multi_kernel<256>), TileCfg<256>::THREADS,
              128 * TileCfg<256>::REGS_CONTROL + 256 * TileCfg<256>::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_streamk_kernel<256>), StreamKCfg<256>::THREADS,
              128 * StreamKCfg<256>::REGS_CONTROL + 256 * StreamKCfg<256>::REGS_EPILOGUE);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_kernel<128, 0>), TileCfg<128, false>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_kernel<256, 0>), TileCfg<256, false>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_cluster_kernel), TileCfg<128, false>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_cluster_rowb_kernel), TileCfg<128, false, 128, 0, true>::SMEM_BYTES);
      regs_ok(reinterpret_cast<const void*>(&gemm_cluster_rowb_kernel), TileCfg<128>::THREADS,
              128 * TileCfg<128>::REGS_CONTROL + 256 * TileCfg<128>::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_cluster_kernel), TileCfg<128>::THREADS,
              128 * TileCfg<128>::REGS_CONTROL + 256 * TileCfg<128>::REGS_EPILOGUE);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_multi_kernel<128>), TileCfg<128, true>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_multi_kernel<256>), TileCfg<256, true>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_rowb_kernel<128>), TileCfg<128, false, 128, 0, true>::SMEM_BYTES);
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_rowb_kernel<128>), TileCfg<128>::THREADS,
              128 * TileCfg<128>::REGS_CONTROL + 256 * TileCfg<128>::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_kernel<128, 0>), TileCfg<128>::THREADS,
              128 * TileCfg<128>::REGS_CONTROL + 256 * TileCfg<128>::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_multi_kernel<128>), TileCfg<128>::THREADS,
              128 * TileCfg<128>::REGS_CONTROL + 256 * TileCfg<128>::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_mc_kernel<128>), TileCfg<128>::THREADS,
              128 * TileCfg<128>::REGS_CONTROL + 256 * TileCfg<128>::REGS_EPILOGUE);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_mc_kernel<128>), TileCfg<128, true>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_mc_kernel<256>), TileCfg<256, true>::SMEM_BYTES);
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_mc_kernel<256>), TileCfg<256>::THREADS,
              128 * TileCfg<256>::REGS_CONTROL + 256 * TileCfg<256>::REGS_EPILOGUE);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_decode_kernel<256, 16>), TileCfg<256, false, 16>::SMEM_BYTES);
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_decode_kernel<256, 16>), TileCfg<256>::THREADS,
              128 * TileCfg<256>::REGS_CONTROL + 256 * TileCfg<256>::REGS_EPILOGUE);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_decode_kernel<256, 64>), TileCfg<256, false, 64>::SMEM_BYTES);
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_decode_kernel<256, 64>), TileCfg<256>::THREADS,
              128 * TileCfg<256>::REGS_CONTROL + 256 * TileCfg<256>::REGS_EPILOGUE);
      opt_in(reinterpret_cast<const void*>(&gemm_tile_kernel<256, 1>), TileCfg<256, false>::SMEM_BYTES);
      regs_ok(reinterpret_cast<const void*>(&gemm_tile_kernel<256, 1>), TileCfg<256>::THREADS,
              128 * TileCfg<256>::REGS_CONTROL + 256 * TileCfg<256>::REGS_EPILOGUE);
      using PairCfg = TileCfg<256, false, 128, 1>;
      using PairMultiCfg = TileCfg<256, true, 128, 1>;
      using PairRowbCfg = TileCfg<256, true, 128, 2, true>;
      opt_in(reinterpret_cast<const void*>(&gemm_pair_rowb_kernel<0>), PairRowbCfg::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_pair_rowb_kernel<1>), PairRowbCfg::SMEM_BYTES);
      regs_ok(reinterpret_cast<const void*>(&gemm_pair_rowb_kernel<0>), PairRowbCfg::THREADS,
              128 * PairRowbCfg::REGS_CONTROL + 256 * PairRowbCfg::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_pair_rowb_kernel<1>), PairRowbCfg::THREADS,
              128 * PairRowbCfg::REGS_CONTROL + 256 * PairRowbCfg::REGS_EPILOGUE);
      opt_in(reinterpret_cast<const void*>(&gemm_pair_kernel<false>), PairCfg::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_pair_kernel<true>), PairCfg::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_pair_multi_kernel<false>), PairMultiCfg::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_pair_multi_kernel<true>), PairMultiCfg::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_pair_multi_sk_kernel), PairMultiCfg::SMEM_BYTES);
      regs_ok(reinterpret_cast<const void*>(&gemm_pair_kernel<false>), PairCfg::THREADS,
              128 * PairCfg::REGS_CONTROL + 256 * PairCfg::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_pair_kernel<true>), PairCfg::THREADS,
              128 * PairCfg::REGS_CONTROL + 256 * PairCfg::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_pair_multi_kernel<false>), PairCfg::THREADS,
              128 * PairCfg::REGS_CONTROL + 256 * PairCfg::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_pair_multi_kernel<true>), PairCfg::THREADS,
              128 * PairCfg::REGS_CONTROL + 256 * PairCfg::REGS_EPILOGUE);
      regs_ok(reinterpret_cast<const void*>(&gemm_pair_multi_sk_kernel), PairCfg::THREADS,
              128 * PairCfg::REGS_CONTROL + 256 * PairCfg::REGS_EPILOGUE);
      if (ok) {
        // how many CTA pairs fit on the device at once (one CTA per SM; not every SM need be pairable)
        cudaLaunchAttribute cattr[1];
        cattr[0].id = cudaLaunchAttributeClusterDimension;
        cattr[0].val.clusterDim.x = 2;
        cattr[0].val.clusterDim.y = 1;
        cattr[0].val.clusterDim.z = 1;
        cudaLaunchConfig_t ccfg = {};
        ccfg.gridDim = dim3(static_cast<unsigned>(d.sm_count & ~1));
        ccfg.blockDim = dim3(PairCfg::THREADS);
        ccfg.dynamicSmemBytes = PairMultiCfg::SMEM_BYTES;
        ccfg.attrs = cattr;
        ccfg.numAttrs = 1;
        int n_clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&n_clusters, gemm_pair_multi_kernel<true>, &ccfg) != cudaSuccess) {
          cudaGetLastError();
          n_clusters = 0;
        }
        d.pair_clusters = n_clusters < d.sm_count / 2 ? n_clusters : d.sm_count / 2;
        ccfg.blockDim = dim3(TileCfg<128>::THREADS);
        ccfg.dynamicSmemBytes = TileCfg<128, false>::SMEM_BYTES;
        for (int c = 2; c <= kClusterMax; ++c) {
          cattr[0].val.clusterDim.x = static_cast<unsigned>(c);
          ccfg.gridDim = dim3(static_cast<unsigned>(d.sm_count / c * c));
          if (cudaOccupancyMaxActiveClusters(&n_clusters, gemm_cluster_kernel, &ccfg) != cudaSuccess) {
            cudaGetLastError();
            n_clusters = 0;
          }
          d.clusters[c] = n_clusters < d.sm_count / c ? n_clusters : d.sm_count / c;
        }
      }
      opt_in(reinterpret_cast<const void*>(&gemm_streamk_kernel<16>), StreamKCfg<16>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_streamk_kernel<32>), StreamKCfg<32>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_streamk_kernel<64>), StreamKCfg<64>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_streamk_kernel<128>), StreamKCfg<128>::SMEM_BYTES);
      opt_in(reinterpret_cast<const void*>(&gemm_streamk_kernel<256>), StreamKCfg<256>::SMEM_BYTES);
      if (!ok) {
        cudaGetLastError();
        return B200FP8_ERR_LAUNCH;
      }
      d.ready.store(1, std::memory_order_release);
    }
  }
  *out = &d;
  return B200FP8_OK;
}

// For the queries: the current device's limits; without a device those of a B200, 148 SMs and as many clusters as they
// hold, but no CTA pairs.
Limits limits_or_default() {
  const DeviceInfo* d = nullptr;
  if (device_info(&d) == B200FP8_OK) return *d;
  cudaGetLastError();
  Limits l;
  l.sm_count = 148;
  for (int c = 2; c <= kClusterMax; ++c) l.clusters[c] = l.sm_count / c;
  return l;
}

int sm_count_or_default() { return limits_or_default().sm_count; }

EncodeTiledFn encode_fn() {
  EncodeTiledFn fn = g_encode.load(std::memory_order_acquire);
  if (fn != nullptr) return fn;
  void* sym = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess || sym == nullptr) {
    cudaGetLastError();
    return nullptr;
  }
  fn = reinterpret_cast<EncodeTiledFn>(sym);
  g_encode.store(fn, std::memory_order_release);
  return fn;
}

// 2-D tensor map over a row-major byte matrix [rows, cols] with row stride ld (bytes),
// box = [box_rows x 128 bytes], 128-byte swizzle, zero fill outside the matrix.
// A tensor map is a pure function of (base, rows, cols, ld, box_rows): the last few are kept per
// host thread (no lock, no shared mutable state) so that a caller that repeats a shape - a decode
// loop, a captured graph being re-recorded - does not pay the driver's encoder on every call.
struct TmapKey {
  const void* base;
  int64_t rows, cols, ld;
  uint32_t box_rows;
  int kind;   // 0: byte matrix, 128-byte boxes, SWIZZLE_128B; 1, 2: fp32 matrix, 128- or 256-element boxes, no swizzle
  bool operator==(const TmapKey& o) const {
    return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld && box_rows == o.box_rows && kind == o.kind;
  }
};
constexpr int kTmapCacheEntries = 16;
struct TmapCache {
  TmapKey key[kTmapCacheEntries];
  CUtensorMap map[kTmapCacheEntries];
  int used = 0, next = 0;
};
thread_local TmapCache t_tmap_cache;

// kind 0: byte matrix [rows, cols], ld in bytes; kind 1 / 2: fp32 matrix [rows, cols], ld in bytes, box = [box_rows x
// 128 / 256 floats]
int make_tmap(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t ld, uint32_t box_rows, int kind) {
  const TmapKey k = {base, rows, cols, ld, box_rows, kind};
  TmapCache& c = t_tmap_cache;
  for (int i = 0; i < c.used; ++i)
    if (c.key[i] == k) {
      *map = c.map[i];
      return B200FP8_OK;
    }
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return B200FP8_ERR_DRIVER;
  const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld)};
  const cuuint32_t box[2] = {kind == 2 ? 256u : 128u, box_rows};
  const cuuint32_t elem[2] = {1u, 1u};
  const CUresult r = fn(map, kind >= 1 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2,
                        const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        kind >= 1 ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return B200FP8_ERR_DRIVER;
  const int slot = c.used < kTmapCacheEntries ? c.used++ : c.next;
  c.next = (slot + 1) % kTmapCacheEntries;
  c.key[slot] = k;
  c.map[slot] = *map;
  return B200FP8_OK;
}

int make_tmap_u8(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t ld, uint32_t box_rows) {
  return make_tmap(map, base, rows, cols, ld, box_rows, 0);
}

// Launch with programmatic stream serialisation: the kernel may be put on the device while the one before it in the
// stream drains, and waits for it (pdl_wait) before it touches memory. Hides the launch latency between consecutive
// kernels of a stream: 4096 x 8192 activations 18.4 -> 15.7 us call after call, a row-scaled 512 x 512 x 2048 product, with
// two prep launches then, 20.5 -> 17.6. (The weight quantiser, one launch of many blocks, gained nothing.)
template <typename... P, typename... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, cudaStream_t stream, A... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);   // (a refusal is what launch_status reports)
}

int launch_status() { return cudaGetLastError() == cudaSuccess ? B200FP8_OK : B200FP8_ERR_LAUNCH; }

// Scratch of b200fp8_gemm_decode_static: lives in the module image of every device that
// loads the library, from load until process exit. In host code the NAME of a __device__
// array is only a host-side stand-in, not a device address; the address a kernel may use
// comes from cudaGetSymbolAddress, taken once per device with that device current.
constexpr size_t kStaticScratchBytes = B200FP8_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];
std::atomic<void*> g_static_scratch_addr[kMaxDevices];

int static_scratch_address(void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return B200FP8_ERR_ARCH;
  void* p = g_static_scratch_addr[dev].load(std::memory_order_acquire);
  if (p == nullptr) {
    if (cudaGetSymbolAddress(&p, g_static_scratch) != cudaSuccess || p == nullptr) {
      cudaGetLastError();
      return B200FP8_ERR_DRIVER;
    }
    g_static_scratch_addr[dev].store(p, std::memory_order_release);
  }
  *out = p;
  return B200FP8_OK;
}

int streamk_mp(int64_t M) {
  if (M <= 16) return 16;
  if (M <= 32) return 32;
  if (M <= 64) return 64;
  if (M <= 128) return 128;
  return 256;
}

int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

struct StreamKPlan {
  int mp;
  int num_kb;
  int64_t num_tiles;
  int64_t grid;
  int64_t ast_bytes;      // AsT region (first)
  int64_t partial_bytes;  // partial-sum region (second)
};

StreamKPlan streamk_plan(int64_t M, int64_t N, int64_t K, int sm_count) {
  StreamKPlan p;
  p.mp = streamk_mp(M);
  p.num_kb = static_cast<int>((K + 127) / 128);
  p.num_tiles = (N + 127) / 128;
  const int64_t total = p.num_tiles * p.num_kb;
  p.grid = total < sm_count ? total : sm_count;
  if (p.grid < 1) p.grid = 1;
  p.ast_bytes = align_up(static_cast<int64_t>(p.num_kb) * p.mp * 4, 256);
  p.partial_bytes = 2 * p.grid * p.mp * 128 * 4;
  return p;
}

// tile variants: AsT [ceil(K/128)][M rounded up to 128] fp32
int64_t tile_ast_bytes(int64_t M, int64_t K) { return align_up(((K + 127) / 128) * align_up(M, 128) * 4, 256); }
// + a 16-row copy of A (zero-padded) when M <= 16
int64_t tile_workspace_bytes(int64_t M, int64_t K) {
  if (M == 0 || K == 0) return 0;
  return tile_ast_bytes(M, K) + (M <= 16 ? 16 * align_up(K, 16) : 0);
}

// b200fp8_linear: scales K-block-major + the quantised activations (at least 16 rows, 16-byte row pitch)
int64_t linear_prefix_bytes(int64_t M, int64_t K) {
  if (M == 0 || K == 0) return 0;
  return tile_ast_bytes(M, K) + align_up((M < 16 ? 16 : M) * align_up(K, 16), 256);
}

// row-scaled B: the K-block-major copy of the B scales
int64_t bst_bytes(int64_t N, int64_t K) { return align_up(((K + 127) / 128) * align_up(N, 128) * 4, 256); }

// 128x256 tiles with the last, partly empty wave split along K (B200FP8_VARIANT_TILE256_SK)
struct TileSkPlan {
  int num_m, num_n, num_kb;
  int full;      // tiles handed out whole, round-robin
  int tail;      // remaining tiles (< grid)
  int split;     // K ranges per tail tile; < 2 means the shape gains nothing and runs as plain tiles
  int kb_per;    // K blocks per range
  int64_t grid;
  int64_t ast_bytes, partial_bytes;
};

TileSkPlan tile_sk_plan(int64_t M, int64_t N, int64_t K, int sm_count) {
  TileSkPlan p;
  p.num_m = static_cast<int>((M + 127) / 128);
  p.num_n = static_cast<int>((N + 255) / 256);
  p.num_kb = static_cast<int>((K + 127) / 128);
  const int64_t tiles = static_cast<int64_t>(p.num_m) * p.num_n;
  p.grid = sm_count;
  p.full = static_cast<int>((tiles / sm_count) * sm_count);
  p.tail = static_cast<int>(tiles - p.full);
  p.split = p.tail > 0 ? sm_count / p.tail : 1;
  if (p.split > p.num_kb / 4) p.split = p.num_kb / 4;   // keep ranges of at least 4 K blocks
  if (p.split < 1) p.split = 1;
  p.kb_per = (p.num_kb + p.split - 1) / p.split;
  p.ast_bytes = tile_workspace_bytes(M, K);
  p.partial_bytes = p.split >= 2 ? static_cast<int64_t>(p.tail) * p.split * 128 * 256 * 4 : 0;
  return p;
}

// The same for 256 x 256 tiles on CTA pairs (B200FP8_VARIANT_PAIR256_SPLIT_SK): the workers are the pairs,
// and every K range leaves two partial tiles (one per CTA of the pair).
TileSkPlan pair_sk_plan(int64_t M, int64_t N, int64_t K, int pairs) {
  TileSkPlan p;
  p.num_m = static_cast<int>((M + 255) / 256);
  p.num_n = static_cast<int>((N + 255) / 256);
  p.num_kb = static_cast<int>((K + 127) / 128);
  const int64_t tiles = static_cast<int64_t>(p.num_m) * p.num_n;
  if (pairs < 1) pairs = 1;
  p.grid = 2 * static_cast<int64_t>(pairs);
  p.full = static_cast<int>((tiles / pairs) * pairs);
  p.tail = static_cast<int>(tiles - p.full);
  p.split = p.tail > 0 ? pairs / p.tail : 1;
  if (p.split > p.num_kb / 4) p.split = p.num_kb / 4;   // keep ranges of at least 4 K blocks
  if (p.split < 1) p.split = 1;
  p.kb_per = (p.num_kb + p.split - 1) / p.split;
  p.ast_bytes = tile_workspace_bytes(M, K);
  p.partial_bytes = p.split >= 2 ? static_cast<int64_t>(p.tail) * p.split * 2 * 128 * 256 * 4 : 0;
  return p;
}

// AUTO's estimate of each form's time in us, fitted to graph replays of 46 shapes with 129..8192 rows, 512..28672 columns
// and 1024..8192 deep (single launches on B200): a start-up, then per wave of tiles the K blocks at the form's rate
// and the end of a tile (register stores in the split single-CTA form, staged ones otherwise), and 6 us for the
// fix-up pass of a split last wave. Over 46 other sizes of the same ranges (graph replays, two operand sets) its choice and the
// cluster form's take 1.0 % more than the fastest of the five in the mean; the worst wrong choice is 209 x 544 x 1408 (128 x
// 128 tiles 11.1 us, 128 x 256 10.1). For instance, measured
// 128 x 128 / 128 x 256 / its split tail / pairs / their split tail: 1611 x 7000 x 4208 79.5 / 69.9 / 70.8 / 57.7 / 57.5,
// 2545 x 1920 x 6272 64.1 / 54.0 / 44.3 / 53.4 / 42.7, 317 x 24832 x 2432 41.9 / 27.6 / 28.2 / 36.5 / 36.5,
// 1394 x 1536 x 1152 10.7 / 11.1 / 14.8 / 11.1 / 16.0, 4096 x 4096 x 8192 184.3 / 149.3 / 143.2 / 151.6 / 135.0.
struct Pick {
  int variant;
  double us;
};

double split_waves_us(const TileSkPlan& p, int workers, double per_kb, double per_tile) {
  return (p.full / workers) * (per_kb * p.num_kb + per_tile) + per_kb * p.kb_per + per_tile + 6.0;
}

Pick pick_form(int64_t M, int64_t N, int64_t K, int sm_count, int pairs) {
  const bool pair_ok = pairs > 0;
  const double kb = static_cast<double>((K + 127) / 128);
  const int64_t num_m = (M + 127) / 128;
  auto waves = [](int64_t tiles, int64_t workers) { return static_cast<double>((tiles + workers - 1) / workers); };
  // Decode shapes (M <= 256) are weight-streaming and HBM-bound. Measured on B200 at N = 28672,
  // K = 8192: the plain 128x256 tile kernel (46 us at M = 16, 5.1 TB/s with 112 of 148 SMs busy)
  // beats the swap-AB stream-K kernel (65 us), so AUTO does not pick that one.
  // (two row blocks, M in 129..256, go to the CTA pairs below when the device runs them: 79.5 vs 84-86 us at M = 256)
  // One row block: 128-wide tiles as long as each has an SM to itself - more SMs pull on the weight, and four accumulator
  // stages instead of two are in flight (29 x 13952 x 1680 9.2 vs 11.9 us, 50 x 1024 x 464 4.8 vs 6.9, 1 x 8704 x 544 5.2 vs
  // 6.2) - and 256-wide ones beyond (3 x 21376 x 7808, 167 narrow tiles: 58.0 vs 32.6).
  if (M <= 128) {
    const int64_t narrow = (N + 127) / 128;
    if (narrow <= sm_count) return {B200FP8_VARIANT_TILE128, 4.5 + 0.30 * kb};
    return {B200FP8_VARIANT_TILE256, 6.0 + 0.43 * kb * waves((N + 255) / 256, sm_count)};
  }
  if (M <= 256 && (N <= 128 || !pair_ok))
    return {N > 128 ? B200FP8_VARIANT_TILE256 : B200FP8_VARIANT_TILE128, 6.0 + 0.43 * kb};
  // (128 x 128 tiles: 0.31 us per K block on a few SMs, 0.385 when all of them load operands from L2)
  const int64_t tiles = num_m * ((N + 127) / 128);
  const double share = 0.385 * static_cast<double>(tiles < sm_count ? tiles : sm_count) / sm_count;
  Pick best = {B200FP8_VARIANT_TILE128, 5.5 + waves(tiles, sm_count) * ((share > 0.31 ? share : 0.31) * kb + 0.5)};
  auto consider = [&best](int variant, double us) {
    if (us < best.us) best = {variant, us};
  };
  const TileSkPlan t = tile_sk_plan(M, N, K, sm_count);
  consider(B200FP8_VARIANT_TILE256, 5.0 + waves(static_cast<int64_t>(t.num_m) * t.num_n, sm_count) * (0.52 * kb + 1.3));
  if (t.split >= 2) consider(B200FP8_VARIANT_TILE256_SK, 5.0 + split_waves_us(t, sm_count, 0.54, 2.5));
  if (pair_ok) {
    const TileSkPlan p = pair_sk_plan(M, N, K, pairs);
    consider(B200FP8_VARIANT_PAIR256_SPLIT, 5.3 + waves(static_cast<int64_t>(p.num_m) * p.num_n, pairs) * (0.50 * kb + 1.3));
    if (p.split >= 2) consider(B200FP8_VARIANT_PAIR256_SPLIT_SK, 5.3 + split_waves_us(p, pairs, 0.50, 1.3));
  }
  return best;
}

// CTAs per tile (2..8) for products whose 128 x 128 tiles leave SMs idle: the K blocks of a tile are cut over a cluster
// (gemm_cluster_kernel), as far as all clusters are resident at once. 1: another form is estimated to be faster.
// Cutting costs 1-2 us (two cluster barriers and the addition through distributed shared memory), so that products of
// fewer than 12 K blocks stay whole. Measured, one / two / four CTAs per tile, us: 4 x 2560 x 2048 12.9 / 9.0 / 8.1,
// 64 x 2048 x 4096 20.1 / 12.3 / 9.4, 512 x 512 x 2048 11.4 / 11.3 / 9.2, 512 x 512 x 8192 28.9 / 19.5 / 13.3,
// 1 x 8192 x 8192 34.0 / 17.6 / - (more clusters than fit: 22.3).
// With row-scaled B a K block takes longer and cutting pays more: 512 x 512 x 2048 16.0 -> 11.5 us, 38 x 1024 x 4096 21.7 -> 9.6,
// 2 x 512 x 8192 39.2 -> 12.0, 256 x 2048 x 4096 (split tail of pair tiles before) 19.9 -> 14.5.
int cluster_split(int64_t M, int64_t N, int64_t K, const int* clusters, double other_us, bool rowb) {
  const int64_t tiles = ((M + 127) / 128) * ((N + 127) / 128);
  const int64_t kblocks = (K + 127) / 128;
  int best = 1;
  if (kblocks < 12) return best;
  for (int c = 2; c <= kClusterMax; ++c) {
    if (tiles > clusters[c] || kblocks < 2 * c) continue;
    const double kb = static_cast<double>((kblocks + c - 1) / c);
    const double us = rowb ? 10.0 + 0.56 * kb : (M <= 128 ? 5.3 : 7.5) + 0.33 * kb;
    if (us < other_us) {
      other_us = us;
      best = c;
    }
  }
  return best;
}

// Row-scaled B: 128 x 128 tiles, or 256 x 256 tiles on CTA pairs (with the last wave split along K where that can be
// done), whichever a straight-line fit to measured times says is faster. Per wave and K block a 128 x 128 tile takes
// 0.56 us and a pair tile, four times the area on two SMs, 0.87; both start with about 8 us of launches and
// prologue, the fix-up pass of the split tail takes 5. Measured, 128 x 128 / pair / pair with split tail, us:
// 4096 x 4096 x 8192 268.6 / 241.8 / 221.8, 2048 x 2048 x 4096 46.8 / 36.9 / 36.8, 256 x 4096 x 4096 25.2 / 35.1 / 20.5,
// 512 x 2048 x 2048 16.7 / 22.0 / 17.6, 8192 x 4096 x 7168 469.8 / 386.4 / 395.5.
Pick pick_rowb(int64_t M, int64_t N, int64_t K, int sm_count, int pairs) {
  const int64_t tiles = ((M + 127) / 128) * ((N + 127) / 128);
  const double kb = static_cast<double>((K + 127) / 128);
  const double t128 = 0.56 * kb * static_cast<double>((tiles + sm_count - 1) / sm_count);
  if (pairs < 1 || M <= 128) return {B200FP8_VARIANT_TILE128, 8.0 + t128};
  const TileSkPlan p = pair_sk_plan(M, N, K, pairs);
  const double full = 0.87 * kb * static_cast<double>(p.full / pairs);
  const double t_pair = full + (p.tail > 0 ? 0.87 * kb : 0.0);
  const double t_sk = p.split >= 2 ? full + 0.87 * p.kb_per + 5.0 : t_pair;
  if (t128 <= t_pair && t128 <= t_sk) return {B200FP8_VARIANT_TILE128, 8.0 + t128};
  if (t_sk < t_pair) return {B200FP8_VARIANT_PAIR256_SPLIT_SK, 8.0 + t_sk};
  return {B200FP8_VARIANT_PAIR256_SPLIT, 8.0 + t_pair};
}

int64_t partial_bytes(int variant, int64_t M, int64_t N, int64_t K, const Limits& lim) {
  if (variant == B200FP8_VARIANT_TILE256_SK) return tile_sk_plan(M, N, K, lim.sm_count).partial_bytes;
  if (variant == B200FP8_VARIANT_PAIR256_SPLIT_SK) return pair_sk_plan(M, N, K, lim.pair_clusters).partial_bytes;
  return 0;
}

int without_split_tail(int variant) {
  if (variant == B200FP8_VARIANT_TILE256_SK) return B200FP8_VARIANT_TILE256;
  if (variant == B200FP8_VARIANT_PAIR256_SPLIT_SK) return B200FP8_VARIANT_PAIR256_SPLIT;
  return variant;
}

double wave_efficiency(int64_t tiles, int sms) {
  return static_cast<double>(tiles) / static_cast<double>((tiles + sms - 1) / sms * sms);
}

// Several destinations (the N-sharded exchange), or one multicast address (no pairs). The estimates above are of single
// destinations, whose last wave may be split and whose stores stay on the device: they do not say what an exchange takes,
// which is bound by the links, so this rule is the one that exchanges over NVLink were measured with. 256-wide tiles move 25 %
// fewer operand bytes per flop and are taken unless their last wave is much emptier, on CTA pairs beyond 128 rows: the
// pair kernel's smaller pipeline stages leave room for a second set of output staging buffers, which keeps the links busy
// through the next tile's K loop (2 GPUs, 8192 x 18432 x 7168: 0.596 ms, 0.608 for the pair form with whole K blocks; 4 GPUs
// 0.538 against 0.540 for single CTAs).
int pick_several(int64_t M, int64_t N, int sm_count, int pairs) {
  if (M <= 128 || (M <= 256 && (N <= 128 || pairs < 1))) return N > 128 ? B200FP8_VARIANT_TILE256 : B200FP8_VARIANT_TILE128;
  const int64_t num_m = (M + 127) / 128;
  const double e128 = wave_efficiency(num_m * ((N + 127) / 128), sm_count);
  const double e256 = wave_efficiency(num_m * ((N + 255) / 256), sm_count);
  if (e256 * 1.15 < e128) return B200FP8_VARIANT_TILE128;
  return pairs > 0 ? B200FP8_VARIANT_PAIR256_SPLIT : B200FP8_VARIANT_TILE256;
}

// The form AUTO runs, decided here for the launches and for every query: a variant, and with
// B200FP8_VARIANT_TILE128 the CTAs that share a tile. call: B200FP8_CALL_*; staged: the rows of every destination are
// multiples of 16 bytes (only then do the pair forms pay, which stage their output).
struct Form {
  int variant;
  int cluster;
};

Form auto_form(int64_t M, int64_t N, int64_t K, int call, bool staged, const Limits& lim) {
  if (call == B200FP8_CALL_SEVERAL || call == B200FP8_CALL_MULTICAST)
    return {pick_several(M, N, lim.sm_count, call == B200FP8_CALL_SEVERAL ? lim.pair_clusters : 0), 1};
  const bool rowb = call == B200FP8_CALL_ROWSCALE;
  const int pairs = staged ? lim.pair_clusters : 0;
  const Pick p = rowb ? pick_rowb(M, N, K, lim.sm_count, pairs) : pick_form(M, N, K, lim.sm_count, pairs);
  const int cluster = cluster_split(M, N, K, lim.clusters, p.us, rowb);
  return {cluster > 1 ? B200FP8_VARIANT_TILE128 : p.variant, cluster};
}

// The partial tiles of whatever AUTO may run for this shape, with a destination that can be staged and with one that can't.
int64_t auto_partial_bytes(int64_t M, int64_t N, int64_t K, int call, const Limits& lim) {
  const int64_t a = partial_bytes(auto_form(M, N, K, call, true, lim).variant, M, N, K, lim);
  const int64_t b = partial_bytes(auto_form(M, N, K, call, false, lim).variant, M, N, K, lim);
  return a > b ? a : b;
}

// Whether the GEMM kernel reads the token scales (and, with up to 16 rows, A) where they are instead of copies that a
// prep launch lays out for it: one launch less, 1.0-1.5 us a call, 3 us with up to 16 rows. Rows of As whose length and
// address let a group of K blocks (two for 128-wide tiles, four otherwise) be loaded at once always do (4096 x 4096 x
// 8192 133.3 -> 130.6 us, 256 x 28672 x 8192 79.0 -> 76.7, 37 x 28672 x 8192 43.4 -> 42.3, 4 x 2560 x 2048 8.2 -> 6.3);
// one load of 32 sectors per K block keeps that gain up to about 64 K blocks per SM (345 x 1664 x 7808 17.0 -> 16.0,
// 918 x 9216 x 6272, 95 of them, 58.5 -> 59.4).
bool direct_scales(int variant, int64_t M, int64_t N, int64_t K, const float* As, int64_t ld_as, int sm_count) {
  const int64_t bn = variant == B200FP8_VARIANT_TILE128 ? 128 : 256;
  const int64_t group = bn == 128 ? 2 : 4;
  if (ld_as % group == 0 && reinterpret_cast<uintptr_t>(As) % (group * 4) == 0) return true;
  return ((M + 127) / 128) * ((N + bn - 1) / bn) * ((K + 127) / 128) <= 64 * static_cast<int64_t>(sm_count);
}

template <int BN>
int launch_tile(const void* A, const void* B, GemmArgs args, int64_t lda, int64_t ldb, int sm_count,
                cudaStream_t stream, int64_t sk_grid = 0, int cluster = 1) {
  CUtensorMap ta, tb;
  // Weight-streaming shapes: kernel forms with 16- or 64-row A slots and six or five pipeline stages
  // (measured 3-4 % faster than the 128-row form at N = 28672, K = 8192: 44.5-46 us at M <= 17).
  // A copy of A that the prep kernel makes for M <= 16 has 16 rows. Without a prep launch the box is over the caller's
  // own rows: a load 4 % slower than from the 16-row copy, and the launch saved is worth more (direct_scales).
  const bool decode = BN == 256 && args.M <= 64 && args.sk_split < 2 && args.n_dst == 1 && !args.mc_store &&
                      args.BsT == nullptr;
  const uint32_t a_rows = !decode ? 128u : args.M <= 16 ? 16u : 64u;
  // (no copy of A: a box of the rows that exist; the slot's other rows keep what they held and give accumulator rows
  // that are never stored)
  const uint32_t box_rows = args.direct && args.M < static_cast<int64_t>(a_rows) ? static_cast<uint32_t>(args.M) : a_rows;
  args.a_box_bytes = static_cast<int>(box_rows) * 128;
  int st = make_tmap_u8(&ta, A, (args.a_from_prep && args.M < 16) ? 16 : args.M, args.K, lda, box_rows);
  if (st != B200FP8_OK) return st;
  st = make_tmap_u8(&tb, B, args.N, args.K, ldb, BN);
  if (st != B200FP8_OK) return st;
  const int64_t tiles = ((args.M + 127) / 128) * ((args.N + BN - 1) / BN);
  const int grid = sk_grid > 0 ? static_cast<int>(sk_grid) : static_cast<int>(tiles < sm_count ? tiles : sm_count);
  // Programmatic dependent launch: the kernel may begin (barrier set-up, TMEM allocation, and behind a prep
  // launch of the same call also operand loads) while the kernel enqueued just before it is still running.
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(TileCfg<BN, false>::THREADS);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t err;
  if (BN == 128 && cluster > 1 && args.BsT == nullptr) {
    cfg.gridDim = dim3(static_cast<unsigned>(tiles * cluster));
    cfg.numAttrs = 2;
    cfg.dynamicSmemBytes = TileCfg<128, false>::SMEM_BYTES;
    err = cudaLaunchKernelEx(&cfg, gemm_cluster_kernel, ta, tb, args);
  } else if (decode && a_rows == 16u) {
    cfg.dynamicSmemBytes = TileCfg<256, false, 16>::SMEM_BYTES;
    err = cudaLaunchKernelEx(&cfg, gemm_tile_decode_kernel<256, 16>, ta, tb, args);
  } else if (decode) {
    cfg.dynamicSmemBytes = TileCfg<256, false, 64>::SMEM_BYTES;
    err = cudaLaunchKernelEx(&cfg, gemm_tile_decode_kernel<256, 64>, ta, tb, args);
  } else if (BN == 256 && args.sk_split >= 2) {
    cfg.dynamicSmemBytes = TileCfg<256, false>::SMEM_BYTES;
    err = cudaLaunchKernelEx(&cfg, gemm_tile_kernel<256, 1>, ta, tb, args);
  } else if (BN == 128 && args.BsT != nullptr) {
    // the K-block-major copy of the row scales as an fp32 matrix [K blocks, n_pad]: one box = the
    // table of one tile (used when it fits the shared-memory table)
    CUtensorMap tbst;
    const int64_t kblocks = (args.K + 127) / 128;
    st = make_tmap(&tbst, args.BsT, kblocks, args.n_pad, args.n_pad * 4,
                   static_cast<uint32_t>(kblocks < kRowbTableKb ? kblocks : kRowbTableKb), 1);
    if (st != B200FP8_OK) return st;
    cfg.dynamicSmemBytes = TileCfg<128, false, 128, 0, true>::SMEM_BYTES;
    if (cluster > 1) {
      cfg.gridDim = dim3(static_cast<unsigned>(tiles * cluster));
      cfg.numAttrs = 2;
      err = cudaLaunchKernelEx(&cfg, gemm_cluster_rowb_kernel, ta, tb, tbst, args);
    } else {
      err = cudaLaunchKernelEx(&cfg, gemm_tile_rowb_kernel<128>, ta, tb, tbst, args);
    }
  } else if (args.mc_store) {
    cfg.dynamicSmemBytes = TileCfg<BN, true>::SMEM_BYTES;
    err = cudaLaunchKernelEx(&cfg, gemm_tile_mc_kernel<BN>, ta, tb, args);
  } else if (args.n_dst > 1 || (BN == 256 && args.staged_store)) {
    // Several destinations, and the 256-wide tile with one: the output leaves through shared memory
    // and TMA stores instead of 16-byte stores of row pieces from registers (32 sectors per warp
    // instruction), which shortens the stretch at the end of a tile in which nothing drains TMEM.
    // One byte-matrix tensor map per destination: [M rows, N * element size], 32 x 128-byte boxes
    DstMaps dm;
    const int64_t esize = args.out_fp32 ? 4 : 2;
    for (int d = 0; d < 8; ++d) {
      const int src = d < args.n_dst ? d : 0;
      st = make_tmap_u8(&dm.m[d], args.dst[src], args.M, args.N * esize, args.dst_ld[src] * esize, 32);
      if (st != B200FP8_OK) return st;
    }
    cfg.dynamicSmemBytes = TileCfg<BN, true>::SMEM_BYTES;
    err = cudaLaunchKernelEx(&cfg, gemm_tile_multi_kernel<BN>, ta, tb, args, dm);
  } else {
    cfg.dynamicSmemBytes = TileCfg<BN, false>::SMEM_BYTES;
    err = cudaLaunchKernelEx(&cfg, gemm_tile_kernel<BN, 0>, ta, tb, args);
  }
  if (err != cudaSuccess) {
    cudaGetLastError();
    return B200FP8_ERR_LAUNCH;
  }
  return launch_status();
}

// CTA-pair kernels: 256 x 256 tiles, one cluster of two CTAs per tile, persistent over the pairs that
// fit on the device. The B map's box is this CTA's share of the B rows of one MMA.
template <bool SPLIT>
int launch_pair(const void* A, const void* B, const GemmArgs& args, int64_t lda, int64_t ldb, int pair_clusters,
                cudaStream_t stream) {
  if (pair_clusters < 1) return B200FP8_ERR_LAUNCH;
  CUtensorMap ta, tb;
  int st = make_tmap_u8(&ta, A, args.M, args.K, lda, 128);
  if (st != B200FP8_OK) return st;
  st = make_tmap_u8(&tb, B, args.N, args.K, ldb, SPLIT ? 64 : 128);
  if (st != B200FP8_OK) return st;
  const int64_t tiles = ((args.M + 255) / 256) * ((args.N + 255) / 256);
  // (the split-K plan counts on every pair the device can hold)
  const int pairs = args.sk_split >= 2 ? pair_clusters : static_cast<int>(tiles < pair_clusters ? tiles : pair_clusters);
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 2;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs));
  cfg.blockDim = dim3(TileCfg<256, false>::THREADS);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaError_t err;
  if (args.n_dst > 1 || args.staged_store) {
    DstMaps dm;
    const int64_t esize = args.out_fp32 ? 4 : 2;
    for (int d = 0; d < 8; ++d) {
      const int src = d < args.n_dst ? d : 0;
      st = make_tmap_u8(&dm.m[d], args.dst[src], args.M, args.N * esize, args.dst_ld[src] * esize, 32);
      if (st != B200FP8_OK) return st;
    }
    cfg.dynamicSmemBytes = TileCfg<256, true, 128, 1>::SMEM_BYTES;
    if (args.BsT != nullptr) {
      CUtensorMap tbst;
      st = make_tmap(&tbst, args.BsT, (args.K + 127) / 128, args.n_pad, args.n_pad * 4, kRowbChunkKb, 2);
      if (st != B200FP8_OK) return st;
      cfg.dynamicSmemBytes = TileCfg<256, true, 128, 2, true>::SMEM_BYTES;
      err = args.sk_split >= 2 ? cudaLaunchKernelEx(&cfg, gemm_pair_rowb_kernel<1>, ta, tb, tbst, args, dm)
                               : cudaLaunchKernelEx(&cfg, gemm_pair_rowb_kernel<0>, ta, tb, tbst, args, dm);
    } else if (args.sk_split >= 2) err = cudaLaunchKernelEx(&cfg, gemm_pair_multi_sk_kernel, ta, tb, args, dm);   // (SPLIT form only)
    else err = cudaLaunchKernelEx(&cfg, gemm_pair_multi_kernel<SPLIT>, ta, tb, args, dm);
  } else {
    cfg.dynamicSmemBytes = TileCfg<256, false, 128, 1>::SMEM_BYTES;
    err = cudaLaunchKernelEx(&cfg, gemm_pair_kernel<SPLIT>, ta, tb, args);
  }
  if (err != cudaSuccess) {
    cudaGetLastError();
    return B200FP8_ERR_LAUNCH;
  }
  return launch_status();
}

template <int MP>
int launch_streamk(const void* A, const void* B, const StreamKArgs& args, int64_t lda, int64_t ldb, int64_t grid,
                   cudaStream_t stream) {
  CUtensorMap tw, tx;
  int st = make_tmap_u8(&tw, B, args.N, args.K, ldb, 128);
  if (st != B200FP8_OK) return st;
  st = make_tmap_u8(&tx, A, args.M, args.K, lda, MP);
  if (st != B200FP8_OK) return st;
  gemm_streamk_kernel<MP><<<static_cast<int>(grid), StreamKCfg<MP>::THREADS, StreamKCfg<MP>::SMEM_BYTES, stream>>>(
      tw, tx, args);
  return launch_status();
}

}  // namespace

extern "C" {

int b200fp8_version(void) { return 100; }

const char* b200fp8_strerror(int status) {
  switch (status) {
    case B200FP8_OK: return "ok";
    case B200FP8_ERR_NULL: return "a required pointer is NULL";
    case B200FP8_ERR_SHAPE: return "bad shape or leading dimension";
    case B200FP8_ERR_ALIGN: return "pointer or leading dimension violates a 16-byte alignment rule";
    case B200FP8_ERR_DTYPE: return "unknown output dtype";
    case B200FP8_ERR_VARIANT: return "unknown kernel variant, or variant cannot run this shape";
    case B200FP8_ERR_WORKSPACE: return "workspace missing or too small";
    case B200FP8_ERR_ARCH: return "current CUDA device is not compute capability 10.x (B200)";
    case B200FP8_ERR_DRIVER: return "cuTensorMapEncodeTiled unavailable or rejected the tensor";
    case B200FP8_ERR_LAUNCH: return "CUDA runtime refused the kernel launch";
    case B200FP8_ERR_TOO_LARGE: return "request exceeds a fixed capacity of this entry point";
    default: return "unknown status";
  }
}

int b200fp8_quant_act(const void* x, void* q, float* s, int64_t M, int64_t K, int64_t ldx, int64_t ldq, int64_t lds,
                      void* stream) {
  if (M < 0 || K < 0) return B200FP8_ERR_SHAPE;
  if (M == 0 || K == 0) return B200FP8_OK;
  if (x == nullptr || q == nullptr || s == nullptr) return B200FP8_ERR_NULL;
  if (ldx < K || ldq < K || lds < (K + 127) / 128) return B200FP8_ERR_SHAPE;
  if (K % 8 != 0 || ldx % 8 != 0 || ldq % 8 != 0 || (reinterpret_cast<uintptr_t>(x) & 15u) != 0 ||
      (reinterpret_cast<uintptr_t>(q) & 7u) != 0)
    return B200FP8_ERR_ALIGN;
  const DeviceInfo* dev = nullptr;
  int st = device_info(&dev);
  if (st != B200FP8_OK) return st;
  const int64_t groups = M * ((K + 127) / 128);
  if (K % 128 == 0 && (M == 1 || (ldx == K && ldq == K && lds == K / 128)) &&
      (reinterpret_cast<uintptr_t>(q) & 15u) == 0 && groups <= (int64_t{1} << 35)) {
    // one unbroken run of 128-element groups: no row / column arithmetic in the kernel
    const unsigned blocks = static_cast<unsigned>((groups + 63) / 64);
    if ((reinterpret_cast<uintptr_t>(x) & 31u) == 0)
      launch_pdl(quant_act_contig_kernel<true>, dim3(blocks), static_cast<cudaStream_t>(stream),
                 static_cast<const uint4*>(x), static_cast<uint4*>(q), s, groups);
    else
      launch_pdl(quant_act_contig_kernel<false>, dim3(blocks), static_cast<cudaStream_t>(stream),
                 static_cast<const uint4*>(x), static_cast<uint4*>(q), s, groups);
    return launch_status();
  }
  const int64_t blocks_needed = (groups * 8 + 255) / 256;
  const int64_t max_blocks = static_cast<int64_t>(dev->sm_count) * 32;
  const int grid = static_cast<int>(blocks_needed < max_blocks ? blocks_needed : max_blocks);
  // (the last pass of the loop steps at most one grid beyond the padded count)
  if (groups + 4 + static_cast<int64_t>(grid) * 32 <= 0xFFFFFFFFll)
    launch_pdl(quant_act_kernel<uint32_t>, dim3(grid), static_cast<cudaStream_t>(stream),
               static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q), s, M, K, ldx, ldq, lds);
  else
    launch_pdl(quant_act_kernel<int64_t>, dim3(grid), static_cast<cudaStream_t>(stream),
               static_cast<const __nv_bfloat16*>(x), static_cast<uint8_t*>(q), s, M, K, ldx, ldq, lds);
  return launch_status();
}

int b200fp8_quant_weight(const void* w, void* q, float* s, int64_t N, int64_t K, int64_t ldw, int64_t ldq, int64_t lds,
                         void* stream) {
  if (N < 0 || K < 0) return B200FP8_ERR_SHAPE;
  if (N == 0 || K == 0) return B200FP8_OK;
  if (w == nullptr || q == nullptr || s == nullptr) return B200FP8_ERR_NULL;
  if (ldw < K || ldq < K || lds < (K + 127) / 128) return B200FP8_ERR_SHAPE;
  if (K % 8 != 0 || ldw % 8 != 0 || ldq % 8 != 0 || (reinterpret_cast<uintptr_t>(w) & 15u) != 0 ||
      (reinterpret_cast<uintptr_t>(q) & 7u) != 0)
    return B200FP8_ERR_ALIGN;
  const DeviceInfo* dev = nullptr;
  int st = device_info(&dev);
  if (st != B200FP8_OK) return st;
  const int64_t blocks = ((N + 127) / 128) * ((K + 127) / 128);
  if (blocks > 0x7FFFFFFF) return B200FP8_ERR_TOO_LARGE;
  const bool wide = K % 16 == 0 && ldw % 16 == 0 && ldq % 16 == 0 && (reinterpret_cast<uintptr_t>(w) & 31u) == 0 &&
                    (reinterpret_cast<uintptr_t>(q) & 15u) == 0;
  if (wide)
    quant_weight_kernel<true><<<static_cast<int>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(w), static_cast<uint8_t*>(q), s, N, K, ldw, ldq, lds);
  else
    quant_weight_kernel<false><<<static_cast<int>(blocks), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(w), static_cast<uint8_t*>(q), s, N, K, ldw, ldq, lds);
  return launch_status();
}

int64_t b200fp8_streamk_first_unit(int64_t cta, int64_t total, int64_t grid) {
  return streamk_first_unit(cta, total, grid);
}
int64_t b200fp8_streamk_owner(int64_t unit, int64_t total, int64_t grid) { return streamk_owner(unit, total, grid); }
int64_t b200fp8_streamk_grid(int64_t M, int64_t N, int64_t K) {
  return streamk_plan(M, N, K, sm_count_or_default()).grid;
}

int b200fp8_gemm_pair_clusters(void) { return limits_or_default().pair_clusters; }

int b200fp8_gemm_auto_form(int64_t M, int64_t N, int64_t K, int call, int* ctas_per_tile) {
  if (M < 1 || N < 1 || K < 1) return -B200FP8_ERR_SHAPE;
  if (call < B200FP8_CALL_ONE || call > B200FP8_CALL_MULTICAST) return -B200FP8_ERR_VARIANT;
  const Form f = auto_form(M, N, K, call, true, limits_or_default());
  if (ctas_per_tile != nullptr) *ctas_per_tile = f.cluster;
  return f.variant;
}

int b200fp8_gemm_pick_variant(int64_t M, int64_t N, int64_t K) {
  return auto_form(M, N, K, B200FP8_CALL_ONE, true, limits_or_default()).variant;
}

int64_t b200fp8_gemm_workspace_bytes(int64_t M, int64_t N, int64_t K, int variant) {
  if (M < 0 || N < 0 || K < 0) return -static_cast<int64_t>(B200FP8_ERR_SHAPE);
  const int sms = sm_count_or_default();
  if (M == 0 || N == 0 || K == 0) return (variant >= B200FP8_VARIANT_AUTO && variant <= B200FP8_VARIANT_PAIR256_SPLIT_SK) ? 0 : -static_cast<int64_t>(B200FP8_ERR_VARIANT);
  if (variant == B200FP8_VARIANT_AUTO)
    return tile_workspace_bytes(M, K) + auto_partial_bytes(M, N, K, B200FP8_CALL_ONE, limits_or_default());
  if (variant == B200FP8_VARIANT_TILE128 || variant == B200FP8_VARIANT_TILE256 ||
      variant == B200FP8_VARIANT_PAIR256 || variant == B200FP8_VARIANT_PAIR256_SPLIT)
    return tile_workspace_bytes(M, K);
  if (variant == B200FP8_VARIANT_TILE256_SK) {
    const TileSkPlan p = tile_sk_plan(M, N, K, sms);
    return p.ast_bytes + p.partial_bytes;
  }
  if (variant == B200FP8_VARIANT_PAIR256_SPLIT_SK) {
    const TileSkPlan p = pair_sk_plan(M, N, K, b200fp8_gemm_pair_clusters());
    return p.ast_bytes + p.partial_bytes;
  }
  if (variant != B200FP8_VARIANT_STREAMK) return -static_cast<int64_t>(B200FP8_ERR_VARIANT);
  if (M > 256) return -static_cast<int64_t>(B200FP8_ERR_VARIANT);
  if (M == 0 || N == 0 || K == 0) return 0;
  const StreamKPlan p = streamk_plan(M, N, K, sms);
  return p.ast_bytes + p.partial_bytes;
}

// Shared body of b200fp8_gemm (n_dst = 1), b200fp8_gemm_scatter (n_dst >= 1) and
// b200fp8_gemm_multicast (n_dst = 1, mc = true: dst[0] is a multimem address).
// x_bf16 != nullptr: the activations arrive unquantised (b200fp8_linear); A and As are then
// produced by tile_prep_quant_kernel in the workspace.
struct FusedQuant {
  const void* x_bf16 = nullptr;
  int64_t ldx = 0;
  // rowb: Bs is [N, ceil(K/128)], one scale per row of B (b200fp8_gemm_rowscale)
  bool rowb = false;
};

static int gemm_impl(bool mc, const void* A, const void* B, const float* As, const float* Bs, int n_dst, void* const* dst,
                     const int64_t* dst_ld, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldb, int64_t ld_as,
                     int64_t ld_bs, int out_dtype, int variant, void* workspace, size_t workspace_bytes,
                     uint32_t* status_word, void* stream_, FusedQuant fq = FusedQuant()) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const bool fused_q = fq.x_bf16 != nullptr;
  if (n_dst < 1 || n_dst > 8 || dst == nullptr || dst_ld == nullptr) return B200FP8_ERR_SHAPE;
  void* C = dst[0];
  const int64_t ldc = dst_ld[0];
  if (M < 0 || N < 0 || K < 0) return B200FP8_ERR_SHAPE;
  if (out_dtype != B200FP8_OUT_BF16 && out_dtype != B200FP8_OUT_FP32) return B200FP8_ERR_DTYPE;
  if (variant < B200FP8_VARIANT_AUTO || variant > B200FP8_VARIANT_PAIR256_SPLIT_SK) return B200FP8_ERR_VARIANT;
  if (M == 0 || N == 0) return B200FP8_OK;
  for (int d = 0; d < n_dst; ++d) {
    if (dst[d] == nullptr) return B200FP8_ERR_NULL;
    if (dst_ld[d] < N) return B200FP8_ERR_SHAPE;
  }

  const DeviceInfo* dev = nullptr;
  int st = device_info(&dev);
  if (st != B200FP8_OK) return st;

  // 16-byte vector stores through the staging path need aligned destinations
  const int64_t esize = out_dtype == B200FP8_OUT_FP32 ? 4 : 2;
  bool staged = (N * esize) % 16 == 0;
  for (int d = 0; d < n_dst; ++d)
    staged = staged && (reinterpret_cast<uintptr_t>(dst[d]) & 15u) == 0 && (dst_ld[d] * esize) % 16 == 0;
  if ((n_dst > 1 || mc) && !staged) return B200FP8_ERR_ALIGN;
  if (mc && n_dst != 1) return B200FP8_ERR_SHAPE;
  auto fill_dst = [&](GemmArgs& a) {
    a.n_dst = n_dst;
    a.staged_store = staged ? 1 : 0;
    a.mc_store = mc ? 1 : 0;
    for (int d = 0; d < 8; ++d) {
      a.dst[d] = d < n_dst ? dst[d] : nullptr;
      a.dst_ld[d] = d < n_dst ? dst_ld[d] : 0;
    }
  };

  if (K == 0) {
    if (n_dst > 1 || mc) return B200FP8_ERR_SHAPE;
    gemm_zero_fill_kernel<<<dev->sm_count, 256, 0, stream>>>(C, M, N, ldc, out_dtype == B200FP8_OUT_FP32);
    return launch_status();
  }
  const int64_t kblocks = (K + 127) / 128;
  if (fused_q) {
    if (B == nullptr || Bs == nullptr) return B200FP8_ERR_NULL;
    if (K % 128 != 0 || fq.ldx < K || ldb < K || ld_bs < kblocks) return B200FP8_ERR_SHAPE;
    if (fq.ldx % 8 != 0 || ldb % 16 != 0 || (reinterpret_cast<uintptr_t>(fq.x_bf16) & 15u) != 0 ||
        (reinterpret_cast<uintptr_t>(B) & 15u) != 0)
      return B200FP8_ERR_ALIGN;
  } else {
    if (A == nullptr || B == nullptr || As == nullptr || Bs == nullptr) return B200FP8_ERR_NULL;
    if (lda < K || ldb < K || ld_as < kblocks || ld_bs < kblocks) return B200FP8_ERR_SHAPE;
    if (lda % 16 != 0 || ldb % 16 != 0 || (reinterpret_cast<uintptr_t>(A) & 15u) != 0 ||
        (reinterpret_cast<uintptr_t>(B) & 15u) != 0)
      return B200FP8_ERR_ALIGN;
  }
  if (M > 0x7FFFFF00 || N > 0x7FFFFF00 || K > 0x7FFFFF00) return B200FP8_ERR_TOO_LARGE;

  const bool multi = n_dst > 1 || mc;
  if (fq.rowb && (multi || fused_q)) return B200FP8_ERR_VARIANT;
  // what every tile form needs of the workspace: the scale copy, the copy of A, and the copy of B's row scales
  const int64_t prefix = fused_q ? linear_prefix_bytes(M, K) : tile_workspace_bytes(M, K);
  const int64_t rowb_bytes = fq.rowb ? bst_bytes(N, K) : 0;
  int cluster = 1;
  if (variant == B200FP8_VARIANT_AUTO || fq.rowb) {
    const int call = fq.rowb ? B200FP8_CALL_ROWSCALE
                     : mc    ? B200FP8_CALL_MULTICAST
                             : n_dst > 1 ? B200FP8_CALL_SEVERAL : B200FP8_CALL_ONE;
    const Form f = auto_form(M, N, K, call, staged, *dev);
    variant = f.variant;
    cluster = f.cluster;
    // (a workspace without room for the partial tiles: the same tiles without the split tail)
    if (static_cast<int64_t>(workspace_bytes) < prefix + rowb_bytes + partial_bytes(variant, M, N, K, *dev))
      variant = without_split_tail(variant);
  }
  if (multi && variant == B200FP8_VARIANT_TILE256_SK) variant = B200FP8_VARIANT_TILE256;
  // the K ranges of the pair split-K form leave through the fix-up pass, which writes one destination,
  // and its whole tiles through the staging area
  if (variant == B200FP8_VARIANT_PAIR256_SPLIT_SK && (multi || !staged || dev->pair_clusters < 1))
    variant = B200FP8_VARIANT_PAIR256_SPLIT;
  const bool pair = variant == B200FP8_VARIANT_PAIR256 || variant == B200FP8_VARIANT_PAIR256_SPLIT ||
                    variant == B200FP8_VARIANT_PAIR256_SPLIT_SK;
  if (pair && mc) return B200FP8_ERR_VARIANT;
  if (multi && !pair && variant != B200FP8_VARIANT_TILE128 && variant != B200FP8_VARIANT_TILE256)
    return B200FP8_ERR_VARIANT;

  TileSkPlan skp = {};
  if (variant == B200FP8_VARIANT_TILE256_SK) {
    skp = tile_sk_plan(M, N, K, dev->sm_count);
    if (skp.split < 2) variant = B200FP8_VARIANT_TILE256;   // nothing to split: same as the plain tile kernel
  }
  if (variant == B200FP8_VARIANT_PAIR256_SPLIT_SK) {
    skp = pair_sk_plan(M, N, K, dev->pair_clusters);
    if (skp.split < 2) variant = B200FP8_VARIANT_PAIR256_SPLIT;
  }

  if (variant == B200FP8_VARIANT_TILE128 || variant == B200FP8_VARIANT_TILE256 ||
      variant == B200FP8_VARIANT_TILE256_SK || pair) {
    const bool pair_sk = variant == B200FP8_VARIANT_PAIR256_SPLIT_SK;
    const bool sk = variant == B200FP8_VARIANT_TILE256_SK || pair_sk;
    const int64_t need = prefix + (sk ? skp.partial_bytes : 0) + rowb_bytes;
    if (workspace == nullptr || static_cast<int64_t>(workspace_bytes) < need) return B200FP8_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0) return B200FP8_ERR_ALIGN;
    GemmArgs args;
    fill_dst(args);
    // the copy of A the prep kernel writes: the quantised activations (b200fp8_linear), or A
    // copied (and zero-padded) to 16 rows when M <= 16
    const bool direct = !fused_q && !fq.rowb && !multi && direct_scales(variant, M, N, K, As, ld_as, dev->sm_count);
    args.direct = direct ? 1 : 0;
    args.a_box_bytes = 0;
    uint8_t* a_pad = (fused_q || (M <= 16 && !direct)) ? static_cast<uint8_t*>(workspace) + tile_ast_bytes(M, K) : nullptr;
    args.a_from_prep = a_pad != nullptr;
    args.sk_full = sk ? skp.full : 0;
    args.sk_split = sk ? skp.split : 0;
    args.sk_kb_per = sk ? skp.kb_per : 0;
    args.partial = sk ? reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + prefix) : nullptr;
    args.AsT = static_cast<const float*>(workspace);
    args.m_pad = align_up(M, 128);
    args.n_pad = align_up(N, 128);
    args.BsT = nullptr;
    args.rowb_table = 0;
    if (fused_q) {
      const int64_t rows_q = M < 16 ? 16 : M;
      const int64_t threads = args.m_pad * kblocks * 8;
      launch_pdl(tile_prep_quant_kernel, dim3(static_cast<unsigned>((threads + 255) / 256)), stream,
                 static_cast<const __nv_bfloat16*>(fq.x_bf16), fq.ldx, a_pad, align_up(K, 16), rows_q,
                 static_cast<float*>(workspace), M, args.m_pad, static_cast<int>(kblocks));
      st = launch_status();
      if (st != B200FP8_OK) return st;
    } else if (!direct) {
      const ScaleCopy token = {As, static_cast<float*>(workspace), M, args.m_pad, ld_as};
      ScaleCopy weight = {nullptr, nullptr, 0, 0, 0};
      if (fq.rowb) {
        // the row scales of B, K-block-major, behind the token scales, the copy of A and the partial tiles
        args.BsT = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + prefix + (sk ? skp.partial_bytes : 0));
        args.rowb_table = kblocks <= kRowbTableKb ? 1 : 0;
        weight = {Bs, const_cast<float*>(args.BsT), N, args.n_pad, ld_bs};
      }
      const int64_t rows = weight.pad > token.pad ? weight.pad : token.pad;
      launch_pdl(tile_prep_kernel,
                 dim3(static_cast<unsigned>(rows / 32), static_cast<unsigned>((kblocks + 31) / 32),
                      a_pad != nullptr ? 3u : fq.rowb ? 2u : 1u),
                 stream, token, weight, static_cast<int>(kblocks), static_cast<const uint8_t*>(A), a_pad, M, K, lda,
                 align_up(K, 16));
      st = launch_status();
      if (st != B200FP8_OK) return st;
    }
    args.As = As;
    args.Bs = Bs;
    args.C = C;
    args.M = M;
    args.N = N;
    args.K = K;
    args.ld_as = ld_as;
    args.ld_bs = ld_bs;
    args.ldc = ldc;
    args.out_fp32 = out_dtype == B200FP8_OUT_FP32;
    args.status_word = status_word;
    const void* a_eff = a_pad ? static_cast<const void*>(a_pad) : A;
    const int64_t lda_eff = a_pad ? align_up(K, 16) : lda;
    if (sk) {
      st = pair_sk ? launch_pair<true>(a_eff, B, args, lda_eff, ldb, dev->pair_clusters, stream)
                   : launch_tile<256>(a_eff, B, args, lda_eff, ldb, dev->sm_count, stream, skp.grid);
      if (st != B200FP8_OK) return st;
      cudaLaunchAttribute fattr[1];
      fattr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      fattr[0].val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t fcfg = {};
      fcfg.gridDim = dim3(static_cast<unsigned>(skp.tail), pair_sk ? 8u : 4u, 4u);
      fcfg.blockDim = dim3(256);
      fcfg.stream = stream;
      fcfg.attrs = fattr;
      fcfg.numAttrs = 1;
      if (cudaLaunchKernelEx(&fcfg, tile_sk_fixup_kernel, static_cast<const float*>(args.partial), C, M, N, skp.num_kb,
                             ldc, static_cast<int>(out_dtype == B200FP8_OUT_FP32), skp.num_m, skp.num_n, skp.full,
                             skp.split, skp.kb_per, pair_sk ? 1 : 0) != cudaSuccess) {
        cudaGetLastError();
        return B200FP8_ERR_LAUNCH;
      }
      return launch_status();
    }
    if (variant == B200FP8_VARIANT_PAIR256)
      return launch_pair<false>(a_eff, B, args, lda_eff, ldb, dev->pair_clusters, stream);
    if (variant == B200FP8_VARIANT_PAIR256_SPLIT)
      return launch_pair<true>(a_eff, B, args, lda_eff, ldb, dev->pair_clusters, stream);
    return variant == B200FP8_VARIANT_TILE128
               ? launch_tile<128>(a_eff, B, args, lda_eff, ldb, dev->sm_count, stream, 0, cluster)
                                              : launch_tile<256>(a_eff, B, args, lda_eff, ldb, dev->sm_count, stream);
  }

  // stream-K decode variant
  if (fused_q) return B200FP8_ERR_VARIANT;
  if (M > 256) return B200FP8_ERR_VARIANT;
  const StreamKPlan p = streamk_plan(M, N, K, dev->sm_count);
  if (workspace == nullptr || static_cast<int64_t>(workspace_bytes) < p.ast_bytes + p.partial_bytes)
    return B200FP8_ERR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(workspace) & 255u) != 0) return B200FP8_ERR_ALIGN;
  float* ast = static_cast<float*>(workspace);
  float* partial = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + p.ast_bytes);

  {
    const int total = p.num_kb * p.mp;
    streamk_prep_kernel<<<(total + 255) / 256, 256, 0, stream>>>(As, ast, M, p.num_kb, ld_as, p.mp);
    st = launch_status();
    if (st != B200FP8_OK) return st;
  }
  StreamKArgs args;
  args.Bs = Bs;
  args.AsT = ast;
  args.partial = partial;
  args.C = C;
  args.M = M;
  args.N = N;
  args.K = K;
  args.ld_bs = ld_bs;
  args.ldc = ldc;
  args.out_fp32 = out_dtype == B200FP8_OUT_FP32;
  args.status_word = status_word;
  switch (p.mp) {
    case 16: st = launch_streamk<16>(A, B, args, lda, ldb, p.grid, stream); break;
    case 32: st = launch_streamk<32>(A, B, args, lda, ldb, p.grid, stream); break;
    case 64: st = launch_streamk<64>(A, B, args, lda, ldb, p.grid, stream); break;
    case 128: st = launch_streamk<128>(A, B, args, lda, ldb, p.grid, stream); break;
    default: st = launch_streamk<256>(A, B, args, lda, ldb, p.grid, stream); break;
  }
  if (st != B200FP8_OK) return st;
  const dim3 fix_grid(static_cast<unsigned>(p.num_tiles), static_cast<unsigned>((M + kFixupRows - 1) / kFixupRows));
  streamk_fixup_kernel<<<fix_grid, 128, 0, stream>>>(
      partial, C, M, N, p.num_kb, ldc, out_dtype == B200FP8_OUT_FP32, p.mp, p.grid);
  return launch_status();
}

int b200fp8_gemm(const void* A, const void* B, const float* As, const float* Bs, void* C, int64_t M, int64_t N,
                 int64_t K, int64_t lda, int64_t ldb, int64_t ld_as, int64_t ld_bs, int64_t ldc, int out_dtype,
                 int variant, void* workspace, size_t workspace_bytes, uint32_t* status_word, void* stream) {
  void* dst[1] = {C};
  const int64_t ld[1] = {ldc};
  return gemm_impl(false, A, B, As, Bs, 1, dst, ld, M, N, K, lda, ldb, ld_as, ld_bs, out_dtype, variant, workspace,
                   workspace_bytes, status_word, stream);
}

int b200fp8_gemm_rowscale(const void* A, const void* B, const float* As, const float* Bs_row, void* C, int64_t M,
                          int64_t N, int64_t K, int64_t lda, int64_t ldb, int64_t ld_as, int64_t ld_bs, int64_t ldc,
                          int out_dtype, void* workspace, size_t workspace_bytes, uint32_t* status_word,
                          void* stream) {
  void* dst[1] = {C};
  const int64_t ld[1] = {ldc};
  FusedQuant fq;
  fq.rowb = true;
  return gemm_impl(false, A, B, As, Bs_row, 1, dst, ld, M, N, K, lda, ldb, ld_as, ld_bs, out_dtype,
                   B200FP8_VARIANT_TILE128, workspace, workspace_bytes, status_word, stream, fq);
}

int64_t b200fp8_gemm_rowscale_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  if (M < 0 || N < 0 || K < 0) return -static_cast<int64_t>(B200FP8_ERR_SHAPE);
  if (M == 0 || N == 0 || K == 0) return 0;
  return tile_workspace_bytes(M, K) + bst_bytes(N, K) +
         auto_partial_bytes(M, N, K, B200FP8_CALL_ROWSCALE, limits_or_default());
}

int b200fp8_linear(const void* x_bf16, const void* B, const float* Bs, void* C, int64_t M, int64_t N, int64_t K,
                   int64_t ldx, int64_t ldb, int64_t ld_bs, int64_t ldc, int out_dtype, int variant, void* workspace,
                   size_t workspace_bytes, uint32_t* status_word, void* stream) {
  if (x_bf16 == nullptr && M > 0 && K > 0) return B200FP8_ERR_NULL;
  void* dst[1] = {C};
  const int64_t ld[1] = {ldc};
  FusedQuant fq;
  fq.x_bf16 = x_bf16;
  fq.ldx = ldx;
  return gemm_impl(false, nullptr, B, nullptr, Bs, 1, dst, ld, M, N, K, 0, ldb, 0, ld_bs, out_dtype, variant, workspace,
                   workspace_bytes, status_word, stream, fq);
}

int64_t b200fp8_linear_workspace_bytes(int64_t M, int64_t N, int64_t K, int variant) {
  if (M < 0 || N < 0 || K < 0) return -static_cast<int64_t>(B200FP8_ERR_SHAPE);
  if (M == 0 || N == 0 || K == 0) return 0;
  const int sms = sm_count_or_default();
  if (variant == B200FP8_VARIANT_AUTO)
    return linear_prefix_bytes(M, K) + auto_partial_bytes(M, N, K, B200FP8_CALL_ONE, limits_or_default());
  if (variant == B200FP8_VARIANT_TILE128 || variant == B200FP8_VARIANT_TILE256 ||
      variant == B200FP8_VARIANT_PAIR256 || variant == B200FP8_VARIANT_PAIR256_SPLIT)
    return linear_prefix_bytes(M, K);
  if (variant == B200FP8_VARIANT_TILE256_SK) return linear_prefix_bytes(M, K) + tile_sk_plan(M, N, K, sms).partial_bytes;
  if (variant == B200FP8_VARIANT_PAIR256_SPLIT_SK)
    return linear_prefix_bytes(M, K) + pair_sk_plan(M, N, K, b200fp8_gemm_pair_clusters()).partial_bytes;
  return -static_cast<int64_t>(B200FP8_ERR_VARIANT);
}

int b200fp8_gemm_multicast(const void* A, const void* B, const float* As, const float* Bs, void* C_multimem,
                           int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldb, int64_t ld_as, int64_t ld_bs,
                           int64_t ldc, int out_dtype, int variant, void* workspace, size_t workspace_bytes,
                           uint32_t* status_word, void* stream) {
  void* dst[1] = {C_multimem};
  const int64_t ld[1] = {ldc};
  return gemm_impl(true, A, B, As, Bs, 1, dst, ld, M, N, K, lda, ldb, ld_as, ld_bs, out_dtype, variant, workspace,
                   workspace_bytes, status_word, stream);
}

int b200fp8_gemm_scatter(const void* A, const void* B, const float* As, const float* Bs, int n_dst, void* const* C_dst,
                         const int64_t* ldc_dst, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldb,
                         int64_t ld_as, int64_t ld_bs, int out_dtype, int variant, void* workspace,
                         size_t workspace_bytes, uint32_t* status_word, void* stream) {
  return gemm_impl(false, A, B, As, Bs, n_dst, C_dst, ldc_dst, M, N, K, lda, ldb, ld_as, ld_bs, out_dtype, variant,
                   workspace, workspace_bytes, status_word, stream);
}

int b200fp8_ipc_export(const void* ptr, void* handle_out_64, int64_t* offset_out) {
  if (ptr == nullptr || handle_out_64 == nullptr || offset_out == nullptr) return B200FP8_ERR_NULL;
  static_assert(sizeof(cudaIpcMemHandle_t) == 64, "handle size");
  // the handle names the whole allocation; the offset of ptr inside it comes from the driver
  using RangeFn = CUresult (*)(CUdeviceptr*, size_t*, CUdeviceptr);
  void* sym = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &sym, cudaEnableDefault, &qres) != cudaSuccess ||
      qres != cudaDriverEntryPointSuccess || sym == nullptr) {
    cudaGetLastError();
    return B200FP8_ERR_DRIVER;
  }
  CUdeviceptr base = 0;
  size_t size = 0;
  if (reinterpret_cast<RangeFn>(sym)(&base, &size, reinterpret_cast<CUdeviceptr>(ptr)) != CUDA_SUCCESS)
    return B200FP8_ERR_DRIVER;
  cudaIpcMemHandle_t h;
  if (cudaIpcGetMemHandle(&h, reinterpret_cast<void*>(base)) != cudaSuccess) {
    cudaGetLastError();
    return B200FP8_ERR_DRIVER;
  }
  memcpy(handle_out_64, &h, 64);
  *offset_out = static_cast<int64_t>(reinterpret_cast<CUdeviceptr>(ptr) - base);
  return B200FP8_OK;
}

int b200fp8_ipc_open(const void* handle_64, void** base_out) {
  if (handle_64 == nullptr || base_out == nullptr) return B200FP8_ERR_NULL;
  cudaIpcMemHandle_t h;
  memcpy(&h, handle_64, 64);
  void* p = nullptr;
  if (cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess) != cudaSuccess || p == nullptr) {
    cudaGetLastError();
    return B200FP8_ERR_DRIVER;
  }
  *base_out = p;
  return B200FP8_OK;
}

int b200fp8_ipc_close(void* base) {
  if (base == nullptr) return B200FP8_ERR_NULL;
  if (cudaIpcCloseMemHandle(base) != cudaSuccess) {
    cudaGetLastError();
    return B200FP8_ERR_DRIVER;
  }
  return B200FP8_OK;
}

int b200fp8_peer_barrier_limited(uint32_t* const* flag_arrays, int n, int rank, uint32_t epoch, int64_t limit_clocks,
                                 uint32_t* status_word, void* stream) {
  if (flag_arrays == nullptr) return B200FP8_ERR_NULL;
  if (n < 1 || n > 8 || rank < 0 || rank >= n || limit_clocks < 1) return B200FP8_ERR_SHAPE;
  PeerFlags f;
  for (int i = 0; i < 8; ++i) {
    f.p[i] = i < n ? flag_arrays[i] : nullptr;
    if (i < n && (f.p[i] == nullptr || (reinterpret_cast<uintptr_t>(f.p[i]) & 3u) != 0)) return B200FP8_ERR_NULL;
  }
  peer_barrier_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(f, n, rank, epoch,
                                                                       static_cast<long long>(limit_clocks), status_word);
  return launch_status();
}

int b200fp8_peer_barrier(uint32_t* const* flag_arrays, int n, int rank, uint32_t epoch, uint32_t* status_word,
                         void* stream) {
  return b200fp8_peer_barrier_limited(flag_arrays, n, rank, epoch, kPeerBarrierDefaultLimitClks, status_word, stream);
}

int b200fp8_gemm_decode_static(const void* A, const void* B, const float* As, const float* Bs, void* C, int64_t M,
                               int64_t N, int64_t K, int64_t lda, int64_t ldb, int64_t ld_as, int64_t ld_bs,
                               int64_t ldc, int out_dtype, uint32_t* status_word, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (M < 0 || N < 0 || K < 0) return B200FP8_ERR_SHAPE;
  if (out_dtype != B200FP8_OUT_BF16 && out_dtype != B200FP8_OUT_FP32) return B200FP8_ERR_DTYPE;
  if (M == 0 || N == 0) return B200FP8_OK;
  if (M > 256) return B200FP8_ERR_TOO_LARGE;
  if (A == nullptr || B == nullptr || As == nullptr || Bs == nullptr || C == nullptr) return B200FP8_ERR_NULL;
  if (K == 0) return B200FP8_ERR_SHAPE;
  const int64_t kblocks = (K + 127) / 128;
  if (ldc < N || lda < K || ldb < K || ld_as < kblocks || ld_bs < kblocks) return B200FP8_ERR_SHAPE;
  if (lda % 16 != 0 || ldb % 16 != 0 || (reinterpret_cast<uintptr_t>(A) & 15u) != 0 ||
      (reinterpret_cast<uintptr_t>(B) & 15u) != 0)
    return B200FP8_ERR_ALIGN;
  if (N > 0x7FFFFF00 || K > 0x7FFFFF00) return B200FP8_ERR_TOO_LARGE;

  const DeviceInfo* dev = nullptr;
  int st = device_info(&dev);
  if (st != B200FP8_OK) return st;
  const StreamKPlan p = streamk_plan(M, N, K, dev->sm_count);
  if (static_cast<size_t>(p.ast_bytes + p.partial_bytes) > kStaticScratchBytes) return B200FP8_ERR_TOO_LARGE;
  void* scratch = nullptr;
  st = static_scratch_address(&scratch);   // first call on a device: cudaGetSymbolAddress
  if (st != B200FP8_OK) return st;
  float* ast = static_cast<float*>(scratch);
  float* partial = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + p.ast_bytes);

  // Nothing in the scratch has to start at zero: the prep kernel rewrites the whole AsT
  // region (padding included) and every partial slot the fix-up kernel reads is written by
  // the stream-K kernel of the same call first.
  const int total = p.num_kb * p.mp;
  streamk_prep_kernel<<<(total + 255) / 256, 256, 0, stream>>>(As, ast, M, p.num_kb, ld_as, p.mp);
  st = launch_status();
  if (st != B200FP8_OK) return st;
  StreamKArgs args;
  args.Bs = Bs;
  args.AsT = ast;
  args.partial = partial;
  args.C = C;
  args.M = M;
  args.N = N;
  args.K = K;
  args.ld_bs = ld_bs;
  args.ldc = ldc;
  args.out_fp32 = out_dtype == B200FP8_OUT_FP32;
  args.status_word = status_word;
  switch (p.mp) {
    case 16: st = launch_streamk<16>(A, B, args, lda, ldb, p.grid, stream); break;
    case 32: st = launch_streamk<32>(A, B, args, lda, ldb, p.grid, stream); break;
    case 64: st = launch_streamk<64>(A, B, args, lda, ldb, p.grid, stream); break;
    case 128: st = launch_streamk<128>(A, B, args, lda, ldb, p.grid, stream); break;
    default: st = launch_streamk<256>(A, B, args, lda, ldb, p.grid, stream); break;
  }
  if (st != B200FP8_OK) return st;
  const dim3 fix_grid(static_cast<unsigned>(p.num_tiles), static_cast<unsigned>((M + kFixupRows - 1) / kFixupRows));
  streamk_fixup_kernel<<<fix_grid, 128, 0, stream>>>(
      partial, C, M, N, p.num_kb, ldc, out_dtype == B200FP8_OUT_FP32, p.mp, p.grid);
  return launch_status();
}

}  // extern "C"
