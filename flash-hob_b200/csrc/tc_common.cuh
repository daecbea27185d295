// Pieces shared by the tensor-core kernels (sm_100a): CTA shape and warp roles, the bounded
// mbarrier wait, the K-step loops that issue tcgen05.mma for a whole tile product, and the TMA
// tensor-map builder.  Included by each .cu file that holds such kernels; everything lives in an
// unnamed namespace.
#pragma once

#include <cuda.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <utility>

#include "fhob_common.cuh"
#include "sm100_ptx.cuh"

namespace fhob {
namespace {

using namespace ptx;

constexpr int BM = 128;
constexpr int BOX_ROWS = 64;  // rows of a TMA box
constexpr int EW_THREADS = 256;
constexpr int MMA_WARP = 0;   // issues the products of chain 1 (group A and the outputs it feeds); owns TMEM
constexpr int MMA_WARP2 = 1;  // issues the products of chain 2 (group B and the outputs it feeds)
constexpr int TMA_WARP = 2;
constexpr int EW_WARP0 = 4;   // elementwise warps 4..11
constexpr int NTHREADS = 384;
constexpr int TMEM_COLS = 512;
constexpr int SMEM_LIMIT = 232448;  // 227 KB per CTA
constexpr int SMEM_TAIL = 1024;     // barriers, TMEM base, abort flag, row-sum exchange
constexpr long long kTimeoutCycles = 2000000000LL;   // about a second
constexpr long long kPeerCheckCycles = 2000000LL;    // after ~1 ms also give up if another CTA timed out

// Bounded wait on an mbarrier phase.  `b` is the CTA's barrier block (any struct with an
// `abort_flag`): a wait that runs out sets FHOB_ERR_TIMEOUT in the status word and the CTA-wide
// abort flag, and every later wait of the CTA returns false at once.
template <class B>
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, B* b, int* status) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long start = clock64();
  uint32_t spins = 0;
  for (;;) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((++spins & 0xFFu) == 0) {
      if (*reinterpret_cast<volatile int*>(&b->abort_flag)) return false;
      long long el = clock64() - start;
      if (el > kTimeoutCycles ||
          (el > kPeerCheckCycles && (*reinterpret_cast<volatile int*>(status) & FHOB_ERR_TIMEOUT))) {
        *reinterpret_cast<volatile int*>(&b->abort_flag) = 1;
        atomicOr(status, FHOB_ERR_TIMEOUT);
        return false;
      }
    }
  }
}

// Bounded wait for something already in flight (a load to land, products to finish) before the CTA exits.
__device__ __forceinline__ void wait_landed(uint64_t* bar, uint32_t parity, int* status) {
  const long long start = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - start > kTimeoutCycles) {
      atomicOr(status, FHOB_ERR_TIMEOUT);
      break;
    }
  }
}

// Descriptor words of 128-byte-swizzled bf16 tiles (rows of 64 elements, 8-row groups 1024 B apart).
constexpr uint32_t kDescHi = umma_desc_hi_sw128(1024);

// D (+)= A . B^T with both tiles K-major in shared memory.  a_lo / b_lo are the low descriptor
// words of the tiles; a K=16 step advances 32 bytes inside a 64-column box, the second box of a
// D=128 tile starts A_BOX / B_BOX bytes after the first.  The number of B rows (N) is in idesc.
template <int D, int A_BOX, int B_BOX, int KS0 = 0, int KS1 = D / 16>
__device__ __forceinline__ void gemm_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                        bool accumulate) {
#pragma unroll
  for (int ks = KS0; ks < KS1; ++ks) {
    const uint32_t a = a_lo + (((ks / 4) * A_BOX + (ks % 4) * 32) >> 4);
    const uint32_t b = b_lo + (((ks / 4) * B_BOX + (ks % 4) * 32) >> 4);
    umma_ss_split(d_tmem, a, b, kDescHi, idesc, (accumulate || ks > 0) ? 1u : 0u);
  }
}

// D (+)= A . B with A = bf16 tile in TMEM (128 x BN, 8 columns per 16 rows of B) and B = streamed
// tile (BN rows x N columns, N in idesc) read MN-major: the contraction runs down the BN rows,
// 2048 bytes per step.  b_lo must carry the leading byte offset (distance between the tile's two
// 64-column boxes; not used when the tile has a single box).
template <int BN>
__device__ __forceinline__ void gemm_ts(uint32_t d_tmem, uint32_t a_region, uint32_t b_lo,
                                        uint32_t idesc, bool accumulate) {
  constexpr int CH = BN / 32;
#pragma unroll
  for (int s = 0; s < BN / 16; ++s) {
    const uint32_t a = a_region + (s / CH) * (BN / 2) + 8 * (s % CH);
    umma_ts_split(d_tmem, a, b_lo + ((s * 2048) >> 4), kDescHi, idesc, (accumulate || s > 0) ? 1u : 0u);
  }
}

__device__ __forceinline__ void load4(uint32_t smem_addr, float (&v)[4]) {
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(smem_addr));
}

__device__ __forceinline__ float2 f2(uint32_t lo, uint32_t hi) {
  return make_float2(__uint_as_float(lo), __uint_as_float(hi));
}

// Loads `ROWS` rows x D columns starting at row `y` of one head: boxes of 64 columns x 64 rows; a
// tile's 64-column blocks are BOX bytes apart, rows are 128 bytes inside a block.
template <int ROWS, int D, int BOX>
__device__ __forceinline__ void load_tile(uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int y, int head, int batch) {
  static_assert(ROWS % BOX_ROWS == 0, "whole boxes");
#pragma unroll
  for (int bx = 0; bx < D / 64; ++bx)
#pragma unroll
    for (int by = 0; by < ROWS / BOX_ROWS; ++by)
      tma_load_4d(dst + bx * BOX + by * (BOX_ROWS * 128), map, bar, bx * 64, y + by * BOX_ROWS, head, batch);
}

// 2^x for two numbers on the FMA and ALU pipes, to relieve the special-function units (16 a clock and SM)
// where they are what a kernel waits for.  x = n + f with n the nearest integer, |f| <= 1/2; 2^f is a
// degree-5 polynomial of small relative error there (Remez exchange; 1.3e-7 with the coefficients rounded as
// written, 2.1e-7 evaluated in fp32, as ex2.approx: 2^-22), times 2^n put together from its exponent field.
// x <= 127; below -126 the result is about 2^-126 or less, never a larger number; NaN stays NaN (a clamp that
// keeps it, and a product: an integer added to the exponent of a NaN makes a number of it).
__device__ __forceinline__ float clamp_exp2(float x) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(-126.f));
  return r;
}
__device__ __forceinline__ float2 exp2_fma(float2 x) {
  constexpr float kMagic = 12582912.f;   // 1.5 * 2^23: adding it leaves the nearest integer in the low bits
  x.x = clamp_exp2(x.x);
  x.y = clamp_exp2(x.y);
  const float2 r = __fadd2_rn(x, make_float2(kMagic, kMagic));
  const float2 n = __fadd2_rn(r, make_float2(-kMagic, -kMagic));
  const float2 f = __ffma2_rn(n, make_float2(-1.f, -1.f), x);
  auto c = [](float v) { return make_float2(v, v); };
  float2 y = __ffma2_rn(c(0.0013276472f), f, c(0.009675541f));
  y = __ffma2_rn(y, f, c(0.05550713f));
  y = __ffma2_rn(y, f, c(0.2402212f));
  y = __ffma2_rn(y, f, c(0.69314694f));
  y = __ffma2_rn(y, f, c(1.0000001f));
  return __fmul2_rn(y, make_float2(__uint_as_float((__float_as_uint(r.x) << 23) + 0x3f800000u),
                                   __uint_as_float((__float_as_uint(r.y) << 23) + 0x3f800000u)));
}

// ---- split streamed axis: a cluster of `split` CTAs shares the streamed tiles of one stationary tile
// and adds up its results through distributed shared memory, in rank order (so bits do not vary).

// What CTA `block` of a kind of CTAs does: part `part` of item `item`, or nothing.
struct CtaWork {
  int item, part;
  bool live;   // false: the CTA only fills up a cluster (item 0 stands in; nothing may be stored)
};
__host__ __device__ __forceinline__ CtaWork cta_work(int block, int split, int items) {
  CtaWork w = {block, 0, true};
  if (split > 1) {
    w.item = block / split;
    w.part = block - w.item * split;
  }
  w.live = w.item < items;
  if (!w.live) w.item = 0;
  return w;
}

// Streamed tiles of part `part` of `split` of the range [begin, end).
__device__ __forceinline__ void split_range(int part, int split, int& begin, int& end) {
  const int n = end - begin, b = begin;
  begin = b + static_cast<int>(static_cast<long long>(n) * part / split);
  end = b + static_cast<int>(static_cast<long long>(n) * (part + 1) / split);
}

// 16 fp32 columns of this thread's row of a finished result at TMEM address taddr (zeros if there was nothing
// to add up).  HALVES: the result is the sum of two accumulators, 64 columns apart (split operands).
template <bool HALVES>
__device__ __forceinline__ void load_result(uint32_t taddr, bool any, uint32_t (&v)[16]) {
  if (any) {
    [[maybe_unused]] uint32_t w[16];
    tmem_ld16(taddr, v);
    if constexpr (HALVES) tmem_ld16(taddr + 64, w);
    tmem_wait_ld();
    if constexpr (HALVES) {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = 0u;
  }
}

// This thread's W fp32 result columns (TMEM addresses taddr..) of its row -> staging area.
template <int W, bool HALVES = false>
__device__ __forceinline__ void stage_row(float* dst, uint32_t taddr, bool any) {
#pragma unroll
  for (int c = 0; c < W; c += 16) {
    uint32_t v[16];
    load_result<HALVES>(taddr + c, any, v);
#pragma unroll
    for (int j = 0; j < 16; j += 4)
      *reinterpret_cast<uint4*>(dst + c + j) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  }
}

// Adds the staged columns [c0, c0 + W) of all parts for this CTA's share of the rows, times `mul`, and stores
// them to `base` (n_rows x d_mem per head).  `stage` = shared address of the staging area (row pitch
// `pitch` floats), `rank0` = cluster rank of part 0, `tid` of 256 threads; ROWS rows in all.
template <int W, bool F32, bool F16, int ROWS = BM>
__device__ __forceinline__ void reduce_store(uint32_t stage, int pitch, int c0, int rank0, int part, int split, int tid, void* base,
                                             int head, int m0, int n_rows, int d_mem, float mul) {
  constexpr int V = F32 ? 4 : 8;
  const int rows = (ROWS + split - 1) / split;
  for (int i = tid; i < rows * (W / V); i += EW_THREADS) {
    const int r = part * rows + i / (W / V), c = (i % (W / V)) * V;
    if (r >= ROWS || m0 + r >= n_rows || c >= d_mem) continue;   // rows are whole 16-byte pieces
    float4 a[V / 4];
#pragma unroll
    for (int h = 0; h < V / 4; ++h) a[h] = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t at = stage + (r * pitch + c0 + c) * 4;
    for (int s = 0; s < split; ++s) {
      const uint32_t from = cluster_map(at, rank0 + s);
#pragma unroll
      for (int h = 0; h < V / 4; ++h) {
        const float4 x = cluster_ld4(from + 16 * h);
        a[h].x += x.x; a[h].y += x.y; a[h].z += x.z; a[h].w += x.w;
      }
    }
    const size_t off = (static_cast<size_t>(head) * n_rows + m0 + r) * d_mem + c;
    if constexpr (F32) {
      *reinterpret_cast<float4*>(static_cast<float*>(base) + off) = make_float4(a[0].x * mul, a[0].y * mul, a[0].z * mul, a[0].w * mul);
    } else {
      *reinterpret_cast<uint4*>(static_cast<uint16_t*>(base) + off) =
          make_uint4(pack16<F16>(a[0].x * mul, a[0].y * mul), pack16<F16>(a[0].z * mul, a[0].w * mul),
                     pack16<F16>(a[V / 4 - 1].x * mul, a[V / 4 - 1].y * mul), pack16<F16>(a[V / 4 - 1].z * mul, a[V / 4 - 1].w * mul));
    }
  }
}

// ------------------------------------------------------------------ host side
int check_device() {
  static thread_local int checked_dev = -1;
  int dev = 0;
  FHOB_CUDA_OK(cudaGetDevice(&dev));
  if (dev != checked_dev) {
    int major = 0;
    FHOB_CUDA_OK(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev));
    if (major != 10) return FHOB_ERR_ARCH;
    checked_dev = dev;
  }
  return FHOB_OK;
}

// Launches with programmatic stream serialization: the kernel's CTAs may start while the kernel in
// front of it drains (it says pdl_launch_dependents), and wait in pdl_wait before they touch memory.
template <class... P, class... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, int cluster, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cluster > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeTiledFn>(f);
  }();
  return fn;
}

// 16-bit matrix of `n` rows x `d` columns per head, heads and batch entries at the strides of `v`:
// a 4-D map (d, n, heads, batches), box = 64 columns x 64 rows of one head, 128-byte swizzle.  Taller
// tiles take several boxes, so one map per tensor serves every kernel of a call.
// Encoded maps are kept in a small per-thread table: a training step calls the operator with the
// same tensors again and again, and an encode costs a few microseconds of host time per map.
struct MapKey {
  const void* base;
  int n, d, f16, heads, batches;
  long long row, head, batch;
  bool operator==(const MapKey& o) const {
    return base == o.base && n == o.n && d == o.d && f16 == o.f16 && heads == o.heads &&
           batches == o.batches && row == o.row && head == o.head && batch == o.batch;
  }
};

int make_map(CUtensorMap* m, const void* base, const View& v, int n, int d, bool f16) {
  constexpr int kSlots = 64;
  struct Entry {
    MapKey key;
    CUtensorMap map;
  };
  static thread_local Entry table[kSlots];
  static thread_local int used = 0, next = 0;
  const MapKey key{base, n, d, f16 ? 1 : 0, v.heads, v.batches, v.row, v.head, v.batch};
  for (int i = 0; i < used; ++i)
    if (table[i].key == key) {
      *m = table[i].map;
      return FHOB_OK;
    }
  EncodeTiledFn fn = encode_fn();
  if (!fn) {
    set_cuda_error_text("cuTensorMapEncodeTiled entry point not available");
    return FHOB_ERR_CUDA;
  }
  // strides of the three outer dims in bytes: multiples of 16, checked by the caller's validation
  // and once more by the driver
  cuuint64_t dims[4] = {static_cast<cuuint64_t>(d), static_cast<cuuint64_t>(n), static_cast<cuuint64_t>(v.heads),
                        static_cast<cuuint64_t>(v.batches)};
  cuuint64_t strides[3] = {static_cast<cuuint64_t>(v.row) * 2, static_cast<cuuint64_t>(v.head) * 2,
                           static_cast<cuuint64_t>(v.batch) * 2};
  cuuint32_t box[4] = {64, BOX_ROWS, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(m, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    char buf[96];
    snprintf(buf, sizeof(buf), "cuTensorMapEncodeTiled failed with CUresult %d", static_cast<int>(r));
    set_cuda_error_text(buf);
    return FHOB_ERR_CUDA;
  }
  Entry& e = table[next];
  e.key = key;
  e.map = *m;
  next = (next + 1) % kSlots;
  if (used < kSlots) ++used;
  return FHOB_OK;
}

// Raises the dynamic shared-memory limit of `kernel` once per device and host thread (it is a
// per-function, per-device attribute; setting it again on every launch costs a driver call).
template <class K>
int allow_smem(K kernel, int bytes) {
  constexpr int kSlots = 96;
  struct Entry {
    const void* fn;
    unsigned long long devices;
  };
  static thread_local Entry table[kSlots];
  static thread_local int used = 0;
  int dev = 0;
  FHOB_CUDA_OK(cudaGetDevice(&dev));
  const unsigned long long bit = (dev >= 0 && dev < 64) ? (1ull << dev) : 0;
  const void* fn = reinterpret_cast<const void*>(kernel);
  Entry* e = nullptr;
  for (int i = 0; i < used && !e; ++i)
    if (table[i].fn == fn) e = &table[i];
  if (e && bit && (e->devices & bit)) return FHOB_OK;
  FHOB_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  if (!e && used < kSlots) {
    e = &table[used++];
    e->fn = fn;
    e->devices = 0;
  }
  if (e) e->devices |= bit;
  return FHOB_OK;
}

// SMs of the current device: how many CTAs run at once of a kernel that has an SM to itself.  0: not known.
int sm_count() {
  constexpr int kDevices = 64;
  static thread_local int table[kDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 0;
  if (table[dev] == 0 && cudaDeviceGetAttribute(&table[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) table[dev] = 0;
  return table[dev];
}

// How many CTAs of a cluster share the streamed tiles of one stationary tile of a head.  That is also the
// number of partial sums its results are added up from, so it is worked out from one head alone: the bits
// of a head must not depend on the heads it is launched with (batches are cut over GPUs and into ranges).
// Two conditions, because nothing is known of the other heads:
//  - the head's stationary tiles together take at most one cluster of the portable size, 8 CTAs: a layer
//    of 16 heads is then still one wave (a B200 runs 132 CTAs at once in clusters of 4, 120 in clusters of 8);
//  - where there are heads enough to fill the GPU unsplit, the parts cost at most a quarter more.  In
//    streamed tiles, a CTA takes about `fixed` besides its own (launch, prologue, first loads, epilogue: 6
//    to 9 us against 1 to 1.7 us a 64-row tile of the tensor-core kernels) and `cluster` more in a cluster (its
//    CTAs start together and meet twice).
// Operator, bf16, D = 64, 100 x 6000, us, unsplit / 4 parts / 8: 4 heads 153 / 50 / 38, 16 heads 156 / 95 / 109,
// 256 heads 959 / 1070 / 1247.
constexpr int kMaxParts = 8;
struct SplitCost {
  float fixed = 5.f, cluster = 1.f;
  float any = 0.f;   // heads of any number of tiles are split if that costs at most this much
};
inline int split_parts(int stationary_tiles, int streamed_tiles, const SplitCost& cost = SplitCost{}) {
  const float unsplit = static_cast<float>(streamed_tiles) + cost.fixed;
  int parts = kMaxParts;
  for (; parts > 1; parts >>= 1) {
    const float more = streamed_tiles + parts * (cost.fixed + cost.cluster) - unsplit;
    if (more <= (stationary_tiles <= kMaxParts / parts ? 0.25f : cost.any) * unsplit) break;
  }
  return parts;
}
// Streamed tiles of `tile` rows that the longest item of `rows` stationary rows sees.
inline int longest(int n, int tile, int rows, int window) {
  const int all = (n + tile - 1) / tile;
  const long long seen = window > 0 ? (static_cast<long long>(rows) + window - 2) / tile + 2 : all;
  return seen < all ? static_cast<int>(seen) : all;
}

// The tensor-core kernels: 128-row stationary tiles, streamed rows in units of 64.
inline int tc_parts(int n_stat, int n_strm, int window) { return split_parts((n_stat + BM - 1) / BM, longest(n_strm, 64, BM, window)); }

}  // namespace

// Grid of a launch that holds query-tiled and key-tiled CTAs (of which either may have none): the CTAs of
// an item (a stationary tile of a head) are neighbours in one cluster, and each kind is padded to whole clusters.
inline PairGrid pair_grid(long long items_q, int split_q, long long items_k, int split_k) {
  PairGrid g;
  g.items_q = static_cast<int>(items_q);
  g.items_k = static_cast<int>(items_k);
  g.split_q = split_q;
  g.split_k = split_k;
  g.cluster = 1;
  if (items_q > 0 && split_q > g.cluster) g.cluster = split_q;
  if (items_k > 0 && split_k > g.cluster) g.cluster = split_k;   // both are powers of two
  auto padded = [&](long long n) { return (n + g.cluster - 1) / g.cluster * g.cluster; };
  g.q_blocks = static_cast<int>(padded(items_q * split_q));
  g.blocks = g.q_blocks + padded(items_k * split_k);
  return g;
}
// Clusters of 4 or 8 leave SMs idle that single CTAs would use: an unsplit kind of many CTAs gets a launch of
// its own.  (us, one launch -> two, operator as above in clusters of 8: 256 heads 1560 -> 1247, 16 heads 109 -> 109,
// 4 heads 38 -> 48; in clusters of 2, 32 heads 100 x 2000 D = 128, 93 -> 110.)
inline bool launch_apart(const PairGrid& g) {
  const int unsplit = g.split_q == 1 ? g.items_q : (g.split_k == 1 ? g.items_k : 0);
  return g.cluster >= 4 && unsplit > 4 * sm_count();
}

}  // namespace fhob
