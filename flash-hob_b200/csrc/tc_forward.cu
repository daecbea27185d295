// Forward of attention on the tensor cores (sm_100a): O and the fp32 logsumexp L, or L alone - the
// producers of what the double-backward operator consumes.  Role of the reference's forward kernel
// and of its produce_L (fhog/triton_flash.py:12-133, :252-258), at O(N) memory.
//
// A CTA owns up to two 128-query tiles of a head, A and B, and streams 128-key tiles.  One thread
// issues all products; four warps per query tile do its softmax, one thread per row:
//
//     tensor pipe:   S_A(t+1) | P_B(t) V(t) | S_B(t+1) | P_A(t+1) V(t+1) | ...
//     softmax A:                 S_A(t+1) -> P_A(t+1)   ...
//     softmax B:     S_B(t) -> P_B(t)             S_B(t+1) -> ...
//
// so while one tile's exponentials run on the special-function units, the other tile's products run
// on the tensor pipe.  P overwrites S in TMEM (16-bit) and is the A operand of P V.
//
// What bounds it: one exponential per score at 16 a clock and SM is 2 048 cycles for the 2 x 128 x 128
// scores of a step, as much as the tensor pipe needs for them at head dim 128 (half of it at 64).  A step
// takes about 3 600 (head dim 128) and 3 050 (64) cycles: the rest is latency that two warps a scheduler
// do not hide (scores -> registers -> maximum -> exponentials -> P), and 5 us of a CTA's own.
//  - A row belongs to one thread: no exchange of maxima, no shuffles, no shared memory in the loop (the
//    kernel before this one split a row over two warps that met at an mbarrier for every tile).
//  - Tiles that need masking have a copy of the code of their own; 128 scores and their masks do not fit
//    the registers together.
//  - Head dims up to 64: 64-key tiles and two score stages per query tile (TMEM has the room), so that the
//    scores of the next tile are there when P is done.  Otherwise 128-key tiles (a 64-row score product
//    is bound by shared memory, 48 cycles for 32 of work) and one stage; P is handed over in halves.
//  - The reference maximum of the online softmax follows the row's maximum lazily (only when that has grown
//    by more than 8 in the log2 domain, so P < 2^8); O is rescaled in TMEM on those occasions.
// Measured, us, kernel before -> this one: 32 heads N=4096 D=128 395 -> 255, causal 258 -> 180; 64 heads
// N=2048 D=64 204 -> 124, L alone 164 -> 92.  Tried and slower: half a step of stagger between A and B,
// loading a tile's scores while the one before is exponentiated, a maximum that lags one tile behind.
#include <type_traits>

#include "tc_common.cuh"

namespace fhob {
namespace {

constexpr int FW_MAX_SLOTS = 10;
constexpr int FW_TAIL = 2048;  // barriers, TMEM base, abort flag, row vectors of a split
constexpr int FW_EW = 128;     // softmax threads per query tile
// Warp 0 issues the products (and owns TMEM), warp 1 the loads, warps 4-7 and 8-11 are the softmax of A and B.
constexpr int FW_TMA_WARP = 1, FW_EW_WARP0 = 4, FW_THREADS = 384;

template <int DQK, int DV, bool OUT>
struct FwCfg {
  static constexpr bool kSmall = DQK == 64 && DV == 64;
  static constexpr int BN = OUT && kSmall ? 64 : 128;       // keys per tile
  static constexpr int STAGES = OUT && !kSmall ? 1 : 2;     // score stages of a query tile; the issuing thread runs that far ahead
  static constexpr int Q_BYTES = BM * DQK * 2;
  // K and V tiles take turns in one ring of slots (K only when no O is wanted)
  static constexpr int SLOT_BYTES = BN * (OUT && DV > DQK ? DV : DQK) * 2;
  static constexpr int NSLOT_FIT = (SMEM_LIMIT - FW_TAIL - 2 * Q_BYTES) / SLOT_BYTES;
  static constexpr int NSLOT = NSLOT_FIT > FW_MAX_SLOTS ? FW_MAX_SLOTS : NSLOT_FIT;
  static constexpr int SMEM_BYTES = 2 * Q_BYTES + NSLOT * SLOT_BYTES + FW_TAIL;
  static constexpr int O_COLS = 128;                                 // TMEM columns reserved for each O
  static constexpr int kPitch = DV + 4;                              // floats per row of the staging area (split keys)
  static_assert(NSLOT >= 4, "two tiles in use, two on the way");
  static_assert(BM * kPitch * 4 <= 2 * Q_BYTES + NSLOT * SLOT_BYTES, "staging area");
};

struct FwParams {
  CUtensorMap q, k, v;
  float* lse_out;
  void* o;
  int* status;
  int n_q, n_k, causal, window;
  int groups;     // CTAs per head: groups of `q_tiles` 128-query tiles
  int q_tiles;    // 1 or 2
  int items;      // heads * groups
  int split;      // CTAs of a cluster that share the keys of an item (with q_tiles == 1)
  int heads;      // heads per batch entry of the input tensor maps
  int d_v;        // columns of O in memory (<= DV)
  float scale;
};

struct FwBars {
  uint64_t q_full[2];
  uint64_t kv_full[FW_MAX_SLOTS];
  uint64_t kv_free[FW_MAX_SLOTS];
  uint64_t s_full[2][2];   // [query tile][stage]: scores finished
  uint64_t s_free[2][2];   // without O: scores are in registers
  uint64_t p_full[2][2];   // P written over S
  uint64_t p_half[2];      // its first half has been
  uint64_t o_done[2];      // a tile's P V has finished
  uint64_t out_full[2];    // the last one has
  uint64_t teardown;
  uint32_t tmem_base;
  int abort_flag;
  float red[2][BM];        // split keys: reference maxima and sums of this part's rows
};
static_assert(sizeof(FwBars) <= FW_TAIL, "tail");

__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

__device__ __forceinline__ void fw_split_pack(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(x, y);
  lo = pack_bf16(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}

// fp32 problems (SPLIT): every fp32 operand as bf16 hi + lo, rows [hi(64) | lo(64)] = the two boxes of a
// 128-wide tile; a contraction is hi.hi + hi.lo + lo.hi (see tc_kernels.cu).  Head dims up to 64.  The small
// terms of P V have an accumulator of their own (see BwCfg in tc_backward.cu).
template <int DQK, int DV, bool F16, bool SPLIT, bool OUT>
__global__ void __launch_bounds__(FW_THREADS, 1) fw_kernel(const __grid_constant__ FwParams p) {
  using C = FwCfg<DQK, DV, OUT>;
  static_assert(!SPLIT || (DQK == 128 && DV == 128 && !F16), "split fp32 operands are [hi(64) | lo(64)] bf16 rows");
  constexpr int BN = C::BN, kStages = C::STAGES;
  constexpr bool kHalves = OUT && BN == 128;   // P handed over in two halves
  constexpr int kO = DV, kRes = SPLIT ? 64 : DV;   // columns of an O accumulator (split: [hi.hi | hi.lo + lo.hi]) and of O
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* ring = smem + 2 * C::Q_BYTES;
  FwBars* bars = reinterpret_cast<FwBars*>(ring + C::NSLOT * C::SLOT_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  int item = blockIdx.x, part = 0;
  if (p.split > 1) {
    item = blockIdx.x / p.split;
    part = blockIdx.x - item * p.split;
  }
  const int head = item / p.groups;
  const int group = p.groups - 1 - (item - head * p.groups);   // causal: longest first
  const int off = p.n_k - p.n_q;
  // key tiles of the two query tiles (a tile beyond the last query has none and is left alone)
  auto m_of = [&](int x) { return (group * p.q_tiles + x) * BM; };
  auto live = [&](int x) { return x < p.q_tiles && m_of(x) < p.n_q; };
  int begin[2], end[2];
#pragma unroll
  for (int x = 0; x < 2; ++x) {
    begin[x] = end[x] = 0;
    if (live(x)) {
      visible_tiles(true, m_of(x), BM, BN, p.n_k, off, p.causal, p.window, begin[x], end[x]);
      if (p.split > 1) split_range(part, p.split, begin[x], end[x]);
    }
  }
  const bool any0 = end[0] > begin[0], any1 = end[1] > begin[1];
  const int t_begin = any0 && any1 ? min(begin[0], begin[1]) : (any0 ? begin[0] : begin[1]);
  const int t_end = any0 && any1 ? max(end[0], end[1]) : (any0 ? end[0] : end[1]);
  const int n_tiles = t_end > t_begin ? t_end - t_begin : 0;

  int fault = 0;   // thread 0: what to report at the end
  if (threadIdx.x == 0) {
    if (smem_u32(smem) & 1023u) fault |= FHOB_ERR_SMEM_ALIGN;
    for (int x = 0; x < 2; ++x) {
      mbar_init(&bars->q_full[x], 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(&bars->s_full[x][i], 1);
        mbar_init(&bars->s_free[x][i], FW_EW);
        mbar_init(&bars->p_full[x][i], FW_EW);
      }
      mbar_init(&bars->p_half[x], FW_EW);
      mbar_init(&bars->o_done[x], 1);
      mbar_init(&bars->out_full[x], 1);
    }
    for (int i = 0; i < FW_MAX_SLOTS; ++i) {
      mbar_init(&bars->kv_full[i], 1);
      mbar_init(&bars->kv_free[i], 1);
    }
    mbar_init(&bars->teardown, 1);
    bars->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == MMA_WARP) {
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == FW_TMA_WARP && lane == 0) {
    prefetch_tensormap(&p.q);
    prefetch_tensormap(&p.k);
    if (OUT) prefetch_tensormap(&p.v);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // the CTA allocates all 512 columns, so the allocation starts at column 0 (checked)
  if (threadIdx.x == 0 && *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base) != 0) fault |= FHOB_ERR_TMEM_BASE;
  // Everything up to here overlaps the end of the kernel in front; from here on memory is touched.
  pdl_wait();
  if (threadIdx.x == 0) {
    pdl_launch_dependents();
    if (blockIdx.x == 0) *p.status = 0;   // every call starts clean
  }
  // TMEM: the stages of S for A and for B (P in place), then O of A and B
  auto s_cols = [](int x, int stage) { return static_cast<uint32_t>((x * kStages + stage) * BN); };
  auto o_cols = [](int x) { return static_cast<uint32_t>(256 + x * C::O_COLS); };
  // Order of the loads, which is the order in which they are used: K0 K1 V0 K2 V1 ... with two stages,
  // K0 V0 K1 V1 ... with one, K alone without O
  auto k_load = [&](int j) { return !OUT ? j : (kStages == 1 ? 2 * j : (j == 0 ? 0 : 2 * j - 1)); };
  auto v_load = [&](int j) { return kStages == 1 || j == n_tiles - 1 ? 2 * j + 1 : 2 * j + 2; };

  if (warp == FW_TMA_WARP) {
    // ================================================= TMA producer: Q tiles, then K and V tiles
    if (n_tiles > 0 && elect_one()) {
      const int head_b = head / p.heads, head_h = head - head_b * p.heads;   // batch entry and head within it
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (end[x] > begin[x]) {
          mbar_arrive_expect_tx(&bars->q_full[x], C::Q_BYTES);
          load_tile<BM, DQK, BM * 128>(smem + x * C::Q_BYTES, &p.q, &bars->q_full[x], m_of(x), head_h, head_b);
        }
      const int n_loads = n_tiles * (OUT ? 2 : 1);
      int issued = 0;
      for (int i = 0; i < n_loads; ++i) {
        const int slot = i % C::NSLOT;
        if (!wait_bar(&bars->kv_free[slot], ((i / C::NSLOT) & 1) ^ 1, bars, p.status)) break;
        const bool is_v = OUT && (kStages == 1 ? (i & 1) != 0 : i > 0 && (i % 2 == 0 || i == n_loads - 1));
        const int j = !OUT ? i : (kStages == 1 ? i >> 1 : (is_v ? (i - 1) >> 1 : (i + 1) >> 1)), n0 = (t_begin + j) * BN;
        uint8_t* dst = ring + slot * C::SLOT_BYTES;
        if (is_v) {
          mbar_arrive_expect_tx(&bars->kv_full[slot], BN * DV * 2);
          load_tile<BN, DV, BN * 128>(dst, &p.v, &bars->kv_full[slot], n0, head_h, head_b);
        } else {
          mbar_arrive_expect_tx(&bars->kv_full[slot], BN * DQK * 2);
          load_tile<BN, DQK, BN * 128>(dst, &p.k, &bars->kv_full[slot], n0, head_h, head_b);
        }
        issued = i + 1;
      }
      // drain: every load issued above must have landed before the CTA may exit
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (end[x] > begin[x]) wait_landed(&bars->q_full[x], 0, p.status);
      for (int i = issued > C::NSLOT ? issued - C::NSLOT : 0; i < issued; ++i)
        wait_landed(&bars->kv_full[i % C::NSLOT], (i / C::NSLOT) & 1, p.status);
    }
  } else if (warp == MMA_WARP) {
    // ================================================= MMA issuer (one thread: the pipe runs its products in order)
    if (n_tiles > 0 && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(BM, BN, false, false, F16);
      constexpr uint32_t idesc_o = umma_idesc_bf16(BM, kO, false, true, F16);
      constexpr uint32_t idesc_o64 = umma_idesc_bf16(BM, 64, false, true, F16);   // split operands: the hi box alone
      constexpr int kBox = BM * 128;
      const uint32_t q_lo = umma_desc_lo(smem_u32(smem), 16), ring_lo = umma_desc_lo(smem_u32(ring), 16);
      constexpr uint32_t kQ16 = C::Q_BYTES >> 4, kSlot16 = C::SLOT_BYTES >> 4;
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        ok = ok && wait_bar(bar, parity, bars, p.status);
        return ok;
      };
      auto active = [&](int x, int t) { return t >= begin[x] && t < end[x]; };
      // S_x(t) = Q_x . K(t)^T; the slot is handed back after its last product
      auto scores = [&](int x, int t) {
        const int i = k_load(t - t_begin), slot = i % C::NSLOT, it = t - begin[x], stage = it % kStages;
        if (it == 0 && !wait(&bars->q_full[x], 0)) return;
        if (!OUT && !wait(&bars->s_free[x][stage], ((it / kStages) & 1) ^ 1)) return;
        if (!wait(&bars->kv_full[slot], (i / C::NSLOT) & 1)) return;
        tc_fence_after();
        const uint32_t a = q_lo + x * kQ16, b = ring_lo + slot * kSlot16;
        if constexpr (SPLIT) {
#pragma unroll
          for (int term = 0; term < 3; ++term)   // (hi, hi), (hi, lo), (lo, hi)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_ss_split(s_cols(x, stage), a + (((term == 2) * kBox + ks * 32) >> 4), b + (((term == 1) * (BN * 128) + ks * 32) >> 4),
                            kDescHi, idesc_s, term > 0 || ks > 0 ? 1u : 0u);
        } else {
          gemm_ss<DQK, kBox, BN * 128>(s_cols(x, stage), a, b, idesc_s, false);
        }
        umma_commit(&bars->s_full[x][stage]);
        if (x == 1 || !active(1, t)) umma_commit(&bars->kv_free[slot]);
      };
      // O_x += P_x . V(t)
      auto output = [&](int x, int t) {
        const int i = v_load(t - t_begin), slot = i % C::NSLOT, it = t - begin[x], stage = it % kStages;
        if (!wait(kHalves ? &bars->p_half[x] : &bars->p_full[x][stage], (it / kStages) & 1)) return;
        if (!wait(&bars->kv_full[slot], (i / C::NSLOT) & 1)) return;
        tc_fence_after();
        // MN-major: leading byte offset = distance between the tile's 64-column boxes
        const uint32_t b = ring_lo + slot * kSlot16 - (1u << 16) + (static_cast<uint32_t>((BN * 128) >> 4) << 16);
        auto pv = [&](int k0, int k1, bool accumulate) {
#pragma unroll
          for (int ks = k0; ks < k1; ++ks)
            umma_ts_split(o_cols(x), s_cols(x, stage) + 8 * ks, b + ((ks * 2048) >> 4), kDescHi, idesc_o, accumulate || ks > k0 ? 1u : 0u);
        };
        constexpr int kFirst = kHalves ? BN / 32 : BN / 16;
        pv(0, kFirst, it > 0);
        if (kHalves) {
          if (!wait(&bars->p_full[x][stage], it & 1)) return;
          tc_fence_after();
          pv(kFirst, BN / 16, true);
        }
        if (SPLIT) {   // above P_hi . [V_hi | V_lo]; here P_lo . V_hi on top of the second half
#pragma unroll
          for (int ks = 0; ks < BN / 16; ++ks)
            umma_ts_split(o_cols(x) + 64, s_cols(x, stage) + BN / 2 + 8 * ks, b + ((ks * 2048) >> 4), kDescHi, idesc_o64, 1u);
        }
        umma_commit(&bars->o_done[x]);
        if (t + 1 == end[x]) umma_commit(&bars->out_full[x]);
        if (x == 1 || !active(1, t)) umma_commit(&bars->kv_free[slot]);
      };
      if (OUT) {
        for (int t = t_begin; ok && t < t_begin + kStages; ++t)
          for (int x = 0; ok && x < 2; ++x)
            if (active(x, t)) scores(x, t);
        for (int t = t_begin; ok && t < t_end; ++t)
          for (int x = 0; ok && x < 2; ++x) {
            if (active(x, t)) output(x, t);
            if (ok && active(x, t + kStages)) scores(x, t + kStages);
          }
      } else {
        for (int t = t_begin; ok && t < t_end; ++t)
          for (int x = 0; ok && x < 2; ++x)
            if (active(x, t)) scores(x, t);
      }
      if (!ok) {
        // abort path: no tcgen05.mma may still be reading shared memory or TMEM at exit
        umma_commit(&bars->teardown);
        wait_landed(&bars->teardown, 0, p.status);
      }
    }
  } else if (warp >= FW_EW_WARP0) {
    // ================================================= softmax warps: 4-7 query tile A, 8-11 query tile B
    const int x = (warp - FW_EW_WARP0) >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const int m0 = m_of(x), g_row = m0 + row;
    const int n_iter = end[x] - begin[x], t0 = begin[x];
    const float sl2 = p.scale * kLog2e, abs_sl2 = fabsf(sl2);
    // visible keys of this row
    int lo = 0, hi = p.n_k - 1;
    if (p.causal && g_row + off < hi) hi = g_row + off;
    if (p.window > 0 && g_row + off - p.window + 1 > 0) lo = g_row + off - p.window + 1;
    float run_m = -INFINITY, run_l = 0.f;   // reference maximum (log2 domain) and sum of exponentials
    bool ok = true;
    const uint32_t o_addr = lane_base + o_cols(x);

    // One key tile; tiles that need masking take a copy of the code of their own.
    auto step = [&](auto masked_tile, int it, int n0, int stage) {
      ok = __all_sync(0xffffffffu, wait_bar(&bars->s_full[x][stage], (it / kStages) & 1, bars, p.status));
      if (!ok) return;
      tc_fence_after();
      const uint32_t s_addr = lane_base + s_cols(x, stage);
      constexpr int NC = BN / 32;
      uint32_t s[NC][32];
#pragma unroll
      for (int c = 0; c < NC; ++c) tmem_ld32(s_addr + 32 * c, s[c]);
      tmem_wait_ld();
      if (!OUT) {
        tc_fence_before();
        mbar_arrive(&bars->s_free[x][stage]);
      }
      if (sl2 < 0.f) {   // a negative scale: the largest scaled score is the smallest raw one
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int j = 0; j < 32; ++j) s[c][j] ^= 0x80000000u;
      }
      if (decltype(masked_tile)::value) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int idx = n0 + 32 * c + j;
            if (idx < lo || idx > hi) s[c][j] = 0xff800000u;   // -inf
          }
      }
      constexpr int MXC = 4;   // independent chains: a warp has little else to issue here
      float mx[MXC];
#pragma unroll
      for (int i = 0; i < MXC; ++i) {
        mx[i] = fmaxf(__uint_as_float(s[i * NC / MXC][(i * (BN / MXC)) % 32]), __uint_as_float(s[i * NC / MXC][(i * (BN / MXC)) % 32 + 1]));
#pragma unroll
        for (int j = 2; j < BN / MXC; j += 2) {
          const int g = i * (BN / MXC) + j;
          mx[i] = max3(mx[i], __uint_as_float(s[g / 32][g % 32]), __uint_as_float(s[g / 32][g % 32 + 1]));
        }
      }
#pragma unroll
      for (int h = MXC / 2; h > 0; h >>= 1)
#pragma unroll
        for (int i = 0; i < h; ++i) mx[i] = fmaxf(mx[i], mx[i + h]);
      const float raw_m = mx[0];
      const float tile_m = raw_m == -INFINITY ? -INFINITY : raw_m * abs_sl2;
      const bool need = tile_m > run_m + 8.f;   // true for the first finite maximum
      if (__any_sync(0xffffffffu, need)) {
        const float alpha = (need && run_m != -INFINITY) ? ex2(run_m - tile_m) : 1.f;
        if (OUT && it > 0) {
          // O is idle once the previous tile's P V has finished; the next one waits for this tile's P
          ok = __all_sync(0xffffffffu, wait_bar(&bars->o_done[x], (it - 1) & 1, bars, p.status));
          if (!ok) return;
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < kO; c += 16) {
            uint32_t v[16];
            tmem_ld16(o_addr + c, v);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
            tmem_st16(o_addr + c, v);
          }
        }
        run_l *= alpha;
        if (need) run_m = tile_m;
      }
      const float neg_m = run_m == -INFINITY ? 0.f : -run_m;
      const float2 mul = make_float2(abs_sl2, abs_sl2), add = make_float2(neg_m, neg_m);
      float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        [[maybe_unused]] uint32_t w[16], w_lo[16];
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 e = __ffma2_rn(f2(s[c][j], s[c][j + 1]), mul, add);
          // (L alone: one exponential in eight on the FMA pipe is 10 % faster; with P to pack and store, none is)
          float2 pr = !OUT && j % 16 == 0 ? exp2_fma(e) : make_float2(ex2(e.x), ex2(e.y));
          if (decltype(masked_tile)::value) {   // (-inf) * 0 is not a number when the scale is 0
            if (s[c][j] == 0xff800000u) pr.x = 0.f;
            if (s[c][j + 1] == 0xff800000u) pr.y = 0.f;
          }
          sum[(j >> 1) % 2] = __fadd2_rn(sum[(j >> 1) % 2], pr);
          if constexpr (OUT && SPLIT) fw_split_pack(pr.x, pr.y, w[j / 2], w_lo[j / 2]);
          else if constexpr (OUT) w[j / 2] = pack16<F16>(pr.x, pr.y);
        }
        // the row's scores are in registers: P goes over them, 16 packed columns per 32 keys
        if constexpr (OUT) tmem_st16(s_addr + 16 * c, w);
        if constexpr (OUT && SPLIT) tmem_st16(s_addr + BN / 2 + 16 * c, w_lo);
        if (kHalves && c == NC / 2 - 1) {
          tmem_wait_st();
          tc_fence_before();
          mbar_arrive(&bars->p_half[x]);
        }
      }
      run_l += (sum[0].x + sum[1].x) + (sum[0].y + sum[1].y);
      if (OUT) {
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(&bars->p_full[x][stage]);
      }
    };
    for (int it = 0; it < n_iter; ++it) {
      const int n0 = (t0 + it) * BN, stage = it % kStages;
      // does any score of this tile need masking?  (uniform over the tile's warps)
      bool masked = n0 + BN > p.n_k;
      if (p.causal) {
        masked = masked || (n0 + BN - 1 > m0 + off);
        if (p.window > 0) masked = masked || (m0 + BM - 1 + off - n0 >= p.window);
      }
      if (masked) step(std::true_type{}, it, n0, stage);
      else step(std::false_type{}, it, n0, stage);
      if (!ok) break;
    }

    // ---- results
    if (OUT && n_iter > 0) ok = ok && __all_sync(0xffffffffu, wait_bar(&bars->out_full[x], 0, bars, p.status));
    tc_fence_after();
    if (p.split > 1) {
      // this part's row: unscaled O, reference maximum and sum (query tile A only)
      if (x == 0) {
        if (OUT) stage_row<kRes, SPLIT>(reinterpret_cast<float*>(smem) + row * C::kPitch, o_addr, n_iter > 0);
        bars->red[0][row] = run_m;
        bars->red[1][row] = run_l;
      }
    } else if (ok && live(x) && (!OUT || g_row - lane < p.n_q)) {
      // a sum of zero: no visible key (a NaN is kept)
      const float inv_l = run_l == 0.f ? 0.f : 1.f / run_l;
      if (g_row < p.n_q)
        p.lse_out[static_cast<size_t>(head) * p.n_q + g_row] = run_l == 0.f ? -INFINITY : (run_m + log2f(run_l)) * 0.6931471805599453f;
      if (OUT) {
        const size_t at = (static_cast<size_t>(head) * p.n_q + g_row) * p.d_v;
#pragma unroll
        for (int c = 0; c < kRes; c += 16) {
          uint32_t v[16];
          load_result<SPLIT>(o_addr + c, n_iter > 0, v);
          if (g_row < p.n_q) {
            if constexpr (SPLIT) {
#pragma unroll
              for (int j = 0; j < 16; j += 4)   // rows are whole 16-byte pieces
                if (c + j < p.d_v)
                  *reinterpret_cast<float4*>(static_cast<float*>(p.o) + at + c + j) =
                      make_float4(__uint_as_float(v[j]) * inv_l, __uint_as_float(v[j + 1]) * inv_l, __uint_as_float(v[j + 2]) * inv_l,
                                  __uint_as_float(v[j + 3]) * inv_l);
            } else {
#pragma unroll
              for (int j = 0; j < 16; j += 8)
                if (c + j < p.d_v) {
                  uint32_t w[4];
#pragma unroll
                  for (int h = 0; h < 4; ++h)
                    w[h] = pack16<F16>(__uint_as_float(v[j + 2 * h]) * inv_l, __uint_as_float(v[j + 2 * h + 1]) * inv_l);
                  *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.o) + at + c + j) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
          }
        }
      }
    }
  }

  // ---- split keys: every part has its own reference maximum; rows are weighted and added in rank order
  if (p.split > 1) {
    __syncwarp();
    cluster_sync();
    const int tid = threadIdx.x - FW_EW_WARP0 * 32, m0 = m_of(0);
    if (tid >= 0) {
      constexpr int V = SPLIT ? 4 : 8, PIECES = OUT ? kRes / V : 1;
      const int rows = (BM + p.split - 1) / p.split;
      const uint32_t stage = smem_u32(smem), red = smem_u32(&bars->red[0][0]);
      for (int i = tid; i < rows * PIECES; i += EW_THREADS) {
        const int r = part * rows + i / PIECES, c = (i % PIECES) * V;
        if (r >= BM || m0 + r >= p.n_q) continue;
        float m = -INFINITY, l = 0.f;
        for (int q = 0; q < p.split; ++q) m = fmaxf(m, cluster_ld(cluster_map(red + r * 4, q)));
        float4 a[V / 4];
#pragma unroll
        for (int h = 0; h < V / 4; ++h) a[h] = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int q = 0; q < p.split; ++q) {
          const float mq = cluster_ld(cluster_map(red + r * 4, q)), lq = cluster_ld(cluster_map(red + (BM + r) * 4, q));
          const float w = mq == -INFINITY ? 1.f : ex2(mq - m);   // (no maximum but a sum: NaN)
          l = fmaf(lq, w, l);
          if (OUT && lq != 0.f) {   // a part without a visible key has nothing to add
            const uint32_t from = cluster_map(stage + (r * C::kPitch + c) * 4, q);
#pragma unroll
            for (int h = 0; h < V / 4; ++h) {
              const float4 y = cluster_ld4(from + 16 * h);
              a[h].x = fmaf(y.x, w, a[h].x); a[h].y = fmaf(y.y, w, a[h].y);
              a[h].z = fmaf(y.z, w, a[h].z); a[h].w = fmaf(y.w, w, a[h].w);
            }
          }
        }
        const size_t g = static_cast<size_t>(head) * p.n_q + m0 + r;
        if (c == 0) p.lse_out[g] = l == 0.f ? -INFINITY : (m + log2f(l)) * 0.6931471805599453f;
        if (OUT && c < p.d_v) {
          const float inv_l = l == 0.f ? 0.f : 1.f / l;
          if constexpr (SPLIT)
            *reinterpret_cast<float4*>(static_cast<float*>(p.o) + g * p.d_v + c) = make_float4(a[0].x * inv_l, a[0].y * inv_l, a[0].z * inv_l, a[0].w * inv_l);
          else
            *reinterpret_cast<uint4*>(static_cast<uint16_t*>(p.o) + g * p.d_v + c) =
                make_uint4(pack16<F16>(a[0].x * inv_l, a[0].y * inv_l), pack16<F16>(a[0].z * inv_l, a[0].w * inv_l),
                           pack16<F16>(a[V / 4 - 1].x * inv_l, a[V / 4 - 1].y * inv_l), pack16<F16>(a[V / 4 - 1].z * inv_l, a[V / 4 - 1].w * inv_l));
        }
      }
    }
    cluster_sync();   // the others are done with this CTA's shared memory
  }

  // ---- teardown
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(0, TMEM_COLS);
  }
  if (threadIdx.x == 0 && fault) atomicOr(p.status, fault);
}

// ------------------------------------------------------------------ host side
template <int DQK, int DV, bool F16, bool SPLIT, bool OUT>
int fw_launch(const FhobProblem& p, void* o_out, float* lse_out, int* status, cudaStream_t s) {
  using C = FwCfg<DQK, DV, OUT>;
  constexpr auto kernel = fw_kernel<DQK, DV, F16, SPLIT, OUT>;
  FwParams tp;
  memset(&tp, 0, sizeof(tp));
  const int dv = head_dim_v(p);
  const void *q = p.q, *k = p.k, *v = p.v;
  View vq = tensor_view(p, kTenQ, p.n_q, p.d), vk = tensor_view(p, kTenK, p.n_k, p.d), vv = tensor_view(p, kTenV, p.n_k, dv);
  if (SPLIT) {   // the bf16 hi/lo copies the caller of this function left in the workspace
    SplitBuffers sb = split_buffers(p);
    q = sb.q; k = sb.k; v = sb.v;
    vq = contiguous_view(p.bh, p.n_q, 128);
    vk = vv = contiguous_view(p.bh, p.n_k, 128);
  }
  int st = make_map(&tp.q, q, vq, p.n_q, SPLIT ? 128 : p.d, F16);
  if (st == FHOB_OK) st = make_map(&tp.k, k, vk, p.n_k, SPLIT ? 128 : p.d, F16);
  if (st == FHOB_OK && OUT) st = make_map(&tp.v, v, vv, p.n_k, SPLIT ? 128 : dv, F16);
  if (st == FHOB_OK) st = allow_smem(kernel, C::SMEM_BYTES);
  if (st != FHOB_OK) return st;
  tp.lse_out = lse_out;
  tp.o = o_out;
  tp.status = status;
  tp.n_q = p.n_q; tp.n_k = p.n_k; tp.causal = p.causal; tp.window = p.window;
  tp.heads = (!SPLIT && p.layout) ? p.layout->heads : p.bh;
  tp.d_v = dv;
  tp.scale = p.scale;
  const int tiles = (p.n_q + BM - 1) / BM;
  if (static_cast<long long>(tiles) * p.bh > 0x7fffffffLL) return FHOB_ERR_SHAPE;
  // A head of one query tile may split its keys (a second tile would cost the parts more than they save).
  tp.split = tiles == 1 ? tc_parts(p.n_q, p.n_k, p.window) : 1;
  // Two query tiles a CTA hide each other's latency and share K and V; a tile takes as long alone, so
  // when single tiles fit the GPU at once, a CTA has one.  (The bits are the same.)
  tp.q_tiles = tiles == 1 || static_cast<long long>(tiles) * p.bh <= sm_count() ? 1 : 2;
  tp.groups = (tiles + tp.q_tiles - 1) / tp.q_tiles;
  tp.items = tp.groups * p.bh;
  const long long blocks = static_cast<long long>(tp.items) * tp.split;
  if (blocks > 0x7fffffffLL) return FHOB_ERR_SHAPE;
  FHOB_CUDA_OK(launch_pdl(kernel, static_cast<unsigned>(blocks), FW_THREADS, C::SMEM_BYTES, tp.split, s, tp));
  return FHOB_OK;
}

template <int DQK, int DV, bool F16, bool SPLIT = false>
int fw_dispatch(const FhobProblem& p, void* o_out, float* lse_out, int* status, cudaStream_t s) {
  // no O wanted: the scores alone (no tile of the second head dim is touched)
  return o_out ? fw_launch<DQK, DV, F16, SPLIT, true>(p, o_out, lse_out, status, s)
               : fw_launch<DQK, DQK, F16, SPLIT, false>(p, o_out, lse_out, status, s);
}

template <bool F16>
int fw_dims(const FhobProblem& p, void* o_out, float* lse_out, int* status, cudaStream_t s) {
  // tile widths: the head dims rounded up to 64 or 128
  const int dv = head_dim_v(p);
  if (p.d <= 64)
    return dv <= 64 ? fw_dispatch<64, 64, F16>(p, o_out, lse_out, status, s) : fw_dispatch<64, 128, F16>(p, o_out, lse_out, status, s);
  return dv <= 64 ? fw_dispatch<128, 64, F16>(p, o_out, lse_out, status, s) : fw_dispatch<128, 128, F16>(p, o_out, lse_out, status, s);
}

}  // namespace

int tc_forward(const FhobProblem& p, void* o_out, float* lse_out, int* status, cudaStream_t s) {
  if (!tc_first_order_supported(p)) return FHOB_ERR_SHAPE;
  int st = check_device();
  if (st != FHOB_OK) return st;
  if (p.dtype == FHOB_F32) {
    st = tc_split_inputs(p, s, kSplitQ | kSplitK | (o_out ? kSplitV : 0));
    return st != FHOB_OK ? st : fw_dispatch<128, 128, false, true>(p, o_out, lse_out, status, s);
  }
  return p.dtype == FHOB_F16 ? fw_dims<true>(p, o_out, lse_out, status, s) : fw_dims<false>(p, o_out, lse_out, status, s);
}

}  // namespace fhob
