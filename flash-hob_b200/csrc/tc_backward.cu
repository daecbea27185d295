// First backward of attention on the tensor cores (sm_100a): dQ, dK, dV from the saved forward results,
// the first-order half of a twice-differentiable attention function.  Role of the reference's dense
// backward (fhog/triton_flash.py:190-220), at O(N) memory; the maths is jax_refs/flash_impl.py:124-173
// with P = exp(S - L) and D = rowsum(dO * O).
//
//   BQ (queries stationary): dS = P (dP - D), dP = dO V^T;   dQ += dS K            3 products
//   BK (keys stationary):    the same tiles transposed;      dV += P^T dO, dK += dS^T Q    4 products
//
// Both halves are one launch (neither needs the other), after the pre-pass that leaves -L*log2(e) and -D.
// One thread issues all products of a CTA.  S has one accumulator, which is free again as soon as the
// elementwise warps have it in registers: the 16-bit tiles (dS, and in BK P) go into dP's columns, of
// which there are two or three in turn, and are the A operands of the output products from there:
//
//     tensor pipe:   S(t+1) | outputs(t) | dP(t+ND) | S(t+2) | outputs(t+1) ...
//     elementwise:   S(t), dP(t) -> P, dS (t)       | S(t+1), dP(t+1) -> ...
//
// so dP is ND tiles ahead and S one, and no wait is for something that waits for its result.
// What bounds it: BQ 128 keys a tile at head dim 128: 1 536 cycles of tensor pipe; BK 64 queries a tile
// (TMEM has no room for more beside dK and dV): 1 280; the elementwise warps need about as long.  The two
// streamed tensors have rings of their own, because V is done with after dP and K only after dQ.
#include <type_traits>

#include "tc_common.cuh"

namespace fhob {
namespace {

constexpr int BW_TAIL = 1024;   // barriers, TMEM base, abort flag
constexpr int BW_RING = 5;      // most slots of a ring

// Two head dims: the first stationary and the first streamed tile are q/k-side tensors (DQK columns), the
// second ones v-side tensors (DV columns).  BQ: Q, dO | K, V.  BK: K, V | Q, dO.
// SPLIT: fp32 operands as bf16 hi + lo pairs, rows [hi(64) | lo(64)] = the two boxes of a 128-wide tile, three
// products per contraction (see tc_kernels.cu); 64 columns a result.  A result's accumulator has 128 columns:
// hi.hi in the first 64, hi.lo and lo.hi in the others, added up at the end.  The tensor core cuts off low bits
// every time it adds to an accumulator, so the two small terms must not be added to the large one tile by
// tile: with all three in 64 columns dV of 8 causal heads N = 2048 is off by 1.25e-5, this way by 7.1e-6.
template <bool KSIDE, int DQK, int DV, bool SPLIT>
struct BwCfg {
  static constexpr int OUT0 = DQK;                                       // TMEM columns of dQ | dK
  static constexpr int OUT1 = KSIDE ? DV : 0;                            // dV
  static constexpr int OUT_COLS = OUT0 + OUT1;
  static constexpr int W0 = SPLIT ? 64 : OUT0, W1 = SPLIT && KSIDE ? 64 : OUT1;   // columns of the results
  // 128 streamed rows a tile if S and two dP of that width fit beside the results
  static constexpr int BN = OUT_COLS + 3 * 128 <= TMEM_COLS && !(SPLIT && KSIDE) ? 128 : 64;
  // split P and dS do not fit dP's columns together: P goes over S then, and S has as many stages as dP
  static constexpr bool P_OVER_S = SPLIT && KSIDE;
  static constexpr int ND = BN == 128 || P_OVER_S ? 2 : 3;
  static constexpr int NS = P_OVER_S ? ND : 1;
  static constexpr int S_COL = OUT_COLS, DP_COL = OUT_COLS + NS * BN;
  static constexpr int STAT0 = BM * DQK * 2, STAT1 = BM * DV * 2;
  static constexpr int VEC_BYTES = KSIDE ? 2 * BN * 4 : 0;               // BK: -L*log2e and -D of the streamed queries
  static constexpr int TILE0 = BN * DQK * 2, TILE1 = BN * DV * 2;
  static constexpr int SLOT0 = TILE0 + (KSIDE ? 1024 : 0), SLOT1 = TILE1;   // tiles stay 1024-byte aligned
  static constexpr int ROOM = SMEM_LIMIT - BW_TAIL - STAT0 - STAT1;
  // the second ring first (its tiles are loaded first), the rest to the first
  static constexpr int N1_FIT = ROOM / (SLOT0 + SLOT1), N1 = N1_FIT > BW_RING ? BW_RING : N1_FIT;
  static constexpr int N0_FIT = (ROOM - N1 * SLOT1) / SLOT0, N0 = N0_FIT > BW_RING ? BW_RING : N0_FIT;
  static constexpr int SMEM_BYTES = STAT0 + STAT1 + N0 * SLOT0 + N1 * SLOT1 + BW_TAIL;
  static constexpr int kPitch = W0 + W1 + 4;                             // floats per row of the staging area (split streamed axis)
  static_assert(DP_COL + ND * BN <= TMEM_COLS, "TMEM budget");
  static_assert(N0 >= 2 && N0 >= NS && N1 >= ND, "slots of a ring: the issuing thread is ND tiles ahead with dP, NS with S");
  static_assert(BM * kPitch * 4 <= SMEM_BYTES - BW_TAIL, "staging area");
};

enum { kBwQ = 0, kBwDO, kBwK, kBwV, kBwMaps };

struct BwParams {
  CUtensorMap map[kBwMaps];
  const float* nlc;   // -L*log2(e) per query
  const float* k1;    // -D per query
  void *dq, *dk, *dv;
  int* status;
  int n_q, n_k, causal, window;
  int tiles_q, tiles_k;   // 128-row tiles of a head
  int items_q, items_k;   // (head, tile) pairs of the two halves
  int q_blocks;           // the first q_blocks CTAs are BQ
  int split_q, split_k;   // CTAs that share the streamed tiles of one pair
  int cluster;            // CTAs of a cluster (a multiple of both)
  int heads;              // heads per batch entry of the input tensor maps (4-D: columns, rows, head, batch)
  int d, d_v;             // columns in memory (<= the tile widths; see bw_launch)
  float scale;
};

struct BwBars {
  uint64_t stat_full;
  uint64_t full0[BW_RING], free0[BW_RING];   // rings of the streamed tensors
  uint64_t full1[BW_RING], free1[BW_RING];
  uint64_t s_full[3], dp_full[3];            // scores of a stage finished
  uint64_t s_free;                           // S is in registers
  uint64_t p_full[3];                        // 16-bit tiles of a stage written
  uint64_t out_full;
  uint64_t teardown;
  uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(BwBars) <= BW_TAIL, "tail");

__device__ __forceinline__ void bw_split_pack(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(x, y);
  lo = pack_bf16(x - __uint_as_float(hi << 16), y - __uint_as_float(hi & 0xffff0000u));
}

// One half over one 128-row tile of one head; `block` numbers the (head, tile, part) triples.
template <bool KSIDE, int DQK, int DV, bool F16, bool SPLIT>
__device__ __forceinline__ void bw_body(const BwParams& p, int block) {
  using C = BwCfg<KSIDE, DQK, DV, SPLIT>;
  static_assert(!SPLIT || (DQK == 128 && DV == 128 && !F16), "split fp32 operands are [hi(64) | lo(64)] bf16 rows");
  constexpr int BN = C::BN, CPT = BN / 2;   // CPT: columns of a score tile per elementwise thread
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* ring0 = smem + C::STAT0 + C::STAT1;
  uint8_t* ring1 = ring0 + C::N0 * C::SLOT0;
  BwBars* bars = reinterpret_cast<BwBars*>(ring1 + C::N1 * C::SLOT1);
  int* status = p.status;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = KSIDE ? p.split_k : p.split_q;
  const CtaWork work = cta_work(block, split, KSIDE ? p.items_k : p.items_q);   // the grid is padded to whole clusters
  const int item = work.item, part = work.part;
  const bool live = work.live;
  const int tiles_per_head = KSIDE ? p.tiles_k : p.tiles_q;
  const int head = item / tiles_per_head;
  const int tile_in_head = item - head * tiles_per_head;
  const int tile = KSIDE ? tile_in_head : tiles_per_head - 1 - tile_in_head;  // causal: longest first
  const int m0 = tile * BM;
  const int n_stat = KSIDE ? p.n_k : p.n_q, n_strm = KSIDE ? p.n_q : p.n_k;
  const int off = p.n_k - p.n_q;
  int t_begin, t_end;
  visible_tiles(!KSIDE, m0, BM, BN, n_strm, off, p.causal, p.window, t_begin, t_end);
  if (split > 1) split_range(part, split, t_begin, t_end);
  const int n_iter = live ? t_end - t_begin : 0;
  auto stat_map = [&](int i) { return &p.map[KSIDE ? kBwK + i : kBwQ + i]; };   // Q, dO | K, V
  auto strm_map = [&](int i) { return &p.map[KSIDE ? kBwQ + i : kBwK + i]; };

  int fault = 0;   // thread 0: what to report at the end
  if (threadIdx.x == 0) {
    if (smem_u32(smem) & 1023u) fault |= FHOB_ERR_SMEM_ALIGN;
    mbar_init(&bars->stat_full, 1);
    for (int i = 0; i < BW_RING; ++i) {
      mbar_init(&bars->full0[i], 1);
      mbar_init(&bars->free0[i], 1);
      mbar_init(&bars->full1[i], 1);
      mbar_init(&bars->free1[i], 1);
    }
    for (int i = 0; i < 3; ++i) {
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->dp_full[i], 1);
      mbar_init(&bars->p_full[i], EW_THREADS);
    }
    mbar_init(&bars->s_free, EW_THREADS);
    mbar_init(&bars->out_full, 1);
    mbar_init(&bars->teardown, 1);
    bars->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == MMA_WARP) {
    tmem_alloc(&bars->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  if (warp == TMA_WARP && lane == 0)
    for (int i = 0; i < kBwMaps; ++i) prefetch_tensormap(&p.map[i]);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // the CTA allocates all 512 columns, so the allocation starts at column 0 (checked)
  if (threadIdx.x == 0 && *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base) != 0) fault |= FHOB_ERR_TMEM_BASE;
  // Everything up to here overlaps the end of the kernel in front; from here on memory is touched.
  pdl_wait();
  if (threadIdx.x == 0) pdl_launch_dependents();

  if (warp == TMA_WARP) {
    // ================================================= TMA producer
    if (n_iter > 0 && elect_one()) {
      const int head_b = head / p.heads, head_h = head - head_b * p.heads;   // batch entry and head within it
      if (KSIDE) fence_proxy_async_global();   // the row vectors the bulk copies read were written by the kernel in front
      mbar_arrive_expect_tx(&bars->stat_full, C::STAT0 + C::STAT1);
      load_tile<BM, DQK, BM * 128>(smem, stat_map(0), &bars->stat_full, m0, head_h, head_b);
      load_tile<BM, DV, BM * 128>(smem + C::STAT0, stat_map(1), &bars->stat_full, m0, head_h, head_b);
      int issued0 = 0, issued1 = 0;
      for (int it = 0; it < n_iter; ++it) {
        const int n0 = (t_begin + it) * BN, s1 = it % C::N1, s0 = it % C::N0;
        if (!wait_bar(&bars->free1[s1], ((it / C::N1) & 1) ^ 1, bars, status)) break;
        mbar_arrive_expect_tx(&bars->full1[s1], C::TILE1);
        load_tile<BN, DV, BN * 128>(ring1 + s1 * C::SLOT1, strm_map(1), &bars->full1[s1], n0, head_h, head_b);
        issued1 = it + 1;
        if (!wait_bar(&bars->free0[s0], ((it / C::N0) & 1) ^ 1, bars, status)) break;
        mbar_arrive_expect_tx(&bars->full0[s0], C::TILE0 + C::VEC_BYTES);
        uint8_t* dst = ring0 + s0 * C::SLOT0;
        load_tile<BN, DQK, BN * 128>(dst, strm_map(0), &bars->full0[s0], n0, head_h, head_b);
        if (KSIDE) {
          const size_t vo = static_cast<size_t>(head) * row_stride(p.n_q) + n0;
          bulk_load(dst + C::TILE0, p.nlc + vo, BN * 4, &bars->full0[s0]);
          bulk_load(dst + C::TILE0 + BN * 4, p.k1 + vo, BN * 4, &bars->full0[s0]);
        }
        issued0 = it + 1;
      }
      // drain: every load issued above must have landed before the CTA may exit
      wait_landed(&bars->stat_full, 0, status);
      for (int i = issued1 > C::N1 ? issued1 - C::N1 : 0; i < issued1; ++i) wait_landed(&bars->full1[i % C::N1], (i / C::N1) & 1, status);
      for (int i = issued0 > C::N0 ? issued0 - C::N0 : 0; i < issued0; ++i) wait_landed(&bars->full0[i % C::N0], (i / C::N0) & 1, status);
    }
  } else if (warp == MMA_WARP) {
    // ================================================= MMA issuer (one thread: the pipe runs its products in order)
    if (n_iter > 0 && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(BM, BN, false, false, F16);
      constexpr uint32_t idesc_o0 = umma_idesc_bf16(BM, C::OUT0, false, true, F16);                 // dQ | dK
      constexpr uint32_t idesc_o1 = umma_idesc_bf16(BM, C::OUT1 ? C::OUT1 : 64, false, true, F16);  // dV
      constexpr uint32_t idesc_o64 = umma_idesc_bf16(BM, 64, false, true, F16);                     // split operands: the hi box alone
      constexpr int kStatBox = BM * 128, kBox = BN * 128;
      const uint32_t stat0 = umma_desc_lo(smem_u32(smem), 16), stat1 = stat0 + (C::STAT0 >> 4);
      const uint32_t r0 = umma_desc_lo(smem_u32(ring0), 16), r1 = umma_desc_lo(smem_u32(ring1), 16);
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        ok = ok && wait_bar(bar, parity, bars, status);
        return ok;
      };
      auto tile0 = [&](int t) { return r0 + (t % C::N0) * (C::SLOT0 >> 4); };
      auto tile1 = [&](int t) { return r1 + (t % C::N1) * (C::SLOT1 >> 4); };
      auto wait0 = [&](int t) { return wait(&bars->full0[t % C::N0], (t / C::N0) & 1); };
      auto wait1 = [&](int t) { return wait(&bars->full1[t % C::N1], (t / C::N1) & 1); };
      // score product over KD columns (or over the hi/lo boxes of split operands)
      auto scores = [&](auto kd, uint32_t d, uint32_t a, uint32_t b) {
        if constexpr (SPLIT) {
#pragma unroll
          for (int term = 0; term < 3; ++term)   // (hi, hi), (hi, lo), (lo, hi)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              umma_ss_split(d, a + (((term == 2) * kStatBox + ks * 32) >> 4), b + (((term == 1) * kBox + ks * 32) >> 4), kDescHi, idesc_s,
                            term > 0 || ks > 0 ? 1u : 0u);
        } else {
          gemm_ss<decltype(kd)::value, kStatBox, kBox>(d, a, b, idesc_s, false);
        }
      };
      auto s_of = [&](int t) {
        scores(std::integral_constant<int, DQK>{}, C::S_COL + (t % C::NS) * BN, stat0, tile0(t));
        umma_commit(&bars->s_full[t % C::NS]);
      };
      auto dp_of = [&](int t) {
        scores(std::integral_constant<int, DV>{}, C::DP_COL + (t % C::ND) * BN, stat1, tile1(t));
        umma_commit(&bars->dp_full[t % C::ND]);
        if (!KSIDE) umma_commit(&bars->free1[t % C::N1]);   // V is done with
      };
      // output product, A = 16-bit tile in TMEM (lo half `lo` columns on), B = streamed tile read MN-major
      // (leading byte offset = distance between its 64-column boxes)
      auto outputs = [&](uint32_t out, uint32_t a, int lo, uint32_t tile, uint32_t idesc, bool accumulate) {
        const uint32_t b = tile - (1u << 16) + (static_cast<uint32_t>(kBox >> 4) << 16);
        gemm_ts<BN>(out, a, b, idesc, accumulate);
        if constexpr (SPLIT) gemm_ts<BN>(out + 64, a + lo, b, idesc_o64, true);   // hi . [hi | lo] above, lo . hi here
      };
      wait(&bars->stat_full, 0);
      for (int t = 0; ok && t < C::ND && t < n_iter; ++t) {
        if (!wait1(t)) break;
        tc_fence_after();
        dp_of(t);
        if (t < C::NS) {
          if (!wait0(t)) break;
          tc_fence_after();
          s_of(t);
        }
      }
      for (int t = 0; ok && t < n_iter; ++t) {
        if (!C::P_OVER_S && t + 1 < n_iter) {
          if (!wait(&bars->s_free, t & 1) || !wait0(t + 1)) break;
          tc_fence_after();
          s_of(t + 1);
        }
        if (!wait(&bars->p_full[t % C::ND], (t / C::ND) & 1)) break;
        tc_fence_after();
        const uint32_t dp = C::DP_COL + (t % C::ND) * BN;
        constexpr int kLo = BN / 4;   // split tiles: the lo half starts this many columns after the hi half
        if (KSIDE) {
          const uint32_t pcol = C::P_OVER_S ? C::S_COL + (t % C::NS) * BN : dp + BN / 4;
          outputs(C::OUT0, pcol, kLo, tile1(t), idesc_o1, t > 0);   // dV += P^T . dO
        }
        outputs(0, dp, kLo, tile0(t), idesc_o0, t > 0);             // dQ += dS . K | dK += dS^T . Q
        umma_commit(&bars->free0[t % C::N0]);
        if (KSIDE) umma_commit(&bars->free1[t % C::N1]);
        if (t + C::ND < n_iter) {
          if (!wait1(t + C::ND)) break;
          tc_fence_after();
          dp_of(t + C::ND);
          if (C::P_OVER_S) {
            if (!wait0(t + C::ND)) break;
            tc_fence_after();
            s_of(t + C::ND);
          }
        }
      }
      if (ok) {
        umma_commit(&bars->out_full);
      } else {
        // abort path: no tcgen05.mma may still be reading shared memory or TMEM at exit
        umma_commit(&bars->teardown);
        wait_landed(&bars->teardown, 0, status);
      }
    }
  } else if (warp >= EW_WARP0) {
    // ================================================= elementwise warps
    const int quad = warp & 3, half = (warp - EW_WARP0) >> 2;
    const int row = quad * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quad * 32) << 16;
    const int g_row = m0 + row;  // stationary row of this thread
    const float sl2 = p.scale * kLog2e;
    float r_nlc = 0.f, r_k1 = 0.f;
    if (!KSIDE && g_row < p.n_q) {
      const size_t vi = static_cast<size_t>(head) * row_stride(p.n_q) + g_row;
      r_nlc = p.nlc[vi];
      r_k1 = p.k1[vi];
    }
    // visible streamed index range of this thread's row
    int lo, hi;
    if (!KSIDE) {
      lo = 0;
      hi = p.n_k - 1;
      if (p.causal && g_row + off < hi) hi = g_row + off;
      if (p.window > 0 && g_row + off - p.window + 1 > 0) lo = g_row + off - p.window + 1;
    } else {
      lo = p.causal ? g_row - off : 0;
      if (lo < 0) lo = 0;
      hi = p.n_q - 1;
      if (p.window > 0 && g_row - off + p.window - 1 < hi) hi = g_row - off + p.window - 1;
    }
    bool ok = true;
    constexpr int NC = CPT / 32;

    // One streamed tile; tiles that need masking take a copy of the code of their own.
    auto step = [&](auto masked_tile, int it, int col_base) {
      constexpr bool kMasked = decltype(masked_tile)::value;
      const int ns = it % C::NS, nd = it % C::ND;
      uint32_t sv = 0;
      if (KSIDE) {
        // the slot's vectors were written by the TMA unit: observe its barrier before reading them
        ok = __all_sync(0xffffffffu, wait_bar(&bars->full0[it % C::N0], (it / C::N0) & 1, bars, status));
        if (!ok) return;
        sv = smem_u32(ring0 + (it % C::N0) * C::SLOT0 + C::TILE0) + half * CPT * 4;
      }
      ok = __all_sync(0xffffffffu, wait_bar(&bars->s_full[ns], (it / C::NS) & 1, bars, status));
      if (!ok) return;
      tc_fence_after();
      const uint32_t s_addr = lane_base + C::S_COL + ns * BN + half * CPT;
      const uint32_t dp_addr = lane_base + C::DP_COL + nd * BN + half * CPT;
      uint32_t s[NC][32];
#pragma unroll
      for (int c = 0; c < NC; ++c) tmem_ld32(s_addr + 32 * c, s[c]);
      tmem_wait_ld();
      if (!C::P_OVER_S) {
        tc_fence_before();
        mbar_arrive(&bars->s_free);
      }
      ok = __all_sync(0xffffffffu, wait_bar(&bars->dp_full[nd], (it / C::ND) & 1, bars, status));
      if (!ok) return;
      tc_fence_after();
      // the 16-bit tiles: dS in the first, P in the second half of the thread's dP columns (split: hi and lo
      // halves of dS there, of P over S).  All of dP is in registers before the first of them is written.
      uint32_t dp[NC][32];
#pragma unroll
      for (int c = 0; c < NC; ++c) tmem_ld32(dp_addr + 32 * c, dp[c]);
      tmem_wait_ld();
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        [[maybe_unused]] uint32_t w_p[16], w_ds[16], w_p_lo[16], w_ds_lo[16];
#pragma unroll
        for (int j4 = 0; j4 < 8; ++j4) {
          float c_nlc[4], c_k1[4];
          if (!KSIDE) {
#pragma unroll
            for (int e = 0; e < 4; ++e) { c_nlc[e] = r_nlc; c_k1[e] = r_k1; }
          } else {
            load4(sv + (32 * c + 4 * j4) * 4, c_nlc);
            load4(sv + (BN + 32 * c + 4 * j4) * 4, c_k1);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int j = 4 * j4 + 2 * h;
            const float2 arg = __ffma2_rn(f2(s[c][j], s[c][j + 1]), make_float2(sl2, sl2), make_float2(c_nlc[2 * h], c_nlc[2 * h + 1]));
            float2 pr = make_float2(ex2(arg.x), ex2(arg.y));
            const float2 dpp = __fadd2_rn(f2(dp[c][j], dp[c][j + 1]), make_float2(c_k1[2 * h], c_k1[2 * h + 1]));
            float2 ds = __fmul2_rn(pr, dpp);
            if (kMasked) {
              const int idx = col_base + 32 * c + j;
              const bool ok0 = idx >= lo && idx <= hi, ok1 = idx + 1 >= lo && idx + 1 <= hi;
              pr.x = ok0 ? pr.x : 0.f; pr.y = ok1 ? pr.y : 0.f;
              ds.x = ok0 ? ds.x : 0.f; ds.y = ok1 ? ds.y : 0.f;
            }
            if constexpr (SPLIT) {
              bw_split_pack(ds.x, ds.y, w_ds[j / 2], w_ds_lo[j / 2]);
              if constexpr (KSIDE) bw_split_pack(pr.x, pr.y, w_p[j / 2], w_p_lo[j / 2]);
            } else {
              w_ds[j / 2] = pack16<F16>(ds.x, ds.y);
              if constexpr (KSIDE) w_p[j / 2] = pack16<F16>(pr.x, pr.y);
            }
          }
        }
        tmem_st16(dp_addr + 16 * c, w_ds);
        if constexpr (SPLIT) tmem_st16(dp_addr + CPT / 2 + 16 * c, w_ds_lo);
        if constexpr (KSIDE && !SPLIT) tmem_st16(dp_addr + CPT / 2 + 16 * c, w_p);
        if constexpr (KSIDE && SPLIT) {
          tmem_st16(s_addr + 16 * c, w_p);
          tmem_st16(s_addr + CPT / 2 + 16 * c, w_p_lo);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(&bars->p_full[nd]);
    };

    for (int it = 0; it < n_iter; ++it) {
      const int n0 = (t_begin + it) * BN;
      bool masked = n0 + BN > n_strm;
      if (p.causal) {
        if (!KSIDE) masked = masked || (n0 + BN - 1 > m0 + off);
        else masked = masked || (n0 + off < m0 + BM - 1);
        if (p.window > 0) {
          if (!KSIDE) masked = masked || (m0 + BM - 1 + off - n0 >= p.window);
          else masked = masked || (n0 + BN - 1 + off - m0 >= p.window);
        }
      }
      if (masked) step(std::true_type{}, it, n0 + half * CPT);
      else step(std::false_type{}, it, n0 + half * CPT);
      if (!ok) break;
    }

    // ---- results
    if (n_iter > 0) ok = ok && __all_sync(0xffffffffu, wait_bar(&bars->out_full, 0, bars, status));
    tc_fence_after();
    if (split > 1) {
      float* dst = reinterpret_cast<float*>(smem) + row * C::kPitch;   // every tile has been read: out_full follows the last product
      stage_row<C::W0 / 2, SPLIT>(dst + half * (C::W0 / 2), lane_base + half * (C::W0 / 2), n_iter > 0);
      if constexpr (KSIDE) stage_row<C::W1 / 2, SPLIT>(dst + C::W0 + half * (C::W1 / 2), lane_base + C::OUT0 + half * (C::W1 / 2), n_iter > 0);
    } else if (ok && live) {
      // `width` columns from TMEM column col0 on; dS was stored without the scale
      auto store_out = [&](auto width, int d_mem, uint32_t col0, void* base, float mul) {
        constexpr int W = decltype(width)::value;   // columns of the result; d_mem <= W of them exist in memory
        const size_t at = (static_cast<size_t>(head) * n_stat + g_row) * d_mem;
#pragma unroll
        for (int c = half * (W / 2); c < (half + 1) * (W / 2); c += 16) {
          uint32_t v[16];
          load_result<SPLIT>(lane_base + col0 + c, n_iter > 0, v);
          if (g_row >= n_stat) continue;
          if constexpr (SPLIT) {
#pragma unroll
            for (int j = 0; j < 16; j += 4)   // rows are whole 16-byte pieces
              if (c + j < d_mem)
                *reinterpret_cast<float4*>(static_cast<float*>(base) + at + c + j) =
                    make_float4(__uint_as_float(v[j]) * mul, __uint_as_float(v[j + 1]) * mul, __uint_as_float(v[j + 2]) * mul, __uint_as_float(v[j + 3]) * mul);
          } else {
#pragma unroll
            for (int j = 0; j < 16; j += 8)
              if (c + j < d_mem) {
                uint32_t w[4];
#pragma unroll
                for (int h = 0; h < 4; ++h) w[h] = pack16<F16>(__uint_as_float(v[j + 2 * h]) * mul, __uint_as_float(v[j + 2 * h + 1]) * mul);
                *reinterpret_cast<uint4*>(static_cast<uint16_t*>(base) + at + c + j) = make_uint4(w[0], w[1], w[2], w[3]);
              }
          }
        }
      };
      store_out(std::integral_constant<int, C::W0>{}, p.d, 0, KSIDE ? p.dk : p.dq, p.scale);
      if constexpr (KSIDE) store_out(std::integral_constant<int, C::W1>{}, p.d_v, C::OUT0, p.dv, 1.f);
    }
  }

  // ---- split streamed axis: add up the parts
  if (p.cluster > 1) {
    __syncwarp();
    cluster_sync();
    const int tid = threadIdx.x - EW_WARP0 * 32, rank0 = static_cast<int>(cluster_rank()) - part;
    if (split > 1 && live && tid >= 0) {
      reduce_store<C::W0, SPLIT, F16>(smem_u32(smem), C::kPitch, 0, rank0, part, split, tid, KSIDE ? p.dk : p.dq, head, m0, n_stat, p.d, p.scale);
      if constexpr (KSIDE) reduce_store<C::W1, SPLIT, F16>(smem_u32(smem), C::kPitch, C::W0, rank0, part, split, tid, p.dv, head, m0, n_stat, p.d_v, 1.f);
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
  if (threadIdx.x == 0 && fault) atomicOr(status, fault);
}

template <int DQK, int DV, bool F16, bool SPLIT>
__global__ void __launch_bounds__(NTHREADS, 1) bw_kernel(const __grid_constant__ BwParams p) {
  const int block = blockIdx.x;
  if (block < p.q_blocks) bw_body<false, DQK, DV, F16, SPLIT>(p, block);
  else bw_body<true, DQK, DV, F16, SPLIT>(p, block - p.q_blocks);
}

// ------------------------------------------------------------------ host side
template <int DQK, int DV, bool F16, bool SPLIT = false>
int bw_launch(const FhobProblem& p, void* dq, void* dk, void* dv, cudaStream_t s) {
  constexpr auto kernel = bw_kernel<DQK, DV, F16, SPLIT>;
  using CQ = BwCfg<false, DQK, DV, SPLIT>;
  using CK = BwCfg<true, DQK, DV, SPLIT>;
  constexpr int kSmem = CQ::SMEM_BYTES > CK::SMEM_BYTES ? CQ::SMEM_BYTES : CK::SMEM_BYTES;
  RowVectors rv = row_vectors(p);
  BwParams tp;
  memset(&tp, 0, sizeof(tp));
  const void* mats[kBwMaps] = {p.q, p.d_o, p.k, p.v};
  const int ids[kBwMaps] = {kTenQ, kTenDO, kTenK, kTenV};
  if (SPLIT) {
    // the bf16 hi/lo copies the caller of this function left in the workspace
    SplitBuffers sb = split_buffers(p);
    mats[kBwQ] = sb.q; mats[kBwDO] = sb.d_o; mats[kBwK] = sb.k; mats[kBwV] = sb.v;
  }
  for (int i = 0; i < kBwMaps; ++i) {
    const int n = i < kBwK ? p.n_q : p.n_k;
    // head dims below the tile widths: the boxes reach past the end of a row and are zero-filled there
    const int d = SPLIT ? 128 : (i == kBwDO || i == kBwV ? head_dim_v(p) : p.d);
    // where each input lives: the caller's layout, or contiguous (always so for the split copies)
    const int st = make_map(&tp.map[i], mats[i], SPLIT ? contiguous_view(p.bh, n, d) : tensor_view(p, ids[i], n, d), n, d, F16);
    if (st != FHOB_OK) return st;
  }
  tp.nlc = rv.nlc;
  tp.k1 = rv.k1;
  tp.status = rv.status;
  tp.dq = dq; tp.dk = dk; tp.dv = dv;
  tp.heads = (!SPLIT && p.layout) ? p.layout->heads : p.bh;
  tp.d = p.d;
  tp.d_v = head_dim_v(p);
  tp.n_q = p.n_q; tp.n_k = p.n_k; tp.causal = p.causal; tp.window = p.window; tp.scale = p.scale;
  tp.tiles_q = (p.n_q + BM - 1) / BM;
  tp.tiles_k = (p.n_k + BM - 1) / BM;
  if (static_cast<long long>(tp.tiles_q > tp.tiles_k ? tp.tiles_q : tp.tiles_k) * p.bh > 0x3fffffffLL) return FHOB_ERR_SHAPE;
  tp.items_q = tp.tiles_q * p.bh;
  tp.items_k = tp.tiles_k * p.bh;
  const int st = allow_smem(kernel, kSmem);
  if (st != FHOB_OK) return st;
  auto go = [&](bool q_side, bool k_side) -> int {
    const PairGrid g = pair_grid(q_side ? tp.items_q : 0, tc_parts(p.n_q, p.n_k, p.window), k_side ? tp.items_k : 0, tc_parts(p.n_k, p.n_q, p.window));
    if (g.blocks > 0x7fffffffLL) return FHOB_ERR_SHAPE;
    tp.split_q = g.split_q; tp.split_k = g.split_k;
    tp.cluster = g.cluster;
    tp.q_blocks = g.q_blocks;
    FHOB_CUDA_OK(launch_pdl(kernel, static_cast<unsigned>(g.blocks), NTHREADS, kSmem, g.cluster, s, tp));
    return FHOB_OK;
  };
  if (!launch_apart(pair_grid(tp.items_q, tc_parts(p.n_q, p.n_k, p.window), tp.items_k, tc_parts(p.n_k, p.n_q, p.window)))) return go(true, true);
  const int first = go(true, false);
  return first != FHOB_OK ? first : go(false, true);
}

template <bool F16>
int bw_dims(const FhobProblem& p, void* dq, void* dk, void* dv, cudaStream_t s) {
  // tile widths: the head dims rounded up to 64 or 128
  const int d_v = head_dim_v(p);
  if (p.d <= 64) return d_v <= 64 ? bw_launch<64, 64, F16>(p, dq, dk, dv, s) : bw_launch<64, 128, F16>(p, dq, dk, dv, s);
  return d_v <= 64 ? bw_launch<128, 64, F16>(p, dq, dk, dv, s) : bw_launch<128, 128, F16>(p, dq, dk, dv, s);
}

// One warp waits on an mbarrier nothing ever arrives on: exercises the give-up branch of wait_bar.
struct ExpireBars {
  uint64_t bar;
  int abort_flag;
};
__global__ void expire_wait_kernel(int* status) {
  __shared__ ExpireBars b;
  if (threadIdx.x == 0) {
    mbar_init(&b.bar, 1);
    b.abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();
  wait_bar(&b.bar, 0, &b, status);
}

}  // namespace

int tc_selftest_expired_wait(int* status, cudaStream_t s) {
  expire_wait_kernel<<<1, 32, 0, s>>>(status);
  FHOB_CUDA_OK(cudaGetLastError());
  return FHOB_OK;
}

// 16-bit problems with head dims up to 128, and fp32 problems with both head dims up to 64 whose workspace
// holds the bf16 hi/lo copies (see tc_split_supported)
bool tc_first_order_supported(const FhobProblem& p) { return tc_supported(p); }

int tc_backward(const FhobProblem& p, void* dq, void* dk, void* dv, cudaStream_t s) {
  if (!tc_first_order_supported(p)) return FHOB_ERR_SHAPE;
  int st = check_device();
  if (st != FHOB_OK) return st;
  if (p.dtype == FHOB_F32) {
    st = tc_split_inputs(p, s, kSplitQ | kSplitK | kSplitV | kSplitDO);
    return st != FHOB_OK ? st : bw_launch<128, 128, false, true>(p, dq, dk, dv, s);
  }
  return p.dtype == FHOB_F16 ? bw_dims<true>(p, dq, dk, dv, s) : bw_dims<false>(p, dq, dk, dv, s);
}

}  // namespace fhob
