// CUDA-core (FFMA) kernels of the double-backward attention operator.
//
// They serve fp32 problems with a head dim above 64, and any problem the caller
// forces onto them.  The algorithm is that of the tensor-core kernels
// (reference: fhog/triton_bwdbwd.py:178-313 for the query-tiled passes, :321-535
// for the key-tiled one): a CTA keeps "stationary" rows in shared memory, streams
// rows of the other side, rebuilds the score-shaped tiles S, A2, dP, X from fp32
// dot products, applies the elementwise formulas of fhob_common.cuh and either
// reduces along the row (the sweep) or feeds the resulting tiles into the output
// products (passes 3, 4).  Arbitrary n_q, n_k and head dims <= 128 are handled by
// bounds checks; pairs outside the matrix or hidden by the mask contribute zero.
// Two head dims: Q, K, ddQ, ddK, dQ2, dK2 have `d` columns, V, ddV, dO, O, ddO, dV2
// have `dv` (jax_refs/flash_impl.py:381-389 has d_in != d_out).
#include <type_traits>

#include "tc_common.cuh"

namespace fhob {
namespace {

constexpr int NT = 256;       // threads per CTA

struct SimtParams {
  const void *q, *k, *v, *d_o, *ddq, *ddk, *ddv;
  void *dq2, *dk2, *dv2, *ddo;
  const float *nlc, *k1;
  float *ndd, *k23;
  int bh, n_q, n_k, d, dv, causal, window;
  float scale;
  int q_blocks;           // the first q_blocks CTAs are query-tiled, the others key-tiled
  int items_q, items_k;   // (head, tile) pairs of either kind
  int split_q, split_k;   // CTAs that share the streamed tiles of such a pair
  int cluster;            // CTAs of a cluster (a multiple of both)
};

template <typename T>
__device__ __forceinline__ float ld_elem(const void* p, size_t i);
template <>
__device__ __forceinline__ float ld_elem<float>(const void* p, size_t i) {
  return static_cast<const float*>(p)[i];
}
template <>
__device__ __forceinline__ float ld_elem<__nv_bfloat16>(const void* p, size_t i) {
  return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}
template <>
__device__ __forceinline__ float ld_elem<__half>(const void* p, size_t i) {
  return __half2float(static_cast<const __half*>(p)[i]);
}
template <typename T>
__device__ __forceinline__ void st_elem(void* p, size_t i, float v);
template <>
__device__ __forceinline__ void st_elem<__half>(void* p, size_t i, float v) {
  static_cast<__half*>(p)[i] = __float2half_rn(v);
}
template <>
__device__ __forceinline__ void st_elem<float>(void* p, size_t i, float v) {
  static_cast<float*>(p)[i] = v;
}
template <>
__device__ __forceinline__ void st_elem<__nv_bfloat16>(void* p, size_t i, float v) {
  static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// ---- the operator's passes and the first backward
//
// What bounds them is the FMA pipe (128 a clock and SM) and, close behind, shared-memory reads: a
// 16-byte read by a warp takes up to four clocks of the SM's one read port, so a thread has to make about
// 16 multiply-adds of every float4 it reads.  A CTA owns OM = 64 stationary rows and streams ON = 32;
// two groups of four warps take one half of the work of each phase:
//
//   scores    group 0: S, A2 (4 x 4 of the 64 x 32 tile a thread, 12 FMA per float4 read)
//             group 1: dP, X                                     (10.7)
//   elements  group 0: P, t, ddP;  then group 1: dS, dS2          (tiles pass through shared memory)
//   outputs   group 0: dQ2 | dK2,  group 1: ddO | dV2             (8 x 8 of 64 x 128 a thread, 16)
//
// Warps w and w + 4 share a scheduler, so the pipe stays busy while the groups' shares differ.  Products
// are packed fp32 pairs (fma.f32x2): over even and odd elements of the contraction in the scores,
// over neighbouring columns in the outputs; a packed FMA takes one issue slot for two.
// Row statistics come from one sweep (MODE 2).  With D known, centred sums need neither dd nor a second pass:
//   dd = scale sum P A2,   k23 = -D dd - b = -sum P (X + (dP - D) scale A2).
// Passes 3 and 4 share a launch, as do the two halves of the first backward.
//
// fp32, 8 heads, N = 1024, D = 128, the operator: 4884 -> 1331 us
// (one 4 x 1 strip of scores a thread, four passes in launches of their own, before).
constexpr int OM = 64;
constexpr int ON = 32;
constexpr int OP = 128 + 4;    // row pitch of the operand tiles: 8 neighbouring rows lie in different banks
constexpr int PP = OM + 4;     // row pitch of the tiles of P and its derivatives, stored [streamed][stationary]

// MODE 2 = sweep, 3, 4 = passes 3 and 4 (dQ2, ddO | dK2, dV2), 5, 6 = first backward (dQ | dK, dV)
template <int MODE>
struct Tiles {
  static constexpr bool kQStat = MODE != 4 && MODE != 6;
  static constexpr bool kFirst = MODE >= 5;                    // first backward: S and dP alone
  static constexpr bool kBoth2 = MODE == 2 || MODE == 3;       // X = dO . ddV^T reads a streamed tile of its own
  // tiles: 0 = Q | K, 1 = ddQ | ddK, 2 = dO | V (streamed: V | dO), 3 = ddV
  static constexpr int NSTAT = kFirst ? 2 : (MODE == 4 ? 4 : 3);
  static constexpr int NSTRM = kFirst ? 2 : (MODE == 4 ? 3 : 4);
  static constexpr int NP = MODE == 3 ? 4 : (MODE == 4 ? 3 : 2);
  static constexpr int SMEM_BYTES = 4 * (NSTAT * OM * OP + NSTRM * ON * OP + NP * ON * PP + 4 * ON);
  static_assert(SMEM_BYTES <= 232448, "shared memory");
};

__device__ __forceinline__ void cp_async16(float* dst, const void* src, bool live) {
  const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(live ? 16 : 0) : "memory");
}

// Rows [row0, row0 + rows) of a head's (n, d) matrix -> [rows][OP] fp32, zero beyond n.  Rows are whole
// 16-byte pieces and the base is 16-byte aligned (checked by the entry points).  fp32 arrives asynchronously.
template <typename T>
__device__ __forceinline__ void load_rows(float* tile, const void* src, size_t head_off, int row0, int rows, int n, int d) {
  constexpr int V = 16 / sizeof(T);
  const int pieces = d / V;
  const T* base = static_cast<const T*>(src) + head_off;
  for (int idx = threadIdx.x; idx < rows * pieces; idx += NT) {
    const int r = idx / pieces, c = (idx - r * pieces) * V;
    const bool live = row0 + r < n;
    const T* from = base + static_cast<size_t>(live ? row0 + r : 0) * d + c;
    float* to = tile + r * OP + c;
    if constexpr (V == 4) {
      cp_async16(to, from, live);
    } else {
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (live) w = *reinterpret_cast<const uint4*>(from);
      const T* e = reinterpret_cast<const T*>(&w);
      *reinterpret_cast<float4*>(to) = make_float4(static_cast<float>(e[0]), static_cast<float>(e[1]), static_cast<float>(e[2]), static_cast<float>(e[3]));
      *reinterpret_cast<float4*>(to + 4) = make_float4(static_cast<float>(e[4]), static_cast<float>(e[5]), static_cast<float>(e[6]), static_cast<float>(e[7]));
    }
  }
}
__device__ __forceinline__ void loads_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

// acc[i][j] += a_i . b_j over four elements, even and odd ones apart
__device__ __forceinline__ void dot4(float2& acc, const float4& a, const float4& b) {
  acc = __ffma2_rn(lo2(a), lo2(b), acc);
  acc = __ffma2_rn(hi2(a), hi2(b), acc);
}

// out (8 rows x 8 columns: 4 at col, 4 at col + 64) += at[c][rows] . b[c][cols] over the ON streamed rows,
// for one or two such products.  WIDE: the second four columns exist.
template <bool TWO, bool WIDE>
__device__ __forceinline__ void outer(float2 (&out)[8][4], const float* a0, const float* b0, const float* a1, const float* b1) {
#pragma unroll 4
  for (int c = 0; c < ON; ++c) {
#pragma unroll
    for (int t = 0; t < (TWO ? 2 : 1); ++t) {
      const float* a = (t ? a1 : a0) + c * PP;
      const float* b = (t ? b1 : b0) + c * OP;
      const float4 al = ld4(a), ah = ld4(a + 4), bl = ld4(b);
      float4 bh = make_float4(0.f, 0.f, 0.f, 0.f);
      if (WIDE) bh = ld4(b + 64);
      const float r[8] = {al.x, al.y, al.z, al.w, ah.x, ah.y, ah.z, ah.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 rr = make_float2(r[i], r[i]);
        out[i][0] = __ffma2_rn(rr, lo2(bl), out[i][0]);
        out[i][1] = __ffma2_rn(rr, hi2(bl), out[i][1]);
        if (WIDE) {
          out[i][2] = __ffma2_rn(rr, lo2(bh), out[i][2]);
          out[i][3] = __ffma2_rn(rr, hi2(bh), out[i][3]);
        }
      }
    }
  }
}

// Four neighbouring columns of a result row.
template <typename T>
__device__ __forceinline__ void store4(void* base, size_t at, const float2& a, const float2& b, float mul) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(static_cast<float*>(base) + at) = make_float4(a.x * mul, a.y * mul, b.x * mul, b.y * mul);
  } else {
    T w[4] = {static_cast<T>(a.x * mul), static_cast<T>(a.y * mul), static_cast<T>(b.x * mul), static_cast<T>(b.y * mul)};
    *reinterpret_cast<uint2*>(static_cast<T*>(base) + at) = *reinterpret_cast<const uint2*>(w);
  }
}

template <typename T, int MODE>
__device__ __forceinline__ void simt_body(const SimtParams& p, int block) {
  using C = Tiles<MODE>;
  constexpr bool kQStat = C::kQStat, kFirst = C::kFirst;
  extern __shared__ float smem[];
  // first backward: tiles 0 and 2 only, stored one after the other
  float* stat[4] = {smem, smem + OM * OP, smem + (kFirst ? 1 : 2) * OM * OP, smem + 3 * OM * OP};
  float* strm0 = smem + C::NSTAT * OM * OP;
  float* strm[4] = {strm0, strm0 + ON * OP, strm0 + (kFirst ? 1 : 2) * ON * OP, strm0 + 3 * ON * OP};
  float* pt0 = strm0 + C::NSTRM * ON * OP;
  float* svec = pt0 + C::NP * ON * PP;   // key-tiled: nlc, ndd, k1, k23 of the streamed queries
  // tiles of P and its derivatives.  t and (unless it is an operand itself) P wait where dS and dS2 go.
  float* pt[4] = {pt0, pt0 + ON * PP, pt0 + 2 * ON * PP, pt0 + 3 * ON * PP};
  float* const p_tile = MODE == 3 ? pt[3] : pt[1];

  const int d = p.d, dv = p.dv;
  const int group = threadIdx.x >> 7, tid = threadIdx.x & 127;
  const int ty = tid >> 3, tx = tid & 7;     // scores: rows 4 ty + i, streamed rows tx + 8 j
  const int ry = tid >> 4, cx = tid & 15;    // outputs: rows 8 ry + i, columns 4 cx.. and 64 + 4 cx..
  // with few tiles a head the streamed axis is split over the CTAs of a cluster
  const int split = kQStat ? p.split_q : p.split_k;
  const CtaWork work = cta_work(block, split, kQStat ? p.items_q : p.items_k);   // the grid is padded to whole clusters
  const int item = work.item, begin_part = work.part;
  const bool padding = !work.live;
  const int tile_no = item / p.bh, bh = item - tile_no * p.bh;   // causal: the longest tiles of all heads first
  const int tiles = ((kQStat ? p.n_q : p.n_k) + OM - 1) / OM;
  const int m0 = (kQStat ? tiles - 1 - tile_no : tile_no) * OM;
  const size_t qoff = static_cast<size_t>(bh) * p.n_q * d, qoff_v = static_cast<size_t>(bh) * p.n_q * dv;
  const size_t koff = static_cast<size_t>(bh) * p.n_k * d, koff_v = static_cast<size_t>(bh) * p.n_k * dv;
  const size_t voff = static_cast<size_t>(bh) * row_stride(p.n_q);
  const int off = p.n_k - p.n_q;
  const int n_stat = kQStat ? p.n_q : p.n_k, n_strm = kQStat ? p.n_k : p.n_q;

  // operands of the (q/k, v) head dims on either side
  const void *q_in[4] = {p.q, p.ddq, p.d_o, nullptr}, *k_in[4] = {p.k, p.ddk, p.v, p.ddv};
  auto load_side = [&](float* const (&dst)[4], bool q_side, int row0, int rows) {
    const int n = q_side ? p.n_q : p.n_k;
    const size_t o = q_side ? qoff : koff, o_v = q_side ? qoff_v : koff_v;
    const void* const* in = q_side ? q_in : k_in;
    load_rows<T>(dst[0], in[0], o, row0, rows, n, d);
    if (!kFirst) load_rows<T>(dst[1], in[1], o, row0, rows, n, d);
    load_rows<T>(dst[2], in[2], o_v, row0, rows, n, dv);
    if (!kFirst && !q_side) load_rows<T>(dst[3], in[3], o_v, row0, rows, n, dv);
  };
  load_side(stat, kQStat, m0, OM);

  float r_nlc[4], r_ndd[4], r_k1[4], r_k23[4];   // constants of the thread's stationary queries
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int qi = m0 + 4 * ty + i;
    const bool ok = kQStat && qi < p.n_q;
    r_nlc[i] = ok ? p.nlc[voff + qi] : 0.f;
    r_k1[i] = ok ? p.k1[voff + qi] : 0.f;
    r_ndd[i] = ok && MODE == 3 ? p.ndd[voff + qi] : 0.f;
    r_k23[i] = ok && MODE == 3 ? p.k23[voff + qi] : 0.f;
  }
  float rowacc[4] = {0.f, 0.f, 0.f, 0.f};   // sweep
  float2 out[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) out[i][j] = make_float2(0.f, 0.f);

  int t_begin, t_end;
  visible_tiles(kQStat, m0, OM, ON, n_strm, off, p.causal, p.window, t_begin, t_end);
  if (split > 1) split_range(begin_part, split, t_begin, t_end);
  if (padding) t_end = t_begin;
  const float sl2 = p.scale * kLog2e;

  for (int t = t_begin; t < t_end; ++t) {
    const int n0 = t * ON;
    __syncthreads();   // the previous step has read its tiles
    load_side(strm, !kQStat, n0, ON);
    if (!kQStat && threadIdx.x < ON) {
      const int qi = n0 + threadIdx.x;
      const bool ok = qi < p.n_q;
      svec[threadIdx.x] = ok ? p.nlc[voff + qi] : 0.f;
      svec[2 * ON + threadIdx.x] = ok ? p.k1[voff + qi] : 0.f;
      if (!kFirst) {
        svec[ON + threadIdx.x] = ok ? p.ndd[voff + qi] : 0.f;
        svec[3 * ON + threadIdx.x] = ok ? p.k23[voff + qi] : 0.f;
      }
    }
    loads_landed();
    __syncthreads();

    // does any pair of this tile need masking?  (uniform over the CTA)
    bool masked = n0 + ON > n_strm;
    if (p.causal) {
      if (kQStat) masked = masked || n0 + ON - 1 > m0 + off || (p.window > 0 && m0 + OM - 1 + off - n0 >= p.window);
      else masked = masked || n0 + off < m0 + OM - 1 || (p.window > 0 && n0 + ON - 1 + off - m0 >= p.window);
    }
    auto allowed = [&](int i, int j) {
      if (!masked) return true;
      const int r = m0 + 4 * ty + i, c = n0 + tx + 8 * j;
      return c < n_strm && pair_visible(kQStat ? r : c, kQStat ? c : r, off, p.causal, p.window);
    };

    float2 u0[4][4], u1[4][4];   // group 0: S, A2; group 1: dP, X
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) u0[i][j] = u1[i][j] = make_float2(0.f, 0.f);
    if (group == 0) {
      const float *sa = stat[0] + 4 * ty * OP, *sb = stat[1] + 4 * ty * OP, *ca = strm[0] + tx * OP, *cb = strm[1] + tx * OP;
#pragma unroll 2
      for (int e = 0; e < d; e += 4) {
        float4 k[4], kk[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          k[j] = ld4(ca + 8 * j * OP + e);
          if (!kFirst) kk[j] = ld4(cb + 8 * j * OP + e);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 q = ld4(sa + i * OP + e);
#pragma unroll
          for (int j = 0; j < 4; ++j) dot4(u0[i][j], q, k[j]);
          if (!kFirst) {
            const float4 qq = ld4(sb + i * OP + e);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              dot4(u1[i][j], q, kk[j]);
              dot4(u1[i][j], qq, k[j]);
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = tx + 8 * j;
        float pr[4], tt[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool ok = allowed(i, j);
          const float s = u0[i][j].x + u0[i][j].y, a2 = u1[i][j].x + u1[i][j].y;
          pr[i] = ok ? exp2f(fmaf(s, sl2, kQStat ? r_nlc[i] : svec[c])) : 0.f;
          if (MODE == 2) {
            tt[i] = ok ? a2 * p.scale : 0.f;
            rowacc[i] = fmaf(pr[i], tt[i], rowacc[i]);
          } else if (!kFirst) {
            tt[i] = ok ? fmaf(a2, p.scale, kQStat ? r_ndd[i] : svec[ON + c]) : 0.f;
          }
        }
        const int at = c * PP + 4 * ty;
        *reinterpret_cast<float4*>(p_tile + at) = make_float4(pr[0], pr[1], pr[2], pr[3]);
        if (!kFirst) *reinterpret_cast<float4*>(pt[0] + at) = make_float4(tt[0], tt[1], tt[2], tt[3]);
        if (MODE == 3 || MODE == 4)
          *reinterpret_cast<float4*>(pt[2] + at) = make_float4(pr[0] * tt[0], pr[1] * tt[1], pr[2] * tt[2], pr[3] * tt[3]);
      }
    } else {
      const float *sa = stat[2] + 4 * ty * OP, *sb = stat[3] + 4 * ty * OP, *ca = strm[2] + tx * OP, *cb = strm[3] + tx * OP;
#pragma unroll 2
      for (int e = 0; e < dv; e += 4) {
        float4 v[4], vv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[j] = ld4(ca + 8 * j * OP + e);
          if (C::kBoth2) vv[j] = ld4(cb + 8 * j * OP + e);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 g = ld4(sa + i * OP + e);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            dot4(u0[i][j], g, v[j]);
            if (C::kBoth2) dot4(u1[i][j], g, vv[j]);
          }
          if (MODE == 4) {
            const float4 gg = ld4(sb + i * OP + e);
#pragma unroll
            for (int j = 0; j < 4; ++j) dot4(u1[i][j], gg, v[j]);
          }
        }
      }
    }
    __syncthreads();   // P and t are there
    if (group == 1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = tx + 8 * j, at = c * PP + 4 * ty;
        const float4 p4 = ld4(p_tile + at);
        float4 t4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!kFirst) t4 = ld4(pt[0] + at);
        const float pr[4] = {p4.x, p4.y, p4.z, p4.w}, tt[4] = {t4.x, t4.y, t4.z, t4.w};
        float ds[4], ds2[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool ok = allowed(i, j);
          const float dpp = u0[i][j].x + u0[i][j].y + (kQStat ? r_k1[i] : svec[2 * ON + c]);
          const float x = u1[i][j].x + u1[i][j].y;
          if (MODE == 2) {
            if (ok) rowacc[i] = fmaf(pr[i], fmaf(dpp, tt[i], x), rowacc[i]);
          } else {
            ds[i] = ok ? pr[i] * dpp : 0.f;
            if (!kFirst) ds2[i] = ok ? pr[i] * fmaf(dpp, tt[i], x + (kQStat ? r_k23[i] : svec[3 * ON + c])) : 0.f;
          }
        }
        if (MODE != 2) *reinterpret_cast<float4*>(pt[0] + at) = make_float4(ds[0], ds[1], ds[2], ds[3]);
        if (MODE == 3 || MODE == 4) *reinterpret_cast<float4*>(pt[1] + at) = make_float4(ds2[0], ds2[1], ds2[2], ds2[3]);
      }
    }
    if constexpr (MODE == 3 || MODE == 4) {
      __syncthreads();   // dS and dS2 are there
      const int ro = 8 * ry, co = 4 * cx;
      if (group == 0) {   // dS . ddK | ddQ + dS2 . K | Q
        if (d > 64) outer<true, true>(out, pt[0] + ro, strm[1] + co, pt[1] + ro, strm[0] + co);
        else outer<true, false>(out, pt[0] + ro, strm[1] + co, pt[1] + ro, strm[0] + co);
      } else {            // ddP . V | dO (+ P . ddV)
        if (dv > 64) outer<MODE == 3, true>(out, pt[2] + ro, strm[2] + co, pt[3] + ro, strm[3] + co);
        else outer<MODE == 3, false>(out, pt[2] + ro, strm[2] + co, pt[3] + ro, strm[3] + co);
      }
    } else if constexpr (kFirst) {
      __syncthreads();
      const int ro = 8 * ry, co = 4 * cx;
      if constexpr (MODE == 5) {   // dS . K, 64 columns a group
        if (64 * group < d) outer<false, false>(out, pt[0] + ro, strm[0] + 64 * group + co, nullptr, nullptr);
      } else if (group == 0) {     // dS . Q
        if (d > 64) outer<false, true>(out, pt[0] + ro, strm[0] + co, nullptr, nullptr);
        else outer<false, false>(out, pt[0] + ro, strm[0] + co, nullptr, nullptr);
      } else {                     // P . dO
        if (dv > 64) outer<false, true>(out, pt[1] + ro, strm[2] + co, nullptr, nullptr);
        else outer<false, false>(out, pt[1] + ro, strm[2] + co, nullptr, nullptr);
      }
    }
  }

  loads_landed();   // a tile without visible pairs has not waited yet

  // Worked out again from the block number: kept in registers through the loop, these cost spills in it.
  uint32_t block_again;
  asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(block_again));
  block_again -= kQStat ? 0 : p.q_blocks;
  const bool live = block_again / split < static_cast<uint32_t>(kQStat ? p.items_q : p.items_k);
  const int part = static_cast<int>(block_again % split);

  // results; the parts of an item are staged in shared memory and added up in rank order
  constexpr int kPitch = 256 + 4;   // floats per staged row: the two results
  static_assert(4 * OM * kPitch <= C::SMEM_BYTES, "staging area");
  if (split > 1) __syncthreads();   // every tile has been read
  const bool first = group == 0 || MODE == 5;
  void *base0 = MODE == 3 || MODE == 5 ? p.dq2 : p.dk2, *base1 = MODE == 3 ? p.ddo : p.dv2;
  if (MODE == 2) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float tot = rowacc[i];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
      const int qi = m0 + 4 * ty + i;
      if (tx != 0) continue;
      if (split > 1) smem[group * OM + 4 * ty + i] = tot;
      else if (live && qi < p.n_q) (group == 0 ? p.ndd : p.k23)[voff + qi] = -tot;
    }
  } else {
    const int cols = first ? d : dv, col = 4 * cx + (MODE == 5 ? 64 * group : 0);
    const size_t head = first ? (kQStat ? qoff : koff) : (kQStat ? qoff_v : koff_v);
    const float mul = first ? p.scale : 1.f;   // dS and dS2 carry no factor `scale`
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (split > 1) {
        const size_t at = (8 * ry + i) * kPitch + (first ? 0 : 128) + col;
        store4<float>(smem, at, out[i][0], out[i][1], 1.f);
        if (MODE != 5) store4<float>(smem, at + 64, out[i][2], out[i][3], 1.f);
        continue;
      }
      const int r = m0 + 8 * ry + i;
      if (!live || r >= n_stat) continue;
      const size_t at = head + static_cast<size_t>(r) * cols + col;
      if (col < cols) store4<T>(first ? base0 : base1, at, out[i][0], out[i][1], mul);
      if (MODE != 5 && col + 64 < cols) store4<T>(first ? base0 : base1, at + 64, out[i][2], out[i][3], mul);
    }
  }
  if (p.cluster > 1) {
    cluster_sync();
    const int rank0 = static_cast<int>(cluster_rank()) - part;
    if (split > 1 && live) {
      if constexpr (MODE == 2) {
        const int row = threadIdx.x & (OM - 1), qi = m0 + row;
        if (part == 0 && threadIdx.x < 2 * OM && qi < p.n_q) {
          float tot = 0.f;
          for (int i = 0; i < split; ++i) tot += cluster_ld(cluster_map(smem_u32(smem) + threadIdx.x * 4, rank0 + i));
          (threadIdx.x < OM ? p.ndd : p.k23)[voff + qi] = -tot;
        }
      } else {
        constexpr bool kF32 = sizeof(T) == 4, kF16 = std::is_same<T, __half>::value;
        reduce_store<128, kF32, kF16, OM>(smem_u32(smem), kPitch, 0, rank0, part, split, threadIdx.x, base0, bh, m0, n_stat, d, p.scale);
        if (MODE != 5)
          reduce_store<128, kF32, kF16, OM>(smem_u32(smem), kPitch, 128, rank0, part, split, threadIdx.x, base1, bh, m0, n_stat, dv, 1.f);
      }
    }
    cluster_sync();   // the others are done with this CTA's shared memory
  }
}

// MODE_Q on the first q_blocks CTAs, MODE_K (if not 0) on the others
template <typename T, int MODE_Q, int MODE_K>
__global__ void __launch_bounds__(NT, 1) simt_pass_kernel(const __grid_constant__ SimtParams p) {
  pdl_wait();
  if (threadIdx.x == 0) pdl_launch_dependents();
  const int block = blockIdx.x;
  if (block < p.q_blocks) simt_body<T, MODE_Q>(p, block);
  else if constexpr (MODE_K != 0) simt_body<T, MODE_K>(p, block - p.q_blocks);
}

// O(N)-memory forward: online softmax.  A CTA owns OM = 64 queries and streams FN = 128 keys; a warp owns eight
// rows of both the scores and the outputs, so a row's maximum and sum never leave the warp and P passes
// through shared memory without a CTA barrier.  The warp's operand on the row side (Q, P) is the same
// address for all lanes; of the other one (K, V) a thread reads one float4 per 32 multiply-adds.  K of the next
// step arrives during P V, V during Q K^T.  Heads of few tiles are split over clusters, as the operator's.
// fp32, D = 128, us, before (32 queries a CTA, two to four FMAs per word read) -> now:
// 8 heads N = 1024 405 -> 129, 32 causal heads N = 512 294 -> 90.  4 heads 200 x 5000, in two parts: 316.
constexpr int FN = 128;
constexpr int kForwardSmem = 4 * ((OM + 2 * FN) * OP + FN * PP);
constexpr int kForwardPitch = 128 + 4;   // floats per staged row of a split problem: the outputs, maximum, sum

// As load_rows for callers whose rows are not whole 16-byte pieces: element by element, zeros up to a multiple of four.
template <typename T>
__device__ __forceinline__ void load_rows_any(float* tile, const void* src, size_t head_off, int row0, int rows, int n, int d, bool vec) {
  if (vec) {
    load_rows<T>(tile, src, head_off, row0, rows, n, d);
    return;
  }
  const int w = (d + 3) & ~3;
  for (int idx = threadIdx.x; idx < rows * w; idx += NT) {
    const int r = idx / w, c = idx - r * w;
    const bool live = row0 + r < n && c < d;
    tile[r * OP + c] = live ? ld_elem<T>(src, head_off + static_cast<size_t>(row0 + r) * d + c) : 0.f;
  }
}

__device__ __forceinline__ void loads_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void loads_landed_but_last() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

template <typename T>
__global__ void __launch_bounds__(NT, 1) simt_forward_kernel(const __grid_constant__ SimtParams p, void* o_out, float* lse_out, int* status, bool vec) {
  pdl_wait();
  if (threadIdx.x == 0) {
    pdl_launch_dependents();
    if (blockIdx.x == 0 && status) *status = 0;   // every call starts clean
  }
  extern __shared__ float smem[];
  float *qs = smem, *ks = qs + OM * OP, *vs = ks + FN * OP, *ps = vs + FN * OP;   // ps: [key][query]
  const int d = p.d, dv = p.dv, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = p.split_q;
  const CtaWork work = cta_work(blockIdx.x, split, p.items_q);
  const int item = work.item, part = work.part;
  const bool live = work.live;
  const int tile_no = item / p.bh, bh = item - tile_no * p.bh;   // causal: the longest tiles of all heads first
  const int m0 = ((p.n_q + OM - 1) / OM - 1 - tile_no) * OM, row0 = m0 + 8 * warp;
  const size_t qoff = static_cast<size_t>(bh) * p.n_q * d, ooff = static_cast<size_t>(bh) * p.n_q * dv;
  const size_t koff = static_cast<size_t>(bh) * p.n_k * d, voff = static_cast<size_t>(bh) * p.n_k * dv;
  const int off = p.n_k - p.n_q;
  int t_begin, t_end;
  visible_tiles(true, m0, OM, FN, p.n_k, off, p.causal, p.window, t_begin, t_end);
  if (split > 1) split_range(part, split, t_begin, t_end);
  if (!live) t_end = t_begin;
  const float sl2 = p.scale * kLog2e;

  float mrow[8], lrow[8];   // maximum (of the row) and sum (of this lane's columns), log2 domain
  float2 acc[8][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    mrow[i] = -INFINITY;
    lrow[i] = 0.f;
    acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
  }
  load_rows_any<T>(qs, p.q, qoff, m0, OM, p.n_q, d, vec);
  if (t_begin < t_end) load_rows_any<T>(ks, p.k, koff, t_begin * FN, FN, p.n_k, d, vec);
  loads_commit();

  for (int t = t_begin; t < t_end; ++t) {
    const int n0 = t * FN;
    if (o_out) load_rows_any<T>(vs, p.v, voff, n0, FN, p.n_k, dv, vec);
    loads_commit();
    loads_landed_but_last();
    __syncthreads();   // Q, K

    float2 s[8][4];   // rows 8 warp + i, keys lane + 32 j; even and odd elements of the contraction apart
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = make_float2(0.f, 0.f);
    const float *qa = qs + 8 * warp * OP, *ka = ks + lane * OP;
#pragma unroll 2
    for (int e = 0; e < d; e += 4) {
      float4 k[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) k[j] = ld4(ka + 32 * j * OP + e);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 q = ld4(qa + i * OP + e);
#pragma unroll
        for (int j = 0; j < 4; ++j) dot4(s[i][j], q, k[j]);
      }
    }
    __syncthreads();   // K has been read
    if (t + 1 < t_end) load_rows_any<T>(ks, p.k, koff, n0 + FN, FN, p.n_k, d, vec);
    loads_commit();

    const bool masked = n0 + FN > p.n_k || (p.causal && (n0 + FN - 1 > m0 + off || (p.window > 0 && m0 + OM - 1 + off - n0 >= p.window)));
    float pr[4][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float sv[4], mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = n0 + lane + 32 * j;
        const bool ok = !masked || (c < p.n_k && pair_visible(row0 + i, c, off, p.causal, p.window));
        sv[j] = ok ? (s[i][j].x + s[i][j].y) * sl2 : -INFINITY;
        mx = fmaxf(mx, sv[j]);
      }
      const float mnew = fmaxf(mrow[i], warp_max(mx));
      const float alpha = mnew == -INFINITY ? 1.f : exp2f(mrow[i] - mnew);
      const float from = mnew == -INFINITY ? 0.f : mnew;   // no maximum yet: P = 0 for hidden keys, NaN for NaN scores
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        pr[j][i] = exp2f(sv[j] - from);
        sum += pr[j][i];
      }
      lrow[i] = lrow[i] * alpha + sum;
      mrow[i] = mnew;
#pragma unroll
      for (int h = 0; h < 2; ++h) acc[i][h] = make_float2(acc[i][h].x * alpha, acc[i][h].y * alpha);
    }
    if (o_out) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float* to = ps + (lane + 32 * j) * PP + 8 * warp;
        *reinterpret_cast<float4*>(to) = make_float4(pr[j][0], pr[j][1], pr[j][2], pr[j][3]);
        *reinterpret_cast<float4*>(to + 4) = make_float4(pr[j][4], pr[j][5], pr[j][6], pr[j][7]);
      }
    }
    loads_landed_but_last();
    __syncthreads();   // V (and this warp's P)
    if (o_out) {
      const float *pa = ps + 8 * warp, *va = vs + 4 * lane;
#pragma unroll 4
      for (int c = 0; c < FN; ++c) {
        const float4 al = ld4(pa + c * PP), ah = ld4(pa + c * PP + 4), v = ld4(va + c * OP);
        const float r[8] = {al.x, al.y, al.z, al.w, ah.x, ah.y, ah.z, ah.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          acc[i][0] = __ffma2_rn(make_float2(r[i], r[i]), lo2(v), acc[i][0]);
          acc[i][1] = __ffma2_rn(make_float2(r[i], r[i]), hi2(v), acc[i][1]);
        }
      }
      __syncthreads();   // V has been read
    }
  }
  loads_landed();
#pragma unroll
  for (int i = 0; i < 8; ++i) lrow[i] = warp_sum(lrow[i]);

  auto store = [&](int row, const float (&o)[4], float m, float l) {   // lane: columns 4 lane..
    const float inv = l == 0.f ? 0.f : 1.f / l;   // a sum of zero: no visible key (a NaN is kept)
    if (o_out) {
      const size_t at = ooff + static_cast<size_t>(row) * dv + 4 * lane;
      if (vec) {
        if (4 * lane < dv) store4<T>(o_out, at, make_float2(o[0], o[1]), make_float2(o[2], o[3]), inv);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (4 * lane + e < dv) st_elem<T>(o_out, at + e, o[e] * inv);
      }
    }
    if (lane == 0)
      lse_out[static_cast<size_t>(bh) * p.n_q + row] = l == 0.f ? -INFINITY : (m + log2f(l)) * 0.6931471805599453f;
  };
  if (split <= 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float o[4] = {acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y};
      if (live && row0 + i < p.n_q) store(row0 + i, o, mrow[i], lrow[i]);
    }
    return;   // launches without a split have no clusters
  }
  // the parts' rows are staged and put on a common maximum, in rank order
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float* to = smem + (8 * warp + i) * kForwardPitch;
    store4<float>(to, 4 * lane, acc[i][0], acc[i][1], 1.f);
    if (lane == 0) {
      to[128] = mrow[i];
      to[129] = lrow[i];
    }
  }
  cluster_sync();
  if (live) {
    const int rank0 = static_cast<int>(cluster_rank()) - part;
    for (int r = part + split * warp; r < OM && m0 + r < p.n_q; r += split * 8) {
      const uint32_t at = smem_u32(smem) + r * kForwardPitch * 4;
      float m = -INFINITY, l = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
      for (int i = 0; i < split; ++i) m = fmaxf(m, cluster_ld(cluster_map(at, rank0 + i) + 128 * 4));
      for (int i = 0; i < split; ++i) {
        const uint32_t from = cluster_map(at, rank0 + i);
        const float mi = cluster_ld(from + 128 * 4), li = cluster_ld(from + 129 * 4);
        if (li == 0.f) continue;   // a part without a visible key
        const float w = mi == -INFINITY ? 1.f : exp2f(mi - m);   // (no maximum but a sum: NaN)
        const float4 x = cluster_ld4(from + 16 * lane);
        l = fmaf(li, w, l);
        o[0] = fmaf(x.x, w, o[0]); o[1] = fmaf(x.y, w, o[1]); o[2] = fmaf(x.z, w, o[2]); o[3] = fmaf(x.w, w, o[3]);
      }
      store(m0 + r, o, m, l);
    }
  }
  cluster_sync();   // the others are done with this CTA's shared memory
}


SimtParams make_params(const FhobProblem& p) {
  RowVectors rv = row_vectors(p);
  SimtParams s;
  s.q = p.q; s.k = p.k; s.v = p.v; s.d_o = p.d_o; s.ddq = p.ddq; s.ddk = p.ddk; s.ddv = p.ddv;
  s.dq2 = p.dq2; s.dk2 = p.dk2; s.dv2 = p.dv2; s.ddo = p.ddo;
  s.nlc = rv.nlc; s.k1 = rv.k1; s.ndd = rv.ndd; s.k23 = rv.k23;
  s.bh = p.bh; s.n_q = p.n_q; s.n_k = p.n_k; s.d = p.d; s.dv = head_dim_v(p); s.causal = p.causal; s.window = p.window; s.scale = p.scale;
  return s;
}

// In streamed tiles (fp32, D = 128: 12 us in passes 3 and 4): what a CTA takes besides its tiles is about one
// tile's time, meeting in a cluster about half of one.  That is little enough for
// heads of any number of tiles to be split in two from about 1000 streamed rows on.  Operator, fp32, D = 128, us,
// unsplit -> split: 1 head 64 x 3000 2497 -> 332, 4 heads 200 x 5000 4156 -> 1086, 1 causal head N = 2000 1719 -> 897;
// 8 heads N = 1024 1326 -> 1337, 64 heads 9333 -> 9596, causal 5174 -> 5371.
constexpr SplitCost kSimtCost = {1.f, 0.5f, 1.f / 16};

PairGrid modes_grid(const FhobProblem& p, bool q_side, bool k_side) {
  const int tiles_q = (p.n_q + OM - 1) / OM, tiles_k = (p.n_k + OM - 1) / OM;
  return pair_grid(q_side ? static_cast<long long>(tiles_q) * p.bh : 0, split_parts(tiles_q, longest(p.n_k, ON, OM, p.window), kSimtCost),
                   k_side ? static_cast<long long>(tiles_k) * p.bh : 0, split_parts(tiles_k, longest(p.n_q, ON, OM, p.window), kSimtCost));
}

template <typename T, int MODE_Q, int MODE_K>
int launch_modes(const FhobProblem& problem, SimtParams& p, bool q_side, bool k_side, cudaStream_t st) {
  constexpr auto kernel = simt_pass_kernel<T, MODE_Q, MODE_K>;
  constexpr int kQ = Tiles<MODE_Q>::SMEM_BYTES, kK = Tiles<MODE_K ? MODE_K : MODE_Q>::SMEM_BYTES, kSmem = kQ > kK ? kQ : kK;
  const int ok = allow_smem(kernel, kSmem);
  if (ok != FHOB_OK) return ok;
  const PairGrid g = modes_grid(problem, q_side, k_side);
  if (g.blocks > 0x7fffffffLL) return FHOB_ERR_SHAPE;
  p.items_q = g.items_q; p.items_k = g.items_k;
  p.split_q = g.split_q; p.split_k = g.split_k;
  p.cluster = g.cluster;
  p.q_blocks = g.q_blocks;
  FHOB_CUDA_OK(launch_pdl(kernel, static_cast<unsigned>(g.blocks), NT, kSmem, g.cluster, st, p));
  return FHOB_OK;
}

// `pass` as in the entry points; passes 1 and 2 are one sweep, whichever is asked for
template <typename T>
int dispatch_pass(int pass, const FhobProblem& p, cudaStream_t st) {
  SimtParams s = make_params(p);
  switch (pass) {
    case 1:
    case 2:
    case 12: return launch_modes<T, 2, 0>(p, s, true, false, st);
    case 3: return launch_modes<T, 3, 4>(p, s, true, false, st);
    case 4: return launch_modes<T, 3, 4>(p, s, false, true, st);
    case 34: return launch_modes<T, 3, 4>(p, s, true, true, st);
  }
  return FHOB_ERR_ARG;
}

template <typename T>
int launch_backward(const FhobProblem& p, void* dq, void* dk, void* dv, cudaStream_t st) {
  SimtParams s = make_params(p);
  s.dq2 = dq; s.dk2 = dk; s.dv2 = dv;
  return launch_modes<T, 5, 6>(p, s, true, true, st);
}

// The forward reads rows element by element if they are not whole, aligned 16-byte pieces.
template <typename T>
int launch_forward(const FhobProblem& p, void* o_out, float* lse_out, int* status, cudaStream_t st) {
  constexpr auto kernel = simt_forward_kernel<T>;
  const int ok = allow_smem(kernel, kForwardSmem);
  if (ok != FHOB_OK) return ok;
  SimtParams s = make_params(p);
  auto whole = [](const void* x, int cols) { return ((reinterpret_cast<uintptr_t>(x) | (cols * sizeof(T))) & 15u) == 0; };
  const bool vec = whole(p.q, s.d) && whole(p.k, s.d) && whole(p.v, s.dv) && whole(o_out, s.dv);
  const long long items = static_cast<long long>((p.n_q + OM - 1) / OM) * p.bh;
  if (items > 0x7fffffffLL) return FHOB_ERR_SHAPE;
  s.items_q = static_cast<int>(items);
  s.split_q = s.cluster = split_parts((p.n_q + OM - 1) / OM, longest(p.n_k, FN, OM, p.window), kSimtCost);
  if (items * s.split_q > 0x7fffffffLL) return FHOB_ERR_SHAPE;
  FHOB_CUDA_OK(launch_pdl(kernel, static_cast<unsigned>(items * s.split_q), NT, kForwardSmem, s.cluster, st, s, o_out, lse_out, status, vec));
  return FHOB_OK;
}

}  // namespace

int simt_grid(const FhobProblem& p, PairGrid* g) {
  *g = modes_grid(p, true, true);
  return g->blocks > 0x7fffffffLL ? FHOB_ERR_SHAPE : FHOB_OK;
}

int simt_backward(const FhobProblem& p, void* dq, void* dk, void* dv, cudaStream_t st) {
  if (p.d > 128 || head_dim_v(p) > 128) return FHOB_ERR_SHAPE;
  if (p.dtype == FHOB_F32) return launch_backward<float>(p, dq, dk, dv, st);
  if (p.dtype == FHOB_F16) return launch_backward<__half>(p, dq, dk, dv, st);
  return launch_backward<__nv_bfloat16>(p, dq, dk, dv, st);
}

int simt_pass(int pass, const FhobProblem& p, cudaStream_t st) {
  if (p.d > 128 || head_dim_v(p) > 128) return FHOB_ERR_SHAPE;
  if (p.dtype == FHOB_F32) return dispatch_pass<float>(pass, p, st);
  if (p.dtype == FHOB_F16) return dispatch_pass<__half>(pass, p, st);
  return dispatch_pass<__nv_bfloat16>(pass, p, st);
}

int simt_forward(const FhobProblem& p, void* o_out, float* lse_out, int* status, cudaStream_t st) {
  if (p.d > 128 || head_dim_v(p) > 128) return FHOB_ERR_SHAPE;
  if (p.dtype == FHOB_F32) return launch_forward<float>(p, o_out, lse_out, status, st);
  if (p.dtype == FHOB_F16) return launch_forward<__half>(p, o_out, lse_out, status, st);
  return launch_forward<__nv_bfloat16>(p, o_out, lse_out, status, st);
}

}  // namespace fhob
