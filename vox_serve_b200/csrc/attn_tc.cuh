// The tcgen05 attention core of prompt rows, shared by prefill_attn_tc.cu (paged cache of the speech LMs) and window_attn_tc.cu
// (sliding windows of the text LMs): one accumulator row of 128 per softmax thread, scores and probabilities in TMEM, K and V
// tiles of 64 keys through two-stage rings.  A kernel brings an object `rows` that says what its thread's row sees:
//   n_tiles, tile(it)        the key tiles to walk, in order (tile i holds keys 64 i ..)
//   scale_log2               what a score is multiplied by, times log2(e)
//   full(tok0), visible(kj)  whether all 64 keys from tok0 / key kj are visible to this thread's row
//   group, q_row(t, g)       accumulator row r is row t = r / group of the tile, head g = r % group of the group: its query row, or nullptr
//                            (a padding row: zeros)
//   finish(m_ref, l)         factor for the accumulated row, given the exponents' reference and the denominator against it
//   store(c0, o, f)          32 output values of this thread's row from column c0, times the factor: either out to memory, or
//   STAGED                   as bf16 through shared memory; out_at(t, g, c) is then where 16-byte chunk c of a row goes (nullptr: a padding
//                            row)
//   HOLE, hole0, hole1       keys [hole0, hole1) are seen by no row of the block: they are neither fetched nor multiplied
// The running maximum, its rescale and the division at the end are the online softmax of M. Milakov and N. Gimelshein ("Online normalizer
// calculation for softmax", 2018) as FlashAttention walks it over key tiles (T. Dao et al., 2022); the roles of the warps and scores
// multiplied one tile ahead follow the published schedule of FlashAttention-3 (J. Shah et al., 2024).
// See prefill_attn_tc.cu for the schedule here and what bounds it.
#pragma once
#include "common.cuh"
#include <cudaTypedefs.h>

namespace vb {

__device__ __forceinline__ void ptc_cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ptc_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void ptc_cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ float ptc_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// two fp32 values in a register pair: one instruction for both
__device__ __forceinline__ uint64_t ptc_pair(uint32_t a, uint32_t b) { return static_cast<uint64_t>(b) << 32 | a; }
__device__ __forceinline__ uint64_t ptc_pair(float a, float b) { return ptc_pair(__float_as_uint(a), __float_as_uint(b)); }
__device__ __forceinline__ float ptc_lo(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float ptc_hi(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
__device__ __forceinline__ uint64_t ptc_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t ptc_add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float ptc_max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// what two bf16 roundings left of their values, as bf16 (the differences are exact)
__device__ __forceinline__ uint32_t ptc_left(float p0, float p1, uint32_t h) {
  float d0, d1;
  asm("{\n\t.reg .b16 h0, h1, m;\n\tmov.b32 {h0, h1}, %2;\n\tmov.b16 m, 0xBF80;\n\tfma.rn.f32.bf16 %0, h0, m, %3;\n\tfma.rn.f32.bf16 %1, h1, m, %4;\n\t}\n"
      : "=f"(d0), "=f"(d1)
      : "r"(h), "f"(p0), "f"(p1));
  return pack_bf16(d0, d1);
}

constexpr int PTC_THREADS = 224;       // 4 softmax warps, 1 MMA warp, 2 loader warps
constexpr int PTC_KT = 64;             // tokens per K / V tile
constexpr int PTC_STAGES = 2;          // K and V tiles in flight, each with barriers of their own
constexpr float PTC_RESCALE = 8.f;     // growth of a row's maximum (base 2) that moves the exponents' reference

template <int D>
struct PtcLayout {
  static constexpr int TILE = PTC_KT * D * 2;               // [D / 64][64 tokens][64 dims] bf16
  static constexpr int Q = 0;                               // [D / 64][128][64]
  static constexpr int K = Q + 128 * D * 2;
  static constexpr int V = K + PTC_STAGES * TILE;
  static constexpr int BAR = V + PTC_STAGES * TILE;
  static constexpr int TOTAL = BAR + 256 + 1024;            // PtcShared, alignment slack
};

// B operand stored [k][n] with the n's contiguous (128-byte swizzled rows of 64 n, 8-row groups of k 1024 bytes apart, blocks of
// 64 n `block_bytes` apart)
__device__ __forceinline__ uint64_t umma_desc_sw128_mnmajor(uint32_t smem_addr, uint32_t block_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3ffffu) >> 4);
  d |= static_cast<uint64_t>(block_bytes >> 4) << 16;      // LBO
  d |= static_cast<uint64_t>(1024 >> 4) << 32;             // SBO
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
__device__ __forceinline__ void ptc_tma_5d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]; A: two bf16 per 32-bit column
__device__ __forceinline__ void umma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void ptc_tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]),
        "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]),
        "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void ptc_tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// barriers and scalars behind the operand tiles
struct PtcShared {
  uint64_t q_full, k_full[PTC_STAGES], k_empty[PTC_STAGES], v_full[PTC_STAGES], v_empty[PTC_STAGES];
  uint64_t s_full[2];       // scores complete
  uint64_t p_full[2];       // probabilities written, O ready to be added to
  uint64_t o_done;          // P V of a tile complete
  uint64_t o_last;          // ... of the last tile
  uint64_t v_part[PTC_STAGES];      // a V tile with rows that no row may see has landed (they are cleared next)
  uint32_t tmem;
  int tile[3];
  int warp_tot[PTC_THREADS / 32];
};

__device__ __forceinline__ void ptc_init(PtcShared* sh, int loader_arrivals) {
  mbar_init(&sh->q_full, 128);
  for (int i = 0; i < PTC_STAGES; ++i) {
    mbar_init(&sh->k_full[i], loader_arrivals);
    mbar_init(&sh->k_empty[i], 1);
    mbar_init(&sh->v_full[i], loader_arrivals);
    mbar_init(&sh->v_empty[i], 1);
    mbar_init(&sh->v_part[i], 1);
  }
  for (int i = 0; i < 2; ++i) {
    mbar_init(&sh->s_full[i], 1);
    mbar_init(&sh->p_full[i], 128);
  }
  mbar_init(&sh->o_done, 1);
  mbar_init(&sh->o_last, 1);
  fence_barrier_init();
  sh->tile[0] = -1;
}

// Accumulator rows r0, r0 + STEP, ... as (row of the tile, head of the group): one division for all of them
template <int STEP>
struct PtcWalk {
  int t, g, dt, dg, group;
  __device__ __forceinline__ PtcWalk(int r0, int group_) : t(r0 / group_), dt(STEP / group_), group(group_) {
    g = r0 - t * group;
    dg = STEP - dt * group;
  }
  __device__ __forceinline__ void next() {
    t += dt;
    g += dg;
    if (g >= group) {
      g -= group;
      ++t;
    }
  }
};
// Results as bf16 on their way out: a thread's row goes to the place of the query rows (the last scores have been multiplied), 16-byte chunk c
// of row r at chunk c ^ (r & 7) of its eight, and leaves in whole rows
template <int D>
__device__ __forceinline__ uint4* ptc_staged(uint8_t* smem, int r, int c) {
  return reinterpret_cast<uint4*>(smem + PtcLayout<D>::Q + r * D * 2) + ((c & ~7) | ((c ^ r) & 7));
}
template <int D>
__device__ __forceinline__ void ptc_put32(uint8_t* smem, int c0, const uint32_t (&o)[32], float f) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = pack_bf16(__uint_as_float(o[c * 8 + 2 * i]) * f, __uint_as_float(o[c * 8 + 2 * i + 1]) * f);
    *ptc_staged<D>(smem, threadIdx.x, (c0 >> 3) + c) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}
// all rows, once the four softmax warps have put theirs; none if one of them has given up
template <int D, class Rows>
__device__ __forceinline__ void ptc_send(uint8_t* smem, const Rows& rows, BoundedWait& bw) {
  constexpr int CPR = D / 8, STEP = 128 / CPR;
  if (warps_any<1, 128>(bw.dead)) {
    bw.dead = true;
    return;
  }
  const int c = threadIdx.x % CPR, r0 = threadIdx.x / CPR;
  PtcWalk<STEP> w(r0, rows.group);
#pragma unroll 4
  for (int i = 0; i < CPR; ++i, w.next()) {
    uint4* dst = rows.out_at(w.t, w.g, c);
    if (dst) *dst = *ptc_staged<D>(smem, r0 + i * STEP, c);
  }
}

// this thread's accumulated row, once the last tile has been multiplied
template <int D, class Rows>
__device__ __forceinline__ void ptc_finish_rows(uint8_t* smem, const Rows& rows, uint32_t t_lane, int n_tiles, float m_ref, float l_run) {
  tc_fence_after();
  const float f = rows.finish(m_ref, l_run);
#pragma unroll 1
  for (int c0 = 0; c0 < D; c0 += 32) {
    uint32_t o[32];
    if (n_tiles > 0) {
      tmem_ld_32x32(t_lane + 128 + c0, o);
      tmem_ld_wait();
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) o[i] = 0u;
    }
    if (rows.STAGED) ptc_put32<D>(smem, c0, o, f);
    else rows.store(c0, o, f);
  }
}

// ================= warps 0..3: softmax =================
template <int D, class Rows>
__device__ __forceinline__ void ptc_softmax(uint8_t* smem, PtcShared* sh, const Rows& rows, BoundedWait& bw) {
  using L = PtcLayout<D>;
  constexpr int KBD = D / 64, CPR = D * 2 / 16;
  const int tid = threadIdx.x, warp = tid >> 5, n_tiles = rows.n_tiles;
  {
    // CPR neighbouring threads take a row: a warp reads whole rows, four or two at a time.  (A row per thread, 16 bytes of 32 rows an
    // instruction: the rows were there after 6 us instead of 2.)
    __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(smem + L::Q);
    constexpr int STEP = 128 / CPR;
    const int c = tid % CPR, r0 = tid / CPR;
    uint4 v[CPR];
    PtcWalk<STEP> w(r0, rows.group);
#pragma unroll
    for (int i = 0; i < CPR; ++i, w.next()) {
      const __nv_bfloat16* src = rows.q_row(w.t, w.g);
      v[i] = make_uint4(0u, 0u, 0u, 0u);
      if (src) v[i] = *reinterpret_cast<const uint4*>(src + c * 8);
    }
#pragma unroll
    for (int i = 0; i < CPR; ++i) *reinterpret_cast<uint4*>(sQ + xt_index(r0 + i * STEP, c * 8, 128, KBD)) = v[i];
    fence_proxy_async();
    mbar_arrive(&sh->q_full);
  }
  const uint32_t t_lane = sh->tmem + (static_cast<uint32_t>(warp * 32) << 16);   // this warp's TMEM lane quarter
  const float scale = rows.scale_log2 > 0.f ? rows.scale_log2 : 1.f;
  float m_ref = -INFINITY, l_run = 0.f;            // the exponents' reference and the denominator against it
  for (int j = 0; j < n_tiles && !bw.dead; ++j) {
    const uint32_t sc = t_lane + (j & 1) * 64;
    bw.wait(&sh->s_full[j & 1], (j >> 1) & 1);
    if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
    tc_fence_after();
    uint32_t v[64];
    {
      uint32_t a[32], c[32];
      tmem_ld_32x32(sc, a);
      tmem_ld_32x32(sc + 32, c);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; ++i) { v[i] = a[i]; v[32 + i] = c[i]; }
    }
    const int tok0 = rows.tile(j) * PTC_KT;
    if (!(rows.scale_log2 > 0.f)) {                            // (a scale that is not positive goes in before the maximum)
#pragma unroll
      for (int i = 0; i < 64; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * rows.scale_log2);
    }
    if (!__all_sync(0xffffffffu, rows.full(tok0))) {           // some row of the warp does not see all of the tile
#pragma unroll
      for (int i = 0; i < 64; ++i)
        if (!rows.visible(tok0 + i)) v[i] = 0xff800000u;       // -inf
    }
    float m0 = -INFINITY, m1 = -INFINITY, m2 = -INFINITY, m3 = -INFINITY;
#pragma unroll
    for (int i = 0; i < 64; i += 8) {
      m0 = ptc_max3(m0, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
      m1 = ptc_max3(m1, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
      m2 = ptc_max3(m2, __uint_as_float(v[i + 4]), __uint_as_float(v[i + 5]));
      m3 = ptc_max3(m3, __uint_as_float(v[i + 6]), __uint_as_float(v[i + 7]));
    }
    const float mx = fmaxf(fmaxf(m0, m1), fmaxf(m2, m3)) * scale;
    const bool move = mx > m_ref + PTC_RESCALE || (m_ref == -INFINITY && mx > -INFINITY);
    if (__any_sync(0xffffffffu, move)) {
      const float alpha = move ? ptc_ex2(m_ref - mx) : 1.f;                  // ex2(-inf) = 0
      if (move) m_ref = mx;
      l_run *= alpha;
      if (j > 0) {
        bw.wait(&sh->o_done, (j - 1) & 1);                                   // tile j - 1 has been added
        if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
        tc_fence_after();
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t o[32];
          tmem_ld_32x32(t_lane + 128 + c0, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          ptc_tmem_st32(t_lane + 128 + c0, o);
        }
      }
    }
    const float u = m_ref == -INFINITY ? 0.f : m_ref;          // every key masked so far
    // a probability goes in as two bf16 terms, its rounding and what that left (relative 2^-17): the reference may lag, and the largest
    // of a row, 1 and exact against the maximum itself, need not be a power of two
    uint64_t l2 = ptc_pair(0.f, 0.f);
    const uint64_t scale2 = ptc_pair(scale, scale), u2 = ptc_pair(-u, -u);
    uint32_t ph[32], pl[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const uint64_t x = ptc_fma2(ptc_pair(v[2 * i], v[2 * i + 1]), scale2, u2);
      const float p0 = ptc_ex2(ptc_lo(x)), p1 = ptc_ex2(ptc_hi(x));
      l2 = ptc_add2(l2, ptc_pair(p0, p1));
      ph[i] = pack_bf16(p0, p1);
      pl[i] = ptc_left(p0, p1, ph[i]);
    }
    l_run += ptc_lo(l2) + ptc_hi(l2);
    ptc_tmem_st32(sc, ph);
    ptc_tmem_st32(sc + 32, pl);
    ptc_tmem_st_wait();
    tc_fence_before();
    mbar_arrive(&sh->p_full[j & 1]);
  }
  // ---- normalise and store this thread's row ----
  if (n_tiles > 0 && !bw.dead) {
    bw.wait(&sh->o_last, 0);
    if (!__all_sync(0xffffffffu, !bw.dead)) bw.dead = true;
  }
  if (!bw.dead) ptc_finish_rows<D>(smem, rows, t_lane, n_tiles, m_ref, l_run);
  if (rows.STAGED) ptc_send<D>(smem, rows, bw);          // (all four warps come here)
}

// ================= warp 4: MMA issuer (the whole warp walks the loop, one elected lane issues: operands stay in uniform registers) =================
template <int D>
__device__ __forceinline__ void ptc_issue(uint8_t* smem, PtcShared* sh, int n_tiles, BoundedWait& bw) {
  using L = PtcLayout<D>;
  constexpr int KBD = D / 64;
  const uint32_t tmem = sh->tmem;
  const uint32_t idesc_s = umma_idesc(128, PTC_KT, 1u), idesc_o = umma_idesc(128, D, 1u) | (1u << 16);   // (B of P V: MN-major)
  const uint64_t q_desc = umma_desc_sw128_kmajor(smem_u32(smem + L::Q));
  auto alive = [&]() {
    if (!__all_sync(0xffffffffu, !bw.dead)) bw.dead = true;
    return !bw.dead;
  };
  auto scores = [&](int j) {
    bw.wait(&sh->k_full[j & 1], (j >> 1) & 1);
    if (!alive()) return;
    tc_fence_after();
    const uint64_t k_desc = umma_desc_sw128_kmajor(smem_u32(smem + L::K + (j & 1) * L::TILE));
    if (elect_one()) {
#pragma unroll
      for (int kb = 0; kb < KBD; ++kb)
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16(tmem + (j & 1) * 64, q_desc + kb * (128 * 128 >> 4) + 2 * k, k_desc + kb * (PTC_KT * 128 >> 4) + 2 * k, idesc_s,
                    (kb > 0 || k > 0) ? 1u : 0u);
      umma_commit(&sh->k_empty[j & 1]);
      umma_commit(&sh->s_full[j & 1]);
    }
    __syncwarp();
  };
  if (n_tiles > 0) {
    bw.wait(&sh->q_full, 0);
    if (alive()) scores(0);
  }
  for (int j = 0; j < n_tiles && !bw.dead; ++j) {
    if (j + 1 < n_tiles) {
      // the other score buffer holds the probabilities of tile j - 1 until they have been multiplied
      if (j > 0) bw.wait(&sh->o_done, (j - 1) & 1);
      if (alive()) scores(j + 1);
    }
    bw.wait(&sh->p_full[j & 1], (j >> 1) & 1);
    bw.wait(&sh->v_full[j & 1], (j >> 1) & 1);
    if (!alive()) break;
    tc_fence_after();
    const uint64_t v_desc = umma_desc_sw128_mnmajor(smem_u32(smem + L::V + (j & 1) * L::TILE), PTC_KT * 128);
    if (elect_one()) {
#pragma unroll
      for (int k = 0; k < PTC_KT / 16; ++k) {        // 16 tokens: 8 columns of either term of the probabilities, two 8-row groups of V
        umma_bf16_ta(tmem + 128, tmem + (j & 1) * 64 + 32 + 8 * k, v_desc + k * (2048 >> 4), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
        umma_bf16_ta(tmem + 128, tmem + (j & 1) * 64 + 8 * k, v_desc + k * (2048 >> 4), idesc_o, 1u);
      }
      umma_commit(&sh->v_empty[j & 1]);
      umma_commit(&sh->o_done);
      if (j + 1 == n_tiles) umma_commit(&sh->o_last);
    }
    __syncwarp();
  }
}

// whether V tile j holds rows to clear: past the last key, or in the hole
template <class Rows>
__device__ __forceinline__ bool ptc_partial(const Rows& rows, int j, int kmax) {
  const int tok0 = rows.tile(j) * PTC_KT;
  return j + 1 == rows.n_tiles || (Rows::HOLE && max(tok0, rows.hole0) < min(tok0 + PTC_KT, rows.hole1));
}

// ================= warps 5 and 6: K tiles, V tiles =================
// Boxes of `bt` keys x 64 dims of one head; place(tok) -> (page, slot in it), fetch(page, slot, box destination, dim, barrier).  A lane finds the
// place of each of a tile's boxes while the tile in front is waited for; one lane issues.  (Found by the issuing lane, box by box, the divisions and
// the load from the page table stood in every tile's way: 0.1 us a box, 1.02 us a tile of 64 keys in pages of 128 and 2.1 in pages of 16; and with one
// warp for K and V a K tile stood behind the wait for a V stage.)
template <int D, class Rows, class Place, class Fetch>
struct PtcBoxes {
  const Rows& rows;
  int kmax, bt;
  Place place;
  Fetch fetch_box;
  __device__ __forceinline__ int2 find(int j) const {
    const int lane = threadIdx.x & 31;
    int2 at = make_int2(-1, 0);
    if (lane < PTC_KT / bt && j < rows.n_tiles) {
      const int tok = rows.tile(j) * PTC_KT + lane * bt;
      // (pages past the last key and pages inside the hole are not the request's)
      if (tok < kmax && !(Rows::HOLE && tok >= rows.hole0 && tok + bt <= rows.hole1)) at = place(tok);
    }
    return at;
  }
  __device__ __forceinline__ void issue(const int2& at, uint32_t dst, uint64_t* bar) const {
    const int lane = threadIdx.x & 31;
    const uint32_t there = __ballot_sync(0xffffffffu, at.x >= 0), mb = smem_u32(bar);
    if (lane == 0) mbar_arrive_expect_tx(bar, __popc(there) * bt * D * 2);
    for (int i = 0; i < PTC_KT / bt; ++i) {
      const int page = __shfl_sync(0xffffffffu, at.x, i), slot = __shfl_sync(0xffffffffu, at.y, i);
      if (lane == 0 && (there >> i & 1u)) {
#pragma unroll
        for (int kb = 0; kb < D / 64; ++kb) fetch_box(page, slot, dst + kb * (PTC_KT * 128) + i * bt * 128, kb * 64, mb);
      }
    }
  }
};
__device__ __forceinline__ void ptc_let_land(bool dead) {                  // copies in flight, before the block may leave
  if (!dead) return;
  const unsigned long long t0 = gtimer();
  while (gtimer() - t0 < 2000000ull) __nanosleep(1000);
}
template <int D, class Rows, class Place, class Fetch>
__device__ __forceinline__ void ptc_load_k(uint8_t* smem, PtcShared* sh, const Rows& rows, int kmax, int bt, BoundedWait& bw, Place place, Fetch fetch_box) {
  using L = PtcLayout<D>;
  const PtcBoxes<D, Rows, Place, Fetch> boxes{rows, kmax, bt, place, fetch_box};
  int2 at = boxes.find(0);
  for (int j = 0; j < rows.n_tiles; ++j) {
    const int2 next = boxes.find(j + 1);
    bw.wait(&sh->k_empty[j & 1], ((j >> 1) & 1) ^ 1);
    if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
    boxes.issue(at, smem_u32(smem + L::K + (j & 1) * L::TILE), &sh->k_full[j & 1]);
    at = next;
  }
  ptc_let_land(bw.dead);
}
// Rows of V tiles that no row may see are multiplied by probability 0: whatever the cache holds there, they must be finite.  The last tile of the walk holds
// key kmax - 1 and rows past it; tiles at the edges of the hole hold rows inside it.  They are cleared once the tile has landed.
template <int D, class Rows, class Place, class Fetch>
__device__ __forceinline__ void ptc_load_v(uint8_t* smem, PtcShared* sh, const Rows& rows, int kmax, int bt, BoundedWait& bw, Place place, Fetch fetch_box) {
  using L = PtcLayout<D>;
  constexpr int KBD = D / 64;
  const PtcBoxes<D, Rows, Place, Fetch> boxes{rows, kmax, bt, place, fetch_box};
  const int lane = threadIdx.x & 31;
  uint32_t turn = 0;                              // bit s: parity of stage s's next partial tile
  int2 at = boxes.find(0);
  for (int j = 0; j < rows.n_tiles; ++j) {
    const int s = j & 1;
    const bool partial = ptc_partial(rows, j, kmax);
    const int2 next = boxes.find(j + 1);
    bw.wait(&sh->v_empty[s], ((j >> 1) & 1) ^ 1);
    if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
    uint8_t* tile = smem + L::V + s * L::TILE;
    boxes.issue(at, smem_u32(tile), partial ? &sh->v_part[s] : &sh->v_full[s]);
    at = next;
    if (!partial) continue;
    bw.wait(&sh->v_part[s], turn >> s & 1u);
    if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
    turn ^= 1u << s;
    const int tok0 = rows.tile(j) * PTC_KT;
    auto clear = [&](int r0, int r1) {            // rows [r0, r1) of the tile
      const int chunks = (r1 - r0) * 8;
      for (int i = lane; i < KBD * chunks; i += 32) {
        const int kb = i / chunks, c = i - kb * chunks;
        *reinterpret_cast<uint4*>(tile + kb * (PTC_KT * 128) + r0 * 128 + c * 16) = make_uint4(0u, 0u, 0u, 0u);
      }
    };
    if (kmax - tok0 < PTC_KT) clear(kmax - tok0, PTC_KT);
    if (Rows::HOLE && max(tok0, rows.hole0) < min(tok0 + PTC_KT, rows.hole1))
      clear(max(rows.hole0 - tok0, 0), min(rows.hole1 - tok0, PTC_KT));
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh->v_full[s]);
  }
  ptc_let_land(bw.dead);
}

inline int ptc_box_tokens(int page_size) { return page_size % 64 == 0 ? 64 : (page_size % 32 == 0 ? 32 : (page_size % 16 == 0 ? 16 : 8)); }
PFN_cuTensorMapEncodeTiled_v12000 encode_fn();      // api.cu

}  // namespace vb
