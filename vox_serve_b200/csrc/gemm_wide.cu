// Dense projections Y[T][N] = X[T][K] * W[N][K]^T for steps of many rows (prompts), on pairs of SMs.
//
// The one-SM kernel of gemm.cu is built to stream weights past a few dozen rows.  With hundreds of rows it is bound by what
// an SM can pull out of L2: its 128 x 256 tile needs 48 KB of operands per 512 tensor-core cycles (94 B / cycle / SM), with a
// ring of two stages and an epilogue that nothing overlaps (395 TFLOP/s on a 1024-row prompt step).  Here
//   * two CTAs of a cluster issue ONE tcgen05.mma.cta_group::2 of 256 weight rows x up to 256 token rows: each CTA loads its
//     own 128 weight rows and HALF of the token rows, so the same product needs 32 KB per SM (64 B / cycle at 256 tokens);
//   * CTAs are persistent (one pair per two SMs) and walk a list of units (split, weight pair, token tile); two accumulators
//     of 256 TMEM columns alternate, so a unit's epilogue runs beside the next unit's products;
//   * the ring holds 3 or 4 stages of 128 k;
//   * the token tile is a launch parameter (a multiple of 16, at most 256): the host picks the one that fills the last wave.
//     With 148 SMs and 1024 rows, 256-token tiles leave the QKV projection of 5120 rows in 80 units on 74 pairs.
// Measured per launch (one-SM kernel -> this one, us): 1024 rows, QKV 5120 x 3072: 63 -> 32, O 3072 x 3072: 40 -> 19, gate/up
// 16384 x 3072: 171 -> 77 (1.34 PFLOP/s), down 3072 x 8192: 79 -> 38; 133 rows: 16 -> 11.4, 13.6 -> 10.4, 32 -> 28.5, 17.5 ->
// 13.7.  What bounds it now: operands out of L2 (with the products left out the copies alone run at 15.5 TB/s over all SMs,
// 0.31 us per 64-k block of a 256-token tile, where the tensor cores need 0.27) and the last wave.
// Operands: weights as vb_pack_weight_tiles lays them out (linear bulk copies); activations in the tiled XT layout (linear
// bulk copies, at most two per k-block where a token tile crosses a block of the layout) or row-major through a tensor map
// whose box is half a token tile.  Epilogues and rounding points are gemm.cu's (modes 0, 1, 2, clamped gate, groups).
//
// Warp roles per CTA: warp 0 producer, warp 1 MMA issuer (leader CTA) or relay (the other CTA: tells the leader that its
// half of a stage has landed), warps 2..9 epilogue (two per TMEM quarter, alternating 16-column chunks).
// Every wait is bounded (BoundedWait): a CTA whose wait runs out sets its flag, stops issuing and leaves.
#include "../../include/vb_api.h"
#define VB_PDL_FAMILY 2
#include "quotient.cuh"
#include <type_traits>

namespace vb {

constexpr int GW_THREADS = 320;
constexpr int GW_BLOCK_K = 64;
constexpr int GW_A_BYTES = 128 * 128;
constexpr int GW_ACC_COLS = 256;
constexpr int GW_KPS = 2;            // k-blocks per ring stage: the hand-shakes of a pair cost about 0.26 us per stage whatever it holds
constexpr int GW_MAX_STAGES = 4;

struct GemmWideParams {
  void* y;
  const uint8_t* w_tiles;
  const uint8_t* x_tiles;      // XT(x_tile) layout, or nullptr: x_map
  const __nv_bfloat16* bias;
  const int32_t* tile_group;   // group of every token tile (nullptr: one group)
  const int4* tiles;           // or a table of token tiles: [0].x of them, then (group, first row, rows, -) each
  int tiles_max;
  long long group_bytes;
  int T, N, K, ldy, mode, split_k, tile_rows, sub, n_out, act, y_tiled, x_tile;
  int n_tok;                   // token rows per tile (multiple of 16, <= 256)
  int stages, num_kb, n_tiles, n_pairs, t_blocks, units, w_kb_stride, group_kb, kb_base;
  float glu_limit, glu_slope;
  unsigned char* wait_flag;
};

__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
// Nothing that a thread wrote travels with these arrivals (operands are written by the copy engine, accumulators read
// through tcgen05), so they need no release at cluster scope; with one, every stage cost the relay a fence of 0.75 us.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void umma2_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on the barrier at this offset in both CTAs of the pair once the MMAs issued so far have completed
__device__ __forceinline__ void umma2_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3))
      : "memory");
}
__device__ __forceinline__ void gw_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void gw_tma_2d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}

__device__ __forceinline__ float gw_act(float v, int act) {
  if (act == 1) { const float r = fmaxf(v, 0.f); return r * r; }
  if (act == 2) return 0.5f * v * (1.f + erff(v * 0.70710678118654752f));
  if (act == 3) return 0.5f * v * (1.f + tanhf(0.79788456080286536f * (v + 0.044715f * v * v * v)));
  return v;
}

// boxes of half a token tile, by its rows: a table's tiles differ, and what a box has beyond its tile is copied for nothing
constexpr int GW_BOXES = 4;
template <bool TABLE>
struct GwMaps {
  CUtensorMap m[TABLE ? GW_BOXES : 1];     // 64, 80, 96, 128 rows; without a table half of n_tok
};
__host__ __device__ __forceinline__ int gw_box(int half) { return half <= 64 ? 0 : half <= 80 ? 1 : half <= 96 ? 2 : 3; }
__host__ __device__ __forceinline__ int gw_box_rows(int i) { return i == 0 ? 64 : i == 1 ? 80 : i == 2 ? 96 : 128; }
struct GwUnit {
  int split, pair, tblk, kb0, kb1, t0, n_cur;    // n_cur: token rows of the tile rounded up to 16
};
struct GwTableUnit : GwUnit {
  int t_end, group;
};
template <bool TABLE>
__device__ __forceinline__ std::conditional_t<TABLE, GwTableUnit, GwUnit> gw_unit(const GemmWideParams& p, const int4* table, int n_tiles, int u) {
  std::conditional_t<TABLE, GwTableUnit, GwUnit> r;
  if constexpr (TABLE) {
    r.split = 0;
    r.pair = u / n_tiles;
    r.tblk = u - r.pair * n_tiles;
    r.kb0 = 0;
    r.kb1 = p.num_kb;
    const int4 t = table[r.tblk];
    r.group = t.x;
    r.t0 = t.y;
    r.t_end = t.y + t.z;
    r.n_cur = (t.z + 15) & ~15;
    return r;
  }
  // token tiles fastest: the pairs that run side by side share weight tiles in L2
  const int per_split = p.n_pairs * p.t_blocks;
  r.split = u / per_split;
  const int rem = u - r.split * per_split;
  r.pair = rem / p.t_blocks;
  r.tblk = rem - r.pair * p.t_blocks;
  r.kb0 = static_cast<int>(static_cast<long long>(r.split) * p.num_kb / p.split_k);
  r.kb1 = static_cast<int>(static_cast<long long>(r.split + 1) * p.num_kb / p.split_k);
  r.t0 = r.tblk * p.n_tok;
  r.n_cur = min(p.n_tok, (p.T - r.t0 + 15) & ~15);
  return r;
}

__device__ __forceinline__ int gw_end(const GemmWideParams& p, const GwUnit&) { return p.T; }
__device__ __forceinline__ int gw_end(const GemmWideParams&, const GwTableUnit& g) { return g.t_end; }
// (bounded to 128 registers: what is left of the file holds the first blocks of the kernel behind this one, which start early)
template <bool TABLE>          // token tiles from a table (p.tiles)
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(480, 1)
    gemm_wide_kernel(const GemmWideParams p, const __grid_constant__ GwMaps<TABLE> maps) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int b_bytes = p.n_tok * 64;                 // half of the token tile's rows (a multiple of 1024)
  const int b_off = GW_KPS * GW_A_BYTES;            // a stage: the weight blocks of GW_KPS k-blocks, then their token blocks
  const int stage_bytes = GW_KPS * (GW_A_BYTES + b_bytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes);   // this CTA's copies have landed
  uint64_t* peer = full + GW_MAX_STAGES;                                          // (leader) the other CTA's have
  uint64_t* empty = peer + GW_MAX_STAGES;                                         // the MMAs have read the stage
  uint64_t* acc_full = empty + GW_MAX_STAGES;                                     // [2]
  uint64_t* acc_empty = acc_full + 2;                                             // (leader) [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const uint32_t gate = smem_u32(tmem_slot + 1);                                  // set once the kernels in front have completed
  int4* table = reinterpret_cast<int4*>(smem + p.stages * stage_bytes + 512);     // of p.tiles

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;
  BoundedWait bw{p.wait_flag, gate};

  if (warp == 0 && lane == 0) {
    tmem_slot[1] = 0u;
    if (!p.x_tiles) prefetch_tmap(&maps.m[0]);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&peer[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 16);                 // eight epilogue warps of either CTA
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * GW_ACC_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
#define GW_UNITS (TABLE ? n_tiles * p.n_pairs : p.units)
  // (the table does not come from the kernel in front, but from one before it: it has completed)
  const int n_tiles = TABLE ? min(__ldcg(reinterpret_cast<const int*>(p.tiles)), p.tiles_max) : 0;
  if (TABLE)
    for (int i = threadIdx.x; i < n_tiles; i += GW_THREADS) table[i] = __ldcg(p.tiles + 1 + i);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ================= producer =================
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      const uint32_t a_rows_bytes = static_cast<uint32_t>(p.tile_rows) * 128u;
      bool waited = false;
      const uint32_t smem_a = smem_u32(smem), bar_full = smem_u32(full);
      for (int u = first; u < GW_UNITS; u += step) {
        const auto g = gw_unit<TABLE>(p, table, n_tiles, u);
        const int w0 = (g.pair * 2 + static_cast<int>(rank)) * p.sub;
        const int n_sub = max(0, min(p.sub, p.n_tiles - w0));
        const size_t w_kbs = p.w_kb_stride ? p.w_kb_stride : p.num_kb;
        const size_t sub_stride = w_kbs * a_rows_bytes;          // from one weight tile to the next
        const int half = g.n_cur >> 1, row0 = g.t0 + static_cast<int>(rank) * half;
        // token rows in the tiled layout: [row0, row0 + half) may cross from one block of x_tile rows into the next
        const int xb = p.x_tiles ? row0 / p.x_tile : 0, in0 = row0 - xb * p.x_tile;
        const uint32_t r0 = static_cast<uint32_t>(p.x_tiles ? min(half, p.x_tile - in0) : 0) * 128u;
        const uint32_t r1 = p.x_tiles ? static_cast<uint32_t>(half) * 128u - r0 : 0u;
        const uint32_t bytes = static_cast<uint32_t>(n_sub) * a_rows_bytes + (p.x_tiles ? r0 + r1 : static_cast<uint32_t>(TABLE ? gw_box_rows(gw_box(half)) * 128 : b_bytes));
        const size_t x_step = static_cast<size_t>(p.x_tile) * 128;
        // a single thread feeds the ring: what it does per stage is kept to a handful of additions
        const uint8_t* wsrc = p.w_tiles + static_cast<size_t>(w0) * sub_stride + static_cast<size_t>(p.kb_base + g.kb0) * a_rows_bytes;
        const uint8_t* xsrc = p.x_tiles ? p.x_tiles + (static_cast<size_t>(xb) * p.num_kb + g.kb0) * x_step + static_cast<size_t>(in0) * 128
                                        : nullptr;
        const uint8_t* xsrc1 = p.x_tiles ? p.x_tiles + (static_cast<size_t>(xb + 1) * p.num_kb + g.kb0) * x_step : nullptr;
        int kx = g.kb0 * GW_BLOCK_K;
        auto load_a = [&](uint32_t dst, int nk, uint32_t bar) {
          if (p.tile_rows == 128) {                     // the tile's k-blocks lie side by side: one copy
            if (n_sub > 0) gw_bulk(dst, wsrc, nk * GW_A_BYTES, bar);
          } else {
            for (int j = 0; j < nk; ++j)
              for (int i = 0; i < n_sub; ++i)
                gw_bulk(dst + j * GW_A_BYTES + i * a_rows_bytes, wsrc + j * a_rows_bytes + i * sub_stride, a_rows_bytes, bar);
          }
          wsrc += nk * a_rows_bytes;
        };
        auto load_b = [&](uint32_t dst, int nk, uint32_t bar) {
          for (int j = 0; j < nk; ++j, dst += b_bytes) {
            if (xsrc) {
              gw_bulk(dst, xsrc, r0, bar);
              if (r1) gw_bulk(dst + r0, xsrc1, r1, bar);
              xsrc += x_step;
              xsrc1 += x_step;
            } else {
              gw_tma_2d(dst, &maps.m[TABLE ? gw_box(half) : 0], bar, kx, row0);
              kx += GW_BLOCK_K;
            }
          }
        };
        int kb = g.kb0;
        if (!waited) {
          // the first ring pass of weights does not depend on the previous kernel (the groups of token tiles do)
          const int npre = min(p.stages, (g.kb1 - g.kb0 + GW_KPS - 1) / GW_KPS);
          auto pre_a = [&]() {
            for (int i = 0; i < npre; ++i) {
              const int nk = min(GW_KPS, g.kb1 - g.kb0 - i * GW_KPS);
              mbar_arrive_expect_tx(&full[i], nk * bytes);
              load_a(smem_a + i * stage_bytes, nk, bar_full + 8 * i);
            }
          };
          if constexpr (TABLE) wsrc += g.group * (p.group_bytes + static_cast<size_t>(p.group_kb) * a_rows_bytes);
          if (TABLE || !p.tile_group) pre_a();
          pdl_wait();
          wait_gate_open(gate);
          pdl_trigger();
          if (!TABLE && p.tile_group) {
            const size_t grp = p.tile_group[g.tblk];
            wsrc += grp * p.group_bytes + grp * p.group_kb * a_rows_bytes;
            pre_a();
          }
          for (int i = 0; i < npre; ++i)
            load_b(smem_a + i * stage_bytes + b_off, min(GW_KPS, g.kb1 - g.kb0 - i * GW_KPS), bar_full + 8 * i);
          kb += npre * GW_KPS;
          s = npre == p.stages ? 0 : npre;
          ph = npre == p.stages ? 1u : 0u;
          waited = true;
        } else if constexpr (TABLE) {
          wsrc += g.group * (p.group_bytes + static_cast<size_t>(p.group_kb) * a_rows_bytes);
        } else if (p.tile_group) {
          const size_t grp = p.tile_group[g.tblk];
          wsrc += grp * p.group_bytes + grp * p.group_kb * a_rows_bytes;
        }
        uint32_t dst = smem_a + s * stage_bytes;
        for (; kb < g.kb1; kb += GW_KPS) {
          const int nk = min(GW_KPS, g.kb1 - kb);
          bw.wait(&empty[s], ph ^ 1u);
          if (bw.dead) break;
          const uint32_t bar = bar_full + 8 * s;
          mbar_arrive_expect_tx(&full[s], nk * bytes);
          load_a(dst, nk, bar);
          load_b(dst + b_off, nk, bar);
          dst += stage_bytes;
          if (++s == p.stages) { s = 0; ph ^= 1u; dst = smem_a; }
        }
        if (bw.dead) break;
      }
      if (!waited) { pdl_wait(); pdl_trigger(); }       // (a pair without units: nobody waits)
      if (bw.dead) {                                    // let the copies in flight land before the block may leave
        const unsigned long long t0 = gtimer();
        while (gtimer() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    int s = 0, it = 0;
    uint32_t ph = 0;
    if (rank == 0) {
      // ================= MMA issuer =================
      // (the whole warp walks the loop and one elected lane issues: the operands stay in uniform registers; with a loop under
      // `if (lane == 0)` moving them there cost 70 cycles per MMA)
      const uint64_t desc0 = umma_desc_sw128_kmajor(smem_u32(smem));
      for (int u = first; u < GW_UNITS && !bw.dead; u += step, ++it) {
        const auto g = gw_unit<TABLE>(p, table, n_tiles, u);
        const int acc = it & 1;
        bw.wait(&acc_empty[acc], ((it >> 1) & 1) ^ 1);
        if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
        tc_fence_after();
        const uint32_t d = tmem_base + acc * GW_ACC_COLS, idesc = umma_idesc(256, g.n_cur, 1u);
        for (int kb = g.kb0; kb < g.kb1; kb += GW_KPS) {
          bw.wait(&full[s], ph);
          bw.wait(&peer[s], ph);
          if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
          tc_fence_after();
          const uint64_t a0 = desc0 + static_cast<uint64_t>(s) * (stage_bytes >> 4), b0 = a0 + (b_off >> 4);
          const int nk = min(GW_KPS, g.kb1 - kb);
          if (elect_one()) {
            for (int j = 0; j < nk; ++j) {
              const uint64_t a_desc = a0 + j * (GW_A_BYTES >> 4), b_desc = b0 + j * (b_bytes >> 4);
#pragma unroll
              for (int k = 0; k < GW_BLOCK_K / 16; ++k)
                umma2_bf16(d, a_desc + 2 * k, b_desc + 2 * k, idesc, (kb > g.kb0 || j > 0 || k > 0) ? 1u : 0u);
            }
            umma2_commit(&empty[s]);
            if (kb + GW_KPS >= g.kb1) umma2_commit(&acc_full[acc]);
          }
          __syncwarp();
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
      }
    } else if (lane == 0) {
      // ================= relay: this CTA's half of a stage has landed =================
      const uint32_t peer0 = cluster_addr(peer, 0);
      for (int u = first; u < GW_UNITS && !bw.dead; u += step) {
        const auto g = gw_unit<TABLE>(p, table, n_tiles, u);
        for (int kb = g.kb0; kb < g.kb1; kb += GW_KPS) {
          bw.wait(&full[s], ph);
          if (bw.dead) break;
          mbar_arrive_cluster(peer0 + 8 * s);
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else {
    // ================= epilogue =================
    const int quarter = warp & 3, wg = (warp - 2) >> 2;      // TMEM lanes [32 quarter, +32); chunks wg, wg + 2, ...
    const int row = quarter * 32 + lane;
    const int sub_i = (quarter * 32) / p.tile_rows;           // which of the CTA's weight tiles this quarter's rows belong to
    const int row_in = row - sub_i * p.tile_rows;
    int it = 0;
    for (int u = first; u < GW_UNITS && !bw.dead; u += step, ++it) {
      const auto g = gw_unit<TABLE>(p, table, n_tiles, u);
      const int acc = it & 1;
      const int tile = (g.pair * 2 + static_cast<int>(rank)) * p.sub + sub_i;
      const bool row_ok = sub_i < p.sub && row_in < p.tile_rows && tile < p.n_tiles;
      bw.wait(&acc_full[acc], (it >> 1) & 1);
      if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * GW_ACC_COLS + (static_cast<uint32_t>(quarter * 32) << 16);
      if (p.mode == 2) {
        const int h = p.tile_rows >> 1, q_in = row_in >> 5;
        const bool hi = lane >= 16;
        const int n_out = tile * h + q_in * 16 + (lane & 15);
        const bool live = row_ok && n_out < p.n_out;
        __nv_bfloat16* y = static_cast<__nv_bfloat16*>(p.y);
        const int nkb_y = (p.n_out + 63) >> 6, yk = (n_out >> 3) & 7;
        for (int c0 = wg * 16; c0 < g.n_cur; c0 += 32) {
          uint32_t v[16];
          tmem_ld_32x16(taddr + c0, v);
          // 16 tokens from a multiple of 16 lie in one block of the tiled layout
          const int tc = g.t0 + c0, tb = p.y_tiled ? tc / p.x_tile : 0, tt = tc - tb * p.x_tile;
          __nv_bfloat16* yc = p.y_tiled ? y + ((static_cast<size_t>(tb) * nkb_y + (n_out >> 6)) * p.x_tile + tt) * 64 + (n_out & 7)
                                        : y + static_cast<size_t>(tc) * p.ldy + n_out;
          tmem_ld_wait();
          // this lane finishes tokens c0 + 2 i + hi: gate from the low half-warp, up from the high one.  The eight values are
          // taken through each step together (no branch inside: uniform choices stand outside the loops), or a warp waits out
          // every exponential and division on its own: 18 us per 256-token unit, more than its products take (gate/up of 1024
          // rows: 86 -> 77 us)
          float gt[8], up[8], o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float mine = __uint_as_float(hi ? v[2 * i + 1] : v[2 * i]);
            const float send = __uint_as_float(hi ? v[2 * i] : v[2 * i + 1]);
            const float other = __shfl_xor_sync(0xffffffffu, send, 16);
            gt[i] = hi ? other : mine;
            up[i] = hi ? mine : other;
          }
          if (p.glu_limit > 0.f) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              gt[i] = fminf(gt[i], p.glu_limit);
              up[i] = fminf(fmaxf(up[i], -p.glu_limit), p.glu_limit);
              o[i] = 1.0f + expf(-p.glu_slope * gt[i]);
            }
            div8(gt, o);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = gt[i] * (up[i] + 1.0f);
          } else if (p.act == 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = gw_act(gt[i], 1) * up[i];
          } else if (p.act == 2) {
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = gw_act(gt[i], 2) * up[i];
          } else if (p.act == 3) {
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = gw_act(gt[i], 3) * up[i];
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              gt[i] = round_bf16(gt[i]);
              o[i] = 1.0f + expf(-gt[i]);
            }
            div8(gt, o);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = round_bf16(gt[i]) * round_bf16(up[i]);
          }
          const int lim = live ? gw_end(p, g) - tc : 0;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int j = 2 * i + (hi ? 1 : 0);
            const size_t yi = p.y_tiled ? static_cast<size_t>(j * 64 + ((yk ^ (j & 7)) << 3)) : static_cast<size_t>(j) * p.ldy;
            if (j < lim) yc[yi] = __float2bfloat16_rn(o[i]);
          }
        }
      } else {
        const int n = tile * p.tile_rows + row_in;
        const bool live = row_ok && n < p.N;
        if (p.mode == 1) {
          float* y = static_cast<float*>(p.y) + static_cast<size_t>(g.split) * p.T * p.ldy + n;
          for (int c0 = wg * 16; c0 < g.n_cur; c0 += 32) {
            uint32_t v[16];
            tmem_ld_32x16(taddr + c0, v);
            tmem_ld_wait();
            if (live) {
              const int t = g.t0 + c0, m = min(16, gw_end(p, g) - t);
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (j < m) y[static_cast<size_t>(t + j) * p.ldy] = __uint_as_float(v[j]);
            }
          }
        } else {
          __nv_bfloat16* y = static_cast<__nv_bfloat16*>(p.y) + n;
          const float bv = (p.bias && live) ? __bfloat162float(p.bias[n]) : 0.f;
          for (int c0 = wg * 16; c0 < g.n_cur; c0 += 32) {
            uint32_t v[16];
            tmem_ld_32x16(taddr + c0, v);
            tmem_ld_wait();
            float a[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) a[j] = __uint_as_float(v[j]) + bv;
            if (p.act == 1) {
#pragma unroll
              for (int j = 0; j < 16; ++j) a[j] = gw_act(a[j], 1);
            } else if (p.act == 2) {
#pragma unroll
              for (int j = 0; j < 16; ++j) a[j] = gw_act(a[j], 2);
            } else if (p.act == 3) {
#pragma unroll
              for (int j = 0; j < 16; ++j) a[j] = gw_act(a[j], 3);
            }
            if (live) {
              const int t = g.t0 + c0, m = min(16, gw_end(p, g) - t);
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (j < m) y[static_cast<size_t>(t + j) * p.ldy] = __float2bfloat16_rn(a[j]);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[acc], 0));
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();          // no CTA leaves while its peer may still arrive on its barriers or multiply its operands
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * GW_ACC_COLS) : "memory");
  }
}

#undef GW_UNITS

static int gw_pairs() { return sm_count() / 2; }

}  // namespace vb

using namespace vb;

extern "C" {

int vb_gemm_wide_timeouts(void) {
  return wait_ran_out(WK_GEMM_WIDE);
}

static int gw_launch(void* d_y, const void* d_w_tiles, const void* const* x_maps, const void* d_x_tiles, int T, int N, int K, int ldy,
                      int mode, int split_k, int tile_rows, int n_out, int y_tiled, const void* d_bias, int act, int n_tok,
                      const int32_t* d_tile_group, const int32_t* d_tiles, int tiles_max, long long group_bytes, int w_kb_stride, int group_kb, int kb_base,
                      float glu_limit, float glu_slope, void* stream) {
  VB_CHECK_ARG(d_y && d_w_tiles && (x_maps || d_x_tiles), "vb_gemm_bf16_wide: null pointer");
  VB_CHECK_ARG(T > 0 && N > 0 && K > 0 && K % 8 == 0, "vb_gemm_bf16_wide: T=%d N=%d K=%d (K a multiple of 8)", T, N, K);
  VB_CHECK_ARG(mode >= 0 && mode <= 2, "vb_gemm_bf16_wide: mode %d", mode);
  VB_CHECK_ARG(mode == 1 || split_k == 1, "vb_gemm_bf16_wide: split_k > 1 needs mode 1 (fp32 partials)");
  VB_CHECK_ARG(act >= 0 && act <= 3 && (act == 0 || mode != 1), "vb_gemm_bf16_wide: activation %d is a mode 0 / 2 option", act);
  VB_CHECK_ARG(!d_bias || mode == 0, "vb_gemm_bf16_wide: bias is a mode 0 option");
  VB_CHECK_ARG(!y_tiled || (mode == 2 && d_x_tiles), "vb_gemm_bf16_wide: tiled output is a mode 2 option beside tiled input");
  VB_CHECK_ARG(tile_rows == 32 || tile_rows == 64 || tile_rows == 96 || tile_rows == 128, "vb_gemm_bf16_wide: tile_rows %d", tile_rows);
  VB_CHECK_ARG(mode != 2 || N % tile_rows == 0, "vb_gemm_bf16_wide: mode 2 needs N %% tile_rows == 0");
  VB_CHECK_ARG(n_tok >= 16 && n_tok <= 256 && n_tok % 16 == 0, "vb_gemm_bf16_wide: n_tok %d outside [16, 256] or not a multiple of 16", n_tok);
  VB_CHECK_ARG(group_bytes >= 0 && w_kb_stride >= 0 && group_kb >= 0 && kb_base >= 0, "vb_gemm_bf16_wide: offsets");
  VB_CHECK_ARG(!(d_tile_group || d_tiles) || x_maps, "vb_gemm_bf16_wide: groups need row-major activations");
  VB_CHECK_ARG(glu_limit >= 0.f && (glu_limit == 0.f || (mode == 2 && act == 0)), "vb_gemm_bf16_wide: a positive limit belongs to mode 2 without an activation");
  VB_CHECK_ARG(!d_tiles || (tiles_max > 0 && tiles_max <= 4096 && reinterpret_cast<uintptr_t>(d_tiles) % 16 == 0 && split_k == 1 && !d_x_tiles && !d_tile_group && n_tok == 256),
               "vb_gemm_bf16_wide: a table of tiles stands alone, on a 16-byte boundary, with up to 4096 of them");
  GemmWideParams p = {};
  VB_CHECK_ARG(p.wait_flag = wait_flag(WK_GEMM_WIDE), "vb_gemm_bf16_wide: no mapped host memory");
  p.num_kb = (K + GW_BLOCK_K - 1) / GW_BLOCK_K;
  VB_CHECK_ARG(split_k >= 1 && split_k <= p.num_kb, "vb_gemm_bf16_wide: split_k %d outside [1, %d]", split_k, p.num_kb);
  p.y = d_y; p.w_tiles = static_cast<const uint8_t*>(d_w_tiles); p.x_tiles = static_cast<const uint8_t*>(d_x_tiles);
  p.bias = static_cast<const __nv_bfloat16*>(d_bias);
  p.tile_group = d_tile_group; p.tiles = reinterpret_cast<const int4*>(d_tiles); p.tiles_max = tiles_max;
  p.group_bytes = group_bytes; p.w_kb_stride = w_kb_stride; p.group_kb = group_kb; p.kb_base = kb_base;
  p.T = T; p.N = N; p.K = K; p.ldy = ldy; p.mode = mode; p.split_k = split_k; p.tile_rows = tile_rows; p.sub = 128 / tile_rows;
  p.n_out = n_out > 0 ? n_out : (mode == 2 ? N / 2 : N);
  p.act = act; p.y_tiled = y_tiled; p.x_tile = vb_gemm_t_tile(T); p.n_tok = n_tok;
  p.glu_limit = glu_limit; p.glu_slope = glu_slope;
  p.n_tiles = (N + tile_rows - 1) / tile_rows;
  p.n_pairs = (p.n_tiles + 2 * p.sub - 1) / (2 * p.sub);
  p.t_blocks = (T + n_tok - 1) / n_tok;
  VB_CHECK_ARG(static_cast<long long>(p.n_pairs) * p.t_blocks * split_k <= 0x3fffffffLL, "vb_gemm_bf16_wide: too many tiles");
  p.units = p.n_pairs * p.t_blocks * split_k;
  const int stage_bytes = GW_KPS * (GW_A_BYTES + n_tok * 64);
  const int tail = 1024 /*barriers*/ + 1024 /*alignment*/ + tiles_max * 16;
  p.stages = min(GW_MAX_STAGES, (VB_MAX_DYN_SMEM - tail) / stage_bytes);
  const int smem = p.stages * stage_bytes + tail;
  if (d_tiles) {
    const int pairs = static_cast<int>(min(static_cast<long long>(p.n_pairs) * tiles_max, static_cast<long long>(gw_pairs())));
    GwMaps<true> maps;
    for (int i = 0; i < GW_BOXES; ++i) {
      VB_CHECK_ARG(x_maps[i], "vb_gemm_bf16_wide: null pointer");
      maps.m[i] = *static_cast<const CUtensorMap*>(x_maps[i]);
    }
    VB_CHECK_CUDA(max_dyn_smem_once(gemm_wide_kernel<true>));
    VB_CHECK_CUDA(launch_kernel(gemm_wide_kernel<true>, dim3(2 * pairs), dim3(GW_THREADS), smem, static_cast<cudaStream_t>(stream), true, p, maps));
    return 0;
  }
  static const GwMaps<false> none = {};
  VB_CHECK_CUDA(max_dyn_smem_once(gemm_wide_kernel<false>));
  VB_CHECK_CUDA(launch_kernel(gemm_wide_kernel<false>, dim3(2 * min(p.units, gw_pairs())), dim3(GW_THREADS), smem, static_cast<cudaStream_t>(stream), true, p,
                              x_maps ? *static_cast<const GwMaps<false>*>(x_maps[0]) : none));
  return 0;
}

int vb_gemm_bf16_wide_grouped(void* d_y, const void* d_w_tiles, const void* x_map, const void* d_x_tiles, int T, int N, int K, int ldy,
                      int mode, int split_k, int tile_rows, int n_out, int y_tiled, const void* d_bias, int act, int n_tok,
                      const int32_t* d_tile_group, long long group_bytes, int w_kb_stride, int group_kb, int kb_base,
                      float glu_limit, float glu_slope, void* stream) {
  return gw_launch(d_y, d_w_tiles, x_map ? &x_map : nullptr, d_x_tiles, T, N, K, ldy, mode, split_k, tile_rows, n_out, y_tiled, d_bias, act, n_tok, d_tile_group,
                   nullptr, 0, group_bytes, w_kb_stride, group_kb, kb_base, glu_limit, glu_slope, stream);
}

int vb_gemm_bf16_wide_tiles(void* d_y, const void* d_w_tiles, const void* const* x_maps, int T, int N, int K, int ldy, int mode, int tile_rows, int n_out, int act,
                            const int32_t* d_tiles, int tiles_max, long long group_bytes, int w_kb_stride, int group_kb, float glu_limit, float glu_slope, void* stream) {
  VB_CHECK_ARG(d_tiles && x_maps, "vb_gemm_bf16_wide_tiles: null pointer");
  return gw_launch(d_y, d_w_tiles, x_maps, nullptr, T, N, K, ldy, mode, 1, tile_rows, n_out, 0, nullptr, act, 256, nullptr, d_tiles, tiles_max, group_bytes, w_kb_stride,
                   group_kb, 0, glu_limit, glu_slope, stream);
}

int vb_gemm_bf16_wide(void* d_y, const void* d_w_tiles, const void* x_map, const void* d_x_tiles, int T, int N, int K, int ldy,
                      int mode, int split_k, int tile_rows, int n_out, int y_tiled, const void* d_bias, int act, int n_tok,
                      void* stream) {
  return vb_gemm_bf16_wide_grouped(d_y, d_w_tiles, x_map, d_x_tiles, T, N, K, ldy, mode, split_k, tile_rows, n_out, y_tiled, d_bias, act,
                                   n_tok, nullptr, 0, 0, 0, 0, 0.f, 0.f, stream);
}

}  // extern "C"
