// Vocoder convolutions over channels-last activations [B][T][C] (fp32), on tcgen05 with fp32-grade products.
//
// The channel-first kernel (snac_mma.cu) gathers its activation operand with one strided load per element, splits it in
// registers and stores both halves to shared memory: 1.5 - 2 us per 32-deep k-block however small the problem, no overlap of
// the epilogue, a 128-row weight tile even for layers of 32 channels, and layers narrower than 128 channels left to CUDA
// cores.  With the channels innermost the convolution is a plain matrix product per tap:
//   D[position][n] += sum_c X[position - shift(tap)][c] * W[tap][n][c]
// whose activation tile (128 positions x 32 channels) is one box of a tensor map -- positions before the start and past the
// end are the map's zero fill, short sequences put several batch entries into one box -- and whose output rows are contiguous.
// A transposed convolution of stride s is the same product with two taps and n = (phase, channel): row n of the result holds
// the s output positions of input position n.
//
// Products: x = hi + lo and w = hi + lo, both halves rounded to tf32 (to nearest), lo_w hi_x + hi_w lo_x + hi_w hi_x with
// fp32 accumulation; what is dropped is below 2^-22 of a product (the channel-first kernel truncates: 2^-20).
//
// Roles of a CTA's eighteen warps: 0 copies (activation box and two weight tiles per stage), 1 issues the MMAs, 2..5 split a
// stage's raw activations into the two halves and put them into TMEM as the MMA's A operand (128 x 32 columns each; through
// shared memory the operand would cost 12 KB of its bandwidth per 8-deep product, and the two tiles another 32 KB of stores),
// 6..17 are the epilogue.  Persistent CTAs, two accumulators, 4 stages (6 where column tiles are 32 wide): TMEM bounds them.
// The width of a column tile (32, 64 or 128) is chosen per launch from the number of tiles: a transformer layer of 640 rows
// has 5 x 4 tiles of 128.
// What bounds it: wide layers of few positions are one chain of 32-deep k-blocks (0.41 us each, the split into halves), narrow
// layers of many positions the epilogue (1x1 with residual, 614400 positions of 64 channels: 393 MB in 126 us).
// Measured (one pass): SNAC 32 windows 1454 us channel-first, 651 here; 1 window 711 and 262; Mimi 32 chunks 6721 and 1930.
// Of that, the residual's rows asked for before the accumulator is waited for: Mimi 2499 -> 2407; 16 columns at a time on twelve warps
// without a spilled register, where 32 on eight spilled 53: Mimi 2403 -> 1933, SNAC 746 -> 647 and 313 -> 266.
#include "../../include/vb_api.h"
#define VB_PDL_FAMILY 32
#include "common.cuh"
#include <cudaTypedefs.h>

namespace vb {
PFN_cuTensorMapEncodeTiled_v12000 encode_fn();      // api.cu

constexpr int CL_THREADS = 576;
constexpr int CL_A_BYTES = 128 * 128;       // 128 positions x 32 channels
constexpr int CL_MAX_STAGES = 6;            // 512 TMEM columns less two accumulators, 64 a stage
constexpr int CL_EPI_WARPS = 12;
constexpr int CL_EPI_BYTES = CL_EPI_WARPS * 2048;      // a transpose of 32 rows x 16 columns per epilogue warp

struct ClConvParams {
  const uint8_t* w;          // [tap * kb][hi | lo][n_pad][32], rows swizzled
  float* y;                  // [b * y_bstride + t * ldy + n]
  float* y2;                 // optional: the activated values; y then holds the plain ones
  const float* bias;         // [cmod], column n takes entry n % cmod
  const float* resid;
  const float* scale;        // [N]
  const float* noise;        // [b * noise_ld + t]
  const float* alpha;        // [cmod] alpha, then [cmod] 1 / (alpha + 1e-9)
  long long y_bstride, r_bstride;
  int ldy, ldr, noise_ld, cmod, epi, act;
  int B, n_lo, n_hi, ksize, dil, N, n_pad, kb_per_tap, ksteps;
  int nt, n_tiles, nr, nb, t_tiles, units, stages, tmem_cols;
  unsigned char* wait_flag;
  int acc_cols;              // TMEM columns of an accumulator: nt, or 2 nt where the two halves of the weights have their own
};
enum ClEpi { CE_PLAIN = 0, CE_RESID = 1, CE_SCALE_RESID = 2, CE_NOISE = 3 };
enum ClAct { CA_NONE = 0, CA_SNAKE = 1, CA_ELU = 2, CA_GELU = 3 };

// round to the 10 mantissa bits of tf32, halves away from zero (integer arithmetic: the conversion instruction runs at a
// quarter of the rate and made the split the longest step of a stage).  Only below CL_ROUND_MAX: from there on up the sum would leave
// the exponent -- the largest finite values would become infinite, and NaN as arithmetic writes it, 0x7fffffff, a zero -- and the
// low bits are cut off instead, so that a NaN or an infinity stays one.
constexpr float CL_ROUND_MAX = 0x1.ffep127f;
__device__ __forceinline__ float tf32_rna_below(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); }
__device__ __forceinline__ float tf32_rna(float x) {
  return __uint_as_float((__float_as_uint(x) + (fabsf(x) < CL_ROUND_MAX ? 0x1000u : 0u)) & 0xffffe000u);
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void cl_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
               : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem], tf32
__device__ __forceinline__ void umma_tf32_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
        "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
      : "memory");
}

// a stage's row split once more, value by value (out of line: hardly any stage needs it, and its registers are the whole kernel's)
__device__ __noinline__ void cl_split_again(const uint8_t* src, uint32_t t, int row) {
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    float hi[16], lo[16];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 v = *reinterpret_cast<const float4*>(src + (((half * 4 + c) ^ (row & 7)) << 4));
      const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        hi[4 * c + e] = tf32_rna(x[e]);
        lo[4 * c + e] = tf32_rna(x[e] - hi[4 * c + e]);
      }
    }
    tmem_st_32x16(t + 16 * half, hi);
    tmem_st_32x16(t + 32 + 16 * half, lo);
  }
}

// sin(x)^2: the square needs x only modulo pi, so one rounding step k = x / pi and two fused steps x - k pi leave
// |r| <= pi / 2, where sin r = r + r^3 P(r^2) with a fitted polynomial of degree 3 (largest relative error 6e-9).  Valid up to
// |x| = 2^16 (k pi exact to 2^-33 there); larger arguments take sinf.  No branch per element: a row of 32 is interleaved.
constexpr float CL_SIN_MAX = 65536.f;
__device__ __forceinline__ float cl_sin_sq(float x) {
  const float k = rintf(x * 0.318309886f);
  float r = fmaf(k, -3.14159274101f, x);
  r = fmaf(k, 8.742278012619e-08f, r);
  const float u = r * r;
  float q = fmaf(u, 2.605780761e-06f, -1.980960296e-04f);
  q = fmaf(u, q, 8.333066247e-03f);
  q = fmaf(u, q, -1.666665955e-01f);
  const float sn = fmaf(r * u, q, r);
  return sn * sn;
}
// ELU without a branch: e^x - 1 = 2^n (e^r - 1) + (2^n - 1) with x = n ln 2 + r, |r| <= ln 2 / 2, and e^r - 1 = r + r^2 Q(r) with a
// fitted polynomial of degree 4.  Largest relative error against 64 bits 8.7e-8 over [-90, 0].
__device__ __forceinline__ float cl_elu(float v) {
  const float x = fmaxf(v, -80.f);
  const float t = fmaf(x, 1.44269504f, 12582912.f), n = t - 12582912.f;        // n in the low bits of t as well
  float r = fmaf(n, -0.693359375f, x);
  r = fmaf(n, 2.12194440e-4f, r);
  float q = fmaf(r, 0.0013882514f, 0.0083665475f);
  q = fmaf(q, r, 0.0416672f);
  q = fmaf(q, r, 0.16666543f);
  q = fmaf(q, r, 0.49999997f);
  const float e = fmaf(r * r, q, r), s = __uint_as_float((__float_as_uint(t) << 23) + 0x3f800000u);
  return v <= 0.f ? fmaf(s, e, s - 1.f) : v;
}
__device__ __forceinline__ float4 cl_snake4(float4 v, const float4& a, const float4& inv) {
  const float4 y = make_float4(a.x * v.x, a.y * v.y, a.z * v.z, a.w * v.w);
  const float big = fmaxf(fmaxf(fabsf(y.x), fabsf(y.y)), fmaxf(fabsf(y.z), fabsf(y.w)));
  float4 s = make_float4(cl_sin_sq(y.x), cl_sin_sq(y.y), cl_sin_sq(y.z), cl_sin_sq(y.w));
  if (!(big <= CL_SIN_MAX)) {
    const float4 t = make_float4(sinf(y.x), sinf(y.y), sinf(y.z), sinf(y.w));
    s = make_float4(t.x * t.x, t.y * t.y, t.z * t.z, t.w * t.w);
  }
  return make_float4(fmaf(inv.x, s.x, v.x), fmaf(inv.y, s.y, v.y), fmaf(inv.z, s.z, v.z), fmaf(inv.w, s.w, v.w));
}
struct ClUnit {
  int n0, n_cur, t0, b0;
};
__device__ __forceinline__ ClUnit cl_unit(const ClConvParams& p, int u) {
  ClUnit r;
  const int m = u / p.n_tiles;                 // column tiles fastest: they share the activation boxes in L2
  r.n0 = (u - m * p.n_tiles) * p.nt;
  r.n_cur = min(p.nt, p.N - r.n0);
  const int bt = m / p.t_tiles;
  r.t0 = p.n_lo + (m - bt * p.t_tiles) * p.nr;
  r.b0 = bt * p.nb;
  return r;
}

// (96 registers a thread: what the epilogue needs.  Spilled registers go to a first-level cache that the stages leave 28 KB)
__global__ void __launch_bounds__(640, 1) cl_conv_kernel(const ClConvParams p, const __grid_constant__ CUtensorMap x_map) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stage_bytes = CL_A_BYTES + p.nt * 256;
  float* epi_sm = reinterpret_cast<float*>(smem + p.stages * stage_bytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.stages * stage_bytes + CL_EPI_BYTES);   // copies have landed
  uint64_t* ready = full + CL_MAX_STAGES;        // the halves are in TMEM
  uint64_t* empty = ready + CL_MAX_STAGES;       // the MMAs have read the stage
  uint64_t* acc_full = empty + CL_MAX_STAGES;    // [2]
  uint64_t* acc_empty = acc_full + 2;            // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const uint32_t gate = smem_u32(tmem_slot + 1);  // set once the kernels in front have completed
  int4* row_tab = reinterpret_cast<int4*>(smem + p.stages * stage_bytes + CL_EPI_BYTES + 512);     // [128]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  BoundedWait bw{p.wait_flag, gate};

  if (warp == 0 && lane == 0) {
    tmem_slot[1] = 0u;
    prefetch_tmap(&x_map);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&ready[s], 4);
      mbar_init(&empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], CL_EPI_WARPS);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, p.tmem_cols);
    tmem_relinquish();
  }
  // tile row -> (batch entry << 16 | position) inside a tile, and where it lies from the tile's first row on in the output and in the
  // residual: the same for every tile (32-bit offsets, the host keeps a launch below 2^31 elements)
  if (warp >= 6 && warp < 10) {
    const int r = (warp - 6) * 32 + lane, bb = r / p.nr, tt = r - bb * p.nr;
    row_tab[r] = make_int4(bb < p.nb ? (bb << 16) | tt : -1, bb * static_cast<int>(p.y_bstride) + tt * p.ldy,
                           bb * static_cast<int>(p.r_bstride) + tt * p.ldr, 0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t a_col0 = tmem_base + 2 * p.acc_cols;    // stage s: hi at + 64 s, lo at + 64 s + 32

  if (warp == 0) {
    // ================= copies =================
    if (lane == 0) {
      const uint32_t box_bytes = static_cast<uint32_t>(p.nr * p.nb) * 128u, smem_a = smem_u32(smem), bar0 = smem_u32(full);
      const size_t half_bytes = static_cast<size_t>(p.n_pad) * 128;
      int s = 0;
      uint32_t ph = 0;
      bool waited = false;
      for (int u = blockIdx.x; u < p.units && !bw.dead; u += gridDim.x) {
        const ClUnit g = cl_unit(p, u);
        const uint32_t w_bytes = static_cast<uint32_t>(g.n_cur) * 128u;
        const uint8_t* wsrc = p.w + static_cast<size_t>(g.n0) * 128;
        auto load_w = [&](int stage) {
          const uint32_t dst = smem_a + stage * stage_bytes + CL_A_BYTES, bar = bar0 + 8 * stage;
          cl_bulk(dst, wsrc, w_bytes, bar);
          cl_bulk(dst + w_bytes, wsrc + half_bytes, w_bytes, bar);
          wsrc += 2 * half_bytes;
        };
        int tap = 0, kb = 0;
        auto load_x = [&](int stage) {
          tma_load_3d(smem_a + stage * stage_bytes, &x_map, bar0 + 8 * stage, kb * 32, g.t0 - (p.ksize - 1 - tap) * p.dil, g.b0);
          if (++kb == p.kb_per_tap) { kb = 0; ++tap; }
        };
        int i = 0;
        if (!waited) {          // weights do not depend on the previous kernel
          const int npre = min(p.stages, p.ksteps);
          for (int j = 0; j < npre; ++j) {
            mbar_arrive_expect_tx(&full[j], box_bytes + 2 * w_bytes);
            load_w(j);
          }
          pdl_wait();
          wait_gate_open(gate);
          pdl_trigger();
          for (int j = 0; j < npre; ++j) load_x(j);
          waited = true;
          i = npre;
          s = npre == p.stages ? 0 : npre;
          ph = npre == p.stages ? 1u : 0u;
        }
        for (; i < p.ksteps; ++i) {
          bw.wait(&empty[s], ph ^ 1u);
          if (bw.dead) break;
          mbar_arrive_expect_tx(&full[s], box_bytes + 2 * w_bytes);
          load_x(s);
          load_w(s);
          if (++s == p.stages) { s = 0; ph ^= 1u; }
        }
      }
      if (bw.dead) {            // let the copies in flight land before the block may leave
        const unsigned long long t0 = gtimer();
        while (gtimer() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================= MMA issuer =================
    // The whole warp walks the loop and one elected lane issues: descriptors and TMEM addresses then stay in uniform registers.
    // Under `if (lane == 0)` every operand of every MMA was moved there first, 70 cycles per instruction whatever its width
    // (64 k-blocks of a 640-row layer: 50 -> 33 us).
    const uint64_t desc0 = umma_desc_sw128_kmajor(smem_u32(smem) + CL_A_BYTES);
    int s = 0, it = 0;
    uint32_t ph = 0;
    for (int u = blockIdx.x; u < p.units && !bw.dead; u += gridDim.x, ++it) {
      const ClUnit g = cl_unit(p, u);
      const int acc = it & 1;
      bw.wait(&acc_empty[acc], ((it >> 1) & 1) ^ 1);
      if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
      tc_fence_after();
      const uint32_t d = tmem_base + acc * p.acc_cols, idesc = umma_idesc(128, g.n_cur, 2u), idesc2 = umma_idesc(128, 2 * g.n_cur, 2u);
      for (int i = 0; i < p.ksteps; ++i) {
        bw.wait(&full[s], ph);
        bw.wait(&ready[s], ph);
        if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
        tc_fence_after();
        const uint64_t b_hi = desc0 + static_cast<uint64_t>(s) * (stage_bytes >> 4), b_lo = b_hi + ((g.n_cur * 128) >> 4);
        const uint32_t a_hi = a_col0 + s * 64, a_lo = a_hi + 32;
        if (elect_one()) {
          if (p.acc_cols != p.nt) {
            // narrow tiles, where an instruction costs more than its columns: hi_x times both halves of the weights (they lie one
            // behind the other) in one instruction, hi_w hi_x and lo_w hi_x in accumulators of their own: Mimi 1929 -> 1881 us, SNAC 32
            // windows 638 -> 623, and a third off the error against 64 bits (tiles of 128 leave no TMEM for it)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              umma_tf32_ta(d, a_hi + 8 * k, b_hi + 2 * k, idesc2, (i > 0 || k > 0) ? 1u : 0u);
              umma_tf32_ta(d, a_lo + 8 * k, b_hi + 2 * k, idesc, 1u);
            }
          } else
#pragma unroll
          for (int k = 0; k < 4; ++k) {                      // small terms first
            umma_tf32_ta(d, a_lo + 8 * k, b_hi + 2 * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
            umma_tf32_ta(d, a_hi + 8 * k, b_lo + 2 * k, idesc, 1u);
            umma_tf32_ta(d, a_hi + 8 * k, b_hi + 2 * k, idesc, 1u);
          }
          umma_commit(&empty[s]);
          if (i + 1 == p.ksteps) umma_commit(&acc_full[acc]);
        }
        __syncwarp();
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp < 6) {
    // ================= split: raw activations -> two halves in TMEM =================
    // A stage is split as if all its values were ordinary ones, with the sum of four times the values kept beside it: that leaves the
    // finite range for a NaN, an infinity and anything from CL_ROUND_MAX on.  Whether it did is asked once the next stage has landed and
    // its values are on the way, when the stores have had their time as well, and only then is the stage handed to the products; one
    // with such a value is split again first.  (The check costs 32 multiply-adds and a vote a stage.  Asked at the end of its own stage: SNAC
    // one window 263 -> 279 us, 32 windows 628 -> 671, Mimi 1904 -> 2047; this way, the second half's low bits left to the product, which
    // reads the upper 19 of a tf32 operand, and the second split out of line: 262, 651, 1929.)
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t t0 = a_col0 + (static_cast<uint32_t>(quarter * 32) << 16);
    int s = 0, last = -1;                          // last: the stage that has been split and not handed over
    uint32_t ph = 0;
    float sum = 0.f;
    auto hand_over = [&]() {
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ready[last]);
    };
    for (int u = blockIdx.x; u < p.units && !bw.dead; u += gridDim.x) {
      for (int i = 0; i < p.ksteps; ++i) {
        bw.wait(&full[s], ph);
        if (!__all_sync(0xffffffffu, !bw.dead && fabsf(sum) < INFINITY)) {
          if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
          cl_split_again(smem + last * stage_bytes + row * 128, t0 + last * 64, row);
        }
        const uint8_t* src = smem + s * stage_bytes + row * 128;
        const uint32_t t = t0 + s * 64;
        float4 in[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) in[c] = *reinterpret_cast<const float4*>(src + ((c ^ (row & 7)) << 4));
        if (last >= 0) hand_over();
        tc_fence_after();            // the products that read this stage's columns before are behind the copy that was waited for
        float odd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float hi[16], lo[16];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float4 v = in[half * 4 + c];
            const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              hi[4 * c + e] = tf32_rna_below(x[e]);
              lo[4 * c + e] = __uint_as_float(__float_as_uint(x[e] - hi[4 * c + e]) + 0x1000u);
              odd[e] = fmaf(x[e], 4.f, odd[e]);
            }
          }
          tmem_st_32x16(t + 16 * half, hi);
          tmem_st_32x16(t + 32 + 16 * half, lo);
        }
        sum = (odd[0] + odd[1]) + (odd[2] + odd[3]);
        last = s;
        if (++s == p.stages) { s = 0; ph ^= 1u; }
      }
    }
    if (last >= 0 && !bw.dead) {
      if (!__all_sync(0xffffffffu, fabsf(sum) < INFINITY)) cl_split_again(smem + last * stage_bytes + row * 128, t0 + last * 64, row);
      hand_over();
    }
  } else {
    // ================= epilogue =================
    // Three warps per TMEM quarter take 16-column chunks in turn.  A lane holds 16 columns of one row, so bias, activation and
    // residual are 16 independent chains, and three warps per scheduler hide each other's loads and transposes.  Rows leave (and
    // residuals come) through a 32 x 16 transpose: 64-byte runs per row.
    const int quarter = warp & 3, group = (warp - 6) >> 2;
    float* st = epi_sm + (warp - 6) * 512;
    float4* my_row = reinterpret_cast<float4*>(st + lane * 16);
    const int cq = lane & 3, rq = lane >> 2, sw = (lane >> 1) & 3;      // transposed side: 16-byte chunk cq of rows rq, rq + 8, ...
    const int tq = ((cq ^ (rq >> 1)) << 2) + rq * 16;                   // (rq + 8 i swizzles as rq does)
    const int4* tab = row_tab + quarter * 32 + rq;               // rows rq, rq + 8, ... of the quarter: tab[0], tab[8], ...
    int it = 0, turn = group;                                    // first chunk of the unit that is this warp's
    for (int u = blockIdx.x; u < p.units && !bw.dead; u += gridDim.x, ++it) {
      const ClUnit g = cl_unit(p, u);
      const int acc = it & 1;
      uint32_t live = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int bt = tab[8 * i].x;
        live |= ((bt >= 0 && g.b0 + (bt >> 16) < p.B && g.t0 + (bt & 0xffff) < p.n_hi) ? 1u : 0u) << i;
      }
      const int y0 = g.b0 * static_cast<int>(p.y_bstride) + (g.t0 - p.n_lo) * p.ldy + g.n0 + cq * 4;
      const int r0 = g.b0 * static_cast<int>(p.r_bstride) + (g.t0 - p.n_lo) * p.ldr + g.n0 + cq * 4;
      bool first = true;
      float nz = 0.f;
#pragma unroll 1
      for (int c0 = turn << 4; c0 < g.n_cur; c0 += 48) {
        const int n0 = g.n0 + c0, nm = n0 % p.cmod;              // 16 columns from a multiple of 16 lie in one group of channels
        // the residual's rows are requested before the accumulator is waited for.  (Its producer is the kernel in front of this
        // one or an earlier one: the first unit waits for it by name, later units follow accumulators that did.)
        float4 rs[4];
        if (p.epi != CE_PLAIN) {
          if (it == 0 && first) pdl_wait();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            rs[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live >> i & 1u) rs[i] = __ldcg(reinterpret_cast<const float4*>(p.resid + (r0 + c0 + tab[8 * i].z)));
          }
          if (p.epi == CE_NOISE) {
            const int r = quarter * 32 + lane, bb = r / p.nr, nb = g.b0 + bb, t = g.t0 + r - bb * p.nr;
            if (bb < p.nb && nb < p.B && t < p.n_hi) nz = __ldcg(&p.noise[static_cast<long long>(nb) * p.noise_ld + t]);
          }
        }
        if (first) {
          bw.wait(&acc_full[acc], (it >> 1) & 1);
          if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
          tc_fence_after();
          first = false;
        }
        const uint32_t taddr = tmem_base + acc * p.acc_cols + (static_cast<uint32_t>(quarter * 32) << 16);
        if (p.epi != CE_PLAIN) {
#pragma unroll
          for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(st + i * 128 + tq) = rs[i];
        }
        uint32_t tv[16];
        tmem_ld_32x16(taddr + c0, tv);
        tmem_ld_wait();
        float v[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c] = __uint_as_float(tv[c]);
        if (p.acc_cols != p.nt) {
          tmem_ld_32x16(taddr + g.n_cur + c0, tv);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; ++c) v[c] += __uint_as_float(tv[c]);
        }
        if (p.bias) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float4 q = __ldg(reinterpret_cast<const float4*>(p.bias + nm) + c);
            v[4 * c] += q.x; v[4 * c + 1] += q.y; v[4 * c + 2] += q.z; v[4 * c + 3] += q.w;
          }
        }
        if (p.epi != CE_PLAIN) {
          __syncwarp();
          if (p.epi == CE_SCALE_RESID) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float4 q = __ldg(reinterpret_cast<const float4*>(p.scale + n0) + c);
              v[4 * c] *= q.x; v[4 * c + 1] *= q.y; v[4 * c + 2] *= q.z; v[4 * c + 3] *= q.w;
            }
          } else if (p.epi == CE_NOISE) {
#pragma unroll
            for (int c = 0; c < 16; ++c) v[c] *= nz;
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float4 q = my_row[c ^ sw];
            v[4 * c] += q.x; v[4 * c + 1] += q.y; v[4 * c + 2] += q.z; v[4 * c + 3] += q.w;
          }
          __syncwarp();
        }
        auto store = [&](float* y) {
#pragma unroll
          for (int c = 0; c < 4; ++c) my_row[c ^ sw] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 q = *reinterpret_cast<const float4*>(st + i * 128 + tq);
            if (live >> i & 1u)
              *reinterpret_cast<float4*>(y + (y0 + c0 + tab[8 * i].y)) = q;
          }
          __syncwarp();
        };
        if (p.y2) store(p.y);
        if (p.act == CA_SNAKE) {
          const float4* al = reinterpret_cast<const float4*>(p.alpha + nm);
          const float4* ia = reinterpret_cast<const float4*>(p.alpha + p.cmod + nm);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float4 o = cl_snake4(make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]), __ldg(al + c), __ldg(ia + c));
            v[4 * c] = o.x; v[4 * c + 1] = o.y; v[4 * c + 2] = o.z; v[4 * c + 3] = o.w;
          }
        } else if (p.act == CA_ELU) {
#pragma unroll
          for (int c = 0; c < 16; ++c) v[c] = cl_elu(v[c]);
        } else if (p.act == CA_GELU) {
#pragma unroll
          for (int c = 0; c < 16; ++c) v[c] = 0.5f * v[c] * (1.f + erff(v[c] * 0.70710678118654752f));
        }
        store(p.y2 ? p.y2 : p.y);
      }
      if (bw.dead) break;
      if (first) {                    // (a warp without a chunk of this unit keeps in step with the accumulators all the same)
        bw.wait(&acc_full[acc], (it >> 1) & 1);
        if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
      }
      turn = (turn + 24 - (g.n_cur >> 4)) % 3;                   // the turns go on over the units (a 32-column tile has two chunks)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

// fp32 weights [N][K] (K = taps x channels, tap-major) -> [K / 32][hi | lo][n_pad][32], 128-byte rows swizzled; rows past N zero
__global__ void __launch_bounds__(256) cl_pack_kernel(float4* __restrict__ dst, const float* __restrict__ w, int N, int K, int n_pad) {
  const int kb = blockIdx.x;
  for (int i = threadIdx.x + blockIdx.y * blockDim.x; i < n_pad * 8; i += blockDim.x * gridDim.y) {
    const int r = i >> 3, c = i & 7;
    float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
    if (r < N) {
      const float4 v = *reinterpret_cast<const float4*>(w + static_cast<size_t>(r) * K + kb * 32 + c * 4);
      const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        hi[e] = tf32_rna(a[e]);
        lo[e] = tf32_rna(a[e] - hi[e]);
      }
    }
    const size_t base = static_cast<size_t>(kb) * 2 * n_pad * 8 + static_cast<size_t>(r) * 8 + (c ^ (r & 7));
    dst[base] = make_float4(hi[0], hi[1], hi[2], hi[3]);
    dst[base + static_cast<size_t>(n_pad) * 8] = make_float4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// ------------------------------------------------------------------------------------------
// depthwise convolution, 7 taps, dilation d, "same" padding; Snake on the input and on the output (optional both)
// ------------------------------------------------------------------------------------------
// A block owns 64 channels x DW_T positions: the (activated) input rows with their halo are staged once in shared memory, so
// every element is read and put through its sine once, in 256-byte rows; a thread finishes four channels of DW_T / 16 rows, whose
// chains interleave (the activation branches once per four values, to the library's sine when an argument is out of range).
// DW_T 128 and four-wide activations against 64 and one by one: 12 to 30 us a layer -> 4 to 14 (SNAC, 32 windows).
constexpr int DW_T = 128;
__global__ void __launch_bounds__(256) cl_dwconv7_kernel(float* __restrict__ y, const float* __restrict__ x, long long x_bstride,
                                                         const float* __restrict__ w, const float* __restrict__ bias,
                                                         const float* __restrict__ alpha_in, const float* __restrict__ alpha_out,
                                                         int C, int T, int dil, int t_lo, int t_hi) {
  extern __shared__ float4 tile[];          // [rows][16]
  const int c4 = threadIdx.x & 15, r0 = threadIdx.x >> 4;
  const int c = blockIdx.y * 64 + c4 * 4, b = blockIdx.z, t0 = t_lo + blockIdx.x * DW_T;
  const int halo = 3 * dil, n_out = min(DW_T, t_hi - t0), rows = n_out + 2 * halo;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  auto ld4 = [&](const float* p) { return p ? __ldg(reinterpret_cast<const float4*>(p + c)) : zero; };
  const float4 ai = ld4(alpha_in), ii = ld4(alpha_in ? alpha_in + C : nullptr), ao = ld4(alpha_out),
               io = ld4(alpha_out ? alpha_out + C : nullptr), bv = ld4(bias);
  float4 wk[7];
#pragma unroll
  for (int k = 0; k < 7; ++k) wk[k] = ld4(w + k * C);
  pdl_sync();
  const float* xb = x + static_cast<size_t>(b) * x_bstride + c;
  for (int rb = r0; rb < rows; rb += 64) {
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = rb + 16 * i, t = t0 - halo + r;
      v[i] = (r < rows && t >= 0 && t < T) ? __ldcg(reinterpret_cast<const float4*>(xb + static_cast<size_t>(t) * C)) : zero;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (alpha_in) v[i] = cl_snake4(v[i], ai, ii);              // (the activation of zero is zero)
      if (rb + 16 * i < rows) tile[(rb + 16 * i) * 16 + c4] = v[i];
    }
  }
  __syncthreads();
  float* yb = y + static_cast<size_t>(b) * T * C + c;
#pragma unroll 2
  for (int r = r0; r < n_out; r += 16) {
    float4 o = bv;
#pragma unroll
    for (int k = 0; k < 7; ++k) {
      const float4 v = tile[(r + k * dil) * 16 + c4];
      o.x = fmaf(wk[k].x, v.x, o.x);
      o.y = fmaf(wk[k].y, v.y, o.y);
      o.z = fmaf(wk[k].z, v.z, o.z);
      o.w = fmaf(wk[k].w, v.w, o.w);
    }
    if (alpha_out) o = cl_snake4(o, ao, io);
    *reinterpret_cast<float4*>(yb + static_cast<size_t>(t0 + r) * C) = o;
  }
}

// ------------------------------------------------------------------------------------------
// last convolution of a decoder: one output channel, ksize taps, `left` positions of context before; optional tanh
// ------------------------------------------------------------------------------------------
constexpr int LC_T = 128;
__global__ void __launch_bounds__(LC_T) cl_last_conv_kernel(float* __restrict__ y, const float* __restrict__ x, long long x_bstride,
                                                            const float* __restrict__ w, const float* __restrict__ bias, int C,
                                                            int T, int ksize, int left, int t0, int t1, int use_tanh) {
  extern __shared__ float lsm[];            // [ksize][C] weights, then [LC_T + ksize - 1][C + 4] rows
  float* ws = lsm;
  float* xs = lsm + ksize * C;
  const int b = blockIdx.y, tb = t0 + blockIdx.x * LC_T, ld = C + 4, rows = min(LC_T, t1 - tb) + ksize - 1, c4n = C >> 2;
  for (int i = threadIdx.x; i < ksize * C; i += LC_T) ws[i] = __ldg(&w[(i % C) * ksize + i / C]);
  const float bv = __ldg(bias);
  pdl_sync();
  const float* xb = x + static_cast<size_t>(b) * x_bstride;
  for (int i = threadIdx.x; i < rows * c4n; i += LC_T) {
    const int r = i / c4n, c = i - r * c4n, t = tb - left + r;
    *reinterpret_cast<float4*>(xs + r * ld + c * 4) =
        (t >= 0 && t < T) ? __ldcg(reinterpret_cast<const float4*>(xb + static_cast<size_t>(t) * C) + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  const int t = tb + threadIdx.x;
  if (t >= t1) return;
  float a0 = bv, a1 = 0.f, a2 = 0.f, a3 = 0.f;
  for (int k = 0; k < ksize; ++k) {
    const float4* xr = reinterpret_cast<const float4*>(xs + (threadIdx.x + k) * ld);
    const float4* wr = reinterpret_cast<const float4*>(ws + k * C);
    for (int c = 0; c < c4n; ++c) {
      const float4 v = xr[c], q = wr[c];
      a0 += v.x * q.x;
      a1 += v.y * q.y;
      a2 += v.z * q.z;
      a3 += v.w * q.w;
    }
  }
  const float o = (a0 + a1) + (a2 + a3);
  y[static_cast<size_t>(b) * (t1 - t0) + (t - t0)] = use_tanh ? tanhf(o) : o;
}

// ------------------------------------------------------------------------------------------
// the small stages in front: code embeddings, upsampling, LayerNorm, attention of one chunk
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) cl_from_codes_kernel(float* __restrict__ z, const int32_t* __restrict__ c0,
                                                            const int32_t* __restrict__ c1, const int32_t* __restrict__ c2,
                                                            const float* __restrict__ cb, const float* __restrict__ pw,
                                                            const float* __restrict__ pb, int C, int T, int cb_size, int cb_dim,
                                                            int s0, int s1, int s2) {
  const int b = blockIdx.y, t = blockIdx.x;
  const int32_t* codes[3] = {c0, c1, c2};
  const int strides[3] = {s0, s1, s2};
  __shared__ float e[3][16];
  pdl_sync();
  if (threadIdx.x < 3 * cb_dim) {
    const int i = threadIdx.x / cb_dim, d = threadIdx.x % cb_dim, tl = T / strides[i];
    int code = codes[i][b * tl + t / strides[i]];
    code = min(max(code, 0), cb_size - 1);
    e[i][d] = cb[(static_cast<size_t>(i) * cb_size + code) * cb_dim + d];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      float a = pb[i * C + c];
      for (int d = 0; d < cb_dim; ++d) a += pw[(static_cast<size_t>(i) * C + c) * cb_dim + d] * e[i][d];
      acc += a;
    }
    z[(static_cast<size_t>(b) * T + t) * C + c] = acc;
  }
}

// z0 [B][T][D] = entry of codebook 0, z1 = sum of the entries of codebooks 1 .. K - 1
__global__ void __launch_bounds__(256) cl_codes_sum_kernel(float* __restrict__ z0, float* __restrict__ z1, const long long* __restrict__ codes,
                                                           const float* __restrict__ emb, int K, int bins, int D, int T) {
  const int t = blockIdx.x, b = blockIdx.y;
  __shared__ int row[64];
  pdl_sync();
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    long long c = codes[(static_cast<size_t>(b) * K + k) * T + t];
    row[k] = k * bins + static_cast<int>(c < 0 ? 0 : (c >= bins ? bins - 1 : c));
  }
  __syncthreads();
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    const size_t o = (static_cast<size_t>(b) * T + t) * D + d;
    z0[o] = emb[static_cast<size_t>(row[0]) * D + d];
    float acc = 0.f;
#pragma unroll 8
    for (int k = 1; k < K; ++k) acc += emb[static_cast<size_t>(row[k]) * D + d];
    z1[o] = acc;
  }
}

// depthwise transposed convolution, 2 s taps, stride s, trimmed on the right: [B][T][C] -> [B][T s][C]; w [C][2 s]
__global__ void __launch_bounds__(256) cl_upsample_kernel(float* __restrict__ y, const float* __restrict__ x, const float* __restrict__ w,
                                                          int C, int T, int s) {
  const int to = blockIdx.x, b = blockIdx.y, t = to / s, r = to - t * s;
  pdl_sync();
  const float* xr = x + (static_cast<size_t>(b) * T + t) * C;
  float* yr = y + (static_cast<size_t>(b) * T * s + to) * C;
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float a = xr[c] * w[c * 2 * s + r];
    if (t > 0) a += xr[c - C] * w[c * 2 * s + s + r];
    yr[c] = a;
  }
}

// one warp per row, row kept in registers (C <= 1024, a multiple of 4)
__global__ void __launch_bounds__(128) cl_layernorm_kernel(float* __restrict__ y, const float* __restrict__ x, const float* __restrict__ w,
                                                           const float* __restrict__ bias, int rows, int C, float eps) {
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, n4 = C >> 2;
  pdl_sync();
  if (row >= rows) return;
  const float4* xr = reinterpret_cast<const float4*>(x + static_cast<size_t>(row) * C);
  float4 v[8];
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = lane + 32 * i;
    v[i] = c < n4 ? __ldcg(xr + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
  }
  const float mean = warp_sum(sum) / static_cast<float>(C);
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (lane + 32 * i < n4) {
      const float a = v[i].x - mean, b = v[i].y - mean, c = v[i].z - mean, d = v[i].w - mean;
      sq += (a * a + b * b) + (c * c + d * d);
    }
  }
  const float rstd = 1.f / sqrtf(warp_sum(sq) / static_cast<float>(C) + eps);
  float4* yr = reinterpret_cast<float4*>(y + static_cast<size_t>(row) * C);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = lane + 32 * i;
    if (c < n4) {
      const float4 ww = __ldg(reinterpret_cast<const float4*>(w) + c), bb = __ldg(reinterpret_cast<const float4*>(bias) + c);
      yr[c] = make_float4((v[i].x - mean) * rstd * ww.x + bb.x, (v[i].y - mean) * rstd * ww.y + bb.y,
                          (v[i].z - mean) * rstd * ww.z + bb.z, (v[i].w - mean) * rstd * ww.w + bb.w);
    }
  }
}

// causal attention inside one chunk of T <= 64 positions, rotary pairs (2j, 2j + 1); qkv [B][T][3 C] -> out [B][T][C].
// One block per (head, batch entry): a chunk is a few dozen positions, so scores and weights stay in shared memory.
__global__ void __launch_bounds__(256) cl_chunk_attention_kernel(float* __restrict__ out, const float* __restrict__ qkv, int C, int H,
                                                                 int T, float max_period) {
  extern __shared__ float asm_[];      // q, k, v [T][D + 4], p [T][T + 1], frequencies
  const int h = blockIdx.x, b = blockIdx.y, D = C / H, ld = D + 4, half = D >> 1;
  float* q = asm_;
  float* k = q + T * ld;
  float* v = k + T * ld;
  float* p = v + T * ld;
  float* freq = p + T * (T + 1);       // [D / 2]
  for (int j = threadIdx.x; j < half; j += blockDim.x)
    freq[j] = expf(static_cast<float>(j) * (-logf(max_period) * 2.f / static_cast<float>(D)));
  pdl_sync();
  __syncthreads();
  const float* base = qkv + static_cast<size_t>(b) * T * 3 * C + h * D;
#pragma unroll 4
  for (int i = threadIdx.x; i < T * half; i += blockDim.x) {
    const int t = i / half, j = i - t * half;
    const float* row = base + static_cast<size_t>(t) * 3 * C + 2 * j;
    const float2 a = __ldcg(reinterpret_cast<const float2*>(row)), e = __ldcg(reinterpret_cast<const float2*>(row + C)),
                 f = __ldcg(reinterpret_cast<const float2*>(row + 2 * C));
    float sn, cs;
    sincosf(static_cast<float>(t) * freq[j], &sn, &cs);
    const int o = t * ld + 2 * j;
    q[o] = a.x * cs - a.y * sn;
    q[o + 1] = a.x * sn + a.y * cs;
    k[o] = e.x * cs - e.y * sn;
    k[o + 1] = e.x * sn + e.y * cs;
    v[o] = f.x;
    v[o + 1] = f.y;
  }
  __syncthreads();
  const float scale = rsqrtf(static_cast<float>(D));
  const int d4 = D >> 2;
  for (int i = threadIdx.x; i < T * T; i += blockDim.x) {
    const int tq = i / T, tk = i - tq * T;
    float s = 0.f;
    if (tk <= tq) {
      const float4* a = reinterpret_cast<const float4*>(q + tq * ld);
      const float4* c = reinterpret_cast<const float4*>(k + tk * ld);
      float s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll 4
      for (int d = 0; d < d4; ++d) {
        const float4 x = a[d], y = c[d];
        s += x.x * y.x;
        s1 += x.y * y.y;
        s2 += x.z * y.z;
        s3 += x.w * y.w;
      }
      s = (s + s1) + (s2 + s3);
    }
    p[tq * (T + 1) + tk] = s * scale;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int tq = warp; tq < T; tq += 8) {
    float mx = -INFINITY;
    for (int tk = lane; tk <= tq; tk += 32) mx = fmaxf(mx, p[tq * (T + 1) + tk]);
    mx = warp_max(mx);
    float den = 0.f;
    for (int tk = lane; tk <= tq; tk += 32) {
      const float e = expf(p[tq * (T + 1) + tk] - mx);
      p[tq * (T + 1) + tk] = e;
      den += e;
    }
    const float inv = 1.f / warp_sum(den);
    __syncwarp();
    for (int d = lane; d < D; d += 32) {
      float a = 0.f;
      for (int tk = 0; tk <= tq; ++tk) a += p[tq * (T + 1) + tk] * v[tk * ld + d];
      out[(static_cast<size_t>(b) * T + tq) * C + h * D + d] = a * inv;
    }
    __syncwarp();
  }
}

static bool on16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }      // (a null pointer is)

static int cl_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 148;
  }
  return sms;
}

}  // namespace vb

using namespace vb;

extern "C" {

int vb_cl_timeouts(void) {
  return wait_ran_out(WK_CL_CONV);
}

long long vb_cl_pack_bytes(int N, int K) {
  if (N <= 0 || K <= 0 || N % 32 || K % 32) return -1;
  return static_cast<long long>(N) * K * 8;
}

int vb_cl_pack(void* d_dst, const float* d_w, int N, int K, void* stream) {
  VB_CHECK_ARG(d_dst && d_w, "vb_cl_pack: null pointer");
  VB_CHECK_ARG(on16(d_dst) && on16(d_w), "vb_cl_pack: pointers must lie on 16-byte boundaries");
  VB_CHECK_ARG(vb_cl_pack_bytes(N, K) > 0, "vb_cl_pack: N = %d and K = %d must be positive multiples of 32", N, K);
  cl_pack_kernel<<<dim3(K / 32, (N * 8 + 2047) / 2048), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<float4*>(d_dst), d_w, N, K, N);
  VB_CHECK_LAUNCH();
  return 0;
}

int vb_cl_conv(float* d_y, float* d_y2, const float* d_x, long long x_bstride, int Tx, const void* d_w, const float* d_bias,
               const float* d_resid, long long r_bstride, const float* d_scale, const float* d_noise, int noise_ld,
               const float* d_alpha, int epilogue, int act, int B, int Cin, int N, int cmod, int ksize, int dil, int n_lo, int n_hi,
               long long y_bstride, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w, "vb_cl_conv: null pointer");
  VB_CHECK_ARG(Cin > 0 && Cin % 32 == 0 && N > 0 && N % 32 == 0, "vb_cl_conv: Cin = %d and N = %d must be positive multiples of 32", Cin, N);
  VB_CHECK_ARG(cmod > 0 && cmod % 32 == 0 && N % cmod == 0, "vb_cl_conv: %d columns do not divide into groups of %d channels", N, cmod);
  VB_CHECK_ARG(ksize >= 1 && dil >= 1 && Tx > 0 && n_lo >= 0, "vb_cl_conv: ksize %d, dilation %d, %d positions, rows from %d", ksize, dil, Tx, n_lo);
  VB_CHECK_ARG(epilogue >= 0 && epilogue <= 3 && act >= 0 && act <= 3, "vb_cl_conv: epilogue %d / activation %d", epilogue, act);
  VB_CHECK_ARG(epilogue == CE_PLAIN || d_resid, "vb_cl_conv: this epilogue needs d_resid");
  VB_CHECK_ARG(epilogue != CE_SCALE_RESID || d_scale, "vb_cl_conv: the scaled residual needs d_scale");
  VB_CHECK_ARG(epilogue != CE_NOISE || d_noise, "vb_cl_conv: the noise epilogue needs d_noise");
  VB_CHECK_ARG(act != CA_SNAKE || d_alpha, "vb_cl_conv: Snake needs d_alpha");
  VB_CHECK_ARG(on16(d_x) && x_bstride % 4 == 0 && on16(d_y) && on16(d_y2) && y_bstride % 4 == 0 && on16(d_resid) && (!d_resid || r_bstride % 4 == 0),
               "vb_cl_conv: rows must start on 16-byte boundaries");
  VB_CHECK_ARG(on16(d_w) && on16(d_bias) && on16(d_scale) && on16(d_alpha), "vb_cl_conv: weights, bias, scale and alpha must lie on 16-byte boundaries");
  if (B <= 0 || n_lo >= n_hi) return 0;
  // the epilogue addresses rows with 32-bit offsets from the first one: what is beyond that runs in several launches
  const long long per_entry = max(y_bstride, r_bstride);
  const int max_b = per_entry >= (1LL << 30) ? 1 : static_cast<int>(((1LL << 31) - 1) / max(per_entry, 1LL)) - 1;
  if (B > max_b) {
    for (int b0 = 0; b0 < B; b0 += max_b) {
      const int rc = vb_cl_conv(d_y + b0 * y_bstride, d_y2 ? d_y2 + b0 * y_bstride : nullptr, d_x + b0 * x_bstride, x_bstride, Tx, d_w, d_bias,
                                d_resid ? d_resid + b0 * r_bstride : nullptr, r_bstride, d_scale,
                                d_noise ? d_noise + static_cast<long long>(b0) * noise_ld : nullptr, noise_ld, d_alpha, epilogue, act,
                                min(max_b, B - b0), Cin, N, cmod, ksize, dil, n_lo, n_hi, y_bstride, stream);
      if (rc != 0) return rc;
    }
    return 0;
  }
  const long long max_rows = max((1LL << 30) / N / 128 * 128, 128LL);
  if (n_hi - n_lo > max_rows) {
    for (long long t = n_lo; t < n_hi; t += max_rows) {
      const int rc = vb_cl_conv(d_y, d_y2, d_x, x_bstride, Tx, d_w, d_bias, d_resid, r_bstride, d_scale, d_noise, noise_ld, d_alpha, epilogue, act,
                                B, Cin, N, cmod, ksize, dil, static_cast<int>(t), static_cast<int>(min(t + max_rows, static_cast<long long>(n_hi))),
                                y_bstride, stream);
      if (rc != 0) return rc;
    }
    return 0;
  }
  VB_CHECK_ARG(N <= (1 << 22), "vb_cl_conv: %d columns", N);
  auto fn = encode_fn();
  VB_CHECK_ARG(fn, "cuTensorMapEncodeTiled not available (no CUDA driver?)");
  ClConvParams p = {};
  VB_CHECK_ARG(p.wait_flag = wait_flag(WK_CL_CONV), "vb_cl_conv: no mapped host memory");
  const int range = n_hi - n_lo;
  p.nr = min(range, 128);
  p.nb = min(B, 128 / p.nr);
  p.t_tiles = (range + p.nr - 1) / p.nr;
  const long long m_tiles = static_cast<long long>(p.t_tiles) * ((B + p.nb - 1) / p.nb);
  p.kb_per_tap = Cin / 32;
  p.ksteps = p.kb_per_tap * ksize;
  // width of a column tile: rounds of units times what a unit costs -- a stage takes the products' 6 cycles a column or the
  // split's 320, whichever is longer, the epilogue about 1000 plus 24 a column where nothing overlaps it
  const int sms = cl_sms();
  long long best = -1;
  for (int nt = 128; nt >= 32; nt >>= 1) {
    if (nt > N && nt > 32) continue;
    const long long units = m_tiles * ((N + nt - 1) / nt), rounds = (units + sms - 1) / sms;
    const long long stage = max(6 * nt, 320), unit = max(stage * p.ksteps, 500LL + 24 * nt);
    const long long cost = rounds * unit + 1000 + 24 * nt;
    if (best < 0 || cost < best) { best = cost; p.nt = nt; p.units = static_cast<int>(units); }
  }
  VB_CHECK_ARG(m_tiles * ((N + p.nt - 1) / p.nt) < 0x7fffffffLL, "vb_cl_conv: too many tiles");
  p.n_tiles = (N + p.nt - 1) / p.nt;
  p.w = static_cast<const uint8_t*>(d_w);
  const long long first = static_cast<long long>(n_lo) * N;
  p.y = d_y + first; p.y2 = d_y2 ? d_y2 + first : nullptr; p.bias = d_bias; p.resid = d_resid ? d_resid + first : nullptr; p.scale = d_scale; p.noise = d_noise; p.alpha = d_alpha;
  p.y_bstride = y_bstride; p.r_bstride = r_bstride; p.ldy = N; p.ldr = N; p.noise_ld = noise_ld; p.cmod = cmod;
  p.epi = epilogue; p.act = act; p.B = B; p.n_lo = n_lo; p.n_hi = n_hi; p.ksize = ksize; p.dil = dil; p.N = N; p.n_pad = N;
  const int stage_bytes = CL_A_BYTES + p.nt * 256, tail = CL_EPI_BYTES + 512 /*barriers*/ + 2048 /*row table*/ + 1024 /*alignment*/;
  p.acc_cols = p.nt <= 64 ? 2 * p.nt : p.nt;
  p.stages = min(min(CL_MAX_STAGES, (512 - 2 * p.acc_cols) / 64), (VB_MAX_DYN_SMEM - tail) / stage_bytes);
  p.tmem_cols = 512;
  CUtensorMap map;
  {
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(Cin), static_cast<cuuint64_t>(Tx), static_cast<cuuint64_t>(B)};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(Cin) * 4, static_cast<cuuint64_t>(x_bstride) * 4};
    cuuint32_t box[3] = {32, static_cast<cuuint32_t>(p.nr), static_cast<cuuint32_t>(p.nb)}, estr[3] = {1, 1, 1};
    const CUresult r = fn(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(d_x), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    VB_CHECK_ARG(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled(channels last) failed: CUresult %d", static_cast<int>(r));
  }
  VB_CHECK_CUDA(max_dyn_smem_once(cl_conv_kernel));
  const int smem = p.stages * stage_bytes + tail;
  VB_CHECK_CUDA(launch_kernel(cl_conv_kernel, dim3(min(p.units, sms)), dim3(CL_THREADS), smem, static_cast<cudaStream_t>(stream), true, p, map));
  return 0;
}

int vb_cl_dwconv7(float* d_y, const float* d_x, long long x_bstride, const float* d_w, const float* d_bias, const float* d_alpha_in,
                  const float* d_alpha_out, int B, int C, int T, int dilation, int t_lo, int t_hi, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w, "vb_cl_dwconv7: null pointer");
  VB_CHECK_ARG(C % 64 == 0 && dilation >= 1 && dilation <= 64 && x_bstride % 4 == 0, "vb_cl_dwconv7: C = %d (a multiple of 64), dilation %d", C, dilation);
  VB_CHECK_ARG(on16(d_y) && on16(d_x) && on16(d_w) && on16(d_bias) && on16(d_alpha_in) && on16(d_alpha_out), "vb_cl_dwconv7: pointers must lie on 16-byte boundaries");
  VB_CHECK_ARG(0 <= t_lo && t_lo <= t_hi && t_hi <= T, "vb_cl_dwconv7: range [%d, %d) outside [0, %d)", t_lo, t_hi, T);
  if (B <= 0 || t_lo == t_hi) return 0;
  VB_CHECK_CUDA(max_dyn_smem_once(cl_dwconv7_kernel));
  VB_LAUNCH_PDL(cl_dwconv7_kernel, dim3((t_hi - t_lo + DW_T - 1) / DW_T, C / 64, B), 256, static_cast<size_t>(DW_T + 6 * dilation) * 256, stream,
                d_y, d_x, x_bstride, d_w, d_bias, d_alpha_in, d_alpha_out, C, T, dilation, t_lo, t_hi);
  return 0;
}

int vb_cl_last_conv(float* d_y, const float* d_x, long long x_bstride, const float* d_w, const float* d_bias, int B, int C, int T,
                    int ksize, int left, int t0, int t1, int use_tanh, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w && d_bias, "vb_cl_last_conv: null pointer");
  VB_CHECK_ARG(C % 4 == 0 && C <= 256 && ksize >= 1 && ksize <= 16 && x_bstride % 4 == 0, "vb_cl_last_conv: C = %d, ksize %d", C, ksize);
  VB_CHECK_ARG(on16(d_x), "vb_cl_last_conv: rows must start on 16-byte boundaries");
  VB_CHECK_ARG(0 <= t0 && t0 < t1 && t1 <= T, "vb_cl_last_conv: bad output range [%d, %d) of %d", t0, t1, T);
  if (B <= 0) return 0;
  VB_CHECK_CUDA(max_dyn_smem_once(cl_last_conv_kernel));
  const size_t smem = (static_cast<size_t>(ksize) * C + static_cast<size_t>(LC_T + ksize - 1) * (C + 4)) * sizeof(float);
  VB_LAUNCH_PDL(cl_last_conv_kernel, dim3((t1 - t0 + LC_T - 1) / LC_T, B), LC_T, smem, stream, d_y, d_x, x_bstride, d_w, d_bias, C, T, ksize,
                left, t0, t1, use_tanh);
  return 0;
}

int vb_cl_from_codes(float* d_z, const int32_t* d_codes0, const int32_t* d_codes1, const int32_t* d_codes2, const float* d_codebooks,
                     const float* d_proj_w, const float* d_proj_b, int B, int C, int T, int cb_size, int cb_dim, int stride0, int stride1,
                     int stride2, void* stream) {
  VB_CHECK_ARG(d_z && d_codes0 && d_codes1 && d_codes2 && d_codebooks && d_proj_w && d_proj_b, "vb_cl_from_codes: null pointer");
  VB_CHECK_ARG(cb_dim <= 16 && T % stride0 == 0 && T % stride1 == 0 && T % stride2 == 0, "vb_cl_from_codes: bad dims");
  if (B <= 0) return 0;
  VB_LAUNCH_PDL(cl_from_codes_kernel, dim3(T, B), 256, 0, stream, d_z, d_codes0, d_codes1, d_codes2, d_codebooks, d_proj_w, d_proj_b, C, T,
                cb_size, cb_dim, stride0, stride1, stride2);
  return 0;
}

int vb_cl_codes_sum(float* d_z0, float* d_z1, const int64_t* d_codes, const float* d_emb, int B, int K, int bins, int D, int T, void* stream) {
  VB_CHECK_ARG(d_z0 && d_z1 && d_codes && d_emb, "vb_cl_codes_sum: null pointer");
  VB_CHECK_ARG(K >= 1 && K <= 64, "vb_cl_codes_sum: %d codebooks", K);
  if (B <= 0 || T <= 0) return 0;
  VB_LAUNCH_PDL(cl_codes_sum_kernel, dim3(T, B), 256, 0, stream, d_z0, d_z1, reinterpret_cast<const long long*>(d_codes), d_emb, K, bins, D, T);
  return 0;
}

int vb_cl_upsample(float* d_y, const float* d_x, const float* d_w, int B, int C, int T, int stride, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w && stride >= 1, "vb_cl_upsample: bad arguments");
  if (B <= 0 || T <= 0) return 0;
  VB_LAUNCH_PDL(cl_upsample_kernel, dim3(T * stride, B), 256, 0, stream, d_y, d_x, d_w, C, T, stride);
  return 0;
}

int vb_cl_layernorm(float* d_y, const float* d_x, const float* d_w, const float* d_b, int rows, int C, float eps, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w && d_b, "vb_cl_layernorm: null pointer");
  VB_CHECK_ARG(on16(d_y) && on16(d_x) && on16(d_w) && on16(d_b), "vb_cl_layernorm: pointers must lie on 16-byte boundaries");
  VB_CHECK_ARG(C > 0 && C % 4 == 0 && C <= 1024, "vb_cl_layernorm: C = %d (a multiple of 4, <= 1024)", C);
  if (rows <= 0) return 0;
  VB_LAUNCH_PDL(cl_layernorm_kernel, (rows + 3) / 4, 128, 0, stream, d_y, d_x, d_w, d_b, rows, C, eps);
  return 0;
}

int vb_cl_chunk_attention(float* d_out, const float* d_qkv, int B, int C, int H, int T, float max_period, void* stream) {
  VB_CHECK_ARG(d_out && d_qkv, "vb_cl_chunk_attention: null pointer");
  VB_CHECK_ARG(reinterpret_cast<uintptr_t>(d_qkv) % 8 == 0, "vb_cl_chunk_attention: rows must start on 8-byte boundaries");
  VB_CHECK_ARG(H >= 1 && C % H == 0 && (C / H) % 4 == 0 && C / H <= 256 && T >= 1 && T <= 64, "vb_cl_chunk_attention: C %d, H %d, T %d (<= 64)", C, H, T);
  if (B <= 0) return 0;
  const size_t smem = (static_cast<size_t>(3) * T * (C / H + 4) + static_cast<size_t>(T) * (T + 1) + C / H / 2) * sizeof(float);
  VB_CHECK_ARG(smem <= VB_MAX_DYN_SMEM, "vb_cl_chunk_attention: head size %d too large", C / H);
  VB_CHECK_CUDA(max_dyn_smem_once(cl_chunk_attention_kernel));
  VB_LAUNCH_PDL(cl_chunk_attention_kernel, dim3(H, B), 256, smem, stream, d_out, d_qkv, C, H, T, max_period);
  return 0;
}

}  // extern "C"
