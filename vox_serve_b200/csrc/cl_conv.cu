// Vocoder convolutions over channels-last activations [B][T][C] (fp32), on tcgen05 with fp32-grade products.
//
// With the channels innermost a convolution is a plain matrix product per tap:
//   D[n][position] += sum_c W[tap][n][c] * X[position - shift(tap)][c]
// The weights are the MMA's first operand (128 output channels = the lanes of the accumulator), the positions its columns: a lane
// of the epilogue owns one channel -- bias, scale and alpha are scalars of the thread -- and 32 lanes store 32 neighbouring channels,
// so rows leave and residuals come without a transpose.  A transposed convolution of stride s is the same product with two taps and
// n = (phase, channel): row n of the result holds the s output positions of input position n.
//
// Products: both operands as two fp16 parts, v = hi + lo / 2048 (the low part scaled into the normal range: 22 bits and a sign), hi_w hi_x in
// one accumulator, hi_w lo_x + lo_w hi_x in a second one; what is dropped is below 2^-22 of a product.  Half the MMA time and half the
// weight bytes of the two tf32 parts that stood here, at the same width; error against 64 bits of a decode 4.7e-6 (Mimi, was 2.8e-5).  Weights are
// scaled per output channel by a power of two when they are packed.  Activations by 16: their parts hold 22 bits of a value in [2^-14, 4092) and smaller
// ones to 2^-40 absolute.  A row's block of 32 channels with a value from 4092 on, an infinity, a NaN, or nothing but values below 2^-14 is kept as
// it is in fp32, and the positions into which it goes are multiplied in fp32 on CUDA cores (cl_exact_chunk).  So every value is held to 2^-26
// of the largest beside it, however quiet the passage; and since a row's code and a position's way follow from what goes into them alone, an
// entry's bits do not depend on its batch.
// What only these convolutions read is written as parts by the kernel that produces it, in the bytes its fp32 values would have taken, and
// fetched by TMA: nothing is converted here, and a tap is the same tile in shared memory read from a later row on.  Activations that come
// as fp32 are split on the way by eight warps, once per tile and 64 channels for all taps.
//
// Warps: 0 copies weights (one bulk copy a stage), 1 issues the MMAs, 2 copies activations, 3 looks at the codes of a tile's rows (with fp32
// activations 2..9 split), the rest is the epilogue.  Persistent CTAs, two accumulator pairs where they fit, weights that stay in shared
// memory where a CTA's units share them.  Long sums of narrow layers are divided over a cluster (cl_splits) and added through
// distributed shared memory in rank order, by the layer alone and not by the number of rows.
// What bounds it (640 rows of 512 x 2048, split in four: 12.8 us, was 28.4; 5120 x 1536 x 1024: 60 us, was 161): the wide layers the bytes
// through L2 and shared memory, 0.6 us for 64 channels and one tap of 128 x 128; the layers of many positions the epilogue's instructions,
// some 50 for the 32 values of a warp (153600 x 128 with residual 61 us, was 71, 30 of DRAM time).
// Measured (one pass): SNAC 32 windows 652 -> 532 us, 1 window 262 -> 242, Mimi 32 chunks 1926 -> 1262, the small kernels below among them; with the fused units of
// cl_unit.cu and the depthwise tiles by their time 487, 183 and 1089.
#include "../../include/vb_api.h"
#define VB_PDL_FAMILY 32
#include "cl_common.cuh"

namespace vb {
constexpr int CL_SPLIT_WARPS = 8;
constexpr int CL_X_STAGES = 4, CL_W_STAGES = 8, CL_TOPS = 8;
constexpr int CL_ROWS = 256;                // rows of a stage of activations: columns of the tile and the halo
constexpr int CL_TAIL = 8192;               // barriers, tables, alignment

struct ClConvParams {
  const uint8_t* w;          // [128 channels][32 of K][128][32 hi | 32 lo], rows of 128 bytes swizzled
  const float* w_inv;        // [n_pad] 1 / (scale of the channel's weights * CL_X_SCALE)
  const float* x;            // fp32, or parts
  const uint8_t* x_code;     // of the parts
  float* y;                  // [b * y_bstride + t * N + n]; the plain values where another output is given
  float* y2;                 // optional: the activated values
  uint32_t* yp;              // optional: the activated values as parts
  uint8_t* yp_code;
  const float* bias;         // [cmod], column n takes entry n % cmod
  const float* resid;
  const float* scale;        // [N]
  const float* noise;        // [b * noise_ld + t]
  const float* alpha;        // [cmod] alpha, then [cmod] 1 / (alpha + 1e-9)
  long long x_bstride, y_bstride, r_bstride;
  int noise_ld, cmod, epi, act;
  int B, Tx, Cin, N, n_lo, n_hi, ksize, dil;
  int group;                 // 32-channel blocks a stage
  int kb;                    // stages of channels
  int taps;                  // taps that one stage of activations serves: all of them, or one
  int halo;                  // rows of an entry in front of its first position (taps == ksize), else 0
  int nr, nb, pitch, cols, rows_pad;      // a tile: nb entries of nr positions, `pitch` rows apart; columns in all
  int m_tiles, t_tiles, units, grid;
  int splits;                // parts of K, each on a CTA of a cluster
  uint32_t m_tiles_inv, t_tiles_inv;      // for cl_div
  int x_stages, w_stages, acc_cols, acc_bufs;
  int resident;              // the weights of a CTA's units are the same and stay in shared memory
  int staged;                // results and residuals pass through boxes of 8 positions x 32 channels in shared memory, four per warp
  int passes;                // rows of a stage that a thread of the split takes: 1, 2, 4, 8 or 16
  unsigned char* wait_flag;
};
enum ClEpi { CE_PLAIN = 0, CE_RESID = 1, CE_SCALE_RESID = 2, CE_NOISE = 3 };

// a / b for 0 <= a < 2^31 with inv = ceil(2^32 / b), 0 for b == 1: the quotient or one more, as a product
__device__ __forceinline__ int cl_div(int a, int b, uint32_t inv) {
  if (inv == 0u) return a;
  const int q = static_cast<int>(__umulhi(static_cast<uint32_t>(a), inv));
  return q * static_cast<long long>(b) > a ? q - 1 : q;
}
struct ClUnit {
  int m0, t0, b0;
};
__device__ __forceinline__ ClUnit cl_unit(const ClConvParams& p, int u) {
  ClUnit r;
  const int m = cl_div(u, p.m_tiles, p.m_tiles_inv);                 // channel tiles fastest: they share the activations in L2
  r.m0 = (u - m * p.m_tiles) * 128;
  const int bt = cl_div(m, p.t_tiles, p.t_tiles_inv);
  r.t0 = p.n_lo + (m - bt * p.t_tiles) * p.nr;
  r.b0 = bt * p.nb;
  return r;
}

// Which of eight columns are outside the parts' range: a bit each.  Of activations as fp32 this block's own channels [blk_lo, blk_hi) count -- all
// tiny, or one too large -- of parts the codes of all of them: in either case what the flag that a unit is looked at for was found from.
template <bool PARTS>
__device__ __noinline__ uint32_t cl_exact_columns(const ClConvParams& p, const int4* col_tab, int t0, int b0, int c0, int blk_lo, int blk_hi) {
  const int lane = threadIdx.x & 31, part = lane >> 3, e = col_tab[c0 + (lane & 7)].x;         // four lanes a column
  uint32_t code = 0u;
  float m = 0.f;
  const int b = b0 + (e >> 16), t = t0 + (e & 0xffff);
  if (e >= 0 && b < p.B && t < p.n_hi) {
#pragma unroll 1
    for (int tap = 0; tap < p.ksize; ++tap) {
      const int ts = t - (p.ksize - 1 - tap) * p.dil;
      if (ts < 0 || ts >= p.Tx) continue;
      const long long row = b * p.x_bstride + static_cast<long long>(ts) * p.Cin;
      if (PARTS) {
#pragma unroll 4
        for (int k = part; k < p.Cin >> 5; k += 4) code |= __ldcg(p.x_code + (row >> 5) + k);
      } else {
#pragma unroll 4
        for (int k = blk_lo * 32 + part * 4; k < blk_hi * 32; k += 16) {
          const float4 v = __ldcg(reinterpret_cast<const float4*>(p.x + row + k));
          m = max3_abs(max3_abs(m, v.x, v.y), v.z, v.w);
        }
      }
    }
  }
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) {
    const float other = __shfl_xor_sync(0xffffffffu, m, o);
    m = max3_abs(m, other, other);
    code |= __shfl_xor_sync(0xffffffffu, code, o);
  }
  return __ballot_sync(0xffffffffu, (PARTS ? code : cl_code(m)) & CB_RAW) & 0xffu;
}
// Four columns of a unit that is looked at: the accumulators in the plain scale, and the columns of `mask` multiplied again in fp32 -- this warp's
// 32 channels, blocks [blk_lo, blk_hi) of K.  The weights come from their packed parts.  The epilogue goes on as if the products had given this,
// the factor of the channel being 1.  A block of 32 inputs at a time: a lane holds its channel's weights and, of every column, the input of its
// number, which goes round by shuffles.  5120 rows of 1536 x 1024 take 50 us, with one value of 5000 132, with nothing but such values 4.3 ms (element
// by element 61 and 141 ms); 640 rows of 2048 x 512 15, 52 and 440 us.  (Four or eight weights more in flight cost the epilogue registers: Mimi 1262 us,
// 1273 and 1285.)
__device__ __noinline__ void cl_exact_chunk(const ClConvParams& p, const int4* col_tab, int m0, int t0, int b0, int c0, int lane_row,
                                            int blk_lo, int blk_hi, uint32_t t_hi, uint32_t t_lo, uint32_t mask, float inv) {
  const int lane = threadIdx.x & 31, blocks_per_tap = p.Cin >> 5, sw = lane_row & 7;
  const uint8_t* wt = p.w + static_cast<size_t>(m0 >> 7) * (blocks_per_tap * p.ksize) * CL_W_BLOCK + lane_row * 128;
  const float w_scale = p.w_inv[m0 + lane_row] * CL_X_SCALE;
  const long long base = b0 * p.x_bstride + static_cast<long long>(t0) * p.Cin;
  float acc[4] = {};
#pragma unroll 1
  for (int tap = 0; tap < p.ksize && mask; ++tap) {
    const int shift = (p.ksize - 1 - tap) * p.dil;
    // lane c: where column c's row lies; the columns that have one
    const int e = col_tab[c0 + (lane & 3)].x, q0 = (e & 0xffff) - shift, at_lane = static_cast<int>((e >> 16) * p.x_bstride) + q0 * p.Cin;
    const uint32_t in = __ballot_sync(0xffffffffu, t0 + q0 >= 0 && t0 + q0 < p.Tx) & mask;
#pragma unroll 1
    for (int blk = blk_lo; blk < blk_hi; ++blk) {
      float x[4];
      const uint32_t parts = __ballot_sync(0xffffffffu, p.x_code && (in >> (lane & 3) & 1u) && !(__ldcg(p.x_code + ((base + at_lane) >> 5) + blk) & CB_RAW));
#pragma unroll
      for (int c = 0; c < 4; ++c) x[c] = in >> c & 1u ? __ldcg(p.x + base + __shfl_sync(0xffffffffu, at_lane, c) + blk * 32 + lane) : 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (parts >> c & 1u) {
          const uint32_t word = __float_as_uint(x[c]);
          const float2 fh = unpack_f16(__shfl_sync(0xffffffffu, word, lane >> 1)), fl = unpack_f16(__shfl_sync(0xffffffffu, word, 16 + (lane >> 1)));
          x[c] = fmaf(lane & 1 ? fl.y : fl.x, 1.f / CL_LO_SCALE, lane & 1 ? fh.y : fh.x) * (1.f / CL_X_SCALE);
        }
      }
      const uint8_t* wb = wt + static_cast<size_t>(tap * blocks_per_tap + blk) * CL_W_BLOCK;
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        const uint4 hi = __ldg(reinterpret_cast<const uint4*>(wb + ((q ^ sw) << 4))), lo = __ldg(reinterpret_cast<const uint4*>(wb + (((q + 4) ^ sw) << 4)));
        const uint32_t h[4] = {hi.x, hi.y, hi.z, hi.w}, l[4] = {lo.x, lo.y, lo.z, lo.w};
        float w[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 fh = unpack_f16(h[i]), fl = unpack_f16(l[i]);
          w[2 * i] = fmaf(fl.x, 1.f / CL_LO_SCALE, fh.x) * w_scale;
          w[2 * i + 1] = fmaf(fl.y, 1.f / CL_LO_SCALE, fh.y) * w_scale;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (!(mask >> c & 1u)) continue;
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[c] = fmaf(__shfl_sync(0xffffffffu, x[c], 8 * q + k), w[k], acc[c]);
        }
      }
    }
  }
  uint32_t hi[4], lo[4];
  tmem_ld_32x4(t_hi, hi);
  tmem_ld_32x4(t_lo, lo);
  tmem_ld_wait();
#pragma unroll
  for (int c = 0; c < 4; ++c)
    if (!(mask >> c & 1u)) acc[c] = fmaf(__uint_as_float(lo[c]), 1.f / CL_LO_SCALE, __uint_as_float(hi[c])) * inv;
  tmem_st_32x4(t_hi, acc);
#pragma unroll
  for (int c = 0; c < 4; ++c) acc[c] = 0.f;
  tmem_st_32x4(t_lo, acc);
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

struct ClEpiState {          // of a thread of the epilogue, for one unit: its channel and where that lies at the unit's first position
  int n;
  float bias, scale, alpha, ialpha;
  float *y, *y2;
  uint32_t* yp;                // the block of 32 channels that the warp holds
  uint8_t* code;
  const float *resid, *noise;
};
// What the epilogue's loops read of the launch's parameters, in registers: behind every asm statement that clobbers memory the compiler reads
// the parameters themselves again, and a dozen such reads were most of a chunk's time (Mimi's 1x1 layer of 153600 x 128: 62 us).
struct ClHot {
  int cols, N, epi, act;
  bool two, res, parts;
};
// where column c0 + (lane & 7) lies: its entry in the table, or x = -1 where there is no such position
__device__ __forceinline__ int4 cl_column(const ClConvParams& p, const ClUnit& g, const int4* col_tab, int c0) {
  int4 tb = col_tab[c0 + (threadIdx.x & (CL_EC - 1))];
  if (!(tb.x >= 0 && g.b0 + (tb.x >> 16) < p.B && g.t0 + (tb.x & 0xffff) < p.n_hi)) tb.x = -1;
  return tb;
}
__device__ __forceinline__ void cl_residual(const ClConvParams& p, const ClHot& h, const ClEpiState& e, const ClUnit& g, const int4* col_tab, int c0, int inside,
                                            float (&rs)[CL_EC]) {
  if (c0 + CL_EC <= inside) {
    const float* r = e.resid + static_cast<long long>(c0) * h.N;
#pragma unroll
    for (int c = 0; c < CL_EC; ++c) rs[c] = __ldcg(r + c * h.N);
    return;
  }
  const int4 tb = cl_column(p, g, col_tab, c0);
#pragma unroll
  for (int c = 0; c < CL_EC; ++c) {
    const bool ok = __shfl_sync(0xffffffffu, tb.x, c) >= 0;
    const int o = __shfl_sync(0xffffffffu, tb.z, c);
    rs[c] = ok ? __ldcg(e.resid + o) : 0.f;
  }
}
__device__ __forceinline__ void cl_linear(const ClConvParams& p, const ClHot& h, const ClEpiState& e, const ClUnit& g, const int4* col_tab, int c0, F2 (&v)[CL_EC / 2],
                                          const float (&rs)[CL_EC]) {
#pragma unroll
  for (int c = 0; c < CL_EC / 2; ++c) v[c] = f2_add(v[c], f2(e.bias));
  if (h.epi == CE_SCALE_RESID) {
#pragma unroll
    for (int c = 0; c < CL_EC / 2; ++c) v[c] = f2_fma(v[c], f2(e.scale), f2(rs[2 * c], rs[2 * c + 1]));
  } else if (h.epi == CE_NOISE) {
    const int4 tb = cl_column(p, g, col_tab, c0);
    const float nz = tb.x >= 0 ? __ldcg(e.noise + tb.w) : 0.f;
#pragma unroll
    for (int c = 0; c < CL_EC / 2; ++c)
      v[c] = f2_fma(v[c], f2(__shfl_sync(0xffffffffu, nz, 2 * c), __shfl_sync(0xffffffffu, nz, 2 * c + 1)), f2(rs[2 * c], rs[2 * c + 1]));
  } else if (h.epi == CE_RESID) {
#pragma unroll
    for (int c = 0; c < CL_EC / 2; ++c) v[c] = f2_add(v[c], f2(rs[2 * c], rs[2 * c + 1]));
  }
}
// eight words of a thread, one a row
__device__ __forceinline__ void cl_store(const ClConvParams& p, const ClHot& h, const ClUnit& g, const int4* col_tab, int c0, int inside, uint32_t* y,
                                         const uint32_t (&w)[CL_EC]) {
  if (c0 + CL_EC <= inside) {
    y += static_cast<long long>(c0) * h.N;
#pragma unroll
    for (int c = 0; c < CL_EC; ++c) y[c * h.N] = w[c];
    return;
  }
  const int4 tb = cl_column(p, g, col_tab, c0);
#pragma unroll
  for (int c = 0; c < CL_EC; ++c) {
    const bool ok = __shfl_sync(0xffffffffu, tb.x, c) >= 0;
    const int o = __shfl_sync(0xffffffffu, tb.y, c);
    if (ok) y[o] = w[c];
  }
}
__device__ __forceinline__ void cl_store(const ClConvParams& p, const ClHot& h, const ClUnit& g, const int4* col_tab, int c0, int inside, float* y,
                                         const F2 (&v)[CL_EC / 2]) {
  uint32_t w[CL_EC];
#pragma unroll
  for (int c = 0; c < CL_EC / 2; ++c) {
    const float2 x = f2_get(v[c]);
    w[2 * c] = __float_as_uint(x.x);
    w[2 * c + 1] = __float_as_uint(x.y);
  }
  cl_store(p, h, g, col_tab, c0, inside, reinterpret_cast<uint32_t*>(y), w);
}
// ... eight of them; the lane's row: whether there is one, and its offset -> the lane's code
__device__ __noinline__ uint32_t cl_odd_store(uint32_t* yp, int ok, int where, F2 a, F2 b, F2 c, F2 d) {
  const F2 v[CL_EC / 2] = {a, b, c, d};
  uint32_t code = 0u;
#pragma unroll
  for (int r = 0; r < CL_EC; ++r) {
    const float2 xy = f2_get(v[r >> 1]);
    int at;
    uint32_t bits;
    const uint32_t row = cl_odd_row(r & 1 ? xy.y : xy.x, at, bits);
    const bool there = __shfl_sync(0xffffffffu, ok, r);
    const int o = __shfl_sync(0xffffffffu, where, r);
    if (there) yp[o + at] = bits;
    if ((threadIdx.x & 7) == r) code = row;
  }
  return code;
}
// eight rows of a block as parts; rows out of range as they are
__device__ __forceinline__ void cl_store_parts(const ClConvParams& p, const ClHot& h, const ClEpiState& e, const ClUnit& g, const int4* col_tab, int c0, int inside,
                                               F2 (&v)[CL_EC / 2]) {
  const int lane = threadIdx.x & 31;
  const int4 tb = cl_column(p, g, col_tab, c0);
  uint32_t code = CB_NORMAL;
  const bool ordinary = cl_ordinary(v, __ballot_sync(0xffffffffu, tb.x >= 0) & 0xffu);
  if (!ordinary) code = cl_odd_store(e.yp, tb.x >= 0, tb.y, v[0], v[1], v[2], v[3]);
  if (lane < CL_EC && tb.x >= 0) e.code[tb.y >> 5] = static_cast<uint8_t>(code);
  if (!ordinary) return;
  uint32_t w[CL_EC];
#pragma unroll
  for (int c = 0; c < CL_EC / 2; ++c) {
    uint32_t hi, lo;
    cl_parts(v[c], CL_X_SCALE, hi, lo);
    cl_exchange(hi, lo, w[2 * c], w[2 * c + 1]);
  }
  cl_store(p, h, g, col_tab, c0, inside, e.yp + (lane & 1 ? 16 : 0) + (lane >> 1), w);
}
__device__ __forceinline__ void cl_finish(const ClConvParams& p, const ClHot& h, const ClEpiState& e, const ClUnit& g, const int4* col_tab, int c0, int inside,
                                          F2 (&v)[CL_EC / 2]) {
  if (h.two) cl_store(p, h, g, col_tab, c0, inside, e.y, v);
  if (h.act == CA_SNAKE) cl_act<CA_SNAKE>(e.alpha, e.ialpha, v);
  else if (h.act == CA_ELU) cl_act<CA_ELU>(e.alpha, e.ialpha, v);
  else if (h.act == CA_GELU) cl_act<CA_GELU>(e.alpha, e.ialpha, v);
  if (h.parts) cl_store_parts(p, h, e, g, col_tab, c0, inside, v);
  else cl_store(p, h, g, col_tab, c0, inside, e.y2 ? e.y2 : e.y, v);
}

struct ClMaps {
  CUtensorMap x, y, last, r;         // activations; boxes of plain values beside others, of the last values (fp32 or parts), of residuals
};
struct ClBoxes {               // a warp's boxes of 8 x 32 words
  uint32_t at;                 // four of them
  uint64_t* res_full;          // the box of residuals has landed
  uint32_t res_ph, flip;
};
// The chunks of a unit whose tile is one run of positions: results leave and residuals come as boxes.  A thread's words lie 128 bytes apart in
// them, so a word costs one instruction with a constant offset (its address in global memory costs two or three more).
template <int ACT>
__device__ __forceinline__ void cl_boxed_chunks(const ClHot& h, const ClMaps& maps, const ClEpiState& e, int n_box, int t0, int b0, int inside,
                                                uint32_t taddr, float inv, int c_first, int c_step, ClBoxes& bx, BoundedWait& bw) {
  const int lane = threadIdx.x & 31, cols = h.cols;
  const bool two = h.two, res = h.res, parts = h.parts;
#pragma unroll 1
  for (int c0 = c_first; c0 < inside; c0 += c_step) {          // (chunks behind the last position have nothing to leave)
    const uint32_t in = bx.at + (bx.flip ? 1024u : 0u) + lane * 4;                       // residuals, or plain values
    const uint32_t out = bx.at + (res ? 2048u : two ? (bx.flip ? 3072u : 1024u) : 2048u) + (res || !two ? (bx.flip ? 1024u : 0u) : 0u);
    const uint32_t plain = bx.at + (bx.flip ? 2048u : 0u);
    if (res) {
      bw.wait(bx.res_full, bx.res_ph);
      if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; return; }
      bx.res_ph ^= 1u;
      if (lane == 0 && c0 + c_step < inside) {         // (the other box has been read: every lane has passed the chunk in front)
        mbar_arrive_expect_tx(bx.res_full, 1024u);
        tma_load_3d(bx.at + (bx.flip ? 0u : 1024u), &maps.r, smem_u32(bx.res_full), n_box, t0 + c0 + c_step, b0);
      }
    }
    F2 v[CL_EC / 2];
    cl_load_acc(taddr + c0, cols, inv, v);
#pragma unroll
    for (int c = 0; c < CL_EC / 2; ++c) v[c] = f2_add(v[c], f2(e.bias));
    if (res) {
      float rs[CL_EC];
#pragma unroll
      for (int c = 0; c < CL_EC; ++c) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(rs[c]) : "r"(in + c * 128) : "memory");
      if (h.epi == CE_RESID) {
#pragma unroll
        for (int c = 0; c < CL_EC / 2; ++c) v[c] = f2_add(v[c], f2(rs[2 * c], rs[2 * c + 1]));
      } else if (h.epi == CE_SCALE_RESID) {
#pragma unroll
        for (int c = 0; c < CL_EC / 2; ++c) v[c] = f2_fma(v[c], f2(e.scale), f2(rs[2 * c], rs[2 * c + 1]));
      } else {
        const float nz = (lane & 7) + c0 < inside ? __ldcg(e.noise + c0 + (lane & 7)) : 0.f;
#pragma unroll
        for (int c = 0; c < CL_EC / 2; ++c)
          v[c] = f2_fma(v[c], f2(__shfl_sync(0xffffffffu, nz, 2 * c), __shfl_sync(0xffffffffu, nz, 2 * c + 1)), f2(rs[2 * c], rs[2 * c + 1]));
      }
    }
    // the boxes stored two chunks ago have been read
    if (lane == 0) bulk_wait_read<1>();
    __syncwarp();
    auto put = [&](uint32_t a) {
#pragma unroll
      for (int c = 0; c < CL_EC / 2; ++c) {
        const float2 x = f2_get(v[c]);
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(a + 2 * c * 128), "f"(x.x) : "memory");
        asm volatile("st.shared.f32 [%0], %1;" ::"r"(a + (2 * c + 1) * 128), "f"(x.y) : "memory");
      }
    };
    if (two) put(plain + lane * 4);
    cl_act<ACT>(e.alpha, e.ialpha, v);
    if (parts) {
      uint32_t code = CB_NORMAL;
      if (cl_ordinary(v, c0 + CL_EC <= inside ? 0xffu : (1u << (inside - c0)) - 1u)) {
        const uint32_t a = out + (lane & 1 ? 64u : 0u) + (lane >> 1) * 4;
#pragma unroll
        for (int c = 0; c < CL_EC / 2; ++c) {
          uint32_t hi, lo, w0, w1;
          cl_parts(v[c], CL_X_SCALE, hi, lo);
          cl_exchange(hi, lo, w0, w1);
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(a + 2 * c * 128), "r"(w0) : "memory");
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(a + (2 * c + 1) * 128), "r"(w1) : "memory");
        }
      } else {
        put(out + lane * 4);
#pragma unroll 1
        for (int r = 0; r < CL_EC; ++r) {          // (every lane has read its value when the lanes have exchanged theirs)
          float x;
          int at;
          uint32_t bits;
          asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(out + r * 128 + lane * 4) : "memory");
          const uint32_t row = cl_odd_row(x, at, bits);
          asm volatile("st.shared.b32 [%0], %1;" ::"r"(out + r * 128 + at * 4), "r"(bits) : "memory");
          if ((lane & 7) == r) code = row;
        }
      }
      if (lane < CL_EC && c0 + lane < inside) e.code[(c0 + lane) * (h.N >> 5)] = static_cast<uint8_t>(code);
    } else {
      put(out + lane * 4);
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) {             // (what a box has past the last position is not written)
      if (two) tma_store_3d(&maps.y, plain, n_box, t0 + c0, b0);
      tma_store_3d(&maps.last, out, n_box, t0 + c0, b0);
      bulk_commit();
    }
    bx.flip ^= 1u;
  }
}

struct ClSplit {
  uint32_t smem0;
  int x_bytes, u_first, u_step, kb_lo, x_steps;
  uint64_t *x_ready, *x_empty, *top_full, *top_empty;
  uint32_t* tops;
  const int2* row_tab;
};
// The split's loop.  A thread takes one 16-byte chunk of every 16th row (32nd where a stage is 32 channels wide): NP rows of a stage, in batches
// of eight loads -- half a stage or several stages.  As soon as a row is converted the row of the next batch that takes its registers is asked
// for, so eight loads a thread are on the way all the time, across stages and units.
template <int NP>
__device__ __forceinline__ void cl_split(const ClConvParams& p, const ClSplit& sp, BoundedWait& bw) {
  constexpr int NJ = 8, PB = NP < NJ ? NP : NJ, SB = NJ / PB, HALVES = NP / PB;      // rows and stages of a batch, batches of a stage
  constexpr int NONE = static_cast<int>(0x80000000u);
  const int wsp = (threadIdx.x >> 5) - 2, lane = threadIdx.x & 31;
  const int lanes = 8 * p.group, ch = lane & (lanes - 1), rows_pass = 256 / lanes, row0 = wsp * (32 / lanes) + lane / lanes;
  const int rows = p.cols + p.halo;
  // (rows_pass is a multiple of 16, so the swizzle of a thread's rows is one)
  const uint32_t dst0 = sp.smem0 + (ch >> 3) * p.rows_pad * 128 + (ch & 1) * 8 + row0 * 128 + ((((ch >> 1) & 3) ^ (row0 & 7)) << 4);
  int off[NP];
  const float* xu = p.x;             // first position of the unit's first entry, this thread's channels
  int u = sp.u_first, st = 0, half = 0;                    // the batch in registers
  // rows of unit `v` (for stage `stage` where every tap has its own)
  auto rows_of = [&](int v, int stage) {
    const ClUnit g = cl_unit(p, v);
    const int shift = p.taps > 1 ? p.halo : (p.ksize > 1 ? (p.ksize - 1 - stage % p.ksize) * p.dil : 0);
    xu = p.x + g.b0 * p.x_bstride + static_cast<long long>(g.t0 - shift) * p.Cin + ch * 4;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int r = i * rows_pass + row0;
      const int2 tab = r < rows ? sp.row_tab[r] : make_int2(-1, 0);
      const int t = g.t0 - shift + (tab.x & 0xffff);
      off[i] = tab.x >= 0 && g.b0 + (tab.x >> 16) < p.B && t >= 0 && t < min(p.Tx, p.n_hi) ? tab.y : NONE;
    }
  };
  const bool by_tap = p.taps == 1 && p.ksize > 1;          // (only with one stage a batch)
  auto channels = [&](int stage) { return xu + (sp.kb_lo + (by_tap ? stage / p.ksize : stage)) * p.group * 32; };
  auto load = [&](const float* xk, int o) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (o != NONE) v = __ldcg(reinterpret_cast<const float4*>(xk + o));
    return v;
  };
  float4 v[NJ];
  if (u < p.units) {
    rows_of(u, 0);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j / PB < sp.x_steps) v[j] = load(channels(j / PB), off[j % PB]);
    }
  }
  int s = 0, it = 0;
  uint32_t ph = 0;
  uint32_t top = 0u, low = 0xffffffffu;        // bits of the largest four-channel magnitude, and of the smallest that is not zero, less one
#pragma unroll 1
  while (u < p.units) {
    int nu = u, ns = st, nh = half + 1;
    if (nh == HALVES) {
      nh = 0;
      ns += SB;
      if (ns >= sp.x_steps) {
        ns = 0;
        nu += sp.u_step;
      }
    }
    const bool more = nu < p.units;
    if (more && (nu != u || (by_tap && ns != st))) rows_of(nu, ns);
    const float* xk = channels(ns);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const bool on = SB == 1 || st + j / PB < sp.x_steps;
      if (on) {
        if (j % PB == 0 && (HALVES == 1 || half == 0)) {
          bw.wait(&sp.x_empty[s], ph ^ 1u);
          if (!__all_sync(0xffffffffu, !bw.dead)) {
            bw.dead = true;
            return;
          }
        }
        const int pass = HALVES == 1 ? j % PB : half * PB + j;
        if (pass * rows_pass < rows) {
          uint32_t h0, h1, l0, l1;
          cl_parts(f2(v[j].x, v[j].y), CL_X_SCALE, h0, l0);
          cl_parts(f2(v[j].z, v[j].w), CL_X_SCALE, h1, l1);
          const uint32_t m = __float_as_uint(max3_abs(max3_abs(v[j].x, v[j].y, v[j].z), v[j].w, v[j].w));         // (a NaN has the largest)
          top = max(top, m);
          low = min(low, m - 1u);
          const uint32_t a = dst0 + s * sp.x_bytes + pass * rows_pass * 128;
          asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(h0), "r"(h1) : "memory");
          asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a ^ 64u), "r"(l0), "r"(l1) : "memory");
        }
      }
      if (more) {
        if (HALVES == 1) {
          if (SB == 1 || ns + j / PB < sp.x_steps) v[j] = load(SB == 1 ? xk : xk + (j / PB) * p.group * 32, off[j % PB]);
        } else {
          v[j] = load(xk, nh == 0 ? off[j] : off[(PB + j) % NP]);
        }
      }
      if (on && j % PB == PB - 1 && (HALVES == 1 || half == HALVES - 1)) {        // the warp's rows of the stage are there
        const bool last = st + j / PB + 1 == sp.x_steps;
        if (last) {
          const bool look = __any_sync(0xffffffffu, top >= __float_as_uint(CL_X_TOP) || low < __float_as_uint(CL_X_LOW) - 1u);
          bw.wait(&sp.top_empty[it & 7], ((it >> 3) & 1) ^ 1);
          if (lane == 0) sp.tops[(it & 7) * CL_SPLIT_WARPS + wsp] = look;
          top = 0u;
          low = 0xffffffffu;
        }
        __syncwarp();
        if (lane == 0) {
          if (last) mbar_arrive(&sp.top_full[it & 7]);
          mbar_arrive(&sp.x_ready[s]);
        }
        if (last) ++it;
        if (++s == p.x_stages) { s = 0; ph ^= 1u; }
      }
    }
    u = nu;
    st = ns;
    half = nh;
  }
}

// PARTS: the activations come as parts, fetched by a tensor map; otherwise as fp32, split on the way
template <bool PARTS>
struct ClRoles {
  static constexpr int FIRST_EPI = PARTS ? 4 : 2 + CL_SPLIT_WARPS, EPI_WARPS = PARTS ? 12 : 8, THREADS = 32 * (FIRST_EPI + EPI_WARPS);
};
template <bool PARTS>
__global__ void __launch_bounds__(ClRoles<PARTS>::THREADS, 1) cl_conv_kernel(const __grid_constant__ ClConvParams p, const __grid_constant__ ClMaps maps) {
  constexpr int FIRST_EPI = ClRoles<PARTS>::FIRST_EPI, EPI_WARPS = ClRoles<PARTS>::EPI_WARPS, THREADS = ClRoles<PARTS>::THREADS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int x_sub = p.rows_pad * 128, x_bytes = p.group * x_sub, w_bytes = p.group * CL_W_BLOCK;
  uint8_t* w_smem = smem + p.x_stages * x_bytes;
  uint8_t* boxes = w_smem + p.w_stages * w_bytes;               // four boxes per epilogue warp
  uint8_t* tail = boxes + (p.staged ? EPI_WARPS * 4096 : 0);
  uint64_t* x_ready = reinterpret_cast<uint64_t*>(tail);        // a stage's parts are in shared memory
  uint64_t* x_empty = x_ready + CL_X_STAGES;                    // the MMAs have read them
  uint64_t* w_full = x_empty + CL_X_STAGES;
  uint64_t* w_empty = w_full + CL_W_STAGES;
  uint64_t* acc_full = w_empty + CL_W_STAGES;                   // [2]
  uint64_t* acc_empty = acc_full + 2;                           // [2]
  uint64_t* top_full = acc_empty + 2;                           // [CL_TOPS] a unit's range of values is known (units taken in turn)
  uint64_t* top_empty = top_full + CL_TOPS;
  uint64_t* res_full = top_empty + CL_TOPS;                     // [EPI_WARPS]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(res_full + 12);
  const uint32_t gate = smem_u32(tmem_slot + 1);                // set once the kernels in front have completed
  uint32_t* tops = reinterpret_cast<uint32_t*>(tail + 640);     // [CL_TOPS][CL_SPLIT_WARPS] whether a unit may have columns out of range (PARTS: one word)
  int2* row_tab = reinterpret_cast<int2*>(tail + 1024);         // [CL_ROWS] (entry << 16 | row of the entry) or -1, offset in x
  int4* col_tab = reinterpret_cast<int4*>(tail + 1024 + CL_ROWS * 8);      // [CL_ROWS] the same or -1, offsets in y, resid, noise
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  BoundedWait bw{p.wait_flag, gate};

  if (warp == 0 && lane == 0) {
    tmem_slot[1] = 0u;
    if (PARTS) prefetch_tmap(&maps.x);
    for (int s = 0; s < CL_X_STAGES; ++s) {
      mbar_init(&x_ready[s], PARTS ? 1 : CL_SPLIT_WARPS);
      mbar_init(&x_empty[s], 1);
    }
    for (int s = 0; s < CL_W_STAGES; ++s) {
      mbar_init(&w_full[s], 1);
      mbar_init(&w_empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], EPI_WARPS);
    }
    for (int i = 0; i < CL_TOPS; ++i) {
      mbar_init(&top_full[i], PARTS ? 1 : CL_SPLIT_WARPS);
      mbar_init(&top_empty[i], EPI_WARPS);
    }
    for (int i = 0; i < EPI_WARPS; ++i) mbar_init(&res_full[i], 1);
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  for (int r = threadIdx.x; r < CL_ROWS; r += THREADS) {      // the same for every tile
    const int e = r / p.pitch, q = r - e * p.pitch;
    row_tab[r] = make_int2(e < p.nb ? (e << 16) | q : -1, static_cast<int>(e * p.x_bstride) + q * p.Cin);
    col_tab[r] = make_int4(e < p.nb && q < p.nr ? (e << 16) | q : -1, static_cast<int>(e * p.y_bstride) + q * p.N,
                           static_cast<int>(e * p.r_bstride) + q * p.N, e * p.noise_ld + q);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // this CTA's units, and its share of a unit's channels
  const int rank = p.splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int u_first = p.splits > 1 ? blockIdx.x / p.splits : blockIdx.x, u_step = p.splits > 1 ? p.units : gridDim.x;
  const int kb_lo = rank * p.kb / p.splits, kb_n = (rank + 1) * p.kb / p.splits - kb_lo;
  const int tap_steps = p.ksize / p.taps, x_steps = kb_n * tap_steps;        // stages of activations a unit takes

  if (warp == 0) {
    // ================= weights =================
    if (lane == 0) {
      const int blocks_per_tap = p.Cin >> 5;
      const size_t tile_bytes = static_cast<size_t>(blocks_per_tap) * p.ksize * CL_W_BLOCK;
      const uint32_t dst0 = smem_u32(w_smem), bar0 = smem_u32(w_full);
      int s = 0, pre = p.w_stages;         // stages filled before the kernels in front have completed: weights do not depend on them
      uint32_t ph = 0;
      auto after_wait = [&]() {
        pdl_wait();
        wait_gate_open(gate);
        pdl_trigger();
      };
      for (int u = u_first; u < p.units && !bw.dead; u += u_step) {
        const uint8_t* src = p.w + static_cast<size_t>(cl_unit(p, u).m0 >> 7) * tile_bytes;
        for (int i = kb_lo; i < kb_lo + kb_n && !bw.dead; ++i) {
          for (int tap = 0; tap < p.ksize; ++tap) {
            if (pre == 0) after_wait();
            --pre;
            if (!p.resident) bw.wait(&w_empty[s], ph ^ 1u);
            if (bw.dead) break;
            mbar_arrive_expect_tx(&w_full[s], w_bytes);
            cl_bulk(dst0 + s * w_bytes, src + static_cast<size_t>(tap * blocks_per_tap + i * p.group) * CL_W_BLOCK, w_bytes, bar0 + 8 * s);
            if (++s == p.w_stages) { s = 0; ph ^= 1u; }
          }
        }
        if (p.resident) break;
      }
      if (pre >= 0) after_wait();
      if (bw.dead) {            // let the copies in flight land before the block may leave
        const unsigned long long t0 = gtimer();
        while (gtimer() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================= MMA issuer =================
    // The whole warp walks the loop and one elected lane issues: descriptors and TMEM addresses stay in uniform registers.
    const uint64_t w_desc0 = umma_desc_sw128_kmajor(smem_u32(w_smem)), x_desc0 = umma_desc_sw128_kmajor(smem_u32(smem));
    const uint32_t idesc = umma_idesc(128, p.cols, 0u);
    int xs = 0, ws = 0, it = 0;
    uint32_t xph = 0, wph = 0;
    for (int u = u_first; u < p.units && !bw.dead; u += u_step, ++it) {
      const int acc = p.acc_bufs > 1 ? it & 1 : 0;
      bw.wait(&acc_empty[acc], ((p.acc_bufs > 1 ? it >> 1 : it) & 1) ^ 1);
      if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
      tc_fence_after();
      const uint32_t d = tmem_base + acc * p.acc_cols, d2 = d + p.cols;
      for (int i = 0; i < x_steps && !bw.dead; ++i) {
        bw.wait(&x_ready[xs], xph);
        // Parts written by threads, to be read by the tensor core.  The fence stands here and not with the writers, where it would wait for the
        // loads that they have on the way.  It orders them all the same: a proxy fence counts anywhere on the path from the writes to the reads,
        // and the writes come before it by the writers' arrivals (release) and this warp's wait (acquire), the MMAs after it in program order.
        if (!PARTS) fence_proxy_async();
        for (int tap = 0; tap < p.taps; ++tap) {
          if (!p.resident || it == 0) bw.wait(&w_full[ws], wph);
          if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
          tc_fence_after();
          if (elect_one()) {
            uint64_t w_hi = w_desc0 + static_cast<uint64_t>(ws) * (w_bytes >> 4);
            uint64_t x_hi = x_desc0 + static_cast<uint64_t>(xs) * (x_bytes >> 4) + tap * p.dil * 8;      // a tap: the tile from a later row on
            for (int g = 0; g < p.group; ++g) {
#pragma unroll
              for (int k = 0; k < 2; ++k) {            // (the low parts lie 64 bytes behind the high ones)
                const uint32_t go = (i | tap | g | k) ? 1u : 0u;
                umma_bf16(d, w_hi + 2 * k, x_hi + 2 * k, idesc, go);
                umma_bf16(d2, w_hi + 2 * k, x_hi + 4 + 2 * k, idesc, go);
                umma_bf16(d2, w_hi + 4 + 2 * k, x_hi + 2 * k, idesc, 1u);
              }
              w_hi += CL_W_BLOCK >> 4;
              x_hi += x_sub >> 4;
            }
            if (!p.resident) umma_commit(&w_empty[ws]);
            if (tap + 1 == p.taps) {
              umma_commit(&x_empty[xs]);
              if (i + 1 == x_steps) umma_commit(&acc_full[acc]);
            }
          }
          __syncwarp();
          if (++ws == p.w_stages) { ws = 0; wph ^= 1u; }
        }
        if (++xs == p.x_stages) { xs = 0; xph ^= 1u; }
      }
    }
  } else if (PARTS && warp == 2) {
    // ================= activations =================
    if (lane == 0) {
      const uint32_t box = static_cast<uint32_t>(p.nb * p.pitch) * 128u, dst0 = smem_u32(smem), bar0 = smem_u32(x_ready);
      int s = 0;
      uint32_t ph = 0;
      pdl_wait();
      for (int u = u_first; u < p.units && !bw.dead; u += u_step) {
        const ClUnit g = cl_unit(p, u);
        for (int i = kb_lo; i < kb_lo + kb_n && !bw.dead; ++i) {
          for (int tap = 0; tap < tap_steps; ++tap) {
            bw.wait(&x_empty[s], ph ^ 1u);
            if (bw.dead) break;
            const int t = g.t0 - (p.taps > 1 ? p.halo : (p.ksize - 1 - tap) * p.dil);
            mbar_arrive_expect_tx(&x_ready[s], p.group * box);
            for (int b = 0; b < p.group; ++b)
              tma_load_3d(dst0 + s * x_bytes + b * x_sub, &maps.x, bar0 + 8 * s, (i * p.group + b) * 64, t, g.b0);
            if (++s == p.x_stages) { s = 0; ph ^= 1u; }
          }
        }
      }
      if (bw.dead) {            // let the copies in flight land before the block may leave
        const unsigned long long t0 = gtimer();
        while (gtimer() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
    __syncwarp();
  } else if (PARTS && warp == 3) {
    // ================= codes of the rows that a unit's outputs are made of =================
    const int cb = p.Cin >> 5, back = (p.ksize - 1) * p.dil;
    pdl_wait();
    int it = 0;
    for (int u = u_first; u < p.units && !bw.dead; u += u_step, ++it) {
      const ClUnit g = cl_unit(p, u);
      uint32_t code = 0u;
      const int ta = max(g.t0 - back, 0), tb = min(min(g.t0 + p.nr, p.n_hi), p.Tx);
      for (int e = 0; e < p.nb && g.b0 + e < p.B && ta < tb; ++e) {
        const uint8_t* base = p.x_code + ((g.b0 + e) * p.x_bstride >> 5);
        const long long lo = static_cast<long long>(ta) * cb, hi = static_cast<long long>(tb) * cb;
        const uintptr_t a = reinterpret_cast<uintptr_t>(base + lo), b = reinterpret_cast<uintptr_t>(base + hi), a4 = min((a + 3) & ~uintptr_t(3), b),
                        b4 = max(b & ~uintptr_t(3), a4);
        for (uintptr_t q = a4 + 4 * lane; q < b4; q += 128) code |= __ldcg(reinterpret_cast<const uint32_t*>(q));
        if (a + lane < a4) code |= __ldcg(reinterpret_cast<const uint8_t*>(a + lane));
        if (b4 + lane < b) code |= __ldcg(reinterpret_cast<const uint8_t*>(b4 + lane));
      }
      code = __reduce_or_sync(0xffffffffu, code);
      code |= code >> 16;
      const bool look = (code | code >> 8) & CB_RAW;
      bw.wait(&top_empty[it & (CL_TOPS - 1)], ((it / CL_TOPS) & 1) ^ 1);
      if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
      if (lane == 0) {
        tops[(it & (CL_TOPS - 1)) * CL_SPLIT_WARPS] = look;
        mbar_arrive(&top_full[it & (CL_TOPS - 1)]);
      }
      __syncwarp();
    }
  } else if (!PARTS && warp < 2 + CL_SPLIT_WARPS) {
    // ================= split: global memory -> registers -> two fp16 parts in shared memory =================
    const ClSplit sp{smem_u32(smem), x_bytes, u_first, u_step, kb_lo, x_steps, x_ready, x_empty, top_full, top_empty, tops, row_tab};
    pdl_wait();
    switch (p.passes) {
      case 1: cl_split<1>(p, sp, bw); break;
      case 2: cl_split<2>(p, sp, bw); break;
      case 4: cl_split<4>(p, sp, bw); break;
      case 8: cl_split<8>(p, sp, bw); break;
      default: cl_split<16>(p, sp, bw); break;
    }
  } else {
    // ================= epilogue =================
    // A lane holds one channel at eight positions, and every store and residual load of a warp is one run of 128
    // bytes.  The four quarters of TMEM hold 128 channels, or copies of 64 or 32 that share the columns; two or three warps a
    // quarter.
    const int quarter = warp & 3, lane_row = quarter * 32 + lane;
    const ClHot h{p.cols, p.N, p.epi, p.act, p.y && (p.y2 || p.yp), p.epi != CE_PLAIN, p.yp != nullptr};
    ClBoxes bx{smem_u32(boxes) + (warp - FIRST_EPI) * 4096, &res_full[warp - FIRST_EPI], 0u, 0u};
    int it = 0, skew = 0;
    for (int u = u_first; u < p.units && !bw.dead; u += u_step, ++it) {
      const ClUnit g = cl_unit(p, u);
      const int acc = p.acc_bufs > 1 ? it & 1 : 0;
      const uint32_t acc_ph = (p.acc_bufs > 1 ? it >> 1 : it) & 1;
      const uint32_t taddr = tmem_base + acc * p.acc_cols + (static_cast<uint32_t>(quarter * 32) << 16);
      const int width = min(128, p.N - g.m0), copies = cl_copies(width);        // (N is a multiple of 32)
      const int row = copies == 1 ? lane_row : lane_row & (width - 1);
      const bool mine = row < width;
      // This warp's chunks of eight columns: every `turns`-th one.  Which warps have one more than the others goes round from unit to unit (there are
      // two accumulators): 16 chunks for the 6 warps of 64 channels are 8 in three units instead of 3 in each.  Mimi, 32 windows in a row of calls: 614400 x 64
      // with residual 117 -> 112 us, 614400 x 32 88 -> 84, 153600 x 256 to two outputs 114 -> 110.
      const int turns = EPI_WARPS / 4 * copies;          // (of a tile's own width: it divides EPI_WARPS, so `skew` is kept modulo that)
      int turn = ((warp - FIRST_EPI) >> 2) * copies + (copies == 4 ? quarter : copies == 2 ? quarter >> 1 : 0) - skew % turns;
      if (turn < 0) turn += turns;
      skew = (skew + h.cols / CL_EC) % EPI_WARPS;
      ClEpiState e;
      e.n = g.m0 + row;
      const int nm = p.cmod == h.N ? e.n : e.n % p.cmod;
      float inv = 0.f;
      e.bias = e.alpha = e.ialpha = 0.f;
      e.scale = 1.f;
      if (mine) {
        inv = __ldg(p.w_inv + g.m0 + lane_row);
        if (p.bias) e.bias = __ldg(p.bias + nm);
        if (p.epi == CE_SCALE_RESID) e.scale = __ldg(p.scale + e.n);
        if (p.act == CA_SNAKE) {
          e.alpha = __ldg(p.alpha + nm);
          e.ialpha = __ldg(p.alpha + p.cmod + nm);
        }
      }
      const long long at = static_cast<long long>(g.t0 - p.n_lo) * p.N + e.n;
      e.y = p.y ? p.y + (g.b0 * p.y_bstride + at) : nullptr;
      e.y2 = p.y2 ? p.y2 + (g.b0 * p.y_bstride + at) : nullptr;
      const long long block = g.b0 * p.y_bstride + (at - (e.n & 31));
      e.yp = p.yp ? p.yp + block : nullptr;
      e.code = p.yp_code + (block >> 5);
      e.resid = p.resid + (g.b0 * p.r_bstride + at);
      e.noise = p.noise + (static_cast<long long>(g.b0) * p.noise_ld + g.t0);
      const int inside = p.nb == 1 ? min(p.nr, p.n_hi - g.t0) : 0;       // columns in front of this one are one run of rows
      if (p.epi != CE_PLAIN && it == 0) pdl_wait();
      bool first = true;
      auto wait_acc = [&]() {
        bw.wait(&top_full[it & (CL_TOPS - 1)], (it / CL_TOPS) & 1);
        bw.wait(&acc_full[acc], acc_ph);
        if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; return; }
        tc_fence_after();
        first = false;
        const bool look = __any_sync(0xffffffffu, tops[(it & (CL_TOPS - 1)) * CL_SPLIT_WARPS + (PARTS ? 0 : lane & 7)] != 0u);
        if (lane == 0) mbar_arrive(&top_empty[it & (CL_TOPS - 1)]);
        if (look) {
          if (mine) {
            const int blk_lo = kb_lo * p.group, blk_hi = (kb_lo + kb_n) * p.group;
#pragma unroll 1
            for (int c0 = turn * CL_EC; c0 < p.cols; c0 += turns * CL_EC) {
              const uint32_t mask = cl_exact_columns<PARTS>(p, col_tab, g.t0, g.b0, c0, blk_lo, blk_hi);
#pragma unroll 1
              for (int c = c0; c < c0 + CL_EC; c += 4)
                cl_exact_chunk(p, col_tab, g.m0, g.t0, g.b0, c, lane_row, blk_lo, blk_hi, taddr + c, taddr + p.cols + c, mask >> (c - c0) & 15u, inv);
            }
          }
          inv = 1.f;
        }
      };
      if (p.staged) {
        const int c_first = turn * CL_EC, c_step = turns * CL_EC, n_box = g.m0 + (row & ~31);
        const bool some = mine && c_first < inside;
        if (some && h.res && lane == 0) {          // the first residuals, asked for before the accumulator is waited for
          mbar_arrive_expect_tx(bx.res_full, 1024u);
          tma_load_3d(bx.at + (bx.flip ? 1024u : 0u), &maps.r, smem_u32(bx.res_full), n_box, g.t0 - p.n_lo + c_first, g.b0);
        }
        wait_acc();
        if (!bw.dead && some) {
          switch (h.act) {
            case CA_SNAKE: cl_boxed_chunks<CA_SNAKE>(h, maps, e, n_box, g.t0 - p.n_lo, g.b0, inside, taddr, inv, c_first, c_step, bx, bw); break;
            case CA_ELU: cl_boxed_chunks<CA_ELU>(h, maps, e, n_box, g.t0 - p.n_lo, g.b0, inside, taddr, inv, c_first, c_step, bx, bw); break;
            case CA_GELU: cl_boxed_chunks<CA_GELU>(h, maps, e, n_box, g.t0 - p.n_lo, g.b0, inside, taddr, inv, c_first, c_step, bx, bw); break;
            default: cl_boxed_chunks<CA_NONE>(h, maps, e, n_box, g.t0 - p.n_lo, g.b0, inside, taddr, inv, c_first, c_step, bx, bw); break;
          }
        }
        if (bw.dead) break;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
      } else if (p.splits == 1) {
        if (mine) {
          float rs[CL_EC];
          int c0 = turn * CL_EC;
          if (h.res && c0 < h.cols) cl_residual(p, h, e, g, col_tab, c0, inside, rs);      // asked for before the accumulator is waited for
#pragma unroll 1
          for (; c0 < h.cols; c0 += turns * CL_EC) {
            if (first) {
              wait_acc();
              if (bw.dead) break;
            }
            F2 v[CL_EC / 2];
            cl_load_acc(taddr + c0, h.cols, inv, v);
            cl_linear(p, h, e, g, col_tab, c0, v, rs);
            if (h.res && c0 + turns * CL_EC < h.cols) cl_residual(p, h, e, g, col_tab, c0 + turns * CL_EC, inside, rs);
            cl_finish(p, h, e, g, col_tab, c0, inside, v);
          }
          if (bw.dead) break;
        }
        if (first) wait_acc();          // (a warp without a chunk of this unit keeps in step with the accumulators all the same)
        if (bw.dead) break;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
      } else {
        // this CTA's part of K into its own shared memory (its stages have been read), then every `splits`-th chunk of all parts
        float* sums = reinterpret_cast<float*>(smem);        // [column][128]
        wait_acc();
        if (!bw.dead) {
#pragma unroll 1
          for (int c0 = turn * CL_EC; c0 < h.cols; c0 += turns * CL_EC) {
            F2 v[CL_EC / 2];
            cl_load_acc(taddr + c0, h.cols, inv, v);
#pragma unroll
            for (int c = 0; c < CL_EC / 2; ++c) {
              const float2 x = f2_get(v[c]);
              sums[(c0 + 2 * c) * 128 + row] = x.x;
              sums[(c0 + 2 * c + 1) * 128 + row] = x.y;
            }
          }
        }
        cluster_sync_all();
        if (!bw.dead && mine) {
#pragma unroll 1
          for (int c0 = (rank + turn * p.splits) * CL_EC; c0 < h.cols; c0 += p.splits * turns * CL_EC) {
            float rs[CL_EC];
            F2 v[CL_EC / 2];
            if (h.res) cl_residual(p, h, e, g, col_tab, c0, inside, rs);
#pragma unroll
            for (int c = 0; c < CL_EC / 2; ++c) v[c] = f2(0.f);
#pragma unroll 1
            for (int k = 0; k < p.splits; ++k) {
#pragma unroll
              for (int c = 0; c < CL_EC / 2; ++c)
                v[c] = f2_add(v[c], f2(ld_dsmem_f32(sums + (c0 + 2 * c) * 128 + row, k), ld_dsmem_f32(sums + (c0 + 2 * c + 1) * 128 + row, k)));
            }
            cl_linear(p, h, e, g, col_tab, c0, v, rs);
            cl_finish(p, h, e, g, col_tab, c0, inside, v);
          }
        }
        cluster_sync_all();
        break;
      }
    }
    if (p.staged && lane == 0) {
      bulk_wait_read<0>();
      if (bw.dead) {            // a box of residuals may be on its way
        const unsigned long long t0 = gtimer();
        while (gtimer() - t0 < 2000000ull) __nanosleep(1000);
      }
    }
    __syncwarp();
  }
  if (p.splits > 1 && warp < FIRST_EPI) {        // (the epilogue's two meetings of the cluster are every warp's)
    __syncwarp();
    cluster_sync_all();
    cluster_sync_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// channel of a packed row: a last tile of 32 or 64 channels is repeated over its 128 rows
__device__ __forceinline__ int cl_packed_row(int r, int N) {
  const int m0 = r & ~127, width = min(128, N - m0);
  return cl_copies(width) > 1 ? m0 + (r & (width - 1)) : r;
}
// scale of every output channel's weights: the power of two that brings the largest finite one into [2^13, 2^14)
__global__ void __launch_bounds__(256) cl_scale_kernel(float* __restrict__ inv, const float* __restrict__ w, int N, int K) {
  const int n = cl_packed_row(blockIdx.x, N);
  __shared__ float sm[8];
  float m = 0.f;
  if (n < N) {
    for (int k = threadIdx.x; k < K; k += 256) {
      const float a = fabsf(w[static_cast<size_t>(n) * K + k]);
      if (a < INFINITY) m = fmaxf(m, a);
    }
  }
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) m = fmaxf(m, sm[i]);
    const int e = m > 0.f ? max(ilogbf(m), -100) : 13;
    inv[blockIdx.x] = ldexpf(1.f / CL_X_SCALE, e - 13);
  }
}

// fp32 weights [N][K] (K = taps x channels, tap-major) -> [128 channels][K / 32][128][32 hi | 32 lo] fp16, 128-byte rows swizzled; channels past N
// zero or (cl_packed_row) repeated
__global__ void __launch_bounds__(256) cl_pack_kernel(uint4* __restrict__ dst, const float* __restrict__ inv, const float* __restrict__ w, int N, int K) {
  const int blk = blockIdx.x, m = blockIdx.y, blocks = gridDim.x;
  uint4* out = dst + (static_cast<size_t>(m) * blocks + blk) * (CL_W_BLOCK / 16);
  for (int i = threadIdx.x; i < 128 * 4; i += 256) {
    const int r = i >> 2, c = i & 3, n = cl_packed_row(m * 128 + r, N);
    uint32_t hi[4] = {0u, 0u, 0u, 0u}, lo[4] = {0u, 0u, 0u, 0u};
    if (n < N) {
      const float s = 1.f / (inv[m * 128 + r] * CL_X_SCALE);
      const float* src = w + static_cast<size_t>(n) * K + blk * 32 + c * 8;
#pragma unroll
      for (int e = 0; e < 4; ++e) cl_parts(f2(src[2 * e], src[2 * e + 1]), s, hi[e], lo[e]);
    }
    out[r * 8 + (c ^ (r & 7))] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    out[r * 8 + ((c + 4) ^ (r & 7))] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// ------------------------------------------------------------------------------------------
// depthwise convolution, 7 taps, dilation d, "same" padding; Snake on the input and on the output (optional both)
// ------------------------------------------------------------------------------------------
// A block owns 64 channels x up to DW_T positions: the (activated) input rows with their halo are staged once in shared memory, so
// every element is read and put through its sine once, in 256-byte rows; a thread finishes four channels of every 16th row, whose
// chains interleave (the activation branches once per four values, to the library's sine when an argument is out of range).
// DW_T 128 and four-wide activations against 64 and one by one: 12 to 30 us a layer -> 4 to 14 (SNAC, 32 windows).
constexpr int DW_T = 128;
__global__ void __launch_bounds__(256) cl_dwconv7_kernel(float* __restrict__ y, uint8_t* __restrict__ code, const float* __restrict__ x, long long x_bstride,
                                                         const float* __restrict__ w, const float* __restrict__ bias,
                                                         const float* __restrict__ alpha_in, const float* __restrict__ alpha_out,
                                                         int C, int T, int dil, int t_lo, int t_hi, int tile_rows) {
  extern __shared__ float4 tile[];          // [rows][16]
  const int c4 = threadIdx.x & 15, r0 = threadIdx.x >> 4;
  const int c = blockIdx.y * 64 + c4 * 4, b = blockIdx.z, t0 = t_lo + blockIdx.x * tile_rows;
  const int halo = 3 * dil, n_out = min(tile_rows, t_hi - t0), rows = n_out + 2 * halo;
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
  const size_t y0 = static_cast<size_t>(b) * T * C + c;
#pragma unroll 2
  for (int r = r0; r < n_out; r += 16) {          // (alike for the sixteen lanes of a row)
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
    const size_t at = y0 + static_cast<size_t>(t0 + r) * C;
    if (code) cl_put4(reinterpret_cast<uint32_t*>(y), code, at, o);
    else *reinterpret_cast<float4*>(y + at) = o;
  }
}

// ------------------------------------------------------------------------------------------
// last convolution of a decoder: one output channel, ksize taps, `left` positions of context before; optional tanh
// ------------------------------------------------------------------------------------------
// Bound by reading x once: sixteen lanes hold sixteen positions, four channels a lane, rows straight from global memory in whole lines and all in
// flight (taps known: 18 rows for 3 taps); sixteen sums a lane then change places in fifteen exchanges, a position a lane.  Against rows staged in
// shared memory and read again for every tap: 32 x 2,048 positions of 64 channels, 7 taps 16.5 us -> 10.9 in a row of calls; 32 x 19,200 positions,
// 3 taps 59 us -> 57, where the kernel in front leaves 157 MB that L2 still has to write back.
constexpr int LC_T = 128, LC_RUN = 16;
template <int KSIZE>          // 0: any
__global__ void __launch_bounds__(LC_T, 4) cl_last_conv_kernel(float* __restrict__ y, const float* __restrict__ x, long long x_bstride,
                                                            const float* __restrict__ w, const float* __restrict__ bias, int C,
                                                            int T, int ksize, int left, int t0, int t1, int use_tanh) {
  // the last rows first: they are what the kernel in front left in L2
  const int b = gridDim.y - 1 - blockIdx.y, lane = threadIdx.x & 15, tb = t0 + (gridDim.x - 1 - blockIdx.x) * LC_T + (threadIdx.x >> 4) * LC_RUN;
  const float* xb = x + static_cast<size_t>(b) * x_bstride;
  float acc[LC_RUN] = {};
  auto tap = [&](int c, int k) {
    return c < C ? make_float4(__ldg(w + (c + 0) * ksize + k), __ldg(w + (c + 1) * ksize + k), __ldg(w + (c + 2) * ksize + k), __ldg(w + (c + 3) * ksize + k))
                 : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto row = [&](int c, int t) {
    return c < C && t >= 0 && t < T ? __ldcg(reinterpret_cast<const float4*>(xb + static_cast<size_t>(t) * C + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto add = [](float& a, const float4& v, const float4& q) { a = fmaf(v.w, q.w, fmaf(v.z, q.z, fmaf(v.y, q.y, fmaf(v.x, q.x, a)))); };
  const float bv = __ldg(bias);
  if constexpr (KSIZE > 0) {
    float4 wk[KSIZE];
#pragma unroll
    for (int k = 0; k < KSIZE; ++k) wk[k] = tap(lane * 4, k);
    pdl_sync();
    for (int c = lane * 4;;) {
      if (tb < t1) {
#pragma unroll
        for (int r = 0; r < LC_RUN + KSIZE - 1; ++r) {
          const float4 v = row(c, tb - left + r);
#pragma unroll
          for (int k = 0; k < KSIZE; ++k)
            if (r - k >= 0 && r - k < LC_RUN) add(acc[r - k], v, wk[k]);
        }
      }
      if ((c += 64) - lane * 4 >= C) break;
#pragma unroll
      for (int k = 0; k < KSIZE; ++k) wk[k] = tap(c, k);
    }
  } else {
    pdl_sync();
    for (int c = lane * 4; tb < t1 && c - lane * 4 < C; c += 64) {
      for (int k = 0; k < ksize; ++k) {
        const float4 q = tap(c, k);
#pragma unroll
        for (int j = 0; j < LC_RUN; ++j) add(acc[j], row(c, tb - left + j + k), q);
      }
    }
  }
#pragma unroll
  for (int o = LC_RUN / 2; o; o >>= 1) {           // (the two halves of a sum are added in the same order for every position)
    const bool up = lane & o;
#pragma unroll
    for (int j = 0; j < o; ++j) {
      const float give = up ? acc[j] : acc[j + o], keep = up ? acc[j + o] : acc[j];
      acc[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  const int t = tb + lane;
  if (t >= t1) return;
  const float o = acc[0] + bv;
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
  const bool wide = cb_dim % 4 == 0 && reinterpret_cast<uintptr_t>(pw) % 16 == 0;
  pdl_sync();
  if (threadIdx.x < 3 * cb_dim) {
    const int i = threadIdx.x / cb_dim, d = threadIdx.x % cb_dim, tl = T / strides[i];
    int code = codes[i][b * tl + t / strides[i]];
    code = min(max(code, 0), cb_size - 1);
    e[i][d] = cb[(static_cast<size_t>(i) * cb_size + code) * cb_dim + d];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float acc = 0.f, a[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) a[i] = __ldg(&pb[i * C + c]);
    for (int d = 0; d < cb_dim; d += 4) {          // (four entries of the three rows in flight together)
      float q[3][4];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const float* r = pw + (static_cast<size_t>(i) * C + c) * cb_dim + d;
        if (wide) {
          const float4 v = __ldg(reinterpret_cast<const float4*>(r));
          q[i][0] = v.x; q[i][1] = v.y; q[i][2] = v.z; q[i][3] = v.w;
        } else {
#pragma unroll
          for (int h = 0; h < 4; ++h) q[i][h] = d + h < cb_dim ? __ldg(r + h) : 0.f;
        }
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (d + h < cb_dim) a[i] += q[i][h] * e[i][d + h];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) acc += a[i];
    z[(static_cast<size_t>(b) * T + t) * C + c] = acc;
  }
}

// z0 [B][T][D] = entry of codebook 0, z1 = sum of the entries of codebooks 1 .. K - 1
__global__ void __launch_bounds__(256) cl_codes_sum_kernel(float* __restrict__ z0, float* __restrict__ z1, uint8_t* __restrict__ code0, uint8_t* __restrict__ code1, const long long* __restrict__ codes,
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
    const float first = emb[static_cast<size_t>(row[0]) * D + d];
    float acc = 0.f;
#pragma unroll 8
    for (int k = 1; k < K; ++k) acc += emb[static_cast<size_t>(row[k]) * D + d];
    if (code0) {                     // (D is a multiple of 32)
      cl_put1(reinterpret_cast<uint32_t*>(z0), code0, o >> 5, first);
      cl_put1(reinterpret_cast<uint32_t*>(z1), code1, o >> 5, acc);
    } else {
      z0[o] = first;
      z1[o] = acc;
    }
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
__global__ void __launch_bounds__(128) cl_layernorm_kernel(float* __restrict__ y, uint8_t* __restrict__ code, const float* __restrict__ x, const float* __restrict__ w,
                                                           const float* __restrict__ bias, int rows, int C, float eps) {
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, n4 = C >> 2;
  float4 ww[8], bb[8];               // (read while the kernel in front still runs)
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (lane + 32 * i < n4) {
      ww[i] = __ldg(reinterpret_cast<const float4*>(w) + lane + 32 * i);
      bb[i] = __ldg(reinterpret_cast<const float4*>(bias) + lane + 32 * i);
    }
  }
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
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = lane + 32 * i;
    if (c < n4) {                    // (with codes: C is a multiple of 32, alike for the eight lanes of a block)
      const float4 o = make_float4((v[i].x - mean) * rstd * ww[i].x + bb[i].x, (v[i].y - mean) * rstd * ww[i].y + bb[i].y,
                                   (v[i].z - mean) * rstd * ww[i].z + bb[i].z, (v[i].w - mean) * rstd * ww[i].w + bb[i].w);
      const size_t at = static_cast<size_t>(row) * C + 4 * c;
      if (code) cl_put4(reinterpret_cast<uint32_t*>(y), code, at, o);
      else *reinterpret_cast<float4*>(y + at) = o;
    }
  }
}

// causal attention inside one chunk of T <= 64 positions, rotary pairs (2j, 2j + 1); qkv [B][T][3 C] -> out [B][T][C].
// One block per (head, batch entry), latency bound: a chunk is a few dozen positions.  The angles do not depend on the input and are found
// while the kernel in front still runs; a thread's rows are all in flight at once; a warp owns four queries (a key of its own per lane, so one read of
// a key serves four sums, and the softmax needs the warp alone), and what it reads in each step of p v are the four weights of a key in
// one load.  32 chunks of 20 positions, 8 heads of 64 dims: 15.8 us of a layer in a row of calls with a block-wide pass per stage; now 9.4.
constexpr int CA_ROWS = 4;
__global__ void __launch_bounds__(256) cl_chunk_attention_kernel(float* __restrict__ out, uint8_t* __restrict__ code, const float* __restrict__ qkv, int C, int H,
                                                                 int T, float max_period) {
  extern __shared__ float4 asm_[];     // p [8 warps][T] of four queries, q, k, v [T][D + 4], frequencies
  const int h = blockIdx.x, b = blockIdx.y, D = C / H, ld = D + 4, half = D >> 1, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float4* p = asm_ + warp * T;
  float* q = reinterpret_cast<float*>(asm_ + 8 * T);
  float* k = q + T * ld;
  float* v = k + T * ld;
  float* freq = v + T * ld;            // [D / 2]
  for (int j = threadIdx.x; j < half; j += blockDim.x)
    freq[j] = expf(static_cast<float>(j) * (-logf(max_period) * 2.f / static_cast<float>(D)));
  __syncthreads();
  const float* base = qkv + static_cast<size_t>(b) * T * 3 * C + h * D;
  for (int i0 = threadIdx.x; i0 - static_cast<int>(threadIdx.x) < T * half; i0 += 4 * 256) {
    float sn[4], cs[4];
    int at[4];
    float2 a[4], e[4], f[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * 256, t = i / half, j = i - t * half;
      at[u] = i < T * half ? t * ld + 2 * j : -1;
      if (at[u] >= 0) sincosf(static_cast<float>(t) * freq[j], &sn[u], &cs[u]);
    }
    if (i0 == static_cast<int>(threadIdx.x)) pdl_sync();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u * 256, t = i / half, j = i - t * half;
      if (at[u] < 0) continue;
      const float* row = base + static_cast<size_t>(t) * 3 * C + 2 * j;
      a[u] = __ldcg(reinterpret_cast<const float2*>(row));
      e[u] = __ldcg(reinterpret_cast<const float2*>(row + C));
      f[u] = __ldcg(reinterpret_cast<const float2*>(row + 2 * C));
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (at[u] < 0) continue;
      *reinterpret_cast<float2*>(q + at[u]) = make_float2(a[u].x * cs[u] - a[u].y * sn[u], a[u].x * sn[u] + a[u].y * cs[u]);
      *reinterpret_cast<float2*>(k + at[u]) = make_float2(e[u].x * cs[u] - e[u].y * sn[u], e[u].x * sn[u] + e[u].y * cs[u]);
      *reinterpret_cast<float2*>(v + at[u]) = f[u];
    }
  }
  __syncthreads();
  const float scale = rsqrtf(static_cast<float>(D));
  const int d4 = D >> 2;
  for (int t0 = warp; t0 < T; t0 += 8 * CA_ROWS) {           // queries t0, t0 + 8, ...; past the end the last one is repeated and not written
    int tq[CA_ROWS];
    float s[2][CA_ROWS], den[CA_ROWS], inv[CA_ROWS];
#pragma unroll
    for (int r = 0; r < CA_ROWS; ++r) tq[r] = min(t0 + 8 * r, T - 1);
    const int last = tq[CA_ROWS - 1];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int tk = lane + 32 * u;
      if (32 * u > last) break;
      const float4* c = reinterpret_cast<const float4*>(k + min(tk, T - 1) * ld);
      float sum[CA_ROWS][4] = {};
#pragma unroll 4
      for (int d = 0; d < d4; ++d) {
        const float4 y = c[d];
#pragma unroll
        for (int r = 0; r < CA_ROWS; ++r) {
          const float4 x = reinterpret_cast<const float4*>(q + tq[r] * ld)[d];
          sum[r][0] += x.x * y.x;
          sum[r][1] += x.y * y.y;
          sum[r][2] += x.z * y.z;
          sum[r][3] += x.w * y.w;
        }
      }
#pragma unroll
      for (int r = 0; r < CA_ROWS; ++r) s[u][r] = ((sum[r][0] + sum[r][1]) + (sum[r][2] + sum[r][3])) * scale;
    }
#pragma unroll
    for (int r = 0; r < CA_ROWS; ++r) {
      float mx = lane <= tq[r] ? s[0][r] : -INFINITY;
      if (lane + 32 <= tq[r]) mx = fmaxf(mx, s[1][r]);
      mx = warp_max(mx);
      s[0][r] = lane <= tq[r] ? expf(s[0][r] - mx) : 0.f;
      s[1][r] = lane + 32 <= tq[r] ? expf(s[1][r] - mx) : 0.f;
      den[r] = warp_sum(s[0][r] + s[1][r]);
      inv[r] = 1.f / den[r];
    }
    __syncwarp();                      // (the weights of the queries before have been read)
    if (lane <= last) p[lane] = make_float4(s[0][0], s[0][1], s[0][2], s[0][3]);
    if (lane + 32 <= last) p[lane + 32] = make_float4(s[1][0], s[1][1], s[1][2], s[1][3]);
    __syncwarp();
    for (int d0 = 0; d0 < D; d0 += 64) {
      float o[2][CA_ROWS] = {};
      const int d = d0 + lane, da = min(d, D - 1), db = min(d + 32, D - 1);
#pragma unroll 4
      for (int tk = 0; tk <= last; ++tk) {
        const float4 w = p[tk];
        const float x = v[tk * ld + da], y = v[tk * ld + db], ws[CA_ROWS] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int r = 0; r < CA_ROWS; ++r) {
          if (tk <= tq[r]) {           // (a key that is not a number stays out of the queries before it)
            o[0][r] += ws[r] * x;
            o[1][r] += ws[r] * y;
          }
        }
      }
#pragma unroll
      for (int r = 0; r < CA_ROWS; ++r) {
        if (t0 + 8 * r >= T) break;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const size_t at = (static_cast<size_t>(b) * T + tq[r]) * C + h * D + d + 32 * u;
          if (d0 + 32 * u >= D) break;
          if (code) cl_put1(reinterpret_cast<uint32_t*>(out), code, at >> 5, o[u][r] * inv[r]);         // (D is a multiple of 32)
          else if (d + 32 * u < D) out[at] = o[u][r] * inv[r];
        }
      }
    }
  }
}

static bool on16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }      // (a null pointer is)

// Rows of a block of the depthwise convolution, by what a launch was measured to take (us): a block alone on its SM 2 and 0.034 a row, each further one on
// it 0.9 and 0.0155 a row, some more for the halo.  Blocks of 128 rows / of the rows chosen here: 80 x 512 of one window 4.7 / 2.5, 330 x 256 of one 6.4 / 2.5, of 4 6.4 /
// 3.4, of 16 8.3 / 6.7, of 32 13.1 / 11.9; 1024 x 256 of 16 15.3 / 15.3 (in blocks of 16 29.3).
static int cl_dw_rows(int range, int channel_blocks, int B, int dil, int sms) {
  static const int kRows[] = {DW_T, 96, 64, 48, 32, 16};
  int best = DW_T;
  double least = 0.0;
  for (int rows : kRows) {
    const long long blocks = static_cast<long long>((range + rows - 1) / rows) * channel_blocks * B, on_sm = (blocks + sms - 1) / sms;
    const int n = min(rows, range);
    const double cost = 2.0 + 0.034 * n + 0.07 * dil + static_cast<double>(on_sm - 1) * (0.9 + 0.0155 * n + 0.03 * dil);
    if (rows == DW_T || cost < least) {
      least = cost;
      best = rows;
    }
  }
  return best;
}

}  // namespace vb

using namespace vb;

extern "C" {

int vb_cl_timeouts(void) {
  return wait_ran_out(WK_CL_CONV);
}

long long vb_cl_pack_bytes(int N, int K) {
  if (N <= 0 || K <= 0 || N % 32 || K % 32) return -1;
  const long long n_pad = (static_cast<long long>(N) + 127) / 128 * 128;
  return n_pad * K * 4 + n_pad * 4;
}

int vb_cl_pack(void* d_dst, const float* d_w, int N, int K, void* stream) {
  VB_CHECK_ARG(d_dst && d_w, "vb_cl_pack: null pointer");
  VB_CHECK_ARG(on16(d_dst) && on16(d_w), "vb_cl_pack: pointers must lie on 16-byte boundaries");
  VB_CHECK_ARG(vb_cl_pack_bytes(N, K) > 0, "vb_cl_pack: N = %d and K = %d must be positive multiples of 32", N, K);
  const int m_tiles = (N + 127) / 128;
  VB_CHECK_ARG(m_tiles <= 65535, "vb_cl_pack: N = %d", N);
  float* inv = reinterpret_cast<float*>(static_cast<uint8_t*>(d_dst) + static_cast<long long>(m_tiles) * 128 * K * 4);
  cl_scale_kernel<<<m_tiles * 128, 256, 0, static_cast<cudaStream_t>(stream)>>>(inv, d_w, N, K);
  VB_CHECK_LAUNCH();
  cl_pack_kernel<<<dim3(K / 32, m_tiles), 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<uint4*>(d_dst), inv, d_w, N, K);
  VB_CHECK_LAUNCH();
  return 0;
}

}  // extern "C"

namespace vb {
// Long sums of narrow layers are one chain of products on few CTAs: 640 rows of 512 x 2048 23.3 us in one part, 15.7 in two, 12.9 in four; 1024 x 3584
// 33.9, 26.0, 23.6.  Shorter sums and wider layers lose (5120 rows of 256 x 1536 20.6 -> 27.9, 640 of 4096 x 2048 38.8 -> 60.6).
// By the layer alone, since the parts round in another order than one sum: what fills the chip without them pays for that.  512 x 2048 / 1024 x 3584 in one
// part and in four (us), by rows: 20 21.4 9.1 / 29.4 11.2; 160 21.7 9.9 / 30.2 13.8; 640 23.1 12.3 / 32.8 22.7; 1280 24.2 27.3 / 40.2 44.9; 2560 27.2
// 41.8 / 55.5 94.4; 10240 71 127 / 213 309.  The line is where 32 streams of ten frames lie, 640 rows: split launches are not persistent, every
// CTA starts, meets its cluster twice and ends for one unit.
static int cl_splits(int blocks, int m_tiles, int kb) {
  return blocks >= 64 && m_tiles <= 8 ? min(4, kb) : 1;
}
// How a launch is divided: columns of a tile, whether a stage of activations serves all taps, boxes for the results.  The fields of p that describe
// the problem are set.  Costs in cycles, per 64 channels and tap: the MMAs' 6 a column; the bytes through L2, some 45 a cycle and SM (32 KB of
// weights, 256 bytes a row of activations, once per stage); the bytes through shared memory, 128 a cycle (the MMAs read 12 times 4 KB of
// weights and 32 bytes a column); a turn of the ring of weights.
template <bool PARTS>
static void cl_plan(ClConvParams& p, int sms) {
  static const int kCols[] = {240, 224, 208, 192, 176, 160, 144, 128, 112, 96, 80, 64, 48, 32, 16};
  const int range = p.n_hi - p.n_lo, blocks = p.Cin / 32;
  p.m_tiles = (p.N + 127) / 128;
  p.group = blocks % 2 ? 1 : 2;
  p.kb = blocks / p.group;
  // Parts of K: by the layer alone, not by the number of positions, so that a result's sum has one order whatever its batch.
  p.splits = cl_splits(p.kb * p.ksize * p.group, p.m_tiles, p.kb);
  const bool two = p.y && (p.y2 || p.yp);
  double best = -1.0;
  for (int per_tap = 0; per_tap < 2; ++per_tap) {
    const long long back = static_cast<long long>(p.ksize - 1) * p.dil;
    if (per_tap == 0 && (p.ksize == 1 || back > 64)) continue;
    const int halo = per_tap ? 0 : static_cast<int>(back), taps = per_tap ? 1 : p.ksize;
    for (int cand : kCols) {
      int nr, nb;
      if (range >= cand) {
        nr = cand; nb = 1;
      } else {
        nr = range;
        nb = max(min((cand + halo) / (nr + halo), p.B), 1);
      }
      const int pitch = nr + halo, cols = (nb * pitch - halo + 15) / 16 * 16, rows = cols + halo;
      if (cols > 240 || rows > CL_ROWS) continue;
      const int t_tiles = (range + nr - 1) / nr;
      const long long units = static_cast<long long>(p.m_tiles) * t_tiles * ((p.B + nb - 1) / nb);
      if (units > 0x7fffffffLL) continue;
      const int pass = PARTS ? 8 : 32 / p.group, rows_pad = (rows + pass - 1) / pass * pass, x_bytes = p.group * rows_pad * 128,
                w_bytes = p.group * CL_W_BLOCK, area = VB_MAX_DYN_SMEM - CL_TAIL;
      for (int staged = 0; staged < 2; ++staged) {
        if (staged && (nb != 1 || p.splits > 1 || (two && p.epi != CE_PLAIN))) continue;
        const int s = p.splits, steps = (p.kb + s - 1) / s * p.ksize, room = area - (staged ? ClRoles<PARTS>::EPI_WARPS * 4096 : 0);
        const bool resident = s == 1 && units > sms && p.m_tiles <= sms && steps <= CL_W_STAGES && steps * w_bytes + 2 * x_bytes <= room;
        int xs = 2, ws = steps;
        if (!resident) {
          if (taps == 1 && 3 * x_bytes + 3 * w_bytes <= room) xs = 3;
          ws = min(CL_W_STAGES, (room - xs * x_bytes) / w_bytes);
          if (ws < 2) continue;
        }
        while (xs < CL_X_STAGES && (xs + 1) * x_bytes + ws * w_bytes <= room) ++xs;
        if (s > 1 && (units * s > 0x7fffffffLL || xs * x_bytes + ws * w_bytes < cols * 512)) continue;
        const long long grid = s > 1 ? units * s : resident ? sms / p.m_tiles * p.m_tiles : min(units, static_cast<long long>(sms));
        const double share = p.group / 2.0, wl = resident ? 0.0 : 32768.0, xl = 256.0 * rows / taps;
        const double stage = fmax(fmax(fmax(6.0 * cols, (wl + xl) / 45), (12 * (4096 + 32.0 * cols) + wl + xl) / 128) * share, resident ? 100.0 : 2400.0 / ws);
        const double epi = 1000 + (staged ? 16.0 : 24.0) * cols * (two ? 1.4 : 1.0) * (p.epi != CE_PLAIN ? 1.2 : 1.0), main = stage * steps + 300;
        double cost;
        if (s > 1) cost = static_cast<double>((units * s + sms - 1) / sms) * (main + epi + 5000);
        else cost = static_cast<double>((units + grid - 1) / grid) * (4 * cols <= 512 ? fmax(main, epi) : main + epi) + epi;
        if (best < 0.0 || cost < best) {
          best = cost;
          p.taps = taps; p.halo = halo; p.nr = nr; p.nb = nb; p.pitch = pitch; p.cols = cols; p.rows_pad = rows_pad; p.resident = resident;
          p.t_tiles = t_tiles; p.units = static_cast<int>(units); p.x_stages = xs; p.w_stages = ws; p.grid = static_cast<int>(grid); p.staged = staged;
        }
      }
    }
  }
  const int rows_pass = 32 / p.group, passes = (p.cols + p.halo + rows_pass - 1) / rows_pass;
  p.passes = passes > 8 ? 16 : passes > 4 || (p.taps == 1 && p.ksize > 1) ? 8 : passes > 2 ? 4 : passes;
  p.m_tiles_inv = p.m_tiles > 1 ? static_cast<uint32_t>(((1ULL << 32) + p.m_tiles - 1) / p.m_tiles) : 0u;
  p.t_tiles_inv = p.t_tiles > 1 ? static_cast<uint32_t>(((1ULL << 32) + p.t_tiles - 1) / p.t_tiles) : 0u;
  p.acc_cols = 2 * p.cols;
  p.acc_bufs = 2 * p.acc_cols <= 512 ? 2 : 1;
}

// boxes of 8 x 32 words of an fp32 (or parts) tensor [B][rows][N]
static bool cl_box_map(CUtensorMap* map, const void* base, int N, int rows, int B, long long bstride) {
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(B)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(N) * 4, static_cast<cuuint64_t>(bstride) * 4};
  cuuint32_t box[3] = {32, CL_EC, 1}, estr[3] = {1, 1, 1};
  return encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool PARTS>
static int cl_launch(ClConvParams p, cudaStream_t stream) {
  cl_plan<PARTS>(p, sm_count());
  VB_CHECK_ARG(p.units > 0, "vb_cl_conv: too many tiles");
  ClMaps maps = {};
  VB_CHECK_ARG((!PARTS && !p.staged) || encode_fn(), "cuTensorMapEncodeTiled not available (no CUDA driver?)");
  if (PARTS) {
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(p.Cin) * 2, static_cast<cuuint64_t>(p.Tx), static_cast<cuuint64_t>(p.B)};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(p.Cin) * 4, static_cast<cuuint64_t>(p.x_bstride) * 4};
    cuuint32_t box[3] = {64, static_cast<cuuint32_t>(p.pitch), static_cast<cuuint32_t>(p.nb)}, estr[3] = {1, 1, 1};
    const CUresult r = encode_fn()(&maps.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<float*>(p.x), dims, strides, box, estr,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    VB_CHECK_ARG(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled(channels last) failed: CUresult %d", static_cast<int>(r));
  }
  if (p.staged) {          // (rows of the results count from n_lo; what a box has past the last one is not written)
    const int rows = p.n_hi - p.n_lo;
    VB_CHECK_ARG((!p.y || cl_box_map(&maps.y, p.y, p.N, rows, p.B, p.y_bstride)) &&
                     cl_box_map(&maps.last, p.y2 ? static_cast<void*>(p.y2) : p.yp ? static_cast<void*>(p.yp) : p.y, p.N, rows, p.B, p.y_bstride) &&
                     (!p.resid || cl_box_map(&maps.r, p.resid, p.N, rows, p.B, p.r_bstride)),
                 "cuTensorMapEncodeTiled(channels last, results) failed");
  }
  const int smem = p.x_stages * p.group * p.rows_pad * 128 + p.w_stages * p.group * CL_W_BLOCK + (p.staged ? ClRoles<PARTS>::EPI_WARPS * 4096 : 0) + CL_TAIL;
  VB_CHECK_CUDA(max_dyn_smem_once(cl_conv_kernel<PARTS>));
  VB_CHECK_CUDA(launch_kernel_cluster(cl_conv_kernel<PARTS>, dim3(p.grid), dim3(ClRoles<PARTS>::THREADS), smem, stream, true, p.splits, p, maps));
  return 0;
}

// rows [n_lo, n_hi) of p's outputs, which point to the first of them
static int cl_run(const ClConvParams& q, cudaStream_t stream) {
  ClConvParams p = q;
  // the epilogue addresses rows with 32-bit offsets from the first one: what is beyond that runs in several launches
  const long long per_entry = max(max(p.y_bstride, p.r_bstride), p.x_bstride);
  const int max_b = per_entry >= (1LL << 30) ? 1 : static_cast<int>(((1LL << 31) - 1) / max(per_entry, 1LL)) - 1;
  const long long max_rows = max((1LL << 30) / p.N / 128 * 128, 128LL);
  auto part = [&](int b0, int b, long long t, long long t1) {
    ClConvParams r = p;
    r.x += b0 * p.x_bstride;
    if (p.x_code) r.x_code += b0 * p.x_bstride >> 5;
    const long long at = b0 * p.y_bstride + (t - p.n_lo) * p.N;
    if (p.y) r.y += at;
    if (p.y2) r.y2 += at;
    if (p.yp) r.yp += at, r.yp_code += at >> 5;
    if (p.resid) r.resid += b0 * p.r_bstride + (t - p.n_lo) * p.N;
    if (p.noise) r.noise += static_cast<long long>(b0) * p.noise_ld;
    r.B = b;
    r.n_lo = static_cast<int>(t);
    r.n_hi = static_cast<int>(t1);
    return cl_run(r, stream);
  };
  if (p.B > max_b) {
    for (int b0 = 0; b0 < p.B; b0 += max_b) {
      const int rc = part(b0, min(max_b, p.B - b0), p.n_lo, p.n_hi);
      if (rc != 0) return rc;
    }
    return 0;
  }
  if (p.n_hi - p.n_lo > max_rows) {
    for (long long t = p.n_lo; t < p.n_hi; t += max_rows) {
      const int rc = part(0, p.B, t, min(t + max_rows, static_cast<long long>(p.n_hi)));
      if (rc != 0) return rc;
    }
    return 0;
  }
  // dense rows without taps are one sequence, whatever entry they belong to
  if (p.ksize == 1 && p.B > 1 && p.n_lo == 0 && p.n_hi == p.Tx && p.x_bstride == static_cast<long long>(p.Tx) * p.Cin &&
      p.y_bstride == static_cast<long long>(p.Tx) * p.N && (!p.resid || p.r_bstride == p.y_bstride) && (!p.noise || p.noise_ld == p.Tx) &&
      static_cast<long long>(p.B) * p.Tx * max(p.N, p.Cin) < (1LL << 30)) {
    p.n_hi = p.Tx = p.B * p.Tx;
    p.B = 1;
  }
  return p.x_code ? cl_launch<true>(p, stream) : cl_launch<false>(p, stream);
}
}  // namespace vb

extern "C" {

int vb_cl_conv_parts(float* d_y, float* d_y2, void* d_yp, void* d_yp_code, const void* d_x, const void* d_x_code, long long x_bstride, int Tx,
                     const void* d_w, const float* d_bias, const float* d_resid, long long r_bstride, const float* d_scale, const float* d_noise,
                     int noise_ld, const float* d_alpha, int epilogue, int act, int B, int Cin, int N, int cmod, int ksize, int dil, int n_lo,
                     int n_hi, long long y_bstride, void* stream) {
  VB_CHECK_ARG((d_y || d_yp) && d_x && d_w, "vb_cl_conv: null pointer");
  VB_CHECK_ARG(!d_y2 || (d_y && !d_yp), "vb_cl_conv: activated values as fp32 or as parts");
  VB_CHECK_ARG(!d_yp == !d_yp_code, "vb_cl_conv: parts come with their codes");
  VB_CHECK_ARG(Cin > 0 && Cin % 32 == 0 && N > 0 && N % 32 == 0, "vb_cl_conv: Cin = %d and N = %d must be positive multiples of 32", Cin, N);
  VB_CHECK_ARG(cmod > 0 && cmod % 32 == 0 && N % cmod == 0, "vb_cl_conv: %d columns do not divide into groups of %d channels", N, cmod);
  VB_CHECK_ARG(ksize >= 1 && dil >= 1 && Tx > 0 && n_lo >= 0, "vb_cl_conv: ksize %d, dilation %d, %d positions, rows from %d", ksize, dil, Tx, n_lo);
  VB_CHECK_ARG(epilogue >= 0 && epilogue <= 3 && act >= 0 && act <= 3, "vb_cl_conv: epilogue %d / activation %d", epilogue, act);
  VB_CHECK_ARG(epilogue == CE_PLAIN || d_resid, "vb_cl_conv: this epilogue needs d_resid");
  VB_CHECK_ARG(epilogue != CE_SCALE_RESID || d_scale, "vb_cl_conv: the scaled residual needs d_scale");
  VB_CHECK_ARG(epilogue != CE_NOISE || d_noise, "vb_cl_conv: the noise epilogue needs d_noise");
  VB_CHECK_ARG(act != CA_SNAKE || d_alpha, "vb_cl_conv: Snake needs d_alpha");
  VB_CHECK_ARG(on16(d_x) && x_bstride % 4 == 0 && on16(d_y) && on16(d_y2) && on16(d_yp) && y_bstride % 4 == 0 && on16(d_resid) &&
                   (!d_resid || r_bstride % 4 == 0),
               "vb_cl_conv: rows must start on 16-byte boundaries");
  VB_CHECK_ARG(on16(d_w) && on16(d_bias) && on16(d_scale) && on16(d_alpha), "vb_cl_conv: weights, bias, scale and alpha must lie on 16-byte boundaries");
  VB_CHECK_ARG((!d_x_code || x_bstride % 32 == 0) && (!d_yp || y_bstride % 32 == 0), "vb_cl_conv: entries of parts must lie multiples of 32 apart");
  VB_CHECK_ARG(N <= (1 << 22), "vb_cl_conv: %d columns", N);
  if (B <= 0 || n_lo >= n_hi) return 0;
  ClConvParams p = {};
  VB_CHECK_ARG(p.wait_flag = wait_flag(WK_CL_CONV), "vb_cl_conv: no mapped host memory");
  const long long first = static_cast<long long>(n_lo) * N, n_pad = (N + 127LL) / 128 * 128;
  p.w = static_cast<const uint8_t*>(d_w);
  p.w_inv = reinterpret_cast<const float*>(p.w + n_pad * Cin * ksize * 4);
  p.x = static_cast<const float*>(d_x); p.x_code = static_cast<const uint8_t*>(d_x_code);
  p.y = d_y ? d_y + first : nullptr; p.y2 = d_y2 ? d_y2 + first : nullptr;
  p.yp = d_yp ? static_cast<uint32_t*>(d_yp) + first : nullptr; p.yp_code = d_yp ? static_cast<uint8_t*>(d_yp_code) + (first >> 5) : nullptr;
  p.bias = d_bias; p.resid = epilogue != CE_PLAIN ? d_resid + first : nullptr; p.scale = d_scale; p.noise = epilogue == CE_NOISE ? d_noise : nullptr;
  p.alpha = d_alpha; p.x_bstride = x_bstride; p.y_bstride = y_bstride; p.r_bstride = p.resid ? r_bstride : 0; p.noise_ld = noise_ld;
  p.cmod = cmod; p.epi = epilogue; p.act = act; p.B = B; p.Tx = Tx; p.Cin = Cin; p.N = N; p.n_lo = n_lo; p.n_hi = n_hi; p.ksize = ksize; p.dil = dil;
  return cl_run(p, static_cast<cudaStream_t>(stream));
}

int vb_cl_conv(float* d_y, float* d_y2, const float* d_x, long long x_bstride, int Tx, const void* d_w, const float* d_bias,
               const float* d_resid, long long r_bstride, const float* d_scale, const float* d_noise, int noise_ld,
               const float* d_alpha, int epilogue, int act, int B, int Cin, int N, int cmod, int ksize, int dil, int n_lo, int n_hi,
               long long y_bstride, void* stream) {
  VB_CHECK_ARG(d_y, "vb_cl_conv: null pointer");
  return vb_cl_conv_parts(d_y, d_y2, nullptr, nullptr, d_x, nullptr, x_bstride, Tx, d_w, d_bias, d_resid, r_bstride, d_scale, d_noise, noise_ld,
                          d_alpha, epilogue, act, B, Cin, N, cmod, ksize, dil, n_lo, n_hi, y_bstride, stream);
}

int vb_cl_dwconv7_parts(float* d_y, void* d_code, const float* d_x, long long x_bstride, const float* d_w, const float* d_bias,
                        const float* d_alpha_in, const float* d_alpha_out, int B, int C, int T, int dilation, int t_lo, int t_hi, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w, "vb_cl_dwconv7: null pointer");
  VB_CHECK_ARG(C % 64 == 0 && dilation >= 1 && dilation <= 64 && x_bstride % 4 == 0, "vb_cl_dwconv7: C = %d (a multiple of 64), dilation %d", C, dilation);
  VB_CHECK_ARG(on16(d_y) && on16(d_x) && on16(d_w) && on16(d_bias) && on16(d_alpha_in) && on16(d_alpha_out), "vb_cl_dwconv7: pointers must lie on 16-byte boundaries");
  VB_CHECK_ARG(0 <= t_lo && t_lo <= t_hi && t_hi <= T, "vb_cl_dwconv7: range [%d, %d) outside [0, %d)", t_lo, t_hi, T);
  if (B <= 0 || t_lo == t_hi) return 0;
  VB_CHECK_CUDA(max_dyn_smem_once(cl_dwconv7_kernel));
  const int tile = cl_dw_rows(t_hi - t_lo, C / 64, B, dilation, sm_count());
  VB_LAUNCH_PDL(cl_dwconv7_kernel, dim3((t_hi - t_lo + tile - 1) / tile, C / 64, B), 256, static_cast<size_t>(tile + 6 * dilation) * 256, stream,
                d_y, static_cast<uint8_t*>(d_code), d_x, x_bstride, d_w, d_bias, d_alpha_in, d_alpha_out, C, T, dilation, t_lo, t_hi, tile);
  return 0;
}
int vb_cl_dwconv7(float* d_y, const float* d_x, long long x_bstride, const float* d_w, const float* d_bias, const float* d_alpha_in,
                  const float* d_alpha_out, int B, int C, int T, int dilation, int t_lo, int t_hi, void* stream) {
  return vb_cl_dwconv7_parts(d_y, nullptr, d_x, x_bstride, d_w, d_bias, d_alpha_in, d_alpha_out, B, C, T, dilation, t_lo, t_hi, stream);
}

int vb_cl_last_conv(float* d_y, const float* d_x, long long x_bstride, const float* d_w, const float* d_bias, int B, int C, int T,
                    int ksize, int left, int t0, int t1, int use_tanh, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w && d_bias, "vb_cl_last_conv: null pointer");
  VB_CHECK_ARG(C % 4 == 0 && C <= 256 && ksize >= 1 && ksize <= 16 && x_bstride % 4 == 0, "vb_cl_last_conv: C = %d, ksize %d", C, ksize);
  VB_CHECK_ARG(on16(d_x), "vb_cl_last_conv: rows must start on 16-byte boundaries");
  VB_CHECK_ARG(0 <= t0 && t0 < t1 && t1 <= T, "vb_cl_last_conv: bad output range [%d, %d) of %d", t0, t1, T);
  if (B <= 0) return 0;
  const dim3 grid((t1 - t0 + LC_T - 1) / LC_T, B);
  if (ksize == 3)
    VB_LAUNCH_PDL(cl_last_conv_kernel<3>, grid, LC_T, 0, stream, d_y, d_x, x_bstride, d_w, d_bias, C, T, ksize, left, t0, t1, use_tanh);
  else if (ksize == 7)
    VB_LAUNCH_PDL(cl_last_conv_kernel<7>, grid, LC_T, 0, stream, d_y, d_x, x_bstride, d_w, d_bias, C, T, ksize, left, t0, t1, use_tanh);
  else
    VB_LAUNCH_PDL(cl_last_conv_kernel<0>, grid, LC_T, 0, stream, d_y, d_x, x_bstride, d_w, d_bias, C, T, ksize, left, t0, t1, use_tanh);
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

int vb_cl_codes_sum_parts(float* d_z0, float* d_z1, void* d_code0, void* d_code1, const int64_t* d_codes, const float* d_emb, int B, int K, int bins,
                          int D, int T, void* stream) {
  VB_CHECK_ARG(d_z0 && d_z1 && d_codes && d_emb, "vb_cl_codes_sum: null pointer");
  VB_CHECK_ARG(K >= 1 && K <= 64, "vb_cl_codes_sum: %d codebooks", K);
  VB_CHECK_ARG(!d_code0 == !d_code1 && (!d_code0 || D % 32 == 0), "vb_cl_codes_sum: parts need both codes and D = %d a multiple of 32", D);
  if (B <= 0 || T <= 0) return 0;
  VB_LAUNCH_PDL(cl_codes_sum_kernel, dim3(T, B), 256, 0, stream, d_z0, d_z1, static_cast<uint8_t*>(d_code0), static_cast<uint8_t*>(d_code1),
                reinterpret_cast<const long long*>(d_codes), d_emb, K, bins, D, T);
  return 0;
}
int vb_cl_codes_sum(float* d_z0, float* d_z1, const int64_t* d_codes, const float* d_emb, int B, int K, int bins, int D, int T, void* stream) {
  return vb_cl_codes_sum_parts(d_z0, d_z1, nullptr, nullptr, d_codes, d_emb, B, K, bins, D, T, stream);
}

int vb_cl_upsample(float* d_y, const float* d_x, const float* d_w, int B, int C, int T, int stride, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w && stride >= 1, "vb_cl_upsample: bad arguments");
  if (B <= 0 || T <= 0) return 0;
  VB_LAUNCH_PDL(cl_upsample_kernel, dim3(T * stride, B), 256, 0, stream, d_y, d_x, d_w, C, T, stride);
  return 0;
}

int vb_cl_layernorm_parts(float* d_y, void* d_code, const float* d_x, const float* d_w, const float* d_b, int rows, int C, float eps, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w && d_b, "vb_cl_layernorm: null pointer");
  VB_CHECK_ARG(on16(d_y) && on16(d_x) && on16(d_w) && on16(d_b), "vb_cl_layernorm: pointers must lie on 16-byte boundaries");
  VB_CHECK_ARG(C > 0 && C % 4 == 0 && C <= 1024, "vb_cl_layernorm: C = %d (a multiple of 4, <= 1024)", C);
  VB_CHECK_ARG(!d_code || C % 32 == 0, "vb_cl_layernorm: parts need C = %d to be a multiple of 32", C);
  if (rows <= 0) return 0;
  VB_LAUNCH_PDL(cl_layernorm_kernel, (rows + 3) / 4, 128, 0, stream, d_y, static_cast<uint8_t*>(d_code), d_x, d_w, d_b, rows, C, eps);
  return 0;
}
int vb_cl_layernorm(float* d_y, const float* d_x, const float* d_w, const float* d_b, int rows, int C, float eps, void* stream) {
  return vb_cl_layernorm_parts(d_y, nullptr, d_x, d_w, d_b, rows, C, eps, stream);
}

int vb_cl_chunk_attention_parts(float* d_out, void* d_code, const float* d_qkv, int B, int C, int H, int T, float max_period, void* stream) {
  VB_CHECK_ARG(d_out && d_qkv, "vb_cl_chunk_attention: null pointer");
  VB_CHECK_ARG(reinterpret_cast<uintptr_t>(d_qkv) % 8 == 0, "vb_cl_chunk_attention: rows must start on 8-byte boundaries");
  VB_CHECK_ARG(H >= 1 && C % H == 0 && (C / H) % 4 == 0 && C / H <= 256 && T >= 1 && T <= 64, "vb_cl_chunk_attention: C %d, H %d, T %d (<= 64)", C, H, T);
  VB_CHECK_ARG(!d_code || (C / H) % 32 == 0, "vb_cl_chunk_attention: parts need heads of a multiple of 32, not %d", C / H);
  if (B <= 0) return 0;
  const size_t smem = (static_cast<size_t>(3) * T * (C / H + 4) + static_cast<size_t>(8) * T * 4 + C / H / 2) * sizeof(float);
  VB_CHECK_ARG(smem <= VB_MAX_DYN_SMEM, "vb_cl_chunk_attention: head size %d too large", C / H);
  VB_CHECK_CUDA(max_dyn_smem_once(cl_chunk_attention_kernel));
  VB_LAUNCH_PDL(cl_chunk_attention_kernel, dim3(H, B), 256, smem, stream, d_out, static_cast<uint8_t*>(d_code), d_qkv, C, H, T, max_period);
  return 0;
}
int vb_cl_chunk_attention(float* d_out, const float* d_qkv, int B, int C, int H, int T, float max_period, void* stream) {
  return vb_cl_chunk_attention_parts(d_out, nullptr, d_qkv, B, C, H, T, max_period, stream);
}

}  // extern "C"
