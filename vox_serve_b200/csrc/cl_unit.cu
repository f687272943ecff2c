// Residual units of the vocoders over channels-last activations [B][T][C] (fp32), a unit in one launch:
//   y = x + W s2(dw7(s1(x)) + b1) + b2       (vb_cl_dw_unit: SNAC; s1, s2 Snakes, dw7 a depthwise convolution of 7 taps with dilation)
// and the end of Mimi's decoder (vb_cl_res_tail, further down).
// A block owns `nr` positions of one channel tile.  What goes into the product never leaves the block: a warp takes 64 channels, two a lane, and walks a
// run of positions `dil` apart, so a row of x is loaded and put through its Snake once for the seven sums that it is part of, all in registers; the sums'
// Snakes are written as the two fp16 parts that the tensor cores multiply (cl_common.cuh) into the operand in shared memory, and the products of 64
// channels are issued as soon as all their runs are done.  The arithmetic -- order of the sums, parts, what is multiplied in fp32 because parts
// cannot hold it -- is that of cl_dwconv7 and cl_conv one after the other, bit for bit.
#include "../../include/vb_api.h"
#define VB_PDL_FAMILY 32
#include "cl_common.cuh"

namespace vb {
constexpr int CU_W_STAGES = 4, CU_MAX_CHUNKS = 16;      // (a block of 32 channels has a bit in a row's word)

struct CuDwParams {
  const float* x;            // [b * x_bstride + t * C + c]
  const float* dw_w;         // [7][C]
  const float* dw_b;         // [C]
  const float* alpha_in;     // [2][C] alpha, 1 / (alpha + 1e-9)
  const float* alpha_mid;
  const uint8_t* w;          // packed (vb_cl_pack)
  const float* w_inv;
  const float* bias;         // [C]
  const float* alpha_out;    // Snake of the result, or null
  float* y;                  // fp32 result, or
  uint32_t* yp;              // the result as parts
  uint8_t* yp_code;
  long long x_bstride, y_bstride;
  int C, T, dil, t_lo, t_hi;
  int nr, cols;              // positions of a block; columns of its products
  int classes, segs, len;    // runs: position (class + dil (seg len + j)) of a block, j < len
  int m_tiles, chunks, w_stages, tmem_cols;
  uint32_t runs_inv, segs_inv, dil_inv, m_tiles_inv;      // for cu_div
  unsigned char* wait_flag;
};
// a / b for 0 <= a < 2^31 with inv = ceil(2^32 / b), 0 for b == 1: the quotient or one more, as a product
__device__ __forceinline__ int cu_div(int a, int b, uint32_t inv) {
  if (inv == 0u) return a;
  const int q = static_cast<int>(__umulhi(static_cast<uint32_t>(a), inv));
  return q * static_cast<long long>(b) > a ? q - 1 : q;
}

// What a warp of an epilogue needs of its unit: a lane is a channel
struct CuOut {
  float bias, alpha, ialpha;
  const float* resid;        // this channel at the block's first position
  float* y;
  uint32_t* yp;              // the warp's block of 32 channels there
  uint8_t* code;
  int N;
};
__device__ __forceinline__ void cu_resid(const CuOut& o, int c0, int inside, float (&rs)[CL_EC]) {
  const float* r = o.resid + static_cast<long long>(c0) * o.N;
  if (c0 + CL_EC <= inside) {
#pragma unroll
    for (int c = 0; c < CL_EC; ++c) rs[c] = __ldcg(r + c * o.N);
    return;
  }
#pragma unroll
  for (int c = 0; c < CL_EC; ++c) rs[c] = c0 + c < inside ? __ldcg(r + c * o.N) : 0.f;
}
// Columns [c_first, inside) in steps of c_step, eight at a time: accumulators + bias + residual, activation, fp32 or parts.  `rs`: the first residuals.
template <int ACT>
__device__ __forceinline__ void cu_chunks(const CuOut& o, uint32_t taddr, int cols, int inside, int c_first, int c_step, float inv, float (&rs)[CL_EC]) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int c0 = c_first; c0 < inside; c0 += c_step) {
    const uint32_t rows = c0 + CL_EC <= inside ? 0xffu : (1u << (inside - c0)) - 1u;
    F2 v[CL_EC / 2];
    cl_load_acc(taddr + c0, cols, inv, v);
#pragma unroll
    for (int c = 0; c < CL_EC / 2; ++c) v[c] = f2_add(f2_add(v[c], f2(o.bias)), f2(rs[2 * c], rs[2 * c + 1]));
    if (c0 + c_step < inside) cu_resid(o, c0 + c_step, inside, rs);
    cl_act<ACT>(o.alpha, o.ialpha, v);
    const long long at = static_cast<long long>(c0) * o.N;
    if (!o.yp) {
      float* y = o.y + at;
      if (rows == 0xffu) {
#pragma unroll
        for (int c = 0; c < CL_EC; ++c) {
          const float2 x = f2_get(v[c >> 1]);
          y[c * o.N] = c & 1 ? x.y : x.x;
        }
        continue;
      }
#pragma unroll
      for (int c = 0; c < CL_EC; ++c) {
        const float2 x = f2_get(v[c >> 1]);
        if (rows >> c & 1u) y[c * o.N] = c & 1 ? x.y : x.x;
      }
      continue;
    }
    uint32_t* yp = o.yp + at;
    uint32_t code = CB_NORMAL;
    if (cl_ordinary(v, rows)) {
      uint32_t* q = yp + (lane & 1 ? 16 : 0) + (lane >> 1);
#pragma unroll
      for (int c = 0; c < CL_EC / 2; ++c) {
        uint32_t hi, lo, w0, w1;
        cl_parts(v[c], CL_X_SCALE, hi, lo);
        cl_exchange(hi, lo, w0, w1);
        if (rows >> (2 * c) & 1u) q[2 * c * o.N] = w0;
        if (rows >> (2 * c) & 2u) q[(2 * c + 1) * o.N] = w1;
      }
    } else {
#pragma unroll
      for (int c = 0; c < CL_EC; ++c) {
        const float2 x = f2_get(v[c >> 1]);
        int word;
        uint32_t bits;
        const uint32_t row = cl_odd_row(c & 1 ? x.y : x.x, word, bits);
        if (rows >> c & 1u) yp[c * o.N + word] = bits;
        if ((lane & 7) == c) code = row;
      }
    }
    if (lane < CL_EC && (rows >> lane & 1u)) o.code[(at + static_cast<long long>(lane) * o.N) >> 5] = static_cast<uint8_t>(code);
  }
}

// The inputs of a product as they lie in shared memory: [block of 32 channels][row][128 bytes, swizzled], parts or (a bit in the row's word) fp32
struct CuOperand {
  uint32_t at;               // first row of the first block
  int blk_bytes, blocks;
  const uint32_t* raw;
};
// The products of four columns that `mask` names again in fp32, for this warp's 32 channels, into the accumulators (plain scale; the columns that are
// not named in the plain scale as well): cl_exact_chunk of cl_conv.cu for one tap with the inputs in shared memory, in the same order.
__device__ __noinline__ void cu_exact_chunk(const CuOperand& x, const uint8_t* w, float w_scale, int lane_row, int c0, uint32_t mask, uint32_t t_hi, uint32_t t_lo,
                                            float inv) {
  const int lane = threadIdx.x & 31, sw = lane_row & 7;
  float acc[4] = {};
#pragma unroll 1
  for (int blk = 0; blk < x.blocks && mask; ++blk) {
    float v[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int r = c0 + c;
      v[c] = 0.f;
      if (!(mask >> c & 1u)) continue;
      const uint32_t row = x.at + blk * x.blk_bytes + r * 128;
      if (x.raw[r] >> blk & 1u) {
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v[c]) : "r"(row + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4));
      } else {
        const uint32_t a = row + (((lane >> 3) ^ (r & 7)) << 4) + (lane & 7) * 2;
        uint16_t hi, lo;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(hi) : "r"(a));
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(lo) : "r"(a ^ 64u));
        v[c] = fmaf(__half2float(__ushort_as_half(lo)), 1.f / CL_LO_SCALE, __half2float(__ushort_as_half(hi))) * (1.f / CL_X_SCALE);
      }
    }
    const uint8_t* wb = w + static_cast<size_t>(blk) * CL_W_BLOCK + lane_row * 128;
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      const uint4 hi = __ldg(reinterpret_cast<const uint4*>(wb + ((q ^ sw) << 4))), lo = __ldg(reinterpret_cast<const uint4*>(wb + (((q + 4) ^ sw) << 4)));
      const uint32_t h[4] = {hi.x, hi.y, hi.z, hi.w}, l[4] = {lo.x, lo.y, lo.z, lo.w};
      float f[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 fh = unpack_f16(h[i]), fl = unpack_f16(l[i]);
        f[2 * i] = fmaf(fl.x, 1.f / CL_LO_SCALE, fh.x) * w_scale;
        f[2 * i + 1] = fmaf(fl.y, 1.f / CL_LO_SCALE, fh.y) * w_scale;
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (!(mask >> c & 1u)) continue;
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[c] = fmaf(__shfl_sync(0xffffffffu, v[c], 8 * q + k), f[k], acc[c]);
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
// ... all columns of a warp that are made of a row kept in fp32
__device__ __noinline__ void cu_exact(const CuOperand& x, const uint8_t* w, const float* w_inv, int lane_row, int inside, int c_first, int c_step, uint32_t taddr,
                                      int cols, float inv) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int c0 = c_first; c0 < inside; c0 += c_step) {
    const uint32_t mask = __ballot_sync(0xffffffffu, lane < CL_EC && c0 + lane < inside && x.raw[c0 + lane]);
#pragma unroll 1
    for (int c = 0; c < CL_EC; c += 4)
      cu_exact_chunk(x, w, w_inv[lane_row] * CL_X_SCALE, lane_row, c0 + c, mask >> c & 15u, taddr + c0 + c, taddr + cols + c0 + c, inv);
  }
}

// sin(y)^2 of arguments past what cl_sin_sq reduces (each value by itself: its result does not depend on the others)
__device__ __noinline__ F2 cu_sin_sq_large(F2 y, F2 s) {
  const float2 p = f2_get(y), q = f2_get(s);
  const float sx = sinf(p.x), sy = sinf(p.y);
  return f2(fabsf(p.x) <= CL_SIN_MAX ? q.x : sx * sx, fabsf(p.y) <= CL_SIN_MAX ? q.y : sy * sy);
}
// The constants of cl_sin_sq, held in registers: the compiler moves them into a pair wherever one is used otherwise
struct CuSine {
  F2 inv_pi, magic, unmagic, pi_hi, pi_lo, c3, c2, c1, c0;
};
__device__ __forceinline__ F2 cu_pin(float x) {
  F2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r.v) : "f"(x));
  return r;
}
__device__ __forceinline__ CuSine cu_sine() {
  return CuSine{cu_pin(0.318309886f), cu_pin(12582912.f), cu_pin(-12582912.f), cu_pin(-3.14159274101f), cu_pin(8.742278012619e-08f), cu_pin(2.605780761e-06f),
                cu_pin(-1.980960296e-04f), cu_pin(8.333066247e-03f), cu_pin(-1.666665955e-01f)};
}
// v + inv sin(a v)^2 of two channels at N positions
template <int N>
__device__ __forceinline__ void cu_snake(F2 (&v)[N], F2 a, F2 inv, const CuSine& K) {
  F2 y[N], s[N];
  float m = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    y[i] = f2_mul(a, v[i]);
    const F2 k = f2_add(f2_fma(y[i], K.inv_pi, K.magic), K.unmagic), r = f2_fma(k, K.pi_lo, f2_fma(k, K.pi_hi, y[i])), u = f2_mul(r, r);
    F2 q = f2_fma(u, K.c3, K.c2);
    q = f2_fma(u, q, K.c1);
    q = f2_fma(u, q, K.c0);
    q = f2_fma(f2_mul(r, u), q, r);
    s[i] = f2_mul(q, q);
    const float2 p = f2_get(y[i]);
    m = max3_abs(m, p.x, p.y);
  }
  if (!(m <= CL_SIN_MAX)) {
#pragma unroll
    for (int i = 0; i < N; ++i) s[i] = cu_sin_sq_large(y[i], s[i]);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) v[i] = f2_fma(inv, s[i], v[i]);
}
struct CuTaps {              // of a lane's two channels
  F2 w[7], b, ai, ii, ao, io;
};
__device__ __forceinline__ CuTaps cu_taps(const CuDwParams& p, int c) {
  auto ld = [&](const float* q) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(q + c));
    return f2(v.x, v.y);
  };
  CuTaps t;
#pragma unroll
  for (int i = 0; i < 7; ++i) t.w[i] = ld(p.dw_w + i * p.C);
  t.b = ld(p.dw_b);
  t.ai = ld(p.alpha_in);
  t.ii = ld(p.alpha_in + p.C);
  t.ao = ld(p.alpha_mid);
  t.io = ld(p.alpha_mid + p.C);
  return t;
}
// A run once more for the blocks of rows that parts cannot hold: those stay fp32, a bit in the row's word.  (Two rows at a time: with the kernel's four, or its constants in
// registers, the kernel spilled around the call and SNAC took 0.5 % longer.)  32 x 6000 positions of 64 channels, dilation 9, with one such value in every tile / nothing but
// such values / zeros: 192 / 848 / 62 us, in two launches 211 / 840 / 87; with the seven inputs of every row anew, and zeros taken for such values, 394 / 1554 / 261.
__device__ __noinline__ void cu_odd_run(const CuDwParams& p, const float* x, int t_first, int n, int r0, int c, int block, uint32_t dst, uint32_t* raw, uint32_t* any) {
  const int lane = threadIdx.x & 31, in = (lane & 15) * 2;
  const CuTaps tp = cu_taps(p, c);
  auto snake = [&](F2 (&v)[2], F2 a, F2 inv) { cl_snake4(v[0], v[1], a, a, inv, inv); };          // (the bits of cu_snake, without its constants in registers)
  F2 h[8], got[2];              // (the walk of the kernel below)
  __syncwarp();                 // (every lane's parts of these rows are written)
  int t = t_first - 3 * p.dil;
  auto load2 = [&]() {
#pragma unroll
    for (int i = 0; i < 2; ++i, t += p.dil) {
      float2 v = make_float2(0.f, 0.f);
      if (t >= 0 && t < p.T) v = __ldcg(reinterpret_cast<const float2*>(x + static_cast<long long>(t) * p.C));
      got[i] = f2(v.x, v.y);
    }
  };
#pragma unroll
  for (int i = 0; i < 6; ++i) h[i] = f2(0.f);
  load2();
#pragma unroll 1
  for (int j = -6; j < n; j += 2) {
    snake(got, tp.ai, tp.ii);
#pragma unroll
    for (int i = 0; i < 2; ++i) h[6 + i] = got[i];
    if (j + 2 < n) load2();
    if (j >= 0) {
      F2 o[2];
      float m[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) o[i] = tp.b;
#pragma unroll
      for (int q = 0; q < 7; ++q)
#pragma unroll
        for (int i = 0; i < 2; ++i) o[i] = f2_fma(tp.w[q], h[i + q], o[i]);
      snake(o, tp.ao, tp.io);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 v = f2_get(o[i]);
        m[i] = max3_abs(v.x, v.y, v.y);
      }
#pragma unroll
      for (int q = 1; q < 16; q <<= 1)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float other = __shfl_xor_sync(0xffffffffu, m[i], q);
          m[i] = max3_abs(m[i], other, other);
        }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (j + i >= n || cl_code(m[i]) != CB_RAW) continue;          // (the parts are there)
        const float2 v = f2_get(o[i]);
        const int r = r0 + (j + i) * p.dil;
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(dst + r * 128 + (((in >> 2) ^ (r & 7)) << 4) + (in & 2) * 4), "f"(v.x), "f"(v.y) : "memory");
        if (in == 0) {
          atomicOr(raw + r, 1u << block);
          *any = 1u;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) h[i] = h[i + 2];
  }
}

template <int P>             // warps that make the operand; one more copies weights and issues the products
__global__ void __launch_bounds__(32 * (P + 1), P == 9 ? 2 : 1) cl_dw_unit_kernel(const __grid_constant__ CuDwParams p) {
  constexpr int EPI_WARPS = P / 4 * 4;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int C = p.C, cols = p.cols, blk_bytes = cols * 128;
  uint8_t* w_smem = smem + 2 * p.chunks * blk_bytes;
  uint64_t* op_full = reinterpret_cast<uint64_t*>(w_smem + p.w_stages * 2 * CL_W_BLOCK);          // 64 channels of all positions are there
  uint64_t* w_full = op_full + CU_MAX_CHUNKS;
  uint64_t* w_empty = w_full + CU_W_STAGES;
  uint64_t* acc_full = w_empty + CU_W_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  uint32_t* any = tmem_slot + 1;
  const uint32_t gate = smem_u32(tmem_slot + 2);
  uint32_t* raw = tmem_slot + 4;                                             // [cols] a bit for every block of a row that is kept in fp32
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tt = cu_div(blockIdx.x, p.m_tiles, p.m_tiles_inv), m0 = (blockIdx.x - tt * p.m_tiles) * 128, t0 = p.t_lo + tt * p.nr, b = blockIdx.y;
  const int inside = min(p.nr, p.t_hi - t0), runs = p.classes * p.segs;
  const uint8_t* w = p.w + static_cast<size_t>(m0 >> 7) * (2 * p.chunks) * CL_W_BLOCK;
  BoundedWait bw{p.wait_flag, gate};

  if (warp == P) {
    if (lane == 0) {
      tmem_slot[2] = 0u;
      *any = 0u;
      for (int i = 0; i < p.chunks; ++i) mbar_init(&op_full[i], runs);
      for (int i = 0; i < CU_W_STAGES; ++i) {
        mbar_init(&w_full[i], 1);
        mbar_init(&w_empty[i], 1);
      }
      mbar_init(acc_full, 1);
      fence_barrier_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, p.tmem_cols);
    tmem_relinquish();
  } else {
    for (int i = threadIdx.x; i < cols; i += 32 * P) raw[i] = 0u;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == P) {
    // ================= weights and products =================
    if (lane == 0) {
      for (int i = 0; i < min(p.w_stages, p.chunks); ++i) {          // (weights do not depend on the kernels in front)
        mbar_arrive_expect_tx(&w_full[i], 2 * CL_W_BLOCK);
        cl_bulk(smem_u32(w_smem) + i * 2 * CL_W_BLOCK, w + static_cast<size_t>(i) * 2 * CL_W_BLOCK, 2 * CL_W_BLOCK, smem_u32(&w_full[i]));
      }
      pdl_wait();
      wait_gate_open(gate);
      pdl_trigger();
    }
    __syncwarp();
    const uint64_t w_desc0 = umma_desc_sw128_kmajor(smem_u32(w_smem)), x_desc0 = umma_desc_sw128_kmajor(smem_u32(smem));
    const uint32_t idesc = umma_idesc(128, cols, 0u);
    for (int k = 0; k < p.chunks && !bw.dead; ++k) {
      const int ws = k % p.w_stages;
      bw.wait(&op_full[k], 0u);
      bw.wait(&w_full[ws], (k / p.w_stages) & 1);
      if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
      tc_fence_after();
      if (elect_one()) {
        uint64_t w_hi = w_desc0 + static_cast<uint64_t>(ws) * (2 * CL_W_BLOCK >> 4), x_hi = x_desc0 + static_cast<uint64_t>(2 * k) * (blk_bytes >> 4);
        // (a loop: unrolled by nvcc 12.9, rows of the result came out of the wrong tile of the weights)
#pragma unroll 1
        for (int g = 0; g < 2; ++g) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {            // (the low parts lie 64 bytes behind the high ones)
            const uint32_t go = (k | g | i) ? 1u : 0u;
            umma_bf16(tmem_base, w_hi + 2 * i, x_hi + 2 * i, idesc, go);
            umma_bf16(tmem_base + cols, w_hi + 2 * i, x_hi + 4 + 2 * i, idesc, go);
            umma_bf16(tmem_base + cols, w_hi + 4 + 2 * i, x_hi + 2 * i, idesc, 1u);
          }
          w_hi += CL_W_BLOCK >> 4;
          x_hi += blk_bytes >> 4;
        }
        umma_commit(&w_empty[ws]);
        if (k + 1 == p.chunks) umma_commit(acc_full);
      }
      __syncwarp();
      if (k >= 1 && k - 1 + p.w_stages < p.chunks) {          // the stage in front is free when its products are done
        const int was = (k - 1) % p.w_stages, next = k - 1 + p.w_stages;
        bw.wait(&w_empty[was], ((k - 1) / p.w_stages) & 1);
        if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
        if (elect_one()) {
          mbar_arrive_expect_tx(&w_full[was], 2 * CL_W_BLOCK);
          cl_bulk(smem_u32(w_smem) + was * 2 * CL_W_BLOCK, w + static_cast<size_t>(next) * 2 * CL_W_BLOCK, 2 * CL_W_BLOCK, smem_u32(&w_full[was]));
        }
        __syncwarp();
      }
    }
    if (bw.dead && lane == 0) {            // let the copies in flight land before the block may leave
      const unsigned long long from = gtimer();
      while (gtimer() - from < 2000000ull) __nanosleep(1000);
    }
    __syncwarp();
  } else {
    // ================= the operand =================
    const int items = p.chunks * runs;
    const float* xb = p.x + b * p.x_bstride + lane * 2;
    const long long step = static_cast<long long>(p.dil) * C;
    const uint32_t at_step = p.dil * 128;
    bool first = true;
    const CuSine K = cu_sine();
#pragma unroll 1
    for (int item = warp; item < items; item += P) {
      const int k = cu_div(item, runs, p.runs_inv), run = item - k * runs, cls = cu_div(run, p.segs, p.segs_inv), seg = run - cls * p.segs;
      const int c = k * 64 + lane * 2, r0 = cls + seg * p.len * p.dil;                      // first position of the run
      const int n = r0 < inside ? min(p.len, cu_div(inside - 1 - r0, p.dil, p.dil_inv) + 1) : 0;
      const CuTaps tp = cu_taps(p, c);
      if (first) {
        pdl_wait();
        first = false;
      }
      const uint32_t dst = smem_u32(smem) + (2 * k + (lane >> 4)) * blk_bytes;
      const int in = (lane & 15) * 2;
      const uint32_t chunk = (in >> 3 << 4) + (in & 6) * 2;
      const float* x = xb + k * 64;
      float top = 0.f, low = CL_X_TOP;
      F2 h[10], got[4];              // six inputs through their Snake from the step before and four new ones; the next four
      int t_next = t0 + r0 - 3 * p.dil;
      const float* from = x + static_cast<long long>(t_next) * C;
      const bool within = t_next >= 0 && t_next + (n + 9) * p.dil < p.T;          // (of every row that may be asked for)
      auto load4 = [&]() {
        if (within) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 v = __ldcg(reinterpret_cast<const float2*>(from));
            got[i] = f2(v.x, v.y);
            from += step;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float2 v = make_float2(0.f, 0.f);
            if (t_next >= 0 && t_next < p.T) v = __ldcg(reinterpret_cast<const float2*>(from));
            got[i] = f2(v.x, v.y);
            from += step;
            t_next += p.dil;
          }
        }
      };
#pragma unroll
      for (int i = 0; i < 6; ++i) h[i] = f2(0.f);
      if (n > 0) load4();
      uint32_t at = dst + (r0 - 6 * p.dil) * 128;            // the row of sum j
#pragma unroll 1
      for (int j = -6; n > 0 && j < n; j += 4) {           // inputs j + 6 .. j + 9, sums j .. j + 3
        cu_snake(got, tp.ai, tp.ii, K);           // (the activation of zero is zero)
#pragma unroll
        for (int i = 0; i < 4; ++i) h[6 + i] = got[i];
        if (j + 4 < n) load4();
        if (j > -4) {
          F2 o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = tp.b;
#pragma unroll
          for (int q = 0; q < 7; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = f2_fma(tp.w[q], h[i + q], o[i]);
          cu_snake(o, tp.ao, tp.io, K);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (j + i >= 0 && j + i < n) {
              const float2 v = f2_get(o[i]);
              top = max3_abs(top, v.x, v.y);
              low = min3_abs(low, v.x, v.y);
              uint32_t hi, lo;
              cl_parts(o[i], CL_X_SCALE, hi, lo);
              const uint32_t q = at + i * at_step, a = q + (chunk ^ (q >> 3 & 0x70u));          // (the row's number modulo 8, swizzled)
              asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(hi) : "memory");
              asm volatile("st.shared.b32 [%0], %1;" ::"r"(a ^ 64u), "r"(lo) : "memory");
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) h[i] = h[i + 4];
        at += 4 * at_step;
      }
      // No value out of range, and in either block a lane none of whose values is tiny: nearly always
      const uint32_t fine = __ballot_sync(0xffffffffu, top < CL_X_TOP), large = __ballot_sync(0xffffffffu, low >= CL_X_LOW);
      if (n > 0 && !(fine == 0xffffffffu && (large & 0xffffu) && large >> 16)) {
        const uint32_t some = __ballot_sync(0xffffffffu, top != 0.f);          // (a block of zeros is its parts)
        if (!(fine == 0xffffffffu && ((large & 0xffffu) || !(some & 0xffffu)) && (large >> 16 || !(some >> 16))))
          cu_odd_run(p, x, t0 + r0, n, r0, c, 2 * k + (lane >> 4), dst, raw, any);
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&op_full[k]);
    }
    if (first) pdl_wait();
  }
  // ================= epilogue =================
  if (warp < EPI_WARPS) {
    const int quarter = warp & 3, lane_row = quarter * 32 + lane, width = min(128, C - m0), copies = cl_copies(width);
    const int row = copies == 1 ? lane_row : lane_row & (width - 1), n = m0 + row;
    const int turns = EPI_WARPS / 4 * copies, c_step = turns * CL_EC;
    const int c_first = ((warp >> 2) * copies + (copies == 4 ? quarter : copies == 2 ? quarter >> 1 : 0)) * CL_EC;
    const bool some = row < width && c_first < inside;
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const long long at = static_cast<long long>(t0) * C;
    float inv = 0.f, rs[CL_EC];
    CuOut o{};
    if (some) {
      o.N = C;
      o.resid = p.x + b * p.x_bstride + at + n;
      cu_resid(o, c_first, inside, rs);          // asked for before the accumulator is waited for
      inv = __ldg(p.w_inv + m0 + lane_row);
      o.bias = __ldg(p.bias + n);
      if (p.alpha_out) o.alpha = __ldg(p.alpha_out + n), o.ialpha = __ldg(p.alpha_out + C + n);
    }
    for (int k = 0; k < p.chunks; ++k) bw.wait(&op_full[k], 0u);          // (what `any` and the rows' words say is seen with them)
    bw.wait(acc_full, 0u);
    const bool alive = __all_sync(0xffffffffu, !bw.dead);
    tc_fence_after();
    if (alive && some) {
      if (*any) {
        const CuOperand x{smem_u32(smem), blk_bytes, 2 * p.chunks, raw};
        cu_exact(x, w, p.w_inv + m0, lane_row, inside, c_first, c_step, taddr, cols, inv);
        inv = 1.f;
      }
      const long long to = b * p.y_bstride + at;
      if (p.y) o.y = p.y + to + n;
      if (p.yp) o.yp = p.yp + to + (n & ~31), o.code = p.yp_code + ((to + (n & ~31)) >> 5);
      if (p.alpha_out) cu_chunks<CA_SNAKE>(o, taddr, cols, inside, c_first, c_step, inv, rs);
      else cu_chunks<CA_NONE>(o, taddr, cols, inside, c_first, c_step, inv, rs);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == P) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

static bool on16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }      // (a null pointer is)

// shared memory of a block
static int cu_dw_smem(int C, int cols, int w_stages) {
  return 1024 + C / 32 * cols * 128 + w_stages * 2 * CL_W_BLOCK + (CU_MAX_CHUNKS + 2 * CU_W_STAGES + 1) * 8 + 16 + cols * 4;
}
// How a launch is divided: positions of a block, and whether two blocks of nine producing warps share an SM or one of eighteen has it.  Positions are
// multiples of nine: runs of the dilations 1, 3 and 9 then come out alike, one for each of the nine warps.
struct CuDwPlan {
  int nr, cols, classes, segs, len, warps, w_stages, smem;
};
static CuDwPlan cu_dw_plan(int C, int dil, long long range, long long B, int sms) {
  static const int kRows[] = {126, 108, 90, 72, 63, 54, 45, 36, 27, 18, 9};
  const int chunks = C / 64, m_tiles = (C + 127) / 128;
  CuDwPlan best{};
  double least = 0.0;
  for (int nr : kRows) {
    const int cols = (nr + 15) / 16 * 16;
    const long long units = m_tiles * ((range + nr - 1) / nr) * B;
    for (int warps = 9; warps <= 18; warps += 9) {
      const int limit = warps == 9 ? 113 * 1024 : VB_MAX_DYN_SMEM;
      int ws = min(chunks, CU_W_STAGES);
      while (ws > min(chunks, 2) && cu_dw_smem(C, cols, ws) > limit) --ws;
      if (cu_dw_smem(C, cols, ws) > limit) continue;
      const int classes = min(dil, nr), want = chunks == 1 ? warps : 9, segs = max(1, (want + classes / 2) / classes);
      const int len = ((nr + dil - 1) / dil + segs - 1) / segs, items = chunks * classes * segs, rounds = (items + warps - 1) / warps;
      // instructions of a run (a row's Snake with its load 24, a sum with its own and its parts 40), of the epilogue; cycles where `warps` or twice
      // as many share an SM
      const double run = (len + 6) * 24.0 + len * 40.0 + 60, epi = cols / 8.0 * min(4, C / 32) * 80;
      const long long slots = static_cast<long long>(sms) * (warps == 9 ? 2 : 1);
      const double waves = static_cast<double>((units + slots - 1) / slots), on_sm = warps == 9 && units > sms ? 18.0 : warps;
      const double cost = waves * (3500 + rounds * run * fmax(2.5, on_sm / 2.2) + epi / (warps == 9 ? 1.2 : 2.2) * (on_sm > warps ? 1.0 : 0.6));
      if (best.nr == 0 || cost < least) {
        least = cost;
        best = CuDwPlan{nr, cols, classes, segs, len, warps, ws, cu_dw_smem(C, cols, ws)};
      }
    }
  }
  return best;
}

// ------------------------------------------------------------------------------------------
// the end of Mimi's decoder: last residual unit, ELU and the convolution to one channel
// ------------------------------------------------------------------------------------------
// out[t] = bl + sum_j wl_j . e(y[t - 2 + j]),  y = x + W3 e(h) + b3,  h[t] = b1 + sum_j W1_j e(x[t - 2 + j]),  e = ELU, 64 channels, 32 hidden ones
//
// Here positions are the lanes of the accumulators and channels their columns: a thread has a position's channels side by side, so parts need no exchange
// between lanes and the last sum over the channels is the thread's own.  A group of eight warps takes 128 positions -- two of them only for the unit's
// first convolution, two more for the last one -- through five steps: the tile of x by TMA, its ELU as parts in its place (a thread keeps its 32 values for the
// residual), three taps of products, ELU of the hidden channels as parts, products, ELU and the taps of the last convolution.  The next tile comes
// while the second half runs.  Nothing but x is read and nothing but the samples is written; two groups run into the gaps of one another.
// What bounds it: instructions, some 12,000 of a warp's a tile (the ELUs more than half) at 45 % of the issue slots, two groups of one SM waiting for products
// between their steps.  32 x 19,200 positions: 117 us (125 with x in local memory, where a call for it had put it), before as three launches 88 + 113 + 60, and the convolution in front writes its result once
// (111 -> 70 us).  With x kept in shared memory and fetched between tiles 143.
// What parts cannot hold is multiplied in fp32 by warps, a lane a channel.  32 x 19,200 positions with one such value in all 128 us, one in every tile 455, one every 16
// positions 556, 10 ms of silence an entry 248, nothing but silence 1340, nothing but loud values 1820; in three launches 283, 884, 1600, 350, 2340 and 3070.  (With a lane
// for all 6144 products of its position 814, 12800, 13000, 1220, 8950 and 10100.)
constexpr int CT_C = 64, CT_H = 32, CT_TAPS = 3, CT_ROWS = 128, CT_OUT = CT_ROWS - 2 * (CT_TAPS - 1), CT_PAD = 8;
constexpr int CT_GROUPS = 2, CT_GROUP_THREADS = 256, CT_THREADS = CT_GROUPS * CT_GROUP_THREADS;
constexpr int CT_X = CT_ROWS * 256, CT_OP1 = 2 * (CT_PAD + CT_ROWS) * 128, CT_OP2 = CT_ROWS * 128, CT_GROUP_BYTES = CT_OP1 + CT_OP2;
constexpr int CT_W1 = CT_TAPS * 2 * 2 * CT_H * 128, CT_W3 = 2 * CT_C * 128;          // every row twice, the second time with its low parts in front
struct CtTables {            // behind the tiles in shared memory
  float inv1[CT_H], b1[CT_H], inv3[CT_C], b3[CT_C], wl[CT_TAPS][CT_C];
  float sums[CT_GROUPS][2][CT_TAPS][CT_ROWS];
  uint8_t raw1[CT_GROUPS][2][CT_PAD + CT_ROWS], raw2[CT_GROUPS][CT_ROWS], odd[CT_GROUPS][2][CT_ROWS];
  uint64_t x_full[CT_GROUPS], m1[CT_GROUPS], m3[CT_GROUPS];
  uint32_t tmem, gate;
};
constexpr int CT_SMEM = 1024 + CT_GROUPS * CT_GROUP_BYTES + CT_W1 + CT_W3 + static_cast<int>(sizeof(CtTables)) + 16;
static_assert(CT_SMEM <= VB_MAX_DYN_SMEM, "tail of Mimi: shared memory");
struct CtParams {
  const uint8_t *w1, *w3;    // packed (vb_cl_pack)
  const float *inv1, *b1, *inv3, *b3, *wl, *bl;
  float* y;                  // [B][T]
  int T, t_tiles, tiles;
  uint32_t t_tiles_inv;
  unsigned char* wait_flag;
};
__device__ __forceinline__ float4 ct_lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void ct_sts4(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// sixteen channels of a row as parts: 16-byte chunks `at` and `at` + 1 of the high ones, four further on the low ones
__device__ __forceinline__ void ct_put16(uint32_t row, int sw, int at, const F2 (&v)[8]) {
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) cl_parts(v[4 * c + i], CL_X_SCALE, hi[i], lo[i]);
    ct_sts4(row + (((at + c) ^ sw) << 4), hi[0], hi[1], hi[2], hi[3]);
    ct_sts4(row + (((at + c + 4) ^ sw) << 4), lo[0], lo[1], lo[2], lo[3]);
  }
}
// what is multiplied for channel c of a row of an operand, and for input c of row n of the weights
__device__ __forceinline__ float ct_value(uint32_t row, int r, int c, bool raw) {
  float f;
  if (raw) {
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(row + (((c >> 2) ^ (r & 7)) << 4) + (c & 3) * 4));
    return f;
  }
  const uint32_t a = row + (((c >> 3) ^ (r & 7)) << 4) + (c & 7) * 2;
  uint16_t hi, lo;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(hi) : "r"(a));
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(lo) : "r"(a ^ 64u));
  return fmaf(__half2float(__ushort_as_half(lo)), 1.f / CL_LO_SCALE, __half2float(__ushort_as_half(hi)));
}
// The hidden channels of a thread's position once more where they may not be parts, kept as what the whole block of 32 says (whether that is fp32).  All lanes
// load, those that `redo` names store.
__device__ __noinline__ bool ct_hidden(const CtTables& tb, int row, uint32_t op2, uint32_t d, bool redo) {
  F2 v[CT_H / 2];
  float m = 0.f;
#pragma unroll
  for (int c = 0; c < CT_H; c += 8) {
    uint32_t hi[8], lo[8];
    tmem_ld_32x8(d + c, hi);
    tmem_ld_32x8(d + CT_H + c, lo);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      float a[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) a[k] = fmaf(fmaf(__uint_as_float(lo[i + k]), 1.f / CL_LO_SCALE, __uint_as_float(hi[i + k])), tb.inv1[c + i + k], tb.b1[c + i + k]);
      v[(c + i) >> 1] = cl_elu(f2(a[0], a[1]));
      const float2 e = f2_get(v[(c + i) >> 1]);
      m = max3_abs(m, e.x, e.y);
    }
  }
  if (!redo) return false;
  const uint32_t o = op2 + row * 128;
  if (cl_code(m) != CB_RAW) {
#pragma unroll
    for (int c = 0; c < 2; ++c) ct_put16(o, row & 7, 2 * c, reinterpret_cast<const F2(&)[8]>(v[8 * c]));
    return false;
  }
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const float2 x = f2_get(v[2 * c]), y = f2_get(v[2 * c + 1]);
    ct_sts4(o + ((c ^ (row & 7)) << 4), __float_as_uint(x.x), __float_as_uint(x.y), __float_as_uint(y.x), __float_as_uint(y.y));
  }
  return true;
}
// eight inputs, 8 q and on, of row n of weights in shared memory
__device__ __forceinline__ void ct_weights(uint32_t row, int n, int q, float scale, float (&f)[8]) {
  const float4 hi = ct_lds4(row + ((q ^ (n & 7)) << 4)), lo = ct_lds4(row + (((q + 4) ^ (n & 7)) << 4));
  const float h[4] = {hi.x, hi.y, hi.z, hi.w}, l[4] = {lo.x, lo.y, lo.z, lo.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 fh = unpack_f16(__float_as_uint(h[i])), fl = unpack_f16(__float_as_uint(l[i]));
    f[2 * i] = fmaf(fl.x, 1.f / CL_LO_SCALE, fh.x) * scale;
    f[2 * i + 1] = fmaf(fl.y, 1.f / CL_LO_SCALE, fh.y) * scale;
  }
}
// The hidden channels in fp32 of the positions row0 + i that `mask` names, those with inputs that are not parts: a lane a channel, four positions at a time, their inputs
// a lane each going round by shuffles.
__device__ __noinline__ void ct_hidden_exact(CtTables& tb, int group, int row0, uint32_t mask, int first, uint32_t op1, uint32_t w1, uint32_t op2) {
  const int lane = threadIdx.x & 31;
  const float scale = tb.inv1[lane] * CL_X_SCALE;
#pragma unroll 1
  while (mask) {
    int row[4];
    float acc[4] = {};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      row[c] = mask ? row0 + __ffs(mask) - 1 : -CT_PAD;
      mask &= mask - 1u;
    }
#pragma unroll 1
    for (int j = 0; j < CT_TAPS; ++j) {
#pragma unroll 1
      for (int b = 0; b < 2; ++b) {
        float x[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int r = CT_PAD + row[c] - 2 + j;
          x[c] = 0.f;
          if (row[c] < 0 || r < first) continue;           // (none, or in front of the entry)
          const bool raw = tb.raw1[group][b][r];
          x[c] = ct_value(op1 + b * (CT_OP1 / 2) + r * 128, r, lane, raw) * (raw ? 1.f : 1.f / CL_X_SCALE);
        }
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          float f[8];
          ct_weights(w1 + (j * 2 + b) * 2 * CT_H * 128 + lane * 128, lane, q, scale, f);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (row[c] < 0 || CT_PAD + row[c] - 2 + j < first) continue;
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[c] = fmaf(__shfl_sync(0xffffffffu, x[c], 8 * q + k), f[k], acc[c]);
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (row[c] < 0) continue;
      const float a = acc[c] + tb.b1[lane];
      int word;
      uint32_t bits;
      const uint32_t code = cl_odd_row(f2_get(cl_elu(f2(a, a))).x, word, bits);
      asm volatile("st.shared.b32 [%0], %1;" ::"r"(op2 + row[c] * 128 + (((word >> 2) ^ (row[c] & 7)) << 4) + (word & 3) * 4), "r"(bits) : "memory");
      if (lane == 0) tb.raw2[group][row[c]] = code == CB_RAW;
    }
  }
}
// What a tile has of either kind: a thread's position, or sixteen of the warp's
__device__ __noinline__ void ct_odd(CtTables& tb, int group, int row, int half, int first, uint32_t op1, uint32_t w1, uint32_t op2, uint32_t d) {
  const int lane = threadIdx.x & 31, row0 = (row & ~31) + half * 16;
  auto exact = [&](int r) {
    bool any = false;
    for (int j = r >= 2 ? 0 : CT_TAPS; j < CT_TAPS; ++j)          // (nothing is made of rows 0 and 1)
      any |= tb.raw1[group][0][CT_PAD + r - 2 + j] || tb.raw1[group][1][CT_PAD + r - 2 + j];
    return any;
  };
  if (half == 0) {
    const bool mine = !exact(row), raw = ct_hidden(tb, row, op2, d, mine && row >= 2 && (tb.odd[group][0][row] || tb.odd[group][1][row]));
    if (mine) tb.raw2[group][row] = raw;
  }
  const uint32_t mask = __ballot_sync(0xffffffffu, lane < 16 && exact(row0 + (lane & 15)));
  if (mask) ct_hidden_exact(tb, group, row0, mask, first, op1, w1, op2);
}
// The last step for a warp some of whose positions have hidden channels that are not parts (`raw`): their channels in fp32, a lane a channel, before the sums that the others
// go through as well
__device__ __noinline__ void ct_last(const CtTables& tb, int row, int half, const F2 (&x)[16], uint32_t w3, uint32_t op2, uint32_t d, bool raw, float (&s)[CT_TAPS]) {
  const int lane = threadIdx.x & 31, n = half * 32 + lane;
  float v[32];
#pragma unroll
  for (int c = 0; c < 32; c += 8) {
    uint32_t hi[8], lo[8];
    tmem_ld_32x8(d + c, hi);
    tmem_ld_32x8(d + CT_C + c, lo);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[c + i] = fmaf(fmaf(__uint_as_float(lo[i]), 1.f / CL_LO_SCALE, __uint_as_float(hi[i])), tb.inv3[half * 32 + c + i], tb.b3[half * 32 + c + i]);
  }
  const float scale = tb.inv3[n] * CL_X_SCALE;
#pragma unroll 1
  for (uint32_t mask = __ballot_sync(0xffffffffu, raw); mask; mask &= mask - 1u) {
    const int p = __ffs(mask) - 1, at = (row & ~31) + p;
    float a = 0.f;
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      float f[8];
      ct_weights(w3 + n * 128, n, q, scale, f);
      const float4 h0 = ct_lds4(op2 + at * 128 + (((2 * q) ^ (at & 7)) << 4)), h1 = ct_lds4(op2 + at * 128 + (((2 * q + 1) ^ (at & 7)) << 4));
      const float h[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) a = fmaf(h[k], f[k], a);
    }
    a += tb.b3[n];
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      const float t = __shfl_sync(0xffffffffu, a, c);
      if (lane == p) v[c] = t;
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    F2 sum[CT_TAPS] = {f2(0.f), f2(0.f), f2(0.f)};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = q * 16 + 2 * i;
      const F2 y = cl_elu(f2_add(f2(v[c], v[c + 1]), x[8 * q + i]));
#pragma unroll
      for (int j = 0; j < CT_TAPS; ++j) {
        const float2 g = *reinterpret_cast<const float2*>(tb.wl[j] + half * 32 + c);
        sum[j] = f2_fma(y, f2(g.x, g.y), sum[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < CT_TAPS; ++j) {
      const float2 e = f2_get(sum[j]);
      s[j] += e.x + e.y;
    }
  }
}

__global__ void __launch_bounds__(CT_THREADS, 1) cl_res_tail_kernel(const __grid_constant__ CtParams p, const __grid_constant__ CUtensorMap xmap) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  CtTables& tb = *reinterpret_cast<CtTables*>(smem + CT_GROUPS * CT_GROUP_BYTES + CT_W1 + CT_W3);
  const int group = threadIdx.x / CT_GROUP_THREADS, tid = threadIdx.x % CT_GROUP_THREADS, warp = tid >> 5, lane = tid & 31;
  const int half = warp >> 2, row = (warp & 3) * 32 + lane, sw = row & 7;
  const uint32_t op1 = smem_u32(smem) + group * CT_GROUP_BYTES, op2 = op1 + CT_OP1;
  const uint32_t w1 = smem_u32(smem) + CT_GROUPS * CT_GROUP_BYTES, w3 = w1 + CT_W1, gate = smem_u32(&tb.gate);
  BoundedWait bw{p.wait_flag, gate};

  if (threadIdx.x == 0) {
    tb.gate = 0u;
    prefetch_tmap(&xmap);
    for (int i = 0; i < CT_GROUPS; ++i) {
      mbar_init(&tb.x_full[i], 1);
      mbar_init(&tb.m1[i], 1);
      mbar_init(&tb.m3[i], 1);
    }
    fence_barrier_init();
  }
  if (threadIdx.x < 32) {
    tmem_alloc(&tb.tmem, 512);
    tmem_relinquish();
  }
  for (int i = threadIdx.x; i < CT_C; i += CT_THREADS) {
    if (i < CT_H) tb.inv1[i] = __ldg(p.inv1 + i), tb.b1[i] = __ldg(p.b1 + i);
    tb.inv3[i] = __ldg(p.inv3 + i);
    tb.b3[i] = __ldg(p.b3 + i);
    for (int j = 0; j < CT_TAPS; ++j) tb.wl[j][i] = __ldg(p.wl + i * CT_TAPS + j);
  }
  // Weights (they do not depend on the kernels in front): the first 32 or 64 of a packed block's 128 rows as high parts, and again as low ones, so that one
  // instruction multiplies the activations' high parts by both
  auto weights = [&](const uint8_t* src, int rows, uint32_t dst) {
    for (int i = threadIdx.x; i < rows * 8; i += CT_THREADS) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(src) + i);
      ct_sts4(dst + i * 16, v.x, v.y, v.z, v.w);
      ct_sts4(dst + rows * 128 + (i ^ 4) * 16, v.x, v.y, v.z, v.w);
    }
  };
  for (int i = 0; i < CT_TAPS * 2; ++i) weights(p.w1 + static_cast<size_t>(i) * CL_W_BLOCK, CT_H, w1 + i * 2 * CT_H * 128);
  weights(p.w3, CT_C, w3);
  for (int i = tid; i < 2 * CT_PAD; i += CT_GROUP_THREADS) tb.raw1[group][i / CT_PAD][i % CT_PAD] = 0;
  for (int i = tid; i < 2 * CT_PAD * 8; i += CT_GROUP_THREADS)          // rows in front of a tile: read for positions that nothing is made of
    ct_sts4(op1 + (i / (CT_PAD * 8)) * (CT_OP1 / 2) + (i % (CT_PAD * 8)) * 16, 0u, 0u, 0u, 0u);
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t d1 = tb.tmem + group * 256, d3 = d1 + 2 * CT_H, lanes = static_cast<uint32_t>((warp & 3) * 32) << 16;
  const float bl = __ldg(p.bl);
  pdl_wait();
  if (threadIdx.x == 0) wait_gate_open(gate);
  pdl_trigger();
  auto tile_of = [&](int i, int& b, int& t0) {
    b = cu_div(i, p.t_tiles, p.t_tiles_inv);
    t0 = (i - b * p.t_tiles) * CT_OUT - 2 * (CT_TAPS - 1);           // position of row 0
  };
  auto fetch = [&](int i) {
    int b, t0;
    tile_of(i, b, t0);
    mbar_arrive_expect_tx(&tb.x_full[group], CT_X);
    for (int k = 0; k < 2; ++k) tma_load_3d(op1 + k * (CT_OP1 / 2) + CT_PAD * 128, &xmap, smem_u32(&tb.x_full[group]), k * 32, t0, b);
  };
  auto meet = [&](bool any) { return group == 0 ? warps_any<1, CT_GROUP_THREADS>(any) : warps_any<2, CT_GROUP_THREADS>(any); };
  const uint64_t a1 = umma_desc_sw128_kmajor(op1 + (CT_PAD - CT_TAPS + 1) * 128), a3 = umma_desc_sw128_kmajor(op2);
  const uint64_t b1 = umma_desc_sw128_kmajor(w1), b3 = umma_desc_sw128_kmajor(w3);
  const int step = CT_GROUPS * gridDim.x;
  int tile = blockIdx.x + group * gridDim.x;
  if (tid == 0 && tile < p.tiles) fetch(tile);
  uint32_t ph = 0;
#pragma unroll 1
  for (; tile < p.tiles; tile += step, ph ^= 1u) {
    int b, t0;
    tile_of(tile, b, t0);
    bw.wait(&tb.x_full[group], ph);
    // ---- ELU of the tile as parts, in its place: a thread's position, 32 of its channels, which it keeps for the residual ----
    const uint32_t o1 = op1 + half * (CT_OP1 / 2) + (CT_PAD + row) * 128;
    F2 x[16];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float4 v = ct_lds4(o1 + ((c ^ sw) << 4));
      x[2 * c] = f2(v.x, v.y);
      x[2 * c + 1] = f2(v.z, v.w);
    }
    float m = 0.f;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      F2 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] = cl_elu(x[8 * q + i]);
        const float2 e = f2_get(v[i]);
        m = max3_abs(m, e.x, e.y);
      }
      ct_put16(o1, sw, 2 * q, v);
    }
    const bool raw = cl_code(m) == CB_RAW;
    if (raw) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float2 e = f2_get(cl_elu(x[2 * c])), f = f2_get(cl_elu(x[2 * c + 1]));
        ct_sts4(o1 + ((c ^ sw) << 4), __float_as_uint(e.x), __float_as_uint(e.y), __float_as_uint(f.x), __float_as_uint(f.y));
      }
    }
    tb.raw1[group][half][CT_PAD + row] = raw;
    fence_proxy_async();
    const bool odd1 = meet(raw);
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
#pragma unroll 1
        for (int i = 0; i < 2 * CT_TAPS; ++i) {          // tap, then block of 32 channels
          const uint64_t a = a1 + (i >> 1) * 8 + (i & 1) * (CT_OP1 / 2 >> 4), w = b1 + i * (2 * CT_H * 128 >> 4);
#pragma unroll 1
          for (int k = 0; k < 2; ++k) {
            umma_bf16(d1, a + 2 * k, w + 2 * k, umma_idesc(128, 2 * CT_H, 0u), (i | k) ? 1u : 0u);
            umma_bf16(d1 + CT_H, a + 4 + 2 * k, w + 2 * k, umma_idesc(128, CT_H, 0u), 1u);
          }
        }
        umma_commit(&tb.m1[group]);
      }
      __syncwarp();
    }
    bw.wait(&tb.m1[group], ph);
    __syncwarp();
    tc_fence_after();
    if (tid == 0 && !odd1 && tile + step < p.tiles) fetch(tile + step);          // (the operand has been read; where fp32 is in it, once more below)
    // ---- ELU of the hidden channels as parts: sixteen of them ----
    {
      uint32_t hi[16], lo[16];
      tmem_ld_32x16(d1 + lanes + half * 16, hi);
      tmem_ld_32x16(d1 + lanes + CT_H + half * 16, lo);
      tmem_ld_wait();
      F2 v[8];
      m = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 s = *reinterpret_cast<const float2*>(tb.inv1 + half * 16 + 2 * i), c = *reinterpret_cast<const float2*>(tb.b1 + half * 16 + 2 * i);
        v[i] = f2_fma(f2(__uint_as_float(lo[2 * i]), __uint_as_float(lo[2 * i + 1])), f2(1.f / CL_LO_SCALE), f2(__uint_as_float(hi[2 * i]), __uint_as_float(hi[2 * i + 1])));
        v[i] = cl_elu(f2_fma(v[i], f2(s.x, s.y), f2(c.x, c.y)));
        const float2 e = f2_get(v[i]);
        m = max3_abs(m, e.x, e.y);
      }
      ct_put16(op2 + row * 128, sw, 2 * half, v);
    }
    // (both halves in range: the block of 32 is)
    tb.odd[group][half][row] = !cl_fits(m);
    fence_proxy_async();
    tc_fence_before();
    const bool odd = meet(odd1 || !cl_fits(m));
    if (odd) {
      tc_fence_after();
      ct_odd(tb, group, row, half, CT_PAD - t0, op1, w1, op2, d1 + lanes);
      fence_proxy_async();
      tc_fence_before();
      meet(false);
    }
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
          umma_bf16(d3, a3 + 2 * k, b3 + 2 * k, umma_idesc(128, 2 * CT_C, 0u), k);
          umma_bf16(d3 + CT_C, a3 + 4 + 2 * k, b3 + 2 * k, umma_idesc(128, CT_C, 0u), 1u);
        }
        umma_commit(&tb.m3[group]);
      }
      __syncwarp();
    }
    bw.wait(&tb.m3[group], ph);
    __syncwarp();
    tc_fence_after();
    // ---- residual, ELU, the taps of the last convolution: 32 channels ----
    float s[CT_TAPS] = {};
    if (!odd || !__any_sync(0xffffffffu, tb.raw2[group][row])) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t hi[16], lo[16];
        tmem_ld_32x16(d3 + lanes + half * 32 + q * 16, hi);
        tmem_ld_32x16(d3 + lanes + CT_C + half * 32 + q * 16, lo);
        const int n0 = half * 32 + q * 16;
        tmem_ld_wait();
        F2 v[8], sum[CT_TAPS];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float4 g = *reinterpret_cast<const float4*>(tb.inv3 + n0 + 4 * c), a = *reinterpret_cast<const float4*>(tb.b3 + n0 + 4 * c);
          auto one = [&](int i, F2 g2, F2 a2, F2 x2) {
            F2 u = f2_fma(f2(__uint_as_float(lo[i]), __uint_as_float(lo[i + 1])), f2(1.f / CL_LO_SCALE), f2(__uint_as_float(hi[i]), __uint_as_float(hi[i + 1])));
            return f2_add(f2_fma(u, g2, a2), x2);
          };
          v[2 * c] = one(4 * c, f2(g.x, g.y), f2(a.x, a.y), x[8 * q + 2 * c]);
          v[2 * c + 1] = one(4 * c + 2, f2(g.z, g.w), f2(a.z, a.w), x[8 * q + 2 * c + 1]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = cl_elu(v[i]);
#pragma unroll
        for (int j = 0; j < CT_TAPS; ++j) {
          sum[j] = f2(0.f);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float4 g = *reinterpret_cast<const float4*>(tb.wl[j] + n0 + 4 * c);
            sum[j] = f2_fma(v[2 * c], f2(g.x, g.y), sum[j]);
            sum[j] = f2_fma(v[2 * c + 1], f2(g.z, g.w), sum[j]);
          }
          const float2 e = f2_get(sum[j]);
          s[j] += e.x + e.y;
        }
      }
    } else {
      F2 kept[16];          // (of its own: what a call is given the address of lives in memory, everywhere)
      float sums[CT_TAPS] = {};
#pragma unroll
      for (int i = 0; i < 16; ++i) kept[i] = x[i];
      ct_last(tb, row, half, kept, w3, op2, d3 + lanes + half * 32, tb.raw2[group][row], sums);
#pragma unroll
      for (int j = 0; j < CT_TAPS; ++j) s[j] = sums[j];
    }
#pragma unroll
    for (int j = 0; j < CT_TAPS; ++j) tb.sums[group][half][j][row] = t0 + row < 0 ? 0.f : s[j];
    tc_fence_before();
    if (meet(bw.dead)) break;
    if (tid == 0 && odd1 && tile + step < p.tiles) fetch(tile + step);
    if (half == 0 && row >= 2 * (CT_TAPS - 1) && t0 + row < p.T) {
      float o = bl;
#pragma unroll
      for (int j = 0; j < CT_TAPS; ++j) o += tb.sums[group][0][j][row - 2 + j] + tb.sums[group][1][j][row - 2 + j];
      p.y[static_cast<long long>(b) * p.T + t0 + row] = o;
    }
  }
  if (__syncthreads_or(bw.dead) && threadIdx.x == 0) {            // let the copies in flight land before the block may leave
    const unsigned long long from = gtimer();
    while (gtimer() - from < 2000000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    tmem_dealloc(tb.tmem, 512);
  }
}
}  // namespace vb

using namespace vb;

extern "C" {

int vb_cl_dw_unit_pays(int B, int C, int rows, int dilation) {
  if (B <= 0 || rows <= 0 || C <= 0 || C % 64 || C > 256 || dilation < 1 || dilation > 64) return 0;
  return C <= 128 || (C + 127) / 128 * ((rows + 125LL) / 126) * B <= sm_count();
}

int vb_cl_dw_unit(float* d_y, void* d_yp, void* d_yp_code, const float* d_x, long long x_bstride, const float* d_dw_w, const float* d_dw_b,
                  const float* d_alpha_in, const float* d_alpha_mid, const void* d_w, const float* d_bias, const float* d_alpha_out, int B, int C, int T,
                  int dilation, int t_lo, int t_hi, void* stream) {
  VB_CHECK_ARG(!d_y != !d_yp && !d_yp == !d_yp_code, "vb_cl_dw_unit: one result, as fp32 or as parts with their codes");
  VB_CHECK_ARG(d_x && d_dw_w && d_dw_b && d_alpha_in && d_alpha_mid && d_w && d_bias, "vb_cl_dw_unit: null pointer");
  VB_CHECK_ARG(C > 0 && C % 64 == 0 && C <= 64 * CU_MAX_CHUNKS && dilation >= 1 && dilation <= 64, "vb_cl_dw_unit: C = %d (a multiple of 64, <= 1024), dilation %d",
               C, dilation);
  VB_CHECK_ARG(x_bstride % 4 == 0 && on16(d_x) && on16(d_y) && on16(d_yp), "vb_cl_dw_unit: rows must start on 16-byte boundaries");
  VB_CHECK_ARG(on16(d_dw_w) && on16(d_dw_b) && on16(d_alpha_in) && on16(d_alpha_mid) && on16(d_w) && on16(d_bias) && on16(d_alpha_out),
               "vb_cl_dw_unit: weights, biases and alphas must lie on 16-byte boundaries");
  VB_CHECK_ARG(0 <= t_lo && t_lo <= t_hi && t_hi <= T, "vb_cl_dw_unit: range [%d, %d) outside [0, %d)", t_lo, t_hi, T);
  VB_CHECK_ARG(B <= 65535, "vb_cl_dw_unit: %d entries", B);
  if (B <= 0 || t_lo == t_hi) return 0;
  const CuDwPlan g = cu_dw_plan(C, dilation, t_hi - t_lo, B, sm_count());
  CuDwParams p = {};
  VB_CHECK_ARG(p.wait_flag = wait_flag(WK_CL_CONV), "vb_cl_dw_unit: no mapped host memory");
  const long long n_pad = (C + 127LL) / 128 * 128;
  p.x = d_x; p.dw_w = d_dw_w; p.dw_b = d_dw_b; p.alpha_in = d_alpha_in; p.alpha_mid = d_alpha_mid;
  p.w = static_cast<const uint8_t*>(d_w);
  p.w_inv = reinterpret_cast<const float*>(p.w + n_pad * C * 4);
  p.bias = d_bias; p.alpha_out = d_alpha_out; p.y = d_y; p.yp = static_cast<uint32_t*>(d_yp); p.yp_code = static_cast<uint8_t*>(d_yp_code);
  p.x_bstride = x_bstride; p.y_bstride = static_cast<long long>(T) * C;
  p.C = C; p.T = T; p.dil = dilation; p.t_lo = t_lo; p.t_hi = t_hi;
  p.nr = g.nr; p.cols = g.cols; p.classes = g.classes; p.segs = g.segs; p.len = g.len; p.m_tiles = (C + 127) / 128; p.chunks = C / 64; p.w_stages = g.w_stages;
  auto inverse = [](int b) { return b > 1 ? static_cast<uint32_t>(((1ULL << 32) + b - 1) / b) : 0u; };
  p.runs_inv = inverse(g.classes * g.segs); p.segs_inv = inverse(g.segs); p.dil_inv = inverse(dilation); p.m_tiles_inv = inverse(p.m_tiles);
  p.tmem_cols = 32;
  while (p.tmem_cols < 2 * g.cols) p.tmem_cols *= 2;
  const long long tiles = static_cast<long long>(p.m_tiles) * ((static_cast<long long>(t_hi) - t_lo + g.nr - 1) / g.nr);
  VB_CHECK_ARG(tiles <= 0x7fffffffLL, "vb_cl_dw_unit: too many tiles");
  const dim3 grid(static_cast<unsigned>(tiles), B);
  if (g.warps == 9) {
    VB_CHECK_CUDA(max_dyn_smem_once(cl_dw_unit_kernel<9>));
    VB_LAUNCH_PDL(cl_dw_unit_kernel<9>, grid, 320, g.smem, stream, p);
  } else {
    VB_CHECK_CUDA(max_dyn_smem_once(cl_dw_unit_kernel<18>));
    VB_LAUNCH_PDL(cl_dw_unit_kernel<18>, grid, 608, g.smem, stream, p);
  }
  return 0;
}

int vb_cl_res_tail(float* d_y, const float* d_x, long long x_bstride, const void* d_w1, const float* d_b1, const void* d_w3, const float* d_b3,
                   const float* d_wl, const float* d_bl, int B, int T, void* stream) {
  VB_CHECK_ARG(d_y && d_x && d_w1 && d_b1 && d_w3 && d_b3 && d_wl && d_bl, "vb_cl_res_tail: null pointer");
  VB_CHECK_ARG(T > 0 && x_bstride % 4 == 0 && on16(d_x) && on16(d_w1) && on16(d_w3), "vb_cl_res_tail: rows and weights must start on 16-byte boundaries");
  if (B <= 0) return 0;
  VB_CHECK_ARG(encode_fn(), "cuTensorMapEncodeTiled not available (no CUDA driver?)");
  CtParams p = {};
  VB_CHECK_ARG(p.wait_flag = wait_flag(WK_CL_CONV), "vb_cl_res_tail: no mapped host memory");
  p.w1 = static_cast<const uint8_t*>(d_w1); p.w3 = static_cast<const uint8_t*>(d_w3);
  p.inv1 = reinterpret_cast<const float*>(p.w1 + static_cast<size_t>(CT_TAPS) * 2 * CL_W_BLOCK); p.inv3 = reinterpret_cast<const float*>(p.w3 + CL_W_BLOCK);
  p.b1 = d_b1; p.b3 = d_b3; p.wl = d_wl; p.bl = d_bl; p.y = d_y; p.T = T;
  p.t_tiles = (T + CT_OUT - 1) / CT_OUT;
  const long long tiles = static_cast<long long>(p.t_tiles) * B;
  VB_CHECK_ARG(tiles < 0x7fffffffLL - 2 * CT_GROUPS * 1024, "vb_cl_res_tail: too many tiles");
  p.tiles = static_cast<int>(tiles);
  p.t_tiles_inv = p.t_tiles > 1 ? static_cast<uint32_t>(((1ULL << 32) + p.t_tiles - 1) / p.t_tiles) : 0u;
  CUtensorMap map;
  cuuint64_t dims[3] = {CT_C, static_cast<cuuint64_t>(T), static_cast<cuuint64_t>(B)};
  cuuint64_t strides[2] = {CT_C * 4, static_cast<cuuint64_t>(B > 1 ? x_bstride : static_cast<long long>(T) * CT_C) * 4};
  cuuint32_t box[3] = {32, CT_ROWS, 1}, estr[3] = {1, 1, 1};
  const CUresult r = encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(d_x), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  VB_CHECK_ARG(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled(tail) failed: CUresult %d", static_cast<int>(r));
  VB_CHECK_CUDA(max_dyn_smem_once(cl_res_tail_kernel));
  VB_LAUNCH_PDL(cl_res_tail_kernel, min(p.tiles, sm_count()), CT_THREADS, CT_SMEM, stream, p, map);
  return 0;
}

}  // extern "C"
