// What the vocoder kernels over channels-last activations share (cl_conv.cu: the convolutions and what stands between them; cl_unit.cu: residual
// units in one launch): activations as two fp16 parts a value, activation functions, pieces of the epilogues.
#pragma once
#include "common.cuh"
#include <cuda_fp16.h>
#include <cudaTypedefs.h>

namespace vb {
PFN_cuTensorMapEncodeTiled_v12000 encode_fn();      // api.cu

constexpr int CL_W_BLOCK = 128 * 128;       // 128 output channels x 32 input channels, high and low parts

constexpr float CL_X_SCALE = 16.f, CL_LO_SCALE = 2048.f;      // of activations; of low parts against high ones
// what the two parts of an activation hold to 2^-22.  Where the largest value is not between these (or zero) -- of a block kept as parts, of what goes
// into one result of fp32 activations -- the products are taken on CUDA cores
constexpr float CL_X_TOP = 65472.f / CL_X_SCALE, CL_X_LOW = 0x1p-10f / CL_X_SCALE;
enum ClCode { CB_NORMAL = 1, CB_RAW = 4 };      // of a block of 32 activations kept as parts (all zero: 0)

enum ClAct { CA_NONE = 0, CA_SNAKE = 1, CA_ELU = 2, CA_GELU = 3 };

__device__ __forceinline__ void cl_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, uint32_t src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(src), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_32x4(uint32_t taddr, uint32_t (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr));
}
__device__ __forceinline__ void tmem_st_32x4(uint32_t taddr, const float (&v)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]) : "memory");
}
__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float2 unpack_f16(uint32_t v) {
  return __half22float2(*reinterpret_cast<const __half2*>(&v));
}
// the larger magnitude of three, NaN if one is
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// the smaller magnitude of three
__device__ __forceinline__ float min3_abs(float a, float b, float c) {
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// two fp32 values in one register pair: an instruction for both
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ float2 f2_get(F2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// parts of two values, v * scale = hi + lo / 2048
__device__ __forceinline__ void cl_parts(F2 a, float scale, uint32_t& hi, uint32_t& lo) {
  const float2 x = f2_get(f2_mul(a, f2(scale))), y = f2_get(f2_mul(a, f2(scale * CL_LO_SCALE)));
  hi = pack_f16(x.x, x.y);
  float l0, l1;          // 2048 (x - hi), both steps exact
  asm("{\n\t.reg .b16 h0, h1, m;\n\tmov.b32 {h0, h1}, %2;\n\tmov.b16 m, 0xE800;\n\tfma.rn.f32.f16 %0, h0, m, %3;\n\tfma.rn.f32.f16 %1, h1, m, %4;\n\t}\n"
      : "=f"(l0), "=f"(l1)
      : "r"(hi), "f"(y.x), "f"(y.y));
  lo = pack_f16(l0, l1);
}
// Two rows of a block whose channels lie in the lanes: neighbouring lanes exchange, even ones keep two high parts, odd ones two low parts of each
// row -> word (lane & 1 ? 16 : 0) + (lane >> 1) of either row
__device__ __forceinline__ void cl_exchange(uint32_t hi, uint32_t lo, uint32_t& w0, uint32_t& w1) {
  const bool odd = threadIdx.x & 1;
  const uint32_t own = odd ? lo : hi, got = __shfl_xor_sync(0xffffffffu, odd ? hi : lo, 1);
  w0 = __byte_perm(own, got, odd ? 0x1054u : 0x5410u);
  w1 = __byte_perm(own, got, odd ? 0x3276u : 0x7632u);
}
// what a block of 32 activations with the largest magnitude m is kept as
__device__ __forceinline__ bool cl_fits(float m) { return __float_as_uint(m) - __float_as_uint(CL_X_LOW) < __float_as_uint(CL_X_TOP) - __float_as_uint(CL_X_LOW); }
__device__ __forceinline__ uint32_t cl_code(float m) { return cl_fits(m) ? CB_NORMAL : m == 0.f ? 0u : CB_RAW; }      // (zeros are the same bits either way)
// Activations kept as parts: 128 bytes per 32 channels as in fp32, [32 high | 32 low] fp16 -- or, where the largest of the 32 is out of range, the fp32
// values themselves, with CB_RAW in the block's code byte.  Here for eight neighbouring lanes that hold a block's channels, four each.
__device__ __forceinline__ void cl_put4(uint32_t* yp, uint8_t* code, size_t at, const float4& v) {
  float m = max3_abs(max3_abs(v.x, v.y, v.z), v.w, v.w);
  const uint32_t eight = 0xffu << (threadIdx.x & 24);
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
    const float other = __shfl_xor_sync(eight, m, o);
    m = max3_abs(m, other, other);
  }
  const uint32_t c = cl_code(m), in = static_cast<uint32_t>(at) & 31u;
  uint32_t* blk = yp + (at - in);
  if (!cl_fits(m)) {
    *reinterpret_cast<float4*>(blk + in) = v;
  } else {
    uint2 hi, lo;
    cl_parts(f2(v.x, v.y), CL_X_SCALE, hi.x, lo.x);
    cl_parts(f2(v.z, v.w), CL_X_SCALE, hi.y, lo.y);
    *reinterpret_cast<uint2*>(blk + (in >> 1)) = hi;
    *reinterpret_cast<uint2*>(blk + 16 + (in >> 1)) = lo;
  }
  if (in == 0) code[at >> 5] = static_cast<uint8_t>(c);
}
// ... and for a warp that holds a block, a channel a lane
__device__ __forceinline__ void cl_put1(uint32_t* yp, uint8_t* code, size_t block, float v) {
  const int lane = threadIdx.x & 31;
  float m = v;
  asm volatile("redux.sync.max.NaN.abs.f32 %0, %0, 0xffffffff;" : "+f"(m));
  const uint32_t c = cl_code(m);
  uint32_t hi, lo, word, unused;
  cl_parts(f2(v, 0.f), CL_X_SCALE, hi, lo);
  cl_exchange(hi, lo, word, unused);
  if (!cl_fits(m)) yp[block * 32 + lane] = __float_as_uint(v);
  else yp[block * 32 + (lane & 1 ? 16 : 0) + (lane >> 1)] = word;
  if (lane == 0) code[block] = static_cast<uint8_t>(c);
}

// sin(x)^2: the square needs x only modulo pi, so one rounding step k = x / pi (in the low bits of a sum with 1.5 2^23) and two fused steps
// x - k pi leave |r| <= pi / 2, where sin r = r + r^3 P(r^2) with a fitted polynomial of degree 3 (largest relative error 6e-9).  Valid up
// to |x| = 2^16 (k pi exact to 2^-33 there); larger arguments take sinf.  Two values an instruction and no branch per element.
constexpr float CL_SIN_MAX = 65536.f;
template <int N>
__device__ __forceinline__ void cl_sin_sq(const F2 (&x)[N], F2 (&s)[N]) {
  F2 k[N], r[N], u[N];
#pragma unroll
  for (int i = 0; i < N; ++i) k[i] = f2_fma(x[i], f2(0.318309886f), f2(12582912.f));
#pragma unroll
  for (int i = 0; i < N; ++i) k[i] = f2_add(k[i], f2(-12582912.f));
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = f2_fma(k[i], f2(-3.14159274101f), x[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = f2_fma(k[i], f2(8.742278012619e-08f), r[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) u[i] = f2_mul(r[i], r[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = f2_fma(u[i], f2(2.605780761e-06f), f2(-1.980960296e-04f));
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = f2_fma(u[i], s[i], f2(8.333066247e-03f));
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = f2_fma(u[i], s[i], f2(-1.666665955e-01f));
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = f2_fma(f2_mul(r[i], u[i]), s[i], r[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = f2_mul(s[i], s[i]);
}
__device__ __forceinline__ F2 cl_sin_sq(F2 x) {
  const F2 in[1] = {x};
  F2 out[1];
  cl_sin_sq(in, out);
  return out[0];
}
// ELU without a branch: e^x - 1 = 2^n (e^r - 1) + (2^n - 1) with x = n ln 2 + r, |r| <= ln 2 / 2, and e^r - 1 = r + r^2 Q(r) with a
// fitted polynomial of degree 4.  Largest relative error against 64 bits 8.7e-8 over [-90, 0].
__device__ __forceinline__ F2 cl_elu(F2 v) {
  const float2 w = f2_get(v);
  const F2 x = f2(fmaxf(w.x, -80.f), fmaxf(w.y, -80.f));
  const F2 t = f2_fma(x, f2(1.44269504f), f2(12582912.f)), n = f2_add(t, f2(-12582912.f));        // n in the low bits of t as well
  F2 r = f2_fma(n, f2(-0.693359375f), x);
  r = f2_fma(n, f2(2.12194440e-4f), r);
  F2 q = f2_fma(r, f2(0.0013882514f), f2(0.0083665475f));
  q = f2_fma(q, r, f2(0.0416672f));
  q = f2_fma(q, r, f2(0.16666543f));
  q = f2_fma(q, r, f2(0.49999997f));
  const F2 e = f2_fma(f2_mul(r, r), q, r);
  const float2 tb = f2_get(t);
  const F2 s = f2(__uint_as_float((__float_as_uint(tb.x) << 23) + 0x3f800000u), __uint_as_float((__float_as_uint(tb.y) << 23) + 0x3f800000u));
  const float2 o = f2_get(f2_fma(s, e, f2_add(s, f2(-1.f))));
  return f2(w.x <= 0.f ? o.x : w.x, w.y <= 0.f ? o.y : w.y);
}
// v + inv sin(a v)^2 of four values, two channels a pair
__device__ __forceinline__ void cl_snake4(F2& v0, F2& v1, F2 a0, F2 a1, F2 i0, F2 i1) {
  const F2 y0 = f2_mul(a0, v0), y1 = f2_mul(a1, v1);
  const float2 p = f2_get(y0), q = f2_get(y1);
  F2 s0 = cl_sin_sq(y0), s1 = cl_sin_sq(y1);
  if (!(max3_abs(max3_abs(p.x, p.y, q.x), q.y, q.y) <= CL_SIN_MAX)) {      // (each value by itself: its result does not depend on the others)
    const float2 a = f2_get(s0), b = f2_get(s1);
    auto one = [](float y, float s) {
      if (fabsf(y) <= CL_SIN_MAX) return s;
      const float sn = sinf(y);
      return sn * sn;
    };
    s0 = f2(one(p.x, a.x), one(p.y, a.y));
    s1 = f2(one(q.x, b.x), one(q.y, b.y));
  }
  v0 = f2_fma(i0, s0, v0);
  v1 = f2_fma(i1, s1, v1);
}
__device__ __forceinline__ float4 cl_snake4(const float4& v, const float4& a, const float4& inv) {
  F2 v0 = f2(v.x, v.y), v1 = f2(v.z, v.w);
  cl_snake4(v0, v1, f2(a.x, a.y), f2(a.z, a.w), f2(inv.x, inv.y), f2(inv.z, inv.w));
  const float2 p = f2_get(v0), q = f2_get(v1);
  return make_float4(p.x, p.y, q.x, q.y);
}

// copies of a channel tile of `width` channels in the 128 rows of its weights: the epilogue's warps share their columns
__host__ __device__ __forceinline__ int cl_copies(int width) { return width == 32 ? 4 : width == 64 ? 2 : 1; }

// The epilogue works on eight columns at a time, in a loop that is short enough for the instruction caches: sixteen columns in straight-line
// code took twice as long (Mimi's 1x1 layer of 153600 x 128 85 us).
constexpr int CL_EC = 8;

__device__ __forceinline__ void cl_load_acc(uint32_t taddr, int cols, float inv, F2 (&v)[CL_EC / 2]) {
  uint32_t hi[CL_EC], lo[CL_EC];
  tmem_ld_32x8(taddr, hi);
  tmem_ld_32x8(taddr + cols, lo);
  tmem_ld_wait();
#pragma unroll
  for (int c = 0; c < CL_EC / 2; ++c)
    v[c] = f2_mul(f2_fma(f2(__uint_as_float(lo[2 * c]), __uint_as_float(lo[2 * c + 1])), f2(1.f / CL_LO_SCALE),
                         f2(__uint_as_float(hi[2 * c]), __uint_as_float(hi[2 * c + 1]))),
                  f2(inv));
}

// act(v), in place
template <int ACT>
__device__ __forceinline__ void cl_act(float alpha, float ialpha, F2 (&v)[CL_EC / 2]) {
  if (ACT == CA_SNAKE) {
#pragma unroll
    for (int c = 0; c < CL_EC / 2; c += 2) cl_snake4(v[c], v[c + 1], f2(alpha), f2(alpha), f2(ialpha), f2(ialpha));
  } else if (ACT == CA_ELU) {
#pragma unroll
    for (int c = 0; c < CL_EC / 2; ++c) v[c] = cl_elu(v[c]);
  } else if (ACT == CA_GELU) {
#pragma unroll
    for (int c = 0; c < CL_EC / 2; ++c) {
      const float2 x = f2_get(v[c]);
      v[c] = f2(0.5f * x.x * (1.f + erff(x.x * 0.70710678118654752f)), 0.5f * x.y * (1.f + erff(x.y * 0.70710678118654752f)));
    }
  }
}

// Whether eight rows of a block are all of ordinary size: no value out of range, and a lane none of whose rows is tiny.  (Nearly always; a chunk that
// this does not hold for is looked at row by row.)  `rows`: a bit for each that there is; the others become 1.  One code for a chunk, its largest
// value's, cost 8 of Mimi's 1262 us less, and let a loud row's neighbours lose what they are made of.
__device__ __forceinline__ bool cl_ordinary(F2 (&v)[CL_EC / 2], uint32_t rows) {
  if (rows != 0xffu) {
#pragma unroll
    for (int c = 0; c < CL_EC / 2; ++c) {
      const float2 x = f2_get(v[c]);
      v[c] = f2(rows >> (2 * c) & 1u ? x.x : 1.f, rows >> (2 * c) & 2u ? x.y : 1.f);
    }
  }
  float top = 0.f, low = CL_X_TOP;
#pragma unroll
  for (int c = 0; c < CL_EC / 2; ++c) {
    const float2 x = f2_get(v[c]);
    top = max3_abs(top, x.x, x.y);
    low = min3_abs(low, x.x, x.y);
  }
  return __all_sync(0xffffffffu, top < CL_X_TOP) && __any_sync(0xffffffffu, low >= CL_X_LOW);
}
// a row of a block on its own: word `at` of the row -> its bits, and the row's code
__device__ __forceinline__ uint32_t cl_odd_row(float x, int& at, uint32_t& bits) {
  const int lane = threadIdx.x & 31;
  float m = x;
  asm volatile("redux.sync.max.NaN.abs.f32 %0, %0, 0xffffffff;" : "+f"(m));
  const uint32_t code = cl_code(m);
  uint32_t hi, lo, unused;
  cl_parts(f2(x, 0.f), CL_X_SCALE, hi, lo);
  cl_exchange(hi, lo, bits, unused);
  at = (lane & 1 ? 16 : 0) + (lane >> 1);
  if (!cl_fits(m)) {
    at = lane;
    bits = __float_as_uint(x);
  }
  return code;
}

}  // namespace vb
