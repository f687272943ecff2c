// Fused multi-codebook sampler: repetition penalty -> temperature -> softmax -> top-k / top-p / min-p
// filter -> draw, plus the repetition-cache update.  Replaces vox_serve/sampling.py (Sampler.run_sampling,
// apply_repetition_penalty, update_repetition_penalty_cache) and the FlashInfer sampling kernels it calls.
//
// Exact + deterministic by construction:
//   * logits are bf16, so after penalty and temperature every token's value is one of 65536 bf16 codes (a
//     monotone 16-bit key) and every token with the same code has the same bf16-rounded probability;
//   * one thread-block cluster per row keeps the whole row on chip after a single pass (sample_kernel below):
//     integer masses, fixed reduction trees, no atomics -- the result does not depend on thread scheduling;
//   * greedy = largest key, smallest index on ties: exactly torch.argmax on the penalised bf16 logits.
#include "../../include/vb_api.h"
#define VB_PDL_FAMILY 16
#include "common.cuh"

namespace vb {

struct SampleParams {
  const __nv_bfloat16* logits;
  const uint8_t* rep_cache;    // [B][W][C][V] or null
  const int32_t* cache_rows;   // optional: batch row b reads / marks cache row cache_rows[b] (slot-resident caches)
  int rows, vocab, ld;
  int W, C_cache, C_logits;
  float penalty, temperature;
  int strategy, top_k;
  float top_p, min_p;
  int mask_token;
  uint64_t seed, offset;
  unsigned long long* rng_state;   // optional device {seed, offset, arrivals}: offset advances by one per call
  int64_t* out;
};

__device__ __forceinline__ uint32_t bf16_key(float v) {  // monotone: larger value <-> larger key
  const uint32_t b = __float_as_uint(v) >> 16;
  return (b & 0x8000u) ? (~b & 0xffffu) : (b | 0x8000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
  const uint32_t b = (k & 0x8000u) ? (k & 0x7fffu) : (~k & 0xffffu);
  return __uint_as_float(b << 16);
}

// penalised (and, for stochastic strategies, temperature-scaled) bf16 value of token i of `row`
__device__ __forceinline__ float token_value(const SampleParams& p, int row, int i, bool scaled) {
  float l = __bfloat162float(p.logits[static_cast<size_t>(row) * p.ld + i]);
  if (p.rep_cache) {
    const int b0 = row / p.C_logits;
    const int b = p.cache_rows ? p.cache_rows[b0] : b0;
    const int c = (p.C_logits == 1 && p.C_cache != 1) ? 0 : row % p.C_logits;   // sampling.py:140-141
    bool seen = false;
    for (int w = 0; w < p.W; ++w)
      seen |= p.rep_cache[((static_cast<size_t>(b) * p.W + w) * p.C_cache + c) * p.vocab + i] != 0;
    if (seen) l = (l > 0.f) ? round_bf16(l / p.penalty) : round_bf16(l * p.penalty);   // sampling.py:143-144
  }
  if (i == p.mask_token) l = -INFINITY;
  if (scaled) l = round_bf16(l / p.temperature);
  return l;
}

// ---- Philox4x32-10 ----
__device__ __forceinline__ void philox_round(uint32_t (&c)[4], uint32_t k0, uint32_t k1) {
  const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
  const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
  const uint32_t n0 = hi1 ^ c[1] ^ k0, n1 = lo1, n2 = hi0 ^ c[3] ^ k1, n3 = lo0;
  c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
}
__device__ __forceinline__ double philox_uniform(uint64_t seed, uint64_t offset, uint32_t stream, uint32_t sub) {
  uint32_t c[4] = {static_cast<uint32_t>(offset), static_cast<uint32_t>(offset >> 32), stream, sub};
  uint32_t k0 = static_cast<uint32_t>(seed), k1 = static_cast<uint32_t>(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    philox_round(c, k0, k1);
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  const uint64_t bits = (static_cast<uint64_t>(c[0]) << 21) ^ (static_cast<uint64_t>(c[1]) >> 11);  // 53 bits
  return static_cast<double>(bits & ((1ull << 53) - 1)) * (1.0 / 9007199254740992.0);
}

// ---------------------------------------------------------------------------------------------------------
// One thread-block CLUSTER per row.  The row's tokens are spread over S CTAs x 1024 threads x (2 * PAIRS) tokens;
// after one pass over the logits (+ repetition cache) every token lives on chip -- its 16-bit value key
// and its bf16 probability in one word of shared memory -- and everything else is on-chip reductions:
// block tree -> one DSMEM store per peer CTA -> one cluster barrier.  No histogram, no atomics, no second
// pass over HBM/L2.
//   max key -> [top-k: 16-step bisection on counts] -> softmax denominator (fp32, fixed summation tree) ->
//   mass q_i = floor(bf16(p_i) * 2^32) -> [min-p: direct filter] -> draw by inverse CDF in (cta, thread, pair)
//   order; top-p by REJECTION: the drawn token j is in the nucleus iff mass{p > p_j} < top_p, otherwise
//   everything with p <= p_j is discarded and the draw repeats on what is left (acceptance >= top_p per round;
//   conditional on acceptance the draw is the renormalised nucleus -- the scheme of FlashInfer's sorting-free
//   sampler, with exact integer masses instead of float partial sums, hence scheduling-independent).
// ---------------------------------------------------------------------------------------------------------
// A token's word in shared memory holds its key above and, once the softmax is known, its probability (bf16) below; a mass is taken
// from the probability where it is needed.  Every pass is then a short loop over the thread's pairs: with the keys in registers the
// passes had to be unrolled forty tokens deep, and reading that code once took longer than running it (top-p, cold: 32 rows of 2,051
// tokens 61 us against 18 here; 32 rows of 156,940 tokens in a row of calls 53 against 39, and 67 with 1024 threads that spilled).
// A row's time (28 us in a row of calls, of which 2.3 are traffic) goes to the loads and the first loop (8 us), the two exponentials a token
// and the conversions to masses (6: those units take 8 cycles a warp), and a microsecond and more for each meeting of the cluster: five where the
// first draw is accepted (largest key, denominator, masses, the draw, the mass above it).
constexpr int SMP_THREADS = 1024;        // (cta, thread, pair) order of the tokens
constexpr int SMP_PAIRS = 20;            // 40 tokens per thread: 40960 tokens per CTA, 327680 per 8-CTA cluster
constexpr int SMP_MAX_CLUSTER = 8;

__device__ __forceinline__ void st_dsmem_u64(unsigned long long* local_ptr, uint32_t cta_rank, unsigned long long v) {
  uint32_t laddr = smem_u32(local_ptr), raddr;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(raddr) : "r"(laddr), "r"(cta_rank));
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(raddr), "l"(v) : "memory");
}

struct SmpCtx {
  int S, rank, buf;
  unsigned long long (*xch)[SMP_MAX_CLUSTER];   // [2][8] exchange slots, written by the peers
  unsigned long long* sh;                       // [33]
  __device__ __forceinline__ void publish(unsigned long long v) {   // one warp: lane r stores into CTA r
    const int lane = threadIdx.x & 31;
    if (S == 1) {
      if (lane == 0) xch[buf][0] = v;
    } else if (lane < S) {
      st_dsmem_u64(&xch[buf][rank], lane, v);
    }
  }
  __device__ __forceinline__ void sync() {
    if (S == 1) __syncthreads(); else cluster_sync_all();
  }
};
enum { SMP_SUM = 0, SMP_MAX = 1, SMP_MIN = 2 };
template <int OP>
__device__ __forceinline__ unsigned long long smp_op(unsigned long long a, unsigned long long b) {
  return OP == SMP_SUM ? a + b : (OP == SMP_MAX ? (a > b ? a : b) : (a < b ? a : b));
}
// cluster-wide reduction of one u64 per thread; every thread of every CTA gets the result
template <int OP>
__device__ __forceinline__ unsigned long long smp_reduce(unsigned long long v, SmpCtx& c) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = smp_op<OP>(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) c.sh[warp] = v;
  __syncthreads();
  if (warp == 0) {
    unsigned long long x = c.sh[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = smp_op<OP>(x, __shfl_xor_sync(0xffffffffu, x, o));
    c.publish(x);
  }
  c.sync();
  unsigned long long r = c.xch[c.buf][0];
  for (int i = 1; i < c.S; ++i) r = smp_op<OP>(r, c.xch[c.buf][i]);
  c.buf ^= 1;
  return r;
}
// fp32 sum with a fixed tree (xor butterfly inside the warp and across warps, CTA partials in rank order)
__device__ __forceinline__ float smp_sum_f32(float v, SmpCtx& c) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  float* shf = reinterpret_cast<float*>(c.sh);
  if (lane == 0) shf[warp] = v;
  __syncthreads();
  if (warp == 0) {
    const float x = warp_sum(shf[lane]);
    c.publish(static_cast<unsigned long long>(__float_as_uint(x)));
  }
  c.sync();
  float r = 0.f;
  for (int i = 0; i < c.S; ++i) r += __uint_as_float(static_cast<uint32_t>(c.xch[c.buf][i]));
  c.buf ^= 1;
  return r;
}

// The kernel is instruction-bound (the whole row is on chip): the softmax uses the hardware exponential
// (ex2.approx, 2 ulp) -- a sampler's masses do not need expf's last bit.
constexpr float kLog2e = 1.4426950408889634f;
__device__ __forceinline__ float smp_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Block-wide exclusive scan of one u64 per thread, thread order; returns exclusive prefix, *total = sum.
__device__ __forceinline__ unsigned long long block_excl_scan(unsigned long long v, unsigned long long* sh, unsigned long long* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) sh[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const unsigned long long w = sh[lane];
    unsigned long long wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long n = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += n;
    }
    sh[lane] = wi - w;
    if (lane == 31) sh[32] = wi;
  }
  __syncthreads();
  const unsigned long long res = sh[warp] + incl - v;
  *total = sh[32];
  __syncthreads();
  return res;
}

// the division, out of line: hardly any token needs it
__device__ __noinline__ float smp_quotient(float a, float b) { return a / b; }
// a / b to the nearest with y = 1 / b, for one divisor of many dividends: quotient by the correctly rounded reciprocal and two corrections by the
// exact remainder (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. R&D 34, 1990).
// `far` grows past SMP_FAR where the product leaves [2^-79, 2^81): extreme dividends, zeros (the remainder loses their sign), infinities
// and NaNs.  Those take the division itself.  (The quotients of bf16 values by one of few bits lie on the middle of two bf16 values so often
// that asking whether the product's rounding is sure costs more than the corrections.)
// The remainder is exact while its last bit, 2^-46 of quotient times divisor, is an fp32 value: divisors from 2^-20 on (2^-79 2^-20 2^-46 = 2^-145).
constexpr uint32_t SMP_FAR = 0xa0000000u;
constexpr float SMP_DIVISOR_LOW = 0x1p-20f;
__device__ __forceinline__ float smp_div(float a, float b, float y, uint32_t& far) {
  float q = a * y;
  far = max(far, (__float_as_uint(q) << 1) - 0x30000000u);
  q = fmaf(fmaf(-q, b, a), y, q);
  return fmaf(fmaf(-q, b, a), y, q);
}
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// the two keys of a pair of bf16 codes, and back (bf16_key / key_value on both halves at once)
__device__ __forceinline__ uint32_t key_pair(uint32_t bits) {
  const uint32_t neg = (bits >> 15) & 0x00010001u;
  return bits ^ (0x80008000u | neg * 0x7fffu);
}
// the value of a token's word whose low half is zero
__device__ __forceinline__ float word_value(uint32_t t) {
  const uint32_t m = static_cast<uint32_t>(~static_cast<int32_t>(t) >> 31);          // all ones where the key is a negative value's
  return __uint_as_float(t ^ (0x80000000u | (m & 0x7fff0000u)));
}
// a probability (bf16 in the low half of a token's word) as a mass: floor(p 2^32), saturating at 2^32 - 1
__device__ __forceinline__ uint32_t smp_mass(uint32_t word) { return __float2uint_rz(bf16_lo(word) * 4294967296.f); }

__global__ void __launch_bounds__(SMP_THREADS, 1) sample_kernel(const SampleParams p, const int npairs) {
  extern __shared__ uint2 tok_sm[];                  // [npairs][1024] token pairs: (key << 16 | probability) each
  __shared__ unsigned long long xch[2][SMP_MAX_CLUSTER];
  __shared__ unsigned long long pick[2];
  __shared__ unsigned long long sh[34];
  SmpCtx c;
  c.S = gridDim.x; c.rank = blockIdx.x; c.buf = 0; c.xch = xch; c.sh = sh;
  const int S = c.S, rank = c.rank, row = blockIdx.y, tid = threadIdx.x;
  const bool scaled = p.strategy != 0;
  const int tr = (tid == 0 && trace_block0()) ? trace_begin(4) : -1;
  pdl_sync();

  // ---- one pass over the row: keys (0 = no token / NaN) ----
  // Load latency first: a thread takes up to ten units of four neighbouring tokens -- one 64-bit load for the logits, one 32-bit load for
  // their repetition flags, all of them in flight together -- and only then finishes them (penalty, mask, temperature: same operations and
  // rounding points as token_value()) in a loop of one unit, whose code is short.  Rows off these boundaries are read by pairs, or token by
  // token.  32 rows of 156,940 tokens, cold: 14.3 us with pairs in two turns of straight-line code, 8.7 now.
  const __nv_bfloat16* lrow = p.logits + static_cast<size_t>(row) * p.ld;
  const uint8_t* rep0 = nullptr;
  size_t rep_wstride = 0;
  if (p.rep_cache) {
    const int b0 = row / p.C_logits;
    const int b = p.cache_rows ? p.cache_rows[b0] : b0;
    const int cc = (p.C_logits == 1 && p.C_cache != 1) ? 0 : row % p.C_logits;   // sampling.py:140-141
    rep_wstride = static_cast<size_t>(p.C_cache) * p.vocab;
    rep0 = p.rep_cache + (static_cast<size_t>(b) * p.W * p.C_cache + cc) * p.vocab;
  }
  const uintptr_t odd = (reinterpret_cast<uintptr_t>(lrow) >> 1) | static_cast<uintptr_t>(p.vocab) | reinterpret_cast<uintptr_t>(rep0) | rep_wstride;
  const bool wide = (odd & 3) == 0, even = (odd & 1) == 0;
  const int n_seen = rep0 ? p.W : 0;
  const float inv_temperature = 1.f / p.temperature;
  const uint32_t far_temperature = p.temperature > SMP_DIVISOR_LOW && p.temperature < 0x1p40f ? 0u : SMP_FAR;
  uint32_t kloc = 0u;
  auto tok_index = [&](int j, int half) { return 2 * ((j * S + rank) * SMP_THREADS + tid) + half; };
  {
    constexpr int UNITS = SMP_PAIRS / 2;
    const int n_units = npairs * (SMP_THREADS / 2);
    auto unit_token = [&](int u) {         // first token of unit u: pairs 2 u and 2 u + 1 of the CTA, in (pair, thread) order
      return 2 * (((2 * u / SMP_THREADS) * S + rank) * SMP_THREADS + 2 * u % SMP_THREADS);
    };
    // as they come, into the place of their keys: the loop that finishes them is a short one
    if (even) {
      uint2 lw[UNITS];
      uint32_t sb[UNITS];
#pragma unroll
      for (int q = 0; q < UNITS; ++q) {
        const int u = q * SMP_THREADS + tid, i0 = unit_token(u);
        const bool in = u < n_units && i0 < p.vocab;
        if (wide) {
          lw[q] = in ? __ldg(reinterpret_cast<const uint2*>(lrow + i0)) : make_uint2(0u, 0u);
          sb[q] = in && n_seen ? __ldg(reinterpret_cast<const uint32_t*>(rep0 + i0)) : 0u;
        } else {
          const bool in2 = in && i0 + 2 < p.vocab;
          lw[q].x = in ? __ldg(reinterpret_cast<const uint32_t*>(lrow + i0)) : 0u;
          lw[q].y = in2 ? __ldg(reinterpret_cast<const uint32_t*>(lrow + i0 + 2)) : 0u;
          sb[q] = in && n_seen ? __ldg(reinterpret_cast<const unsigned short*>(rep0 + i0)) : 0u;
          if (in2 && n_seen) sb[q] |= static_cast<uint32_t>(__ldg(reinterpret_cast<const unsigned short*>(rep0 + i0 + 2))) << 16;
        }
      }
#pragma unroll
      for (int q = 0; q < UNITS; ++q) {
        const int u = q * SMP_THREADS + tid;
        if (u < n_units) *reinterpret_cast<uint4*>(&tok_sm[2 * u]) = make_uint4(lw[q].x, lw[q].y, sb[q], 0u);
      }
    } else {          // token by token, eight of them at a time (more cost registers everywhere): 32 rows of 156,941, greedy, 19.6 us one by one in the loop below, 12.6 so
      constexpr int BATCH = 2;
#pragma unroll 1
      for (int q0 = 0; q0 * SMP_THREADS < n_units; q0 += BATCH) {
        uint32_t lw[BATCH][4], sb[BATCH] = {};
#pragma unroll
        for (int q = 0; q < BATCH; ++q)
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            const int u = (q0 + q) * SMP_THREADS + tid, i = unit_token(u) + h;
            lw[q][h] = u < n_units && i < p.vocab ? __ldg(reinterpret_cast<const unsigned short*>(lrow + i)) : 0u;
          }
#pragma unroll 1
        for (int w = 0; w < n_seen; ++w) {
          const uint8_t* rw = rep0 + w * rep_wstride;
#pragma unroll
          for (int q = 0; q < BATCH; ++q)
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int u = (q0 + q) * SMP_THREADS + tid, i = unit_token(u) + h;
              if (u < n_units && i < p.vocab) sb[q] |= static_cast<uint32_t>(__ldg(rw + i)) << (8 * h);
            }
        }
#pragma unroll
        for (int q = 0; q < BATCH; ++q) {
          const int u = (q0 + q) * SMP_THREADS + tid;
          if (u < n_units) *reinterpret_cast<uint4*>(&tok_sm[2 * u]) = make_uint4(lw[q][0] | lw[q][1] << 16, lw[q][2] | lw[q][3] << 16, sb[q], 0u);
        }
      }
    }
    uint32_t kmax2 = 0u;                   // of the even tokens and of the odd ones
    int i0 = unit_token(tid);
#pragma unroll 1
    for (int u = tid; u < n_units; u += SMP_THREADS, i0 += 4 * S * SMP_THREADS) {
      uint4 raw = *reinterpret_cast<const uint4*>(&tok_sm[2 * u]);
      if (even) {
        for (int w = 1; w < n_seen; ++w)
          for (int h = 0; h < 4 && i0 + h < p.vocab; h += 2)
            raw.z |= static_cast<uint32_t>(__ldg(reinterpret_cast<const unsigned short*>(rep0 + w * rep_wstride + i0 + h))) << (8 * h);
      }
      float l[4] = {bf16_lo(raw.x), bf16_hi(raw.x), bf16_lo(raw.y), bf16_hi(raw.y)};
      if (raw.z) {
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (raw.z >> (8 * h) & 0xffu) l[h] = round_bf16(l[h] > 0.f ? smp_quotient(l[h], p.penalty) : l[h] * p.penalty);   // sampling.py:143-144
      }
      if (static_cast<uint32_t>(p.mask_token - i0) < 4u) {
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (p.mask_token - i0 == h) l[h] = -INFINITY;
      }
      if (scaled) {
        float s[4];
        uint32_t far = far_temperature;
#pragma unroll
        for (int h = 0; h < 4; ++h) s[h] = smp_div(l[h], p.temperature, inv_temperature, far);
        if (far >= SMP_FAR) {
#pragma unroll
          for (int h = 0; h < 4; ++h) s[h] = smp_quotient(l[h], p.temperature);
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) l[h] = s[h];
      }
      uint32_t k0 = key_pair(pack_bf16(l[0], l[1])), k1 = key_pair(pack_bf16(l[2], l[3]));
      const float any_nan = (l[0] + l[1]) + (l[2] + l[3]);
      if (any_nan != any_nan || i0 + 4 > p.vocab) {          // (a sum of both infinities is looked at as well)
        uint32_t keep[2] = {0u, 0u};
#pragma unroll
        for (int h = 0; h < 4; ++h)
          if (i0 + h < p.vocab && l[h] == l[h]) keep[h >> 1] |= h & 1 ? 0xffff0000u : 0xffffu;
        k0 &= keep[0];
        k1 &= keep[1];
      }
      *reinterpret_cast<uint4*>(&tok_sm[2 * u]) = make_uint4(k0 << 16, k0 & 0xffff0000u, k1 << 16, k1 & 0xffff0000u);
      kmax2 = max_u16x2(max_u16x2(kmax2, k0), k1);
    }
    kloc = max(kmax2 & 0xffffu, kmax2 >> 16);
  }

  // ---- max key ----
  const uint32_t kmax = static_cast<uint32_t>(smp_reduce<SMP_MAX>(kloc, c));
  // smallest index holding the max key: the greedy answer and the fallback of degenerate rows
  auto first_max_index = [&]() -> unsigned long long {
    unsigned long long best = 0xffffffffull;
#pragma unroll 4
    for (int j = npairs - 1; j >= 0; --j) {
      const uint2 t = tok_sm[j * SMP_THREADS + tid];
      if ((t.y >> 16) == kmax) best = static_cast<unsigned long long>(tok_index(j, 1));
      if ((t.x >> 16) == kmax) best = static_cast<unsigned long long>(tok_index(j, 0));
    }
    const unsigned long long r = smp_reduce<SMP_MIN>(kmax ? best : 0xffffffffull, c);
    return r == 0xffffffffull ? 0ull : r;
  };
  if (p.strategy == 0) {
    const unsigned long long idx = first_max_index();
    if (rank == 0 && tid == 0) p.out[row] = static_cast<int64_t>(idx);
    return;
  }

  // ---- top-k threshold: smallest key k with #{key_i > k} < top_k (ties at the k-th value are kept) ----
  uint32_t k_floor = 0u;
  if (p.strategy == 1 || p.strategy == 3) {
    uint32_t lo = 0u, hi = 65535u;          // invariant: count(> hi) < top_k; count(> lo - 1) >= top_k or lo == 0
    // bisection over [0, 65535] for the smallest k with count(> k) < top_k
#pragma unroll 1
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1, lim = mid << 16 | 0xffffu;      // (no probabilities yet: the low halves are zero)
      uint32_t cnt = 0u;
#pragma unroll 4
      for (int j = 0; j < npairs; ++j) {
        const uint2 t = tok_sm[j * SMP_THREADS + tid];
        cnt += (t.x > lim ? 1u : 0u) + (t.y > lim ? 1u : 0u);
      }
      const unsigned long long tot = smp_reduce<SMP_SUM>(cnt, c);
      if (tot < static_cast<unsigned long long>(p.top_k)) hi = mid; else lo = mid + 1;
    }
    k_floor = lo;
  }
  const uint32_t z_floor = (p.strategy == 3) ? k_floor : 0u;   // top-k-first: the softmax only sees the top-k

  // ---- softmax denominator (fp32) ----
  const float xmax = key_value(kmax);
  float zpart = 0.f;
  const uint32_t z_word = max(z_floor, 1u) << 16;          // (key 0: no token)
#pragma unroll 4
  for (int j = 0; j < npairs; ++j) {
    const uint2 t = tok_sm[j * SMP_THREADS + tid];
    const float ex = smp_ex2((word_value(t.x) - xmax) * kLog2e), ey = smp_ex2((word_value(t.y) - xmax) * kLog2e);
    if (t.x >= z_word) zpart += ex;
    if (t.y >= z_word) zpart += ey;
  }
  const float Z = smp_sum_f32(zpart, c);
  const float log2Z = log2f(Z);

  // ---- probabilities: bf16-rounded softmax output; filtered tokens get 0 ----
  const uint32_t keep_floor = (p.strategy == 1 || p.strategy == 3) ? k_floor : 0u;
  const float minp_thr = (p.strategy == 4) ? p.min_p * round_bf16(smp_ex2(-log2Z)) : 0.f;
  const uint32_t keep_word = max(max(z_floor, keep_floor), 1u) << 16;
  auto probability = [&](uint32_t t) {
    // softmax output e^(x - max) / Z as ONE exponential: 2^((x - max) log2 e - log2 Z)
    const float e = smp_ex2((word_value(t) - xmax) * kLog2e - log2Z);
    return t >= keep_word ? e : 0.f;
  };
  unsigned long long mine = 0ull;           // this thread's share of the candidates' mass
#pragma unroll 4
  for (int j = 0; j < npairs; ++j) {
    uint2 t = tok_sm[j * SMP_THREADS + tid];
    uint32_t pr = pack_bf16(probability(t.x), probability(t.y));
    if (p.strategy == 4) pr = (bf16_lo(pr) >= minp_thr ? pr & 0xffffu : 0u) | (bf16_hi(pr) >= minp_thr ? pr & 0xffff0000u : 0u);
    t.x = __byte_perm(pr, t.x, 0x7610);
    t.y = __byte_perm(pr, t.y, 0x7632);
    tok_sm[j * SMP_THREADS + tid] = t;
    mine += smp_mass(pr);
    mine += __float2uint_rz(bf16_hi(pr) * 4294967296.f);
  }
  // prefixes of the masses over the cluster in (cta, thread, pair) order, and their sum: the candidates' mass
  unsigned long long Mc, lo;
  auto prefix = [&](unsigned long long v) {
    unsigned long long cta_total;
    const unsigned long long excl = block_excl_scan(v, sh, &cta_total);
    if (tid < 32) c.publish(cta_total);
    c.sync();
    unsigned long long base = 0ull, total = 0ull;
    for (int r = 0; r < S; ++r) {
      if (r == rank) base = total;
      total += c.xch[c.buf][r];
    }
    c.buf ^= 1;
    lo = base + excl;
    return total;
  };
  Mc = prefix(mine);
  const uint64_t seed = p.rng_state ? p.rng_state[0] : p.seed;
  const uint64_t offset = p.rng_state ? p.rng_state[1] : p.offset;
  if (Mc == 0ull || !(Z > 0.f)) {
    // degenerate row (everything masked / non-finite): argmax, like the reference's fallthrough
    const unsigned long long idx = first_max_index();
    if (rank == 0 && tid == 0) p.out[row] = static_cast<int64_t>(idx);
  } else {
    const bool nucleus = (p.strategy == 2 || p.strategy == 3);
    unsigned long long P = static_cast<unsigned long long>(static_cast<double>(p.top_p) * 4294967296.0);
    if (P == 0ull) P = 1ull;
    uint32_t pivot = 0u;                     // candidates: key > pivot
    int pb = 0;
    unsigned long long result = 0ull;
#pragma unroll 1
    for (uint32_t round = 0; round < 64u; ++round) {
      // inverse CDF over the candidates
      const double u = philox_uniform(seed, offset, static_cast<uint32_t>(row), round);
      unsigned long long target = static_cast<unsigned long long>(u * static_cast<double>(Mc));
      if (target >= Mc) target = Mc - 1;
      if (mine != 0ull && lo <= target && target < lo + mine) {
        unsigned long long run = lo;
        unsigned long long found = 0ull;
#pragma unroll 1
        for (int j = 0; j < npairs; ++j) {
          const uint2 t = tok_sm[j * SMP_THREADS + tid];
          const uint32_t qx = (t.x >> 16) > pivot ? smp_mass(t.x) : 0u, qy = (t.y >> 16) > pivot ? smp_mass(t.y) : 0u;
          if (target < run + qx) {
            found = (static_cast<unsigned long long>(t.x >> 16) << 32) | static_cast<uint32_t>(tok_index(j, 0));
            break;
          }
          run += qx;
          if (target < run + qy) {
            found = (static_cast<unsigned long long>(t.y >> 16) << 32) | static_cast<uint32_t>(tok_index(j, 1));
            break;
          }
          run += qy;
        }
        if (S == 1) pick[pb] = found;
        else for (int r = 0; r < S; ++r) st_dsmem_u64(&pick[pb], r, found);
      }
      c.sync();
      result = pick[pb];
      pb ^= 1;
      if (!nucleus) break;
      const uint32_t kj = static_cast<uint32_t>(result >> 32);
      mine = 0ull;                           // what lies above j: this thread's share of the next round, should there be one
#pragma unroll 4
      for (int j = 0; j < npairs; ++j) {
        const uint2 t = tok_sm[j * SMP_THREADS + tid];
        if ((t.x >> 16) > kj) mine += smp_mass(t.x);
        if ((t.y >> 16) > kj) mine += smp_mass(t.y);
      }
      const unsigned long long above = prefix(mine);
      if (above < P) break;                  // j is inside the nucleus: accept
      pivot = kj;                            // nothing with p <= p_j is: drop it and redraw
      Mc = above;
    }
    if (rank == 0 && tid == 0) p.out[row] = static_cast<int64_t>(result & 0xffffffffull);
  }
  // advance the device RNG offset once per call: the last row to get here (every row read the offset above,
  // before its final cluster barrier)
  if (p.rng_state && rank == 0 && tid == 0) {
    const unsigned long long old = atomicAdd(&p.rng_state[2], 1ull);
    if (old == static_cast<unsigned long long>(gridDim.y) - 1ull) {
      p.rng_state[2] = 0ull;
      p.rng_state[1] = offset + 1ull;
    }
  }
  trace_end(tr);
}

// Standard normal draws (SNAC NoiseBlock input, vox_serve/tokenizer/snac.py:208 uses torch.randn): one Philox4x32-10
// block per 4 outputs, counter = (offset, quad index), two Box-Muller pairs.  With a device state {seed, offset,
// arrivals} the offset advances by one per launch (last block to arrive), so CUDA-graph replays keep drawing.
__global__ void __launch_bounds__(256) randn_kernel(float* __restrict__ out, long long n, unsigned long long seed_,
                                                    unsigned long long offset_, unsigned long long* state) {
  pdl_sync();
  const unsigned long long seed = state ? state[0] : seed_, offset = state ? state[1] : offset_;
  const long long q = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (q * 4 < n) {
    uint32_t c[4] = {static_cast<uint32_t>(offset), static_cast<uint32_t>(offset >> 32), static_cast<uint32_t>(q),
                     static_cast<uint32_t>(static_cast<unsigned long long>(q) >> 32) ^ 0x5eed0000u};
    uint32_t k0 = static_cast<uint32_t>(seed), k1 = static_cast<uint32_t>(seed >> 32);
#pragma unroll
    for (int r = 0; r < 10; ++r) {
      philox_round(c, k0, k1);
      k0 += 0x9E3779B9u;
      k1 += 0xBB67AE85u;
    }
    float z[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // u1 in (0, 1], u2 in [0, 1): 2^-32 granularity (torch's curand path uses the same resolution)
      const float u1 = (static_cast<float>(c[2 * h]) + 1.0f) * 2.3283064365386963e-10f;
      const float u2 = static_cast<float>(c[2 * h + 1]) * 2.3283064365386963e-10f;
      const float rad = sqrtf(-2.0f * logf(u1));
      float s, co;
      sincospif(2.0f * u2, &s, &co);
      z[2 * h] = rad * co;
      z[2 * h + 1] = rad * s;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (q * 4 + j < n) out[q * 4 + j] = z[j];
  }
  if (state) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const unsigned long long old = atomicAdd(&state[2], 1ull);
      if (old == static_cast<unsigned long long>(gridDim.x) - 1ull) {
        state[2] = 0ull;
        state[1] = offset + 1ull;
      }
    }
  }
}

__global__ void penalty_kernel(__nv_bfloat16* out, const SampleParams p) {
  const int row = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < p.vocab; i += gridDim.x * blockDim.x)
    out[static_cast<size_t>(row) * p.vocab + i] = __float2bfloat16_rn(token_value(p, row, i, false));
}

// window > 1: cache[:, :-1] = cache[:, 1:]; cache[:, -1] = 0   (sampling.py:166-168)
__global__ void rep_shift_kernel(uint8_t* cache, const int32_t* cache_rows, int B, int W, size_t plane /*C*V*/) {
  pdl_sync();
  const size_t n = static_cast<size_t>(B) * plane;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t b0 = i / plane, r = i - b0 * plane;
    const size_t b = cache_rows ? static_cast<size_t>(cache_rows[b0]) : b0;
    uint8_t* base = cache + b * W * plane + r;
    for (int w = 0; w + 1 < W; ++w) base[w * plane] = base[(w + 1) * plane];
    base[(W - 1) * plane] = 0;
  }
}
// cache[b, w(s), c(s), ids[b', c']] = 1 for every b and every (b', c')   (sampling.py:169-178)
__global__ void rep_mark_kernel(uint8_t* cache, const int32_t* cache_rows, const int64_t* ids, int B, int W, int C,
                                int V, int C_ids, int windowed) {
  pdl_sync();
  const int n_ids = B * C_ids;
  const bool cb0_only = (C_ids == 1 && C != 1);
  const int w_lo = windowed ? W - 1 : 0, w_hi = W;
  const int c_lo = 0, c_hi = cb0_only ? 1 : C;
  const int per_b = (w_hi - w_lo) * (c_hi - c_lo) * n_ids;
  const long long total = static_cast<long long>(B) * per_b;
  for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < total;
       t += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int b0 = static_cast<int>(t / per_b);
    int r = static_cast<int>(t - static_cast<long long>(b0) * per_b);
    const int b = cache_rows ? cache_rows[b0] : b0;
    const int j = r % n_ids; r /= n_ids;
    const int c = c_lo + r % (c_hi - c_lo); r /= (c_hi - c_lo);
    const int w = w_lo + r;
    long long id = ids[j];
    if (id < 0) id += V;
    if (id >= 0 && id < V) cache[((static_cast<size_t>(b) * W + w) * C + c) * V + id] = 1;
  }
}

}  // namespace vb

using namespace vb;

extern "C" {

size_t vb_sample_workspace_bytes(int rows, int vocab) {
  (void)vocab; (void)rows;
  return 256;   // the sampler keeps the row on chip; the workspace is kept in the ABI for callers that size it
}

static int fill_params(SampleParams& p, int64_t* d_out_ids, const void* d_logits, int rows, int vocab, int ld,
                       const uint8_t* d_rep_cache, int W, int C_cache, int C_logits, float penalty, int strategy,
                       int top_k, float top_p, float min_p, float temperature, uint64_t seed, uint64_t offset,
                       int mask_token, void* ws, uint64_t* rng_state = nullptr, const int32_t* cache_rows = nullptr) {
  p.logits = static_cast<const __nv_bfloat16*>(d_logits);
  p.rep_cache = d_rep_cache;
  p.cache_rows = cache_rows;
  p.rows = rows; p.vocab = vocab; p.ld = ld;
  p.W = W; p.C_cache = C_cache; p.C_logits = C_logits > 0 ? C_logits : 1;
  p.penalty = penalty; p.temperature = temperature;
  p.strategy = strategy; p.top_k = top_k; p.top_p = top_p; p.min_p = min_p;
  p.mask_token = mask_token; p.seed = seed; p.offset = offset;
  p.rng_state = reinterpret_cast<unsigned long long*>(rng_state);
  (void)ws;
  p.out = d_out_ids;
  return 0;
}

int vb_sample(int64_t* d_out_ids, const void* d_logits, int rows, int vocab, int ld_logits,
              const uint8_t* d_rep_cache, const int32_t* d_cache_rows, int rep_window_slots, int rep_codebooks,
              int logit_codebooks,
              float penalty, int strategy, int top_k, float top_p, float min_p, float temperature, uint64_t seed,
              uint64_t offset, uint64_t* d_rng_state, int mask_token, void* d_workspace, size_t workspace_bytes,
              void* stream) {
  VB_CHECK_ARG(d_out_ids && d_logits && d_workspace, "vb_sample: null pointer");
  VB_CHECK_ARG(strategy >= 0 && strategy <= 4, "vb_sample: strategy %d", strategy);
  VB_CHECK_ARG(workspace_bytes >= vb_sample_workspace_bytes(rows, vocab), "vb_sample: workspace too small");
  VB_CHECK_ARG(strategy == 0 || temperature > 0.f, "vb_sample: temperature must be > 0 for stochastic sampling");
  VB_CHECK_ARG(!(strategy == 1 || strategy == 3) || top_k > 0, "vb_sample: top_k must be > 0");
  VB_CHECK_ARG(!d_rep_cache || (rep_window_slots > 0 && rep_codebooks > 0), "vb_sample: bad repetition cache dims");
  if (rows <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SampleParams p;
  fill_params(p, d_out_ids, d_logits, rows, vocab, ld_logits, d_rep_cache, rep_window_slots, rep_codebooks,
              logit_codebooks, penalty, strategy, top_k, top_p, min_p, temperature, seed, offset, mask_token,
              d_workspace, d_rng_state, d_cache_rows);
  // smallest cluster (1, 2, 4 or 8 CTAs) whose threads can hold the row on chip
  int S = 1;
  while (S < SMP_MAX_CLUSTER && static_cast<long long>(S) * SMP_THREADS * 2 * SMP_PAIRS < vocab) S <<= 1;
  VB_CHECK_ARG(static_cast<long long>(S) * SMP_THREADS * 2 * SMP_PAIRS >= vocab,
               "vb_sample: vocab %d exceeds the %d tokens one cluster holds on chip", vocab,
               SMP_MAX_CLUSTER * SMP_THREADS * 2 * SMP_PAIRS);
  VB_CHECK_ARG(rows <= 65535, "vb_sample: %d rows exceed the grid limit (65535)", rows);
  const int npairs = (vocab + S * SMP_THREADS * 2 - 1) / (S * SMP_THREADS * 2);
  const size_t smem = static_cast<size_t>(2 * npairs) * SMP_THREADS * sizeof(uint32_t);
  // (static shared memory counts against the same 227 KiB: leave room for it)
  VB_CHECK_CUDA(cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     2 * SMP_PAIRS * SMP_THREADS * static_cast<int>(sizeof(uint32_t))));
  VB_LAUNCH_PDL_CLUSTER(sample_kernel, dim3(S, rows), SMP_THREADS, smem, st, S, p, npairs);
  return 0;
}

int vb_randn(float* d_out, int64_t n, uint64_t seed, uint64_t offset, uint64_t* d_rng_state, void* stream) {
  VB_CHECK_ARG(d_out, "vb_randn: null pointer");
  VB_CHECK_ARG(n >= 0 && n < (static_cast<int64_t>(1) << 40), "vb_randn: bad element count");
  if (n == 0) return 0;
  const long long quads = (n + 3) / 4;
  const unsigned blocks = static_cast<unsigned>((quads + 255) / 256);
  VB_LAUNCH_PDL(randn_kernel, blocks, 256, 0, stream, d_out, static_cast<long long>(n), seed, offset,
                reinterpret_cast<unsigned long long*>(d_rng_state));
  return 0;
}

int vb_apply_repetition_penalty(void* d_out, const void* d_logits, const uint8_t* d_rep_cache,
                                int rep_window_slots, int rep_codebooks, int logit_codebooks, float penalty,
                                int rows, int vocab, void* stream) {
  VB_CHECK_ARG(d_out && d_logits && d_rep_cache, "vb_apply_repetition_penalty: null pointer");
  if (rows <= 0) return 0;
  SampleParams p;
  fill_params(p, nullptr, d_logits, rows, vocab, vocab, d_rep_cache, rep_window_slots, rep_codebooks,
              logit_codebooks, penalty, 0, 0, 0.f, 0.f, 1.f, 0, 0, -1, nullptr);
  const int gx = max(1, min(64, (vocab + 255) / 256));
  VB_LAUNCH_PLAIN(penalty_kernel, dim3(gx, rows), 256, 0, stream, static_cast<__nv_bfloat16*>(d_out), p);
  return 0;
}

int vb_update_repetition_cache(uint8_t* d_cache, const int32_t* d_cache_rows, const int64_t* d_ids, int B, int W,
                               int C, int V, int C_ids, int window, void* stream) {
  VB_CHECK_ARG(d_cache && d_ids, "vb_update_repetition_cache: null pointer");
  VB_CHECK_ARG(B > 0 && W > 0 && C > 0 && V > 0 && C_ids > 0, "vb_update_repetition_cache: bad dims");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int windowed = window > 1;
  if (windowed) {
    const size_t plane = static_cast<size_t>(C) * V;
    size_t nb = (static_cast<size_t>(B) * plane + 255) / 256; if (nb > 4096) nb = 4096; const unsigned blocks = static_cast<unsigned>(nb);
    VB_LAUNCH_PDL(rep_shift_kernel, blocks, 256, 0, st, d_cache, d_cache_rows, B, W, plane);
  }
  VB_LAUNCH_PDL(rep_mark_kernel, 64, 256, 0, st, d_cache, d_cache_rows, d_ids, B, W, C, V, C_ids, windowed);
  return 0;
}

}  // extern "C"

VB_DEFINE_TRACE_SETTER(sampler)
