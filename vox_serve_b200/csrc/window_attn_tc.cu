// Prompt portions of the text LMs' window attention on tcgen05 (bf16, key and value heads of one size, 64 or 128): the masks,
// sink, gates and cache forms of vb_window_attn_tiled on the attention core of attn_tc.cuh.
//
// A CTA owns TQ = min(64, 128 / R) rows of one request x the R query heads of ONE key head (accumulator row r: prompt row r / R,
// head r % R), so a group's K / V tiles are fetched once for all its heads; the mma.sync tiles of window_attn.cu take one query
// head each.  A row tile of 64 is dealt to ceil(64 / TQ) CTAs.  Keys are walked in tiles of 64 positions: first those with kept
// tokens, then from the tile of the first key that the CTA's first row sees; within a tile the mask is per key.  What lies between the two is
// nobody's to read (a page table may name other requests' pages there, or unwritten ones): its boxes are skipped, its V rows cleared.
// Measured (16 query heads on 4 key heads of 128, two prompts of 1001 rows in all): the three-layer prompt step around it 1058 us with
// mma.sync, 884 here (724 with the steps around it since, 720 with a loading warp each for K and V).
#include "../../include/vb_api.h"
#define VB_PDL_FAMILY 1
#include "attn_tc.cuh"

namespace vb {

struct WindowTcParams {
  const __nv_bfloat16* q;        // [T][H][D]
  void* out;                     // [T][H * D] bf16 or fp32
  const float* gate;
  const int32_t* pos;
  const int32_t* page_indptr;
  const int32_t* page_indices;
  const int32_t* qo_indptr;
  const int32_t* tile_req;
  const int32_t* tile_row0;
  const float* sink;             // [H] or nullptr
  int ld_gate, H, G, R, TQ, subs, page_size, window, chunk, keep, v_share, out_f32, head_gate, box_tokens;
  float scale_log2;
  unsigned char* wait_flag;
};

__device__ __forceinline__ void wtc_tma_4d(uint32_t dst, const CUtensorMap* m, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

struct WindowRows {
  static constexpr bool HOLE = true, STAGED = false;
  const WindowTcParams& p;
  int n_tiles, n0, t1;           // tiles 0 .. n0 - 1 hold kept tokens, the rest start at t1
  int hole0, hole1;              // between the kept tokens and the first key that the block's first row sees
  int pos, lo, row, head, D;
  int row0, nrows, head0, group;
  bool ok;
  float scale_log2;
  __device__ __forceinline__ int tile(int it) const { return it < n0 ? it : t1 + (it - n0); }
  __device__ __forceinline__ bool full(int tok0) const { return ok && tok0 + PTC_KT - 1 <= pos && tok0 >= lo; }
  __device__ __forceinline__ bool visible(int kj) const { return ok && kj <= pos && (kj >= lo || kj < p.keep); }
  __device__ __forceinline__ const __nv_bfloat16* q_row(int t, int g) const {
    return t < nrows ? p.q + (static_cast<size_t>(row0 + t) * p.H + head0 + g) * D : nullptr;
  }
  __device__ __forceinline__ uint4* out_at(int, int, int) const { return nullptr; }
  // a sink is one more term of the denominator, a key without a value
  __device__ __forceinline__ float finish(float m_ref, float l) const {
    if (!ok) return 0.f;
    if (!p.sink) return l > 0.f ? 1.f / l : 0.f;
    const float s = p.sink[head] * 1.4426950408889634f, M = fmaxf(m_ref, s), c = exp2f(m_ref - M);
    return c / (l * c + exp2f(s - M));
  }
  __device__ __forceinline__ void store(int c0, const uint32_t (&o)[32], float f) const {
    if (!ok) return;
    const size_t at = (static_cast<size_t>(row) * p.H + head) * D + c0;
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(o[i]) * f;
    if (p.gate) {
      const float* g = p.gate + static_cast<size_t>(row) * p.ld_gate + (p.head_gate ? head : head * D + c0);
      if (p.head_gate) {
        const float w = 1.f / (1.f + expf(-__ldg(g)));
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] *= w;
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] *= 1.f / (1.f + expf(-__ldg(g + i)));
      }
    }
    if (p.out_f32) {
      float4* y = reinterpret_cast<float4*>(static_cast<float*>(p.out) + at);
#pragma unroll
      for (int c = 0; c < 8; ++c) y[c] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    } else {
      uint4* y = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.out) + at);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        y[c] = make_uint4(pack_bf16(v[8 * c], v[8 * c + 1]), pack_bf16(v[8 * c + 2], v[8 * c + 3]), pack_bf16(v[8 * c + 4], v[8 * c + 5]),
                          pack_bf16(v[8 * c + 6], v[8 * c + 7]));
    }
  }
};

template <int D>
__global__ void __launch_bounds__(PTC_THREADS, 2) window_attn_tc_kernel(const WindowTcParams p, const __grid_constant__ CUtensorMap k_map,
                                                                        const __grid_constant__ CUtensorMap v_map) {
  using L = PtcLayout<D>;
  extern __shared__ uint8_t wtc_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(wtc_smem_raw) + 1023) & ~uintptr_t(1023));
  PtcShared* sh = reinterpret_cast<PtcShared*>(smem + L::BAR);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  BoundedWait bw{p.wait_flag};
  if (tid == 0) {
    ptc_init(sh, 1);
    prefetch_tmap(&k_map);
    prefetch_tmap(&v_map);
  }
  if (warp == 4) {
    tmem_alloc(&sh->tmem, 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem;
  pdl_sync();

  // later tiles of a prompt see more keys: they are started first so that the short ones fill the tail
  const int unit = gridDim.x - 1 - blockIdx.x, ti = unit / p.subs, b = p.tile_req[ti], g = blockIdx.y;
  const int row0 = p.tile_row0[ti] + (unit - ti * p.subs) * p.TQ;
  const int nrows = min(min(row0 + p.TQ, p.tile_row0[ti] + 64), p.qo_indptr[b + 1]) - row0;
  if (nrows > 0) {
    auto first_key = [&](int ps) {
      int lo = p.window > 0 ? max(0, ps - p.window + 1) : 0;
      return p.chunk > 0 ? max(lo, ps - ps % p.chunk) : lo;
    };
    const int pos0 = p.pos[row0], kmax = pos0 + nrows, lo0 = first_key(pos0);
    const int n0 = (min(p.keep, lo0) + PTC_KT - 1) / PTC_KT, t1 = max(lo0 / PTC_KT, n0), n_tiles = n0 + (kmax + PTC_KT - 1) / PTC_KT - t1;
    const int t = tid / p.R;
    const bool ok = warp < 4 && t < nrows;
    const WindowRows rows{p, n_tiles, n0, t1, min(p.keep, lo0), lo0, pos0 + t, first_key(pos0 + t), row0 + t, g * p.R + tid - t * p.R, D, row0, nrows, g * p.R, p.R, ok, p.scale_log2};
    if (warp < 4) {
      ptc_softmax<D>(smem, sh, rows, bw);
    } else if (warp == 4) {
      ptc_issue<D>(smem, sh, n_tiles, bw);
    } else {
      const int pbase = p.page_indptr[b], gv = g / p.v_share;
      auto place = [&](int tok) {
        const int i = tok / p.page_size;
        return make_int2(__ldg(&p.page_indices[pbase + i]), tok - i * p.page_size);
      };
      if (warp == 5)
        ptc_load_k<D>(smem, sh, rows, kmax, p.box_tokens, bw, place,
                      [&](int page, int slot, uint32_t dst, int dim, uint32_t bar) { wtc_tma_4d(dst, &k_map, bar, dim, g, slot, page); });
      else
        ptc_load_v<D>(smem, sh, rows, kmax, p.box_tokens, bw, place,
                      [&](int page, int slot, uint32_t dst, int dim, uint32_t bar) { wtc_tma_4d(dst, &v_map, bar, dim, gv, slot, page); });
      __syncwarp();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// one head size for keys and values, 64 or 128; pages of whole 8-token groups; rows that a tensor map can step over
bool window_attn_tc_takes(int H, int G, int dim, int vdim, int page_size, int k_ld, int v_ld, const void* q, const void* k, const void* v,
                          const void* out) {
  auto aligned = [](const void* x) { return reinterpret_cast<uintptr_t>(x) % 16 == 0; };
  return dim == vdim && (dim == 64 || dim == 128) && H / G <= 128 && page_size % 8 == 0 && k_ld % 8 == 0 && v_ld % 8 == 0 && aligned(q) &&
         aligned(k) && aligned(v) && aligned(out) && encode_fn() != nullptr;
}

int window_attn_tc(void* out, const void* q, const void* k_cache, const void* v_cache, const float* gate, int ld_gate, const int32_t* pos,
                   const int32_t* page_indptr, const int32_t* page_indices, const int32_t* qo_indptr, const int32_t* tile_req,
                   const int32_t* tile_row0, int n_tiles, int H, int G, int dim, int page_size, int window, float scale, int chunk, int k_ld,
                   int v_ld, int v_share, int out_f32, const float* sink, int keep_first, int head_gate, cudaStream_t stream) {
  WindowTcParams p{};
  VB_CHECK_ARG(p.wait_flag = wait_flag(WK_WINDOW_ATTN), "vb_window_attn_tiled: no mapped host memory");
  p.q = static_cast<const __nv_bfloat16*>(q); p.out = out; p.gate = gate; p.pos = pos; p.page_indptr = page_indptr;
  p.page_indices = page_indices; p.qo_indptr = qo_indptr; p.tile_req = tile_req; p.tile_row0 = tile_row0; p.sink = sink;
  p.ld_gate = ld_gate; p.H = H; p.G = G; p.R = H / G; p.TQ = min(64, 128 / p.R); p.subs = (64 + p.TQ - 1) / p.TQ;
  p.page_size = page_size; p.window = window; p.chunk = chunk; p.keep = keep_first; p.v_share = v_share; p.out_f32 = out_f32;
  p.head_gate = head_gate; p.box_tokens = ptc_box_tokens(page_size); p.scale_log2 = scale * 1.4426950408889634f;
  CUtensorMap maps[2];
  for (int i = 0; i < 2; ++i) {
    const cuuint64_t D = dim, P = page_size, ld = i ? v_ld : k_ld, heads = i ? G / v_share : G;
    cuuint64_t dims[4] = {D, heads, P, 1ull << 30};     // how many pages there are is the caller's: every box starts at a page of the table
    cuuint64_t strides[3] = {D * 2, ld * 2, P * ld * 2};
    cuuint32_t box[4] = {64, 1, static_cast<cuuint32_t>(p.box_tokens), 1}, estr[4] = {1, 1, 1, 1};
    const CUresult r = encode_fn()(&maps[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(i ? v_cache : k_cache), dims, strides, box,
                                   estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    VB_CHECK_ARG(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled(window cache) failed: CUresult %d", static_cast<int>(r));
  }
  const dim3 grid(n_tiles * p.subs, G);
  if (dim == 128) {
    VB_CHECK_CUDA(cudaFuncSetAttribute(window_attn_tc_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, PtcLayout<128>::TOTAL));
    VB_LAUNCH_PDL(window_attn_tc_kernel<128>, grid, PTC_THREADS, PtcLayout<128>::TOTAL, stream, p, maps[0], maps[1]);
  } else {
    VB_CHECK_CUDA(cudaFuncSetAttribute(window_attn_tc_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, PtcLayout<64>::TOTAL));
    VB_LAUNCH_PDL(window_attn_tc_kernel<64>, grid, PTC_THREADS, PtcLayout<64>::TOTAL, stream, p, maps[0], maps[1]);
  }
  return 0;
}

}  // namespace vb

extern "C" int vb_window_attn_tc_timeouts(void) {
  return vb::wait_ran_out(vb::WK_WINDOW_ATTN);
}
