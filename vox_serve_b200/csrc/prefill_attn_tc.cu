// Tiled paged prefill attention on the 5th-generation tensor cores (tcgen05 + TMEM): the FlashAttention schedule of
// prefill_attn.cu with both contractions issued as tcgen05.mma and their accumulators in tensor memory.  Same inputs, same
// result contract (FlashInferPrefillWrapper.run, flashinfer_utils.py:68-80, 132).
//
//  * a CTA owns (Q tile, kv head).  The Q tile is M = 128 accumulator rows = TQ = 128 / G consecutive prompt rows of ONE
//    request x the G grouped query heads of the kv head (row r = token r / G, head r % G): the GQA group rides in the MMA's
//    M dimension, so a K/V tile is fetched once for all of them;
//  * warps 0..3 are the softmax: thread r owns accumulator row r = TMEM lane r.  It reads its 64 scores at once, keeps the
//    running maximum and denominator in registers (no shuffles: a row is one thread) and writes its probabilities (bf16) over
//    the scores in TMEM, where they are the A operand of O += P V;
//  * O stays in TMEM for the whole sequence.  The maximum that the exponents are taken against is only moved when a row's
//    maximum has grown by more than 8 (base 2), and only then is O rescaled.  Probabilities stay below 2^8 but a row's largest is no
//    longer 1, which bf16 holds exactly (error before the output's own rounding 6.0e-4 -> 1.03e-3 for scores of standard deviation 3), so
//    they are multiplied as two bf16 terms, rounding and remainder, side by side where the scores were.  997 rows on cached tokens, error
//    after the output's rounding / a plan of two layers: 1.94e-3 / 89 us with one term and the lag, 1.92e-3 / 101 us with one term and
//    the exact maximum (most tiles rescale), 1.59e-3 / 102 us with two terms and the lag;
//  * warp 4 issues the MMAs: the scores of tile j + 1 are multiplied while the softmax works on tile j (two score buffers);
//  * warp 5 brings K tiles and warp 6 V tiles as boxes of a tensor map over the paged cache (pages of a multiple of 8 tokens; cp.async
//    per token row otherwise), the 128-byte-swizzled images that the MMAs read.  V is
//    the B operand of P V as it lies in memory, [token][dim] (MN-major): nothing is transposed.
// 98 KB of shared memory and 256 TMEM columns per CTA: two CTAs share an SM and fill each other's waits.
// The form before this one had one warp group for everything -- loads, an element-wise transpose of every V tile, softmax, both
// waits on the tensor cores -- one after the other (2.5 us per 64-token tile), and the kernel for smaller prompts ran on
// mma.sync.  Measured per launch (mma.sync / this kernel, us, back to back): one 133-row prompt 12.0 / 10.3, eight of them 29 / 13,
// four portions of 997 rows, two of them on some 1000 cached tokens, 88 / 33, three prompts of 1024 rows each 186 / 53, four of 600 with 64-wide
// heads 74 / 31.
// Query rows come and results leave in whole rows, a few neighbouring threads each (a row per thread took 6 us until the rows were there and 3 us
// at the end of a launch of cold data, 2 and 2 now).  The 997 rows above: 45 us a layer of cold data, 36 with whole rows.
// A row's result depends on its own request alone, whatever else is in the step and whichever portion it comes in: the tiles of its keys are
// walked in order by one block.  (Sharing them between two blocks where a launch leaves room, 26 us, moved its roundings with its neighbours.)
// What bounds it: the serial chain of a tile (scores -> maximum -> exponentials -> P V, 0.95 us whatever the pages; 1.02 in pages of 128 keys and 2.1 in pages
// of 16 when one lane looked up and fetched K and V box by box), some 5 us around it.  Two softmax threads a row, 32 scores each, change nothing: 0.95
// us alone, 38.8 us instead of 37.3 for the 997 rows above.
// Every wait is bounded (BoundedWait): a block whose wait runs out sets its flag, stops issuing and leaves.
#include "../../include/vb_api.h"
#define VB_PDL_FAMILY 1
#include "attn_tc.cuh"

namespace vb {

struct PrefillTcParams {
  __nv_bfloat16* out;
  const __nv_bfloat16* q;
  const __nv_bfloat16* kv;       // whole cache [slabs][2][page_size][n_kv][D]
  const int32_t* qo_indptr;      // [n_req + 1]
  const int32_t* kv_indptr;      // [n_req + 1]
  const int32_t* kv_indices;
  const int32_t* row_kvlen;      // [n_rows] keys visible to the row
  int slab_base;
  int n_req, n_rows, n_q, n_kv, G, TQ, page_size;
  int out_xt_tile;
  int box_tokens;
  float scale_log2;
  unsigned char* wait_flag;
};

// what this thread's row sees: the first kl keys of its request
struct PagedRows {
  static constexpr bool HOLE = false, STAGED = true;
  static constexpr int hole0 = 0, hole1 = 0;
  const PrefillTcParams& p;
  int n_tiles, kl, row0, nrows, head0, group, D;
  float scale_log2;
  __device__ __forceinline__ int tile(int it) const { return it; }
  __device__ __forceinline__ bool full(int tok0) const { return tok0 + PTC_KT <= kl; }
  __device__ __forceinline__ bool visible(int kj) const { return kj < kl; }
  __device__ __forceinline__ const __nv_bfloat16* q_row(int t, int g) const {
    return t < nrows ? p.q + (static_cast<size_t>(row0 + t) * p.n_q + head0 + g) * D : nullptr;
  }
  __device__ __forceinline__ float finish(float, float l) const { return l > 0.f ? 1.f / l : 0.f; }
  __device__ __forceinline__ void store(int, const uint32_t (&)[32], float) const {}
  __device__ __forceinline__ uint4* out_at(int t, int g, int c) const {
    if (t >= nrows) return nullptr;
    const int row = row0 + t, e = (head0 + g) * D + c * 8;
    const size_t at = p.out_xt_tile ? xt_index(row, e, p.out_xt_tile, (p.n_q * D + 63) >> 6) : static_cast<size_t>(row) * p.n_q * D + e;
    return reinterpret_cast<uint4*>(p.out + at);
  }
};

template <int D, bool TMA>
__global__ void __launch_bounds__(PTC_THREADS, 2) paged_prefill_attn_tc_kernel(const PrefillTcParams p,
                                                                               const __grid_constant__ CUtensorMap kv_map) {
  using L = PtcLayout<D>;
  constexpr int CPR = D * 2 / 16;      // 16-byte chunks per K / V row
  extern __shared__ uint8_t ptc_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ptc_smem_raw) + 1023) & ~uintptr_t(1023));
  PtcShared* sh = reinterpret_cast<PtcShared*>(smem + L::BAR);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  BoundedWait bw{p.wait_flag};
  if (tid == 0) {
    ptc_init(sh, TMA ? 1 : 64);
    if (TMA) prefetch_tmap(&kv_map);
  }
  if (warp == 4) {
    tmem_alloc(&sh->tmem, 256);                   // scores at 0 and 64, O at 128
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem;
  pdl_sync();

  // rows beyond the last request (CUDA-graph padding) produce zeros
  const int hk = blockIdx.x;                        // key heads fastest
  if (blockIdx.x == 0) {
    const int n_valid = p.qo_indptr[p.n_req];
    for (int row = n_valid + blockIdx.y; row < p.n_rows && blockIdx.z == 0; row += gridDim.y)
      for (int i = tid; i < p.n_q * D / 8; i += PTC_THREADS) {
        const int e = i * 8;
        const size_t o = p.out_xt_tile ? xt_index(row, e, p.out_xt_tile, (p.n_q * D + 63) >> 6)
                                       : static_cast<size_t>(row) * p.n_q * D + e;
        *reinterpret_cast<uint4*>(p.out + o) = make_uint4(0u, 0u, 0u, 0u);
      }
  }

  // ---- which (request, rows) is this block's tile?  prefix sum of ceil(n_new / TQ) over the requests.  Blocks take the tiles
  // from the last one back: late rows see the most keys, and the longest tiles should not start last ----
  const int TQ = p.TQ, b = static_cast<int>(gridDim.y * gridDim.z - 1 - (blockIdx.z * gridDim.y + blockIdx.y));
  int base = 0;
  for (int r0 = 0; r0 < p.n_req; r0 += PTC_THREADS) {
    __syncthreads();
    const int r = r0 + tid;
    int nt = 0, row0 = 0, nnew = 0;
    if (r < p.n_req) {
      row0 = p.qo_indptr[r];
      nnew = p.qo_indptr[r + 1] - row0;
      nt = (nnew + TQ - 1) / TQ;
    }
    int incl = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    if (lane == 31) sh->warp_tot[warp] = incl;
    __syncthreads();
    int woff = 0, tot = 0;
    for (int w = 0; w < PTC_THREADS / 32; ++w) {
      const int v = sh->warp_tot[w];
      if (w < warp) woff += v;
      tot += v;
    }
    const int excl = base + woff + incl - nt;
    if (nt > 0 && b >= excl && b < excl + nt) {
      sh->tile[0] = r;
      sh->tile[1] = row0 + (b - excl) * TQ;
      sh->tile[2] = min(TQ, nnew - (b - excl) * TQ);
    }
    base += tot;
  }
  __syncthreads();
  const int req = sh->tile[0];
  if (req >= 0) {
    const int row0 = sh->tile[1], nrows = sh->tile[2];
    // the tile's largest bound (the bounds do not decrease inside a request: the last row's)
    const int kmax = p.row_kvlen[row0 + nrows - 1];
    const int n_tiles = (kmax + PTC_KT - 1) / PTC_KT;
    const int t = tid / p.G;                      // (softmax) this thread's accumulator row: prompt row t of the tile, head tid % G
    const bool ok = warp < 4 && t < nrows;
    const PagedRows rows{p, n_tiles, ok ? p.row_kvlen[row0 + t] : 0, row0, nrows, hk * p.G, p.G, D, p.scale_log2};
    if (warp < 4) {
      ptc_softmax<D>(smem, sh, rows, bw);
    } else if (warp == 4) {
      ptc_issue<D>(smem, sh, n_tiles, bw);
    } else if (TMA) {
      const int pbase = p.kv_indptr[req];
      auto place = [&](int tok) {
        const int i = tok / p.page_size;
        return make_int2(__ldg(&p.kv_indices[pbase + i]), tok - i * p.page_size);
      };
      auto box = [&](int is_v) {
        return [&, is_v](int page, int slot, uint32_t dst, int dim, uint32_t bar) { ptc_tma_5d(dst, &kv_map, bar, dim, hk, slot, is_v, p.slab_base + page); };
      };
      if (warp == 5) ptc_load_k<D>(smem, sh, rows, kmax, p.box_tokens, bw, place, box(0));
      else ptc_load_v<D>(smem, sh, rows, kmax, p.box_tokens, bw, place, box(1));
      __syncwarp();
    } else {
      // ================= loaders for pages that do not divide into 8-token groups: one token's K / V row per thread =================
      const int ltok = tid - 160, pbase = p.kv_indptr[req];
      const size_t page_elems = static_cast<size_t>(p.page_size) * p.n_kv * D;
      auto fetch = [&](int j, int is_v) {
        const int tok = j * PTC_KT + ltok;
        const uint32_t dst = smem_u32(smem + (is_v ? L::V : L::K) + (j & 1) * L::TILE) + ltok * 128;
        if (tok < kmax) {
          const int page = __ldg(&p.kv_indices[pbase + tok / p.page_size]);
          const __nv_bfloat16* src = p.kv + (static_cast<size_t>(p.slab_base + page) * 2 + is_v) * page_elems +
                                     (static_cast<size_t>(tok % p.page_size) * p.n_kv + hk) * D;
#pragma unroll
          for (int ch = 0; ch < CPR; ++ch) {
            ptc_cp_async16(dst + (ch >> 3) * (PTC_KT * 128) + (((ch & 7) ^ (ltok & 7)) << 4), src + ch * 8);
          }
        } else {                       // rows past the last key are multiplied by probability 0: they must be finite
#pragma unroll
          for (int ch = 0; ch < CPR; ++ch) {
            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(dst + (ch >> 3) * (PTC_KT * 128) + (((ch & 7) ^ (ltok & 7)) << 4)),
                         "r"(0) : "memory");
          }
        }
        ptc_cp_commit();
      };
      // K(j) and V(j) are requested one after the other; a tile is announced once a later group is in flight behind it
      for (int j = 0; j < n_tiles && !bw.dead; ++j) {
        bw.wait(&sh->k_empty[j & 1], ((j >> 1) & 1) ^ 1);
        if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
        fetch(j, 0);
        if (j > 0) {                   // V(j - 1)
          ptc_cp_wait<1>();
          fence_proxy_async();
          mbar_arrive(&sh->v_full[(j - 1) & 1]);
        }
        bw.wait(&sh->v_empty[j & 1], ((j >> 1) & 1) ^ 1);
        if (!__all_sync(0xffffffffu, !bw.dead)) { bw.dead = true; break; }
        fetch(j, 1);
        ptc_cp_wait<1>();              // K(j)
        fence_proxy_async();
        mbar_arrive(&sh->k_full[j & 1]);
      }
      ptc_cp_wait<0>();
      if (n_tiles > 0 && !bw.dead) {
        fence_proxy_async();
        mbar_arrive(&sh->v_full[(n_tiles - 1) & 1]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

template <int D, bool TMA>
static int launch_prefill_tc(const PrefillTcParams& p, const CUtensorMap& map, dim3 grid, cudaStream_t stream) {
  auto kern = paged_prefill_attn_tc_kernel<D, TMA>;
  // (a fixed size per instantiation -- safe under CUDA-graph replay)
  constexpr int smem_bytes = PtcLayout<D>::TOTAL;
  VB_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
  VB_LAUNCH_PDL(kern, grid, PTC_THREADS, smem_bytes, stream, p, map);
  return 0;
}
}  // namespace vb

using namespace vb;

extern "C" {

int vb_prefill_attn_tc_timeouts(void) {
  return wait_ran_out(WK_PREFILL_ATTN);
}

int vb_prefill_attn_tc_tile_rows(int n_q, int n_kv) {
  if (n_kv < 1 || n_q < n_kv || n_q % n_kv != 0 || n_q / n_kv > 128) return -1;
  return 128 / (n_q / n_kv);
}

int vb_paged_prefill_attn_tc(void* d_out, const void* d_q, const void* d_kv, int64_t slab_base,
                             const int32_t* d_qo_indptr, const int32_t* d_kv_indptr, const int32_t* d_kv_indices,
                             const int32_t* d_row_kvlen, int n_req, int n_rows, int n_q, int n_kv, int head_dim,
                             int page_size, float sm_scale, int out_xt_tile, void* stream) {
  VB_CHECK_ARG(d_out && d_q && d_kv && d_qo_indptr && d_kv_indptr && d_kv_indices && d_row_kvlen,
               "vb_paged_prefill_attn_tc: null pointer");
  VB_CHECK_ARG(n_kv > 0 && n_q % n_kv == 0 && n_q / n_kv <= 128, "vb_paged_prefill_attn_tc: %d query heads / %d kv heads",
               n_q, n_kv);
  VB_CHECK_ARG(head_dim == 64 || head_dim == 128, "vb_paged_prefill_attn_tc: head_dim %d unsupported (64, 128)", head_dim);
  VB_CHECK_ARG(page_size >= 1, "vb_paged_prefill_attn_tc: page_size %d", page_size);
  if (n_rows <= 0 || n_req <= 0) return 0;
  PrefillTcParams p;
  VB_CHECK_ARG(p.wait_flag = wait_flag(WK_PREFILL_ATTN), "vb_paged_prefill_attn_tc: no mapped host memory");
  p.out = static_cast<__nv_bfloat16*>(d_out);
  p.q = static_cast<const __nv_bfloat16*>(d_q);
  p.kv = static_cast<const __nv_bfloat16*>(d_kv);
  p.qo_indptr = d_qo_indptr;
  p.kv_indptr = d_kv_indptr;
  p.kv_indices = d_kv_indices;
  p.row_kvlen = d_row_kvlen;
  p.slab_base = static_cast<int>(slab_base);
  p.n_req = n_req; p.n_rows = n_rows; p.n_q = n_q; p.n_kv = n_kv; p.G = n_q / n_kv; p.page_size = page_size;
  p.TQ = 128 / p.G;
  p.out_xt_tile = out_xt_tile;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
  const unsigned tiles = static_cast<unsigned>((n_rows + p.TQ - 1) / p.TQ) + static_cast<unsigned>(n_req), slices = (tiles + 65534) / 65535;
  const dim3 grid(n_kv, (tiles + slices - 1) / slices, slices);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  p.box_tokens = ptc_box_tokens(page_size);
  CUtensorMap map = {};
  if (page_size % 8 == 0) {
    auto fn = encode_fn();
    VB_CHECK_ARG(fn, "cuTensorMapEncodeTiled not available (no CUDA driver?)");
    // (dim, head, token, K | V, page); how many pages there are is the caller's: every box starts at a page of the table
    const cuuint64_t H = n_kv, P = page_size, Dd = head_dim;
    cuuint64_t dims[5] = {Dd, H, P, 2, 1ull << 30};
    cuuint64_t strides[4] = {Dd * 2, H * Dd * 2, P * H * Dd * 2, 2 * P * H * Dd * 2};
    cuuint32_t box[5] = {64, 1, static_cast<cuuint32_t>(p.box_tokens), 1, 1}, estr[5] = {1, 1, 1, 1, 1};
    const CUresult r = fn(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(d_kv), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    VB_CHECK_ARG(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled(paged K/V) failed: CUresult %d", static_cast<int>(r));
    return head_dim == 128 ? launch_prefill_tc<128, true>(p, map, grid, st) : launch_prefill_tc<64, true>(p, map, grid, st);
  }
  return head_dim == 128 ? launch_prefill_tc<128, false>(p, map, grid, st) : launch_prefill_tc<64, false>(p, map, grid, st);
}

}  // extern "C"
