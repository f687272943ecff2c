// Shared device helpers for the sm_100a kernels: mbarrier, TMA (cp.async.bulk.tensor), tcgen05/TMEM,
// ldmatrix / mma.sync, bf16 packing.  Inline PTX only; no CUTLASS.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace vb {

// ---------------------------------------------------------------------------------------------
// error plumbing (host)
// ---------------------------------------------------------------------------------------------
void set_error(const char* fmt, ...);
#define VB_CHECK_ARG(cond, ...)          \
  do {                                   \
    if (!(cond)) {                       \
      ::vb::set_error(__VA_ARGS__);      \
      return -1;                         \
    }                                    \
  } while (0)
#define VB_CHECK_CUDA(expr)                                                        \
  do {                                                                             \
    cudaError_t _e = (expr);                                                       \
    if (_e != cudaSuccess) {                                                       \
      ::vb::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e), __FILE__, __LINE__); \
      return -2;                                                                   \
    }                                                                              \
  } while (0)
#define VB_CHECK_LAUNCH() VB_CHECK_CUDA(cudaGetLastError())
// Largest opt-in dynamic shared memory of an sm_100 CTA.  Kernels raise their limit to this ONCE (not to the size
// of the launch at hand): a per-launch value would be baked into nothing -- CUDA-graph kernel nodes replay
// against whatever the function attribute was set to last, so a later, smaller launch would break them.
constexpr int VB_MAX_DYN_SMEM = 227 * 1024;
// SMs of the device in use, asked for once (the devices of a machine are alike); 148 where there is none to ask
inline int sm_count() {
  static std::atomic<int> known{0};
  int sms = known.load(std::memory_order_relaxed), dev = 0;
  if (sms) return sms;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  known.store(sms, std::memory_order_relaxed);
  return sms;
}
// ... once per kernel and device (one flag per instantiation: call it with the kernel itself, not with a pointer that may
// name several; two threads that arrive together both set the same value)
template <typename Kernel>
inline cudaError_t max_dyn_smem_once(Kernel kernel) {
  static std::atomic<unsigned long long> done{0ull};
  static std::atomic<const void*> whose{nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const void* fn = reinterpret_cast<const void*>(kernel);
  const bool mine = whose.load(std::memory_order_acquire) == fn;
  if (mine && dev < 64 && (done.load(std::memory_order_acquire) >> dev & 1ull)) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, VB_MAX_DYN_SMEM);
  if (e != cudaSuccess || dev >= 64) return e;
  const void* none = nullptr;
  if (mine || whose.compare_exchange_strong(none, fn) || none == fn) done.fetch_or(1ull << dev, std::memory_order_release);
  return cudaSuccess;
}

// ---------------------------------------------------------------------------------------------
// programmatic dependent launch (PDL)
// ---------------------------------------------------------------------------------------------
// Every kernel of the decode chain is launched with cudaLaunchAttributeProgrammaticStreamSerialization, calls
// pdl_wait() before it touches anything its stream predecessor wrote, and pdl_trigger() right after.  Kernel k+1
// can therefore start as soon as every CTA of kernel k is past its own wait -- i.e. while k runs, k+1 already does
// whatever does not depend on k: launch latency, barrier / TMEM set-up, and above all streaming WEIGHTS (GEMM)
// and the KV of earlier steps (attention) into shared memory.  Because the trigger comes after the wait, when
// k+1 starts every kernel <= k-1 has completed: pre-wait code may read anything but k's outputs.
// (VB_PDL=0 disables it everywhere; VB_PDL_OFF=<mask> per source file, a debugging aid: 1 attention, 2 projections,
// 4 elementwise, 8 multi-codebook glue, 16 sampler)
#ifndef VB_PDL_FAMILY
#define VB_PDL_FAMILY 0
#endif
bool pdl_enabled(int family);
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel_cluster(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                         cudaStream_t stream, bool pdl, int cluster_x, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl && pdl_enabled(VB_PDL_FAMILY)) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (cluster_x > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster_x;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel_cluster3(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                          cudaStream_t stream, bool pdl, dim3 cluster, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (pdl && pdl_enabled(VB_PDL_FAMILY)) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (cluster.x * cluster.y * cluster.z > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = cluster.x;
    attr[n].val.clusterDim.y = cluster.y;
    attr[n].val.clusterDim.z = cluster.z;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                 bool pdl, Args... args) {
  return launch_kernel_cluster(kernel, grid, block, smem, stream, pdl, 1, args...);
}
// launch as a programmatic dependent of the previous kernel in the stream / as a plain launch (after a memset,
// or for kernels that do not call pdl_wait)
#define VB_LAUNCH_PDL(kernel, grid, block, smem, stream, ...)                                                \
  VB_CHECK_CUDA(::vb::launch_kernel(kernel, dim3(grid), dim3(block), smem, static_cast<cudaStream_t>(stream), \
                                    true, __VA_ARGS__))
#define VB_LAUNCH_PDL_CLUSTER(kernel, grid, block, smem, stream, cluster_x, ...)                                      \
  VB_CHECK_CUDA(::vb::launch_kernel_cluster(kernel, dim3(grid), dim3(block), smem, static_cast<cudaStream_t>(stream), \
                                            true, cluster_x, __VA_ARGS__))
#define VB_LAUNCH_PLAIN(kernel, grid, block, smem, stream, ...)                                              \
  VB_CHECK_CUDA(::vb::launch_kernel(kernel, dim3(grid), dim3(block), smem, static_cast<cudaStream_t>(stream), \
                                    false, __VA_ARGS__))
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// for kernels with nothing to do before their predecessor has finished
__device__ __forceinline__ void pdl_sync() {
  pdl_wait();
  pdl_trigger();
}

// ---------------------------------------------------------------------------------------------
// in-situ timeline (dev tool): with a buffer installed by vb_set_trace, block 0 of the instrumented kernels
// records %globaltimer at its start / end and at a few internal marks.  Buffer (u64): [0] = records used,
// [1] = capacity, records from [4] on, 4 words each: t0, t1, id, aux.  One copy of the pointer per translation unit.
// ---------------------------------------------------------------------------------------------
static __device__ unsigned long long* g_trace_buf = nullptr;
#define VB_DEFINE_TRACE_SETTER(name)                                                  \
  namespace vb {                                                                      \
  cudaError_t trace_set_##name(unsigned long long* p) {                               \
    return cudaMemcpyToSymbol(g_trace_buf, &p, sizeof(p));                            \
  }                                                                                   \
  }
__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)::"memory");   // also a compiler barrier: marks stay in place
  return t;
}
__device__ __forceinline__ int trace_begin(int id, int aux = 0) {
  unsigned long long* b = g_trace_buf;
  if (!b) return -1;
  const unsigned long long i = atomicAdd(b, 1ull);
  if (i >= b[1]) return -1;
  unsigned long long* r = b + 4 + 4 * i;
  r[0] = gtimer(); r[1] = 0ull; r[2] = static_cast<unsigned long long>(id); r[3] = static_cast<unsigned long long>(aux);
  return static_cast<int>(i);
}
__device__ __forceinline__ void trace_end(int rec) {
  if (rec >= 0) g_trace_buf[4 + 4 * rec + 1] = gtimer();
}
__device__ __forceinline__ void trace_mark(int id, int aux = 0) {
  const int r = trace_begin(id, aux);
  trace_end(r);
}
__device__ __forceinline__ bool trace_block0() { return blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0; }
// fine-grained marks: word [2] of the buffer = offset of a [roles][256] u64 area.  The base is resolved once per
// thread (trace_fine_base: the only loads); a mark is then a single predicated store -- no round trip.
__device__ __forceinline__ unsigned long long* trace_fine_base() {
  unsigned long long* b = g_trace_buf;
  if (!b || !trace_block0()) return nullptr;
  const unsigned long long off = b[2];
  return off ? b + off : nullptr;
}
__device__ __forceinline__ void trace_fine(unsigned long long* fine, int role, unsigned idx) {
  if (fine && idx < 256u) fine[role * 256 + idx] = gtimer();
}

// ---------------------------------------------------------------------------------------------
// small device utilities
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// "Tiled" activation layout XT(t_tile): what a GEMM B-operand stage looks like in shared memory, kept in global
// memory: [token block][k-block of 64][t_tile rows][64] bf16 with the 128-byte swizzle applied (16-byte chunk c of
// row r at chunk c ^ (r & 7)).  A (token block, k-block) tile is one contiguous t_tile * 128-byte run, fetched with a
// single linear bulk copy instead of a tensor-map box (t_tile row requests on the TMA unit).  Element index:
__device__ __forceinline__ size_t xt_index(int t, int k, int t_tile, int num_kb) {
  const int tb = t / t_tile, tt = t - tb * t_tile;
  return ((static_cast<size_t>(tb) * num_kb + (k >> 6)) * t_tile + tt) * 64 + ((((k >> 3) & 7) ^ (tt & 7)) << 3) + (k & 7);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(pred));
  return pred != 0;
}

// ---------------------------------------------------------------------------------------------
// thread-block cluster helpers (distributed shared memory)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_dsmem_f32(const float* local_ptr, uint32_t cta_rank) {
  uint32_t laddr = static_cast<uint32_t>(__cvta_generic_to_shared(local_ptr)), raddr;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(raddr) : "r"(laddr), "r"(cta_rank));
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(raddr) : "memory");
  return v;
}

// ---------------------------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: a protocol bug traps (launch error surfaced to the host) instead of hanging the GPU.
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity) {
#pragma unroll 1
  for (uint32_t spin = 0; spin < (1u << 26); ++spin) {
    if (mbar_try_wait(bar, parity)) return;
  }
  __trap();
}

// A wait that gives up.  After 2 s it sets its kind's flag in host memory (vb_wait_flags: whoever collects results looks there) and
// every later wait of the thread returns at once, so that the block can stop issuing, let its copies land and leave with the
// context usable.  `gate`: shared-memory word that the block sets once the kernels in front have completed (0: they have); the
// clock starts there, or a predecessor's running time would count as the wait's own.
enum WaitKind { WK_GEMM_WIDE = 0, WK_CL_CONV = 1, WK_PREFILL_ATTN = 2, WK_WINDOW_ATTN = 3, WK_CHECK = 4, WK_KINDS = 8 };
unsigned char* wait_flag(WaitKind kind);      // api.cu: its address on the device, nullptr if the flags could not be allocated
int wait_ran_out(WaitKind kind);              // api.cu: after all work on the device
struct BoundedWait {
  unsigned char* flag;
  uint32_t gate = 0u;
  unsigned long long limit = 2000000000ull;
  bool dead = false;
  __device__ __forceinline__ void wait(uint64_t* bar, uint32_t parity) {
    if (dead) return;
    unsigned long long t0 = 0ull;
#pragma unroll 1
    for (uint32_t spin = 1;; ++spin) {
      if (mbar_try_wait(bar, parity)) return;
      if ((spin & 255u) == 0u) {
        uint32_t open = 1u;
        if (gate) asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(open) : "r"(gate) : "memory");
        const unsigned long long now = gtimer();
        if (t0 == 0ull || !open) t0 = now;
        else if (now - t0 > limit) {
          dead = true;
          *reinterpret_cast<volatile unsigned char*>(flag) = 1;
          __threadfence_system();
          return;
        }
      }
    }
  }
};
// Several warps that meet behind waits of their own: true in all of them if it is in one.  (A warp that gave up has to come here all the same: the
// others would wait for it without a limit.)
template <int BARRIER, int THREADS>
__device__ __forceinline__ bool warps_any(bool dead) {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, %2, %3, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
               : "=r"(r)
               : "r"(dead ? 1u : 0u), "n"(BARRIER), "n"(THREADS)
               : "memory");
  return r != 0u;
}
__device__ __forceinline__ void wait_gate_open(uint32_t gate) {
  asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(gate), "r"(1u) : "memory");
}

// ---------------------------------------------------------------------------------------------
// TMA
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_hint(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1),
      "l"(policy)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2,
                                            int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2),
      "r"(c3), "r"(c4)
      : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// ---------------------------------------------------------------------------------------------
// ldmatrix / mma.sync (bf16, fp32 accumulate) -- used by the paged attention kernels
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---------------------------------------------------------------------------------------------
// tcgen05 / TMEM
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem desc] * B[smem desc]; kind::f16 covers bf16 inputs with fp32 accumulation.
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A * B with tf32 inputs (fp32 storage).
__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on an mbarrier once all previously issued tcgen05.mma of this thread have completed
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// 32 lanes x 32 columns of fp32: thread i of the warp receives row (lane base + i), 32 consecutive columns
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor for a K-major operand tile stored as rows of 128 bytes with the
// 128-byte swizzle (what TMA SWIZZLE_128B writes): 8-row groups are 1024 B apart (SBO), LBO unused.
// Bit layout (PTX ISA "shared memory descriptor", sm_100): [0,14) addr>>4, [16,30) LBO>>4,
// [32,46) SBO>>4, [46,48) version = 1, [61,64) layout type (2 = SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc_sw128_kmajor(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3ffffu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;            // LBO (ignored for swizzled K-major), canonical value 1
  d |= static_cast<uint64_t>(1024 >> 4) << 32;    // SBO
  d |= static_cast<uint64_t>(1) << 46;            // descriptor version (Blackwell)
  d |= static_cast<uint64_t>(2) << 61;            // SWIZZLE_128B
  return d;
}
// Instruction descriptor, kind::f16 / kind::tf32, dense, fp32 accumulate, both operands K-major.
// [4,6) D fmt (1 = f32), [7,10) A fmt, [10,13) B fmt (f16: 0 f16 / 1 bf16; tf32: 2), [15] A major,
// [16] B major (0 = K), [17,23) N>>3, [24,29) M>>4.
__host__ __device__ constexpr uint32_t umma_idesc(uint32_t m, uint32_t n, uint32_t ab_fmt) {
  return (1u << 4) | (ab_fmt << 7) | (ab_fmt << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

}  // namespace vb
