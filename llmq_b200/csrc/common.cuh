// common.cuh — shared helpers for libb200q (sm_100a only).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/b200q.h"

namespace b200q {

// ---- error plumbing (never throw across the C ABI) -------------------------------------
void set_error(const char* fmt, ...);
extern thread_local char g_err[512];
void count_launch(int n = 1);
// bumped by every test/tuning setter: cached CUDA graphs bake kernel choices in and must be rebuilt
// prompt attention (prefill_attn.cu): which kernel takes a step's portions, and the call
int prefill_attn_route(const int32_t* desc, int n_desc, int n_seqs, int n_tiles, int bt_stride, int n_q, int n_kv, int D, int window);
int prefill_attn(int route, const void* q, int q_stride, void* out, const void* kv_layer, const int32_t* block_table, int bt_stride,
                 const int32_t* tiles, int n_tiles, int n_q, int n_kv, int D, int block_size, float scale, float softcap, int window,
                 cudaStream_t st);
void bump_tuning_epoch();
int tuning_epoch();

// single-token attention (attn.cu) as a forward pass calls it.  tables_known: block table and context lengths were there before the pass, so
// that the pages can be asked into L2 while the kernels before this one still run (see linear).
int decode_attn(const void* q, int q_stride, void* out, const void* kv_layer, const int32_t* block_table, int bt_stride,
                const int32_t* ctx_lens, int n_seqs, int n_q, int n_kv, int D, int block_size, float scale, float softcap, int window,
                bool tables_known, cudaStream_t st);
// The projections (gemm_tcgen05.cu) as a forward pass calls them.  fixed_w: no kernel that may still run when this one begins writes the
// weights, so they are fetched before follow_previous; that holds where the first kernel of the same pass was not launched early.
int linear(const void* A, const void* W, void* C, int M, int N, int K, bool fixed_w, cudaStream_t st);
int linear_parts(const void* A, const void* W, int M, int N, int K, bool fixed_w, cudaStream_t st, const float** partials_out,
                 int* splits_out);
int linear_gated(bool gelu, const void* A, const void* W, void* C, int M, int N, int K, bool fixed_w, cudaStream_t st);
// parts of one split reduction: up to 2048 rows x parts of 8192 columns (256 rows in 6, 768 in 2, 128 in 8), 64 MiB
constexpr size_t SPLIT_BYTES = (size_t)8 * 256 * 8192 * sizeof(float);
// While one of these lives, split products that the calling thread asks for leave their parts there: a pass runs under its model's
class SplitScratchOf {
 public:
  SplitScratchOf(void* p, size_t bytes);
  ~SplitScratchOf();
  SplitScratchOf(const SplitScratchOf&) = delete;

 private:
  void* p_;
  size_t bytes_;
};

#define B200Q_CHECK_ARG(cond, ...)          \
  do {                                      \
    if (!(cond)) {                          \
      ::b200q::set_error(__VA_ARGS__);      \
      return B200Q_EINVAL;                  \
    }                                       \
  } while (0)

#define B200Q_CUDA(expr)                                                              \
  do {                                                                                \
    cudaError_t _e = (expr);                                                          \
    if (_e != cudaSuccess) {                                                          \
      ::b200q::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e),      \
                         __FILE__, __LINE__);                                         \
      return B200Q_ECUDA;                                                             \
    }                                                                                 \
  } while (0)

#define B200Q_LAUNCH_CHECK()                                                          \
  do {                                                                                \
    cudaError_t _e = cudaGetLastError();                                              \
    if (_e != cudaSuccess) {                                                          \
      ::b200q::set_error("kernel launch failed: %s (%s:%d)", cudaGetErrorString(_e),  \
                         __FILE__, __LINE__);                                         \
      return B200Q_ECUDA;                                                             \
    }                                                                                 \
    ::b200q::count_launch();                                                          \
  } while (0)

using bf16 = __nv_bfloat16;

// ---- small device helpers ---------------------------------------------------------------
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// round-to-nearest-even fp32 -> bf16 bits (matches torch .to(bfloat16))
__device__ __forceinline__ uint32_t f2bf_bits(float f) {
  return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(f));
}
__device__ __forceinline__ float round_bf16(float f) {
  return __bfloat162float(__float2bfloat16_rn(f));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  // cvt.rn.bf16x2.f32 d, a, b : d.hi = a, d.lo = b
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

__device__ __forceinline__ uint4 ld_nc_v4(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p));
  return r;
}
// read once, not to be kept in L1; unlike ld_nc_v4 also right for what another kernel writes while this one is already on the chip
__device__ __forceinline__ uint4 ld_once_v4(const void* p) {
  uint4 r;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p)
               : "memory");
  return r;
}
__device__ __forceinline__ uint4 ld_v4(const void* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void st_v4(void* p, uint4 v) { *reinterpret_cast<uint4*>(p) = v; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ---- mbarrier ------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity) {
  while (!mbar_try_wait(bar, parity)) {
  }
}

// ---- TMA -------------------------------------------------------------------------------------
// 1-D bulk copy global -> shared, completion on an mbarrier
__device__ __forceinline__ void tma_bulk_g2s(void* smem_dst, const void* gsrc, uint32_t bytes,
                                             uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// so many bytes (a multiple of 16) into L2 only; as with tma_prefetch_2d, nothing is read by it
__device__ __forceinline__ void bulk_prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
// 2-D tiled tensor-map load
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const void* tmap, int c0, int c1,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
// the same box into L2 only.  Nothing is read by it as far as the memory model goes, so that it may run ahead of follow_previous.
__device__ __forceinline__ void tma_prefetch_2d(const void* tmap, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(tmap), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const void* tmap, int c0, int c1, int c2, int c3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}

// ---- warp-level tensor core pieces used by the attention kernels ---------------------------
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                        uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t& r0, uint32_t& r1,
                                          uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// D(16x8,f32) += A(16x16,bf16,row) * B(16x8,bf16,col)
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1,
                                               uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- kernels that begin while the one before them on the stream still runs -------------------
// launch_early starts a kernel as soon as every block of the one before it has called follow_previous (or has ended), wherever an SM has
// room: the launch, barriers, tensor memory and what may be asked into L2 ahead no longer lie between the two.  follow_previous waits
// until that kernel has ended and what it wrote can be seen; nothing that another kernel may write is read, and nothing is written,
// before it.  Every thread calls it, so the kernel two places back has ended as well; and it is called once the block has its tensor
// memory (a block barrier between), which a block of the next kernel could otherwise take from it and hold until this one ends.  What
// another kernel may write while this one waits is not read-only for this one's lifetime: no __ldg or ld.global.nc in such a kernel, and
// the pointers that it reads through go through follow_previous, so that the compiler makes no such loads of const __restrict__ ones.
// B200, in a graph of dependent kernels: 2.0 us instead of 3.4 from one small kernel to the next; the routed feed-forward of 128 rows
// (8 kernels) 73.2 -> 58.9 us, a decode step of four layers of the 1B model at 48 sequences (37 kernels) 371 -> 349 us.
// (Blocks that take the places which the kernel before leaves may come to lie two on one SM and none on another: kernels that lose more by
// that than a start costs, 1 to 1.5 us, are launched plainly for those sizes, see launch_prefill in attn.cu and prefill_attn.cu.)
// (pinned as an address of global memory, which the compiler would otherwise forget that it is)
template <typename T>
__device__ __forceinline__ T* pinned_global(T* p) {
  size_t at = __cvta_generic_to_global(p);
  asm volatile("" : "+l"(at)::"memory");
  return reinterpret_cast<T*>(__cvta_global_to_generic(at));
}
template <typename T>
__device__ __forceinline__ void pin_behind(T*& p) {
  p = pinned_global(p);
}
template <typename T>
__device__ __forceinline__ void pin_behind(T* __restrict__& p) {
  p = pinned_global<T>(p);
}
// (the wait alone, where a block may find that it has nothing to do; follow_previous comes behind it once the block has its tensor memory)
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... P>
__device__ __forceinline__ void follow_previous(P&... p) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  wait_for_previous();
  (pin_behind(p), ...);
}
template <typename... P, typename... A>
inline cudaError_t launch_early(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, int cluster, A&&... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<A&&>(args)...);
}

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

}  // namespace b200q
