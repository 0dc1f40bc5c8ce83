// tcgen05.cuh — tensor-core pieces shared by the kernels that issue tcgen05.mma (gemm_tcgen05.cu, gemm_skinny.cu, ...): PTX
// wrappers, the shared-memory descriptor, bounded barrier waits, the gated units of the feed-forwards, the tensor-map cache.
#pragma once
#include <cuda.h>

#include "layered_common.cuh"

namespace b200q {

// ---- tcgen05 PTX wrappers ------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]; kind::f16 covers bf16 inputs with fp32 accumulate
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on an mbarrier once all previously issued tcgen05.mma of this thread have completed
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
        "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

// One lane of a converged warp, the same one every time.  Products are issued behind this and not behind `lane == 0`: ptxas keeps the
// operands of what follows in uniform registers, while behind a lane test every product moves its descriptors there one by one: 50
// against 150 cycles per product on an SM whose other warps are busy (46 where they idle), more than a 128 x 128 x 16 product takes.
__device__ __forceinline__ bool elect_one() {
  uint32_t on;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(on));
  return on != 0;
}

// 32 (16) columns of this warp's lanes, one value per lane and column
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};" ::"r"(v[0]),
      "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
      "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
      "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]),
      "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::"r"(v[0]),
      "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
      "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// wait with a limit: false when it ran out, or once another role of the CTA has given up (*dead); then *failed is set, which the engine
// and b200q_wait_failures report.  A limit below 0 counts as run out at once.  The flag and the clock are looked at after EVERY
// tries (a try suspends the thread for a while by itself).
constexpr long long WAIT_CYCLES = 4000000000ll;  // about two seconds
template <int EVERY = 1>
__device__ __forceinline__ bool mbar_wait_or_fail(uint64_t* bar, uint32_t parity, volatile int* dead, int* failed,
                                                  long long limit = WAIT_CYCLES) {
  if (limit >= 0) {
    if (EVERY == 1 && mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (int n = 1;; ++n) {
      if (mbar_try_wait(bar, parity)) return true;
      if (n % EVERY == 0 && (*dead || clock64() - t0 > limit)) break;
    }
  }
  *dead = 1;
  __threadfence_block();
  *(volatile int*)failed = 1;
  return false;
}

// the same for a whole warp, whose lanes agree on the outcome; flag and clock are looked at every 64 tries (a look in between costs 140
// cycles where the data is about to come)
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* dead, int* failed, long long limit) {
  if (limit >= 0) {
    long long t0 = 0;
    for (int n = 0;; ++n) {
      if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
      if (n % 64 != 63) continue;
      if (n == 63) t0 = clock64();
      if (__any_sync(0xffffffffu, *dead || clock64() - t0 > limit)) break;
    }
  }
  *dead = 1;
  __threadfence_block();
  *(volatile int*)failed = 1;
  return false;
}

// ---- q-tiles of prompt attention: {block table row, first row, rows, first position} -----------
// keys that the last token of tile i's portion sees (a whole warp asks; neighbouring tiles of one sequence that continue each other are a
// portion), as far as 31 tiles on: exact for a comparison with up to 512
__device__ __forceinline__ int portion_keys(const int4* tiles, int n_tiles, int i, int lane) {
  const int4 t = tiles[min(i + lane, n_tiles - 1)];
  const int n = min(max(t.z, 0), 16);
  const int x = __shfl_up_sync(0xffffffffu, t.x, 1), y = __shfl_up_sync(0xffffffffu, t.y + n, 1), w = __shfl_up_sync(0xffffffffu, t.w + n, 1);
  const uint32_t ends = __ballot_sync(0xffffffffu, lane > 0 && (i + lane >= n_tiles || x != t.x || y != t.y || w != t.w));
  return __shfl_sync(0xffffffffu, t.w + n, ends ? __ffs(ends) - 2 : 31);
}

// ---- thread-block clusters ------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `p` (a shared-memory object of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_shared(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_cluster_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// UMMA shared-memory descriptor, K-major operand, SWIZZLE_128B, 8-row groups 1024 B apart
// (cute/arch/mma_sm100_desc.hpp SmemDescriptor: start[0,14) lbo[16,30) sbo[32,46) version[46,48)
//  layout_type[61,64)).
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr, uint32_t sbo = 1024, uint32_t lbo = 16) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3ffffu) >> 4);        // start address, 16 B units
  d |= (uint64_t)(lbo >> 4) << 16;                     // LBO (N-major: from one 64-column slice to the next; else ignored)
  d |= (uint64_t)(sbo >> 4) << 32;                     // SBO: from eight rows to the next eight, 1024 B where they are dense
  d |= (uint64_t)1 << 46;                              // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;                              // SWIZZLE_128B
  return d;
}

// kAct: 0 = plain GEMM, 1 = SwiGLU (Llama), 2 = GeGLU with the tanh approximation (Gemma-2):
// out = bf16(bf16(gelu_tanh(bf16(g))) * bf16(u)), gelu_tanh evaluated in fp32 like torch's kernel:
// 0.5 * g * (1 + tanh(sqrt(2/pi) * (g + 0.044715 g^3)))
// 3 = clamped unit (Lipedra: with biases; Fimilorn: without): g' sigmoid(1.702 g') (u' + 1), g' = min(g + bg, limit), u' = clamp(u + bu,
// -limit, limit), in fp32 from the accumulators (one rounding); bias: fp32, this tile's [gate (BN/2) | up (BN/2)], or NULL
constexpr int ACT_NONE = 0, ACT_SWIGLU = 1, ACT_GEGLU = 2, ACT_CLAMPED = 3;
struct GateArgs {
  const float* bias;
  float limit;
};

template <int kAct>
__device__ __forceinline__ float gated_unit(uint32_t gb, uint32_t ub) {
  const float g = round_bf16(__uint_as_float(gb)), u = round_bf16(__uint_as_float(ub));
  if constexpr (kAct == ACT_GEGLU) {
    const float inner = 0.7978845608028654f * (g + 0.044715f * (g * g * g));
    return round_bf16(0.5f * g * (1.f + tanhf(inner))) * u;
  } else {
    return round_bf16(g / (1.f + __expf(-g))) * u;
  }
}
__device__ __forceinline__ float clamped_unit(uint32_t gb, uint32_t ub, float b0, float b1, float limit) {
  const float g = fminf(__uint_as_float(gb) + b0, limit);
  const float w = fminf(fmaxf(__uint_as_float(ub) + b1, -limit), limit);
  return g / (1.f + __expf(-1.702f * g)) * (w + 1.f);
}

// B200Q_BATCH_INVARIANT=1 (read once): what a row of a step gives must not depend on the other rows, so every kernel is taken whose
// order of sums would otherwise change with them (gemm_tcgen05.cu)
bool batch_invariant();

// bf16 row-major [rows, cols] -> tiled map with box {64 cols, box_rows rows}, 128B swizzle (ld: elements between rows, 0 = dense);
// maps are cached by address and shape (gemm_tcgen05.cu)
int get_tmap(const void* ptr, long long rows, long long cols, int box_rows, CUtensorMap* out, long long ld = 0);

// pages of 16 cached rows of D bf16 values, from `kv` on (as many as there are; the caller knows).  One box is a page, laid down as
// [two groups of 8 rows][64-column slices][8 rows][128 bytes]; coordinates {0, 0, 0, page * 2}.
int get_page_tmap(const void* kv, int D, CUtensorMap* out);

// rows of n_q heads of D bf16 values, `stride` elements apart, from p on (as many as there are; the caller knows).  One box is `cols` (32 or
// 64) columns of `heads` heads of `rows` rows, with a swizzle as wide as its columns; coordinates {column, head, row}.
int get_head_rows_tmap(const void* p, int n_q, int D, long long stride, int heads, int rows, int cols, CUtensorMap* out);

// prompt portions over short contexts (attn.cu); long_keys > 0: portions of so many keys and more are left out
int prefill_tiles(const void* q, int q_stride, void* out, const void* kv, const int32_t* bt, int bt_stride, const int32_t* tiles,
                  int n_tiles, int n_q, int n_kv, int D, float scale, float softcap, int window, int long_keys, cudaStream_t st);

int num_sms();  // of the device (gemm_tcgen05.cu)
// products of up to 128 rows (gemm_skinny.cu)
bool gemm_skinny_ok(int M, int N, int K, bool gated);
int gemm_skinny_splits(int M, int N, int K);
int gemm_skinny(const void* A, const void* W, void* C, int M, int N, int K, int act, long long ldc, const float* bias, float limit,
                float* parts, bool fixed_w, cudaStream_t st);

// tiles of 256 weight rows and `rows` rows of A (gemm_rows.cu): a multiple of 32 up to 256, of 64 beyond; N a multiple of 128
// with splits > 1 (of the K / 64 blocks, at least one each) the sums of its parts go to ws[split][M][N] and C is not looked at
int gemm_rows(const void* A, const void* W, void* C, int M, int N, int K, int rows, int splits, float* ws, bool fixed_w, cudaStream_t st);

}  // namespace b200q
