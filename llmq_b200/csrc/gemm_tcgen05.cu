// gemm_tcgen05.cu — C[M,N] = A[M,K] . W[N,K]^T (bf16 in, fp32 accumulate in TMEM, bf16 out)
// for the QKV / O / gate_up / down / LM-head projections,
// the only dense contractions of the hot path.  Hand-written for sm_100a:
//
//   * persistent, warp-specialised CTA (192 threads): warp 0 = TMA producer (128B
//     swizzle), warp 1 = tcgen05.mma issuer (one lane; also owns the TMEM allocation),
//     warps 2-5 = epilogue (tcgen05.ld -> bf16 -> global).
//   * tile 128 x BN x 64 (BN in {64,128,256}), smem ring of 4..8 stages (<= 192 KB), operands
//     K-major in shared memory exactly as TMA lays them down (SWIZZLE_128B), described to the
//     tensor core by UMMA shared-memory descriptors; UMMA shape M=128, N=BN, K=16.
//   * two TMEM accumulator stages (2 x BN fp32 columns): the MMA warp runs tile i+1 while the
//     epilogue warps drain tile i.
//   * tile order is m-fastest so concurrently running CTAs share one weight tile through L2
//     (weights stream from HBM exactly once; activations are L2-resident).
//
// Roofline: decode-sized M is HBM-bound on the weight stream (N*K*2 bytes), M >= ~256 is
// tensor-bound (2*M*N*K flops against the measured bf16 peak).
#include <stdlib.h>

#include <atomic>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "tcgen05.cuh"

namespace b200q {

constexpr int GEMM_BM = 128;
constexpr int GEMM_BK = 64;  // 64 bf16 = 128 B = one swizzle span
constexpr int GEMM_THREADS = 192;
constexpr int GEMM_SMEM_BUDGET = 196608;  // ring bytes

template <int BN>
struct GemmCfg {
  static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2;  // 16 KB
  static constexpr int B_BYTES = BN * GEMM_BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = GEMM_SMEM_BUDGET / STAGE_BYTES > 8 ? 8 : GEMM_SMEM_BUDGET / STAGE_BYTES;
  static constexpr int TMEM_COLS = 2 * BN;  // 128 / 256 / 512: powers of two >= 32
  static constexpr int SMEM_TOTAL = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/ + 4 * 4096 /*epilogue*/;
};

// instruction descriptor for kind::f16: D=f32, A=B=bf16, both K-major, M=128, N=BN
__host__ __device__ constexpr uint32_t make_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(GEMM_BM >> 4) << 24);
}

// Drain one warp's 32 x BN slice of the fp32 accumulator tile (TMEM lanes 32q..32q+31, one row per
// thread) to global memory.  Each thread converts 64 columns of its row to bf16 (128 B), the warp
// transposes them through a 4 KB XOR-swizzled shared-memory patch and stores them back as
// 4 rows x 128 contiguous bytes per instruction — full 128 B lines instead of 32 scattered 16 B
// pieces, which matters because the L2 request rate is shared with the TMA operand stream.
// kSwiGLU (K9+K10 fused): the weight rows were interleaved at load time so that the tile's
// columns are [gate (BN/2) | up (BN/2)] of the SAME BN/2 output columns; the epilogue applies
// out = bf16(bf16(silu(bf16(g))) * bf16(u)) — identical rounding points to the unfused path
// (GEMM output rounded to bf16, then oracle/ops.py::swiglu) — and writes BN/2 columns, so the
// [T, 2I] intermediate never touches HBM.
constexpr int EPI_SMEM_PER_WARP = 32 * 128;  // 32 rows x 64 bf16

template <int BN, int kAct>
__device__ __forceinline__ void epilogue_rows(uint32_t taddr, bf16* ctile, long long ldc,
                                              int row0, int M, uint8_t* patch, int lane,
                                              const float* gate_bias = nullptr, float limit = 0.f, int cols = BN, int c_begin = 0,
                                              int c_step = 64) {
  constexpr bool kSwiGLU = kAct != ACT_NONE;  // gated epilogue: tile = [gate (BN/2) | up (BN/2)]
  constexpr int OUT_BN = kSwiGLU ? BN / 2 : BN;
  // (no row of this warp exists: its accumulators are sums of zeros, which the gated units' division treats as a special case: 384 rows
  // x 2048 x 512 gated 29 us, 15 without)
  if (row0 >= M) return;
  // (kRagged: columns of C in this tile, a multiple of 32; the last tile of a row may have fewer than BN)
  constexpr bool kRagged = BN % 128 != 0 && BN > 64;
  const uint32_t patch_s = smem_u32(patch);
#pragma unroll 1
  for (int c0 = c_begin; c0 < (kRagged ? cols : OUT_BN); c0 += c_step) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // two 32-column TMEM loads -> 64 output columns of this row
      uint32_t v[32];
      uint4 o[4];
      if (kRagged && c0 + 32 * h >= cols) break;
      if constexpr (!kSwiGLU) {
        tmem_ld32(taddr + (uint32_t)(c0 + 32 * h), v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          o[j].x = pack_bf16x2(__uint_as_float(v[8 * j + 0]), __uint_as_float(v[8 * j + 1]));
          o[j].y = pack_bf16x2(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
          o[j].z = pack_bf16x2(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
          o[j].w = pack_bf16x2(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
        }
      } else {
        uint32_t u[32];
        tmem_ld32(taddr + (uint32_t)(c0 + 32 * h), v);
        tmem_ld32(taddr + (uint32_t)(BN / 2 + c0 + 32 * h), u);
        tmem_ld_wait();
        // (a row that does not exist, beside rows that do: as above; 300 rows of 16384 x 2048 64.4 -> 35.2 us, 200 of 28672 x 4096
        // 88.3 -> 64.0, 2001 403 -> 354)
        if (row0 + lane >= M) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0x3f800000u;
        }
        if constexpr (kAct == ACT_CLAMPED) {
          const float4* bg = reinterpret_cast<const float4*>(gate_bias + c0 + 32 * h);
          const float4* bu = reinterpret_cast<const float4*>(gate_bias + BN / 2 + c0 + 32 * h);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 x = gate_bias ? bg[j] : zero, y = gate_bias ? bu[j] : zero;
            v[4 * j + 0] = __float_as_uint(clamped_unit(v[4 * j + 0], u[4 * j + 0], x.x, y.x, limit));
            v[4 * j + 1] = __float_as_uint(clamped_unit(v[4 * j + 1], u[4 * j + 1], x.y, y.y, limit));
            v[4 * j + 2] = __float_as_uint(clamped_unit(v[4 * j + 2], u[4 * j + 2], x.z, y.z, limit));
            v[4 * j + 3] = __float_as_uint(clamped_unit(v[4 * j + 3], u[4 * j + 3], x.w, y.w, limit));
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            o[j].x = pack_bf16x2(__uint_as_float(v[8 * j + 0]), __uint_as_float(v[8 * j + 1]));
            o[j].y = pack_bf16x2(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
            o[j].z = pack_bf16x2(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
            o[j].w = pack_bf16x2(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
          }
        } else
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          o[j].x = pack_bf16x2(gated_unit<kAct>(v[8 * j + 0], u[8 * j + 0]), gated_unit<kAct>(v[8 * j + 1], u[8 * j + 1]));
          o[j].y = pack_bf16x2(gated_unit<kAct>(v[8 * j + 2], u[8 * j + 2]), gated_unit<kAct>(v[8 * j + 3], u[8 * j + 3]));
          o[j].z = pack_bf16x2(gated_unit<kAct>(v[8 * j + 4], u[8 * j + 4]), gated_unit<kAct>(v[8 * j + 5], u[8 * j + 5]));
          o[j].w = pack_bf16x2(gated_unit<kAct>(v[8 * j + 6], u[8 * j + 6]), gated_unit<kAct>(v[8 * j + 7], u[8 * j + 7]));
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // chunk (4h + j) of this thread's 128 B row
        const uint32_t a = patch_s + lane * 128 + (((4 * h + j) ^ (lane & 7)) << 4);
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(o[j].x), "r"(o[j].y),
                     "r"(o[j].z), "r"(o[j].w)
                     : "memory");
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // 4 rows x 128 B per instruction
      const int rr = i * 4 + (lane >> 3), c = lane & 7;
      uint4 o;
      const uint32_t a = patch_s + rr * 128 + ((c ^ (rr & 7)) << 4);
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(o.x), "=r"(o.y), "=r"(o.z), "=r"(o.w)
                   : "r"(a));
      if (row0 + rr < M && (!kRagged || c0 + c * 8 < cols)) st_v4(ctile + (long long)rr * ldc + c0 + c * 8, o);
    }
    __syncwarp();
  }
}

template <int BN, int kAct = ACT_NONE>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a,
                     const __grid_constant__ CUtensorMap tmap_b, bf16* __restrict__ C, int M,
                     int N, int K, int splits, float* __restrict__ ws, int a_bytes,
                     long long ldc, GateArgs gate, int fixed_w) {
  constexpr bool kSwiGLU = kAct != ACT_NONE;
  // a_bytes: bytes one A k-block really carries.  For M < 128 the tensor map's box holds only the
  // rows that exist (rounded up to the 8-row swizzle atom), not 128: the other rows of the UMMA's A
  // tile are stale shared memory whose products land in output rows >= M, which are never stored.
  // A decode-sized GEMM re-reads the whole activation matrix in EVERY CTA — with 128 x 128 tiles as
  // many L2->SM bytes as the weights themselves — so rows that do
  // not exist should not be paid for.
  // splits > 1 (split-K for decode-sized M, where a projection has too few output tiles to put
  // every SM on the weight stream): tile space = m x split x n, each CTA accumulates K/splits of
  // the reduction and writes an fp32 partial tile to ws[split][M][N]; splitk_reduce_kernel sums the
  // partials in a fixed order (deterministic) and rounds to bf16.
  using Cfg = GemmCfg<BN>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tmem_full = empty + STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  uint8_t* epi_smem = smem + STAGES * Cfg::STAGE_BYTES + 256;  // 4 warps x 4 KB transpose patches

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int m_tiles = (M + GEMM_BM - 1) / GEMM_BM;
  const int n_tiles = N / BN;
  const int num_tiles = m_tiles * n_tiles * splits;
  const int k_blocks = (K / GEMM_BK) / splits;  // k-blocks per tile (per split)

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    mbar_init(tmem_full + 0, 1);
    mbar_init(tmem_full + 1, 1);
    mbar_init(tmem_empty + 0, 4);
    mbar_init(tmem_empty + 1, 4);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  int early = 0;  // k-blocks whose weights are asked for while the kernel before this one ends
  if (warp == 0 && lane == 0) {
    const int rest = blockIdx.x / m_tiles, n_blk = rest / splits, kb0 = (rest % splits) * k_blocks;
    for (int kb = 0; kb < STAGES && kb < k_blocks; ++kb) {
      if (fixed_w) {
        mbar_expect_tx(full + kb, (uint32_t)(a_bytes + Cfg::B_BYTES));
        tma_load_2d(smem + kb * Cfg::STAGE_BYTES + Cfg::A_BYTES, &tmap_b, (kb0 + kb) * GEMM_BK, n_blk * BN, full + kb);
        ++early;
      } else {
        tma_prefetch_2d(&tmap_b, (kb0 + kb) * GEMM_BK, n_blk * BN);
      }
    }
  }
  __syncwarp();
  follow_previous(gate.bias);

  if (warp == 0) {
    // ===== TMA producer =====
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
        const int m_blk = tile % m_tiles, rest = tile / m_tiles;
        const int n_blk = rest / splits, kb0 = (rest % splits) * k_blocks;
        int kb = 0;
        // The first tile's stages 0, 1, ..., whose weights are on their way, have a loop of their own: asked about in the loop below, they
        // cost every k-block of every tile some 20 ns (750 x 2048 x 8192 29.9 -> 31.4 us, 300 x 3584 x 14336 49.5 -> 52.3; so 29.2 and 48.7)
        for (; kb < early; ++kb)
          tma_load_2d(smem + kb * Cfg::STAGE_BYTES, &tmap_a, (kb0 + kb) * GEMM_BK, m_blk * GEMM_BM, full + kb);
        if (early > 0) {
          stage = early % STAGES;
          phase = early / STAGES;
          early = 0;
        }
        for (; kb < k_blocks; ++kb) {
          uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          mbar_wait(empty + stage, phase ^ 1u);
          mbar_expect_tx(full + stage, (uint32_t)(a_bytes + Cfg::B_BYTES));
          tma_load_2d(sb, &tmap_b, (kb0 + kb) * GEMM_BK, n_blk * BN, full + stage);
          tma_load_2d(sa, &tmap_a, (kb0 + kb) * GEMM_BK, m_blk * GEMM_BM, full + stage);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ===== MMA issuer =====
    constexpr uint32_t idesc = make_idesc(BN);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      mbar_wait(tmem_empty + acc, acc_phase ^ 1u);
      tc_fence_after();
      const uint32_t tmem_d = tmem_base + (uint32_t)(acc * BN);
      for (int kb = 0; kb < k_blocks; ++kb) {
        mbar_wait(full + stage, phase);
        tc_fence_after();
        if (elect_one()) {
          const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
          const uint32_t sb = sa + Cfg::A_BYTES;
#pragma unroll
          for (int k = 0; k < GEMM_BK / 16; ++k) {
            const uint64_t ad = make_smem_desc(sa + k * 32);
            const uint64_t bd = make_smem_desc(sb + k * 32);
            umma_bf16(tmem_d, ad, bd, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit(empty + stage);  // smem stage free once these MMAs retire
          if (kb == k_blocks - 1) umma_commit(tmem_full + acc);
        }
        __syncwarp();
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  } else {
    // ===== epilogue warps 2..5: TMEM lane quarter = warp % 4 =====
    const int quarter = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      const int m_blk = tile % m_tiles, rest = tile / m_tiles;
      const int n_blk = rest / splits, split = rest % splits;
      mbar_wait(tmem_full + acc, acc_phase);
      tc_fence_after();
      const int row0 = m_blk * GEMM_BM + quarter * 32;
      constexpr int OUT_BN = kSwiGLU ? BN / 2 : BN;
      bf16* ctile = C + (long long)row0 * ldc + (long long)n_blk * OUT_BN;
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN);
      if (splits > 1) {
        // fp32 partial of this K-slice: ws[split][row][col]; one full 128 B line per thread per load
        const int row = row0 + lane;
        float* wrow = ws + ((long long)split * M + row) * N + (long long)n_blk * BN;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
          uint32_t v[32];
          tmem_ld32(taddr + (uint32_t)c0, v);
          tmem_ld_wait();
          if (row < M) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              st_v4(wrow + c0 + 4 * j, make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
          }
        }
      } else {
        epilogue_rows<BN, kAct>(taddr, ctile, ldc, row0, M, epi_smem + (warp - 2) * EPI_SMEM_PER_WARP, lane,
                                kAct == ACT_CLAMPED && gate.bias ? gate.bias + (long long)n_blk * BN : nullptr, gate.limit);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tmem_empty + acc);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// out[m][n] = bf16(sum_s ws[s][m][n]), partials added in split order (deterministic), four parts asked for at once
__global__ void __launch_bounds__(256)
    splitk_reduce_kernel(const float4* __restrict__ ws, uint4* __restrict__ out, long long mn8,
                         int splits) {
  follow_previous(ws, out);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < mn8;
       i += (long long)gridDim.x * blockDim.x) {
    float4 a, b;
    for (int s0 = 0; s0 < splits; s0 += 4) {
      float4 c[4], d[4];
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (s0 + x < splits) {
          c[x] = ws[2 * (i + (s0 + x) * mn8)];
          d[x] = ws[2 * (i + (s0 + x) * mn8) + 1];
        }
#pragma unroll
      for (int x = 0; x < 4; ++x)
        if (s0 + x < splits) {
          if (s0 + x == 0) {
            a = c[x];
            b = d[x];
          } else {
            a.x += c[x].x; a.y += c[x].y; a.z += c[x].z; a.w += c[x].w;
            b.x += d[x].x; b.y += d[x].y; b.z += d[x].z; b.w += d[x].w;
          }
        }
    }
    uint4 o;
    o.x = pack_bf16x2(a.x, a.y);
    o.y = pack_bf16x2(a.z, a.w);
    o.z = pack_bf16x2(b.x, b.y);
    o.w = pack_bf16x2(b.z, b.w);
    out[i] = o;
  }
}

// ==================================================================================================
// 2-CTA variant (cta_group::2): a CTA pair on one TPC computes a 256 x BN tile.  Each CTA stages
// its own 128 rows of A and HALF of the B tile (BN/2 weight rows), the leader issues
// tcgen05.mma.cta_group::2 (UMMA M=256) which reads both CTAs' shared memory, and each CTA drains
// its own 128 x BN accumulator from its TMEM.  Per-SM operand ingest per k-block drops from
// 16 KB + BN*128 B to 16 KB + BN*64 B for the same MMA work — the 1-CTA kernel is ingest-bound,
// this one moves the bound back to the tensor pipe.
// ==================================================================================================
// Eight warps store: a gated tile takes four of them some 14 us, which is longer than its products up to K = 2304 and stands behind the last
// tile of any reduction.
constexpr int GEMM2_THREADS = 320;
template <int BN>
struct Gemm2Cfg {
  static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2;        // 16 KB: this CTA's 128 rows
  static constexpr int B_BYTES = (BN / 2) * GEMM_BK * 2;       // this CTA's half of the B tile
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = GEMM_SMEM_BUDGET / STAGE_BYTES > 8 ? 8 : GEMM_SMEM_BUDGET / STAGE_BYTES;
  static constexpr int TMEM_COLS = BN > 128 ? 512 : 256;       // two accumulators, a power of two
  static constexpr int SMEM_TOTAL = STAGES * STAGE_BYTES + 1024 + 256 + 8 * 4096;
};

__device__ __forceinline__ void mbar_expect_tx_cluster(uint32_t bar_cluster_addr, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(
                   bar_cluster_addr),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr)
               : "memory");
}
__device__ __forceinline__ void tma_load_2d_2sm(void* smem_dst, const void* tmap, int c0, int c1,
                                                uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(tmap), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_2sm(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_2sm(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void umma_bf16_2sm(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                              uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive on the barrier at the same shared-memory offset in BOTH CTAs of the pair
__device__ __forceinline__ void umma_commit_2sm(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
__host__ __device__ constexpr uint32_t make_idesc_2sm(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(256 >> 4) << 24);
}

template <int BN, int kAct = ACT_NONE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM2_THREADS, 1)
    gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a,
                      const __grid_constant__ CUtensorMap tmap_b, bf16* __restrict__ C, int M,
                      int N, int K, long long ldc, GateArgs gate, int fixed_w) {
  constexpr bool kSwiGLU = kAct != ACT_NONE;
  using Cfg = Gemm2Cfg<BN>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tmem_full = empty + STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  uint8_t* epi_smem = smem + STAGES * Cfg::STAGE_BYTES + 256;  // 8 warps x 4 KB transpose patches

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int m_tiles = (M + 255) / 256;
  const int n_tiles = (N + BN - 1) / BN;  // (BN = 160, 192: the last one may be ragged, its rows of W behind the end are zeros)
  const int num_tiles = m_tiles * n_tiles;
  const int k_blocks = K / GEMM_BK;
  const int cluster_id = blockIdx.x >> 1, num_clusters = gridDim.x >> 1;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full + s, 2);   // (leader's copy is the live one) one arrive per CTA's producer
      mbar_init(empty + s, 1);  // multicast tcgen05.commit from the leader
    }
    mbar_init(tmem_full + 0, 1);
    mbar_init(tmem_full + 1, 1);
    mbar_init(tmem_empty + 0, 16);  // 8 epilogue warps x 2 CTAs, all arriving at the leader
    mbar_init(tmem_empty + 1, 16);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc_2sm(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // peer barriers are initialised before anybody signals them
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  int early = 0;  // (as above)
  if (warp == 0 && lane == 0) {
    const int row = cluster_id / m_tiles * BN + (int)rank * (BN / 2);
    for (int kb = 0; kb < STAGES && kb < k_blocks; ++kb) {
      if (fixed_w) {
        const uint32_t lfull = mapa_shared(full + kb, 0);
        mbar_expect_tx_cluster(lfull, Cfg::STAGE_BYTES);
        tma_load_2d_2sm(smem + kb * Cfg::STAGE_BYTES + Cfg::A_BYTES, &tmap_b, kb * GEMM_BK, row, lfull);
        ++early;
      } else {
        tma_prefetch_2d(&tmap_b, kb * GEMM_BK, row);
      }
    }
  }
  __syncwarp();
  follow_previous(gate.bias);

  if (warp == 0) {
    // ===== TMA producer (both CTAs): own A rows + own half of B, completion on the LEADER =====
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int tile = cluster_id; tile < num_tiles; tile += num_clusters) {
        const int m_blk = tile % m_tiles, n_blk = tile / m_tiles;
        int kb = 0;  // (as above)
        for (; kb < early; ++kb)
          tma_load_2d_2sm(smem + kb * Cfg::STAGE_BYTES, &tmap_a, kb * GEMM_BK, m_blk * 256 + (int)rank * 128, mapa_shared(full + kb, 0));
        if (early > 0) {
          stage = early % STAGES;
          phase = early / STAGES;
          early = 0;
        }
        for (; kb < k_blocks; ++kb) {
          uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          const uint32_t lfull = mapa_shared(full + stage, 0);
          mbar_wait(empty + stage, phase ^ 1u);
          mbar_expect_tx_cluster(lfull, Cfg::STAGE_BYTES);
          tma_load_2d_2sm(sb, &tmap_b, kb * GEMM_BK, n_blk * BN + (int)rank * (BN / 2), lfull);
          tma_load_2d_2sm(sa, &tmap_a, kb * GEMM_BK, m_blk * 256 + (int)rank * 128, lfull);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ===== MMA issuer: leader CTA only =====
    if (leader) {
      constexpr uint32_t idesc = make_idesc_2sm(BN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int tile = cluster_id; tile < num_tiles; tile += num_clusters) {
        mbar_wait(tmem_empty + acc, acc_phase ^ 1u);
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(acc * BN);
        for (int kb = 0; kb < k_blocks; ++kb) {
          mbar_wait(full + stage, phase);
          tc_fence_after();
          if (elect_one()) {
            const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
            const uint32_t sb = sa + Cfg::A_BYTES;
#pragma unroll
            for (int k = 0; k < GEMM_BK / 16; ++k) {
              umma_bf16_2sm(tmem_d, make_smem_desc(sa + k * 32), make_smem_desc(sb + k * 32), idesc,
                            (kb > 0 || k > 0) ? 1u : 0u);
            }
            umma_commit_2sm(empty + stage);
            if (kb == k_blocks - 1) umma_commit_2sm(tmem_full + acc);
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1u;
      }
    }
  } else {
    // ===== epilogue (both CTAs): own 128 rows of the 256-row tile, every other 64 columns to four of the warps =====
    const int quarter = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = cluster_id; tile < num_tiles; tile += num_clusters) {
      const int m_blk = tile % m_tiles, n_blk = tile / m_tiles;
      mbar_wait(tmem_full + acc, acc_phase);
      tc_fence_after();
      const int row0 = m_blk * 256 + (int)rank * 128 + quarter * 32;
      constexpr int OUT_BN = kSwiGLU ? BN / 2 : BN;
      bf16* ctile = C + (long long)row0 * ldc + (long long)n_blk * OUT_BN;
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN);
      epilogue_rows<BN, kAct>(taddr, ctile, ldc, row0, M, epi_smem + (warp - 2) * EPI_SMEM_PER_WARP, lane,
                                kAct == ACT_CLAMPED && gate.bias ? gate.bias + (long long)n_blk * BN : nullptr, gate.limit,
                                min(BN, N - n_blk * BN), (warp - 2) / 4 * 64, 128);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_shared(tmem_empty + acc, 0));
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // nobody frees TMEM / exits while the peer may still signal or read
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_2sm(tmem_base, Cfg::TMEM_COLS);
  }
}

// ---- host side: tensor maps + launch ---------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) ==
            cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
    else
      cudaGetLastError();
  });
  return fn;
}

struct TmapKey {
  const void* ptr;
  long long rows, cols;
  int box_rows;
  bool operator==(const TmapKey& o) const {
    return ptr == o.ptr && rows == o.rows && cols == o.cols && box_rows == o.box_rows;
  }
};
struct TmapKeyHash {
  size_t operator()(const TmapKey& k) const {
    size_t h = std::hash<const void*>()(k.ptr);
    h ^= std::hash<long long>()(k.rows * 1315423911LL + k.cols * 2654435761LL + k.box_rows) +
         0x9e3779b97f4a7c15ULL + (h << 6) + (h >> 2);
    return h;
  }
};

// bf16 row-major [rows, cols] -> tiled map with box {64 cols, box_rows rows}, 128B swizzle
// (ld: elements between rows, 0 = dense)
int get_tmap(const void* ptr, long long rows, long long cols, int box_rows, CUtensorMap* out, long long ld) {
  static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
  static std::mutex mu;
  if (ld == 0) ld = cols;
  TmapKey key{ptr, rows, cols + (ld << 24), box_rows};
  {
    std::lock_guard<std::mutex> g(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
      *out = it->second;
      return B200Q_OK;
    }
  }
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled entry point unavailable (driver too old / no driver)");
    return B200Q_ECUDA;
  }
  cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)GEMM_BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMap m;
  CUresult r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), gdim, gstride,
                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d) for [%lld,%lld] box_rows=%d ptr=%p", (int)r,
              rows, cols, box_rows, ptr);
    return B200Q_ECUDA;
  }
  {
    std::lock_guard<std::mutex> g(mu);
    if (cache.size() > 4096) cache.clear();
    cache[key] = m;
  }
  *out = m;
  return B200Q_OK;
}

int get_page_tmap(const void* kv, int D, CUtensorMap* out) {
  static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
  static std::mutex mu;
  const TmapKey key{kv, 0, D, 16};
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return B200Q_OK;
  }
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled entry point unavailable (driver too old / no driver)");
    return B200Q_ECUDA;
  }
  cuuint64_t gdim[4] = {64, 8, (cuuint64_t)(D / 64), 0x0ffffffeull};
  cuuint64_t gstride[3] = {(cuuint64_t)D * 2, 128, (cuuint64_t)D * 16};
  cuuint32_t box[4] = {64, 8, (cuuint32_t)(D / 64), 2};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUtensorMap m;
  CUresult r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(kv), gdim, gstride, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d) for a page pool at %p", (int)r, kv);
    return B200Q_ECUDA;
  }
  if (cache.size() > 4096) cache.clear();
  cache[key] = m;
  *out = m;
  return B200Q_OK;
}

int get_head_rows_tmap(const void* p, int n_q, int D, long long stride, int heads, int rows, int cols, CUtensorMap* out) {
  static std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> cache;
  static std::mutex mu;
  const TmapKey key{p, stride << 16 | n_q, D, (heads * 128 + rows) * 64 + cols - 1};
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return B200Q_OK;
  }
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled entry point unavailable (driver too old / no driver)");
    return B200Q_ECUDA;
  }
  cuuint64_t gdim[3] = {(cuuint64_t)D, (cuuint64_t)n_q, 0x0ffffffeull};
  cuuint64_t gstride[2] = {(cuuint64_t)D * 2, (cuuint64_t)stride * 2};
  cuuint32_t box[3] = {(cuuint32_t)cols, (cuuint32_t)heads, (cuuint32_t)rows};
  cuuint32_t estr[3] = {1, 1, 1};
  CUtensorMap m;
  CUresult r = enc(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled failed (%d) for rows of %d heads of %d at %p", (int)r, n_q, D, p);
    return B200Q_ECUDA;
  }
  if (cache.size() > 4096) cache.clear();
  cache[key] = m;
  *out = m;
  return B200Q_OK;
}

int num_sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

// ---- scratch of partial tiles -----------------------------------------------------------------------
// Whoever orders its products by itself has its own, so that nobody's parts are overwritten before they are added: a model (its passes run
// one behind the other; a piece of its workspace), a stream, and a graph in the making, whose replays may run beside the stream that it was
// captured on.  Nothing here waits for the device or frees: either would end other threads' captures.  A stream's buffer stays with its
// handle (which comes back for another stream only once the work of the one before is done), a graph's comes back with the last of the
// graph and its executables and serves whoever asks next.  Sizes go by powers of two from 1 MiB, so that streams hold twice what their
// largest product needs at most.
struct ModelScratch {
  void* p = nullptr;
  size_t bytes = 0;
};
static thread_local ModelScratch t_model_scratch;
SplitScratchOf::SplitScratchOf(void* p, size_t bytes) : p_(t_model_scratch.p), bytes_(t_model_scratch.bytes) { t_model_scratch = {p, bytes}; }
SplitScratchOf::~SplitScratchOf() { t_model_scratch = {p_, bytes_}; }

namespace {
struct SplitBuffer {
  void* p = nullptr;
  size_t bytes = 0;
  int device = 0;
  cudaStream_t stream = nullptr;
  unsigned long long capture = 0;  // of the graph that owns it; 0: the stream does
  std::atomic<bool> free{false};   // the graph is gone
};
std::mutex g_split_mu;
std::vector<SplitBuffer*> g_split;  // (entries stay: a graph's callback names its own)
}  // namespace

static int splitk_scratch(int splits, int M, int N, cudaStream_t st, float** out) {
  const size_t need = (size_t)splits * M * N * sizeof(float);
  B200Q_CHECK_ARG(need <= SPLIT_BYTES, "split-K scratch too small for M=%d N=%d splits=%d", M, N, splits);
  if (need <= t_model_scratch.bytes) {
    *out = (float*)t_model_scratch.p;
    return B200Q_OK;
  }
  int device = 0;
  unsigned long long capture = 0;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  cudaGraph_t graph = nullptr;
  const cudaGraphNode_t* nodes = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  size_t n_nodes = 0;
  cudaGetDevice(&device);
  if (cudaStreamGetCaptureInfo_v3(st, &status, &capture, &graph, &nodes, &edges, &n_nodes) != cudaSuccess ||
      status != cudaStreamCaptureStatusActive) {
    cudaGetLastError();  // (a product that cannot run here fails at its launch)
    capture = 0;
  }
  std::lock_guard<std::mutex> lock(g_split_mu);
  SplitBuffer *own = nullptr, *spare = nullptr;
  for (SplitBuffer* b : g_split) {
    if (b->device != device || b->bytes < need) continue;
    if (b->free.load()) {
      if (!spare || b->bytes < spare->bytes) spare = b;
    } else if (b->stream == st && b->capture == capture && (!own || b->bytes > own->bytes)) {
      own = b;
    }
  }
  if (!own) {
    own = spare;
    if (!own) {
      size_t bytes = (size_t)1 << 20;
      while (bytes < need) bytes *= 2;
      // (refused to every thread while any stream is captured in the default mode, unless the thread says that it knows)
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      void* p = nullptr;
      cudaThreadExchangeStreamCaptureMode(&mode);
      const cudaError_t e = cudaMalloc(&p, bytes);
      cudaThreadExchangeStreamCaptureMode(&mode);
      B200Q_CUDA(e);
      own = new SplitBuffer;
      own->p = p;
      own->bytes = bytes;
      own->device = device;
      own->free.store(true);
      g_split.push_back(own);
    }
    if (capture) {
      cudaUserObject_t held;
      B200Q_CUDA(cudaUserObjectCreate(&held, own, [](void* b) { static_cast<SplitBuffer*>(b)->free.store(true); }, 1,
                                      cudaUserObjectNoDestructorSync));
      B200Q_CUDA(cudaGraphRetainUserObject(graph, held, 1, cudaGraphUserObjectMove));
    }
    own->stream = st;
    own->capture = capture;
    own->free.store(false);
  }
  *out = (float*)own->p;
  return B200Q_OK;
}

// (no other thread's product on the same stream between a product and the sum of its parts, whichever kernels they take)
static std::mutex g_split_pair;
// product leaves its parts in ws; they are summed into C, or by whoever reads C where partials_out asks for them
template <typename F>
static int split_product(float* ws, void* C, int M, int N, int splits, cudaStream_t st, const float** partials_out, F&& product) {
  std::unique_lock<std::mutex> together(g_split_pair, std::defer_lock);
  if (!partials_out) together.lock();
  const int rc = product();
  if (rc) return rc;
  if (partials_out) {
    *partials_out = ws;
    return B200Q_OK;
  }
  const long long mn8 = (long long)M * N / 8;
  const int most = 8 * num_sms(), grid = (int)((mn8 + 255) / 256 < most ? (mn8 + 255) / 256 : most);
  B200Q_CUDA(launch_early(splitk_reduce_kernel, grid, 256, 0, st, 1, (const float4*)ws, (uint4*)C, mn8, splits));
  count_launch();
  return B200Q_OK;
}

template <int BN, int kAct = ACT_NONE>
static int launch_gemm(const void* A, const void* W, void* C, int M, int N, int K,
                       cudaStream_t st, int splits = 1, const float** partials_out = nullptr, long long ldc = 0,
                       GateArgs gate = {nullptr, 0.f}, bool fixed_w = false) {
  using Cfg = GemmCfg<BN>;
  CUtensorMap ta, tb;
  const int a_rows = M < GEMM_BM ? (M + 7) & ~7 : GEMM_BM;  // one m-tile: load only the rows that exist
  int rc = get_tmap(A, M, K, a_rows, &ta);
  if (rc) return rc;
  rc = get_tmap(W, N, K, BN, &tb);
  if (rc) return rc;
  auto kern = gemm_bf16_kernel<BN, kAct>;
  static bool attr_set = false;
  if (!attr_set) {
    B200Q_CUDA(
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_TOTAL));
    attr_set = true;
  }
  const int tiles = ((M + GEMM_BM - 1) / GEMM_BM) * (N / BN) * splits;
  const int grid = tiles < num_sms() ? tiles : num_sms();
  float* ws = nullptr;
  if (splits > 1 && (rc = splitk_scratch(splits, M, N, st, &ws))) return rc;
  auto product = [&]() -> int {
    B200Q_CUDA(launch_early(kern, grid, GEMM_THREADS, Cfg::SMEM_TOTAL, st, 1, ta, tb, (bf16*)C, M, N, K, splits, ws, a_rows * GEMM_BK * 2,
                            ldc > 0 ? ldc : (kAct != ACT_NONE ? N / 2 : N), gate, (int)fixed_w));
    count_launch();
    return B200Q_OK;
  };
  return splits > 1 ? split_product(ws, C, M, N, splits, st, partials_out, product) : product();
}

static int g_gemm2_pairs = 0;  // co-resident CTA pairs reported by the occupancy query

template <int BN, int kAct = ACT_NONE>
static int launch_gemm2(const void* A, const void* W, void* C, int M, int N, int K,
                        cudaStream_t st, long long ldc = 0, GateArgs gate = {nullptr, 0.f}, bool fixed_w = false) {
  using Cfg = Gemm2Cfg<BN>;
  CUtensorMap ta, tb;
  int rc = get_tmap(A, M, K, GEMM_BM, &ta);
  if (rc) return rc;
  rc = get_tmap(W, N, K, BN / 2, &tb);
  if (rc) return rc;
  auto kern = gemm2_bf16_kernel<BN, kAct>;
  static bool attr_set = false;
  if (!attr_set) {
    B200Q_CUDA(
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_TOTAL));
    attr_set = true;
  }
  const int tiles = ((M + 255) / 256) * ((N + BN - 1) / BN);
  // the tile loop is static round-robin over CO-RESIDENT CTA pairs: size the grid by what the
  // hardware can really keep resident at once (GPC/TPC pairing can make this < SMs/2)
  static int pairs = 0;
  if (pairs == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(num_sms() & ~1);
    cfg.blockDim = dim3(GEMM2_THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM_TOTAL;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = num_sms() / 2;
    }
    pairs = n < num_sms() / 2 ? n : num_sms() / 2;
    g_gemm2_pairs = pairs;
  }
  const int grid = 2 * (tiles < pairs ? tiles : pairs);
  B200Q_CUDA(launch_early(kern, grid, GEMM2_THREADS, Cfg::SMEM_TOTAL, st, 1, ta, tb, (bf16*)C, M, N, K,
                          ldc > 0 ? ldc : (kAct != ACT_NONE ? N / 2 : N), gate, (int)fixed_w));
  count_launch();
  return B200Q_OK;
}

// Which kernel and tile: the least (rounds of the persistent loop) x (time of a round).  Rounds: tiles over 148 SMs, or tiles of 256 rows
// over 74 CTA pairs.  A round's time beside the 128 x 256 tile's (K 14336, one round, us: 85.5; pair 256 x 256 70-74, pair 256 x 128
// 50.7, 128 x 128 55, 128 x 64 50; pairs of 256 x 192 59, 256 x 160 55, whose last tile of a row may be ragged; K 8192 the same shares,
// 49.5 / 41.5 / 29.8 / 32 / 29): the pair kernels fetch half the weight rows per SM, narrow tiles are bound by what they fetch.  Before, the pair kernel was taken for whole rounds of 74 tiles only:
// 768 x 3584 x 14336 86 -> 71 us, 512 x 4096 x 14336 58 -> 53, 1536 x 2048 x 8192 50 -> 43.  The widths of 160 and 192 fill rounds that 256
// leaves half empty: 750 x 3584 x 14336 69 -> 59 us, 1500 x 4096 x 14336 140 -> 125, 1024 x 6144 x 4096 42 -> 37, 3000 x 2048 x 8192 81 -> 73
// (108 sizes looked at: the rule is within 1 % of the best tile for 94 of them, at worst 16 % off at 300 x 2048).
struct TileChoice {
  bool pair;
  int bn;
  double rounds;  // rounds x a round's time, in rounds of 128 x 256 tiles
};
static TileChoice choose_tile(int M, int N, bool gated, bool pairs) {
  const struct {
    bool pair;
    int bn;
    double cost;
  } all[7] = {{true, 256, 0.84},  {false, 256, 1.0},   {true, 192, 0.70},  {true, 160, 0.65},
              {true, 128, 0.595}, {false, 128, 0.645}, {false, 64, 0.585}};
  TileChoice best{false, N % 256 == 0 ? 256 : N % 128 == 0 ? 128 : 64, 1e30};
  for (const auto& c : all) {
    const bool ragged = c.bn == 160 || c.bn == 192;
    if ((ragged ? N < c.bn : N % c.bn != 0) || (gated && c.bn != 256) || (c.pair && (!pairs || M <= GEMM_BM))) continue;
    const long long rows = c.pair ? 256 : GEMM_BM, slots = c.pair ? num_sms() / 2 : num_sms();
    const long long tiles = (M + rows - 1) / rows * ((N + c.bn - 1) / c.bn);
    const double t = (double)((tiles + slots - 1) / slots) * c.cost;
    if (t < best.rounds - 1e-9) best = {c.pair, c.bn, t};
  }
  return best;
}

// Rows of A in a tile of gemm_rows.cu, 0 where the tiles above are faster.  A round there costs, in the same measure (0.38 us a k-block of
// 64), what stands here, its start and end 2 us more.  Measured with 13 shapes of the built-in models x 25 row counts from 80 to 4608 and
// every tile: the rule takes 0.956 of the time without these tiles on average, at worst 1.008, where always knowing the best would take
// 0.949.  us, without / with: 300 x 128256 x 4096 317 / 248, 513 rows 497 / 416, 128 rows 181 / 171; 300 x 8192 x 3584 22.9 / 18.3; 900 x
// 3584 x 4096 24 / 21; 1600 x 4096 x 14336 148 / 130; 4608 x 3584 x 14336 373 / 331.  Up to 128 rows only for vocabulary sizes, whose tiles
// of 256 columns leave the last round half empty (what has fewer columns goes to gemm_skinny.cu).  Gated products gain nothing here: a
// gate and an up tile per CTA leave fewer tiles than the rounds want.
//
// Parts of K (up to 8, of 4 k-blocks or more, M x parts up to 1536: 800 rows in two are 4 % slower, 750 10 % faster, and a model's scratch
// holds 2048) are what fills the rounds of a product of few columns.  A round is then bound by its products or, with few pairs at work, by
// the weights they fetch; the parts are written and summed in 0.3 us a MB, 0.2 us each and 1.1 us (the two kernels overlap), another round
// costs 2 us; 3 % have to be gained.  17 shapes x 20 row counts from 129 to 1000, sums included: the rule takes 0.937 of the time without
// parts on average and 1.002 at worst, where always knowing the best would take 0.92.  us, without / with: 150 x 3584 x 14336 38.2 / 29.3,
// 200 x 4096 x 14336 39.0 / 34.5; 256 x 2560 x 10240 32.4 / 20.5; 300 x 2048 x 8192 27.3 / 17.5, 512 rows 28.0 / 20.9, 750 rows 28.8 / 26.3;
// 400 x 4096 x 14336 49.1 / 46.0.  From K = 2560 to 3584 parts have to gain 0.8 us more: another 1469 sizes (128 to 8192 columns, K 512 to 14336,
// 129 to 768 rows, every tile and number of parts) showed 2 to 9 % lost there (513 x 1536 x 3072 14.6 in two parts, 13.4 whole; 256 x 3072 x 3072
// 14.6 / 13.6).  With that and the parts that choose_splits still has, the rule takes 1.008 of the best's time there and 0.857 of the
// time without these tiles, at worst 1.044 (20 sizes above 1.02).
struct RowsTile {
  int rows, splits;
};
static RowsTile rows_tile(int M, int N, int K, const TileChoice& other, bool may_split) {
  if (M <= 64 || (M <= GEMM_BM && N < num_sms() * 256) || N % 128 != 0) return {0, 1};
  const struct {
    int rows;
    double cost;
  } all[8] = {{64, 0.43}, {96, 0.45}, {128, 0.49}, {160, 0.575}, {192, 0.645}, {224, 0.70}, {256, 0.83}, {320, 1.12}};
  const int pairs = num_sms() / 2, kb = K / GEMM_BK, most = may_split && N <= 8192 ? 8 : 1;
  const double k_block = 0.3817;
  double least = 0.95 * k_block * kb * other.rounds;
  RowsTile best{0, 1};
  for (const auto& c : all)
    for (int s = 1; s <= most && (s == 1 || (kb / s >= 4 && s * M <= 1536)); ++s) {
      const long long tiles = (long long)((N / 128 + 1) / 2) * ((M + c.rows - 1) / c.rows) * s;
      const double rounds = (double)((tiles + pairs - 1) / pairs);
      double t = rounds * c.cost * k_block * ((kb + s - 1) / s);
      if (s > 1) {
        const double weights = 0.124e-6 * 2.0 * N * K * pairs / (tiles < pairs ? tiles : pairs);
        t = 1.03 * ((t > weights ? t : weights) + 2.0 * rounds + 1.1 + s * (0.2 + 0.3e-6 * 4.0 * M * N)) + (kb >= 40 && kb <= 56 ? 0.8 : 0.0);
      } else {
        t += 2.0;
      }
      if (t < least) {
        least = t;
        best = {c.rows, s};
      }
    }
  return best;
}

int g_gemm_force_bn = 0;  // test hook: 0 = heuristic
int g_gemm_splitk = 0;    // 0 = auto, 1 = never, n > 1 = force n splits where legal (tests)

bool batch_invariant() {
  static const bool v = [] {
    const char* e = getenv("B200Q_BATCH_INVARIANT");
    return e && e[0] == '1';
  }();
  return v || g_gemm_splitk == 1;  // (the hook without splits stands for the variable)
}

// split-K factor for a decode-sized projection that gemm_skinny.cu leaves (1 = do not split): when it has too few 128-wide
// output tiles to put every SM on the weight stream, split the reduction so that tiles x splits ~ #SMs.
// 193 to 256 rows whose tiles and parts are 128 CTAs (1024 columns in 8 parts, 2048 in 4), parts of 10 to 28 k-blocks: faster than the
// parts of gemm_rows.cu, whose tiles of 256 columns leave a poor choice there (us, here / there: 256 x 1024 x 5120 11.1 / 12.6, x 12288
// 14.9 / 16.2; 256 x 2048 x 3072 11.6 / 13.5, x 4096 12.9 / 14.6, x 7168 15.7 / 16.3; but x 12288 20.5 / 20.4, 2048 x 2048 10.4 / 10.0 in
// whole tiles; 112, 120 or 144 CTAs lose 2 to 10 %, fewer rows are even).  Others of 129 to 256 rows are split here only where a test
// asks for a count.
static int choose_splits(int M, int N, int K, bool invariant, int forced_bn) {
  const int want = invariant ? 1 : g_gemm_splitk;  // 0 = auto, 1 = off, >1 = forced (tests)
  if (want == 1 || forced_bn != 0 || M > 256 || N % 128 != 0 || N > 8192) return 1;
  const int tiles = ((M + GEMM_BM - 1) / GEMM_BM) * (N / 128);
  const int kb = K / GEMM_BK;
  if (want == 0 && M > GEMM_BM) {
    for (int s = 8; s >= 4; s /= 2)
      if (M > 192 && tiles * s == 128 && kb % s == 0 && kb / s >= 10 && kb / s <= 28) return s;
    return 1;
  }
  int splits = want > 1 ? want : 1;
  if (want == 0 && tiles * 2 <= num_sms()) {
    for (int sN = 8; sN >= 2; --sN)
      if (kb % sN == 0 && kb / sN >= 8 && tiles * sN <= num_sms() + num_sms() / 8) {
        splits = sN;
        break;
      }
  }
  return (splits > 1 && splits <= 8 && kb % splits == 0) ? splits : 1;
}
int g_gemm_mode = 0;      // 0 = auto, 1 = force 1-CTA kernels, 2 = force the 2-CTA kernel

// Up to 128 rows go to gemm_skinny.cu unless a hook asks for one of the kernels here, or results must not depend on the number of
// rows (its splits depend on it, and the kernels here that larger steps use add in another order).
static bool use_skinny(int M, int N, int K, bool gated) {
  return g_gemm_mode == 0 && g_gemm_force_bn == 0 && g_gemm_splitk == 0 && !batch_invariant() && gemm_skinny_ok(M, N, K, gated);
}

// the tile of gemm_rows.cu that a product takes, none where a hook asks for other kernels; parts only where the sums may depend on the rows
static RowsTile rows_tile_of(int M, int N, int K) {
  if (g_gemm_mode != 0 || g_gemm_force_bn != 0) return {0, 1};
  return rows_tile(M, N, K, choose_tile(M, N, false, true), g_gemm_splitk == 0 && !batch_invariant());
}
// the same for a product that may go to the kernels that `linear` looks at first
static RowsTile rows_tile_behind(int M, int N, int K) {
  if (use_skinny(M, N, K, false) || choose_splits(M, N, K, batch_invariant(), g_gemm_force_bn) > 1) return {0, 1};
  return rows_tile_of(M, N, K);
}
// choose_splits for a product on st; more than 128 rows go on without parts where there is no memory for them
static int choose_splits(int M, int N, int K, int forced_bn, cudaStream_t st) {
  const int splits = choose_splits(M, N, K, batch_invariant(), forced_bn);
  float* ws = nullptr;
  if (splits <= 1 || M <= GEMM_BM || splitk_scratch(splits, M, N, st, &ws) == B200Q_OK) return splits;
  cudaGetLastError();
  return 1;
}
// the same for the tiles of gemm_rows.cu
static RowsTile rows_tile_of(int M, int N, int K, cudaStream_t st, float** ws) {
  const RowsTile r = rows_tile_of(M, N, K);
  if (r.splits <= 1 || splitk_scratch(r.splits, M, N, st, ws) == B200Q_OK) return r;
  cudaGetLastError();
  return rows_tile(M, N, K, choose_tile(M, N, false, true), false);
}


// ------------------------------------------------------------------------------------------------
// Grouped GEMM: many small GEMMs that share K and N run as ONE persistent launch — the experts of a
// routed feed-forward (group = expert, rows = the (token, choice) pairs sorted by expert) or per-head
// projections (group = head, every group has all rows and its own column slice of A and C).
//   C[row, g*c_gx + n] = sum_k A[row, g*a_gx + k] * W[g*N + n, k]
// Same pipeline as gemm_bf16_kernel (TMA producer warp, tcgen05.mma issuer warp, 4 epilogue warps, smem
// ring, two TMEM accumulator stages); only the tile walk differs: m-tile i is {group, first row, end row}
// read from a device table that the routing kernel wrote (tab != NULL, *n_mt entries), or computed
// (tab == NULL: every group has ceil(M/128) m-tiles).  An A box always holds 128 rows: rows past a
// group's end belong to the next group (or are zero-filled past the matrix) and their products are
// never stored.  kOutF32: fp32 output (logits, latent-space queries) instead of bf16.
// ------------------------------------------------------------------------------------------------
struct GroupedArgs {
  const int4* tab;     // [*n_mt] {group, row0, row_end, 0} or NULL
  const int32_t* n_mt; // device count of m-tiles (tab != NULL)
  int M, groups;       // tab == NULL: rows of every group, number of groups
  int a_gx, c_gx;      // column offset per group in A / in C (elements)
  long long ldc;
  int ahead;           // k-blocks of weights per CTA that are asked into L2 before the kernel before has ended
  int max_mt;          // entries that the table has room for
};
constexpr int GROUPED_TAB = 64;  // entries that a CTA keeps
constexpr long long GROUPED_AHEAD_BYTES = 64000000;

template <int BN, bool kOutF32>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_grouped_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                        void* __restrict__ Cv, int N, int K, GroupedArgs ga) {
  using Cfg = GemmCfg<BN>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tmem_full = empty + STAGES;
  uint64_t* tmem_empty = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  uint8_t* epi_smem = smem + STAGES * Cfg::STAGE_BYTES + 256;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    mbar_init(tmem_full + 0, 1);
    mbar_init(tmem_full + 1, 1);
    mbar_init(tmem_empty + 0, 4);
    mbar_init(tmem_empty + 1, 4);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  if (warp == 0 && lane == 0 && ga.ahead > 0 && (int)blockIdx.x < ga.groups * (N / BN)) {
    // (the table is not known yet: this CTA's first tile if every group has one m-tile)
    const int row = (int)blockIdx.x % ga.groups * N + (int)blockIdx.x / ga.groups * BN;
    for (int kb = 0; kb < min(ga.ahead, K / GEMM_BK); ++kb) tma_prefetch_2d(&tmap_b, kb * GEMM_BK, row);
  }
  __syncwarp();
  follow_previous();
  // (the first entries come while their number does, not behind it)
  __shared__ int4 first_tab[GROUPED_TAB];
  const int mt_per_group = (ga.M + GEMM_BM - 1) / GEMM_BM;
  int m_tiles = mt_per_group * ga.groups;
  if (ga.tab) {
    if ((int)threadIdx.x < min(ga.max_mt, GROUPED_TAB)) first_tab[threadIdx.x] = ga.tab[threadIdx.x];
    m_tiles = *ga.n_mt;
    __syncthreads();
  }
  const int n_tiles = N / BN;
  const int num_tiles = m_tiles * n_tiles;
  const int k_blocks = K / GEMM_BK;
  auto tile_of = [&](int tile, int& g, int& row0, int& row_end, int& n_blk) {
    const int mt = tile % m_tiles;
    n_blk = tile / m_tiles;
    if (ga.tab) {
      const int4 e = mt < GROUPED_TAB ? first_tab[mt] : ga.tab[mt];
      g = e.x;
      row0 = e.y;
      row_end = e.z;
    } else {
      g = mt / mt_per_group;
      row0 = (mt % mt_per_group) * GEMM_BM;
      row_end = ga.M;
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
        int g, row0, row_end, n_blk;
        tile_of(tile, g, row0, row_end, n_blk);
        for (int kb = 0; kb < k_blocks; ++kb) {
          mbar_wait(empty + stage, phase ^ 1u);
          uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          mbar_expect_tx(full + stage, (uint32_t)(Cfg::A_BYTES + Cfg::B_BYTES));
          tma_load_2d(sa, &tmap_a, g * ga.a_gx + kb * GEMM_BK, row0, full + stage);
          tma_load_2d(sb, &tmap_b, kb * GEMM_BK, g * N + n_blk * BN, full + stage);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = make_idesc(BN);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      mbar_wait(tmem_empty + acc, acc_phase ^ 1u);
      tc_fence_after();
      const uint32_t tmem_d = tmem_base + (uint32_t)(acc * BN);
      for (int kb = 0; kb < k_blocks; ++kb) {
        mbar_wait(full + stage, phase);
        tc_fence_after();
        if (elect_one()) {
          const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
          const uint32_t sb = sa + Cfg::A_BYTES;
#pragma unroll
          for (int k = 0; k < GEMM_BK / 16; ++k)
            umma_bf16(tmem_d, make_smem_desc(sa + k * 32), make_smem_desc(sb + k * 32), idesc,
                      (kb > 0 || k > 0) ? 1u : 0u);
          umma_commit(empty + stage);
          if (kb == k_blocks - 1) umma_commit(tmem_full + acc);
        }
        __syncwarp();
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  } else {
    const int quarter = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      int g, row0, row_end, n_blk;
      tile_of(tile, g, row0, row_end, n_blk);
      mbar_wait(tmem_full + acc, acc_phase);
      tc_fence_after();
      const int r0 = row0 + quarter * 32;
      const long long col0 = (long long)g * ga.c_gx + (long long)n_blk * BN;
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN);
      if constexpr (kOutF32) {
        const int row = r0 + lane;
        float* crow = reinterpret_cast<float*>(Cv) + (long long)row * ga.ldc + col0;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
          uint32_t v[32];
          tmem_ld32(taddr + (uint32_t)c0, v);
          tmem_ld_wait();
          if (row < row_end) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              st_v4(crow + c0 + 4 * j, make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
          }
        }
      } else {
        bf16* ctile = reinterpret_cast<bf16*>(Cv) + (long long)r0 * ga.ldc + col0;
        epilogue_rows<BN, ACT_NONE>(taddr, ctile, ga.ldc, r0, row_end, epi_smem + (warp - 2) * EPI_SMEM_PER_WARP, lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tmem_empty + acc);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

template <int BN, bool kOutF32>
static int launch_grouped(const CUtensorMap& ta, const CUtensorMap& tb, void* C, int N, int K, const GroupedArgs& ga,
                          int max_tiles, cudaStream_t st) {
  using Cfg = GemmCfg<BN>;
  auto kern = gemm_grouped_kernel<BN, kOutF32>;
  static bool attr_set = false;
  if (!attr_set) {
    B200Q_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_TOTAL));
    attr_set = true;
  }
  const int grid = max_tiles < num_sms() ? max_tiles : num_sms();
  B200Q_CUDA(launch_early(kern, grid, GEMM_THREADS, Cfg::SMEM_TOTAL, st, 1, ta, tb, C, N, K, ga));
  count_launch();
  return B200Q_OK;
}

}  // namespace b200q

using namespace b200q;

// shared body of the fused gate_up GEMMs (SwiGLU / GeGLU)
template <int kAct>
static int gemm_gated(const char* what, const void* A, const void* W, void* C, int M, int N, int K,
                      void* stream, long long ldc = 0, GateArgs gate = {nullptr, 0.f}, bool fixed_w = false) {
  B200Q_CHECK_ARG(M >= 0 && N > 0 && K > 0 && K % GEMM_BK == 0 && N % 256 == 0,
                  "%s: unsupported shape M=%d N=%d K=%d (need K%%64==0, N%%256==0)", what, M, N, K);
  B200Q_CHECK_ARG((reinterpret_cast<uintptr_t>(A) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(W) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(C) & 15) == 0,
                  "%s: operands must be 16-byte aligned", what);
  if (M == 0) return B200Q_OK;
  cudaStream_t st = as_stream(stream);
  if (use_skinny(M, N, K, true))
    return gemm_skinny(A, W, C, M, N, K, kAct, ldc > 0 ? ldc : N / 2, gate.bias, gate.limit, nullptr, fixed_w, st);
  if ((g_gemm_mode == 2 && M > GEMM_BM) || (g_gemm_mode == 0 && choose_tile(M, N, true, true).pair))
    return launch_gemm2<256, kAct>(A, W, C, M, N, K, st, ldc, gate, fixed_w);
  return launch_gemm<256, kAct>(A, W, C, M, N, K, st, 1, nullptr, ldc, gate, fixed_w);
}

namespace b200q {

static int rows_product(const void* A, const void* W, void* C, int M, int N, int K, RowsTile r, float* ws, bool fixed_w, cudaStream_t st,
                        const float** partials_out) {
  return split_product(ws, C, M, N, r.splits, st, partials_out,
                       [&]() { return gemm_rows(A, W, nullptr, M, N, K, r.rows, r.splits, ws, fixed_w, st); });
}

int linear(const void* A, const void* W, void* C, int M, int N, int K, bool fixed_w, cudaStream_t st) {
  B200Q_CHECK_ARG(M >= 0 && N > 0 && K > 0 && K % GEMM_BK == 0 && N % 64 == 0,
                  "gemm: unsupported shape M=%d N=%d K=%d (need K%%64==0, N%%64==0)", M, N, K);
  B200Q_CHECK_ARG((reinterpret_cast<uintptr_t>(A) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(W) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(C) & 15) == 0,
                  "gemm: operands must be 16-byte aligned");
  if (M == 0) return B200Q_OK;
  if (use_skinny(M, N, K, false)) return gemm_skinny(A, W, C, M, N, K, ACT_NONE, N, nullptr, 0.f, nullptr, fixed_w, st);
  int bn = g_gemm_force_bn;
  if (g_gemm_mode == 2 && M > GEMM_BM) {
    if ((bn == 0 || bn == 256) && N % 256 == 0) return launch_gemm2<256>(A, W, C, M, N, K, st, 0, GateArgs{nullptr, 0.f}, fixed_w);
    if ((bn == 0 || bn == 128) && N % 128 == 0) return launch_gemm2<128>(A, W, C, M, N, K, st, 0, GateArgs{nullptr, 0.f}, fixed_w);
  }
  {
    // split-K for decode-sized batches: when a projection has too few 128-wide output tiles to
    // put every SM on the weight stream, split the reduction so that tiles x splits ~ #SMs
    // B200Q_BATCH_INVARIANT=1 (read once): never split K, so every output element is reduced in
    // one sequential pass (the attention kernels do likewise) and a request's tokens cannot depend on its batch-mates (like
    // VLLM_BATCH_INVARIANT); costs decode-sized GEMMs up to 2x
    const int splits = choose_splits(M, N, K, bn, st);
    if (splits > 1) return launch_gemm<128>(A, W, C, M, N, K, st, splits, nullptr, 0, GateArgs{nullptr, 0.f}, fixed_w);
  }
  if (bn == 0) {
    float* ws = nullptr;
    const RowsTile r = rows_tile_of(M, N, K, st, &ws);
    if (r.splits > 1) return rows_product(A, W, C, M, N, K, r, ws, fixed_w, st, nullptr);
    if (r.rows > 0) return gemm_rows(A, W, C, M, N, K, r.rows, 1, nullptr, fixed_w, st);
    const TileChoice t = choose_tile(M, N, false, g_gemm_mode == 0);
    auto pair = [&](auto width) {
      return launch_gemm2<decltype(width)::value>(A, W, C, M, N, K, st, 0, GateArgs{nullptr, 0.f}, fixed_w);
    };
    if (t.pair)
      return t.bn == 256   ? pair(std::integral_constant<int, 256>{})
             : t.bn == 192 ? pair(std::integral_constant<int, 192>{})
             : t.bn == 160 ? pair(std::integral_constant<int, 160>{})
                           : pair(std::integral_constant<int, 128>{});
    bn = t.bn;
  }
  if (N % bn != 0) bn = (N % 128 == 0) ? 128 : 64;
  if (bn == 256) return launch_gemm<256>(A, W, C, M, N, K, st, 1, nullptr, 0, GateArgs{nullptr, 0.f}, fixed_w);
  if (bn == 128) return launch_gemm<128>(A, W, C, M, N, K, st, 1, nullptr, 0, GateArgs{nullptr, 0.f}, fixed_w);
  return launch_gemm<64>(A, W, C, M, N, K, st, 1, nullptr, 0, GateArgs{nullptr, 0.f}, fixed_w);
}

int linear_parts(const void* A, const void* W, int M, int N, int K, bool fixed_w, cudaStream_t st, const float** partials_out,
                 int* splits_out) {
  B200Q_CHECK_ARG(partials_out && splits_out, "gemm_splitk: null output argument");
  *partials_out = nullptr;
  *splits_out = 1;
  B200Q_CHECK_ARG(M >= 0 && N > 0 && K > 0 && K % GEMM_BK == 0 && N % 64 == 0,
                  "gemm: unsupported shape M=%d N=%d K=%d (need K%%64==0, N%%64==0)", M, N, K);
  B200Q_CHECK_ARG((reinterpret_cast<uintptr_t>(A) & 15) == 0 && (reinterpret_cast<uintptr_t>(W) & 15) == 0,
                  "gemm: operands must be 16-byte aligned");
  if (M == 0 || g_gemm_mode == 2 || g_gemm_force_bn != 0) return B200Q_OK;
  if (use_skinny(M, N, K, false)) {
    const int n = gemm_skinny_splits(M, N, K);
    if (n <= 1 || N > 8192) return B200Q_OK;
    float* ws = nullptr;
    int rc = splitk_scratch(n, M, N, st, &ws);
    if (!rc) rc = gemm_skinny(A, W, nullptr, M, N, K, ACT_NONE, N, nullptr, 0.f, ws, fixed_w, st);
    if (rc) return rc;
    *partials_out = ws;
    *splits_out = n;
    return B200Q_OK;
  }
  const int splits = choose_splits(M, N, K, 0, st);
  if (splits <= 1) {
    float* ws = nullptr;
    const RowsTile r = rows_tile_of(M, N, K, st, &ws);
    if (r.splits <= 1) return B200Q_OK;
    int rc = rows_product(A, W, nullptr, M, N, K, r, ws, fixed_w, st, partials_out);
    if (!rc) *splits_out = r.splits;
    return rc;
  }
  int rc = launch_gemm<128>(A, W, nullptr, M, N, K, st, splits, partials_out, 0, GateArgs{nullptr, 0.f}, fixed_w);
  if (rc) return rc;
  *splits_out = splits;
  return B200Q_OK;
}

int linear_gated(bool gelu, const void* A, const void* W, void* C, int M, int N, int K, bool fixed_w, cudaStream_t st) {
  return gelu ? gemm_gated<ACT_GEGLU>("gemm_geglu", A, W, C, M, N, K, st, 0, GateArgs{nullptr, 0.f}, fixed_w)
              : gemm_gated<ACT_SWIGLU>("gemm_swiglu", A, W, C, M, N, K, st, 0, GateArgs{nullptr, 0.f}, fixed_w);
}

}  // namespace b200q

extern "C" {

// Grouped / per-head GEMM on the tensor cores, see gemm_grouped_kernel.  Returns B200Q_EINVAL for shapes
// it does not take (the caller falls back): K, N multiples of 64, 16-byte aligned operands and slices.
int b200q_gemm_grouped_bf16(const void* A, long long a_rows, long long lda, int a_gx, const void* W, int groups,
                            void* C, long long ldc, int c_gx, int M, int N, int K, const void* tab_dev,
                            const int32_t* n_mt_dev, int max_mtiles, int out_f32, void* stream) {
  B200Q_CHECK_ARG(A && W && C && groups > 0 && N > 0 && K > 0 && a_rows > 0, "gemm_grouped: bad argument");
  B200Q_CHECK_ARG(b200q_gemm_grouped_ok(A, lda, a_gx, W, C, ldc, c_gx, N, K, out_f32),
                  "gemm_grouped: unsupported shape N=%d K=%d lda=%lld ldc=%lld", N, K, lda, ldc);
  B200Q_CHECK_ARG(tab_dev ? (n_mt_dev && max_mtiles > 0) : M >= 0, "gemm_grouped: bad tile description");
  if (!tab_dev && M == 0) return B200Q_OK;
  CUtensorMap ta, tb;
  int rc = get_tmap(A, a_rows, lda, GEMM_BM, &ta);  // the whole matrix; a group's slice is a column offset
  if (rc) return rc;
  const int bn = N % 256 == 0 ? 256 : (N % 128 == 0 ? 128 : 64);
  rc = get_tmap(W, (long long)groups * N, K, bn, &tb);
  if (rc) return rc;
  GroupedArgs ga{(const int4*)tab_dev, n_mt_dev, M, groups, a_gx, c_gx, ldc, 0, tab_dev ? max_mtiles : 0};
  const long long mt = tab_dev ? max_mtiles : (long long)groups * ((M + GEMM_BM - 1) / GEMM_BM);
  const long long tiles = mt * (N / bn);
  const int cap = (int)(tiles < (1 << 30) ? tiles : (1 << 30));
  // Routed rows, two or more per group on average (so that few groups stay without any) and no more than one m-tile: the weights are
  // what bounds the product, and the kernels that route and gather the rows leave the memory idle (128 rows, 16 experts of 2048 x 1024,
  // 4 of them each: the second product 15.0 -> 12.6 us, the whole layer 60.7 -> 58.7).
  if (tab_dev && a_rows >= 2LL * groups && a_rows <= (long long)GEMM_BM * groups) {
    const long long first = (long long)groups * (N / bn), ctas = first < num_sms() ? first : num_sms();
    ga.ahead = (int)(GROUPED_AHEAD_BYTES / (ctas * bn * GEMM_BK * 2));
  }
  cudaStream_t st = as_stream(stream);
  if (out_f32) {
    if (bn == 256) return launch_grouped<256, true>(ta, tb, C, N, K, ga, cap, st);
    if (bn == 128) return launch_grouped<128, true>(ta, tb, C, N, K, ga, cap, st);
    return launch_grouped<64, true>(ta, tb, C, N, K, ga, cap, st);
  }
  if (bn == 256) return launch_grouped<256, false>(ta, tb, C, N, K, ga, cap, st);
  if (bn == 128) return launch_grouped<128, false>(ta, tb, C, N, K, ga, cap, st);
  return launch_grouped<64, false>(ta, tb, C, N, K, ga, cap, st);
}

int b200q_gemm_grouped_ok(const void* A, long long lda, int a_gx, const void* W, const void* C, long long ldc,
                          int c_gx, int N, int K, int out_f32) {
  const int ca = out_f32 ? 4 : 8;  // elements of C per 16 bytes
  return K % GEMM_BK == 0 && N % 64 == 0 && lda % 8 == 0 && a_gx % 8 == 0 && ldc % ca == 0 && c_gx % ca == 0 &&
         ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(C)) & 15) == 0;
}

// test/tuning hook (not part of the reference-facing surface): force the N tile (0 = auto)
int b200q_gemm_set_tile_n(int bn) {
  B200Q_CHECK_ARG(bn == 0 || bn == 64 || bn == 128 || bn == 256, "gemm tile N must be 0/64/128/256");
  g_gemm_force_bn = bn;
  bump_tuning_epoch();
  return B200Q_OK;
}

// test/tuning hook: 0 = auto, 1 = 1-CTA kernels only, 2 = 2-CTA (cta_group::2) kernel whenever legal
// diagnostics: co-resident CTA pairs the 2-CTA kernel's grid is sized to (0 until first use)
int b200q_gemm_resident_pairs(void) { return g_gemm2_pairs; }

// test hooks: rows of A in the tiles of gemm_rows.cu that a product takes (0: none of them), and the parts of K (1: not split)
int b200q_gemm_rows_tile(int M, int N, int K) { return rows_tile_behind(M, N, K).rows; }
int b200q_gemm_rows_splits(int M, int N, int K) { return rows_tile_behind(M, N, K).splits; }

// test hook: columns of the tiles of a product of more than 128 rows whose reduction is not split
int b200q_gemm_tile_n(int M, int N) { return g_gemm_force_bn ? g_gemm_force_bn : choose_tile(M, N, false, g_gemm_mode == 0).bn; }

// test/tuning hook: 0 = auto split-K, 1 = off, n > 1 = force n splits (decode-sized M only)
int b200q_gemm_set_splitk(int n) {
  B200Q_CHECK_ARG(n >= 0 && n <= 16, "split-K factor must be in [0,16]");
  g_gemm_splitk = n;
  bump_tuning_epoch();
  return B200Q_OK;
}

int b200q_gemm_set_mode(int mode) {
  B200Q_CHECK_ARG(mode >= 0 && mode <= 2, "gemm mode must be 0/1/2");
  g_gemm_mode = mode;
  bump_tuning_epoch();
  return B200Q_OK;
}

int b200q_gemm_bf16(const void* A, const void* W, void* C, int M, int N, int K, void* stream) {
  return linear(A, W, C, M, N, K, false, as_stream(stream));
}

// The split-K half of b200q_gemm_bf16 on its own: when the dispatcher would split the reduction
// (decode-sized M, few output tiles) the fp32 partial tiles are left in the library's scratch
// ([splits][M][N], *partials_out) and NO reduce pass runs — the caller folds the fixed-order sum and
// the bf16 rounding into the kernel that consumes the projection (b200q_add_rmsnorm_splitk,
// b200q_rope_kvwrite_splitk), saving a launch and a round trip per projection.  *splits_out = 1
// means nothing was launched: call b200q_gemm_bf16 instead.  The scratch is the stream's, or the graph's that is being captured, and
// is overwritten by the next split product there (a call of b200q_gemm_bf16 may be one); passes of a model leave it alone.
int b200q_gemm_bf16_splitk(const void* A, const void* W, int M, int N, int K, void* stream, const float** partials_out, int* splits_out) {
  return linear_parts(A, W, M, N, K, false, as_stream(stream), partials_out, splits_out);
}

// K9+K10 fused: out[M, N/2] = swiglu(A . W^T) where W [N, K] holds gate/up rows interleaved in
// blocks of 128 (rows [256j, 256j+128) = gate rows [128j, 128j+128), next 128 = the matching up
// rows).  Same rounding points as b200q_gemm_bf16 followed by b200q_swiglu.
int b200q_gemm_swiglu_bf16(const void* A, const void* W, void* C, int M, int N, int K,
                           void* stream) {
  return linear_gated(false, A, W, C, M, N, K, false, as_stream(stream));
}

// Gemma-2's GeGLU (gelu_tanh(gate) * up) in the same fused epilogue, same weight interleaving
int b200q_gemm_geglu_bf16(const void* A, const void* W, void* C, int M, int N, int K, void* stream) {
  return linear_gated(true, A, W, C, M, N, K, false, as_stream(stream));
}

// the clamped gated unit (with biases unless NULL) in the same epilogue; C has rows of ldc elements
int b200q_gemm_clamped_glu_bf16(const void* A, const void* W, const float* bias, void* C, int ldc, int M, int N, int K,
                                float limit, void* stream) {
  B200Q_CHECK_ARG(ldc >= N / 2 && ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(bias) & 15) == 0 && limit >= 0.f,
                  "gemm_clamped_glu: bad bias, row stride (%d) or limit", ldc);
  return gemm_gated<ACT_CLAMPED>("gemm_clamped_glu", A, W, C, M, N, K, stream, ldc, GateArgs{bias, limit});
}

}  // extern "C"
