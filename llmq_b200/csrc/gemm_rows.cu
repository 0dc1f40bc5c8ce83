// gemm_rows.cu — C[M,N] = A[M,K] . W[N,K]^T for row counts that tiles of 256 rows fill badly, bf16 operands, fp32 accumulation.
//
// Bound: the tensor pipe, and below some 200 rows the weight stream.  gemm_tcgen05.cu pays for 256 rows wherever there are 129 (300 rows
// cost 512), and whole rounds of its tiles.  Here the weights are the tensor core's M side (256 rows of W per CTA pair, cta_group::2) and
// the rows of A its N side: any multiple of 32 up to 256 of them to an accumulator, one or two accumulators to a tile (two share what is
// fetched of W), so that M is cut into parts that waste little and fill the rounds.
//   * CTA pair, persistent, warp-specialised: two threads fetch (128 rows of W each, half of the tile's rows of A), warp 1 of the leader
//     issues the products, eight warps store.  Two tiles' accumulators in tensor memory where they fit.
//   * a lane of an accumulator is a column of C: 32 rows x 128 columns at a time are turned in shared memory and leave by TMA, which also
//     leaves out what lies behind the last row or column.
//   * where the tiles are too few for the chip, K is cut as well and the fp32 sums of its parts leave by plain stores, for another kernel to add.
// The parts of a row of tiles follow each other, so that CTA pairs share weights through L2; every element of C is one sequential sum, in
// the same order as in gemm_tcgen05.cu, or one such sum to a part of K.  Times and the rule that takes these tiles: rows_tile in
// gemm_tcgen05.cu.
#include "tcgen05.cuh"

namespace b200q {

constexpr int GR_THREADS = 352;
constexpr int GR_BK = 64;
constexpr int GR_W_BYTES = 128 * GR_BK * 2;  // 128 rows of W of one k-block
constexpr int GR_MAX_STAGES = 8, GR_RING = 192 * 1024, GR_PATCH = 8192;  // patch: 32 rows x 128 columns of C
constexpr int GR_SMEM = GR_RING + 4 * GR_PATCH + 1024;

struct GemmRowsArgs {
  int* failed;
  int M, N, K, nt, stages, parts, n_blocks;  // a tile has HALVES * nt rows of A; n_blocks: of 128 columns of C
  int fixed_w;                               // see linear() in common.cuh
  int splits;                                // parts of K, each a tile of its own
  float* ws;                                 // their sums, [split][M][N], for splits > 1
};

__device__ __forceinline__ void gr_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void gr_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cluster.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void gr_load(void* to, const void* tmap, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(to)),
      "l"(tmap), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void gr_store(const void* tmap, int c0, int c1, uint32_t from) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(tmap), "r"(c0), "r"(c1), "r"(from)
               : "memory");
}
__device__ __forceinline__ void gr_product(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t add) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(add)
      : "memory");
}
// arrive on the barrier at this place in both CTAs of the pair
__device__ __forceinline__ void gr_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}

// HALVES: accumulators side by side that share a tile's weights (of nt rows of A each).  PARTS: a tile is a part of K (a kernel of its own, since
// what places it costs every other tile 0.3 us)
template <int HALVES, bool PARTS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GR_THREADS, 1)
    gemm_rows_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                     const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ GemmRowsArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* patches = smem + GR_RING;
  __shared__ __align__(8) uint64_t full[GR_MAX_STAGES], empty[GR_MAX_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int dead;  // a wait ran out: the other roles stop as well
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int per_pair = PARTS ? a.parts * a.splits : a.parts, n_tiles = (a.n_blocks + 1) / 2 * per_pair, k_blocks = a.K / GR_BK;
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int a_bytes = a.nt / 2 * (GR_BK * 2), stage_bytes = GR_W_BYTES + HALVES * a_bytes;
  const int rows_all = HALVES * a.nt, accs = 2 * rows_all <= 512 ? 2 : 1;  // accumulators of a whole tile

  if (warp == 0 && lane == 0) {
    dead = 0;
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_c);
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(full + s, 4);   // (the leader's) an arrival from each CTA's two fetching threads
      mbar_init(empty + s, 1);  // the leader's products, in both CTAs
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(acc_full + s, 1);
      mbar_init(acc_empty + s, 16);  // (the leader's) eight warps of each CTA
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // (the peer's barriers are there before anybody signals them)
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
  // (flag and clock are looked at every 64 tries)
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    long long t0 = 0;
    for (int n = 0; !mbar_try_wait(bar, parity); ++n) {
      if (n % 64 != 63) continue;
      if (n == 63) t0 = clock64();
      if (*(volatile int*)&dead) break;
      if (clock64() - t0 > WAIT_CYCLES) {
        dead = 1;
        __threadfence_block();
        *(volatile int*)a.failed = 1;
        break;
      }
    }
  };
  // the first row of W of this CTA's part of a tile
  auto w_row = [&](int tile) { return (tile / per_pair * 2 + rank) * 128; };
  // the k-blocks of a tile: parts of K behind one another, each with all parts of M
  auto k_begin = [&](int tile) { return PARTS ? tile % per_pair / a.parts * k_blocks / a.splits : 0; };
  auto k_end = [&](int tile) { return PARTS ? (tile % per_pair / a.parts + 1) * k_blocks / a.splits : k_blocks; };

  // the first weights while the kernel before this one ends: into the ring where nobody can still be writing them, into L2 otherwise
  const uint32_t full0 = mapa_shared(full, 0);
  int early = 0;
  if (warp == 0 && lane == 0) {
    const int k0 = k_begin(pair), n = min(a.stages, k_end(pair) - k0);
    for (int s = 0; s < n; ++s) {
      if (a.fixed_w) {
        gr_expect_tx(full0 + s * 8, GR_W_BYTES);
        gr_load(smem + s * stage_bytes, &tmap_w, (k0 + s) * GR_BK, w_row(pair), full0 + s * 8);
        ++early;
      } else {
        tma_prefetch_2d(&tmap_w, (k0 + s) * GR_BK, w_row(pair));
      }
    }
  }
  __syncwarp();
  follow_previous();

  // Weights and rows of A are fetched by a thread each: what one thread has to do for both takes 600 cycles a k-block, longer than the
  // products of up to 160 rows
  if (warp == 0 || warp == 10) {
    if (lane == 0) {
      const bool weights = warp == 0;
      const void* map = weights ? &tmap_w : &tmap_a;
      const uint32_t bytes = weights ? GR_W_BYTES : HALVES * a_bytes;
      uint8_t* const to = smem + (weights ? 0 : GR_W_BYTES);
      int stage = early % a.stages, done = early;
      uint32_t phase = early / a.stages;
      for (int tile = pair; tile < n_tiles; tile += pairs) {
        const int row = weights ? w_row(tile) : tile % a.parts * rows_all + rank * (a.nt / 2);
        const int k1 = k_end(tile);
        for (int kb = k_begin(tile) + done; kb < k1; ++kb) {
          const uint32_t bar = full0 + stage * 8;
          uint8_t* at = to + stage * stage_bytes;
          wait(empty + stage, phase ^ 1u);
          gr_expect_tx(bar, bytes);
          gr_load(at, map, kb * GR_BK, row, bar);
          if (HALVES == 2 && !weights) gr_load(at + a_bytes, map, kb * GR_BK, row + a.nt, bar);
          if (++stage == a.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        done = 0;
        if (*(volatile int*)&dead) break;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.nt >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool on = true;  // (waits that the whole warp agrees on: ptxas keeps what follows in uniform registers)
      const uint32_t ring = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
      for (int tile = pair; on && tile < n_tiles; tile += pairs) {
        if (!(on = mbar_wait_warp(acc_empty + acc, acc_phase ^ 1u, &dead, a.failed, WAIT_CYCLES))) break;
        tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(acc * rows_all);
        const int k0 = k_begin(tile), k1 = k_end(tile);
        for (int kb = k0; kb < k1; ++kb) {
          if (!(on = mbar_wait_warp(full + stage, phase, &dead, a.failed, WAIT_CYCLES))) break;
          tc_fence_after();
          if (elect_one()) {
            const uint32_t sw = ring + (uint32_t)(stage * stage_bytes), sa = sw + GR_W_BYTES;
#pragma unroll
            for (int k = 0; k < GR_BK / 16; ++k)
#pragma unroll
              for (int h = 0; h < HALVES; ++h)
                gr_product(d + (uint32_t)(h * a.nt), make_smem_desc(sw + k * 32), make_smem_desc(sa + h * a_bytes + k * 32), idesc,
                           (kb > k0 || k > 0) ? 1u : 0u);
            gr_commit(empty + stage);
            if (kb == k1 - 1) gr_commit(acc_full + acc);
          }
          __syncwarp();
          if (++stage == a.stages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (++acc == accs) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else {
    // two groups of four warps, which take every other 32 rows, with two patches each
    const int quarter = warp & 3, group = (warp - 2) >> 2;
    const bool copies = warp == 2 + 4 * group && lane == 0;
    auto all = [&]() { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
    const uint32_t patch0 = smem_u32(patches) + (uint32_t)group * (2 * GR_PATCH);
    int acc = 0, n_out = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair; tile < n_tiles; tile += pairs) {
      const int block = tile / per_pair * 2 + rank, row0 = tile % a.parts * rows_all;
      const int rows = min(rows_all, a.M - row0);
      wait(acc_full + acc, acc_phase);
      __syncwarp();
      tc_fence_after();
      const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * rows_all);
      if (block < a.n_blocks) {
#pragma unroll 1
        for (int m0 = 32 * group; m0 < rows; m0 += 64, ++n_out) {
          uint32_t v[32];
          tmem_ld32(at + (uint32_t)m0, v);
          tmem_ld_wait();
          if constexpr (PARTS) {  // a warp's row of a part is 128 bytes
            float* to = a.ws + ((long long)(tile % per_pair / a.parts) * a.M + row0 + m0) * a.N + block * 128 + quarter * 32 + lane;
            const int n = rows - m0;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < n) to[(long long)j * a.N] = __uint_as_float(v[j]);
          } else {
            const uint32_t patch = patch0 + (uint32_t)(n_out & 1) * GR_PATCH;
            if (copies) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            all();  // (the copy that read this patch has)
            // row j of the patch, column quarter * 32 + lane: two boxes of 64 columns, as the copy's 128-byte swizzle
            const uint32_t col = (uint32_t)((quarter & 1) * 64 + lane * 2), base = patch + (uint32_t)(quarter >> 1) * 4096 + (col & 15u);
#pragma unroll
            for (int j = 0; j < 32; ++j)
              asm volatile("st.shared.b16 [%0], %1;" ::"r"(base + j * 128 + (((col >> 4) ^ (j & 7)) << 4)),
                           "h"((unsigned short)f2bf_bits(__uint_as_float(v[j])))
                           : "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            all();
            if (copies) {
              gr_store(&tmap_c, block * 128, row0 + m0, patch);
              gr_store(&tmap_c, block * 128 + 64, row0 + m0, patch + 4096);
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) gr_arrive(mapa_shared(acc_empty + acc, 0));
      if (++acc == accs) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
    if (copies) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  tc_fence_before();
  __syncthreads();
  if (dead) {  // (copies in flight end before the block's memory is given back)
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000ll) {
    }
    __syncthreads();
  }
  cluster_sync_all();  // nobody frees tensor memory or leaves while the peer may still signal or read
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

template <int HALVES, bool PARTS>
static int launch_rows(const void* A, const void* W, void* C, int M, int N, int K, int rows, int splits, float* ws, bool fixed_w,
                       cudaStream_t st) {
  GemmRowsArgs a{};
  a.M = M;
  a.N = N;
  a.K = K;
  a.nt = rows / HALVES;
  a.parts = (M + rows - 1) / rows;
  a.n_blocks = N / 128;
  a.fixed_w = fixed_w;
  a.splits = splits;
  a.ws = ws;
  a.stages = GR_RING / (GR_W_BYTES + rows / 2 * GR_BK * 2);
  if (a.stages > GR_MAX_STAGES) a.stages = GR_MAX_STAGES;
  CUtensorMap tw, ta, tc;
  int rc = get_tmap(W, N, K, 128, &tw);
  if (!rc) rc = get_tmap(A, M, K, a.nt / 2, &ta);
  if (!rc) rc = PARTS ? get_tmap(A, M, K, a.nt / 2, &tc) : get_tmap(C, M, N, 32, &tc);  // (parts leave by plain stores)
  if (rc) return rc;
  if (!wait_flag(&a.failed)) {
    set_error("gemm: no host-visible flag for bounded waits");
    return B200Q_ECUDA;
  }
  auto kern = gemm_rows_kernel<HALVES, PARTS>;
  static int pairs = 0;  // as many as can be resident at once
  if (pairs == 0) {
    B200Q_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GR_SMEM));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(num_sms() & ~1);
    cfg.blockDim = dim3(GR_THREADS);
    cfg.dynamicSmemBytes = GR_SMEM;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      n = num_sms() / 2;
    }
    pairs = n < num_sms() / 2 ? n : num_sms() / 2;
  }
  const int tiles = (a.n_blocks + 1) / 2 * a.parts * splits;
  B200Q_CUDA(launch_early(kern, 2 * (tiles < pairs ? tiles : pairs), GR_THREADS, GR_SMEM, st, 1, tw, ta, tc, a));
  count_launch();
  return B200Q_OK;
}

int gemm_rows(const void* A, const void* W, void* C, int M, int N, int K, int rows, int splits, float* ws, bool fixed_w, cudaStream_t st) {
  auto launch = [&](auto halves, auto parts) {
    return launch_rows<decltype(halves)::value, decltype(parts)::value>(A, W, C, M, N, K, rows, splits, ws, fixed_w, st);
  };
  const std::integral_constant<int, 1> one;
  const std::integral_constant<int, 2> two;
  if (splits > 1) return rows > 256 ? launch(two, std::true_type{}) : launch(one, std::true_type{});
  return rows > 256 ? launch(two, std::false_type{}) : launch(one, std::false_type{});
}

}  // namespace b200q
