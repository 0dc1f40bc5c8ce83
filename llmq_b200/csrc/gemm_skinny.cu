// gemm_skinny.cu — C[M,N] = A[M,K] . W[N,K]^T for up to 128 rows of A (decode steps), bf16 operands, fp32 accumulation.
//
// Bound: the weight stream from HBM (2 N K bytes); everything else has to stay out of its way.
//   * the weights are the tensor core's M side (128 or 256 rows of W per CTA), the rows of A its N side, padded to 16 and not
//     to 128: a step of few rows pays for few;
//   * the reduction is split over a cluster of up to 8 CTAs so that every shape puts enough CTAs on the stream; the fp32
//     partial tiles meet in distributed shared memory, are added in the order of the splits (deterministic) and stored once:
//     no scratch round trip and no second launch;
//   * no tile loop: a CTA works one tile, and where the ring takes half of an SM's memory the second CTA of the SM covers its
//     start and its end;
//   * the first weights are asked for before the kernel before this one has ended (follow_previous): into the ring where nobody can
//     still be writing them (fixed_w), into L2 otherwise.
// A gated unit (SwiGLU, GeGLU, clamped) works on a 128-row tile of 64 gate rows and the 64 rows that they gate: few or no splits whose
// parts would have to meet (28672 x 4096, 100 rows: 45.7 us, 48.0 with tiles of 128 + 128 rows; 16384 x 2048, 48 rows: 14.4, 16.3;
// but 6144 x 4096, 100 rows 17.9, 17.0: few tiles, each of which fetches all rows of A).
#include "tcgen05.cuh"

namespace b200q {

constexpr int SK_THREADS = 192;
constexpr int SK_BK = 64;
constexpr int SK_TILE_BYTES = 128 * SK_BK * 2;  // 128 weight rows of one k-block
constexpr int SK_MAX_STAGES = 8;
constexpr int SK_MAX_SPLITS = 8;
constexpr long long SK_AHEAD_BYTES = 24000000;  // weights of a product that are asked for before the kernel before it has ended

struct SkinnyArgs {
  bf16* C;
  float* parts;  // != NULL: the fp32 partial tiles go here ([splits][M][N]) and the caller adds them
  const float* bias;
  int* failed;
  long long ldc, patience;  // patience: cycles that the product warp waits for a stage
  float limit;
  int M, N, K, mp, stages, a_bytes, cols, chunk;  // mp: M padded to 16; chunk: columns (rows of A) per exchange
  int fixed_w;  // see linear() in common.cuh
  int ahead;    // k-blocks of weights that are asked for before the kernel before this one has ended
};

// After a wait ran out, before the block's memory is given back: what the first thread asked for has come, and what was issued has been
// made (`done` is committed behind the last product in any case)
__device__ __noinline__ void skinny_end_copies(uint64_t* full, uint64_t* done, int asked, int stages) {
  if (threadIdx.x == 0)
    for (int i = asked > stages ? asked - stages : 0; i < asked; ++i) mbar_wait_limited(full + i % stages, (uint32_t)(i / stages) & 1u);
  mbar_wait_limited(done, 0);
  __syncthreads();
}

// WT: 128-row weight tiles per CTA
template <int WT, int kAct>
__global__ void __launch_bounds__(SK_THREADS, 2)
    gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a, const SkinnyArgs a) {
  constexpr int NT = WT * 128;
  // (a gated unit's tile is 64 gate rows and the 64 rows that they gate, out of a block of 256 weight rows)
  constexpr bool kGated = kAct != ACT_NONE;
  static_assert(!kGated || WT == 1, "a gated unit's tile is 128 rows");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[SK_MAX_STAGES], empty[SK_MAX_STAGES], done;
  __shared__ uint32_t tmem_slot;
  __shared__ int dead;  // a wait ran out: the other roles stop as well
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int split = blockIdx.x, splits = gridDim.x, tile = blockIdx.y;
  const int gate_row = tile / 2 * 256 + tile % 2 * 64;
  const int kb_all = a.K / SK_BK, kb0 = split * kb_all / splits, kb1 = (split + 1) * kb_all / splits;
  const int stage_bytes = WT * SK_TILE_BYTES + a.mp * (SK_BK * 2);

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_a);
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    mbar_init(&done, 1);
    mbar_fence_init();
    dead = 0;
  }
  if (warp == 1) tmem_alloc(&tmem_slot, a.cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
  int asked = 0;  // (of the fetching thread) stages asked for
  // every tile begins at another k-block: all of them asking for the same rows of A at once cost 2-4 % at 64 rows and more
  // (short reductions keep the order that the kernels for larger steps add in)
  const int kb_first = kb0 + (kb1 - kb0 >= 16 ? tile * 5 % (kb1 - kb0) : 0), early = min(a.stages, kb1 - kb0);
  auto load_w = [&](uint8_t* to, int kb, uint64_t* bar) {
    if constexpr (kGated) {
      tma_load_2d(to, &tmap_w, kb * SK_BK, gate_row, bar);
      tma_load_2d(to + SK_TILE_BYTES / 2, &tmap_w, kb * SK_BK, gate_row + 128, bar);
    } else {
      tma_load_2d(to, &tmap_w, kb * SK_BK, tile * NT, bar);
    }
  };
  if (warp == 0 && lane == 0) {  // the first weights while the kernels before this one end
    int kb = kb_first;
    for (int i = 0; i < min(a.ahead, kb1 - kb0); ++i, kb = kb + 1 < kb1 ? kb + 1 : kb0) {
      if (a.fixed_w && i < early) {
        mbar_expect_tx(full + i, (uint32_t)(WT * SK_TILE_BYTES + a.a_bytes));
        load_w(smem + i * stage_bytes, kb, full + i);
      } else if constexpr (kGated) {
        tma_prefetch_2d(&tmap_w, kb * SK_BK, gate_row);
        tma_prefetch_2d(&tmap_w, kb * SK_BK, gate_row + 128);
      } else {
        tma_prefetch_2d(&tmap_w, kb * SK_BK, tile * NT);
      }
    }
  }
  __syncwarp();
  const float* bias = a.bias;
  follow_previous(bias);

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int kb = kb_first;
      for (; asked < kb1 - kb0; ++asked, kb = kb + 1 < kb1 ? kb + 1 : kb0) {
        uint8_t* sw = smem + stage * stage_bytes;
        if (!a.fixed_w || asked >= early) {
          if (!mbar_wait_or_fail(empty + stage, phase ^ 1u, &dead, a.failed)) break;
          mbar_expect_tx(full + stage, (uint32_t)(WT * SK_TILE_BYTES + a.a_bytes));
          load_w(sw, kb, full + stage);
        }
        tma_load_2d(sw + WT * SK_TILE_BYTES, &tmap_a, kb * SK_BK, 0, full + stage);
        if (++stage == a.stages) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.mp >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    int stage = 0;
    uint32_t phase = 0;
    for (int i = kb0; i < kb1; ++i) {
      if (!mbar_wait_warp(full + stage, phase, &dead, a.failed, a.patience)) break;
      tc_fence_after();
      if (elect_one()) {
        const uint32_t sw = smem_u32(smem + stage * stage_bytes), sa = sw + WT * SK_TILE_BYTES;
#pragma unroll
        for (int h = 0; h < WT; ++h)
#pragma unroll
          for (int k = 0; k < SK_BK / 16; ++k)
            umma_bf16(tmem + (uint32_t)(h * a.mp), make_smem_desc(sw + h * SK_TILE_BYTES + k * 32), make_smem_desc(sa + k * 32), idesc,
                      (i > kb0 || k > 0) ? 1u : 0u);
        umma_commit(empty + stage);
      }
      __syncwarp();
      if (++stage == a.stages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    __syncwarp();
    if (elect_one()) umma_commit(&done);
    __syncwarp();
  }

  // ---- the accumulators: lane = weight row, column = row of A ----
  const bool epi = warp >= 2;
  const int quarter = warp & 3, row = quarter * 32 + lane;
  if (epi) {
    mbar_wait_or_fail<16>(&done, 0, &dead, a.failed);
    __syncwarp();
    tc_fence_after();
  }
  // (products that stop early say so before `done`: copies may then still arrive in the ring, which is left alone)
  const bool give = epi && *(volatile int*)&dead == 0;
  // 32 columns of the accumulator: a load takes some 0.2 us, so that both are asked for before the first is used (2048 x 2048 in five
  // parts, 48 rows: 1.6 -> 0.6 us from the last product to the end of the CTA; 64 columns at a time are no faster and take the registers
  // that the next kernel's CTAs need beside this one's)
  auto columns = [&](int h, int c, int n, uint32_t(&v)[2][16]) {
#pragma unroll
    for (int x = 0; x < 2; ++x)
      if (16 * x < n) tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(h * a.mp + c + 16 * x), v[x]);
    tmem_ld_wait();
  };
  if (a.parts) {
    if (epi) {
      float* dst = a.parts + (long long)split * a.M * a.N + (long long)tile * NT + row;
#pragma unroll 1
      for (int h = 0; h < WT; ++h)
#pragma unroll 1
        for (int c = 0; c < a.M; c += 32) {
          uint32_t v[2][16];
          columns(h, c, a.M - c, v);
          float* d = dst + h * 128 + (long long)c * a.N;
          const int n = a.M - c;
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int j = 0; j < 16; ++j, d += a.N)
              if (16 * x + j < n) *d = __uint_as_float(v[x][j]);
        }
    }
  } else {
    float* red = reinterpret_cast<float*>(smem);
    for (int c0 = 0; c0 < a.M; c0 += a.chunk) {
      if (give) {
        const int cn = min(a.chunk, a.mp - c0);
#pragma unroll 1
        for (int h = 0; h < WT; ++h)
#pragma unroll 1
          for (int c = 0; c < cn; c += 32) {
            uint32_t v[2][16];
            columns(h, c0 + c, cn - c, v);
#pragma unroll
            for (int x = 0; x < 2; ++x)
              if (c + 16 * x < cn) {
#pragma unroll
                for (int j = 0; j < 16; ++j) red[(c + 16 * x + j) * NT + h * 128 + row] = __uint_as_float(v[x][j]);
              }
          }
      }
      if (splits > 1)
        cluster_sync_all();
      else
        __syncthreads();
      // rows split, split + splits, ... of the chunk are this CTA's to add and store, four columns of C per thread
      constexpr int OUT = kGated ? NT / 2 : NT, GR = OUT / 4;
      const int rows = min(a.chunk, a.M - c0), mine = rows > split ? (rows - split + splits - 1) / splits : 0;
      for (int i = threadIdx.x; i < mine * GR; i += SK_THREADS) {
        const int r = (i / GR) * splits + split, n = (i % GR) * 4;
        const float* src = red + r * NT + n;
        // (all partial sums are asked for before the first is added: a remote read takes about 200 cycles)
        float4 p[SK_MAX_SPLITS], q[kGated ? SK_MAX_SPLITS : 1];
        if (splits > 1) {
#pragma unroll
          for (int s = 0; s < SK_MAX_SPLITS; ++s)
            if (s < splits) {
              const uint32_t at = mapa_shared(src, s);
              p[s] = ld_cluster_v4(at);
              if constexpr (kGated) q[s] = ld_cluster_v4(at + OUT * 4);
            }
        } else {
          p[0] = *reinterpret_cast<const float4*>(src);
          if constexpr (kGated) q[0] = *reinterpret_cast<const float4*>(src + OUT);
        }
        float4 x = p[0], y = x;
        if constexpr (kGated) y = q[0];
#pragma unroll
        for (int s = 1; s < SK_MAX_SPLITS; ++s)
          if (s < splits) {
            x.x += p[s].x; x.y += p[s].y; x.z += p[s].z; x.w += p[s].w;
            if constexpr (kGated) { y.x += q[s].x; y.y += q[s].y; y.z += q[s].z; y.w += q[s].w; }
          }
        float o[4] = {x.x, x.y, x.z, x.w};
        if constexpr (kGated) {
          const float u[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if constexpr (kAct == ACT_CLAMPED) {
              const float* b = bias + gate_row + n + j;
              o[j] = clamped_unit(__float_as_uint(o[j]), __float_as_uint(u[j]), bias ? b[0] : 0.f, bias ? b[128] : 0.f,
                                  a.limit);
            } else {
              o[j] = gated_unit<kAct>(__float_as_uint(o[j]), __float_as_uint(u[j]));
            }
          }
        }
        *reinterpret_cast<uint2*>(a.C + (long long)(c0 + r) * a.ldc + (long long)tile * OUT + n) =
            make_uint2(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]));
      }
      if (splits > 1)  // nobody writes over, or leaves with, what a peer still reads
        cluster_sync_all();
      else if (c0 + a.chunk < a.M)
        __syncthreads();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (dead) skinny_end_copies(full, &done, asked, a.stages);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, a.cols);
  }
}

constexpr int SK_RING_ALONE = 208 * 1024, SK_RING_SHARED = 108 * 1024;  // ring bytes with one and with two CTAs per SM

// How many clusters of `splits` CTAs fit at once, one CTA per SM (asked for once per size).  The occupancy query knows one CTA per SM
// for kernels that hold tensor memory; the hardware keeps two of them (256 columns or less each) where shared memory allows.
template <int WT, int kAct>
static int resident_clusters(int splits) {
  static int known[SK_MAX_SPLITS + 1];
  int& n = known[splits];
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(splits, 148);
    cfg.blockDim = dim3(SK_THREADS);
    cfg.dynamicSmemBytes = SK_RING_ALONE + 1024;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = splits;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int v = 0;
    if (cudaOccupancyMaxActiveClusters(&v, gemm_skinny_kernel<WT, kAct>, &cfg) != cudaSuccess || v <= 0) {
      cudaGetLastError();
      v = 1;
    }
    n = v;
  }
  return n;
}

bool g_gemm_give_up = false;  // test hook: the product warp's first wait counts as run out

struct SkinnyPlan {
  bool alone;
  int splits;
};
// Measured on B200, weights from HBM, back to back in a graph, us (here / the kernels of gemm_tcgen05.cu; both begin while the product
// before them ends):
//   rows                        1            48           100          128
//   3072 x 2048             5.2 /  6.3   6.8 /  8.0   8.0 /  9.6   8.5 / 10.5
//   4096 x 4096             8.6 /  9.2  10.4 / 10.6  11.2 / 11.7  11.8 / 13.1
//   4096 x 14336           21.3 / 22.4  23.8 / 24.7  24.3 / 26.7  25.2 / 28.9
//   16384 x 2048 gated     13.9 / 25.8  15.3 / 25.9  18.4 / 26.2  19.4 / 26.2
//   28672 x 4096 gated     38.5 / 49.1  41.6 / 49.7  46.3 / 50.8  49.1 / 52.1
// Splits: up to 64 rows two CTAs per SM with three or more stages each are best; with more rows a stage grows and one CTA per SM
// with the whole memory as its ring is (28.7 against 29.7 us at 4096 x 14336, 100 rows), unless the tiles alone would leave half
// of the SMs idle.  All clusters have to be resident at once: a cluster lies within a processing cluster of the chip, and one
// that does not fit doubles the time (2048 x 8192, 100 rows: 23.8 us with 16 clusters of 8, 14.8 with 16 of 6).
template <int WT, int kAct>
static SkinnyPlan skinny_plan(int M, int N, int K) {
  const int kb = K / SK_BK, tiles = N / (128 * WT);
  SkinnyPlan p{((M + 15) & ~15) > 64 && tiles <= 74, 1};
  for (int s = 2; s <= SK_MAX_SPLITS && kb / s >= 6; ++s)  // (fewer than 6 k-blocks each: no faster)
    if (tiles <= resident_clusters<WT, kAct>(s) * (p.alone ? 1 : 2)) p.splits = s;
  return p;
}

template <int WT, int kAct>
static int prepare_kernel() {
  static bool attr_set = false;
  if (!attr_set) {
    B200Q_CUDA(cudaFuncSetAttribute(gemm_skinny_kernel<WT, kAct>, cudaFuncAttributeMaxDynamicSharedMemorySize, SK_RING_ALONE + 1024));
    attr_set = true;
  }
  return B200Q_OK;
}

template <int WT, int kAct>
static int launch_skinny(const void* A, const void* W, SkinnyArgs a, cudaStream_t st) {
  int rc = prepare_kernel<WT, kAct>();
  if (rc) return rc;
  const SkinnyPlan p = skinny_plan<WT, kAct>(a.M, a.N, a.K);
  const int a_rows = (a.M + 7) & ~7;  // only the rows that exist travel; the rest of the padded tile is never stored
  a.mp = (a.M + 15) & ~15;
  a.a_bytes = a_rows * SK_BK * 2;
  a.cols = 32;
  while (a.cols < WT * a.mp) a.cols *= 2;
  const int stage = WT * SK_TILE_BYTES + a.mp * SK_BK * 2;
  a.stages = (p.alone ? SK_RING_ALONE : SK_RING_SHARED) / stage;
  if (a.stages > SK_MAX_STAGES) a.stages = SK_MAX_STAGES;
  a.chunk = a.stages * stage / (WT * 512) & ~15;
  if (a.chunk > a.mp) a.chunk = a.mp;
  a.ahead = (int)(SK_AHEAD_BYTES / ((long long)(a.N / (WT * 128)) * p.splits * WT * SK_TILE_BYTES));
  if (a.ahead < a.stages) a.ahead = a.stages;
  CUtensorMap tw, ta;
  rc = get_tmap(W, a.N, a.K, kAct != ACT_NONE ? 64 : WT * 128, &tw);
  if (rc) return rc;
  rc = get_tmap(A, a.M, a.K, a_rows, &ta);
  if (rc) return rc;
  if (!wait_flag(&a.failed)) {
    set_error("gemm: no host-visible flag for bounded waits");
    return B200Q_ECUDA;
  }
  B200Q_CUDA(launch_early(gemm_skinny_kernel<WT, kAct>, dim3(p.splits, a.N / (WT * 128)), SK_THREADS, a.stages * stage + 1024, st,
                          a.parts ? 1 : p.splits, tw, ta, a));
  count_launch();
  return B200Q_OK;
}

// Tiles of 256 rows halve what a CTA re-reads of A, tiles of 128 give twice the CTAs: 256 only where 128 would give more than
// two for every SM.
static bool wide_tiles(int N) { return N % 256 == 0 && N / 256 >= 148; }

// Which products the kernel above takes; us, here / kernels of gemm_tcgen05.cu:
//   * plain, K < 1024: few k-blocks leave no splits to share out the end of a tile, and the narrower tiles there are done sooner: K = 512
//     5 / 4.5 at one row, 7.7 / 4.6 at 128, K = 64 6.1 / 3.2, for all N up to 8192; K = 768 even at 16 rows; 24576 x 512 8.8 / 9.4 at 32.
//   * plain, up to 64 tiles of 128, so that at least two CTAs work on each: always (1024 x 1024 6-9 / 6.5-8.6, 2048 x 2048 6-9 / 8-10,
//     5120 x 4096 0.7 of the time there).
//   * plain, more tiles, a CTA to each: the longer the reduction, the less the start and the end of a tile count, which the persistent
//     kernels hide.  Share of the time there, 12288 columns: K = 2048 0.99 at 16 rows, 1.07 at 48, 1.31 at 128; K = 4096 0.98 at 80, 1.06
//     at 128; K = 8192 1.02 at 100; two CTAs per SM hide some of it: 24576 x 2048 0.97 at 64 rows, 1.08 at 128.
//   * plain, tiles of 256 (vocabulary sizes): up to 32 rows (128256 x 2048 84 / 87); where K >= 4096 and the tiles fill rounds of two CTAs
//     per SM (128256 x 4096 178 / 183 at 64 rows, 1.7 rounds; but 50176 x 5120 98 / 89, 0.66) up to 64, or 112 if there is one round.  From
//     65 rows on there are the tiles of gemm_rows.cu: 128256 x 4096 181 / 172 at 65, 193 / 176 at 100, 197 / 179 at 112; 151552 x 4096 208 /
//     205, 206 / 202, 211 / 202; one round: 60672 x 4096 83.1 / 87.5, 87.1 / 87.1, 89.1 / 88.5, 65536 x 8192 185 / 193, 189 / 191, 193 / 192.
//   * gated: always (16384 x 2048 13.9 / 25.8 at one row, 19.4 / 26.2 at 128; 28672 x 4096 47.7 / 51.6 at 112, 49.1 / 52.1 at 128; 2048 x 512
//     5.4 / 14.3, 10.5 / 14.6; 9 shapes x 11 row counts: 0.32 to 0.94 of the time there).
bool gemm_skinny_ok(int M, int N, int K, bool gated) {
  if (M < 1 || M > 128 || K % SK_BK != 0 || N % (gated ? 256 : 128) != 0 || N / 128 > 65535) return false;
  if (gated) return true;
  if (wide_tiles(N)) {
    const int tiles = N / 256, rounds = (tiles + 295) / 296;
    return M <= 32 || (M <= (rounds == 1 ? 112 : 64) && K >= 4096 && 5 * tiles >= 4 * 296 * rounds);
  }
  const int tiles = N / 128;
  if (K < 1024) return M <= (tiles > 148 ? 32 : K >= 768 ? 16 : 0);
  return M <= (tiles <= 64 ? 128 : K >= 8192 ? 112 : K >= 4096 ? 80 : tiles > 148 ? 64 : 16);
}

int gemm_skinny_splits(int M, int N, int K) {
  if (wide_tiles(N)) return prepare_kernel<2, ACT_NONE>() ? 1 : skinny_plan<2, ACT_NONE>(M, N, K).splits;
  return prepare_kernel<1, ACT_NONE>() ? 1 : skinny_plan<1, ACT_NONE>(M, N, K).splits;
}

// C (or, `parts`: the fp32 partial tiles [splits][M][N]) of up to 128 rows; `act`: ACT_*
int gemm_skinny(const void* A, const void* W, void* C, int M, int N, int K, int act, long long ldc, const float* bias, float limit,
                float* parts, bool fixed_w, cudaStream_t st) {
  SkinnyArgs a{};
  a.fixed_w = fixed_w;
  a.C = (bf16*)C;
  a.parts = parts;
  a.bias = bias;
  a.limit = limit;
  a.ldc = ldc;
  a.patience = g_gemm_give_up ? -1 : WAIT_CYCLES;
  a.M = M;
  a.N = N;
  a.K = K;
  if (act == ACT_SWIGLU) return launch_skinny<1, ACT_SWIGLU>(A, W, a, st);
  if (act == ACT_GEGLU) return launch_skinny<1, ACT_GEGLU>(A, W, a, st);
  if (act == ACT_CLAMPED) return launch_skinny<1, ACT_CLAMPED>(A, W, a, st);
  return wide_tiles(N) ? launch_skinny<2, ACT_NONE>(A, W, a, st) : launch_skinny<1, ACT_NONE>(A, W, a, st);
}

}  // namespace b200q

using namespace b200q;

extern "C" {

// test hook: 1 = products of up to 128 rows give up at their first wait (wrong values, and b200q_wait_failures() says so), 0 = normal
int b200q_gemm_set_give_up(int on) {
  g_gemm_give_up = on != 0;
  bump_tuning_epoch();
  return B200Q_OK;
}

}  // extern "C"
