// prefill_attn.cu — softmax attention of prompt portions over the paged cache on the 5th-generation tensor cores (page layout: attn.cu).
//
// Bound: tensor pipe and exponentials (a 128 x 128 block of scores costs 1024 cycles of products at D = 128 and 1024 cycles of the
// exponential unit); the cache is read once per 256 query rows.  At D = 256 shared memory: 64 keys of 128 query rows move 192 KB through
// it (operands in, 128 bytes a cycle), 1.5k of the 2.1k cycles that a step takes.
// us, when warps found their runs themselves, stored rows through shared memory and shared a step's columns (D = 256) / now: 36 prompts of
// 128 tokens 32.9 / 25.2 (D = 128), three of 333 to 2048 tokens 85 / 66 (D = 256), one of 6000 335 / 275 (D = 128), 270 / 226 (D = 64).
//   * A CTA works a block of consecutive q-tiles (<= 16 tokens each) for one kv head.  Neighbouring tiles of one portion form a run; the
//     run's rows are (token, head of the group) pairs, 128 of them to a tensor-core tile: all heads of a group share what is fetched.
//   * Pages arrive by tiled TMA copies, one each, without a swizzle of their own: the cache stores its 16-byte chunks permuted within
//     eight rows as the tensor core's 128-byte swizzle does, so groups of eight rows cut into 64-column slices are operands as they are
//     (keys K-major, values N-major).
//   * Scores and outputs live in tensor memory; probabilities go back there as bf16 and are the A operand of the second product.
//     D = 64, 128: two query tiles per CTA (four warps of softmax each), one's exponentials behind the other's products; 128 keys at a
//     time.  D = 256: one query tile (its outputs take 256 columns), 64 keys at a time, four blocks of scores; three warpgroups take the
//     steps in turns.
//   * The running maximum moves only when a row's grows by more than 2^8 (exponents stay far from overflow; at D = 256 the first 512
//     keys follow it exactly, so that short contexts round as the plain form does); the outputs in tensor memory are scaled in place.
//   * Persistent: one CTA per SM walks its blocks, last tiles (the longest ones of a prompt) first; the page ring runs on across them.
#include <type_traits>

#include "tcgen05.cuh"

namespace b200q {

template <int D>
struct FaCfg {
  static constexpr int NQ = D > 128 ? 1 : 2;       // query tiles of 128 rows per CTA
  static constexpr int KT = D > 128 ? 64 : 128;    // keys per step
  static constexpr int STG = D == 64 ? 3 : 2;      // ring stages of keys and of values
  static constexpr int MAX_G = D > 128 ? 4 : 8;
  static constexpr int GROUPS = D > 128 ? 3 : 2;   // warpgroups of softmax
  static constexpr int SW = 4 * GROUPS;            // the warp that fetches pages; behind it the one that issues products, two that fetch queries
  static constexpr int THREADS = 32 * (SW + 4);
  static constexpr int CH = D / 64;                // 64-column slices of a row
  static constexpr int Q_BYTES = 128 * D * 2, T_BYTES = KT * D * 2;
  static constexpr int BUFS = D > 128 ? 1 : 2;       // patches of 32 rows x 32 columns per warp, through which outputs leave
  static constexpr int SMEM = NQ * Q_BYTES + 2 * STG * T_BYTES + SW * BUFS * 2048 + 1024;
  static constexpr int O_COL = 256;  // tensor memory: scores from column 0, outputs from here
};

struct FaArgs {
  const bf16* q;
  bf16* out;
  const uint8_t* kv;
  const int32_t* block_table;
  const int4* tiles;
  int* failed;
  int q_stride, bt_stride, n_tiles, per_block, n_q, n_kv, G, window;
  int long_keys;    // (kSplit) portions of fewer keys are left to the kernel of 16-token tiles
  float c0, c1;  // of a score: plain s * c0 in base 2; capped c1 * tanh(s * c0); c0 > 0
  uint32_t q_flip;  // the queries' sign bits turned (a negative scale)
  int vec;          // rows of q and out are 16-byte aligned
  int whole_tokens;  // the 32 rows of a warp are whole tokens, and q and out may be read and written by TMA as they are
  uint32_t inv_g;   // 65536 / G + 1: f / G = f * inv_g >> 16 for the rows of a CTA
};

struct FaRun {
  int bt_row, row0, n, pos0;
};
// A run and its kv head as the page warp hands it to the other roles: keys from k0 on in n0 steps for the first query tile, n1 for the
// second (0: no rows there); n0 = 0: there are no more.  Runs go through a ring in shared memory: found by every warp for itself, they cost
// 1400 to 2000 cycles between two runs.
struct __align__(16) FaWork {
  int bt_row, row0, n, pos0, kvh, k0, n0, n1;
};
constexpr int FA_RING = 8;

// Which units (block of tiles, kv head) a CTA works, and in which order: blocks by the number of their steps, longest first, dealt out
// back and forth over the CTAs (0 .. n-1, n-1 .. 0, ...), so that every CTA gets long and short ones: three prompts of 333 to 2048
// tokens, D = 256, 448 units: 89 us, 110 to 150 with blocks dealt out in the order of the list.
constexpr int FA_SORTED = 512;  // more blocks than this keep the order of the list, last ones first
struct FaOrder {
  const uint16_t* sorted;
  int n_blocks, units;
  __device__ __forceinline__ int block(int rank) const { return sorted ? sorted[rank] : n_blocks - 1 - rank; }
};
struct FaUnit {  // a CTA's place: unit u, at x of its round
  int u = blockIdx.x, x = blockIdx.x;
  __device__ __forceinline__ void step() {
    const int g = gridDim.x;
    u += 2 * (g - x) - 1;
    x = g - 1 - x;
  }
};

// An entry of a table (tiles, pages).  D = 64: a load instruction of its own; as the compiler places plain ones, one prompt of 6000 tokens
// takes 287 us instead of 270 and 4 of 300 to 1200 43.9 instead of 41.2.  D = 128 and 256 lose 1 to 2 % by it.
template <int D, typename T>
__device__ __forceinline__ T table_entry(const T* p) {
  if constexpr (D == 64)
    return __ldca(p);
  else
    return *p;
}

// portion_keys of the tiles first .. first + 15, one per lane
template <int D>
__device__ __forceinline__ int block_portion_keys(const FaArgs& a, int first, int lane) {
  uint64_t ends = 0;  // bit p: tile first + p does not continue the one before it
  int keys[2], x = 0, y = 0, w = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = first + 32 * h + lane;
    const int4 t = table_entry<D>(a.tiles + min(i, a.n_tiles - 1));
    const int n = min(max(t.z, 0), 16);
    keys[h] = t.w + n;
    // (lane 0 compares with lane 31 of the half before)
    const int px = __shfl_up_sync(0xffffffffu, t.x, 1);
    const int x0 = __shfl_sync(0xffffffffu, x, 31), y0 = __shfl_sync(0xffffffffu, y, 31), w0 = __shfl_sync(0xffffffffu, w, 31);
    const int py = __shfl_up_sync(0xffffffffu, t.y + n, 1), pw = __shfl_up_sync(0xffffffffu, t.w + n, 1);
    const bool on = (lane ? px : x0) == t.x && (lane ? py : y0) == t.y && (lane ? pw : w0) == t.w && i < a.n_tiles;
    ends |= (uint64_t)__ballot_sync(0xffffffffu, !on) << (32 * h);
    x = t.x;
    y = t.y + n;
    w = t.w + n;
  }
  const uint64_t later = ends >> (lane + 1);
  const int last = lane + min(later ? __ffsll((long long)later) - 1 : 31, 31);
  const int k0 = __shfl_sync(0xffffffffu, keys[0], last & 31), k1 = __shfl_sync(0xffffffffu, keys[1], last & 31);
  return last < 32 ? k0 : k1;
}

// the runs of a block, seen by a whole warp: lane l holds tile l of the block
template <int D>
struct FaBlock {
  int4 t, ahead;
  uint32_t starts;  // bit l: tile l begins a run
  int count, ahead_count, ahead_first;
  // the tiles of unit u are asked for one unit ahead
  __device__ __forceinline__ void fetch(const FaArgs& a, const FaOrder& o, int u, int lane) {
    ahead_first = u < o.units ? o.block(u / a.n_kv) * a.per_block : a.n_tiles;
    ahead_count = min(a.per_block, a.n_tiles - ahead_first);
    ahead = lane < ahead_count ? table_entry<D>(a.tiles + ahead_first + lane) : make_int4(0, 0, 0, 0);
  }
  template <bool kSplit>
  __device__ __forceinline__ void begin(const FaArgs& a, const FaOrder& o, FaUnit at, int lane) {
    const int first = ahead_first;
    count = ahead_count;
    t = ahead;
    at.step();
    fetch(a, o, at.u, lane);
    t.z = min(max(t.z, 0), 16);
    if constexpr (kSplit)
      if (block_portion_keys<D>(a, first, lane) < a.long_keys) t.z = 0;  // (no rows: no run)
    const int br = __shfl_up_sync(0xffffffffu, t.x, 1), r0 = __shfl_up_sync(0xffffffffu, t.y, 1), nn = __shfl_up_sync(0xffffffffu, t.z, 1),
              p0 = __shfl_up_sync(0xffffffffu, t.w, 1);
    const bool next = lane > 0 && lane < count && br == t.x && r0 + nn == t.y && p0 + nn == t.w;
    starts = __ballot_sync(0xffffffffu, lane < count && !next);
  }
  // run that begins at tile `at`; returns the tile behind it
  __device__ __forceinline__ int run(int at, FaRun& r) const {
    const uint32_t later = at < 31 ? starts & (0xfffffffeu << at) : 0u;
    const int end = later ? __ffs(later) - 1 : count;
    r.bt_row = __shfl_sync(0xffffffffu, t.x, at);
    r.row0 = __shfl_sync(0xffffffffu, t.y, at);
    r.pos0 = __shfl_sync(0xffffffffu, t.w, at);
    r.n = __shfl_sync(0xffffffffu, t.y, end - 1) + __shfl_sync(0xffffffffu, t.z, end - 1) - r.row0;
    return end;
  }
};

// (D = 256) a wait that gives up after about two seconds, or once another role of the CTA has
__device__ __forceinline__ bool fa_wait(uint64_t* bar, uint32_t parity, volatile int* dead, int* failed) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (*dead) return false;
    if (clock64() - t0 > WAIT_CYCLES) {
      *dead = 1;
      *(volatile int*)failed = 1;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const void* tmap, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_store_3d(const void* tmap, int c0, int c1, int c2, uint32_t smem_src) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(tmap), "r"(c0), "r"(c1), "r"(c2),
               "r"(smem_src)
               : "memory");
}
__device__ __forceinline__ float fa_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// two numbers at once, as neighbouring registers (one issue slot)
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair_of(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 halves_of(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float fa_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// One query row of one head once more, by a whole warp, over the keys lo .. pos and no others
template <int D, bool kCap>
__device__ __forceinline__ void fa_row_again(const FaArgs& a, const int32_t* bt, const bf16* q_row, bf16* out_row, int kvh, int lo, int pos) {
  const int lane = threadIdx.x & 31;
  constexpr int NW = D / 64;  // 32-bit words of the output per lane
  const long long page_bytes = 16 * D * 2;
  const uint32_t* q4 = reinterpret_cast<const uint32_t*>(q_row);
  float m = -INFINITY, l = 0.f, acc[NW][2];
#pragma unroll
  for (int w = 0; w < NW; ++w) acc[w][0] = acc[w][1] = 0.f;
  lo = max(lo, 0);
  for (int j0 = lo & ~31; j0 <= pos; j0 += 32) {
    const int j = j0 + lane, t = j & 15;
    const bool seen = j >= lo && j <= pos;
    const int blk = seen ? table_entry<D>(bt + (j >> 4)) : 0;
    float s = -INFINITY;
    if (seen) {
      const uint8_t* row = a.kv + ((long long)blk * 2 * a.n_kv + kvh) * page_bytes + t * (D * 2);
      float dot = 0.f;
#pragma unroll 4
      for (int c = 0; c < D / 8; ++c) {
        const uint4 k = *reinterpret_cast<const uint4*>(row + ((c ^ (t & 7)) << 4));
        const uint32_t kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const uint32_t q = q4[4 * c + x] ^ a.q_flip;
          dot = fmaf(bf16_lo(q), bf16_lo(kk[x]), dot);
          dot = fmaf(bf16_hi(q), bf16_hi(kk[x]), dot);
        }
      }
      s = kCap ? a.c1 * tanhf(dot * a.c0) : dot * a.c0;
    }
    float top = s;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (top > m) {
      const float alpha = fa_ex2(m - top);
      m = top;
      l *= alpha;
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        acc[w][0] *= alpha;
        acc[w][1] *= alpha;
      }
    }
    const float p = seen ? fa_ex2(s - (m == -INFINITY ? 0.f : m)) : 0.f;
    l += p;
    const float p16 = round_bf16(p);
    for (int i = max(lo - j0, 0); i < 32 && j0 + i <= pos; ++i) {  // (the warp agrees on i)
      const float pi = __shfl_sync(0xffffffffu, p16, i);
      const int bi = __shfl_sync(0xffffffffu, blk, i), ti = (j0 + i) & 15;
      const uint8_t* row = a.kv + (((long long)bi * 2 + 1) * a.n_kv + kvh) * page_bytes + ti * (D * 2);
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const int word = w * 32 + lane;
        const uint32_t v = *reinterpret_cast<const uint32_t*>(row + (((word >> 2) ^ (ti & 7)) << 4) + (word & 3) * 4);
        acc[w][0] = fmaf(pi, bf16_lo(v), acc[w][0]);
        acc[w][1] = fmaf(pi, bf16_hi(v), acc[w][1]);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
  for (int w = 0; w < NW; ++w)
    reinterpret_cast<uint32_t*>(out_row)[w * 32 + lane] = pack_bf16x2(acc[w][0] * inv, acc[w][1] * inv);
}

// The rows of this CTA's units whose outputs are NaN, once more, by its softmax warps behind their loops.  In the products of the kernel
// below a hidden key's probability is 0, and times a value that is not finite that is NaN, for every row of the query tile that shares the
// step.  (A row that sees such a value itself comes here too, and gets what it sees.)
template <int D, bool kCap, bool kSplit>
__device__ __noinline__ void fa_rows_again(const FaArgs& a, const FaOrder order) {  // (by the softmax warps)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (FaUnit w; w.u < order.units; w.step()) {
    const int kvh = w.u % a.n_kv, first = order.block(w.u / a.n_kv) * a.per_block, count = min(a.per_block, a.n_tiles - first);
    int keys = 0;
    if constexpr (kSplit) keys = block_portion_keys<D>(a, first, lane);
    for (int i = 0; i < count; ++i) {
      const int4 t = table_entry<D>(a.tiles + first + i);
      if (kSplit && __shfl_sync(0xffffffffu, keys, i) < a.long_keys) continue;
      const int rows = min(max(t.z, 0), 16) * a.G;
      for (int f = warp; f < rows; f += FaCfg<D>::SW) {
        const int tok = f / a.G, head = kvh * a.G + f - tok * a.G, pos = t.w + tok;
        bf16* out_row = a.out + (long long)(t.y + tok) * a.n_q * D + (long long)head * D;
        bool nan = false;
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          const uint32_t v = reinterpret_cast<const uint32_t*>(out_row)[c * 32 + lane];
          nan |= bf16_lo(v) != bf16_lo(v) || bf16_hi(v) != bf16_hi(v);
        }
        if (__any_sync(0xffffffffu, nan))
          fa_row_again<D, kCap>(a, a.block_table + (long long)t.x * a.bt_stride,
                                a.q + (long long)(t.y + tok) * a.q_stride + (long long)head * D, out_row, kvh,
                                a.window > 0 ? pos + 1 - a.window : 0, pos);
      }
    }
  }
}

// kSplit: only the portions of long_keys keys and more (a variant of its own: the code to look at them costs the other one 1 to 2 % in
// instruction fetches, where CTAs walk many short units)
template <int D, bool kCap, bool kSplit>
__global__ void __launch_bounds__(FaCfg<D>::THREADS, 1) prefill_attn_kernel(const __grid_constant__ CUtensorMap kv_map, const __grid_constant__ CUtensorMap q_map,
                    const __grid_constant__ CUtensorMap out_map, const __grid_constant__ FaArgs a) {
  using C = FaCfg<D>;
  constexpr int NQ = C::NQ, KT = C::KT, STG = C::STG, CH = C::CH, PAGES = KT / 16, FA_THREADS = C::THREADS, GROUPS = C::GROUPS, SW = C::SW;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* q_s = smem;
  uint8_t* k_s = smem + NQ * C::Q_BYTES;
  uint8_t* v_s = k_s + STG * C::T_BYTES;
  constexpr int SLOTS = NQ == 1 ? 4 : 2;  // blocks of scores in tensor memory (D = 256: of consecutive steps; else one per query tile)
  __shared__ __align__(8) uint64_t k_full[STG], k_empty[STG], v_full[STG], v_empty[STG], q_ready[2], q_empty[2], s_full[SLOTS], p_ready[SLOTS],
      o_full[2], pv_done[4], o_read, m_ready[SW], l_ready[2 * SW], work_full[FA_RING], work_empty[FA_RING];
  __shared__ FaWork ring[FA_RING];
  uint8_t* patches = v_s + STG * C::T_BYTES;
  __shared__ float row_max[NQ == 1 ? 128 : 1], part[2][GROUPS][NQ == 1 ? 128 : 1];  // D = 256: running maxima; sums of every warpgroup's steps, in turns
  __shared__ uint32_t tmem_slot;
  __shared__ int dead, redo;  // a wait ran out; some output is NaN although its row's sum is finite
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  __shared__ uint16_t sorted[FA_SORTED];
  int* steps_in = reinterpret_cast<int*>(patches);  // (free until the first rows leave)
  const int n_blocks = (a.n_tiles + a.per_block - 1) / a.per_block;
  const bool sort = n_blocks <= FA_SORTED && n_blocks * a.n_kv > (int)gridDim.x;  // (one unit each: nothing to deal out)
  const FaOrder order{sort ? sorted : nullptr, n_blocks, n_blocks * a.n_kv};

  if (threadIdx.x == 0) {
    dead = redo = 0;
    for (int s = 0; s < STG; ++s) {
      mbar_init(k_full + s, 1);
      mbar_init(k_empty + s, 1);
      mbar_init(v_full + s, 1);
      mbar_init(v_empty + s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(q_ready + i, 2);
      mbar_init(q_empty + i, 1);
      mbar_init(o_full + i, 1);
    }
    for (int i = 0; i < 4; ++i) mbar_init(pv_done + i, 1);
    for (int i = 0; i < SLOTS; ++i) {
      mbar_init(s_full + i, 1);
      mbar_init(p_ready + i, 4);
    }
    mbar_init(&o_read, SW);
    for (int i = 0; i < SW; ++i) {
      mbar_init(m_ready + i, 1);
      mbar_init(l_ready + i, 1);
      mbar_init(l_ready + SW + i, 1);
    }
    for (int i = 0; i < FA_RING; ++i) {
      mbar_init(work_full + i, 1);
      mbar_init(work_empty + i, SW + 3);  // (softmax, products, queries)
    }
    mbar_fence_init();
  }
  if (sort)
    for (int i = threadIdx.x; i < n_blocks; i += FA_THREADS) steps_in[i] = 0;
  for (int i = 8 * ((int)blockIdx.x + (int)gridDim.x * (int)threadIdx.x); i < a.n_tiles; i += 8 * (int)gridDim.x * FA_THREADS)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(a.tiles + i));
  if constexpr (kSplit) {  // no tile sees so many keys: nothing to do here
    wait_for_previous();
    bool any = false;
    for (int i = threadIdx.x; i < a.n_tiles; i += FA_THREADS) {
      const int4 t = table_entry<D>(a.tiles + i);
      any |= t.w + min(max(t.z, 0), 16) >= a.long_keys;
    }
    if (!__syncthreads_or(any)) return;
  }
  if (warp == SW + 1) tmem_alloc(&tmem_slot, 512);
  __syncthreads();
  follow_previous();
  if (sort) {
    for (int i = threadIdx.x; i < a.n_tiles; i += FA_THREADS) {  // the last token of a run sees most keys
      const int4 t = table_entry<D>(a.tiles + i), n = table_entry<D>(a.tiles + min(i + 1, a.n_tiles - 1));
      const bool ends = i + 1 == a.n_tiles || (i + 1) % a.per_block == 0 || n.x != t.x || n.y != t.y + t.z || n.w != t.w + t.z;
      const int all = t.w + t.z, keys = a.window > 0 ? min(all, a.window) : all;
      if (ends && (!kSplit || all >= a.long_keys)) atomicAdd(steps_in + i / a.per_block, max(keys, 0) / KT + 2);  // (start and end: about one step)
    }
    __syncthreads();
    const int by = n_blocks <= FA_THREADS / 4 ? 4 : 1;  // threads that look through the blocks for one of them
    for (int i0 = 0; i0 < n_blocks; i0 += FA_THREADS) {
      const int i = i0 + threadIdx.x / by, mine = i < n_blocks ? steps_in[i] : 0;
      int rank = 0;
      for (int k = threadIdx.x % by; k < n_blocks; k += by) rank += steps_in[k] > mine || (steps_in[k] == mine && k > i);
      if (by == 4) {
        rank += __shfl_xor_sync(0xffffffffu, rank, 1);
        rank += __shfl_xor_sync(0xffffffffu, rank, 2);
      }
      if (i < n_blocks) sorted[rank] = (uint16_t)i;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_slot, 0);
  // (the loop that looks at the flag every 16 tries and has no try before it spares registers: one prompt of 8000 tokens, D = 128, 607 ->
  // 505 us; D = 256 has none to spare for it, 450 -> 468)
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if constexpr (NQ == 2)
      return mbar_wait_or_fail<16>(bar, parity, &dead, a.failed);
    else
      return fa_wait(bar, parity, &dead, a.failed);
  };
  // the x-th run of this CTA (a whole warp asks)
  auto take = [&](int x) {
    const int slot = x % FA_RING;
    const bool ok = __all_sync(0xffffffffu, wait(work_full + slot, (uint32_t)(x / FA_RING) & 1u));
    FaWork r = ring[slot];
    if (!ok) r.n0 = 0;
    __syncwarp();
    if (lane == 0) mbar_arrive(work_empty + slot);
    return r;
  };
  // steps of KT keys that query tile i of a run walks: from the page of the first token's first visible key to the tile's last token
  auto first_key = [&](const FaRun& r) { return a.window > 0 && r.pos0 + 1 > a.window ? (r.pos0 + 1 - a.window) / 16 * 16 : 0; };
  auto steps_of = [&](const FaRun& r, int i, int k0) {
    const int rows = min(r.n * a.G, (i + 1) * 128);
    return rows > i * 128 ? (r.pos0 + (int)((uint32_t)(rows - 1) * a.inv_g >> 16) + 1 - k0 + KT - 1) / KT : 0;
  };

  // (384 threads were launched with 168 registers each: 2 x 208 + 88 = 3 x 168; D = 256 512 with 128: 3 x 144 + 80 = 4 x 128)
  if (warp >= SW) {
  if constexpr (NQ == 2)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
  else
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
  if (warp == SW) {
    // ===== pages =====
    if (lane == 0) tma_prefetch_desc(&kv_map);
    int n_keys = 0, n_values = 0, n_work = 0, at = 0;
    FaBlock<D> b;
    FaUnit w;
    b.count = 0;
    b.fetch(a, order, blockIdx.x, lane);
    // finds the next run and hands it to the other roles
    auto next = [&](FaWork& x) {
      FaRun r;
      for (r.n = 0; r.n <= 0;) {
        if (at >= b.count) {
          if (w.u >= order.units) break;
          b.template begin<kSplit>(a, order, w, lane);
          x.kvh = w.u % a.n_kv;
          w.step();
          at = 0;
        }
        at = b.run(at, r);
      }
      x.n0 = x.n1 = 0;
      if (r.n > 0) {
        x.bt_row = r.bt_row;
        x.row0 = r.row0;
        x.n = r.n;
        x.pos0 = r.pos0;
        x.k0 = first_key(r);
        x.n0 = steps_of(r, 0, x.k0);
        if (NQ == 2) x.n1 = steps_of(r, 1, x.k0);
      }
      const int slot = n_work % FA_RING;
      const bool ok = __all_sync(0xffffffffu, wait(work_empty + slot, ((uint32_t)(n_work / FA_RING) & 1u) ^ 1u));
      ++n_work;
      if (!ok) x.n0 = x.n1 = 0;  // (the readers give up as well)
      if (ok && lane == 0) {
        ring[slot] = x;
        mbar_arrive(work_full + slot);
      }
      __syncwarp();
    };
    constexpr int AHEAD = NQ == 1 ? SLOTS : 1;  // steps by which keys are asked for before values, whose slot is free that much later
    auto page_of = [&](const FaWork& r, int j) {
      const int i = j * PAGES + lane;
      return lane < PAGES && i < (r.pos0 + r.n + 15) / 16 - r.k0 / 16 && j < max(r.n0, r.n1)
                 ? table_entry<D>(a.block_table + (long long)r.bt_row * a.bt_stride + r.k0 / 16 + i)
                 : 0;
    };
    // Every run is found while the pages of the one before it are still to be asked for, so that the places of its own first pages are
    // known when it is their turn.
    FaWork r, after;
    r.n0 = r.n1 = after.kvh = 0;
    int blk[AHEAD + 3];  // of steps j .. j + AHEAD + 2
    for (;;) {
      next(after);
      const int page0 = after.n0 > 0 ? page_of(after, 0) : 0, page1 = after.n0 > 0 ? page_of(after, 1) : 0;
      const int total = r.pos0 + r.n, steps = max(r.n0, r.n1);
      auto load = [&](int which, int j, int page_at) {
        const int valid = min(KT, total - (r.k0 + j * KT)), mine = min(16, valid - 16 * lane);
        const int n = which ? n_values++ : n_keys++, st = n % STG;
        const uint32_t par = (uint32_t)(n / STG) & 1u;
        uint64_t* full = which ? v_full + st : k_full + st;
        wait(which ? v_empty + st : k_empty + st, par ^ 1u);
        __syncwarp();
        uint8_t* dst = (which ? v_s : k_s) + st * C::T_BYTES;
        if (which && valid < KT) {  // probabilities of keys that are not there are zero: their values must not be NaN
          for (int i = lane; i < (KT - valid) * CH * 8; i += 32) {
            const int row = valid + i / (CH * 8), c = i % (CH * 8);
            *reinterpret_cast<uint4*>(dst + (row >> 3) * (CH * 1024) + (c >> 3) * 1024 + (row & 7) * 128 + (c & 7) * 16) =
                make_uint4(0, 0, 0, 0);
          }
          fence_async_shared();
          __syncwarp();
        }
        if (lane == 0) mbar_expect_tx(full, (uint32_t)(valid * D * 2));
        __syncwarp();
        if (lane < PAGES && mine > 0) {
          const long long page = ((long long)page_at * 2 + which) * a.n_kv + r.kvh;
          uint8_t* to = dst + lane * (CH * 2048);
          if (mine == 16) {
            tma_load_4d(to, &kv_map, 0, 0, 0, (int)(page * 2), full);
          } else {  // the rows that exist, one by one
            const uint8_t* src = a.kv + page * (16 * D * 2);
            for (int row = 0; row < mine; ++row)
#pragma unroll
              for (int c = 0; c < CH; ++c)
                tma_bulk_g2s(to + (row >> 3) * (CH * 1024) + c * 1024 + (row & 7) * 128, src + row * (D * 2) + c * 128, 128, full);
          }
        }
        __syncwarp();
      };
#pragma unroll 1
      for (int j = -AHEAD; j < steps; ++j) {
        blk[AHEAD + 2] = page_of(r, j + AHEAD + 2);
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {
          const int i = which ? j : j + AHEAD;
          if (i >= 0 && i < steps) load(which, i, which ? blk[0] : blk[AHEAD]);
        }
#pragma unroll
        for (int i = 0; i < AHEAD + 2; ++i) blk[i] = blk[i + 1];
      }
      if (after.n0 == 0) break;
      r = after;
      blk[AHEAD] = page0;
      blk[AHEAD + 1] = page1;
    }
  } else if (warp == SW + 1) {
    // ===== products =====
    constexpr uint32_t base_desc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 4) << 24);
    constexpr uint32_t qk_desc = base_desc | ((uint32_t)(KT >> 3) << 17);
    constexpr uint32_t pv_desc = base_desc | (1u << 16) | ((uint32_t)(D >> 3) << 17);  // values: N-major
    auto issue_qk = [&](int i, int slot, int st) {
      const uint32_t qa = smem_u32(q_s + i * C::Q_BYTES), kb = smem_u32(k_s + st * C::T_BYTES);
#pragma unroll
      for (int k = 0; k < D / 16; ++k)
        umma_bf16(tmem + (uint32_t)(slot * KT), make_smem_desc(qa + (k >> 2) * 16384 + (k & 3) * 32),
                  make_smem_desc(kb + (k >> 2) * 1024 + (k & 3) * 32, CH * 1024), qk_desc, k > 0 ? 1u : 0u);
    };
    auto issue_pv = [&](int i, int slot, int st, bool add) {
      const uint32_t vb = smem_u32(v_s + st * C::T_BYTES);
#pragma unroll
      for (int k = 0; k < KT / 16; ++k)
        umma_bf16_ts(tmem + (uint32_t)(C::O_COL + i * D), tmem + (uint32_t)(slot * KT + k * 8),
                     make_smem_desc(vb + k * (CH * 2048), CH * 1024, 1024), pv_desc, add || k > 0 ? 1u : 0u);
    };
    int n_k = 0, n_v = 0, n_p[2] = {0, 0}, n_s = 0;
    uint32_t q_par[2] = {0, 0};
    auto next_k = [&]() {
      wait(k_full + n_k % STG, (uint32_t)(n_k / STG) & 1u);
      __syncwarp();
      tc_fence_after();
    };
    for (int x = 0;; ++x) {
      const FaWork r = take(x);
      // (from one lane: the compiler then knows that the warp agrees)
      const int n0 = __shfl_sync(0xffffffffu, r.n0, 0), n1 = NQ == 2 ? __shfl_sync(0xffffffffu, r.n1, 0) : 0, steps = n1 > 0 ? n1 : n0;
      if (steps == 0) break;
#pragma unroll
      for (int i = 0; i < NQ; ++i)
        if (i == 0 || n1 > 0) {
          wait(q_ready + i, q_par[i]);
          q_par[i] ^= 1u;
        }
      if constexpr (NQ == 2) {
        next_k();
        if (elect_one()) {
          issue_qk(0, 0, n_k % STG);
          umma_commit(s_full + 0);
          if (n0 == 1) umma_commit(q_empty + 0);
          if (n1 > 0) {
            issue_qk(1, 1, n_k % STG);
            umma_commit(s_full + 1);
            if (n1 == 1) umma_commit(q_empty + 1);
          }
          umma_commit(k_empty + n_k % STG);
        }
        __syncwarp();
        ++n_k;
        for (int j = 0; j < steps; ++j) {
          const bool more = j + 1 < steps;
          if (more) next_k();
          wait(v_full + n_v % STG, (uint32_t)(n_v / STG) & 1u);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int n = i ? n1 : n0;
            if (j < n) {
              wait(p_ready + i, (uint32_t)n_p[i] & 1u);
              __syncwarp();
              ++n_p[i];
              tc_fence_after();
              if (elect_one()) {
                issue_pv(i, i, n_v % STG, j > 0);
                if (j + 1 < n) {  // (products are made in order: the scores are written once the probabilities have been read)
                  issue_qk(i, i, n_k % STG);
                  umma_commit(s_full + i);
                  if (j + 2 == n) umma_commit(q_empty + i);
                } else {
                  umma_commit(o_full + i);
                }
              }
              __syncwarp();
            }
          }
          if (elect_one()) {
            umma_commit(v_empty + n_v % STG);
            if (more) umma_commit(k_empty + n_k % STG);
          }
          __syncwarp();
          ++n_v;
          if (more) ++n_k;
        }
      } else {
        // scores are as many steps ahead as there is room for them: those of step j come behind the product of step j - SLOTS
        auto scores = [&](int j) {
          next_k();
          const int slot = (n_s + j) % SLOTS;
          if (elect_one()) {
            issue_qk(0, slot, n_k % STG);
            umma_commit(s_full + slot);
            if (j + 1 == steps) umma_commit(q_empty + 0);
            umma_commit(k_empty + n_k % STG);
          }
          __syncwarp();
          ++n_k;
        };
#pragma unroll 1
        for (int j = 0; j < min(SLOTS, steps); ++j) scores(j);
        for (int j = 0; j < steps; ++j) {
          const int g = n_s + j, slot = g % SLOTS;
          wait(v_full + n_v % STG, (uint32_t)(n_v / STG) & 1u);
          wait(p_ready + slot, (uint32_t)(g / SLOTS) & 1u);
          if (j == 0) wait(&o_read, ((uint32_t)x & 1u) ^ 1u);  // (the outputs of the run before have been read)
          __syncwarp();
          tc_fence_after();
          if (elect_one()) {
            issue_pv(0, slot, n_v % STG, j > 0);
            umma_commit(v_empty + n_v % STG);
            umma_commit(pv_done + slot);
            if (j + 1 == steps) umma_commit(o_full + 0);
          }
          __syncwarp();
          ++n_v;
          if (j + SLOTS < steps) scores(j + SLOTS);
        }
        n_s += steps;
      }
    }
  } else {
    // ===== queries into shared memory, as the tensor core reads them =====
    constexpr int LPR = D / 8, RPP = 64 / LPR;  // lanes per row, rows per pass of the two warps
    const int tid = threadIdx.x - 32 * (SW + 2), c = tid % LPR;
    uint32_t par[2] = {1, 1};
    for (int x = 0;; ++x) {
      const FaWork r = take(x);
      if (r.n0 == 0) break;
      {
        const int rows = r.n * a.G, kvh = r.kvh;
        const bf16* src0 = a.q + (long long)r.row0 * a.q_stride + (long long)kvh * a.G * D + c * 8;
        auto source = [&](int f) {
          const int t = (int)((uint32_t)f * a.inv_g >> 16);
          return src0 + (long long)t * a.q_stride + (f - t * a.G) * D;
        };
        // (a tile whose rows all exist comes by TMA; of the others there is one at most, the run's last)
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
          if (i * 128 >= rows) break;
          wait(q_empty + i, par[i]);
          __syncwarp();
          par[i] ^= 1u;
          if (a.whole_tokens && (i + 1) * 128 <= rows) {
            if (lane == 0) {
              if (warp == SW + 2) {
                mbar_expect_tx(q_ready + i, C::Q_BYTES);
#pragma unroll
                for (int h = 0; h < CH; ++h)
                  tma_load_3d(q_s + i * C::Q_BYTES + h * 16384, &q_map, h * 64, kvh * a.G, r.row0 + (int)((uint32_t)(i * 128) * a.inv_g >> 16),
                              q_ready + i);
              } else {
                mbar_arrive(q_ready + i);
              }
            }
            __syncwarp();
            continue;
          }
          uint8_t* dst = q_s + i * C::Q_BYTES + (c >> 3) * 16384;
          if (a.vec && a.q_flip == 0) {
#pragma unroll 4
            for (int x = tid / LPR; x < 128; x += RPP) {
              const int f = i * 128 + x;
              const bool on = f < rows;
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + x * 128 + (((c & 7) ^ (x & 7)) << 4))),
                           "l"(on ? source(f) : src0), "r"(on ? 16 : 0)
                           : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 0;" ::: "memory");
          } else {
            for (int x = tid / LPR; x < 128; x += RPP) {
              const int f = i * 128 + x;
              uint4 v = make_uint4(0, 0, 0, 0);
              if (f < rows) {
                const uint32_t* s4 = reinterpret_cast<const uint32_t*>(source(f));
                v = make_uint4(s4[0] ^ a.q_flip, s4[1] ^ a.q_flip, s4[2] ^ a.q_flip, s4[3] ^ a.q_flip);
              }
              *reinterpret_cast<uint4*>(dst + x * 128 + (((c & 7) ^ (x & 7)) << 4)) = v;
            }
          }
          fence_async_shared();
          __syncwarp();
          if (lane == 0) mbar_arrive(q_ready + i);
        }
      }
    }
  }
  } else {
    if constexpr (NQ == 2)
      asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    else
      asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
    // ===== softmax: a row per thread =====
    const int wg = warp >> 2, i_tile = NQ == 2 ? wg : 0;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t s_count = 0, o_par = 0;  // steps so far (D = 256: of all warpgroups)
    const float c0e = 2.8853900817779268f * a.c0;  // 2 log2 e c0
    auto capped = [&](float v) {  // c1 tanh(c0 v) = c1 - 2 c1 / (1 + e^(2 c0 v))
      return fmaf(-2.f * a.c1, fa_rcp(fa_ex2(v * c0e) + 1.f), a.c1);
    };
    // c1 tanh(z) - base, z = c0 v, from the first terms of its series: five for |z| <= 0.3 (the next one is below 6e-8 of the sum); three
    // for |z| <= 0.1, whose coefficients make up for the fourth (economised: w^3, w = z^2, less the Chebyshev polynomial of degree 3 on
    // that interval with a zero at 0; 3e-9 of the sum, 5e-8 without).  On the FMA pipe beside the exponential unit.
    const float t3 = a.c1 * (-1.f / 3.f), t5 = a.c1 * (2.f / 15.f), t7 = a.c1 * (-17.f / 315.f), t9 = a.c1 * (62.f / 2835.f);
    const float u3 = a.c1 * -0.333331008f, u5 = a.c1 * 0.132581935f;
    auto exponents = [&](float v0, float v1, float base, bool three) {
      const f32x2 b = pair_of(-base, -base);
      if constexpr (kCap) {
        const f32x2 z = mul2(pair_of(v0, v1), pair_of(a.c0, a.c0)), w = mul2(z, z);
        f32x2 t;
        if (three) {
          t = fma2(w, pair_of(u5, u5), pair_of(u3, u3));
        } else {
          t = fma2(w, pair_of(t9, t9), pair_of(t7, t7));
          t = fma2(w, t, pair_of(t5, t5));
          t = fma2(w, t, pair_of(t3, t3));
        }
        return halves_of(fma2(z, fma2(w, t, pair_of(a.c1, a.c1)), b));
      }
      return halves_of(fma2(pair_of(v0, v1), pair_of(a.c0, a.c0), b));
    };
    auto both = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(SW * 32) : "memory"); };
    const float no_key = -INFINITY;
    for (int x = 0;; ++x) {
      const FaWork r = take(x);
      if (r.n0 == 0) break;
      const int steps = i_tile ? r.n1 : r.n0, rows = r.n * a.G;
      if (steps == 0) continue;
      const int f = min(i_tile * 128 + row, rows - 1);
      const int tok = (int)((uint32_t)f * a.inv_g >> 16);
      const int pos = r.pos0 + tok, lo = a.window > 0 ? pos + 1 - a.window : 0;
      const int pos_lo = __shfl_sync(0xffffffffu, pos, 0), pos_hi = __shfl_sync(0xffffffffu, pos, 31);  // (rows of later tokens behind)
      float m = no_key, l = 0.f;
      int key0 = r.k0;  // first key of the step
      // chunks of 32 columns: those that no row of the warp sees are left out; whole: every row sees all of the step
      auto used = [&](int c) { return key0 + 32 * c <= pos_hi && (a.window <= 0 || key0 + 32 * c + 31 > pos_lo - a.window); };
      auto whole = [&]() { return key0 + KT - 1 <= pos_lo && (a.window <= 0 || key0 > pos_hi - a.window); };
      // the step's scores: the row's largest (-inf: no key seen), and whether the series serves for all of the warp's
      auto fetch_scores = [&](uint32_t s_at, uint32_t(&s)[KT / 32][32], int& terms) {
#pragma unroll
        for (int c = 0; c < KT / 32; ++c)
          tmem_ld32(s_at + (uint32_t)(32 * c), s[c]);
        tmem_ld_wait();
        float mx[4] = {no_key, no_key, no_key, no_key}, big[2] = {0.f, 0.f};
        // What the warps have to fetch to execute a step counts: the same code for whole steps and for others behind their masks, which lie
        // apart (one prompt of 6000 tokens: D = 64 284 -> 236 us, D = 128 337 -> 272, than with masks between the chunks)
        const bool all = whole();
        if (!all) {
#pragma unroll
          for (int c = 0; c < KT / 32; ++c) {
            const int end = min(max(pos + 1 - key0 - 32 * c, 0), 32), begin = min(max(lo - key0 - 32 * c, 0), 32);
            const uint32_t seen = (end < 32 ? (1u << end) - 1u : ~0u) & (a.window > 0 ? begin < 32 ? ~0u << begin : 0u : ~0u);
#pragma unroll
            for (int y = 0; y < 32; ++y) {
              // (of visible keys only: rows behind the last key hold whatever was in shared memory before)
              if constexpr (kCap) big[y & 1] = fmaxf(big[y & 1], seen >> y & 1u ? fabsf(__uint_as_float(s[c][y])) : 0.f);
              if (!(seen >> y & 1u)) s[c][y] = 0xff800000u;
            }
          }
        }
#pragma unroll
        for (int c = 0; c < KT / 32; ++c)
#pragma unroll
          for (int y = 0; y < 32; y += 2)
            mx[y / 2 & 3] = max3(mx[y / 2 & 3], __uint_as_float(s[c][y]), __uint_as_float(s[c][y + 1]));
        if (kCap && all) {
#pragma unroll
          for (int c = 0; c < KT / 32; ++c)
#pragma unroll
            for (int y = 0; y < 32; y += 2)
              big[y / 2 & 1] = max3(big[y / 2 & 1], fabsf(__uint_as_float(s[c][y])), fabsf(__uint_as_float(s[c][y + 1])));
        }
        const float z = fmaxf(big[0], big[1]) * a.c0;
        terms = !kCap ? 0 : !__all_sync(0xffffffffu, z <= 0.3f) ? 0 : __all_sync(0xffffffffu, z <= 0.1f) ? 3 : 5;
        const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        // (c0 > 0 and tanh grows: the largest product gives the largest score; -inf, no key seen, stays -inf)
        if constexpr (kCap)
          return top == no_key ? top : capped(top);
        else
          return top * a.c0;
      };
      // probabilities in the scores' place, as bf16; returns their sum
      auto give_probabilities = [&](uint32_t s_at, uint32_t(&s)[KT / 32][32], int terms) {
        const float base = m == no_key ? 0.f : m;
        f32x2 sum[2] = {pair_of(0.f, 0.f), pair_of(0.f, 0.f)};
        auto take_all = [&](int c, auto give) {
#pragma unroll
          for (int y = 0; y < 32; y += 2) {
            const float2 p = give(__uint_as_float(s[c][y]), __uint_as_float(s[c][y + 1]));
            sum[y / 2 & 1] = add2(sum[y / 2 & 1], pair_of(p.x, p.y));
            s[c][y / 2] = pack_bf16x2(p.x, p.y);
          }
          tmem_st16(s_at + (uint32_t)(16 * c), s[c]);
        };
        auto simple = [&](float v0, float v1) {
          const float2 e = exponents(v0, v1, base, true);
          return make_float2(fa_ex2(e.x), fa_ex2(e.y));
        };
        auto nothing = [&](int c) {
#pragma unroll
          for (int y = 0; y < 16; ++y) s[c][y] = 0u;
          tmem_st16(s_at + (uint32_t)(16 * c), s[c]);
        };
        // (a hidden key's product is -inf; plain scores carry that through by themselves)
        if (whole() && (!kCap || terms == 3)) {
#pragma unroll
          for (int c = 0; c < KT / 32; ++c) take_all(c, simple);
        } else if (!kCap) {
#pragma unroll
          for (int c = 0; c < KT / 32; ++c)
            if (used(c))
              take_all(c, simple);
            else
              nothing(c);
        } else if (terms == 0) {
#pragma unroll
          for (int c = 0; c < KT / 32; ++c)
            take_all(c, [&](float v0, float v1) {
              return make_float2(fa_ex2(v0 == no_key ? v0 : capped(v0) - base), fa_ex2(v1 == no_key ? v1 : capped(v1) - base));
            });
        } else {
#pragma unroll
          for (int c = 0; c < KT / 32; ++c)
            if (used(c))
              take_all(c, [&](float v0, float v1) {
                const float2 e = exponents(v0, v1, base, false);
                return make_float2(fa_ex2(v0 == no_key ? v0 : e.x), fa_ex2(v1 == no_key ? v1 : e.y));
              });
            else
              nothing(c);
        }
        const float2 s0 = halves_of(sum[0]), s1 = halves_of(sum[1]);
        return (s0.x + s0.y) + (s1.x + s1.y);
      };
      // `n` columns of the outputs so far times alpha
      auto rescale = [&](uint32_t o_at, auto n, auto at_once, float alpha) {
        constexpr int AT_ONCE = decltype(at_once)::value;
#pragma unroll 1
        for (int c = 0; c < decltype(n)::value; c += 32 * AT_ONCE) {
          uint32_t o[AT_ONCE][32];
#pragma unroll
          for (int h = 0; h < AT_ONCE; ++h) tmem_ld32(o_at + (uint32_t)(c + 32 * h), o[h]);
          tmem_ld_wait();
#pragma unroll
          for (int h = 0; h < AT_ONCE; ++h) {
#pragma unroll
            for (int y = 0; y < 32; ++y) o[h][y] = __float_as_uint(__uint_as_float(o[h][y]) * alpha);
            tmem_st32(o_at + (uint32_t)(c + 32 * h), o[h]);
          }
        }
      };
      if constexpr (NQ == 2) {
        const uint32_t s_at = tmem + lanes + (uint32_t)(i_tile * KT);
        for (int j = 0; j < steps; ++j, key0 += KT) {
          wait(s_full + i_tile, s_count & 1u);
          __syncwarp();
          ++s_count;
          tc_fence_after();
          int terms;
          uint32_t s[KT / 32][32];
          const float top = fetch_scores(s_at, s, terms);
          const bool grew = top > m + 8.f;
          if (__any_sync(0xffffffffu, grew)) {
            const float m_new = grew ? top : m;
            const float alpha = grew ? fa_ex2(m - m_new) : 1.f;
            m = m_new;
            l *= alpha;
            if (j > 0) {
              __syncwarp();
              tc_fence_after();
              rescale(tmem + lanes + (uint32_t)(C::O_COL + i_tile * D), std::integral_constant<int, D>{}, std::integral_constant<int, 1>{}, alpha);
            }
          }
          l += give_probabilities(s_at, s, terms);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_ready + i_tile);
        }
      } else {
        // The warpgroups take the steps in turns, whole rows each: a step's running maximum follows from the one before it, which another
        // warpgroup hands over; exponentials, the scaling of the outputs and the sums of a step run beside the next ones'.
        const int quarter = warp & 3, first = (wg + GROUPS - (int)(s_count % GROUPS)) % GROUPS;
        key0 += first * KT;
        for (int j = first; j < steps; j += GROUPS, key0 += GROUPS * KT) {
          const uint32_t g = s_count + j, slot = g % SLOTS;
          const uint32_t s_at = tmem + lanes + slot * KT;
          wait(s_full + slot, g / SLOTS & 1u);
          __syncwarp();
          tc_fence_after();
          int terms;
          uint32_t s[KT / 32][32];
          const float top = fetch_scores(s_at, s, terms);
          float before = no_key;
          if (j > 0) {
            wait(m_ready + (g - 1) % GROUPS * 4 + quarter, (g - 1) / GROUPS & 1u);
            __syncwarp();
            before = row_max[row];
          }
          const bool grew = top > before + (j < 8 ? 0.f : 8.f);
          const float now = grew ? top : before;
          row_max[row] = now;
          __syncwarp();
          if (lane == 0) mbar_arrive(m_ready + wg * 4 + quarter);
          l *= m == now ? 1.f : fa_ex2(m - now);
          m = now;
          l += give_probabilities(s_at, s, terms);
          if (j > 0 && __any_sync(0xffffffffu, grew)) {
            // (this step's scores came behind the product of SLOTS steps before, so that the parity tells)
            wait(pv_done + (g - 1) % SLOTS, (g - 1) / SLOTS & 1u);
            __syncwarp();
            tc_fence_after();
            rescale(tmem + lanes + (uint32_t)C::O_COL, std::integral_constant<int, D>{}, std::integral_constant<int, 2>{},
                    grew ? fa_ex2(before - now) : 1.f);
          }
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_ready + slot);
        }
        s_count += steps;
        // ---- the row's sum: every warpgroup's steps, against the last maximum ----
        const uint32_t last = s_count - 1;
        if (last % GROUPS != (uint32_t)wg) {
          wait(m_ready + last % GROUPS * 4 + quarter, last / GROUPS & 1u);
          __syncwarp();
          const float end = row_max[row];
          l *= m == end ? 1.f : fa_ex2(m - end);
        }
        part[x & 1][wg][row] = l;
        __syncwarp();
        // (barriers of every other run: a warpgroup may give the next run's sum before another one has looked for this run's, but not the one
        // behind it, for which that one has to have given the next)
        if (lane == 0) mbar_arrive(l_ready + (x & 1) * SW + wg * 4 + quarter);
        l = 0.f;
#pragma unroll
        for (int i = 0; i < GROUPS; ++i) {
          wait(l_ready + (x & 1) * SW + i * 4 + quarter, (uint32_t)x / 2 & 1u);
          l += part[x & 1][i][row];
        }
        __syncwarp();
      }
      // ---- out = O / l ----
      wait(o_full + i_tile, o_par);
      __syncwarp();
      o_par ^= 1u;
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      // (D = 256: 96, 96 and 64 columns)
      const int c_begin = NQ == 2 ? 0 : wg * 96, c_end = NQ == 2 ? D : min(c_begin + 96, D);
      const uint32_t o_at = tmem + lanes + (uint32_t)(C::O_COL + (NQ == 2 ? i_tile * D : 0));
      // The warp's 32 rows x 32 columns leave through shared memory: by one TMA copy where the rows are whole tokens that exist (a
      // thread's own stores of rows turned there took 4000 cycles a run of 128 columns, these 1500), by stores of full sectors otherwise.
      const uint32_t patches_at = smem_u32(patches + warp * (C::BUFS * 2048));
      const int first_row = i_tile * 128 + (warp & 3) * 32;
      const bool by_tma = a.whole_tokens && first_row + 32 <= rows;
      __nv_bfloat162 check = __float2bfloat162_rn(0.f);  // NaN once a column of the row is not finite
#pragma unroll 1
      for (int c0 = c_begin; c0 < c_end; c0 += 32 * C::BUFS) {
        uint32_t o[C::BUFS][32];
#pragma unroll
        for (int h = 0; h < C::BUFS; ++h) tmem_ld32(o_at + (uint32_t)(c0 + 32 * h), o[h]);
        tmem_ld_wait();
#pragma unroll
        for (int h = 0; h < C::BUFS; ++h) {
          const uint32_t patch = patches_at + h * 2048;
          const int c = c0 + 32 * h;
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(C::BUFS - 1) : "memory");
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint32_t w[4];
#pragma unroll
            for (int z = 0; z < 4; ++z) {
              w[z] = pack_bf16x2(__uint_as_float(o[h][8 * k + 2 * z]) * inv, __uint_as_float(o[h][8 * k + 2 * z + 1]) * inv);
              check = __hfma2(*reinterpret_cast<__nv_bfloat162*>(&w[z]), __float2bfloat162_rn(0.f), check);
            }
            // (as the copy's 64-byte swizzle)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(patch + lane * 64 + ((k ^ (lane >> 1 & 3)) << 4)), "r"(w[0]),
                         "r"(w[1]), "r"(w[2]), "r"(w[3])
                         : "memory");
          }
          if (by_tma) {
            fence_async_shared();
            __syncwarp();
            if (lane == 0) tma_store_3d(&out_map, c, r.kvh * a.G, r.row0 + (int)((uint32_t)first_row * a.inv_g >> 16), patch);
          } else {
            __syncwarp();
#pragma unroll 1
            for (int y = 0; y < 4; ++y) {
              const int rr = y * 8 + lane / 4, k = lane % 4;
              uint4 v;
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                           : "r"(patch + rr * 64 + ((k ^ (rr >> 1 & 3)) << 4)));
              const int g = first_row + rr;
              if (g < rows) {
                const int t = (int)((uint32_t)g * a.inv_g >> 16);
                bf16* dst = a.out + (long long)(r.row0 + t) * a.n_q * D + (long long)(r.kvh * a.G + g - t * a.G) * D + c + k * 8;
                if (a.vec) {
                  st_v4(dst, v);
                } else {
                  uint32_t* d4 = reinterpret_cast<uint32_t*>(dst);
                  d4[0] = v.x; d4[1] = v.y; d4[2] = v.z; d4[3] = v.w;
                }
              }
            }
            __syncwarp();
          }
          // (a group for every use of a patch, an empty one where nothing was copied: the wait above counts groups)
          if (lane == 0) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      tc_fence_before();
      __syncwarp();
      if (NQ == 1 && lane == 0) mbar_arrive(&o_read);
      // (a sum that is not finite comes from the scores, which are the row's own)
      if ((__hisnan(check.x) || __hisnan(check.y)) && l < INFINITY && i_tile * 128 + row < rows) redo = 1;
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
    both();  // (every row of the CTA has left)
    if (*(volatile int*)&redo) fa_rows_again<D, kCap, kSplit>(a, order);
  }
  __syncthreads();
  if (dead) {  // (copies in flight end before the block's memory is given back)
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000ll) {
    }
    __syncthreads();
  }
  if (warp == SW + 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// q-tiles to a block: as many as fill the query tiles; fewer where the SMs would not all get a unit (27 prompts of 10 to 31 tokens at
// D = 256, 4 kv heads: 24.6 us with full blocks, whose CTAs walk several short runs one after the other)
constexpr int FA_SMS = 148;
static int tiles_per_block(int n_tiles, int n_kv, int G, int D) {
  int n = (D > 128 ? 128 : 256) / (16 * G);
  while (n > 1 && (long long)((n_tiles + n - 1) / n) * n_kv < FA_SMS) n = (n + 1) / 2;
  return n;
}

template <int D, bool kCap, bool kSplit>
static int launch_prefill(FaArgs a, cudaStream_t st) {
  using C = FaCfg<D>;
  B200Q_CHECK_ARG(a.G <= C::MAX_G, "prefill_attn: GQA group %d too large for D=%d (max %d)", a.G, D, C::MAX_G);
  a.per_block = tiles_per_block(a.n_tiles, a.n_kv, a.G, D);
  CUtensorMap map;
  int rc = get_page_tmap(a.kv, D, &map);
  if (rc) return rc;
  if (!wait_flag(&a.failed)) {
    set_error("prefill_attn: no host-visible flag for bounded waits");
    return B200Q_ECUDA;
  }
  CUtensorMap q_map{}, out_map{};
  // (a tensor map takes rows of queries that lie one behind the other; others are read as they were before there was one)
  a.whole_tokens = a.vec && a.q_flip == 0 && 32 % a.G == 0 && a.q_stride >= a.n_q * D;
  if (a.whole_tokens) {
    rc = get_head_rows_tmap(a.out, a.n_q, D, (long long)a.n_q * D, a.G, 32 / a.G, 32, &out_map);
    if (!rc) rc = get_head_rows_tmap(a.q, a.n_q, D, a.q_stride, a.G, 128 / a.G, 64, &q_map);
    if (rc) return rc;
  }
  auto kern = prefill_attn_kernel<D, kCap, kSplit>;
  static bool attr_set = false;
  if (!attr_set) {
    B200Q_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    attr_set = true;
  }
  const int blocks = (a.n_tiles + a.per_block - 1) / a.per_block;
  const long long units = (long long)blocks * a.n_kv;
  const int grid = units < FA_SMS ? (int)units : FA_SMS;
  // Launched early where a CTA has no more than two units, or units of one step of keys.  CTAs that find their SMs as those of the kernel
  // before leave them come to lie elsewhere than the launch of an empty chip puts them, and where long units are dealt out over several
  // rounds that costs more than the start that is saved (D = 128, us, plainly / early: 12 portions of 100 to 700 tokens 56.8 / 61.3, 8 of 512
  // 47.0 / 50.5, 16 of 256 37.4 / 39.5, 4 of 300 to 1200 51.0 / 53.0; but one of 512 22.2 / 21.5, 36 of 128 32.8 / 32.5; D = 64 60 of 128
  // 44.5 / 42.7, 8 of 512 37.6 / 40.2; D = 256, 4 heads, 8 of 512 30.8 / 29.9, 40 of 50 to 200 41.0 / 43.0).  At D = 256 up to 64 blocks gain or
  // are even with any number of heads (8 heads: 16 of 256 45.9 / 45.1, 3 of 333 to 2048 88.4 / 87.2, 8 of 512 even; 6 of 300 to 600 46.8 / 48.4).
  if (units <= 2 * FA_SMS || a.bt_stride * 16 <= C::KT || (D == 256 && blocks <= 64)) {
    B200Q_CUDA(launch_early(kern, grid, C::THREADS, C::SMEM, st, 1, map, q_map, out_map, a));
    count_launch();
  } else {
    kern<<<grid, C::THREADS, C::SMEM, st>>>(map, q_map, out_map, a);
    B200Q_LAUNCH_CHECK();
  }
  return B200Q_OK;
}

// ---- which kernel -------------------------------------------------------------------------------
// Times of both kernels from a step's portions, us.  The kernel of 16-token tiles (attn.cu): the tile with most pages, or all pages and
// tiles over the SMs.  The kernel above: its longest unit, or all runs and steps over the SMs.  (The smaller of the two counts in part:
// `less`.)  Fitted to 3300 (the first kernel) and 1600 (the second) measured times: 1 to 200 portions of 2 to 3000 tokens, up to 2000 cached
// ones before them, groups of 1 to 8 heads; each kernel within 10 to 17 %.  Taking the faster one by these sums costs 0.3 to 0.4 % against
// always knowing it (at worst half as much again).  tiles / tensor memory at D = 128, 32 / 8 heads: 36 x 128 tokens 50 / 27, 16 x 128 25 / 18,
// one of 512 25 / 20, one of 2000 191 / 40, 40 behind 1500 48 / 30, but one of 200 9 / 12, 32 x 16 5 / 14, 200 x 8-40 42 / 75.
struct PromptCosts {
  double start, page, pages, pages_per_head, tile_per_head, less;
  double fa_start, fa_run, fa_step, fa_less;
};
class PromptTimes {
 public:
  PromptTimes(int n_tiles, int n_q, int n_kv, int D, int window)
      : c_(D == 64    ? PromptCosts{3.31, 0.33, 0.044, 0.041, 0.12, 0.74, 3.41, 3.29, 1.33, 0.27}
           : D == 128 ? PromptCosts{3.85, 0.49, 0.049, 0.082, 0.33, 0.58, 3.86, 4.17, 1.58, 0.25}
                      : PromptCosts{3.70, 1.19, 0.647, 0.081, 0.60, 0.44, 5.36, 5.36, 0.93, 0.33}),
        n_kv_(n_kv),
        G_(n_q / n_kv),
        window_(window),
        step_(D > 128 ? 64 : 128),
        per_(tiles_per_block(n_tiles, n_kv, n_q / n_kv, D)) {}
  void add(int n, int past) {
    if (n <= 0) return;
    const int t = (n + 15) / 16;
    // pages of the first to the last tile, one more each, no more than the window holds
    const long long a = (past + (n < 16 ? n : 16) + 15) / 16, b = a + t - 1, cap = window_ > 0 ? window_ / 16 + 2 : b;
    const long long m = b < cap ? b : cap, below = m >= a ? m - a + 1 : 0;
    pages_ += (double)(below * (a + m) / 2 + (t - below) * cap);
    if (m > most_pages_) most_pages_ = m;
    for (int at = 0; at < t;) {
      const int block = (tile_ + at) / per_, left = per_ - (tile_ + at) % per_, len = left < t - at ? left : t - at;
      const int begin = past + 16 * at, end = past + (16 * (at + len) < n ? 16 * (at + len) : n);
      const int k0 = window_ > 0 && begin + 1 > window_ ? begin + 1 - window_ : 0;
      const double us = c_.fa_run + c_.fa_step * ((end - k0 + step_ - 1) / step_);
      unit_ = block == block_ ? unit_ + us : us;
      block_ = block;
      if (unit_ > longest_) longest_ = unit_;
      all_ += us;
      at += len;
    }
    tile_ += t;
  }
  double tiles_us() const {
    return c_.start + both(c_.page * most_pages_,
                           ((c_.pages + c_.pages_per_head * G_) * pages_ + c_.tile_per_head * G_ * tile_) * n_kv_ / FA_SMS, c_.less);
  }
  double tensor_us() const { return c_.fa_start + both(longest_, all_ * n_kv_ / FA_SMS, c_.fa_less); }

 private:
  static double both(double x, double y, double less) { return x > y ? x + less * y : y + less * x; }
  PromptCosts c_;
  int n_kv_, G_, window_, step_, per_, tile_ = 0, block_ = -1;
  long long most_pages_ = 0;
  double pages_ = 0, all_ = 0, unit_ = 0, longest_ = 0;
};

// keys from which a portion alone is faster above (us, tiles / tensor memory): D = 64 one of 512 tokens 18 / 19, D = 128 one of 300 14 / 15,
// four of 300 28 / 23, D = 256 one of 128 12 / 12, one of 200 19 / 14
static int long_portion(int D) { return D == 64 ? 512 : D == 128 ? 320 : 160; }

// 0: the kernel of 16-token tiles, 1: the one above, 2: both, each for its portions (`long_keys` divides them).
// desc: the portions as {.., tokens, cached tokens before them, ..}, or NULL where the caller does not know them.  Then n_seqs is how many
// portions there are at most (0: unknown), and three steps are looked at: that many like portions without cached tokens (if they go to the
// kernel above, longer contexts do), as many behind what the block table could hold, and as few as it could hold.  If only the second or
// third would go there: where little is lost if that is wrong, the portions are taken to be as long as the table is wide (a second launch
// costs 2 to 4 us: 40 tokens behind 1500 35 us, 39 with it; 16 tokens of a table of 2048 that are all there is take 9 instead of 4);
// otherwise each portion is looked at on the GPU: the tile kernel's CTAs of long portions leave at once, the kernel above passes over the
// short ones (200 x 8-40 tokens, a table of 2048: 47 us, 82 above, 42 with a table of 64).
// B200Q_BATCH_INVARIANT=1: always the tile kernel, where a row's sums follow from its own sequence; here they depend on how the tiles of
// all portions are cut into blocks.
static int g_route = -1;  // test hook: >= 0 forces one

int prefill_attn_route(const int32_t* desc, int n_desc, int n_seqs, int n_tiles, int bt_stride, int n_q, int n_kv, int D, int window) {
  if (g_route >= 0) return g_route;
  if (batch_invariant() || n_tiles <= 0 || n_q / n_kv < 1) return 0;
  auto tensor = [](const PromptTimes& t) { return t.tensor_us() < t.tiles_us(); };
  if (desc) {
    PromptTimes t(n_tiles, n_q, n_kv, D, window);
    for (int i = 0; i < n_desc; ++i) t.add(desc[4 * i + 1], desc[4 * i + 2]);
    return tensor(t) ? 1 : 0;
  }
  const long long width = bt_stride > 0 ? 16LL * bt_stride : 16;
  const int many = n_seqs > 0 && n_seqs < n_tiles ? n_seqs : n_tiles;
  auto even = [&](int k, bool cached) {  // the tiles in k like portions
    PromptTimes t(n_tiles, n_q, n_kv, D, window);
    for (int i = 0; i < k; ++i) {
      const long long n = 16 * (n_tiles * (i + 1LL) / k - n_tiles * (long long)i / k);
      t.add((int)n, cached && width > n ? (int)(width - n) : 0);
    }
    return t;
  };
  const PromptTimes none = even(many, false);
  if (tensor(none)) return 1;
  if (2 * width < 3 * long_portion(D)) return 0;  // (near the line there is nothing to gain)
  const bool full = tensor(even(many, true));
  // (a table four times as wide as the portions are on average holds other sequences too, or a few of the portions are long)
  if (!full && !(width * many >= 64LL * n_tiles && tensor(even((int)((16LL * n_tiles + width - 1) / width), false)))) return 0;
  return full && none.tensor_us() < none.tiles_us() + 6 ? 1 : 2;
}

int prefill_attn(int route, const void* q, int q_stride, void* out, const void* kv_layer, const int32_t* block_table, int bt_stride,
                 const int32_t* tiles, int n_tiles, int n_q, int n_kv, int D, int block_size, float scale, float softcap, int window,
                 cudaStream_t st) {
  B200Q_CHECK_ARG(n_tiles >= 0 && n_kv > 0 && n_q % n_kv == 0 && n_q / n_kv <= 8,
                  "prefill_attn: unsupported heads n_q=%d n_kv=%d (GQA group must be <= 8)", n_q, n_kv);
  B200Q_CHECK_ARG(block_size == 16 && (D == 64 || D == 128 || D == 256),
                  "prefill_attn: unsupported D=%d block_size=%d (D in {64,128,256}, block 16)", D, block_size);
  if (n_tiles == 0 || n_q == 0) return B200Q_OK;
  const int long_keys = route == 2 ? long_portion(D) : 0;
  if (route != 1) {
    const int rc = prefill_tiles(q, q_stride, out, kv_layer, block_table, bt_stride, tiles, n_tiles, n_q, n_kv, D, scale, softcap, window,
                                 long_keys, st);
    if (rc || route == 0) return rc;
  }
  const float log2e = 1.4426950408889634f;
  FaArgs a{};
  a.q = (const bf16*)q;
  a.out = (bf16*)out;
  a.kv = (const uint8_t*)kv_layer;
  a.block_table = block_table;
  a.tiles = (const int4*)tiles;
  a.q_stride = q_stride;
  a.bt_stride = bt_stride;
  a.n_tiles = n_tiles;
  a.n_q = n_q;
  a.n_kv = n_kv;
  a.G = n_q / n_kv;
  a.window = window;
  a.long_keys = long_keys;
  a.q_flip = scale < 0.f ? 0x80008000u : 0u;
  const float s = scale < 0.f ? -scale : scale;
  a.c0 = softcap > 0.f ? s / softcap : s * log2e;
  a.inv_g = 65536u / (uint32_t)a.G + 1u;
  if (!(a.c0 > 1e-37f)) a.c0 = a.c0 >= 0.f ? 1e-37f : a.c0;  // (0: all scores equal; times a hidden key's -inf it would be NaN)
  a.c1 = softcap * log2e;
  a.vec = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) == 0 && q_stride % 8 == 0;
  auto launch = [&](auto cap) {
    constexpr bool c = decltype(cap)::value;
    if (D == 64) return long_keys ? launch_prefill<64, c, true>(a, st) : launch_prefill<64, c, false>(a, st);
    if (D == 128) return long_keys ? launch_prefill<128, c, true>(a, st) : launch_prefill<128, c, false>(a, st);
    return long_keys ? launch_prefill<256, c, true>(a, st) : launch_prefill<256, c, false>(a, st);
  };
  return softcap > 0.f ? launch(std::true_type{}) : launch(std::false_type{});
}

}  // namespace b200q

using namespace b200q;

extern "C" {

int b200q_prefill_attn_seqs(const void* q, int q_stride, void* out, const void* kv_layer, const int32_t* block_table, int bt_stride,
                            int n_seqs, const int32_t* tiles, int n_tiles, int n_q, int n_kv, int D, int block_size, float scale,
                            float softcap, int window, void* stream) {
  const int route = n_kv > 0 && n_q >= n_kv ? prefill_attn_route(nullptr, 0, n_seqs, n_tiles, bt_stride, n_q, n_kv, D, window) : 0;
  return prefill_attn(route, q, q_stride, out, kv_layer, block_table, bt_stride, tiles, n_tiles, n_q, n_kv, D, block_size, scale, softcap,
                      window, as_stream(stream));
}

int b200q_prefill_attn_ex(const void* q, int q_stride, void* out, const void* kv_layer, const int32_t* block_table, int bt_stride,
                          const int32_t* tiles, int n_tiles, int n_q, int n_kv, int D, int block_size, float scale, float softcap,
                          int window, void* stream) {
  return b200q_prefill_attn_seqs(q, q_stride, out, kv_layer, block_table, bt_stride, 0, tiles, n_tiles, n_q, n_kv, D, block_size, scale,
                                 softcap, window, stream);
}

int b200q_prefill_attn(const void* q, int q_stride, void* out, const void* kv_layer, const int32_t* block_table, int bt_stride,
                       const int32_t* tiles, int n_tiles, int n_q, int n_kv, int D, int block_size, float scale, void* stream) {
  return b200q_prefill_attn_seqs(q, q_stride, out, kv_layer, block_table, bt_stride, 0, tiles, n_tiles, n_q, n_kv, D, block_size, scale,
                                 0.f, 0, stream);
}

// test hooks: one route for all calls (-1: choose)
int b200q_prefill_attn_set_route(int route) {
  B200Q_CHECK_ARG(route >= -1 && route <= 2, "prefill route must be -1..2");
  g_route = route;
  bump_tuning_epoch();
  return B200Q_OK;
}

// the route of a step (prefill_attn_route; desc is host memory, [n_desc][4], or NULL)
int b200q_prefill_attn_route(const int32_t* desc, int n_desc, int n_seqs, int n_tiles, int bt_stride, int n_q, int n_kv, int D,
                             int window) {
  return prefill_attn_route(desc, n_desc, n_seqs, n_tiles, bt_stride, n_q, n_kv, D, window);
}

}  // extern "C"
