// elementwise.cu — the HBM-bound, coalesced, 16-byte-vectorised kernels of the hot path:
// embedding gather (K1), RMSNorm / fused add+RMSNorm (K2), RoPE + paged KV write (K4+K5),
// SwiGLU (K10), row gather and greedy argmax (K13), in place of vLLM's ops.  All rounding points follow the oracle (oracle/ops.py), which follows
// vLLM's native op definitions / HF transformers' Llama.
#include <limits.h>
#include <stdarg.h>

#include <type_traits>

#include "tcgen05.cuh"

namespace b200q {

thread_local char g_err[512] = {0};
static long long g_launches = 0;

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}
void count_launch(int n) { __atomic_fetch_add(&g_launches, (long long)n, __ATOMIC_RELAXED); }
static int g_epoch = 0;
void bump_tuning_epoch() { __atomic_fetch_add(&g_epoch, 1, __ATOMIC_RELAXED); }
int tuning_epoch() { return __atomic_load_n(&g_epoch, __ATOMIC_RELAXED); }

// ------------------------------------------------------------------------------------------
// K1 embedding gather.  One warp per 512 B (32 lanes x 16 B); grid-stride over (token, chunk).
// ------------------------------------------------------------------------------------------
// A negative id is an indirection into `prev_out`, the sampled ids of the PREVIOUS forward step
// (id = prev_out[-1 - ids[t]]): the engine enqueues step k+1 before it has read step k's tokens
// back, so a decode row's input token is still on the device (engine.cu, async stepping).
__device__ __forceinline__ int resolve_token(const int32_t* __restrict__ ids,
                                             const int32_t* __restrict__ prev_out, int t) {
  int id = ids[t];
  if (id < 0) id = prev_out[-1 - id];  // plain load: written by the previous step's sampler
  return id;
}

__global__ void __launch_bounds__(256) embed_kernel(const int32_t* __restrict__ ids,
                                                    const int32_t* __restrict__ prev_out,
                                                    const uint4* __restrict__ table,
                                                    uint4* __restrict__ out, int T, int chunks) {
  follow_previous(ids, prev_out, table, out);
  long long total = (long long)T * chunks;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    int t = (int)(i / chunks), c = (int)(i % chunks);
    int id = resolve_token(ids, prev_out, t);
    out[i] = ld_once_v4(table + (long long)id * chunks + c);
  }
}

// Gemma: out = bf16(table[id] * scale) (the normaliser sqrt(H), itself rounded to bf16 by the host)
__global__ void __launch_bounds__(256) embed_scaled_kernel(const int32_t* __restrict__ ids,
                                                           const int32_t* __restrict__ prev_out,
                                                           const uint4* __restrict__ table,
                                                           uint4* __restrict__ out, int T, int chunks,
                                                           float scale) {
  follow_previous(ids, prev_out, table, out);
  long long total = (long long)T * chunks;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    int t = (int)(i / chunks), c = (int)(i % chunks);
    int id = resolve_token(ids, prev_out, t);
    uint4 a = ld_once_v4(table + (long long)id * chunks + c);
    uint32_t* ap = reinterpret_cast<uint32_t*>(&a);
#pragma unroll
    for (int k = 0; k < 4; ++k) ap[k] = pack_bf16x2(bf16_lo(ap[k]) * scale, bf16_hi(ap[k]) * scale);
    out[i] = a;
  }
}

// ------------------------------------------------------------------------------------------
// K2 RMSNorm / fused add + RMSNorm.  One 256-thread CTA per token row; the row lives in
// registers between the reduction and the scale (one HBM read, one write per tensor).
// ------------------------------------------------------------------------------------------
constexpr int NORM_THREADS = 256;
constexpr int NORM_MAX_CHUNKS = 4;  // H <= 256*4*8 = 8192
// The kernels are made for 1, 2 and 4 chunks of a row per thread, and a thread asks for two or more of them, and of their weights, before it
// stores the first: pointers that went through follow_previous are not known to lie apart, so that the compiler leaves every load behind
// the store ahead of it.  us, add + norm before kernels began early / with the loads as the compiler left them / now: 48 rows of 8192
// 4.0 / 4.3 / 3.1, 750 of 8192 6.8 / 8.7 / 6.6, 750 of 4096 4.5 / 5.0 / 4.1, 4608 of 2048 10.0 / 9.7 / 9.4.  Registers decide the rest: a
// kernel for four chunks whatever the width takes 11.0 for the last of these, norms alone with all four weights of a thread at once 32.9
// instead of 28.2 for 4608 rows of 8192.
template <typename F>
static int norm_chunks(int H, F&& launch) {
  const int n = (H / 8 + NORM_THREADS - 1) / NORM_THREADS;
  return n <= 1 ? launch(std::integral_constant<int, 1>{}) : n == 2 ? launch(std::integral_constant<int, 2>{})
                                                                    : launch(std::integral_constant<int, NORM_MAX_CHUNKS>{});
}

// C pieces of 8 consecutive outputs of a split-K GEMM, from off[i] on: the fp32 partials ws[s][row][col] added in split order (the same order
// and rounding as the stand-alone reduction) and rounded to bf16.  These kernels are chains of reads from L2: AT_ONCE parts of every piece
// are asked for before the first is added.  More than the callers' 4 or 2 x 2 take registers that longer rows or fuller SMs want back.
// 48 rows of 4 parts, us, part after part / so: a norm of 4096 3.6 / 3.2; of 2048 2.7 / 2.5; with 8 parts 4.4 / 4.2.
template <int C, int AT_ONCE>
__device__ __forceinline__ void sum_partials_bf16(const float* ws, const long long (&off)[C], long long mn, int splits, uint4 (&out)[C]) {
  float4 a[C][2];
  for (int s0 = 0; s0 < splits; s0 += AT_ONCE) {
    float4 p[C][AT_ONCE][2];
#pragma unroll
    for (int i = 0; i < C; ++i)
#pragma unroll
      for (int x = 0; x < AT_ONCE; ++x)
        if (s0 + x < splits) {
          p[i][x][0] = *reinterpret_cast<const float4*>(ws + (s0 + x) * mn + off[i]);
          p[i][x][1] = *reinterpret_cast<const float4*>(ws + (s0 + x) * mn + off[i] + 4);
        }
#pragma unroll
    for (int i = 0; i < C; ++i)
#pragma unroll
      for (int x = 0; x < AT_ONCE; ++x)
        if (s0 + x < splits) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 c = p[i][x][h];
            if (s0 + x == 0) {
              a[i][h] = c;
            } else {
              a[i][h].x += c.x; a[i][h].y += c.y; a[i][h].z += c.z; a[i][h].w += c.w;
            }
          }
        }
  }
#pragma unroll
  for (int i = 0; i < C; ++i)
    out[i] = make_uint4(pack_bf16x2(a[i][0].x, a[i][0].y), pack_bf16x2(a[i][0].z, a[i][0].w), pack_bf16x2(a[i][1].x, a[i][1].y),
                        pack_bf16x2(a[i][1].z, a[i][1].w));
}

// kPartials: x is not read from x_in but reduced on the fly from the fp32 partials of a split-K GEMM
// (up to 768 rows): the projection's reduce pass, the residual add and the norm become ONE
// launch instead of two, and the bf16 GEMM output never makes a round trip through memory.
template <int CH, bool kAdd, bool kPartials = false>
__global__ void __launch_bounds__(NORM_THREADS)
    rmsnorm_kernel(const uint4* __restrict__ x_in, uint4* __restrict__ residual,
                   const uint4* __restrict__ w, uint4* __restrict__ y, int chunks, float inv_h,
                   float eps, const float* __restrict__ ws, int splits, long long mn) {
  follow_previous(x_in, residual, w, y, ws);
  const long long row = blockIdx.x;
  const uint4* xr = x_in + row * chunks;
  // (sums of parts: what does not wait for them is asked for first; otherwise the residual's chunks go two at a time behind the row's)
  uint4 v[CH], res[kPartials ? CH : 2], weight[CH];
  float ss = 0.f;
  if constexpr (kPartials) {
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      const int c = threadIdx.x + j * NORM_THREADS;
      if (c < chunks) {
        if (kAdd) res[j] = ld_v4(residual + row * chunks + c);
        weight[j] = ld_v4(w + c);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < CH; ++j) {
    int c = threadIdx.x + j * NORM_THREADS;
    if (c < chunks) {
      if constexpr (kPartials) {
        const long long off[1] = {(row * chunks + c) * 8};
        uint4 sum[1];
        sum_partials_bf16<1, 4>(ws, off, mn, splits, sum);
        v[j] = sum[0];
      } else {
        v[j] = ld_v4(xr + c);
        weight[j] = ld_v4(w + c);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < CH; ++j) {
    int c = threadIdx.x + j * NORM_THREADS;
    if (kAdd && !kPartials && j % 2 == 0) {
#pragma unroll
      for (int i = 0; i < 2 && j + i < CH; ++i)
        if (c + i * NORM_THREADS < chunks) res[i] = ld_v4(residual + row * chunks + c + i * NORM_THREADS);
    }
    if (c < chunks) {
      uint4 a = v[j];
      if (kAdd) {
        uint4 r = res[kPartials ? j : j % 2];
        uint32_t* ap = reinterpret_cast<uint32_t*>(&a);
        const uint32_t* rp = reinterpret_cast<const uint32_t*>(&r);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float lo = bf16_lo(ap[k]) + bf16_lo(rp[k]);
          float hi = bf16_hi(ap[k]) + bf16_hi(rp[k]);
          ap[k] = pack_bf16x2(lo, hi);  // residual stream is kept in bf16 (rounded sum)
        }
        st_v4(residual + row * chunks + c, a);
      }
      v[j] = a;
      const uint32_t* ap = reinterpret_cast<const uint32_t*>(&a);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float lo = bf16_lo(ap[k]), hi = bf16_hi(ap[k]);
        ss += lo * lo + hi * hi;
      }
    }
  }
  __shared__ float red[NORM_THREADS / 32];
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < NORM_THREADS / 32; ++i) tot += red[i];
  const float inv = __frsqrt_rn(tot * inv_h + eps);
#pragma unroll
  for (int j = 0; j < CH; ++j) {
    int c = threadIdx.x + j * NORM_THREADS;
    if (c < chunks) {
      uint4 a = v[j];
      uint4 ww = weight[j];
      uint32_t* ap = reinterpret_cast<uint32_t*>(&a);
      const uint32_t* wp = reinterpret_cast<const uint32_t*>(&ww);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // y = bf16( bf16(x * inv) * w )  — the normalised value is rounded to the weight
        // dtype before the weight multiply (vllm/ir/ops/layernorm.py:19-20)
        float lo = round_bf16(bf16_lo(ap[k]) * inv) * bf16_lo(wp[k]);
        float hi = round_bf16(bf16_hi(ap[k]) * inv) * bf16_hi(wp[k]);
        ap[k] = pack_bf16x2(lo, hi);
      }
      st_v4(y + row * chunks + c, a);
    }
  }
}

// ------------------------------------------------------------------------------------------
// Gemma-2 norms.  GemmaRMSNorm multiplies by (1 + w) and rounds ONCE:
//   y = bf16( (x * rsqrt(mean(x^2) + eps)) * (1 + w) )      all in fp32 until the final cast.
// gemma_norm_add_norm fuses the sandwich around a residual add (two row reductions, the row
// stays in registers):  a = norm(x, w_post);  residual = bf16(residual + a);  x = norm(residual, w_next)
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ float block_sum_256(float v, float* red) {
  v = warp_sum(v);
  __syncthreads();  // red may still be read by the previous reduction
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float tot = 0.f;
#pragma unroll
  for (int i = 0; i < NORM_THREADS / 32; ++i) tot += red[i];
  return tot;
}

__device__ __forceinline__ float chunk_sumsq(const uint4& a) {
  const uint32_t* ap = reinterpret_cast<const uint32_t*>(&a);
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float lo = bf16_lo(ap[k]), hi = bf16_hi(ap[k]);
    ss += lo * lo + hi * hi;
  }
  return ss;
}

// a <- bf16((a * inv) * (1 + w))
__device__ __forceinline__ void gemma_scale_chunk(uint4& a, const uint4& ww, float inv) {
  uint32_t* ap = reinterpret_cast<uint32_t*>(&a);
  const uint32_t* wp = reinterpret_cast<const uint32_t*>(&ww);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float lo = (bf16_lo(ap[k]) * inv) * (1.f + bf16_lo(wp[k]));
    float hi = (bf16_hi(ap[k]) * inv) * (1.f + bf16_hi(wp[k]));
    ap[k] = pack_bf16x2(lo, hi);
  }
}

template <int CH, bool kSandwich>
__global__ void __launch_bounds__(NORM_THREADS)
    gemma_norm_kernel(const uint4* __restrict__ x_in, uint4* __restrict__ residual,
                      const uint4* __restrict__ w_post, const uint4* __restrict__ w_next,
                      uint4* __restrict__ y, int chunks, float inv_h, float eps) {
  __shared__ float red[NORM_THREADS / 32];
  follow_previous(x_in, residual, w_post, w_next, y);
  const long long row = blockIdx.x;
  const uint4* xr = x_in + row * chunks;
  uint4 v[CH], res[2], weight[2];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < CH; ++j) {
    int c = threadIdx.x + j * NORM_THREADS;
    if (c < chunks) {
      v[j] = ld_v4(xr + c);
      ss += chunk_sumsq(v[j]);
    }
  }
  float inv = __frsqrt_rn(block_sum_256(ss, red) * inv_h + eps);
  if (kSandwich) {
    // a = norm(x, w_post); residual <- bf16(residual + a); then the second norm over the new residual
    ss = 0.f;
#pragma unroll
    for (int j = 0; j < CH; ++j) {
      int c = threadIdx.x + j * NORM_THREADS;
      if (j % 2 == 0) {
#pragma unroll
        for (int i = 0; i < 2 && j + i < CH; ++i)
          if (c + i * NORM_THREADS < chunks) {
            weight[i] = ld_v4(w_post + c + i * NORM_THREADS);
            res[i] = ld_v4(residual + row * chunks + c + i * NORM_THREADS);
          }
      }
      if (c < chunks) {
        uint4 a = v[j];
        gemma_scale_chunk(a, weight[j % 2], inv);
        uint4 r = res[j % 2];
        uint32_t* ap = reinterpret_cast<uint32_t*>(&a);
        const uint32_t* rp = reinterpret_cast<const uint32_t*>(&r);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          ap[k] = pack_bf16x2(bf16_lo(rp[k]) + bf16_lo(ap[k]), bf16_hi(rp[k]) + bf16_hi(ap[k]));
        st_v4(residual + row * chunks + c, a);
        v[j] = a;
        ss += chunk_sumsq(a);
      }
    }
    inv = __frsqrt_rn(block_sum_256(ss, red) * inv_h + eps);
  }
  const uint4* w_out = kSandwich ? w_next : w_post;
#pragma unroll
  for (int j = 0; j < CH; ++j) {
    int c = threadIdx.x + j * NORM_THREADS;
    if (j % 2 == 0) {
#pragma unroll
      for (int i = 0; i < 2 && j + i < CH; ++i)
        if (c + i * NORM_THREADS < chunks) weight[i] = ld_v4(w_out + c + i * NORM_THREADS);
    }
    if (c < chunks) {
      uint4 a = v[j];
      gemma_scale_chunk(a, weight[j % 2], inv);
      st_v4(y + row * chunks + c, a);
    }
  }
}

// final-logit soft-capping with every eager bf16 rounding: l <- bf16(bf16(tanh(bf16(l / cap))) * cap)
__global__ void __launch_bounds__(256)
    softcap_kernel(uint4* __restrict__ logits, long long n_chunks, float cap) {
  follow_previous(logits);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_chunks;
       i += (long long)gridDim.x * blockDim.x) {
    uint4 a = ld_v4(logits + i);
    uint32_t* ap = reinterpret_cast<uint32_t*>(&a);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float lo = round_bf16(tanhf(round_bf16(__fdiv_rn(bf16_lo(ap[k]), cap)))) * cap;
      float hi = round_bf16(tanhf(round_bf16(__fdiv_rn(bf16_hi(ap[k]), cap)))) * cap;
      ap[k] = pack_bf16x2(lo, hi);
    }
    st_v4(logits + i, a);
  }
}

// ------------------------------------------------------------------------------------------
// K4+K5 RoPE (neox pairs i, i+D/2) on q and k, and the paged KV write.
// One CTA per token.  Work items: q heads x (D/16) chunk-pairs (in place), k heads x (D/16)
// chunk-pairs (rotated, written to the cache only), v heads x (D/8) chunks (copied to the cache).
// Cache rows are [token][D] with 16 B chunk c stored at chunk (c ^ (token_in_block & 7)) so
// that the attention kernels' ldmatrix reads of TMA-copied pages are bank-conflict free.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void rope_chunk_pair(uint4& x1, uint4& x2, const uint4& cs,
                                                const uint4& sn) {
  uint32_t* a = reinterpret_cast<uint32_t*>(&x1);
  uint32_t* b = reinterpret_cast<uint32_t*>(&x2);
  const uint32_t* c = reinterpret_cast<const uint32_t*>(&cs);
  const uint32_t* s = reinterpret_cast<const uint32_t*>(&sn);
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    // bf16 arithmetic with a rounding after every op, as HF / vLLM eager do on bf16 tensors:
    // o1 = x1*cos - x2*sin ; o2 = x2*cos + x1*sin
    float x1l = bf16_lo(a[k]), x1h = bf16_hi(a[k]);
    float x2l = bf16_lo(b[k]), x2h = bf16_hi(b[k]);
    float cl = bf16_lo(c[k]), ch = bf16_hi(c[k]);
    float sl = bf16_lo(s[k]), sh = bf16_hi(s[k]);
    float o1l = round_bf16(x1l * cl) - round_bf16(x2l * sl);
    float o1h = round_bf16(x1h * ch) - round_bf16(x2h * sh);
    float o2l = round_bf16(x2l * cl) + round_bf16(x1l * sl);
    float o2h = round_bf16(x2h * ch) + round_bf16(x1h * sh);
    a[k] = pack_bf16x2(o1l, o1h);
    b[k] = pack_bf16x2(o2l, o2h);
  }
}

// kPartials: the qkv row is reduced on the fly from the fp32 partials of the split-K qkv projection
// (up to 768 rows) instead of being read back as bf16 — reduce + RoPE + KV write in one launch
template <bool kPartials>
__global__ void __launch_bounds__(kPartials ? 128 : 256)
    rope_kvwrite_kernel(uint4* __restrict__ qkv, const uint4* __restrict__ cos_sin,
                        const int32_t* __restrict__ positions,
                        const int32_t* __restrict__ slot_mapping, uint4* __restrict__ kv_layer,
                        int n_q, int n_kv, int D, int block_size, const float* __restrict__ ws,
                        int splits, long long mn) {
  follow_previous(qkv, cos_sin, positions, slot_mapping, kv_layer, ws);
  const int t = blockIdx.x;
  const int cpr = D / 8;        // 16 B chunks per head row
  const int half = cpr / 2;     // chunk pairs per head
  const int row_chunks = (n_q + 2 * n_kv) * cpr;
  uint4* row = qkv + (long long)t * row_chunks;
  const int pos = positions[t];
  const int slot = slot_mapping[t];
  const uint4* cs_row = cos_sin + (long long)pos * cpr;  // [cos (D/2) | sin (D/2)]
  const int blk = slot >= 0 ? slot / block_size : 0;
  const int off = slot >= 0 ? slot % block_size : 0;
  const int n_rope_items = (n_q + n_kv) * half;
  const int n_items = n_rope_items + n_kv * cpr;
  for (int it = blockIdx.y * blockDim.x + threadIdx.x; it < n_items; it += gridDim.y * blockDim.x) {
    if (it < n_rope_items) {
      int head = it / half, c = it % half;
      uint4 x1, x2;
      uint4 cs = ld_v4(cs_row + c);
      uint4 sn = ld_v4(cs_row + half + c);
      if constexpr (kPartials) {
        const long long e = ((long long)t * row_chunks + head * cpr + c) * 8, off2[2] = {e, e + (long long)half * 8};
        uint4 x[2];
        sum_partials_bf16<2, 2>(ws, off2, mn, splits, x);
        x1 = x[0];
        x2 = x[1];
      } else {
        x1 = ld_v4(row + head * cpr + c);
        x2 = ld_v4(row + head * cpr + c + half);
      }
      rope_chunk_pair(x1, x2, cs, sn);
      if (head < n_q) {
        st_v4(row + head * cpr + c, x1);
        st_v4(row + head * cpr + c + half, x2);
      } else if (slot >= 0) {
        int h = head - n_q;
        uint4* dst =
            kv_layer + ((((long long)blk * 2 + 0) * n_kv + h) * block_size + off) * cpr;
        int sw = off & 7;
        st_v4(dst + (c ^ sw), x1);
        st_v4(dst + ((c + half) ^ sw), x2);
      }
    } else if (slot >= 0) {
      int j = it - n_rope_items;
      int h = j / cpr, c = j % cpr;
      uint4 v;
      if constexpr (kPartials) {
        const long long off1[1] = {((long long)t * row_chunks + (n_q + n_kv + h) * cpr + c) * 8};
        uint4 sum[1];
        sum_partials_bf16<1, 4>(ws, off1, mn, splits, sum);
        v = sum[0];
      } else
        v = ld_v4(row + (n_q + n_kv + h) * cpr + c);
      uint4* dst = kv_layer + ((((long long)blk * 2 + 1) * n_kv + h) * block_size + off) * cpr;
      st_v4(dst + (c ^ (off & 7)), v);
    }
  }
}

// ------------------------------------------------------------------------------------------
// K10 SwiGLU.  grid-stride over 16 B chunks of the output.
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    swiglu_kernel(const uint4* __restrict__ gate_up, uint4* __restrict__ out, int T, int ichunks) {
  follow_previous(gate_up, out);
  long long total = (long long)T * ichunks;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    long long t = i / ichunks;
    int c = (int)(i % ichunks);
    uint4 g = ld_once_v4(gate_up + t * 2 * ichunks + c);
    uint4 u = ld_once_v4(gate_up + t * 2 * ichunks + ichunks + c);
    uint32_t* gp = reinterpret_cast<uint32_t*>(&g);
    const uint32_t* up = reinterpret_cast<const uint32_t*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float gl = bf16_lo(gp[k]), gh = bf16_hi(gp[k]);
      // silu rounded to bf16, then the product rounded to bf16 (two bf16 ops, as eager torch)
      float sl = round_bf16(gl / (1.f + __expf(-gl)));
      float sh = round_bf16(gh / (1.f + __expf(-gh)));
      gp[k] = pack_bf16x2(sl * bf16_lo(up[k]), sh * bf16_hi(up[k]));
    }
    out[i] = g;
  }
}

__global__ void __launch_bounds__(256)
    gather_rows_kernel(const uint4* __restrict__ x, const int32_t* __restrict__ rows,
                       uint4* __restrict__ out, int n, int chunks) {
  follow_previous(x, rows, out);
  long long total = (long long)n * chunks;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    int r = (int)(i / chunks), c = (int)(i % chunks);
    out[i] = ld_v4(x + (long long)rows[r] * chunks + c);
  }
}

// ------------------------------------------------------------------------------------------
// K13 greedy argmax over bf16 logits; lowest index wins ties (torch.argmax behaviour).
// A cluster of gridDim.x CTAs shares a row, four 16-byte loads in flight per thread (48 rows of 128256 logits: 15.3 us with the end of the
// step, 9.7 so).  V need not be a multiple of 8 (tail handled scalar).
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void amax_update(float v, int i, float& best, int& bi) {
  if (v > best || (v == best && i < bi)) {
    best = v;
    bi = i;
  }
}

// the largest of the block's threads and then of the cluster's CTAs; thread 0 of CTA 0 returns with it
template <int THREADS>
__device__ __forceinline__ void amax_cluster(float& best, int& bi) {
  const int split = blockIdx.x, splits = gridDim.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float ov = __shfl_xor_sync(0xffffffffu, best, o);
    int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    amax_update(ov, oi, best, bi);
  }
  __shared__ float sv[THREADS / 32];
  __shared__ int si[THREADS / 32];
  if ((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = best;
    si[threadIdx.x >> 5] = bi;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    best = threadIdx.x < THREADS / 32 ? sv[threadIdx.x] : -INFINITY;
    bi = threadIdx.x < THREADS / 32 ? si[threadIdx.x] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, best, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      amax_update(ov, oi, best, bi);
    }
    if (threadIdx.x == 0) {
      sv[0] = best;
      si[0] = bi;
    }
  }
  if (splits > 1) {
    cluster_sync_all();
    if (split == 0 && threadIdx.x == 0)
      for (int s = 1; s < splits; ++s)
        amax_update(ld_cluster_f32(mapa_shared(sv, s)), __float_as_int(ld_cluster_f32(mapa_shared(si, s))), best, bi);
    cluster_sync_all();
  }
}

constexpr int ARGMAX_THREADS = 512;
__global__ void __launch_bounds__(ARGMAX_THREADS)
    argmax_kernel(const bf16* __restrict__ logits, int32_t* __restrict__ ids, int V) {
  follow_previous(logits, ids);
  const int split = blockIdx.x, r_ = blockIdx.y;
  const bf16* row = logits + (long long)r_ * V;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  const int nvec = ((reinterpret_cast<uintptr_t>(row) & 15) == 0) ? V / 8 : 0;
  const uint4* rv = reinterpret_cast<const uint4*>(row);
  const int step = gridDim.x * ARGMAX_THREADS, first = split * ARGMAX_THREADS + threadIdx.x;
  for (int c0 = first; c0 < nvec; c0 += 4 * step) {
    uint4 a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + u * step < nvec) a[u] = ld_once_v4(rv + c0 + u * step);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c0 + u * step < nvec) {
        const uint32_t* ap = reinterpret_cast<const uint32_t*>(&a[u]);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          amax_update(bf16_lo(ap[k]), (c0 + u * step) * 8 + 2 * k, best, bi);
          amax_update(bf16_hi(ap[k]), (c0 + u * step) * 8 + 2 * k + 1, best, bi);
        }
      }
  }
  for (int i = nvec * 8 + first; i < V; i += step) amax_update(__bfloat162float(row[i]), i, best, bi);
  amax_cluster<ARGMAX_THREADS>(best, bi);
  if (split == 0 && threadIdx.x == 0) ids[r_] = bi == 0x7fffffff ? 0 : bi;
}

// ------------------------------------------------------------------------------------------
// K13 sampler at temperature > 0: the reference's default path (SamplingParams(temperature=0.7),
// ref:llmq/workers/vllm_worker.py:161-165; vLLM: probs = softmax(logits/T); probs.div_(q).argmax
// with q ~ Exp(1), vllm/v1/sample/ops/topk_topp_sampler.py:395-416).  argmax_i p_i/q_i ==
// argmax_i (logit_i/T - log q_i), so no softmax pass is needed: one read of the bf16 logits row.
// q_i = -log(u_i), u_i from Philox4x32-10 keyed by the request's seed with counter
// (element index / 4, token position) — counter-based, so a request's samples do not depend on
// its batch-mates.  temperature == 0 rows fall back to the greedy argmax (lowest index on ties).
// params: int32[B][4] = {float bits of temperature, seed lo, seed hi, position}.
// ------------------------------------------------------------------------------------------
// counter (c0, c1, 0, 0); k0, k1: the key of every round
__device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, const uint32_t (&k0)[10], const uint32_t (&k1)[10], uint32_t (&out)[4]) {
  uint32_t c2 = 0, c3 = 0;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = (uint64_t)0xD2511F53u * c0, p1 = (uint64_t)0xCD9E8D57u * c2;
    c0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0[r];
    c1 = (uint32_t)p1;
    c2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1[r];
    c3 = (uint32_t)p0;
  }
  out[0] = c0;
  out[1] = c1;
  out[2] = c2;
  out[3] = c3;
}

// -log(-log u), u = (n + 1/2) / 2^24 with n = the upper 24 bits.  n + 1/2 takes 25 bits from 2^23 on and rounds half a step up or down (to
// u = 1 for the largest n, whose noise is 17.3 and not infinite): what was rounded off, d = +-2^-25, comes back as log u = log u' + d / u',
// 1 / u' = 2 - u' being near enough (off by 1.5e-8 of 0.69 at u' = 1/2).  Below 2^23, d = 0.
__device__ __forceinline__ float gumbel_from_bits(uint32_t x) {
  const float n = (float)(x >> 8), n5 = n + 0.5f, u = n5 * (1.0f / 16777216.0f);
  const float d = ((n - n5) + 0.5f) * (1.0f / 16777216.0f);
  return -logf(-fmaf(d, 2.f - u, logf(u)));
}

// A cluster of gridDim.x CTAs shares a row.  Bound: integer work of the random numbers.  The two logarithms of a logit's noise are taken
// only where the logit could still win: its value t + noise exceeds the best so far only if -log u < e^(t - best), and -log u >= 1 - u,
// which the bits give directly; four logits (one block of random numbers) are looked at together, by the largest t and the largest u among
// them.  The margin covers the roundings of t, best and the exponential (|best| * 1e-6 + 1.5e-3 in base 2, some ten times what they are),
// so what is left out is smaller than the best, and the result is the one that all logarithms give.  The best so far is the CTA's, in
// shared memory: a warp sees a few thousand logits only, and would take logarithms for a third of them on its own.  128 rows of 128256
// logits 35 -> 25 us, 1024 rows 181 -> 133 (issue slots 58 % busy, half of them the random numbers).  Two CTAs per SM:
// with three, which leave 40 registers to a thread, 28 and 142.  Rows of temperature 0:
// 48 / 128 / 300 / 1024 of them 6.4 / 10.0 / 22 / 69 us (8.6 / 14.7 / 30 / 92 before).
constexpr int SAMPLE_THREADS = 512;
__device__ __forceinline__ int order_float(float v) {  // integers of the same order
  const int o = __float_as_int(v);
  return o ^ ((o >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float unorder_float(int o) { return __int_as_float(o ^ ((o >> 31) & 0x7fffffff)); }

__global__ void __launch_bounds__(SAMPLE_THREADS, 2)
    sample_kernel(const bf16* __restrict__ logits, const int32_t* __restrict__ params,
                  int32_t* __restrict__ ids, int V) {
  __shared__ int top_s;  // the CTA's best so far, through order_float
  if (threadIdx.x == 0) top_s = INT_MIN;
  __syncthreads();
  follow_previous(logits, params, ids);
  const int split = blockIdx.x, splits = gridDim.x, r_ = blockIdx.y;
  const bf16* row = logits + (long long)r_ * V;
  const float temp = __int_as_float(params[4 * r_ + 0]);
  // (the round keys are kept: 1024 rows 132.6 us, 133.4 with keys made again for every block; 128 rows 24.6 either way)
  uint32_t k0[10], k1[10];
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    k0[i] = (uint32_t)params[4 * r_ + 1] + (uint32_t)i * 0x9E3779B9u;
    k1[i] = (uint32_t)params[4 * r_ + 2] + (uint32_t)i * 0xBB67AE85u;
    asm volatile("" : "+r"(k0[i]), "+r"(k1[i]));
  }
  const uint32_t pos = (uint32_t)params[4 * r_ + 3];
  const bool greedy = !(temp > 0.f);
  const float inv_t = greedy ? 1.f : 1.f / temp;
  const float log2e = 1.4426950408889634f;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  // groups of 4 consecutive elements share one Philox block: counter = (group, position, 0, 0)
  constexpr int AT_ONCE = 2;
  const int n4 = V / 4, step = splits * SAMPLE_THREADS, first = split * SAMPLE_THREADS + threadIdx.x;
  const uint2 none = make_uint2(0xff80ff80u, 0xff80ff80u);
  auto fetch = [&](int g) { return g < n4 ? *reinterpret_cast<const uint2*>(row + 4 * (long long)g) : none; };  // (8 B aligned: V*2 B rows)
  if (greedy) {
    auto take = [&](int g, uint2 q) {
      const float v[4] = {bf16_lo(q.x), bf16_hi(q.x), bf16_lo(q.y), bf16_hi(q.y)};
#pragma unroll
      for (int k = 0; k < 4; ++k) amax_update(v[k], 4 * g + k, best, bi);
    };
    int g = first;
    auto round = [&](auto at_once) {  // so many loads in flight
      constexpr int N = decltype(at_once)::value;
      for (; g < n4 - (N - 1) * step; g += N * step) {
        uint2 a[N];
#pragma unroll
        for (int x = 0; x < N; ++x) a[x] = fetch(g + x * step);
#pragma unroll
        for (int x = 0; x < N; ++x) take(g + x * step, a[x]);
      }
    };
    round(std::integral_constant<int, 4>{});
    round(std::integral_constant<int, 2>{});
    round(std::integral_constant<int, 1>{});
  } else {
    auto take = [&](int g, uint2 q) {  // the four logits of group g with their noise
      uint32_t r[4];
      philox4x32_10((uint32_t)g, pos, k0, k1, r);
      const float v[4] = {bf16_lo(q.x), bf16_hi(q.x), bf16_lo(q.y), bf16_hi(q.y)};
#pragma unroll
      for (int k = 0; k < 4; ++k) amax_update(v[k] * inv_t + gumbel_from_bits(r[k]), 4 * g + k, best, bi);
    };
    uint2 a[AT_ONCE];
#pragma unroll
    for (int x = 0; x < AT_ONCE; ++x) a[x] = fetch(first + x * step);
    // (a row of one round: nothing to compare with before it has been looked at)
    const bool one_round = n4 <= AT_ONCE * step;
    if (one_round) {
#pragma unroll
      for (int x = 0; x < AT_ONCE; ++x)
        if (first + x * step < n4) take(first + x * step, a[x]);
    }
    for (int g0 = first; !one_round && g0 - (int)threadIdx.x < n4; g0 += AT_ONCE * step) {  // (whole CTAs go round together)
      uint2 next[AT_ONCE];
#pragma unroll
      for (int x = 0; x < AT_ONCE; ++x) next[x] = fetch(g0 + (AT_ONCE + x) * step);
      const float top = unorder_float(*(volatile int*)&top_s);  // (nothing yet: not a number, and every logit is looked at)
      const float bound = fmaf(top, log2e, -(1.5e-3f + fabsf(top) * 1e-6f));
      bool look[AT_ONCE], any = false;
#pragma unroll
      for (int x = 0; x < AT_ONCE; ++x) {
        uint32_t r[4];
        philox4x32_10((uint32_t)(g0 + x * step), pos, k0, k1, r);
        const __nv_bfloat162 m = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a[x].x), *reinterpret_cast<const __nv_bfloat162*>(&a[x].y));
        const float t = fmaxf(__low2float(m), __high2float(m)) * inv_t;
        float least;  // e^(t - best), a little more
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(least) : "f"(fmaf(t, log2e, -bound)));
        // 1 - u >= 2 - f - 2^-23 with f = 1 + the upper 23 bits
        const uint32_t most = max(max(r[0], r[1]), max(r[2], r[3]));
        const float one_less_u = (2.f - __uint_as_float(0x3f800000u | (most >> 9))) - 1.1920929e-7f;
        look[x] = !(one_less_u > least) && g0 + x * step < n4;
        any |= look[x];
      }
      if (__any_sync(0xffffffffu, any)) {
#pragma unroll
        for (int x = 0; x < AT_ONCE; ++x)
          if (look[x]) take(g0 + x * step, a[x]);  // (seldom: its random numbers once more)
        const int o = __reduce_max_sync(0xffffffffu, order_float(best));
        if ((threadIdx.x & 31) == 0) atomicMax(&top_s, o);
      }
#pragma unroll
      for (int x = 0; x < AT_ONCE; ++x) a[x] = next[x];
    }
  }
  amax_cluster<SAMPLE_THREADS>(best, bi);
  if (split == 0 && threadIdx.x == 0) ids[r_] = bi == 0x7fffffff ? 0 : bi;
}

// CTAs per row: the least rounds x (a CTA's share of a row and its start) + what a cluster and every CTA cost, in the time of one logit of a
// CTA that works alone (of the argmax 0.05 ns, of the sampler 0.13).  Rounds: rows over the clusters that are resident at once, a last one
// that is not full counted in part (`last`), because rows do not end together.  A cluster lies within one of the chip's eight processing clusters,
// which has room for `room` CTAs (17 SMs counted, so that 48 clusters of 6 do not count as resident: 48 rows of 128256 logits 14.9 us with 5
// CTAs each, 18.7 with 6).  Fitted to 1 to 1024 rows of 4096 to 256000 logits with 1 to 8 CTAs each: 1 (sampler) and 2 % (argmax) behind
// the best number on average.  Sampler, us: 128 rows of 128256 24.8 with 2 CTAs each, 30 with 3, 35 with 1; 1024 rows 133 / 149 with 1 / 2;
// one row 7.4 with 8, 12.9 with 2.  Argmax: 128 rows of 32000 4.1 / 4.8 / 5.3 with 1 / 2 / 4, of 128256 12.1 / 10.0 / 8.9; 300 rows of
// 128256 20.8 / 16.8 / 17.4 with 1 / 2 / 3.
struct RowCosts {
  int room, per_cta;  // CTAs that a processing cluster has room for; logits below which a row is not shared any further
  double cluster, last;
};
constexpr RowCosts ARGMAX_COSTS{4 * 17, 16 * ARGMAX_THREADS, 20000, 0.4}, SAMPLE_COSTS{2 * 17, 8 * SAMPLE_THREADS, 5000, 0.3};
static int row_splits(int rows, int V, const RowCosts& c) {
  int best = 1;
  double least = 1e30;
  for (int s = 1; s <= 8 && s <= V / c.per_cta + 1; ++s) {
    const int resident = 8 * (c.room / s);
    const double full = (double)rows / resident, rounds = c.last * ((rows + resident - 1) / resident) + (1.0 - c.last) * (full > 1.0 ? full : 1.0);
    const double t = rounds * ((double)V / s + 4000.0) + (s > 1 ? c.cluster : 0.0) + 20.0 * rows * s;
    if (t < least) {
      least = t;
      best = s;
    }
  }
  return best;
}

}  // namespace b200q

using namespace b200q;

extern "C" {

int b200q_version(void) { return B200Q_VERSION; }
const char* b200q_last_error(void) { return g_err; }
int64_t b200q_launch_count(void) { return (int64_t)__atomic_load_n(&g_launches, __ATOMIC_RELAXED); }

int b200q_device_check(void) {
  int dev = 0;
  cudaDeviceProp p;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaGetDeviceProperties(&p, dev) != cudaSuccess) {
    cudaGetLastError();
    set_error("no CUDA device available: libb200q has no CPU fallback");
    return B200Q_ENODEV;
  }
  if (p.major != 10) {
    set_error("device %s is sm_%d%d; libb200q is built for sm_100a only", p.name, p.major,
              p.minor);
    return B200Q_ENODEV;
  }
  return B200Q_OK;
}

int b200q_embed_ex(const int32_t* ids, const int32_t* prev_out, const void* table, void* out, int T,
                   int H, float scale, void* stream) {
  B200Q_CHECK_ARG(T >= 0 && H > 0 && H % 8 == 0, "embed: bad shape T=%d H=%d", T, H);
  if (T == 0) return B200Q_OK;
  int chunks = H / 8;
  if (scale > 0.f && scale != 1.f)
    embed_scaled_kernel<<<grid_for((long long)T * chunks, 256), 256, 0, as_stream(stream)>>>(
        ids, prev_out, (const uint4*)table, (uint4*)out, T, chunks, scale);
  else
    embed_kernel<<<grid_for((long long)T * chunks, 256), 256, 0, as_stream(stream)>>>(
        ids, prev_out, (const uint4*)table, (uint4*)out, T, chunks);
  B200Q_LAUNCH_CHECK();
  return B200Q_OK;
}

int b200q_embed(const int32_t* ids, const void* table, void* out, int T, int H, void* stream) {
  return b200q_embed_ex(ids, nullptr, table, out, T, H, 0.f, stream);
}

int b200q_embed_scaled(const int32_t* ids, const void* table, void* out, int T, int H, float scale,
                       void* stream) {
  B200Q_CHECK_ARG(scale > 0.f, "embed_scaled: scale must be positive");
  if (scale == 1.f) return b200q_embed_ex(ids, nullptr, table, out, T, H, 0.f, stream);
  return b200q_embed_ex(ids, nullptr, table, out, T, H, scale, stream);
}

int b200q_gemma_rmsnorm(const void* x, const void* w, void* y, int T, int H, float eps,
                        void* stream) {
  B200Q_CHECK_ARG(T >= 0 && H > 0 && H % 8 == 0 && H <= NORM_THREADS * NORM_MAX_CHUNKS * 8,
                  "gemma_rmsnorm: bad shape T=%d H=%d", T, H);
  if (T == 0) return B200Q_OK;
  return norm_chunks(H, [&](auto ch) -> int {
    B200Q_CUDA(launch_early(gemma_norm_kernel<decltype(ch)::value, false>, T, NORM_THREADS, 0, as_stream(stream), 1, (const uint4*)x, nullptr,
                            (const uint4*)w, nullptr, (uint4*)y, H / 8, 1.f / (float)H, eps));
    count_launch();
    return B200Q_OK;
  });
}

int b200q_gemma_norm_add_norm(void* x, void* residual, const void* w_post, const void* w_next, int T,
                              int H, float eps, void* stream) {
  B200Q_CHECK_ARG(T >= 0 && H > 0 && H % 8 == 0 && H <= NORM_THREADS * NORM_MAX_CHUNKS * 8,
                  "gemma_norm_add_norm: bad shape T=%d H=%d", T, H);
  B200Q_CHECK_ARG(x && residual && w_post && w_next, "gemma_norm_add_norm: null argument");
  if (T == 0) return B200Q_OK;
  return norm_chunks(H, [&](auto ch) -> int {
    B200Q_CUDA(launch_early(gemma_norm_kernel<decltype(ch)::value, true>, T, NORM_THREADS, 0, as_stream(stream), 1, (const uint4*)x, (uint4*)residual,
                            (const uint4*)w_post, (const uint4*)w_next, (uint4*)x, H / 8, 1.f / (float)H, eps));
    count_launch();
    return B200Q_OK;
  });
}

int b200q_softcap_bf16(void* logits, int64_t n, float cap, void* stream) {
  B200Q_CHECK_ARG(n >= 0 && n % 8 == 0 && cap > 0.f, "softcap: bad arguments n=%lld cap=%f",
                  (long long)n, (double)cap);
  B200Q_CHECK_ARG((reinterpret_cast<uintptr_t>(logits) & 15) == 0, "softcap: logits not 16-byte aligned");
  if (n == 0) return B200Q_OK;
  B200Q_CUDA(launch_early(softcap_kernel, grid_for(n / 8, 256), 256, 0, as_stream(stream), 1, (uint4*)logits, n / 8, cap));
  count_launch();
  return B200Q_OK;
}

int b200q_rmsnorm(const void* x, const void* w, void* y, int T, int H, float eps, void* stream) {
  B200Q_CHECK_ARG(T >= 0 && H > 0 && H % 8 == 0 && H <= NORM_THREADS * NORM_MAX_CHUNKS * 8,
                  "rmsnorm: bad shape T=%d H=%d", T, H);
  if (T == 0) return B200Q_OK;
  return norm_chunks(H, [&](auto ch) -> int {
    B200Q_CUDA(launch_early(rmsnorm_kernel<decltype(ch)::value, false>, T, NORM_THREADS, 0, as_stream(stream), 1, (const uint4*)x, nullptr,
                            (const uint4*)w, (uint4*)y, H / 8, 1.f / (float)H, eps, nullptr, 0, 0));
    count_launch();
    return B200Q_OK;
  });
}

int b200q_add_rmsnorm(void* x, void* residual, const void* w, int T, int H, float eps,
                      void* stream) {
  B200Q_CHECK_ARG(T >= 0 && H > 0 && H % 8 == 0 && H <= NORM_THREADS * NORM_MAX_CHUNKS * 8,
                  "add_rmsnorm: bad shape T=%d H=%d", T, H);
  if (T == 0) return B200Q_OK;
  return norm_chunks(H, [&](auto ch) -> int {
    B200Q_CUDA(launch_early(rmsnorm_kernel<decltype(ch)::value, true>, T, NORM_THREADS, 0, as_stream(stream), 1, (const uint4*)x, (uint4*)residual,
                            (const uint4*)w, (uint4*)x, H / 8, 1.f / (float)H, eps, nullptr, 0, 0));
    count_launch();
    return B200Q_OK;
  });
}

int b200q_add_rmsnorm_splitk(void* x, void* residual, const void* w, const float* partials,
                             int splits, int T, int H, float eps, void* stream) {
  B200Q_CHECK_ARG(T >= 0 && H > 0 && H % 8 == 0 && H <= NORM_THREADS * NORM_MAX_CHUNKS * 8,
                  "add_rmsnorm_splitk: bad shape T=%d H=%d", T, H);
  B200Q_CHECK_ARG(partials && splits >= 1 && splits <= 16, "add_rmsnorm_splitk: bad partials (splits=%d)", splits);
  if (T == 0) return B200Q_OK;
  return norm_chunks(H, [&](auto ch) -> int {
    B200Q_CUDA(launch_early(rmsnorm_kernel<decltype(ch)::value, true, true>, T, NORM_THREADS, 0, as_stream(stream), 1, nullptr, (uint4*)residual,
                            (const uint4*)w, (uint4*)x, H / 8, 1.f / (float)H, eps, partials, splits, (long long)T * H));
    count_launch();
    return B200Q_OK;
  });
}

int b200q_rope_kvwrite(void* qkv, const void* cos_sin, const int32_t* positions,
                       const int32_t* slot_mapping, void* kv_layer, int T, int n_q, int n_kv,
                       int D, int block_size, void* stream) {
  B200Q_CHECK_ARG(T >= 0 && (D == 64 || D == 128 || D == 256) && n_q > 0 && n_kv > 0 && block_size > 0,
                  "rope_kvwrite: bad shape T=%d n_q=%d n_kv=%d D=%d bs=%d", T, n_q, n_kv, D,
                  block_size);
  if (T == 0) return B200Q_OK;
  // A row is (n_q + n_kv) D/16 + n_kv D/8 items.  Up to 320 rows a row's rounds of 256 items go to blocks of their own, of equal size (128 rows
  // of 32 + 8 + 8 heads, D = 128: 3.05 -> 2.61 us); above, the chip is full and one block to a row reads with more in flight (1000: 6.1, 6.7).
  const int items = (n_q + n_kv) * D / 16 + n_kv * D / 8, blocks = T <= 320 ? (items + 255) / 256 : 1;
  const int threads = blocks > 1 ? ((items + blocks - 1) / blocks + 31) / 32 * 32 : 256;
  B200Q_CUDA(launch_early(rope_kvwrite_kernel<false>, dim3(T, blocks), threads, 0, as_stream(stream), 1, (uint4*)qkv, (const uint4*)cos_sin, positions,
                          slot_mapping, (uint4*)kv_layer, n_q, n_kv, D, block_size, nullptr, 0, 0));
  count_launch();
  return B200Q_OK;
}

int b200q_rope_kvwrite_splitk(void* qkv, const float* partials, int splits, const void* cos_sin,
                              const int32_t* positions, const int32_t* slot_mapping, void* kv_layer,
                              int T, int n_q, int n_kv, int D, int block_size, void* stream) {
  B200Q_CHECK_ARG(T >= 0 && (D == 64 || D == 128 || D == 256) && n_q > 0 && n_kv > 0 && block_size > 0,
                  "rope_kvwrite_splitk: bad shape T=%d n_q=%d n_kv=%d D=%d bs=%d", T, n_q, n_kv, D,
                  block_size);
  B200Q_CHECK_ARG(partials && splits >= 1 && splits <= 16, "rope_kvwrite_splitk: bad partials (splits=%d)", splits);
  if (T == 0) return B200Q_OK;
  // One item to a thread, in blocks of 128: a thread that goes on to a second item begins its reads anew.  Four parts, us, a block of 256
  // to a row / so: 48 rows of 32 + 8 + 8 heads, D = 128 5.2 / 3.2; 16 + 8 + 8, D = 256 5.7 / 3.3; 128 rows of the first 5.5 / 3.7.
  const int items = (n_q + n_kv) * D / 16 + n_kv * D / 8;
  B200Q_CUDA(launch_early(rope_kvwrite_kernel<true>, dim3(T, (items + 127) / 128), 128, 0, as_stream(stream), 1, (uint4*)qkv, (const uint4*)cos_sin, positions,
                          slot_mapping, (uint4*)kv_layer, n_q, n_kv, D, block_size, partials, splits, (long long)T * (n_q + 2 * n_kv) * D));
  count_launch();
  return B200Q_OK;
}

int b200q_swiglu(const void* gate_up, void* out, int T, int I, void* stream) {
  B200Q_CHECK_ARG(T >= 0 && I > 0 && I % 8 == 0, "swiglu: bad shape T=%d I=%d", T, I);
  if (T == 0) return B200Q_OK;
  int ic = I / 8;
  B200Q_CUDA(launch_early(swiglu_kernel, grid_for((long long)T * ic, 256), 256, 0, as_stream(stream), 1, (const uint4*)gate_up, (uint4*)out,
                          T, ic));
  count_launch();
  return B200Q_OK;
}

int b200q_gather_rows(const void* x, const int32_t* rows, void* out, int n, int H, void* stream) {
  B200Q_CHECK_ARG(n >= 0 && H > 0 && H % 8 == 0, "gather_rows: bad shape n=%d H=%d", n, H);
  if (n == 0) return B200Q_OK;
  int chunks = H / 8;
  B200Q_CUDA(launch_early(gather_rows_kernel, grid_for((long long)n * chunks, 256), 256, 0, as_stream(stream), 1, (const uint4*)x, rows,
                          (uint4*)out, n, chunks));
  count_launch();
  return B200Q_OK;
}

int b200q_argmax_bf16(const void* logits, int32_t* ids, int B, int V, void* stream) {
  B200Q_CHECK_ARG(B >= 0 && V > 0, "argmax: bad shape B=%d V=%d", B, V);
  if (B == 0) return B200Q_OK;
  for (int at = 0; at < B; at += 65535) {  // (a grid's second dimension ends at 65535 rows)
    const int rows = B - at < 65535 ? B - at : 65535, splits = row_splits(rows, V, ARGMAX_COSTS);
    B200Q_CUDA(launch_early(argmax_kernel, dim3(splits, rows), ARGMAX_THREADS, 0, as_stream(stream), splits,
                            (const bf16*)logits + (long long)at * V, ids + at, V));
    count_launch();
  }
  return B200Q_OK;
}

int b200q_sample_bf16(const void* logits, const int32_t* params, int32_t* ids, int B, int V,
                      void* stream) {
  B200Q_CHECK_ARG(B >= 0 && V > 0 && V % 4 == 0, "sample: bad shape B=%d V=%d (V %% 4 == 0)", B, V);
  B200Q_CHECK_ARG(params != nullptr, "sample: params is null");
  if (B == 0) return B200Q_OK;
  // (a grid's second dimension ends at 65535 rows)
  for (int at = 0; at < B; at += 65535) {
    const int rows = B - at < 65535 ? B - at : 65535;
    const int splits = row_splits(rows, V, SAMPLE_COSTS);
    B200Q_CUDA(launch_early(sample_kernel, dim3(splits, rows), SAMPLE_THREADS, 0, as_stream(stream), splits,
                            (const bf16*)logits + (long long)at * V, params + 4 * (long long)at, ids + at, V));
    count_launch();
  }
  return B200Q_OK;
}

}  // extern "C"
