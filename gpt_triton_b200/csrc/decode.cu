// Token-by-token generation on top of the forward path: key/value cache, one-query attention, sampling.
// The reference project lists "KV cache + sampling" among the things it never built (README.md:55), so nothing
// here has a counterpart there; the arithmetic follows the reference's flash_attention_v1 (kernels.py:417-474:
// 64-key blocks, fp16 dot operands, fp32 running maximum and denominator, P rounded to fp16 relative to the
// running maximum of its block), so that a cached step gives what re-running the whole sequence would.
//
// Everything that changes from one generated token to the next is read from DEVICE memory (the int32 pair
// `pos` = {tokens in the cache, prompt length}), so that the kernels of a decode step can be recorded once in a
// CUDA graph and replayed for every step.  All of these kernels are HBM-bound gathers and streams:
//   kv_cache_fill_kernel      cache[b, l, 0:2H] = qkv[b, l, H:3H] after the prompt's forward   (2 x B L 2H bytes)
//   attention_decode_kernel   appends the new token's k, v and attends its q over the cache    (B (pos+1) 2H elements read)
//   sample_rows_kernel        top-k filter + Gumbel-max draw over a row of logits              (passes over B V logits, mostly L2)
//   decode_append_kernel      tokens[b, column] = next id (also into the buffer the next step embeds); pos += 1
#include <atomic>

#include "common.cuh"
#include "mma_sync.cuh"

namespace b200 {
namespace {

// codes left in the status word (site numbers above those of the tensor-core kernels)
constexpr int kSiteCachePosition = 41;  // the cache has no room for the position being written
constexpr int kSiteTokenColumn = 42;    // the token buffer has no column for the id being appended

// ------------------------------------------------------------------ prompt -> cache
// One warp per (batch, position) row: 2H elements as 16-byte vectors.
__global__ void __launch_bounds__(256)
kv_cache_fill_kernel(const uint4* __restrict__ qkv, uint4* __restrict__ cache, int64_t rows, int64_t L, int64_t cache_len, int vec_per_h) {
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int64_t stride = (int64_t)gridDim.x * 8;
  for (int64_t t = warp0; t < rows; t += stride) {
    const int64_t b = t / L, l = t % L;
    const uint4* src = qkv + (t * 3 + 1) * vec_per_h;
    uint4* dst = cache + (b * cache_len + l) * 2 * vec_per_h;
    for (int c = lane; c < 2 * vec_per_h; c += 32) dst[c] = src[c];
  }
}

// ------------------------------------------------------------------ one-query attention over the cache
// The value a dot product sees: fp32 storage is rounded to fp16 first (kernels.py:229, 234 of the reference cast every
// dot operand to fp16); 16-bit storage is used as it is.
template <typename T>
__device__ __forceinline__ float dot_operand(float v) {
  return v;
}
template <>
__device__ __forceinline__ float dot_operand<float>(float v) {
  return __half2float(__float2half_rn(v));
}
__device__ __forceinline__ float ex2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// eight 16-bit elements that were loaded as 16 bytes
template <typename T>
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t;
    if constexpr (DType<T>::code == B200_F16) t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
    else t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
    f[2 * i] = t.x, f[2 * i + 1] = t.y;
  }
}
// N consecutive elements moved as one access (N * sizeof(T) is 2, 4, 8 or 16 bytes; the address is aligned to it)
template <typename T, int N>
struct alignas(sizeof(T) * N) Vec {
  T v[N];
};
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// qkv_new [B, 3H] holds the new token's q | k | v; cache [B, cache_len, 2H] holds k | v of the earlier positions.
// The pos + 1 keys are walked in the reference's blocks of 64 (kernels.py:509).  A PAIR of lanes owns a key: lane
// 2i takes the first D/2 elements of the key and value rows of keys i, i + 16, i + 32, i + 48 of the block, lane
// 2i + 1 the second D/2, read as 16-byte vectors, so one warp-wide load covers whole 32-byte sectors of 16 rows;
// the two halves of a dot product meet in one shuffle.  All loads of a block are independent of each other, so many
// are in flight per lane.  The softmax reference point of a block is the running maximum over the blocks up
// to and including it, exactly as in the reference's loop (kernels.py:440-468): P = exp(s - that maximum) is
// rounded to fp16 before it multiplies V, the denominator sums the unrounded P.  Every lane keeps a private D/2-wide
// piece of the output row in registers (the rescale factor of a block is the same for all lanes); at the end the
// 16 pieces of each half are added by a halving exchange (D/2 -> D/32 values per lane in four shuffle rounds) that
// leaves lane l with output columns (l & 1) * D/2 + (l >> 1) * D/32 + [0, D/32).
// SPLIT = 1: one warp per (batch, head), four per block, no block-level synchronisation.  SPLIT > 1: the SPLIT warps of a block
// share one (batch, head) and take the 64-key blocks of a group of SPLIT side by side; the block maxima of a group go through
// shared memory (one block-level barrier per group), so that a warp still uses the running maximum over the blocks up to its own;
// the warps' partial rows are merged through shared memory at the end.
// What bounds it: the bytes of the cache with many sequences, the chain position -> keys -> scores -> values with few.  AHEAD (half
// rows of 16-bit data of at most 64 bytes): all keys and values of a block are loaded into registers before the first is used, one
// trip to memory per block instead of two; worth it while the warps that these registers cost are not missed.
// Before (four warps, or one from 16 per SM on, values loaded behind the softmax) -> now, us (HBM alone), 12 heads of 64, bf16: 8
// sequences, 330 keys 17.5 -> 6.7; 16 17.6 -> 10.2; 32 18.2 -> 13.4; 197 56.7 -> 39.3 (31).
// STAGED (one warp per row, 16-bit data): with many sequences what bounds it is how much of the cache is on its way, and registers
// hold too little of that.  Keys and values of a block come by cp.async into two slots of shared memory per warp; a slot is
// refilled as soon as it has been read, so that 8 to 16 KB per warp are in flight at 12 warps an SM.  The same bits as the other
// variants of one warp.  us, before -> now (HBM alone), 330 and 1000 keys: 128 sequences 31.3 -> 26.3 (20) and 78.7 -> 62.6 (61); 256
// 56.2 -> 47.1 (40) and 155 -> 121 (122); 512 102 -> 89 (81) and 272 -> 240 (244); 25 heads of 32, 256 sequences 58 -> 49 and 154 -> 132.
constexpr int kStagedWarps = 2;  // per block
template <int D>
constexpr int kStagedSlot = 64 * D * 2;  // bytes of a block of 16-bit keys, or of values
template <int SPLIT, bool STAGED>
constexpr int kDecodeWarps = SPLIT > 1 ? SPLIT : STAGED ? kStagedWarps : 4;

template <typename T, int D, int SPLIT, bool AHEAD, bool STAGED = false>
__global__ void __launch_bounds__(32 * kDecodeWarps<SPLIT, STAGED>)
attention_decode_kernel(const T* qkv_new, T* __restrict__ cache, T* __restrict__ out, int64_t BH, int NH, int64_t cache_len, float scale_log2e,
                        const int* pos_dev, int* status_word) {
  constexpr int WARPS = kDecodeWarps<SPLIT, STAGED>;
  static_assert(!STAGED || (SPLIT == 1 && !AHEAD && sizeof(T) == 2), "one warp per row, 16-bit rows");
  extern __shared__ __align__(128) uint8_t ring[];  // STAGED: per warp a slot for keys and one for values
  __shared__ __align__(16) float q_s[WARPS][D + 4];  // the second half of q sits 4 floats further on: the two lanes of a pair read different banks
  __shared__ float part_o[SPLIT == 1 ? 1 : WARPS][D];
  __shared__ float part_ml[WARPS][2];
  __shared__ float group_max[2][WARPS];
  constexpr int DPL = D / 32;  // output columns per lane
  constexpr int DH = D / 2;    // elements of a row per lane of a pair
  constexpr int VECS = DH * (int)sizeof(T) / 16;  // 16-byte pieces of that
  static_assert(!AHEAD || (sizeof(T) == 2 && VECS <= 4), "a block's keys and values fit the registers");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int side = lane & 1, kl = lane >> 1;  // which half of the rows; which of the 16 key slots
  const int64_t w = SPLIT == 1 ? (int64_t)blockIdx.x * WARPS + warp : (int64_t)blockIdx.x;
  const int part = SPLIT == 1 ? 0 : warp;
  const int64_t b = w / NH;
  const int h = (int)(w % NH);
  const int64_t H = (int64_t)NH * D, pitch = 2 * H;
  const T* qn = qkv_new + b * 3 * H + (int64_t)h * D;
  const T* kn = qn + H;
  const T* vn = kn + H;
  T* kc = cache + b * cache_len * pitch + (int64_t)h * D;
  T* vc = kc + H;
  pdl_launch_dependents();
  // Ahead of the kernel in front: this warp's first block of keys and values towards L2.  (The position may still be the previous
  // step's, or anything at all: it only decides which lines of the cache are prefetched.)
  if (AHEAD && SPLIT > 2 && w < BH) {
    const int64_t end = min((int64_t)*reinterpret_cast<const volatile int*>(pos_dev), cache_len);
#pragma unroll
    for (int r = 0; r < 64; r += 32) {
      const int64_t key = part * 64 + r + lane;
      if (key < end) {
#pragma unroll
        for (int c = 0; c < D * (int)sizeof(T); c += 128) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(kc + key * pitch) + c));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(vc + key * pitch) + c));
        }
      }
    }
  }
  pdl_wait();
  // (an ordinary load behind the wait, on which every load of the cache depends: the cache may stay __restrict__, see common.cuh)
  const int pos = pos_dev[0];
  if (pos < 0 || pos >= cache_len) {
    if (threadIdx.x == 0 && status_word) atomicCAS(status_word, 0, kSiteCachePosition);
    return;
  }
  if (w >= BH) return;  // (SPLIT > 1: the whole block leaves together)
  // one block of keys: the first warp alone (the host knows how long the cache is, not how many keys it holds; without AHEAD the
  // registers that this takes cost more than it gives)
  const bool solo = SPLIT == 1 || (AHEAD && pos < 64);
  if (solo && part != 0) return;
  if constexpr (SPLIT == 1) {  // (all loads ahead of the stores; with several warps the registers are dearer)
    T q_new[DPL], k_new[DPL], v_new[DPL];
#pragma unroll
    for (int r = 0; r < DPL; ++r) q_new[r] = qn[r * 32 + lane], k_new[r] = kn[r * 32 + lane], v_new[r] = vn[r * 32 + lane];
#pragma unroll
    for (int r = 0; r < DPL; ++r) {
      const int i = r * 32 + lane;
      q_s[warp][i + (i >= D / 2 ? 4 : 0)] = dot_operand<T>(to_float(q_new[r]));
      kc[(int64_t)pos * pitch + i] = k_new[r];
      vc[(int64_t)pos * pitch + i] = v_new[r];
    }
  } else {
    for (int i = lane; i < D; i += 32) {
      q_s[warp][i + (i >= D / 2 ? 4 : 0)] = dot_operand<T>(to_float(qn[i]));
      if (part == 0) {
        kc[(int64_t)pos * pitch + i] = kn[i];
        vc[(int64_t)pos * pitch + i] = vn[i];
      }
    }
  }
  __syncwarp();
  // (the new token's own key and value are read from qkv_new below, not back from the cache)
  const int n_keys = pos + 1;
  // STAGED: a block's rows on their way into a slot; a warp-wide copy covers whole rows, and the 16-byte pieces of a row are permuted by
  // its number, so that the lanes' reads fall into different banks
  constexpr int ROW = D * (int)sizeof(T), PIECES = ROW / 16;
  uint8_t* const keys_s = ring + (STAGED ? warp * 2 * kStagedSlot<D> : 0);
  uint8_t* const values_s = keys_s + (STAGED ? kStagedSlot<D> : 0);
  auto fetch = [&](uint8_t* slot, const T* rows, const T* newest, int k0) {
    if (k0 < n_keys) {
      const uint32_t to = (uint32_t)__cvta_generic_to_shared(slot);
      const int c = lane % PIECES;
#pragma unroll
      for (int i = 0; i < 64 * PIECES / 32; ++i) {
        const int r = i * (32 / PIECES) + lane / PIECES, key = k0 + r;
        const T* src = (key == pos ? newest : rows + (int64_t)min(key, pos) * pitch) + c * 8;
        warp_mma::cp_async16(to + (uint32_t)(r * ROW + ((c ^ (r & (PIECES - 1))) << 4)), src, key < n_keys);
      }
    }
    warp_mma::cp_async_commit();  // (possibly empty: the waits count groups)
  };
  auto staged = [&](const uint8_t* slot, int r, int piece) { return *reinterpret_cast<const uint4*>(slot + r * ROW + ((piece ^ (r & (PIECES - 1))) << 4)); };
  if constexpr (STAGED) {
    fetch(keys_s, kc, kn, 0);
    fetch(values_s, vc, vn, 0);
  }
  const int n_groups = (n_keys + 64 * SPLIT - 1) / (64 * SPLIT);
  float m_run = -INFINITY;  // reference maximum of this warp's latest block
  float m_all = -INFINITY;  // running maximum over all blocks of the groups done so far
  float l_lane = 0.f;
  float o[DH];
#pragma unroll
  for (int d = 0; d < DH; ++d) o[d] = 0.f;
  const float* q_mine = q_s[warp] + side * (DH + 4);
  for (int g = 0; g < n_groups; ++g) {
    const int k0 = (g * SPLIT + part) * 64;
    uint4 kraw[AHEAD ? 4 : 1][AHEAD ? VECS : 1], vraw[AHEAD ? 4 : 1][AHEAD ? VECS : 1];
    if constexpr (AHEAD) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = k0 + j * 16 + kl;
        const uint4* kr = reinterpret_cast<const uint4*>((key == pos ? kn : kc + (int64_t)key * pitch) + side * DH);
#pragma unroll
        for (int c = 0; c < VECS; ++c) kraw[j][c] = key < n_keys ? kr[c] : make_uint4(0u, 0u, 0u, 0u);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = k0 + j * 16 + kl;
        const uint4* vr = reinterpret_cast<const uint4*>((key == pos ? vn : vc + (int64_t)key * pitch) + side * DH);
#pragma unroll
        for (int c = 0; c < VECS; ++c) vraw[j][c] = key < n_keys ? vr[c] : make_uint4(0u, 0u, 0u, 0u);
      }
    }
    if constexpr (STAGED) {
      warp_mma::cp_async_wait<1>();  // the keys are there (the values may not be)
      __syncwarp();
    }
    float s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int key = k0 + j * 16 + kl;
      float a = 0.f;
      if (AHEAD || key < n_keys) {
        const T* kr = (key == pos ? kn : kc + (int64_t)key * pitch) + side * DH;
#pragma unroll
        for (int c = 0; c < DH; c += 8) {
          float f[8];
          if constexpr (AHEAD) unpack8<T>(kraw[j][c / 8], f);
          else if constexpr (STAGED) unpack8<T>(staged(keys_s, j * 16 + kl, side * (PIECES / 2) + c / 8), f);
          else load8(kr + c, f);
#pragma unroll
          for (int i = 0; i < 8; ++i) a = fmaf(q_mine[c + i], dot_operand<T>(f[i]), a);
        }
      }
      a += __shfl_xor_sync(0xffffffffu, a, 1);                      // the other half of the dot product
      s[j] = key < n_keys ? a * scale_log2e : -INFINITY;            // score in log2 units
    }
    if constexpr (STAGED) {
      __syncwarp();
      fetch(keys_s, kc, kn, k0 + 64);
    }
    const float bm = warp_max(fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3])));
    float m_new = fmaxf(m_all, bm);
    if (!solo) {
      if (lane == 0) group_max[g & 1][warp] = bm;
      __syncthreads();
#pragma unroll
      for (int p2 = 0; p2 < SPLIT; ++p2) {
        const float other = group_max[g & 1][p2];
        if (p2 < part) m_new = fmaxf(m_new, other);
        m_all = fmaxf(m_all, other);
      }
    } else {
      m_all = m_new;
    }
    if (bm == -INFINITY) continue;  // no key of this block exists (warp-uniform; SPLIT > 1 only)
    const float mult = ex2_ftz(m_run - m_new);  // 0 for the warp's first block
    m_run = m_new;
    float ph[4], psum = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float pj = ex2_ftz(s[j] - m_new);  // 0 for keys beyond the last
      psum += pj;
      ph[j] = __half2float(__float2half_rn(pj));
    }
    l_lane = fmaf(l_lane, mult, side == 0 ? psum : 0.f);  // (both lanes of a pair hold the same scores: count them once)
#pragma unroll
    for (int d = 0; d < DH; ++d) o[d] *= mult;
    if constexpr (STAGED) {
      warp_mma::cp_async_wait<1>();  // the values are there (the next keys may not be)
      __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int key = k0 + j * 16 + kl;
      if (key < n_keys) {
        const T* vr = (key == pos ? vn : vc + (int64_t)key * pitch) + side * DH;
#pragma unroll
        for (int c = 0; c < DH; c += 8) {
          float f[8];
          if constexpr (AHEAD) unpack8<T>(vraw[j][c / 8], f);
          else if constexpr (STAGED) unpack8<T>(staged(values_s, j * 16 + kl, side * (PIECES / 2) + c / 8), f);
          else load8(vr + c, f);
#pragma unroll
          for (int i = 0; i < 8; ++i) o[c + i] = fmaf(ph[j], dot_operand<T>(f[i]), o[c + i]);
        }
      }
    }
    if constexpr (STAGED) {
      __syncwarp();
      fetch(values_s, vc, vn, k0 + 64);
    }
  }
  // add up the lanes' pieces and denominators (all relative to the same maximum m_run)
  float l_warp = warp_sum(l_lane);
#pragma unroll
  for (int n = DH / 2, off = 16; off > 1; n >>= 1, off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float mine = upper ? o[i + n] : o[i];
      const float theirs = upper ? o[i] : o[i + n];
      o[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, off);
    }
  }
  const int col0 = side * DH + kl * DPL;  // first of this lane's DPL output columns
  // o[0 .. DPL) now holds output columns col0 + j of this warp's blocks
  if (!solo) {
#pragma unroll
    for (int j = 0; j < DPL; ++j) part_o[warp][col0 + j] = o[j];
    if (lane == 0) part_ml[warp][0] = m_run, part_ml[warp][1] = l_warp;
    __syncthreads();
    if (warp != 0) return;
    l_warp = 0.f;
#pragma unroll
    for (int j = 0; j < DPL; ++j) o[j] = 0.f;
#pragma unroll
    for (int p2 = 0; p2 < SPLIT; ++p2) {
      const float mp = part_ml[p2][0];
      const float f = mp == -INFINITY ? 0.f : ex2_ftz(mp - m_all);  // (m_all is the maximum over every block by now)
      l_warp = fmaf(part_ml[p2][1], f, l_warp);
#pragma unroll
      for (int j = 0; j < DPL; ++j) o[j] = fmaf(part_o[p2][col0 + j], f, o[j]);
    }
  }
  const float inv = 1.0f / l_warp;
  Vec<T, DPL> res;
#pragma unroll
  for (int d = 0; d < DPL; ++d) res.v[d] = from_float<T>(o[d] * inv);
  *reinterpret_cast<Vec<T, DPL>*>(out + b * H + (int64_t)h * D + col0) = res;
}

template <typename T, int D, int SPLIT, bool AHEAD, bool STAGED = false>
int attention_decode_split(const void* qkv_new, void* cache, void* out, int64_t BH, int64_t NH, int64_t cache_len, float sl, const int* pos_dev,
                           int* status_word, cudaStream_t stream) {
  constexpr int warps = kDecodeWarps<SPLIT, STAGED>;
  const int64_t blocks = SPLIT == 1 ? (BH + warps - 1) / warps : BH;
  // (an early start helps blocks that all find room; 3072 of them in the way of the product in front cost a step with 256 sequences 10 %)
  LaunchSetup ls(dim3((unsigned)blocks), dim3(32 * warps), STAGED ? warps * 2 * kStagedSlot<D> : 0, stream, 1, pdl_enabled() || blocks <= 2 * sm_count());
  const cudaError_t e = cudaLaunchKernelEx(&ls.cfg, attention_decode_kernel<T, D, SPLIT, AHEAD, STAGED>, (const T*)qkv_new, (T*)cache, (T*)out, BH, (int)NH,
                                           cache_len, sl, pos_dev, status_word);
  note_launches(1);
  return status_from_cuda(e);
}

// How many (batch, head) pairs of a variant the current device has room for at once (0 if it cannot be asked).
template <typename T, int D, int SPLIT, bool AHEAD, bool STAGED = false>
int64_t heads_at_once() {
  static std::atomic<int> per_sm[kMaxDevices];  // blocks, + 1; 0: not asked yet
  const int slot = device_slot();
  if (slot < 0) return 0;
  constexpr int warps = kDecodeWarps<SPLIT, STAGED>;
  int n = per_sm[slot].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, attention_decode_kernel<T, D, SPLIT, AHEAD, STAGED>, 32 * warps,
                                                      STAGED ? warps * 2 * kStagedSlot<D> : 0) != cudaSuccess)
      return 0;
    per_sm[slot].store(++n, std::memory_order_relaxed);
  }
  return (int64_t)(n - 1) * sm_count() * (SPLIT == 1 ? warps : 1);
}

template <typename T, int D>
int attention_decode_sized(const void* qkv_new, void* cache, void* out, int64_t BH, int64_t NH, int64_t cache_len, float sl, const int* pos_dev,
                           int* status_word, cudaStream_t stream) {
#define B200_DECODE(SPLIT, AHEAD) return attention_decode_split<T, D, SPLIT, AHEAD>(qkv_new, cache, out, BH, NH, cache_len, sl, pos_dev, status_word, stream)
#define B200_DECODE_IF_ROOM(SPLIT, AHEAD) \
  if (BH <= heads_at_once<T, D, SPLIT, AHEAD>()) B200_DECODE(SPLIT, AHEAD)
  if constexpr (sizeof(T) == 2 && D <= 64) {
    // Most warps per (batch, head) whose launch still finds room at once: a second wave of blocks costs nearly as much as the first
    // (12 heads of 64, bf16, 222 sequences are one wave at one warp, 1.1 at two: 52.8 us against 58.4 at 330 keys, 14 against 21 at
    // 60; 173 sequences are one wave at two: 36 against 47).  A cache of one block of keys has nothing to share out (96 heads, 16
    // keys: 2.8 us with one warp, 3.8 with eight).  Four warps that load values behind the softmax, against one that loads ahead,
    // 64 sequences, 100 / 330 / 1000 keys: 11.8 / 20.5 / 42.3 us against 9.8 / 20.0 / 48.5.
    // Many rows of more than one block: keys and values staged in shared memory (see the kernel).  Below 6 pairs per SM (10 of half the
    // size) several warps per pair can be faster (12 heads of 64, 330 / 1000 keys: 32 sequences 13.7 / 30.5 us against 15.9 / 37.5, 64
    // 20.5 / 42.6 against 18.6 / 45.0, but 128 31.3 / 78.7 against 26.3 / 62.6; 25 heads of 32: 32 sequences 12.8 / 23.8 against 12.9 /
    // 29.5, 64 16.9 / 40.2 against 15.9 / 37.3).  At head size 64 an SM has room for 12 pairs, and a second wave that is not half
    // full costs what it would save: 170 sequences 35.9 / 91.9 against 40.2 / 105.7, 197 39.7 / 102 against 41.8 / 116, but 222 52.7 / 145
    // against 44.9 / 118.  At 32 it pays from one wave on (170 x 25 heads 42.0 / 117 against 37.6 / 98.7).
    if (cache_len > 64 && BH >= (D == 64 ? 6 : 10) * (int64_t)sm_count()) {
      const int64_t room = heads_at_once<T, D, 1, false, true>();
      if (BH <= room || D == 32 || 2 * BH >= 3 * room)
        return attention_decode_split<T, D, 1, false, true>(qkv_new, cache, out, BH, NH, cache_len, sl, pos_dev, status_word, stream);
    }
    if (cache_len > 64) {
      B200_DECODE_IF_ROOM(8, true);
      B200_DECODE_IF_ROOM(4, true);
      B200_DECODE_IF_ROOM(2, true);
      if (cache_len > 256) B200_DECODE_IF_ROOM(4, false);
    }
    B200_DECODE_IF_ROOM(1, true);
    if (cache_len > 64) B200_DECODE_IF_ROOM(2, false);
    B200_DECODE_IF_ROOM(1, false);
    B200_DECODE(1, false);
  } else {
    // rows too wide to be held: one warp per (batch, head) fills the GPU from about 16 warps per SM on; below that, four share one
    if (BH >= (int64_t)sm_count() * 16) B200_DECODE(1, false);
    B200_DECODE(4, false);
  }
#undef B200_DECODE_IF_ROOM
#undef B200_DECODE
}

template <typename T>
int attention_decode_typed(const void* qkv_new, void* cache, void* out, int64_t B, int64_t NH, int64_t D, int64_t cache_len, float scale,
                           const int* pos_dev, int* status_word, cudaStream_t stream) {
  const float sl = scale * 1.4426950408889634f;
  if (D == 32) return attention_decode_sized<T, 32>(qkv_new, cache, out, B * NH, NH, cache_len, sl, pos_dev, status_word, stream);
  if (D == 64) return attention_decode_sized<T, 64>(qkv_new, cache, out, B * NH, NH, cache_len, sl, pos_dev, status_word, stream);
  if (D == 128) return attention_decode_sized<T, 128>(qkv_new, cache, out, B * NH, NH, cache_len, sl, pos_dev, status_word, stream);
  return B200_ERR_UNSUPPORTED;
}

// ------------------------------------------------------------------ append + advance
// One block: every thread reads the position before thread 0 moves it.
__global__ void __launch_bounds__(256)
decode_append_kernel(const int64_t* __restrict__ next_ids, int64_t* __restrict__ tokens, int64_t ld_tokens, int64_t n_cols, int64_t B, int* pos_dev,
                     int advance, int64_t* __restrict__ feedback, int* status_word) {
  const int64_t col = (int64_t)pos_dev[0] - pos_dev[1] + (advance ? 1 : 0);
  __syncthreads();
  if (col < 0 || col >= n_cols) {
    if (threadIdx.x == 0 && status_word) atomicCAS(status_word, 0, kSiteTokenColumn);
    return;
  }
  for (int64_t b = threadIdx.x; b < B; b += blockDim.x) {
    const int64_t id = next_ids[b];
    tokens[b * ld_tokens + col] = id;
    if (feedback) feedback[b] = id;  // what the next decode step embeds
  }
  if (advance && threadIdx.x == 0) pos_dev[0] += 1;
}

// ------------------------------------------------------------------ sampling
// Counter-based uniform numbers: the 64-bit finaliser of SplitMix64 (Steele, Lea, Flood 2014) applied to
// seed + golden ratio * (step + 1) and then, xored with (row, column), once more; 23 random bits -> u = (n + 1/2) / 2^23 in (0, 1), exact in fp32.
__host__ __device__ inline uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float uniform01(uint64_t stream_key, uint32_t row, uint32_t col) {
  const uint64_t x = mix64(stream_key ^ (((uint64_t)row << 32) | col));
  return ((float)(uint32_t)(x >> 41) + 0.5f) * (1.0f / 8388608.0f);
}
// Unsigned key with the order of the floats (larger float <-> larger key).
__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

constexpr int kSampleThreads = 512;

// One block per row.  top_k > 0: four 8-bit radix passes find the key of the top_k-th largest logit; every logit at
// or above it stays in (ties at the threshold all stay, as with the usual `logits < kth_value -> -inf` filter).
// Then Gumbel-max: id = argmax_j (logit_j / temperature - log(-log(u_j))), lowest j on ties, which draws from
// softmax(logits / temperature) over the kept columns.
template <typename T>
__global__ void __launch_bounds__(kSampleThreads)
sample_rows_kernel(const T* __restrict__ logits, int64_t ld, int V, float inv_temperature, int top_k, uint64_t seed, const int* __restrict__ step_dev,
                   int64_t* __restrict__ ids_out) {
  __shared__ int hist[256];
  __shared__ int sel_bin, sel_want;
  __shared__ float red_val[kSampleThreads / 32];
  __shared__ int red_idx[kSampleThreads / 32];
  const int row = blockIdx.x, tid = threadIdx.x;
  const T* x = logits + (int64_t)row * ld;
  uint32_t thr_key = 0;
  if (top_k > 0 && top_k < V) {
    uint32_t prefix = 0, mask = 0;
    int want = top_k;
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass;
      if (tid < 256) hist[tid] = 0;
      __syncthreads();
      for (int i = tid; i < V; i += kSampleThreads) {
        const uint32_t key = order_key(to_float(x[i]));
        if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255], 1);
      }
      __syncthreads();
      if (tid == 0) {
        int cum = 0, bin = 255;
        for (; bin > 0; --bin) {
          if (cum + hist[bin] >= want) break;
          cum += hist[bin];
        }
        sel_bin = bin, sel_want = want - cum;
      }
      __syncthreads();
      prefix |= (uint32_t)sel_bin << shift;
      mask |= 255u << shift;
      want = sel_want;
      __syncthreads();
    }
    thr_key = prefix;
  }
  const uint64_t stream_key = mix64(seed + 0x9E3779B97F4A7C15ull * ((uint64_t)(uint32_t)(step_dev ? step_dev[0] : 0) + 1));
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  for (int i = tid; i < V; i += kSampleThreads) {
    const float f = to_float(x[i]);
    if (!(f == f) || order_key(f) < thr_key) continue;  // NaN or filtered out
    const float g = -logf(-logf(uniform01(stream_key, (uint32_t)row, (uint32_t)i)));
    const float sc = fmaf(f, inv_temperature, g);
    if (sc > best) best = sc, best_i = i;  // ascending i within a thread: the first maximum stays
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
    if (ov > best || (ov == best && oi < best_i)) best = ov, best_i = oi;
  }
  if ((tid & 31) == 0) red_val[tid >> 5] = best, red_idx[tid >> 5] = best_i;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kSampleThreads / 32; ++w)
      if (red_val[w] > best || (red_val[w] == best && red_idx[w] < best_i)) best = red_val[w], best_i = red_idx[w];
    ids_out[row] = best_i == 0x7fffffff ? 0 : best_i;
  }
}

}  // namespace

int launch_kv_cache_fill(const void* qkv, void* cache, int64_t B, int64_t L, int64_t H, int64_t cache_len, int dtype, cudaStream_t stream) {
  if (B == 0 || L == 0 || H == 0) return B200_OK;
  const int64_t row_bytes = H * dtype_size(dtype);
  if (row_bytes % 16 || ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(cache)) & 15)) return B200_ERR_ALIGNMENT;
  if (L > cache_len || row_bytes / 16 > 0x3fffffff) return B200_ERR_BAD_ARGUMENT;
  const int64_t rows = B * L;
  int64_t blocks = (rows + 7) / 8;
  const int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  kv_cache_fill_kernel<<<(unsigned)blocks, 256, 0, stream>>>((const uint4*)qkv, (uint4*)cache, rows, L, cache_len, (int)(row_bytes / 16));
  note_launches(1);
  return status_from_cuda(cudaGetLastError());
}

int launch_attention_decode(const void* qkv_new, void* cache, void* out, int64_t B, int64_t NH, int64_t D, int64_t cache_len, float scale, int dtype,
                            const int* pos_dev, int* status_word, cudaStream_t stream) {
  if (B == 0 || NH == 0) return B200_OK;
  // half key rows are read as 16-byte vectors
  if (((reinterpret_cast<uintptr_t>(qkv_new) | reinterpret_cast<uintptr_t>(cache)) & 15) || (D / 2 * dtype_size(dtype)) % 16) return B200_ERR_ALIGNMENT;
  if (B * NH > 0x7fffffffLL * 4 || NH > 0x7fffffff) return B200_ERR_BAD_ARGUMENT;
  switch (dtype) {
    case B200_F32: return attention_decode_typed<float>(qkv_new, cache, out, B, NH, D, cache_len, scale, pos_dev, status_word, stream);
    case B200_F16: return attention_decode_typed<__half>(qkv_new, cache, out, B, NH, D, cache_len, scale, pos_dev, status_word, stream);
    case B200_BF16: return attention_decode_typed<__nv_bfloat16>(qkv_new, cache, out, B, NH, D, cache_len, scale, pos_dev, status_word, stream);
  }
  return B200_ERR_BAD_ARGUMENT;
}

int launch_decode_append(const int64_t* next_ids, int64_t* tokens, int64_t ld_tokens, int64_t n_cols, int64_t B, int* pos_dev, int advance,
                         int64_t* feedback, int* status_word, cudaStream_t stream) {
  decode_append_kernel<<<1, 256, 0, stream>>>(next_ids, tokens, ld_tokens, n_cols, B, pos_dev, advance, feedback, status_word);
  note_launches(1);
  return status_from_cuda(cudaGetLastError());
}

int launch_sample_rows(const void* logits, int64_t ld, int64_t B, int64_t V, int dtype, float temperature, int top_k, uint64_t seed,
                       const int* step_dev, int64_t* ids_out, cudaStream_t stream) {
  if (B == 0) return B200_OK;
  if (V <= 0 || V > 0x7fffffff || B > 0x7fffffff || !(temperature > 0.f) || top_k < 0) return B200_ERR_BAD_ARGUMENT;
  const float inv_t = 1.0f / temperature;
  switch (dtype) {
    case B200_F32: sample_rows_kernel<float><<<(unsigned)B, kSampleThreads, 0, stream>>>((const float*)logits, ld, (int)V, inv_t, top_k, seed, step_dev, ids_out); break;
    case B200_F16: sample_rows_kernel<__half><<<(unsigned)B, kSampleThreads, 0, stream>>>((const __half*)logits, ld, (int)V, inv_t, top_k, seed, step_dev, ids_out); break;
    case B200_BF16:
      sample_rows_kernel<__nv_bfloat16><<<(unsigned)B, kSampleThreads, 0, stream>>>((const __nv_bfloat16*)logits, ld, (int)V, inv_t, top_k, seed, step_dev, ids_out);
      break;
    default: return B200_ERR_BAD_ARGUMENT;
  }
  note_launches(1);
  return status_from_cuda(cudaGetLastError());
}

}  // namespace b200
