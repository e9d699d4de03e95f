// Causal flash attention on the 5th-generation tensor cores: fp16 or bf16 storage, head sizes 32 and 64 (32 columns are zero-filled by
// the loads).  The arithmetic is that of attention_sm100.cu (64-key blocks, P in fp16 relative to the running maximum of its block:
// kernels.py:417-474 of the reference), bit for bit; what differs is how the work sits on an SM.
//
// A block of a tile is one chain: S = Q K^T, scores to registers, maximum, exponentials, P, rescaled O, P V.  An SM keeps FOUR
// query tiles of 128 rows in flight, one per CTA, so that four such chains fill each other's waits:
//   warp 0      one thread loads (TMA) and issues the MMAs; what it waits for next is always the one thing that can happen next
//   warps 1-4   softmax, one thread per query row: nothing to exchange between threads
// Tensor memory is what limits the number of tiles (512 columns an SM): 64 columns of S, whose first 32 take P once the scores are in
// registers (P V reads its A operand from there: no shared-memory round trip, and 16 KB less per CTA), and 64 columns of O.  S of
// block j + 1 is therefore issued when P V of block j is done; the other three CTAs use that time.
// Shared memory: Q (one buffer: the next item's tile is on its way as soon as the item's last S is computed) and two stages of K and V.
//
// What bounds it: the chain of a block, 2900 cycles of which 1400 are the two MMAs and their hand-overs, 750 the exponentials, 320 the
// maximum, 310 the rescaling of O; four chains an SM come to 725 cycles a block, where the special-function unit needs 512 for its
// 8192 exponentials (54 % busy).  Two tiles an SM with two threads per row (attention_sm100.cu): 1040 cycles.  us, fp16 | bf16, before ->
// now, batch x heads x rows x columns, ten calls on views of a fused projection after a pause (calls without end, the clock pulled down):
// 16 x 12 x 2048 x 64 229 -> 184 | 252 -> 199 (248 -> 208 | 263 -> 218), 64 x 12 x 300 x 64 48 -> 36 | 51 -> 39 (46 -> 37 | 49 -> 38; in a replayed graph
// 42 -> 31 | 46 -> 34), 16 x 16 x 1024 x 64 95 -> 74 | 103 -> 82; 16 x 12 x 1024 x 32 159 -> 55 | 157 -> 61 (generic kernel before).
// Tried: three tiles with tensor memory for S, P and O apart, S issued a block ahead (189 us at 16 x 12 x 2048: the three tiles' exponentials
// fall together, 1450 cycles each, and nothing overlaps them); the same with a turn per scheduler for the exponentials (231) and with two
// threads per row (222: 72 registers, spills).
#include <atomic>

#include "attention_sm100.cuh"

namespace b200 {
namespace attn_causal {

using namespace attn100;

constexpr int HEAD = 64;  // columns of the tiles
constexpr int Q_BYTES = BLOCK_M * HEAD * 2;
constexpr int KV_BYTES = BLOCK_N * HEAD * 2;  // each of K and V
constexpr int STAGE_BYTES = 2 * KV_BYTES;
constexpr int NUM_THREADS = 32 * 5;
constexpr int CTAS_PER_SM = 4;
constexpr int CTRL_BYTES = 128;
constexpr int SMEM_BYTES = 1024 + Q_BYTES + 2 * STAGE_BYTES + CTRL_BYTES;
static_assert(CTAS_PER_SM * (SMEM_BYTES + 1024) <= 228 * 1024, "shared memory budget");
constexpr int TMEM_COLS = 128;  // S (P in its first half), O

struct Params {
  void* out;
  int64_t so_b, so_h, so_l;
  int B, NH, L, D;
  float scale_log2e;  // softmax scale times log2(e)
  int out_vec32;      // output rows may be written with 32-byte stores
  int q_head_inner, k_head_inner, v_head_inner;  // tensor map dimension order is {D, head, row, batch} instead of {D, row, head, batch}
  int* status_word;
};

// The items of one CTA, longest first.  (Dealt to and fro, so that who got a long one gets a short one next, the busiest CTA had 4 %
// more than the mean instead of 16, and it took 4 % longer: a CTA that ends early leaves its share of the SM to the other three, and
// neighbours read the same keys.)
struct Deal {
  int64_t idx, n_items;
  __device__ __forceinline__ explicit Deal(int64_t n) : idx(blockIdx.x), n_items(n) {}
  __device__ __forceinline__ bool any() const { return idx < n_items; }
  __device__ __forceinline__ void next() { idx += gridDim.x; }
};

struct Item {
  int b, h, q0, q_end, nblk;
};
__device__ __forceinline__ Item decode_item(int64_t idx, int bh_total, int n_qt, int NH, int L) {
  const int qt = n_qt - 1 - (int)(idx / bh_total);
  const int bh = (int)(idx % bh_total);
  Item it;
  it.b = bh / NH;
  it.h = bh % NH;
  it.q0 = qt == 0 ? 0 : tile_end(qt - 1, n_qt, L);
  it.q_end = tile_end(qt, n_qt, L);
  it.nblk = (it.q_end - 1) / BLOCK_N + 1;
  return it;
}

// p = exp(s - max) of 32 scores, rounded to fp16 pairs; returns the sum of the unrounded values (even and odd ones apart).
__device__ __forceinline__ float exponentials(const uint32_t (&v)[32], float scale_log2e, float m, uint32_t (&w)[16]) {
  float s0 = 0.f, s1 = 0.f;
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    const float p0 = ex2f(fmaf(__uint_as_float(v[i]), scale_log2e, -m));
    const float p1 = ex2f(fmaf(__uint_as_float(v[i + 1]), scale_log2e, -m));
    s0 += p0, s1 += p1;
    const __half2 h = __floats2half2_rn(p0, p1);
    w[i / 2] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return s0 + s1;
}
// Maximum of 32 scores, those beyond `lim` (this row's last visible one) set to -inf if `masked`.
__device__ __forceinline__ float maximum(uint32_t (&v)[32], bool masked, int lim) {
  float m0 = -INFINITY, m1 = -INFINITY;
  if (masked) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if (i > lim) v[i] = 0xff800000u;
      m0 = fmaxf(m0, __uint_as_float(v[i]));
    }
    return m0;
  }
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    m0 = fmax3(m0, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
    m1 = fmax3(m1, __uint_as_float(v[i + 2]), __uint_as_float(v[i + 3]));
  }
  return fmaxf(m0, m1);
}

template <typename T>
__global__ void __launch_bounds__(NUM_THREADS, CTAS_PER_SM)
causal_attention_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                        Params p, uint32_t idesc_s, uint32_t idesc_pv) {
  constexpr bool IS_FP16 = DType<T>::code == B200_F16;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t smem_q = base, smem_kv = smem_q + Q_BYTES;  // [2]{K[64][64], V[64][64]}
  uint8_t* ctrl = smem_raw + (base - raw) + Q_BYTES + 2 * STAGE_BYTES;
  const uint32_t bars = smem_u32(ctrl);
  const uint32_t bar_q_full = bars;         // Q of an item has landed
  const uint32_t bar_kv_full = bars + 8;    // [2] K and V of a block have landed
  const uint32_t bar_s_full = bars + 24;    // S of a block is in tensor memory (and P V of the block before it is done)
  const uint32_t bar_p_full = bars + 32;    // P of a block is in tensor memory, O rescaled, V (bf16 storage) converted
  const uint32_t bar_pv_done = bars + 40;   // P V of a block is done: its K and V are free, O is current
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ctrl + 48);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(ctrl + 56);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int n_qt = (p.L + BLOCK_M - 1) / BLOCK_M;
  const int bh_total = p.B * p.NH;
  Deal deal((int64_t)n_qt * bh_total);
  auto item_at = [&](const Deal& d) { return decode_item(d.idx, bh_total, n_qt, p.NH, p.L); };

  if (threadIdx.x == 0) {
    mbar_init(bar_q_full, 1);
    mbar_init(bar_kv_full, 1);
    mbar_init(bar_kv_full + 8, 1);
    mbar_init(bar_s_full, 1);
    mbar_init(bar_p_full, 4);
    mbar_init(bar_pv_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_s = *tmem_slot, tmem_o = tmem_s + BLOCK_N;
  // set-up done (own shared and tensor memory only); global memory from here on
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    if (elect_one()) {
      auto load_q = [&](const Item& it) {
        mbar_arrive_expect_tx(bar_q_full, Q_BYTES);
        tma_load_4d(smem_q, &map_q, bar_q_full, 0, p.q_head_inner ? it.h : it.q0, p.q_head_inner ? it.q0 : it.h, it.b);
      };
      // K and V of the next block in the order of the work, whose stage is free
      Deal load_deal = deal;
      Item load_it = item_at(load_deal);
      int load_j = 0;
      uint32_t loads = 0;
      auto load_kv = [&]() {
        if (!load_deal.any()) return;
        const uint32_t dst = smem_kv + (loads & 1) * STAGE_BYTES, bar = bar_kv_full + 8 * (loads & 1);
        const int key = load_j * BLOCK_N;
        mbar_arrive_expect_tx(bar, STAGE_BYTES);
        tma_load_4d(dst, &map_k, bar, 0, p.k_head_inner ? load_it.h : key, p.k_head_inner ? key : load_it.h, load_it.b);
        tma_load_4d(dst + KV_BYTES, &map_v, bar, 0, p.v_head_inner ? load_it.h : key, p.v_head_inner ? key : load_it.h, load_it.b);
        ++loads;
        if (++load_j == load_it.nblk) {
          load_deal.next(), load_j = 0;
          if (load_deal.any()) load_it = item_at(load_deal);
        }
      };
      uint32_t n = 0, qn = 0;  // blocks and items so far
      bool alive = true;
      load_q(load_it);
      load_kv();
      const int k_steps = (p.D + 15) / 16;
      for (; alive && deal.any(); deal.next(), ++qn) {
        const Item it = item_at(deal);
        Deal after = deal;
        after.next();
        if (!mbar_wait(bar_q_full, qn & 1, abort_flag, p.status_word, 15)) break;
        for (int j = 0; j < it.nblk; ++j, ++n) {
          const uint32_t stage = smem_kv + (n & 1) * STAGE_BYTES;
          alive = false;
          // P V of the block before has read its P (where S goes) and its stage (where the next block's K and V go)
          if (n > 0 && !mbar_wait(bar_pv_done, (n - 1) & 1, abort_flag, p.status_word, 19)) break;
          if (!mbar_wait(bar_kv_full + 8 * (n & 1), (n >> 1) & 1, abort_flag, p.status_word, 13)) break;
          tc_fence_after();
          {
            const uint64_t da = desc_kmajor(smem_q), db = desc_kmajor(stage);
            for (int k = 0; k < k_steps; ++k) umma_f16(tmem_s, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc_s, (uint32_t)(k != 0));
          }
          umma_commit(bar_s_full);
          load_kv();
          if (j + 1 == it.nblk && after.any()) {
            // the item's last S: behind it Q is free
            if (!mbar_wait(bar_s_full, n & 1, abort_flag, p.status_word, 12)) break;
            load_q(item_at(after));
          }
          if (!mbar_wait(bar_p_full, n & 1, abort_flag, p.status_word, 16)) break;
          tc_fence_after();
          const uint64_t db = desc_mnmajor(stage + KV_BYTES, 1024);
#pragma unroll
          for (int k = 0; k < BLOCK_N / 16; ++k)  // A: +16 keys = 8 columns of tensor memory; B: +16 keys = two 8-key groups = +2048 bytes
            umma_f16_ts(tmem_o, tmem_s + (uint32_t)(8 * k), db + (uint64_t)(128 * k), idesc_pv, (uint32_t)((j | k) != 0));
          umma_commit(bar_pv_done);
          alive = true;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ softmax warps: one thread per query row
    const int quarter = warp & 3;  // tensor-memory lanes [32 * quarter, +32) are this warp's rows
    const int r_in_tile = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_addr = tmem_s + lane_addr, o_addr = tmem_o + lane_addr;
    uint32_t n = 0;
    bool alive = true;
    for (; alive && deal.any(); deal.next()) {
      const Item it = item_at(deal);
      const int row = it.q0 + r_in_tile;
      const int warp_row0 = it.q0 + quarter * 32;   // first query row of this warp
      const bool warp_live = warp_row0 < it.q_end;  // a warp whose 32 rows all lie beyond the tile's end only keeps the handshakes going
      float m_run = -INFINITY, l_lo = 0.f, l_hi = 0.f;  // denominators of the blocks' first and last 32 keys
      for (int j = 0; j < it.nblk; ++j, ++n) {
        if (!mbar_wait(bar_s_full, n & 1, abort_flag, p.status_word, 18)) {
          alive = false;
          break;
        }
        tc_fence_after();
        const int k0 = j * BLOCK_N;
        const bool live = warp_live && k0 <= warp_row0 + 31;  // (warp-uniform) else every key is masked for all its rows
        float mult = 1.f;
        if (live) {
          uint32_t lo[32], hi[32];
          tmem_ld_32x32(s_addr, lo);
          tmem_ld_32x32(s_addr + 32, hi);
          tmem_ld_wait();
          // maximum of the raw scores (the scale is positive, so it commutes with max); a masked score is -inf: 2^-inf = 0
          const float bm = fmaxf(maximum(lo, k0 + 31 > warp_row0, row - k0), maximum(hi, k0 + 63 > warp_row0, row - k0 - 32));
          const float m_new = fmaxf(m_run, bm * p.scale_log2e);  // running maximum, in log2 units
          mult = ex2f(m_run - m_new);
          m_run = m_new;
          uint32_t w[16];
          const float s_lo = exponentials(lo, p.scale_log2e, m_new, w);
          tmem_st_32x16(s_addr, w);
          const float s_hi = exponentials(hi, p.scale_log2e, m_new, w);
          tmem_st_32x16(s_addr + 16, w);
          l_lo = l_lo * mult + s_lo, l_hi = l_hi * mult + s_hi;
        } else if (warp_live) {
          // masked for every row of the warp: P = 0 (rows beyond L may keep whatever is there: nothing reads their output)
          const uint32_t none[16] = {};
          tmem_st_32x16(s_addr, none);
          tmem_st_32x16(s_addr + 16, none);
        }
        if constexpr (!IS_FP16) {
          // bf16 storage: V -> fp16 in place, 64 bytes per softmax thread (the swizzle is address-agnostic)
          const uint32_t vaddr = smem_kv + (n & 1) * STAGE_BYTES + KV_BYTES + (uint32_t)(threadIdx.x - 32) * 16u;
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint32_t w4[4];
            ld_shared_v4(vaddr + g * 2048, w4);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 f2 = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w4[i]));
              const __half2 h2 = __floats2half2_rn(f2.x, f2.y);
              w4[i] = *reinterpret_cast<const uint32_t*>(&h2);
            }
            st_shared_v4(vaddr + g * 2048, w4[0], w4[1], w4[2], w4[3]);
          }
        }
        // o = o * exp(m_old - m_new), unless no row's maximum moved (S of this block was issued behind the last P V: O is current)
        if (j > 0 && live && __any_sync(0xffffffffu, mult != 1.0f)) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t a[32];
            tmem_ld_32x32(o_addr + c * 32, a);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) a[i] = __float_as_uint(__uint_as_float(a[i]) * mult);
            tmem_st_32x32(o_addr + c * 32, a);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        if constexpr (!IS_FP16) fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_p_full);
      }
      if (!alive) break;
      // the last block's P V, then normalise and store the row
      if (!mbar_wait(bar_pv_done, (n - 1) & 1, abort_flag, p.status_word, 21)) break;
      tc_fence_after();
      if (warp_live) {  // (warp-uniform: the tensor-memory load below is a warp-wide instruction)
        const float inv = 1.0f / (l_lo + l_hi);
        T* dst = reinterpret_cast<T*>(p.out) + (int64_t)it.b * p.so_b + (int64_t)it.h * p.so_h + (int64_t)row * p.so_l;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int room = p.D - c * 32;  // columns of these 32 that exist (a multiple of 8)
          if (room <= 0) break;
          uint32_t a[32];
          tmem_ld_32x32(o_addr + c * 32, a);
          tmem_ld_wait();
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = pack_out<T>(__uint_as_float(a[2 * i]) * inv, __uint_as_float(a[2 * i + 1]) * inv);
          if (row < it.q_end) {
            if (p.out_vec32 && room >= 32) {
              st_global_v8(dst + c * 32, &w[0]);
              st_global_v8(dst + c * 32 + 16, &w[8]);
            } else {
#pragma unroll
              for (int g = 0; g < 4; ++g)
                if (g * 8 < room) *reinterpret_cast<uint4*>(dst + c * 32 + g * 8) = make_uint4(w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]);
            }
          }
        }
      }
      // (this warp's reads of O are ordered before its next arrival on bar_p_full, which is what lets the next item's first P V
      // overwrite O)
      tc_fence_before();
    }
  }

  // ------------------------------------------------------------ teardown
  __syncwarp();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) {
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_s, TMEM_COLS);
  }
}

}  // namespace attn_causal

int launch_causal_attention_sm100(const void* q, const void* k, const void* v, void* out, int64_t B, int64_t NH, int64_t L, int64_t D,
                                  const int64_t* qs, const int64_t* ks, const int64_t* vs, const int64_t* os, float scale, int dtype, int* status_word,
                                  cudaStream_t stream) {
  using namespace attn_causal;
  if (D > HEAD || D % 8 || !(scale > 0.f) || (dtype != B200_F16 && dtype != B200_BF16)) return B200_ERR_UNSUPPORTED;
  if (!view_ok(q, qs, B, NH) || !view_ok(k, ks, B, NH) || !view_ok(v, vs, B, NH) || !view_ok(out, os, B, NH)) return B200_ERR_UNSUPPORTED;
  if (B * NH > 0x7fffffffLL || L > 0x7fffff00LL || B > 0x7fffffffLL) return B200_ERR_UNSUPPORTED;
  CUtensorMap mq, mk, mv;
  Params p;
  int st = make_map(&mq, q, B, NH, L, D, qs, BLOCK_M, dtype, &p.q_head_inner);
  if (st == B200_OK) st = make_map(&mk, k, B, NH, L, D, ks, BLOCK_N, dtype, &p.k_head_inner);
  if (st == B200_OK) st = make_map(&mv, v, B, NH, L, D, vs, BLOCK_N, dtype, &p.v_head_inner);
  if (st != B200_OK) return B200_ERR_UNSUPPORTED;  // e.g. strides the tensor map cannot express
  static std::atomic<bool> attr_set[kMaxDevices];  // kernel attributes are per device
  const int slot = device_slot();
  if (slot < 0) return B200_ERR_CUDA;
  if (!attr_set[slot].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(causal_attention_kernel<__half>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess ||
        cudaFuncSetAttribute(causal_attention_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess)
      return B200_ERR_CUDA;
    attr_set[slot].store(true, std::memory_order_release);
  }
  p.out = out;
  p.so_b = os[0], p.so_h = os[1], p.so_l = os[2];
  p.B = (int)B, p.NH = (int)NH, p.L = (int)L, p.D = (int)D;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.out_vec32 = (reinterpret_cast<uintptr_t>(out) & 31) == 0 && os[0] % 16 == 0 && os[1] % 16 == 0 && os[2] % 16 == 0;
  p.status_word = status_word;
  const int64_t n_items = ((L + BLOCK_M - 1) / BLOCK_M) * B * NH;
  int64_t grid = (int64_t)sm_count() * CTAS_PER_SM;
  if (grid > n_items) grid = n_items;
  LaunchSetup ls(dim3((unsigned)grid), dim3(NUM_THREADS), SMEM_BYTES, stream);
  // S = Q K^T in the storage format; P V always fp16 x fp16 (one MMA has one operand format)
  const cudaError_t e = dtype == B200_BF16
                            ? cudaLaunchKernelEx(&ls.cfg, causal_attention_kernel<__nv_bfloat16>, mq, mk, mv, p, idesc(1, 1, 0, BLOCK_N), idesc(0, 0, 1, HEAD))
                            : cudaLaunchKernelEx(&ls.cfg, causal_attention_kernel<__half>, mq, mk, mv, p, idesc(0, 0, 0, BLOCK_N), idesc(0, 0, 1, HEAD));
  note_launches(1);
  return status_from_cuda(e);
}

}  // namespace b200
