// Causal attention with online softmax over 64-key blocks (fp16 operands, fp32 statistics): the
// generic kernel (any storage type, head size 16..256, any alignment) on mma.sync tensor-core
// instructions, and one for aligned float32 rows of head sizes up to 64 that fetches ahead.  Most
// 16-bit calls are routed to the tcgen05/TMA kernels instead (launch_attention_sm100).
//
// One CTA = 64 query rows of one (batch, head); 4 warps x 16 rows.  Q, K, V are read through
// (batch, head, row) element strides, so the fused [tokens, 3*hidden] output of the c_attn
// projection is consumed in place and the result is written straight into [batch, seq, hidden].
// Inputs of any storage type are rounded to fp16 when staged in shared memory, P is rounded to
// fp16 relative to the running maximum of each 64-key block and the running maximum and
// denominator are fp32 -- the arithmetic of the reference's flash_attention_v1 kernel.  Key
// blocks that the causal mask removes entirely are skipped (they contribute exact zeros).
#include <atomic>

#include "common.cuh"
#include "mma_sync.cuh"

namespace b200 {
namespace attn {

using warp_mma::cp_async16, warp_mma::cp_async_commit, warp_mma::cp_async_wait;

constexpr int BLOCK = 64;  // query rows per CTA == keys per block
constexpr int NUM_WARPS = 4;
constexpr int PAD = 8;  // halves of padding per shared-memory row (keeps ldmatrix conflict-free)

struct Strides {
  int64_t b, h, l;
};

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// exp for the softmax: correctly-rounded-ish expf when the storage type is fp32 (the 1e-4 parity
// path: a fast exp flips too many fp16 roundings of P), the ex2-based intrinsic otherwise.
template <typename TIn>
__device__ __forceinline__ float softmax_exp(float x) {
  if constexpr (sizeof(TIn) == 4) {
    return expf(x);
  } else {
    return __expf(x);
  }
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
  __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&h);
}

// Stage rows [row0, row0+64) x D of one (batch, head) slice into shared memory as fp16; rows >= L are zero.
template <int D, typename TIn>
__device__ __forceinline__ void stage_tile(__half* dst, const TIn* src, int64_t row_stride, int row0, int L, bool vec) {
  constexpr int LDS = D + PAD;
  constexpr int VPR = D / 8;  // 8-element vectors per row
  for (int i = threadIdx.x; i < BLOCK * VPR; i += NUM_WARPS * 32) {
    const int r = i / VPR, c = (i % VPR) * 8;
    float f[8];
    if (row0 + r < L) {
      const TIn* p = src + (int64_t)(row0 + r) * row_stride + c;
      if (vec) {
        load8(p, f);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = to_float(p[j]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) f[j] = 0.f;
    }
    store8(dst + r * LDS + c, f);
  }
}

// One 64-key step of a warp's 16 rows: S = Q K^T, softmax against the running maximum, O += P V.  qf: the rows' fragments (head
// sizes up to 64), or sQ_lane their place in shared memory; sK_lane, sV_lane: the lane's ldmatrix addresses in the block's tiles.
template <int D, typename TIn>
__device__ __forceinline__ void key_step(const uint32_t (&qf)[D <= 64 ? D / 16 : 1][4], uint32_t sQ_lane, uint32_t sK_lane, uint32_t sV_lane, float scale,
                                         bool diagonal, int k0, const int (&row_g)[2], int t4, float (&o)[D / 8][4], float (&m_run)[2], float (&l_run)[2]) {
  constexpr int LDS = D + PAD;
  // S = Q K^T  (16 rows x 64 keys per warp)
  float s[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks) {
    uint32_t a[4];
    if constexpr (D <= 64) {
      a[0] = qf[ks][0], a[1] = qf[ks][1], a[2] = qf[ks][2], a[3] = qf[ks][3];
    } else {
      ldmatrix_x4(a, sQ_lane + ks * 32);
    }
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      uint32_t bfr[4];
      ldmatrix_x4(bfr, sK_lane + (uint32_t)((np * 16 * LDS + ks * 16) * 2));
      mma_16816(s[2 * np], a, bfr[0], bfr[1]);
      mma_16816(s[2 * np + 1], a, bfr[2], bfr[3]);
    }
  }

  // scale, causal mask, block maximum
  float bm[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = e >> 1;
      float x = __fmul_rn(s[nt][e], scale);  // (rounded before the maximum is subtracted: no fused multiply-add)
      if (diagonal && row_g[r] < k0 + nt * 8 + t4 * 2 + (e & 1)) x = -INFINITY;
      s[nt][e] = x;
      bm[r] = fmaxf(bm[r], x);
    }
  }
  float mult[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    bm[r] = fmaxf(bm[r], __shfl_xor_sync(0xffffffffu, bm[r], 1));
    bm[r] = fmaxf(bm[r], __shfl_xor_sync(0xffffffffu, bm[r], 2));
    const float m_new = fmaxf(m_run[r], bm[r]);
    mult[r] = softmax_exp<TIn>(m_run[r] - m_new);
    m_run[r] = m_new;
  }
  float psum[2] = {0.f, 0.f};
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = e >> 1;
      const float p = softmax_exp<TIn>(s[nt][e] - m_run[r]);
      s[nt][e] = p;
      psum[r] += p;
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    psum[r] += __shfl_xor_sync(0xffffffffu, psum[r], 1);
    psum[r] += __shfl_xor_sync(0xffffffffu, psum[r], 2);
    l_run[r] = l_run[r] * mult[r] + psum[r];
  }
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
    o[i][0] *= mult[0], o[i][1] *= mult[0];
    o[i][2] *= mult[1], o[i][3] *= mult[1];
  }

  // O += P V   (P rounded to fp16)
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    uint32_t a[4];
    a[0] = pack_half2(s[2 * kk][0], s[2 * kk][1]);
    a[1] = pack_half2(s[2 * kk][2], s[2 * kk][3]);
    a[2] = pack_half2(s[2 * kk + 1][0], s[2 * kk + 1][1]);
    a[3] = pack_half2(s[2 * kk + 1][2], s[2 * kk + 1][3]);
#pragma unroll
    for (int dp = 0; dp < D / 16; ++dp) {
      uint32_t bfr[4];
      ldmatrix_x4_trans(bfr, sV_lane + (uint32_t)((kk * 16 * LDS + dp * 16) * 2));
      mma_16816(o[2 * dp], a, bfr[0], bfr[1]);
      mma_16816(o[2 * dp + 1], a, bfr[2], bfr[3]);
    }
  }
}

// Normalise, stage the CTA's rows in shared memory, then store them with wide accesses.
template <int D, int WARPS, typename TOut>
__device__ __forceinline__ void store_rows(uint8_t* smem_raw, const float (&o)[D / 8][4], const float (&l_run)[2], int warp, int g, int t4, int q0, int L,
                                           TOut* op, int64_t so_l, int vec_out) {
  __syncthreads();
  constexpr int LDO = D + (sizeof(TOut) == 4 ? 4 : 8);
  TOut* sO = reinterpret_cast<TOut*>(smem_raw);
  const float inv_l[2] = {1.0f / l_run[0], 1.0f / l_run[1]};
#pragma unroll
  for (int i = 0; i < D / 8; ++i) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      TOut* p = sO + (warp * 16 + g + r * 8) * LDO + i * 8 + t4 * 2;
      p[0] = from_float<TOut>(o[i][2 * r] * inv_l[r]);
      p[1] = from_float<TOut>(o[i][2 * r + 1] * inv_l[r]);
    }
  }
  __syncthreads();
  constexpr int VPR = D / 8;
  for (int i = threadIdx.x; i < WARPS * 16 * VPR; i += WARPS * 32) {
    const int r = i / VPR, c = (i % VPR) * 8;
    if (q0 + r < L) {
      TOut* dst = op + (int64_t)(q0 + r) * so_l + c;
      const TOut* src = sO + r * LDO + c;
      if (vec_out) {
        if (sizeof(TOut) == 4) {
          *reinterpret_cast<float4*>(dst) = *reinterpret_cast<const float4*>(src);
          *reinterpret_cast<float4*>(dst + 4) = *reinterpret_cast<const float4*>(src + 4);
        } else {
          *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[j] = src[j];
      }
    }
  }
}

template <int D, typename TIn, typename TOut>
__global__ void __launch_bounds__(NUM_WARPS * 32)
attention_kernel(const TIn* __restrict__ q, const TIn* __restrict__ k, const TIn* __restrict__ v, TOut* __restrict__ out,
                 int NH, int L, Strides sq, Strides sk, Strides sv, Strides so, float scale, int vec_in, int vec_out) {
  constexpr int LDS = D + PAD;
  constexpr bool Q_IN_REGS = D <= 64;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __half* sQ = reinterpret_cast<__half*>(smem_raw);
  __half* sK = sQ + BLOCK * LDS;
  __half* sV = sK + BLOCK * LDS;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int n_qblocks = (L + BLOCK - 1) / BLOCK;
  const int qb = n_qblocks - 1 - (int)blockIdx.x;  // longest rows first
  const int bh = blockIdx.y;
  const int b = bh / NH, h = bh % NH;
  const TIn* qp = q + (int64_t)b * sq.b + (int64_t)h * sq.h;
  const TIn* kp = k + (int64_t)b * sk.b + (int64_t)h * sk.h;
  const TIn* vp = v + (int64_t)b * sv.b + (int64_t)h * sv.h;
  const int q0 = qb * BLOCK;

  stage_tile<D, TIn>(sQ, qp, sq.l, q0, L, vec_in);
  __syncthreads();

  const uint32_t sQ_u = (uint32_t)__cvta_generic_to_shared(sQ);
  const uint32_t sK_u = (uint32_t)__cvta_generic_to_shared(sK);
  const uint32_t sV_u = (uint32_t)__cvta_generic_to_shared(sV);
  // per-lane ldmatrix offsets (bytes)
  const uint32_t q_off = (uint32_t)(((warp * 16 + (lane & 15)) * LDS + (lane >> 4) * 8) * 2);
  const uint32_t k_off = (uint32_t)((((lane & 7) + ((lane >> 4) << 3)) * LDS + ((lane >> 3) & 1) * 8) * 2);
  const uint32_t v_off = (uint32_t)((((lane & 7) + ((lane >> 3) & 1) * 8) * LDS + (lane >> 4) * 8) * 2);

  uint32_t qf[Q_IN_REGS ? D / 16 : 1][4];
  if constexpr (Q_IN_REGS) {
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) ldmatrix_x4(qf[ks], sQ_u + q_off + ks * 32);
  }

  float o[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY};
  float l_run[2] = {0.f, 0.f};
  const int row_g[2] = {q0 + warp * 16 + g, q0 + warp * 16 + g + 8};

  for (int kb = 0; kb <= qb; ++kb) {
    const int k0 = kb * BLOCK;
    __syncthreads();  // previous block's K/V fully consumed
    stage_tile<D, TIn>(sK, kp, sk.l, k0, L, vec_in);
    stage_tile<D, TIn>(sV, vp, sv.l, k0, L, vec_in);
    __syncthreads();

    key_step<D, TIn>(qf, sQ_u + q_off, sK_u + k_off, sV_u + v_off, scale, kb == qb, k0, row_g, t4, o, m_run, l_run);
  }

  store_rows<D, NUM_WARPS, TOut>(smem_raw, o, l_run, warp, g, t4, q0, L, out + (int64_t)b * so.b + (int64_t)h * so.h, so.l, vec_out);
}

// Float32 rows of head sizes up to 64 at 16-byte addresses: the same arithmetic (key_step), another way in.  attention_kernel loads a
// block, waits for it, converts it and only then works: one latency of L2 or HBM per 64 keys, and at 16 x 300 tokens twice the time
// of the work itself.  Here the next block comes by cp.async while this one is worked on, as float32 into a place of its own, and
// each thread converts what it has fetched; with two pairs of fp16 tiles that takes one barrier per block instead of two.  Blocks
// masked for all of a warp's rows are left out warp by warp, and only the warp's diagonal blocks are masked.  12 heads of 64, fp16 out,
// us, attention_kernel | this: 1 x 300 tokens 17.0 | 9.4, 16 x 300 40.0 | 24.1, 64 x 300 202 | 95, 8 x 1024 231 | 81, 16 x 2048 1389 |
// 535.  What is left is the instructions of the exponentials, the conversions and mma.sync.  Where four CTAs, or two of eight warps, share
// an SM the registers end at 128, and heads of 64 spill 16 to 24 bytes per thread, heads of 32 with one pair of tiles 8.
template <int D, int WARPS, int BUFS, typename TOut>
struct F32Cfg {
  static constexpr int ROWS = WARPS * 16, THREADS = WARPS * 32, LDS = D + PAD;
  static constexpr int RAW = 2 * BLOCK * D * 4;        // one block's keys and values as they come (float32)
  static constexpr int TILES = 2 * BLOCK * LDS * 2;    // and as fp16 tiles (BUFS of these)
  static constexpr int LDO = D + (sizeof(TOut) == 4 ? 4 : 8);
  static constexpr int SMEM = RAW + BUFS * TILES;
  static_assert(ROWS * LDS * 2 <= TILES && ROWS * LDO * (int)sizeof(TOut) <= SMEM, "Q lies in the last pair of tiles, the output over everything");
};

template <int D, int WARPS, int BUFS, typename TOut>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : (BUFS == 1 ? 4 : 3))
attention_f32_kernel(const float* q, const float* k, const float* v, TOut* out, int BH, int NH, int L, Strides sq, Strides sk, Strides sv, Strides so,
                     float scale, int vec_out) {
  using C = F32Cfg<D, WARPS, BUFS, TOut>;
  constexpr int LDS = C::LDS, CHUNKS = D / 4;  // 16-byte pieces of a float32 row
  static_assert(C::THREADS % CHUNKS == 0 && BLOCK * CHUNKS % C::THREADS == 0, "every thread fetches the same number of pieces");
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const uint32_t raw_u = (uint32_t)__cvta_generic_to_shared(smem_raw);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t4 = lane & 3;
  const int n_qtiles = (L + C::ROWS - 1) / C::ROWS;
  const int qt = n_qtiles - 1 - (int)(blockIdx.x / (unsigned)BH);  // longest rows first
  const int bh = (int)(blockIdx.x % (unsigned)BH);
  const int b = bh / NH, h = bh % NH;
  const float* qp = q + (int64_t)b * sq.b + (int64_t)h * sq.h;
  const float* kp = k + (int64_t)b * sk.b + (int64_t)h * sk.h;
  const float* vp = v + (int64_t)b * sv.b + (int64_t)h * sv.h;
  const int q0 = qt * C::ROWS;
  const int n_kb = (min(q0 + C::ROWS, L) + BLOCK - 1) / BLOCK;

  // A thread fetches, and later converts, the same 16-byte pieces: between the two it waits for its own copies only.
  constexpr int STEP = C::THREADS / CHUNKS;  // rows that the CTA fetches at a time
  const int my_row = (int)threadIdx.x / CHUNKS, my_col = (int)threadIdx.x % CHUNKS * 4;
  const float *kt = kp + (int64_t)my_row * sk.l + my_col, *vt = vp + (int64_t)my_row * sv.l + my_col;  // the next row to fetch
  auto fetch = [&](int kb) {
#pragma unroll
    for (int j = 0; j < BLOCK / STEP; ++j) {
      const bool ok = kb * BLOCK + j * STEP + my_row < L;  // (the rest is zero-filled)
      cp_async16(raw_u + (threadIdx.x + j * C::THREADS) * 16, ok ? kt : kp, ok);
      cp_async16(raw_u + C::RAW / 2 + (threadIdx.x + j * C::THREADS) * 16, ok ? vt : vp, ok);
      kt += STEP * sk.l, vt += STEP * sv.l;
    }
    cp_async_commit();
  };
  pdl_launch_dependents();
  pdl_wait();
  fetch(0);
  __half* sQ = reinterpret_cast<__half*>(smem_raw + C::RAW + (BUFS - 1) * C::TILES);
  for (int i = threadIdx.x; i < C::ROWS * (D / 8); i += C::THREADS) {
    const int r = i / (D / 8), c = i % (D / 8) * 8;
    float f[8] = {};
    if (q0 + r < L) load8(qp + (int64_t)(q0 + r) * sq.l + c, f);
    store8(sQ + r * LDS + c, f);
  }
  __syncthreads();
  uint32_t qf[D / 16][4];
#pragma unroll
  for (int ks = 0; ks < D / 16; ++ks)
    ldmatrix_x4(qf[ks], (uint32_t)__cvta_generic_to_shared(sQ) + (uint32_t)(((warp * 16 + (lane & 15)) * LDS + (lane >> 4) * 8) * 2) + ks * 32);

  const uint32_t k_off = (uint32_t)((((lane & 7) + ((lane >> 4) << 3)) * LDS + ((lane >> 3) & 1) * 8) * 2);
  const uint32_t v_off = (uint32_t)((((lane & 7) + ((lane >> 3) & 1) * 8) * LDS + (lane >> 4) * 8) * 2);
  float o[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_run[2] = {-INFINITY, -INFINITY};
  float l_run[2] = {0.f, 0.f};
  const int row0 = q0 + warp * 16;
  const int row_g[2] = {row0 + g, row0 + g + 8};

  for (int kb = 0; kb < n_kb; ++kb) {
    const int k0 = kb * BLOCK;
    uint8_t* tiles = smem_raw + C::RAW + (BUFS == 2 ? kb & 1 : 0) * C::TILES;
    cp_async_wait<0>();
    if (BUFS == 1) __syncthreads();  // (two pairs: this one was last read in front of the previous block's barrier)
#pragma unroll
    for (int j = 0; j < BLOCK / STEP; ++j) {
      const int i = (int)threadIdx.x + j * C::THREADS;
      const uint32_t at = (uint32_t)((my_row + j * STEP) * LDS + my_col) * 2;
#pragma unroll
      for (int kv = 0; kv < 2; ++kv) {
        const float4 f = *reinterpret_cast<const float4*>(smem_raw + kv * (C::RAW / 2) + i * 16);
        *reinterpret_cast<uint2*>(tiles + kv * (C::TILES / 2) + at) = make_uint2(pack_half2(f.x, f.y), pack_half2(f.z, f.w));
      }
    }
    if (kb + 1 < n_kb) fetch(kb + 1);
    __syncthreads();
    if (row0 < L && k0 <= row0 + 15) {  // (a block behind a row adds exact zeros: left out)
      const uint32_t t = raw_u + C::RAW + (BUFS == 2 ? kb & 1 : 0) * C::TILES;
      key_step<D, float>(qf, 0u, t + k_off, t + C::TILES / 2 + v_off, scale, k0 + BLOCK > row0, k0, row_g, t4, o, m_run, l_run);
    }
  }
  store_rows<D, WARPS, TOut>(smem_raw, o, l_run, warp, g, t4, q0, L, out + (int64_t)b * so.b + (int64_t)h * so.h, so.l, vec_out);
}

template <int D>
constexpr size_t smem_bytes() {
  size_t in = (size_t)3 * BLOCK * (D + PAD) * 2;
  size_t o = (size_t)BLOCK * (D + 4) * 4;
  return in > o ? in : o;
}

template <int D, int WARPS, int BUFS, typename TOut>
static int launch_f32(const float* q, const float* k, const float* v, TOut* out, int64_t B, int64_t NH, int64_t L, Strides sq, Strides sk, Strides sv,
                      Strides so, float scale, int vec_out, cudaStream_t stream) {
  using C = F32Cfg<D, WARPS, BUFS, TOut>;
  static std::atomic<bool> attr_set[kMaxDevices];  // kernel attributes are per device
  const int slot = device_slot();
  if (slot < 0) return B200_ERR_CUDA;
  if (!attr_set[slot].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(attention_f32_kernel<D, WARPS, BUFS, TOut>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) != cudaSuccess) return B200_ERR_CUDA;
    attr_set[slot].store(true, std::memory_order_release);
  }
  const int64_t tiles = (L + C::ROWS - 1) / C::ROWS * B * NH;
  const bool early = B * L <= 128 || (B * L <= kManyRowsPdl && (L <= BLOCK || (L + BLOCK - 1) / BLOCK * B * NH >= 6 * (int64_t)sm_count()));
  LaunchSetup ls(dim3((unsigned)tiles), dim3(C::THREADS), C::SMEM, stream, 1, pdl_enabled() || early);
  const cudaError_t e = cudaLaunchKernelEx(&ls.cfg, attention_f32_kernel<D, WARPS, BUFS, TOut>, q, k, v, out, (int)(B * NH), (int)NH, (int)L, sq, sk, sv, so, scale, vec_out);
  note_launches(1);
  return status_from_cuda(e);
}

template <int D, typename TIn, typename TOut>
static int launch_typed(const void* q, const void* k, const void* v, void* out, int64_t B, int64_t NH, int64_t L,
                        Strides sq, Strides sk, Strides sv, Strides so, float scale, cudaStream_t stream) {
  constexpr size_t smem = smem_bytes<D>();
  static std::atomic<bool> attr_set[kMaxDevices];  // kernel attributes are per device
  const int slot = device_slot();
  if (slot < 0) return B200_ERR_CUDA;
  if (smem > 48 * 1024 && !attr_set[slot].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(attention_kernel<D, TIn, TOut>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return B200_ERR_CUDA;
    attr_set[slot].store(true, std::memory_order_release);
  }
  auto ok_in = [](const void* p, const Strides& s) {
    const int64_t m = sizeof(TIn) == 4 ? 4 : 8;
    return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && s.b % m == 0 && s.h % m == 0 && s.l % m == 0;
  };
  const int vec_in = ok_in(q, sq) && ok_in(k, sk) && ok_in(v, sv);
  const int64_t mo = sizeof(TOut) == 4 ? 4 : 8;
  const int vec_out = (reinterpret_cast<uintptr_t>(out) & 15) == 0 && so.b % mo == 0 && so.h % mo == 0 && so.l % mo == 0;
  const int64_t n_qblocks = (L + BLOCK - 1) / BLOCK;
  const int64_t bh = B * NH;
  if constexpr (sizeof(TIn) == 4 && D <= 64) {
    // The same bits from each, so the choice may follow the batch.  us, 12 heads of 64, fp16 out, four warps with two pairs of tiles |
    // with one (four CTAs on an SM instead of three) | eight warps: 8 x 300 (480 tiles) 15.6 | 18.7 | 14.4, 16 x 300 (960) 25.0 |
    // 24.1 | 26.1, 256 x 64 (3072) 55.9 | 54.2 | 65.4, 8 x 1024 (1536) 90.9 | 86.7 | 81.0, 16 x 2048 643 | 584 | 535.
    if (vec_in && NH <= 65535 && L <= INT32_MAX - 2 * BLOCK && n_qblocks * bh <= INT32_MAX) {
      auto* run = n_qblocks * bh <= 4 * (int64_t)sm_count() ? launch_f32<D, 4, 2, TOut> : L <= 512 ? launch_f32<D, 4, 1, TOut> : launch_f32<D, 8, 2, TOut>;
      return run((const float*)q, (const float*)k, (const float*)v, (TOut*)out, B, NH, L, sq, sk, sv, so, scale, vec_out, stream);
    }
  }
  if (bh > 65535) {
    // fold very large batch*head counts into several launches of whole batches
    const int64_t b_per = 65535 / NH;
    if (b_per < 1) return B200_ERR_BAD_ARGUMENT;
    for (int64_t b0 = 0; b0 < B; b0 += b_per) {
      const int64_t nb = (B - b0 < b_per) ? B - b0 : b_per;
      int st = launch_typed<D, TIn, TOut>((const TIn*)q + b0 * sq.b, (const TIn*)k + b0 * sk.b, (const TIn*)v + b0 * sv.b,
                                          (TOut*)out + b0 * so.b, nb, NH, L, sq, sk, sv, so, scale, stream);
      if (st != B200_OK) return st;
    }
    return B200_OK;
  }
  dim3 grid((unsigned)n_qblocks, (unsigned)bh);
  attention_kernel<D, TIn, TOut><<<grid, NUM_WARPS * 32, smem, stream>>>((const TIn*)q, (const TIn*)k, (const TIn*)v, (TOut*)out, (int)NH,
                                                                        (int)L, sq, sk, sv, so, scale, vec_in, vec_out);
  note_launches(1);
  return status_from_cuda(cudaGetLastError());
}

template <typename TIn, typename TOut>
static int dispatch_d(int64_t D, const void* q, const void* k, const void* v, void* out, int64_t B, int64_t NH, int64_t L,
                      Strides sq, Strides sk, Strides sv, Strides so, float scale, cudaStream_t stream) {
  switch (D) {
    case 16: return launch_typed<16, TIn, TOut>(q, k, v, out, B, NH, L, sq, sk, sv, so, scale, stream);
    case 32: return launch_typed<32, TIn, TOut>(q, k, v, out, B, NH, L, sq, sk, sv, so, scale, stream);
    case 64: return launch_typed<64, TIn, TOut>(q, k, v, out, B, NH, L, sq, sk, sv, so, scale, stream);
    case 128: return launch_typed<128, TIn, TOut>(q, k, v, out, B, NH, L, sq, sk, sv, so, scale, stream);
    case 256: return launch_typed<256, TIn, TOut>(q, k, v, out, B, NH, L, sq, sk, sv, so, scale, stream);
  }
  return B200_ERR_BAD_ARGUMENT;
}

}  // namespace attn

int launch_attention(const void* q, const void* k, const void* v, void* out, int64_t B, int64_t NH, int64_t L,
                     int64_t D, const int64_t* qs, const int64_t* ks, const int64_t* vs, const int64_t* os, float scale,
                     int in_dtype, int out_dtype, int* status_word, cudaStream_t stream) {
  using namespace attn;
  if (B == 0 || NH == 0 || L == 0) return B200_OK;
  if (L > 0x7fffffffLL - BLOCK) return B200_ERR_BAD_ARGUMENT;
  {
    // tensor-core path for the shapes it covers; everything else takes the generic kernel below
    const int st = launch_attention_sm100(q, k, v, out, B, NH, L, D, qs, ks, vs, os, scale, in_dtype, out_dtype, status_word, stream);
    if (st != B200_ERR_UNSUPPORTED) return st;
  }
  Strides sq{qs[0], qs[1], qs[2]}, sk{ks[0], ks[1], ks[2]}, sv{vs[0], vs[1], vs[2]}, so{os[0], os[1], os[2]};
  if (in_dtype == B200_F32 && out_dtype == B200_F32) return dispatch_d<float, float>(D, q, k, v, out, B, NH, L, sq, sk, sv, so, scale, stream);
  if (in_dtype == B200_F32 && out_dtype == B200_F16) return dispatch_d<float, __half>(D, q, k, v, out, B, NH, L, sq, sk, sv, so, scale, stream);
  if (in_dtype == B200_F16 && out_dtype == B200_F16) return dispatch_d<__half, __half>(D, q, k, v, out, B, NH, L, sq, sk, sv, so, scale, stream);
  if (in_dtype == B200_BF16 && out_dtype == B200_BF16) return dispatch_d<__nv_bfloat16, __nv_bfloat16>(D, q, k, v, out, B, NH, L, sq, sk, sv, so, scale, stream);
  return B200_ERR_BAD_ARGUMENT;
}

}  // namespace b200
