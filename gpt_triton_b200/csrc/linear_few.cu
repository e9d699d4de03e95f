// Products of at most 16 bf16 rows around a deferred RMS norm (b200_linear: LN == 3, 4 and 5 of gemm_sm100.cuh), cut along K.
//
// Such a product is the read of its weights.  A block computes 64 columns over one of S ranges of K, the S blocks of 64 columns form a
// cluster, and the eight warps of a block cut its range again, in steps of 32.  Weights go from global memory to the registers of
// mma.sync fragments directly: a dot product does not care about the order of its terms, so the 16 bytes that a lane loads of a row
// are its elements of two k-steps, and the activations are taken in the same order.  The 16-row operand of the MMA is the weights, the
// 8-column one the rows.  Partial sums meet in shared memory, then every rank of the cluster gets some of the rows, whole 64-column
// slices, for the epilogue.
//
// What bounds it: fixed costs of 3 us (hand-over from the kernel in front 0.7-0.9, first load 0.9, two cluster barriers with the sums
// between them 0.9, epilogue 0.3) and the read of the weights behind them at 5.5-6 TB/s; at 9 to 16 rows also the MMAs.  gemm_few_kernel
// computes each sum as one chain of MMAs, K / 16 of them behind one another, on N / 16 to N / 64 SMs.  us per launch in a replayed
// graph of such launches on weights that are not in L2, gemm_few_kernel -> this kernel (HBM alone), N x K, 1 | 16 rows:
//   act(z)  2048 x 2048 6.0 -> 4.1 | 6.0 -> 5.2 (1.3), 8192 x 2048 10.1 -> 8.6 | 10.2 -> 9.9 (5.2), 4096 x 4096 11.2 -> 8.8 | 11.2 -> 9.9 (5.2)
//   x += z  1024 x 4096 9.8 -> 4.6 | 9.9 -> 5.2 (1.3), 2048 x 8192 18.0 -> 9.2 | 18.2 -> 11.0 (5.2), 4096 x 16384 35.8 -> 29.0 | 35.0 -> 30.5 (20.8)
#include "gemm_sm100.cuh"
#include "mma_sync.cuh"

namespace b200 {
namespace {

using namespace sm100;
using warp_mma::mma_bf16;

constexpr int kCols = gemm::NARROW_BN;  // per cluster: a slice of the sums of squares (LN == 4), a block of gate and up columns (LN == 5)
constexpr int kWarps = 8;
constexpr int kStep = 32;               // k per warp and step: four lanes' 16 bytes of every row
constexpr int kPitch = kCols + 4;       // floats per row of a partial tile: the MMA's accumulators land in different banks
constexpr int kMaxSplit = 8;

// 16 bytes of weights: read once and by this block only
__device__ __forceinline__ uint4 ld_weights(const __nv_bfloat16* w) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(w));
  return v;
}
__device__ __forceinline__ void prefetch_l2_bulk(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// MG: groups of eight rows.  Shared memory: kWarps partial tiles of [8 * MG][kPitch] floats, and behind them, for a cluster, what the
// ranks send: [S][8 * MG / S][kPitch].
template <typename OutT, int LN, int MG>
__global__ void __launch_bounds__(32 * kWarps, 2)
linear_few_kernel(const __nv_bfloat16* a, const __nv_bfloat16* __restrict__ w, gemm::EpilogueArgs<OutT> epi, int M, int64_t N, int K, int64_t lda,
                  int64_t ldb) {
  constexpr int ROWS = 8 * MG, TILE = ROWS * kPitch;
  constexpr int kOwn = ROWS / kWarps;  // rows per warp in the epilogue, at most (one block per cluster)
  extern __shared__ __align__(16) float part[];
  float* got = part + kWarps * TILE;
  const int warp = warp_index(), lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int splits = (int)gridDim.x, rank = (int)blockIdx.x;
  const int64_t n0 = (int64_t)blockIdx.y * kCols;
  const int steps = (K + kStep - 1) / kStep;
  const int first = (int)((int64_t)steps * rank / splits), last = (int)((int64_t)steps * (rank + 1) / splits);
  // (L2 is where writes of other SMs meet as well: a prefetch may run ahead of the wait whoever wrote the weights)
  if (threadIdx.x < kCols && n0 + threadIdx.x < N) {
    const int k0 = first * kStep, bytes = (min(last * kStep, K) - k0) * 2;
    if (bytes > 0) prefetch_l2_bulk(w + (n0 + threadIdx.x) * ldb + k0, (uint32_t)bytes);
  }
  pdl_launch_dependents();
  if (splits > 1) cluster_arrive();  // (waited for in front of the first access to another block's shared memory)
  pdl_wait();

  float acc[kCols / 16][MG][4];
#pragma unroll
  for (int i = 0; i < kCols / 16; ++i)
#pragma unroll
    for (int j = 0; j < MG; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
  // (columns beyond the last and rows beyond M: the last one's, not stored)
  const __nv_bfloat16* wbase = w + n0 * ldb + t * 8;
  const int last_col = (int)min((int64_t)kCols, N - n0) - 1;
  auto weights = [&](int i, int k) { return ld_weights(wbase + (int64_t)min(i * 8 + g, last_col) * ldb + k); };
  const __nv_bfloat16* abase = a + t * 8;
  auto rows = [&](int j, int k) { return *reinterpret_cast<const uint4*>(abase + (int64_t)min(j * 8 + g, M - 1) * lda + k); };
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 wv[kCols / 8], av[MG];
  int s = first + warp;
  auto load_rows = [&](bool ok, int k) {
#pragma unroll
    for (int j = 0; j < MG; ++j) av[j] = ok ? rows(j, k) : zero;
  };
  {
    const int k = s * kStep;
    const bool ok = s < last && k + t * 8 < K;  // K is a multiple of 8
    load_rows(ok, k);
#pragma unroll
    for (int i = 0; i < kCols / 8; ++i) wv[i] = ok ? weights(i, k) : zero;
  }
  // the rows of this warp's epilogue: what does not depend on the product is on its way while the weights stream
  const int own = ROWS / splits;  // rows of this block
  float scale[kOwn];
  float2 xr[kOwn], gn = make_float2(0.f, 0.f), fb = gn;
  const int64_t c0 = n0 + (LN == 5 ? lane : 2 * lane), c1 = c0 + (LN == 5 ? 32 : 1);
  const bool in0 = c0 < N, in1 = c1 < N;
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    const int lr = warp + i * kWarps, row = rank * own + lr;
    scale[i] = 0.f;
    xr[i] = make_float2(0.f, 0.f);
    if (lr >= own || row >= M) continue;  // (warp-uniform)
    if (epi.sq_in) {
      float s2 = 0.f;
      for (int j = lane; j < epi.sq_slices; j += 32) s2 += epi.sq_in[(int64_t)j * epi.sq_in_ld + row];
      scale[i] = s2;  // (this lane's part)
    }
    if constexpr (LN == 4) {
      if (in0) xr[i].x = epi.x[row * epi.ld_x + c0];
      if (in1) xr[i].y = epi.x[row * epi.ld_x + c1];
    }
  }
  if constexpr (LN == 4) {
    if (epi.gain) gn = make_float2(in0 ? __ldg(epi.gain + c0) : 0.f, in1 ? __ldg(epi.gain + c1) : 0.f);
  } else {
    if (epi.fbias) fb = make_float2(in0 ? __ldg(epi.fbias + c0) : 0.f, in1 ? __ldg(epi.fbias + c1) : 0.f);
  }

  for (; s < last; s += kWarps) {
    // a register is loaded for the next step as soon as its MMAs have read it: 4 KB of weights in flight per warp
    const int k = (s + kWarps) * kStep;
    const bool ok = s + kWarps < last && k + t * 8 < K;
#pragma unroll
    for (int i = 0; i < kCols / 16; ++i) {
      const uint32_t lo[4] = {wv[2 * i].x, wv[2 * i + 1].x, wv[2 * i].y, wv[2 * i + 1].y}, hi[4] = {wv[2 * i].z, wv[2 * i + 1].z, wv[2 * i].w, wv[2 * i + 1].w};
#pragma unroll
      for (int j = 0; j < MG; ++j) mma_bf16(acc[i][j], lo, av[j].x, av[j].y);
#pragma unroll
      for (int j = 0; j < MG; ++j) mma_bf16(acc[i][j], hi, av[j].z, av[j].w);
      wv[2 * i] = ok ? weights(2 * i, k) : zero;
      wv[2 * i + 1] = ok ? weights(2 * i + 1, k) : zero;
    }
    load_rows(ok, k);
  }

  // accumulator element (column g or g + 8 of its 16, row 2 t or 2 t + 1 of its 8) -> [row][column]
  float* mine = part + warp * TILE;
#pragma unroll
  for (int i = 0; i < kCols / 16; ++i)
#pragma unroll
    for (int j = 0; j < MG; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) mine[(j * 8 + 2 * t + (e & 1)) * kPitch + i * 16 + g + (e >> 1) * 8] = acc[i][j][e];
  __syncthreads();
  if (splits > 1) cluster_wait();
  for (int i = threadIdx.x; i < ROWS * (kCols / 4); i += 32 * kWarps) {
    const int row = i / (kCols / 4), c = i % (kCols / 4) * 4;
    float4 v[kWarps];
#pragma unroll
    for (int j = 0; j < kWarps; ++j) v[j] = *reinterpret_cast<const float4*>(part + j * TILE + row * kPitch + c);
#pragma unroll
    for (int d = kWarps / 2; d > 0; d >>= 1)
#pragma unroll
      for (int j = 0; j < d; ++j) v[j].x += v[j + d].x, v[j].y += v[j + d].y, v[j].z += v[j + d].z, v[j].w += v[j + d].w;
    if (splits > 1) {
      const uint32_t to = mapa_shared(smem_u32(got + (rank * own + row % own) * kPitch + c), (uint32_t)(row / own));
      asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to), "f"(v[0].x), "f"(v[0].y), "f"(v[0].z), "f"(v[0].w) : "memory");
    } else {
      *reinterpret_cast<float4*>(part + row * kPitch + c) = v[0];  // (this thread alone has read these four of the first tile)
    }
  }
  if (splits > 1) cluster_arrive();
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    if (warp + i * kWarps >= own) continue;
    scale[i] = epi.sq_in ? epi.out_scale / sqrtf(warp_sum(scale[i]) / epi.sq_cols + epi.eps) : epi.out_scale;
  }
  if (splits > 1) {
    cluster_wait();  // nobody touches another block's shared memory from here on
  } else {
    __syncthreads();
  }

#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    const int lr = warp + i * kWarps;
    const int64_t row = rank * own + lr;
    if (lr >= own || row >= M) continue;  // (warp-uniform)
    const float* src = (splits > 1 ? got : part) + lr * kPitch;
    const float mult = scale[i];
    const int at0 = LN == 5 ? lane : 2 * lane, at1 = LN == 5 ? lane + 32 : 2 * lane + 1;
    float p0[kMaxSplit], p1[kMaxSplit];
#pragma unroll
    for (int r = 0; r < kMaxSplit; ++r) {
      const bool there = r < splits;
      p0[r] = there ? src[r * own * kPitch + at0] : 0.f, p1[r] = there ? src[r * own * kPitch + at1] : 0.f;
    }
#pragma unroll
    for (int d = kMaxSplit / 2; d > 0; d >>= 1)
#pragma unroll
      for (int r = 0; r < d; ++r) p0[r] += p0[r + d], p1[r] += p1[r + d];
    const float z0 = p0[0], z1 = p1[0];
    if constexpr (LN == 4) {
      const float v0 = fmaf(mult, z0, xr[i].x), v1 = fmaf(mult, z1, xr[i].y);
      if (in0) epi.x[row * epi.ld_x + c0] = v0;
      if (in1) epi.x[row * epi.ld_x + c1] = v1;
      if (epi.gain) {
        if (in0) epi.gx[row * epi.ld_gx + c0] = __float2bfloat16_rn(v0 * gn.x);
        if (in1) epi.gx[row * epi.ld_gx + c1] = __float2bfloat16_rn(v1 * gn.y);
        const float sq = warp_sum((in0 ? v0 * v0 : 0.f) + (in1 ? v1 * v1 : 0.f));
        if (lane == 0) epi.sq_out[(int64_t)blockIdx.y * epi.sq_out_ld + row] = sq;
      }
    } else if constexpr (LN == 5) {
      const float gate = fminf(fmaf(z0, mult, fb.x), epi.pair_limit);
      const float up = fminf(fmaxf(fmaf(z1, mult, fb.y), -epi.pair_limit), epi.pair_limit);
      const int64_t c = n0 / 2 + lane;
      if (c < epi.pair_cols) epi.out[row * epi.ld_out + c] = from_float<OutT>(gate * gemm::sigmoid_fast(epi.pair_alpha * gate) * (up + 1.0f));
    } else {
      float f[2] = {z0 * mult + fb.x, z1 * mult + fb.y};
      gemm::activate_chunk(f, (int)c0, epi.act_lo, epi.act_hi, epi.act_split, epi.act_param);
      OutT* out = epi.out + row * epi.ld_out;
      if (in0) out[c0] = from_float<OutT>(f[0]);
      if (in1) out[c1] = from_float<OutT>(f[1]);
    }
  }
}

template <typename OutT, int LN, int MG>
int launch_groups(const b200_linear_args& p, const gemm::EpilogueArgs<OutT>& epi, int splits, cudaStream_t stream) {
  constexpr int tile = 8 * MG * kPitch * 4;
  static_assert((kWarps + 1) * tile <= 48 * 1024, "no opt-in needed");
  LaunchSetup ls(dim3((unsigned)splits, (unsigned)((p.N + kCols - 1) / kCols)), dim3(32 * kWarps), (size_t)(kWarps + (splits > 1 ? 1 : 0)) * tile, stream, splits, true);
  const cudaError_t e = cudaLaunchKernelEx(&ls.cfg, linear_few_kernel<OutT, LN, MG>, static_cast<const __nv_bfloat16*>(p.a),
                                           static_cast<const __nv_bfloat16*>(p.b), epi, (int)p.M, p.N, (int)p.K, p.lda, p.ldb);
  note_launches(1);
  return status_from_cuda(e);
}

// Blocks per cluster: doubled while all blocks find room at once, one per SM, or two per SM as long as each keeps 512 of K.  us at one
// row, N x K: 2048 x 2048 4.6 with 4 x 32 blocks, 4.7 with 8 x 32 (16 rows: 5.5 and 6.9: with the SMs full the next kernel's blocks
// cannot start ahead); 2048 x 8192 11.2 with 4 x 32, 8.6 with 8 x 32; 8192 x 2048 10.2 with 128, 8.4 with 2 x 128.
int few_splits(int64_t N, int64_t K) {
  const int64_t slices = (N + kCols - 1) / kCols;
  int s = 1;
  while (s < kMaxSplit && K >= (int64_t)kStep * kWarps * s * 2 &&
         (slices * s * 2 <= sm_count() || (slices * s * 2 <= 2 * (int64_t)sm_count() && K >= 512 * (int64_t)s * 2)))
    s *= 2;
  return s;
}

}  // namespace

// Where this kernel is the better one, up to 16 rows at once: which one it is depends on N and K alone, so that a row's result does not
// depend on how many of them there are (gemm_few_kernel sums in another order).  From 9 rows on the sums take twice the MMAs and twice
// the shared memory.  us, gemm_few_kernel -> this, N x K, 1 to 8 | 9 to 16 rows:
//   act(z)  1024 x 512 3.1 -> 3.2 | 3.1 -> 3.9, 1024 x 1024 4.1 -> 3.3 | 4.1 -> 3.9, 1552 x 1024 4.7 -> 3.4 | 4.7 -> 4.2, 3088 x 1024 5.1 -> 4.3 | 5.1 ->
//           5.2, 4096 x 1024 4.7 -> 4.6 | 4.6 -> 5.7, 2048 x 2048 6.0 -> 4.6 | 6.0 -> 5.4, 8192 x 2048 10.9 -> 9.2 | 10.9 -> 10.3
//   pairs   5504 x 1024 5.4 -> 4.9 | 5.4 -> 5.9, 4096 x 2048 8.3 -> 5.8 | 8.4 -> 6.4, 8192 x 2048 10.0 -> 9.1 | 10.0 -> 10.0, 9408 x 2048 10.5 -> 10.1 |
//           10.4 -> 11.1
// Beyond one slice per SM gemm_few_kernel streams as fast (10880 x 2048 11.6 against 12.2 us at one row), except for LN == 4, whose tiles it
// cuts to 16 columns (22 against 13).
bool linear_few_takes(const b200_linear_args& p, int ln) {
  if (p.M < 1 || p.M > 16 || p.K < 512 || p.K % 8 || p.op_dtype != B200_BF16) return false;
  const int64_t slices = (p.N + kCols - 1) / kCols, sms = sm_count();
  if (slices > 65535) return false;
  if (ln == 4) return true;
  if (p.K < 2048) return p.K >= 1024 && 3 * slices <= sms;
  return 8 * slices <= (ln == 5 ? 7 : 8) * sms;
}

template <typename OutT, int LN>
int launch_linear_few(const b200_linear_args& p, const gemm::EpilogueArgs<OutT>& epi, cudaStream_t stream) {
  const int splits = few_splits(p.N, p.K);
  return p.M <= 8 ? launch_groups<OutT, LN, 1>(p, epi, splits, stream) : launch_groups<OutT, LN, 2>(p, epi, splits, stream);
}
template int launch_linear_few<float, 3>(const b200_linear_args&, const gemm::EpilogueArgs<float>&, cudaStream_t);
template int launch_linear_few<__nv_bfloat16, 3>(const b200_linear_args&, const gemm::EpilogueArgs<__nv_bfloat16>&, cudaStream_t);
template int launch_linear_few<float, 4>(const b200_linear_args&, const gemm::EpilogueArgs<float>&, cudaStream_t);
template int launch_linear_few<__nv_bfloat16, 5>(const b200_linear_args&, const gemm::EpilogueArgs<__nv_bfloat16>&, cudaStream_t);

}  // namespace b200
