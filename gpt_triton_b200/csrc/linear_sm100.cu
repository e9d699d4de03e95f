// 16-bit instantiations of the tcgen05 GEMM behind b200_linear: products over rows whose RMS norm is deferred to the
// epilogue (gemm_sm100.cuh, LN == 3 and 4), and the gated pairs of a feed-forward (LN == 5).
#include "gemm_sm100.cuh"

namespace b200 {

// linear_few.cu: at most 16 rows, cut along K
bool linear_few_takes(const b200_linear_args& p, int ln);
template <typename OutT, int LN>
int launch_linear_few(const b200_linear_args& p, const gemm::EpilogueArgs<OutT>& epi, cudaStream_t stream);

namespace {

template <typename OutT, int LN>
int launch(const b200_linear_args& p, const gemm::EpilogueArgs<OutT>& epi, cudaStream_t stream) {
  const gemm::LnArgs none;
  if constexpr (!std::is_same<OutT, __half>::value) {
    if (linear_few_takes(p, LN)) return launch_linear_few<OutT, LN>(p, epi, stream);
  }
  // LN == 4 promises its sums of squares per 64 columns up to kNarrowMaxRows rows, which the wide kernel does not leave; LN == 5 needs an
  // output that a tensor map takes there, and beyond those rows everywhere.
  const bool mapped = LN != 5 || ((reinterpret_cast<uintptr_t>(p.out) & 15) == 0 && p.ld_out % 8 == 0);
  const bool small = LN == 4 ? gemm::narrow_is_faster(p.M, p.N, LN) : gemm::takes_few_rows(p.M, p.N, LN) || gemm::narrow_is_faster(p.M, p.N, LN);
  if (p.M <= gemm::kNarrowMaxRows ? small || LN == 4 || !mapped : small && mapped)
    return gemm::launch_narrow<OutT, false, LN>(p.a, p.b, epi, p.M, p.N, p.K, p.lda, p.ldb, p.op_dtype, none, p.status_word, stream);
  return gemm::launch_wide<OutT, false, 0, LN>(p.a, p.b, epi, p.M, p.N, p.K, p.lda, p.ldb, p.op_dtype, none, p.status_word, stream);
}

template <typename OutT, int LN>
int fill_and_launch(const b200_linear_args& p, cudaStream_t stream) {
  gemm::EpilogueArgs<OutT> e;
  memset(&e, 0, sizeof(e));
  e.out = static_cast<OutT*>(p.out), e.ld_out = p.ld_out;
  e.sq_in = p.row_sumsq, e.sq_in_ld = p.row_sumsq_ld, e.sq_slices = p.row_sumsq_slices, e.sq_cols = (float)p.row_sumsq_cols;
  e.eps = p.eps, e.out_scale = p.out_scale;
  e.act_lo = p.act_lo, e.act_hi = p.act_hi, e.act_split = p.act_split;
  e.act_param = p.act_param, e.fbias = p.bias;
  e.pair_cols = p.pair_cols, e.pair_limit = p.pair_limit, e.pair_alpha = p.pair_alpha;
  e.x = p.x, e.ld_x = p.ld_x, e.gain = p.gain, e.gx = static_cast<__nv_bfloat16*>(p.gx), e.ld_gx = p.ld_gx;
  e.sq_out = p.sumsq_out, e.sq_out_ld = p.sumsq_out_ld;
  return launch<OutT, LN>(p, e, stream);
}

}  // namespace

// fp16([gelu](A B^T + bias)) from fp16 operands with a float32 bias: a product of a float32 model whose result is only ever an
// operand.  GELU and rounding are those of the float32 epilogue and of pack_kernel behind it: the same bits in one pass.  16 x 300
// tokens, 768 -> 3072 with GELU: 52 us + 13 us of pack_kernel on the next product's side before.
int launch_gemm_operand(const void* a, const void* b, const float* bias, void* out, int64_t M, int64_t N, int64_t K, int64_t lda, int64_t ldb,
                        int64_t ld_out, int add_gelu, int* status_word, cudaStream_t stream) {
  if (((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(bias)) & 15) || lda % 8 || ldb % 8) return B200_ERR_ALIGNMENT;
  b200_linear_args p;
  memset(&p, 0, sizeof(p));
  p.a = a, p.b = b, p.M = M, p.N = N, p.K = K, p.lda = lda, p.ldb = ldb, p.out = out, p.ld_out = ld_out, p.op_dtype = B200_F16, p.out_dtype = B200_F16;
  p.bias = bias, p.out_scale = 1.f, p.status_word = status_word;
  p.act_lo = add_gelu ? B200_ACT_GELU_TANH : 0, p.act_hi = p.act_lo, p.act_split = N;
  return fill_and_launch<__half, 3>(p, stream);
}

int64_t linear_sm100_slice_cols(int64_t M) { return M <= gemm::kNarrowMaxRows ? gemm::NARROW_BN : gemm::EPI_COLS; }

int launch_linear_sm100(const b200_linear_args& p, cudaStream_t stream) {
  if (p.op_dtype != B200_BF16) return B200_ERR_UNSUPPORTED;
  if ((reinterpret_cast<uintptr_t>(p.a) & 15) || (reinterpret_cast<uintptr_t>(p.b) & 15) || p.lda % 8 || p.ldb % 8) return B200_ERR_ALIGNMENT;
  if (reinterpret_cast<uintptr_t>(p.bias) & 15) return B200_ERR_ALIGNMENT;
  if (p.x) return fill_and_launch<float, 4>(p, stream);
  if (p.pair_cols) return p.out_dtype == B200_BF16 ? fill_and_launch<__nv_bfloat16, 5>(p, stream) : B200_ERR_UNSUPPORTED;
  if (p.out_dtype == B200_BF16) return fill_and_launch<__nv_bfloat16, 3>(p, stream);
  if (p.out_dtype == B200_F32) return fill_and_launch<float, 3>(p, stream);
  return B200_ERR_UNSUPPORTED;
}

}  // namespace b200
