/*
 * Whole passes over a model as one host call each: libb200passes.so, a client of the C ABI in b200_gpt.h.  A pass makes the entry
 * point calls that the Python operators make one by one, in the same order and with the same arguments; it saves what those cost on the
 * host (15-30 us each).  No kernel code lives here and nothing is kept between calls.
 */
#ifndef B200_PASSES_H_
#define B200_PASSES_H_

#include "b200_gpt.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Counts changes of the structures below; b200_passes_version gives the library's.  A caller in another language, whose structures repeat
 * these by hand, compares their sizes too: b200_gpt_block, b200_gpt_pass_args, b200_sublayer, b200_decoder_pass_args. */
#define B200_PASSES_VERSION 1
int b200_passes_version(void);
void b200_passes_struct_bytes(int64_t sizes[4]);

/* One block of a FusedGPT.  Operands are [N, ld] K-major 16-bit (b200_pack_operand; qkv and up with the LayerNorm in front folded in:
 * b200_fold_layernorm, whose extension they then have instead of a bias); biases and LayerNorm vectors in the storage type. */
typedef struct {
  const void *ln1_w, *ln1_b, *ln2_w, *ln2_b;
  const void *qkv, *qkv_bias, *qkv_ext, *proj, *proj_bias, *up, *up_bias, *up_ext, *down, *down_bias;
  int64_t ld_qkv, ld_proj, ld_up, ld_down;
  void* kv; /* [B, cache_len, 2 H], or NULL: nothing is remembered */
} b200_gpt_block;

/* ids [B, L] -> the residual stream behind the last block, out [B * L, H].  pos_dev: a decode step (L == 1, every block with kv) at the
 * device-side position pos_dev[0].  H % 8 == 0; folded: 16-bit types only.  The workspace's size follows from the arguments, `out` and the
 * blocks' biases included (a 16-byte aligned `out` holds the stream between blocks). */
typedef struct {
  const b200_gpt_block* blocks;
  const int64_t* ids;
  const void *wte, *wpe;
  const int32_t* pos_dev;
  void* out;
  int64_t n_blocks, heads, B, L, V, P, H, cache_len;
  float eps;
  int dtype, folded;
  void* workspace; /* 256-byte aligned */
  int64_t workspace_bytes;
  int* status_word;
} b200_gpt_pass_args;
int64_t b200_gpt_pass_workspace_bytes(const b200_gpt_pass_args* args);
int b200_gpt_pass(const b200_gpt_pass_args* args, void* stream);

enum { B200_SUB_LIGHTNING = 0, B200_SUB_LATENT = 1, B200_SUB_DENSE = 2, B200_SUB_DIFFERENTIAL = 3, B200_SUB_DELTA = 4, B200_SUB_GATED = 5 };

/* One sublayer of a decoder with an fp32 residual stream, bf16 weights. */
typedef struct {
  int kind, act;
  const void* w_in; /* the products that read the rows in front, stacked: sections from the output columns off[] on */
  int64_t n_in, ld_in, off[6];
  const void* w_out;
  int64_t k_out, ld_out;
  const void *w_mid, *w_uk, *w_uv; /* latent: uk | uv stacked (values from the column off_mid on), and each alone */
  int64_t n_mid, ld_mid, off_mid;
  const double* decay;                                       /* lightning */
  const float *norm, *norm2, *sink, *freq, *lambda_, *conv_w; /* lightning, delta, latent: norm; differential: norm (queries), norm2 (keys) */
  const float *a_log, *dt_bias, *bias_in, *bias_out;
  int64_t heads, kv_heads, dim, vdim, rank, window, reach, rot_dims, taps, conv_cols, ff;
  int64_t source; /* latent: the sublayer whose latents it reads (itself: it owns them) */
  float scale, softcap, eps, out_scale, limit, alpha, q_scale, unit_eps;
  int v_dtype;
  const float *gain, *behind, *shift; /* gain: weights of the norm behind (norm in front only: of the next sublayer's); both norms: in front */
  int add_embedding;                  /* both norms: the embeddings join the stream in front of this sublayer */
} b200_sublayer;

/* ids [B * n] -> rows behind the final norm, out [B * n, W] (pitch ld_out) bf16.  both_norms == 0: rows as b200_linear takes them with
 * sumsq_out [b200_linear_slice_cols slices, B * n]; else normed.  mem0, mem1, ring: the memory of every sublayer (latents | state |
 * keys, values | state, convolution inputs; NULL entries: none), arrays of n_subs, or NULL when nothing is remembered.  pos_dev: a
 * decode step (n == 1); else the first token stands at position start. */
typedef struct {
  const b200_sublayer* subs;
  void* const* mem0;
  void* const* mem1;
  const int64_t* ring;
  const int64_t* ids;
  const void* table;
  const float *first_gain, *final_gain;
  const int32_t* pos_dev;
  void* out;
  float* sumsq_out;
  int64_t n_subs, B, n, start, V, W, ld_out;
  float eps, table_scale;
  int both_norms;
  void* workspace; /* 256-byte aligned */
  int64_t workspace_bytes;
  int* status_word;
} b200_decoder_pass_args;
int64_t b200_decoder_pass_workspace_bytes(const b200_decoder_pass_args* args);
int b200_decoder_pass(const b200_decoder_pass_args* args, void* stream);

#ifdef __cplusplus
}
#endif
#endif /* B200_PASSES_H_ */
