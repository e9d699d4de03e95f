// Whole passes as one host call each (include/b200_passes.h).  Every pass is written once and runs in two modes: with an arena that only
// counts, which gives the workspace size, and with the caller's workspace, which makes the calls.
#include "../../include/b200_passes.h"

#include <math.h>
#include <string.h>

#include <algorithm>
#include <vector>

namespace {

// Bump allocator over the workspace; without memory it counts.
struct Arena {
  uint8_t* base;
  int64_t capacity, used, peak;
  bool full;

  Arena(void* p, int64_t bytes) : base(static_cast<uint8_t*>(p)), capacity(bytes), used(0), peak(0), full(false) {}
  bool counting() const { return base == nullptr; }
  template <typename T = void>
  T* take(int64_t bytes) {
    const int64_t at = used;
    used += (bytes + 255) & ~(int64_t)255;
    peak = std::max(peak, used);
    if (!counting() && used > capacity) {
      full = true;
      return nullptr;
    }
    return reinterpret_cast<T*>(counting() ? reinterpret_cast<uint8_t*>(256) : base + at);  // (never dereferenced while counting)
  }
};

// Gives back what a scope took.
struct Scope {
  Arena& arena;
  int64_t mark;
  explicit Scope(Arena& a) : arena(a), mark(a.used) {}
  ~Scope() { arena.used = mark; }
};

#define B200_RUN(call)                            \
  do {                                            \
    if (arena.full) return B200_ERR_WORKSPACE;    \
    if (!arena.counting()) {                      \
      const int status_ = (call);                 \
      if (status_ != B200_OK) return status_;     \
    }                                             \
  } while (0)

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// ------------------------------------------------------------------ FusedGPT
int gpt_pass(const b200_gpt_pass_args& p, Arena& arena, void* stream) {
  const int64_t T = p.B * p.L, H = p.H, D = H / p.heads;
  const int es = p.dtype == B200_F32 ? 4 : 2;
  const int op = p.dtype == B200_BF16 ? B200_BF16 : B200_F16;
  const float scale = (float)(1.0 / sqrt((double)D));
  const int64_t in_strides[3] = {p.L * 3 * H, D, 3 * H}, out_strides[3] = {p.L * H, D, H};
  // Float32 storage: every product takes fp16 operands; with more than 128 rows they leave their producers as such (except in a decode
  // step, whose attention leaves float32 rows), else a pass converts them in front of the product.
  const bool f32 = p.dtype == B200_F32;
  auto attention_operands = [&](const b200_gpt_block& b) { return f32 && T > 128 && !p.pos_dev && aligned16(b.qkv_bias); };
  auto mlp_operands = [&](const b200_gpt_block& b) { return f32 && T > 128 && aligned16(b.up_bias); };
  int attention_es = f32 ? 2 : es, mlp_es = attention_es;  // of the widest rows of any block between its products
  for (int64_t i = 0; f32 && i < p.n_blocks; ++i) {
    if (!attention_operands(p.blocks[i])) attention_es = 4;
    if (!mlp_operands(p.blocks[i])) mlp_es = 4;
  }
  // No more than the operators hold at a time.  The stream: x in front of a block's attention, x2 behind it.  x is the caller's out (the
  // last product does not read it), and between attention and the end of the block, while x2 is the stream, it holds the normed rows.
  void* x = p.out && aligned16(p.out) ? p.out : arena.take(T * H * es);
  void* x2 = arena.take(T * H * es);
  const int64_t qkv_bytes = (T * 3 * H * es + 255) & ~(int64_t)255;
  void* wide = arena.take(std::max(qkv_bytes + T * H * attention_es, T * 4 * H * mlp_es));  // q | k | v and rows, later the feed-forward's middle
  void* rows = static_cast<uint8_t*>(wide) + qkv_bytes;                                     // attention's output, normed rows in front of it

  auto attend = [&](const b200_gpt_block& b, int out_dtype) -> int {
    if (p.pos_dev) {
      B200_RUN(b200_attention_decode(wide, b.kv, rows, p.B, p.heads, D, p.cache_len, scale, p.dtype, p.pos_dev, p.status_word, stream));
      return B200_OK;
    }
    if (b.kv) B200_RUN(b200_kv_cache_fill(wide, b.kv, p.B, p.L, H, p.cache_len, p.dtype, stream));
    const uint8_t* q = static_cast<const uint8_t*>(wide);
    B200_RUN(b200_attention(q, q + H * es, q + 2 * H * es, rows, p.B, p.heads, p.L, D, in_strides, in_strides, in_strides, out_strides, scale, p.dtype, out_dtype,
                            p.status_word, stream));
    return B200_OK;
  };

  if (p.folded) {
    float* stats = arena.take<float>(T * 8);
    void* ext = arena.take(T * B200_LN_EXT_COLS * es);
    const size_t need = b200_gemm_ln_workspace_bytes(T, H);
    void* ws = arena.take((int64_t)need);
    // raw rows -> product with their LayerNorm folded in; rows -> product + bias + residual that leaves the result's row statistics
    auto consume = [&](const void* a, const void* w, int64_t ld, const void* w_ext, void* out, int64_t N, int gelu) {
      return b200_gemm_ln(a, w, nullptr, nullptr, out, T, N, H, H, ld, N, N, p.dtype, p.dtype, gelu, stats, ext, w_ext, nullptr, nullptr, p.eps, nullptr, 0,
                          p.status_word, stream);
    };
    auto produce = [&](const void* a, const void* w, int64_t ld, const void* bias, const void* residual, void* out, int64_t K) {
      return b200_gemm_ln(a, w, bias, residual, out, T, H, K, K, ld, H, H, p.dtype, p.dtype, 0, nullptr, nullptr, nullptr, stats, ext, p.eps, ws, need,
                          p.status_word, stream);
    };
    if (p.pos_dev) B200_RUN(b200_embedding_at(p.ids, p.wte, p.wpe, x, p.B, p.L, p.V, p.P, H, p.dtype, nullptr, p.eps, stats, ext, p.pos_dev, stream));
    else B200_RUN(b200_embedding_ln_stats(p.ids, p.wte, p.wpe, x, p.B, p.L, p.V, p.P, H, p.dtype, nullptr, p.eps, stats, ext, stream));
    for (int64_t i = 0; i < p.n_blocks; ++i) {
      const b200_gpt_block& b = p.blocks[i];
      B200_RUN(consume(x, b.qkv, b.ld_qkv, b.qkv_ext, wide, 3 * H, 0));
      const int st = attend(b, p.dtype);
      if (st != B200_OK) return st;
      B200_RUN(produce(rows, b.proj, b.ld_proj, b.proj_bias, x, x2, H));
      B200_RUN(consume(x2, b.up, b.ld_up, b.up_ext, wide, 4 * H, 1));
      if (i + 1 < p.n_blocks) {
        B200_RUN(produce(wide, b.down, b.ld_down, b.down_bias, x2, x, 4 * H));
      } else {
        B200_RUN(b200_gemm(wide, b.down, b.down_bias, x2, p.out, T, H, 4 * H, 4 * H, b.ld_down, H, H, op, p.dtype, 0, p.status_word, stream));
      }
    }
    return B200_OK;
  }

  // Operator by operator.
  void* packed = f32 && (attention_es == 4 || mlp_es == 4) ? arena.take(T * (mlp_es == 4 ? 4 : 1) * H * 2) : nullptr;
  auto product = [&](const void* a, bool is_operand, const void* w, int64_t ld, const void* bias, const void* residual, void* out, int64_t N, int64_t K,
                     int gelu) -> int {
    if (f32 && !is_operand) {
      const int st = b200_pack_operand(a, packed, T, K, K, K, 0, B200_F32, B200_F16, stream);
      if (st != B200_OK) return st;
      a = packed;
    }
    return b200_gemm(a, w, bias, residual, out, T, N, K, K, ld, N, N, op, p.dtype, gelu, p.status_word, stream);
  };
  if (p.pos_dev) B200_RUN(b200_embedding_at(p.ids, p.wte, p.wpe, x, p.B, p.L, p.V, p.P, H, p.dtype, nullptr, p.eps, nullptr, nullptr, p.pos_dev, stream));
  else B200_RUN(b200_embedding(p.ids, p.wte, p.wpe, x, p.B, p.L, p.V, p.P, H, p.dtype, nullptr, stream));
  for (int64_t i = 0; i < p.n_blocks; ++i) {
    const b200_gpt_block& b = p.blocks[i];
    bool operands = attention_operands(b);
    B200_RUN(b200_layernorm(x, b.ln1_w, b.ln1_b, rows, T, H, p.eps, p.dtype, operands ? B200_F16 : p.dtype, stream));
    B200_RUN(product(rows, operands, b.qkv, b.ld_qkv, b.qkv_bias, nullptr, wide, 3 * H, H, 0));
    const int st = attend(b, operands ? B200_F16 : p.dtype);
    if (st != B200_OK) return st;
    B200_RUN(product(rows, operands, b.proj, b.ld_proj, b.proj_bias, x, x2, H, H, 0));
    operands = mlp_operands(b);
    B200_RUN(b200_layernorm(x2, b.ln2_w, b.ln2_b, x, T, H, p.eps, p.dtype, operands ? B200_F16 : p.dtype, stream));
    if (operands) {
      B200_RUN(b200_gemm_operand(x, b.up, static_cast<const float*>(b.up_bias), wide, T, 4 * H, H, H, b.ld_up, 4 * H, 1, p.status_word, stream));
    } else {
      B200_RUN(product(x, false, b.up, b.ld_up, b.up_bias, nullptr, wide, 4 * H, H, 1));
    }
    B200_RUN(product(wide, operands, b.down, b.ld_down, b.down_bias, x2, i + 1 < p.n_blocks ? x : p.out, H, 4 * H, 0));
  }
  return B200_OK;
}

// ------------------------------------------------------------------ decoders with an fp32 residual stream
int64_t pitch(int64_t cols) { return (cols + 31) / 32 * 32; }  // 64 bytes of bf16: what wide stores and tensor maps want

// Rows as a product reads them: a matrix and, behind a deferred norm, the sums of squares of its rows' slices.
struct Rows {
  const void* data;
  int64_t ld, cols;
  const float* sumsq;
  int64_t slices, norm_cols;
  float eps;
};
struct Latents {
  const void* data;
  int64_t hist;
};

struct Decoder {
  const b200_decoder_pass_args& p;
  Arena& arena;
  void* stream;
  int64_t T;
  std::vector<Latents> latents;

  Decoder(const b200_decoder_pass_args& args, Arena& a, void* s) : p(args), arena(a), stream(s), T(args.B * args.n), latents((size_t)args.n_subs) {}

  void* matrix(int64_t rows, int64_t cols) { return arena.take(rows * pitch(cols) * 2); }
  void* mem(void* const* table, int64_t i) const { return table ? table[i] : nullptr; }
  Rows plain(const void* data, int64_t ld, int64_t cols) const { return {data, ld, cols, nullptr, 0, 0, 0.f}; }

  b200_linear_args args(const Rows& in, int64_t rows, const void* w, int64_t N, int64_t ldw) const {
    b200_linear_args q;
    memset(&q, 0, sizeof(q));
    q.a = in.data, q.b = w, q.M = rows, q.N = N, q.K = in.cols, q.lda = in.ld, q.ldb = ldw;
    q.op_dtype = B200_BF16, q.out_dtype = B200_BF16, q.out_scale = 1.f, q.act_split = N, q.status_word = p.status_word;
    if (in.sumsq)
      q.row_sumsq = in.sumsq, q.row_sumsq_slices = (int)in.slices, q.row_sumsq_cols = in.norm_cols, q.row_sumsq_ld = rows, q.eps = in.eps;
    return q;
  }
  int linear(const Rows& in, int64_t rows, const void* w, int64_t N, int64_t ldw, void* out, int act, int64_t split, int act_after, const float* bias) {
    b200_linear_args q = args(in, rows, w, N, ldw);
    q.out = out, q.ld_out = pitch(N), q.act_lo = act, q.act_hi = act_after, q.act_split = split, q.bias = bias;
    B200_RUN(b200_linear(&q, stream));
    return B200_OK;
  }
  // x += product; the next norm's rows into gx and sumsq
  int residual(const Rows& in, const b200_sublayer& s, float* x, void* gx, int64_t ld_gx, float* sumsq) {
    b200_linear_args q = args(in, T, s.w_out, p.W, s.ld_out);
    q.out_dtype = B200_F32, q.act_split = 0;
    q.x = x, q.ld_x = p.W, q.gain = s.gain, q.gx = gx, q.ld_gx = ld_gx, q.sumsq_out = sumsq, q.sumsq_out_ld = T;
    B200_RUN(b200_linear(&q, stream));
    return B200_OK;
  }

  // The mixer or the inner half of a feed-forward: rows -> what the output product reads.
  int inner(int64_t i, const Rows& in, Rows& y) {
    const b200_sublayer& s = p.subs[i];
    int st = B200_OK;
    if (s.kind == B200_SUB_DENSE || s.kind == B200_SUB_GATED) {
      void* mid = matrix(T, s.ff);
      y = plain(mid, pitch(s.ff), s.ff);
      if (s.kind == B200_SUB_DENSE) return linear(in, T, s.w_in, s.n_in, s.ld_in, mid, s.act, s.n_in, 0, nullptr);
      b200_linear_args q = args(in, T, s.w_in, s.n_in, s.ld_in);
      q.out = mid, q.ld_out = pitch(s.ff), q.bias = s.bias_in, q.pair_cols = s.ff, q.pair_limit = s.limit, q.pair_alpha = s.alpha;
      B200_RUN(b200_linear(&q, stream));
      return B200_OK;
    }
    void* z = matrix(T, s.n_in);
    const int64_t ldz = pitch(s.n_in), hv = s.heads * s.vdim;
    auto column = [&](int64_t c) { return static_cast<const uint8_t*>(z) + c * 2; };
    if (s.kind == B200_SUB_LIGHTNING) st = linear(in, T, s.w_in, s.n_in, s.ld_in, z, B200_ACT_SILU, s.off[3], B200_ACT_SIGMOID, nullptr);
    else if (s.kind == B200_SUB_DIFFERENTIAL) st = linear(in, T, s.w_in, s.n_in, s.ld_in, z, 0, s.off[3], B200_ACT_SIGMOID, nullptr);
    else if (s.kind == B200_SUB_DELTA) st = linear(in, T, s.w_in, s.n_in, s.ld_in, z, 0, s.off[5], B200_ACT_SILU, nullptr);
    else st = linear(in, T, s.w_in, s.n_in, s.ld_in, z, 0, s.n_in, 0, nullptr);
    if (st != B200_OK) return st;
    void* out = matrix(T, hv);
    y = plain(out, pitch(hv), hv);
    const bool fresh = !p.pos_dev && p.start == 0;
    void* state = mem(p.mem0, i);

    if (s.kind == B200_SUB_LIGHTNING) {
      if (!state) state = arena.take(p.B * s.heads * s.dim * s.vdim * 4);
      const int64_t slices = b200_decayed_attention_slices(p.n, s.heads, s.dim, s.vdim, B200_BF16);
      float* sumsq = arena.take<float>(slices * T * 4);
      const size_t need = b200_decayed_attention_workspace_bytes(p.B, p.n, s.heads, s.dim, s.vdim, B200_BF16);
      void* ws = need ? arena.take((int64_t)need) : nullptr;
      B200_RUN(b200_decayed_attention(z, ldz, s.off[1], s.off[2], s.off[3], s.decay, s.norm, static_cast<float*>(state), fresh, out, pitch(hv), sumsq, T, p.B, p.n,
                                      s.heads, s.dim, s.vdim, B200_BF16, ws, need, p.status_word, stream));
      y.sumsq = sumsq, y.slices = slices, y.norm_cols = hv, y.eps = s.eps;
      return B200_OK;
    }
    if (s.kind == B200_SUB_LATENT) {
      const int64_t R = s.rank;
      void* cache = mem(p.mem0, s.source);
      const int64_t ring = p.ring ? p.ring[s.source] : 0;
      if (p.pos_dev) {
        if (s.source == i)
          B200_RUN(b200_latent_append(column(s.off[1]), ldz, s.norm, s.eps, nullptr, cache, p.B, 1, R, 0, ring, 0, p.pos_dev, B200_BF16, stream));
        const int64_t window = std::min(s.window, ring);
        const size_t need = b200_latent_decode_workspace_bytes(p.B, s.heads, R, window, B200_BF16);
        void* ws = arena.take((int64_t)need);
        B200_RUN(b200_latent_decode(z, ldz, s.w_uk, s.w_uv, cache, out, pitch(hv), p.B, s.heads, s.dim, s.vdim, R, ring, window, s.scale, s.sink, B200_BF16,
                                    p.pos_dev, ws, need, stream));
        return B200_OK;
      }
      if (s.source == i) {
        void* work = const_cast<void*>(latents[(size_t)i].data);
        const int64_t hist = latents[(size_t)i].hist;
        if (hist) B200_RUN(b200_latent_gather(cache, work, p.B, p.n, R, hist, ring, p.start, B200_BF16, stream));
        B200_RUN(b200_latent_append(column(s.off[1]), ldz, s.norm, s.eps, work, cache, p.B, p.n, R, hist, ring, p.start, nullptr, B200_BF16, stream));
      }
      const Latents& c = latents[(size_t)s.source];
      const int64_t m = p.B * (c.hist + p.n), ldk = pitch(s.n_mid);
      void* kv = matrix(m, s.n_mid);
      st = linear(plain(c.data, R, R), m, s.w_mid, s.n_mid, s.ld_mid, kv, 0, s.n_mid, 0, nullptr);
      if (st != B200_OK) return st;
      B200_RUN(b200_window_attention(z, ldz, kv, ldk, static_cast<uint8_t*>(kv) + s.off_mid * 2, ldk, out, pitch(hv), p.B, p.n, c.hist, s.heads, s.dim, s.vdim,
                                     s.window, s.scale, s.sink, B200_BF16, p.status_word, stream));
      return B200_OK;
    }
    if (s.kind == B200_SUB_DIFFERENTIAL) {
      const int64_t kc = s.kv_heads * 2 * s.dim, vc = s.kv_heads * s.vdim, ring = p.ring ? p.ring[i] : 0;
      const int64_t hist = p.pos_dev ? 0 : std::min(p.start, s.window - 1), m = hist + p.n;
      b200_rotary_args r;
      memset(&r, 0, sizeof(r));
      r.rows = z, r.ld = ldz, r.off_k = s.off[1], r.off_v = s.off[2], r.q_weight = s.norm, r.k_weight = s.norm2, r.freq = s.freq, r.rot_dims = s.rot_dims;
      r.B = p.B, r.n = p.n, r.q_heads = 2 * s.heads, r.kv_heads = s.kv_heads, r.maps = 2, r.dim = s.dim, r.vdim = s.vdim, r.hist = hist;
      r.start = p.pos_dev ? 0 : p.start, r.eps = s.eps, r.dtype = B200_BF16, r.pos_dev = p.pos_dev, r.v_rows_dtype = s.v_dtype;
      r.k_cache = state, r.v_cache = mem(p.mem1, i), r.ring = state ? ring : 0;
      b200_pair_attention_args a;
      memset(&a, 0, sizeof(a));
      a.q = z, a.ld_q = ldz, a.gate = column(s.off[3]), a.ld_gate = ldz, a.lambda = s.lambda_, a.out = out, a.ld_out = pitch(hv);
      a.B = p.B, a.n = p.n, a.heads = s.heads, a.kv_heads = s.kv_heads, a.dim = s.dim, a.vdim = s.vdim;
      a.scale = s.scale, a.softcap = s.softcap, a.eps = s.eps, a.out_scale = s.out_scale, a.dtype = B200_BF16, a.status_word = p.status_word;
      if (p.pos_dev) {
        a.k = r.k_cache, a.v = r.v_cache, a.v_dtype = B200_BF16, a.ring = ring, a.window = std::min(s.window, ring), a.pos_dev = p.pos_dev;
        a.k_row = 2 * s.dim, a.v_row = s.vdim, a.k_head = ring * a.k_row, a.v_head = ring * a.v_row, a.k_batch = s.kv_heads * a.k_head, a.v_batch = s.kv_heads * a.v_head;
      } else {
        r.k_rows = matrix(p.B * m, kc), r.ld_k = pitch(kc), r.v_rows = matrix(p.B * m, vc), r.ld_v = pitch(vc);
        a.k = r.k_rows, a.v = r.v_rows, a.v_dtype = s.v_dtype, a.hist = hist, a.window = std::min(s.window, m);
        a.k_row = r.ld_k, a.v_row = r.ld_v, a.k_batch = m * a.k_row, a.k_head = 2 * s.dim, a.v_batch = m * a.v_row, a.v_head = s.vdim;
      }
      B200_RUN(b200_rotary_append(&r, stream));
      a.workspace_bytes = b200_pair_attention_workspace_bytes(&a);
      a.workspace = a.workspace_bytes ? arena.take(a.workspace_bytes) : nullptr;
      B200_RUN(b200_pair_attention(&a, stream));
      return B200_OK;
    }
    if (s.kind != B200_SUB_DELTA) return B200_ERR_BAD_ARGUMENT;
    b200_delta_args d;
    memset(&d, 0, sizeof(d));
    d.rows = z, d.ld = ldz, d.off_k = s.off[1], d.off_v = s.off[2], d.off_a = s.off[3], d.off_b = s.off[4], d.off_g = s.off[5];
    d.conv_w = s.conv_w, d.conv_state = mem(p.mem1, i), d.conv_cols = s.conv_cols, d.taps = s.taps;
    d.mixed = matrix(T, s.conv_cols), d.ld_mixed = pitch(s.conv_cols);
    d.norms = arena.take<float>(2 * s.kv_heads * T * 4), d.gates = arena.take<float>(2 * s.heads * T * 4);
    d.a_log = s.a_log, d.dt_bias = s.dt_bias, d.norm_w = s.norm, d.y = out, d.ld_y = pitch(hv), d.pos_dev = p.pos_dev;
    d.state = static_cast<float*>(state ? state : arena.take(p.B * s.heads * s.dim * s.vdim * 4));
    d.B = p.B, d.n = p.n, d.start = p.pos_dev ? 0 : p.start, d.heads = s.heads, d.kv_heads = s.kv_heads, d.dim = s.dim, d.vdim = s.vdim;
    d.eps = s.eps, d.unit_eps = s.unit_eps, d.q_scale = s.q_scale, d.fresh = fresh, d.dtype = B200_BF16, d.status_word = p.status_word;
    d.workspace_bytes = b200_delta_workspace_bytes(&d);
    d.workspace = d.workspace_bytes ? arena.take(d.workspace_bytes) : nullptr;
    B200_RUN(b200_delta(&d, stream));
    return B200_OK;
  }

  int run() {
    float* x = arena.take<float>(T * p.W * 4);
    // latents that several sublayers of this pass read
    if (!p.pos_dev) {
      for (int64_t i = 0; i < p.n_subs; ++i) {
        const b200_sublayer& s = p.subs[i];
        if (s.kind != B200_SUB_LATENT || s.source != i) continue;
        const int64_t hist = std::min(p.start, s.reach - 1);
        latents[(size_t)i] = {arena.take(p.B * (hist + p.n) * s.rank * 2), hist};
      }
    }
    return p.both_norms ? run_both(x) : run_front(x);
  }

  int run_front(float* x) {
    const int64_t slice = b200_linear_slice_cols(T, B200_BF16), slices = (p.W + slice - 1) / slice;
    void* gx[2] = {matrix(T, p.W), matrix(T, p.W)};
    float* sq[2] = {arena.take<float>(slices * T * 4), arena.take<float>(slices * T * 4)};
    B200_RUN(b200_embedding_rms(p.ids, p.table, p.first_gain, x, gx[0], sq[0], T, p.V, p.W, pitch(p.W), B200_BF16, stream));
    Rows rows{gx[0], pitch(p.W), p.W, sq[0], 1, p.W, p.eps};
    for (int64_t i = 0; i < p.n_subs; ++i) {
      const Scope scope(arena);
      Rows y;
      int st = inner(i, rows, y);
      if (st != B200_OK) return st;
      const bool last = i + 1 == p.n_subs;
      void* g = last ? p.out : gx[(i + 1) & 1];
      float* q = last ? p.sumsq_out : sq[(i + 1) & 1];
      st = residual(y, p.subs[i], x, g, last ? p.ld_out : pitch(p.W), q);
      if (st != B200_OK) return st;
      rows = Rows{g, last ? p.ld_out : pitch(p.W), p.W, q, slices, p.W, p.eps};
    }
    return B200_OK;
  }

  int run_both(float* x) {
    void* h = matrix(T, p.W);
    void* y = matrix(T, p.W);
    b200_stream_args u;
    auto update = [&](int64_t i) {  // in front of sublayer i (n_subs: the final norm)
      memset(&u, 0, sizeof(u));
      const b200_sublayer* s = i < p.n_subs ? &p.subs[i] : nullptr;
      u.x = x, u.T = T, u.W = p.W, u.table_scale = p.table_scale, u.eps = p.eps, u.keep = i > 0, u.dtype = B200_BF16;
      if (i > 0) u.y = y, u.ld_y = pitch(p.W), u.y_gain = p.subs[i - 1].behind;
      if (i == 0 || (s && s->add_embedding)) u.ids = p.ids, u.table = p.table, u.V = p.V;
      u.shift = s ? s->shift : nullptr;
      u.gain = s ? s->gain : p.final_gain;
      u.h = s ? h : p.out, u.ld_h = s ? pitch(p.W) : p.ld_out;
      return b200_stream_update(&u, stream);
    };
    for (int64_t i = 0; i < p.n_subs; ++i) {
      const Scope scope(arena);
      const b200_sublayer& s = p.subs[i];
      B200_RUN(update(i));
      Rows z;
      int st = inner(i, plain(h, pitch(p.W), p.W), z);
      if (st == B200_OK) st = linear(z, T, s.w_out, p.W, s.ld_out, y, 0, p.W, 0, s.bias_out);
      if (st != B200_OK) return st;
    }
    B200_RUN(update(p.n_subs));
    return B200_OK;
  }
};

bool gpt_args_ok(const b200_gpt_pass_args* p) {
  return p && p->blocks && p->n_blocks >= 1 && p->heads >= 1 && p->B >= 1 && p->L >= 1 && p->H >= 8 && p->H % 8 == 0 && p->H % p->heads == 0 &&
         (!p->pos_dev || p->L == 1) && (!p->folded || p->dtype != B200_F32) && p->B * p->L <= 0x7fffffffLL;
}
bool decoder_args_ok(const b200_decoder_pass_args* p) {
  if (!p || !p->subs || p->n_subs < 1 || p->B < 1 || p->n < 1 || p->start < 0 || p->W < 1 || (p->pos_dev && p->n != 1) || p->B * p->n > 0x7fffffffLL) return false;
  for (int64_t i = 0; i < p->n_subs; ++i) {
    const b200_sublayer& s = p->subs[i];
    if (s.kind < B200_SUB_LIGHTNING || s.kind > B200_SUB_GATED) return false;
    if (s.k_out != (s.kind == B200_SUB_DENSE || s.kind == B200_SUB_GATED ? s.ff : s.heads * s.vdim)) return false;  // what w_out reads
    if (s.kind == B200_SUB_LATENT && (s.source < 0 || s.source > i || p->subs[s.source].kind != B200_SUB_LATENT || p->subs[s.source].source != s.source)) return false;
  }
  return true;
}

}  // namespace

extern "C" {

int b200_passes_version(void) { return B200_PASSES_VERSION; }
void b200_passes_struct_bytes(int64_t sizes[4]) {
  sizes[0] = sizeof(b200_gpt_block), sizes[1] = sizeof(b200_gpt_pass_args), sizes[2] = sizeof(b200_sublayer), sizes[3] = sizeof(b200_decoder_pass_args);
}

int64_t b200_gpt_pass_workspace_bytes(const b200_gpt_pass_args* args) {
  if (!gpt_args_ok(args)) return 0;
  Arena arena(nullptr, 0);
  gpt_pass(*args, arena, nullptr);
  return arena.peak;
}

int b200_gpt_pass(const b200_gpt_pass_args* args, void* stream) {
  if (!gpt_args_ok(args) || !args->ids || !args->wte || !args->wpe || !args->out) return B200_ERR_BAD_ARGUMENT;
  for (int64_t i = 0; args->pos_dev && i < args->n_blocks; ++i)
    if (!args->blocks[i].kv) return B200_ERR_BAD_ARGUMENT;
  if (!args->workspace || (reinterpret_cast<uintptr_t>(args->workspace) & 255)) return B200_ERR_WORKSPACE;
  Arena arena(args->workspace, args->workspace_bytes);
  return gpt_pass(*args, arena, stream);
}

int64_t b200_decoder_pass_workspace_bytes(const b200_decoder_pass_args* args) {
  if (!decoder_args_ok(args)) return 0;
  Arena arena(nullptr, 0);
  Decoder(*args, arena, nullptr).run();
  return arena.peak;
}

int b200_decoder_pass(const b200_decoder_pass_args* args, void* stream) {
  if (!decoder_args_ok(args) || !args->ids || !args->table || !args->out || (!args->both_norms && !args->sumsq_out)) return B200_ERR_BAD_ARGUMENT;
  if (!args->workspace || (reinterpret_cast<uintptr_t>(args->workspace) & 255)) return B200_ERR_WORKSPACE;
  Arena arena(args->workspace, args->workspace_bytes);
  return Decoder(*args, arena, stream).run();
}

}  // extern "C"
