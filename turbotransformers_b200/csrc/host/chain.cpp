#include "chain.h"

#include "../ttb_chain_rules.cuh"

#include <algorithm>
#include <cmath>
#include <initializer_list>

namespace turbo_transformers {
namespace layers {

using core::Check;
using core::DeviceContext;
using core::Tensor;

namespace {

constexpr int64_t kHead = 64;

bool Aligned(std::initializer_list<const Tensor*> ts) {
  uintptr_t x = 0;
  for (const Tensor* t : ts) x |= reinterpret_cast<uintptr_t>(t->raw());
  return (x & 15) == 0;
}
bool Half(const Tensor& t, const Tensor& like) {
  return t.on_gpu() && core::SameType(t.dtype(), core::kFloat16) && t.device_id() == like.device_id();
}
bool Vector(const Tensor& t, int64_t n, const Tensor& like) { return Half(t, like) && t.numel() == n; }

int64_t Ctas(const Tensor& x) { return ttb_ctx_sm_count(DeviceContext(x.device_id())); }
// A [K, N] product with a bias over rows like `x`.
bool LinearFits(const PackedLinear& l, bool trans, int64_t K, int64_t N, const Tensor& x) {
  return !l.use_int8() && Half(l.weight(), x) && l.weight().n_dim() == 2 && l.in_dim(trans) == K && l.out_dim(trans) == N && N % 8 == 0 &&
         N <= ttb::chain::bias_columns(Ctas(x)) &&
         Vector(l.bias(), N, x) && Aligned({&l.bias()});
}
bool NormFits(const Tensor& gamma, const Tensor& beta, int64_t H, const Tensor& x) {
  return Vector(gamma, H, x) && Vector(beta, H, x) && Aligned({&gamma, &beta});
}
// (How many keys those rows may have: history_fits and memory_fits of ttb_chain_rules.cuh.)
// The rows up to which one kernel is the faster route: above 32 the rows are eight tiles for the kernel, and every CTA's reading of all of them outweighs
// the launches saved. us, one kernel / layer by layer. GPT-2 small, a step with 30 cached tokens: 1 row 171 / 398, 16 234 / 414, 24 303 / 420,
// 32 339 / 417, 40 539 / 422, 64 601 / 448; BERT-base, tokens: 1 161 / 426, 16 218 / 425, 24 288 / 421, 32 310 / 425, 33 490 / 423; BERT-large 16 474 / 875,
// 24 676 / 878, 32 764 / 874. Layers with context attention are more launches, and Python, for the same products: a step of six layers, 45
// source tokens, 1 row 215 / 592, 32 234 / 623, 64 381 / 621.
// From 25 rows on, stacks of four layers and more: 12 layers 303 / 395, four 108 / 143. What shorter ones would gain is a few launches, and their
// layer-by-layer pass gives bit for bit the results of its layers called one by one.
constexpr int64_t kMostRows = 24, kMostRowsDeep = 32, kDeep = 4, kMostRowsContext = TTB_CHAIN_MAX_ROWS;
int64_t MostRows(int64_t layers) { return layers >= kDeep ? kMostRowsDeep : kMostRows; }
bool RowsFit(const Tensor& x, int64_t heads, int64_t inner, int64_t most) {
  if (x.n_dim() != 3 || !x.on_gpu() || !core::SameType(x.dtype(), core::kFloat16)) return false;
  const int64_t rows = x.numel() ? x.rows() : 0, H = x.shape(2);
  // (narrower models keep the layer-by-layer pass, whose results are bit for bit those of its layers called one by one)
  return rows > 0 && H == heads * kHead && H >= 512 && Aligned({&x}) && rows <= std::min(most, ttb_chain_rows(H, inner)) &&
         ttb::chain::rows_have_writers(rows, Ctas(x));
}

// The call's scratch memory: what operations hand on to others, every result in a place of its own in the order in which they write them.
struct Flow {
  Tensor buffer{nullptr};
  int64_t bytes = 0, at = 0;
  char* base = nullptr;
  static int64_t Size(int64_t rows, int64_t columns) { return (rows * columns * 2 + 255) / 256 * 256; }
  void Allocate(int64_t n, int dev) {
    bytes = n;
    base = reinterpret_cast<char*>(buffer.Reshape(core::kInt8, {n}, kDLCUDA, dev, "chain/flow"));
  }
  void* Next(int64_t rows, int64_t columns) {
    TT_ENFORCE(at + Size(rows, columns) <= bytes, "chain: the flow is too short");
    void* p = base + at;
    at += Size(rows, columns);
    return p;
  }
};

struct Ops {
  std::vector<ttb_chain_op> list;
  int M;
  ttb_chain_linear* Linear(const void* A, int64_t K, const void* W, const void* bias, int64_t N, void* out, int act = TTB_CHAIN_ACT_NONE,
                           const void* residual = nullptr) {
    list.emplace_back();
    ttb_chain_linear& o = list.back().u.linear;
    list.back().kind = TTB_CHAIN_LINEAR;
    o = ttb_chain_linear{};
    o.A = A; o.W = W; o.bias = bias; o.residual = residual; o.out = out;
    o.M = M; o.N = (int32_t)N; o.K = (int32_t)K; o.lda = (int32_t)K; o.ldr = (int32_t)N; o.ldo = (int32_t)N; o.act = act;
    return &o;
  }
  void Norm(ttb_chain_linear* o, const Tensor& gamma, const Tensor& beta, float eps, void* normed = nullptr) {
    o->gamma = gamma.raw(); o->beta = beta.raw(); o->eps = eps; o->normed = normed;
  }
  ttb_chain_attention* Attention(int keys, const void* q, int64_t ldq, int64_t heads, int64_t length, void* out) {
    list.emplace_back();
    ttb_chain_attention& o = list.back().u.attention;
    list.back().kind = TTB_CHAIN_ATTENTION;
    o = ttb_chain_attention{};
    o.keys = keys; o.q = q; o.ldq = (int32_t)ldq; o.out = out; o.ldo = (int32_t)(heads * kHead); o.rows = M; o.heads = (int32_t)heads;
    o.length = (int32_t)length; o.scale = 1.0f / std::sqrt((float)kHead);
    return &o;
  }
};

}  // namespace

bool Chain::EncoderTakes(const BertAttention& attention, const BertIntermediate& intermediate, const Tensor& x, int64_t layers) {
  return !x.is_null() && RowsFit(x, attention.num_attention_heads_, intermediate.dense_.out_dim(false), MostRows(layers));
}

bool Chain::DecoderTakes(const MultiHeadedAttention& attention, const PositionwiseFeedForward& ffn, bool trans_f, const Tensor& x, int64_t past, int64_t memory_keys,
                         int64_t layers) {
  const bool context = memory_keys > 0;
  const int64_t heads = attention.num_attention_heads_;
  if (x.is_null() || !RowsFit(x, heads, ffn.dense1_.out_dim(trans_f), context ? kMostRowsContext : MostRows(layers))) return false;
  if (((past > 0 || context) && x.shape(1) != 1) || past > (1 << 24)) return false;
  if (context) return ttb::chain::memory_fits(x.rows(), heads, Ctas(x), memory_keys, past);
  return past == 0 || ttb::chain::history_fits(x.rows(), heads, Ctas(x), past);
}

bool Chain::Encoder(const std::vector<EncoderBlock>& blocks, const Tensor& x, const Tensor& mask, Tensor* out) {
  if (blocks.empty() || 5 * blocks.size() + 1 > TTB_CHAIN_MAX_OPS || !EncoderTakes(*blocks[0].attention, *blocks[0].intermediate, x, (int64_t)blocks.size())) return false;
  const int64_t heads = blocks[0].attention->num_attention_heads_;
  const int64_t F = blocks[0].intermediate->dense_.out_dim(false);
  const int64_t B = x.shape(0), L = x.shape(1), H = x.shape(2), M = B * L;
  const float* mask_ptr = nullptr;
  if (!mask.is_null()) {  // one row of L keys per sequence; everything else is the general path's business
    if (!mask.on_gpu() || mask.device_id() != x.device_id() || !core::SameType(mask.dtype(), core::kFloat32) || mask.n_dim() < 2 || mask.n_dim() > 4 ||
        mask.shape(-1) != L || mask.numel() != B * L || mask.shape(0) != B)
      return false;
    mask_ptr = mask.data<float>();
  }
  for (const EncoderBlock& b : blocks) {
    const MultiHeadedAttention& a = *b.attention;
    if (a.num_attention_heads_ != heads || a.causal_ || a.qkv_.weight().is_null() || !LinearFits(a.qkv_, false, H, 3 * H, x) ||
        !LinearFits(a.dense_, false, H, H, x) || !NormFits(a.layernorm_gamma_, a.layernorm_beta_, H, x) ||
        !LinearFits(b.intermediate->dense_, false, H, F, x) || !LinearFits(b.output->dense_, false, F, H, x) ||
        !NormFits(b.output->layer_norm_weight_, b.output->layer_norm_bias_, H, x))
      return false;
  }
  const int dev = x.device_id();
  ttb_ctx* c = DeviceContext(dev);
  Flow f;
  f.Allocate((int64_t)blocks.size() * (Flow::Size(M, 3 * H) + 5 * Flow::Size(M, H) + Flow::Size(M, F)), dev);
  out->Reshape(x.dtype(), {B, L, H}, kDLCUDA, dev, "chain/out");
  Ops ops;
  ops.M = (int)M;
  ops.list.reserve(5 * blocks.size() + 1);
  const EncoderBlock* before = nullptr;
  const void *in = x.raw(), *residual = x.raw();  // what the block before has added up, and the layer norm of that: this block's residual
  for (const EncoderBlock& b : blocks) {
    const MultiHeadedAttention& a = *b.attention;
    void* normed = before ? f.Next(M, H) : nullptr;
    void* qkv = f.Next(M, 3 * H);
    ttb_chain_linear* o = ops.Linear(in, H, a.qkv_.Packed(false), a.qkv_.bias().raw(), 3 * H, qkv);
    if (before) {
      ops.Norm(o, before->output->layer_norm_weight_, before->output->layer_norm_bias_, 1e-12f, normed);
      residual = normed;
    }
    void* context = f.Next(M, H);
    ttb_chain_attention* at = ops.Attention(TTB_CHAIN_KEYS_ROWS, qkv, 3 * H, heads, L, context);
    at->mask = mask_ptr;
    at->mask_pitch = (int32_t)L;
    void* sum = f.Next(M, H);
    ops.Linear(context, H, a.dense_.Packed(false), a.dense_.bias().raw(), H, sum, TTB_CHAIN_ACT_NONE, residual);
    normed = f.Next(M, H);
    void* inter = f.Next(M, F);
    o = ops.Linear(sum, H, b.intermediate->dense_.Packed(false), b.intermediate->dense_.bias().raw(), F, inter, TTB_CHAIN_ACT_GELU);
    ops.Norm(o, a.layernorm_gamma_, a.layernorm_beta_, 1e-12f, normed);
    void* next = f.Next(M, H);
    ops.Linear(inter, F, b.output->dense_.Packed(false), b.output->dense_.bias().raw(), H, next, TTB_CHAIN_ACT_NONE, normed);
    in = next;
    before = &b;
  }
  ops.Norm(ops.Linear(in, H, nullptr, nullptr, 0, nullptr), before->output->layer_norm_weight_, before->output->layer_norm_bias_, 1e-12f, out->raw_mut());
  Check(ttb_chain_forward_flow(c, TTB_F16, ops.list.data(), (int)ops.list.size(), f.base, f.at), c, "encoder chain");
  return true;
}

bool Chain::Decoder(const std::vector<DecoderBlock>& blocks, const Tensor& x, bool trans_a, bool trans_f, const LayerNorm* final, const class Linear* head,
                    const Tensor* memory, const Tensor* memory_mask, Tensor* hidden, Tensor* logits, Tensor* attn) {
  const bool context = !blocks.empty() && blocks[0].context;
  if (blocks.empty() || x.n_dim() != 3 || (context ? 8 : 5) * blocks.size() + 1 > TTB_CHAIN_MAX_OPS) return false;
  const int64_t heads = blocks[0].attention->num_attention_heads_;
  const int64_t F = blocks[0].ffn->dense1_.out_dim(trans_f);
  const int64_t B = x.shape(0), L = x.shape(1), H = x.shape(2), M = B * L;
  const bool cached = blocks[0].self_keys != nullptr;
  const int64_t past = cached && !blocks[0].self_keys->is_null() ? blocks[0].self_keys->shape(0) : 0;
  int64_t Lk = 0;
  if (context) {
    const Tensor* k = blocks[0].memory_keys;
    if (!k || !memory_mask || !attn) return false;
    Lk = !k->is_null() && k->n_dim() == 4 ? k->shape(2) : (memory && memory->n_dim() == 3 ? memory->shape(1) : 0);
    if (Lk < 1 || !memory_mask->on_gpu() || memory_mask->device_id() != x.device_id() || !core::SameType(memory_mask->dtype(), core::kFloat32) ||
        memory_mask->shape(-1) != Lk || memory_mask->numel() != B * Lk)
      return false;
  }
  if (!DecoderTakes(*blocks[0].attention, *blocks[0].ffn, trans_f, x, past, Lk, (int64_t)blocks.size())) return false;
  for (const DecoderBlock& b : blocks) {
    const MultiHeadedAttention& a = *b.attention;
    const PositionwiseFeedForward& f = *b.ffn;
    if (a.num_attention_heads_ != heads || a.qkv_.weight().is_null() || !LinearFits(a.qkv_, trans_a, H, 3 * H, x) || !LinearFits(a.dense_, trans_a, H, H, x) ||
        !NormFits(a.layernorm_gamma_, a.layernorm_beta_, H, x) || a.causal_ != blocks[0].attention->causal_ || !LinearFits(f.dense1_, trans_f, H, F, x) ||
        !LinearFits(f.dense2_, trans_f, F, H, x) || !NormFits(f.layer_norm_weight_, f.layer_norm_bias_, H, x) || (b.context != nullptr) != context)
      return false;
    if ((b.self_keys != nullptr) != cached || (b.self_values != nullptr) != cached) return false;
    if (cached) {  // every block has cached the same tokens of this batch
      for (const Tensor* t : {b.self_keys, b.self_values}) {
        if (t->is_null() ? past != 0 : (past == 0 || t->n_dim() != 3 || t->shape(0) != past || t->shape(1) != B || t->shape(2) != H || !Half(*t, x) || !Aligned({t})))
          return false;
      }
    }
    if (context) {
      const MultiHeadedAttention& m = *b.context;
      if (m.num_attention_heads_ != heads || m.q_.weight().is_null() || m.k_.weight().is_null() || m.v_.weight().is_null() || !LinearFits(m.q_, trans_a, H, H, x) ||
          !LinearFits(m.dense_, trans_a, H, H, x) || !NormFits(m.layernorm_gamma_, m.layernorm_beta_, H, x) || !b.memory_keys || !b.memory_values)
        return false;
      const bool filled = !b.memory_keys->is_null() && !b.memory_values->is_null();
      if (filled) {
        for (const Tensor* t : {b.memory_keys, b.memory_values})
          if (!Half(*t, x) || !Aligned({t}) || t->n_dim() != 4 || t->shape(0) != B || t->shape(1) != heads || t->shape(2) != Lk || t->shape(3) != kHead) return false;
      } else if (!memory || memory->n_dim() != 3 || memory->shape(0) != B || memory->shape(1) != Lk || memory->shape(2) != H || !Half(*memory, x) ||
                 m.k_.use_int8() || m.v_.use_int8() || !Half(m.k_.weight(), x) || !Half(m.v_.weight(), x) || m.k_.in_dim(trans_a) != H || m.v_.in_dim(trans_a) != H ||
                 m.k_.out_dim(trans_a) != H || m.v_.out_dim(trans_a) != H || m.k_.bias().is_null() || m.v_.bias().is_null()) {
        return false;
      }
    }
  }
  if (final && !NormFits(final->gamma_, final->beta_, H, x)) return false;
  int64_t V = 0;
  if (head) {
    const PackedLinear& l = head->dense_;
    if (!final || !logits || l.use_int8() || !Half(l.weight(), x) || l.in_dim(head->is_trans_) != H || !l.bias().is_null()) return false;
    V = l.out_dim(head->is_trans_);
    if (V < 1 || V > (1 << 24)) return false;
  }
  const int dev = x.device_id();
  ttb_ctx* c = DeviceContext(dev);
  for (const DecoderBlock& b : blocks)
    if (context && (b.memory_keys->is_null() || b.memory_values->is_null())) b.context->ProjectMemory(*memory, *memory, b.memory_keys, b.memory_values, trans_a);
  Flow f;
  f.Allocate((int64_t)blocks.size() * (Flow::Size(M, 3 * H) + (context ? 6 : 3) * Flow::Size(M, H) + Flow::Size(M, F)), dev);
  Tensor scores(nullptr);
  hidden->Reshape(x.dtype(), {B, L, H}, kDLCUDA, dev, "chain/hidden");
  if (head) logits->Reshape(x.dtype(), {B, L, V}, kDLCUDA, dev, "chain/logits");
  if (context) {
    attn->Reshape(x.dtype(), {B, 1, Lk}, kDLCUDA, dev, "chain/attention");
    scores.Reshape<float>({M, Lk}, kDLCUDA, dev, "chain/scores");
  }
  Ops ops;
  ops.M = (int)M;
  ops.list.reserve(8 * blocks.size() + 1);
  const void* in = x.raw();  // the residual stream: the caller's tensor until the first block has added to it
  auto add = [&](const void* A, int64_t K, const PackedLinear& l, bool trans) {
    void* sum = f.Next(M, H);
    ops.Linear(A, K, l.Packed(trans), l.bias().raw(), H, sum, TTB_CHAIN_ACT_NONE, in);
    in = sum;
  };
  for (const DecoderBlock& b : blocks) {
    const MultiHeadedAttention& a = *b.attention;
    const PositionwiseFeedForward& ffn = *b.ffn;
    const bool last = &b == &blocks.back();
    void *qkv = f.Next(M, 3 * H), *ctx = f.Next(M, H);
    ops.Norm(ops.Linear(in, H, a.qkv_.Packed(trans_a), a.qkv_.bias().raw(), 3 * H, qkv), a.layernorm_gamma_, a.layernorm_beta_, a.pre_ln_eps_);
    ttb_chain_attention* at = ops.Attention(past > 0 ? TTB_CHAIN_KEYS_CACHE : TTB_CHAIN_KEYS_ROWS, qkv, 3 * H, heads, L, ctx);
    at->past = (int32_t)past;
    at->causal = a.causal_ ? 1 : 0;
    if (cached) {
      EnsureCacheRows(b.self_keys, x.dtype(), past, L, B, H, dev);
      EnsureCacheRows(b.self_values, x.dtype(), past, L, B, H, dev);
      at->k_cache = b.self_keys->raw_mut();
      at->v_cache = b.self_values->raw_mut();
    }
    add(ctx, H, a.dense_, trans_a);
    if (context) {
      const MultiHeadedAttention& m = *b.context;
      void* q = f.Next(M, H);
      ctx = f.Next(M, H);
      ops.Norm(ops.Linear(in, H, m.q_.Packed(trans_a), m.q_.bias().raw(), H, q), m.layernorm_gamma_, m.layernorm_beta_, m.pre_ln_eps_);
      at = ops.Attention(TTB_CHAIN_KEYS_MEMORY, q, H, heads, Lk, ctx);
      at->k = b.memory_keys->raw();
      at->v = b.memory_values->raw();
      at->mask = memory_mask->data<float>();
      at->mask_pitch = (int32_t)Lk;
      if (last) {
        at->probs = attn->raw_mut();
        at->scores = scores.mutableData<float>();
      }
      add(ctx, H, m.dense_, trans_a);
    }
    const int act = ffn.act_ == TTB_ACT_GELU ? TTB_CHAIN_ACT_GELU : TTB_CHAIN_ACT_RELU;
    void* inter = f.Next(M, F);
    ops.Norm(ops.Linear(in, H, ffn.dense1_.Packed(trans_f), ffn.dense1_.bias().raw(), F, inter, act), ffn.layer_norm_weight_, ffn.layer_norm_bias_, ffn.eps_);
    if (last && !final) ops.Linear(inter, F, ffn.dense2_.Packed(trans_f), ffn.dense2_.bias().raw(), H, hidden->raw_mut(), TTB_CHAIN_ACT_NONE, in);
    else add(inter, F, ffn.dense2_, trans_f);
  }
  if (final) {
    ttb_chain_linear* o = ops.Linear(in, H, head ? head->dense_.Packed(head->is_trans_) : nullptr, nullptr, V, head ? logits->raw_mut() : nullptr);
    ops.Norm(o, final->gamma_, final->beta_, final->eps_, hidden->raw_mut());
  }
  Check(ttb_chain_forward_flow(c, TTB_F16, ops.list.data(), (int)ops.list.size(), f.base, f.at), c, "decoder chain");
  return true;
}

}  // namespace layers
}  // namespace turbo_transformers
