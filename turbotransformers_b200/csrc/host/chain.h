// Stacks of layers over few rows as one kernel (ttb_chain_forward_flow): which calls take that route, and their list of operations.
#pragma once
#include <utility>
#include <vector>

#include "layers.h"

namespace turbo_transformers {
namespace layers {

// Every function returns false, having done nothing, for a call that the route does not take: anything but fp16, many rows,
// a width below 512, heads of other than 64, int8 weights, shapes and alignments that the kernel refuses. The caller then runs the
// layers one by one, with the same results up to the order of sums.
class Chain {
 public:
  struct DecoderBlock {
    const MultiHeadedAttention* attention;
    const MultiHeadedAttention* context;  // or null
    const PositionwiseFeedForward* ffn;
    core::Tensor *self_keys, *self_values;      // the block's layer_cache entries, or null (no cache)
    core::Tensor *memory_keys, *memory_values;  // with `context`; filled by this call when empty
  };
  struct EncoderBlock {
    const BertAttention* attention;
    const BertIntermediate* intermediate;
    const BertOutput* output;
  };
  // Whether a call on x could take the route, by what costs nothing to look at: type, width, rows, layers and keys (`past` cached tokens;
  // memory_keys of context attention, 0 without). The two calls below check the rest.
  static bool EncoderTakes(const BertAttention& attention, const BertIntermediate& intermediate, const core::Tensor& x, int64_t layers);
  static bool DecoderTakes(const MultiHeadedAttention& attention, const PositionwiseFeedForward& ffn, bool is_trans_weight_ffn, const core::Tensor& x, int64_t past,
                           int64_t memory_keys, int64_t layers);
  // Post-LN encoder layers: x [B, L, H] -> out. mask: null tensor, or additive fp32 with one row per sequence.
  static bool Encoder(const std::vector<EncoderBlock>& blocks, const core::Tensor& x, const core::Tensor& mask, core::Tensor* out);
  // Pre-LN decoder blocks: x [B, L, H] -> hidden. Without cached tokens any L (causal where the attention says so), with them L = 1. final
  // (a layer norm) and head (then hidden is its input) may be null. memory [B, Lk, H] (read, and not null, only where a block's memory entries are empty), memory_mask fp32 [B, 1, Lk] and attn [B, 1, Lk]
  // (the last block's context attention of head 0) belong to blocks with context attention.
  static bool Decoder(const std::vector<DecoderBlock>& blocks, const core::Tensor& x, bool is_trans_weight_attention, bool is_trans_weight_ffn,
                      const LayerNorm* final, const Linear* head, const core::Tensor* memory, const core::Tensor* memory_mask, core::Tensor* hidden,
                      core::Tensor* logits, core::Tensor* attn);
};

}  // namespace layers
}  // namespace turbo_transformers
