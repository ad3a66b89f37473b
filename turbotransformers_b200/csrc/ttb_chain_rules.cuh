// Rules of the chain kernel (ttb_chain.cu) that do not depend on its data: who computes and writes what on a grid of any size. Host code
// as well, so that they can be checked without a GPU.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define TTB_CHAIN_FN __host__ __device__ __forceinline__
#else
#define TTB_CHAIN_FN inline
#endif

namespace ttb {
namespace chain {

constexpr int kBiasUnits = 16;  // units of eight columns whose biases a CTA has room for

// A product's units are dealt out as evenly as they go: CTA `cta` of `ctas` computes units [first_unit(cta), first_unit(cta + 1)). (Of a
// product of 2^24 columns the products below stay under 2^32 on up to 2047 CTAs.)
TTB_CHAIN_FN uint32_t first_unit(uint32_t units, uint32_t cta, uint32_t ctas) { return units * cta / ctas; }

// Every CTA normalises all rows for itself; their copy in memory is written a row by one CTA, so that there have to be as many: the grid is one
// CTA for each SM that the process sees. (Dealt out round the grid instead, 17 tokens of BERT-base took 357 us for 352.)
TTB_CHAIN_FN bool writes_row(int row, int cta) { return row == cta; }
TTB_CHAIN_FN bool rows_have_writers(int64_t rows, int64_t ctas) { return rows <= ctas; }

// The widest product with a bias that a grid takes, in columns (dealt out unevenly, a CTA may have a unit more than another).
TTB_CHAIN_FN int64_t bias_columns(int64_t ctas) { return (kBiasUnits - 1) * 8 * ctas; }

// ---- attention: up to how many keys the chain is the faster route ------------------------------------------------------------
// A (row, head) is one CTA's: where a CTA has `pairs` of them, its eight warps are shared out among them, kWarps / pairs each (a power of two). Layer by
// layer a long history is split over up to sixteen CTAs a head, so that the chain, which wins by the launches it saves, loses again where a
// warp walks far. Both sides were measured up to 4000 keys (fp16, a step of the whole model, us, chain / layer by layer).
constexpr int kWarps = 8;  // of a CTA

TTB_CHAIN_FN int64_t pairs_of_cta(int64_t rows, int64_t heads, int64_t ctas) { return (rows * heads + ctas - 1) / ctas; }

// Tokens in a decoder-only model's cache. Eight warps a pair: GPT-2 small 1 row, 3000 tokens 448 / 511, 4000 542 / 529; 4 rows, 4000 661 / 599; 8 rows, 3000
// 579 / 646, 4000 716 / 697; 8 heads of 64, 18 rows, 2500 498 / 603. Four: 8 heads, 20 rows, 1000 418 / 476, 1600 561 / 540; 12 heads, 16 rows, 1000 469 / 592, 2000 743 / 687; 24 rows, 1000 554 / 635; 16 heads (24
// layers), 10 rows, 1600 1130 / 1298. Two: 12 heads, 32 rows, 300 433 / 550, 600 559 / 617, 1000 730 / 707; 16 heads, 24 rows, 700 1152 / 1321, 32 rows 1355 / 1463.
// (The lines lie where they lay when the chain was slower: a few hundred tokens short of where the two meet now, which differ by a tenth there.)
TTB_CHAIN_FN bool history_fits(int64_t rows, int64_t heads, int64_t ctas, int64_t tokens) {
  const int64_t pairs = pairs_of_cta(rows, heads, ctas);
  if (pairs <= 1) return tokens <= (rows < 8 ? 2400 + 140 * rows : 3500);
  if (pairs == 2) return tokens <= 550 + 80 * heads;
  return pairs <= 4 && tokens <= 640;
}

// Keys of an encoder memory (and tokens in the cache, as many again to walk). Layer by layer the host is the limit, about 600 us for six layers,
// and beyond the 1024 keys of its one-kernel cross attention (ttb_context_attention_step) that pass takes twice as long. Six layers, a pass of six steps with the
// memory's projections, us a step: 8 heads: 64 rows, 200 keys 491 / 616, 400 645 / 657, 700 877 / 900, 1000 1115 / 1180; 48 rows, 700 742 / 789; 32 rows, 1000
// 610 / 804. 16 heads: 32 rows, 400 608 / 723, 1000 1106 / 1211. (The line lies where it lay when the chain was slower: beyond it the two are equal.)
TTB_CHAIN_FN bool memory_fits(int64_t rows, int64_t heads, int64_t ctas, int64_t keys, int64_t tokens) {
  return keys > 1024 || pairs_of_cta(rows, heads, ctas) * (keys + tokens) <= 300 * heads;
}

}  // namespace chain
}  // namespace ttb
